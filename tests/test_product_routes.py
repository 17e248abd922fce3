"""Which kernel a product goes to, as far as that is decided on the host: no GPU is needed."""
import pytest
import torch

from vitna_anchor_b200 import ops


class _OnDevice(torch.Tensor):
    """A tensor of the host that says it lies on the device, for the checks in front of a launch; no launch may follow."""

    @property
    def is_cuda(self):
        return True


def _device(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16).as_subclass(_OnDevice)


# few rows (the tcgen05 few-rows product's sizes among them) and many
@pytest.mark.parametrize("M,N,K", [(8, 64, 64), (1, 49152, 576), (40, 2048, 2048), (100, 64, 64)])
def test_rows_on_the_host_are_refused(M, N, K):
    """Operands that lie on the host must not reach a launch, whatever the sizes choose."""
    x, w, out = torch.zeros(M, K, dtype=torch.bfloat16), _device(N, K), torch.zeros(M, N).as_subclass(_OnDevice)
    assert not ops.tcgen05_takes(x, w) and not ops.rows_tcgen05_takes(x, w, out) and not ops.rows_tcgen05_pays(x, w, out)
    with pytest.raises(ops.KernelError):
        ops.linear(x, w, out, ops.LINEAR_F32)
    for kernel in (ops.linear_tcgen05, lambda a, b, o, _: ops.linear_rows_tcgen05(a, b, o, ops.EPI_F32)):
        with pytest.raises(ops.KernelError):
            kernel(x, w, out, ops.LINEAR_F32)
    with pytest.raises(ops.KernelError):
        ops.linear_gated(x, w, torch.zeros(M, N, dtype=torch.bfloat16).as_subclass(_OnDevice), _device(M, N // 2), "silu")
    with pytest.raises(ops.KernelError):
        ops.linear_act(x, w, _device(M, N), "relu2")


def test_weights_that_are_no_matrix_are_refused():
    with pytest.raises(ops.KernelError):
        ops.linear(_device(40, 64), _device(4096), torch.zeros(40, 4096).as_subclass(_OnDevice), ops.LINEAR_F32)
