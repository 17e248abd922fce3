"""The tcgen05 products' float32 epilogues where rows do not start on 16 bytes, tiles end inside a warp's 32 x 32 and a block has several tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# narrow tiles of 64 and 128 columns with odd and even row lengths; wide tiles (K >= 2,048, or many tiles) with one tile a block and with several
@pytest.mark.parametrize("shape", [(65, 33, 72), (130, 1746, 576), (97, 2051, 64), (513, 1747, 2048), (2050, 2052, 512), (4100, 1093, 520), (4099, 2304, 512)])
def test_float32_results_and_sums(shape):
    from vitna_anchor_b200 import ops
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    base = torch.randn(M, N, generator=g, device="cuda")
    want = x.double() @ w.double().T
    room = torch.full((M * N + 1024,), 5.0, device="cuda")          # what lies behind the matrix stays as it is
    out = room[:M * N].view(M, N)
    ops.linear_tcgen05(x, w, out, ops.LINEAR_F32)
    acc = base.clone()
    ops.linear_tcgen05(x, w, acc, ops.LINEAR_ACC_F32)
    ops.check_device_errors()
    # K products exact in float32 and K float32 sums, each off by at most 2^-23 of the sum of the terms' sizes
    bound = K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - want).abs() <= bound).all())
    assert bool(((acc.double() - want - base.double()).abs() <= bound + 2.0 ** -23 * (base.double().abs() + want.abs())).all())
    assert bool((room[M * N:] == 5.0).all())
