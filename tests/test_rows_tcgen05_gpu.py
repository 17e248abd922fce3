"""The few-rows tcgen05 product (weights as the 128-row operand, K split over a cluster) at the edges of its tiles, steps and splits, and the norm with a warp a row."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    return g, x, w, x.double() @ w.double().T, K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)      # sums, and what K float32 sums may be off by


# 16, 32 and 64 columns of batch rows, full and not; tiles that end inside 128 rows; K of one step, of a ragged last step, of fewer and more steps than a cluster's
# blocks and than the ring's stages; one to eight blocks a tile, and more tiles than multiprocessors
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (9, 136, 72), (16, 1600, 960), (17, 392, 1032), (32, 2048, 8192), (33, 5120, 968), (64, 6144, 2048), (63, 20016, 136),
                                   (64, 128, 512), (40, 960, 2560)])
def test_results_and_sums(M, N, K):
    from vitna_anchor_b200 import ops
    g, x, w, want, off = _operands(M, N, K, M * N + K)
    base = torch.randn(M, N, generator=g, device="cuda")
    room = torch.full((M * N + 1024,), 5.0, device="cuda")          # what lies behind the matrix stays as it is
    out, acc = room[:M * N].view(M, N), base.clone()
    ops.linear_rows_tcgen05(x, w, out, ops.EPI_F32)
    ops.linear_rows_tcgen05(x, w, acc, ops.EPI_ACC)
    same, act = (torch.full((M, N), 5.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ops.linear_rows_tcgen05(x, w, same, ops.EPI_SAME)
    ops.linear_rows_tcgen05(x, w, act, ops.EPI_SAME, act=4)
    ops.check_device_errors()
    assert bool(((out.double() - want).abs() <= off).all())
    assert bool(((acc.double() - want - base.double()).abs() <= off + 2.0 ** -23 * (base.double().abs() + want.abs())).all())
    assert bool(((same.double() - want).abs() <= off + 2.0 ** -8 * (want.abs() + off)).all())
    squared, off2 = want.clamp(min=0.0) ** 2, 2 * want.abs() * off + off * off + 2.0 ** -23 * want * want
    assert bool(((act.double() - squared).abs() <= off2 + 2.0 ** -8 * (squared + off2)).all())
    assert bool((room[M * N:] == 5.0).all())
    # a row's bits hang neither on the number of rows nor on the others
    for lo, n in ((M - 1, 1), (M // 2, M - M // 2)):
        part = torch.empty(n, N, device="cuda")
        ops.linear_rows_tcgen05(x[lo:lo + n], w, part, ops.EPI_F32)
        assert torch.equal(part, out[lo:lo + n])


# one block a tile, two, three, seven and eight; 16, 32 and 64 columns of batch rows
@pytest.mark.parametrize("M,N,K", [(1, 49152, 576), (8, 32000, 1024), (8, 32768, 768), (24, 49152, 960), (16, 8192, 2048), (40, 5120, 960), (64, 16384, 2048), (64, 6144, 2048), (32, 2560, 2560),
                                   (64, 2048, 8192)])
def test_sums_are_as_exact_as_the_kernel_it_stands_in_for(M, N, K):
    """What is cut off of a sum in tensor memory grows with the products added one after another: no more of them than the mma.sync kernel's warps add, or, for many
    columns and more than eight rows, the tile kernel."""
    from vitna_anchor_b200 import ops
    _, x, w, want, _ = _operands(M, N, K, M + N + K)
    out, other = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    ops.linear_rows_tcgen05(x, w, out, ops.EPI_F32)
    if M > 8 and N > 8192:
        ops.linear_tcgen05(x, w, other, ops.LINEAR_F32)
    else:
        ops.linear_skinny(x, w, other, ops.EPI_F32)
    ops.check_device_errors()
    mine, theirs = float((out.double() - want).norm()), float((other.double() - want).norm())
    # both are norms over thousands of sums' rounding errors, which depend on their order: measured within 7 % of each other where the chains are as long
    assert mine <= 1.15 * theirs, (mine / float(want.norm()), theirs / float(want.norm()))


@pytest.mark.parametrize("M,inter,K,kind", [(9, 4, 64, 0), (17, 68, 200, 0), (64, 2560, 960, 0), (33, 1000, 1096, 2), (64, 8192, 256, 0)])
def test_gated(M, inter, K, kind):
    from vitna_anchor_b200 import ops
    _, x, w, want, off = _operands(M, 2 * inter, K, inter + K)
    out = torch.full((M, inter), 5.0, device="cuda", dtype=torch.bfloat16)
    ops.linear_rows_tcgen05(x, w, out, ops.EPI_SWIGLU, act=kind)
    ops.check_device_errors()
    f = torch.nn.functional.silu if kind == 0 else (lambda t: torch.nn.functional.gelu(t, approximate="tanh"))
    a, b, e = want[:, :inter], want[:, inter:], off + 2.0 ** -8 * (want.abs() + off)      # both are rounded to bfloat16 before the gate
    ea, eb = e[:, :inter], e[:, inter:]
    bound = 1.2 * ea * b.abs() + 1.2 * (a.abs() + ea) * eb + 2.0 ** -8 * (f(a) * b).abs()       # the functions' slopes stay below 1.2
    assert bool(((out.double() - f(a) * b).abs() <= 1.01 * bound + 1e-6).all())


@pytest.mark.parametrize("M,nh,nkv,hd,ps,K", [(64, 15, 5, 64, 16, 960), (9, 3, 1, 128, 8, 136), (33, 32, 32, 64, 16, 512), (20, 1, 1, 64, 1, 2056)])
def test_rotation_and_cache(M, nh, nkv, hd, ps, K):
    from vitna_anchor_b200 import ops
    N = (nh + 2 * nkv) * hd
    g, x, w, _, _ = _operands(M, N, K, N + K)
    pos = torch.randint(0, 300, (M,), generator=g, device="cuda", dtype=torch.int32)
    ang = torch.rand(300, hd // 2, generator=g, device="cuda") * 6.28
    cos, sin = torch.cos(ang), torch.sin(ang)
    pages = -(-2 * M // ps)
    slot = torch.randperm(pages * ps, generator=g, device="cuda")[:M].to(torch.int32)
    slot[M // 3] = -1
    got_c, want_c = (torch.full((pages, 2, nkv, ps, hd), 3.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    got_q, want_q = (torch.zeros(M, nh * hd, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ops.linear_rows_tcgen05(x, w, got_q, ops.EPI_ROPE, rope=(pos, cos, sin, slot, got_c, nh, nkv, hd))
    qkv = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    ops.linear_rows_tcgen05(x, w, qkv, ops.EPI_SAME)
    ops.rope_store(qkv, pos, cos, sin, slot, want_q, want_c, nh, nkv, hd, hd, ps)
    ops.check_device_errors()
    # the same rounded sums; the rotation's two products may be contracted differently: an ulp of the larger one, then a rounding to bfloat16
    size = torch.maximum(want_q.float().abs(), want_q.float().view(M, nh, 2, hd // 2).flip(2).reshape(M, -1).abs())
    assert bool(((got_q.float() - want_q.float()).abs() <= 2.0 ** -7 * size + 1e-6).all())
    assert bool(((got_c.float() - want_c.float()).abs() <= 2.0 ** -7 * want_c.float().abs().amax(-1, keepdim=True)).all())
    assert torch.equal(got_c[:, 1], want_c[:, 1])                        # the values as they are


@pytest.mark.parametrize("stage", [0, 5])
def test_gives_up_a_wait_and_says_so(stage):
    from vitna_anchor_b200 import ops
    _, x, w, want, off = _operands(40, 2048, 8192, 3)
    out = torch.zeros(40, 2048, device="cuda")
    ops.set_wait_limit_ms(5.0)
    try:
        ops.skip_stage_once("linear_tcgen05", stage)
        ops.linear_rows_tcgen05(x, w, out, ops.EPI_F32)
        torch.cuda.synchronize()
        with pytest.raises(ops.KernelGaveUp, match=r"code 7[123]\)"):          # a code of no other kernel
            ops.check_device_errors()
    finally:
        ops.set_wait_limit_ms(0)
    ops.linear_rows_tcgen05(x, w, out, ops.EPI_F32)
    ops.check_device_errors()
    assert bool(((out.double() - want).abs() <= off).all())


# a warp a row (`rows` in all and 77 of them) and eight rows a block
@pytest.mark.parametrize("n,rows,warps", [(4, 2048, True), (4, 2500, False), (512, 2048, True), (576, 5000, True), (576, 3000, None), (640, 5001, False), (644, 5000, True), (700, 7001, False),
                                          (1024, 5000, True), (1028, 5000, True), (2048, 5000, True), (2052, 200, False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_rows(n, rows, warps, dtype):
    from vitna_anchor_b200 import ops
    warps = dtype == torch.float32 if warps is None else warps         # (None: it is the result's type that decides)
    assert bool(ops.lib().vk_rmsnorm_warp_blocks(rows, n, 0 if dtype == torch.float32 else 1)) == warps
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(rows, n, generator=g, device="cuda") * 3
    w = torch.randn(n, generator=g, device="cuda")
    picked = torch.randperm(rows, generator=g, device="cuda")[:77].to(torch.int32)
    out, some = torch.empty(rows, n, device="cuda", dtype=dtype), torch.empty(77, n, device="cuda", dtype=dtype)
    ops.rmsnorm_rows(x, w, 1e-5, out)
    ops.rmsnorm_rows(x, w, 1e-5, some, picked)
    assert torch.equal(some, out[picked.long()])                       # the same order of sums in both forms
    want = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) * w.double()
    assert bool(((out.double() - want).abs() <= ((n / 32 + 8) * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)) * want.abs() + 1e-9).all())
