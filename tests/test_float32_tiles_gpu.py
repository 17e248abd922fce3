"""The true 32-bit path's kernels for many rows give the bits of the kernels for few: every output is one chain of sums in one order."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# one shape for every tile the launch may choose, at the tiles' edges: 16 x 16, 16 x 32, 32 x 32, 64 x 64; a slab of 32, its remainders, one piece
@pytest.mark.parametrize("shape", [(1, 7, 4), (16, 16, 32), (15, 4737, 36), (16, 4800, 64), (17, 3201, 100), (33, 3200, 576), (64, 131, 1536), (1024, 800, 96),
                                   (1025, 833, 132)])
def test_a_product_has_the_same_bits_in_every_tile(shape):
    from vitna_anchor_b200 import ops
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    apart = torch.zeros(M + 1, K + 1, device="cuda")[:M, :K].copy_(x)       # rows that do not start on 16 bytes: the general kernel
    for mode in (ops.LINEAR_SAME, ops.LINEAR_ACC_F32):
        base = torch.randn(M, N, generator=g, device="cuda")
        a, b = base.clone(), base.clone()
        ops.linear_simt(x, w, a, mode, few_rows=0)
        ops.linear_simt(apart, w, b, mode, few_rows=0)
        assert torch.equal(a, b)
        want = x.double() @ w.double().T + (base.double() if mode == ops.LINEAR_ACC_F32 else 0)
        # a chain of K roundings, each at most 2^-24 of a partial sum of at most sum |x w|
        bound = (K + 2) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + base.double().abs())
        assert bool(((a.double() - want).abs() <= bound).all())


# (heads, kv heads, head size, value size, page, window, bias, values in keys, key heads a value, gate)
@pytest.mark.parametrize("form", [(3, 1, 64, 64, 16, 0, False, False, 1, False), (4, 2, 16, 16, 4, 0, True, False, 1, False), (2, 2, 128, 96, 8, 0, False, False, 1, True),
                                  (4, 4, 20, 36, 16, 130, False, False, 2, False), (2, 1, 68, 60, 16, 0, True, True, 1, False), (2, 2, 64, 128, 16, 7, False, False, 1, True),
                                  (1, 1, 4, 4, 1, 300, False, False, 1, False)])
def test_attention_of_portions_has_the_bits_of_attention_token_by_token(form):
    from vitna_anchor_b200 import ops
    nh, nkv, hd, vd, ps, window, bias, v_in_key, v_share, gated = form
    g = torch.Generator(device="cuda").manual_seed(hd * 7 + window)
    segs = [(0, 1 + 64), (127, 2), (300, 130), (5, 33), (63, 64)]            # (position of the first token, tokens): tiles of 1, 2, 33 and 64 rows
    longest = max(p + n for p, n in segs)
    blocks = -(-longest // ps)
    elems = ps * (nkv * hd if v_in_key else nkv * hd + nkv // v_share * vd)
    pages = torch.randn(len(segs) * blocks, elems, generator=g, device="cuda")
    bt = torch.randperm(len(segs) * blocks, generator=g, device="cuda").view(len(segs), blocks).to(torch.int32)
    T = sum(n for _, n in segs)
    pos = torch.cat([torch.arange(p, p + n) for p, n in segs]).to(torch.int32).cuda()
    seg = torch.cat([torch.full((n,), i) for i, (_, n) in enumerate(segs)]).to(torch.int32).cuda()
    tiles, at = [], 0
    for i, (p, n) in enumerate(segs):
        tiles += [(at + o, min(64, n - o), p + o, i) for o in range(0, n, 64)]
        at += n
    tiles = torch.tensor(sorted(tiles, key=lambda t: t[2] + t[1]), dtype=torch.int32, device="cuda")
    q = 2 * torch.randn(T, nh * hd, generator=g, device="cuda")
    table = torch.randn(90, nh, generator=g, device="cuda") if bias else None
    gate = torch.randn(T, nh + 3, generator=g, device="cuda")[:, :nh] if gated else None
    one = torch.zeros(T, nh * vd + 5, device="cuda")
    two = one.clone()
    ops.attention_rows_biased(q, pages, bt, seg, pos, one[:, :nh * vd], nh, nkv, hd, vd, ps, hd ** -0.5, window, table, None, v_in_key, v_share, gate)
    ops.attention_rows_tile(q, pages, bt, tiles, two[:, :nh * vd], nh, nkv, hd, vd, ps, hd ** -0.5, window, table, v_in_key, v_share, gate)
    assert torch.equal(one, two)


def test_a_key_that_is_not_finite_reaches_no_earlier_query():
    from vitna_anchor_b200 import ops
    nh, hd, T = 2, 64, 200
    g = torch.Generator(device="cuda").manual_seed(5)
    pages = torch.randn(1, T * 2 * nh * hd, generator=g, device="cuda")
    pages.view(2, nh, T, hd)[1, :, 150] = float("inf")
    q = torch.randn(T, nh * hd, generator=g, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    tiles = i32([(o, min(64, T - o), o, 0) for o in range(0, T, 64)])
    bt, seg, pos = i32([[0]]), torch.zeros(T, dtype=torch.int32, device="cuda"), torch.arange(T, dtype=torch.int32, device="cuda")
    one, two = (torch.empty(T, nh * hd, device="cuda") for _ in range(2))
    ops.attention_rows_biased(q, pages, bt, seg, pos, one, nh, nh, hd, hd, T, hd ** -0.5)
    ops.attention_rows_tile(q, pages, bt, tiles, two, nh, nh, hd, hd, T, hd ** -0.5)
    assert bool(torch.isfinite(two[:150]).all()) and np.array_equal(one.cpu().numpy(), two.cpu().numpy(), equal_nan=True)
