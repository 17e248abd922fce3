"""The tcgen05 prompt attention for keys and values of 64 and 128 values against the general kernel, which takes every query by itself: tiles of all sizes up to 128 rows, the
diagonal inside a step, windows that begin inside and at a step's edge, pages on either side of a step's length, rows that lie apart, gates."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(128, 128), (64, 128), (128, 64)])
@pytest.mark.parametrize("form", [(4, 2, 16, 0, False), (3, 1, 8, 100, False), (2, 2, 32, 64, True), (2, 1, 64, 1, False), (6, 3, 128, 65, True), (1, 1, 16, 1000, False)])
def test_dims_against_the_general_kernel(dims, form):
    from vitna_anchor_b200 import ops
    hd, vd = dims
    nh, nkv, ps, window, gated = form
    g = torch.Generator(device="cuda").manual_seed(hd + vd + window)
    segs = [(0, 257), (127, 2), (300, 130), (5, 60), (63, 65), (1000, 128)]       # (position of the first token, tokens)
    longest = max(p + n for p, n in segs)
    blocks = -(-longest // ps)
    pages = torch.randn(len(segs) * blocks, ps * nkv * (hd + vd), generator=g, device="cuda").to(torch.bfloat16)
    bt = torch.randperm(len(segs) * blocks, generator=g, device="cuda").view(len(segs), blocks).to(torch.int32)
    T = sum(n for _, n in segs)
    pos = torch.cat([torch.arange(p, p + n) for p, n in segs]).to(torch.int32).cuda()
    seg = torch.cat([torch.full((n,), i) for i, (_, n) in enumerate(segs)]).to(torch.int32).cuda()
    tiles, at = [], 0
    for i, (p, n) in enumerate(segs):
        tiles += [(at + o, min(128, n - o), p + o, i) for o in range(0, n, 128)]
        at += n
    tiles = torch.tensor(sorted(tiles, key=lambda t: t[2] + t[1]), dtype=torch.int32, device="cuda")
    q = (2 * torch.randn(T, nh * hd, generator=g, device="cuda")).to(torch.bfloat16)
    gate = torch.randn(T, nh + 3, generator=g, device="cuda")[:, :nh] if gated else None
    one = torch.full((T + 1, nh * vd + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    two = one.clone()
    ops.attention_rows_biased(q, pages, bt, seg, pos, one[:T, :nh * vd], nh, nkv, hd, vd, ps, hd ** -0.5, window, None, None, False, 1, gate)
    ops.attention_prefill_tcgen05_dims(q, pages, bt, tiles, two[:T, :nh * vd], nh, nkv, hd, vd, ps, hd ** -0.5, window, gate)
    torch.cuda.synchronize()
    ops.check_device_errors()
    a, b = one.float(), two.float()
    # both are sums of float32 products of the same inputs, the probabilities in two bfloat16 parts (2^-16 of a value); then rounded to bfloat16, once each
    assert bool(((a - b).abs() <= 2.0 ** -7 * a.abs() + 2.0 ** -14 * float(a[:T, :nh * vd].abs().max())).all())
    assert bool((two[T] == 7).all()) and bool((two[:, nh * vd:] == 7).all())
