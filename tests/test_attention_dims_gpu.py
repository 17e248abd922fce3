"""The tcgen05 prompt attention for keys and values of 64 and 128 values against the general kernel, which takes every query by itself: tiles of all sizes up to 128 rows, the
diagonal inside a step, windows that begin inside and at a step's edge, pages on either side of a step's length, rows that lie apart, gates."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(128, 128), (64, 128), (128, 64)])
# (the last four: more than 148 blocks, which come two to a multiprocessor)
@pytest.mark.parametrize("form", [(4, 2, 16, 0, False), (3, 1, 8, 100, False), (2, 2, 32, 64, True), (2, 1, 64, 1, False), (6, 3, 128, 65, True), (1, 1, 16, 1000, False), (32, 4, 16, 0, False), (24, 8, 8, 65, True), (20, 4, 128, 300, False),
                                  (17, 17, 64, 1, True)])
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


@pytest.mark.parametrize("dims", [(128, 128), (64, 128), (128, 64)])
def test_which_kernel_a_portion_takes(dims, monkeypatch):
    """Short portions take the kernel with tiles of 64 rows, longer ones the tcgen05 kernel; both sides of the line give what the general kernel gives."""
    from types import SimpleNamespace
    from vitna_anchor_b200 import ops
    hd, vd = dims
    nh, nkv, ps, line = 4, 2, 16, 128 if hd == 64 else 48
    taken = []
    for name in ("_prefill_tcgen05_dims", "attention_prefill_biased"):
        monkeypatch.setattr(ops, name, lambda *a, _f=getattr(ops, name), _n=name, **k: (taken.append(_n), _f(*a, **k))[1])
    for lens, fast in (((line,), False), ((line + 1,), True), ((line, line), False), ((line + 9, line - 8), True), ((2,), False)):
        g = torch.Generator(device="cuda").manual_seed(sum(lens))
        blocks = -(-max(lens) // ps)
        pages = torch.randn(len(lens) * blocks, ps * nkv * (hd + vd), generator=g, device="cuda").to(torch.bfloat16)
        i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
        bt = torch.arange(len(lens) * blocks, device="cuda").view(len(lens), blocks).to(torch.int32)
        starts = [sum(lens[:i]) for i in range(len(lens))]
        tiles = lambda rows: i32(sorted([(starts[i] + o, min(rows, n - o), o, i) for i, n in enumerate(lens) for o in range(0, n, rows)], key=lambda t: t[2] + t[1]))
        T = sum(lens)
        ctx = SimpleNamespace(num_dec=0, dec_tokens=None, num_pre=T, num_segments=len(lens), pre_tokens=None, pre_tiles=tiles(64), pre_tiles_big=tiles(128),
                              token_seg=i32([i for i, n in enumerate(lens) for _ in range(n)]), positions=i32([j for n in lens for j in range(n)]),
                              max_context=max(lens), workspace=SimpleNamespace(max_context=1024))
        q = torch.randn(T, nh * hd, generator=g, device="cuda").to(torch.bfloat16)
        one, two = (torch.empty(T, nh * vd, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        ops.attention_rows_biased(q, pages, bt, ctx.token_seg, ctx.positions, one, nh, nkv, hd, vd, ps, hd ** -0.5)
        del taken[:]
        ops.attention_biased(q, pages, SimpleNamespace(block_tables=bt), ctx, two, nh, nkv, hd, vd, ps, hd ** -0.5)
        assert taken == ["_prefill_tcgen05_dims" if fast else "attention_prefill_biased"], lens
        a, b = one.float(), two.float()
        # sums of float32 products of the same inputs; the older kernel's probabilities are one bfloat16 (2^-9 of a value), then rounded to bfloat16, once each
        assert bool(((a - b).abs() <= 2.0 ** -7 * a.abs() + 2.0 ** -8 * float(a.abs().max())).all())
