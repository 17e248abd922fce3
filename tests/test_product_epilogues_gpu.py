"""The tcgen05 products' epilogues where rows do not start on 16 bytes, tiles end inside a warp's 32 x 32 and a block has several tiles, and the products of row
groups where row tiles without a group lie between the others."""
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


# wide tiles (1,024 columns and more) and narrow ones; columns that end inside a tile, on a piece of eight and off it; bfloat16 (plain and relu squared) and float32
@pytest.mark.parametrize("mode,act", [(0, 0), (0, 4), (1, 0)])
@pytest.mark.parametrize("N,K,tiles", [(1024, 72, 19), (1064, 520, 16), (1027, 136, 40), (2304, 1056, 37), (1096, 72, 2), (520, 264, 9)])
def test_row_groups(N, K, tiles, mode, act):
    from vitna_anchor_b200 import ops
    E, M = 5, tiles * 128
    g = torch.Generator(device="cuda").manual_seed(N * K + tiles)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(E, N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    group = torch.randint(-1, E, (tiles,), generator=g, device="cuda", dtype=torch.int32)
    group[tiles // 2] = -1
    group[0] = 3
    group[-max(1, tiles // 8):] = -1
    dtype = torch.float32 if mode else torch.bfloat16
    room = torch.full((M * N + 1024,), 5.0, device="cuda", dtype=dtype)
    ops._check(ops.lib().vk_linear_tcgen05_grouped(ops._p(x), ops._p(w), ops._p(room), M, N, K, K, E, ops._p(group), mode, 0, act,
                                                   ops._p(ops.error_word()), ops._stream()), "linear_tcgen05_grouped")
    ops.check_device_errors()
    out = room[:M * N].view(tiles, 128, N)
    for i, e in enumerate(group.tolist()):
        if e < 0:
            assert bool((out[i] == 5.0).all())                       # rows without a group are left alone
            continue
        a, b = x[i * 128:(i + 1) * 128].double(), w[e].double()
        want, off = a @ b.T, K * 2.0 ** -23 * (a.abs() @ b.abs().T)       # (as above)
        if act:
            off = 2 * want.abs() * off + off * off + 2.0 ** -23 * want * want
            want = want.clamp(min=0.0) ** 2
        if mode == 0:
            off = off + 2.0 ** -8 * (want.abs() + off)                 # rounded to bfloat16
        assert bool(((out[i].double() - want).abs() <= off).all())
    assert bool((room[M * N:] == 5.0).all())


def _route(kind, M, N, K):
    """The wide tiles' weight rows, one more with pairs of blocks; 0 for the narrow kernel."""
    from vitna_anchor_b200 import ops
    return ops.lib().vk_linear_tcgen05_route(kind, M, N, K)


# pairs of blocks: row tiles of 256 with an empty half, with rows in both; widths of 160, 192 and 256 whose last tile ends inside a block's half; one round and several
@pytest.mark.parametrize("M,N,K,route", [(2048, 2576, 3000, 161), (1900, 2576, 3000, 161), (2048, 5152, 2048, 193), (2048, 6160, 2048, 257), (3000, 4112, 1800, 257),
                                         (2049, 2048, 8200, 257)])
def test_pairs_of_blocks(M, N, K, route):
    from vitna_anchor_b200 import ops
    assert [_route(kind, M, N, K) for kind in (0, 1, 2)] == [route] * 3
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    want, off = x.double() @ w.double().T, K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)      # (as above)
    f32 = torch.full((M * N + 1024,), 5.0, device="cuda")
    ops.linear_tcgen05(x, w, f32[:M * N].view(M, N), ops.LINEAR_F32)
    assert bool(((f32[:M * N].view(M, N).double() - want).abs() <= off).all()) and bool((f32[M * N:] == 5.0).all())
    base = torch.randn(M, N, generator=g, device="cuda")
    acc = base.clone()
    ops.linear_tcgen05(x, w, acc, ops.LINEAR_ACC_F32)
    assert bool(((acc.double() - want - base.double()).abs() <= off + 2.0 ** -23 * (base.double().abs() + want.abs())).all())
    same = torch.full((M, N), 5.0, device="cuda", dtype=torch.bfloat16)
    ops.linear_tcgen05(x, w, same, ops.LINEAR_SAME)
    ops.check_device_errors()
    assert bool(((same.double() - want).abs() <= off + 2.0 ** -8 * (want.abs() + off)).all())
    # a row's bits do not hang on the number of rows
    part = torch.empty(M - 128, N, device="cuda")
    ops.linear_tcgen05(x[128:], w, part, ops.LINEAR_F32)
    assert torch.equal(part, f32[128 * N:M * N].view(M - 128, N))


@pytest.mark.parametrize("M,inter,K,route", [(2048, 2584, 2048, 193), (2000, 8192, 2048, 257), (1100, 3080, 2048, 257), (8192, 1536, 576, 192)])
def test_gated_pairs_of_blocks(M, inter, K, route):
    from vitna_anchor_b200 import ops
    assert _route(3, M, inter, K) == route
    g = torch.Generator(device="cuda").manual_seed(M + inter + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * inter, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    gated = torch.full((M, inter), 5.0, device="cuda", dtype=torch.bfloat16)
    ops.linear_tcgen05_swiglu(x, w, gated)
    ops.check_device_errors()
    want, off = x.double() @ w.double().T, K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)      # (as above)
    # both halves are rounded to bfloat16 first; silu's slope stays below 1.1, its own error is a few 2^-22
    a, b, e = want[:, :inter], want[:, inter:], off + 2.0 ** -8 * (want.abs() + off)
    ea, eb, f = e[:, :inter], e[:, inter:], torch.nn.functional.silu(a)
    bound = 1.1 * ea * b.abs() + (f.abs() + 1.1 * ea) * eb + (2.0 ** -8 + 2.0 ** -18) * (f * b).abs()
    assert bool(((gated.double() - f * b).abs() <= 1.01 * bound + 1e-6).all())


# rows that do not begin on 16 bytes, written value by value: bfloat16 in narrow tiles up to K = 600 and in wide ones, sums in tiles of 160 and 192 columns, never by pairs
@pytest.mark.parametrize("shape,routes", [((4100, 1093, 520), (0, 160)), ((3000, 1001, 1000), (192, 192)), ((4096, 1178, 4472), (160, 160)), ((2048, 1249, 376), (0, 160)),
                                          ((16384, 142, 112), (0, 0))])
def test_rows_off_16_bytes(shape, routes):
    from vitna_anchor_b200 import ops
    M, N, K = shape
    assert (_route(0, M, N, K), _route(2, M, N, K)) == routes
    test_float32_results_and_sums(shape)
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    same = torch.full((M, N), 5.0, device="cuda", dtype=torch.bfloat16)
    ops.linear_tcgen05(x, w, same, ops.LINEAR_SAME)
    ops.check_device_errors()
    want, off = x.double() @ w.double().T, K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)      # (as above)
    assert bool(((same.double() - want).abs() <= off + 2.0 ** -8 * (want.abs() + off)).all())


# the edge of a round of narrow tiles (296 of 64 rows, 333 go to wide ones; 148 of 128 rows, 152), wide tiles of a short K and of few columns, sums in tiles of 160
# and 192 columns with and without whole rows of 16 bytes
@pytest.mark.parametrize("shape", [(4736, 512, 72), (4700, 520, 72), (4736, 2048, 768), (500, 4736, 768), (1000, 2426, 776), (8190, 576, 64), (8190, 570, 136),
                                   (2999, 2046, 264), (2999, 2052, 128), (20000, 100, 72)])
def test_products_at_the_edge_of_a_round(shape):
    test_float32_results_and_sums(shape)


# the fused turn in wide tiles where the last tile holds one, two and three heads of four (64 columns) and one of two (128)
@pytest.mark.parametrize("nh,nkv,hd,K", [(9, 3, 64, 576), (3, 1, 64, 264), (6, 2, 64, 64), (5, 3, 128, 136)])
def test_turned_heads_at_the_edge_of_a_round(nh, nkv, hd, K, M=8100, route=256):
    from vitna_anchor_b200 import ops
    ps, N = 16, (nh + 2 * nkv) * hd
    assert _route(4 if hd == 64 else 5, M, N, K) == route
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    pos = torch.randint(0, 500, (M,), generator=g, device="cuda", dtype=torch.int32)
    slot = torch.randperm(M + 60, generator=g, device="cuda")[:M].to(torch.int32)
    slot[::7] = -1
    pages = (M + 60 + ps - 1) // ps
    ang = torch.rand(500, hd // 2, generator=g, device="cuda") * 6.0
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    cache = torch.full((pages, 2, nkv, ps, hd), 7.0, device="cuda", dtype=torch.bfloat16)
    q = torch.full((M, nh * hd), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.linear_tcgen05_rope(x, w, q, pos, cos, sin, slot, cache, nh, nkv, hd)
    ops.check_device_errors()
    p, off = x.double() @ w.double().T, K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    p, off = p.view(M, nh + 2 * nkv, hd), (off + 2.0 ** -8 * (p.abs() + off)).view(M, nh + 2 * nkv, hd)      # the projections are rounded to bfloat16 first
    c, s = cos.double()[pos.long()][:, None], sin.double()[pos.long()][:, None]
    t, o = p[:, :nh + nkv], off[:, :nh + nkv]
    a, b, oa, ob = t[..., :hd // 2], t[..., hd // 2:], o[..., :hd // 2], o[..., hd // 2:]
    turned = torch.cat([a * c - b * s, b * c + a * s], -1)
    slack = torch.cat([oa * c.abs() + ob * s.abs(), ob * c.abs() + oa * s.abs()], -1) + 2.0 ** -22 * (torch.cat([a, a], -1).abs() + torch.cat([b, b], -1).abs())
    slack = slack + 2.0 ** -8 * (turned.abs() + slack)                       # rounded to bfloat16
    assert bool(((q.view(M, nh, hd).double() - turned[:, :nh]).abs() <= slack[:, :nh]).all())
    held = torch.full((pages * ps, 2, nkv, hd), 7.0, device="cuda", dtype=torch.float64)
    room = torch.zeros_like(held)
    on = slot >= 0
    held[slot[on].long(), 0], room[slot[on].long(), 0] = turned[on, nh:], slack[on, nh:]
    held[slot[on].long(), 1], room[slot[on].long(), 1] = p[on, nh + nkv:], off[on, nh + nkv:]
    got = cache.permute(0, 3, 1, 2, 4).reshape(pages * ps, 2, nkv, hd).double()
    assert bool(((got - held).abs() <= room).all())


# by pairs of blocks: row tiles with rows in both halves and with an empty one, a last tile of one head of four and of one of two
@pytest.mark.parametrize("nh,nkv,hd,K,M", [(29, 16, 64, 2048, 2100), (17, 2, 128, 4096, 2049)])
def test_turned_heads_by_pairs(nh, nkv, hd, K, M):
    test_turned_heads_at_the_edge_of_a_round(nh, nkv, hd, K, M, 257)


@pytest.mark.parametrize("stage", [0, 7, 90])        # of the first tile and of a later one: the first block's tensor warp, then both blocks' copying and adding-up warps give up
def test_pairs_of_blocks_give_up_a_wait_and_say_so(stage):
    """Neither block leaves before both know of it and their copies have had time to land; the next launch is right."""
    from vitna_anchor_b200 import ops
    M, N, K = 2048, 6160, 2048
    assert _route(1, M, N, K) == 257
    g = torch.Generator(device="cuda").manual_seed(stage)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    out = torch.zeros(M, N, device="cuda")
    ops.set_wait_limit_ms(5.0)
    try:
        ops.skip_stage_once("linear_tcgen05_wide", stage)
        ops.linear_tcgen05(x, w, out, ops.LINEAR_F32)
        torch.cuda.synchronize()
        with pytest.raises(ops.KernelGaveUp):
            ops.check_device_errors()
    finally:
        ops.set_wait_limit_ms(0)
    ops.linear_tcgen05(x, w, out, ops.LINEAR_F32)
    ops.check_device_errors()
    want, off = x.double() @ w.double().T, K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)      # (as above)
    assert bool(((out.double() - want).abs() <= off).all())
