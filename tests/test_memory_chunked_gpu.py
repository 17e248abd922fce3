"""The matrix memories' chunked kernels against the same recurrences token after token, written out in 64 bits: at the edges of the pieces of 16 tokens and
of the chunks of 64, for heads that fill a tile and heads that do not, over two steps of which the second carries the first's states, on scattered
slots, with gates and decays from hardly any to almost all."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STEPS = (((1, 2, 15, 16, 17, 0, 64), (3, 0, 6, 2, 5, -1, 7)), ((63, 130, 1, 65, 48, 3, 129), (0, 3, 2, -1, 7, 4, 5)))
SIZES = ((2, 64, 256), (1, 128, 256), (3, 20, 36), (2, 4, 4), (2, 68, 132), (4, 128, 64))
# A product of tf32 parts is exact to 2^-22 of its size and up to 200 such products meet in float32 sums that the tensor cores truncate, so a sum is
# off by at most 2^-18 of the sum of its terms' sizes; an output divides two such sums and then its head's root mean square.
PART = 2.0 ** -18


def _ctx(lens, slots):
    starts = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return starts, SimpleNamespace(seg_starts=torch.from_numpy(starts).cuda(), seg_slots=torch.tensor(slots, dtype=torch.int32, device="cuda"),
                                   num_segments=len(lens), decode_only=False)


def _close(got, want, bound, what):
    got = got.double().cpu().numpy()
    assert np.isfinite(got).all(), what
    worst = (np.abs(got - want) / (bound + 1e-30)).max()
    assert worst <= 1.0, (what, worst)


def _rms(x, eps):
    return np.sqrt((x ** 2).mean(-1, keepdims=True) + eps)


@pytest.mark.parametrize("strong", [False, True])
@pytest.mark.parametrize("sizes", SIZES)
def test_mlstm_in_chunks(sizes, strong):
    from vitna_anchor_b200 import ops
    H, dk, dv = sizes
    rng = np.random.default_rng(dk + dv)
    cap, eps = 15.0, 1e-5
    N = (2 * H * dk + 2 * H * dv + 2 * H + 3) // 4 * 4
    dev = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float32)).cuda()
    bias = np.concatenate([rng.standard_normal(H), (-6.0 if strong else 3.0) + rng.standard_normal(H)]).astype(np.float32)
    nw = (1 + 0.1 * rng.standard_normal(H * dv)).astype(np.float32)
    state = torch.zeros(8, ops.mlstm_state_floats(H, dk, dv), device="cuda")
    state[1] = 7.0                                                          # a slot nobody holds stays as it is
    S, n_, m_ = np.zeros((8, H, dk, dv)), np.zeros((8, H, dk)), np.zeros((8, H))
    S_size, n_size = S.copy(), n_.copy()                                    # the same sums of the terms' sizes
    for lens, slots in STEPS:
        T = sum(lens)
        proj = rng.standard_normal((T, N)).astype(np.float32)
        proj[:, 2 * H * dk + 2 * H * dv:] *= 6.0 if strong else 1.0
        starts, ctx = _ctx(lens, slots)
        out = torch.empty(T, H * dv, device="cuda")
        scratch = torch.empty(ops.mlstm_chunked_scratch_bytes(T, len(lens), H, dk, dv), dtype=torch.uint8, device="cuda").fill_(0xff)
        assert ops.memory_chunked_takes(N, dk, dv)
        ops.mlstm(dev(proj), dev(bias), cap, dev(nw), eps, ctx, state, torch.empty(T, H * (dv + 2), device="cuda"), out, H, dk, dv, chunk_scratch=scratch)
        p = proj.astype(np.float64)
        q, k = p[:, :H * dk].reshape(T, H, dk) * dk ** -0.5, p[:, H * dk:2 * H * dk].reshape(T, H, dk)
        v, gate = (p[:, 2 * H * dk + i * H * dv:2 * H * dk + (i + 1) * H * dv].reshape(T, H, dv) for i in (0, 1))
        at = 2 * H * dk + 2 * H * dv
        ig = cap * np.tanh((p[:, at:at + H] + bias[:H]) / cap)
        fg = -np.logaddexp(0.0, -cap * np.tanh((p[:, at + H:at + 2 * H] + bias[H:]) / cap))
        want, size = np.zeros((T, H, dv)), np.zeros((T, H, dv))
        for s, slot in enumerate(slots):
            St, n, m, Sz, nz = (x[slot].copy() if slot >= 0 else np.zeros_like(x[0]) for x in (S, n_, m_, S_size, n_size))
            for t in range(starts[s], starts[s + 1]):
                new = np.maximum(fg[t] + m, ig[t])
                a, b = np.exp(fg[t] + m - new), np.exp(ig[t] - new)
                St = a[:, None, None] * St + b[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
                n, m = a[:, None] * n + b[:, None] * k[t], new
                Sz = a[:, None, None] * Sz + b[:, None, None] * np.abs(k[t][:, :, None] * v[t][:, None, :])
                nz = a[:, None] * nz + b[:, None] * np.abs(k[t])
                den = (np.maximum(np.abs((n * q[t]).sum(1)), np.exp(-m)) + 1e-6)[:, None]
                want[t] = np.einsum("hkv,hk->hv", St, q[t]) / den
                size[t] = (np.einsum("hkv,hk->hv", Sz, np.abs(q[t])) + np.abs(want[t]) * (nz * np.abs(q[t])).sum(1)[:, None]) / den
            if slot >= 0:
                S[slot], n_[slot], m_[slot], S_size[slot], n_size[slot] = St, n, m, Sz, nz
        scale = nw.reshape(H, dv) / (1 + np.exp(-gate)) / _rms(want, eps)
        bound = PART * (size + np.abs(want) * (1 + _rms(size, 0) / _rms(want, eps))) * np.abs(scale)
        _close(out, (want * scale).reshape(T, H * dv), bound.reshape(T, H * dv), (sizes, lens))
    assert float((state[1] - 7.0).abs().max()) == 0.0
    for slot in (0, 2, 3, 4, 5, 6, 7):
        row = state[slot].cpu()
        _close(row[:H * dk * dv], S[slot].reshape(-1), PART * S_size[slot].reshape(-1), ("S", slot))
        _close(row[H * dk * dv:H * dk * dv + H * dk], n_[slot].reshape(-1), PART * n_size[slot].reshape(-1), ("n", slot))
        _close(row[H * dk * dv + H * dk:], m_[slot], 2.0 ** -18 * (1 + np.abs(m_[slot])), ("m", slot))


@pytest.mark.parametrize("tau", [16.0, 1.0, 0.05])         # a decay of about 0.95, 0.5 and 1e-6 a token: the sums of logarithms reach -900 in a chunk
@pytest.mark.parametrize("sizes", SIZES)
def test_gated_linear_attention_in_chunks(sizes, tau):
    from vitna_anchor_b200 import ops
    H, dk, dv = sizes
    rng = np.random.default_rng(dk * 3 + dv)
    rank, eps = 4, 1e-5
    N = 2 * H * dk + 2 * H * dv + rank
    dev = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float32)).cuda()
    a2, bias, nw = (x.astype(np.float32) for x in (rng.standard_normal((H * dk, rank)) * 0.5, rng.standard_normal(H * dk), 1 + 0.2 * rng.standard_normal(dv)))
    state = torch.zeros(8, H * dk * dv, device="cuda")
    state[1] = 7.0
    S = np.zeros((8, H, dk, dv))
    S_size = S.copy()
    for lens, slots in STEPS:
        T = sum(lens)
        proj = rng.standard_normal((T, N)).astype(np.float32)
        starts, ctx = _ctx(lens, slots)
        out = torch.empty(T, H * dv, device="cuda")
        scratch = torch.empty(ops.gla_chunked_scratch_bytes(T, len(lens), H, dk, dv), dtype=torch.uint8, device="cuda").fill_(0xff)
        ops.gla(dev(proj), N - rank, dev(a2.T.copy()), dev(bias), tau, dev(nw), eps, ctx, state, torch.empty(T, H * dk, device="cuda"),
                torch.empty(T, H * dv, device="cuda"), out, H, dk, dv, 2 * H * dk + H * dv, chunk_scratch=scratch)
        p = proj.astype(np.float64)
        q, k = p[:, :H * dk].reshape(T, H, dk) * dk ** -0.5, p[:, H * dk:2 * H * dk].reshape(T, H, dk)
        v, g = (p[:, 2 * H * dk + i * H * dv:2 * H * dk + (i + 1) * H * dv].reshape(T, H, dv) for i in (0, 1))
        a = np.exp(-np.logaddexp(0.0, -(p[:, N - rank:] @ a2.astype(np.float64).T + bias)) / tau).reshape(T, H, dk)
        want, size = np.zeros((T, H, dv)), np.zeros((T, H, dv))
        for s, slot in enumerate(slots):
            St, Sz = (x[slot].copy() if slot >= 0 else np.zeros((H, dk, dv)) for x in (S, S_size))
            for t in range(starts[s], starts[s + 1]):
                St = a[t][:, :, None] * St + k[t][:, :, None] * v[t][:, None, :]
                Sz = a[t][:, :, None] * Sz + np.abs(k[t][:, :, None] * v[t][:, None, :])
                want[t], size[t] = np.einsum("hkv,hk->hv", St, q[t]), np.einsum("hkv,hk->hv", Sz, np.abs(q[t]))
            if slot >= 0:
                S[slot], S_size[slot] = St, Sz
        scale = nw * (g / (1 + np.exp(-g))) / _rms(want, eps)
        bound = PART * (size + np.abs(want) * (1 + _rms(size, 0) / _rms(want, eps))) * np.abs(scale)
        _close(out, (want * scale).reshape(T, H * dv), bound.reshape(T, H * dv), (sizes, lens))
    assert float((state[1] - 7.0).abs().max()) == 0.0
    for slot in (0, 2, 3, 4, 5, 6, 7):
        _close(state[slot].cpu(), S[slot].reshape(-1), PART * S_size[slot].reshape(-1), ("S", slot))


@pytest.mark.parametrize("rank", [764, 768, 1100])          # around the most whose 16 tokens the chunks' kernel stages (767; rows come in whole pieces of four), and far more
def test_ranks_around_what_the_chunks_take(rank, monkeypatch):
    """A prompt's step through the part: a rank that the chunks do not take runs token after token, with the same results."""
    from vitna_anchor_b200 import ops
    from vitna_anchor_b200.cache import CacheManager
    from vitna_anchor_b200.engine.context import ContextBuilder
    from vitna_anchor_b200.parts.base import Workspace
    from vitna_anchor_b200.parts.gla import GatedLinearAttention
    W, H, dk, dv, T = 64, 1, 16, 16, 600
    assert ops.memory_chunked_takes(2 * H * dk + 2 * H * dv + rank, dk, dv, rank) == (rank <= 767)
    g = torch.Generator(device="cuda").manual_seed(rank)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    part = GatedLinearAttention(W, H, dk, dv, 8.0, (r(2 * H * dk + 2 * H * dv + rank, W) * W ** -0.5).bfloat16(), r(H * dk, rank) * rank ** -0.5, r(H * dk), 1 + 0.1 * r(dv),
                                (r(W, H * dv) * dv ** -0.5).bfloat16(), 1e-6)
    x, got = r(T, W).bfloat16(), []
    for chunked in (True, False):
        if not chunked:
            monkeypatch.setattr(ops, "memory_chunked_takes", lambda *a: False)
        cache = CacheManager([part.cache_spec()], page_size=16, num_pages=T // 16 + 1, max_requests=1, dtype=torch.bfloat16, device="cuda")
        builder = ContextBuilder(cache, torch.bfloat16, Workspace(torch.device("cuda"), T, 1, T), max_batch_tokens=T, max_segments=1, max_model_len=608, device="cuda")
        cache.open(0)
        cache.reserve_step([(0, T)])
        ctx, _ = builder.build([(0, [0] * T, [])])
        ctx.caches[0].state.zero_()
        y = torch.zeros(T, W, device="cuda")
        part.forward(x, ctx, ctx.caches[0], y)
        got.append(y)
    assert float((got[0] - got[1]).abs().max()) <= 2e-2 * float(got[1].abs().max())         # bfloat16 outputs of the head in front of the last product


@pytest.mark.parametrize("kind", ["mlstm", "gla"])
def test_a_norm_weight_that_begins_anywhere(kind):
    """A weight at an address off 8 bytes gives the bits of the same weight on 16."""
    from vitna_anchor_b200 import ops
    H, dk, dv, T, rank = 2, 20, 36, 100, 4
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    n_nw = H * dv if kind == "mlstm" else dv
    proj, bias, a2t, longer = r(T, 2 * H * dk + 2 * H * dv + 4), r(2 * H if kind == "mlstm" else H * dk), r(rank, H * dk), r(n_nw + 1)
    got = []
    for nw in (longer[1:], longer[1:].clone()):
        ctx, out = _ctx((T,), (0,))[1], torch.empty(T, H * dv, device="cuda")
        if kind == "mlstm":
            ops.mlstm(proj, bias, 15.0, nw, 1e-5, ctx, torch.zeros(1, ops.mlstm_state_floats(H, dk, dv), device="cuda"), torch.empty(T, H * (dv + 2), device="cuda"), out, H, dk,
                      dv, chunk_scratch=torch.empty(ops.mlstm_chunked_scratch_bytes(T, 1, H, dk, dv), dtype=torch.uint8, device="cuda"))
        else:
            ops.gla(proj, proj.shape[1] - rank, a2t, bias, 8.0, nw, 1e-5, ctx, torch.zeros(1, H * dk * dv, device="cuda"), torch.empty(T, H * dk, device="cuda"),
                    torch.empty(T, H * dv, device="cuda"), out, H, dk, dv, 2 * H * dk + H * dv,
                    chunk_scratch=torch.empty(ops.gla_chunked_scratch_bytes(T, 1, H, dk, dv), dtype=torch.uint8, device="cuda"))
        got.append(out)
    assert longer[1:].data_ptr() % 8 == 4 and torch.equal(got[0], got[1])


def _part_and_batch(kind, lens, max_tokens, max_requests):
    from vitna_anchor_b200.cache import CacheManager
    from vitna_anchor_b200.engine.context import ContextBuilder
    from vitna_anchor_b200.parts.base import Workspace
    from vitna_anchor_b200.parts.gla import GatedLinearAttention
    from vitna_anchor_b200.parts.mlstm import MatrixLSTM
    W, H, dk, dv, rank = 64, 2, 16, 32, 4
    g = torch.Generator(device="cuda").manual_seed(len(lens))
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    m = lambda rows, cols: (r(rows, cols) * cols ** -0.5).bfloat16()
    if kind == "mlstm":
        part = MatrixLSTM(W, H, dk, dv, 15.0, m(2 * H * dk + 2 * H * dv + 2 * H, W), r(2 * H), 1 + 0.1 * r(H * dv), m(W, H * dv), 1e-6)
    else:
        part = GatedLinearAttention(W, H, dk, dv, 8.0, m(2 * H * dk + 2 * H * dv + rank, W), r(H * dk, rank) * 0.5, r(H * dk), 1 + 0.1 * r(dv), m(W, H * dv), 1e-6)
    cache = CacheManager([part.cache_spec()], page_size=16, num_pages=64, max_requests=max_requests, dtype=torch.bfloat16, device="cuda")
    builder = ContextBuilder(cache, torch.bfloat16, Workspace(torch.device("cuda"), max_tokens, max_requests, 4096), max_batch_tokens=max_tokens, max_segments=max_requests,
                             max_model_len=4096, device="cuda")
    for i in range(len(lens)):
        cache.open(i)
    cache.reserve_step([(i, n) for i, n in enumerate(lens)])
    ctx, _ = builder.build([(i, [0] * n, []) for i, n in enumerate(lens)])
    ctx.caches[0].state.copy_(0.1 * r(*ctx.caches[0].state.shape))
    return part, ctx, r(sum(lens), W).bfloat16()


@pytest.mark.parametrize("lens", [(600, 1, 1, 32, 33, 1), (1, 433, 2), (33, 32, 700), (1, 1, 40, 1), (500,), (1200, 900)])
@pytest.mark.parametrize("few", [1, 100])
@pytest.mark.parametrize("kind", ["mlstm", "gla"])
def test_a_step_of_segments_of_every_length(kind, lens, few, monkeypatch):
    """Long segments in chunks, with short ones token after token or among them: all have the results and states of the token-by-token kernels, and those that run token
    after token their bits."""
    from vitna_anchor_b200.parts.base import StepContext
    got = []
    for plain in (False, True):
        if plain:
            monkeypatch.setattr(StepContext, "chunk_plan", lambda *a: None)
        part, ctx, x = _part_and_batch(kind, lens, sum(lens), len(lens))
        part.chunk_rule = part.chunk_rule._replace(few=few)
        assert plain or (ctx.chunk_plan(part.chunk_rule) is not None) == (max(lens) > 432)
        y = torch.zeros(x.shape[0], 64, device="cuda")
        part.forward(x, ctx, ctx.caches[0], y)
        got.append((y, ctx.caches[0].state.clone(), ctx.host_seg_slots))
    (y, st, slots), (want, want_st, _) = got
    assert float((y - want).abs().max()) <= 2e-2 * float(want.abs().max())         # bfloat16 outputs of the heads in front of the last product
    assert float((st - want_st).abs().max()) <= 2e-4 * float(want_st.abs().max())
    for n, slot in zip(lens, slots):
        if n <= 32 and few == 1:
            assert torch.equal(st[slot], want_st[slot]), n


def test_scratch_follows_the_segments_that_can_be_long():
    """Steps of up to 2,048 tokens and 256 requests: of more than 32 tokens there are at most 62 segments, and only those have chunks."""
    from vitna_anchor_b200 import ops
    assert ops.mlstm_chunked_scratch_bytes(2048, 256, 8, 128, 256, 32) == ops.mlstm_chunked_scratch_bytes(2048, 62, 8, 128, 256)
    assert 3 * ops.mlstm_chunked_scratch_bytes(2048, 256, 8, 128, 256, 32) < ops.mlstm_chunked_scratch_bytes(2048, 256, 8, 128, 256)
