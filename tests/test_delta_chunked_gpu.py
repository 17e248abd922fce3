"""The delta rule's chunked kernels against the token-by-token ones at the edges of the pieces of 16 tokens, of the chunks of 64 and of the state's slices, over two
steps on scattered slots, with decays from hardly any to almost all."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STEPS = (((1, 2, 15, 16, 17, 64, 31), (3, 0, 6, 2, 5, 7, 4)), ((63, 130, 1, 65, 48, 3, 129), (0, 3, 2, 6, 7, 4, 5)))


@pytest.mark.parametrize("dt", [-6.0, 0.0, 4.0])            # a decay of about 0.997, 0.5 and 0.02 a token
@pytest.mark.parametrize("sizes", [(1, 3, 64, 64, 4), (2, 4, 128, 128, 4), (2, 2, 8, 4, 1), (1, 1, 68, 36, 3), (1, 2, 128, 256, 2), (3, 3, 60, 68, 4), (1, 1, 64, 132, 6)])
@pytest.mark.parametrize("channel", [False, True])
def test_chunks_against_tokens(channel, sizes, dt):
    from vitna_anchor_b200 import ops
    G, H, dk, dv, taps = sizes
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    C, rank = 2 * G * dk + H * dv, 3
    conv, a_log, nw = r(C, taps) * 0.6, r(H) * 0.5, 1 + 0.1 * r(dv)
    state = 0.1 * r(8, ops.delta_state_floats(G, H, dk, dv, taps))
    states = [state.clone(), state.clone()]
    bias = dt + r(H * dk if channel else H)
    a2t, g2t = r(rank, H * dk) * 0.3, r(rank, H * dv)
    for lens, slots in STEPS:
        T, S = sum(lens), len(lens)
        i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device="cuda")
        starts, tseg, seg_slots = i32(np.concatenate([[0], np.cumsum(lens)])), i32(np.repeat(np.arange(S), lens)), i32(slots)
        N = C + H + 2 * rank if channel else C + H * dv + 2 * H
        proj = r(T, N)
        outs = []
        for chunked in (False, True):
            st, out, o = states[chunked], torch.empty(T, H * dv, device="cuda"), torch.empty(T, H * dv, device="cuda")
            if channel:
                scratch = torch.full((ops.channel_delta_chunked_scratch_floats(T, S, H, dk, dv),), float("nan"), device="cuda") if chunked else None
                ops.channel_delta_rule(proj, conv, a_log, bias, a2t, g2t, nw, 1e-5, tseg, starts, seg_slots, st,
                                       torch.empty(T, ops.channel_delta_prep_width(G, H, dk, dv), device="cuda"),
                                       torch.empty(ops.channel_delta_group_floats(T, H, dk), device="cuda"), o, out, G, H, dk, dv, taps, chunk_scratch=scratch)
            else:
                scratch = torch.full((ops.delta_chunked_scratch_floats(T, S, H, dk, dv),), float("nan"), device="cuda") if chunked else None
                ops.delta_rule(proj, conv, a_log, bias, nw, 1e-5, tseg, starts, seg_slots, st, torch.empty(T, ops.delta_prep_width(G, H, dk, dv), device="cuda"), o, out,
                               G, H, dk, dv, taps, chunk_scratch=scratch)
            outs.append((o, out))
        # both forms are float32 sums of up to 130 tokens' contributions; the unit keys keep every sum's terms below the largest value
        for a, b in [(x, y) for x, y in zip(outs[0], outs[1]) if y is outs[1][1] or channel or dv > 128]:       # (o only where the chunks' kernel does not gate)
            assert bool(torch.isfinite(b).all()) and float((a - b).abs().max()) <= 2e-5 * max(1.0, float(a.abs().max()))
    assert float((states[0] - states[1]).abs().max()) <= 2e-5 * max(1.0, float(states[0].abs().max()))
    assert torch.equal(states[1][1], state[1])                 # a slot nobody holds


def test_a_wait_that_runs_out_is_reported():
    """The scan's copies: one chunk's is left out, the wait for it runs out, the kernel returns by itself and the host learns of it."""
    from vitna_anchor_b200 import ops
    G, H, dk, dv, taps, T = 1, 2, 64, 64, 4, 200
    C, N = 2 * G * dk + H * dv, 2 * G * dk + 2 * H * dv + 2 * H
    z = lambda *s: torch.zeros(*s, device="cuda")
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    go = lambda: ops.delta_rule(torch.ones(T, N, device="cuda"), torch.ones(C, taps, device="cuda"), z(H), z(H), torch.ones(dv, device="cuda"), 1e-5, z(T).int(), i32([0, T]),
                                i32([0]), z(1, ops.delta_state_floats(G, H, dk, dv, taps)), z(T, ops.delta_prep_width(G, H, dk, dv)), z(T, H * dv), z(T, H * dv), G, H, dk,
                                dv, taps, chunk_scratch=z(ops.delta_chunked_scratch_floats(T, 1, H, dk, dv)))
    ops.set_wait_limit_ms(5)
    try:
        ops.skip_stage_once("delta_chunked", 1)
        go()
        torch.cuda.synchronize()
        with pytest.raises(ops.KernelGaveUp, match=r"code 61\)"):
            ops.check_device_errors()
        out = go()
        torch.cuda.synchronize()
        ops.check_device_errors()
        assert bool(torch.isfinite(out).all())
    finally:
        ops.set_wait_limit_ms(0)


def _prepare(lens, G, H, dk, dv, taps, first=0, count=None):
    """Rows first .. first + count of the prepared inputs of a step of segments `lens`, by a step that holds these rows alone (their first segment's memory is
    then the inputs before them)."""
    import ctypes
    from vitna_anchor_b200 import ops
    C = 2 * G * dk + H * dv
    N, T = C + H * dv + 2 * H, sum(lens)
    g = torch.Generator(device="cuda").manual_seed(taps)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    proj, conv, a_log, bias, state = r(T, N), r(C, taps), r(H), r(H), r(len(lens), ops.delta_state_floats(G, H, dk, dv, taps))
    count = T - first if count is None else count
    ids, at = np.unique(np.repeat(np.arange(len(lens)), lens)[first:first + count], return_index=True)
    seg, start = np.repeat(np.arange(len(lens)), lens)[first:first + count] - ids[0], np.concatenate([[0], np.cumsum(lens)])
    if taps > 1 and start[ids[0]] < first:
        memory = state[ids[0], H * dv * dk:H * dv * dk + (taps - 1) * C].view(taps - 1, C)        # oldest input first
        memory.copy_(torch.cat([memory, proj[start[ids[0]]:first, :C]])[-(taps - 1):].clone())
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device="cuda")
    rows, out = proj[first:first + count].contiguous(), torch.zeros(count, ops.delta_prep_width(G, H, dk, dv), device="cuda")
    tseg, starts, slots = i32(seg), i32(np.append(at, count)), i32(ids)
    assert ops.lib().vk_delta_prepare(ops._p(rows), ops._p(conv), ops._p(a_log), ops._p(bias), ops._p(tseg), ops._p(starts), ops._p(slots), ops._p(state),
                                      ctypes.c_size_t(state.shape[1]), ops._p(out), count, G, H, dk, dv, taps, ops._stream()) == 0
    return out[:, :C + 2 * H]


# one slice of q and k heads and several, a last one that is not full, heads of one channel, of a slice and of more; one slice of v and several, full and not; the longest
# head that eight tokens have room for, 1,533 channels, and the next, which a block a token takes
@pytest.mark.parametrize("taps", [1, 3, 4])
@pytest.mark.parametrize("G,H,dk,dv,sliced", [(2, 2, 20, 12, True), (3, 9, 64, 64, True), (5, 5, 60, 52, True), (3, 6, 100, 43, True), (1, 1, 256, 256, True), (2, 2, 300, 130, True),
                                              (130, 130, 1, 2, True), (1, 1, 1533, 8, True), (1, 1, 1534, 8, False), (12, 12, 64, 4, True)])
def test_neighbouring_tokens_are_prepared_as_single_ones(G, H, dk, dv, sliced, taps):
    """A step whose tokens are prepared eight a block, a slice of the channels each, gives the bits of the same tokens in steps that a block a token prepares: across
    segments' borders, carried memories and odd lengths."""
    from vitna_anchor_b200 import ops
    lens = [1, 2, 3, 700, 4, 487, 1, 1]
    T = sum(lens)
    slices = ops.lib().vk_delta_prepare_slices
    assert (slices(T, G, H, dk, dv, taps) > 0) == sliced
    whole = _prepare(lens, G, H, dk, dv, taps)
    for lo in range(0, T, 61):
        n = min(61, T - lo)
        assert slices(n, G, H, dk, dv, taps) == 0
        assert torch.equal(_prepare(lens, G, H, dk, dv, taps, lo, n), whole[lo:lo + n]), lo


@pytest.mark.parametrize("strong", [3.0, 200.0, 1e30, float("inf")])       # sums to -100, -6,400, and beyond what any sum holds
@pytest.mark.parametrize("dk", [64, 128])
def test_strong_decays_beside_weak_ones(dk, strong):
    """Tokens that leave almost nothing of the state in front of tokens that leave almost all, inside one chunk, against the recurrence in 64 bits."""
    from vitna_anchor_b200 import ops
    G, H, dv, taps, T = 1, 2, 32, 1, 192
    rng = np.random.default_rng(dk)
    N = 2 * G * dk + 2 * H * dv + 2 * H
    proj = rng.standard_normal((T, N)).astype(np.float32)
    a = np.where((np.arange(T) // 8) % 4 < 2, strong, -2.25)[:, None] + 0.05 * rng.standard_normal((T, H))      # softplus(-2.25) is 0.1
    proj[:, N - H:] = a
    conv, nw = rng.standard_normal((2 * G * dk + H * dv, taps)).astype(np.float32), np.ones(dv, np.float32)
    dev = lambda x: torch.from_numpy(x).cuda()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    state = torch.zeros(1, ops.delta_state_floats(G, H, dk, dv, taps), device="cuda")
    out = torch.empty(T, H * dv, device="cuda")
    ops.delta_rule(dev(proj), dev(conv), torch.zeros(H, device="cuda"), torch.zeros(H, device="cuda"), dev(nw), 1e-6, i32([0] * T), i32([0, T]), i32([0]), state,
                   torch.empty(T, ops.delta_prep_width(G, H, dk, dv), device="cuda"), torch.empty(T, H * dv, device="cuda"), out, G, H, dk, dv, taps,
                   chunk_scratch=torch.full((ops.delta_chunked_scratch_floats(T, 1, H, dk, dv),), float("nan"), device="cuda"))
    p = proj.astype(np.float64)
    z = p[:, :2 * G * dk + H * dv] * conv[:, 0]
    act = z / (1 + np.exp(-z))
    unit = lambda x: x / np.sqrt((x ** 2).sum(-1, keepdims=True) + 1e-6)
    q, k, v = unit(act[:, :dk]) * dk ** -0.5, unit(act[:, dk:2 * dk]), act[:, 2 * dk:].reshape(T, H, dv)
    gate, beta = p[:, 2 * dk + H * dv:2 * dk + 2 * H * dv].reshape(T, H, dv), 1 / (1 + np.exp(-p[:, N - 2 * H:N - H]))
    g = np.exp(-np.logaddexp(0.0, p[:, N - H:]))
    S, want = np.zeros((H, dk, dv)), np.zeros((T, H, dv))
    for t in range(T):
        S *= g[t][:, None, None]
        S += k[t][None, :, None] * (beta[t][:, None] * (v[t] - np.einsum("hkv,k->hv", S, k[t])))[:, None, :]
        want[t] = np.einsum("hkv,k->hv", S, q[t])
    want = want / np.sqrt((want ** 2).mean(-1, keepdims=True) + 1e-6) * gate / (1 + np.exp(-gate))
    # float32 sums of up to 64 tokens' contributions, as in test_chunks_against_tokens; a ratio of decays from float32 sums of -6,400 would be 5e-4 off
    assert np.abs(out.double().cpu().numpy().reshape(T, H, dv) - want).max() <= 2e-5 * np.abs(want).max()
    got = state[0, :H * dv * dk].double().cpu().numpy().reshape(H, dv, dk).transpose(0, 2, 1)
    assert np.abs(got - S).max() <= 2e-5 * max(1.0, np.abs(S).max())


@pytest.mark.parametrize("lens", [(600, 1, 1, 32, 33, 1), (1, 161, 2), (33, 32, 700), (1, 1, 40, 1), (200,), (1200, 900)])
@pytest.mark.parametrize("few", [1, 100])
@pytest.mark.parametrize("channel,dk,dv", [(False, 16, 32), (False, 72, 132), (True, 16, 32), (True, 72, 36)])
def test_a_step_of_segments_of_every_length(channel, dk, dv, lens, few, monkeypatch):
    """Long segments in chunks, with short ones token after token or among them: all have the results and states of the token-by-token kernels, and those that run token
    after token their bits."""
    from vitna_anchor_b200.cache import CacheManager
    from vitna_anchor_b200.engine.context import ContextBuilder
    from vitna_anchor_b200.parts.base import StepContext, Workspace
    from vitna_anchor_b200.parts.delta import ChannelDeltaRule, GatedDeltaRule
    W, G, H, taps, rank, T = 64, 1, 2, 4, 4, sum(lens)
    got = []
    for plain in (False, True):
        if plain:
            monkeypatch.setattr(StepContext, "chunk_plan", lambda *a: None)
        g = torch.Generator(device="cuda").manual_seed(dk)
        r = lambda *s: torch.randn(*s, generator=g, device="cuda")
        m = lambda rows, cols: (r(rows, cols) * cols ** -0.5).bfloat16()
        C = 2 * G * dk + H * dv
        if channel:
            part = ChannelDeltaRule(W, H, G, dk, dv, taps, m(C + H + 2 * rank, W), r(C, taps), 0.5 * r(H), r(H * dk) - 2, 0.5 * r(H * dk, rank), r(H * dv, rank), 1 + 0.1 * r(dv),
                                    m(W, H * dv), 1e-6)
        else:
            part = GatedDeltaRule(W, H, G, dk, dv, taps, m(C + H * dv + 2 * H, W), r(C, taps), 0.5 * r(H), r(H) - 2, 1 + 0.1 * r(dv), m(W, H * dv), 1e-6)
        cache = CacheManager([part.cache_spec()], page_size=16, num_pages=64, max_requests=len(lens), dtype=torch.bfloat16, device="cuda")
        builder = ContextBuilder(cache, torch.bfloat16, Workspace(torch.device("cuda"), T, len(lens), 4096), max_batch_tokens=T, max_segments=len(lens), max_model_len=4096,
                                 device="cuda")
        for i in range(len(lens)):
            cache.open(i)
        cache.reserve_step([(i, n) for i, n in enumerate(lens)])
        ctx, _ = builder.build([(i, [0] * n, []) for i, n in enumerate(lens)])
        ctx.caches[0].state.copy_(0.1 * r(*ctx.caches[0].state.shape))
        x, y = r(T, W).bfloat16(), torch.zeros(T, W, device="cuda")
        part.chunk_rule = part.chunk_rule._replace(few=few)
        assert plain or (ctx.chunk_plan(part.chunk_rule) is not None) == (max(lens) > 160)
        part.forward(x, ctx, ctx.caches[0], y)
        got.append((y, ctx.caches[0].state.clone(), ctx.host_seg_slots))
    (y, st, slots), (want, want_st, _) = got
    assert float((y - want).abs().max()) <= 2e-2 * float(want.abs().max())         # bfloat16 outputs of the heads in front of the last product
    assert float((st - want_st).abs().max()) <= 2e-5 * max(1.0, float(want_st.abs().max()))
    for n, slot in zip(lens, slots):
        if n <= 32 and few == 1:
            assert torch.equal(st[slot], want_st[slot]), n



def test_a_captured_step_is_not_played_for_one_with_longer_segments(tmp_path):
    """Two steps whose counts of tokens, requests and tiles are the same (70 + 60 and 100 + 30 tokens) take different launches, because only the second has a segment
    long enough for chunks: the graph captured for the one must not be played for the other."""
    import lupanex_models as LM
    from vitna_anchor_b200.engine.loading import load_model
    from vitna_anchor_b200.engine.runner import ModelRunner, StepEntry
    model_dir = LM.make_model(str(tmp_path / "m"), "streams", 5)
    rows = {}
    for graphs in (True, False):
        model = load_model(model_dir, "bfloat16", "cuda")
        assert model.chunk_rules
        runner = ModelRunner(model, page_size=16, num_pages=64, max_requests=2, max_batch_tokens=256, max_model_len=model.max_positions, device="cuda", cuda_graphs=graphs)
        rng, got = np.random.default_rng(3), []
        for lens in ((70, 60), (70, 60), (70, 60), (100, 30), (30, 100), (100, 30), (70, 60)):
            for i, n in enumerate(lens):
                runner.open(i)
            ids = [rng.integers(0, model.vocab_size, n).tolist() for n in lens]
            got.append(runner.step([StepEntry(i, t, [len(t) - 1]) for i, t in enumerate(ids)]).clone())
            for i in range(2):
                runner.close(i)
        runner.check(sync=True)
        rows[graphs] = torch.stack(got)
        assert not graphs or runner.graph_replays > 0
    assert float((rows[True] - rows[False]).abs().max()) <= 1e-5 * max(1.0, float(rows[False].abs().max()))        # the same launches either way
