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
        for a, b in zip(outs[0], outs[1]):
            assert bool(torch.isfinite(b).all()) and float((a - b).abs().max()) <= 2e-5 * max(1.0, float(a.abs().max()))
    assert float((states[0] - states[1]).abs().max()) <= 2e-5 * max(1.0, float(states[0].abs().max()))
    assert torch.equal(states[1][1], state[1])                 # a slot nobody holds
