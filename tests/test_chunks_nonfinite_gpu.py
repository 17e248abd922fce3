"""What is not finite in the chunked recurrences: a NaN that the device made, or an infinity, in one token's operands or in a carried state is to be found where the
token-by-token kernels have it."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENS, SLOTS = (70, 200, 1, 66), (3, 0, 2, 1)
AT = 70 + 100                               # the token that carries it: the second request's hundredth, inside its second chunk


def _made(kind):
    """A NaN as the arithmetic instructions make it (inf - inf), or an infinity."""
    inf = torch.full((1,), float("inf"), device="cuda")
    return inf - inf if kind == "nan" else inf


def _meta():
    starts = np.concatenate([[0], np.cumsum(LENS)]).astype(np.int32)
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device="cuda")
    return sum(LENS), len(LENS), i32(starts), i32(np.repeat(np.arange(len(LENS)), LENS)), i32(SLOTS)


def _memory(kind, H, dk, dv, place, what):
    """mLSTM and gated linear attention: (outputs, states) token after token and in chunks, with `what` at one place."""
    from vitna_anchor_b200 import ops
    T, S, starts, tseg, slots = _meta()
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    rank = 4
    N = 2 * H * dk + 2 * H * dv + (2 * H if kind == "mlstm" else rank)
    proj = r(T, N)
    state = 0.1 * r(4, (ops.mlstm_state_floats if kind == "mlstm" else ops.gla_state_floats)(H, dk, dv))
    cols = {"q": dk + 3, "k": H * dk + dk + 3, "v": 2 * H * dk + dv + 5, "gate": 2 * H * dk + H * dv + dv + 5, "rest": 2 * H * dk + 2 * H * dv + 1,
            "rest_last": N - 1}
    if place == "state":
        state[0, dv + 7] = _made(what)[0]
    else:
        proj[AT, cols[place]] = _made(what)[0]
    bias, nw = r(2 * H if kind == "mlstm" else H * dk), 1 + 0.1 * r(H * dv if kind == "mlstm" else dv)
    a2t = r(rank, H * dk)
    ctx = SimpleNamespace(seg_starts=starts, seg_slots=slots, num_segments=S, decode_only=False)
    got = []
    for chunked in (False, True):
        st, out = state.clone(), torch.empty(T, H * dv, device="cuda")
        nbytes = (ops.mlstm_chunked_scratch_bytes if kind == "mlstm" else ops.gla_chunked_scratch_bytes)(T, S, H, dk, dv)
        scratch = torch.full((nbytes,), 0xff, dtype=torch.uint8, device="cuda") if chunked else None
        if kind == "mlstm":
            ops.mlstm(proj, bias, 15.0, nw, 1e-5, ctx, st, torch.empty(T, H * (dv + 2), device="cuda"), out, H, dk, dv, chunk_scratch=scratch)
        else:
            ops.gla(proj, N - rank, a2t, bias, 8.0, nw, 1e-5, ctx, st, torch.empty(T, H * dk, device="cuda"), torch.empty(T, H * dv, device="cuda"), out, H, dk, dv,
                    2 * H * dk + H * dv, chunk_scratch=scratch)
        got.append((out, st))
    return got


def _delta(kind, G, H, dk, dv, place, what):
    from vitna_anchor_b200 import ops
    T, S, starts, tseg, slots = _meta()
    taps, rank, C, channel = 4, 3, 2 * G * dk + H * dv, kind == "channel"
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    N = C + H + 2 * rank if channel else C + H * dv + 2 * H
    proj, conv, a_log, nw = r(T, N), r(C, taps) * 0.6, r(H) * 0.5, 1 + 0.1 * r(dv)
    bias, a2t, g2t = r(H * dk if channel else H) - 2.0, r(rank, H * dk) * 0.3, r(rank, H * dv)
    state = 0.1 * r(4, ops.delta_state_floats(G, H, dk, dv, taps))
    cols = {"q": 3, "k": G * dk + 3, "v": 2 * G * dk + 5, "gate": N - 1 if channel else C + 5, "rest": C if channel else N - 2 * H, "rest_last": C + H if channel else N - 1}
    if place == "state":
        state[0, 9] = _made(what)[0]
    else:
        proj[AT, cols[place]] = _made(what)[0]
    got = []
    for chunked in (False, True):
        st, out, o = state.clone(), torch.empty(T, H * dv, device="cuda"), torch.empty(T, H * dv, device="cuda")
        if channel:
            scratch = torch.full((ops.channel_delta_chunked_scratch_floats(T, S, H, dk, dv),), float("nan"), device="cuda") if chunked else None
            ops.channel_delta_rule(proj, conv, a_log, bias, a2t, g2t, nw, 1e-5, tseg, starts, slots, st,
                                   torch.empty(T, ops.channel_delta_prep_width(G, H, dk, dv), device="cuda"),
                                   torch.empty(ops.channel_delta_group_floats(T, H, dk), device="cuda"), o, out, G, H, dk, dv, taps, chunk_scratch=scratch)
        else:
            scratch = torch.full((ops.delta_chunked_scratch_floats(T, S, H, dk, dv),), float("nan"), device="cuda") if chunked else None
            ops.delta_rule(proj, conv, a_log, bias, nw, 1e-5, tseg, starts, slots, st, torch.empty(T, ops.delta_prep_width(G, H, dk, dv), device="cuda"), o, out,
                           G, H, dk, dv, taps, chunk_scratch=scratch)
        got.append((out, st))
    return got


RUNS = [("mlstm", (2, 64, 256)), ("mlstm", (2, 128, 64)), ("gla", (2, 64, 256)), ("gla", (2, 128, 64)), ("delta", (1, 2, 64, 64)), ("delta", (2, 2, 128, 256)),
        ("channel", (1, 2, 64, 64)), ("channel", (2, 2, 128, 128))]
PLACES = ("q", "k", "v", "gate", "rest", "rest_last", "state")


@pytest.mark.parametrize("place", PLACES)
@pytest.mark.parametrize("kind,sizes", RUNS)
def test_a_nan_is_kept(kind, sizes, place):
    tokens, chunks = (_memory if kind in ("mlstm", "gla") else _delta)(kind, *sizes, place, "nan")
    assert bool(torch.isnan(tokens[0]).any())
    for a, b in zip(tokens, chunks):
        assert not bool((torch.isnan(a) & ~torch.isnan(b)).any()), (kind, place)


def _heads(kind, sizes, out):
    H, dv = sizes[-3] if kind in ("mlstm", "gla") else sizes[1], sizes[-1]
    return out.view(-1, H, dv)


@pytest.mark.parametrize("place", PLACES)
@pytest.mark.parametrize("kind,sizes", RUNS)
def test_a_nan_stays_where_it_belongs(kind, sizes, place):
    """The tokens in front of it, inside its chunk too, the other columns, heads and requests are what the token-by-token kernels make them."""
    tokens, chunks = (_memory if kind in ("mlstm", "gla") else _delta)(kind, *sizes, place, "nan")
    for a, b in zip(tokens, chunks):
        on = torch.isfinite(a)
        assert torch.equal(on, torch.isfinite(b)), (kind, place, int((on & ~torch.isfinite(b)).sum()), int((~on & torch.isfinite(b)).sum()))
        # float32 sums of up to 200 tokens' contributions, 6e-7 apart at their size; mLSTM divides by one that nearly cancels in some rows
        assert float((a[on] - b[on]).abs().max()) <= (1e-3 if kind == "mlstm" else 2e-5) * max(1.0, float(a[on].abs().max()))


@pytest.mark.parametrize("place", PLACES)
@pytest.mark.parametrize("kind,sizes", [r for r in RUNS if r[0] != "channel"])
def test_an_infinity_stays_where_it_belongs(kind, sizes, place):
    """A head's row without anything but finite values token after token has finite values here, and one with something else has something else here.  (Which of a row's
    values, and of what kind, hangs on the order of the sums: an infinity of each sign is a NaN, and a head's norm spreads the one and not the other.)"""
    tokens, chunks = (_memory if kind in ("mlstm", "gla") else _delta)(kind, *sizes, place, "inf")
    a, b = (torch.isfinite(_heads(kind, sizes, x[0])).all(-1) for x in (tokens, chunks))
    assert torch.equal(a, b), (kind, place)
    assert torch.equal(torch.isfinite(tokens[1]), torch.isfinite(chunks[1]))
