"""The recurrences in chunks of tokens on values that are no ordinary numbers, against the walk token by token over the same inputs: what
is NaN or Inf at a token reaches that token and later ones, the columns and requests that it reaches in the walk and no others."""
import math

import pytest
import torch

from test_delta_chunks_gpu import DEV, tables

pytestmark = pytest.mark.gpu


def inputs(kind, H, dk, dv, lengths, g):
    from hk_b200.csrc import ops
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)       # noqa: E731
    n, R, K, V = sum(lengths), len(lengths), H * dk, H * dv
    dvp = ops.mlstm_padded(dv) if kind == "memory" else dv
    t = {"proj": rand(n, 3 * K + V + 4 * H), "state": rand(R, H, dk, dvp), "m": rand(R, H), "bias": rand(2 * K) - 1.0, "wl": rand(n, K)}
    if kind == "memory":
        t["state"][..., dv + 1:] = 0.0
    return t


def scan(kind, H, dk, dv, lengths, t, first_chunked, eps=1e-6):
    """(out, state) with the requests from `first_chunked` on in chunks."""
    from hk_b200.csrc import ops
    short, long, chunks, requests = tables(lengths, first_chunked)
    more = {"chunks": chunks, "requests": requests, "most_rows": max(lengths)} if first_chunked < len(lengths) else {}
    n, K, V, p, state = sum(lengths), H * dk, H * dv, t["proj"], t["state"].clone()
    q, k, v, x, logits = p[:, :K], p[:, K:2 * K], p[:, 2 * K:2 * K + V], p[:, 2 * K + V:3 * K + V], p[:, 3 * K + V:]
    out = torch.full((n, H * state.shape[3]), 7.0, device=DEV)
    if kind == "general":
        ops.delta_rule_scan(q, k, v, x, t["wl"], t["bias"][:K], t["bias"][K:], short, state, out, H, dk, dv, math.exp(-0.5), eps, **more)
    elif kind == "gated":
        ops.gated_delta_scan(q, k, v, logits[:, :H], logits[:, H:2 * H], t["bias"][:H].abs(), t["bias"][H:2 * H], short, state, out, H, H, dk, dv,
                             dk ** -0.5, eps, **more)
    elif kind == "retention":
        pos = torch.cat([torch.arange(c) for c in lengths]).int().to(DEV)
        angle = torch.arange(max(lengths), device=DEV)[:, None] * torch.rand(1, 2, generator=torch.Generator(DEV).manual_seed(1), device=DEV)
        ops.retention_scan(q, k, v, angle.cos(), angle.sin(), 4, pos, 1 - t["bias"][:H].abs() * 0.05, short, state, out, H, dk, dv, 0.3, **more)
    else:
        gates = torch.empty(n, H, 3, device=DEV)
        ops.mlstm_scan(q, k, v, logits[:, :H], logits[:, H:2 * H], t["bias"][:H], t["bias"][H:2 * H] + 4, short, state, t["m"].clone(), out, gates,
                       H, dk, dv, 15.0, 0.5, **({**more, "long_segments": long} if more else {}))
    return out, state


def same(got, want, more_finite=False):
    for a, b, what in zip(got, want, ("outputs", "states")):
        finite = torch.isfinite(b)
        # (the walk runs the matrix memory as a delta rule that removes nothing: 0 times a NaN entry reaches the column's others)
        assert torch.equal(torch.isfinite(a) & finite if more_finite else torch.isfinite(a), finite), what
        worst = float((a - b)[finite].abs().max() / b[finite].abs().max())
        assert worst <= 6e-5, f"{what}: {worst:.3g} of the largest value"      # float32 rounding of both


@pytest.mark.parametrize("kind", ["general", "gated", "retention", "memory"])
@pytest.mark.parametrize("dk,dv", [(64, 64), (24, 20), (64, 132)])
@pytest.mark.parametrize("what", ["value", "key", "read", "gate"])
@pytest.mark.parametrize("at", [0, 17, 31, 63, 69])
def test_what_is_not_finite_reaches_no_earlier_token(kind, dk, dv, what, at):
    H, lengths = 2, [40, 70, 65]
    if what == "gate" and kind == "retention":
        return                          # its decays are the model's
    t = inputs(kind, H, dk, dv, lengths, torch.Generator(DEV).manual_seed(dk + dv + at))
    K, V, row = H * dk, H * dv, lengths[0] + at
    col = {"read": 3, "key": K + 3, "value": 2 * K + dv // 2, "gate": 3 * K + V if kind in ("gated", "memory") else 2 * K + V + 3}[what]
    for spoil in (float("nan"), float("inf")) if what == "value" else (float("nan"),):
        t["proj"][row, col] = spoil     # of head 0 of the second request
        want = scan(kind, H, dk, dv, lengths, t, len(lengths))
        assert bool(torch.isfinite(want[0][:row]).all()) and not bool(torch.isfinite(want[0][row]).all())
        same(scan(kind, H, dk, dv, lengths, t, 0), want, kind == "memory" and what == "key")
        if kind == "gated" and what == "gate":      # the decay's logit instead of the step's
            t["proj"][row, col], t["proj"][row, col + H] = 0.5, spoil
            same(scan(kind, H, dk, dv, lengths, t, 0), scan(kind, H, dk, dv, lengths, t, len(lengths)))
        if kind == "general" and what == "gate":    # the channel's decay
            t["proj"][row, col], t["wl"][row, 3] = 0.5, spoil
            same(scan(kind, H, dk, dv, lengths, t, 0), scan(kind, H, dk, dv, lengths, t, len(lengths)))


@pytest.mark.parametrize("kind", ["general", "gated"])
@pytest.mark.parametrize("lengths", [[33], [1, 70, 95]])
def test_chunks_that_are_not_full_without_an_epsilon(kind, lengths):
    """Rows that fill a chunk up have no key whose length could be divided by."""
    t = inputs(kind, 2, 64, 64, lengths, torch.Generator(DEV).manual_seed(len(lengths)))
    got, want = (scan(kind, 2, 64, 64, lengths, t, first, eps=0.0) for first in (0, len(lengths)))
    assert all(bool(torch.isfinite(x).all()) for x in want)
    same(got, want)


@pytest.mark.parametrize("first_chunked", [0, 2])
def test_gates_and_maxima_of_the_matrix_memory(first_chunked):
    """What `mlstm_scan` leaves in `gates` and `m_state`, for requests in chunks and beside them, from the logits alone."""
    from hk_b200.csrc import ops
    H, dk, dv, lengths, cap = 3, 8, 8, [5, 33, 70, 129], 15.0
    g = torch.Generator(DEV).manual_seed(7)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)       # noqa: E731
    n, R, at = sum(lengths), len(lengths), H * (2 * dk + dv)
    wide, ib, fb, m0 = rand(n, at + 2 * H + 2) * 3, rand(H), rand(H) + 2, rand(R, H)
    short, long, chunks, requests = tables(lengths, first_chunked)
    state, m, gates = torch.zeros(R, H, dk, ops.mlstm_padded(dv), device=DEV), m0.clone(), torch.full((n, H, 3), 7.0, device=DEV)
    out = torch.empty(n, H * ops.mlstm_padded(dv), device=DEV)
    ops.mlstm_scan(wide[:, :H * dk], wide[:, H * dk:2 * H * dk], wide[:, 2 * H * dk:at], wide[:, at:at + H], wide[:, at + H:at + 2 * H], ib, fb,
                   short, state, m, out, gates, H, dk, dv, cap, 0.5, long_segments=long, chunks=chunks, requests=requests, most_rows=max(lengths))
    soft = lambda x: cap * torch.tanh(x.double() / cap)              # noqa: E731
    i, f = soft(wide[:, at:at + H] + ib), torch.nn.functional.logsigmoid(soft(wide[:, at + H:at + 2 * H] + fb))
    row = 0
    for r, count in enumerate(lengths):
        top = m0[r].double()
        for t in range(row, row + count):
            new = torch.maximum(f[t] + top, i[t])
            want = torch.stack([torch.exp(f[t] + top - new), torch.exp(i[t] - new), torch.exp(-new)], dim=1)
            # exponents of up to 2 cap and a sum of up to 129 terms, each rounded in float32
            assert bool(((gates[t].double() - want).abs() <= 5e-5 * want + 1e-30).all())
            top = new
        assert bool(((m[r].double() - top).abs() <= 5e-5 * (1 + top.abs())).all())
        row += count


def test_more_walked_requests_than_a_grid_is_high():
    lengths = [1] * 65536 + [64]
    t = inputs("general", 1, 4, 4, lengths, torch.Generator(DEV).manual_seed(3))
    same(scan("general", 1, 4, 4, lengths, t, 65536), scan("general", 1, 4, 4, lengths, t, len(lengths)))


@pytest.mark.parametrize("kind", ["general", "gated", "retention", "memory"])
@pytest.mark.parametrize("dk,dv", [(64, 68), (60, 64), (8, 72), (64, 128)])
def test_value_columns_around_a_pass(kind, dk, dv):
    """One, two and three passes over the value columns, the last of them with columns that a pass of 64 leaves over."""
    lengths = [33, 100]
    t = inputs(kind, 3, dk, dv, lengths, torch.Generator(DEV).manual_seed(dk * dv))
    same(*(scan(kind, 3, dk, dv, lengths, t, first) for first in (0, len(lengths))))


@pytest.mark.parametrize("kind", ["general", "gated", "retention", "memory"])
@pytest.mark.parametrize("at", [0, 17, 40])
def test_the_largest_finite_values_reach_no_earlier_token(kind, at):
    """A value that bfloat16 would round to infinity, at a token with a small key: the bits of the tokens before it as without it, and
    finite everywhere as in the walk (the generalised rule divides by a chunk's decays, which leaves it no room there)."""
    H, d, lengths = 2, 64, [70]
    t = inputs(kind, H, d, d, lengths, torch.Generator(DEV).manual_seed(at))
    K = H * d
    t["proj"][at, K:2 * K] *= 1e-2
    clean, _ = scan(kind, H, d, d, lengths, t, 0)
    t["proj"][at, 2 * K + 5] = 3.4e38
    got, want = (scan(kind, H, d, d, lengths, t, first) for first in (0, len(lengths)))
    assert torch.equal(got[0][:at], clean[:at]) and all(bool(torch.isfinite(x).all()) for x in want)
    if kind != "general":
        same(got, want)
