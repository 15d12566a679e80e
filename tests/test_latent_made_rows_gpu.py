"""The two kernels over keys and values made for a step (`attention_fast.run_made`), on arrays whose every row outside a request's
own is NaN: against the softmax in float64, windows shorter than a request's first rows among them.  And what a row of the cache that
holds NaN or Inf does to other requests of the step, and to rows of its own request that do not see it: nothing."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
H, R, DR, GUARD = 2, 64, 64, 256


def made_case(spans, window, layout, seed=0, tile=1, spoilt=(), spoil=float("nan"), gate=None, dr=DR):
    """(out of `run_made`, the same in float64, positions): spans (cached, new) of requests whose rows lie as `layout` says, the rest
    of their tiles zeros; `spoilt` = (request, row of its own) whose cache row and values are `spoil`."""
    from hk_b200.csrc import attention_fast, gemm_fast
    g = torch.Generator(DEV).manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)       # noqa: E731
    lens, starts = [n for _, n in spans], [c for c, _ in spans]
    q_starts = np.cumsum([0] + lens[:-1]).tolist()
    items, segments, firsts, rows = layout(list(range(len(spans))), q_starts, lens, starts, window)

    def guarded(width):
        """A matrix of `rows` rows, NaN, inside one with NaN on both sides."""
        return torch.full((GUARD + rows + GUARD, width), float("nan"), dtype=torch.bfloat16, device=DEV)[GUARD:GUARD + rows]
    c, rope, kv = guarded(R), guarded(dr), guarded(H * 256)
    w = (rand(H, 256, R) * R ** -0.5).bfloat16()
    n = sum(lens)
    q, want, pos = (rand(n, H * (128 + dr)) * 0.5).bfloat16(), torch.empty(n, H, 128, dtype=torch.float64), []
    for (_, first, count, row0), qs, ql, p0 in zip(segments.tolist(), q_starts, lens, starts):
        part, whole = slice(row0, row0 + count), slice(row0 // tile * tile, -(-(row0 + count) // tile) * tile)
        c[whole], rope[whole], kv[whole] = 0.0, 0.0, 0.0
        c[part], rope[part] = rand(count, R).bfloat16(), rand(count, dr).bfloat16()
        kv[part] = (c[part].float() @ w.float().flatten(0, 1).t()).bfloat16()
        keys = torch.cat([kv[part].view(count, H, 256)[..., :128], rope[part][:, None].expand(count, H, dr)], dim=2).double()
        values = torch.einsum("tr,hvr->thv", c[part].double(), w[:, 128:].double())
        for i in range(ql):
            p, lo = p0 + i, max(0, p0 + i - window + 1) if window else 0
            see = slice(lo - first, p + 1 - first)
            s = torch.einsum("hd,thd->ht", q[qs + i].view(H, 128 + dr).double(), keys[see]) * 192 ** -0.5
            want[qs + i] = torch.einsum("ht,thv->hv", torch.softmax(s, dim=1), values[see]).cpu()
            pos.append(p)
    for request, own in spoilt:
        c[segments[request][3] + own], kv[segments[request][3] + own] = spoil, spoil
    out = torch.full((n, H * 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    logits = rand(n, H if gate == "head" else H * 128) if gate else None
    if gate:
        want *= 0.7 * torch.sigmoid(logits.double().cpu().view(n, H, -1))
    attention_fast.run_made(q, kv, rope if dr else None, torch.from_numpy(items).to(DEV), out, H, window, 192 ** -0.5, c, w[:, 128:].contiguous(),
                            torch.from_numpy(firsts).to(DEV), logits, gate == "head", 0.7)
    gemm_fast.check_status(torch.device(DEV, 0))
    return out.double().cpu().view(n, H, 128), want, np.asarray(pos)


@pytest.mark.parametrize("span,window", [((12, 70), 8), ((15, 64), 7), ((3, 64), 1), ((15, 300), 15), ((5, 64), 16), ((0, 70), 7)])
def test_a_window_that_leaves_out_the_first_positions(span, window):
    """The request is the step's first: the place of its position 0 may lie before the arrays."""
    from hk_b200.csrc import attention_fast
    got, want, pos = made_case([span], window, attention_fast.made_items)
    scale = float(want.abs().max())
    assert bool(torch.isfinite(got).all()) and float((got - want).abs().max()) <= 3e-2 * scale      # probabilities and values in bfloat16
    # the first positions: values that are never rounded, so half a unit of the result and float32 sums
    early = pos < attention_fast.MADE_FIRST
    assert bool(((got - want).abs()[early] <= 2.0 ** -8 * want.abs()[early] + 1e-4 * scale).all())


def tiled(*args):
    from hk_b200.csrc import attention_fast
    return attention_fast.made_items(*args, attention_fast.MADE_TILE)


NEIGHBOURS = [([(0, 70), (0, 200), (0, 65)], 0), ([(0, 129), (37, 127), (200, 300)], 0), ([(300, 90), (0, 257), (5, 64)], 50),
              ([(700, 129), (15, 64), (140, 70)], 130), ([(15, 64), (16, 64), (3, 70)], 7)]


@pytest.mark.parametrize("spans,window", NEIGHBOURS)
@pytest.mark.parametrize("spoil", [float("nan"), float("inf")])
def test_a_request_that_is_not_finite_leaves_the_others_alone(spans, window, spoil):
    clean, want, _ = made_case(spans, window, tiled, tile=128)
    scale = float(want.abs().max())
    assert float((clean - want).abs().max()) <= 3e-2 * scale       # probabilities and values in bfloat16
    ends = np.cumsum([n for _, n in spans]).tolist()
    for bad, (cached, n) in enumerate(spans):
        rows = cached + n - max(0, cached - window + 1 if window else 0)
        got, _, _ = made_case(spans, window, tiled, tile=128, spoilt=[(bad, i) for i in range(rows)], spoil=spoil)
        own = slice(ends[bad] - n, ends[bad])
        assert not bool(torch.isfinite(got[own]).any())
        got[own] = clean[own]
        assert torch.equal(got, clean)


@pytest.mark.parametrize("spans,window", NEIGHBOURS)
def test_neighbours_in_a_step_of_the_part(spans, window):
    """The same through `LatentAttention`: a request whose inputs are NaN and Inf, the others' results equal to the bit."""
    from test_latent_made_gpu import part_of, run
    from test_parts_gpu import bind_random
    part = part_of(2, 64, 512, window or None)
    prec, _ = bind_random(part, torch.bfloat16, std=0.08)
    rows = [torch.randn(c + n, 192, device=DEV).to(torch.bfloat16) for c, n in spans]
    clean, _ = run(part, prec, rows, spans, 64)
    assert bool(torch.isfinite(clean).all())
    ends = np.cumsum([n for _, n in spans]).tolist()
    for bad, (_, n) in enumerate(spans):
        spoilt = [x.clone() for x in rows]
        spoilt[bad][::2], spoilt[bad][1::2] = float("nan"), float("inf")
        got, _ = run(part, prec, spoilt, spans, 64)
        own = slice(ends[bad] - n, ends[bad])
        assert not bool(torch.isfinite(got[own]).any())
        got[own] = clean[own]
        assert torch.equal(got, clean)


@pytest.mark.parametrize("tile", [1, 128])
@pytest.mark.parametrize("dr", [0, 8])
def test_latent_rows_fill_up_their_tiles(tile, dr):
    from hk_b200.csrc import attention_fast, ops
    spans, r, pt = [(0, 127), (300, 90), (130, 129), (5, 123), (0, 128)], 16, 16
    per = 32
    pages = torch.randn(per * len(spans), 1, pt, r + dr, device=DEV).bfloat16()
    table = torch.randperm(per * len(spans)).int().view(len(spans), per).to(DEV)
    lens = [n for _, n in spans]
    _, segments, _, rows = attention_fast.made_items(range(len(spans)), np.cumsum([0] + lens[:-1]).tolist(), lens, [c for c, _ in spans], 50, tile)
    c = torch.full((rows, r), float("nan"), dtype=torch.bfloat16, device=DEV)
    rope = torch.full((rows, dr), float("nan"), dtype=torch.bfloat16, device=DEV) if dr else None
    ops.latent_rows(pages, table, torch.from_numpy(segments).to(DEV), int(segments[:, 2].max()), c, rope, tile)
    want = torch.zeros(rows, r + dr, dtype=torch.bfloat16, device=DEV)
    for slot, first, count, row in segments.tolist():
        pos = torch.arange(first, first + count, device=DEV)
        want[row:row + count] = pages[table[slot, pos // pt].long(), 0, pos % pt]
    assert torch.equal(torch.cat([c, rope], dim=1) if dr else c, want)


@pytest.mark.parametrize("spans,window,gate,dr", [([(0, 70)], 0, None, 64), ([(0, 300), (37, 127)], 0, "each", 64), ([(300, 90), (0, 257)], 50, "head", 64),
                                                  ([(15, 64), (3, 400)], 7, "each", 0), ([(0, 129)], 0, "head", 0)])
@pytest.mark.parametrize("at", [0.0, 0.04, 0.5, 1.0])
def test_rows_that_see_only_finite_rows_stay_finite(spans, window, gate, dr, at):
    """One position of every request holds NaN: the rows before it, and those that it has left the window of, are as they were."""
    places = [min(cached + n - 1, (max(0, cached - window + 1) if window else 0) + int(at * (cached + n))) for cached, n in spans]
    spoilt = [(i, p - (max(0, cached - window + 1) if window else 0)) for i, (p, (cached, _)) in enumerate(zip(places, spans))]
    got, want, pos = made_case(spans, window, tiled, tile=128, spoilt=spoilt, gate=gate, dr=dr)
    place = np.concatenate([np.full(n, p) for p, (_, n) in zip(places, spans)])
    sees = torch.from_numpy((place <= pos) & ((place > pos - window) if window else True))
    scale = float(want.abs().max())
    assert not bool(torch.isfinite(got[sees]).any()) and bool(torch.isfinite(got[~sees]).all())
    assert bool(((got - want).abs()[~sees] <= 3e-2 * scale).all())       # probabilities and values in bfloat16


@pytest.mark.parametrize("spans", [[(0, 64)], [(3, 70), (0, 200), (15, 64)]])
def test_values_of_the_first_positions_are_never_rounded(spans):
    """The first positions' results are off by half a unit of themselves and float32 sums; values in bfloat16 would show."""
    from hk_b200.csrc import attention_fast
    got, want, pos = made_case(spans, 0, tiled, tile=128)
    scale, early = float(want.abs().max()), pos < attention_fast.MADE_FIRST
    off = (got - want).abs() - 2.0 ** -8 * want.abs()
    assert bool((off[early] <= 1e-4 * scale).all())
    assert bool((off[~early] > 1e-4 * scale).any())         # (as later ones do)


def test_sizes_that_the_host_shares_with_the_kernels():
    from hk_b200.csrc import attention_fast, build, ops
    made, first, runs = build.load("attention_prefill_tc"), build.load("attention_latent"), build.load("attention_generic")
    assert made.hk_attention_made_tile() == attention_fast.MADE_TILE and made.hk_attention_made_tokens() == attention_fast.MADE_TOKENS
    assert first.hk_latent_first_rows_count() == attention_fast.MADE_FIRST
    assert [runs.hk_attention_f32_tokens(g) for g in (1, 3, 32, 33)] == [ops.RUN_ROWS, ops.RUN_ROWS // 3, 1, 0]


@pytest.mark.parametrize("rank", [8, 72, 504, 512, 520, 1000, 1032])
def test_first_rows_of_any_rank(rank, monkeypatch):
    """Fewer pieces of a latent row than the block has warps, a number that does not divide, one to three stagings of the
    weights."""
    from hk_b200.csrc import attention_fast
    monkeypatch.setitem(made_case.__globals__, "R", rank)
    got, want, pos = made_case([(0, 70), (3, 40)], 0, tiled, tile=128)
    scale, early = float(want.abs().max()), pos < attention_fast.MADE_FIRST
    assert bool(torch.isfinite(got).all()) and float((got - want).abs().max()) <= 3e-2 * scale
    assert bool(((got - want).abs()[early] <= 2.0 ** -8 * want.abs()[early] + 1e-4 * scale).all())
