"""The two kernels over keys and values made for a step (`attention_fast.run_made`), on arrays whose every row outside a request's
own is NaN: against the softmax in float64, windows shorter than a request's first rows among them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
H, R, DR, GUARD = 2, 64, 64, 256


def made_case(spans, window, layout, seed=0):
    """(out of `run_made`, the same in float64, positions): spans (cached, new) of requests whose rows lie as `layout` says."""
    from hk_b200.csrc import attention_fast, gemm_fast
    g = torch.Generator(DEV).manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)       # noqa: E731
    lens, starts = [n for _, n in spans], [c for c, _ in spans]
    q_starts = np.cumsum([0] + lens[:-1]).tolist()
    items, segments, firsts, rows = layout(list(range(len(spans))), q_starts, lens, starts, window)

    def guarded(width):
        """A matrix of `rows` rows, NaN, inside one with NaN on both sides."""
        return torch.full((GUARD + rows + GUARD, width), float("nan"), dtype=torch.bfloat16, device=DEV)[GUARD:GUARD + rows]
    c, rope, kv = guarded(R), guarded(DR), guarded(H * 256)
    w = (rand(H, 256, R) * R ** -0.5).bfloat16()
    n = sum(lens)
    q, want, pos = (rand(n, H * 192) * 0.5).bfloat16(), torch.empty(n, H, 128, dtype=torch.float64), []
    for (_, first, count, row0), qs, ql, p0 in zip(segments.tolist(), q_starts, lens, starts):
        part = slice(row0, row0 + count)
        c[part], rope[part] = rand(count, R).bfloat16(), rand(count, DR).bfloat16()
        kv[part] = (c[part].float() @ w.float().flatten(0, 1).t()).bfloat16()
        keys = torch.cat([kv[part].view(count, H, 256)[..., :128], rope[part][:, None].expand(count, H, DR)], dim=2).double()
        values = torch.einsum("tr,hvr->thv", c[part].double(), w[:, 128:].double())
        for i in range(ql):
            p, lo = p0 + i, max(0, p0 + i - window + 1) if window else 0
            see = slice(lo - first, p + 1 - first)
            s = torch.einsum("hd,thd->ht", q[qs + i].view(H, 192).double(), keys[see]) * 192 ** -0.5
            want[qs + i] = torch.einsum("ht,thv->hv", torch.softmax(s, dim=1), values[see]).cpu()
            pos.append(p)
    out = torch.full((n, H * 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    attention_fast.run_made(q, kv, rope, torch.from_numpy(items).to(DEV), out, H, window, 192 ** -0.5, c, w[:, 128:].contiguous(),
                            torch.from_numpy(firsts).to(DEV))
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
