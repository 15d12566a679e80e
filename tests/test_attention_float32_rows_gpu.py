"""The float32 attention over runs of tokens beside rows that are NaN or Inf: a row's result is that of the kernel of a block per
token and head, which reads what the row sees alone."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H,G,hd,vd,spans,window,chunk", [
    (4, 2, 64, 64, [(0, 130)], 0, 0), (16, 8, 128, 128, [(0, 65), (63, 16), (0, 1), (200, 33)], 0, 0), (2, 2, 40, 72, [(0, 64), (7, 163)], 20, 0),
    (6, 2, 128, 64, [(30, 90)], 0, 48), (32, 1, 72, 128, [(0, 40), (64, 3)], 20, 0),
])
@pytest.mark.parametrize("spoil", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["values", "keys", "both"])
def test_rows_that_are_not_finite_reach_who_sees_them(H, G, hd, vd, spans, window, chunk, spoil, where):
    from hk_b200.csrc import ops
    g = torch.Generator(DEV).manual_seed(H * 100 + hd + vd)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)       # noqa: E731
    pt = 8
    per = max(-(-(c + n) // pt) for c, n in spans)
    table = torch.from_numpy(np.random.default_rng(hd).permutation(per * len(spans)).astype(np.int32).reshape(len(spans), per)).to(DEV)
    k, v = rand(per * len(spans), G, pt, hd), rand(per * len(spans), G, pt, vd)
    for slot, (c, n) in enumerate(spans):       # a few columns of a position inside, of the last, and of one that a window leaves behind
        for p in {c + n // 2, c + n - 1} | ({c // 2} if window or chunk else set()):
            page = int(table[slot, p // pt])
            if where != "keys":
                v[page, :, p % pt, 1::5] = spoil
            if where != "values":
                k[page, :, p % pt, 2] = float("nan")
    n = sum(c for _, c in spans)
    pos = torch.cat([torch.arange(p, p + c) for p, c in spans]).int().to(DEV)
    slot = torch.cat([torch.full((c,), i) for i, (_, c) in enumerate(spans)]).int().to(DEV)
    starts = np.cumsum([0] + [c for _, c in spans[:-1]]).tolist()
    runs = ops.float32_runs(range(len(spans)), starts, [c for _, c in spans], [p for p, _ in spans], H // G)
    args, sizes = (rand(n, H * hd), k, v, table, pos, slot), (H, G, hd, pt, window, hd ** -0.5)
    got, want = torch.full((n, H * vd), 7.0, device=DEV), torch.empty(n, H * vd, device=DEV)
    ops.paged_attention(*args, want, *sizes, chunk=chunk)
    before = ops.launch_count()
    ops.paged_attention(*args, got, *sizes, chunk=chunk, runs=torch.from_numpy(runs).to(DEV))
    assert ops.launch_count() == before + 1
    finite = torch.isfinite(want)
    assert 0 < int(finite.sum()) < finite.numel() and torch.equal(torch.isfinite(got), finite)
    worst = float((got - want)[finite].abs().max() / want[finite].abs().max())
    assert worst <= 1e-5, f"{worst:.3g} of the largest value"      # sums of up to 230 keys and 128 dims in other orders
