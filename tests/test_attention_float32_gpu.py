"""The float32 kernel over runs of tokens (`hk_attention_f32`) against the kernel of a block per token and head, which holds the plain reference:
every option of the scores, head and value sizes inside its tile, groups that do not divide its rows, runs at its edges, cached
keys, pages of odd sizes, several requests."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H,G,hd,vd,pt,spans,options", [
    (4, 2, 128, 128, 16, [(0, 130)], {}), (16, 8, 128, 128, 16, [(0, 65), (63, 16), (0, 1), (200, 33)], {}),
    (3, 3, 40, 40, 5, [(0, 64), (7, 63)], {"window": 20}), (6, 2, 64, 64, 7, [(100, 129)], {"window": 1}),
    (5, 1, 4, 8, 3, [(2, 31), (0, 9)], {"softcap": 3.0}), (32, 1, 72, 128, 16, [(0, 40)], {"sink": True}),
    (6, 2, 128, 64, 16, [(30, 90)], {"sink": True, "sinks": True, "chunk": 48}), (4, 4, 128, 128, 16, [(0, 70), (5, 20)], {"gate": True}),
    (8, 2, 64, 128, 16, [(0, 150)], {"dist": 17, "softcap": 10.0}), (7, 7, 100, 36, 16, [(33, 95)], {"dist": 1, "window": 70}),
    (2, 1, 96, 40, 16, [(0, 64)], {"one_tensor": True}),
])
def test_float32_runs_match_the_kernel_of_a_block_per_head(H, G, hd, vd, pt, spans, options):
    from hk_b200.csrc import ops
    g = torch.Generator(DEV).manual_seed(H * 100 + hd + vd)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)       # noqa: E731
    per = max(-(-(c + n) // pt) for c, n in spans)
    pages = per * len(spans) + 2
    order = np.random.default_rng(hd).permutation(pages)[:per * len(spans)].astype(np.int32).reshape(len(spans), per)
    table = torch.from_numpy(order).to(DEV).contiguous()
    k = rand(pages, G, pt, hd)
    v = None if options.get("one_tensor") else rand(pages, G, pt, vd)
    n = sum(c for _, c in spans)
    pos = torch.cat([torch.arange(p, p + c) for p, c in spans]).int().to(DEV)
    slot = torch.cat([torch.full((c,), i) for i, (_, c) in enumerate(spans)]).int().to(DEV)
    q, gate = rand(n, H * hd), rand(n, H * vd + 8)[:, 4:4 + H * vd]
    more = {"sink": bool(options.get("sink")), "sinks": rand(H) if options.get("sinks") else None, "softcap": options.get("softcap", 0.0),
            "chunk": options.get("chunk", 0), "gate": gate if options.get("gate") else None, "gate_scale": 0.7,
            "dist": rand(H, options["dist"]) if options.get("dist") else None}
    starts = np.cumsum([0] + [c for _, c in spans[:-1]]).tolist()
    runs = ops.float32_runs(range(len(spans)), starts, [c for _, c in spans], [p for p, _ in spans], H // G)
    assert runs[:, 1].sum() == n and runs[:, 1].max() <= 32 // (H // G)
    got, want = torch.full((n, H * vd), float("nan"), device=DEV), torch.empty(n, H * vd, device=DEV)
    args = (q, k, v, table, pos, slot)
    sizes = (H, G, hd, pt, options.get("window", 0), hd ** -0.5)
    ops.paged_attention(*args, want, *sizes, **more)
    before = ops.launch_count()
    ops.paged_attention(*args, got, *sizes, runs=torch.from_numpy(runs).to(DEV), **more)
    assert ops.launch_count() == before + 1
    alone = torch.empty_like(got)           # token by token: the same bits
    single = np.asarray([(r, 1, s, p) for r, (s, p) in enumerate(zip(slot.tolist(), pos.tolist()))], dtype=np.int32)
    ops.paged_attention(*args, alone, *sizes, runs=torch.from_numpy(single).to(DEV), **more)
    assert torch.equal(alone, got)
    worst = float((got - want).abs().max() / want.abs().max())
    assert worst <= 1e-5, f"{worst:.3g} of the largest value"      # sums of up to 300 keys and 128 dims in other orders


def test_groups_that_the_kernel_does_not_take():
    from hk_b200.csrc import ops
    assert ops.float32_runs([0], [0], [40], [0], 33) is None
    assert ops.float32_runs([2], [3], [9], [4], 8).tolist() == [[11, 1, 2, 12], [7, 4, 2, 8], [3, 4, 2, 4]]
