"""Latent attention with keys and values made for a step (`LatentAttention._forward_made`) against the same part in the latent space
and, whole prompts, against the plain implementation: tile edges, several requests, rows in the cache before, windows, both kinds
of gate, a query latent, no rotated part, and requests of both kinds in one step."""
import numpy as np
import pytest
import torch

import plain_padodra as K
from test_parts_gpu import bind_random, make_ctx

pytestmark = pytest.mark.gpu


def part_of(H, dr, r, window=None, gate=True, q_rank=None):
    from hk_b200.parts import LatentAttention, RotaryEmbedding
    rope = RotaryEmbedding(10000.0, dr, 4096) if dr else None
    return LatentAttention(192, H, 128, dr, 128, r, "m.", 1e-6, (128 + dr) ** -0.5, position=rope, gate=gate, window=window, q_rank=q_rank,
                           out_scale=0.5 if gate else 1.0)


def run(part, prec, rows, spans, made_from):
    """The part's result for the spans' new rows; `rows` [request][cached + new, d]."""
    from hk_b200.cache.device import PagedCache
    part.MADE_FROM, part.MADE_BESIDE = made_from, 0
    cache = PagedCache([[part.cache_spec()]], prec, 16, sum(-(-(c + n) // 16) for c, n in spans), len(spans), 4096)
    slots = [cache.open() for _ in spans]

    def step(which):
        ctx = make_ctx(prec, which, cache, page_tokens=16, part=part)
        x = torch.cat([rows[s][p:p + n] for s, p, n in [(slots.index(s), p, n) for s, p, n in which]])
        y = torch.full((x.shape[0], part.hidden), float("nan"), device="cuda")
        part.forward(x, y, ctx, cache.layers[0][0], accumulate=False)
        return y, ctx
    for s, (c, _) in zip(slots, spans):
        if c:
            step([(s, 0, c)])
    return step([(s, c, n) for s, (c, n) in zip(slots, spans)])


@pytest.mark.parametrize("H,dr,r,window,gate,q_rank,spans", [
    (2, 64, 512, None, True, None, [(0, 64)]), (3, 64, 256, None, True, None, [(0, 127), (0, 129)]),
    (2, 64, 512, None, True, None, [(0, 256), (0, 257), (0, 383)]),
    (2, 64, 128, None, False, None, [(37, 70), (200, 128), (1, 300)]),         # rows in the cache before
    (2, 64, 512, 50, True, None, [(300, 90), (0, 200)]), (2, 0, 512, 130, True, None, [(700, 129)]),
    (4, 64, 512, 64, "head", 96, [(100, 256), (0, 64)]), (2, 0, 256, None, "head", None, [(0, 300)]),
    (2, 64, 512, None, True, None, [(0, 200), (63, 1), (900, 1), (5, 40)]),    # both kinds in one step, single tokens among them
    (2, 64, 512, None, True, None, [(77, 1), (30, 1), (0, 65), (12, 90)]), (2, 64, 512, 7, True, None, [(3, 70), (15, 64), (16, 64)]),
])
def test_made_keys_and_values_match_the_latent_space(H, dr, r, window, gate, q_rank, spans):
    torch.manual_seed(H * 1000 + dr + r)
    part = part_of(H, dr, r, window, gate, q_rank)
    prec, w = bind_random(part, torch.bfloat16, std=0.08)
    rows = [torch.randn(c + n, 192, device="cuda").to(torch.bfloat16) for c, n in spans]
    from hk_b200.csrc import gemm_fast
    from hk_b200.parts.latent_attention import LatentInfo
    want, ctx = run(part, prec, rows, spans, 1 << 30)
    assert not isinstance(ctx.tables[part.step_tables_key()][1], LatentInfo)
    got, ctx = run(part, prec, rows, spans, 64)
    assert isinstance(ctx.tables[part.step_tables_key()][1], LatentInfo)
    gemm_fast.check_status(torch.device("cuda", 0))
    scale = float(want.abs().max())
    assert bool(torch.isfinite(got).all()) and float((got - want).abs().max()) <= 3e-2 * scale      # as other bfloat16 parts: 8-bit factors
    if window is None and gate is True and q_rank is None and dr and all(c == 0 for c, _ in spans):
        m = {"heads": H, "dim": 128, "rot_dim": dr, "vdim": 128, "kv_rank": r, "scale": part.scale,
             "rot": {"base": 10000.0, "dims": dr, "scaling": {"factor": 1.0, "fast": 32.0, "slow": 1.0, "original": 4096}}}
        plain = np.concatenate([K.latent_attention(x.double().cpu().numpy(), w, "m.", m, 1e-6) for x in rows])
        # out_scale 0.5 rides on the gate
        assert np.abs(got.double().cpu().numpy() - 0.5 * plain).max() <= 3e-2 * np.abs(0.5 * plain).max()


def test_requests_that_see_too_many_rows_stay_in_the_latent_space():
    from hk_b200.csrc import attention_fast
    part = part_of(2, 64, 512)
    prec, _ = bind_random(part, torch.bfloat16, std=0.08)
    ctx = make_ctx(prec, [(0, 64 * 16, 64)], part=part)
    assert "made_items" not in ctx.tables[part.step_tables_key()][0]
    ctx = make_ctx(prec, [(0, 64 * 15, 64)], part=part)
    assert "made_items" in ctx.tables[part.step_tables_key()][0]
    items, segments, firsts, rows = attention_fast.made_items([3, 1, 2], [0, 300, 310], [300, 10, 70], [0, 90, 9], 20)
    assert firsts.tolist() == [[0, 0, 0, 16], [310, 329, 9, 7]]
    items, segments, firsts, rows = attention_fast.made_items([3, 1], [0, 300], [300, 10], [0, 90], 20)
    assert rows == 300 + 29 and segments.tolist() == [[3, 0, 300, 0], [1, 71, 29, 300]]
    assert [i[:6] for i in items.tolist()] == [[0, 256, 0, 0, 0, 256], [256, 44, 0, 256, 237, 300], [300, 10, 229, 90, 71, 100]]
