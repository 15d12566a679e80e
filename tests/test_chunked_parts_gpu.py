"""The recurrent mixers that take long portions in chunks, as parts: the same requests in the same steps, in chunks and walked token by
token, over steps that change between the two, with short requests beside; every row's result and every state, the convolution's
tail and the matrix memory's maxima among them."""
import pytest
import torch

from test_parts_gpu import bind_random, make_ctx

pytestmark = pytest.mark.gpu
D = 128


def part_of(kind):
    from hk_b200.parts import MLSTM, GatedDeltaRule, GeneralDeltaRule, Retention, RotaryEmbedding
    if kind == "delta":
        return GeneralDeltaRule(D, 3, 64, "m.", norm_eps=1e-5, decay_rank=16)
    if kind == "gated":
        return GatedDeltaRule(D, 4, 2, 32, 64, 4, "m.", norm_eps=1e-6)
    if kind == "retention":
        return Retention(D, 2, 64, 36, [0.9, 0.99], "m.", 1e-6, position=RotaryEmbedding(5e5, 32, 1024))
    return MLSTM(D, 2, 64, 64, 15.0, "m.", norm_eps=1e-6)


# what every request brings to a step: long ones beside short ones, then all walked, then in chunks again, then single tokens
STEPS = [[200, 5, 97, 1], [40, 63, 1, 2], [65, 30, 0, 130], [1, 1, 1, 1], [0, 96, 64, 0], [1, 1, 1, 1]]
CHUNKED = [[200, 97], [], [65, 130], [], [96, 64], []]


@pytest.mark.parametrize("kind", ["delta", "gated", "retention", "mlstm"])
def test_steps_in_chunks_and_walked(kind):
    from hk_b200.cache.device import PagedCache
    from hk_b200.parts.parallel import mixer_cache_specs, mixer_caches
    part = part_of(kind)
    prec, _ = bind_random(part, torch.bfloat16, std=0.08)
    assert part._chunks
    requests = len(STEPS[0])
    inputs = [[torch.randn(n, D, device="cuda").bfloat16() for n in step] for step in STEPS]

    def walk(longest_from):
        part.LONGEST_FROM, part.ROWS_FROM, part.BESIDE = longest_from, 1 << 40, 1 << 20
        cache = PagedCache([mixer_cache_specs(part)], prec, 16, 16 * requests, requests, 1024)
        slots, at, results = [cache.open() for _ in range(requests)], [0] * requests, []
        for step, rows in zip(STEPS, inputs):
            who = [r for r in (2, 0, 3, 1) if step[r]]
            ctx = make_ctx(prec, [(slots[r], at[r], step[r]) for r in who], cache, page_tokens=16, part=part)
            x = torch.cat([rows[r] for r in who])
            y = torch.full((x.shape[0], D), float("nan"), device="cuda")
            part.forward(x, y, ctx, mixer_caches(part, cache.layers[0]), accumulate=False)
            chunked = ctx.tables[part.step_tables_key()][0]["long"][:, 2].tolist()
            results.append((y, [c.state[slots].clone() for c in cache.layers[0]], sorted(chunked)))
            for r in who:
                at[r] += step[r]
        return results
    got, want = walk(64), walk(1 << 30)
    for i, ((y, states, chunked), (y0, states0, none)) in enumerate(zip(got, want)):
        assert chunked == sorted(CHUNKED[i]) and none == []
        assert bool(torch.isfinite(y).all())
        # float32 rounding in the scan moves a bfloat16 factor of the last product here and there: a few units of 2^-8
        assert float((y - y0).norm() / y0.norm()) <= 2e-3 and float((y - y0).abs().max()) <= 2e-2 * float(y0.abs().max())
        for a, b in zip(states, states0):
            assert float((a - b).abs().max()) <= 6e-5 * max(1.0, float(b.abs().max())), f"step {i}"      # float32 rounding of both
