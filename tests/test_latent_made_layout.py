"""Where the rows of requests lie whose keys and values are made for a step (`attention_fast.made_items`)."""
import random

import pytest


@pytest.mark.parametrize("window", [0, 1, 7, 15, 16, 50, 128, 130, 1000])
def test_a_tile_holds_one_requests_rows(window):
    from hk_b200.csrc import attention_fast
    T = attention_fast.MADE_TILE
    rng = random.Random(window)
    for _ in range(200):
        n = rng.randrange(1, 6)
        lens = [rng.choice([64, 127, 128, 129, rng.randrange(64, 600)]) for _ in range(n)]
        starts = [rng.choice([0, 3, 12, 15, 16, 127, 128, rng.randrange(900)]) for _ in range(n)]
        q_starts = [sum(lens[:i]) for i in range(n)]
        items, segments, firsts, rows = attention_fast.made_items(range(n), q_starts, lens, starts, window, T)
        own, free = {}, 0
        for (slot, first, count, row), ql, p0 in zip(segments.tolist(), lens, starts):
            assert first == (max(0, p0 - window + 1) if window else 0) and first + count == p0 + ql
            lo, hi = row // T * T, -(-(row + count) // T) * T
            assert lo == free                   # whole tiles, side by side
            own[slot], free = (lo, hi, row - first), hi
        assert free == rows
        request = {q + i: s for s, (q, ql) in enumerate(zip(q_starts, lens)) for i in range(ql)}
        for q_row, count, base, pos0, lo, hi, _, _ in items.tolist():
            r0, r1, base0 = own[request[q_row]]
            assert base == base0 and base % T == 0 and r0 <= base + lo // T * T and base + -(-hi // T) * T <= r1
        for q_row, base, pos0, count in firsts.tolist():
            # the rows that the kernel of a request's first positions reads: those that its own window leaves
            r0, r1, base0 = own[request[q_row]]
            first = max(0, pos0 - window + 1) if window else 0
            assert base == base0 and r0 <= base + first and base + pos0 + count <= r1 and pos0 + count <= attention_fast.MADE_FIRST


def test_rows_side_by_side_without_tiles():
    """Without tiles the place of a request's position 0 may lie before the arrays: only the positions that its window leaves are there."""
    from hk_b200.csrc import attention_fast
    _, segments, firsts, rows = attention_fast.made_items([0], [0], [70], [12], 8)
    assert firsts.tolist() == [[0, -5, 12, 4]] and segments.tolist() == [[0, 5, 77, 0]] and rows == 77
    _, segments, firsts, rows = attention_fast.made_items([0], [0], [70], [12], 8, 128)
    assert firsts.tolist() == [[0, 0, 12, 4]] and segments.tolist() == [[0, 5, 77, 5]] and rows == 128


def latent_part(H=32):
    from hk_b200.parts import LatentAttention
    part = LatentAttention(4096, H, 128, 64, 128, 512, "m.", 1e-6, 192 ** -0.5)
    part._w_ukv, part._wide, part._sm_count, part._tables_key = True, True, 148, ("latent",)      # as bound in bfloat16
    return part


@pytest.mark.parametrize("spans,stays", [
    ([(30000, 2048)], []), ([(50000, 4096)], []), ([(120000, 8192)], [0]), ([(60000, 4000), (0, 4096)], [0]), ([(0, 100000)], []),
    ([(30000, 2100), (20000, 1500), (15000, 1100)], [0]), ([(0, 64)] * 3, [])])
def test_what_a_step_makes_is_bounded(spans, stays):
    """The arrays of a step stay below MADE_SCRATCH or what the latent space would take; what does not fit stays there."""
    from types import SimpleNamespace
    part, T = latent_part(), 128
    lens, starts = [n for _, n in spans], [c for c, _ in spans]
    ctx = SimpleNamespace(slots=list(range(len(spans))), q_starts=[sum(lens[:i]) for i in range(len(lens))], q_lens=lens, start_positions=starts,
                          n_tokens=sum(lens), fixed_shape=False, max_context=200000, page_tokens=16)
    tables = part._made_tables(ctx)
    if len(stays) == len(spans):
        assert tables is None
        return
    kept = sorted(tables.arrays["made_segments"][:, 0].tolist())
    assert kept == [i for i in range(len(spans)) if i not in stays]
    n = sum(lens[i] for i in kept)
    made = 2 * (n * 32 * 192 + tables.info.rows * (576 + 32 * 256))
    assert made <= max(part.MADE_SCRATCH, 2 * n * 32 * (128 + 576 + 512))
    # without the bound they would all have been made
    part.MADE_SCRATCH = 1 << 50
    assert sorted(part._made_tables(ctx).arrays["made_segments"][:, 0].tolist()) == list(range(len(spans)))
