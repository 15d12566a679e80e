"""Which steps of the chunked recurrences go in chunks, by their requests' lengths: what was in chunks for its longest request stays so,
several middling requests go by the walk's estimated time."""
import pytest


def part_of(kind, heads, dim):
    from hk_b200.parts import MLSTM, GatedDeltaRule, GeneralDeltaRule, Retention
    if kind == "delta":
        return GeneralDeltaRule(64, heads, dim, "m.", norm_eps=1e-5)
    if kind == "gated":
        return GatedDeltaRule(64, heads, heads, dim, dim, 4, "m.", norm_eps=1e-6)
    if kind == "retention":
        return Retention(64, heads, dim, dim, [0.9] * heads, "m.", 1e-6)
    return MLSTM(64, heads, dim, dim, 15.0, "m.", norm_eps=1e-6)


@pytest.mark.parametrize("kind,heads,dim,lengths,chunks", [
    ("delta", 64, 64, [2048], True), ("delta", 64, 64, [512] * 4, True), ("delta", 64, 64, [320], True), ("delta", 32, 64, [640], True),
    ("retention", 64, 64, [512], True), ("delta", 64, 64, [200], False), ("delta", 32, 64, [320], False), ("delta", 16, 64, [512], False),
    ("delta", 64, 64, [300, 120, 90], True), ("gated", 32, 64, [300, 290, 200, 120], True), ("mlstm", 64, 64, [227] * 9, True),
    ("delta", 32, 64, [227] * 9, True), ("delta", 16, 64, [128] * 16, False), ("retention", 64, 64, [227] * 9, False),
    ("delta", 64, 64, [64] * 8, False), ("delta", 64, 32, [300, 120, 90], False), ("mlstm", 32, 64, [64], False),
])
def test_which_steps_go_in_chunks(kind, heads, dim, lengths, chunks):
    assert part_of(kind, heads, dim)._chunks_pay(lengths) is chunks


def test_kinds_that_weigh_chunks_differently_share_no_tables():
    """The choice follows from a kind's walk and its chunks' time; the tables of a step are shared by their key."""
    parts = [part_of(kind, 64, 64) for kind in ("delta", "gated", "retention", "mlstm", "delta")]
    for part in parts:
        part._chunks = True
    keys = [part.step_tables_key() for part in parts]
    assert keys[0] == keys[4] and len(set(keys)) == 4
    assert not parts[0]._chunks_pay([157] * 6) and parts[1]._chunks_pay([157] * 6)
