"""Which kernel and which tile a shape gets: pure functions of the shape, checked without a GPU."""


def test_tile_widths_the_tcgen05_product_chooses():
    from hk_b200.csrc import gemm_fast
    cfg = gemm_fast.tc_config
    assert cfg(2048, 24576, 4096, 148, swiglu=True) == (256, 1)         # 1,536 tiles: the widest
    assert cfg(2048, 6144, 4096, 148) == (240, 1)                        # 416 tiles in 3 waves instead of 384 of 256
    assert cfg(2048, 4096, 12288, 148) == (240, 1)                       # 288 tiles in 2 waves
    bn, splits = cfg(64, 24576, 4096, 148, swiglu=True)                  # one wave, every SM a tile
    assert splits == 1 and bn % 32 == 0 and 120 <= -(-24576 // bn) <= 148
    bn, splits = cfg(64, 4096, 12288, 148)
    assert bn in (128, 256) and splits > 1                               # narrow output: K slices


def test_tile_widths_of_one_row_tile():
    """Wide outputs in one wave of narrow tiles, unless the rows of a are few and short."""
    from hk_b200.csrc import gemm_fast
    cfg = gemm_fast.tc_config
    assert cfg(31, 8256, 2048, 148) == (128, 2) and cfg(32, 8256, 2048, 148) == (64, 1) and cfg(17, 8256, 4096, 148) == (64, 1)
    assert cfg(17, 12288, 2048, 148)[1] == 1 and cfg(24, 10304, 2048, 148) == (80, 1)


def test_tile_widths_of_a_few_hundred_rows():
    """Several row tiles, few waves: every choice is one that the kernel takes, and none leaves half of the SMs idle."""
    from hk_b200.csrc import gemm_fast
    for m in (129, 200, 257, 384, 527, 1000):
        for n, k in ((4096, 4096), (4096, 12288), (6144, 4096), (2056, 2048), (72, 512), (10304, 2048)):
            bn, splits = gemm_fast.tc_config(m, n, k, 148)
            assert bn % 16 == 0 and 64 <= bn <= 256 and 1 <= splits <= -(-k // 64)
            tiles = -(-m // 128) * -(-n // bn) * splits
            assert n < 4000 or tiles > 74
        for n, k in ((24576, 4096), (12288, 2048), (1056, 256)):
            bn, splits = gemm_fast.tc_config(m, n, k, 148, swiglu=True)
            assert bn % 32 == 0 and (splits == 1 or (n // 2) % (bn // 2) == 0)
    assert gemm_fast.tc_config(527, 4096, 12288, 148) == (144, 1)       # 145 tiles in one wave


def test_which_steps_of_a_recurrence_go_in_chunks():
    import types

    import numpy as np

    from hk_b200.parts import recurrent
    part = types.SimpleNamespace()

    def taken(heads, rows):
        scan = recurrent._ChunkedScan.__new__(recurrent._ChunkedScan)
        scan.H, scan._chunks = heads, True
        starts = np.cumsum([0] + rows[:-1])
        seg = np.asarray([(i, int(s), n) for i, (s, n) in enumerate(zip(starts, rows))], dtype=np.int32).reshape(-1, 3)
        part.arrays = {"segments": seg}
        old, recurrent.segment_tables = recurrent.segment_tables, lambda ctx: part
        try:
            t = scan.step_tables(None).arrays
        finally:
            recurrent.segment_tables = old
        assert sorted(t["short"].tolist() + t["long"].tolist()) == sorted(seg.tolist()) and len(t["requests"]) == len(t["long"])
        assert int(t["chunks"][:, 1].sum()) == int(t["long"][:, 2].sum())
        return t["long"][:, 2].tolist()

    assert taken(64, [319]) == [] and taken(64, [320]) == [320] and taken(64, [1] * 9) == []
    assert taken(64, [512] * 4) == [512] * 4 and taken(64, [512] * 5) == [] and taken(32, [640] * 8) == [640] * 8
    assert taken(32, [700, 301, 77, 1]) == [700, 301, 77] and taken(32, [1500, 100, 63]) == [1500, 100]
    assert taken(32, [639]) == [] and taken(8, [1000]) == [1000] and taken(320, [319]) == []
    assert taken(300, [400]) == [400] and taken(300, [400, 64]) == []


def test_scratch_of_a_walk_beside_chunks():
    from hk_b200.csrc import ops
    assert ops.walk_rows(1079, 1, 1) == (1, 1)              # one token beside 1,078 rows in chunks
    assert ops.walk_rows(1079, 3, 63) == (189, 63) and ops.walk_rows(400, 20, 1) == (20, 1)
    assert ops.walk_rows(206, 2, 130) == (206, 0)           # as many as the step has: its rows
    assert ops.walk_rows(500, 7, 0) == (500, 0)             # nothing beside
    assert ops.walk_rows(70000, 65536, 1) == (70000, 0) and ops.walk_rows(70000, 65535, 1) == (65535, 1)
