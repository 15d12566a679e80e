"""The product on pairs of SMs: rows, columns and K off every tile's edge, several tiles a pair, K slices, every epilogue; and the
rule that chooses it."""
import ctypes

import pytest
import torch


def test_rule_gives_what_the_kernel_takes():
    from hk_b200.csrc import gemm_fast
    for refused in ((128, 24576, 4096), (527, 4096, 512), (256, 2048, 6144), (256, 10304, 2048)):
        assert gemm_fast.pair_config(*refused, 148) is None
    for m in (129, 200, 257, 384, 527, 1000, 2048, 4096, 8192):
        for n, k in ((4096, 4096), (4096, 12288), (6144, 4096), (20544, 4096), (10304, 2048), (2048, 6144), (72, 512), (151936, 4096)):
            for gated in (False, True):
                got = gemm_fast.pair_config(m, n, k, 148, gated)
                if got is None:
                    assert k < 1024 or m < 600 or n < 4096          # what many rows by long rows of weights never get
                    continue
                tiles_m, slices = got
                units = -(-m // 32)
                assert 1 <= tiles_m <= units and -(-units // tiles_m) <= 8 and 1 <= slices <= -(-k // 64)


def test_rule_picks():
    """Some of the choices (tiles along the rows, K slices), as the times that the models were fitted to have them."""
    from hk_b200.csrc import gemm_fast
    picks = {(527, 6144, 4096, False): (3, 1),
             (527, 24576, 4096, True): (3, 1),
             (527, 4096, 12288, False): (4, 1),
             (2048, 24576, 4096, True): (9, 1),
             (300, 4096, 4096, False): (4, 1),
             (256, 8256, 2048, False): (2, 1),
             (1000, 4096, 12288, False): (4, 1),
             (200, 4096, 12288, False): (2, 2)}
    assert {s: gemm_fast.pair_config(*s[:3], 148, s[3]) for s in picks} == picks


def _reference(a, w, epilogue, start, limit, slope):
    z = a.double() @ w.double().T
    if epilogue in (2, 3, 4):
        g, u = z.chunk(2, dim=1)
        if epilogue == 4:
            g, u = g.clamp(max=limit), u.clamp(-limit, limit) + 1
            return g * torch.sigmoid(slope * g) * u
        return (torch.nn.functional.silu(g) if epilogue == 2 else torch.nn.functional.gelu(g, approximate="tanh")) * u
    return {0: z, 1: start.double() + z, 5: slope * z.clamp(min=0) ** 2, 6: z}[epilogue]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,tiles_m,slices,pairs", [
    (1, 256, 64, 1, 1, 74), (33, 256, 72, 1, 1, 74), (100, 300, 200, 1, 1, 74), (129, 770, 1000, 1, 4, 74), (256, 512, 256, 1, 1, 1),
    (250, 4098, 192, 1, 3, 2), (700, 514, 328, 4, 2, 5), (300, 1000, 520, 2, 1, 3), (527, 1030, 1024, 3, 1, 74), (2048, 1536, 136, 9, 1, 74)])
@pytest.mark.parametrize("epilogue", range(7))
def test_pair_product(M, N, K, tiles_m, slices, pairs, epilogue):
    from hk_b200.csrc import build, gemm_fast, ops
    gen = torch.Generator().manual_seed(M * 7 + K + epilogue)
    a, w = torch.randn(M, K, generator=gen).bfloat16(), (torch.randn(N, K, generator=gen) / K ** 0.5).bfloat16()
    columns, kind = (N // 2 if epilogue in (2, 3, 4) else N), (torch.float32 if epilogue < 2 else torch.bfloat16)
    guard = torch.full((M + 40, columns), 5.0, dtype=kind, device="cuda")
    start = torch.randn(M, columns, generator=gen).to(kind)
    guard[:M] = start.cuda()
    lib = build.load("gemm_pair")
    lib.hk_gemm_pair_partial_floats.restype = ctypes.c_longlong
    partial = torch.full((int(lib.hk_gemm_pair_partial_floats(M, N, tiles_m, slices)),), float("nan"), device="cuda")
    da, dw = a.cuda(), w.cuda()
    p = lambda t: ctypes.c_void_p(t.data_ptr())      # noqa: E731
    limit, slope = 0.8, 1.702
    assert lib.hk_gemm_pair(p(da), p(dw), p(guard), M, N, K, ctypes.c_longlong(columns), epilogue, tiles_m, slices, pairs, p(partial),
                            p(gemm_fast.status_flag(guard.device)), ctypes.c_float(limit), ctypes.c_float(slope), ops._stream()) == 0
    gemm_fast.check_status(guard.device)
    want, got = _reference(a, w, epilogue, start, limit, slope), guard[:M].double().cpu()
    # 32-bit sums of exact products: each of at most K + slices additions rounds by 2^-24 of the sum of magnitudes; the tensor
    # core may cut instead of round within a step of 16, which doubles that.  A narrowed result is rounded by 2^-9 of itself, and an
    # activation's slope is at most 1.2 (a squared relu's 2 |z|): the sums are of order 1, so their error vanishes beside that
    sums = (a.double().abs() @ w.double().abs().T) * (K + slices) * 2 ** -23
    if epilogue < 2:
        bound = sums + (start.double().abs() * 2 ** -23 if epilogue else 0)
    else:
        bound = want.abs() * 2 ** -8 + 16 * sums.max() + 1e-6
    assert bool(((got - want).abs() <= bound).all())
    assert bool((guard[M:] == 5.0).all())
    assert float((got - want).norm() / want.norm()) < (1e-5 if epilogue < 2 else 3e-3)       # a dropped K block would be 1e-1


@pytest.mark.gpu
def test_pair_refusals():
    from hk_b200.csrc import gemm_fast
    a, w = torch.zeros(300, 512, dtype=torch.bfloat16, device="cuda"), torch.zeros(4096, 512, dtype=torch.bfloat16, device="cuda")
    out = torch.full((300, 4096), 3.0, device="cuda")
    for tiles_m, slices in ((0, 1), (1, 1), (11, 1), (2, 0), (2, 9)):
        assert not gemm_fast.run_pair(a, w, out, 0, 4096, tiles_m, slices)
    assert not gemm_fast.run_pair(a, w[:4095], out, 2, 4096, 2, 1)
    assert bool((out == 3.0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("counts,N,K,tile_rows", [([1, 0, 3], 256, 64, 32), ([70, 1, 33, 0, 64], 300, 136, 64), ([257, 5, 128], 514, 200, 128),
                                                  ([300, 0, 31, 513], 1030, 72, 256), ([0, 0, 9], 4096, 520, 64)])
@pytest.mark.parametrize("epilogue", [0, 2, 4])
def test_pair_product_by_group(counts, N, K, tile_rows, epilogue):
    from hk_b200.csrc import gemm_fast
    gen = torch.Generator().manual_seed(N + K)
    E, M = len(counts), sum(counts)
    a, w = torch.randn(M, K, generator=gen).bfloat16(), (torch.randn(E, N, K, generator=gen) / K ** 0.5).bfloat16()
    offsets, tiles, want = [0], [], []
    limit, slope = 0.8, 1.702
    for e, count in enumerate(counts):
        tiles += [(e, offsets[-1] + r) for r in range(0, count, tile_rows)]
        want.append(_reference(a[offsets[-1]:offsets[-1] + count], w[e], epilogue, torch.zeros(()), limit, slope))
        offsets.append(offsets[-1] + count)
    tiles += [(-1, 0)] * 3
    columns, kind = (N if epilogue == 0 else N // 2), (torch.float32 if epilogue == 0 else torch.bfloat16)
    guard = torch.full((M + 40, columns), 5.0, dtype=kind, device="cuda")
    table = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")      # noqa: E731
    assert gemm_fast.run_pair_grouped(a.cuda(), w.cuda(), guard[:M], table(tiles), table(offsets), tile_rows, epilogue != 0,
                                      2 if epilogue == 4 else 0, limit, slope)
    gemm_fast.check_status(guard.device)
    want, got = torch.cat(want), guard[:M].double().cpu()
    # as in test_pair_product; the sums are of order 1
    sums = K * 2 ** -23 * float((a.double().abs().max() * w.double().abs().max()) * K)
    bound = torch.full_like(want, sums) if epilogue == 0 else want.abs() * 2 ** -8 + 16 * sums + 1e-6
    assert bool(((got - want).abs() <= bound).all())
    assert bool((guard[M:] == 5.0).all())
    assert float((got - want).norm() / want.norm()) < (1e-5 if epilogue == 0 else 3e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [1, 6, 7, 8, 11, 12, 13, 25])
def test_pair_products_one_after_the_other(blocks):
    """K blocks below, at and beyond what the rings hold (12 stages at 32 rows, 7 at 256): the last releases of a launch must have come
    before its blocks leave, or they would strike the barriers of the next one's, whose rings lie elsewhere."""
    from hk_b200.csrc import gemm_fast
    gen = torch.Generator("cuda").manual_seed(blocks)
    w = torch.randn(74 * 256 + 256, blocks * 64, generator=gen, device="cuda").bfloat16()
    cases = []
    for rows, columns in ((256, 1024), (32, 256), (200, w.shape[0]), (96, 2048)):
        a = torch.randn(rows, w.shape[1], generator=gen, device="cuda").bfloat16()
        cases.append((a, w[:columns], torch.empty(rows, columns, device="cuda"), (a.double() @ w[:columns].double().T)))
    for turn in range(40):
        for a, wc, out, _ in cases:
            assert gemm_fast.run_pair(a, wc, out, 0, out.shape[1], 1, 1)
        if turn % 13 == 0:
            for a, wc, out, want in cases:        # K exact products of bf16 summed in 32 bits, cut at most twice as far as rounded
                bound = (a.double().abs() @ wc.double().abs().T) * (blocks * 64 + 1) * 2 ** -23
                assert bool(((out.double() - want).abs() <= bound).all())
                out.fill_(float("nan"))
    gemm_fast.check_status(w.device)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [40, 300])
def test_pinned_products(rows, monkeypatch):
    """'tc' is the product of one SM a tile and 'pair' the one on pairs, through every epilogue and whatever the rule would take."""
    from hk_b200.csrc import ops
    gen = torch.Generator("cuda").manual_seed(rows)
    a, w = (torch.randn(n, 1024, generator=gen, device="cuda").bfloat16() for n in (rows, 4096))
    ran, check = [], ops._check
    monkeypatch.setattr(ops, "_check", lambda code, what, **more: (ran.append(what), check(code, what, **more)))
    results = {}
    for kernel in ("tc", "pair"):
        with ops.force(gemm=kernel):
            outs = [torch.empty(rows, n, dtype=t, device="cuda") for n, t in ((4096, torch.float32), (2048, torch.bfloat16), (4096, torch.bfloat16),
                                                                              (4096, torch.bfloat16))]
            ops.gemm(a, w, outs[0])
            ops.gemm_swiglu(a, w, outs[1])
            ops.gemm_squared_relu(a, w, outs[2], 0.5)
            ops.gemm_narrow(a, w, outs[3])
        assert len(ran) == 4 and all(("pairs" in name) == (kernel == "pair") and "tcgen05" in name for name in ran), ran
        ran.clear()
        results[kernel] = outs
    for x, y in zip(results["tc"], results["pair"]):        # float32 sums in another order, then at most one rounding to bfloat16
        assert float((x.double() - y.double()).norm() / x.double().norm()) <= (2e-6 if x.dtype == torch.float32 else 1e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [4_200_000, 40_000_000, 2 ** 31 - 33])
def test_more_rows_than_the_tiles_count_are_refused(rows):
    """Before anything is launched: the addresses belong to nothing."""
    from hk_b200.csrc import build
    lib = build.load("gemm_pair")
    for epilogue in (0, 2):
        assert lib.hk_gemm_pair(1 << 20, 1 << 20, 1 << 20, rows, 4096, 4096, 4096, epilogue, -(-rows // 256), 1, 74, 0, 1 << 20, 0.0, 1.0, 0) == 100001
