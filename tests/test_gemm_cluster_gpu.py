"""The product whose K slices are added inside a cluster: rows, columns and K off every tile's edge, each number of slices,
stored and added, and the rule that chooses it."""
import pytest
import torch


def test_rule_keeps_all_clusters_resident():
    from hk_b200.csrc import gemm_fast
    assert gemm_fast.cluster_config(64, 8192, 4096, 148) is None and gemm_fast.cluster_config(129, 4096, 4096, 148) is None
    for m in (17, 64, 100, 128):
        for n in (64, 260, 1024, 2048, 2560, 4096, 6144):
            for k in (776, 2048, 4096, 12288):
                got = gemm_fast.cluster_config(m, n, k, 148)
                if got is None:
                    continue
                bn, slices = got
                assert 64 <= bn <= 256 and bn % 32 == 0 and 4 * slices <= -(-k // 64)
                assert -(-n // bn) <= gemm_fast.CLUSTERS_AT_ONCE[slices]
    assert gemm_fast.cluster_config(64, 4096, 4096, 148) == (192, 6)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,bn,slices", [(1, 64, 128, 64, 2), (8, 64, 136, 64, 2), (9, 68, 520, 64, 3), (33, 260, 1000, 96, 3),
                                             (64, 4096, 4096, 192, 6), (65, 516, 776, 160, 6), (127, 1028, 2048, 256, 8),
                                             (128, 6144, 4096, 192, 4), (128, 252, 512, 256, 8)])
@pytest.mark.parametrize("add", [False, True])
def test_cluster_product(M, N, K, bn, slices, add):
    from hk_b200.csrc import gemm_fast
    gen = torch.Generator().manual_seed(M * 7 + K)
    a = torch.randn(M, K, generator=gen).bfloat16()
    w = torch.randn(N, K, generator=gen).bfloat16()
    start = torch.randn(M, N, generator=gen)
    guard = torch.cat([start, torch.full((1, N), 5.0)]).cuda()
    assert gemm_fast.run_cluster(a.cuda(), w.cuda(), guard[:M], add, bn, slices)
    gemm_fast.check_status(guard.device)
    want = a.double() @ w.double().T + (start.double() if add else 0)
    # 32-bit sums of exact products: each of at most K + slices additions rounds by 2^-24 of the sum of magnitudes; the tensor
    # core may cut instead of round within a step of 16, which doubles that
    bound = (a.double().abs() @ w.double().abs().T + start.double().abs()) * (K + slices) * 2 ** -23
    assert bool(((guard[:M].double().cpu() - want).abs() <= bound).all())
    assert bool((guard[M] == 5.0).all())
    rel = (guard[:M].double().cpu() - want).norm() / want.norm()
    assert rel < 1e-5       # and what such sums really lose: a dropped K block would be 1e-1


@pytest.mark.gpu
def test_cluster_refusals():
    from hk_b200.csrc import gemm_fast
    a, w = torch.zeros(64, 512, dtype=torch.bfloat16, device="cuda"), torch.zeros(256, 512, dtype=torch.bfloat16, device="cuda")
    out = torch.full((64, 256), 3.0, device="cuda")
    for bn, slices in ((48, 2), (80, 2), (288, 2), (64, 1), (64, 9)):
        assert not gemm_fast.run_cluster(a, w, out, False, bn, slices)
    assert bool((out == 3.0).all())
