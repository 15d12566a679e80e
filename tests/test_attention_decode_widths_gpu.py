"""Decode attention fed by TMA in its two widths (four consumer warps over tiles of 64 keys, two over 32): batches of one
more thread block than a wave of the wide form holds take the narrow one."""
import pytest
import torch

from test_kernels_gpu import DEV, attention_case, close_probabilities_in_bfloat16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,pt,requests,splits", [(128, 16, 38, 1), (128, 32, 74, 1), (128, 64, 40, 1), (128, 128, 19, 2),
                                                   (64, 16, 56, 1), (64, 128, 31, 2), (128, 16, 37, 1)])
@pytest.mark.parametrize("window", [0, 45])
def test_decode_batches_about_one_wave(hd, pt, requests, splits, window):
    # lengths about the narrow and the wide tile's edges, one of several tiles more than the ring holds
    lens = [(1, 31, 32, 33, 63, 64, 65, 97, 129, 331)[i % 10] for i in range(requests)]
    out, want, _ = attention_case("flash", torch.bfloat16, 16, 8, hd, pt, window, lens, [(n - 1, 1) for n in lens],
                                  fixed_splits=splits, mass=True)
    close_probabilities_in_bfloat16(out, want, attention_case.mass)
    from hk_b200.csrc import gemm_fast
    gemm_fast.check_status(torch.device(DEV))


@pytest.mark.parametrize("splits", [2, 3, 5, 7, 8])
@pytest.mark.parametrize("H,G,hd,pt,sink,window,requests", [(32, 8, 128, 16, False, 0, 4), (16, 1, 64, 128, True, 0, 11), (5, 5, 128, 32, True, 77, 3),
                                                            (12, 2, 64, 16, False, 300, 1), (32, 8, 128, 64, False, 0, 40)])
def test_splits_merged_in_a_cluster(splits, H, G, hd, pt, sink, window, requests, monkeypatch):
    """Every number of splits, some without a key, against the same splits merged by a kernel of their own, which gives the same bits;
    forty requests are more clusters than the GPU holds and take that kernel both times."""
    from dataclasses import replace

    from hk_b200.csrc import attention_fast, gemm_fast, ops
    g = torch.Generator(DEV).manual_seed(splits)
    lens = [(700, 1, 64, 129, 1333, 65, 31, 512)[i % 8] for i in range(requests)]
    pages = [-(-n // pt) for n in lens]
    table = torch.full((requests, max(pages)), -1, dtype=torch.int32)
    at = 0
    for r, n in enumerate(pages):
        table[r, :n] = torch.arange(at, at + n)
        at += n
    k, v = (torch.randn(at, G, pt, hd, generator=g, device=DEV).bfloat16() for _ in range(2))
    q, sinks = torch.randn(requests, H * hd, generator=g, device=DEV).bfloat16(), torch.randn(H, generator=g, device=DEV) if sink else None
    plan = attention_fast.build_plan(list(range(requests)), list(range(requests)), [1] * requests, [n - 1 for n in lens], requests, window, H, G, 148,
                                     lambda a: torch.from_numpy(a.copy()).to(DEV), fixed_splits=splits)
    ran, check = [], ops._check
    monkeypatch.setattr(ops, "_check", lambda code, what: (ran.append(what), check(code, what)))
    outs = []
    for p in (plan, replace(plan, splits=0)):
        out = torch.full((requests, H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
        assert attention_fast.run(q, k, v, table.to(DEV), out, H, G, hd, pt, window, hd ** -0.5, p, sink=sink, sinks=sinks)
        outs.append(out.float())
    assert ("cluster" in ran[0]) == (requests < 40) and "combine" in ran[-1]
    assert torch.equal(outs[0], outs[1])
    gemm_fast.check_status(torch.device(DEV))
