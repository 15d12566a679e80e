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
