"""What a launch may ask of shared memory: the limit belongs to a kernel, not to a launcher of it, and counts the static part.  Each
case is a process of its own, since a limit that an earlier test has raised would hide what is looked for."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def forms(first_context, second_context, requests):
    """Decode attention over (requests, splits) one after the other, each with its own bound on the context (page lists of other
    lengths), against the softmax in float64."""
    import torch
    from hk_b200.csrc import attention_fast, gemm_fast, ops
    H, G, hd, pt, kept = 32, 8, 128, 16, 40
    dev = torch.device("cuda", 0)
    g = torch.Generator(dev).manual_seed(3)
    most = max(requests)
    lens = [(kept * pt, 1, 17, 333)[r % 4] for r in range(most)]
    table = torch.randperm(most * kept, generator=g, device=dev).int().view(most, kept)
    k, v = (torch.randn(most * kept, G, pt, hd, generator=g, device=dev).bfloat16() for _ in range(2))
    q = torch.randn(most, H * hd, generator=g, device=dev).bfloat16()
    ran, check = [], ops._check
    ops._check = lambda code, what, **more: (ran.append(what), check(code, what, **more))
    for step, R in enumerate(requests):
        splits = attention_fast.decode_splits(R, G, 148)
        plan = attention_fast.build_plan(list(range(R)), list(range(R)), [1] * R, [n - 1 for n in lens[:R]], R, 0, H, G, 148,
                                         lambda a: torch.from_numpy(a.copy()).to(dev), fixed_splits=splits,
                                         max_context=second_context if step == 1 else first_context)
        out = torch.full((R, H * hd), float("nan"), dtype=torch.bfloat16, device=dev)
        assert attention_fast.run(q[:R], k, v, table, out, H, G, hd, pt, 0, hd ** -0.5, plan)
        for r in range(R):
            keys, values = (x[table[r].long()].transpose(0, 1).reshape(G, kept * pt, hd)[:, :lens[r]].double() for x in (k, v))
            p = torch.softmax(torch.einsum("gjd,gtd->gjt", q[r].view(G, H // G, hd).double(), keys) * hd ** -0.5, dim=2)
            want, mass = torch.einsum("gjt,gtd->gjd", p, values), torch.einsum("gjt,gtd->gjd", p, values.abs())
            # probabilities and the result rounded to bfloat16
            assert bool(((out[r].view(G, H // G, hd).double() - want).abs() <= 2 ** -7 * mass + 1e-3).all()), (step, r)
    gemm_fast.check_status(dev)
    print([name for name in ran if "attention" in name])


def engine():
    """A context of 8,192 and batches of 24, 8 and 32 requests in turn, against the plain model."""
    import tempfile

    import numpy as np
    import torch

    import helpers
    import plain_qwen3 as P
    from hk_b200.engine import Engine, StepEntry
    helpers.TINY["wide"] = (dict(helpers.TINY_E, num_attention_heads=32, num_key_value_heads=8, max_position_embeddings=8192), 3, 0.03, 0.05)
    with tempfile.TemporaryDirectory() as folder:
        path = helpers.make_model_dir(folder, "wide", torch.bfloat16)
        cfg, w = helpers.load_plain(path)
        eng = Engine(path, dtype="bfloat16", page_tokens=16, max_tokens=32 * 64, max_requests=32, max_context=8192, max_batch_tokens=1024)
        rng = np.random.default_rng(1)
        ids = [rng.integers(0, 1000, 20 + r % 5).tolist() for r in range(32)]
        for r in range(32):
            eng.open_request(r)
            eng.step([StepEntry(r, ids[r])])
        for batch in (24, 8, 32):
            new = rng.integers(0, 1000, batch).tolist()
            for r in range(batch):
                ids[r].append(new[r])
            got = eng.step([StepEntry(r, [new[r]], [0]) for r in range(batch)]).double().cpu().numpy()
            for r in (0, 3, batch - 1):
                want = P.forward(cfg, w, ids[r])[-1]
                assert np.linalg.norm(got[r] - want) <= 3e-2 * np.linalg.norm(want), (batch, r)     # two layers in bfloat16


def first_rows(rank):
    import test_latent_made_rows_gpu as rows
    import torch
    rows.R = rank
    got, want, pos = rows.made_case([(0, 70), (3, 40)], 0, rows.tiled, tile=128)
    scale, early = float(want.abs().max()), pos < 16
    assert bool(torch.isfinite(got).all()) and float((got - want).abs().max()) <= 3e-2 * scale
    assert bool(((got - want).abs()[early] <= 2.0 ** -8 * want.abs()[early] + 1e-4 * scale).all())


def most_ranks():
    """The largest rank that the first rows' kernel takes runs, the next one is refused and not tried."""
    import torch
    from hk_b200.csrc import build
    first_rows(2128)
    lib, t = build.load("attention_latent"), torch.zeros(64, dtype=torch.int32, device="cuda")
    p = t.data_ptr()
    assert lib.hk_latent_first_rows(p, p, 0, p, p, p, 1, p, 1, 0, 2136, 0, 1.0, 0, 0, 0, 1.0, 0) == 100001


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["forms(8192, 8192, (24, 8, 32))", "forms(20000, 2048, (8, 24, 8))", "forms(2048, 8192, (32, 4, 32))",
                                  "forms(8192, 300, (1, 24, 1))", "engine()", "first_rows(8)", "first_rows(192)", "first_rows(256)", "first_rows(360)",
                                  "first_rows(504)", "most_ranks()"])
def test_first_launches_of_a_process(case):
    ran = subprocess.run([sys.executable, "-c", f"import test_shared_memory_limits_gpu as t; t.{case}"], capture_output=True, text=True, timeout=300,
                         env=dict(os.environ, PYTHONPATH=os.pathsep.join([HERE, os.path.join(HERE, os.pardir)])))
    assert ran.returncode == 0, ran.stderr[-3000:]
    if case.startswith("forms"):
        assert ("cluster" in ran.stdout) and ("decode" in ran.stdout)
