"""Gates divide as float32 divides, whatever their results are narrowed to: far out, where the denominator lies between 2^126 and 2^128
and a quick division gives 0, and in the last place."""
import math

import pytest
import torch

from test_delta_chunks_gpu import DEV, tables

pytestmark = pytest.mark.gpu
HALF = 2.0 ** -7        # a rounding to bfloat16, and of 2^-16 for an exponential of 88 from a float32 argument


@pytest.mark.parametrize("rows,K", [(20, 64), (100, 64), (300, 1024)])      # one SM a tile, and pairs
@pytest.mark.parametrize("act,gate", [("silu", -88.0), ("gelu_tanh", -10.0), ("swish_clamped", -51.5)])
def test_gated_products(rows, K, act, gate):
    from hk_b200.csrc import ops
    F, limit, slope = 2048, 1e30, 1.702
    a, w = torch.zeros(rows, K, dtype=torch.bfloat16, device=DEV), torch.zeros(2 * F, K, dtype=torch.bfloat16, device=DEV)
    a[:, 0], w[:F, 0], w[F:, 0] = 1.0, gate, 1e30
    w[F - 1, 0] = 0.0
    out = torch.empty(rows, F, dtype=torch.bfloat16, device=DEV)
    ops.gemm_swiglu(a, w, out, act=act, limit=limit, slope=slope)
    z = {-88.0: gate, -10.0: 2 * math.sqrt(2 / math.pi) * (gate + 0.044715 * gate ** 3), -51.5: slope * gate}[gate]
    up = float(w[F, 0])
    want = gate / (1 + math.exp(-z)) * (min(up, limit) + 1 if gate == -51.5 else up)
    assert float(((out[:, :-1].double() - want) / want).abs().max()) <= HALF
    assert not bool(out[:, -1].any())


@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "swish_clamped"])
@pytest.mark.parametrize("kernel", ["tc", "pair"])
def test_gated_epilogues_divide_like_the_streaming_product(kernel, act):
    """Products of one exact term: the same gates and ups, so the same bits as from the kernel that divides plainly, but for the few that
    lie on the edge between two bfloat16 numbers."""
    from hk_b200.csrc import ops
    rows, K, F, apart = 20, 64, 16384, 0
    g = torch.Generator(DEV).manual_seed(11)
    for low, high in ((-1.0, 1.0), (-20.0, 20.0), (-89.0, 89.0)):
        a, w = torch.zeros(rows, K, dtype=torch.bfloat16, device=DEV), torch.zeros(2 * F, K, dtype=torch.bfloat16, device=DEV)
        a[:, 0] = torch.rand(rows, generator=g, device=DEV) + 0.5
        w[:F, 0] = torch.rand(F, generator=g, device=DEV) * (high - low) + low
        w[F:, 0] = torch.randn(F, generator=g, device=DEV)
        outs = []
        for name in (kernel, "stream"):
            outs.append(torch.empty(rows, F, dtype=torch.bfloat16, device=DEV))
            with ops.force(gemm=name):
                ops.gemm_swiglu(a, w, outs[-1], act=act, limit=60.0, slope=1.702)
        assert bool(torch.isfinite(outs[1].float()).all())
        apart += int((outs[0] != outs[1]).sum())
        # normal results: one rounding to bfloat16 apart at most
        assert bool(((outs[0].double() - outs[1].double()).abs() <= 2.0 ** -7 * outs[1].double().abs() + 2.0 ** -126).all())
    assert apart <= 3 * rows * F * 1e-5


@pytest.mark.parametrize("kernel", ["tc", "pair"])
def test_gates_that_are_not_finite(kernel):
    from hk_b200.csrc import ops
    a, w, inf = torch.zeros(20, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(64, 64, dtype=torch.bfloat16, device=DEV), float("inf")
    a[:, 0] = 1.0
    w[:32, 0], w[32:, 0] = torch.tensor([inf, -inf, float("nan"), 0.0, -200.0, 200.0, 3e38, -3e38] * 4), 1.0
    out = torch.empty(20, 32, dtype=torch.bfloat16, device=DEV)
    with ops.force(gemm=kernel):
        ops.gemm_swiglu(a, w, out)
    want = torch.tensor([inf, float("nan"), float("nan"), 0.0, 0.0, 200.0, 3e38, 0.0] * 4, device=DEV).bfloat16()
    assert torch.equal(out.nan_to_num(nan=7.0), want.nan_to_num(nan=7.0).expand(20, 32))


def test_short_convolution_and_norms():
    from hk_b200.csrc import ops
    n, C = 64, 4096
    x, y = torch.full((n, C), -88.0, device=DEV), torch.empty(n, C, dtype=torch.bfloat16, device=DEV)
    segs = torch.tensor([[0, 0, n]], dtype=torch.int32, device=DEV)
    ops.short_conv(x, torch.ones(C, 1, device=DEV), segs, torch.zeros(1, 1, C, device=DEV), y)
    want = -88.0 / (1 + math.exp(88.0))
    assert float(((y.double() - want) / want).abs().max()) <= HALF
    ops.gated_part_norm(torch.full_like(x, 1e37), x, torch.ones(C, device=DEV), 0.0, y, C // 64)        # 4,096 parts: a warp each
    assert float((y.double() + 1).abs().max()) <= HALF
    for act, value in (("sigmoid", 1 / (1 + math.exp(88.0))), ("silu", want)):
        ops.head_out_gate(torch.ones(n, C, device=DEV), x, torch.full((C,), 1e30, device=DEV), 0.0, y, C // 64, 64, act=act)
        assert float((y.double() / (1e30 * value) - 1).abs().max()) <= HALF


@pytest.mark.parametrize("kind", ["general", "gated"])
def test_step_sizes_of_chunks_are_those_of_the_walk(kind):
    """A first token alone has a step size a, its key a unit vector; its value 1 makes a state of a (gated rule), or a state of 1 loses
    a (generalised rule): to the bit."""
    from hk_b200.csrc import ops
    H, d, n = 256, 64, 64
    g = torch.Generator(DEV).manual_seed(5)
    q = k = torch.zeros(n, H, d, device=DEV)
    k = k.clone()
    k[..., 0] = 1.0
    v = torch.zeros(n, H * d, device=DEV)
    v[0] = float(kind == "gated")
    step = torch.full((n, H, 1 if kind == "gated" else d), -float("inf"), device=DEV)
    step[0] = torch.randn(step.shape[1:], generator=g, device=DEV).abs() * 3
    got = []
    for first in (0, 1):
        short, _, chunks, requests = tables([n], first)
        more = {"chunks": chunks, "requests": requests, "most_rows": n} if first == 0 else {}
        state, out = torch.zeros(1, H, d, d, device=DEV), torch.empty(n, H * d, device=DEV)
        state[:, :, 0] = float(kind == "general")
        wide = torch.cat([q.reshape(n, -1), k.reshape(n, -1), v, step.reshape(n, -1)], dim=1)
        cols = [wide[:, i * H * d:(i + 1) * H * d] for i in range(3)] + [wide[:, 3 * H * d:]]
        if kind == "gated":
            far = torch.full((n, H), -1e30, device=DEV)
            logits = torch.cat([cols[3], far], dim=1)
            ops.gated_delta_scan(*cols[:3], logits[:, :H], logits[:, H:], torch.zeros(H, device=DEV), torch.zeros(H, device=DEV), short, state, out,
                                 H, H, d, d, 1.0, 0.0, **more)
        else:
            ops.delta_rule_scan(*cols[:4], torch.full((n, H * d), -1e30, device=DEV), torch.zeros(H * d, device=DEV), torch.zeros(H * d, device=DEV),
                                short, state, out, H, d, d, math.exp(-0.5), 0.0, **more)
        got.append(state)
    assert len(got[1][0, :, 0].unique()) > H // 2 and not bool(got[1][0, :, 1:].any())
    assert torch.equal(*got)
