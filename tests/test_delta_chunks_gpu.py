"""The recurrences walked in chunks of tokens (`csrc/delta_chunks.cu`) against the recurrence in float64, token by token: chunk
edges, keys and values that no tile divides, several requests, a state that is there already, and a call whose other requests
are walked token by token."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def recurrence(keys, values, decay, reads, S, remove=None):
    """S <- decay S - remove (read^T S) + key value^T, out = S^T q over the tokens, float64."""
    out = []
    for t in range(keys.shape[0]):
        new = decay[t][..., None] * S
        if remove is not None:
            new = new - remove[1][t][..., None] * torch.einsum("hk,hkv->hv", remove[0][t], S)[:, None, :]
        S = new + keys[t][..., None] * values[t][:, None, :]
        out.append(torch.einsum("hk,hkv->hv", reads[t], S))
    return torch.stack(out).flatten(1), S


def tables(lengths, first_chunked):
    """(short segments, long segments, chunks, requests); the requests from `first_chunked` on go in chunks."""
    from hk_b200.csrc import ops
    short, long, chunks, requests, row = [], [], [], [], 0
    for i, n in enumerate(lengths):
        (long if i >= first_chunked else short).append((i, row, n))
        if i >= first_chunked:
            requests.append((i, len(chunks), -(-n // ops.DELTA_CHUNK)))
            chunks += [(row + t, min(ops.DELTA_CHUNK, n - t)) for t in range(0, n, ops.DELTA_CHUNK)]
        row += n
    as_table = lambda rows, width: torch.tensor(rows, dtype=torch.int32, device=DEV).reshape(-1, width)      # noqa: E731
    return as_table(short, 3), as_table(long, 3), as_table(chunks, 2), as_table(requests, 3)


def unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def run(kind, H, dk, dv, lengths, tab, g):
    """(out, state) of the kernels and what the recurrence makes of the same inputs, per request."""
    from hk_b200.csrc import ops
    n, R = sum(lengths), len(lengths)
    short, long, chunks, requests = tab
    more = {"chunks": chunks, "requests": requests, "most_rows": max(lengths)}
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)       # noqa: E731
    G = H // 2 if kind == "gated" else H
    K, V = G * dk, H * dv
    dvp = ops.mlstm_padded(dv) if kind == "memory" else dv
    proj, logits = rand(n, 3 * K + V), rand(n, 4 * H)
    state = rand(R, H, dk, dvp)
    if kind == "memory":
        state[..., dv + 1:] = 0.0
    start, out = state.double(), torch.full((n, H * dvp), float("nan"), device=DEV)
    q, k, v, x = proj[:, :K], proj[:, K:2 * K], proj[:, 2 * K:2 * K + V], proj[:, 2 * K + V:]
    per = lambda t, heads, size: t.double().reshape(n, heads, size)        # noqa: E731
    remove = None
    if kind == "general":
        wl, ab, wb = rand(n, K), rand(K), rand(K) * 2 - 2
        ops.delta_rule_scan(q, k, v, x, wl, ab, wb, short, state, out, H, dk, dv, math.exp(-0.5), 1e-6, **more)
        keys, reads = per(k, H, dk), per(q, H, dk)
        decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(per(wl + wb, H, dk)))
        remove = (unit(keys), torch.sigmoid(per(x + ab, H, dk)) * unit(keys))
        values = per(v, H, dv)
    elif kind == "gated":
        al, db = rand(H).abs(), rand(H) - 2
        ops.gated_delta_scan(q, k, v, logits[:, :H], logits[:, H:2 * H], al, db, short, state, out, H, G, dk, dv, dk ** -0.5, 1e-6, **more)
        kk = unit(per(k, G, dk)).repeat_interleave(H // G, dim=1)
        reads = unit(per(q, G, dk)).repeat_interleave(H // G, dim=1) * dk ** -0.5
        beta = torch.sigmoid(logits[:, :H].double())[..., None]
        decay = torch.exp(-torch.exp(al.double()) * torch.nn.functional.softplus(logits[:, H:2 * H].double() + db.double()))[..., None].expand(n, H, dk)
        keys, values, remove = kk * beta, per(v, H, dv), (kk, kk * beta * decay)
    elif kind == "retention":
        rot = min(32, dk // 4 * 2)
        pos = torch.cat([torch.arange(c) for c in lengths]).int().to(DEV)
        angle = torch.rand(max(lengths), rot // 2, generator=g, device=DEV) * 6
        cos, sin, dec = angle.cos(), angle.sin(), 1 - torch.rand(H, generator=g, device=DEV) * 0.1
        ops.retention_scan(q, k, v, cos, sin, rot, pos, dec, short, state, out, H, dk, dv, 0.3, **more)
        c, s = (t.double()[pos.long()][:, None] for t in (cos, sin))

        def turn(t):
            a, b = t[..., :rot // 2], t[..., rot // 2:rot]
            return torch.cat([a * c - b * s, b * c + a * s, t[..., rot:]], -1)
        keys, values, reads = turn(per(k, H, dk)) * 0.3, per(v, H, dv), turn(per(q, H, dk))
        decay = dec.double()[None, :, None].expand(n, H, dk)
    else:
        wide = torch.cat([proj[:, :2 * K + V], logits], dim=1).contiguous()
        ib, fb, m_state, gates = rand(H) - 3, rand(H) + 3, rand(R, H), torch.empty(n, H, 3, device=DEV)
        at = 2 * K + V
        ops.mlstm_scan(wide[:, :K], wide[:, K:2 * K], wide[:, 2 * K:at], wide[:, at:at + H], wide[:, at + H:at + 2 * H], ib, fb, short, state,
                       m_state, out, gates, H, dk, dv, 15.0, 0.5, long_segments=long, **more)
        keys, reads = per(k, H, dk) * gates[..., 1:2].double(), per(q, H, dk) * 0.5      # the gates have tests of their own
        decay = gates[..., 0:1].double().expand(n, H, dk)
        values = torch.cat([per(v, H, dv), torch.ones(n, H, 1, device=DEV).double(), torch.zeros(n, H, dvp - dv - 1, device=DEV).double()], dim=2)
    want, row = [], 0
    for i, c in enumerate(lengths):
        part = slice(row, row + c)
        want.append(recurrence(keys[part], values[part], decay[part], reads[part], start[i],
                               None if remove is None else tuple(t[part] for t in remove)))
        row += c
    return out, state, torch.cat([o for o, _ in want]), torch.stack([s for _, s in want])


@pytest.mark.parametrize("kind", ["general", "gated", "retention", "memory"])
@pytest.mark.parametrize("H,dk,dv,lengths,first_chunked", [
    (2, 64, 64, [1, 31, 32, 33, 64, 65], 0),       # a chunk's edges
    (2, 8, 4, [70], 0), (4, 36, 20, [5, 97], 0),   # keys and values inside a tile
    (2, 64, 132, [40], 0), (2, 12, 68, [33], 0),   # value columns over several tiles, a few in the last
    (2, 64, 64, [3, 9, 130, 64], 2),               # two of the requests token by token
    (6, 64, 64, [80] * 30, 0),                     # enough requests for the walk's wider blocks
])
def test_chunks_match_the_recurrence(kind, H, dk, dv, lengths, first_chunked):
    g = torch.Generator(DEV).manual_seed(len(kind) * 1000 + dk + dv)
    got, got_state, want, want_state = run(kind, H, dk, dv, lengths, tables(lengths, first_chunked), g)
    for a, b, what in ((got, want, "outputs"), (got_state, want_state, "states")):
        worst = float((a.double() - b).abs().max() / b.abs().max())
        assert bool(torch.isfinite(a).all()) and worst <= 3e-5, f"{what}: {worst:.3g} of the largest value"     # accumulated float32 rounding


def test_chunks_refuse_what_they_cannot_do():
    from hk_b200.csrc import ops
    assert ops.delta_chunks_take(64, 64) and not ops.delta_chunks_take(68, 64) and not ops.delta_chunks_take(64, 66)
    assert ops.delta_chunks_take(64, 64, 1.38) and not ops.delta_chunks_take(64, 64, 2.0)
    short, _, chunks, requests = tables([64], 0)
    z = torch.zeros(64, 4 * 64, device=DEV)
    with pytest.raises(ops.KernelError):
        ops.delta_rule_scan(z[:, :64], z[:, 64:128], z[:, 128:192], z[:, 192:], z[:, :64], z[0, :64], z[0, :64], short,
                            torch.zeros(1, 1, 64, 64, device=DEV), torch.zeros(64, 64, device=DEV), 1, 64, 64, 2.0, 1e-6, chunks=chunks,
                            requests=requests)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,dv,act,weight,memory", [(3, 4, "silu", "shared", False), (5, 32, "sigmoid", "all", False), (2, 36, "silu", None, False),
                                                    (7, 64, "sigmoid", "all", True), (3, 68, "silu", "shared", False), (1, 128, "sigmoid", "all", True)])
def test_head_out_gate_of_whole_pieces(dtype, H, dv, act, weight, memory):
    """A head's norm and gate with 8, 16 and 32 lanes a head, heads that leave lanes idle, items that leave a block unfilled."""
    from hk_b200.csrc import ops
    g = torch.Generator(DEV).manual_seed(dv * 10 + H)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)       # noqa: E731
    n, ldo = 37, ops.mlstm_padded(dv) if memory else dv
    o, logits = rand(n, H * ldo), rand(n, H * dv + 8)[:, 4:4 + H * dv]
    w = None if weight is None else rand(dv if weight == "shared" else H * dv)
    gates = rand(n, H, 3).abs() if memory else None
    out = torch.empty(n, H * dv, dtype=dtype, device=DEV)
    ops.head_out_gate(o, logits, w, 1e-5, out, H, dv, act=act, gates=gates, den_eps=1e-6)
    x = o.double().view(n, H, ldo)
    if memory:
        x = x / (torch.maximum(x[..., dv:dv + 1].abs(), gates[..., 2:].double()) + 1e-6)
    x = x[..., :dv]
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)
    if w is not None:
        y = y * w.double().view(-1, dv)
    z = logits.double().view(n, H, dv)
    want = (y * torch.sigmoid(z) * (z if act == "silu" else 1.0)).flatten(1)
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5              # half a unit of the storage type; float32 rounding
    assert bool(((out.double() - want).abs() <= rel * want.abs() + 1e-6).all())
