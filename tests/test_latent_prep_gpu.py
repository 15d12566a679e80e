"""What a token brings to a latent attention (`ops.latent_prep`): heads a warp each and four heads a warp, against the same in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("H,dn,dr,rot,r,pairing,packed,shift,write", [
    (1, 4, 4, 4, 4, "half", False, 0, True), (3, 128, 64, 64, 512, "half", True, 0, True), (4, 100, 64, 32, 132, "adjacent", False, 0, True),
    (5, 128, 64, 0, 128, "half", True, 4, True), (33, 64, 32, 20, 260, "adjacent", True, 0, False), (8, 128, 48, 46, 8, "half", False, 8, True),
    (2, 132, 64, 64, 64, "half", False, 0, True), (3, 128, 68, 64, 64, "half", True, 0, True),      # more than a warp's lanes hold at once
    (3, 126, 62, 62, 66, "adjacent", False, 0, True), (4, 128, 64, 64, 512, "half", True, 1, True),  # no whole pieces; rows that begin off them
])
def test_latent_prep(dtype, H, dn, dr, rot, r, pairing, packed, shift, write):
    from hk_b200.csrc import ops
    g = torch.Generator(DEV).manual_seed(H + dn + r)
    n, pt, dims = 37, 8, dict(generator=g, device=DEV)
    wide = torch.randn(n, H * (dn + dr) + r + dr + 2 * shift, **dims)
    q, kv = wide[:, shift:shift + H * (dn + dr)], wide[:, shift + H * (dn + dr):shift + H * (dn + dr) + r + dr]
    w, angle = torch.rand(r, **dims) + 0.5, torch.rand(64, max(rot // 2, 1), **dims) * 6
    pos = torch.randint(0, 64, (n,), generator=g, device=DEV, dtype=torch.int32)
    slots = torch.arange(n, device=DEV, dtype=torch.int32)
    table = torch.randperm(n * 8, generator=g, device=DEV).to(torch.int32).view(n, 8)
    pages = torch.full((n * 8, 1, pt, r + dr), float("nan"), dtype=dtype, device=DEV)
    plain, full, both = (torch.full((n, H * x), float("nan"), dtype=dtype, device=DEV) for x in (dn, r + dr, dn + dr))
    ops.latent_prep(q, kv, plain, full, w, 1e-5, angle.cos(), angle.sin(), rot, pairing, pos, slots, table, pages, H, dn, dr, r, pt, write_kv=write,
                    q_packed=both if packed else None)

    def turned(x):
        x, a = x.double().clone(), angle[pos.long()][:, None].double()
        one, two = (slice(0, rot, 2), slice(1, rot, 2)) if pairing == "adjacent" else (slice(0, rot // 2), slice(rot // 2, rot))
        if rot:
            u, v = x[..., one].clone(), x[..., two].clone()
            x[..., one], x[..., two] = u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()
        return x
    heads = q.reshape(n, H, dn + dr)
    got = both.view(n, H, dn + dr) if packed else torch.cat([plain.view(n, H, dn), full.view(n, H, r + dr)[..., r:]], dim=2)
    want = torch.cat([heads[..., :dn].double(), turned(heads[..., dn:])], dim=2)
    row = kv[:, :r].double()
    cache = torch.cat([row / (row.square().mean(1, keepdim=True) + 1e-5).sqrt() * w, turned(kv[:, None, r:])[:, 0]], dim=1)
    tol = 2e-6 if dtype == torch.float32 else 2 ** -8        # a few float32 roundings of turned pairs; half a unit of bfloat16
    assert bool(((got.double() - want).abs() <= tol * (want.abs() + 2)).all())
    if not packed:
        assert bool(torch.isnan(full.view(n, H, r + dr)[..., :r]).all())
    at = pages[table.long()[torch.arange(n, device=DEV), (pos // pt).long()], 0, (pos % pt).long()]
    if write:
        assert bool(((at.double() - cache).abs() <= tol * (cache.abs() + 2)).all())
    assert int(torch.isfinite(pages).any(-1).sum()) == (n if write else 0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("r,rot,pairing", [(512, 64, "half"), (132, 32, "adjacent"), (4, 0, "half")])
def test_both_ways_give_the_same_bits(dtype, r, rot, pairing):
    """Rows that begin on a 16-byte boundary and rows that do not."""
    from hk_b200.csrc import ops
    g = torch.Generator(DEV).manual_seed(r)
    n, H, dn, dr, pt = 37, 5, 128, 64, 8
    values, w, angle = torch.randn(n, H * (dn + dr) + r + dr, generator=g, device=DEV), torch.rand(r, generator=g, device=DEV), \
        torch.rand(64, max(rot // 2, 1), generator=g, device=DEV) * 6
    pos, slots = (torch.arange(n, device=DEV) * 7 % 64).int(), torch.arange(n, device=DEV, dtype=torch.int32)
    table = torch.arange(n * 8, device=DEV, dtype=torch.int32).view(n, 8)
    got = []
    for shift in (0, 1):
        wide = torch.zeros(n, values.shape[1] + 4, device=DEV)
        wide[:, shift:shift + values.shape[1]] = values
        q, kv = wide[:, shift:shift + H * (dn + dr)], wide[:, shift + H * (dn + dr):shift + values.shape[1]]
        plain, full, both = (torch.zeros(n, H * x, dtype=dtype, device=DEV) for x in (dn, r + dr, dn + dr))
        pages = torch.zeros(n * 8, 1, pt, r + dr, dtype=dtype, device=DEV)
        ops.latent_prep(q, kv, plain, full, w, 1e-5, angle.cos(), angle.sin(), rot, pairing, pos, slots, table, pages, H, dn, dr, r, pt, q_packed=both)
        got.append((both, pages))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and all(bool(x.any()) for x in got[0])
