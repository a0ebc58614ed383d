"""The route plan over one and over several CTAs: a partition of the local routes by expert, in tiles of at most nt."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("routes,e,base,nt", [(1, 1, 0, 8), (30, 256, 0, 8), (4096, 256, 64, 32), (4097, 32, 32, 64), (50000, 256, 0, 64),
                                              (70001, 1500, 100, 16)])
def test_plan(routes, e, base, nt):
    from minisgl.ops import native as nv

    g = torch.Generator().manual_seed(routes)
    idx = torch.randint(-1, base + e + 40, (routes,), generator=g, dtype=torch.int32)
    w = torch.rand(routes, generator=g)
    tiles = min(e, routes) + routes // nt + 1
    plan = torch.full((4 + 3 * tiles + 3 * routes,), -9, dtype=torch.int32, device=DEV)
    held = idx.to(DEV), w.to(DEV)
    nv.call("moe_plan", nv.ptr(held[0]), nv.ptr(held[1]), nv.I(routes), nv.I(e), nv.I(base), nv.I(nt), nv.ptr(plan), nv.I(tiles))
    plan = plan.cpu()
    local = (idx >= base) & (idx < base + e)
    n_tiles, n = plan[:2].tolist()
    assert n == int(local.sum())
    t = plan[4:4 + 3 * n_tiles].view(-1, 3)
    at = 4 + 3 * tiles
    order, pos, sw = plan[at:at + n], plan[at + routes:at + 2 * routes], plan[at + 2 * routes:at + 2 * routes + n].view(torch.float32)
    assert torch.equal(order.sort().values, local.nonzero().flatten().to(torch.int32)) and torch.equal(sw, w[order.long()])
    assert torch.equal(pos[order.long()], torch.arange(n, dtype=torch.int32)) and bool((pos[~local] == -1).all())
    assert bool((t[:, 2] >= 1).all()) and bool((t[:, 2] <= nt).all()) and int(t[:, 2].sum()) == n
    assert torch.equal(t[:, 1], torch.cumsum(t[:, 2], 0).to(torch.int32) - t[:, 2])
    assert torch.equal(torch.repeat_interleave(t[:, 0], t[:, 2]), idx[order.long()] - base)
    full = torch.bincount((idx[local] - base).long(), minlength=e)
    assert n_tiles == int(((full + nt - 1) // nt).sum())
