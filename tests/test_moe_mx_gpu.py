"""Expert products on the block-scaled MMA: tiles that are filled in part, and permutations of many routes per token."""
import pytest
import torch

from minisgl.ops import quant

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("t,topk,drop,nt", [(3, 1, 0, 8), (5, 32, 0, 64), (4, 128, 0, 32), (3, 129, 0, 16), (3, 300, 0, 64), (5, 7, 4, 8), (3, 140, 130, 32)])
def test_permute_many_routes(t, topk, drop, nt):
    """``drop``: routes that the last token lacks.  Every route's rows and scales are those of its token."""
    from minisgl.ops import native as nv

    h, e, routes = 256, 6, t * topk - drop
    g = torch.Generator().manual_seed(topk)
    x = torch.randn(t, h, generator=g).bfloat16()
    idx = torch.randint(-1, e + 1, (routes,), generator=g, dtype=torch.int32)         # some belong to experts that are not here
    max_tiles = min(e, routes) + routes // nt + 1
    held = x.to(DEV), idx.to(DEV), torch.rand(routes, generator=g).to(DEV)
    plan = torch.zeros(4 + 3 * max_tiles + 3 * routes, dtype=torch.int32, device=DEV)
    xq, sf = torch.zeros(2 * routes, h, dtype=torch.uint8, device=DEV), torch.zeros(max_tiles, h // 128, 512, dtype=torch.uint8, device=DEV)
    nv.read_status(clear=True)
    nv.call("moe_plan", nv.ptr(held[1]), nv.ptr(held[2]), nv.I(routes), nv.I(e), nv.I(0), nv.I(nt), nv.ptr(plan), nv.I(max_tiles))
    nv.call("moe_mx_permute", nv.ptr(held[0]), nv.ptr(xq), nv.ptr(sf), nv.ptr(plan), nv.I(routes), nv.I(max_tiles), nv.I(topk), nv.I(h),
            nv.I(nt))
    torch.cuda.synchronize()
    assert nv.read_status(clear=True)[0] == 0
    plan, xq, sf = plan.cpu(), xq.cpu(), sf.cpu()
    hi, lo, eh, el = quant.mx_split(x)
    pos = plan[4 + 3 * max_tiles + routes:4 + 3 * max_tiles + 2 * routes].tolist()
    starts = plan[4:4 + 3 * int(plan[0])].view(-1, 3)
    blk = torch.arange(h // 32)
    for r, p in enumerate(pos):
        assert (p >= 0) == bool(0 <= idx[r] < e)
        if p < 0:
            continue
        tile = int((starts[:, 1] <= p).sum()) - 1
        n, token = p - int(starts[tile, 1]), r // topk
        off = lambda row: (row % 32) * 16 + (row // 32) * 4 + blk % 4  # noqa: E731
        assert torch.equal(xq[2 * p], hi[token].view(torch.uint8).flatten()) and torch.equal(xq[2 * p + 1], lo[token].view(torch.uint8).flatten())
        assert torch.equal(sf[tile, blk // 4, off(2 * n)].int(), eh[token].flatten().int())
        assert torch.equal(sf[tile, blk // 4, off(2 * n + 1)].int(), el[token].flatten().int())


def test_wide_tiles_filled_in_part():
    """Tiles of 64 routes that hold 1 to 64 of them: up to 32 one box of rows is loaded and narrower instructions are issued.  Against the
    fp16-operand kernel, which computes the same products in another order."""
    from minisgl.ops import cuda as C

    counts = [1, 8, 31, 32, 33, 64, 65, 97, 0, 49, 16, 40]
    h, inter, e = 512, 256, len(counts)
    g = torch.Generator().manual_seed(3)
    w13 = torch.randint(0, 256, (e, 2 * inter, h // 2), generator=g, dtype=torch.uint8).view(torch.int8)
    s13 = torch.randint(119, 122, (e, 2 * inter, h // 32), generator=g, dtype=torch.uint8)
    w2 = torch.randint(0, 256, (e, h, inter // 2), generator=g, dtype=torch.uint8).view(torch.int8)
    s2 = torch.randint(119, 122, (e, h, inter // 32), generator=g, dtype=torch.uint8)
    idx = torch.repeat_interleave(torch.arange(e), torch.tensor(counts))
    idx = idx[torch.randperm(len(idx), generator=g)].to(torch.int32)[:, None]
    assert C.route_tile(len(idx), e, "mx") == 64
    y = torch.randn(len(idx), h, generator=g).bfloat16()
    dev = [a.to(DEV) for a in (y, idx, torch.ones(len(idx), 1), w13, s13, w2, s2)]

    def rows():
        out, plan, _ = C.moe_routed(*dev, 7.0)
        torch.cuda.synchronize()
        return out.float()

    assert C.MOE_KERNEL == "mx"
    C.MOE_KERNEL = "f16"
    try:
        want = rows()
    finally:
        C.MOE_KERNEL = "mx"
    got = rows()
    # per row: an error in one tile must not hide behind the others.  bf16 results of bf16 activations: 2^-9 each, now and then one apart
    err = (got - want).norm(dim=1) / want.norm(dim=1)
    assert float(err.max()) < 3e-3, err.max()
