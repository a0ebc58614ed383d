"""Selecting the largest scores of a row at the edges of its routes: rows on both sides of what registers hold, rows that end inside a
group of four, equal values, values far from the rest."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _topk(logits, pos, k):
    from minisgl.ops import cuda

    t, width = logits.shape
    idx, n = torch.full((t, k), -7, dtype=torch.int32, device=DEV), torch.full((t,), -7, dtype=torch.int32, device=DEV)
    cuda.nv.call("topk", cuda.nv.ptr(logits), cuda.I(width), cuda.nv.ptr(pos), cuda.nv.ptr(idx), cuda.nv.ptr(n), cuda.I(t), cuda.I(k))
    return idx.cpu(), n.cpu()


@pytest.mark.parametrize("width,k", [(9, 8), (513, 512), (1023, 512), (8192, 512), (8193, 512), (16385, 1), (32768, 2048), (33001, 512)])
def test_topk_rows(width, k):
    g = torch.Generator().manual_seed(width)
    lg = torch.randn(8, width, generator=g)
    lg[1] = (lg[1] * 2).round() / 2                     # many equal scores: the first of them by index
    lg[2] = 0.25
    lg[3, width // 2] = 3e38                            # all others in one part of the range
    lg[3, 0] = -3e38
    lg[4, ::2], lg[4, 1::2] = 0.0, -0.0                 # the order of keys: -0 comes after 0
    lg[5, width - 1] = float("nan")
    lg[6] = lg[6].exp()
    n = torch.tensor([width, width, width - 1, width, width, width, k + 1, k], dtype=torch.int32)
    idx, got = _topk(lg.to(DEV), (4 * n - 1).to(DEV), k)
    for r in range(8):
        m = int(n[r])
        if m <= k:
            assert got[r] == m and idx[r].tolist() == [i if i < m else -1 for i in range(k)]
            continue
        if r == 5:
            assert got[r] == -1 and bool((idx[r] == -1).all())
            continue
        row = lg[r, :m].double()
        row = torch.where(torch.signbit(row) & (row == 0), torch.full_like(row, -1e-300), row)
        want = torch.sort(row, descending=True, stable=True).indices[:k].sort().values
        assert got[r] == k and torch.equal(idx[r].long(), want), r
