"""Sampling from a row of logits at the edges of its routes: rows that start off 16 bytes, equal logits, masked ones, one far above."""
import pytest
import torch

from minisgl.ops import api as O
from minisgl.ops import ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _near_a_step(lg, t, k, p, u, mask, got, eps=1e-6):
    """Whether single-precision masses may end at ``got``: their sum over a row is off by less than 1e-6 (2^-24 of each, times an exponent
    of a few units; 2^-40 for each entry), so a draw, or the end of top_p, that close to a step of the running mass may fall on either side."""
    x = lg.double().clone()
    if mask is not None:
        x[mask.long()] = float("-inf")
    prob = torch.softmax(x / t, -1)
    order = torch.sort(prob, descending=True, stable=True).indices
    before = prob[order].cumsum(0) - prob[order]
    for limit in (p - eps, p, p + eps) if p < 1.0 else (2.0,):
        kept = order[(before < limit) & (torch.arange(len(x)) < (k if k > 0 else len(x)))]
        mass = torch.zeros_like(prob)
        mass[kept] = prob[kept]
        end = mass.cumsum(0)
        if mass[got] > 0 and end[got] - mass[got] - eps <= u * end[-1] <= end[got] + eps:
            return True
    return False


@pytest.mark.parametrize("v", [1, 2, 37, 1009, 4099, 32771, 65536])
def test_sample_rows(v):
    """Against the definition in 64 bits."""
    g = torch.Generator().manual_seed(v)
    rows = [(k, p, t) for k in (0, 1, 3, 7, 256, 300, 4000) for p in (1.0, 0.87, 0.31) for t in (0.7, 1.6)]
    lg = torch.randn(len(rows), v, generator=g) * 2.5
    lg[1::5] = lg[1::5].round()                                           # ties
    lg[2::5] = 1.5                                                        # only ties: the longest lists
    lg[3::5, v // 3 + 1:] = float("-inf")
    lg[4::5, 0] = 40.0
    k, p, t = (torch.tensor(c) for c in zip(*rows))
    k, u = k.to(torch.int32), torch.rand(len(rows), generator=g)
    mask = torch.randint(0, v, (len(rows), 2), generator=g, dtype=torch.int32) if v > 1000 else None
    x = torch.empty(lg.numel() + 1, device=DEV)[1:].view_as(lg).copy_(lg)   # rows off 16 bytes
    for logits in (lg.to(DEV), x):
        got = O.sample(logits, t.to(DEV), k.to(DEV), p.to(DEV), u.to(DEV), None if mask is None else mask.to(DEV)).cpu()
        want = ref.sample(lg, t, k, p, u, mask)
        for r in (got != want).nonzero().flatten().tolist():
            m = None if mask is None else mask[r]
            assert _near_a_step(lg[r], float(t[r]), int(k[r]), float(p[r]), float(u[r]), m, int(got[r])), (rows[r], int(got[r]), int(want[r]))


ROWS = {
    "equal": lambda g, v: torch.full((v,), 0.5),
    "two values": lambda g, v: torch.where(torch.rand(v, generator=g) < 0.4, 1.0, 1.0 + 2.0 ** -20),
    "close": lambda g, v: torch.randn(v, generator=g) * 0.003,                   # thousands of values in one part of the histogram
    "about zero": lambda g, v: torch.randn(v, generator=g) * 1e-12,              # keys of both signs in one part
    "rounded": lambda g, v: (torch.randn(v, generator=g) * 2.5).round(),
    "ten left": lambda g, v: torch.where(torch.arange(v) % (v // 10) == 5, torch.randn(v, generator=g), float("-inf")),
    "half masked": lambda g, v: torch.where(torch.arange(v) < v // 2, torch.zeros(v), float("-inf")),
    "far below": lambda g, v: torch.where(torch.arange(v) < 7, torch.randn(v, generator=g), -60.0),     # no mass in 2^-40
}


@pytest.mark.parametrize("kind", list(ROWS))
def test_rows_that_fill_the_list(kind):
    """Rows whose kept set ends among more entries than the list holds, and rows where few entries have a mass."""
    g = torch.Generator().manual_seed(len(kind))
    v = 40001
    rows = [(k, p) for k in (0, 50, 256, 1000, 30000) for p in (1.0, 0.95, 0.5)]
    lg = torch.stack([ROWS[kind](g, v) for _ in rows])
    k, p = (torch.tensor(c) for c in zip(*rows))
    k, t, u = k.to(torch.int32), torch.ones(len(rows)), torch.rand(len(rows), generator=g)
    got = O.sample(lg.to(DEV), t.to(DEV), k.to(DEV), p.to(DEV), u.to(DEV)).cpu()
    want = ref.sample(lg, t, k, p, u)
    for r in (got != want).nonzero().flatten().tolist():
        assert _near_a_step(lg[r], 1.0, int(k[r]), float(p[r]), float(u[r]), None, int(got[r])), (rows[r], int(got[r]), int(want[r]))
