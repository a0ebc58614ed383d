"""The tcgen05 form of the sparse latent attention (64 heads): several tokens per CTA, masked keys, padded rows, maxima that grow from
tile to tile, splits without keys; and a 4:1 history attended whole, without a selection, at every number of local heads."""
import types

import pytest
import torch

from minisgl.ops import api as O

pytestmark = pytest.mark.gpu
DEV, PS, D, H = "cuda", 256, 512, 64


def _state(ratio, t, seed, longest=2048):
    g = torch.Generator().manual_seed(seed)
    pages = longest // PS
    table = torch.zeros(2, longest, dtype=torch.int32)
    for k, p in enumerate(torch.randperm(pages, generator=g).tolist()):
        table[1, k * PS:(k + 1) * PS] = torch.arange(p * PS, (p + 1) * PS, dtype=torch.int32)
    pos = torch.randint(0, longest, (t,), generator=g, dtype=torch.int32)
    pos[:3] = torch.tensor([0, 127, longest - 1], dtype=torch.int32)[:t]
    fb = types.SimpleNamespace(positions=pos, slots=torch.ones(t, dtype=torch.int32), page_table=table, max_context=longest,
                               num_valid=None, is_prefill=False)
    rows = lambda n: torch.randn(n, D, generator=g).bfloat16()  # noqa: E731
    swa_map = torch.randperm(pages + 1, generator=g).to(torch.int32)
    return (fb, rows((pages + 1) * PS), swa_map, rows((pages + 1) * max(PS // max(ratio, 1), 1)) if ratio else None,
            torch.randn(t, H, D, generator=g).bfloat16(), torch.randn(H, generator=g))


def _on(fb):
    return types.SimpleNamespace(**{k: v.to(DEV) if torch.is_tensor(v) else v for k, v in vars(fb).items()})


def _close(got, want):
    # bf16 weights and results: relative errors of about 2^-9 each
    assert ((got.float().cpu() - want.float()).norm() / want.float().norm()).item() < 8e-3


@pytest.mark.parametrize("t,ratio", [(1, 0), (3, 4), (40, 128), (301, 4)])
def test_tokens_of_several_rounds(t, ratio):
    from minisgl.ops import cuda

    fb, swa, swa_map, comp, q, sink = _state(ratio, t, 17 * t + ratio)
    q = q * 6                                      # scores of several units: maxima that move between tiles
    idx = n = None
    if ratio == 4:
        k = 512
        idx = torch.full((t, k), -1, dtype=torch.int32)
        n = ((fb.positions + 1) // 4).clamp(max=k)
        for r in range(t):
            idx[r, : int(n[r])] = torch.randperm(int((fb.positions[r] + 1) // 4))[: int(n[r])].to(torch.int32)
        idx[2::7, 3] = -1                          # entries that do not exist are passed over
    args = lambda d: (d(q), _on(fb) if d(q).is_cuda else fb, d(swa), d(swa_map), None if comp is None else d(comp), ratio,  # noqa: E731
                      None if idx is None else d(idx), None if n is None else d(n), d(sink), D ** -0.5, PS, 128)
    want = O.attention(*args(lambda x: x))
    for ns in (1, 2, 9):
        _close(cuda.attention(*args(lambda x: x.to(DEV)), nsplit=ns), want)


def test_rows_behind_the_valid_ones_are_zero():
    fb, swa, swa_map, comp, q, sink = _state(128, 20, 5)
    want = O.attention(q, fb, swa, swa_map, comp, 128, None, None, sink, D ** -0.5, PS, 128)
    fbd = _on(fb)
    fbd.num_valid = torch.tensor([13], dtype=torch.int32, device=DEV)
    got = O.attention(q.to(DEV), fbd, swa.to(DEV), swa_map.to(DEV), comp.to(DEV), 128, None, None, sink.to(DEV), D ** -0.5, PS, 128)
    assert not got[13:].any()
    _close(got[:13], want[:13])


def test_a_whole_history_is_the_selection_of_all_its_entries():
    fb, swa, swa_map, comp, q, sink = _state(4, 30, 9)
    n = (fb.positions + 1) // 4
    idx = torch.arange(512, dtype=torch.int32).repeat(30, 1)
    idx[idx >= n[:, None]] = -1
    one = lambda i, m, f, *x: O.attention(x[0], f, x[1], x[2], x[3], 4, i, m, x[4], D ** -0.5, PS, 128)  # noqa: E731
    cpu, dev = (q, swa, swa_map, comp, sink), tuple(x.to(DEV) for x in (q, swa, swa_map, comp, sink))
    assert torch.equal(one(None, None, fb, *cpu), one(idx, n, fb, *cpu))
    assert torch.equal(one(None, None, _on(fb), *dev), one(idx.to(DEV), n.to(DEV), _on(fb), *dev))


@pytest.mark.parametrize("heads", [8, 16, 32, 64])
@pytest.mark.parametrize("t,prefill", [(1, False), (7, False), (200, True)])
def test_whole_histories_of_sharded_heads(heads, t, prefill):
    """4:1 entries without a list, in a layer's shards too: as many splits as the wrapper takes, and numbers that leave some without keys."""
    from minisgl.ops import cuda

    fb, swa, swa_map, comp, q, sink = _state(4, t, heads + t)
    fb.is_prefill = prefill
    q, sink = q[:, :heads].contiguous() * 6, sink[:heads].contiguous()
    want = O.attention(q, fb, swa, swa_map, comp, 4, None, None, sink, D ** -0.5, PS, 128)
    dev = [x.to(DEV) for x in (q, swa, swa_map, comp, sink)]
    for ns in (0, 1, 3, 32):
        _close(cuda.attention(dev[0], _on(fb), dev[1], dev[2], dev[3], 4, None, None, dev[4], D ** -0.5, PS, 128, nsplit=ns), want)
