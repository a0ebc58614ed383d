"""Row kernels that take several heads or blocks of a token at once: counts that leave remainders, rows off 16 bytes."""
import pytest
import torch

from minisgl.ops import api as O
from minisgl.ops.ref import RopeSpec

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROPE = RopeSpec.make(64, 10000.0, 65536, 16.0, 32, 1)


@pytest.mark.parametrize("t,heads", [(1, 1), (3, 5), (9, 64), (130, 6)])
def test_heads_in_groups(t, heads):
    g = torch.Generator().manual_seed(t * heads)
    pos = torch.randint(0, 5000, (t,), generator=g, dtype=torch.int32)
    q = torch.randn(t, heads, 128, generator=g).bfloat16() * 3
    w = torch.randn(t, heads, generator=g).bfloat16()
    codes, folded = O.indexer_q_encode(q.to(DEV), w.to(DEV), pos.to(DEV), ROPE, 0.1, 0.2)
    want, wf = O.indexer_q_encode(q, w, pos, ROPE, 0.1, 0.2)
    assert (codes.cpu() == want).float().mean() > 0.995               # a rotation's last place moves a few codes
    assert torch.allclose(folded.cpu(), wf, rtol=1e-3, atol=1e-6)

    q, wide = torch.randn(t, heads, 512, generator=g).bfloat16(), torch.randn(t, 1024 + 512, generator=g).bfloat16()
    gain, loc = 1 + torch.randn(512, generator=g).bfloat16() * 0.1, torch.randperm(512, generator=g)[:t].to(torch.int32)
    loc[0] = -1
    swa_map = torch.tensor([1, -1] if t < 9 else [1, 0], dtype=torch.int32)
    outs = []
    for dev in ("cpu", DEV):
        swa = torch.zeros(2 * 256, 512, dtype=torch.bfloat16, device=dev)
        a = [x.clone().to(dev) for x in (q, wide, pos, gain, loc, swa_map)]
        qq, kv = O.q_kv_norm_rope_store(a[0], a[1][:, 1024:], a[2], a[3], 1e-6, ROPE, swa, a[4], a[5], 256, True)
        outs.append([x.float().cpu() for x in (qq, kv, swa)])
    for a, b in zip(*outs):
        # results of a few units rounded to bf16, codes of e4m3 that go the other way (a sixteenth) now and then
        assert (a - b).norm() <= 4e-3 * a.norm() + 1e-6


@pytest.mark.parametrize("rows,k,off", [(1, 128, 0), (7, 384, 0), (5, 4096, 4), (9001, 1152, 0), (8192, 1280, 8)])
def test_fp8_quant_rows(rows, k, off):
    g = torch.Generator().manual_seed(rows)
    x = (torch.randn(rows, k + 8, generator=g) * 30).bfloat16().to(DEV)[:, off:off + k] if off else \
        (torch.randn(rows, k, generator=g) * 30).bfloat16().to(DEV)
    q, s = O.fp8_quant(x)
    want, ws = O.fp8_quant(x.cpu())
    assert torch.equal(s.cpu(), ws) and torch.equal(q.cpu().view(torch.uint8), want.view(torch.uint8))
