"""The persistent FP8 projection against one CTA per tile: both multiply exact products of the same scales and codes."""
import pytest
import torch

from minisgl.ops import gemm

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("m,n,k", [(8192, 192, 128), (12700, 130, 256), (1300, 2000, 1152), (257, 9700, 384), (3000, 1536, 4096)])
def test_many_rows(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m + k)
    x = torch.randn(m, k, generator=g, device=DEV).mul_(60).to(torch.float8_e4m3fn)
    w = torch.randn(n, k, generator=g, device=DEV).mul_(60).to(torch.float8_e4m3fn)
    pow2 = lambda *s: torch.exp2(torch.randint(-9, -4, s, generator=g, device=DEV).float())  # noqa: E731
    sx, sw = pow2(m, k // 128), pow2(-(-n // 128), k // 128)
    want = (x.double().view(m, -1, 128) * sx.double()[..., None]).flatten(1) @ (
        w.double() * sw.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)).T
    from minisgl.ops import native as nv

    def run(out, accumulate=False):
        nv.call("gemm_prefill_fp8", nv.ptr(x), nv.ptr(w), nv.ptr(out), nv.ptr(sx), nv.ptr(sw), nv.I(m), nv.I(n), nv.I(k), nv.I(k),
                nv.I(k), nv.I(out.stride(0)), nv.I(int(out.dtype == torch.float32)), nv.I(int(accumulate)), nv.I(148))
        return out

    err = lambda y: ((y.double() - want).norm() / want.norm()).item()  # noqa: E731
    got, old = run(torch.empty(m, n, device=DEV)), gemm.gemm_fp8(x, sx, w, sw, out_dtype=torch.float32, bn=128, splits=1)
    assert err(got) < max(1.5 * err(old), 2e-7)
    wide = torch.zeros(m, n + 5, dtype=torch.bfloat16, device=DEV)          # rows off 16 bytes
    run(wide[:, :n], True)
    assert err(wide[:, :n]) < 3e-3 and not wide[:, n:].any()
    assert torch.equal(run(torch.empty(m, n, dtype=torch.bfloat16, device=DEV)), got.bfloat16())
