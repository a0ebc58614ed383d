"""FP8 projections report block scales that are not powers of two, whichever kernel the number of rows takes them to."""
import pytest
import torch

from minisgl.ops import gemm
from minisgl.ops import native as nv

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("m,n,k", [(1, 16, 128), (5, 200, 512), (16, 4096, 1024), (24, 130, 384), (25, 130, 384), (128, 256, 256),
                                   (3000, 1536, 256)])
def test_scales_that_are_not_powers_of_two_are_reported(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m + n)
    x = torch.randn(m, k, generator=g, device=DEV).to(torch.float8_e4m3fn)
    w = torch.randn(n, k, generator=g, device=DEV).to(torch.float8_e4m3fn)
    pow2 = lambda *s: torch.exp2(torch.randint(-9, 4, s, generator=g, device=DEV).float())  # noqa: E731
    sx, sw = pow2(m, k // 128), pow2(-(-n // 128), k // 128)

    def status():
        gemm.gemm_fp8(x, sx, w, sw)
        torch.cuda.synchronize()
        return nv.read_status(clear=True)[:2]

    nv.read_status(clear=True)
    try:
        assert status()[0] == 0
        for scales in (sx, sw):
            for at in {0, scales.numel() // 2, scales.numel() - 1}:
                good = scales.view(-1)[at].clone()
                for bad in (0.75, -0.5):
                    scales.view(-1)[at] = bad
                    assert status() == [2, 41], (at, bad)
                scales.view(-1)[at] = good
        assert status()[0] == 0
    finally:
        nv.read_status(clear=True)
