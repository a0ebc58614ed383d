"""Projections of a few rows against 64 bits and against the tiled kernel: remainders of rows, columns and of the shares of K."""
import pytest
import torch

from minisgl.ops import gemm

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("m", [1, 8, 13, 24])
@pytest.mark.parametrize("n,k", [(16, 128), (130, 384), (1536, 4096), (4100, 1152)])
def test_fp8(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m * n + k)
    x = torch.randn(m, k, generator=g, device=DEV).mul_(60).to(torch.float8_e4m3fn)
    w = torch.randn(n, k, generator=g, device=DEV).mul_(60).to(torch.float8_e4m3fn)
    pow2 = lambda *s: torch.exp2(torch.randint(-9, -4, s, generator=g, device=DEV).float())  # noqa: E731
    sx, sw = pow2(m, k // 128), pow2(-(-n // 128), k // 128)
    want = (x.double().view(m, -1, 128) * sx.double()[..., None]).flatten(1) @ (
        w.double() * sw.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)).T
    err = lambda y: ((y.double() - want).norm() / want.norm()).item()  # noqa: E731
    old = gemm.gemm_fp8(x, sx, w, sw, out_dtype=torch.float32, bn=32, splits=1)
    got = gemm.gemm_fp8(x, sx, w, sw, out_dtype=torch.float32)
    assert err(got) < max(1.5 * err(old), 3e-7)            # sums of 32 bits
    assert err(gemm.gemm_fp8(x, sx, w, sw)) < 3e-3         # one rounding to bf16
    gemm.gemm_fp8(x, sx, w, sw, out=got, accumulate=True)
    assert err(got / 2) < max(1.5 * err(old), 3e-7)


@pytest.mark.parametrize("m", [1, 7, 16, 23])
@pytest.mark.parametrize("n,k,groups", [(40, 32, 1), (2560, 4096, 1), (1024, 4096, 8), (72, 160, 3)])
def test_bf16(m, n, k, groups):
    g = torch.Generator(device=DEV).manual_seed(m * n + k)
    x = torch.randn(m, groups * k, generator=g, device=DEV).bfloat16()
    w = torch.randn(groups * n, k, generator=g, device=DEV).bfloat16()
    want = torch.einsum("tgk,gnk->tgn", x.double().view(m, groups, k), w.double().view(groups, n, k)).flatten(1)
    err = lambda y: ((y.double() - want).norm() / want.norm()).item()  # noqa: E731
    assert err(gemm.gemm_bf16_grouped(x, w, groups)) < 3e-3
    if groups == 1:
        old = gemm.gemm_bf16(x, w, out_dtype=torch.float32, bn=32, splits=1)
        got = gemm.gemm_bf16(x, w, out_dtype=torch.float32)
        assert err(got) < max(1.5 * err(old), 3e-7)
        wide = torch.zeros(m, n + 3, device=DEV)
        gemm.gemm_bf16(x, w, out=wide[:, :n], accumulate=True)
        assert torch.equal(wide[:, :n], got) and not wide[:, n:].any()
