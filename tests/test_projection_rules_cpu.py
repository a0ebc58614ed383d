"""Which kernel a projection runs on: the sizes that were measured on both sides of each line."""
import pytest
import torch

from minisgl.ops import gemm


@pytest.mark.parametrize("m,n,k,groups,fp8,want", [
    (0, 4096, 4096, 1, False, False), (1, 64, 4096, 1, False, True), (8, 16384, 4096, 1, True, True), (8, 4096, 256, 1, True, True),
    (9, 4096, 4096, 1, True, True), (16, 32768, 1024, 1, True, True), (16, 4096, 512, 1, True, True), (17, 1536, 4096, 1, True, False),
    (9, 4096, 256, 1, True, False), (15, 129280, 4096, 1, False, True), (16, 129280, 4096, 1, False, False),
    (16, 12480, 4096, 1, False, False), (24, 8192, 4096, 1, False, True), (25, 4096, 4096, 1, False, False), (24, 1024, 4096, 8, False, True),
    (9, 2048, 4096, 8, False, False), (13, 4096, 128, 1, False, False), (17, 256, 256, 1, False, False), (20, 1024, 16384, 1, False, False),
    (17, 512, 512, 1, False, True)])
def test_few_rows(m, n, k, groups, fp8, want):
    assert gemm.few_rows(m, n, k, groups, fp8) is want


@pytest.mark.parametrize("m,n,groups,fp8,want", [
    (8192, 4096, 1, False, True), (12763, 256, 1, False, True), (12763, 128, 1, False, False), (18907, 64, 1, False, False),
    (9563, 264, 1, False, False), (12763, 264, 1, False, True), (9435, 264, 1, False, True), (6363, 640, 1, False, False),
    (4699, 896, 1, False, True), (4827, 896, 1, False, False), (1700, 1024, 8, False, True),
    (8192, 1536, 1, True, True), (5339, 512, 1, True, True), (4315, 512, 1, True, False), (3163, 640, 1, True, False),
    (19163, 64, 1, True, True), (128, 129280, 1, True, False), (257, 9700, 1, True, True)])
def test_fewer_waves(m, n, groups, fp8, want):
    assert gemm.fewer_waves(m, n, groups, fp8) is want


def test_results_off_16_bytes():
    on = torch.empty(5, 24, dtype=torch.bfloat16)
    assert gemm._rows_on_16(on, 24, 1) and gemm._rows_on_16(on[:, :8], 8, 1) and gemm._rows_on_16(on, 8, 3)
    assert not gemm._rows_on_16(on[:, 1:], 23, 1) and not gemm._rows_on_16(on, 12, 2)
    assert not gemm._rows_on_16(torch.empty(5, 300, dtype=torch.bfloat16), 300, 1)
    assert gemm._rows_on_16(torch.empty(5, 300), 300, 1)
