"""Which kernel a projection runs on: the sizes that were measured on both sides of each line."""
import pytest

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
