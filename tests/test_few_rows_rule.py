"""Which products of a few rows go to the kernel made for them: both sides of every line of the rule, as measured on 148 multiprocessors, and the same lines on another device."""
import pytest

from hyperion_b200.ops import gemm


@pytest.mark.parametrize("m,n,k,pieces,pays", [
    (8, 896, 896, False, True), (1, 1152, 896, False, True), (8, 4096, 2048, False, True),
    (8, 160, 4096, False, True), (8, 288, 8192, False, False), (1, 640, 16384, False, False),      # narrow: whole sums over long k
    (8, 288, 8192, True, True), (1, 640, 16384, True, True), (8, 896, 4864, True, True),           # in pieces
    (8, 2560, 3072, True, False), (8, 5120, 2048, True, False), (8, 2048, 8192, True, False),      # more tiles than SMs: no pieces
    (8, 5120, 1024, False, True), (8, 5120, 2048, False, False), (8, 8192, 2048, False, True),     # a second turn of tiles
    (8, 10240, 256, False, True), (8, 10240, 1024, False, False), (8, 32768, 256, False, False),
    (8, 1024, 4096, False, True), (8, 1792, 4096, False, False), (8, 4096, 4096, False, False),    # the last by its bytes
    (8, 1536, 4096, False, True), (8, 1536, 6144, False, True), (8, 2560, 2048, True, True),       # the split product's second turn
    (16, 1024, 1024, False, True), (16, 896, 4864, False, False), (16, 896, 4864, True, True), (16, 5120, 1024, False, False), (16, 2304, 768, False, True),
    (16, 4096, 256, False, False), (16, 2048, 2048, False, False), (16, 2560, 2048, False, True), (16, 1536, 6144, False, False), (16, 768, 8192, True, False), (16, 160, 8192, True, True),
])
def test_lines(m, n, k, pieces, pays):
    assert gemm.pays_few_rows(m, n, k, pieces, 148) is pays


def test_tiles_follow_the_device():
    assert gemm.pays_few_rows(8, 4096, 1536, False, 148) and not gemm.pays_few_rows(8, 4096, 1536, False, 96)  # 256 tiles: one turn of 296 blocks, two of 192 with most of the second idle
