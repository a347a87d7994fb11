"""Which products are this library's and which cuBLAS's (kernels/ops.py, gemm_f32_sizes and rows_gemm_sizes): at sizes where one of the
two was measured to be slower it must not be the one that is taken."""

import pytest

from paged_llm_rs_b200.kernels import ops


@pytest.mark.parametrize("M,N,K", [(4, 512, 512), (16, 1024, 256), (64, 1024, 256), (257, 512, 512), (256, 1024, 256), (17, 32768, 1024), (32, 32768, 1024),
                                   (17, 12288, 4096), (64, 6144, 1024), (33, 8192, 1024), (128, 4096, 1024), (192, 2048, 1024), (300, 1024, 2048),
                                   (6, 4096, 12288), (32, 1024, 4096), (3, 1024, 1024), (1, 4096, 1024), (2048, 4096, 1024)])
def test_float32_products_of_the_library(M, N, K):
    assert not ops.gemm_f32_sizes(M, N, K)


@pytest.mark.parametrize("M,N,K", [(4, 4096, 1024), (8, 1024, 2048), (16, 151936, 1024), (4, 151936, 1024), (17, 4096, 1024), (32, 6144, 1024), (33, 4096, 1024),
                                   (64, 1024, 2048), (64, 4096, 12288), (128, 1024, 3072), (128, 2048, 2048), (256, 1024, 2048), (252, 1024, 3072),
                                   (16, 12288, 4096), (24, 1024, 512), (16, 2048, 512)])
def test_float32_products_of_this_library(M, N, K):
    assert ops.gemm_f32_sizes(M, N, K)


@pytest.mark.parametrize("M,N,K", [(33, 6144, 4096), (48, 4096, 4096), (64, 4096, 12288), (64, 1024, 256), (48, 512, 1024), (65, 1024, 2048), (16, 4096, 1024)])
def test_plain_products_of_the_library_or_the_weight_streaming_kernel(M, N, K):
    assert not ops.rows_gemm_sizes(M, N, K, N * K, True)


@pytest.mark.parametrize("M,N,K,rows_of_w,plain", [(8, 6144, 4096, 6144, True), (32, 4096, 12288, 4096, True), (64, 1024, 2048, 1024, True), (17, 256, 256, 256, True),
                                                   (64, 151936, 1024, 151936, True), (64, 12288, 4096, 24576, False), (48, 512, 1024, 1024, False)])
def test_products_with_the_weights_as_the_128_row_operand(M, N, K, rows_of_w, plain):
    assert ops.rows_gemm_sizes(M, N, K, rows_of_w * K, plain)
