"""The float32 path's own kernels: the product on the CUDA cores (csrc/gemm_f32.cu) at the edges of its tiles and splits, and
the attention (csrc/attention_generic.cu) where a value is an infinity that its rows do not see."""

import pytest
import torch

import test_kernels_gpu as K
from paged_llm_rs_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,K", [(4, 4), (257, 36), (64, 128), (1000, 1024), (65, 3072), (300, 68)])
@pytest.mark.parametrize("M", [1, 4, 16, 17, 32, 33, 128, 129, 256])
def test_float32_product(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + 7 * N + 13 * K)
    x = torch.randn(M, K, device=DEV, generator=g)
    w = torch.randn(N, K, device=DEV, generator=g) * 0.05
    want = x.double() @ w.double().T
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)      # K roundings of the sum of the products' sizes, at most
    for tile in (0, 16, 32, 128):
        for splits in (0, 1, 3, 8):
            if splits > -(-K // 32):
                continue
            assert ((ops.gemm_f32(x, w, tile=tile, splits=splits).double() - want).abs() <= bound).all()


def test_float32_product_is_the_engines_route_and_leaves_the_rest():
    x, w = torch.randn(8, 1024, device=DEV), torch.randn(2048, 1024, device=DEV)
    assert ops.gemm_f32_takes(x, w) and torch.equal(ops.linear(x, w), ops.gemm_f32(x, w))
    assert ops.gemm_f32_takes(torch.randn(256, 2048, device=DEV), torch.randn(1024, 2048, device=DEV))
    odd = torch.randn(8 * 1024 + 1, device=DEV)[1:].view(8, 1024)
    # too few rows, a tiny product, many tiles, k no multiple of four, an address off 16 bytes: the library
    for a, b in ((x[:3], w), (x, w[:64]), (torch.randn(512, 1024, device=DEV), w), (x[:, :1022].contiguous(), w[:, :1022].contiguous()), (odd, w)):
        assert not ops.gemm_f32_takes(a, b)
        torch.testing.assert_close(ops.linear(a, b), (a.double() @ b.double().T).float(), atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("nh,nkv,hd", [(4, 4, 16), (16, 8, 128), (8, 1, 48), (6, 2, 256)])
def test_an_infinite_value_reaches_only_the_rows_that_see_it(nh, nkv, hd):
    # the last token of a portion, of a short one (few rows) and of a decoded one holds infinities; the rows before it must not
    def craft(r, q, k, v):
        v[-1] = float("inf")
    reqs = [(0, 70), (63, 2), (130, 33), (200, 1)]
    res, _ = K.run_attention(torch.float32, reqs, nh, nkv, hd, 16, None, 1, craft=craft)
    plain, _ = K.run_attention(torch.float32, reqs, nh, nkv, hd, 16, None, 1)
    for (got, _), (without, want) in zip(res, plain):
        assert torch.isinf(got[-1]).all() and torch.equal(got[:-1], without[:-1])
        torch.testing.assert_close(without, want, **K.tol(torch.float32))


@pytest.mark.parametrize("nh,nkv,hd,window", [(8, 1, 256, None), (16, 2, 256, None), (6, 2, 208, 40), (5, 5, 144, None)])
def test_single_tokens_of_long_heads(nh, nkv, hd, window):
    # (a step of decoded tokens alone takes a kernel without place for many rows, 32 keys a turn; split items among them)
    reqs = [(0, 1), (31, 1), (32, 1), (33, 1), (700, 1), (63, 1), (255, 1)]
    for target in (1, 296):
        for (got, want) in K.run_attention(torch.float32, reqs, nh, nkv, hd, 16, window, target, kinds=1, idle_items=2)[0]:
            torch.testing.assert_close(got, want, **K.tol(torch.float32))


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("n", [15, 16, 17, 33, 47, 49, 63, 65])
def test_turns_that_are_not_full(hd, n):
    # (a turn of 64 keys leaves out the sixteens that it does not have)
    for (got, want) in K.run_attention(torch.float32, [(0, n), (40, n)], 8, 4, hd, 16, None, 1)[0]:
        torch.testing.assert_close(got, want, **K.tol(torch.float32))
