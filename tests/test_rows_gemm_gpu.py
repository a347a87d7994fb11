"""The product with the weights as the tensor cores' 128-row operand (csrc/rows_gemm_tcgen05.cu) against float32, at the
edges of its tiles (128 rows of W, 128 values of k a stage, 16 rows of x) and for every number of splits of k."""

import pytest
import torch

from paged_llm_rs_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def inputs(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + 7 * N + 13 * K)
    return torch.randn(M, K, device=DEV, generator=g).bfloat16(), (torch.randn(N, K, device=DEV, generator=g) * 0.05).bfloat16()


# n and k on, one off and far from a tile's edge; a single tile of k; more stages than the ring holds; the wide head
@pytest.mark.parametrize("N,K", [(64, 64), (128, 128), (136, 192), (1000, 320), (256, 4160), (2048, 8192), (33000, 128)])
@pytest.mark.parametrize("M", [1, 16, 17, 63, 64])
def test_rows_product(M, N, K):
    x, w = inputs(M, N, K)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = x.double() @ w.double().T
    # a float sum of K products: at most K roundings of 2^-24 of the sum of their sizes
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    for splits in (0, 1, 2, 4, 8):
        if splits > -(-K // 128):
            continue
        y = ops.rows_gemm(x, w, status=st, splits=splits, out_dtype=torch.float32)
        assert ((y.double() - want).abs() <= bound).all()
        assert torch.equal(ops.rows_gemm(x, w, status=st, splits=splits), y.bfloat16())       # the bfloat16 result is that sum, rounded once
    assert st.item() == 0


@pytest.mark.parametrize("I,K", [(64, 64), (72, 128), (200, 1088), (3072, 1024)])
@pytest.mark.parametrize("M", [1, 17, 64])
def test_rows_product_with_activations(M, I, K):
    x, w = inputs(M, 2 * I, K)
    gu = ops.rows_gemm(x, w, splits=1).float()
    scale = 1 + gu[:, :I].abs() + gu[:, I:].abs()
    for splits in (0, 1, 2, 8):
        if splits > -(-K // 128):
            continue
        for act, limit, f in (("silu", 0.0, lambda g, u: g * torch.sigmoid(g) * u), ("relu", 0.0, lambda g, u: g.clamp(min=0) * u),
                              ("clamped", 2.0, lambda g, u: g.clamp(max=2.0) * torch.sigmoid(1.702 * g.clamp(max=2.0)) * (u.clamp(-2.0, 2.0) + 1))):
            y = ops.rows_gemm(x, w, glu=True, act=act, limit=limit, splits=splits)
            # (another order of the sums flips a rounding of gate or up now and then, which the activation scales by the other factor)
            assert ((y.float() - f(gu[:, :I], gu[:, I:])).abs() / scale).max().item() < 2e-2
        y = ops.rows_gemm(x, w, unary="squared_relu", splits=splits)
        want = gu.clamp(min=0).square()
        assert ((y.float() - want).abs() / (1 + want)).max().item() < 2e-2


@pytest.mark.parametrize("N", [136, 1000, 1992])
def test_ragged_widths_whose_splits_leave_one_another_at_once(N):
    # a cluster's CTAs read one another's shared memory; where the last tile is not full, one of them has nothing to add and
    # store for a column past the width, and must neither read for it nor leave before its peers have read
    x, w = inputs(40, N, 2048)
    xf, wf = x.float(), w.float()
    for splits in (2, 4, 8):
        first = ops.rows_gemm(x, w, splits=splits, out_dtype=torch.float32), ops.rows_gemm(x, w[: N // 16 * 16], glu=True, splits=splits), \
            ops.gemm_f32(xf, wf, splits=splits)
        for _ in range(200):
            again = ops.rows_gemm(x, w, splits=splits, out_dtype=torch.float32), ops.rows_gemm(x, w[: N // 16 * 16], glu=True, splits=splits), \
                ops.gemm_f32(xf, wf, splits=splits)
        assert all(torch.equal(a, b) for a, b in zip(first, again))
        for y in (first[0], first[2]):       # (the same operands in both: K roundings of the sum of the products' sizes, at most)
            assert ((y.double() - x.double() @ w.double().T).abs() <= 2048 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)).all()


def test_rows_product_is_the_engines_route_and_leaves_the_rest():
    x, w = inputs(24, 256, 256)
    assert ops.rows_gemm_takes(x, w, 256) and torch.equal(ops.linear(x, w), ops.rows_gemm(x, w))
    assert torch.equal(ops.linear_glu(x, w), ops.rows_gemm(x, w, glu=True))
    assert torch.equal(ops.linear_act(x, w, "squared_relu"), ops.rows_gemm(x, w, unary="squared_relu"))
    few, large = torch.randn(2, 4096, device=DEV).bfloat16(), torch.randn(4096, 4096, device=DEV).bfloat16()
    assert ops.rows_gemm_takes(few, large, 4096) and not ops.rows_gemm_takes(few, large[:2048], 2048)
    # rows of more than 64, a k that is no multiple of 64, rows that do not lie together, an address off 16 bytes: the other kernels
    for a, b in ((inputs(65, 256, 256)), (inputs(24, 256, 200)), (inputs(24, 256, 512)[0][:, :256], w),
                 (torch.randn(24 * 256 + 1, device=DEV).bfloat16()[1:].view(24, 256), w)):
        assert not ops.rows_gemm_takes(a, b, 256)
        torch.testing.assert_close(ops.linear(a, b).float(), a.float() @ b.float().T, atol=3e-2, rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_product_into_a_buffer_that_the_kernels_do_not_write_is_the_librarys(dtype):
    x, w = torch.randn(32, 1024, device="cuda").to(dtype), torch.randn(2048, 1024, device="cuda").to(dtype)
    want = ops.linear(x, w)
    wide = torch.zeros(32, 2 * 2048, dtype=dtype, device="cuda")
    for out in (torch.zeros(32, 2048, dtype=dtype, device="cuda"), wide[:, ::2], torch.zeros(0, dtype=dtype, device="cuda")):
        got = ops.linear(x, w, out)
        assert got.data_ptr() == out.data_ptr() and got.shape == (32, 2048)
        # (two float sums of 1024 products in another order, then one rounding to bfloat16, an ulp apart at most)
        torch.testing.assert_close(got, want, atol=1e-2 if dtype == torch.bfloat16 else 1e-3, rtol=2 ** -7 if dtype == torch.bfloat16 else 1e-4)
    assert not wide[:, 1::2].any()


def test_rows_that_do_not_lie_together_are_refused():
    from paged_llm_rs_b200.errors import KernelError
    x, w = inputs(24, 256, 512)
    wide = torch.zeros(24, 512, dtype=torch.bfloat16, device=DEV)
    for f, a, b, out in ((ops.rows_gemm, x[:, :256], w[:, :256].contiguous(), None), (ops.rows_gemm, x, w.t().contiguous().t(), None),
                         (ops.rows_gemm, x, w, wide[:, ::2]), (ops.gemm_f32, x.float()[:, :256], w.float()[:, :256].contiguous(), None),
                         (ops.gemm_f32, x.float(), w.float(), wide.float()[:, ::2])):
        with pytest.raises(KernelError):
            f(a, b, out)
