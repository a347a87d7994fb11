"""Float32 products on the tensor cores (csrc/gemm_f32_tcgen05.cu) at the edges of their tiles, splits and parts."""

import pytest
import torch

from paged_llm_rs_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _bound(x, w):
    """Three roundings a value's parts, one a block of 64 values and split, and what the tensor cores cut off inside a block (twelve
    instructions, an ulp each at most), of the sum of the products' sizes."""
    return (2.0 ** -22 * 4) * (x.double().abs() @ w.double().abs().T) + 1e-37


@pytest.mark.parametrize("N,K", [(4, 64), (132, 72), (128, 128), (300, 200), (1024, 1032)])
@pytest.mark.parametrize("M", [1, 31, 33, 64, 65, 129, 256, 257])
def test_products_in_parts(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + 7 * N + 13 * K)
    x = torch.randn(M, K, device=DEV, generator=g)
    any_w = torch.randn(N, K, device=DEV, generator=g) * 0.05
    short = any_w.bfloat16().float()
    mixed = short.clone()                                # some turns and blocks of W with one part, some with two, some with three
    mixed[:, K // 2:][N // 3:] = any_w[:, K // 2:][N // 3:]
    mixed[:, :40] += short[:, :40] * 2.0 ** -9
    for w in (short, any_w, mixed):
        want, bound = x.double() @ w.double().T, _bound(x, w)
        for tile, splits in ((0, 0), (32, 1), (64, 2), (128, 3), (256, 8)):
            if splits <= -(-K // 64):
                got = ops.gemm_f32_tcgen05(x, w, tile=tile, splits=splits)
                assert ((got.double() - want).abs() <= bound).all(), (tile, splits)


@pytest.mark.parametrize("splits", [1, 2])
def test_values_that_cannot_be_split(splits):
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w = torch.randn(40, 192, device=DEV, generator=g), torch.randn(264, 192, device=DEV, generator=g)
    x[3, 5], x[7, 9], x[9, 1], x[12, 190] = float("inf"), float("nan"), 3.4e38, float("-inf")
    x[11] *= 1e-36                                       # (its parts would be below the smallest normal number)
    # w[0, 100] below meets small values only: where a product of finite values leaves float's range, float arithmetic goes on with an
    # infinity and may meet one of the other sign, and 64 bits do not
    x[:, 100] *= 0.05
    w[0, 1] = 0.0
    for bad in (False, True):
        if bad:
            w[200, 3], w[0, 100], w[261, 191] = float("-inf"), 3.4028e38, float("nan")
        want = (x.double() @ w.double().T).float()
        got = ops.gemm_f32_tcgen05(x, w, splits=splits)
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
        bound = _bound(x, w)
        live = torch.isfinite(want) & (bound < 1e30)
        assert ((got.double() - want.double()).abs() <= bound)[live].all()
        tiny = want[11, 1:200].double()
        assert (got[11, 1:200].double() - tiny).norm() <= 2.0 ** -20 * tiny.norm()


def test_the_route_and_what_it_leaves():
    x, w = torch.randn(256, 1024, device=DEV), torch.randn(2048, 1024, device=DEV)
    assert ops.gemm_f32_tcgen05_takes(x, w) and torch.equal(ops.linear(x, w), ops.gemm_f32_tcgen05(x, w))
    out = torch.empty(256, 2048, device=DEV)
    assert ops.linear(x, w, out=out) is out and torch.equal(out, ops.gemm_f32_tcgen05(x, w))
    odd = torch.randn(256 * 1024 + 1, device=DEV)[1:].view(256, 1024)
    # few rows, a small product, k no multiple of eight, columns no multiple of four, an address off 16 bytes, rows that do not lie together
    for a, b in ((x[:32], w), (x, w[:512]), (x[:, :1020].contiguous(), w[:, :1020].contiguous()), (x, w[:2047]), (odd, w), (x[:, ::2], w[:, ::2])):
        assert not ops.gemm_f32_tcgen05_takes(a, b)
        torch.testing.assert_close(ops.linear(a, b), (a.double() @ b.double().T).float(), atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("at", [0, 700, 1031])
@pytest.mark.parametrize("M,tile,splits", [(1, 32, 8), (33, 64, 8), (33, 64, 5), (200, 256, 8)])
def test_every_cta_of_a_cluster_learns_of_a_value_that_cannot_be_split(M, tile, splits, at):
    # (33 rows in eight CTAs: the last five have no entries of the tile to add, and leave as the others do)
    g = torch.Generator(device=DEV).manual_seed(M + at)
    x, w = torch.randn(M, 1032, device=DEV, generator=g), torch.randn(264, 1032, device=DEV, generator=g)
    w[77, at], w[262, at] = float("inf"), 3.4028e38
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    for _ in range(20):
        got = ops.gemm_f32_tcgen05(x, w, status=st, tile=tile, splits=splits)
    want = x.double() @ w.double().T
    assert st.item() == 0 and torch.equal(torch.isinf(got), torch.isinf(want.float())) and not got.isnan().any()
    live = torch.isfinite(want.float())
    assert ((got.double() - want).abs() <= _bound(x, w))[live].all()
