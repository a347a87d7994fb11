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


@pytest.mark.parametrize("K,splits", [(192, 1), (1032, 1), (192, 2), (1032, 8)])
@pytest.mark.parametrize("M,tile", [(1, 32), (40, 64), (130, 256)])
def test_small_weights(M, tile, K, splits):
    # what is below 2^-110 keeps fewer than 24 bits in three parts: rows of W that hold nothing larger, wholly or in some CTA's share of k
    g = torch.Generator(device=DEV).manual_seed(M + K)
    x, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(264, K, device=DEV, generator=g)
    small = [5, 31, 32, 127, 128, 200, 263]
    w[small] *= torch.tensor([1e-36, 1e-35, 1e-34, 1e-36, 1e-37, 1e-33, 1e-36], device=DEV)[:, None]
    w[40, :K // 2] *= 1e-37
    w[41, K - 70:] *= 1e-37
    w[42] = (w[42] * 1e-36).bfloat16().float()
    got, want = ops.gemm_f32_tcgen05(x, w, tile=tile, splits=splits).double(), x.double() @ w.double().T
    norm = (x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)).clamp(min=1e-300)
    # (as _bound, of the row's own size: K products of it at most)
    assert ((got - want).abs() / norm).max().item() < 2.0 ** -20


@pytest.mark.parametrize("splits", [1, 2])
def test_sums_that_leave_the_range_on_their_way(splits):
    # a first part is rounded up and may take a product out of float's range that is in it; what the further parts bring then has the other sign
    g = torch.Generator(device=DEV).manual_seed(8)
    x, w = torch.randn(40, 192, device=DEV, generator=g) * 0.1, torch.randn(264, 192, device=DEV, generator=g)
    x[:, 7], w[:, 7], x[:, 150], w[:, 150] = 0.0, 0.0, 0.0, 0.0
    x[4, 7], w[9, 7], w[130, 7] = 1.9999 * 2.0 ** 100, 2.0 ** 27, -2.0 ** 120
    x[39, 150], w[263, 150] = -1.9999 * 2.0 ** 90, 2.0 ** 37
    got, want = ops.gemm_f32_tcgen05(x, w, splits=splits), (x.double() @ w.double().T).float()
    assert want[4, 9].isfinite() and want[4, 130] == -float("inf") and want[39, 263].isfinite()
    assert torch.equal(torch.isinf(got), torch.isinf(want)) and not got.isnan().any()
    live = torch.isfinite(want)
    assert ((got.double() - want.double()).abs() <= _bound(x, w))[live].all()


def test_few_tiny_weights_beside_others():
    # A weight that decays: tiny in every row beside weights of the usual size, where what its third part loses is nothing.  Rows of bfloat16's
    # least numbers are their own first part; a product of such a number is cut off by where its leading zeros stand, six bits earlier
    g = torch.Generator(device=DEV).manual_seed(11)
    x, w = torch.randn(70, 512, device=DEV, generator=g), torch.randn(140, 512, device=DEV, generator=g) * 0.02
    w[:, 100] *= 1e-37
    w[50] = 3 * 2.0 ** -133
    x[:, 7] *= 2.0 ** 60
    got, want, bound = ops.gemm_f32_tcgen05(x, w).double(), x.double() @ w.double().T, _bound(x, w)
    bound[:, 50] *= 2 ** 6
    assert ((got - want).abs() <= bound).all() and (bound[:, 50] < 2e-4 * want[:, 50].abs()).all()
