"""The tcgen05 product with two CTAs to a tile of 256 x 256 (csrc/gemm_tcgen05.cu) against the kernel with one, at sizes on and off
its tiles: the two add up the same products in the same order."""

import pytest
import torch

from paged_llm_rs_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,tiles_n,K", [(256, 74, 64), (200, 74, 72), (129, 80, 1024), (1024, 19, 320), (833, 22, 4160), (2048, 12, 1024), (2000, 10, 136)])
@pytest.mark.parametrize("glu", [False, True])
def test_pairs_of_ctas(M, tiles_n, K, glu):
    g = torch.Generator(device=DEV).manual_seed(M + tiles_n + K)
    n_out = tiles_n * (128 if glu else 256)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn((2 if glu else 1) * n_out, K, device=DEV, generator=g) * 0.05).bfloat16()
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    y = ops.gemm_tcgen05(x, w, glu=glu, status=st)
    assert st.item() == 0
    # rows one tile at a time are below the rule's line: the kernel with one CTA a tile
    one = torch.cat([ops.gemm_tcgen05(x[r:r + 128].contiguous(), w, glu=glu, status=st) for r in range(0, M, 128)])
    assert st.item() == 0 and torch.equal(y, one)
    if not glu:
        torch.testing.assert_close(y.float(), x.float() @ w.float().T, atol=3e-2, rtol=2e-2)


@pytest.mark.parametrize("M", [256, 900])
@pytest.mark.parametrize("act,limit,f", [("relu", 0.0, lambda g, u: g.clamp(min=0) * u),
                                         ("clamped", 2.0, lambda g, u: g.clamp(max=2.0) * torch.sigmoid(1.702 * g.clamp(max=2.0)) * (u.clamp(-2.0, 2.0) + 1)),
                                         ("squared_relu", None, lambda g: g.clamp(min=0).square())])
def test_pairs_of_ctas_with_the_other_activations(M, act, limit, f):
    g = torch.Generator(device=DEV).manual_seed(M)
    K, n_out = 320, 80 * 256
    glu = limit is not None
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn((2 if glu else 1) * n_out, K, device=DEV, generator=g) * 0.05).bfloat16()
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    run = (lambda r: ops.gemm_tcgen05(r, w, glu=True, status=st, act=act, limit=limit)) if glu else (lambda r: ops.linear_act(r, w, act, status=st))
    y = run(x)
    one = torch.cat([run(x[r:r + 128].contiguous()) for r in range(0, M, 128)])
    assert st.item() == 0 and torch.equal(y, one)
    h = ops.gemm_tcgen05(x, w, status=st).float()       # (the product as it is rounded before the activation reads it)
    want = f(h[:, :n_out], h[:, n_out:]) if glu else f(h)
    # (the activation's result is rounded to bfloat16, and formed with the fast exponential and division)
    torch.testing.assert_close(y.float(), want, atol=1e-3, rtol=2 ** -7)
