"""The passes that take whole vectors where rows and addresses allow it, against float64 at the sizes where that rule turns:
widths on and off a vector, at and past what a row's team holds, and addresses that are no vector's."""

import pytest
import torch

from paged_llm_rs_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = {torch.float32: dict(atol=2e-5, rtol=2e-5), torch.bfloat16: dict(atol=2e-2, rtol=1e-2)}      # (the result's rounding and sums of up to 4100 squares)


def at(shape, dtype, g, off, scale=1.0, add=0.0):
    """Random values whose first entry lies ``off`` entries past a 256-byte boundary."""
    n = 1
    for d in shape:
        n *= d
    t = torch.empty(n + off, dtype=dtype, device=DEV)
    t[off:] = (torch.randn(n, device=DEV, generator=g) * scale + add).to(dtype)
    return t[off:].view(shape)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n,W", [(1, 4), (3, 36), (70, 1024), (65, 130), (5, 4096), (2, 4100)])
def test_sandwich_norm(dtype, n, W, off):
    g = torch.Generator(device=DEV).manual_seed(n + W + off)
    eps = 1e-6

    def norm(v, gain):
        return v * torch.rsqrt(v.square().mean(-1, keepdim=True) + eps) * gain
    a, bias, ga, gy = at((n, W), dtype, g, off), at((W,), torch.float32, g, off, 0.1), at((W,), torch.float32, g, off, 0.1, 1.0), at((W,), torch.float32, g, 0, 0.1, 1.0)
    for use_a, use_bias, use_y, picked in ((1, 1, 1, 0), (1, 0, 1, 0), (0, 0, 1, 0), (1, 1, 0, 0), (1, 1, 1, 1), (0, 0, 1, 1)):
        x = at((n, W), torch.float32, g, off)
        was = x.clone()
        rows = torch.tensor([n - 1, 0], dtype=torch.int32, device=DEV) if picked else None
        y = at((2 if picked else n, W), dtype, g, off) if use_y else None
        ops.sandwich_norm32(x, a if use_a else None, bias if use_bias else None, ga if use_a else None, gy if use_y else None, y, eps, rows=rows)
        want = was.double() + (norm(a.double() + (bias.double() if use_bias else 0.0), ga.double()) if use_a else 0.0)
        torch.testing.assert_close(x.double(), was.double() if picked else want, **TOL[torch.float32])
        if use_y:
            out = norm(want, gy.double())
            torch.testing.assert_close(y.double(), out[rows.long()] if picked else out, **TOL[dtype])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n,width", [(1, 8), (3, 20), (130, 1024), (1025, 3072), (7, 1032), (127, 1024), (128, 1032)])
def test_biased_gated_activation_and_gate(dtype, n, width, off):
    g = torch.Generator(device=DEV).manual_seed(n + width + off)
    gu, bias = at((n, 2 * width), dtype, g, off), at((2 * width,), torch.float32, g, off, 0.3)
    v = gu.double() + bias.double()
    gate, up = v[:, :width], v[:, width:]
    out = at((n, width), dtype, g, off)
    for act, limit, want in (("silu", 0.0, gate * torch.sigmoid(gate) * up), ("relu", 0.0, gate.clamp(min=0) * up),
                             ("clamped", 1.5, gate.clamp(max=1.5) * torch.sigmoid(1.702 * gate.clamp(max=1.5)) * (up.clamp(-1.5, 1.5) + 1))):
        torch.testing.assert_close(ops.swiglu_bias(gu, bias, out, act, limit).double(), want, **TOL[dtype])
    # the gate as a column range of a wider tensor
    z = gu[:, width:]
    for kind, f in (("sigmoid", torch.sigmoid), ("silu", lambda t: t * torch.sigmoid(t))):
        y = at((n, width), dtype, g, off)
        want = y.double() * f(z.double())
        torch.testing.assert_close(ops.gate_mul(y, z, kind).double(), want, **TOL[dtype])
