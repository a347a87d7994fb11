"""Smaller pieces where a step has too few or too many of the usual ones: gated products in tiles of 32 columns
(csrc/gemm_tcgen05.cu) and single tokens' attention by CTAs of two and of eight consumer
warps (csrc/attention_decode_tma.cu)."""

import numpy as np
import pytest
import torch

import test_kernels_gpu as K
from paged_llm_rs_b200.kernels import attention_plan, ops
from paged_llm_rs_b200.parts.base import AttentionWork

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one tile, as many tiles as SMs and a few more, an odd number of blocks of k, the last rows of a tile missing
@pytest.mark.parametrize("M,n_out,k", [(1, 64, 64), (65, 64, 72), (100, 3072, 1024), (128, 4672, 320), (128, 4736, 320), (129, 2304, 136), (255, 2368, 1096)])
@pytest.mark.parametrize("act", ["silu", "relu", "clamped"])
def test_gated_products_in_narrow_tiles(M, n_out, k, act):
    g = torch.Generator(device=DEV).manual_seed(M + n_out + k)
    x = torch.randn(M, k, device=DEV, generator=g).bfloat16()
    w = (torch.randn(2 * n_out, k, device=DEV, generator=g) * 0.05).bfloat16()
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    y = ops.gemm_tcgen05(x, w, glu=True, status=st, act=act, limit=2.0 if act == "clamped" else 0.0).float()
    assert st.item() == 0
    gate, up = ((x.float() @ h.float().T).bfloat16().float() for h in (w[:n_out], w[n_out:]))
    if act == "silu":
        want = gate * torch.sigmoid(gate) * up
    elif act == "relu":
        want = gate.clamp(min=0) * up
    else:
        c = gate.clamp(max=2.0)
        want = c * torch.sigmoid(1.702 * c) * (up.clamp(-2.0, 2.0) + 1)
    # (another order of the sums flips a rounding of gate or up now and then, which the activation scales by the other factor)
    assert ((y - want).abs() / (1 + gate.abs() + up.abs())).max().item() < 2e-2


@pytest.mark.parametrize("many", [True, False])
@pytest.mark.parametrize("nh,nkv,hd,page", [(16, 8, 128, 16), (32, 8, 128, 64), (8, 8, 64, 8), (24, 8, 128, 32), (64, 8, 64, 16), (4, 2, 128, 256)])
def test_steps_of_single_tokens(nh, nkv, hd, page, many):
    # more CTAs than two an SM; or one for an SM at most, which take whole items by eight warps
    B = ops.sm_count() * 2 // nkv + 5 if many else min(ops.sm_count() // nkv, 18)
    rng = np.random.default_rng(nh + page)
    ctxs = [0, 1, 15, 16, 31, 32, 33, 63, 64, 127, 700, 128, 129, 511, 383, 1400][:B] + [int(c) for c in rng.integers(0, 300, max(0, B - 16))]
    width = max(c // page + 1 for c in ctxs)
    n_pages = sum(c // page + 1 for c in ctxs) + 2
    order = iter(rng.permutation(n_pages).tolist())
    tables = np.full((B, width), -1, np.int32)
    for r, c in enumerate(ctxs):
        for b in range(c // page + 1):
            tables[r, b] = next(order)
    g = torch.Generator(device=DEV).manual_seed(nh)
    kp, vp = (torch.randn(n_pages, nkv, page, hd, device=DEV, generator=g).bfloat16() for _ in range(2))
    qkv = torch.randn(B, (nh + 2 * nkv) * hd, device=DEV, generator=g).bfloat16()
    gain = 1 + 0.1 * torch.randn(hd, device=DEV, generator=g)
    for target in (1, 10 ** 6) if many else (1,):            # whole; split
        work, red, parts = attention_plan.plan_attention([(r, 1, c) for r, c in enumerate(ctxs)], 1, None, nkv, target, min_split_keys=64)
        dev = lambda a, n: torch.from_numpy(np.ascontiguousarray(a if len(a) else np.zeros((1, n), np.int32))).to(DEV)
        w = AttentionWork(dev(work, 8), torch.tensor([len(work)], dtype=torch.int32, device=DEV), len(work), dev(red, 4),
                          torch.tensor([len(red)], dtype=torch.int32, device=DEV), len(red), torch.zeros(max(parts, 1), nh, hd, device=DEV),
                          torch.zeros(max(parts, 1), nh, 2, device=DEV), kinds=1, reduces=many)
        k2, v2, out, st = kp.clone(), vp.clone(), torch.zeros(B, nh * hd, dtype=torch.bfloat16, device=DEV), K.status()
        ops.decode_attention_fused(qkv, gain, gain, 1e-6, None, None, k2, v2, torch.from_numpy(tables).to(DEV), w, out, nh, nkv, hd, hd ** -0.5, st)
        assert st.item() == 0

        def rows(pool, r, n):                                # a request's rows as they lie: chunk c of the row at offset o at c ^ (o & 7)
            t = torch.cat([pool[p] for p in tables[r, :(n - 1) // page + 1]], 1)[:, :n]
            at = torch.arange(n, device=DEV) % page & 7
            idx = (torch.arange(hd // 8, device=DEV)[None, :] ^ at[:, None])[None, :, :, None].expand(nkv, n, hd // 8, 8)
            return t.view(nkv, n, hd // 8, 8).gather(2, idx).reshape(nkv, n, hd).double()
        norm = lambda x: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * gain.double()
        for r, c in enumerate(ctxs):
            f = qkv[r].double().view(nh + 2 * nkv, hd)
            q, k_new, v_new = norm(f[:nh]), norm(f[nh:nh + nkv]), f[nh + nkv:]
            k, v = rows(k2, r, c + 1), rows(v2, r, c + 1)
            assert torch.equal(v[:, c], v_new) and (k[:, c] - k_new).abs().max().item() < 2 ** -7 * (1 + k_new.abs().max().item())
            assert torch.equal(k[:, :c], rows(kp, r, c + 1)[:, :c])
            s = torch.einsum("gpd,gnd->gpn", q.view(nkv, nh // nkv, hd).bfloat16().double(), k) * hd ** -0.5
            want = torch.einsum("gpn,gnd->gpd", torch.softmax(s, -1), v).reshape(-1)
            # weights rounded to bfloat16 (2^-9 each, of values up to 4.5) and the result once more; q's rounding may differ by an ulp
            assert (out[r].double() - want).abs().max().item() < 5e-2


# (a lane holds a chunk of a head and its rotation's partner: heads of 8, 16 and 32 chunks, numbers of heads that leave lanes and warps without one)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd", [(16, 8, 128), (5, 1, 64), (3, 3, 256), (33, 11, 128), (1, 1, 32)])
@pytest.mark.parametrize("rope,norm", [(True, True), (False, True), (True, False)])
def test_norm_and_rotation_of_many_tokens(dtype, nh, nkv, hd, rope, norm):
    T, page = 300, 16
    chunks = hd * (4 if dtype == torch.float32 else 2) // 16
    swizzled = chunks % 8 == 0
    g = torch.Generator(device=DEV).manual_seed(nh + hd)
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, device=DEV, generator=g).to(dtype)
    qg, kg = (1 + 0.1 * torch.randn(hd, device=DEV, generator=g) for _ in range(2)) if norm else (None, None)
    cos, sin = (torch.randn(400, hd // 2, device=DEV, generator=g) for _ in range(2)) if rope else (None, None)
    pos = torch.randperm(400, device=DEV, generator=g)[:T].to(torch.int32)
    slots = torch.randperm(20 * page, device=DEV, generator=g)[:T].to(torch.int32)
    slots[7] = -1
    pools = [torch.zeros(20, nkv, page, hd, device=DEV, dtype=dtype) for _ in range(2)]
    q, st = torch.empty(T, nh * hd, device=DEV, dtype=dtype), K.status()
    ops.qk_norm_rope_kv(qkv, q, qg, kg, 1e-6, cos, sin, hd if rope else 0, pos, slots, *pools, nh, nkv, hd, st, swizzled=swizzled)
    assert st.item() == 0
    x = qkv.double().view(T, nh + 2 * nkv, hd)

    def made(y, gain):
        if gain is not None:
            y = y * torch.rsqrt((y * y).mean(-1, keepdim=True) + 1e-6) * gain.double()
        if rope:
            c, s = cos.double()[pos.long()][:, None], sin.double()[pos.long()][:, None]
            a, b = y[..., :hd // 2], y[..., hd // 2:]
            y = torch.cat([a * c - b * s, b * c + a * s], -1)
        return y
    want_q, want_k, want_v = made(x[:, :nh], qg), made(x[:, nh:nh + nkv], kg), x[:, nh + nkv:]
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21          # one rounding, and some of float's before it
    near = lambda a, b: ((a.double() - b).abs() <= eps * (1 + b.abs().amax(-1, keepdim=True))).all()
    assert near(q.view(T, nh, hd), want_q)
    for pool, want in zip(pools, (want_k, want_v)):
        rows = pool.transpose(1, 2).reshape(20 * page, nkv, hd)
        got = rows[slots.long().clamp(min=0)]
        if swizzled:
            at = slots.clamp(min=0) % page & 7
            idx = (torch.arange(chunks, device=DEV)[None, :] ^ at[:, None])[:, None, :, None].expand(T, nkv, chunks, hd // chunks)
            got = got.view(T, nkv, chunks, -1).gather(2, idx.long()).reshape(T, nkv, hd)
        keep = slots >= 0
        assert near(got[keep], want[keep])
        untouched = torch.ones(20 * page, dtype=torch.bool, device=DEV)
        untouched[slots[keep].long()] = False
        assert not rows[untouched].any()


def test_gains_and_tables_off_sixteen_bytes():
    # (the vector loads ask for such boundaries: elsewhere the values are fetched one by one)
    nh, nkv, hd, page, T = 8, 4, 128, 16, 300
    g = torch.Generator(device=DEV).manual_seed(3)
    off = lambda t: torch.cat([torch.zeros(1, device=DEV), t.reshape(-1)])[1:].view(t.shape)
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, device=DEV, generator=g).bfloat16()
    qg, kg, cos, sin = (torch.randn(*s, device=DEV, generator=g) for s in ((hd,), (hd,), (T, hd // 2), (T, hd // 2)))
    pos = torch.arange(T, device=DEV, dtype=torch.int32)
    got = []
    for f in (lambda t: t, off):
        for n in (40, T):
            pools = [torch.zeros(T // page + 1, nkv, page, hd, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
            q, st = torch.empty(n, nh * hd, device=DEV, dtype=torch.bfloat16), K.status()
            ops.qk_norm_rope_kv(qkv[:n], q, f(qg), f(kg), 1e-6, f(cos), f(sin), hd, pos[:n], pos[:n], *pools, nh, nkv, hd, st, swizzled=True)
            got.append((q, *pools))
        work, red, parts = attention_plan.plan_attention([(r, 1, 0) for r in range(9)], 1, None, nkv, 1)
        w = AttentionWork(torch.from_numpy(work).to(DEV), torch.tensor([9], dtype=torch.int32, device=DEV), 9, torch.zeros(1, 4, dtype=torch.int32, device=DEV),
                          torch.zeros(1, dtype=torch.int32, device=DEV), 0, torch.zeros(1, nh, hd, device=DEV), torch.zeros(1, nh, 2, device=DEV), kinds=1)
        pools = [torch.zeros(9, nkv, page, hd, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
        out, st = torch.zeros(9, nh * hd, dtype=torch.bfloat16, device=DEV), K.status()
        ops.decode_attention_fused(qkv[:9], f(qg), f(kg), 1e-6, f(cos), f(sin), *pools, torch.arange(9, dtype=torch.int32, device=DEV).view(9, 1), w, out,
                                   nh, nkv, hd, hd ** -0.5, st)
        got.append((out, *pools))
        gu = torch.randn(200, 2048, device=DEV, generator=torch.Generator(device=DEV).manual_seed(9)).bfloat16()
        got.append((ops.swiglu_bias(gu, f(qg.repeat(16)), torch.empty(200, 1024, dtype=torch.bfloat16, device=DEV)),))
    for a, b in zip(got[:4], got[4:]):
        for x, y in zip(a, b):
            # another order of a row's sum flips a rounding now and then: an ulp of bfloat16
            torch.testing.assert_close(x.float(), y.float(), atol=1e-2, rtol=2 ** -7)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd", [(16, 8, 128), (5, 1, 64), (33, 11, 128), (1, 1, 32), (6, 2, 256)])
def test_many_tokens_get_the_same_bits_as_few(dtype, nh, nkv, hd):
    # a CTA a token (from 256 tokens on) and some lanes a head (below): the same sums in the same order, so that a token's key does not
    # depend on how many others its step brings
    T, page = 300, 16
    g = torch.Generator(device=DEV).manual_seed(nh * hd)
    qkv = (torch.randn(T, (nh + 2 * nkv) * hd, device=DEV, generator=g) * 3).to(dtype)
    qg, kg = (1 + 0.1 * torch.randn(hd, device=DEV, generator=g) for _ in range(2))
    angle = torch.rand(T, hd // 2, device=DEV, generator=g) * 6.3
    pos = torch.arange(T, device=DEV, dtype=torch.int32)

    def made(rows):
        pools = [torch.zeros(T // page + 1, nkv, page, hd, device=DEV, dtype=dtype) for _ in range(2)]
        q, st = torch.empty(T, nh * hd, device=DEV, dtype=dtype), K.status()
        for a in range(0, T, rows):
            b = slice(a, min(T, a + rows))
            ops.qk_norm_rope_kv(qkv[b], q[b], qg, kg, 1e-6, angle.cos(), angle.sin(), hd, pos[b], pos[b], *pools, nh, nkv, hd, st)
        assert st.item() == 0
        return (q, *pools)
    for many, few in zip(made(T), made(100)):
        assert torch.equal(many, few)


def _single_tokens(ctxs, work, nh, nkv, hd, page, rope):
    """A step of single tokens whose items are not cut, of which item r begins at its own first key, against 64 bits."""
    B, total, last = len(ctxs), nh + 2 * nkv, max(ctxs)
    rng = np.random.default_rng(B * hd + page)
    n_pages = sum(c // page + 1 for c in ctxs) + 2
    order = iter(rng.permutation(n_pages).tolist())
    tables = np.full((B, last // page + 1), -1, np.int32)
    for r, c in enumerate(ctxs):
        for b in range(c // page + 1):
            tables[r, b] = next(order)
    g = torch.Generator(device=DEV).manual_seed(nh + last)
    kp, vp = (torch.randn(n_pages, nkv, page, hd, device=DEV, generator=g).bfloat16() for _ in range(2))
    qkv = torch.randn(B, total * hd, device=DEV, generator=g).bfloat16()
    qg, kg = (1 + 0.1 * torch.randn(hd, device=DEV, generator=g) for _ in range(2))
    angle = torch.rand(last + 1, hd // 2, device=DEV, generator=g) * 6.3
    cos, sin = (angle.cos(), angle.sin()) if rope else (None, None)
    one = torch.zeros(1, dtype=torch.int32, device=DEV)
    w = AttentionWork(torch.from_numpy(work).to(DEV), one + B, B, torch.zeros(1, 4, dtype=torch.int32, device=DEV), one, 0,
                      torch.zeros(1, nh, hd, device=DEV), torch.zeros(1, nh, 2, device=DEV), kinds=1, reduces=False)
    out, st = torch.zeros(B, nh * hd, dtype=torch.bfloat16, device=DEV), K.status()
    ops.decode_attention_fused(qkv, qg, kg, 1e-6, cos, sin, kp, vp, torch.from_numpy(tables).to(DEV), w, out, nh, nkv, hd, hd ** -0.5, st)
    assert st.item() == 0

    def made(x, gain, c):
        x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * gain.double()
        if rope:
            a, b, co, si = x[..., :hd // 2], x[..., hd // 2:], cos[c].double(), sin[c].double()
            x = torch.cat([a * co - b * si, b * co + a * si], -1)
        return x.bfloat16().double()
    for r, c in enumerate(ctxs):
        f = qkv[r].double().view(total, hd)
        begin, n = int(work[r, 4]), c + 1
        at = torch.arange(n, device=DEV) % page & 7
        idx = (torch.arange(hd // 8, device=DEV)[None, :] ^ at[:, None])[None, :, :, None].expand(nkv, n, hd // 8, 8)
        k, v = (torch.cat([p[i] for i in tables[r, :c // page + 1]], 1)[:, :n].reshape(nkv, n, hd // 8, 8).gather(2, idx).reshape(nkv, n, hd).double()
                for p in (kp, vp))                           # (the step has written its own key and value)
        near = (k[:, c] - made(f[nh:nh + nkv], kg, c)).abs()
        assert near.max().item() < 2 ** -6 and torch.equal(v[:, c], f[nh + nkv:])
        s = torch.einsum("gpd,gnd->gpn", made(f[:nh], qg, c).view(nkv, nh // nkv, hd), k[:, begin:]) * hd ** -0.5
        want = torch.einsum("gpn,gnd->gpd", torch.softmax(s, -1), v[:, begin:]).reshape(-1)
        # weights rounded to bfloat16 (2^-9 each, of values up to 4.5) and the result once more; q's rounding may differ by an ulp
        assert (out[r].double() - want).abs().max().item() < 5e-2, (r, c)


# A key range may begin at any multiple of 64, whichever kernel takes it (the eight warps' tiles have 128 keys; pages of 128 tokens and more do
# not hold a whole tile that begins in their middle)
@pytest.mark.parametrize("nh,nkv,hd,page", [(16, 8, 128, 16), (8, 2, 64, 64), (16, 8, 128, 128), (4, 1, 128, 256)])
@pytest.mark.parametrize("chunk", [64, 192])
@pytest.mark.parametrize("ctxs", [[64, 700], [70, 127, 191, 192, 200, 383, 384, 447, 511, 1000]])
def test_key_ranges_that_begin_within_a_tile(nh, nkv, hd, page, chunk, ctxs):
    work, _, parts = attention_plan.plan_attention([(r, 1, c) for r, c in enumerate(ctxs)], 1, None, nkv, 1, chunk=chunk)
    assert parts == 0 and (work[:, 4] % 128 == 64).any()
    _single_tokens(ctxs, work, nh, nkv, hd, page, True)


# One or two requests (eight consumer warps, a ring of three stages of 128 keys) and some more (a ring of two): the edges of a tile, of the ring's
# first turn and of the second, the token's own key in each place of the ring
@pytest.mark.parametrize("rope", [True, False])
@pytest.mark.parametrize("nh,nkv,hd,page", [(16, 8, 128, 16), (32, 8, 64, 64), (6, 1, 128, 8), (2, 2, 64, 256)])
@pytest.mark.parametrize("ctxs", [[0, 1], [126, 127], [128, 129], [255, 256], [383, 384], [385, 511], [767, 768], [900, 15],
                                  [0, 127, 128, 255, 256, 257, 384, 511, 512, 640, 1000]])
def test_whole_contexts_by_eight_warps(nh, nkv, hd, page, rope, ctxs):
    if nkv * len(ctxs) > ops.sm_count():
        pytest.skip("more CTAs than SMs: other kernels")
    work, _, parts = attention_plan.plan_attention([(r, 1, c) for r, c in enumerate(ctxs)], 1, None, nkv, 1)
    assert parts == 0
    _single_tokens(ctxs, work, nh, nkv, hd, page, rope)


@pytest.mark.parametrize("nh,nkv,hd,page", [(16, 8, 128, 16), (8, 4, 64, 32)])
def test_many_requests_with_a_rotation(nh, nkv, hd, page):
    # (more CTAs than two an SM: two consumer warps and tiles of 32 keys)
    ctxs = [(37 * r) % 300 for r in range(2 * ops.sm_count() // nkv + 5)]
    work, _, parts = attention_plan.plan_attention([(r, 1, c) for r, c in enumerate(ctxs)], 1, None, nkv, 1)
    assert parts == 0
    _single_tokens(ctxs, work, nh, nkv, hd, page, True)


@pytest.mark.parametrize("nh,nkv,hd", [(16, 8, 128), (32, 8, 128), (8, 8, 64), (6, 2, 64), (5, 1, 128), (16, 2, 64)])
@pytest.mark.parametrize("many", [2.0, 1.5, 0.0])
def test_weights_in_two_parts(nh, nkv, hd, many):
    # two, four or eight warps to a CTA (by CTAs an SM), groups of one to eight heads: only the result is rounded to bfloat16
    B, page = int(many * ops.sm_count() / nkv + 1), 16
    ctxs = [(97 * r) % 500 + 3 for r in range(B)]
    g = torch.Generator(device=DEV).manual_seed(nh * hd + B)
    width = max(ctxs) // page + 1
    tables = torch.arange(B * width, device=DEV, dtype=torch.int32).view(B, width)
    kp, vp = (torch.randn(B * width, nkv, page, hd, device=DEV, generator=g).bfloat16() for _ in range(2))
    qkv = torch.randn(B, (nh + 2 * nkv) * hd, device=DEV, generator=g).bfloat16()
    work, _, _ = attention_plan.plan_attention([(r, 1, c) for r, c in enumerate(ctxs)], 1, None, nkv, 1)
    one = torch.zeros(1, dtype=torch.int32, device=DEV)
    w = AttentionWork(torch.from_numpy(work).to(DEV), one + B, B, torch.zeros(1, 4, dtype=torch.int32, device=DEV), one, 0,
                      torch.zeros(1, nh, hd, device=DEV), torch.zeros(1, nh, 2, device=DEV), kinds=1, reduces=False)
    out, st = torch.zeros(B, nh * hd, dtype=torch.bfloat16, device=DEV), K.status()
    ops.decode_attention_fused(qkv, None, None, 0.0, None, None, kp, vp, tables, w, out, nh, nkv, hd, hd ** -0.5, st)
    assert st.item() == 0
    for r, c in enumerate(ctxs):
        n = c + 1
        at = torch.arange(n, device=DEV) % page & 7
        idx = (torch.arange(hd // 8, device=DEV)[None, :] ^ at[:, None])[None, :, :, None].expand(nkv, n, hd // 8, 8)
        k, v = (p[tables[r].long()].transpose(0, 1).reshape(nkv, -1, hd)[:, :n].reshape(nkv, n, hd // 8, 8).gather(2, idx).reshape(nkv, n, hd).double()
                for p in (kp, vp))
        s = torch.einsum("gpd,gnd->gpn", qkv[r].double().view(-1, hd)[:nh].view(nkv, nh // nkv, hd), k) * hd ** -0.5
        want = torch.einsum("gpn,gnd->gpd", torch.softmax(s, -1), v).reshape(-1)
        # half a step of the result's bfloat16, and of the weights 2^-17 each (and float's roundings), of values up to 5
        assert ((out[r].double() - want).abs() <= 2.0 ** -8 * want.abs() + 5 * 2.0 ** -16).all(), r
