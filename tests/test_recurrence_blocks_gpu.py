"""The matrix LSTM and the gated delta rule in blocks of tokens (csrc/mlstm_blocks.cuh, csrc/delta_blocks.cuh) against the plain recurrences in float64 and against the kernels
that go token by token: segments that end on and off a block's edge, that begin with and without a state, beside shorter ones
and empty ones."""

import pytest
import torch

import plain_pamarax as P
from paged_llm_rs_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
EPS, CAP = 1e-6, 15.0


def plain(u, gates, ib, fb, gain, H, d, E):
    """One whole sequence, float64 on the CPU; and what float32 may be off by.  A numerator is a sum over d entries of a state
    that is a sum over tokens: its roundings, and those of the weights, are at most some (d + 80) 2^-24 of the same sum of sizes
    (a block adds 64 tokens at a time), which the head's norm divides by the root mean square of the numerators."""
    T = u.shape[0]
    q, k, v, g = torch.split(u.double(), [H * d, H * d, H * E, H * E], 1)
    i = P.capped(gates[:, :H].double() + ib.double(), CAP)
    f = P.logsigmoid(P.capped(gates[:, H:].double() + fb.double(), CAP))
    q, k, v = q.view(T, H, d) * d ** -0.5, k.view(T, H, d), v.view(T, H, E)
    o = P.matrix_memory(q, k, v, i, f)
    F = f.cumsum(0)
    out, off = torch.zeros(T, H, E, dtype=torch.float64), torch.zeros(T, H, E, dtype=torch.float64)
    for h in range(H):
        e = (F[:, None, h] - F[None, :, h] + i[None, :, h]).masked_fill(torch.ones(T, T, dtype=torch.bool).triu(1), float("-inf"))
        m = torch.maximum(e.max(1).values, F[:, h])
        w = torch.exp(e - m[:, None])
        den = torch.maximum((w * (q[:, h] @ k[:, h].T)).sum(1).abs(), torch.exp(-m)) + 1e-6
        size = (w * (q[:, h].abs() @ k[:, h].abs().T)) @ v[:, h].abs() / den[:, None]
        rms = torch.sqrt(o[:, h].pow(2).mean(1, keepdim=True) + EPS)
        out[:, h], off[:, h] = o[:, h] / rms, (size + o[:, h].abs() / rms * size.pow(2).mean(1, keepdim=True).sqrt()) / rms
    after = gain.double() * torch.sigmoid(g)
    return out.reshape(T, H * E) * after, ((d + 80) * 2.0 ** -24 * off + 4 * 2.0 ** -24 * out.abs()).reshape(T, H * E) * after.abs()


def steps(blocks, dtype, cuts, seqs, ib, fb, gain, H, d, E, longest=64):
    """Every sequence through ``cuts`` steps: cuts[s] lists the tokens each takes in step s (0: it is not in the step)."""
    was, ops.MLSTM_BLOCKS, ops.MLSTM_LONGEST = ops.MLSTM_LONGEST, blocks, longest       # (blocks from the first length that has two)
    try:
        state = torch.full((len(seqs) + 1, ops.mlstm_state_floats(H, d, E)), 7.0, device=DEV)       # (whatever an older request left)
        done, outs = [0] * len(seqs), [[] for _ in seqs]
        for cut in cuts:
            segs, us, gs, at = [], [], [], 0
            for r, n in enumerate(cut):
                segs.append((at, n, done[r], r + 1))
                us.append(seqs[r][0][done[r]:done[r] + n])
                gs.append(seqs[r][1][done[r]:done[r] + n])
                at += n
            u, g = torch.cat(us).to(DEV, dtype).contiguous(), torch.cat(gs).to(DEV).contiguous()
            out = torch.empty(at, H * E, dtype=dtype, device=DEV)
            ops.mlstm_mix(u, g, ib.to(DEV), fb.to(DEV), CAP, gain.to(DEV), torch.tensor(segs, dtype=torch.int32, device=DEV), state, out, H, d, E, EPS,
                          max(cut))
            for r, (a, n, _, _) in enumerate(segs):
                outs[r].append(out[a:a + n].cpu())
                done[r] += n
        return [torch.cat(o) for o in outs]
    finally:
        ops.MLSTM_BLOCKS, ops.MLSTM_LONGEST = True, was


@pytest.mark.parametrize("H,d,E", [(2, 8, 4), (1, 36, 68), (4, 128, 256), (1, 256, 64)])
@pytest.mark.parametrize("cuts", [[(65, 1, 0)], [(64, 128, 3), (129, 0, 65)], [(3, 200, 66), (130, 1, 127)]])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_matrix_lstm_in_blocks(dtype, cuts, H, d, E):
    g = torch.Generator().manual_seed(d + E + len(cuts))
    n = [sum(c[r] for c in cuts) for r in range(3)]
    # (strong and weak forget gates, input gates that move the running maximum about)
    seqs = [((torch.randn(t, H * (2 * d + 2 * E), generator=g) * 0.7).to(dtype).float(), torch.randn(t, 2 * H, generator=g) * 6.0) for t in n]
    ib, fb, gain = torch.randn(H, generator=g), torch.randn(H, generator=g) * 3.0, 1 + 0.1 * torch.randn(H * E, generator=g)
    want = [plain(u, gt, ib, fb, gain, H, d, E) if len(u) else None for u, gt in seqs]
    for blocks in (True, False):
        for both, got in zip(want, steps(blocks, dtype, cuts, seqs, ib, fb, gain, H, d, E)):
            if both is None:
                continue
            w, off = both
            # (bfloat16: the same arithmetic, and the result's rounding)
            assert ((got.double() - w).abs() <= off + (2.0 ** -8 * w.abs() if dtype == torch.bfloat16 else 0.0)).all(), blocks


def test_a_later_infinite_value_reaches_no_earlier_token():
    H, d, E = 1, 32, 64
    g = torch.Generator().manual_seed(1)
    u, gates = torch.randn(100, H * (2 * d + 2 * E), generator=g), torch.randn(100, 2 * H, generator=g)
    bad = u.clone()
    bad[70, 2 * H * d:2 * H * d + H * E] = float("inf")
    one = torch.zeros(H), torch.zeros(H), torch.ones(H * E)
    a, b = (steps(True, torch.float32, [(100,)], [(x, gates)], *one, H, d, E)[0] for x in (u, bad))
    assert torch.equal(a[:70], b[:70])


def plain_delta(u, conv_w, ba, a_log, dt, gain, H, G, d, E):
    T = u.shape[0]
    c = 2 * G * d + H * E
    x = P.causal_conv_silu(u[:, :c].double(), conv_w.double())
    q, k, v = x[:, :G * d].view(T, G, d), x[:, G * d:2 * G * d].view(T, G, d), x[:, 2 * G * d:].view(T, H, E)
    beta = torch.sigmoid(ba[:, :H].double())
    g = torch.exp(-torch.exp(a_log.double()) * P.softplus(ba[:, H:].double() + dt.double()))
    o = P.unit_rms(P.gated_delta_rule(P.unit_vector(q) * d ** -0.5, P.unit_vector(k), v, beta, g), EPS) * gain.double()
    return o.reshape(T, H * E) * P.silu(u[:, c:].double())


def delta_steps(blocks, dtype, cuts, seqs, conv_w, a_log, dt, gain, H, G, d, E, most=max, longest=64):
    was, ops.DELTA_BLOCKS, ops.DELTA_LONGEST = ops.DELTA_LONGEST, blocks, longest
    try:
        taps = conv_w.shape[1]
        state = torch.full((len(seqs) + 1, ops.delta_state_floats(H, G, d, E, taps)), 7.0, device=DEV)
        done, outs = [0] * len(seqs), [[] for _ in seqs]
        for cut in cuts:
            segs, us, gs, at = [], [], [], 0
            for r, n in enumerate(cut):
                segs.append((at, n, done[r], r + 1))
                us.append(seqs[r][0][done[r]:done[r] + n])
                gs.append(seqs[r][1][done[r]:done[r] + n])
                at += n
            u, ba = torch.cat(us).to(DEV, dtype).contiguous(), torch.cat(gs).to(DEV).contiguous()
            out = torch.empty(at, H * E, dtype=dtype, device=DEV)
            ops.delta_mix(u, conv_w.to(DEV, dtype), ba, a_log.to(DEV), dt.to(DEV), gain.to(DEV), torch.tensor(segs, dtype=torch.int32, device=DEV),
                          most(cut), state, out, H, G, d, E, taps, EPS)
            for r, (a, n, _, _) in enumerate(segs):
                outs[r].append(out[a:a + n].cpu())
                done[r] += n
        return [torch.cat(o) for o in outs]
    finally:
        ops.DELTA_BLOCKS, ops.DELTA_LONGEST = True, was


@pytest.mark.parametrize("H,G,d,E,taps", [(2, 1, 8, 4, 4), (1, 1, 36, 68, 3), (8, 4, 128, 128, 4), (2, 2, 64, 200, 6), (1, 1, 16, 16, 1)])
@pytest.mark.parametrize("cuts", [[(65, 1, 0)], [(64, 128, 3), (129, 0, 65)], [(3, 200, 66), (130, 1, 127)]])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_delta_rule_in_blocks(dtype, cuts, H, G, d, E, taps):
    g = torch.Generator().manual_seed(d + E + len(cuts))
    n = [sum(c[r] for c in cuts) for r in range(3)]
    c = 2 * G * d + H * E
    # (keys with much in common, so that a token's write depends on many before it; decays from next to none to strong)
    seqs = [((torch.randn(t, c + H * E, generator=g) + 0.7).to(dtype).float(), torch.randn(t, 2 * H, generator=g) * 3.0) for t in n]
    conv_w = (torch.randn(c, taps, generator=g) * 0.5 + 0.3).to(dtype).float()
    a_log, dt, gain = torch.randn(H, generator=g), torch.randn(H, generator=g), 1 + 0.1 * torch.randn(E, generator=g)
    want = [plain_delta(u, conv_w, ba, a_log, dt, gain, H, G, d, E) for u, ba in seqs]
    got, scan = (delta_steps(b, dtype, cuts, seqs, conv_w, a_log, dt, gain, H, G, d, E) for b in (True, False))
    for r in range(3):
        if not n[r]:
            continue
        off, base = (float((x.double() - want[r]).norm() / want[r].norm()) for x in (got[r], scan[r]))
        # float32: the recurrence's own error, which the substitution repeats, within the order of the sums; bfloat16: the result's rounding
        assert off <= (max(2e-6, 1.5 * base) if dtype == torch.float32 else 4e-3), (r, off, base)
        assert ((got[r].double() - want[r]).abs().max() / want[r].abs().max()) <= (1e-4 if dtype == torch.float32 else 2e-2)


def test_a_later_infinite_value_reaches_no_earlier_token_of_the_delta_rule():
    H, G, d, E, taps = 1, 1, 32, 64, 4
    g = torch.Generator().manual_seed(1)
    c = 2 * d + E
    u, ba = torch.randn(100, c + E, generator=g), torch.randn(100, 2 * H, generator=g)
    bad = u.clone()
    bad[70, 2 * d:c] = float("inf")
    rest = torch.rand(c, taps, generator=g), torch.zeros(H), torch.zeros(H), torch.ones(E)
    a, b = (delta_steps(True, torch.float32, [(100,)], [(x, ba)], *rest, H, G, d, E)[0] for x in (u, bad))
    assert torch.equal(a[:70], b[:70])


@pytest.mark.parametrize("gate", [float("inf"), 1e30, 5000.0])
def test_a_gate_that_resets_the_state_resets_it_in_a_block_too(gate):
    # tokens whose decay is exactly zero (one at a block's start, two in a row, one in the last block) beside heads without any
    H, G, d, E, taps = 2, 1, 32, 64, 4
    g = torch.Generator().manual_seed(3)
    c = 2 * G * d + H * E
    u, ba = torch.randn(200, c + H * E, generator=g), torch.randn(200, 2 * H, generator=g)
    ba[[64, 90, 91, 150], H] = gate
    conv_w, a_log, dt, gain = torch.rand(c, taps, generator=g), torch.zeros(H), torch.zeros(H), torch.ones(E)
    want = plain_delta(u, conv_w, ba, a_log, dt, gain, H, G, d, E)
    for blocks in (True, False):
        # (the second step starts from the state that the first one left)
        got = delta_steps(blocks, torch.float32, [(130,), (70,)], [(u, ba)], conv_w, a_log, dt, gain, H, G, d, E)[0]
        assert float((got.double() - want).norm() / want.norm()) <= 2e-6, blocks


@pytest.mark.parametrize("n", [33, 64, 200])
def test_the_delta_rule_takes_segments_of_unknown_length(n):
    # (max_segment_tokens 0: no block path, and every token convolved)
    H, G, d, E, taps = 2, 1, 16, 24, 4
    g = torch.Generator().manual_seed(n)
    c = 2 * G * d + H * E
    u, ba, rest = torch.randn(n, c + H * E, generator=g), torch.randn(n, 2 * H, generator=g), (torch.zeros(H), torch.zeros(H), torch.ones(E), H, G, d, E)
    conv_w = torch.rand(c, taps, generator=g)
    a, b = (delta_steps(False, torch.float32, [(n,)], [(u, ba)], conv_w, *rest, most=most)[0] for most in (lambda cut: 0, max))
    want = plain_delta(u, conv_w, ba, *rest)
    assert torch.equal(a, b) and float((a.double() - want).norm() / want.norm()) <= 2e-6


def test_the_delta_rules_blocks_are_no_further_from_64_bits_than_the_recurrence():
    H, G, d, E, taps = 8, 4, 128, 128, 4
    c = 2 * G * d + H * E
    for off, strength, shift in ((0.7, 3.0, 0.0), (0.0, 3.0, 0.0), (0.0, 1.0, -4.0)):       # (keys alike or not, strong and weak decays)
        ratio = 1.0
        for seed in range(4):
            g = torch.Generator().manual_seed(seed)
            seqs = [(torch.randn(193, c + H * E, generator=g) + off, torch.randn(193, 2 * H, generator=g) * strength)]
            conv_w = torch.randn(c, taps, generator=g) * 0.5 + 0.3
            rest = torch.randn(H, generator=g), torch.randn(H, generator=g) + shift, 1 + 0.1 * torch.randn(E, generator=g), H, G, d, E
            want = plain_delta(*seqs[0][:1], conv_w, seqs[0][1], *rest)
            a, b = (delta_steps(blocks, torch.float32, [(193,)], seqs, conv_w, *rest)[0].double() for blocks in (True, False))
            ratio *= float((a - want).norm() / (b - want).norm())
        # (0.93 to 1.005 measured; the rest is what another four draws move it by)
        assert ratio ** 0.25 <= 1.03, (off, strength, shift, ratio ** 0.25)


@pytest.mark.parametrize("tokens,longest", [(64, 64), (512, 512), (384, 512)])
def test_segments_up_to_the_longest_go_token_by_token(tokens, longest):
    L = ops.lib()
    assert L.pllm_mlstm_block_floats(None, 4 * 768, 2000, 3, tokens, longest, 4, 128, 256) == 0
    assert L.pllm_delta_block_floats(2000, 3, tokens, longest, 8, 4, 128, 128) == 0
    assert L.pllm_mlstm_block_floats(None, 4 * 768, 2000, 3, longest + 1, longest, 4, 128, 256) > 0
    assert L.pllm_delta_block_floats(2000, 3, longest + 1, longest, 8, 4, 128, 128) > 0


@pytest.mark.parametrize("cut", [(70, 300, 90, 512, 40), (513, 100, 640, 385, 3)])
def test_a_step_of_segments_on_both_sides_of_the_longest(cut):
    # (at the lengths the engine uses: some go token by token beside others in blocks, and each keeps its own state)
    H, d, E, G, taps = 2, 32, 64, 2, 4
    g = torch.Generator().manual_seed(sum(cut))
    one = torch.zeros(H), torch.zeros(H), torch.ones(H * E)
    seqs = [(torch.randn(n, H * (2 * d + 2 * E), generator=g), torch.randn(n, 2 * H, generator=g)) for n in cut]
    was = ops.MLSTM_LONGEST, ops.DELTA_LONGEST
    assert min(was) >= 384
    for got, (u, gt) in zip(steps(True, torch.float32, [cut], seqs, *one, H, d, E, longest=was[0]), seqs):
        want, off = plain(u, gt, *one, H, d, E)
        assert ((got.double() - want).abs() <= off).all()
    c = 2 * G * d + H * E
    seqs = [(torch.randn(n, c + H * E, generator=g), torch.randn(n, 2 * H, generator=g)) for n in cut]
    conv_w, rest = torch.rand(c, taps, generator=g), (torch.zeros(H), torch.zeros(H), torch.ones(E), H, G, d, E)
    for got, (u, ba) in zip(delta_steps(True, torch.float32, [cut], seqs, conv_w, *rest, longest=was[1]), seqs):
        want = plain_delta(u, conv_w, ba, *rest)
        assert float((got.double() - want).norm() / want.norm()) <= 2e-6


@pytest.mark.parametrize("taps", [1, 2, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_delta_rules_convolution_from_step_to_step(dtype, taps):
    # (a portion shorter than the taps, then single tokens, a step of single tokens alone having a convolution of its own, then a portion again)
    H, G, d, E = 2, 1, 16, 24
    g = torch.Generator().manual_seed(taps)
    c = 2 * G * d + H * E
    cuts = [(3, 20), (1, 1), (1, 1), (1, 0), (9, 1), (1, 30)]
    n = [sum(cut[r] for cut in cuts) for r in range(2)]
    seqs = [(torch.randn(t, c + H * E, generator=g).to(dtype).float(), torch.randn(t, 2 * H, generator=g)) for t in n]
    conv_w, rest = (torch.randn(c, taps, generator=g) * 0.4).to(dtype).float(), (torch.zeros(H), torch.zeros(H), torch.ones(E), H, G, d, E)
    for got, (u, ba) in zip(delta_steps(True, dtype, cuts, seqs, conv_w, *rest), seqs):
        want = plain_delta(u, conv_w, ba, *rest)
        assert float((got.double() - want).norm() / want.norm()) <= (2e-6 if dtype == torch.float32 else 4e-3)
