"""Steps of single tokens with short contexts, which are not cut (attention_plan.whole_keys): the native packer and the array planner
keep one rule."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from paged_llm_rs_b200.cache.manager import CacheManager
from paged_llm_rs_b200.engine.runner import group_plans
from paged_llm_rs_b200.engine.step import GroupPlanConfig, NativeDecodePacker, StepCaps, StepEntry, StepPacker
from paged_llm_rs_b200.errors import ConfigError
from paged_llm_rs_b200.kernels import attention_plan as P
from paged_llm_rs_b200.parts.attention import GQAttention
from paged_llm_rs_b200.parts.base import PlanWish
from paged_llm_rs_b200.parts.spec import PartSpec
from test_step_pack import FULL, WIN, setup


@pytest.mark.parametrize("target", [64, 296])
@pytest.mark.parametrize("needs,plans", [([FULL], [GroupPlanConfig(8, 8, None, whole=True)]),
                                         ([FULL, WIN], [GroupPlanConfig(8, 2, None, whole=True), GroupPlanConfig(16, 1, 300, whole=True)])])
def test_the_native_packer_leaves_whole_what_the_python_packer_does(needs, plans, target):
    rng = np.random.default_rng(target)
    cache, packer, caps, work_caps, native, out = setup(needs, plans, 2500, 16, 40, 64, target)
    cut = 0
    for trial in range(40):
        n = int(rng.integers(1, 13))
        ids = [f"r{trial}_{i}" for i in range(n)]
        c = 8 * n if len(plans) == 1 else 2 * n
        edge = P.whole_keys(c, target) - 1
        for r in ids:
            ctx = int(rng.choice([0, 63, 64, 300, min(edge, 1000), min(edge + 1, 1000) if trial % 2 else 5]))
            cache.open(r)
            assert cache.reserve(r, ctx + 1)
            cache.commit(r, ctx)
        entries = [StepEntry(r, [int(rng.integers(0, 1000))], [0]) for r in ids]
        want, layout, _ = packer.pack(entries, caps, work_caps, None, None)
        native.pack(entries, None, None)
        assert np.array_equal(out, want), np.nonzero(out != want)[0][:10]
        cut += int(want[layout["g0.n_red"][0]] > 0)
        for r in ids:
            cache.close(r)
    assert 0 < cut < 40


def test_only_short_contexts_of_single_tokens_are_left_whole():
    for ctas, target, n in ((8, 296, 1), (8, 296, 4), (8, 296, 16), (1, 296, 30)):
        most = P.whole_keys(n * ctas, target)
        for longest, whole in ((most, True), (most + 1, False)):
            segments = [(i, 1, 40 + i) for i in range(n - 1)] + [(n - 1, 1, longest - 1)]
            for small in (P.SMALL_PLAN, -1):
                was, P.SMALL_PLAN = P.SMALL_PLAN, small
                try:
                    work, red, parts = P.plan_attention(segments, 8, None, ctas, target, whole=True)
                finally:
                    P.SMALL_PLAN = was
                assert (len(red) == 0) == whole and (len(work) == n) == whole
    mixed = [(0, 1, 600), (1, 9, 30)]
    a, b = (P.plan_attention(mixed, 8, None, 2, 296, whole=w) for w in (False, True))
    assert (a[0] == b[0]).all() and (a[1] == b[1]).all()


def _mixer(rotary, head_dim=128):
    """An attention layer as the planner sees it (no device is touched); ``rotary``: entries of a head that turn, None without an encoding."""
    rt = SimpleNamespace(device=torch.device("cuda"), dtype=torch.bfloat16, trace=None, status=None)
    turn = SimpleNamespace(rotary=lambda: (None, None, rotary) if rotary else None)
    params = dict(hidden_size=256, num_heads=16, num_kv_heads=8, head_dim=head_dim, scale=1.0, **({} if rotary is None else dict(position_encoding="p")))
    return GQAttention(PartSpec("gqa_attention", params, "m"), rt, {"p": turn})


def test_contexts_are_left_whole_for_the_kernel_that_gains_by_it():
    # (a rotation of part of a head: forward() norms and rotates by a kernel of its own, and the attention has four warps)
    assert [_mixer(r).plan_wish(16).whole for r in (None, 0, 128, 64)] == [True, True, True, False]


def test_layers_of_one_group_that_differ_in_how_ranges_are_cut():
    whole, cut = _mixer(128), _mixer(64)
    of = lambda *mixers: (CacheManager([m.cache_need() for m in mixers], 16, 10, 4, torch.bfloat16, "cpu", allocate_device=False), list(mixers).__getitem__)
    for mixers, lenders, want in (((whole, whole), (), True), ((whole, cut), (), False), ((whole, whole), {1}, False), ((cut,), (), False)):
        plan, = group_plans(*of(*mixers), 16, lenders)
        assert plan.whole == want and plan.part_keys == 0
    # a mixer of a caller's own beside them says nothing about it
    wish = whole.plan_wish(16)
    own = SimpleNamespace(cache_need=whole.cache_need, plan_wish=lambda page: PlanWish(wish.tile_tokens, wish.ctas_per_item, wish.heads, wish.head_dim))
    assert not group_plans(*of(whole, own), 16)[0].whole
    parts = lambda n: SimpleNamespace(cache_need=whole.cache_need, plan_wish=lambda page: PlanWish(8, 2, 16, 128, part_keys=n))
    assert group_plans(*of(parts(192), parts(192)), 16)[0].part_keys == 192 and group_plans(*of(parts(192), parts(0)), 16)[0].part_keys == 0
    other = SimpleNamespace(cache_need=whole.cache_need, plan_wish=lambda page: PlanWish(7, 2, 16, 128))
    with pytest.raises(ConfigError):
        group_plans(*of(parts(0), other), 16)


@pytest.mark.parametrize("target,ctas", [(296, 8), (296, 4), (296, 1), (200, 2)])
def test_contexts_of_very_different_lengths_are_cut(target, ctas):
    # one long context beside short ones: its CTAs would walk on alone when the others have left
    for n in (2, 5, 12, 16, 17, 20, 32, 34, 60):
        if n * ctas >= target:
            continue
        most = P.whole_keys(n * ctas, target)
        for longest, rest in ((most, most), (most, most * 7 // 8), (most, 40), (700, 40), (300, 250), (min(most, 200), 40)):
            segments = [(i, 1, rest - 1) for i in range(n - 1)] + [(n - 1, 1, longest - 1)]
            keys = [rest] * (n - 1) + [longest]
            near = P.even_enough(max(keys), sum(keys), n, n * ctas, target) and max(keys) <= most
            for small in (P.SMALL_PLAN, -1):
                was, P.SMALL_PLAN = P.SMALL_PLAN, small
                try:
                    work, _, _ = P.plan_attention(segments, 8, None, ctas, target, whole=True, even=True)
                    cut, _, _ = P.plan_attention(segments, 8, None, ctas, target)
                finally:
                    P.SMALL_PLAN = was
                assert np.array_equal(work, cut) or near
                assert not near or len(work) == n
    # (what was measured: 20 requests of which one has 4000 tokens took 2009 us whole and 1472 cut, 32 of 2000 to 1500 1453 and 1559)
    assert not P.even_enough(4000, 4000 + 19 * 60, 20, 160, 296) and P.even_enough(2000, 32 * 1750, 32, 256, 296)


@pytest.mark.parametrize("ctas", [1, 2, 8])
def test_the_native_packer_weighs_lengths_as_the_python_packer_does(ctas):
    rng = np.random.default_rng(ctas)
    cache = CacheManager([FULL], 16, 8000, 36, torch.float32, "cpu", prefix_cache=False, allocate_device=False)
    packer = StepPacker(cache, [GroupPlanConfig(8, ctas, None, whole=True)], 296, vocab_size=1000, max_positions=5000, device="cpu")
    caps, work_caps = StepCaps(tokens=36, wanted=36, segments=36, table_width=130), [P.plan_limits(36, 8, 296, ctas)]
    host, layout, _ = packer.pack([], caps, work_caps)
    out = np.zeros_like(host)
    native = NativeDecodePacker(packer, caps, work_caps, layout, out)
    cut = 0
    for trial in range(60):
        n = int(rng.integers(2, 37))
        ids = [f"r{trial}_{i}" for i in range(n)]
        rest = int(rng.choice([30, 200, 700]))
        for i, r in enumerate(ids):
            # the longest context at the edge of what is left whole, and one key beyond it
            fifths, keys = P.EVEN_LARGE if 16 * n * ctas <= 7 * 296 else P.EVEN_CROWDED if 296 < 2 * n * ctas and 9 * n * ctas <= 8 * 296 else P.EVEN
            edge = (5 * n * keys + fifths * rest * (n - 1)) // (5 * n - fifths)
            ctx = max(rest, edge - (trial % 2 == 0)) if i == n - 1 else rest - 1
            cache.open(r)
            assert cache.reserve(r, ctx + 1)
            cache.commit(r, ctx)
        entries = [StepEntry(r, [int(rng.integers(0, 1000))], [0]) for r in ids]
        want, layout, _ = packer.pack(entries, caps, work_caps, None, None)
        native.pack(entries, None, None)
        assert np.array_equal(out, want), np.nonzero(out != want)[0][:10]
        cut += int(want[layout["g0.n_red"][0]] > 0)
        for r in ids:
            cache.close(r)
    assert 0 < cut < 60
