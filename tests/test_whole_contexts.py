"""Steps of single tokens with short contexts, which are not cut (attention_plan.whole_keys): the native packer and the array planner
keep one rule."""

import numpy as np
import pytest

from paged_llm_rs_b200.cache.manager import CacheManager
from paged_llm_rs_b200.engine.step import GroupPlanConfig, StepEntry
from paged_llm_rs_b200.kernels import attention_plan as P
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
