"""Steps cut into parts of few keys (attention_plan.plan_attention, part_keys): every key once, within the capacities of a captured step."""

import random

import numpy as np
import pytest

from paged_llm_rs_b200.kernels import attention_plan as P


@pytest.mark.parametrize("tile,ctas,window", [(16, 8, None), (8, 4, 300), (32, 2, None), (4, 64, None), (32, 1, 70)])
def test_parts_cover_every_key_once(tile, ctas, window):
    rng = random.Random(7 * tile + ctas)
    target = 296
    for _ in range(60):
        segments, at = [], 0
        for _ in range(rng.randint(1, 6)):
            n = rng.choice([1, 1, rng.randint(2, 40), rng.randint(2, 250)])
            segments.append((at, n, rng.choice([0, rng.randint(0, 90), rng.randint(0, 30000)])))
            at += n
        work, red, parts = P.plan_attention(segments, tile, window, ctas, target, part_keys=P.F32_PART_KEYS)
        most = P.plan_limits(at, tile, target, ctas, len(segments))
        assert len(work) <= most[0] and len(red) <= most[1] and parts <= most[2]
        whole, _, _ = P.plan_attention(segments, tile, window, ctas, 1, chunk=0)
        tiles = {}
        for seg, q0, qn, p0, begin, end, part, split in work.tolist():
            tiles.setdefault((seg, q0, qn, p0), []).append((begin, end, part, split))
        assert set(tiles) == {tuple(r[:4]) for r in whole.tolist()}
        rows = []
        for seg, q0, qn, p0, begin, end, _, _ in whole.tolist():
            mine = tiles[seg, q0, qn, p0]
            assert mine[0][0] == begin and mine[-1][1] == end and all(a[1] == b[0] for a, b in zip(mine, mine[1:])) and len(mine) <= P.MAX_SPLITS
            assert all((b - begin) % P.SPLIT_ALIGN == 0 for b, _, _, _ in mine)
            if len(mine) == 1:
                assert mine[0][2:] == (-1, 0)
            else:
                assert [s for _, _, _, s in mine] == [len(mine) << 16 | k for k in range(len(mine))]
                rows += [p + t for _, _, p, _ in mine for t in range(qn)]
        assert sorted(rows) == list(range(parts))
        want = {(q0 + t, m[0][2] + t, len(m), qn) for (_, q0, qn, _), m in tiles.items() if len(m) > 1 for t in range(qn)}
        assert want == {tuple(r) for r in red.tolist()}


def test_single_tokens_alone_are_cut_as_before():
    segments = [(i, 1, 100 * i + 5) for i in range(9)]
    a = P.plan_attention(segments, 16, None, 8, 296)
    b = P.plan_attention(segments, 16, None, 8, 296, part_keys=P.F32_PART_KEYS)
    assert (a[0] == b[0]).all() and (a[1] == b[1]).all() and a[2] == b[2]


@pytest.mark.parametrize("most", [5, 37, 148, 592])
def test_a_part_is_the_smallest_that_leaves_few_enough(most):
    rng = random.Random(most)
    for _ in range(300):
        keys = np.array([rng.choice([1, rng.randint(1, 300), rng.randint(1, 40000)]) for _ in range(rng.randint(1, most - 1))])
        part = rng.choice([64, P.F32_PART_KEYS, 1000])
        size = P.part_size(keys, part, most)

        def fits(n):
            return int((-(-keys // n)).sum()) <= most and int(keys.max()) <= P.MAX_SPLITS * n
        assert size >= part and (size - part) % P.SPLIT_ALIGN == 0 and fits(size) and (size == part or not fits(size - P.SPLIT_ALIGN))


def test_long_ranges_are_planned_without_trying_every_size():
    # (a portion behind 30 000 tokens: counted, as a time says little on a busy machine)
    sums = []

    class Counted(np.ndarray):
        def sum(self, *a, **k):
            sums.append(1)
            return np.asarray(self).sum(*a, **k)
    P.part_size(np.arange(30000, 30256, 2).view(Counted), P.F32_PART_KEYS, 148)
    assert len(sums) <= 20             # (of some 470 sizes: two logarithms of that, and the sum of the keys)
