"""Cutting a step's attention into work items for the kernels.

A segment is the run of consecutive tokens one request brings to a step.  It is
cut into tiles of at most ``tile_tokens`` query tokens; a tile attends over the
keys from the start of its first token's window or chunk (or 0) up to its last token.  When a step has
too few tiles to fill the GPU and a tile's key range is long (decoding, or a
short portion late in a long prompt), the range is split and the splits are
combined by the reduce kernel, always in the same order.

Item layout (int32 x 8): seg, first query token (index in the step), query
tokens, position of the first query token, first key, one past the last key,
first partial row or -1 when not split, (splits << 16 | index of this split)
or 0 when not split.  The splits of a tile are consecutive items.
Reduction layout (int32 x 4): token index, first partial row, splits, stride
between the token's partial rows.
"""

from __future__ import annotations

from typing import List, Optional, Sequence, Tuple

import numpy as np

SPLIT_ALIGN = 64   # split boundaries fall on multiples of the kernels' key tiles (32 and 64)
# The shortest split: one tile of keys.  Measured on captured steps of the 0.6B shape (decoded tokens a second
# with 64 / 128 / 256 / 512 keys): batch 1 at context 4096: 1343 / 1266 / 1267 / 1081; batch 1 at context 512:
# 1478 / 1480 / 1450 / 1266; batch 8 at context 512: 10484 / 10490 / 9700 / 8648.  (Before the reduction's list
# was fetched ahead of its wait and the products' tiles were chosen anew, 256 was the best of these.)
MIN_SPLIT_KEYS = 64
MAX_SPLITS = 128   # the reduce kernel holds the weights of up to 256 splits in shared memory
# A tile of many query tokens is cut only where every part still has this many keys: its partial results are
# a tile of rows each, not one row (a 512-token portion behind 1024 tokens of context beside one decoded
# token, 0.6B shape: cut in four from 256 keys on, the attention took 25 us a layer and the reduction 17;
# whole, see profiles/prefill_2048_tokens.md).
MULTI_MIN_SPLIT_KEYS = 2048
# The float32 kernel on the CUDA cores needs some 10 us for 64 keys of its tile of 32 rows, so there a part of few keys is worth its partial
# results (part_keys below; us a step of the 0.6B shape whole / in parts of 64 / 128 / 192 / 256 keys: 4 decoded tokens beside 252 behind 100
# 4534 / 4208 / 4207 / 4153 / 4354; 2 beside 60 behind 600 5116 / 2989 / 3051 / 3106 / 3379; 250 alone 3914 / 3709 / 3635 / 3811 / 3909;
# 4 at 1500 beside 40 2732 / 2791 / 2787 / 2513 / 2619).
F32_PART_KEYS = 192


# Single tokens whole (the bulk-copy kernel, csrc/attention_decode_tma.cu, then has eight consumer warps where every CTA gets an SM, here with a ring of three stages) or cut and
# their parts reduced, us a step of the 0.6B shape cut / whole:
#   requests x 8 CTAs   1: 500 tokens 675 / 635, 620 687 / 682, 700 682 / 699    4: 620 769 / 733, 700 744 / 749, 800 750 / 764
#   6: 800 828 / 792, 1200 864 / 864                                             8: 900 849 / 825, 1200 882 / 874, 1400 906 / 915
#   12: 1000 912 / 897, 1500 991 / 983, 2000 1089 / 1104                         16: 300 818 / 791, 1500 1098 / 1069, 4000 1722 / 1670
#   20: 2000 1731 / 1546, 4000 2466 / 2179                                       32: 300 1171 / 1012, 1200 1559 / 1453, 4000 2847 / 2786
WHOLE_KEYS, WHOLE_KEYS_A_CTA, WHOLE_KEYS_MANY = 512, 6, 4096


def whole_keys(ctas: int, target_ctas: int) -> int:
    """The most keys of a single token that is left whole in a step of so many CTAs uncut (csrc/step_pack.cu has the same rule)."""
    return WHOLE_KEYS_MANY if 8 * ctas >= 3 * target_ctas else WHOLE_KEYS + WHOLE_KEYS_A_CTA * ctas


# Contexts of very different lengths: the longest one's CTAs walk on alone when the others have left, where cut in two they walk half as far.  A step
# whole / cut (0.6B shape, 8 CTAs a request; lengths from the longest down by a quarter | a half | nine tenths | one long, the rest an eighth of it):
#   requests  8: 520 tokens .97 .98 1.00 1.02, 760 1.00 1.01 1.01 1.02             12: 640 .96 .97 1.01 1.00, 900 .99 1.01 1.03 1.10
#            16: 640 .95 .95 .97 .95, 1200 .98 .98 1.01 1.06, 4000 .98 1.03 1.10 1.18   (eight warps to a CTA, each CTA an SM)
#            18: 300 .94 .94 .97 .99, 640 .97 .99 1.01 1.04, 1600 .98 1.02 1.07 1.12, 4000 1.03 1.09 1.24 1.30
#            20: 420 .89 .90 .98 1.01, 1200 .88 .92 1.02 1.07, 4000 .87 1.01 1.17 1.30   (cut, its CTAs are more than the SMs have places for)
#            28: 420 .89 .88 .88 1.00, 1200 .91 .93 .96 1.07, 4000 .99 1.05 1.13 1.33    32: 420 .92 .90 .90 1.01, 2200 .95 .98 1.02 1.19
#            36: 300 .98 .99 .98 1.01, 900 .96 1.01 1.03 1.12, 4000 1.01 1.05 1.16 1.32  (small CTAs, for which the cut ones have places again)
# So the longest may be longer than a share of the mean (in fifths) by so many keys: what is then left whole takes .86 to 1.03 of its time cut, and before there was
# this bound 4000 tokens beside 60 took up to 1.39.
EVEN_LARGE, EVEN_CROWDED, EVEN = (4, 480), (6, 320), (5, 192)


def even_enough(longest: int, total: int, items: int, ctas: int, target_ctas: int) -> bool:
    """Whether the contexts of a step of ``items`` single tokens (``total`` keys in all, in ``ctas`` CTAs uncut) are near enough to one another
    to be left whole (csrc/step_pack.cu has the same rule)."""
    fifths, keys = EVEN_LARGE if 16 * ctas <= 7 * target_ctas else EVEN_CROWDED if target_ctas < 2 * ctas and 9 * ctas <= 8 * target_ctas else EVEN
    return 5 * items * longest - fifths * total <= 5 * items * keys


def part_size(keys: np.ndarray, part_keys: int, most: int) -> int:
    """The least of ``part_keys``, ``part_keys`` + 64, .. that cuts key ranges ``keys`` (fewer than ``most``) into ``most`` parts at most and none into
    more than MAX_SPLITS.  From the size that their sum and the longest ask for on, by steps that double and then by halves: tried one
    after the other from ``part_keys`` on, 256 tokens behind 30 000 took 398 us to plan, 100 of them for the rest."""
    def fits(step):
        return int((-(-keys // (part_keys + step * SPLIT_ALIGN))).sum()) <= most
    low = max(0, -(-(max(-(-int(keys.sum()) // most), -(-int(keys.max()) // MAX_SPLITS)) - part_keys) // SPLIT_ALIGN))
    if fits(low):
        return part_keys + low * SPLIT_ALIGN
    by = 1
    while not fits(low + by):
        low, by = low + by, by * 2
    high = low + by                      # (it fits there, and not at low)
    while high - low > 1:
        mid = (low + high) // 2
        low, high = (low, mid) if fits(mid) else (mid, high)
    return part_keys + high * SPLIT_ALIGN


def plan_attention(segments: Sequence[Tuple[int, int, int]], tile_tokens: int, window: Optional[int],
                   ctas_per_item: int, target_ctas: int,
                   min_split_keys: int = MIN_SPLIT_KEYS,
                   multi_min_split_keys: int = MULTI_MIN_SPLIT_KEYS, chunk: int = 0, part_keys: int = 0, whole: bool = False, even: bool = False) -> Tuple[np.ndarray, np.ndarray, int]:
    """segments: (first token index, token count, position of the first token) per
    segment, in step order; ``chunk``: a query reads keys of its own chunk of that many positions only; ``part_keys``: a step with tiles of
    several tokens is cut into parts of that many keys, or of so many more that they stay within twice the target; ``whole``: a step of single
    tokens of which none has more keys than ``whole_keys`` says is not cut; ``even``: nor more than ``even_enough`` allows beside the others.
    Returns (work [n, 8], red [m, 4], partial rows used)."""
    in_parts = part_keys > 0 and any(c > 1 for _, c, _ in segments)
    if len(segments) <= SMALL_PLAN:
        small = _small_plan(segments, tile_tokens, window, ctas_per_item, target_ctas, min_split_keys, multi_min_split_keys, chunk,
                            part_keys if in_parts else 0, whole, even)
        if small is not None:
            return small
    seg_ids, q0s, qns, p0s = [], [], [], []
    if segments and all(c == 1 for _, c, _ in segments):
        # a decode step: one tile per segment, no per-segment array work
        a = np.asarray(segments, dtype=np.int64)
        seg_ids, q0s, qns, p0s = [np.arange(len(a))], [a[:, 0]], [a[:, 1]], [a[:, 2]]
        segments = ()
    for si, (tok0, count, pos0) in enumerate(segments):
        if count <= 0:
            continue
        # last tile first: it has the longest key range, and the kernels deal items to the
        # SMs in list order, so the long ones start early and the short ones fill the end
        starts = np.arange(0, count, tile_tokens, dtype=np.int64)[::-1]
        seg_ids.append(np.full(len(starts), si, dtype=np.int64))
        q0s.append(tok0 + starts)
        qns.append(np.minimum(tile_tokens, count - starts))
        p0s.append(pos0 + starts)
    if not seg_ids:
        return np.zeros((0, 8), np.int32), np.zeros((0, 4), np.int32), 0
    seg = np.concatenate(seg_ids); q0 = np.concatenate(q0s); qn = np.concatenate(qns); p0 = np.concatenate(p0s)
    kv_end = p0 + qn
    kv_begin = np.maximum(0, p0 - (window - 1)) if window else (p0 - p0 % chunk if chunk else np.zeros_like(p0))
    n_tiles = len(seg)
    keys = kv_end - kv_begin

    splits = np.ones(n_tiles, dtype=np.int64)
    if in_parts:
        most = 2 * target_ctas // ctas_per_item
        if n_tiles < most:
            splits = -(-keys // part_size(keys, part_keys, most))
            # (single tokens are cut as finely as by the rule below where that stays within the bound too)
            finer = np.where(qn == 1, np.maximum(splits, np.minimum(min(target_ctas // (n_tiles * ctas_per_item), MAX_SPLITS),
                                                                    keys // min_split_keys)), splits)
            if int(finer.sum()) <= most:
                splits = finer
    elif n_tiles * ctas_per_item < target_ctas:
        # as many splits as keep the launch within the target (one or two full waves of
        # CTAs), rounded down so that the last wave is not a sliver.  A step of single tokens that
        # falls short of the target is cut in two at least; tiles of many tokens are not (their
        # partial results are large, and a portion that nearly fills the GPU is better left whole).
        want = target_ctas // (n_tiles * ctas_per_item)
        if want < 2:
            want = 2 if int(qn.max()) == 1 else 1
        floor = np.where(qn > 1, max(min_split_keys, multi_min_split_keys), min_split_keys)
        if not whole or int(qn.max()) > 1 or int(keys.max()) > whole_keys(n_tiles * ctas_per_item, target_ctas) or \
                even and not even_enough(int(keys.max()), int(keys.sum()), n_tiles, n_tiles * ctas_per_item, target_ctas):
            splits = np.clip(np.minimum(want, keys // floor), 1, MAX_SPLITS)
    if (splits == 1).all():
        work = np.stack([seg, q0, qn, p0, kv_begin, kv_end, np.full(n_tiles, -1), np.zeros(n_tiles, np.int64)], 1)
        return work.astype(np.int32), np.zeros((0, 4), np.int32), 0

    # every tile into its splits, without a Python loop over tiles
    chunk = -(-keys // splits)
    chunk = -(-chunk // SPLIT_ALIGN) * SPLIT_ALIGN
    n_split = np.where(splits > 1, -(-keys // chunk), 1)           # splits that really hold keys
    total = int(n_split.sum())
    tile_of = np.repeat(np.arange(n_tiles), n_split)
    first = np.cumsum(n_split) - n_split
    k = np.arange(total) - first[tile_of]                          # which split of its tile
    is_split = n_split > 1
    begin = kv_begin[tile_of] + k * chunk[tile_of]
    end = np.where(is_split[tile_of], np.minimum(begin + chunk[tile_of], kv_end[tile_of]), kv_end[tile_of])
    rows_of = np.where(is_split, n_split * qn, 0)                  # partial rows a tile uses
    base = np.cumsum(rows_of) - rows_of
    part = np.where(is_split[tile_of], base[tile_of] + k * qn[tile_of], -1)
    # which split of how many
    split = np.where(is_split[tile_of], (n_split[tile_of] << 16) | k, 0)
    work = np.stack([seg[tile_of], q0[tile_of], qn[tile_of], p0[tile_of], begin, end, part, split], 1)
    st = np.nonzero(is_split)[0]
    tile_r = np.repeat(st, qn[st])                                 # one reduction per token of a split tile
    t_in = np.arange(len(tile_r)) - np.repeat(np.cumsum(qn[st]) - qn[st], qn[st])
    red = np.stack([q0[tile_r] + t_in, base[tile_r] + t_in, n_split[tile_r], qn[tile_r]], 1)
    return work.astype(np.int32), red.astype(np.int32).reshape(-1, 4), int(rows_of.sum())


SMALL_PLAN = 32        # segments, and tiles, of a step that is planned number by number


def _small_plan(segments, tile_tokens, window, ctas_per_item, target_ctas, min_split_keys, multi_min_split_keys, chunk, part_keys=0, whole=False, even=False):
    """``plan_attention`` for a step of few tiles of which none is split (a prompt's portion, as a rule): the same list without the
    forty array operations that cost such a step more than its work (35 to 80 us).  None when it is not one."""
    items, most = [], 0
    for si, (tok0, count, pos0) in enumerate(segments):
        if count <= 0:
            continue
        if len(items) + (count - 1) // tile_tokens >= SMALL_PLAN:
            return None
        for start in range((count - 1) // tile_tokens * tile_tokens, -1, -tile_tokens):
            n, p = min(tile_tokens, count - start), pos0 + start
            begin = max(0, p - (window - 1)) if window else (p - p % chunk if chunk else 0)
            if part_keys and p + n - begin > part_keys:
                return None
            items.append((si, tok0 + start, n, p, begin, p + n, -1, 0))
            most = max(most, n)
    if not items:
        return None
    if len(items) * ctas_per_item < target_ctas:
        want = target_ctas // (len(items) * ctas_per_item)
        if want < 2:
            want = 2 if most == 1 else 1
        if want > 1 and whole and most == 1:
            keys, ctas = [end - begin for _, _, _, _, begin, end, _, _ in items], len(items) * ctas_per_item
            if max(keys) <= whole_keys(ctas, target_ctas) and (not even or even_enough(max(keys), sum(keys), len(items), ctas, target_ctas)):
                want = 1
        if want > 1:
            for _, _, n, _, begin, end, _, _ in items:
                if end - begin >= 2 * (max(min_split_keys, multi_min_split_keys) if n > 1 else min_split_keys):
                    return None       # (in parts, a tile of several tokens has been looked at above)
    return np.array(items, dtype=np.int32), np.zeros((0, 4), np.int32), 0


def plan_limits(max_step_tokens: int, tile_tokens: int, target_ctas: int, ctas_per_item: int = 1,
                max_segments: Optional[int] = None) -> Tuple[int, int, int]:
    """Upper bounds (work items, reductions, partial rows) for any step of at most
    ``max_step_tokens`` tokens (in at most ``max_segments`` segments, when given), so that
    buffers and launch grids can be sized once.  Tight, because a captured step launches the
    bound and the idle CTAs cost time (a CTA of the tcgen05 kernel holds an SM's whole shared
    memory even to find that it has nothing to do)."""
    # Unsplit: one item per tile; a segment of n tokens has at most n / tile + 1 tiles, and there
    # is at most one tile per token.  Split: tiles * ctas_per_item is below the target and each
    # tile is cut into max(2, target // (tiles * ctas_per_item)) parts, which is at most
    # 2 * target / ctas_per_item items in all.
    split_items = -(-2 * target_ctas // max(1, ctas_per_item))
    tiles = max_step_tokens
    if max_segments is not None:
        tiles = min(tiles, max_segments + max_step_tokens // max(1, tile_tokens))
    max_work = max(tiles, split_items)
    max_red = max_step_tokens
    max_parts = split_items * tile_tokens
    return max_work, max_red, max_parts


def many_splits(n_tokens: int, ctas_per_item: int, target_ctas: int) -> bool:
    """Whether a step of this many single tokens is cut into eight splits a tile or more (the
    planner's arithmetic): the reduction kernel then shares an entry's splits out over four
    groups of threads."""
    return target_ctas // max(1, n_tokens * ctas_per_item) >= 8
