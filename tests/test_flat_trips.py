"""Flat scoring calls whose pairs take a CTA of LegacyFlatScoreKernel
(beam_gb300/csrc/legacy_scoring.cu) several trips round its loop.

On the CPU: the kernel's passes and barriers restated warp by warp under random
schedules. The flags of the long pairs are read by passes that may be skipped,
and a skipped pass has no barrier, so a trip that is not the last has to end with one.

On the GPU: more than four trips of pairs, long and short ones changing places
from trip to trip, against the oracle. Integer work: every value must be equal."""

import random
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))

WARPS = 8
TRIP = 152 * 16 * WARPS  # pairs of one trip of the whole grid


class Stuck(Exception):
    pass


def run_cta(pairs, closing, rng):
    """One CTA over `pairs` ((long?, value) each, WARPS a trip), one step of one
    warp at a time; returns the results. closing: a barrier between two trips."""
    is_long, part, out = [False] * WARPS, [0] * WARPS, [None] * len(pairs)

    def warp(me):
        for w0 in range(0, len(pairs), WARPS):
            for p in range(WARPS + 1):
                which = me if p == 0 else p - 1
                if p > 0:
                    yield "step"
                    if not is_long[which]:
                        continue
                w = w0 + which
                mine = w < len(pairs) and (p > 0 or not pairs[w][0])
                share = 0
                if mine:
                    yield "step"  # the rows
                    share = pairs[w][1] * (me + 1) if p > 0 else pairs[w][1]
                if p > 0:
                    part[me] = share
                    yield "barrier"
                    share = sum(part)
                if mine and (p == 0 or me == 0):
                    out[w] = share
                if p == 0:
                    is_long[me] = w < len(pairs) and not mine
                yield "barrier"
            if closing and w0 + WARPS < len(pairs):
                yield "barrier"

    warps = {i: warp(i) for i in range(WARPS)}
    waiting = set()
    while warps:
        ready = [i for i in warps if i not in waiting]
        if not ready:
            waiting.clear()
            continue
        i = rng.choice(ready)
        for _ in range(rng.choice((1, 1, 3, 30))):  # some warps run far ahead
            try:
                if next(warps[i]) == "barrier":
                    waiting.add(i)
                    break
            except StopIteration:
                if waiting:
                    raise Stuck
                del warps[i]
                break
    return out


def want(pairs):
    return [v * sum(range(1, WARPS + 1)) if long else v for long, v in pairs]


def test_flags_are_read_before_the_next_trip_writes_them():
    rng = random.Random(3)
    wrong = 0
    for trial in range(400):
        pairs = [(rng.random() < rng.choice((0.0, 0.2, 0.6)), rng.randint(1, 1000)) for _ in range(rng.randint(9, 45))]
        assert run_cta(pairs, True, rng) == want(pairs)
        try:
            wrong += run_cta(pairs, False, rng) != want(pairs)
        except Stuck:
            wrong += 1
    assert wrong > 0  # what the closing barrier is for


@pytest.mark.gpu
@pytest.mark.parametrize("count", [TRIP + 1, 2 * TRIP + 7, 4 * TRIP + 4099])
def test_gpu_matches_oracle_over_several_trips(count):
    from beam_gb300 import FlatScorer
    from oracle import legacy_flat_gains
    rng = np.random.default_rng(count)
    rows, ids = 600, 30000
    size_of = rng.integers(1, 50, size=ids)
    reps = np.sort(rng.choice(ids, size=rows, replace=False))
    nb = [np.unique(rng.integers(0, ids, size=rng.integers(300, 900) if i % 2 else rng.integers(0, 12)))
          for i in range(rows)]
    offsets = np.concatenate([[0], np.cumsum([len(x) for x in nb])])
    nb = np.concatenate(nb)
    owner = np.repeat(np.arange(rows), np.diff(offsets))
    s, sx = size_of[reps][owner], size_of[nb]
    cap = np.where(nb == reps[owner], s * (s - 1) // 2, s * sx)
    flat = {"offsets": offsets, "reps": reps, "rsz": size_of[reps], "self": size_of[reps] // 3, "nb": nb,
            "wt": 1 + rng.integers(0, 1 << 30, size=len(nb)) % np.maximum(cap, 1), "nsz": sx}
    # odd rows are long: a slot's pair is long in one trip and short in the next
    at = np.arange(count)
    odd = (at // TRIP + at + at // WARPS) % 3 == 0
    a = 2 * rng.integers(0, rows // 2, size=count) + odd
    b = (a + 2 * rng.integers(1, rows // 2, size=count)) % rows
    pairs = np.stack([a, b], 1).astype(np.int32)
    want_gain, want_before = legacy_flat_gains(flat, pairs)
    with FlatScorer() as scorer:
        for _ in range(5):
            gain, before = scorer.score(flat, pairs)
            assert np.array_equal(gain, want_gain)
            assert np.array_equal(before, want_before)


def steps(first, end, lane, stride, deep, wrap):
    """Positions that one lane visits of the row entries [first, end): four steps
    of `stride` in flight, in 32-bit arithmetic of the given kind."""
    k0, seen, turns = wrap(first + lane), [], 0
    while k0 < end and turns < 40:  # (a position that wraps never ends)
        for d in range(deep):
            k = wrap(k0 + d * stride)
            if k < end:
                seen.append(k)
        k0 = wrap(k0 + stride * deep)
        turns += 1
    return seen


def lower_bound_mids(lo, hi, at, wrap, mid):
    out = []
    span = hi - lo
    while span > 0:
        if lo < hi:
            m = mid(lo, hi, wrap)
            out.append(m)
            if m < at:
                lo = m + 1
            else:
                hi = m
        span >>= 1
    return out, lo


def test_positions_near_the_largest_entry_count():
    """LegacyRows and FlatLowerBounds on rows that end at 2^31 - 1, the most
    entries a call takes: every position once and none outside the row."""
    def unsigned(x):
        return x % (1 << 32)

    def signed(x):
        return (x + (1 << 31)) % (1 << 32) - (1 << 31)

    top = (1 << 31) - 1
    for length, stride in ((1, 32), (33, 32), (700, 32), (5000, 256), (4096, 256)):
        for end in (top, top - 1, top - 1023, 5000):
            first = end - length
            seen = sorted(k for lane in range(stride) for k in steps(first, end, lane, stride, 4, unsigned))
            assert seen == list(range(first, end))
    wrapped = [k for lane in range(32) for k in steps(top - 33, top, lane, 32, 4, signed)]
    assert min(wrapped) < 0  # what signed positions did there
    rng = random.Random(2)
    for _ in range(2000):
        lo = rng.choice((0, 1 << 30, top - 5000))
        hi = min(top, lo + rng.choice((1, 2, 31, 4999, 1 << 29)))
        at = rng.randint(lo, hi)
        mids, found = lower_bound_mids(lo, hi, at, signed, lambda l, h, w: w(l + ((h - l) >> 1)))
        assert found == at and all(lo <= m < hi for m in mids)
    mids, _ = lower_bound_mids(1 << 30, (1 << 30) + 9, 1 << 30, signed, lambda l, h, w: w(l + h) >> 1)
    assert min(mids) < 0  # what the sum of both ends did there
