"""Canonical masks where the row-by-row form can go wrong: every set size,
sets made of whole lines (rows that are empty or full leave the top rows
undecided), subsets of one line, the longest candidate lists (48 and 49
points), and batch sizes around the kernel's groups of four and sixteen."""

from __future__ import annotations

import random

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

FULL = (1 << 49) - 1


def line_sets(rng, n):
    """Unions of parallel lines, some with a point flipped or thinned out."""
    out = []
    while len(out) < n:
        a, b = rng.choice([(1, 0), (0, 1), (1, 1), (1, 3), (2, 5)])
        lines = rng.sample(range(7), rng.randint(1, 6))
        m = sum(1 << i for i in range(49) if (a * (i // 7) + b * (i % 7)) % 7 in lines)
        kind = rng.randrange(3)
        if kind == 1:
            m ^= 1 << rng.randrange(49)
        elif kind == 2:
            m &= rng.getrandbits(49)
        if m:
            out.append(m)
    return out


def random_sets(rng, n, k):
    return [sum(1 << p for p in rng.sample(range(49), k)) for _ in range(n)]


@pytest.mark.parametrize("case", ["sizes", "lines", "full", 1, 3, 5, 15, 17, 33])
def test_masks_vs_oracle(canon_oracle, case):
    rng = random.Random(str(case))
    if case == "sizes":
        masks = [m for k in range(1, 50) for m in random_sets(rng, 4, k)]
    elif case == "lines":
        masks = line_sets(rng, 200)
    elif case == "full":
        masks = [FULL, FULL ^ 1, FULL ^ (1 << 48), FULL ^ 0b1001] * 3
    else:
        masks = random_sets(rng, case, 9)
    masks = np.array(masks, dtype=np.uint64)
    assert np.array_equal(canon_oracle.compute_masks(masks), orc.canonical_masks(masks))
