"""Host model of the canonical form by image rows (csrc/canon_form.cuh) against the oracle's minimum
over all 2016 matrices: stage 1 keeps, row by row, the maps whose lines reach the smallest patterns;
stage 2 compares what is left.  Sets of every size, unions of parallel lines (whose top rows stay
undecided), and the full set, which every map fixes."""

from __future__ import annotations

import random

import numpy as np
import pytest

from oracle import oracle as orc

FULL = (1 << 49) - 1
POINTS = [(x, y) for x in range(7) for y in range(7)]  # bit 7 x + y


def rot(p, s):
    return (p << s | p >> (7 - s)) & 127


def scaled(p, mu):
    return sum(1 << mu * b % 7 for b in range(7) if p >> b & 1)


def best_shift(p):
    return min(range(7), key=lambda s: (rot(p, s), s))


CANON = [min(rot(scaled(p, mu), s) for mu in range(1, 7) for s in range(7)) for p in range(128)]
MUS = [[mu for mu in range(1, 7) if rot(scaled(p, mu), best_shift(scaled(p, mu))) == CANON[p]]
       for p in range(128)]
INV = [0, 1, 4, 5, 2, 3, 6]  # 1 / q mod 7


def lines_of(S, d):
    """The seven lines of a direction as 7-bit rows."""
    rows = [0] * 7
    for x, y in POINTS:
        if S >> (7 * x + y) & 1:
            if d == 7:
                rows[x] |= 1 << y
            else:  # column x of line y + d x
                rows[(y + d * x) % 7] |= 1 << x
    return rows


def canonical(S):
    if S == FULL:
        return S
    img = [lines_of(S, d) for d in range(8)]
    cand = [(d, l6, dl) for d in range(8) for l6 in range(7) for dl in range(1, 7)
            if img[d][(l6 - dl) % 7]]
    prefix, p = 0, 0
    for r in range(6, 0, -1):
        def value(c, r=r):
            return CANON[img[c[0]][(c[1] + (6 - r) * c[2]) % 7]]
        v = min(map(value, cand))
        cand = [c for c in cand if value(c) == v]
        prefix = prefix << 7 | v
        if v not in (0, 127):
            p = r
            break
    best = None
    for d, l6, dl in cand:
        line = (l6 + (6 - p) * dl) % 7
        for mu in MUS[img[d][line]] if p else range(1, 7):
            rho = best_shift(scaled(img[d][line], mu)) if p else 0
            top = p - 1 if p else 0
            at = (line + dl) % 7 if p else (l6 - dl) % 7
            rows = {}
            for r in range(top, -1, -1):
                rows[r] = scaled(img[d][at], mu)
                at = (at + dl) % 7
            for point in (b for b in range(7) if rows[0] >> b & 1):
                nu = (7 - point) % 7
                neg = (nu - rho) * INV[p] % 7 if p else 0
                s = (rho + neg) % 7 if p else nu
                cur = prefix
                for r in range(top, -1, -1):
                    cur = cur << 7 | rot(rows[r], s)
                    s = (s + neg) % 7
                best = cur if best is None else min(best, cur)
    return best


def line_unions(rng, n):
    out = []
    while len(out) < n:
        a, b = rng.choice([(1, 0), (0, 1), (1, 1), (1, 3), (2, 5)])
        lines = rng.sample(range(7), rng.randint(1, 6))
        m = sum(1 << i for i, (x, y) in enumerate(POINTS) if (a * x + b * y) % 7 in lines)
        if rng.randrange(2):
            m ^= 1 << rng.randrange(49)
        if m:
            out.append(m)
    return out


@pytest.mark.parametrize("case", ["sizes", "lines", "full"])
def test_rows_give_the_smallest_image(case):
    rng = random.Random(case)
    if case == "sizes":
        masks = [sum(1 << i for i in rng.sample(range(49), k)) for k in range(1, 50)
                 for _ in range(3)]
    elif case == "lines":
        masks = line_unions(rng, 60)
    else:
        masks = [FULL, FULL ^ 1, FULL ^ 1 << 48, FULL ^ 0b1001]
    want = orc.canonical_masks(np.array(masks, dtype=np.uint64)).tolist()
    assert [canonical(m) for m in masks] == want
