"""Host model of the toric walk (csrc/toric_walk.cuh).

  * tw_next: the stages a code goes through, whatever its best weight does
    meanwhile, end, each has work, and the bounds they rest on hold (checked
    by enumerating whole toric codes).
  * tw_us / tw_u / tw_pair: the u's and pairs of every pivot row give each
    message of a stage once; the pieces of a batch tile its pairs.
  * tw_count: the carry-save counter tells exactly which sums reach the top.
"""

from __future__ import annotations

import itertools
import random
from math import comb

import pytest

from generalized_toric_gpu_search_b200.tables import build_eval_matrix, gf8_mul

N = 49
MAX_K = 21
COMBS = {b: sorted(itertools.combinations(range(MAX_K), b), key=lambda r: r[::-1])
         for b in range(1, 5)}


def cdiv(a, b):
    return -(-a // b)


def tw_next(k, best, wthr, level, p1):
    """(stage, level after, p1 after) or None when the code is settled; a
    stage is (w, a, b_lo, b_hi, avoid, forced)."""
    if best < wthr or level >= k or cdiv(N * (level + 1), k) >= best:
        return None
    w = level + 1
    if p1 and cdiv(N * w, k - 1) >= best:
        return None
    avoid = -1
    while avoid < 3 and k - (avoid + 1) >= w and cdiv(N * (w + 1), k + avoid + 1) >= best:
        avoid += 1
    last_row = not p1 and cdiv(N * w, k - 1) >= best
    if last_row and (avoid < 0 or comb(k - 1, w - 1) <= comb(k - avoid, w)) or (
            not p1 and w > 4 and avoid < 0):
        return (w, 0, 1), level, True
    if avoid > 0 or p1:
        return (w, max(avoid, 1), 0), (k if avoid > 0 else w), False
    return (w, 0, 0), w, p1


def n_us(k, stage, p):
    w, avoid, forced = stage
    rows, picks = k - avoid - 1 - p - forced, w - 3 - forced
    return comb(rows, picks) * 7 ** (w - 3) if rows >= picks and p >= 2 else 0


def n_pairs(p):
    return 49 * (p * (p - 1) // 2)


def u_rows(k, stage, p, o):
    """Message {row: exponent} of u number o of pivot row p."""
    w, avoid, forced = stage
    picks = w - 3 - forced
    msg = {p: 0}
    if forced:
        msg[k - 1] = o % 7
        o //= 7
    dig = []
    for _ in range(picks):
        dig.append(o % 7)
        o //= 7
    if 0 < picks <= 4:
        rows = COMBS[picks][o]
    else:
        rows, r = [], k
        for j in range(picks, 0, -1):
            r -= 1
            while comb(r, j) > o:
                r -= 1
            o -= comb(r, j)
            rows.append(r)
    for r, d in zip(rows, dig):
        assert p + 1 + r not in msg
        msg[p + 1 + r] = d
    return msg


def pair_rows(e):
    lo, hi = COMBS[2][e // 49]
    return {lo: e % 49 // 7, hi: e % 7}


def stage_messages(k, stage):
    for p in range(k):
        for o in range(n_us(k, stage, p)):
            u = u_rows(k, stage, p, o)
            for e in range(n_pairs(p)):
                v = pair_rows(e)
                assert not set(u) & set(v)
                yield {**u, **v}


def wanted_messages(k, stage):
    w, avoid, forced = stage
    for sup in itertools.combinations(range(k - avoid), w):
        if forced and sup[-1] != k - 1:
            continue
        pivot = sup[2]
        free = [r for r in sup if r != pivot]
        for d in itertools.product(range(7), repeat=w - 1):
            yield dict(zip(free, d)) | {pivot: 0}


@pytest.mark.parametrize("k, stage", [
    (4, (4, 0, 0)), (4, (4, 0, 1)), (5, (4, 0, 0)), (6, (4, 1, 0)), (6, (4, 0, 1)),
    (6, (5, 0, 1)), (6, (5, 1, 0)), (5, (5, 0, 0)), (6, (6, 0, 0))])
def test_lists_cover_a_stage_once(k, stage):
    got = sorted(tuple(sorted(m.items())) for m in stage_messages(k, stage))
    want = sorted(tuple(sorted(m.items())) for m in wanted_messages(k, stage))
    assert got == want


def test_deep_levels_unrank_every_pick():
    for k, stage in ((11, (8, 0, 0)), (12, (9, 0, 1)), (12, (8, 2, 0))):
        for p in range(2, k):
            n = n_us(k, stage, p) // 7 ** (stage[0] - 3)
            picks = {tuple(sorted(u_rows(k, stage, p, c * 7 ** (stage[0] - 3)))) for c in range(n)}
            assert len(picks) == n
            assert all(min(x) == p and max(x) < k - stage[1] for x in picks)


def test_stages_have_work_and_pieces_tile_it():
    seen = set()
    for k in range(4, MAX_K + 1):
        for best in range(2, N - k + 2):
            level, p1 = 3, False
            while (nx := tw_next(k, best, 1, level, p1)) is not None:
                stage, level, p1 = nx
                if (k, stage) in seen:
                    continue
                seen.add((k, stage))
                assert sum(n_us(k, stage, p) for p in range(k)) > 0
                assert max(p for p in range(k) if n_us(k, stage, p)) <= k - 2  # pairs laid out
    for groups in range(1, 27):
        for cut in range(4):
            per = (groups + (1 << cut) - 1) >> cut
            got = [g for q in range(1 << cut) for g in range(q * per, min(groups, (q + 1) * per))]
            assert got == list(range(groups))


def griesmer(k):
    return max(d for d in range(1, N + 1) if sum(cdiv(d, 8 ** i) for i in range(k)) <= N)


@pytest.mark.parametrize("k", range(2, MAX_K + 1))
def test_stages_end(k):
    """From any best weight a code can have, falling or not, the stages end
    by level 11, within 16 of them."""
    rng = random.Random(k)
    for start in range(1, griesmer(k) + 8):
        for _ in range(20):
            level, p1, n = 3, False, 0
            best = start
            while (nx := tw_next(k, best, 1, level, p1)) is not None:
                stage, level, p1 = nx
                n += 1
                # the true distance is at most the Griesmer bound, and a code
                # that reaches a level has met every lighter message
                if stage[0] >= 5:
                    best = min(best, griesmer(k))
                if rng.random() < 0.5:
                    best = max(1, best - rng.randint(0, 3))
                assert stage[0] <= 11 and n <= 16


def codewords(rows):
    """All GF(8) combinations of bit-plane rows, as (message, weight)."""
    k = len(rows)
    mult = []
    for r in rows:
        m = [(0, 0, 0)]
        x = r
        for _ in range(7):
            m.append(x)
            x = (x[2], x[0] ^ x[2], x[1])
        mult.append(m)
    for msg in itertools.product(range(8), repeat=k):
        p = [0, 0, 0]
        for i, c in enumerate(msg):
            for q in range(3):
                p[q] ^= mult[i][c][q]
        yield msg, bin(p[0] | p[1] | p[2]).count("1")


def systematic(M, S):
    """Planes of the generator of S reduced as toric_prep_kernel reduces it
    (row r takes its own first nonzero column)."""
    inv = [0] + [next(x for x in range(1, 8) if gf8_mul(a, x) == 1) for a in range(1, 8)]
    G = [[int(x) for x in M[i]] for i in S]
    for r in range(len(G)):
        col = next(j for j in range(N) if G[r][j])
        f = inv[G[r][col]]
        G[r] = [gf8_mul(f, x) for x in G[r]]
        for q in range(len(G)):
            if q != r and G[q][col]:
                c = G[q][col]
                G[q] = [x ^ gf8_mul(c, y) for x, y in zip(G[q], G[r])]
    return [tuple(sum(((x >> b) & 1) << j for j, x in enumerate(g)) for b in range(3)) for g in G]


@pytest.mark.parametrize("seed", range(6))
def test_part_bounds_on_whole_codes(seed):
    """Every codeword whose translates all escape a stage weighs at least the
    stage's bound.  The code is invariant under the torus, so the light
    messages of E stand for those of every translate: it is enough that the
    lightest codeword of the whole code that is heavier than everything met
    on E respects the bound."""
    rng = random.Random(seed)
    k = rng.choice([4, 5])
    S = sorted(rng.sample(range(N), k))
    words = list(codewords(systematic(build_eval_matrix(), S)))[1:]
    d = min(wt for _, wt in words)

    def met(pred):
        return min((wt for m, wt in words if pred([i for i, c in enumerate(m) if c])), default=N + 1)

    for w in range(1, k + 1):
        for r in range(0, min(3, k - w) + 1):
            best = met(lambda s: len(s) < w or len(s) == w and not any(i >= k - r for i in s))
            assert d >= min(best, cdiv(N * (w + 1), k + r))
        best = met(lambda s: len(s) < w or len(s) == w and k - 1 in s)
        assert d >= min(best, cdiv(N * w, k - 1))


@pytest.mark.parametrize("columns", [30, 32, 36, 42])
def test_counter_reaches_its_top(columns):
    """tw_count on one-bit rows (an int of many lanes), every bias."""
    rng = random.Random(columns)
    lanes = 512
    full = (1 << lanes) - 1
    levels = 5 if columns <= 32 else 6
    density = [rng.random() for _ in range(lanes)]
    rows = [sum((rng.random() < density[i]) << i for i in range(lanes)) for _ in range(columns)]
    count = [sum(r >> i & 1 for r in rows) for i in range(lanes)]

    def add(n, level, a, b):
        s = n[level]
        n[level] = s ^ a ^ b
        return s & a | s & b | a & b

    for bias in range((1 << levels) - columns, 1 << levels):
        if bias < 0:
            continue
        n = [full if bias >> i & 1 else 0 for i in range(levels)]
        wait = [0] * (levels + 1)
        for i in range(columns // 2):
            carry = add(n, 0, rows[2 * i], rows[2 * i + 1])
            for l in range(1, levels + 1):
                if l == levels or not i >> (l - 1) & 1:
                    wait[l] = carry
                    break
                carry = add(n, l, wait[l], carry)
        carry, have = 0, False
        for l in range(1, levels):
            waits = columns // 2 >> (l - 1) & 1
            if waits or have:
                carry = add(n, l, wait[l] if waits else 0, carry if have else 0)
                have = True
        over = (wait[levels] if columns // 2 >> (levels - 1) else 0) | carry
        for i in range(lanes):
            assert over >> i & 1 == (count[i] + bias >= 1 << levels)
