"""The toric walk (csrc/toric_walk.cuh) against the other enumerations.

The general walk runs on the same code with its columns permuted (not a toric
matrix as it stands, every weight the same); k <= 8 also against the CPU
oracle."""

import random

import numpy as np
import pytest

from generalized_toric_gpu_search_b200 import DistanceOracleCUDABP, build_eval_matrix

pytestmark = pytest.mark.gpu

M = build_eval_matrix()
PERMUTED = M[:, np.random.default_rng(5).permutation(49)]


def _sets(rng, n, lo, hi):
    return [rng.sample(range(49), rng.randint(lo, hi)) for _ in range(n)]


@pytest.mark.parametrize("n, lo, hi", [
    (1, 4, 4), (1, 5, 5), (3, 7, 7),       # a level with few supports
    (1, 12, 12), (2, 13, 13), (1, 14, 14),  # either layout, a lone code on all CTAs
    (40, 2, 8), (300, 4, 13),              # more codes than CTAs
    (9, 15, 16), (4, 17, 19), (1, 21, 21)])  # one to three blocks of pairs
def test_matches_the_general_walk(n, lo, hi):
    rng = random.Random(1000 * n + lo)
    sets = _sets(rng, n, lo, hi)
    got = DistanceOracleCUDABP(0, M).max_zeros_batch(sets, 1)
    assert got == DistanceOracleCUDABP(0, PERMUTED).max_zeros_batch(sets, 1)
    if hi <= 8:
        from oracle import oracle as cpu

        assert got == cpu.max_zeros_batch(M, sets, 1)


@pytest.mark.parametrize("lo, hi", [(4, 9), (10, 13), (14, 16)])
def test_targets(lo, hi):
    """A set below its target may stop early, at a witness; the others are
    exact."""
    rng = random.Random(lo)
    sets = _sets(rng, 60, lo, hi)
    exact = DistanceOracleCUDABP(0, M).max_zeros_batch(sets, 1)
    for shift in (-1, 0, 1, 3):
        td = [max(1, 49 - z + shift) for z in exact]
        got = DistanceOracleCUDABP(0, M).max_zeros_batch(sets, np.array(td, dtype=np.int32))
        for z, g, t in zip(exact, got, td):
            assert g == z if 49 - z >= t else 49 - t < g <= z


def test_degenerate_rows_among_others():
    """Repeated rows, single rows and empty sets beside codes that walk."""
    rng = random.Random(3)
    sets = _sets(rng, 30, 8, 14)
    for i, s in enumerate(sets[:12]):
        sets[i] = [[], s[:1], s[:2], s + s[:1]][i % 4]
    got = DistanceOracleCUDABP(0, M).max_zeros_batch(sets, 1)
    assert got == DistanceOracleCUDABP(0, PERMUTED).max_zeros_batch(sets, 1)
