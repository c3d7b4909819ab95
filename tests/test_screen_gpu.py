"""Sampled screening at the edges of its kernel: row counts around the five-row chunks of its
tables and the change of hashing at k = 21, sample counts around a CTA's pass, from one set on few
SMs to many CTAs per set."""

from __future__ import annotations

import random

import numpy as np
import pytest

from generalized_toric_gpu_search_b200 import DistanceOracleCUDABP, build_eval_matrix
from oracle import oracle as cpu

pytestmark = pytest.mark.gpu

M = build_eval_matrix()


@pytest.mark.parametrize("count", [1, 31, 127, 128, 129, 2500])
def test_every_row_count(count):
    rng = random.Random(count)
    # sets of one size per call to the oracle; one mixed batch on the device
    sets = [sorted(rng.sample(range(49), k)) for k in range(1, 50)]
    got = DistanceOracleCUDABP(0, M).max_zeros_batch(sets, 1, sample_count=count, sample_seed=77)
    for i, s in enumerate(sets):
        # the oracle's set id is the position in its batch
        want = cpu.max_zeros_batch(M, [s] * (i + 1), 1, sample_count=count, sample_seed=77)
        assert got[i] == want[i], (len(s), count)


@pytest.mark.parametrize("n, k, count", [(1, 9, 100_000), (3, 25, 70_000), (700, 22, 1500)])
def test_pieces(n, k, count):
    rng = random.Random(n)
    sets = [sorted(rng.sample(range(49), k)) for _ in range(n)]
    got = DistanceOracleCUDABP(0, M).max_zeros_batch(sets, 1, sample_count=count, sample_seed=3)
    assert got == cpu.max_zeros_batch(M, sets, 1, sample_count=count, sample_seed=3)


def test_other_matrix_and_repeated_rows():
    rng = random.Random(8)
    other = np.array([[rng.randrange(8) for _ in range(49)] for _ in range(49)], dtype=M.dtype)
    for k in (4, 21, 23):
        sets = [[rng.randrange(49) for _ in range(k)] for _ in range(20)]
        got = DistanceOracleCUDABP(0, other).max_zeros_batch(sets, 1, sample_count=900)
        assert got == cpu.max_zeros_batch(other, sets, 1, sample_count=900)
