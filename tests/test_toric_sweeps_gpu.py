"""Levels 1 to 4 of the toric preparation: row counts around the change from counting all columns
to the first 32 of them first, and around the two limits of its level 4, where few codes leave the
longer ones to the walk and many do not."""

from __future__ import annotations

import random

import numpy as np
import pytest

from generalized_toric_gpu_search_b200 import DistanceOracleCUDABP, build_eval_matrix

pytestmark = pytest.mark.gpu

M = build_eval_matrix()
PERMUTED = M[:, np.random.default_rng(1).permutation(49)]  # same codes, the general walk


@pytest.mark.parametrize("n, lo, hi", [(5, 2, 5), (20, 9, 12), (600, 2, 11), (320, 12, 15)])
def test_matches_the_general_walk(n, lo, hi):
    rng = random.Random(10 * n + lo)
    sets = [rng.sample(range(49), rng.randint(lo, hi)) for _ in range(n)]
    want = DistanceOracleCUDABP(0, PERMUTED).max_zeros_batch(sets, 1)
    assert DistanceOracleCUDABP(0, M).max_zeros_batch(sets, 1) == want
