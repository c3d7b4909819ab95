"""Sampled screening with thresholds where a set's work is spread over many CTAs and most sets fail
early: CTAs of a set start, look at its fail flag and raise it at the same time.  A set that fails
reports the zeros of one of its sampled codewords, so never more than the full sampled maximum."""

from __future__ import annotations

import random

import numpy as np
import pytest

from generalized_toric_gpu_search_b200 import DistanceOracleCUDABP, build_eval_matrix
from oracle import oracle as cpu

pytestmark = pytest.mark.gpu

M = build_eval_matrix()
COUNT = 20_000  # 157 rounds of 128 work ids


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("lo, hi", [(6, 20), (22, 40), (45, 49)])
def test_failing_sets_report_a_sampled_codeword(lo, hi, seed):
    rng = random.Random(100 * lo + seed)
    sets = [sorted(rng.sample(range(49), rng.randint(lo, hi))) for _ in range(40)]
    full = cpu.max_zeros_batch(M, sets, 1, sample_count=COUNT, sample_seed=seed)
    oracle = DistanceOracleCUDABP(0, M)
    for shift in (0, 1, 2, 5, 12):  # over the sampled distance: 0 passes, 12 fails at once
        td = np.array([49 - z + shift - (i % 4 == 3) for i, z in enumerate(full)], dtype=np.int32)
        for _ in range(5):
            got = oracle.max_zeros_batch(sets, td, sample_count=COUNT, sample_seed=seed)
            for z, g, t in zip(full, got, td):
                if 49 - z >= t:
                    assert g == z
                else:
                    assert 49 - t < g <= z
