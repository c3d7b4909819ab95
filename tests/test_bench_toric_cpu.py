"""bench.py's claims about a toric batch: its launches and its roofline follow the two kernels that
run (csrc/abi.cu: bind_distance; csrc/distance.cu: run_prepare, run_walk)."""

from __future__ import annotations

import pytest

import bench


@pytest.mark.parametrize("k_max, enumeration, launches", [
    (14, "auto", 2), (2, "auto", 2), (21, "infoset", 2),  # toric_prep_kernel, toric_walk_kernel
    (1, "auto", 3), (14, "orbit", 3), (14, "projective", 3)])
def test_launches_of_a_toric_batch(k_max, enumeration, launches):
    assert bench.step_launches(k_max, enumeration) == launches
    assert bench.takes_toric_walk(k_max, enumeration) == (launches == 2)


def test_roofline_counts_the_kernels_own_codewords():
    paths = {"infoset_codewords": 9_000, "enumeration_codewords": 500}
    pipes = {"lop3_per_clk_sm": 64.0, "popc_per_clk_sm": 16.0}
    walk = bench.roofline(True, 1e-6, 0.0, 3e-6, 2_000, paths, pipes, 10, 1000.0)
    assert walk["kernel"] == "toric_walk_kernel" and walk["codewords"] == 7_000
    assert walk["codewords_per_clk_sm"] == pytest.approx(7_000 / (3e-6 * 10 * 1e9))
    # the ALU's 64 LOP3 and 54 of them per 32 codewords
    assert walk["frac"] == pytest.approx(walk["codewords_per_clk_sm"] * 54 / 32 / 64)
    assert walk["kernel_share"] == pytest.approx(0.75)
    prep = bench.roofline(True, 4e-6, 0.0, 3e-6, 2_000, paths, pipes, 10, 1000.0)
    assert prep["kernel"] == "toric_prep_kernel" and prep["codewords"] == 2_000
    assert prep["frac"] == pytest.approx(2_000 * 8 / 7 / (4e-6 * 10 * 1e9 * 16))
    enum = bench.roofline(False, 1e-6, 2e-6, 0.0, 0, paths, pipes, 10, 1000.0)
    assert enum["kernel"] == "walk_hist_kernel" and enum["codewords"] == 500
