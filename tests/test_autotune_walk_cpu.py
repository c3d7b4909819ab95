"""The information-set knobs are timed on, and chosen for, the walk that reads them (host logic; the
toric walk has a fixed shape and reads none)."""

from __future__ import annotations

import numpy as np
import pytest

from generalized_toric_gpu_search_b200 import _lib, autotune, distance
from generalized_toric_gpu_search_b200.tables import build_eval_matrix

M = build_eval_matrix()


class FakeContext:
    """Says of a matrix what the library does."""

    made: list = []

    def __init__(self, device_id, matrix):
        self.device_id, self.matrix = device_id, np.asarray(matrix)
        self.is_toric = bool(np.array_equal(self.matrix, M))
        FakeContext.made.append(self)

    def close(self):
        pass


@pytest.fixture
def host(monkeypatch):
    FakeContext.made = []
    monkeypatch.setattr(distance, "ToricContext", FakeContext)
    monkeypatch.setattr(_lib, "device_info", lambda d: (148, 10, 0, "GPU"))
    monkeypatch.setattr(distance.torch.cuda, "Stream", lambda device=None: None)


def test_tuning_runs_the_general_walk(host, monkeypatch, tmp_path):
    monkeypatch.setattr(autotune, "measure",
                        lambda factory, sets, cfg: 1.0 / (1 + cfg.is_max_task_units))
    table = autotune.tune(0, ks=[6, 8], path=tmp_path / "t.json", walk="infoset")
    assert [c.is_toric for c in FakeContext.made] == [False]
    # codes of the same weights: the same columns in another order
    order = lambda A: sorted(map(tuple, np.asarray(A).T.tolist()))
    assert order(FakeContext.made[0].matrix) == order(M)
    assert autotune.choose(table, 8).is_max_task_units == 2401


def test_entries_timed_on_toric_batches_are_not_used(host, monkeypatch, tmp_path):
    path = tmp_path / "t.json"
    old = dict(is_blocks_per_sm=4, is_tasks_per_thread=16, is_max_task_units=343,
               infoset_seconds=1e-4, tail_rows=5)
    autotune.save_table("GPU", {k: dict(old) for k in autotune.INFOSET_KS}, path)
    got = autotune.choose(autotune.load_table("GPU", path), 9)
    assert got == distance.LaunchConfig(tail_rows=5)
    calls = []
    monkeypatch.setattr(autotune, "tune", lambda *a, **kw: calls.append(list(kw["ks"])) or {})
    autotune.ensure_table(0, path=path)
    assert calls == [list(autotune.INFOSET_KS)]
    # entries of one's own making, with no timing in them, are taken as they are
    assert autotune.choose({9: dict(is_tasks_per_thread=16)}, 9).is_tasks_per_thread == 16


@pytest.mark.parametrize("toric", [True, False])
def test_the_oracle_tunes_only_what_reads_the_knobs(host, monkeypatch, toric):
    calls = []
    table = {6: dict(is_blocks_per_sm=4), 14: dict(is_blocks_per_sm=5, is_tasks_per_thread=8)}
    monkeypatch.setattr(autotune, "ensure_table", lambda d: calls.append(d) or table)
    oracle = distance.DistanceOracleCUDABP(0, M if toric else np.roll(M, 1, axis=1))
    assert calls == ([] if toric else [0])
    one, other = oracle._runner_for(6, False), oracle._runner_for(14, False)
    assert (one is other) == toric  # one runner, one workspace
    assert one.config == distance.LaunchConfig(is_blocks_per_sm=0 if toric else 4)
    assert oracle._runner_for(14, True).config == distance.LaunchConfig()
