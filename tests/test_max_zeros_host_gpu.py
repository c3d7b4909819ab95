"""tg_max_zeros_host: what it refuses before anything runs, batches whose buffers an oracle does not
keep, and oracles called from several threads at once."""

from __future__ import annotations

import ctypes
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

from generalized_toric_gpu_search_b200 import DistanceOracleCUDABP, _lib, build_eval_matrix

pytestmark = pytest.mark.gpu

M = build_eval_matrix()


def test_refusals_and_a_call():
    oracle = DistanceOracleCUDABP(0, M)
    p = oracle.runner.params(2, 3, 1)
    h_idx = torch.tensor([0, 8, 16, 1, 9, 20], dtype=torch.int32).pin_memory()
    h_off = torch.tensor([0, 3, 6], dtype=torch.int64).pin_memory()
    h_out = torch.full((3,), -1, dtype=torch.int32).pin_memory()
    buf = torch.empty(3 * 256 + 8, dtype=torch.uint8, device="cuda")  # offsets, indices, values
    ws = oracle.runner.workspace(p)
    torch.cuda.synchronize()
    good = dict(ctx=oracle.ctx.handle, idx=h_idx.data_ptr(), n=6, off=h_off.data_ptr(),
                out=h_out.data_ptr(), buf=buf.data_ptr(), size=buf.numel(), ws=ws.data_ptr(),
                ws_size=ws.numel())

    def call(**kw):
        a = {**good, **kw}
        return _lib.load().tg_max_zeros_host(
            a["ctx"], ctypes.byref(p), a["idx"], a["n"], a["off"], None, a["out"], a["buf"],
            a["size"], a["ws"], a["ws_size"], oracle._stream.cuda_stream)

    invalid, workspace = _lib.TG_ERR_INVALID_ARGUMENT, _lib.TG_ERR_WORKSPACE
    for name in ("ctx", "idx", "off", "out", "buf", "ws"):
        assert call(**{name: None}) == invalid, name
    assert call(n=-1) == invalid
    assert call(buf=buf.data_ptr() + 8, size=buf.numel() - 8) == invalid
    assert call(ws=ws.data_ptr() + 8) == invalid
    assert call(size=2 * 256 + 7) == workspace
    assert call(ws_size=255) == workspace
    assert call() == _lib.TG_OK
    want = oracle.max_zeros_batch([[0, 8, 16], [1, 9, 20]], 1)
    assert h_out.tolist() == want + [_lib.TG_OK]


def test_buffers_above_the_kept_size():
    rng = random.Random(1)
    pool = [sorted(rng.sample(range(49), rng.randint(2, 4))) for _ in range(60)]
    oracle = DistanceOracleCUDABP(0, M)
    oracle.KEEP_BYTES = 1 << 15
    want = oracle.max_zeros_batch(pool, 1)
    n = oracle.KEEP_BYTES // 4 + 1000  # the results alone are larger
    big = [i % 60 for i in range(n)]
    for td in (1, np.ones(n, dtype=np.int32)):
        got = oracle.max_zeros_batch([pool[i] for i in big], td)
        assert got == [want[i] for i in big]
        assert oracle._buffer is None and oracle._h_out is None
        assert oracle.max_zeros_batch(pool, 1) == want
        assert oracle._buffer is not None and oracle._h_out is not None


def test_threads_with_oracles_of_their_own_and_a_shared_one():
    rng = random.Random(2)
    batches = [[sorted(rng.sample(range(49), rng.randint(4, hi))) for _ in range(n)]
               for n, hi in ((1, 14), (40, 13), (700, 11), (3, 16), (300, 14), (64, 8))]
    shared = DistanceOracleCUDABP(0, M)
    want = [shared.max_zeros_batch(b, 1) for b in batches]
    oracles = [shared, shared, DistanceOracleCUDABP(0, M), DistanceOracleCUDABP(0, M)]

    def work(i):
        order = random.Random(i).sample(range(len(batches)), len(batches)) * 5
        return all(oracles[i].max_zeros_batch(batches[b], 1) == want[b] for b in order)

    with ThreadPoolExecutor(4) as pool:
        assert all(pool.map(work, range(4)))
