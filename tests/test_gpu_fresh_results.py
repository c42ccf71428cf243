"""Results of many megabytes into arrays whose pages are not there yet (a new mapping, as
a large NumPy allocation is), into read pages and into arrays in use: the same bytes, and
what surrounds the arrays stays as it was. A call into new pages may take a few times as
long as one into pages in use, not tens of times.
"""
import ctypes as C
import mmap
import time

import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig, _lib
from omg_audio_gb300 import materials as M
from omg_audio_gb300.engine import jobs_to_c, panels_to_c
from omg_audio_gb300.surrogate import Mlp

pytestmark = pytest.mark.gpu

GUARD = 256   # floats before and after each array, in its first and last page


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _fresh(n, read=False):
    """n floats in a new anonymous mapping, off its page boundary (and all pages read, or none touched)."""
    m = np.frombuffer(mmap.mmap(-1, 4 * (n + 2 * GUARD)), np.float32)
    if read:
        m[::256].sum()
    return m, m[GUARD:GUARD + n]


def _check(call, sizes):
    """call(*arrays) into arrays in use, into new ones and into read ones."""
    warm = [np.full(n, 7.0, np.float32) for n in sizes]
    call(*warm)
    times = {"warm": [], "fresh": []}
    for k in range(5):
        t0 = time.perf_counter()
        call(*warm)
        t1 = time.perf_counter()
        pairs = [_fresh(n, read=k == 4) for n in sizes]
        t2 = time.perf_counter()
        call(*[v for _, v in pairs])
        t3 = time.perf_counter()
        times["warm"].append(t1 - t0)
        if k < 4:
            times["fresh"].append(t3 - t2)
        for (m, v), w in zip(pairs, warm):
            assert np.array_equal(v, w)
            assert not m[:GUARD].any() and not m[GUARD + len(v):].any()
    # 77 MB: 1.1 ms in use, 2.7 ms new (43 ms where the device brought the pages in)
    assert np.median(times["fresh"]) <= 12 * np.median(times["warm"]), times


@pytest.mark.parametrize("n", [3000, 100000])
def test_query_and_predict(n):
    with Context(TraceConfig(timeout_ms=60000)) as ctx:
        net = Mlp(ctx, 38, 64, 2, 192, 2)
        x = np.random.default_rng(1).normal(size=(n, 38)).astype(np.float32)
        spread = np.empty(n, np.float32)

        def query(mean):
            assert _lib.lib().omg_surrogate_query(ctx.h, net.id, _p(x), n, _p(mean), _p(spread), -30.0) == 0

        def predict(mean, std):
            assert _lib.lib().omg_surrogate_predict(ctx.h, net.id, _p(x), n, _p(mean), _p(std)) == 0

        _check(query, [n * 192])
        _check(predict, [n * 192, n * 192])


@pytest.mark.parametrize("n_jobs", [16, 1200])
def test_batch(n_jobs):
    walls = [M.CONCRETE] * 4 + [M.WOOD_PANEL, M.CONCRETE]
    with Context(TraceConfig(timeout_ms=60000, n_bins=2000, bin_dt=0.001, max_time=2.0)) as ctx:
        jobs = [Job((1.5, 1, 1.5), (4.5, 3, 1.6), 16, seed=i + 1, box_size=(6, 4, 3), box_walls=walls)
                for i in range(n_jobs)]
        arr, nbf, ndf = jobs_to_c(jobs, ctx.cfg)
        panels, rv = panels_to_c(()), (_lib.omg_reverb * n_jobs)()

        def trace(bins, dirs):
            assert _lib.lib().omg_trace_batch(ctx.h, arr, n_jobs, panels, 0, _p(bins), _p(dirs), rv) == 0

        _check(trace, [nbf, ndf])
