"""Buffers that could not be grown are grown again by the next call: an early solve
whose records would take tens of terabytes is refused for want of memory (nothing is
launched), and the calls after it equal those before it."""
import ctypes as C

import numpy as np
import pytest

from omg_audio_gb300 import Context, TraceConfig, _lib
from omg_audio_gb300 import workloads as W
from omg_audio_gb300.early import WorldEarly

from test_gpu_parity import gpu_scene

pytestmark = pytest.mark.gpu


def test_early_after_a_solve_too_large():
    with Context(TraceConfig()) as ctx:
        case = W.multiroom(seed=6, nx=2, ny=2)
        early = WorldEarly(ctx, gpu_scene(ctx, case.recorder), [])
        src, lis = case.pairs[0][:2]
        chains = early.discover(lis, 256)
        want = early.solve([(0, src)], chains, lis).copy()
        n = 1 << 20
        ids, pos = np.zeros(n, np.uint16), np.zeros((n, 3), np.float32)
        many, rec = np.zeros((n, 4), np.uint16), np.zeros(1, np.dtype(_lib.omg_mesh_record))

        def p(a):
            return a.ctypes.data_as(C.c_void_p)

        rc = _lib.lib().omg_early_solve(ctx.h, early.id, p(ids), p(pos), n, p(many), n, p(np.asarray(lis, np.float32)),
                                        p(np.zeros(9, np.float32)), 0, p(rec))
        assert rc == _lib.E_OOM
        assert early.discover(lis, 256) == chains
        got = early.solve([(0, src)], chains, lis)
        assert all(np.array_equal(got[f], want[f]) for f in want.dtype.names)
