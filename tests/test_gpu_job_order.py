"""Batches of more rays than the chip holds take their rays from the job whose
rays are expected to live longest first. The results stay each job's own, in the
batch's order: rooms of falling and rising absorption, boxes and meshes, other
histogram lengths; and a call of the same layout with other walls, whose order
differs from the one the plan was made for.

Tolerance: segment counts equal, bins within 1e-5 relative (test_gpu_parity.py).
"""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig
from omg_audio_gb300 import workloads as W
from omg_audio_gb300.materials import Material

from test_gpu_parity import GOLDEN, gpu_scene, rel_bins

pytestmark = pytest.mark.gpu


def _jobs(scene, case, alphas, n):
    _, size, _, src, lis, _ = GOLDEN[0]
    jobs = [Job(src, lis, n + 64 * i, seed=50 + i, box_size=size, box_walls=[Material((a,) * 3, 0.1, (0.0,) * 3)] * 6,
                n_bins=100 + 50 * i, max_time=1.0 + 0.5 * i) for i, a in enumerate(alphas)]
    jobs.insert(1, Job(case.src, case.lis, n, seed=70, scene=scene, n_bins=200))
    return jobs


@pytest.mark.parametrize("n", [1000, 40000])
def test_every_job_keeps_its_results(n):
    with Context(TraceConfig()) as ctx, Context(TraceConfig()) as alone:
        case = W.shoebox12(seed=4)
        scene, own = gpu_scene(ctx, case.recorder), gpu_scene(alone, case.recorder)
        for alphas in ((0.6, 0.3, 0.1, 0.02), (0.05, 0.1, 0.4, 0.8), (0.05, 0.1, 0.4, 0.8)):
            got = ctx.trace_batch(_jobs(scene, case, alphas, n))
            for j, (e, rv) in zip(_jobs(own, case, alphas, n), got):
                (es, rs), = alone.trace_batch([j])
                assert rv.segments == rs.segments
                assert e.bins.shape == es.bins.shape
                assert rel_bins(e.bins, es.bins) <= 1e-5
                assert np.allclose(rv.rt60, rs.rt60, rtol=1e-4, atol=1e-5, equal_nan=True)
        # a batch on the device: the same, launch after launch
        b = ctx.batch(_jobs(scene, case, (0.6, 0.3, 0.1, 0.02), n))
        first = None
        for _ in range(2):
            b.launch()
            segs = [rv.segments for _, rv in b.read()]
            assert b.segments() == sum(segs)
            assert first is None or first == segs
            first = segs
        b.destroy()
        scene.release()
        own.release()
