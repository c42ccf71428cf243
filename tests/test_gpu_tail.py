"""Launches whose last rays are handed to a second launch, a warp per ray: by
the number of rays (none, 28 or 56 a multiprocessor), the hit rule, the bands
and the geometries in one batch. Each job equals its own launch of few rays at
a time: the same rays (a job's streams are numbered from its ray base, so the
job is one launch here and part of a batch there), whichever kernel ends them.

Tolerance: segment counts equal; bins within 1e-5 relative, as for any job in a
batch against its single launch (test_gpu_parity.py).
"""
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig, _lib
from omg_audio_gb300 import workloads as W

from test_gpu_parity import GOLDEN, gpu_scene, rel_bins

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("tie", [0, 1])
@pytest.mark.parametrize("unit_rays", [2.9, 3.2, 9.5])
def test_jobs_equal_their_single_launches(tie, unit_rays):
    n = int(unit_rays * 28 * _sms()) // 4
    with Context(TraceConfig(tie_mode=tie)) as ctx:
        case = W.multiroom(seed=6)
        big = gpu_scene(ctx, case.recorder)
        box12 = W.shoebox12(seed=4)
        small = gpu_scene(ctx, box12.recorder)
        _, size, walls, bsrc, blis, _ = GOLDEN[0]
        k = len(case.panels)
        jobs = [Job(case.pairs[0][0], case.pairs[0][1], n, seed=31, scene=big, panel_offset=0, n_panels=k),
                Job(box12.src, box12.lis, n, seed=32, scene=small),
                Job(case.pairs[7][0], case.pairs[7][1], n, seed=33, scene=big, panel_offset=0, n_panels=k),
                Job(bsrc, blis, n, seed=34, box_size=size, box_walls=walls)]
        b = ctx.batch(jobs, case.panels)
        assert b.kernel_count() == (3 if unit_rays < 3 else 4)
        for _ in range(2):                    # the second launch reuses the recorded graph
            b.launch()
            got = b.read()
            for j, (e, rv) in zip(jobs, got):
                one = ctx.batch([j], case.panels)
                # no second launch: the single job walks with another kernel shape throughout
                one.set_shape(mode=0, epochs=1)
                one.launch()
                (es, rs), = one.read()
                assert rv.segments == rs.segments
                assert rel_bins(e.bins, es.bins) <= 1e-5
                one.destroy()
        b.destroy()
        big.release()
        small.release()


@pytest.mark.parametrize("bvh", [_lib.BVH_SAH, _lib.BVH_SAH3])
def test_eight_bands_and_one_ray_over(bvh):
    """8 bands (the saved energies fill both words), at the first size with a tail."""
    n = 3 * 28 * _sms()
    with Context(TraceConfig(tie_mode=1)) as ctx:
        case = W.city(seed=3, nx=3, ny=2, n_sources=1, n_dome=1)
        scene = gpu_scene(ctx, case.recorder, bvh, 8)
        src, lis = (tuple(map(float, p[0])) for p in (case.sources, case.listeners))
        segs = []
        for m, count in ((n - 1, 3), (n, 4)):
            b = ctx.batch([Job(src, lis, m, seed=41, scene=scene, n_bands=8)])
            b.set_shape(mode=0, epochs=0)     # (a shape set on a batch is the context's next default)
            assert b.kernel_count() == count
            b.launch()
            (e, rv), = b.read()
            b.set_shape(mode=0, epochs=1)
            b.launch()
            (es, rs), = b.read()
            assert rv.segments == rs.segments
            assert rel_bins(e.bins, es.bins) <= 1e-5
            segs.append(rv.segments)
            b.destroy()
        assert segs[1] > segs[0] > 0
        scene.release()
