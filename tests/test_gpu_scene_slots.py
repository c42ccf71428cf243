"""A scene table slot given to another scene: the plan kept for calls of one
layout, and a batch recorded before, run on what the slot holds now. The new
scene's tree is built on the device and has no 4-wide form, so the calls' kernels
differ; before and after, the results are those of a context of its own.

Tolerance: segment counts equal, bins within 1e-5 relative (test_gpu_parity.py).
"""
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig, _lib
from omg_audio_gb300 import workloads as W

from test_gpu_parity import gpu_scene, rel_bins

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tie", [0, 1])
@pytest.mark.parametrize("kinds", [(_lib.BVH_SAH, _lib.BVH_LBVH), (_lib.BVH_LBVH, _lib.BVH_SAH)])
@pytest.mark.parametrize("n_rays", [700, 20000])
def test_calls_follow_the_scene_in_the_slot(tie, kinds, n_rays):
    a, b = W.shoebox12(seed=4), W.multiroom(seed=2)
    src, lis = b.pairs[0]
    with Context(TraceConfig(tie_mode=tie)) as ctx:
        first = gpu_scene(ctx, a.recorder, kinds[0])
        ctx.trace_world(first, a.src, a.lis, n_rays, seed=3)          # keeps a plan
        old = ctx.batch([Job(src, lis, n_rays, seed=3, scene=first)])
        old.launch()
        old.read()
        slot = first.id
        first.release()
        second = gpu_scene(ctx, b.recorder, kinds[1])
        assert second.id == slot
        e, rv = ctx.trace_world(second, src, lis, n_rays, seed=3)
        old.launch()
        (eb, rb), = old.read()
        with Context(TraceConfig(tie_mode=tie)) as fresh:
            sc = gpu_scene(fresh, b.recorder, kinds[1])
            ref, rr = fresh.trace_world(sc, src, lis, n_rays, seed=3)
            sc.release()
        assert rv.segments == rr.segments == rb.segments
        assert rel_bins(e.bins, ref.bins) <= 1e-5
        assert rel_bins(eb.bins, ref.bins) <= 1e-5
        old.destroy()
        second.release()
