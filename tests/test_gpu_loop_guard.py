"""A lowered loop guard under the first-found rule: every launch shape counts two
iterations a segment of the longest path, a walk and a shading pass, and one more that
finds the queue empty. Twice the bounces and one is therefore enough, however many rounds
a walk takes and however many rays share a warp; half of it is not. Launches of a warp per
ray, of one and of several rays a warp, and of lanes with a tail."""
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig, _lib
from omg_audio_gb300 import workloads as W

from test_gpu_parity import gpu_scene

pytestmark = pytest.mark.gpu

BOUNCES = 20


@pytest.mark.parametrize("rays", [512, 8000, 20000])
def test_guard_counts_segments(rays):
    with Context(TraceConfig(tie_mode=0, max_bounces=BOUNCES)) as ctx:
        case = W.multiroom(seed=6)
        scene = gpu_scene(ctx, case.recorder, _lib.BVH_SAH)
        src, lis = case.pairs[0][:2]
        b = ctx.batch([Job(src, lis, rays, seed=3, scene=scene, panel_offset=0, n_panels=len(case.panels))],
                      case.panels)

        def run(guard):
            ctx.set_limits(loop_guard=guard)
            b.launch()
            (e, rv), = b.read()
            return rv.segments, e.bins.tobytes()

        want = run(0)
        assert run(2 * BOUNCES + 1) == want
        with pytest.raises(_lib.OmgError) as err:
            run(BOUNCES)
        assert err.value.status == _lib.E_OVERFLOW and ctx.last_flags() & 8
        assert run(0) == want
        b.destroy()
        scene.release()


@pytest.mark.parametrize("rays", [512, 20000])
def test_guard_of_queued_walks(rays):
    """Mode 1 with a whole walk an iteration: a walk and a shading pass a segment, and a few
    iterations in which the queues run dry."""
    with Context(TraceConfig(tie_mode=0, max_bounces=BOUNCES)) as ctx:
        case = W.multiroom(seed=6)
        scene = gpu_scene(ctx, case.recorder, _lib.BVH_SAH)
        src, lis = case.pairs[0][:2]
        b = ctx.batch([Job(src, lis, rays, seed=3, scene=scene)])
        b.set_shape(mode=1, walk_steps=0, wf_rounds=0, epochs=0)
        got = []
        for guard in (0, 2 * BOUNCES + 8):
            ctx.set_limits(loop_guard=guard)
            b.launch()
            (e, rv), = b.read()
            got.append((rv.segments, e.bins.tobytes()))
        assert got[0] == got[1]
        b.destroy()
        scene.release()
