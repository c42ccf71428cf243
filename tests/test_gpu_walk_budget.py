"""A lowered walk budget under the first-found rule: the persistent kernels, whose
walks go ahead of their leaves, accept and refuse what the wavefront rounds do, which
visit the nodes of the reference's walk alone. At the least budget that the rounds
accept, and one below, over warps of one to 32 rays, warp-local queues, panels and
trees of both kinds. The dome's escapes of one event accept and refuse what a ray
query along the same fan does."""
import numpy as np
import pytest

from omg_audio_gb300 import Context, DomeProbe, Job, TraceConfig, _lib
from omg_audio_gb300 import workloads as W

from test_gpu_parity import gpu_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bvh", [_lib.BVH_SAH, _lib.BVH_LBVH])
@pytest.mark.parametrize("rays", [10000, 60001])
def test_budget_of_the_reference_walk(bvh, rays):
    with Context(TraceConfig(tie_mode=0, max_bounces=24)) as ctx:
        case = W.multiroom(seed=6)
        scene = gpu_scene(ctx, case.recorder, bvh)
        src, lis = case.pairs[0][:2]
        b = ctx.batch([Job(src, lis, rays, seed=3, scene=scene, panel_offset=0, n_panels=len(case.panels))],
                      case.panels)

        def accepted(budget):
            ctx.set_limits(walk_budget=budget)
            b.launch()
            try:
                (e, rv), = b.read()
            except _lib.OmgError as err:
                assert err.status == _lib.E_OVERFLOW and ctx.last_flags() & 4
                return None
            return rv.segments, e.bins.tobytes()

        b.set_shape(mode=0, wf_rounds=24, wf_tail=0, epochs=0)
        lo, hi = 1, 4096
        while lo < hi:
            mid = (lo + hi) // 2
            if accepted(mid):
                hi = mid
            else:
                lo = mid + 1
        want = accepted(lo)
        assert want and not accepted(lo - 1)
        for shape in (dict(mode=0), dict(mode=1, walk_steps=8), dict(mode=0, epochs=4)):
            b.set_shape(**{**dict(mode=0, wf_rounds=0, epochs=0, walk_steps=0), **shape})
            assert accepted(lo) == want, shape
            assert accepted(lo - 1) is None, shape
        ctx.set_limits(0, 0)
        b.destroy()
        scene.release()


def test_dome_budget():
    """One event a ray: the walks are those of a ray query along the fan."""
    with Context(TraceConfig(tie_mode=0)) as ctx:
        case = W.multiroom(seed=6)
        scene = gpu_scene(ctx, case.recorder)
        n = 512
        probe = DomeProbe(ctx, scene, [], n)
        eyes = np.array([case.pairs[k][1] for k in range(40)], np.float32)
        i = np.arange(n)
        z = (1.0 - 2.0 * (i + np.float32(0.5)).astype(np.float32) / np.float32(n)).astype(np.float32)
        r = np.sqrt(np.maximum(np.float32(1.0) - z * z, np.float32(0.0)))
        ga = np.float32(np.pi) * (np.float32(3.0) - np.sqrt(np.float32(5.0)))
        phi = (ga * i.astype(np.float32)).astype(np.float64)
        fan = np.stack([r * np.cos(phi).astype(np.float32), r * np.sin(phi).astype(np.float32), z], 1)
        o, d = np.repeat(eyes, n, 0), np.tile(fan, (len(eyes), 1)).astype(np.float32)

        def accepted(fn, budget):
            ctx.set_limits(walk_budget=budget)
            try:
                return fn()
            except _lib.OmgError as err:
                assert err.status == _lib.E_OVERFLOW
                return None

        lo, hi = 1, 4096
        while lo < hi:
            mid = (lo + hi) // 2
            if accepted(lambda: ctx.raycast(scene, o, d), mid):
                hi = mid
            else:
                lo = mid + 1
        ctx.set_limits(0, 0)
        want = probe.sample(eyes, max_events=1)
        got = accepted(lambda: probe.sample(eyes, max_events=1), lo)
        assert got and all(np.array_equal(got[k], want[k]) for k in ("escape", "ray_tp", "raw"))
        assert accepted(lambda: probe.sample(eyes, max_events=1), lo - 1) is None
        ctx.set_limits(0, 0)
        scene.release()
