"""A lowered walk budget counts the lanes' visits whatever the number of rays: few rays,
which a warp each would walk, accept what the same rays among many do, and under the
first-found rule refuse what the wavefront rounds do, which visit the nodes of the
reference's walk alone. (A near-tie walk goes on while other lanes of its warp look for
their leaves, so rays with fewer in their warp may do with less.) Early reflections count the walks of every pair, also of those that the
pair's geometry ends after them."""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig, _lib
from omg_audio_gb300 import workloads as W
from omg_audio_gb300.early import WorldEarly

from test_gpu_parity import gpu_scene

pytestmark = pytest.mark.gpu


def _least(accepted):
    lo, hi = 1, 4096
    while lo < hi:
        mid = (lo + hi) // 2
        if accepted(mid):
            hi = mid
        else:
            lo = mid + 1
    return lo


@pytest.mark.parametrize("tie", [0, 1])
@pytest.mark.parametrize("mesh", ["rooms", "box"])
@pytest.mark.parametrize("rays", [64, 5000])
def test_trace_of_few_rays(tie, mesh, rays):
    with Context(TraceConfig(tie_mode=tie, max_bounces=24)) as ctx:
        if mesh == "rooms":
            case = W.multiroom(seed=6)
            src, lis = case.pairs[0][:2]
        else:
            case = W.shoebox12(seed=1)
            src, lis = case.src, case.lis
        scene = gpu_scene(ctx, case.recorder)
        few = ctx.batch([Job(src, lis, rays, seed=3, scene=scene)])
        # the same streams and no others: jobs of one seed
        many = ctx.batch([Job(src, lis, rays, seed=3, scene=scene)] * (1 + 60000 // rays))
        if tie == 0:
            many.set_shape(mode=0, wf_rounds=24, wf_tail=0, epochs=0)
            few.set_shape(mode=0, wf_rounds=0, epochs=0)

        def accepted(b, budget):
            ctx.set_limits(walk_budget=budget)
            b.launch()
            try:
                e, rv = b.read()[0]
            except _lib.OmgError as err:
                assert err.status == _lib.E_OVERFLOW and ctx.last_flags() & 4
                return None
            return rv.segments, e.bins.tobytes()

        lo = _least(lambda m: accepted(many, m))
        want = accepted(many, lo)
        assert want and accepted(few, lo) == want
        assert lo == 1 or tie == 1 or accepted(few, lo - 1) is None
        assert lo <= 2 or accepted(few, lo // 2) is None
        ctx.set_limits(0, 0)
        assert accepted(few, 0) == want
        few.destroy()
        many.destroy()
        scene.release()


def test_early_pairs_count_their_walks():
    with Context(TraceConfig()) as ctx:
        case = W.multiroom(seed=6)
        scene = gpu_scene(ctx, case.recorder)
        early, lis = WorldEarly(ctx, scene), case.pairs[0][1]
        chains = [c for c in early.discover(lis, 768, 1) if c[1] == 1]
        # sources far behind every surface that the chains name: no path, after a walk each
        sources = [(k, (lis[0] + d[0], lis[1] + d[1], lis[2] + d[2]))
                   for k, d in enumerate(np.vstack([np.eye(3), -np.eye(3)]) * 55.0)]
        want = early.solve(sources, chains, lis)

        def accepted(budget):
            ctx.set_limits(walk_budget=budget)
            try:
                return early.solve(sources, chains, lis)
            except _lib.OmgError as err:
                assert err.status == _lib.E_OVERFLOW
                return None

        lo = _least(lambda m: accepted(m) is not None)
        assert np.array_equal(accepted(lo), want)
        # the reference's walk to the first chain's surface alone visits more than this
        assert lo > 8 and accepted(8) is None
        ctx.set_limits(0, 0)
        early.close()
        scene.release()


def test_early_pair_that_geometry_ends():
    """A source below the floor that its chain names: the walk to the floor comes first."""
    with Context(TraceConfig()) as ctx:
        case = W.shoebox12(seed=1)
        scene = gpu_scene(ctx, case.recorder)
        early, lis = WorldEarly(ctx, scene), (4.0, 3.0, 2.0)
        chains = [c for c in early.discover(lis, 768, 1) if c[1] == 1]
        up = early.solve([(1, (4.5, 3.2, 1.5))], chains, lis)[0]
        floor = [c for c, r in zip(chains, up) if r["valid"] and r["dir"][2] < -0.5]
        assert len(floor) == 1
        below = [(1, (4.5, 3.2, -1.5))]
        assert not early.solve(below, floor, lis)["valid"].any()
        ctx.set_limits(walk_budget=1)
        with pytest.raises(_lib.OmgError) as err:
            early.solve(below, floor, lis)
        assert err.value.status == _lib.E_OVERFLOW
        ctx.set_limits(0, 0)
        assert not early.solve(below, floor, lis)["valid"].any()
        early.close()
        scene.release()
