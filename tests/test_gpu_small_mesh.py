"""Few rays in meshes of few primitives (near-tie rule): up to 128 primitives are
all tested by the warp's lanes, 1 to 4 each, larger meshes are walked. Rooms on
either side of each step, with walls authored once or twice (coincident: the
lowest surface wins), against the oracle on the same streams; watertight
contexts against the walk a lane per ray.

Tolerance: segment counts equal, bins within the compensated sums' 1e-5.
"""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, MeshBuilder, TraceConfig, _lib
from omg_audio_gb300 import materials as M

from test_gpu_parity import oparams, rel_bins
from test_oracle_golden import omat

pytestmark = pytest.mark.gpu

SRC, LIS = (0.7, 0.8, 0.9), (1.4, 1.1, 1.2)


def _quads(k, twice, extra):
    """A 2 x 2.1 x 2.2 m room, its walls k x k quads each, `extra` quads more in mid-air."""
    size = (2.0, 2.1, 2.2)
    for _ in range(2 if twice else 1):
        for ax in range(3):
            a, b = [i for i in range(3) if i != ax]
            for v in (0.0, size[ax]):
                for i in range(k):
                    for j in range(k):
                        q = []
                        for u, w in ((i, j), (i + 1, j), (i + 1, j + 1), (i, j + 1)):
                            p = [0.0, 0.0, 0.0]
                            p[ax], p[a], p[b] = v, size[a] * u / k, size[b] * w / k
                            q.append(np.float32(p))
                        yield ax * 2 + (v > 0), q
    for e in range(extra):
        x, z = 0.05 + 0.01 * e, 0.1 + 0.02 * e
        yield 6, [np.float32(p) for p in ((x, 0.1, z), (x + 0.1, 0.1, z), (x + 0.1, 0.2, z), (x, 0.2, z))]


def _build(mb, mats, k, twice, extra):
    last = None
    for s, q in _quads(k, twice, extra):
        if s != last:
            mb.begin_surface()
            last = s
        mb.quad(*q, mats[s % len(mats)])


# (walls split, authored twice, quads more): 12, 32, 34, 64, 66, 96, 98, 128 and 130 triangles
ROOMS = [(1, False, 0), (1, False, 10), (1, False, 11), (1, True, 20), (1, True, 21), (2, True, 0), (2, True, 1),
         (2, True, 16), (2, True, 17)]
WALLS = (M.CONCRETE, M.DRYWALL, M.WOOD_PANEL, M.BRICK, M.CARPET, M.ACOUSTIC_TILE)


@pytest.mark.parametrize("room", ROOMS)
@pytest.mark.parametrize("bvh", [_lib.BVH_SAH, _lib.BVH_SAH3])
def test_few_rays_equal_the_oracle(oracle, room, bvh):
    O = oracle
    with Context(TraceConfig(tie_mode=1, max_bounces=40, timeout_ms=60000)) as ctx:
        mb, ob = MeshBuilder(), O.MeshBuilder()
        _build(mb, [mb.material(m) for m in WALLS], *room)
        _build(ob, [ob.material(omat(O, m)) for m in WALLS], *room)
        scene = ctx.upload_builder(mb, 3, bvh)
        mesh = ob.build("f32")
        for n in (1, 700):
            b, _, st = O.trace_mesh(mesh, SRC, LIS, n, P=oparams(O, ctx.cfg), seed=5, threads=8, acc64=True)
            e, rv = ctx.trace_world(scene, SRC, LIS, n, seed=5)
            assert rv.segments == st["segments"]
            assert rel_bins(e.bins, b) <= 1e-5
        scene.release()


@pytest.mark.parametrize("room", ROOMS[::3])
def test_watertight_equals_the_lane_walk(room):
    with Context(TraceConfig(tie_mode=1, tri_test=1, max_bounces=40, timeout_ms=60000)) as ctx:
        mb = MeshBuilder()
        _build(mb, [mb.material(m) for m in WALLS], *room)
        scene = ctx.upload_builder(mb)
        b = ctx.batch([Job(SRC, LIS, 900, seed=6, scene=scene)])
        b.set_shape(mode=0, epochs=0)
        b.launch()
        (e, rv), = b.read()
        b.set_shape(mode=0, epochs=1)
        b.launch()
        (el, rl), = b.read()
        assert rv.segments == rl.segments
        assert rel_bins(e.bins, el.bins) <= 1e-5
        b.destroy()
        scene.release()
