"""Panel overlays and the job thresholds: traces against the f32 oracle, which
tests panel after panel with the reference's divisions and compares quotients
and square roots. Group sizes 1 to 5, many groups, panels that touch, overlap,
repeat (the exact-tie rule) or enclose the listener, in a shoebox (every job a
box: the shoebox kernel; mixed with a mesh: the general one) and on a mesh.
Segment counts equal, bins within the compensated sums' 1e-5."""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, Material, MeshBuilder, TraceConfig
from omg_audio_gb300 import materials as M
from omg_audio_gb300 import workloads as W

from test_gpu_parity import oparams, rel_bins
from test_oracle_golden import omat

pytestmark = pytest.mark.gpu

SIZE, SRC, LIS = (7.0, 5.0, 3.0), (1.5, 1.2, 1.5), (5.0, 3.5, 1.4)
WALLS = [M.CONCRETE, M.DRYWALL, M.WOOD_PANEL, M.BRICK, M.CARPET, M.ACOUSTIC_TILE]


def _panels(n, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k in range(n):
        c = rng.uniform([0.3, 0.3, 0.2], [6.7, 4.7, 2.8])
        half = rng.uniform(0.02, 0.8, 3)
        half[int(rng.integers(3))] = 0.02                      # a pane
        m = Material(tuple(rng.uniform(0.05, 0.6, 3)), float(rng.uniform(0, 0.5)), tuple(rng.uniform(0, 0.6, 3)))
        out.append((tuple(map(float, c - half)), tuple(map(float, c + half)), m))
        if k % 7 == 3:
            out.append((out[-1][0], out[-1][1], M.GRASS))      # the same box again: the first one counts
    out = out[:n]
    if n > 4:
        out[4] = ((4.0, 2.5, 0.5), (6.0, 4.5, 2.4), Material((0.1,) * 3, 0.0, (0.5,) * 3))   # around the listener
    return out


def _oracle(O, cfg, panels, mesh=None, seed=3, rays=3000):
    pan = [(mn, mx, omat(O, m)) for mn, mx, m in panels]
    P = oparams(O, cfg)
    if mesh is None:
        return O.trace_box(SIZE, [omat(O, m) for m in WALLS], SRC, LIS, rays, seed=seed, P=P, panels=pan, acc64=True)
    return O.trace_mesh(mesh, SRC, LIS, rays, seed=seed, P=P, panels=pan, acc64=True, threads=8)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 33, 140])
@pytest.mark.parametrize("tie", [0, 1], ids=["first-found", "near-tie"])
def test_panels_equal_the_oracle(oracle, tie, n):
    O = oracle
    pan = _panels(n, 100 + n)
    with Context(TraceConfig(tie_mode=tie, max_bounces=40, timeout_ms=60000)) as ctx:
        rec = W.Recorder()
        ids = [rec.material(m) for m in WALLS]
        W._abox(rec, (0.0, 0.0, 0.0), SIZE, ids[0])
        mb = MeshBuilder()
        rec.replay(mb)
        scene = ctx.upload_builder(mb)
        ob = O.MeshBuilder()
        rec.replay(ob, lambda m: omat(O, m))
        mesh = ob.build("f32")
        box = dict(box_size=SIZE, box_walls=WALLS)
        both = ctx.trace_batch([Job(SRC, LIS, 3000, seed=3, panel_offset=0, n_panels=n, **box),
                                Job(SRC, LIS, 3000, seed=3, panel_offset=0, n_panels=n, scene=scene)], pan)
        alone = ctx.trace_batch([Job(SRC, LIS, 3000, seed=3, panel_offset=0, n_panels=n, **box)], pan)
        b, _, st = _oracle(O, ctx.cfg, pan)
        bm, _, sm = _oracle(O, ctx.cfg, pan, mesh)
        for (e, rv), (rb, rs) in ((both[0], (b, st)), (alone[0], (b, st)), (both[1], (bm, sm))):
            assert rv.segments == rs["segments"]
            assert rel_bins(e.bins, rb) <= 1e-5


@pytest.mark.parametrize("radius,max_time,c", [(0.5, 3.0, 343.0), (0.1234567, 0.0317, 331.3), (3.3e-3, 0.5, 1.0),
                                               (1e30, 1e30, 343.0), (0.25, 1e-9, 343.0)])
def test_receiver_and_time_limits_equal_the_oracle(oracle, radius, max_time, c):
    O = oracle
    with Context(TraceConfig(receiver_radius=radius, max_time=max_time, speed_of_sound=c, max_bounces=40)) as ctx:
        e, rv = ctx.trace_box(SIZE, WALLS, SRC, LIS, 4000, seed=11)
        b, _, st = O.trace_box(SIZE, [omat(O, m) for m in WALLS], SRC, LIS, 4000, seed=11, P=oparams(O, ctx.cfg),
                               acc64=True)
        assert rv.segments == st["segments"]
        assert rel_bins(e.bins, b) <= 1e-5


def test_thresholds_are_the_comparisons_they_replace():
    """DJob's bisection restated: for radii and limits at random the found f32
    is where the rounded comparison changes, checked at it and its neighbours."""
    f = np.float32
    rng = np.random.default_rng(1)
    for _ in range(200):
        r, t, c = f(10.0 ** rng.uniform(-6, 6)), f(10.0 ** rng.uniform(-6, 4)), f(10.0 ** rng.uniform(-2, 4))

        def least(pred):
            lo, hi = 0, 0x7F800000
            while lo < hi:
                mid = (lo + hi) // 2
                if pred(np.array(mid, np.uint32).view(f)[()]):
                    hi = mid
                else:
                    lo = mid + 1
            return np.array(lo, np.uint32).view(f)[()]

        with np.errstate(over="ignore"):
            s = least(lambda v: not (np.sqrt(v) < r))
            for v in (np.nextafter(s, f(0)), s, np.nextafter(s, f(np.inf))):
                assert (np.sqrt(v) < r) == (v < s)
            first = least(lambda v: v / c > t)
            dmax = np.nextafter(first, f(0))
            for v in (dmax, first, np.nextafter(first, f(np.inf)), np.nextafter(dmax, f(0))):
                assert (v / c > t) == (v > dmax)
