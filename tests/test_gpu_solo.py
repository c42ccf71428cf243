"""Launches of few rays on meshes (a warp per ray, solo.cu) against the oracle on
the same streams, segment counts equal and bins within the compensated sums'
1e-5: both hit rules, the reference's and the three-axis tree, 3 and 8 bands,
panels, shoebox jobs in the same batch, a scene of one leaf, and scenes on which
its lists fill (hundreds of coincident sheets) so that the lane walk takes over.
The first-found rule is compared on rooms that share walls, where most walls
are authored twice and the tree's order decides."""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, Material, MeshBuilder, TraceConfig, _lib
from omg_audio_gb300 import materials as M
from omg_audio_gb300 import workloads as W

from test_gpu_parity import oparams, rel_bins
from test_oracle_golden import omat

pytestmark = pytest.mark.gpu


def _both(ctx, O, rec, nb=3, bvh=_lib.BVH_SAH):
    mb = MeshBuilder()
    rec.replay(mb)
    ob = O.MeshBuilder()
    rec.replay(ob, lambda m: omat(O, m))
    return ctx.upload_builder(mb, nb, bvh), ob.build("f32")


@pytest.mark.parametrize("tie,bvh", [(0, _lib.BVH_SAH), (1, _lib.BVH_SAH), (1, _lib.BVH_SAH3)])
@pytest.mark.parametrize("seed,nx,ny", [(2, 4, 3), (9, 2, 1), (5, 8, 5)])
def test_shared_walls_and_panels(oracle, tie, bvh, seed, nx, ny):
    O = oracle
    case = W.multiroom(seed=seed, nx=nx, ny=ny, n_pairs=4)
    with Context(TraceConfig(tie_mode=tie, n_bins=300, bin_dt=0.01, max_bounces=64, timeout_ms=60000)) as ctx:
        scene, mesh = _both(ctx, O, case.recorder, bvh=bvh)
        pan = [(mn, mx, omat(O, m)) for mn, mx, m in case.panels]
        P = oparams(O, ctx.cfg)
        for k, (src, lis) in enumerate(case.pairs):
            b, _, st = O.trace_mesh(mesh, src, lis, 4000, seed=40 + k, P=P, panels=pan, threads=8, acc64=True)
            e, rv = ctx.trace_world(scene, src, lis, 4000, case.panels, seed=40 + k)
            assert rv.segments == st["segments"], k
            assert rel_bins(e.bins, b) <= 1e-5, k


@pytest.mark.parametrize("tie", [0, 1])
def test_eight_bands_and_mixed_jobs(oracle, tie):
    O = oracle
    rooms = W.room_batch(seed=11, n_rooms=6, tri_median=300, tri_hi=900, ray_lo=300, ray_hi=1200)
    with Context(TraceConfig(tie_mode=tie, n_bins=400, bin_dt=0.005, max_bounces=50, timeout_ms=60000)) as ctx:
        jobs, want = [], []
        P = oparams(O, ctx.cfg)
        for k, r in enumerate(rooms):
            scene, mesh = _both(ctx, O, r.recorder, r.n_bands)
            jobs.append(Job(r.src, r.lis, r.n_rays, seed=7 + k, scene=scene, n_bands=r.n_bands))
            Pk = oparams(O, ctx.cfg)
            Pk.n_bands = r.n_bands
            want.append(O.trace_mesh(mesh, r.src, r.lis, r.n_rays, energy=[1.0] * r.n_bands, seed=7 + k, P=Pk,
                                     threads=8, acc64=True))
        walls = [M.CONCRETE, M.DRYWALL, M.WOOD_PANEL, M.BRICK, M.CARPET, M.ACOUSTIC_TILE]
        jobs.append(Job((1.5, 1, 1.5), (4.5, 3, 1.6), 500, seed=3, box_size=(6, 4, 3), box_walls=walls))
        want.append(O.trace_box((6, 4, 3), [omat(O, m) for m in walls], (1.5, 1, 1.5), (4.5, 3, 1.6), 500, seed=3, P=P,
                                acc64=True))
        assert sum(j.n_rays for j in jobs) < 8000
        for (e, rv), (b, _, st) in zip(ctx.trace_batch(jobs), want):
            assert rv.segments == st["segments"]
            assert rel_bins(e.bins, b) <= 1e-5


def _sheets(n, gap):
    """A 6 x 4 x 3 m room whose far wall is n sheets, `gap` apart, each of another material."""
    rng = np.random.default_rng(n)
    rec = W.Recorder()
    room = rec.material(M.CONCRETE)
    W._abox(rec, (0.0, 0.0, 0.0), (6.0, 4.0, 3.0), room)
    rec.coarse(1e9)
    for k in range(n):
        m = rec.material(Material(tuple(rng.uniform(0.02, 0.5, 3)), 0.2, tuple(rng.uniform(0.0, 0.5, 3))))
        x = 5.0 + gap * k
        rec.begin_surface()
        rec.quad((x, 0.1, 0.1), (x, 3.9, 0.1), (x, 3.9, 2.9), (x, 0.1, 2.9), m)
    return rec


@pytest.mark.parametrize("tie", [0, 1])
@pytest.mark.parametrize("n,gap", [(2, 0.0), (40, 0.0), (200, 0.0), (200, 1e-7), (300, 1e-5), (12, 3e-4)])
def test_coincident_sheets(oracle, tie, n, gap):
    O = oracle
    with Context(TraceConfig(tie_mode=tie, n_bins=300, bin_dt=0.01, max_bounces=24, timeout_ms=60000)) as ctx:
        scene, mesh = _both(ctx, O, _sheets(n, gap))
        P = oparams(O, ctx.cfg)
        b, _, st = O.trace_mesh(mesh, (1.5, 1, 1.5), (4.5, 3, 1.6), 2000, seed=5, P=P, threads=8, acc64=True)
        e, rv = ctx.trace_world(scene, (1.5, 1, 1.5), (4.5, 3, 1.6), 2000, seed=5)
        assert rv.segments == st["segments"]
        assert rel_bins(e.bins, b) <= 1e-5


@pytest.mark.parametrize("tie", [0, 1])
def test_a_scene_of_one_leaf(oracle, tie):
    O = oracle
    rec = W.Recorder()
    m = rec.material(Material((0.1, 0.2, 0.3), 0.5, (0.0,) * 3))
    rec.coarse(1e9)
    rec.begin_surface()
    rec.quad((-5, -5, 0), (5, -5, 0), (5, 5, 0), (-5, 5, 0), m)
    with Context(TraceConfig(tie_mode=tie, max_bounces=8)) as ctx:
        scene, mesh = _both(ctx, O, rec)
        P = oparams(O, ctx.cfg)
        b, _, st = O.trace_mesh(mesh, (0, 0, 1), (1, 1, 1.5), 3000, seed=5, P=P, acc64=True)
        e, rv = ctx.trace_world(scene, (0, 0, 1), (1, 1, 1.5), 3000, seed=5)
        assert rv.segments == st["segments"]
        assert rel_bins(e.bins, b) <= 1e-5
