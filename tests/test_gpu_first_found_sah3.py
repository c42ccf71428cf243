"""The first-found rule on the three-axis tree, whose order decides between equal
hits: launches of few rays (a warp per ray), of lanes, and with a second launch for
their last rays, against the wavefront rounds, which walk the same tree node by node
in the reference's order. Rooms that share walls and coincident sheets (most walls are
there twice or more), with panels, 3 and 8 bands; then the early reflections of a
room against the oracle. Segments and echograms equal (the sums are exact)."""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, MeshBuilder, TraceConfig, _lib
from omg_audio_gb300 import materials as M
from omg_audio_gb300 import workloads as W
from omg_audio_gb300.early import WorldEarly

from test_gpu_early import _chain_list
from test_gpu_early_paths import _same
from test_gpu_parity import gpu_scene
from test_gpu_solo import _sheets
from test_oracle_early import BOX_QUADS, box_mesh, omat

pytestmark = pytest.mark.gpu

BOUNCES = 24


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _agree(ctx, job, panels, sizes):
    for rays, kernels in sizes:
        b = ctx.batch([job(rays)], panels)
        b.set_shape(mode=0, wf_rounds=BOUNCES, wf_tail=0, epochs=0)
        b.launch()
        (want, wr), = b.read()
        b.set_shape(mode=0, wf_rounds=0, epochs=0)
        assert b.kernel_count() == kernels, rays
        b.launch()
        (got, gr), = b.read()
        assert gr.segments == wr.segments > 0, rays
        assert np.array_equal(got.bins, want.bins) and np.array_equal(got.dirs, want.dirs), rays
        b.destroy()


def _sizes():
    unit = 28 * _sms()
    return [(500, 3), (2 * unit, 3), (2 * unit + 1, 3), (3 * unit - 1, 3), (3 * unit, 4), (9 * unit + 7, 4)]


@pytest.mark.parametrize("seed,nx,ny", [(2, 4, 3), (9, 2, 1)])
def test_shared_walls_and_panels(seed, nx, ny):
    case = W.multiroom(seed=seed, nx=nx, ny=ny, n_pairs=2)
    with Context(TraceConfig(tie_mode=0, max_bounces=BOUNCES)) as ctx:
        scene = gpu_scene(ctx, case.recorder, _lib.BVH_SAH3)
        for k, (src, lis) in enumerate(case.pairs):
            _agree(ctx, lambda n: Job(src, lis, n, seed=40 + k, scene=scene, panel_offset=0, n_panels=len(case.panels)),
                   case.panels, _sizes())


def test_eight_bands():
    case = W.city(seed=3, nx=3, ny=2, n_sources=1, n_dome=1)
    src, lis = (tuple(map(float, p[0])) for p in (case.sources, case.listeners))
    with Context(TraceConfig(tie_mode=0, max_bounces=BOUNCES)) as ctx:
        scene = gpu_scene(ctx, case.recorder, _lib.BVH_SAH3, 8)
        _agree(ctx, lambda n: Job(src, lis, n, seed=4, scene=scene, n_bands=8), [], _sizes())


@pytest.mark.parametrize("n,gap", [(2, 0.0), (40, 0.0), (200, 1e-7), (300, 1e-5), (12, 3e-4)])
def test_coincident_sheets(n, gap):
    with Context(TraceConfig(tie_mode=0, max_bounces=BOUNCES)) as ctx:
        scene = gpu_scene(ctx, _sheets(n, gap), _lib.BVH_SAH3)
        _agree(ctx, lambda r: Job((1.5, 1, 1.5), (4.5, 3, 1.6), r, seed=5, scene=scene), [], _sizes()[:5])


@pytest.mark.parametrize("tie", [0, 1])
def test_early_reflections(oracle, tie):
    with Context(TraceConfig(tie_mode=tie)) as ctx:
        mb = MeshBuilder()
        mat = mb.material(M.CONCRETE)
        for q, _ in BOX_QUADS:
            mb.begin_surface()
            mb.quad(*[np.float32(p) for p in q], mat)
        scene = ctx.upload_builder(mb, 3, _lib.BVH_SAH3)
        mn, mx = (2.0, 1.5, 0.0), (3.0, 2.5, 0.8)
        early = WorldEarly(ctx, scene, [(mn, mx, M.WOOD_PANEL)])
        oe = oracle.Early(box_mesh(oracle, [M.CONCRETE] * 6), [(mn, mx, omat(oracle, M.WOOD_PANEL))])
        lis = (4.03, 2.07, 1.61)
        for n_rays in (40, 768, 9000):
            assert early.discover(lis, n_rays, 1) == oe.discover(lis, n_rays, 1), n_rays
        sources = [(k, (0.53 + 0.61 * k, 1.13 + 0.27 * k, 1.07 + 0.13 * k)) for k in range(9)]
        assert _same(early, oe, sources, _chain_list(oe, lis), lis, ()) > 20
        early.close()
        scene.release()
