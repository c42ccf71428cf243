"""The early reflections' launches: discovery with a warp or a lane per fan ray
(by the number of rays), closest hits by whole warps (trees numbered on the
host) or by one lane (trees built on the device), in first-found and near-tie
contexts, with more blockers than a warp has lanes. All equal the oracle.

Tolerance: chains, validity, delays and directions equal; gains within 2e-6
relative, as in test_gpu_early.py (exp of the air attenuation).
"""
import numpy as np
import pytest

from omg_audio_gb300 import Context, MeshBuilder, TraceConfig, _lib
from omg_audio_gb300 import materials as M
from omg_audio_gb300.early import WorldEarly
from omg_audio_gb300.materials import Material
from omg_audio_gb300.world import build_world_mesh

from test_gpu_early import SOURCES, SPOTS, _chain_list
from test_oracle_early import BOX_QUADS, box_mesh, omat
from walkthrough import furniture_world, oracle_world, product_world

pytestmark = pytest.mark.gpu


def _same(early, oe, sources, chains, lis, extras):
    rec = early.solve(sources, chains, lis, extras)
    ref, valid = oe.solve(sources, chains, lis, extras, threads=8)
    gv = rec["valid"].astype(bool)
    assert np.array_equal(gv, valid), np.argwhere(gv != valid)[:5]
    r, o = rec[gv], ref[valid]
    assert np.array_equal(r["delay_s"], o[:, 0])
    assert np.array_equal(r["dir"], o[:, 1:4])
    assert np.all(np.abs(r["gains"] - o[:, 4:7]) <= 2e-6 * np.abs(o[:, 4:7]) + 1e-30)
    return int(valid.sum())


@pytest.mark.parametrize("tie", [0, 1])
def test_world_by_number_of_rays_and_blockers(oracle, tie):
    O = oracle
    with Context(TraceConfig(tie_mode=tie)) as ctx:
        R, D = product_world()
        mb = MeshBuilder()
        build_world_mesh(mb, R, D)
        scene = ctx.upload_builder(mb, 3, _lib.BVH_SAH)
        furn_g, _ = furniture_world(lambda m: Material(tuple(m["absorption"]), m["scattering"],
                                                       tuple(m["transmission"])))
        furn_o, _ = furniture_world(lambda m: O.Material.make(m["absorption"], m["scattering"], m["transmission"]))
        early = WorldEarly(ctx, scene, furn_g)
        ob = O.MeshBuilder()
        O.world_build(ob, *oracle_world(O))
        oe = O.Early(ob.build("f32"), furn_o)
        lis = SPOTS[1]
        for n_rays in (1, 31, 65, 9000):
            assert early.discover(lis, n_rays, 3) == oe.discover(lis, n_rays, 3), n_rays
        chains = _chain_list(oe, lis, 120)
        # 45 thin blockers about the listener: more than the lanes of a warp
        extras = [((lis[0] - 1.0 + 0.04 * k, lis[1] - 0.6, 0.0), (lis[0] - 0.99 + 0.04 * k, lis[1] + 0.6, 2.0),
                   (0.9, 0.95, 0.99)) for k in range(45)]
        for n_src in (1, len(SOURCES)):
            assert _same(early, oe, SOURCES[:n_src], chains, lis, extras) > 0
        early.close()
        scene.release()


@pytest.mark.parametrize("bvh", [_lib.BVH_SAH, _lib.BVH_LBVH])
def test_box_over_both_trees(oracle, bvh):
    with Context(TraceConfig()) as ctx:
        mb = MeshBuilder()
        mat = mb.material(M.CONCRETE)
        for q, _ in BOX_QUADS:
            mb.begin_surface()
            mb.quad(*[np.float32(p) for p in q], mat)
        scene = ctx.upload_builder(mb, 3, bvh)
        mn, mx = (2.0, 1.5, 0.0), (3.0, 2.5, 0.8)
        early = WorldEarly(ctx, scene, [(mn, mx, M.WOOD_PANEL)])
        oe = oracle.Early(box_mesh(oracle, [M.CONCRETE] * 6), [(mn, mx, omat(oracle, M.WOOD_PANEL))])
        lis = (4.03, 2.07, 1.61)
        for n_rays in (40, 768, 9000):
            assert early.discover(lis, n_rays, 1) == oe.discover(lis, n_rays, 1), n_rays
        chains = _chain_list(oe, lis)
        sources = [(k, (0.53 + 0.61 * k, 1.13 + 0.27 * k, 1.07 + 0.13 * k)) for k in range(9)]
        assert _same(early, oe, sources, chains, lis, ()) > 20
        early.close()
        scene.release()
