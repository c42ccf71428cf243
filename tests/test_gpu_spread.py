"""Launches of few rays: the rays are spread over more warps (fewer than 32 a
warp, launch_trace). At ray counts around the steps of that rule a trace equals
the f32 oracle on the same streams: the segment counts exactly, the bins within
the compensated sums' 1e-5 (bins holding >= 1e-6 of the band total)."""
import pytest

from omg_audio_gb300 import Context, MeshBuilder, TraceConfig
from omg_audio_gb300 import materials as M
from omg_audio_gb300 import workloads as W

from test_gpu_parity import oparams, rel_bins
from test_oracle_golden import omat

pytestmark = pytest.mark.gpu

# 1 ray; one short of and one past a ray a warp on the small rule (16 warps x 152) and on the deep one (32)
RAYS = [1, 33, 2431, 2433, 4865, 9729, 40000, 77825]


@pytest.mark.parametrize("rays", RAYS)
@pytest.mark.parametrize("tie", [0, 1], ids=["first-found", "near-tie"])
def test_small_launch_on_a_mesh_equals_the_oracle(oracle, tie, rays):
    O = oracle
    case = W.shoebox12(seed=1) if rays != 4865 else W.multiroom(nx=2, ny=2, n_pairs=2)
    src, lis = (case.src, case.lis) if rays != 4865 else case.pairs[0]
    with Context(TraceConfig(tie_mode=tie, n_bins=300, bin_dt=0.01, max_bounces=24, timeout_ms=60000)) as ctx:
        mb = MeshBuilder()
        case.recorder.replay(mb)
        scene = ctx.upload_builder(mb)
        ob = O.MeshBuilder()
        case.recorder.replay(ob, lambda m: omat(O, m))
        P = oparams(O, ctx.cfg)
        b, _, st = O.trace_mesh(ob.build("f32"), src, lis, rays, P=P, seed=9, threads=8, acc64=True)
        e, rv = ctx.trace_world(scene, src, lis, rays, seed=9)
        assert rv.segments == st["segments"]
        assert rel_bins(e.bins, b) <= 1e-5


@pytest.mark.parametrize("rays", RAYS)
def test_small_launch_in_a_box_equals_the_oracle(oracle, rays):
    O = oracle
    walls = [M.CONCRETE, M.DRYWALL, M.WOOD_PANEL, M.BRICK, M.CARPET, M.ACOUSTIC_TILE]
    with Context(TraceConfig(max_bounces=24, timeout_ms=60000)) as ctx:
        e, rv = ctx.trace_box((6, 4, 3), walls, (1.5, 1, 1.5), (4.5, 3, 1.6), rays, seed=7)
        b, _, st = O.trace_box((6, 4, 3), [omat(O, m) for m in walls], (1.5, 1, 1.5), (4.5, 3, 1.6), rays, seed=7,
                               P=oparams(O, ctx.cfg), acc64=True)
        assert rv.segments == st["segments"]
        assert rel_bins(e.bins, b) <= 1e-5
