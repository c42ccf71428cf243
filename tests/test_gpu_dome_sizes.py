"""The dome's launches by size: few (listener, ray) pairs spread one to a warp,
many fill the warps, and panels are tested a lane each when a warp holds few
rays. A listener's escapes and bins do not depend on how many share the call
(the fan is fixed per listener): a call of many listeners equals calls of one,
bit for bit, and the escapes equal the f32 oracle's under both hit rules.

Tolerance: none; the arithmetic per ray is the same in every launch shape.
"""
import numpy as np
import pytest

from omg_audio_gb300 import DomeProbe, MeshBuilder
from omg_audio_gb300 import workloads as W
from omg_audio_gb300.world import door_panels

from test_gpu_dome import _oracle_probe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tie", [False, True])
@pytest.mark.parametrize("n_eyes,n_rays", [(1, 1), (3, 33), (17, 512), (150, 384)])
def test_listeners_do_not_depend_on_their_company(ctx, ctx_tie, oracle, tie, n_eyes, n_rays):
    c = ctx_tie if tie else ctx
    case = W.multiroom(seed=5)
    mb = MeshBuilder()
    case.recorder.replay(mb)
    scene = c.upload_builder(mb)
    probe = DomeProbe(c, scene, case.glass, n_fan=n_rays)
    base = np.asarray(case.listeners, np.float32)
    eyes = np.concatenate([base + np.float32(0.01 * k) for k in range(1 + n_eyes // len(base))])[:n_eyes]
    doors = [d for d in case.doors if not d.glass]
    doors[0].openness, doors[2].openness = 0.0, 0.5
    leaves = door_panels(doors)
    g = probe.sample(eyes, leaves, n_rays=n_rays)
    for e in sorted({0, n_eyes // 2, n_eyes - 1}):
        one = probe.sample(eyes[e:e + 1], leaves, n_rays=n_rays)
        assert np.array_equal(one["escape"][0], g["escape"][e])
        assert np.array_equal(one["raw"][0], g["raw"][e])
    _, p32 = _oracle_probe(oracle, case, "f32", n_rays, tie=tie)
    ref = p32.sample(eyes[0], [l.as_dict() for l in leaves], n_rays=n_rays)
    assert np.array_equal(g["escape"][0], ref["escape"])
    scene.release()
