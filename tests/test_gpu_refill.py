"""A call that is refused after its walls or panels were taken in leaves nothing
behind: the corrected call, of the same layout, equals that of a context which was
never asked the refused one, bit for bit. One-shot batches and the late field, with new walls, with new panels, with both."""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig, _lib
from omg_audio_gb300 import materials as M
from omg_audio_gb300 import workloads as W
from omg_audio_gb300.sim import LateField

from test_gpu_parity import gpu_scene

pytestmark = pytest.mark.gpu

CFG = dict(n_bins=300, max_bounces=64, tie_mode=1)
ROOM = W.shoebox12(seed=4)


def _jobs(scene, walls, bad=False):
    """A shoebox with panels, then a mesh whose source the caller may have got wrong."""
    src = (float("nan"), 1.0, 1.0) if bad else ROOM.src
    return [Job((1.0, 1.0, 1.5), (4.0, 3.0, 1.5), 2048, seed=1, box_size=(6.0, 4.0, 3.0), box_walls=[walls] * 6,
                panel_offset=0, n_panels=4),
            Job(src, ROOM.lis, 2048, seed=2, scene=scene)]


def _panels(z, m):
    return [((2.0 + 0.2 * k, 1.0, 0.0), (2.1 + 0.2 * k, 3.0, z), m) for k in range(4)]


OLD = (M.CONCRETE, 1.0, M.DRYWALL)
CHANGES = [(M.CARPET, 1.0, M.DRYWALL), (M.CONCRETE, 2.0, M.DRYWALL), (M.CARPET, 2.0, M.WOOD_PANEL)]


def _one_shot(ctx, scene, walls, z, pm, bad=False):
    return [e for e, _ in ctx.trace_batch(_jobs(scene, walls, bad), _panels(z, pm))]


def _late(field, scene, walls, z, pm, bad=False):
    field.submit([0, 1], _jobs(scene, walls, bad), _panels(z, pm), alpha=[1.0, 1.0])
    field.poll(wait=True)
    return [field.read(s) for s in (0, 1)]


@pytest.mark.parametrize("late", [False, True], ids=["one-shot", "late"])
@pytest.mark.parametrize("change", CHANGES, ids=["walls", "panels", "both"])
def test_refused_call_leaves_nothing_behind(late, change):
    def ready(ctx):
        scene = gpu_scene(ctx, ROOM.recorder)
        if not late:
            return lambda *a, **k: _one_shot(ctx, scene, *a, **k)
        field = LateField(ctx, 2)
        return lambda *a, **k: _late(field, scene, *a, **k)

    with Context(TraceConfig(**CFG)) as ctx:
        run = ready(ctx)
        old = run(*OLD)
        with pytest.raises(_lib.OmgError) as e:
            run(*change, bad=True)
        assert e.value.status == _lib.E_INVALID
        got = run(*change)
    with Context(TraceConfig(**CFG)) as ctx:
        run = ready(ctx)
        run(*OLD)                             # (the field averages over both)
        ctx.trace_batch([Job((1.0, 1.0, 1.5), (2.0, 2.0, 1.5), 64, box_size=(4.0, 4.0, 3.0),
                             box_walls=[M.BRICK] * 6)])   # another layout: nothing kept for the next call
        want = run(*change)
    assert not np.array_equal(got[0].bins, old[0].bins)
    for g, w in zip(got, want):
        assert np.array_equal(g.bins, w.bins) and np.array_equal(g.dirs, w.dirs)
