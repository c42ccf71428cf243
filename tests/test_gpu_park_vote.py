"""The park signal of an epoch, taken up by each warp of the wavefront kernels as one:
many launches with thresholds that raise it early and late, their segments those of
the single launch each time and their echograms equal to the first launch's."""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig
from omg_audio_gb300 import workloads as W

from test_gpu_parity import gpu_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [dict(mode=1, tail_mode=1), dict(mode=2, tail_mode=2), dict(mode=0, tail_mode=2)],
                         ids=["wavefront", "cooperative", "tail"])
@pytest.mark.parametrize("epochs,pct", [(2, 5), (8, 50), (32, 95)])
def test_launches_repeat(shape, epochs, pct):
    with Context(TraceConfig(tie_mode=1, max_bounces=64)) as ctx:
        case = W.multiroom(seed=6, nx=3, ny=2)
        scene = gpu_scene(ctx, case.recorder)
        b = ctx.batch([Job(*case.pairs[k][:2], 12001 + k, seed=k, scene=scene) for k in range(3)])
        b.set_shape(mode=0, tail_mode=0, epochs=0)
        b.launch()
        alone = [rv.segments for _, rv in b.read()]
        b.set_shape(epochs=epochs, park_pct=pct, **shape)
        first = None
        for _ in range(8):
            b.launch()
            got = b.read()
            assert [rv.segments for _, rv in got] == alone
            first = first or [(e.bins.copy(), e.dirs.copy()) for e, _ in got]
            for (bins, dirs), (e, _) in zip(first, got):
                assert np.array_equal(bins, e.bins) and np.array_equal(dirs, e.dirs)
        b.destroy()
        scene.release()
