"""The hand-over of a launch's last rays, decided by each warp as one: many launches
at the sizes where the threshold is met early, late or by a batch of jobs that end at
different times. Every launch equals the first bit for bit (the sums are exact and a
ray's stream is its own), and the segments are those of the same batch without a
second launch."""
import numpy as np
import pytest

from omg_audio_gb300 import Context, Job, TraceConfig
from omg_audio_gb300 import workloads as W

from test_gpu_parity import gpu_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tie", [0, 1])
@pytest.mark.parametrize("units", [3.0, 4.5, 9.0, 20.0])
def test_launches_repeat(tie, units):
    import torch
    total = int(units * 28 * torch.cuda.get_device_properties(0).multi_processor_count)
    with Context(TraceConfig(tie_mode=tie, max_bounces=64)) as ctx:
        case = W.multiroom(seed=6, nx=3, ny=2)
        scene = gpu_scene(ctx, case.recorder)
        room = W.shoebox12(seed=4)
        small = gpu_scene(ctx, room.recorder)
        a = total // 3
        jobs = [Job(*case.pairs[0][:2], a, seed=1, scene=scene), Job(room.src, room.lis, a, seed=2, scene=small),
                Job(*case.pairs[1][:2], total - 2 * a, seed=3, scene=scene)]
        b = ctx.batch(jobs)
        b.set_shape(mode=0, epochs=1)
        b.launch()
        alone = [rv.segments for _, rv in b.read()]
        b.set_shape(mode=0, epochs=0)
        assert b.kernel_count() == 4
        first = None
        for _ in range(12):
            b.launch()
            got = b.read()
            assert [rv.segments for _, rv in got] == alone
            first = first or [(e.bins.copy(), e.dirs.copy()) for e, _ in got]
            for (bins, dirs), (e, _) in zip(first, got):
                assert np.array_equal(bins, e.bins) and np.array_equal(dirs, e.dirs)
        b.destroy()
        scene.release()
        small.release()
