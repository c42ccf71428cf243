"""The packed job, panel and chain records equal the field-by-field ones, byte
for byte, over bands, numpy values and values that only a field assignment
takes (an integer out of range wraps, a float beyond f32 becomes infinity)."""
import ctypes as C

import numpy as np
import pytest

from omg_audio_gb300 import _lib
from omg_audio_gb300 import engine as E
from omg_audio_gb300.early import chains_to_c
from omg_audio_gb300.engine import Job, TraceConfig
from omg_audio_gb300.materials import BRICK, CARPET, CONCRETE, Material


class _Scene:
    def __init__(self, sid, nb):
        self.id, self.n_bands = sid, nb


def _mat(rng, nb):
    return Material(tuple(map(float, rng.random(nb))), float(rng.random()), tuple(rng.random(nb)))


def _jobs(rng):
    out = [Job((1, 2, 3), (4.5, 5, 6), 100, box_size=(7, 8, 9), box_walls=[CONCRETE, BRICK, CARPET] * 2),
           Job(np.array([1, 2, 3.0]), np.float32([4, 5, 6]), np.int64(7), seed=-3, scene=_Scene(5, 8), n_bins=400,
               max_time=2.5, panel_offset=3, n_panels=2),
           Job([1, 2, 3, 99], (4, 5, 6), 7, scene=_Scene(9, 1), energy=[0.5, 0.25, 3.0]),
           Job((1, 2, 3), (4, 5, 6), 7, seed=1 << 40, box_size=[1, 1, 1], n_bands=8, energy=np.arange(8) / 3,
               box_walls=[_mat(rng, 8) for _ in range(6)])]
    return out


ODD = [Job((1e40, 2, 3), (4, 5, 6), 7, scene=_Scene(1, 3)), Job((1, 2, 3), (4, 5, 6), -1, scene=_Scene(1, 3)),
       Job((1, 2, 3), (4, 5, 6), 1 << 33, box_size=(1, 2, 3), box_walls=[CONCRETE] * 6)]


@pytest.mark.parametrize("odd", [None, 0, 1, 2])
def test_jobs(odd):
    jobs = _jobs(np.random.default_rng(1)) + ([] if odd is None else [ODD[odd]])
    cfg = TraceConfig(n_bins=300)
    arr, nbf, ndf = E.jobs_to_c(jobs, cfg)
    assert bytes(arr) == bytes(E._jobs_by_field(jobs, cfg))
    assert nbf == sum(j.bins_len(cfg) * j.bands(cfg) for j in jobs) and ndf == 3 * sum(j.bins_len(cfg) for j in jobs)
    assert len(arr) == len(jobs) and arr[1].scene_id == 5 and arr[0].box_walls[1].scattering == np.float32(0.12)


def test_panels_and_box_jobs():
    rng = np.random.default_rng(2)
    pan = [((0, 0, 0), (1, 1, 1), CONCRETE), (np.zeros(3), np.float32([1, 2, 3]), _mat(rng, 8)),
           ([0, 1, 2], (3, 4, 1e300), _mat(rng, 1)), ((0, 0, 0), (1, 1, 1), Material((), 0.5, ()))]
    for k in range(len(pan) + 1):
        assert bytes(E.panels_to_c(pan[:k])) == bytes(E._panels_by_field(pan[:k]))
    for args in (((6, 4, 3), [CONCRETE, BRICK, CARPET] * 2, (1, 2, 3), (4, 5, 6), 100, None, 7, 3),
                 (np.ones(3), [_mat(rng, 8)] * 6, [1, 2, 3], (4, 5, 6), -5, range(8), -1, 8)):
        size, walls, src, lis, n, energy, seed, nb = args
        j = E._box_job(*args)
        want = _lib.omg_box_job()
        for k in range(3):
            want.size[k], want.src[k], want.lis[k] = size[k], src[k], lis[k]
        for w in range(6):
            want.walls[w] = walls[w].to_c()
        want.n_rays, want.seed = n, seed & 0xFFFFFFFF
        for b in range(nb):
            want.energy[b] = 1.0 if energy is None else energy[b]
        assert bytes(j) == bytes(want)


def test_more_bands_than_a_record_holds_are_refused():
    with pytest.raises(IndexError):
        E.panels_to_c([((0, 0, 0), (1, 1, 1), Material((0.1,) * 9, 0.1, (0.0,) * 9))])


def test_chains():
    chains = [((1, 2, 3), 3), ((65535, 65535, 65535), 0), ((70000, -1, 5), 2)]
    arr = chains_to_c(chains)
    for a, (c, o) in zip(arr, chains):
        assert [a.surf[k] for k in range(3)] == [v & 0xFFFF for v in c] and a.order == o
    assert C.sizeof(chains_to_c([])) == C.sizeof(_lib.omg_chain)
