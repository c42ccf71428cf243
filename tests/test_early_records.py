"""Chains and blockers as the C records of a solve: what a field takes is packed to the
same bytes, what a field refuses is refused."""
import ctypes as C

import numpy as np
import pytest

from omg_audio_gb300 import _lib
from omg_audio_gb300.early import chains_to_c, extras_to_c


def _chains_by_field(chains):
    arr = (_lib.omg_chain * max(1, len(chains)))()
    for i, (c, o) in enumerate(chains):
        for k in range(3):
            arr[i].surf[k] = c[k]
        arr[i].order = o
    return arr


def _extras_by_field(extras):
    ex = (_lib.omg_aabb * max(1, len(extras)))()
    for i, (mn, mx, tr) in enumerate(extras):
        for k in range(3):
            ex[i].mn[k], ex[i].mx[k], ex[i].transmission[k] = mn[k], mx[k], tr[k]
    return ex


CHAINS = [[], [((1, 2, 3), 3)], [((0, 65535, 7), 1), ((-1, 65536, 1 << 70), 2)],
          [((np.uint16(5), np.int64(6), np.int32(-2)), np.int64(3))], [((True, False, 4), 2), ([9, 8, 7, 6], 3)]]


@pytest.mark.parametrize("chains", CHAINS)
def test_chains_equal_their_fields(chains):
    assert bytes(chains_to_c(chains)) == bytes(_chains_by_field(chains))


@pytest.mark.parametrize("bad", [1.5, 1.0, np.float32(2.0), np.float64(3.0), "4", None, b"5", 1j])
@pytest.mark.parametrize("place", range(4))
def test_chains_refuse_what_a_field_refuses(bad, place):
    v = [1, 2, 3, 3]
    v[place] = bad
    chains = [((0, 1, 2), 1), (tuple(v[:3]), v[3])]
    with pytest.raises(TypeError):
        _chains_by_field(chains)
    with pytest.raises(TypeError):
        chains_to_c(chains)


EXTRAS = [[], [((0, 1, 2), (3, 4, 5), (0.1, 0.2, 0.3))],
          [((np.float64(0.1), np.float32(0.2), -0.0), np.arange(3.0), [1e-40, 1e39, -1e300]),
           ((float("inf"), True, 1 << 60), (float("-inf"), 2, 3), (4, 5, 6))]]


@pytest.mark.parametrize("extras", EXTRAS)
def test_extras_equal_their_fields(extras):
    assert extras_to_c(extras).tobytes() == bytes(_extras_by_field(extras))
    assert C.sizeof(_lib.omg_aabb) == 36


@pytest.mark.parametrize("bad", ["1.0", None, 1j, b"2"])
@pytest.mark.parametrize("place", range(9))
def test_extras_refuse_what_a_field_refuses(bad, place):
    v = [0.0] * 9
    v[place] = bad
    extras = [(v[:3], v[3:6], v[6:])]
    with pytest.raises(TypeError):
        _extras_by_field(extras)
    with pytest.raises(TypeError):
        extras_to_c(extras)
