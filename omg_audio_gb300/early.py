"""World early reflections over the C ABI (include/omg_cuda.h, "world early
reflections"): the surface table of an uploaded world mesh plus furniture
faces, chain discovery from the listener (the WorldDiscovery seam,
crates/omg-scene/src/early_world.rs:18-26; mesh_chains, pt_mesh.rs:382-457)
and the batched exact solve of every (source, chain) pair (the WorldSolve
seam, early_world.rs:36-48; mesh_record, pt_mesh.rs:186-337)."""
from __future__ import annotations

import ctypes as C
import operator
from array import array
from typing import List, Sequence, Tuple

import numpy as np

from . import _lib
from ._lib import lib
from .engine import panels_to_c

NO_SURF = _lib.NO_SURF
Chain = Tuple[Tuple[int, int, int], int]


def _p(a: np.ndarray):
    return a.ctypes.data_as(C.c_void_p)


def _f3(v):
    return np.ascontiguousarray(np.asarray(v, np.float32).reshape(3))


_RECORD = np.dtype(_lib.omg_mesh_record)


def chains_to_c(chains: Sequence[Chain]):
    """omg_chain records (three u16 surfaces and the u16 order each). Integers alone;
    one beyond 16 bits keeps its low ones, as assigned to a field."""
    arr = (_lib.omg_chain * max(1, len(chains)))()
    if len(chains):
        flat = [v for c, o in chains for v in (c[0], c[1], c[2], o)]
        try:
            flat = array("H", flat)
        except OverflowError:
            flat = array("H", [operator.index(v) & 0xFFFF for v in flat])
        C.memmove(arr, flat.buffer_info()[0], C.sizeof(_lib.omg_chain) * len(chains))
    return arr


def extras_to_c(extras: Sequence):
    """omg_aabb records of (mn, mx, transmission) triples, one of zeros for none."""
    flat = array("f", [x for mn, mx, tr in extras
                       for x in (mn[0], mn[1], mn[2], mx[0], mx[1], mx[2], tr[0], tr[1], tr[2])])
    return np.frombuffer(flat, np.float32) if len(flat) else np.zeros(9, np.float32)


class WorldEarly:
    """SurfaceTable::build + append_box over an uploaded scene (early_world.rs:114-120).
    furniture: (min, max, Material) triples; their faces reflect, and discovery
    rays bounce off the boxes."""

    def __init__(self, ctx, scene, furniture: Sequence = ()):
        self.ctx = ctx
        self.scene = scene
        pan = [(tuple(mn), tuple(mx), m) for (mn, mx, m) in furniture]
        arr = panels_to_c(pan)
        eid = C.c_uint32()
        ctx._check(lib().omg_early_create(ctx.h, scene.id, arr, len(pan), C.byref(eid)), "omg_early_create")
        self.id = eid.value
        b, n = C.c_uint32(), C.c_uint32()
        ctx._check(lib().omg_early_info(ctx.h, self.id, C.byref(b), C.byref(n)), "omg_early_info")
        self.base_overlay, self.n_surfaces = b.value, n.value

    def close(self):
        if getattr(self, "id", None) and self.ctx.h:
            lib().omg_early_destroy(self.ctx.h, self.id)
            self.id = None

    def __del__(self):
        self.close()

    def discover(self, listener, n_rays: int = 768, rot: int = 0, use_boxes: bool = True) -> List[Chain]:
        """mesh_chains: unique chains in the reference's first-found order."""
        cap = 3 * max(n_rays, 1)
        out = np.empty((cap, 4), np.uint16)
        n = C.c_uint32()
        self.ctx._check(lib().omg_early_discover(self.ctx.h, self.id, _p(_f3(listener)), n_rays, rot,
                                                 int(use_boxes), _p(out), cap, C.byref(n)), "omg_early_discover")
        return [((a, b, c), o) for a, b, c, o in out[:min(n.value, cap)].tolist()]

    def solve(self, sources: Sequence[Tuple[int, Sequence[float]]], chains: Sequence[Chain], listener,
              extras: Sequence = ()):
        """mesh_record for every (source, chain) pair: a structured array
        (n_sources, n_chains) with delay_s, dir, gains, key, valid.
        extras: (min, max, transmission3) blockers."""
        ns, nc = len(sources), len(chains)
        ids = np.array([s[0] for s in sources], np.uint16)
        pos = np.ascontiguousarray(np.array([s[1] for s in sources], np.float32).reshape(-1, 3))
        ex = extras_to_c(extras)
        out = np.empty(max(1, ns * nc), _RECORD)   # every record is written by the call
        self.ctx._check(lib().omg_early_solve(self.ctx.h, self.id, _p(ids), _p(pos), ns, chains_to_c(chains), nc,
                                              _p(_f3(listener)), _p(ex), len(extras), _p(out)), "omg_early_solve")
        return out[:ns * nc].reshape(ns, nc)
