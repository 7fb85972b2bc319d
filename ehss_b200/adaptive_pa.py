"""Adaptive finite-grid PA on the device (ccs_cli.adaptive_pa, ccs_cli.py:142-160).

For each of ``directions`` Sobol(2, seed) directions the atom disks are
projected on a ``grid_size`` x ``grid_size`` midpoint grid and the covered
pixels are counted exactly (libehss_b200: ehss_pa_grid); the PA is the mean of
count * spacing^2 over the directions, as in the reference.
"""
from __future__ import annotations

import ctypes as ct
import time

import numpy as np

from . import _lib
from .device import empty, ptr, stream_handle, torch


def _enqueue_grid(scene, directions, grid_size, seed, xy=None):
    """Enqueue the pixel counts of one (structure, seed); returns the device
    buffer [2, directions] of counts and spacings (8 bytes each, so that both
    come back in one copy)."""
    lib = _lib.load()
    t = torch()
    n_dirs, n = int(directions), int(grid_size)
    wb = ct.c_uint64()
    _lib.check(lib.ehss_pa_grid_workspace_bytes(scene.n_atoms, n_dirs, n, ct.byref(wb)), 'adaptive PA')
    ws = empty(int(wb.value) + 256, t.uint8, scene.device)
    both = empty((2, n_dirs), t.int64, scene.device)
    _lib.check(lib.ehss_pa_grid(scene.ptr, scene.n_atoms, n_dirs, int(seed), n, ptr(both[0]), ptr(both[1]), ptr(xy),
                                (ws.data_ptr() + 255) & ~255, int(wb.value), stream_handle(scene.device)),
               'adaptive PA')
    return both


def _read_grid(both):
    host = both.cpu().numpy()
    return host[0], host[1].view(np.float64)


def grid_counts(scene, directions, grid_size, seed, with_xy=False):
    """Per-direction covered-pixel counts, pixel spacings (and projections)."""
    xy = empty((int(directions), scene.n_atoms, 2), torch().float64, scene.device) if with_xy else None
    out = _read_grid(_enqueue_grid(scene, directions, grid_size, seed, xy))
    return out + ((xy.cpu().numpy(),) if with_xy else ())


def adaptive_pa(spheres, directions, grid_size, seed, scene=None):
    from .engine import Scene
    tick = time.perf_counter()
    scene = scene or Scene(spheres.centers, spheres.radii)
    setup_s = time.perf_counter() - tick
    return adaptive_pa_runs([(scene, seed)], directions, grid_size, setup_s)[0]


def adaptive_pa_runs(items, directions, grid_size, setup_s=0.):
    """``adaptive_pa`` of many (scene, seed) pairs: every pair is enqueued
    before the first count is read, so the device does not wait for the host
    between them; query_s is each pair's share."""
    tick = time.perf_counter()
    queued = [_enqueue_grid(scene, directions, grid_size, seed) for scene, seed in items]
    found = [_read_grid(both) for both in queued]
    query_s = (time.perf_counter() - tick) / len(items)
    out = []
    for counts, spacing in found:
        tick = time.perf_counter()
        value = float(np.mean([float(c) * float(sp) ** 2 for c, sp in zip(counts, spacing)]))
        out.append(dict(pa_angstrom2=value, source_s=0., projection_s=setup_s, query_s=query_s,
                        readout_s=time.perf_counter() - tick))
    return out
