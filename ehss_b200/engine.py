"""The reference's EHSS / PA plugin objects, backed by the CUDA library.

Drop-in counterparts of (paths relative to the reference project root):

* ``PreparedStaticGPUEHSS``  PreparedStaticCPUEHSS  src/support_exchange_transport/ehss_static.py:62-101
* ``GPUEHSSTransport.trace`` CPUEHSSTransport.trace ehss_cpu.py:118-142
* ``external_source``        ehss_state.external_source ehss_state.py:42-53
* ``SphereIndex.query``      pa_spatial.SphereIndex.query pa_spatial.py:157-164

Arguments, validation and error types follow the reference (ValueError for
bad caps, identities, groups).  Geometry lives on the device in a ``Scene``;
the host arrays of a source/result are numpy, as in the reference.
"""
from __future__ import annotations

import ctypes as ct
import time
from types import SimpleNamespace

import numpy as np

from . import _lib
from .device import empty, ptr, require_cuda, stream_handle, to_device, torch
from .state import EHSSResult, EHSSSource, Spheres

PRECISIONS = {'fp64': _lib.PREC_FP64, 'fp32': _lib.PREC_FP32}


def _precision(p):
    if isinstance(p, str):
        if p not in PRECISIONS:
            raise ValueError(f'precision must be one of {sorted(PRECISIONS)}')
        return PRECISIONS[p]
    if p not in (0, 1):
        raise ValueError('precision must be 0 (fp64) or 1 (fp32)')
    return int(p)


def _aligned_buffer(nbytes, device):
    """uint8 device buffer with a 256-byte aligned start; returns (tensor, address)."""
    buf = empty(int(nbytes) + 256, torch().uint8, device)
    addr = (buf.data_ptr() + 255) & ~255
    return buf, addr


class Scene:
    """One structure resident on the device: atoms plus the LBVH.

    Owns its coordinates (a device copy), so later changes to the caller's
    arrays cannot invalidate it, like the reference's prepared scene
    (ehss_static.py:68-69).
    """

    def __init__(self, centers, radii, leaf_size=_lib.DEFAULT_LEAF, device=None, exterior=False):
        lib = _lib.load()
        self.device = require_cuda(device)
        c = np.ascontiguousarray(centers, dtype=np.float64)
        r = np.ascontiguousarray(radii, dtype=np.float64)
        if c.ndim != 2 or c.shape[1] != 3 or r.shape != (len(c),) or len(c) == 0:
            raise ValueError('Expected nonempty centers (N,3) and radii (N,).')
        self.n_atoms = len(r)
        self._radii = r.copy()
        self.leaf_size = int(leaf_size)
        sb, wb = ct.c_uint64(), ct.c_uint64()
        _lib.check(lib.ehss_scene_bytes(self.n_atoms, self.leaf_size, ct.byref(sb), ct.byref(wb)), 'scene size')
        stream = stream_handle(self.device)
        self._buf, self.ptr = _aligned_buffer(sb.value, self.device)
        self.nbytes = sb.value
        xyz_d = to_device(c, np.float64, self.device)
        r_d = to_device(r, np.float64, self.device)
        ws, ws_addr = _aligned_buffer(wb.value, self.device)
        if exterior:
            # buried atoms left out of the tree: valid for the fused block trace only
            _lib.check(lib.ehss_scenes_build_ex(1, (ct.c_void_p * 1)(xyz_d.data_ptr()),
                                                (ct.c_void_p * 1)(r_d.data_ptr()), (ct.c_int64 * 1)(self.n_atoms),
                                                self.leaf_size, (ct.c_void_p * 1)(self.ptr), (ct.c_uint64 * 1)(sb.value),
                                                ws_addr, wb.value, _lib.BUILD_EXTERIOR, stream), 'scene build')
        else:
            _lib.check(lib.ehss_scene_build(self.n_atoms, xyz_d.data_ptr(), r_d.data_ptr(), self.leaf_size, self.ptr,
                                            sb.value, ws_addr, wb.value, stream), 'scene build')
        self._read_info('scene build')   # synchronises
        del ws, xyz_d, r_d

    def _read_info(self, what):
        info = _lib.SceneInfo()
        _lib.check(_lib.load().ehss_scene_info_get(self.ptr, ct.byref(info), stream_handle(self.device)), what)
        self.info = info
        self.exterior = bool(info.exterior)
        self.n_active = int(info.n_active)
        self.center = np.array(info.center[:])
        self.radius = float(info.radius)

    def refit(self, centers, radii=None):
        """New coordinates (and optionally radii) for the same atoms, tree
        topology kept (ehss_scenes_refit; SphereIndex.refit, pa_spatial.py:166-170).
        The header and atom records become those of a build of the new
        coordinates and every node box the union of its atoms' boxes, so
        traces return what a rebuilt scene returns.  Full scenes only."""
        if self.exterior:
            raise ValueError('an exterior scene cannot be refit: its tree holds the atoms exposed in the built coordinates')
        c = np.ascontiguousarray(centers, dtype=np.float64)
        r = self._radii if radii is None else np.ascontiguousarray(radii, dtype=np.float64)
        if c.shape != (self.n_atoms, 3) or r.shape != (self.n_atoms,):
            raise ValueError('Refit requires fixed primitive identities.')
        if not np.isfinite(c).all() or not np.isfinite(r).all() or np.any(r <= 0):
            raise ValueError('Finite centers (N,3) and positive finite radii required.')
        lib = _lib.load()
        sb, wb = ct.c_uint64(), ct.c_uint64()
        _lib.check(lib.ehss_scene_bytes(self.n_atoms, self.leaf_size, ct.byref(sb), ct.byref(wb)), 'scene size')
        xyz_d = to_device(c, np.float64, self.device)
        r_d = to_device(r, np.float64, self.device)
        ws, ws_addr = _aligned_buffer(wb.value, self.device)
        _lib.check(lib.ehss_scenes_refit(1, (ct.c_void_p * 1)(xyz_d.data_ptr()), (ct.c_void_p * 1)(r_d.data_ptr()),
                                         (ct.c_int64 * 1)(self.n_atoms), (ct.c_void_p * 1)(self.ptr), ws_addr,
                                         wb.value, stream_handle(self.device)), 'scene refit')
        self._read_info('scene refit')   # synchronises
        del ws, xyz_d, r_d
        self._radii = r.copy()
        return self

    @classmethod
    def from_spheres(cls, spheres, leaf_size=_lib.DEFAULT_LEAF, device=None):
        return cls(spheres.centers, spheres.radii, leaf_size, device)

    def source_rays(self, power, seed, first=0, n=None):
        """Device impact-disk rays (origins, directions) as torch tensors."""
        lib = _lib.load()
        total = 1 << int(power)
        n = total - first if n is None else int(n)
        o = empty((n, 3), torch().float64, self.device)
        d = empty((n, 3), torch().float64, self.device)
        _lib.check(lib.ehss_source_rays(self.ptr, int(power), int(seed), int(first), n, ptr(o), ptr(d),
                                        stream_handle(self.device)), 'source')
        return o, d


def _check_seed(seed):
    if isinstance(seed, (bool, np.bool_)) or not isinstance(seed, (int, np.integer)) or not 0 <= int(seed) < 2 ** 64:
        raise ValueError('seed must be an integer in 0..2**64-1')
    return int(seed)


def external_source(spheres, power, seed, scene=None):
    """Impact-disk source generated on the device from bit-exact Sobol points.

    Same contract as the reference's external_source: 2**power rays, weight
    pi R^2 / n each, no initial collider.  The ray arrays are numpy arrays
    over page-locked host memory, which a trace reads where they lie.
    """
    power = int(power)
    if not 0 <= power <= 30:
        raise ValueError('power must be 0..30')
    seed = _check_seed(seed)
    scene = scene or Scene.from_spheres(spheres)
    o, d = scene.source_rays(power, seed)
    t = torch()
    # page-locked host arrays: the copy back runs as DMA, and a later trace reads them in place
    host = t.empty((3, o.shape[0], 3), dtype=t.float64, pin_memory=True)
    host[0].copy_(o, non_blocking=True)
    host[1].copy_(d, non_blocking=True)
    host[2].copy_(d, non_blocking=True)
    t.cuda.current_stream(scene.device).synchronize()
    origins, directions, incoming = (a.numpy() for a in host)
    n = len(origins)
    R = scene.radius
    return EHSSSource(origins, directions, incoming, np.full(n, np.pi * R * R / n),
                      np.full(n, -1), np.zeros(n, dtype=np.int64), "external impact disk")


def _host_array(a, dtype):
    """``a`` as a C-contiguous array whose elements lie on their own alignment,
    as kernels need them: itself where it is one, else a copy."""
    a = np.ascontiguousarray(a, dtype=dtype)
    return a if a.flags.aligned else a.copy()


def _per_ray(a, dtype, shape):
    """The entries of ``shape[0]`` rays, as _host_array: longer arrays are read
    up to there, and one entry for all rays is repeated."""
    a = np.asarray(a)
    if a.shape != shape:
        a = np.broadcast_to(a[:shape[0]], shape)
    return _host_array(a, dtype)


def _rows(a, dtype, n, width):
    """The first n rows of ``width`` entries, as _host_array."""
    a = _host_array(np.atleast_1d(a), dtype)
    if len(a) < n or a.size != width * len(a):
        raise ValueError('One origin, direction and owner per ray required')
    return a.reshape(-1, width)[:n]


def _reachable(a, device, hold):
    """Address of a contiguous host array that kernels can read where it lies
    (page-locked memory), or of a device copy; ``hold`` keeps it alive."""
    host = torch().from_numpy(a)
    t = host if host.is_pinned() else host.to(device)
    hold.append(t)
    return t.data_ptr()


def _page_locked(device, sizes):
    """uint8 views of one new page-locked buffer, one per size, each on a 64-byte boundary."""
    starts, total = [], 0
    for n in sizes:
        starts.append(total)
        total += -(-n // 64) * 64
    buf = torch().empty(max(total, 1), dtype=torch().uint8, pin_memory=True)
    host = buf.numpy()
    return buf, [host[s:s + n] for s, n in zip(starts, sizes)]


# Rays from which on a pass over an array of them (65,536: 8 us where they are in a cache, 37 where not; 262,144: 36 and
# 132) is made while the device works.
_LONG = 65536
# fractions spread evenly over [0, 1), without a period that an array could share
_SPREAD = np.arange(1024) * ((5 ** .5 - 1) / 2) % 1


def _all(a, value):
    """Whether every entry of an int64 array is ``value``, -1 or 0."""
    return len(a) > 0 and (np.bitwise_and if value else np.bitwise_or).reduce(a) == value


def _seems_all(a, value):
    """The same of a thousand entries (5 us)."""
    return _all(a[(_SPREAD * len(a)).astype(np.int64)], value)


def _unless(a, value):
    """None for an int64 array whose every entry is ``value``, -1 or 0 (the rule), else the
    array.  One pass, left out where a sample of a long array shows that it is not."""
    return None if (len(a) <= _LONG or _seems_all(a, value)) and _all(a, value) else a


# Bytes of an int64 array up to which a copy in page-locked memory, read by the kernel over the link, costs less than
# a copy to the device (65,536 rays: 17 us and 10 over the link against 53; 262,144: 133 and 38 against 154).
_STAGE_BYTES = 1 << 20


def _ahead(a, device, hold):
    """Address of a device copy of a long page-locked array, which crosses the link
    while the host reads others through (_unless; 262,144 traced rays of 2000 atoms:
    911 us, read where they lie after that 1000); None for any other array."""
    host = torch().from_numpy(a)
    if len(a) <= _LONG or not host.is_pinned():
        return None
    with torch().cuda.device(device):
        hold.append(host.to(device, non_blocking=True))
    return hold[-1].data_ptr()


def _stage_bytes(a):
    return 0 if a is None or a.nbytes > _STAGE_BYTES else a.nbytes


def _staged(a, space, device, hold):
    """Address of an int64 array that kernels can read: as _reachable, but a short
    array is copied into ``space`` (page-locked, _stage_bytes)."""
    if a is None:
        return None
    if not len(space) or torch().from_numpy(a).is_pinned():
        return _reachable(a, device, hold)
    space.view(np.int64)[...] = a
    return space.ctypes.data


class GPUEHSSTransport:
    """EHSS tracer on one prepared scene (CPUEHSSTransport.trace contract).

    ``trace`` takes and returns host arrays, as the reference does.  One
    launch reads the rays from page-locked host memory (rays in pageable
    arrays, and more than 65,536 of them, are copied to the device first),
    traces them and writes the results into a page-locked buffer whose parts
    become the returned arrays.
    """

    def __init__(self, scene, precision='fp32', threads=1):
        if getattr(scene, 'exterior', False):
            raise ValueError('an exterior scene holds only atoms reachable from outside; trace needs a full scene')
        self.scene = scene
        self.precision = _precision(precision)
        self.threads = threads

    def trace(self, source, cap=64, record_history=False):
        if type(cap) is not int or cap < 1 or cap > np.iinfo(np.int32).max:
            raise ValueError('Positive cap and zero/one initial collision required')
        start = time.perf_counter()
        n = len(source.weights)
        try:
            origins, directions = (_per_ray(a, np.float64, (n, 3)) for a in (source.origins, source.directions))
            last, bounces = (_per_ray(a, np.int64, (n,)) for a in (source.last_atom, source.initial_bounces))
        except (ValueError, IndexError):
            raise ValueError('One origin, direction, initial identity and bounce count per weight required') from None
        wait = torch().cuda.current_stream(self.scene.device).synchronize
        hold = []
        try:
            ahead = [_ahead(a, self.scene.device, hold) for a in (origins, directions)]
            # a source starts without colliders and collisions as a rule, and then needs neither array
            last, bounces = _unless(last, -1), _unless(bounces, 0)
            if bounces is not None and np.any(source.initial_bounces > 1):
                raise ValueError('Positive cap and zero/one initial collision required')
            if last is not None and (np.any(last < -1) or np.any(last >= self.scene.n_atoms)):
                raise ValueError('Invalid initial physical identity')
            (P, D, b, esc, unres, st), hist_out = self._enqueue(ahead, origins, directions, last, bounces, cap, record_history)
        finally:
            wait()
        if st[_lib.STAT_ERRORS]:
            raise _lib.EHSSDeviceError(f'{int(st[_lib.STAT_ERRORS])} rays reported a bounded device failure')
        history = hist_out.numpy() if record_history else np.full((n, 0), -1, dtype=np.int32)
        return EHSSResult(P, D, esc, unres, b, history, source,
                          dict(query_s=time.perf_counter() - start, sphere_tests=int(st[_lib.STAT_SPHERE]),
                               box_tests=int(st[_lib.STAT_BOX]), queries=int(st[_lib.STAT_QUERIES]),
                               grazing_queries=int(st[_lib.STAT_GRAZING]),
                               fp64_fallback_queries=int(st[_lib.STAT_FALLBACK]),
                               fp64_sphere_tests=int(st[_lib.STAT_FP64]), backend='B200 CUDA',
                               precision='fp64' if self.precision == _lib.PREC_FP64 else 'fp32',
                               threads=self.threads, history_recorded=bool(record_history),
                               response_reuse=False))

    def _enqueue(self, ahead, origins, directions, last, bounces, cap, record_history):
        """Enqueue one trace (no wait); returns the host arrays that it fills."""
        # the scene's device, whichever is the thread's current one: the handle of a default stream names no device
        with torch().cuda.device(self.scene.device):
            return self._launch(ahead, origins, directions, last, bounces, cap, record_history)

    def _launch(self, ahead, origins, directions, last, bounces, cap, record_history):
        lib, t, dev = _lib.load(), torch(), self.scene.device
        n = len(origins)
        hold = []
        rays = [p or _reachable(a, dev, hold) for p, a in zip(ahead, (origins, directions))]
        wb = ct.c_uint64()
        _lib.check(lib.ehss_trace_host_workspace_bytes(n, ct.byref(wb)), 'trace')
        ws = t.empty(wb.value, dtype=t.uint8, device=dev)
        buf, (P, D, b, esc, unres, st, *space) = _page_locked(dev, (24 * n, 24 * n, 8 * n, n, n, 8 * _lib.NSTATS) + tuple(
            map(_stage_bytes, (last, bounces))))
        initial = [_staged(a, v, dev, hold) for a, v in zip((last, bounces), space)]
        hist = t.full((n, cap), -1, dtype=t.int32, device=dev) if record_history else None
        hist_out = t.empty((n, cap), dtype=t.int32, pin_memory=True) if record_history else None
        out = [a.ctypes.data for a in (P, D, b, esc, unres)]
        _lib.check(lib.ehss_trace_host(self.scene.ptr, n, cap, self.precision, *rays, *initial, *out, ptr(hist), st.ctypes.data,
                                       ws.data_ptr(), wb.value, stream_handle(dev)), 'trace')
        if hist is not None:
            hist_out.copy_(hist, non_blocking=True)
        f8 = np.float64
        return (P.view(f8).reshape(n, 3), D.view(f8).reshape(n, 3), b.view(np.int64), esc.view(np.bool_),
                unres.view(np.bool_), st.view(np.uint64)), hist_out


def _check_groups(groups, n):
    g = np.asarray(groups)
    if g.shape != (n,) or not np.issubdtype(g.dtype, np.integer):
        raise ValueError('One integer group per atom required')
    unique = np.unique(g)
    if not np.array_equal(unique, np.arange(len(unique))):
        raise ValueError('Contiguous nonempty groups required')


class PreparedStaticGPUEHSS:
    """Owned geometry for repeated sampling of one unchanged structure.

    ``groups`` and ``threads`` are accepted and validated as in the
    reference; neither affects results (the device LBVH replaces the
    reference's median-split groups, and the GPU replaces worker threads).
    """

    def __init__(self, spheres, groups=None, leaf_size=None, threads=1, boundary='sphere', simplify=False,
                 coverage_depth=4, precision='fp32', device=None):
        # leaf_size bounds the device LBVH leaves (capped at 16); left out, the fast default is used
        if type(threads) is not int or threads < 1:
            raise ValueError('Threads must be a positive integer')
        leaf_size = _lib.DEFAULT_LEAF if leaf_size is None else leaf_size
        if type(leaf_size) is not int or leaf_size < 1:
            raise ValueError('Positive integer leaf size required')
        start = time.perf_counter()
        s = Spheres(spheres.centers, spheres.radii, deduplicate=False)
        if groups is not None:
            _check_groups(groups, len(s.radii))
        scene = Scene.from_spheres(s, leaf_size=min(leaf_size, 16), device=device)
        self.model = SimpleNamespace(spheres=s, scene=scene)
        self.scene = scene
        tick = time.perf_counter()
        from .compact import CompactBoundary
        # incidence boundary, as the reference's prepared engine carries it (ehss_static.py:94)
        self.boundary = CompactBoundary.fit(s, boundary, device=scene.device)
        boundary_s = time.perf_counter() - tick
        self.engine = GPUEHSSTransport(scene, precision=precision, threads=threads)
        self.setup = dict(total_s=time.perf_counter() - start, preparation='static device LBVH',
                          nodes=int(scene.info.n_nodes), depth=int(scene.info.depth), threads=threads,
                          boundary_s=boundary_s)


class SphereIndex:
    """Any-hit PA index (SphereIndex(spheres, kind, leaf_size).query)."""

    def __init__(self, spheres, kind='bvh', leaf_size=None, device=None):
        leaf_size = _lib.DEFAULT_LEAF if leaf_size is None else leaf_size
        if kind not in ('bvh', 'octree') or leaf_size < 1:
            raise ValueError('Valid kind, positive leaf size and nonempty primitives required.')
        self.spheres = spheres
        self.scene = Scene.from_spheres(spheres, leaf_size=min(int(leaf_size), 16), device=device)

    def refit(self, spheres):
        """Same atoms at new positions (SphereIndex.refit, pa_spatial.py:166-170):
        the device tree is refit in place (ehss_scenes_refit)."""
        if len(spheres.radii) != len(self.spheres.radii):
            raise ValueError('Refit requires fixed primitive identities.')
        self.scene.refit(spheres.centers, spheres.radii)
        self.spheres = spheres

    def query(self, source):
        owners = getattr(source, 'owners', None)
        if owners is None:
            owners = source.last_atom
        n = len(source.origins)
        origins, directions = (_rows(a, np.float64, n, 3) for a in (source.origins, source.directions))
        own = _rows(owners, np.int64, n, 1).reshape(-1)
        blocked, st = self._enqueue(origins, directions, own)
        torch().cuda.current_stream(self.scene.device).synchronize()
        if st[_lib.STAT_ERRORS]:
            raise _lib.EHSSDeviceError('PA query reported a bounded device failure')
        # an array of its own: the page-locked buffer serves the next call, also while the caller keeps the result
        return blocked.copy(), int(st[_lib.STAT_BOX]), int(st[_lib.STAT_SPHERE])

    def _enqueue(self, origins, directions, owners):
        """Enqueue one any-hit query (no wait); returns the host arrays that it fills."""
        with torch().cuda.device(self.scene.device):      # as in GPUEHSSTransport._enqueue
            return self._launch(origins, directions, owners)

    def _launch(self, origins, directions, owners):
        lib, t, dev = _lib.load(), torch(), self.scene.device
        n = len(origins)
        hold = []
        # Rays without owners are the rule (_unless); rays that are copied to the device take theirs with them from where
        # that copy costs little more than the look.  The origins are enough to cross the link ahead: the look takes less
        # than those of a trace (200,000 rays: 313 us, with nothing ahead 400).
        P = _ahead(origins, dev, hold)
        if P or n <= 16384 or t.from_numpy(origins).is_pinned():
            owners = _unless(owners, -1)
        P, D = P or _reachable(origins, dev, hold), _reachable(directions, dev, hold)
        buf, (blocked, st, space) = _page_locked(dev, (n, 8 * _lib.NSTATS, _stage_bytes(owners)))
        own = _staged(owners, space, dev, hold)
        stats = t.zeros(_lib.NSTATS, dtype=t.int64, device=dev)
        _lib.check(lib.ehss_pa_anyhit(self.scene.ptr, n, P, D, own, blocked.ctypes.data if n else None, ptr(stats),
                                      stream_handle(dev)), 'PA query')
        t.from_numpy(st.view(np.int64)).copy_(stats, non_blocking=True)
        return blocked.view(np.bool_), st.view(np.int64)
