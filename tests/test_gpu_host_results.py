"""Explicit rays whose results the kernel writes to page-locked host memory:
they equal the results in device memory, run after run, also where several warps
finish one run of rays; and arrays off their elements' alignment are copied."""
import ctypes as ct

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _source(o, d):
    import ehss_b200 as eb
    n = len(o)
    return eb.EHSSSource(o, d, d, np.ones(n), np.full(n, -1), np.zeros(n, dtype=np.int64), 'test')


@pytest.mark.parametrize('atoms,n', [(3, 300000), (300, 60001)])
def test_every_run_of_results_reaches_the_host(atoms, n):
    import torch
    import ehss_b200 as eb
    from ehss_b200 import _lib, workloads as W
    c, r = W.triatomic()[:2] if atoms == 3 else W.globule(atoms, 5)[:2]
    src = O.external_source(c, r, (n - 1).bit_length(), 5)
    o, d = src['origins'][:n].copy(), src['directions'][:n].copy()
    prep = eb.PreparedStaticGPUEHSS(eb.Spheres(c, r, deduplicate=False))
    P, D = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    last, b = torch.full((n,), -1, device='cuda'), torch.zeros(n, dtype=torch.int64, device='cuda')
    esc, unres = (torch.zeros(n, dtype=torch.uint8, device='cuda') for _ in range(2))
    _lib.check(_lib.load().ehss_trace(prep.scene.ptr, n, 32, 1, P.data_ptr(), D.data_ptr(), last.data_ptr(), b.data_ptr(),
                                      esc.data_ptr(), unres.data_ptr(), None, None, torch.cuda.current_stream().cuda_stream))
    want = [a.cpu().numpy() for a in (P, D, b, esc.bool(), unres.bool())]
    source = _source(_pinned(o), _pinned(d))
    for _ in range(10):
        got = prep.engine.trace(source, 32)
        for a, w in zip((got.positions, got.outgoing, got.bounces, got.escaped, got.unresolved), want):
            assert np.array_equal(a, w)


def _off_by(a, k):
    """The array in page-locked memory, k bytes behind an aligned address."""
    import torch
    raw = torch.empty(a.nbytes + 8, dtype=torch.uint8, pin_memory=True).numpy()
    out = np.frombuffer(raw, dtype=a.dtype, count=a.size, offset=k).reshape(a.shape)
    out[...] = a
    return out


def test_misaligned_page_locked_arrays():
    import torch
    import ehss_b200 as eb
    from ehss_b200 import _lib, workloads as W
    c, r, _ = W.globule(100, 7)
    src = O.external_source(c, r, 10, 7)
    o, d = src['origins'], src['directions']
    ref = O.StaticTree(c, r, 4).trace(o, d, cap=8)
    prep = eb.PreparedStaticGPUEHSS(eb.Spheres(c, r, deduplicate=False))
    source = _source(o, d)
    source.origins, source.directions = _off_by(o, 4), _off_by(d, 1)
    assert not source.origins.flags.aligned
    got = prep.engine.trace(source, 8)
    for f in ('positions', 'outgoing', 'escaped', 'unresolved', 'bounces'):
        assert np.array_equal(getattr(got, f), ref[f])
    source.owners = _off_by(np.full(1024, -1), 4)
    blocked = eb.SphereIndex(eb.Spheres(c, r, deduplicate=False)).query(source)[0]
    assert np.array_equal(blocked, O.PATree(c, r, 8).query(o, d, np.full(1024, -1))[0])
    # the library refuses such addresses instead of reading them
    lib = _lib.load()
    wb = ct.c_uint64()
    _lib.check(lib.ehss_trace_host_workspace_bytes(1024, ct.byref(wb)))
    ws = torch.empty(wb.value, dtype=torch.uint8, device='cuda')
    out = torch.empty(1024 * 58 + 64, dtype=torch.uint8, pin_memory=True)
    p = out.data_ptr()
    rest = (p, p + 24576, p + 49152, p + 57344, p + 58368, None, p + 59392, ws.data_ptr(), wb.value, None)
    good = _pinned(o).ctypes.data, _pinned(d).ctypes.data
    for ray in ((source.origins.ctypes.data, good[1]), (good[0], source.directions.ctypes.data)):
        assert lib.ehss_trace_host(prep.scene.ptr, 1024, 8, 1, *ray, None, None, *rest) == _lib.ERR_VALUE
        assert lib.ehss_pa_anyhit(prep.scene.ptr, 1024, *ray, None, p, None, None) == _lib.ERR_VALUE
