"""Explicit rays at the edges of the trace kernel's refill and of its copies
to the host: ray counts around a warp, a run of results and a full grid;
page-locked, pageable and device-resident callers; sources whose first and
last rays start without a collider while others do not; origins beyond the
FP32 bounds.  Outcomes are FP64 in the reference's operation order, so every
comparison with the oracle is for equality."""
import ctypes as ct

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(n, atoms, seed, far=False):
    from ehss_b200 import workloads as W
    c, r, _ = W.globule(atoms, seed)
    src = O.external_source(c, r, max(1, (n - 1).bit_length()), seed)
    o, d = src['origins'][:n].copy(), src['directions'][:n].copy()
    if far:
        o[::3] -= 900. * d[::3]
    return c, r, o, d


def _source(o, d, last=None, bounces=None, pinned=False):
    import torch
    import ehss_b200 as eb
    n = len(o)
    if pinned:
        def keep(a):
            t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
            t.numpy()[...] = a
            return t.numpy()
        o, d = keep(o), keep(d)
    last = np.full(n, -1) if last is None else last
    bounces = np.zeros(n, dtype=np.int64) if bounces is None else bounces
    return eb.EHSSSource(o, d, d, np.ones(n), last, bounces, 'test')


def _equal(got, ref, history=False):
    for f in ('positions', 'outgoing', 'escaped', 'unresolved', 'bounces') + (('collider_ids',) if history else ()):
        np.testing.assert_array_equal(getattr(got, f), ref[f], err_msg=f)


@pytest.mark.parametrize('precision', ['fp32', 'fp64'])
@pytest.mark.parametrize('n,atoms,pinned,far', [
    (1, 3, True, False), (31, 40, False, False), (33, 40, True, False), (65, 300, False, True), (4097, 300, True, True),
    (30000, 300, True, False), (150001, 60, True, False)])
def test_ray_counts_equal_the_oracle(precision, n, atoms, pinned, far):
    import ehss_b200 as eb
    c, r, o, d = _case(n, atoms, 3, far)
    prep = eb.PreparedStaticGPUEHSS(eb.Spheres(c, r, deduplicate=False), precision=precision)
    ref = O.StaticTree(c, r, 4).trace(o, d, cap=16, threads=O.host_cores())
    _equal(prep.engine.trace(_source(o, d, pinned=pinned), 16), ref)


@pytest.mark.parametrize('history', [False, True])
def test_mixed_initial_states(history):
    import ehss_b200 as eb
    c, r, o, d = _case(2000, 200, 5)
    prep = eb.PreparedStaticGPUEHSS(eb.Spheres(c, r, deduplicate=False))
    tree = O.StaticTree(c, r, 4)
    first = tree.trace(o, d, cap=8, record=True)
    last, bounces = np.full(2000, -1), np.zeros(2000, dtype=np.int64)
    on = np.flatnonzero(first['bounces'] > 0)[:600]
    on = on[(on > 0) & (on < 1999)]                       # the ends start without a collider
    last[on] = first['collider_ids'][on, 0]
    bounces[on[::2]] = 1
    ref = tree.trace(o, d, last, bounces, cap=8, record=history)
    _equal(prep.engine.trace(_source(o, d, last, bounces), 8, record_history=history), ref, history)
    bad = last.copy()
    bad[700] = 200
    with pytest.raises(ValueError, match='identity'):
        prep.engine.trace(_source(o, d, bad, np.zeros(2000, dtype=np.int64)), 8)
    two = np.zeros(2000, dtype=np.int64)
    two[700] = 2
    with pytest.raises(ValueError, match='initial collision'):
        prep.engine.trace(_source(o, d, np.where(np.arange(2000) == 700, 3, -1), two), 8)
    short = _source(o, d)
    short.origins = short.origins[:1999]
    with pytest.raises(ValueError):
        prep.engine.trace(short, 8)


@pytest.mark.parametrize('n', [1, 40, 3000, 200000])
def test_device_arrays_in_place_equal_the_host_call(n):
    import torch
    import ehss_b200 as eb
    from ehss_b200 import _lib
    c, r, o, d = _case(n, 120, 7)
    prep = eb.PreparedStaticGPUEHSS(eb.Spheres(c, r, deduplicate=False))
    got = prep.engine.trace(_source(o, d), 32)
    P, D = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    last, b = torch.full((n,), -1, device='cuda'), torch.zeros(n, dtype=torch.int64, device='cuda')
    esc, unres = (torch.full((n,), 7, dtype=torch.uint8, device='cuda') for _ in range(2))
    stats = torch.zeros(_lib.NSTATS, dtype=torch.int64, device='cuda')
    _lib.check(_lib.load().ehss_trace(prep.scene.ptr, n, 32, 1, P.data_ptr(), D.data_ptr(), last.data_ptr(), b.data_ptr(),
                                      esc.data_ptr(), unres.data_ptr(), None, stats.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream))
    _equal(got, dict(positions=P.cpu().numpy(), outgoing=D.cpu().numpy(), escaped=esc.cpu().numpy().astype(bool),
                     unresolved=unres.cpu().numpy().astype(bool), bounces=b.cpu().numpy()))
    assert int(stats[_lib.STAT_QUERIES]) == got.metrics['queries'] and int(stats[_lib.STAT_ERRORS]) == 0


def test_host_call_refuses_pageable_memory():
    import torch
    import ehss_b200 as eb
    from ehss_b200 import _lib
    c, r, o, d = _case(64, 40, 9)
    scene = eb.Scene(c, r)
    wb = ct.c_uint64()
    lib = _lib.load()
    _lib.check(lib.ehss_trace_host_workspace_bytes(64, ct.byref(wb)))
    ws = torch.empty(wb.value, dtype=torch.uint8, device='cuda')
    pin = torch.empty(64 * 58 + 64, dtype=torch.uint8, pin_memory=True)
    p = pin.data_ptr()
    out = (p, p + 1536, p + 3072, p + 3584, p + 3648, None, p + 3712, ws.data_ptr())
    args = (scene.ptr, 64, 8, 1, o.ctypes.data, d.ctypes.data, None, None) + out
    assert lib.ehss_trace_host(*args, wb.value, None) == 1          # EHSS_ERR_VALUE
    assert b'page-locked' in lib.ehss_last_error()
    dev = torch.from_numpy(np.stack([o, d])).cuda()
    ok = (scene.ptr, 64, 8, 1, dev[0].data_ptr(), dev[1].data_ptr(), None, None) + out
    assert lib.ehss_trace_host(*ok, wb.value - 1, None) != 0        # one byte short
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.ehss_trace_host(*ok, wb.value, stream) == 0
    torch.cuda.synchronize()
    ref = O.StaticTree(c, r, 4).trace(o, d, cap=8)
    assert np.array_equal(pin[:1536].numpy().view(np.float64).reshape(64, 3), ref['positions'])


@pytest.mark.parametrize('n,pinned', [(1, False), (33, True), (5000, True)])
def test_any_hit_owners(n, pinned):
    import ehss_b200 as eb
    c, r, o, d = _case(n, 80, 11, far=True)
    index, tree = eb.SphereIndex(eb.Spheres(c, r, deduplicate=False)), O.PATree(c, r, 8)
    rng = np.random.default_rng(2)
    for owners in (np.full(n, -1), np.where(rng.random(n) < .3, rng.integers(0, 80, n), -1)):
        if n > 2:
            owners[0] = owners[-1] = -1
        src = _source(o, d, pinned=pinned)
        src.owners = owners
        blocked, box, sphere = index.query(src)
        assert blocked.dtype == bool and box + sphere > 0      # far origins test every atom and no box
        np.testing.assert_array_equal(blocked, tree.query(o, d, owners)[0])


@pytest.mark.parametrize('scale', [1. - 3e-12, 1. + 1e-6, .5, 3.])
def test_fp64_directions_off_unit_length(scale):
    """The FP64 reject takes unit directions and is switched off for others."""
    import torch
    import ehss_b200 as eb
    from ehss_b200 import _lib
    c, r, o, d = _case(3000, 150, 13)
    d = d * scale
    scene = eb.Scene(c, r)
    ref = O.trace_flat(c, r, o, d, cap=16)
    P, D = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    last, b = torch.full((3000,), -1, device='cuda'), torch.zeros(3000, dtype=torch.int64, device='cuda')
    esc, unres = (torch.zeros(3000, dtype=torch.uint8, device='cuda') for _ in range(2))
    _lib.check(_lib.load().ehss_trace(scene.ptr, 3000, 16, 0, P.data_ptr(), D.data_ptr(), last.data_ptr(), b.data_ptr(),
                                      esc.data_ptr(), unres.data_ptr(), None, None, torch.cuda.current_stream().cuda_stream))
    for got, f in ((P, 'positions'), (D, 'outgoing'), (b, 'bounces'), (esc.bool(), 'escaped')):
        np.testing.assert_array_equal(got.cpu().numpy(), ref[f], err_msg=f)


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('atoms,log2,exterior', [(1, 12, False), (3, 10, True), (300, 13, True), (2000, 12, False)])
def test_pa_of_traced_blocks_equals_the_any_hit_query(precision, atoms, log2, exterior):
    import ehss_b200 as eb
    from ehss_b200 import _lib, workloads as W
    from ehss_b200.blocks import BlockJob, BlockPlan
    c, r = (np.zeros((1, 3)), np.array([2.7])) if atoms == 1 else W.globule(atoms, 17)[:2]
    scene = eb.Scene(c, r, exterior=exterior)
    kinds = ((True, True), (False, True), (True, False))
    plan = BlockPlan([BlockJob(scene, log2, 5 + s, cap=32, precision=precision, ehss=e, pa=p) for s in range(3) for e, p in kinds])
    plan.enqueue()
    out = plan.collect()
    for s in range(3):
        both, only_pa, only_ehss = out[3 * s:3 * s + 3]
        assert both['pa_blocked_rays'] == only_pa['pa_blocked_rays'] > 0
        assert both['ehss_angstrom2'] == only_ehss['ehss_angstrom2']
        assert both['collision_histogram'] == only_ehss['collision_histogram']
    # the instance without the any-hit query reports a block that asks for it
    wrong = BlockPlan([BlockJob(scene, log2, 5, precision=precision, pa=True)])
    wrong.launch.options |= _lib.LAUNCH_NO_PA
    wrong.enqueue()
    with pytest.raises(_lib.EHSSDeviceError):
        wrong.collect()
