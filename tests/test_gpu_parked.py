"""Queries that overflow the FP32 walk's two candidate slots are parked and
finished with the FP64 search: structures whose every atom lies five times in
the same place make nearly every hit one.  Outcomes equal the oracle's, and the
FP64 blocks' word for word."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _five(atoms, seed):
    from ehss_b200 import workloads as W
    c, r, _ = W.globule(atoms, seed)
    return np.repeat(c, 5, axis=0), np.repeat(r, 5)


@pytest.mark.parametrize('atoms,cap', [(1, 4), (40, 3), (200, 64)])
def test_explicit_rays(atoms, cap):
    import ehss_b200 as eb
    c, r = _five(atoms, 3)
    src = O.external_source(c, r, 12, 5)
    o, d = src['origins'], src['directions']
    n = len(o)
    prep = eb.PreparedStaticGPUEHSS(eb.Spheres(c, r, deduplicate=False))
    got = prep.engine.trace(eb.EHSSSource(o, d, d, np.ones(n), np.full(n, -1), np.zeros(n, dtype=np.int64), 't'), cap,
                            record_history=True)
    ref = O.StaticTree(c, r, 4).trace(o, d, cap=cap, record=True, threads=O.host_cores())
    for f in ('positions', 'outgoing', 'escaped', 'unresolved', 'bounces', 'collider_ids'):
        np.testing.assert_array_equal(getattr(got, f), ref[f], err_msg=f)
    assert got.metrics['fp64_fallback_queries'] > 0


@pytest.mark.parametrize('exterior', [False, True])
@pytest.mark.parametrize('boundary', [None, 'box'])
@pytest.mark.parametrize('pa', [False, True])
@pytest.mark.parametrize('count', [False, True])
def test_blocks_equal_fp64(exterior, boundary, pa, count):
    from ehss_b200 import _lib
    from ehss_b200.batch import BatchCCS
    structures = [_five(n, n) for n in (3, 60, 200)]
    out = []
    for precision in ('fp32', 'fp64'):
        bc = BatchCCS(structures, [9, 11, 10], [1, 2, 3], repeats=2, cap=6, precision=precision, pa=pa, exterior=exterior,
                      boundary=boundary, launch=dict(count_tests=count))
        bc.upload(); bc.build(); bc.plan.enqueue()
        out.append(bc.plan.collect())
    for a, b in zip(*out):
        assert a['fp64_fallback_queries'] > 0
        for key in ('ehss_angstrom2', 'pa_from_same_rays_angstrom2', 'unresolved_rays', 'escaped_rays', 'collision_histogram',
                    'collision_contribution_angstrom2', 'queries') + (('pa_blocked_rays',) if pa else ()):
            assert a[key] == b[key], key


def test_cap_extension_of_parked_rays():
    from ehss_b200.batch import BatchCCS
    structures = [_five(60, 8), _five(150, 9)]
    runs = []
    for kw in (dict(cap=2, cap_ladder=(4, 64), tail_fraction=0.), dict(cap=64)):
        runs.append(BatchCCS(structures, 12, [5, 6], repeats=2, **kw).run())
    for a, b in zip(*runs):
        assert a['ehss_angstrom2'] == b['ehss_angstrom2']
        for x, y in zip(a['runs'], b['runs']):             # the ladder ends once nothing is unresolved
            top = len(x['collision_histogram'])
            assert x['collision_histogram'] == y['collision_histogram'][:top] and not any(y['collision_histogram'][top:])


@pytest.mark.parametrize('scale', [1e-2, 30.])
def test_structures_far_from_protein_scale(scale):
    """The bounds follow the structure's scale: outcomes equal FP64's on it."""
    import ehss_b200 as eb
    from ehss_b200 import workloads as W
    c, r, _ = W.globule(500, 21)
    c, r = c * scale, r * (scale if scale < 1 else 1.)         # a thousand angstrom across with ordinary atoms
    src = O.external_source(c, r, 13, 2)
    o, d = src['origins'], src['directions']
    n = len(o)
    ref = O.StaticTree(c, r, 4).trace(o, d, cap=32, threads=O.host_cores())
    for precision in ('fp32', 'fp64'):
        prep = eb.PreparedStaticGPUEHSS(eb.Spheres(c, r, deduplicate=False), precision=precision)
        got = prep.engine.trace(eb.EHSSSource(o, d, d, np.ones(n), np.full(n, -1), np.zeros(n, dtype=np.int64), 't'), 32)
        for f in ('positions', 'outgoing', 'escaped', 'unresolved', 'bounces'):
            np.testing.assert_array_equal(getattr(got, f), ref[f], err_msg=f)
