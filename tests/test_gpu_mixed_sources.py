"""A few rays of a long source that start otherwise than the rest: outcomes and
histories are the oracle's, and the queries counted are those of its paths."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['fp32', 'fp64'])
@pytest.mark.parametrize('history,n', [(False, 40000), (True, 40000), (False, 150000)])
def test_few_rays_with_a_collider(precision, history, n):
    import ehss_b200 as eb
    from ehss_b200 import workloads as W
    rows = np.array([1, 777, 20011, n - 2])
    c, r, _ = W.globule(200, 5)
    src = O.external_source(c, r, 18, 5)
    o, d = src['origins'][:n].copy(), src['directions'][:n].copy()
    tree = O.StaticTree(c, r, 4)
    last, bounces = np.full(n, -1), np.zeros(n, dtype=np.int64)
    first = tree.trace(o[rows], d[rows], cap=8, record=True)
    last[rows] = np.where(first['bounces'] > 0, first['collider_ids'][:, 0], 7)
    bounces[rows[::2]] = 1
    prep = eb.PreparedStaticGPUEHSS(eb.Spheres(c, r, deduplicate=False), precision=precision)
    source = eb.EHSSSource(o, d, d, np.ones(n), last, bounces, 'test')
    got = prep.engine.trace(source, 8, record_history=history)
    ref = tree.trace(o, d, last, bounces, cap=8, record=history, threads=O.host_cores())
    for f in ('positions', 'outgoing', 'escaped', 'unresolved', 'bounces') + (('collider_ids',) if history else ()):
        np.testing.assert_array_equal(getattr(got, f), ref[f], err_msg=f)
    assert got.metrics['queries'] == int((ref['bounces'] - bounces).sum()) + n
    source.last_atom[777] = 200
    with pytest.raises(ValueError, match='identity'):
        prep.engine.trace(source, 8)


@pytest.mark.parametrize('n', [40000, 150000])
def test_few_rays_with_an_owner(n):
    from types import SimpleNamespace
    import ehss_b200 as eb
    from ehss_b200 import workloads as W
    rows = np.array([1, 777, 20011, n - 2])
    c, r, _ = W.globule(200, 5)
    src = O.external_source(c, r, 18, 5)
    o, d = src['origins'][:n].copy(), src['directions'][:n].copy()
    owners = np.full(n, -1)
    owners[rows] = [0, 50, 100, 199]
    index = eb.SphereIndex(eb.Spheres(c, r, deduplicate=False))
    blocked, box, sphere = index.query(SimpleNamespace(origins=o, directions=d, owners=owners))
    np.testing.assert_array_equal(blocked, O.PATree(c, r, 8).query(o, d, owners)[0])
    # counters are those of the rays as they are: the sum of two calls, one of those rays alone
    parts = [index.query(SimpleNamespace(origins=o[k], directions=d[k], owners=owners[k])) for k in
             (rows, np.setdiff1d(np.arange(n), rows))]
    assert (box, sphere) == (parts[0][1] + parts[1][1], parts[0][2] + parts[1][2])
