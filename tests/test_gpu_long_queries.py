"""Any-hit queries around the number of rays from which page-locked origins are
copied to the device ahead: hits, and counters as from parts of the rays."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('pinned', [False, True])
@pytest.mark.parametrize('n', [65536, 65537, 131075])
def test_long_queries(n, pinned):
    from types import SimpleNamespace
    import torch
    import ehss_b200 as eb
    from ehss_b200 import workloads as W
    c, r, _ = W.globule(90, 3)
    src = O.external_source(c, r, 18, 3)
    o, d = src['origins'][:n].copy(), src['directions'][:n].copy()
    index, tree = eb.SphereIndex(eb.Spheres(c, r, deduplicate=False)), O.PATree(c, r, 8)
    po, pd = o, d
    if pinned:
        po, pd = (torch.empty(a.shape, dtype=torch.float64, pin_memory=True).numpy() for a in (o, d))
        po[...], pd[...] = o, d
    plain = np.full(n, -1)
    late, early, every = plain.copy(), plain.copy(), np.arange(n) % 91 - 1
    late[n - 3], early[2] = 40, 41
    for name, owners in (('plain', plain), ('late', late), ('early', early), ('every', every)):
        blocked, box, sphere = index.query(SimpleNamespace(origins=po, directions=pd, owners=owners))
        np.testing.assert_array_equal(blocked, tree.query(o, d, owners)[0], err_msg=name)
        parts = [index.query(SimpleNamespace(origins=o[k], directions=d[k], owners=owners[k]))
                 for k in (slice(0, 30000), slice(30000, None))]
        assert (box, sphere) == tuple(sum(p[i] for p in parts) for i in (1, 2)), name
