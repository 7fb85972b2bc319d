"""Results of any-hit queries belong to the caller: ordinary writable arrays,
unchanged by later queries."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_results_are_kept():
    from types import SimpleNamespace
    import torch
    import ehss_b200 as eb
    from ehss_b200 import workloads as W
    c, r, _ = W.globule(60, 3)
    src = O.external_source(c, r, 12, 3)
    o, d, owners = src['origins'], src['directions'], np.full(4096, -1)
    index = eb.SphereIndex(eb.Spheres(c, r, deduplicate=False))
    kept = [index.query(SimpleNamespace(origins=o, directions=x, owners=owners))[0] for x in (d, -d, d)]
    for got, x in zip(kept, (d, -d, d)):
        assert got.flags.owndata and got.flags.writeable and got.dtype == bool
        assert not torch.from_numpy(got).is_pinned()
        np.testing.assert_array_equal(got, O.PATree(c, r, 8).query(o, x, owners)[0])
