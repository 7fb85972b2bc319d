"""Host staging and block preparation (no GPU): the native copies, checks,
centres and radii equal numpy's on one thread and on several, and blocks that
share a seed get the enumeration they would get alone."""
import ctypes as ct

import numpy as np
import pytest

from ehss_b200 import _lib


def _stage(structures):
    lib = _lib.load()
    S = len(structures)
    n = np.array([len(r) for _, r in structures], dtype=np.int64)
    N = int(n.sum())
    out = np.full((N, 3), -7.), np.full(N, -7.), np.empty((S, 3)), np.empty(S)
    rc = lib.ehss_stage_structures(S, (ct.c_void_p * S)(*[c.ctypes.data for c, _ in structures]),
                                   (ct.c_void_p * S)(*[r.ctypes.data for _, r in structures]), n.ctypes.data,
                                   *[a.ctypes.data for a in out])
    return rc, out


@pytest.mark.parametrize('sizes', [(1,), (2, 1, 7), (300, 5, 41000), (900,) * 150])
def test_staging_equals_numpy(sizes):
    rng = np.random.default_rng(len(sizes))
    structures = [(rng.normal(scale=20., size=(n, 3)) + 5., rng.uniform(1., 3., n)) for n in sizes]
    rc, (xyz, r, centers, radii) = _stage(structures)
    assert rc == 0
    assert np.array_equal(xyz, np.concatenate([c for c, _ in structures]))
    assert np.array_equal(r, np.concatenate([q for _, q in structures]))
    for k, (c, q) in enumerate(structures):
        center = c.mean(axis=0)
        assert np.array_equal(centers[k], center)
        d = c - center
        assert radii[k] == np.max(np.sqrt((d[:, 0] ** 2 + d[:, 1] ** 2) + d[:, 2] ** 2) + q) * 1.000000001


@pytest.mark.parametrize('value,where', [(np.nan, 'c'), (np.inf, 'c'), (-1., 'r'), (0., 'r'), (np.inf, 'r')])
def test_invalid_input_stages_nothing(value, where):
    structures = [(np.ones((50, 3)) * k, np.ones(50)) for k in range(4)]
    structures[2][0 if where == 'c' else 1].reshape(-1)[17] = value
    rc, (xyz, r, _, _) = _stage(structures)
    assert rc == _lib.ERR_VALUE and np.all(xyz == -7.) and np.all(r == -7.)


def test_blocks_that_share_a_seed_are_prepared_alike():
    lib = _lib.load()
    cases = [(5, 10), (5, 10), (6, 10), (5, 11), (5, 10), (2 ** 40 + 5, 10), (6, 10), (5, 11)]

    def prepare(group):
        blocks = (_lib.Block * len(group))()
        for b, (_, log2) in zip(blocks, group):
            b.scene, b.log2_rays, b.cap, b.precision, b.flags, b.hist_offset = 256, log2, 8, 1, _lib.BLOCK_EHSS, -1
        seeds = (ct.c_uint64 * len(group))(*[s for s, _ in group])
        total = ct.c_int64()
        assert lib.ehss_blocks_prepare(blocks, len(group), seeds, 64, ct.byref(total)) == 0
        return blocks
    together = prepare(cases)
    for b, case in zip(together, cases):
        alone = prepare([case])[0]
        assert bytes(b.basis) == bytes(alone.basis) and bytes(b.base) == bytes(alone.base)
