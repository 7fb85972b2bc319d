"""Directions that are not of unit length: explicit rays in both precisions
equal the oracle's all-atom search."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rays(atoms, n, seed):
    from ehss_b200 import workloads as W
    c, r, _ = W.globule(atoms, seed)
    src = O.external_source(c, r, (n - 1).bit_length(), seed)
    return c, r, src['origins'][:n].copy(), src['directions'][:n].copy()


def _trace(c, r, o, d, cap, precision):
    import torch
    import ehss_b200 as eb
    from ehss_b200 import _lib
    n = len(o)
    scene = eb.Scene(c, r)
    P, D = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    last, b = torch.full((n,), -1, device='cuda'), torch.zeros(n, dtype=torch.int64, device='cuda')
    esc, unres = (torch.zeros(n, dtype=torch.uint8, device='cuda') for _ in range(2))
    stats = torch.zeros(_lib.NSTATS, dtype=torch.int64, device='cuda')
    _lib.check(_lib.load().ehss_trace(scene.ptr, n, cap, precision, P.data_ptr(), D.data_ptr(), last.data_ptr(), b.data_ptr(),
                                      esc.data_ptr(), unres.data_ptr(), None, stats.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream))
    out = dict(positions=P, outgoing=D, bounces=b, escaped=esc.bool(), unresolved=unres.bool())
    return {f: a.cpu().numpy() for f, a in out.items()}, stats.cpu().numpy()


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('scale', [1e-5, 1e-3, 1. - 1e-7, 1. + 1e-6, 40., 1e3, 1e5])
def test_explicit_rays_equal_the_oracle(scale, precision):
    c, r, o, d = _rays(400, 6000, 13)
    d = d * scale
    got, stats = _trace(c, r, o, d, 16, precision)
    assert stats[6] == 0
    ref = O.trace_flat(c, r, o, d, cap=16)
    for f in ('positions', 'outgoing', 'bounces', 'escaped', 'unresolved'):
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
