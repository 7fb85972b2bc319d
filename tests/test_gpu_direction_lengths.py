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


SCALES = [1e-5, .5, 1. - 1e-7, 1. + 3e-12, 1. + 1e-7, 1. + 1e-4, 3., 1e3, 1e7]


@pytest.mark.parametrize('scale', SCALES)
def test_ray_blocks_equal_fp64_and_the_oracle(scale):
    import torch
    import ehss_b200 as eb
    from ehss_b200 import _lib
    from ehss_b200.blocks import BlockJob, BlockPlan
    c, r, o, d = _rays(400, 4096, 17)
    d = d * scale

    class Rays:
        def fill_ray_buffer(self, power, seed, buf):
            buf.copy_(torch.from_numpy(np.concatenate([o.ravel(), d.ravel(), np.ones(4096)])))

        def max_projected_area(self):
            return 4096. * (1. + 1e-9)
    scene = eb.Scene(c, r)
    plan = BlockPlan([BlockJob(scene, 12, 0, cap=16, precision=p, pa=True, boundary=Rays())
                      for p in (_lib.PREC_FP32, _lib.PREC_FP64)])
    plan.run()
    f32, f64 = plan.collect()
    for key in ('ehss_angstrom2', 'collision_histogram', 'unresolved_rays', 'escaped_rays', 'pa_blocked_rays'):
        assert f32[key] == f64[key], key
    ref = O.trace_flat(c, r, o, d, cap=16)
    assert f32['collision_histogram'] == np.bincount(ref['bounces'], minlength=17).tolist()
    assert f32['escaped_rays'] == np.count_nonzero(ref['escaped'])
    assert f32['pa_blocked_rays'] == np.count_nonzero(_any_hit(c, r, o, d, np.full(4096, -1)))


def _any_hit(c, r, o, d, owners):
    """sphere_hit of every ray and atom, each operation rounded once."""
    out = np.zeros(len(o), dtype=bool)
    for k in range(len(r)):
        x = o - c[k]
        b = (x[:, 0] * d[:, 0] + x[:, 1] * d[:, 1]) + x[:, 2] * d[:, 2]
        disc = b * b - (((x[:, 0] * x[:, 0] + x[:, 1] * x[:, 1]) + x[:, 2] * x[:, 2]) - r[k] * r[k])
        out |= (disc >= 0) & (-b + np.sqrt(np.maximum(disc, 0.)) > 0) & (owners != k)
    return out


@pytest.mark.parametrize('scale', SCALES + ['32 bits'])
def test_any_hit_equals_every_atom(scale):
    """Rays from 2.5 S out, from inside the structure, just past the spheres (few
    of a scaled ray's hits are its unit ray's), and along lines up to 2 S out."""
    from types import SimpleNamespace
    import ehss_b200 as eb
    c, r, o, d = _rays(400, 8192, 19)
    S = np.max(np.linalg.norm(c - c.mean(axis=0), axis=1) + r)
    rng = np.random.default_rng(3)
    o[::4] -= 1.5 * S * d[::4]
    o[1::4] = c.mean(axis=0) + rng.normal(size=o[1::4].shape) * .4 * S
    side = np.cross(d[2::4], rng.normal(size=d[2::4].shape))
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    k = rng.integers(0, 400, len(side))
    o[2::4] = c[k] + side * (r[k] * (1. + 10. ** rng.uniform(-7., -1., len(k))))[:, None] - 1.8 * S * d[2::4]
    side = np.cross(d[3::4], rng.normal(size=d[3::4].shape))
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    o[3::4] += side * S * rng.uniform(0., 1.2, (len(side), 1))
    d = d.astype(np.float32).astype(np.float64) if scale == '32 bits' else d * scale
    index = eb.SphereIndex(eb.Spheres(c, r, deduplicate=False))
    for owners in (np.full(8192, -1), rng.integers(-1, 400, 8192)):
        blocked = index.query(SimpleNamespace(origins=o, directions=d, owners=owners))[0]
        assert np.array_equal(blocked, _any_hit(c, r, o, d, owners))


def test_any_hit_of_rounded_directions_walks_the_tree():
    from types import SimpleNamespace
    import ehss_b200 as eb
    c, r, o, d = _rays(5000, 2048, 23)
    index = eb.SphereIndex(eb.Spheres(c, r, deduplicate=False))
    tests = [index.query(SimpleNamespace(origins=o, directions=x, owners=np.full(2048, -1)))[2]
             for x in (d, d.astype(np.float32).astype(np.float64))]
    assert tests[1] < 2 * tests[0]
