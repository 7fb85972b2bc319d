"""The work that users of this package have it do, as timed cases.

Each case goes through one of the package's public entry points at sizes taken
from its command line's defaults, its benchmark workloads and its tests:

* ``rays``    explicit rays in host arrays through ``PreparedStaticGPUEHSS(...).engine.trace``
* ``pa``      explicit rays through ``SphereIndex(...).query`` (any-hit projection approximation)
* ``grid``    ``adaptive_pa.grid_counts``, the command line's default PA
* ``batch``   ``BatchCCS(...).run()``: host coordinates in, per-structure cross sections out
* ``cli``     ``ccs_cli.solve_frames``: what ``ccs.py`` computes between reading and writing files
* ``served``  ``serve.DeviceExecutor``: scenes built for newly admitted requests, then one round
* ``refit``   moved frames of the same atoms: ``BatchScenes.refit``, then one block per frame

Structures are the package's synthetic globules (random sequential addition,
van der Waals radii plus probe) and the bent triatomic; rays are those of the
impact disk that every cross section is an average over.
"""
import math

import numpy as np
import torch


def listed():
    return [
        # the smallest molecule, few rays, double precision: a call that is all latency
        dict(name='rays_triatomic', kind='rays', atoms=3, rays=4096, precision='fp64', cap=64),
        # a 650-atom structure sampled in double precision throughout
        dict(name='rays_650_fp64', kind='rays', atoms=650, rays=65536, precision='fp64', cap=64),
        # a 2000-atom structure at production sampling, default precision
        dict(name='rays_2000', kind='rays', atoms=2000, rays=262144, precision='fp32', cap=64),
        # projection approximation by rays on the same structure, a ragged ray count
        dict(name='pa_2000', kind='pa', atoms=2000, rays=200001),
        # the command line's default PA on a small structure
        dict(name='grid_650', kind='grid', atoms=650, directions=64, grid=512),
        # a large protein on a finer grid
        dict(name='grid_20000', kind='grid', atoms=20000, directions=64, grid=1024),
        # the benchmark: 256 structures of 20-5000 atoms, 2^14-2^18 rays, three replicates
        dict(name='batch_256', kind='batch', count=256, lo=20, hi=5000, log2_lo=14, log2_hi=18, repeats=3,
             precision='fp32', pa=False, boundary='', cap=64),
        # one structure, 20 replicates, double precision, EHSS and PA from the same launch
        dict(name='batch_650_fp64_pa', kind='batch', count=1, lo=650, hi=650, log2_lo=16, log2_hi=16, repeats=20,
             precision='fp64', pa=True, boundary='', cap=64),
        # production incidence: rays on an enclosing box, a high cap
        dict(name='batch_box', kind='batch', count=3, lo=300, hi=5000, log2_lo=16, log2_hi=16, repeats=8,
             precision='fp32', pa=False, boundary='box', cap=1024),
        # ccs.py with its default options on one structure: EHSS and adaptive PA, three replicates
        dict(name='cli_default', kind='cli', frames=1, atoms=650, log2=14, repeats=3, pa_method='adaptive', grid=512,
             directions=64),
        # a serving round that has just admitted six requests of 10-20000 atoms
        dict(name='served_round', kind='served', requests=6, lo=10, hi=20000, log2=15, blocks=2),
        # an ensemble of moved frames, tree topology kept
        dict(name='refit_200', kind='refit', frames=200, atoms=1500, log2=15),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['rays', 'rays', 'pa', 'grid', 'batch', 'batch', 'cli', 'served', 'refit'])
    if kind == 'rays':
        return dict(kind=kind, atoms=_log_int(rng, 3, 20000), rays=_log_int(rng, 100, 262144),
                    precision=rng.choice(['fp32', 'fp64']), cap=rng.choice([8, 64, 512]))
    if kind == 'pa':
        return dict(kind=kind, atoms=_log_int(rng, 3, 20000), rays=_log_int(rng, 100, 262144))
    if kind == 'grid':
        # directions and grid are powers of two by the entry point's rule
        return dict(kind=kind, atoms=_log_int(rng, 3, 20000), directions=1 << rng.randint(0, 6), grid=1 << rng.randint(4, 10))
    if kind == 'batch':
        hi = _log_int(rng, 40, 5000)
        log2 = rng.randint(10, 16)
        return dict(kind=kind, count=_log_int(rng, 1, 64), lo=max(3, hi // rng.randint(1, 20)), hi=hi, log2_lo=log2 - 2,
                    log2_hi=log2, repeats=rng.randint(1, 8), precision=rng.choice(['fp32', 'fp32', 'fp64']),
                    pa=rng.random() < 0.4, boundary=rng.choice(['', '', 'box', 'ellipsoid', 'sphere']),
                    cap=rng.choice([12, 64, 512]))
    if kind == 'cli':
        return dict(kind=kind, frames=_log_int(rng, 1, 12), atoms=_log_int(rng, 3, 5000), log2=rng.randint(8, 16),
                    repeats=rng.randint(1, 4), pa_method=rng.choice(['adaptive', 'bvh']), grid=rng.choice([128, 256, 512]),
                    directions=rng.choice([16, 32, 64]))
    if kind == 'served':
        return dict(kind=kind, requests=_log_int(rng, 1, 20), lo=10, hi=_log_int(rng, 100, 20000), log2=rng.randint(12, 15),
                    blocks=rng.randint(1, 2))
    return dict(kind=kind, frames=_log_int(rng, 2, 200), atoms=_log_int(rng, 20, 1500), log2=rng.randint(10, 15))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _structure(atoms, seed):
    from ehss_b200 import workloads
    if atoms == 3:
        xyz, radii, _ = workloads.triatomic()
        return xyz @ workloads.random_rotation(seed).T, radii
    xyz, radii, _ = workloads.globule(atoms, seed)
    return xyz, radii


def _structures(case, seed):
    """[(centers, radii)] of a batch: sizes log-uniform over the case's range."""
    rng = np.random.default_rng(seed)
    n = case.get('count', case.get('requests'))
    sizes = np.exp(rng.uniform(math.log(case['lo']), math.log(case['hi']), n)).round().astype(int)
    return [_structure(int(a), int(s)) for a, s in zip(sizes, rng.integers(0, 2 ** 31, n))]


def _log2s(case, seed):
    # every seed has the same amount of work: an even spread of ray budgets, in a random order
    spread = np.linspace(case['log2_lo'], case['log2_hi'], case['count']).round().astype(int)
    return [int(x) for x in np.random.default_rng([seed, 1]).permutation(spread)]


def _disk_rays(u, centers, radii):
    """Impact-disk rays of the unit-cube points u [n, 4]."""
    centers, radii = np.asarray(centers), np.asarray(radii)
    center = centers.mean(axis=0)
    radius = float(np.max(np.linalg.norm(centers - center, axis=1) + radii)) * (1. + 1e-9)
    z, phi = 1 - 2 * u[:, 0], 2 * np.pi * u[:, 1]
    rho = np.sqrt(np.maximum(0, 1 - z * z))
    d = np.column_stack((rho * np.cos(phi), rho * np.sin(phi), z))
    axes = np.zeros_like(d)
    axes[:, 2] = 1
    axes[np.abs(d[:, 2]) > .9] = [1, 0, 0]
    t = np.cross(axes, d)
    t /= np.linalg.norm(t, axis=1)[:, None]
    b = np.cross(d, t)
    rho, phi = radius * np.sqrt(u[:, 2]), 2 * np.pi * u[:, 3]
    o = center - radius * d + rho[:, None] * (np.cos(phi)[:, None] * t + np.sin(phi)[:, None] * b)
    return o, d, radius


def _ray_inputs(case, seed):
    centers, radii = _structure(case['atoms'], seed)
    o, d, radius = _disk_rays(np.random.default_rng([seed, 2]).random((case['rays'], 4)), centers, radii)
    return centers, radii, o, d, radius


def _pinned(a):
    """The array in page-locked memory, as the package's own sources return their rays."""
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _frames(case, seed):
    from ehss_b200 import workloads
    base, radii = _structure(case['atoms'], seed)
    return [(workloads.ensemble_frame(base, k, seed=seed), radii) for k in range(case['frames'])], (base, radii)


def _cli_args(case, seed):
    from ehss_b200 import ccs_cli
    return ccs_cli.parser().parse_args(
        ['unused.xyz', '--method', 'both', '--pa-method', case['pa_method'], '--rays', str(1 << case['log2']),
         '--directions', str(case['directions']), '--grid-size', str(case['grid']), '--repeats', str(case['repeats']),
         '--seed', str(seed % 2 ** 32)])


def prepare(case, seed):
    import ehss_b200 as eh
    kind = case['kind']
    if kind in ('rays', 'pa'):
        centers, radii, o, d, radius = _ray_inputs(case, seed)
        n = len(o)
        o, d = _pinned(o), _pinned(d)
        spheres = eh.Spheres(centers, radii, deduplicate=False)
        source = eh.EHSSSource(o, d, d, np.full(n, np.pi * radius * radius / n), np.full(n, -1),
                               np.zeros(n, dtype=np.int64), 'external impact disk')
        if kind == 'rays':
            return dict(kind=kind, engine=eh.PreparedStaticGPUEHSS(spheres, precision=case['precision']).engine,
                        source=source, cap=case['cap'])
        return dict(kind=kind, index=eh.SphereIndex(spheres), source=source)
    if kind == 'grid':
        centers, radii = _structure(case['atoms'], seed)
        return dict(kind=kind, scene=eh.Scene(centers, radii), directions=case['directions'], grid=case['grid'], seed=seed)
    if kind == 'batch':
        from ehss_b200.batch import BatchCCS
        structures, log2s = _structures(case, seed), _log2s(case, seed)
        seeds = [(seed + 7919 * k) % 2 ** 32 for k in range(len(structures))]
        return dict(kind=kind, job=BatchCCS(structures, log2s, seeds, repeats=case['repeats'], cap=case['cap'],
                                            precision=case['precision'], pa=case['pa'], boundary=case['boundary'] or None))
    if kind == 'cli':
        frames, _ = _frames(case, seed)
        return dict(kind=kind, frames=[eh.Spheres(c, r, deduplicate=False) for c, r in frames], args=_cli_args(case, seed))
    if kind == 'served':
        from ehss_b200.serve import DeviceExecutor
        return dict(kind=kind, executor=DeviceExecutor(), structures=_structures(case, seed), log2=case['log2'],
                    blocks=case['blocks'], seed=seed)
    from ehss_b200.batch import BatchScenes
    frames, base = _frames(case, seed)
    scenes = BatchScenes([base] * len(frames))
    scenes.build()
    return dict(kind=kind, scenes=scenes, frames=frames, log2=case['log2'], seed=seed)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _stat(results, key, field):
    return np.array([float('nan') if r[key][field] is None else r[key][field] for r in results])


def run(state):
    kind = state['kind']
    if kind == 'rays':
        r = state['engine'].trace(state['source'], state['cap'])
        return dict(positions=r.positions, outgoing=r.outgoing, escaped=r.escaped, unresolved=r.unresolved,
                    bounces=r.bounces)
    if kind == 'pa':
        return dict(blocked=state['index'].query(state['source'])[0])
    if kind == 'grid':
        from ehss_b200.adaptive_pa import grid_counts
        counts, spacing = grid_counts(state['scene'], state['directions'], state['grid'], state['seed'])
        return dict(counts=counts, spacing=spacing)
    if kind == 'batch':
        results = state['job'].run()
        out = dict(mean=_stat(results, 'ehss_angstrom2', 'mean'), sd=_stat(results, 'ehss_angstrom2', 'sd'),
                   tail=np.array([r['ehss_tail_bound_mean_angstrom2'] for r in results]),
                   unresolved=np.array([r['ehss_unresolved_rays_total'] for r in results]))
        if state['job'].pa:
            out.update(pa_mean=_stat(results, 'pa_angstrom2', 'mean'), pa_sd=_stat(results, 'pa_angstrom2', 'sd'))
        return out
    if kind == 'cli':
        from ehss_b200.ccs_cli import solve_frames
        rows = [row for r in solve_frames(state['frames'], state['args'], progress=False) for row in r['runs']]
        return dict(ehss=np.array([r['ehss']['ehss_angstrom2'] for r in rows]),
                    tail=np.array([r['ehss']['tail_bound_angstrom2'] for r in rows]),
                    histogram=np.array([r['ehss']['collision_histogram'] for r in rows]),
                    contribution=np.array([r['ehss']['collision_contribution_angstrom2'] for r in rows]),
                    pa=np.array([r['pa']['pa_angstrom2'] for r in rows]))
    if kind == 'served':
        from ehss_b200.blocks import seed_schedule
        executor = state['executor']
        handles = executor.build(state['structures'])
        jobs = [(h, state['log2'], s) for h in handles for s in seed_schedule(state['seed'], state['blocks'])]
        results = np.array(executor.trace(jobs))
        for h in handles:
            executor.release(h)
        return dict(ehss=results[:, 0], tail=results[:, 1])
    from ehss_b200.blocks import BlockJob, BlockPlan
    scenes = state['scenes']
    scenes.refit(state['frames'])
    plan = BlockPlan([BlockJob(s, state['log2'], state['seed'] % 2 ** 32) for s in scenes.scenes])
    plan.enqueue()
    blocks = plan.collect()
    return dict(ehss=np.array([b['ehss_angstrom2'] for b in blocks]),
                tail=np.array([b['tail_bound_angstrom2'] for b in blocks]),
                hits=np.array([b['pa_from_same_rays_angstrom2'] for b in blocks]))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: coordinates and rays read once, results written once.  Operations:
    a ray that hits (about half of the impact disk's) makes one query more than
    it has collisions, 1.8 per ray on these structures; a query cannot do
    without one box test a level of a binary tree (27 operations) and the tests
    of the spheres that it nearly meets (about 4, of 35 operations)."""
    kind = case['kind']

    def query(atoms):
        return 27. * math.log2(max(2, atoms)) + 35. * min(4, atoms)

    if kind == 'rays':
        return dict(bytes=case['rays'] * (64 + 58.) + 32. * case['atoms'], flops=case['rays'] * 1.8 * query(case['atoms']))
    if kind == 'pa':
        return dict(bytes=case['rays'] * (56 + 1.) + 32. * case['atoms'], flops=case['rays'] * query(case['atoms']))
    if kind == 'grid':
        # every atom projected (12 operations) and its rows' two ends found (10 a row); the mean atom spans
        # 2 r of the structure's width, which grows as the cube root of its atoms
        width = 2 * (1.1 * (case['atoms'] / (4 / 3 * math.pi * 0.1)) ** (1 / 3) + 2.9)
        rows = 2 * 2.9 / width * case['grid']
        return dict(bytes=32. * case['atoms'] + 16. * case['directions'],
                    flops=case['directions'] * case['atoms'] * (12. + 10. * rows))
    if kind == 'batch':
        lo, hi, n = case['lo'], case['hi'], case['count']
        mean = lo if hi == lo else (hi - lo) / math.log(hi / lo)
        rays = case['repeats'] * float(sum(1 << int(round(x)) for x in np.linspace(case['log2_lo'], case['log2_hi'], n)))
        each = (2.8 if case['pa'] else 1.8) * query(math.sqrt(lo * hi))
        return dict(bytes=32. * n * mean + 48. * n, flops=rays * (each + 100.))
    if kind == 'cli':
        rays = float(case['frames'] * case['repeats'] << case['log2'])
        bvh = case['pa_method'] == 'bvh'
        grid = 0. if bvh else work(dict(case, kind='grid'))['flops'] * case['frames'] * case['repeats']
        return dict(bytes=case['frames'] * 32. * case['atoms'], flops=rays * ((2.8 if bvh else 1.8) * query(case['atoms']) + 100.) + grid)
    if kind == 'served':
        mean = (case['hi'] - case['lo']) / math.log(case['hi'] / case['lo'])
        rays = float(case['requests'] * case['blocks'] << case['log2'])
        return dict(bytes=case['requests'] * 32. * mean, flops=rays * (1.8 * query(math.sqrt(case['lo'] * case['hi'])) + 100.))
    rays = float(case['frames'] << case['log2'])
    return dict(bytes=case['frames'] * 32. * case['atoms'], flops=rays * (1.8 * query(case['atoms']) + 100.))


# ---------------------------------------------------------------------------
# the same results from plain 64-bit arithmetic, every ray against every atom
# ---------------------------------------------------------------------------
_MAX_PAIRS = 2e10 if torch.cuda.is_available() else 1e8


def _nearest(o, d, c, r, last):
    """Entry distance and index of the nearest sphere of each ray (infinite: none)."""
    aa = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    x = [o[:, k, None] - c[None, :, k] for k in range(3)]
    proj = ((x[0] * d[:, 0, None] + x[1] * d[:, 1, None]) + x[2] * d[:, 2, None]) / aa[:, None]
    p = [x[k] - proj * d[:, k, None] for k in range(3)]
    disc = (r * r)[None] - ((p[0] * p[0] + p[1] * p[1]) + p[2] * p[2])
    near = -proj - torch.sqrt(disc.clamp_min(0.) / aa[:, None])
    miss = (disc < 0) | (proj >= 0) | (near < (-64. * np.finfo(float).eps) * r[None])
    t = near.clamp_min(0.).masked_fill(miss, math.inf)
    rows = torch.nonzero(last >= 0)[:, 0]
    t[rows, last[rows]] = math.inf
    return t.min(dim=1)


def _trace(o, d, centers, radii, cap):
    """(positions, directions, escaped, bounces) of rays followed to escape or to cap."""
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    o, d, c, r = (torch.tensor(np.asarray(a), dtype=torch.float64, device=dev) for a in (o, d, centers, radii))
    n, step = len(o), max(1, int(3e7) // len(r))
    bounces, escaped = torch.zeros(n, dtype=torch.int64, device=dev), torch.zeros(n, dtype=torch.bool, device=dev)
    last, live = torch.full((n,), -1, dtype=torch.int64, device=dev), torch.arange(n, device=dev)
    while len(live):
        left = []
        for i in live.split(step):
            t, k = _nearest(o[i], d[i], c, r, last[i])
            escaped[i[t == math.inf]] = True
            on = (t != math.inf) & (bounces[i] < cap)
            i, t, k = i[on], t[on, None], k[on]
            m = o[i] + t * d[i] - c[k]
            m = m / torch.sqrt((m[:, 0] * m[:, 0] + m[:, 1] * m[:, 1]) + m[:, 2] * m[:, 2])[:, None]
            o[i] = c[k] + r[k, None] * m
            dot = (d[i, 0] * m[:, 0] + d[i, 1] * m[:, 1]) + d[i, 2] * m[:, 2]
            e = d[i] - (2. * dot)[:, None] * m
            d[i] = e / torch.sqrt((e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1]) + e[:, 2] * e[:, 2])[:, None]
            bounces[i] += 1
            last[i] = k
            left.append(i)
        live = torch.cat(left)
    return o.cpu().numpy(), d.cpu().numpy(), escaped.cpu().numpy(), bounces.cpu().numpy()


# Joe and Kuo's direction numbers: degree, coefficients, first values of dimensions 2 to 5
_JOE_KUO = [(1, 0, (1,)), (2, 1, (1, 3)), (3, 1, (1, 3, 1)), (3, 2, (1, 1, 1))]


def _sobol(dim, log2, seed):
    """2**log2 points of scipy's scrambled Sobol sequence (30 bits, linear matrix scramble and digital shift)."""
    bits = 30
    v = np.zeros((dim, bits), dtype=np.int64)
    v[0] = 1 << np.arange(bits - 1, -1, -1)
    for j in range(1, dim):
        s, a, m = _JOE_KUO[j - 1]
        for k in range(bits):
            if k < s:
                v[j, k] = m[k] << (bits - 1 - k)
            else:
                v[j, k] = v[j, k - s] ^ (v[j, k - s] >> s)
                for t in range(1, s):
                    if (a >> (s - 1 - t)) & 1:
                        v[j, k] ^= v[j, k - t]
    rng = np.random.default_rng(seed)
    shift = (rng.integers(2, size=(dim, bits), dtype=np.uint32).astype(np.int64) << np.arange(bits)).sum(axis=1)
    lower = np.tril(rng.integers(2, size=(dim, bits, bits), dtype=np.uint32)).astype(np.int64)
    place = np.arange(bits - 1, -1, -1)
    lower[:, np.arange(bits), np.arange(bits)] = 1
    digits = (v[:, :, None] >> place) & 1
    v = ((np.einsum('jil,jkl->jki', lower, digits) & 1) << place).sum(axis=2)
    index = np.arange(1 << log2)
    gray, q = index ^ (index >> 1), np.tile(shift, (1 << log2, 1))
    for k in range(log2):
        q[(gray >> k) & 1 == 1] ^= v[:, k]
    return q * 2. ** -bits


def _box_rays(u, centers, radii):
    """Rays on an enclosing box (origins, directions, projected areas)."""
    low, high = np.min(centers - radii[:, None], axis=0), np.max(centers + radii[:, None], axis=0)
    center, ax = (low + high) / 2, (high - low) / 2 * (1 + 1e-9)
    z, phi = 1 - 2 * u[:, 0], 2 * np.pi * u[:, 1]
    rho = np.sqrt(np.maximum(0, 1 - z * z))
    d = np.column_stack((rho * np.cos(phi), rho * np.sin(phi), z))
    proj = np.abs(d) * (4 * np.prod(ax) / ax)
    area = proj.sum(axis=1)
    face = np.minimum((u[:, 2, None] * area[:, None] >= np.cumsum(proj, axis=1)).sum(axis=1), 2)
    p = np.empty_like(d)
    for k in range(3):
        i = np.flatnonzero(face == k)
        p[i, k] = -np.sign(d[i, k]) * ax[k]
        other = [j for j in range(3) if j != k]
        p[np.ix_(i, other)] = (2 * u[i, 3:5] - 1) * ax[other]
    return center + p - 1e-10 * max(1., ax.max()) * d, d, area


def _block(centers, radii, log2, seed, cap, boundary=''):
    """One replicate: (ehss, tail, hit area, collision histogram, contribution by collisions)."""
    n = 1 << log2
    if boundary == 'box':
        o, d, area = _box_rays(_sobol(5, log2, seed), centers, radii)
    else:
        o, d, radius = _disk_rays(_sobol(4, log2, seed), centers, radii)
        area = np.full(n, np.pi * radius * radius)
    _, out, escaped, bounces = _trace(o, d, centers, radii, cap)
    w = area / n
    part = w * np.clip(1 - (d * out).sum(axis=1), 0., 2.) * escaped
    return (part.sum(), 2 * w[~escaped].sum(), w[(bounces > 0) | ~escaped].sum(), np.bincount(bounces, minlength=cap + 1),
            np.bincount(bounces, weights=part, minlength=cap + 1), int((~escaped).sum()))


def _grid(centers, radii, directions, grid, seed):
    """Covered pixels and pixel spacing of each direction's midpoint grid."""
    rel = centers - centers.mean(axis=0)
    points = _sobol(2, max(1, (directions - 1).bit_length()), seed)[:directions]
    counts, spacings = [], []
    for u0, u1 in points:
        z = 1 - 2 * u0
        rho = math.sqrt(max(0., 1 - z * z))
        d = np.array([rho * math.cos(2 * np.pi * u1), rho * math.sin(2 * np.pi * u1), z])
        d /= np.linalg.norm(d)
        a = np.cross([0., 0., 1.] if abs(d[2]) < .9 else [1., 0., 0.], d)
        a /= np.linalg.norm(a)
        x, y = rel @ a, rel @ np.cross(d, a)
        extent = max(np.max(np.abs(x) + radii), np.max(np.abs(y) + radii)) * 1.0000000001
        spacing = 2 * extent / grid
        at = -extent + (np.arange(grid) + .5) * spacing
        lo, hi = np.searchsorted(at, y - radii), np.searchsorted(at, y + radii)
        rows = hi - lo
        i = np.repeat(np.arange(len(x)), rows)
        row = np.arange(rows.sum()) - np.repeat(np.cumsum(rows) - rows, rows) + lo[i]
        half = np.sqrt(np.maximum(0., radii[i] ** 2 - (at[row] - y[i]) ** 2))
        edge = np.zeros((grid, grid + 1), dtype=np.int64)
        np.add.at(edge, (row, np.searchsorted(at, x[i] - half)), 1)
        np.add.at(edge, (row, np.searchsorted(at, x[i] + half, side='right')), -1)
        counts.append(int((np.cumsum(edge, axis=1) > 0).sum()))
        spacings.append(spacing)
    return np.array(counts), np.array(spacings)


def _sd(values):
    return values.std(axis=1, ddof=1) if values.shape[1] > 1 else np.full(len(values), np.nan)


def exact(case, seed):
    """None where every ray against every atom would take too long."""
    kind = case['kind']
    schedule = [(seed + 104729 * k) % 2 ** 32 for k in range(case.get('repeats', case.get('blocks', 1)))]
    if kind == 'rays':
        if 2. * case['rays'] * case['atoms'] > _MAX_PAIRS:
            return None
        centers, radii, o, d, _ = _ray_inputs(case, seed)
        position, out, escaped, bounces = _trace(o, d, centers, radii, case['cap'])
        return dict(positions=position, outgoing=out, escaped=escaped, unresolved=~escaped, bounces=bounces)
    if kind == 'pa':
        if 2. * case['rays'] * case['atoms'] > _MAX_PAIRS:
            return None
        centers, radii, o, d, _ = _ray_inputs(case, seed)
        _, _, _, bounces = _trace(o, d, centers, radii, 1)
        return dict(blocked=bounces > 0)
    if kind == 'grid':
        if case['directions'] * case['atoms'] > 2e5:
            return None
        counts, spacing = _grid(*_structure(case['atoms'], seed), case['directions'], case['grid'], seed)
        return dict(counts=counts, spacing=spacing)
    if kind == 'batch':
        rays = case['repeats'] * float(case['count'] << case['log2_hi'])
        if 2. * rays * case['hi'] > _MAX_PAIRS or rays > 3e6 or case['boundary'] not in ('', 'box'):
            return None
        blocks = [[_block(c, r, log2, (seed + 7919 * k + 104729 * j) % 2 ** 32, case['cap'], case['boundary'])
                   for j in range(case['repeats'])]
                  for k, ((c, r), log2) in enumerate(zip(_structures(case, seed), _log2s(case, seed)))]
        ehss, tail, hit, left = (np.array([[b[f] for b in row] for row in blocks]) for f in (0, 1, 2, 5))
        out = dict(mean=ehss.mean(axis=1), sd=_sd(ehss), tail=tail.mean(axis=1), unresolved=left.sum(axis=1))
        if case['pa']:
            out.update(pa_mean=hit.mean(axis=1), pa_sd=_sd(hit))
        return out
    if kind == 'cli':
        rays = float(case['frames'] * case['repeats'] << case['log2'])
        grids = case['frames'] * case['repeats'] * case['directions'] * case['atoms']
        if 2. * rays * case['atoms'] > _MAX_PAIRS or rays > 3e6 or grids > 2e5:
            return None
        rows = []
        for c, r in _frames(case, seed)[0]:
            for s in schedule:
                b = _block(c, r, case['log2'], s, 64)
                if case['pa_method'] == 'adaptive':
                    counts, spacing = _grid(c, r, case['directions'], case['grid'], s)
                    b = b[:2] + (np.mean(counts * spacing ** 2),) + b[3:]
                rows.append(b)
        return dict(zip(('ehss', 'tail', 'pa', 'histogram', 'contribution'), (np.array(x) for x in list(zip(*rows))[:5])))
    if kind == 'served':
        rays = float(case['requests'] * case['blocks'] << case['log2'])
        if 2. * rays * case['hi'] > _MAX_PAIRS or rays > 3e6:
            return None
        blocks = [_block(c, r, case['log2'], s, 64) for c, r in _structures(case, seed) for s in schedule]
        return dict(ehss=np.array([b[0] for b in blocks]), tail=np.array([b[1] for b in blocks]))
    rays = float(case['frames'] << case['log2'])
    if 2. * rays * case['atoms'] > _MAX_PAIRS or rays > 3e6:
        return None
    blocks = [_block(c, r, case['log2'], seed % 2 ** 32, 64) for c, r in _frames(case, seed)[0]]
    return dict(ehss=np.array([b[0] for b in blocks]), tail=np.array([b[1] for b in blocks]),
                hits=np.array([b[2] for b in blocks]))
