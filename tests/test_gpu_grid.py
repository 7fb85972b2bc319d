"""Adaptive-grid PA at the edges of the raster kernel: grids narrower than a
mask word and of the largest size, atom counts around the staging size, disks
below a pixel, sparse structures whose atoms do not hide one another, exterior
scenes.  Pixel counts are integers, so every comparison is for equality."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _structure(atoms, kind, seed=0):
    rng = np.random.default_rng([atoms, seed])
    if kind == 'sparse':       # no atom hides another
        return rng.uniform(-40., 40., (atoms, 3)), rng.uniform(.02, .3, atoms)
    side = (atoms / .1) ** (1. / 3.)
    return rng.uniform(-side / 2, side / 2, (atoms, 3)), rng.uniform(2.4, 3.2, atoms)


@pytest.mark.parametrize('atoms,kind,directions,grid', [
    (1, 'dense', 4, 8), (1, 'dense', 2, 8192), (3, 'dense', 1, 16), (7, 'dense', 64, 32), (8, 'sparse', 2, 64),
    (1023, 'dense', 2, 256), (1024, 'sparse', 2, 512), (1025, 'dense', 64, 128), (2100, 'dense', 128, 512),
    (20000, 'dense', 2, 1024), (30000, 'sparse', 1, 1024), (9000, 'sparse', 1, 4096)])
def test_counts_equal_the_oracle(atoms, kind, directions, grid):
    import ehss_b200 as eb
    from ehss_b200.adaptive_pa import grid_counts
    c, r = _structure(atoms, kind)
    scene = eb.Scene(c, r)
    counts, spacing, xy = grid_counts(scene, directions, grid, 5, with_xy=True)
    again, _ = grid_counts(scene, directions, grid, 5)
    assert np.array_equal(counts, again)
    for k in range(0, directions, max(1, directions // 3)):
        lower = np.array([-spacing[k] * grid / 2] * 2)
        assert counts[k] == O.union_count(xy[k], r, lower, spacing[k], grid), k


@pytest.mark.parametrize('atoms,kind', [(40, 'dense'), (1500, 'dense'), (5000, 'dense'), (300, 'sparse')])
def test_exterior_scene_counts_equal_the_full_scene(atoms, kind):
    import ehss_b200 as eb
    from ehss_b200.adaptive_pa import grid_counts
    c, r = _structure(atoms, kind, 1)
    full, exterior = eb.Scene(c, r), eb.Scene(c, r, exterior=True)
    assert kind == 'sparse' or atoms < 1000 or exterior.n_active < full.n_active
    for grid in (64, 512):
        a, b = grid_counts(full, 16, grid, 3), grid_counts(exterior, 16, grid, 3)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


# both sides of the line between the two cover kernels (grid^3 against 4096 atoms), of the number of CTAs that share a
# direction's atoms, and one CTA a direction
@pytest.mark.parametrize('atoms,kind,directions,grid', [
    (2, 'dense', 4, 16), (8, 'dense', 2, 32), (9, 'dense', 2, 32), (128, 'sparse', 2, 64), (129, 'sparse', 2, 64),
    (512, 'dense', 4, 128), (513, 'dense', 4, 128), (700, 'dense', 512, 64), (2000, 'dense', 256, 16),
    (4096, 'dense', 2, 256), (4097, 'sparse', 2, 256), (20000, 'dense', 1, 8), (20000, 'dense', 64, 64),
    (33000, 'sparse', 1, 512), (300000, 'sparse', 1, 1024), (2000, 'dense', 4, 1024), (257, 'dense', 1, 512)])
def test_coarse_grids_and_shared_directions(atoms, kind, directions, grid):
    test_counts_equal_the_oracle(atoms, kind, directions, grid)
