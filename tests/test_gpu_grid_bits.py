"""Hydration grids on bitmaps: boxes whose rows end before, on and after a
32-voxel word, fewer planes than the fill has slabs, a box larger than the
fill's shared memory (the sweeps), closed hollows, spheres that end on voxel
centres, and a coordinate far from the origin.  Site sets and their order are
compared exactly with the oracle's per-voxel tests and breadth-first fill."""
import numpy as np
import pytest

import crabsaxs_b200 as cs
import oracle as O

pytestmark = pytest.mark.gpu


def _cloud(seed, extent, n):
    """n atoms in a box of the given extents, with atoms in two corners."""
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(0.0, 1.0, (n, 3)) * np.asarray(extent)
    xyz[0], xyz[-1] = 0.0, extent
    return xyz, rng.choice([0, 1, 2, 3, 5], n).astype(np.int32)


def _hollow(radius, n):
    """A closed sphere of atoms: the voxels inside are not exterior."""
    k = np.arange(n) + 0.5
    t, f = np.arccos(1.0 - 2.0 * k / n), np.pi * (1.0 + 5.0**0.5) * k
    return radius * np.stack([np.cos(f) * np.sin(t), np.sin(f) * np.sin(t), np.cos(t)], 1)


def _check(engine, xyz, el, spacing, **kw):
    s = cs.Structure(xyz, el)
    got, _ = cs.hydration_grid_exterior(s, spacing, engine=engine, **kw)
    ref, _ = O.exterior_grid(xyz, el, spacing, *kw.values())
    assert got.shape == ref.shape and np.array_equal(got, ref)
    got, _ = cs.hydration_grid_adaptive(s, spacing, engine=engine)
    ref, _ = O.adaptive_grid(xyz, spacing)
    assert got.shape == ref.shape and np.array_equal(got, ref)


@pytest.mark.parametrize("nx", [31, 32, 33, 63, 64, 65, 97])
def test_rows_around_whole_words(engine, nx):
    # margin of the exterior box: 1.8 (largest radius, S) + 1.4 + 3.0 + 1.0 on each side
    xyz, el = _cloud(nx, (nx - 15.5, 21.0, 17.0), 60)
    _check(engine, xyz, el, 1.0)


@pytest.mark.parametrize("extent,spacing", [((40.0, 30.0, 0.0), 4.0), ((0.0, 0.0, 300.0), 4.0), ((3.0, 90.0, 2.0), 2.0),
                                            ((0.0, 0.0, 0.0), 30.0)])
def test_flat_and_thin_boxes(engine, extent, spacing):
    xyz, el = _cloud(7, extent, 40)
    _check(engine, xyz, el, spacing)


@pytest.mark.parametrize("radius", [6.0, 13.0])
def test_closed_hollow(engine, radius):
    xyz = _hollow(radius, int(6 * radius * radius))
    _check(engine, xyz, np.full(len(xyz), 1, np.int32), 1.0)


def test_box_beyond_the_shared_memory_fill(engine):
    xyz, el = _cloud(11, (18.0, 264.0, 264.0), 300)  # 33 x 280 x 280 voxels
    xyz = np.concatenate([xyz, _hollow(8.0, 400) + [9.0, 100.0, 150.0]])
    _check(engine, xyz, np.concatenate([el, np.full(400, 1, np.int32)]), 1.0)


@pytest.mark.parametrize("shift", [0.0, 4096.0, 1.0e7])
def test_spheres_that_end_on_voxel_centres(engine, shift):
    """Atoms on the grid's own lattice with radii of whole spacings: the
    distances of the outermost voxels equal the radius to the last bits."""
    rng = np.random.default_rng(5)
    xyz = rng.integers(0, 12, (30, 3)).astype(float) + shift
    el = np.full(30, 1, np.int32)  # carbon, 1.7
    _check(engine, xyz, el, 1.0, probe=1.3, thickness=2.0)
    _check(engine, xyz, el, 0.5, probe=0.8, thickness=1.5)
