"""Coordinate P(r) on the GPU (metrics.rs:236-270, 475-583) against the oracle.

Bins are index work and must be the reference's bit for bit: with unit
weights every bin holds an integer count, which f64 sums exactly in any
order, so those histograms must equal the oracle's exactly.  Weighted sums
differ only by summation order: 1e-12 of the largest bin.  Rg and dmax are
computed in the reference's own order and must be equal.
"""
import math

import numpy as np
import pytest

import crabsaxs_b200 as cs
import oracle as O
from crabsaxs_b200 import synth

pytestmark = pytest.mark.gpu

C_, H_, N_, O_, S_ = 1, 0, 2, 3, 4
SUM_RTOL = 1e-12


def _oracle_atoms(s: cs.Structure):
    return O.Atoms(s.xyz, s.element, s.group, s.occupancy)


def _check_features(s: cs.Structure, bins, engine):
    got = cs.coordinate_features(s, cs.PrOptions(bins=bins), engine=engine)
    ref = O.coordinate_features(_oracle_atoms(s), bins)
    assert got.rg == ref["rg"] and got.dmax == ref["dmax"]
    assert np.array_equal(got.p_r.r, ref["r"])
    scale = np.max(np.abs(ref["p"]))
    assert np.max(np.abs(got.p_r.p - ref["p"])) <= SUM_RTOL * scale
    assert got.p_r.rg == pytest.approx(ref["pr_rg"], rel=SUM_RTOL)
    assert got.p_r.dmax == ref["pr_dmax"]
    return got


def test_coordinate_features_report_pair_distance(engine):  # metrics.rs:678-684
    s = cs.Structure(np.array([[0.0, 0.0, 0.0], [4.0, 0.0, 0.0]]), np.array([C_, C_]))
    f = _check_features(s, 160, engine)
    assert abs(f.dmax - 4.0) < 1e-12 and f.rg > 1.0 and len(f.p_r.p) > 0


@pytest.mark.parametrize("n,bins", [(300, 160), (1000, 16), (2500, 160), (2500, 1000), (777, 7)])
def test_protein_features_match_oracle(engine, n, bins):
    s = synth.protein(40 + n, n, 6.0 + n ** (1.0 / 3.0))
    _check_features(s, bins, engine)


def test_groups_occupancy_and_hydrogen_floor(engine):
    """United-atom groups change the weights, occupancies scale them, and
    hydrogens (form factor 0 with implicit hydrogens) take the 1e-6 floor."""
    base = synth.protein(91, 1500, 14.0)
    rng = np.random.default_rng(5)
    n = len(base.xyz)
    el = base.element.copy()
    el[rng.random(n) < 0.1] = H_
    group = np.where(el == C_, rng.integers(-1, 4, n), -1).astype(np.int8)
    group[(el == N_) & (rng.random(n) < 0.5)] = 7
    occ = np.where(rng.random(n) < 0.2, 0.5, 1.0)
    s = cs.Structure(base.xyz, el, occ, group)
    _check_features(s, 200, engine)


def _mode(engine):
    return cs.pr_last_timing(engine)[3]


def test_unit_weight_bins_are_exact(engine):
    """Unit weights: one weight class, integer pair counts (mode 0)."""
    s = synth.protein(17, 3000, 20.0)
    for bins in (16, 160, 4096):
        dmax, hist = cs.pair_distance_histogram(s.xyz, np.ones(len(s.xyz)), bins, engine=engine)
        assert _mode(engine) == 0
        rd, rh = O.pair_distance_histogram(s.xyz, np.ones(len(s.xyz)), bins)
        assert dmax == rd and np.array_equal(hist, rh), bins


def test_integer_weight_bins_are_exact_in_the_f64_mode(engine):
    """100 distinct integer weights exceed the 64 weight classes, so the
    products go through the per-warp f64 histograms (mode 1); integer sums
    below 2^53 are exact in any order, so the bins must equal the oracle's."""
    s = synth.protein(18, 2800, 19.0)
    w = 1.0 + (np.arange(len(s.xyz)) % 100)
    for bins in (16, 160, 3000):
        dmax, hist = cs.pair_distance_histogram(s.xyz, w, bins, engine=engine)
        assert _mode(engine) == 1
        rd, rh = O.pair_distance_histogram(s.xyz, w, bins)
        assert dmax == rd and np.array_equal(hist, rh), bins


def test_several_weight_classes_count_exactly(engine):
    """A few distinct weights: per-class-pair counts (mode 0) combined as
    count * w_a * w_b against the oracle's pair-by-pair sums."""
    s = synth.protein(19, 2000, 16.0)
    w = np.array([1.0, 6.5, 7.25, 8.0, 16.125])[np.arange(len(s.xyz)) % 5]
    dmax, hist = cs.pair_distance_histogram(s.xyz, w, 160, engine=engine)
    assert _mode(engine) == 0
    rd, rh = O.pair_distance_histogram(s.xyz, w, 160)
    assert dmax == rd and np.array_equal(hist, rh)


def test_pairs_on_exact_bin_edges(engine):
    """Integer distances with step 1 sit exactly on bin edges; distance 16 is
    capped into the last bin (metrics.rs:515-516)."""
    xyz = np.zeros((17, 3))
    xyz[:, 0] = np.arange(17)
    dmax, hist = cs.pair_distance_histogram(xyz, np.ones(17), 16, engine=engine)
    expected = np.array([0.0] + [17.0 - k for k in range(1, 16)])
    expected[15] += 1.0
    assert dmax == 16.0 and np.array_equal(hist, expected)
    # a cubic lattice away from the origin: many equal distances at every radius
    g = np.stack(np.meshgrid(*[np.arange(9) * 1.25] * 3, indexing="ij"), -1).reshape(-1, 3) + 500.0
    for bins in (20, 160, 333):
        d, h = cs.pair_distance_histogram(g, np.ones(len(g)), bins, engine=engine)
        rd, rh = O.pair_distance_histogram(g, np.ones(len(g)), bins)
        assert d == rd and np.array_equal(h, rh), bins


def test_many_bins_use_the_global_histogram(engine):
    """Above ~6,000 bins (f64) or ~8,000 (counts) the histograms no longer fit
    in shared memory and each block accumulates into its own row in device
    memory (mode 2).  20,000 bins still take the FP32 fast path with a wide
    edge margin; above 75,000 bins the margin reaches a quarter bin and every
    pair takes the exact f64 path; above 2^20 bins as well."""
    s = synth.protein(23, 1200, 13.0)
    w = np.random.default_rng(2).uniform(1.0, 16.0, len(s.xyz))
    dmax, hist = cs.pair_distance_histogram(s.xyz, w, 20000, engine=engine)
    assert _mode(engine) == 2
    rd, rh = O.pair_distance_histogram(s.xyz, w, 20000)
    assert dmax == rd
    assert np.max(np.abs(hist - rh)) <= SUM_RTOL * np.max(rh)
    small = synth.protein(24, 300, 8.0)
    for atoms, bins in ((s, 20000), (s, 100000), (small, 1_200_000)):
        n = len(atoms.xyz)
        d1, h1 = cs.pair_distance_histogram(atoms.xyz, np.ones(n), bins, engine=engine)
        assert _mode(engine) == 2
        r1 = O.pair_distance_histogram(atoms.xyz, np.ones(n), bins)[1]
        assert np.array_equal(h1, r1), bins


def test_single_point_and_invalid_inputs(engine):  # metrics.rs:241-244, 489-498
    same = cs.Structure(np.tile([1.0, -2.0, 3.0], (300, 1)), np.full(300, C_))
    for s in (same, cs.Structure(np.array([[5.0, 5.0, 5.0]]), np.array([O_]))):
        f = cs.coordinate_features(s, engine=engine)
        assert f.dmax == 0.0 and list(f.p_r.r) == [0.0] and list(f.p_r.p) == [1.0]
        assert f.p_r.rg == 0.0 and f.p_r.dmax == 0.0
    d, h = cs.pair_distance_histogram(np.zeros((0, 3)), np.zeros(0), 16, engine=engine)
    assert d == 0.0 and not h.any()
    with pytest.raises(cs.InvalidInput):
        cs.coordinate_features(cs.Structure(np.zeros((0, 3)), np.zeros(0, dtype=np.int8)), engine=engine)
    with pytest.raises(cs.InvalidInput):
        cs.pair_distance_histogram(np.zeros((3, 3)), np.ones(3), 0, engine=engine)
    with pytest.raises(cs.InvalidInput):
        cs.pair_distance_histogram(np.array([[0.0, 0, 0], [1e101, 0, 0]]), np.ones(2), 16, engine=engine)


def test_large_structure_matches_oracle(engine):
    """30,000 atoms (4.5e8 pairs): P(r) against the oracle, with the element
    weights (class counts) and with random per-atom weights (f64 mode)."""
    s = synth.protein(29, 30000, 40.0)
    _check_features(s, 160, engine)
    assert _mode(engine) == 0
    w = np.random.default_rng(4).uniform(0.5, 9.0, len(s.xyz))
    dmax, hist = cs.pair_distance_histogram(s.xyz, w, 160, engine=engine)
    assert _mode(engine) == 1
    rd, rh = O.pair_distance_histogram(s.xyz, w, 160)
    assert dmax == rd and np.max(np.abs(hist - rh)) <= SUM_RTOL * np.max(rh)


def test_100k_atoms_size_properties(engine):
    """100,000 atoms (R 80 Å): unit weights count every pair exactly once
    (sum n(n-1)/2, exact in f64), weighted sums total ((Σw)² - Σw²)/2, and
    dmax is at least the largest distance between extreme atoms."""
    w_ = synth.ATOMS_100K
    s = synth.protein(w_.seed, w_.n_atoms, w_.radius)
    n = len(s.xyz)
    _, h1 = cs.pair_distance_histogram(s.xyz, np.ones(n), 160, engine=engine)
    assert h1.sum() == n * (n - 1) / 2 and np.all(h1 == np.round(h1))
    w = np.random.default_rng(8).uniform(0.5, 9.0, n)
    dmax, h = cs.pair_distance_histogram(s.xyz, w, 160, engine=engine)
    total = (math.fsum(w) ** 2 - math.fsum(w * w)) / 2.0
    assert abs(h.sum() - total) <= 1e-11 * total
    ext = s.xyz[np.concatenate([np.argmin(s.xyz, 0), np.argmax(s.xyz, 0)])]
    dd = ext[:, None, :] - ext[None, :, :]
    assert dmax >= math.sqrt(np.max(np.sum(dd * dd, -1))) - 1e-9
    total_ms, hist_ms, pairs, mode = cs.pr_last_timing(engine)
    assert pairs == n * (n - 1) / 2 and 0.0 < hist_ms <= total_ms and mode == 1


@pytest.mark.parametrize("n", [2, 31, 33, 63, 65, 127, 129, 257, 500])
@pytest.mark.parametrize("classes", [1, 3, 60, 70])
@pytest.mark.parametrize("bins", [1, 37, 1600])
def test_tile_and_class_edges_are_exact(engine, n, classes, bins):
    """Whole and ragged warps, half tiles and tiles, one class to more than can be counted (70), and bins on both
    sides of 32 counters a bin: integer weights, so every bin is exact in any order and must equal the oracle's."""
    rng = np.random.default_rng(n + 7 * classes + bins)
    xyz = np.round(rng.uniform(-9.0, 9.0, size=(n, 3)), 1) + 55.0  # distances on a grid: many near or on edges
    w = rng.integers(1, classes + 1, size=n).astype(float)
    dmax, hist = cs.pair_distance_histogram(xyz, w, bins, engine=engine)
    rd, rh = O.pair_distance_histogram(xyz, w, bins)
    assert dmax == rd and np.array_equal(hist, rh)


def test_longest_pair_is_found_in_shells_and_rods(engine):
    """The atoms that can end the longest pair are found from one pair and its middle: a hollow sphere (all of them),
    a bent rod (the middle lies off the atoms), two clusters, and equal atoms."""
    rng = np.random.default_rng(8)
    v = rng.normal(size=(3000, 3))
    sphere = 40.0 * v / np.sqrt((v ** 2).sum(axis=1))[:, None]
    t = rng.uniform(0.0, 2.2, size=2500)
    rod = np.stack([60 * np.cos(t), 60 * np.sin(t), np.zeros_like(t)], axis=1) + rng.normal(size=(2500, 3))
    two = np.concatenate([rng.normal(size=(400, 3)), rng.normal(size=(700, 3)) + [90.0, 3.0, -8.0]])
    for xyz in (sphere, rod, two, np.repeat(two[:5], 40, axis=0)):
        d, h = cs.pair_distance_histogram(xyz, np.ones(len(xyz)), 50, engine=engine)
        rd, rh = O.pair_distance_histogram(xyz, np.ones(len(xyz)), 50)
        assert d == rd and np.array_equal(h, rh)


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e101])
def test_bad_coordinates_are_refused_in_every_mode(engine, bad):
    rng = np.random.default_rng(1)
    xyz = rng.normal(size=(300, 3))
    xyz[211, 2] = bad
    for w in (np.ones(300), rng.uniform(size=300)):
        with pytest.raises(cs.InvalidInput):
            cs.pair_distance_histogram(xyz, w, 20, engine=engine)
    d, h = cs.pair_distance_histogram(xyz[:200], np.ones(200), 20, engine=engine)
    assert d > 0 and h.sum() == 200 * 199 / 2


def _longest(xyz):
    """Largest squared pair distance in the reference's order of operations."""
    best = 0.0
    for i in range(0, len(xyz), 256):
        d = xyz[i:i + 256, None, :] - xyz[None, :, :]
        best = max(best, np.max(d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2]))
    return best


@pytest.mark.parametrize("shape", ["ball", "rod", "outlier", "shell", "far", "huge", "tiny", "equal"])
@pytest.mark.parametrize("n", [130, 4096, 4097, 8191, 8192])
def test_dmax_is_the_longest_pair(engine, n, shape):
    """The longest pair from the rim atoms, with and without moves of the
    centre, where FP32 squares apply and where they would overflow or vanish,
    and with many equally long pairs: dmax equals the f64 maximum exactly."""
    rng = np.random.default_rng(n)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    ball = u * rng.uniform(size=(n, 1)) ** (1.0 / 3.0) * 30.0
    xyz = {"ball": ball, "rod": ball * [4.0, 0.2, 0.2], "outlier": np.vstack([ball[1:], [[200.0, 3.0, -7.0]]]),
           "shell": 30.0 * u, "far": ball + 1.0e6, "huge": ball * 1.0e20, "tiny": ball * 1.0e-20,
           "equal": np.sign(ball) * 10.0}[shape]
    s = cs.Structure(xyz, np.ones(n, np.int8))
    got = cs.coordinate_features(s, cs.PrOptions(bins=40), engine=engine).dmax
    assert got == np.sqrt(_longest(xyz))


@pytest.mark.parametrize("scale", [1e-150, 1e-60, 1e-42, 1e-39, 1e-36, 1e30, 1e36, 3e37, 1e38, 3e39, 2e44, 7e45, 3e46, 1e60, 1e98])
@pytest.mark.parametrize("n", [200, 4500])
def test_steps_whose_inverse_is_not_an_fp32_number(engine, scale, n):
    """The counting kernel's bins are addresses: where 1/step is subnormal, zero or past FP32's largest number, every
    pair is placed by its f64 distance.  Whole numbers, equal to the oracle's."""
    rng = np.random.default_rng(n)
    xyz = rng.uniform(-0.5, 0.5, size=(n, 3)) * scale
    for bins in (1, 16, 160):
        d, h = cs.pair_distance_histogram(xyz, np.ones(n), bins, engine=engine)
        assert _mode(engine) == 0
        rd, rh = O.pair_distance_histogram(xyz, np.ones(n), bins)
        assert d == rd and np.array_equal(h, rh), bins


@pytest.mark.parametrize("n,k,bins", [(3, 3, 5449), (40, 1, 6112), (150, 58, 6386), (344, 3, 7296), (500, 2, 1500),
                                      (500, 2, 8000), (427, 41, 200), (700, 3, 100000 // 13)])
def test_few_pairs_and_many_bins(engine, n, k, bins):
    """Both widths of the shared counters, with class pairs of fewer pairs than bins among them: whole numbers, equal
    to the oracle's for products that f64 sums exactly."""
    rng = np.random.default_rng(n + bins)
    xyz = rng.uniform(-9.0, 9.0, size=(n, 3))
    w = 1.0 + rng.integers(0, k, size=n)
    w[: k] = 1.0 + np.arange(k)  # classes of very different sizes
    w[rng.random(n) < 0.5] = 1.0
    d, h = cs.pair_distance_histogram(xyz, w, bins, engine=engine)
    assert _mode(engine) == 0
    rd, rh = O.pair_distance_histogram(xyz, w, bins)
    assert d == rd and np.array_equal(h, rh)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("shape", ["sphere", "bent rod", "two clusters", "equal atoms"])
def test_longest_pair_past_the_size_that_looks_at_every_pair(engine, shape, weighted):
    """Above 4,096 atoms the longest pair is searched from one pair, a centre moved off its middle (with more than 64
    weights the box's) and the atoms about the rim: shapes whose middle lies off the atoms, or whose atoms all lie on
    the rim."""
    rng = np.random.default_rng(18)
    v = rng.normal(size=(5000, 3))
    t = rng.uniform(0.0, 2.2, size=9000)
    two = np.concatenate([rng.normal(size=(1600, 3)), rng.normal(size=(2800, 3)) + [90.0, 3.0, -8.0]])
    xyz = {"sphere": 40.0 * v / np.sqrt((v ** 2).sum(axis=1))[:, None],
           "bent rod": np.stack([60 * np.cos(t), 60 * np.sin(t), 0.0 * t], axis=1) + rng.normal(size=(9000, 3)),
           "two clusters": two, "equal atoms": np.repeat(two[:5], 1000, axis=0)}[shape]
    w = 1.0 + (np.arange(len(xyz)) % 100 if weighted else np.zeros(len(xyz)))
    d, h = cs.pair_distance_histogram(xyz, w, 50, engine=engine)
    assert _mode(engine) == (1 if weighted else 0)
    rd, rh = O.pair_distance_histogram(xyz, w, 50)
    assert d == rd and np.array_equal(h, rh)
