"""The distance histogram at the limits of its shared memory, its inputs and its tables."""
import ctypes as C

import numpy as np
import pytest

import crabsaxs_b200 as cs
import oracle as O
from crabsaxs_b200 import _native as N

pytestmark = pytest.mark.gpu

HIST = 16  # the histogram's variant code


@pytest.fixture(scope="module")
def hist_engine():
    """A context whose pair sums take the histogram wherever it fits, also where the recurrence is faster."""
    from crabsaxs_b200.api import Engine

    e = Engine(0)
    e.check(N.lib.crab_ctx_set_pair_variant(e.handle, HIST))
    yield e
    e.close()


def _mirrored(n, reach, rng):
    """n points in a ball of that diameter, symmetric about the origin (so the centroid is there), two of them one
    diameter apart."""
    h = rng.normal(size=(n // 2, 3))
    h *= (0.5 * reach * rng.random(n // 2) ** (1 / 3) / np.sqrt((h * h).sum(axis=1)))[:, None]
    h[0] = [reach / 2, 0.0, 0.0]
    return np.concatenate([h, -h])


def _tol(q, reach):
    """Per type pair and q, relative to Σ|w_i w_j|: bins of at most 0.0075 / q_max, and distances off by 2^-24 of the
    reach for each of the rounded coordinates and themselves (as for the histogram's tile edges)."""
    return 0.0075 ** 2 / 36.0 + 0.44 * q.max() * 2.0 ** -24 * reach * (2 * np.sqrt(3.0) + 3.0) + 1e-12


# q_max x reach / 0.005 is the number of bins: those that two 64-bit sums a bin leave in shared memory beside the
# staging (up to 11,424), its last 448 past what the counting kernel takes, then those whose sums are in device memory.
@pytest.mark.parametrize("bins", [5200, 10960, 10980, 11100, 11250, 11405, 11430, 12000, 16000, 22300])
@pytest.mark.parametrize("weights", ["few", "distinct"])
def test_loose_weights_over_the_range_of_bins(hist_engine, bins, weights):
    rng = np.random.default_rng(bins)
    reach = (0.005 * bins / 0.5 - 1e-3) / 1.0001
    xyz = _mirrored(520, reach, rng)
    w = rng.uniform(0.2, 1.0, size=520)
    if weights == "few":
        w = np.where(rng.random(520) < 0.1, 0.4, 0.75)
    t = rng.integers(0, 3, size=520)
    q = np.sort(np.concatenate([[0.0], rng.uniform(0.0, 0.5, size=60), [0.5]]))
    got, _ = cs.debye_partials(xyz, w, t, 3, q, engine=hist_engine)
    ref, _ = O.debye_partials(xyz, w, t, 3, q)
    s = np.array([w[t == a].sum() for a in range(3)])
    scale = np.array([s[a] * s[b] for a in range(3) for b in range(a, 3)])[:, None]
    assert (np.abs(got - ref) / scale).max() <= _tol(q, reach)


def _plan(engine, xyz, w, t, n_types, q):
    plan = C.c_void_p()
    xyz, w, q = (np.ascontiguousarray(v, dtype=np.float64) for v in (xyz, w, q))
    t = np.ascontiguousarray(t, dtype=np.int32)
    engine.check(N.lib.crab_pair_plan_create(engine.handle, xyz.ctypes.data_as(N.D), w.ctypes.data_as(N.D),
                                             t.ctypes.data_as(N.I32P), len(w), n_types, q.ctypes.data_as(N.D), len(q),
                                             C.byref(plan)))
    return plan


@pytest.mark.parametrize("where", ["x", "z", "w"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e39])
def test_what_is_not_finite_takes_the_recurrence(engine, where, bad):
    """A pair's bin is an address: a plan with values that have none (1e39: in FP32) is refused the histogram and made
    of the recurrence, which takes them as it always did; q = 0 is the product of the weights."""
    rng = np.random.default_rng(7)
    xyz, w, t = rng.uniform(-9.0, 9.0, size=(200, 3)), np.ones(200), np.zeros(200, dtype=int)
    if where == "w":
        w[150] = bad
    else:
        xyz[150, "xyz".index(where)] = bad
    q = np.array([0.0, 0.01, 0.2, 0.4])
    plan = _plan(engine, xyz, w, t, 1, q)
    try:
        assert N.lib.crab_pair_plan_select(engine.handle, plan, HIST) == N.EINVAL
    finally:
        N.lib.crab_pair_plan_destroy(plan)
    got, _ = cs.debye_partials(xyz, w, t, 1, q, engine=engine)
    assert got.shape == (1, 4)
    if where != "w":
        assert got[0, 0] == 200 * 199 / 2


@pytest.mark.parametrize("scale", [1e15, 1e17, 1e19, 1e21, 1e30])
def test_reach_whose_squares_leave_fp32(engine, hist_engine, scale):
    """Distances of 1e15 and more, with q_max x reach small: the histogram while the squares are FP32 numbers, refused
    beyond."""
    rng = np.random.default_rng(11)
    xyz = _mirrored(64, 2.0 * scale, rng)
    w, t = np.ones(64), np.zeros(64, dtype=int)
    q = np.linspace(0.5, 6.0, 12) / scale
    plan = _plan(engine, xyz, w, t, 1, q)
    try:
        fits = N.lib.crab_pair_plan_select(engine.handle, plan, HIST) == N.OK
    finally:
        N.lib.crab_pair_plan_destroy(plan)
    assert fits == (scale < 1e18)
    got, _ = cs.debye_partials(xyz, w, t, 1, q, engine=hist_engine)
    if fits:
        ref, _ = O.debye_partials(xyz, w, t, 1, q)
        assert np.abs(got - ref).max() / 64.0 ** 2 <= _tol(q * scale, 2.0)
    one = cs.debye_intensity(cs.Structure(xyz, np.full(64, 1, dtype=np.int8)), q, engine=engine)
    assert one.shape == q.shape


@pytest.mark.parametrize("weights", ["ones", "distinct"])
def test_allocation_failure_inside_a_change_of_kernel(weights):
    """Every allocation of a change to the histogram (and back) fails once; the plan is then as it was, refuses to run,
    or has the new kernel, and the next change works."""
    from crabsaxs_b200.api import Engine

    rng = np.random.default_rng(3)
    n, q = 400, np.linspace(0.01, 0.4, 30)
    xyz, t = rng.uniform(-10.0, 10.0, size=(n, 3)), rng.integers(0, 2, size=n)
    w = np.ones(n) if weights == "ones" else rng.uniform(0.2, 1.0, size=n)
    ref, _ = O.debye_partials(xyz, w, t, 2, q)
    s = np.array([w[t == a].sum() for a in range(2)])
    scale = np.array([s[a] * s[b] for a in range(2) for b in range(a, 2)])[:, None]

    def check(engine, plan):
        out = np.empty((3, len(q)))
        engine.check(N.lib.crab_pair_plan_run(engine.handle, plan, 1, 0, None))
        engine.check(N.lib.crab_pair_plan_read(engine.handle, plan, out.ctypes.data_as(N.D), None))
        assert (np.abs(out - ref) / scale).max() <= 96 * 2.0 ** -23  # at most 96 recurrence steps, two roundings each

    engine = Engine(0)
    engine.check(N.lib.crab_ctx_set_pair_variant(engine.handle, 64 * 16 + 2))
    for variant in (16, 96 * 16 + 2):
        for after in range(12):
            plan = _plan(engine, xyz, w, t, 2, q)
            if variant != 16:
                engine.check(N.lib.crab_pair_plan_select(engine.handle, plan, 16))
            engine.fail_allocations(after)
            status = N.lib.crab_pair_plan_select(engine.handle, plan, variant)
            engine.fail_allocations(None)
            if status == N.OK:
                break
            if N.lib.crab_pair_plan_run(engine.handle, plan, 1, 0, None) == N.OK:
                check(engine, plan)
            engine.check(N.lib.crab_pair_plan_select(engine.handle, plan, variant))
            check(engine, plan)
            N.lib.crab_pair_plan_destroy(plan)
        assert after > 0 and status == N.OK
        check(engine, plan)
        N.lib.crab_pair_plan_destroy(plan)
    engine.close()


def test_sites_and_cells_past_the_kept_slots(engine):
    """23 million sites (552 MB, their cells 276 MB): the grid's slots are above the size that a context keeps, and the
    call still reads them.  A shard without the site-site sums, against the sites themselves: the share is their last
    tiles, as many sites as the sum says near q = 0.  The call leaves no such slot behind."""
    s = cs.Structure(np.array([[3.0, -2.0, 1.0]]), np.array([1], dtype=np.int8))
    p = cs.SolventParams(shell_thickness_angstrom=176.0, hydration_model=cs.HydrationModel.Grid)
    q = np.array([1e-9, 0.004, 0.05, 0.3])
    got = cs.debye_solvent_basis(s, q, p, engine=engine, shard=(1, 2))
    held = C.c_int64()
    engine.check(N.lib.crab_ctx_workspace_bytes(engine.handle, C.byref(held)))
    few, _ = cs.hydration_grid_exterior(s, 1.0, 1.4, 3.0, engine=engine)  # releases what a call may have left
    left = C.c_int64()
    engine.check(N.lib.crab_ctx_workspace_bytes(engine.handle, C.byref(left)))
    assert held.value - left.value < 1 << 28
    sites, _ = cs.hydration_grid_exterior(s, 1.0, 1.4, 176.0, engine=engine)
    assert len(sites) > 22_400_000
    # v h sinc: the whole sum at q ~ 0 from the FP64 path's definition of both amplitudes
    site = cs.debye_solvent_basis(s, q, cs.SolventParams(hydration_model=cs.HydrationModel.Grid), engine=engine,
                                  fp64=True)
    v = np.sqrt(site[0])  # one atom: vv = v²
    r = np.sqrt(((few - s.xyz) ** 2).sum(axis=1))
    h = site[4] / (v * np.sinc(q[:, None] * r / np.pi).sum(axis=1))  # the site's amplitude
    count = got[4, 0] / (v[0] * h[0])
    assert abs(count - round(count)) <= 1e-3 and 0 < round(count) < len(sites)
    r = np.sqrt(((sites[len(sites) - round(count):] - s.xyz) ** 2).sum(axis=1))
    ref = np.array([np.sinc(k * r / np.pi).sum() for k in q])
    assert np.abs(got[4] / (v * h) - ref).max() / count <= _tol(q, 2.0 * r.max())


def _site_row(engine, s, q, p, grid):
    got = cs.debye_solvent_basis(s, q, p, engine=engine)
    ref = O.debye_solvent_basis(O.Atoms(s.xyz, s.element, s.group, s.occupancy), q, 1.0, 0.0,
                                spacing=p.hydration_grid_spacing_angstrom, model=grid)
    return np.abs(got[2] - ref[2]).max() / np.abs(ref[2]).max()


def test_lattice_refused_by_a_bound_only():
    """Two atoms 131,053 Å apart with a 4 Å shell: the cells' own squared span is 131,050 below 2^30, the span of the
    atoms' box with its shell above."""
    from crabsaxs_b200.api import Engine

    s = cs.Structure(np.array([[0.0, 0.0, 0.0], [131053.0, 0.3, -0.2]]), np.array([1, 3], dtype=np.int8))
    engine = Engine(0)
    p = cs.SolventParams(hydration_model=cs.HydrationModel.AdaptiveGrid)
    assert _site_row(engine, s, np.array([4e-4, 1.1e-3]), p, 2) <= 1e-9
    engine.close()


def _pair_counts(cells):
    """Ordered pairs per squared distance, as whole numbers (autocorrelation of the cells)."""
    cells = cells - cells.min(axis=0)
    span = cells.max(axis=0) + 1
    box = np.zeros(2 * span)
    box[tuple(cells.T)] = 1.0
    f = np.fft.rfftn(box)
    count = np.rint(np.fft.irfftn(f * f.conj(), s=box.shape, axes=(0, 1, 2))).astype(np.int64)
    axes = [np.minimum(np.arange(2 * n), 2 * n - np.arange(2 * n)) ** 2 for n in span]
    n2 = axes[0][:, None, None] + axes[1][None, :, None] + axes[2][None, None, :]
    return np.bincount(n2.ravel(), weights=count.ravel())


@pytest.mark.parametrize("side", [30.0, 43.5, 44.5, 45.5, 46.1, 54.0])
def test_lattices_about_the_shared_counters(engine, side):
    """A 1 Å shell around the corners of a cube: spans on both sides of 11,264 squared cells, by the bound and by the
    cells themselves.  Against whole numbers of pairs per distance (the oracle's running sum of 1e8 terms is itself off
    by 1e-9)."""
    p = cs.SolventParams(hydration_model=cs.HydrationModel.AdaptiveGrid, hydration_grid_spacing_angstrom=1.0)
    q = np.linspace(0.0, 0.5, 9)

    def row(xyz):
        s = cs.Structure(xyz, np.full(len(xyz), 1, dtype=np.int8))
        sites, _ = cs.hydration_grid_adaptive(s, 1.0, engine=engine)
        cells = np.rint(sites - sites[0]).astype(np.int64)
        count = _pair_counts(cells)
        r = np.sqrt(np.arange(len(count)))
        total = np.array([(count * np.sinc(k * r / np.pi)).sum() for k in q])
        return cs.debye_solvent_basis(s, q, p, engine=engine)[2] / total, (np.ptp(cells, axis=0) ** 2).sum()

    site2, _ = row(np.array([[0.37, 0.37, 0.37]]))  # a site's squared amplitude
    got, span2 = row(np.stack(np.meshgrid(*[[0.0, side]] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.37)
    assert (span2 >= 11264) == (side >= 46.0)
    assert np.abs(got / site2 - 1.0).max() <= 1e-9


@pytest.mark.parametrize("weights", ["ones", "few", "distinct"])
@pytest.mark.parametrize("n,T", [(2, 1), (31, 1), (33, 2), (64, 1), (65, 1), (127, 1), (129, 1), (257, 3), (700, 14),
                                 (300, 90)])
def test_tile_edges_on_the_histogram(hist_engine, n, T, weights):
    """The sizes of the histogram's tile edges, on the histogram whatever the choice for them is."""
    rng = np.random.default_rng(n + T)
    xyz = rng.uniform(-12.0, 12.0, size=(n, 3)) + 31.0
    w = rng.uniform(0.2, 1.0, size=n)
    if weights != "distinct":
        w = np.where((rng.random(n) < 0.1) & (weights == "few"), 0.4, 0.75)
        w[rng.random(n) < (0.05 if weights == "few" else 0.0)] = 0.0
    t = rng.integers(0, T, size=n)
    q = np.sort(np.concatenate([[0.0], rng.uniform(0.0, 0.6, size=40)]))
    got, _ = cs.debye_partials(xyz, w, t, T, q, engine=hist_engine)
    ref, _ = O.debye_partials(xyz, w, t, T, q)
    s = np.array([w[t == a].sum() for a in range(T)])
    scale = np.array([max(s[a] * s[b], 1e-12) for a in range(T) for b in range(a, T)])[:, None]
    assert (np.abs(got - ref) / scale).max() <= _tol(q, 42.0)
    parts = [cs.debye_partials(xyz, w, t, T, q, engine=hist_engine, shard=(k, 3))[0] for k in range(3)]
    assert np.abs(sum(parts) - got).max() <= 1e-12 * max(np.abs(got).max(), 1e-300)


def _launches(engine, call):
    before = engine.stats()[0]
    out = call()
    return out, engine.stats()[0] - before


@pytest.mark.parametrize("n,T,nq,weights,hist", [
    (4000, 4, 100, "ones", True), (20000, 14, 8, "ones", True), (3000, 14, 300, "distinct", True),
    (1386, 14, 8, "distinct", False), (330, 66, 17, "distinct", False), (2500, 250, 100, "ones", False),
    (960, 60, 6, "distinct", False), (9000, 250, 5, "few", False), (310, 2, 9, "distinct", False)])
def test_the_faster_kernels_are_taken(engine, n, T, nq, weights, hist):
    """Where bins cost more than pairs the recurrence runs, in one launch; shards take the same kernels as the whole."""
    rng = np.random.default_rng(n)
    R = 0.8 * n ** (1.0 / 3.0) + 4.0
    xyz, t = rng.uniform(-R, R, size=(n, 3)), np.arange(n) % T
    w = np.ones(n) if weights == "ones" else rng.uniform(0.2, 1.0, size=n)
    if weights == "few":
        w = np.where(rng.random(n) < 0.1, 0.4, 1.0)
    q = np.linspace(0.5 / nq, 0.5, nq)
    (got, _), launches = _launches(engine, lambda: cs.debye_partials(xyz, w, t, T, q, engine=engine))
    assert (launches > 1) == hist
    parts = [cs.debye_partials(xyz, w, t, T, q, engine=engine, shard=(k, 2))[0] for k in range(2)]
    assert np.abs(sum(parts) - got).max() <= 1e-12 * np.abs(got).max()


@pytest.mark.parametrize("n,nq,solvent,hist", [(2790, 2, False, False), (700, 5, False, False), (300, 200, False, True),
                                               (1500, 100, True, True), (1881, 3, True, False)])
def test_structure_calls_take_the_faster_path(engine, n, nq, solvent, hist):
    """Few q of many classes: the general path with the recurrence.  Both against the FP64 path, relative to the terms
    at q = 0 of positive amplitudes."""
    rng = np.random.default_rng(n)
    codes = [(e, -1) for e in range(1, 15)] + [(1, g) for g in range(14)]
    pick = rng.integers(0, len(codes), size=n)
    el, group = (np.array([codes[k][i] for k in pick], dtype=np.int8) for i in (0, 1))
    R = 0.9 * n ** (1.0 / 3.0) + 3.0
    xyz = rng.uniform(-R, R, size=(n, 3))
    s = cs.Structure(xyz, el, np.where(rng.random(n) < 0.1, 0.4, 1.0), group)
    q = np.linspace(0.5 / nq, 0.5, nq)
    if solvent:
        p = cs.SolventParams(c1=1.0, c2=0.7, hydration_model=cs.HydrationModel.AdaptiveGrid)
        got, launches = _launches(engine, lambda: cs.debye_solvent_basis(s, q, p, engine=engine))
        ref = cs.debye_solvent_basis(s, q, p, engine=engine, fp64=True)[0]
        top = cs.debye_solvent_basis(s, [0.0], p, engine=engine, fp64=True)[0, 0]
        got = got[0]
        assert (launches > 9) == hist
    else:
        got, launches = _launches(engine, lambda: cs.debye_intensity(s, q, engine=engine))
        p = cs.SolventParams()
        ref = cs.debye_solvent_basis(s, q, p, engine=engine, fp64=True)[0]
        top = cs.debye_solvent_basis(s, [0.0], p, engine=engine, fp64=True)[0, 0]
        assert (launches > 1) == hist
    assert np.abs(got - ref).max() / top <= 1e-5


def test_sums_that_would_not_fit_the_device(engine):
    """600 types at 22,400 bins with one odd weight: 65 GB of sums, refused before anything is allocated."""
    rng = np.random.default_rng(2)
    n, T = 1800, 600
    reach = 0.005 * 22300 / 0.5
    xyz = _mirrored(n, reach, rng)
    w, t = np.ones(n), np.arange(n) % T
    w[7] = 0.5
    q = np.array([0.01, 0.2, 0.5])
    plan = _plan(engine, xyz, w, t, T, q)
    held, after = C.c_int64(), C.c_int64()
    try:
        engine.check(N.lib.crab_ctx_workspace_bytes(engine.handle, C.byref(held)))
        assert N.lib.crab_pair_plan_select(engine.handle, plan, HIST) == N.EINVAL
        engine.check(N.lib.crab_ctx_workspace_bytes(engine.handle, C.byref(after)))
        engine.check(N.lib.crab_pair_plan_run(engine.handle, plan, 1, 0, None))
    finally:
        N.lib.crab_pair_plan_destroy(plan)
    assert after.value == held.value
    got, _ = cs.debye_partials(xyz, w, t, T, q, engine=engine)
    ref, _ = cs.debye_partials(xyz, w, t, T, q, engine=engine, fp64=True)
    assert np.abs(got - ref).max() <= 9.0 * 1e-4 and np.isfinite(got).all()  # nine pairs a row, FP32 phases q r


def test_no_room_for_the_histogram_falls_back(engine):
    """The histogram was not asked for: where its buffers cannot be had the recurrence serves, with those it has."""
    from crabsaxs_b200.api import Engine

    rng = np.random.default_rng(4)
    n, T, q = 3000, 4, np.linspace(0.005, 0.5, 200)
    xyz, t, w = rng.uniform(-15.0, 15.0, size=(n, 3)), rng.integers(0, T, size=n), np.ones(n)
    ref, launches = _launches(engine, lambda: cs.debye_partials(xyz, w, t, T, q, engine=engine)[0])
    assert launches > 1  # the histogram, where there is room
    fresh = Engine(0)
    fresh.check(N.lib.crab_ctx_set_pair_variant(fresh.handle, 100 * 16 + 7))
    rec = cs.debye_partials(xyz, w, t, T, q, engine=fresh)[0]
    fresh.check(N.lib.crab_ctx_set_pair_variant(fresh.handle, 0))
    fresh.fail_allocations(0)
    got, launches = _launches(fresh, lambda: cs.debye_partials(xyz, w, t, T, q, engine=fresh)[0])
    fresh.fail_allocations(None)
    assert launches == 1 and np.array_equal(got, rec)
    got, launches = _launches(fresh, lambda: cs.debye_partials(xyz, w, t, T, q, engine=fresh)[0])
    assert launches > 1 and np.array_equal(got, ref)
    fresh.close()


def test_autotune_that_fails_leaves_a_plan_that_works():
    from crabsaxs_b200.api import Engine, Other

    rng = np.random.default_rng(6)
    fresh = Engine(0)
    structures = [cs.Structure(rng.uniform(-9.0, 9.0, size=(150, 3)), np.full(150, 1, dtype=np.int8)) for _ in range(4)]
    q, cand = np.linspace(0.01, 0.5, 60), np.array([[1.0, 0.5]])
    c = cs.ensemble_curves(structures, q, cs.SolventParams(), cand, engine=fresh)[0]
    y, sigma = c.mean(axis=0) * 1.1 + 3.0, 0.02 * c.mean(axis=0) + 1.0
    plan = cs.EnsemblePlan(structures, q, candidates=cand, engine=fresh)
    want = plan.score(y, sigma)
    for after in (0, 1, 3, 6, 9):
        fresh.fail_allocations(after)
        with pytest.raises(Other, match="ENOMEM"):
            plan.autotune()
        fresh.fail_allocations(None)
        plan.autotune()
        got = plan.score(y, sigma)
        assert np.abs(got["kl_weights"] - want["kl_weights"]).max() <= 1e-3
        assert got["kl_reduced_chi2"] == pytest.approx(want["kl_reduced_chi2"], rel=1e-3)
    plan.close()
    fresh.close()


def test_no_room_for_a_structure_call_falls_back(engine):
    """As above for a structure's own call, whose histogram comes after its other buffers."""
    from crabsaxs_b200.api import Engine

    rng = np.random.default_rng(8)
    n, q = 900, np.linspace(0.005, 0.5, 150)
    xyz, el = rng.uniform(-12.0, 12.0, size=(n, 3)), rng.integers(1, 6, size=n).astype(np.int8)
    whole, odd = (cs.Structure(xyz, el, occ) for occ in (np.ones(n), np.where(rng.random(n) < 0.2, 0.4, 1.0)))
    fresh = Engine(0)
    fresh.check(N.lib.crab_ctx_set_pair_variant(fresh.handle, 150 * 16 + 6))
    rec = cs.debye_intensity(odd, q, engine=fresh)
    fresh.check(N.lib.crab_ctx_set_pair_variant(fresh.handle, 0))
    ref = cs.debye_intensity(whole, q, engine=fresh)
    fresh.fail_allocations(0)
    got, launches = _launches(fresh, lambda: cs.debye_intensity(odd, q, engine=fresh))
    assert launches == 1 and np.array_equal(got, rec)
    assert np.array_equal(cs.debye_intensity(whole, q, engine=fresh), ref)
    fresh.fail_allocations(None)
    got, launches = _launches(fresh, lambda: cs.debye_intensity(odd, q, engine=fresh))
    assert launches > 1 and np.array_equal(got, cs.debye_intensity(odd, q, engine=engine))
    fresh.close()


def test_offsets_of_one_bin_at_their_largest(hist_engine):
    """Two clusters of 18,000 coincident atoms 4,088.4999 bins apart: every pair between them adds the largest positive
    offset to one bin, and every CTA counts whole runs of such pairs between two flushes.  Against sinc itself; the
    tolerance is that of the histogram's tile edges (4,096 bins over the reach)."""
    n, d = 18000, 1.32246
    xyz = np.zeros((2 * n, 3))
    xyz[0::2, 0], xyz[1::2, 0] = -d / 2, d / 2
    t = np.arange(2 * n) % 2
    q = np.linspace(0.5, 12.0, 24)
    got, _ = cs.debye_partials(xyz, np.ones(2 * n), t, 2, q, engine=hist_engine)
    sinc = np.sinc(q * d / np.pi)
    tol = (12.0 * d / 4000.0) ** 2 / 36.0 + 0.44 * 12.0 * 2.0 ** -24 * d * (2 * np.sqrt(3.0) + 3.0) + 1e-12
    assert np.abs(got[1] / n ** 2 - sinc).max() <= tol
    assert np.abs(got[0] / (0.5 * n * (n - 1)) - 1.0).max() <= tol


def test_large_sums_are_given_back():
    """140 types with weights of their own at 12,000 bins: 3.8 GB of sums, which a one-shot call does not leave behind;
    the next calls are the same to the bit."""
    from crabsaxs_b200.api import Engine

    rng = np.random.default_rng(12)
    n, T = 3000, 140
    xyz, t = _mirrored(n, 119.0, rng), np.arange(n) % T
    w, q = rng.uniform(0.2, 1.0, size=n), np.linspace(0.1, 0.5, 8)
    fresh = Engine(0)
    fresh.check(N.lib.crab_ctx_set_pair_variant(fresh.handle, HIST))
    (got, _), launches = _launches(fresh, lambda: cs.debye_partials(xyz, w, t, T, q, engine=fresh))
    assert launches > 1
    held = C.c_int64()
    fresh.check(N.lib.crab_ctx_workspace_bytes(fresh.handle, C.byref(held)))
    assert held.value < 1 << 29
    assert np.array_equal(cs.debye_partials(xyz, w, t, T, q, engine=fresh)[0], got)
    ref, _ = cs.debye_partials(xyz, w, t, T, q, engine=fresh, fp64=True)
    assert np.abs(got - ref).max() <= 22.0 ** 2 * _tol(q, 119.0)
    fresh.close()


def test_sites_of_a_size_query_outlive_calls_without_a_grid(engine):
    """A size query leaves its sites on the device (12 million, above the kept slots) for the fill call that follows;
    calls in between that build no grid leave them alone, one that builds a grid makes the fill call build again."""
    one = cs.Structure(np.array([[1.0, 2.0, 3.0]]), np.array([1], dtype=np.int8))
    other = cs.Structure(np.random.default_rng(0).uniform(-9.0, 9.0, size=(300, 3)), np.full(300, 2, dtype=np.int8))
    args = (1.0, 1.4, 142.0)
    want, _ = cs.hydration_grid_exterior(one, *args, engine=engine)
    assert len(want) * 24 > 1 << 28
    q = np.linspace(0.01, 0.4, 40)
    plain, grid = cs.SolventParams(), cs.SolventParams(hydration_model=cs.HydrationModel.AdaptiveGrid)
    between = [lambda: None, lambda: cs.debye_solvent_basis(other, q, plain, engine=engine),
               lambda: cs.debye_intensity(other, q, engine=engine),
               lambda: cs.multipole_solvent_basis(other, q, 12, plain, engine=engine),
               lambda: cs.debye_solvent_basis(other, q, grid, engine=engine)]
    h = one.handle(engine)
    for call in between:
        m, vol = C.c_int64(), C.c_double()
        engine.check(N.lib.crab_hydration_grid_exterior(engine.handle, h, *args, None, 0, C.byref(m), C.byref(vol)))
        call()
        got = np.empty((m.value, 3))
        engine.check(N.lib.crab_hydration_grid_exterior(engine.handle, h, *args, got.ctypes.data_as(N.D), m.value,
                                                        C.byref(m), C.byref(vol)))
        assert np.array_equal(got, want)


def test_a_shard_without_room_does_not_fall_back():
    """Shards split the pairs of the two kernels differently: one that falls back alone would leave the sum wrong."""
    from crabsaxs_b200.api import Engine, Other

    rng = np.random.default_rng(14)
    n, T, q = 3000, 4, np.linspace(0.005, 0.5, 200)
    xyz, t, w = rng.uniform(-15.0, 15.0, size=(n, 3)), rng.integers(0, T, size=n), np.ones(n)
    el = rng.integers(1, 6, size=n).astype(np.int8)
    whole, odd = (cs.Structure(xyz, el, occ) for occ in (w, np.where(rng.random(n) < 0.2, 0.4, 1.0)))
    fresh = Engine(0)
    fresh.check(N.lib.crab_ctx_set_pair_variant(fresh.handle, 100 * 16 + 7))
    cs.debye_partials(xyz, w, t, T, q, engine=fresh, shard=(0, 2))  # the recurrence's buffers
    cs.debye_solvent_basis(odd, q, cs.SolventParams(), engine=fresh, shard=(0, 2))
    fresh.check(N.lib.crab_ctx_set_pair_variant(fresh.handle, 0))
    fresh.fail_allocations(0)
    with pytest.raises(Other, match="ENOMEM"):
        cs.debye_partials(xyz, w, t, T, q, engine=fresh, shard=(0, 2))
    fresh.fail_allocations(None)
    cs.debye_solvent_basis(whole, q, cs.SolventParams(), engine=fresh, shard=(0, 2))
    fresh.fail_allocations(0)
    with pytest.raises(Other, match="ENOMEM"):
        cs.debye_solvent_basis(odd, q, cs.SolventParams(), engine=fresh, shard=(0, 2))
    fresh.close()
