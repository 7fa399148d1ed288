"""An ensemble plan called again: its captured graph against the options and limits of every call."""
import numpy as np
import pytest

import crabsaxs_b200 as cs

pytestmark = pytest.mark.gpu


def _ensemble(k, nq, rng):
    structures = []
    for _ in range(k):
        n = int(rng.integers(20, 60))
        structures.append(cs.Structure(rng.uniform(-8.0, 8.0, size=(n, 3)) * rng.uniform(0.7, 1.5),
                                       rng.choice([1, 2, 3], size=n).astype(np.int8)))
    return structures, np.linspace(0.01, 0.5, nq), np.array([[1.0, 0.5], [1.02, 1.5], [0.98, -0.4]])


def _observed(structures, q, cand, rng, engine):
    curves = cs.ensemble_curves(structures, q, cs.SolventParams(), cand, engine=engine)
    y = 1.7 * (rng.dirichlet(np.full(len(structures), 0.3)) @ curves[1]) + 0.02 * curves[1].mean()
    sigma = 0.02 * y + 1e-3 * y.max()
    return y + sigma * rng.normal(size=len(q)), sigma


def _equal(a, b):
    return all(np.array_equal(a[k], b[k]) for k in a if k != "elapsed_ms")


Fixed, Bg, Me, Fit = cs.ScaleMode.Fixed, cs.BackgroundMode, cs.MaximumEntropyOptions, cs.FitOptions


@pytest.mark.parametrize("other", [
    dict(fit=Fit(scale_mode=Fixed(0.9))),
    dict(fit=Fit(background_mode=Bg.FixedZero)),
    dict(fit=Fit(background_mode=Bg.Fixed(40.0))),
    dict(reweight=Me(kl_strength=7.0)),
    dict(reweight=Me(step_size=0.05, max_iterations=20)),
    dict(reweight=Me(max_iterations=3)),
    dict(reweight=Me(tolerance=0.2)),
    dict(reweight=Me(min_weight=0.05)),
    dict(reweight=Me(fit=Fit(scale_mode=Fixed(1.2)))),
    dict(reweight=Me(fit=Fit(background_mode=Bg.Fixed(25.0)))),
])
def test_every_call_has_its_own_options(engine, other):
    """One plan with the default options, others, and the defaults again: each equal to a fresh plan's to the bit."""
    rng = np.random.default_rng(21)
    structures, q, cand = _ensemble(7, 60, rng)
    y, sigma = _observed(structures, q, cand, rng, engine)

    def fresh(**options):
        plan = cs.EnsemblePlan(structures, q, candidates=cand, engine=engine)
        try:
            return plan.score(y, sigma, **options)
        finally:
            plan.close()

    base, changed = fresh(), fresh(**other)
    assert not _equal(base, changed)
    plan = cs.EnsemblePlan(structures, q, candidates=cand, engine=engine)
    try:
        got = [plan.score(y, sigma), plan.score(y, sigma, **other), plan.score(y, sigma, **other),
               plan.score(y, sigma)]
    finally:
        plan.close()
    for g, want in zip(got, [base, changed, changed, base]):
        assert _equal(g, want)


@pytest.mark.parametrize("variant", [0, 16])
def test_wait_that_runs_out_is_reported_by_every_ensemble_call(engine, variant):
    """The pair kernel's bounded wait shortened to nothing, for the plan's own kernel and the distance histogram: the
    calls report it instead of returning what incomplete sums give, and the context goes on."""
    from crabsaxs_b200 import _native as N
    from crabsaxs_b200.api import Engine, Other

    rng = np.random.default_rng(5)
    structures, q, cand = _ensemble(5, 50, rng)
    y, sigma = _observed(structures, q, cand, rng, engine)
    exp = cs.ExperimentalCurve(q, y, sigma)
    fresh = Engine(0)
    fresh.check(N.lib.crab_ctx_set_pair_variant(fresh.handle, variant))
    plan = cs.EnsemblePlan(structures, q, candidates=cand, engine=fresh)
    fitter = cs.EnsembleFitter(structures, [str(k) for k in range(5)], exp, engine=fresh)
    calls = [lambda: plan.score(y, sigma), fitter.fit,
             lambda: cs.ensemble_curves(structures, q, cs.SolventParams(), cand, engine=fresh)]
    before = [calls[0](), calls[1]().weights, calls[2]()]
    fresh.set_wait_budget(0)
    for call in calls:
        for _ in range(2):
            with pytest.raises(Other, match="ETIMEOUT"):
                call()
    fresh.set_wait_budget(None)
    assert _equal(calls[0](), before[0])
    assert np.array_equal(calls[1]().weights, before[1]) and np.array_equal(calls[2](), before[2])
    plan.close()
    fresh.close()


def _uneven(k, classes, rng, loose):
    """Conformers of one atom to several tiles, of extents 4 to 120 Å, each with some of the classes."""
    out = []
    for c in range(k):
        n = [1, 2, 127, 128, 129, 400][c % 6] + int(rng.integers(0, 3))
        el = rng.integers(1, 15, size=n).astype(np.int8) if classes > 4 else rng.integers(1, 5, size=n).astype(np.int8)
        group = np.where(el == 1, rng.integers(-1, 4, size=n), -1).astype(np.int8)
        occ = np.ones(n)
        if loose:
            occ[rng.random(n) < 0.2] = 0.35
            occ[rng.random(n) < 0.05] = 0.0
        out.append(cs.Structure(rng.uniform(-1.0, 1.0, size=(n, 3)) * [2.0, 15.0, 60.0][c % 3], el, occ, group))
    return out


@pytest.mark.parametrize("k,classes,loose", [(1, 4, False), (6, 4, True), (7, 14, False), (48, 14, False),
                                             (13, 14, True)])
def test_histogram_of_many_structures(engine, k, classes, loose):
    """The distance histogram of a whole ensemble (variant 16, chosen before the plan is made): every structure has its
    own bins, rows are resident in groups of 96 MB (48 conformers of 17 classes: several), and a structure may lack
    classes.  Against the FP64 path of each conformer, relative to its curve at q = 0 with positive amplitudes: bins of
    at most 0.0075 / q_max leave 0.0075² / 36, FP32 distances 2^-24 of the reach."""
    from crabsaxs_b200 import _native as N
    from crabsaxs_b200.api import Engine

    rng = np.random.default_rng(100 + k)
    structures = _uneven(k, classes, rng, loose)
    q = np.concatenate([[0.0], np.linspace(0.01, 0.5, 40)])
    cand = np.array([[1.0, 0.0], [1.03, 0.8]])
    hist = Engine(0)
    hist.check(N.lib.crab_ctx_set_pair_variant(hist.handle, 16))
    got = cs.ensemble_curves(structures, q, cs.SolventParams(), cand, engine=hist)
    again = cs.ensemble_curves(structures, q, cs.SolventParams(), cand, engine=hist)
    rec = cs.ensemble_curves(structures, q, cs.SolventParams(), cand, engine=engine)
    assert np.array_equal(got, again)
    for c, s in enumerate(structures):
        reach = 2.0 * np.sqrt(((s.xyz - s.xyz.mean(axis=0)) ** 2).sum(axis=1).max()) + 1e-3
        tol = 0.0075 ** 2 / 36.0 + 0.44 * 0.5 * 2.0 ** -24 * reach * (2 * np.sqrt(3.0) + 3.0) + 1e-12
        b = cs.debye_solvent_basis(s, q, cs.SolventParams(), True, engine=engine, fp64=True)
        top = cs.debye_solvent_basis(s, [0.0], cs.SolventParams(), True, engine=engine, fp64=True)[:, 0]
        for i, (c1, c2) in enumerate(cand):
            ref = cs.combine_solvent_basis(b, q, c1, c2)
            parts = [1.0, 1.3, c2 * c2, 2.3, 2.3 * c2, 2.3 * c2]
            scale = max(float(np.abs(top) @ parts), 1e-9)
            assert np.abs(got[i, c] - ref).max() / scale <= tol, (c, i)
            assert np.abs(rec[i, c] - ref).max() / scale <= 168 * 2.0 ** -23 + tol, (c, i)
    hist.close()


@pytest.mark.parametrize("k,nq", [(33, 800), (32, 800), (20, 1200), (50, 520), (1000, 20), (300, 40), (513, 9)])
def test_forms_of_the_reweighting(engine, k, nq):
    """One CTA, eight that search step lengths and eight that split the curves, about the lines between them and with
    threads by the curves instead of the q: the outcome restated from the weights in f64 (1e-9, as the fit's test)."""
    rng = np.random.default_rng(k + nq)
    structures = [cs.Structure(rng.uniform(-6.0, 6.0, size=(9, 3)) * rng.uniform(0.6, 1.6),
                               rng.choice([1, 2, 3], size=9).astype(np.int8)) for _ in range(k)]
    q, cand = np.linspace(0.01, 0.5, nq), np.array([[1.0, 0.5]])
    c = cs.ensemble_curves(structures, q, cs.SolventParams(), cand, engine=engine)[0]
    y = 1.3 * (rng.dirichlet(np.full(k, 0.3)) @ c)
    sigma = 0.02 * y + 1e-3 * y.max()
    y = y + sigma * rng.normal(size=nq)
    plan = cs.EnsemblePlan(structures, q, candidates=cand, engine=engine)
    try:
        r, again = plan.score(y, sigma), plan.score(y, sigma)
    finally:
        plan.close()
    assert _equal(r, again)
    v = r["kl_weights"]
    assert v.min() > 0.0 and abs(v.sum() - 1.0) <= 1e-9
    res = (r["kl_scale"] * (v @ c) + r["kl_background"] - y) / sigma
    assert r["kl_reduced_chi2"] == pytest.approx((res ** 2).sum() / (nq - 1), rel=1e-9)
    assert r["kl_divergence"] == pytest.approx((v * np.log(v * k)).sum(), abs=1e-9)
