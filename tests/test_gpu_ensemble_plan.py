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
