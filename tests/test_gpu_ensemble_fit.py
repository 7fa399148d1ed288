"""The ensemble's weight fit and KL reweighting at the sizes where their kernels change form: one conformer, whole and
ragged warps, the counting sort (up to 128) against the network, curves in and out of shared memory, one CTA against a
cluster, and q grids too long for the per-q tables.

The test restates one step's outcome from the returned weights in f64: χ², its gradient in the weights, and the KL
objective's stationarity.  Sums of m f64 terms in another order differ by at most m 2^-53 of their absolute sum, and
the fit of scale and background passes that on with the conditioning of a 2 x 2 system: 1e-9 leaves a factor 1e4.
"""
import numpy as np
import pytest

import crabsaxs_b200 as cs

pytestmark = pytest.mark.gpu


def _conformers(k, rng):
    out = []
    for _ in range(k):
        n = int(rng.integers(8, 20))
        out.append(cs.Structure(rng.uniform(-6.0, 6.0, size=(n, 3)) * rng.uniform(0.6, 1.6),
                                rng.choice([1, 2, 3], size=n).astype(np.int8)))
    return out


@pytest.mark.parametrize("k,nq", [(1, 20), (2, 33), (31, 64), (33, 300), (88, 300), (90, 300), (128, 40), (129, 40), (200, 300), (300, 500),
                                  (1024, 40), (40, 3300), (1024, 3300)])
def test_fit_and_reweighting_are_consistent(engine, k, nq):
    rng = np.random.default_rng(1000 * k + nq)
    structures = _conformers(k, rng)
    q = np.linspace(0.01, 0.5, nq)
    cand = np.array([[1.0, 0.5], [1.02, 1.5]])
    sol = cs.SolventParams()
    curves = cs.ensemble_curves(structures, q, sol, cand, engine=engine)
    true = rng.dirichlet(np.full(k, 0.3))
    y = 2.0 * (true @ curves[1]) + 0.01 * curves[1].mean()
    sigma = 0.02 * y + 1e-3 * y.max()
    y = y + sigma * rng.normal(size=nq)
    plan = cs.EnsemblePlan(structures, q, solvent=sol, candidates=cand, engine=engine)
    try:
        r = plan.score(y, sigma)
        again = plan.score(y, sigma)
    finally:
        plan.close()
    assert np.array_equal(r["weights"], again["weights"]) and np.array_equal(r["kl_weights"], again["kl_weights"])
    c, w, dof = curves[r["candidate"]], r["weights"], max(nq - 1, 1)
    assert w.min() >= 0.0 and abs(w.sum() - 1.0) <= 1e-12 * k
    res = (r["scale"] * (w @ c) + r["background"] - y) / sigma
    assert r["reduced_chi2"] == pytest.approx((res ** 2).sum() / dof, rel=1e-9)
    terms = 2.0 * res * r["scale"] * c / sigma / dof
    assert np.abs(r["dchi2_dw"] - terms.sum(axis=1)).max() <= 1e-9 * np.abs(terms).sum(axis=1).max()
    v = r["kl_weights"]
    assert v.min() > 0.0 and abs(v.sum() - 1.0) <= 1e-9
    res = (r["kl_scale"] * (v @ c) + r["kl_background"] - y) / sigma
    assert r["kl_reduced_chi2"] == pytest.approx((res ** 2).sum() / dof, rel=1e-9)
    assert r["kl_divergence"] == pytest.approx((v * np.log(v * k)).sum(), abs=1e-9)
    # descent from the uniform start: the objective is no higher there
    u = np.full(k, 1.0 / k)
    A = np.stack([u @ c, np.ones(nq)], axis=1) / sigma[:, None]
    s0, b0 = np.linalg.lstsq(A, y / sigma, rcond=None)[0]
    start = (((max(s0, 0.0) * (u @ c) + b0 - y) / sigma) ** 2).sum() / dof
    assert r["kl_reduced_chi2"] + r["kl_divergence"] <= start * (1 + 1e-9) + 1e-9
