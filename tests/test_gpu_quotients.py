"""Quotients by a reciprocal (the ensemble weight fit's gradient terms) against the division, to the bit."""
import numpy as np
import pytest

import crabsaxs_b200 as cs
from crabsaxs_b200 import _native as N

pytestmark = pytest.mark.gpu


def _check(engine, a, b):
    a, b = (np.ascontiguousarray(v, dtype=np.float64) for v in (a, b))
    by, div = np.empty_like(a), np.empty_like(a)
    engine.check(N.lib.crab_probe_quotients(engine.handle, *(v.ctypes.data_as(N.D) for v in (a, b)), len(a),
                                            *(v.ctypes.data_as(N.D) for v in (by, div))))
    zero = a == 0.0
    assert np.all(by[zero] == 0.0)
    assert np.array_equal(by[~zero].view(np.uint64), div[~zero].view(np.uint64))
    with np.errstate(all="ignore"):
        assert np.array_equal(div[~zero].view(np.uint64), (a / b)[~zero].view(np.uint64))


def _doubles(rng, n, lo, hi, ends):
    """Exponents lo .. hi, mantissas random or (ends) within 64 of either end."""
    m = rng.integers(0, 1 << 52, size=n, dtype=np.uint64)
    if ends:
        near = rng.integers(0, 64, size=n, dtype=np.uint64)
        m = np.where(rng.random(n) < 0.5, near, np.uint64((1 << 52) - 1) - near)
    e = rng.integers(lo + 1023, hi + 1024, size=n).astype(np.uint64)
    return (e << np.uint64(52) | m).view(np.float64)


@pytest.mark.parametrize("ends_a", [False, True])
@pytest.mark.parametrize("ends_b", [False, True])
@pytest.mark.parametrize("lo,hi", [(-10, 10), (-482, -478), (478, 482), (-480, 480), (-1022, 1023)])
def test_equal_to_the_division(engine, lo, hi, ends_a, ends_b):
    rng = np.random.default_rng(abs(lo) + 2 * ends_a + ends_b)
    a = _doubles(rng, 400_000, lo, hi, ends_a) * rng.choice([-1.0, 1.0], size=400_000)
    for b_lo, b_hi in ((-8, 8), (-332, -328), (328, 331), (-332, 331)):  # 1e-100 = 2^-332.2, 1e100 = 2^332.2
        _check(engine, a, _doubles(rng, len(a), b_lo, b_hi, ends_b))


def test_values_outside_the_range(engine):
    a = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** -1022, 1.7976931348623157e308,
                  2.0 ** -481, 2.0 ** -480, 2.0 ** 480, 2.0 ** 481, np.nextafter(2.0 ** 481, 0.0)])
    b = np.array([1e-100, 1.0, 3.0, 0.1, 1e100, np.nextafter(2.0, 1.0), np.nextafter(1.0, 2.0)])
    _check(engine, np.repeat(a, len(b)), np.tile(b, len(a)))


def test_a_sigma_outside_the_range_takes_the_division(engine):
    """One sigma past 1e100 switches the fit to plain quotients: its outcome restated in f64."""
    rng = np.random.default_rng(3)
    structures = [cs.Structure(rng.uniform(-6.0, 6.0, size=(12, 3)) * rng.uniform(0.6, 1.6),
                               rng.choice([1, 2, 3], size=12).astype(np.int8)) for _ in range(9)]
    q, cand = np.linspace(0.01, 0.5, 40), np.array([[1.0, 0.5]])
    c = cs.ensemble_curves(structures, q, cs.SolventParams(), cand, engine=engine)[0]
    y = 1.3 * (rng.dirichlet(np.full(9, 0.3)) @ c)
    sg = 0.02 * y + 1.0
    y = y + sg * rng.normal(size=40)
    sg[17] = 1e101
    plan = cs.EnsemblePlan(structures, q, candidates=cand, engine=engine)
    try:
        r = plan.score(y, sg)
    finally:
        plan.close()
    w = r["weights"]
    assert w.min() >= 0.0 and abs(w.sum() - 1.0) <= 1e-11
    res = (r["scale"] * (w @ c) + r["background"] - y) / sg
    assert r["reduced_chi2"] == pytest.approx((res ** 2).sum() / 39, rel=1e-9)
    terms = 2.0 * res * r["scale"] * c / sg / 39
    assert np.abs(r["dchi2_dw"] - terms.sum(axis=1)).max() <= 1e-9 * np.abs(terms).sum(axis=1).max()
