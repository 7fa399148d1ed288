"""The distance-histogram Debye kernels at the edges of their tiles, bins and weights.

Tolerance, per type pair and q, relative to Σ|w_i w_j| (no pair's sinc exceeds one): a straight line over a bin of
width h leaves at most (q h)²/12 |sinc''| with |sinc''| <= 1/3, and an FP32 distance is off by at most the rounding of
two centred coordinates in three axes and its own, 2^-24 R (2 sqrt(3) + 3), times q |sinc'| <= 0.44 q.
"""
import numpy as np
import pytest

import crabsaxs_b200 as cs
import oracle as O
from crabsaxs_b200 import _native as N

pytestmark = pytest.mark.gpu

HIST = 16  # the histogram's variant code


def _bound(xyz, q):
    c = xyz - xyz.mean(axis=0)
    reach = 2.0 * np.sqrt((c * c).sum(axis=1).max()) * 1.0001 + 1e-3
    h = reach / 4000.0 if q.max() * reach <= 20.0 else 0.0075 / q.max()
    return (q.max() * h) ** 2 / 36.0 + 0.44 * q.max() * 2.0 ** -24 * reach * (2 * np.sqrt(3.0) + 3.0) + 1e-12


def _weights(kind, n, rng):
    if kind == "ones":
        return np.ones(n)
    if kind == "few":  # a few atoms off the commonest weight, some without any, some negative
        w = np.full(n, 0.75)
        w[rng.random(n) < 0.1] = 0.4
        w[rng.random(n) < 0.05] = 0.0
        w[rng.random(n) < 0.05] = -0.3
        return w
    return rng.uniform(0.2, 1.0, size=n)


@pytest.mark.parametrize("weights", ["ones", "few", "distinct"])
@pytest.mark.parametrize("n,T", [(2, 1), (31, 1), (33, 2), (64, 1), (65, 1), (127, 1), (129, 1), (257, 3), (700, 14)])
def test_tile_edges_match_the_oracle(engine, n, T, weights):
    rng = np.random.default_rng(n + T)
    xyz = rng.uniform(-12.0, 12.0, size=(n, 3)) + 31.0
    w, t = _weights(weights, n, rng), rng.integers(0, T, size=n)
    q = np.sort(np.concatenate([[0.0], rng.uniform(0.0, 0.6, size=40)]))
    got, _ = cs.debye_partials(xyz, w, t, T, q, engine=engine)
    ref, _ = O.debye_partials(xyz, w, t, T, q)
    s = np.array([np.abs(w[t == a]).sum() for a in range(T)])
    scale = np.array([max(s[a] * s[b], 1e-12) for a in range(T) for b in range(a, T)])[:, None]
    assert (np.abs(got - ref) / scale).max() <= _bound(xyz, q)
    again, _ = cs.debye_partials(xyz, w, t, T, q, engine=engine)
    assert np.array_equal(again, got)
    parts = [cs.debye_partials(xyz, w, t, T, q, engine=engine, shard=(k, 3))[0] for k in range(3)]
    assert np.abs(sum(parts) - got).max() <= 1e-12 * max(np.abs(got).max(), 1e-300)


@pytest.mark.parametrize("reach", [20.0, 215.0, 330.0, 345.0, 3000.0])
def test_bins_from_the_smallest_to_past_the_largest(engine, reach):
    """q_max x reach from 10 to 1500: the smallest histogram, the largest, coarser steps, and beyond 168 the
    recurrence; plus coincident atoms and atoms exactly one reach apart."""
    rng = np.random.default_rng(int(reach))
    xyz = rng.normal(size=(300, 3))
    xyz *= (0.5 * reach * rng.random(300) ** (1 / 3) / np.sqrt((xyz ** 2).sum(axis=1)))[:, None]
    xyz[0], xyz[1] = [reach / 2, 0, 0], [-reach / 2, 0, 0]
    xyz[2] = xyz[3]
    q = np.linspace(0.001, 0.5, 120)
    w, t = np.ones(300), np.zeros(300, dtype=int)
    got, _ = cs.debye_partials(xyz, w, t, 1, q, engine=engine)
    ref, _ = O.debye_partials(xyz, w, t, 1, q)
    tol = _bound(xyz, q) if reach < 340 else 2e-6 + 0.44 * 0.5 * 2.0 ** -24 * reach * 8
    assert np.abs(got - ref).max() / 300.0 ** 2 <= tol


def test_select_refuses_bins_that_do_not_fit(engine):
    import ctypes as C

    xyz = np.array([[0.0, 0, 0], [3000.0, 0, 0], [10.0, 0, 0]])
    q, w, t = np.linspace(0.01, 0.5, 20), np.ones(3), np.zeros(3, dtype=np.int32)
    plan = C.c_void_p()
    engine.check(N.lib.crab_pair_plan_create(engine.handle, xyz.ctypes.data_as(N.D), w.ctypes.data_as(N.D),
                                             t.ctypes.data_as(N.I32P), 3, 1, q.ctypes.data_as(N.D), len(q),
                                             C.byref(plan)))
    try:
        assert N.lib.crab_pair_plan_select(engine.handle, plan, HIST) == N.EINVAL
        engine.check(N.lib.crab_pair_plan_run(engine.handle, plan, 1, 0, None))
    finally:
        N.lib.crab_pair_plan_destroy(plan)


def _occupancy(kind, n, rng):
    occ = np.ones(n)
    if kind == "altloc":
        at = rng.random(n) < 0.1
        occ[at] = np.round(rng.uniform(0.3, 0.7, size=int(at.sum())), 2)
    elif kind == "odd first":  # every class's first atom has a weight of its own, some atoms none, some negative
        occ[:] = 0.8
        occ[:40] = rng.uniform(0.1, 0.5, size=min(40, n))
        occ[rng.random(n) < 0.05] = 0.0
        occ[rng.random(n) < 0.02] = -0.4
    elif kind == "distinct":
        occ = rng.uniform(0.2, 1.0, size=n)
    return occ


@pytest.mark.parametrize("hydration", [cs.HydrationModel.Analytic, cs.HydrationModel.AdaptiveGrid,
                                       cs.HydrationModel.Grid])
@pytest.mark.parametrize("kind", ["ones", "altloc", "odd first", "distinct"])
@pytest.mark.parametrize("n,implicit", [(1, True), (129, True), (700, False)])
def test_structure_calls_match_the_fp64_path(engine, n, implicit, kind, hydration):
    """The one-structure calls type, place and recombine on the device; the FP64 option keeps the general path.  Terms
    relative to their q = 0 value with all occupancies positive, which bounds every |X_i Y_j| sum."""
    rng = np.random.default_rng(n)
    xyz = rng.uniform(-11.0, 11.0, size=(n, 3)) - 40.0
    el = rng.choice([0, 1, 2, 3, 4, 14], size=n, p=[0.1, 0.5, 0.15, 0.15, 0.05, 0.05]).astype(np.int8)
    group = np.where(el == 1, rng.integers(-1, 4, size=n), np.where(el == 2, 7, -1)).astype(np.int8)
    occ = _occupancy(kind, n, rng)
    s = cs.Structure(xyz, el, occ, group)
    p = cs.SolventParams(c1=1.02, c2=0.9, hydration_model=hydration)
    q = np.concatenate([[0.0], np.linspace(0.004, 0.45, 45)])
    got = cs.debye_solvent_basis(s, q, p, implicit, engine=engine)
    ref = cs.debye_solvent_basis(s, q, p, implicit, engine=engine, fp64=True)
    top = cs.debye_solvent_basis(cs.Structure(xyz, el, np.abs(occ), group), [0.0], p, implicit, engine=engine, fp64=True)
    shell = np.concatenate([xyz - 14.0, xyz + 14.0])  # reach of the sites
    tol = _bound(shell if hydration != cs.HydrationModel.Analytic else xyz, q)
    assert (np.abs(got - ref) / np.maximum(np.abs(top), 1e-9)).max() <= tol
    parts = [cs.debye_solvent_basis(s, q, p, implicit, engine=engine, shard=(k, 3)) for k in range(3)]
    assert np.abs(sum(parts) - got).max() <= 1e-12 * np.abs(got).max()
    assert np.array_equal(cs.debye_solvent_basis(s, q, p, implicit, engine=engine), got)
    vac = cs.debye_intensity(s, q, implicit, engine=engine)
    v = ref[0]
    if hydration == cs.HydrationModel.Analytic:
        assert (np.abs(vac - np.maximum(v, 0.0)) / max(abs(top[0, 0]), 1e-9)).max() <= tol
