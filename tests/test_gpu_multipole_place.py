"""Multipole points placed on the device from one word per atom: atoms that a
hydrogen option drops, united-atom groups, zero and fractional occupancies, hydration sites,
few and many q (one and four q a lane in the q pass), no atom left, and items
of the moment GEMM cut to fill several rounds of the SMs.  The oracle's f64
sums are the reference: 1e-9 relative for the FP64 path and 1e-5 for the
default one, basis terms relative to each term's largest magnitude."""
import numpy as np
import pytest

import crabsaxs_b200 as cs
import oracle as O
from crabsaxs_b200 import _native as N
from crabsaxs_b200 import synth

pytestmark = pytest.mark.gpu


def _mixed(seed, n):
    rng = np.random.default_rng(seed)
    s = synth.protein(seed, n, 4.0 + 1.2 * n ** (1.0 / 3.0))
    el = rng.integers(0, 14, n).astype(np.int8)
    occ = rng.choice([1.0, 1.0, 1.0, 0.5, 0.0], n)
    return cs.Structure(s.xyz, el, occ, rng.integers(-1, 4, n).astype(np.int8))


def _atoms(s):
    return O.Atoms(s.xyz, s.element, s.group, s.occupancy)


@pytest.mark.parametrize("implicit", [True, False])
@pytest.mark.parametrize("n,nq,l_max", [(1, 3, 4), (31, 40, 0), (257, 7, 15), (700, 600, 20)])
def test_mixed_atoms_match_oracle(engine, n, nq, l_max, implicit):
    s = _mixed(n, n)
    q = np.linspace(0.0, 0.6, nq)
    ref = O.multipole_intensity(_atoms(s), q, l_max, implicit)
    scale = np.maximum(np.abs(ref), 1e-12)
    for prec, tol in ((N.PREC_FP64, 1e-9), (N.PREC_TF32_SPLIT, 1e-5)):
        got = cs.multipole_intensity(s, q, l_max, implicit, precision=prec, engine=engine)
        assert np.max(np.abs(got - ref) / scale) <= tol, prec


@pytest.mark.parametrize("model,spacing", [(0, 4.0), (1, 3.0)])
@pytest.mark.parametrize("n,nq", [(40, 5), (900, 300)])
def test_basis_with_and_without_sites_matches_oracle(engine, n, nq, model, spacing):
    s = _mixed(n + 1, n)
    q = np.linspace(0.001, 0.5, nq)
    p = cs.SolventParams(c1=1.02, c2=0.8, hydration_model=cs.HydrationModel(model),
                         hydration_grid_spacing_angstrom=spacing)
    ref = O.multipole_solvent_basis(_atoms(s), q, 18, p.c1, p.c2, model=model, spacing=spacing)
    for prec, tol in ((N.PREC_FP64, 1e-9), (N.PREC_TF32_SPLIT, 1e-5)):
        got = cs.multipole_solvent_basis(s, q, 18, p, precision=prec, engine=engine)
        for k in range(6):
            assert np.max(np.abs(got[k] - ref[k])) <= tol * max(np.max(np.abs(ref[k])), 1e-12), (prec, k)


def test_only_dropped_atoms(engine):
    s = cs.Structure(np.arange(9.0).reshape(3, 3), [0, 0, 0])
    q = np.array([0.0, 0.1, 0.5])
    ref = O.multipole_intensity(_atoms(s), q, 10, True)
    got = cs.multipole_intensity(s, q, 10, True, engine=engine)
    assert np.allclose(got, ref, rtol=1e-5, atol=1e-12)


def test_gemm_items_over_several_rounds(engine):
    s = synth.protein(77, 33000, 44.0)
    q = np.array([0.05, 0.2, 0.45])
    ref = O.multipole_intensity(_atoms(s), q, 50)
    for prec, tol in ((N.PREC_FP64, 1e-9), (N.PREC_TF32_SPLIT, 1e-5)):
        got = cs.multipole_intensity(s, q, 50, precision=prec, engine=engine)
        assert np.max(np.abs(got - ref) / np.abs(ref)) <= tol


def _general(call, *args, **kw):
    """The general path's result: two ranks' shares of the moments, one after the other."""
    other = []
    call(*args, shard=(1, 2), moment_sum=lambda m: other.append(np.array(m)), **kw)

    def add(m):
        m += other[0].reshape(m.shape)

    return call(*args, shard=(0, 2), moment_sum=add, **kw)


@pytest.mark.parametrize("extent,qmax", [(90.0, 0.6), (170.0, 0.6), (400.0, 0.6), (900.0, 0.7)])
@pytest.mark.parametrize("n", [3, 500])
def test_several_radial_segments_match_the_general_path(engine, n, extent, qmax):
    """One to over ten segments: points and sites of each, the outermost atom on
    the last border, and none or one atom in a segment.  (Beyond q r = l + 24
    the reference's downward Bessel recurrence is not j_l, nor smooth between
    the radial nodes: there the general path is what a call has to equal, and
    the oracle only for the first extent.  The ranks' shares put other points
    into one FP32 sum of 32, so the TF32 mode agrees as FP32 does.)"""
    rng = np.random.default_rng(n)
    xyz = rng.uniform(-0.5, 0.5, (n, 3)) * [extent, 0.3 * extent, 0.2 * extent]
    el = rng.integers(0, 8, n).astype(np.int8)
    el[0] = 1
    s = cs.Structure(xyz, el, rng.choice([1.0, 0.5], n))
    q = np.linspace(0.0, qmax, 40)
    p = cs.SolventParams(c1=1.01, c2=0.9, hydration_model=cs.HydrationModel(2), hydration_grid_spacing_angstrom=4.0)
    for prec, tol in ((N.PREC_FP64, 1e-9), (N.PREC_TF32_SPLIT, 1e-5)):
        kw = dict(precision=prec, engine=engine)
        got = cs.multipole_intensity(s, q, 16, **kw)
        ref = _general(cs.multipole_intensity, s, q, 16, **kw)
        assert np.max(np.abs(got - ref)) <= tol * np.max(np.abs(ref)), prec
        basis = cs.multipole_solvent_basis(s, q, 16, p, **kw)
        ref_b = _general(cs.multipole_solvent_basis, s, q, 16, p, **kw)
        for k in range(6):
            assert np.max(np.abs(basis[k] - ref_b[k])) <= tol * np.max(np.abs(ref_b[k])), (prec, k)
        if extent > 90.0:
            continue
        exact = O.multipole_intensity(_atoms(s), q, 16)
        assert np.max(np.abs(got - exact)) <= tol * np.max(exact), prec
        exact = O.multipole_solvent_basis(_atoms(s), q, 16, p.c1, p.c2, model=2, spacing=4.0)
        for k in range(6):
            assert np.max(np.abs(basis[k] - exact[k])) <= tol * np.max(np.abs(exact[k])), (prec, k)
