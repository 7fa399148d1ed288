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
