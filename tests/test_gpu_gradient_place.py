"""The gradient's atoms as the forward pass left them on the device against
the general path (a context with a pair kernel of its own choice types the
atoms and lays them out on the host): atoms without weight, loose
weights, partial tiles, and distance tables in and out of shared memory.

Both are FP32 sums over the same pairs.  The forward curves differ by 2e-6,
which the residuals (half the curve here) double and the sum over q of terms of
both signs raises by about ten: 1e-4 of the largest component."""
import numpy as np
import pytest

import crabsaxs_b200 as cs
from crabsaxs_b200 import _native as N
from crabsaxs_b200.api import Engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def general():
    e = Engine(0)
    e.check(N.lib.crab_ctx_set_pair_variant(e.handle, 168 * 16 + 5))
    yield e
    e.close()


@pytest.mark.parametrize("n,extent,mixed", [(1, 10.0, False), (2, 10.0, True), (127, 20.0, True), (129, 20.0, False),
                                            (700, 40.0, True), (300, 260.0, True)])
def test_placed_atoms_give_the_general_gradient(engine, general, n, extent, mixed):
    rng = np.random.default_rng(n)
    xyz = rng.uniform(-0.5, 0.5, (n, 3)) * extent
    el = rng.choice([0, 1, 2, 3, 4] if mixed else [1, 3], n).astype(np.int8)
    el[0] = 1
    occ = rng.choice([1.0, 1.0, 0.5, 0.25, 0.0], n) if mixed else np.ones(n)
    occ[0] = 1.0
    s = cs.Structure(xyz, el, occ)
    q = np.arange(1, 61) * 0.006
    p = cs.SolventParams(c1=1.02, c2=0.7)
    curve = cs.combine_solvent_basis(cs.debye_solvent_basis(s, q, p, engine=engine), q, p.c1, p.c2)
    y, sigma = 0.5 * curve, 0.05 * curve + 1e-3 * curve.max()
    chi, g, gp = cs.chi2_grad(s, q, y, sigma, p, 1.0, 0.0, engine=engine)
    chi_r, g_r, gp_r = cs.chi2_grad(s, q, y, sigma, p, 1.0, 0.0, engine=general)
    assert abs(chi - chi_r) <= 1e-4 * chi_r
    assert np.max(np.abs(np.asarray(gp) - gp_r) / np.abs(gp_r)) <= 1e-4
    assert np.max(np.abs(g - g_r)) <= 1e-4 * np.max(np.abs(g_r)) + 1e-12
    assert np.all(g[occ == 0.0] == 0.0)
