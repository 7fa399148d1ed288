"""Site-site sums of hydration lattices: one tile of sites and less, whole and
ragged tiles, more tile pairs than CTAs, and spans whose squared distances do
not fit the shared counters.  The counts are integers and the transform f64:
the hydration row equals the oracle's f64 pair sum to 1e-9 of its largest
value (the site coordinates' own rounding is 1e-15 of a distance)."""
import numpy as np
import pytest

import crabsaxs_b200 as cs
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,extent,spacing", [(1, 0.0, 9.0), (1, 0.0, 4.0), (2, 14.0, 3.0), (60, 40.0, 4.0),
                                              (60, 40.0, 2.0), (2, 700.0, 4.0)])
def test_site_rows_match_oracle(engine, n, extent, spacing):
    rng = np.random.default_rng(n)
    xyz = rng.uniform(-0.5, 0.5, (n, 3)) * [extent, 0.8 * extent, 0.6 * extent]
    s = cs.Structure(xyz, np.ones(n, np.int8))
    q = np.linspace(0.0, 0.5, 31)
    p = cs.SolventParams(hydration_model=cs.HydrationModel.AdaptiveGrid, hydration_grid_spacing_angstrom=spacing)
    got = cs.debye_solvent_basis(s, q, p, engine=engine)
    a = O.Atoms(s.xyz, s.element, s.group, s.occupancy)
    ref = O.debye_solvent_basis(a, q, 1.0, 0.0, model=2, spacing=spacing)
    assert np.max(np.abs(got[2] - ref[2])) <= 1e-9 * np.max(np.abs(ref[2]))
