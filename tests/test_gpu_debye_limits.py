"""The distance histogram at the limits of its shared memory, its inputs and its tables."""
import numpy as np
import pytest

import crabsaxs_b200 as cs
import oracle as O

pytestmark = pytest.mark.gpu


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
def test_loose_weights_over_the_range_of_bins(engine, bins, weights):
    rng = np.random.default_rng(bins)
    reach = (0.005 * bins / 0.5 - 1e-3) / 1.0001
    xyz = _mirrored(520, reach, rng)
    w = rng.uniform(0.2, 1.0, size=520)
    if weights == "few":
        w = np.where(rng.random(520) < 0.1, 0.4, 0.75)
    t = rng.integers(0, 3, size=520)
    q = np.sort(np.concatenate([[0.0], rng.uniform(0.0, 0.5, size=60), [0.5]]))
    got, _ = cs.debye_partials(xyz, w, t, 3, q, engine=engine)
    ref, _ = O.debye_partials(xyz, w, t, 3, q)
    s = np.array([w[t == a].sum() for a in range(3)])
    scale = np.array([s[a] * s[b] for a in range(3) for b in range(a, 3)])[:, None]
    assert (np.abs(got - ref) / scale).max() <= _tol(q, reach)
