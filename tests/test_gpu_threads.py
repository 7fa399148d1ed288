"""Two contexts on two threads: calls whose kernels need different amounts of shared memory."""
import threading

import numpy as np
import pytest

import crabsaxs_b200 as cs
from crabsaxs_b200.api import Engine

pytestmark = pytest.mark.gpu


def _structure(n, classes, rng):
    """That many scattering classes: elements 1 .. 14, then united groups of carbon and nitrogen."""
    codes = [(e, -1) for e in range(1, 15)] + [(e, g) for e in (1, 2) for g in range(14)]
    codes = codes[:classes]
    assert len(codes) == classes
    pick = np.concatenate([np.arange(classes), rng.integers(0, classes, size=n - classes)])
    el = np.array([codes[k][0] for k in pick], dtype=np.int8)
    group = np.array([codes[k][1] for k in pick], dtype=np.int8)
    return cs.Structure(rng.uniform(-9.0, 9.0, size=(n, 3)), el, np.ones(n), group)


def _beside(calls, rounds):
    """Each call many times on a thread of its own; its result must stay the one it has alone."""
    alone = [call() for call in calls]
    failed = []
    start = threading.Barrier(len(calls))

    def work(k):
        try:
            start.wait()
            for _ in range(rounds):
                if not np.array_equal(calls[k](), alone[k]):
                    raise AssertionError("another result beside the other thread")
        except Exception as e:  # noqa: BLE001
            failed.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_class_counts_of_two_threads_do_not_meet():
    rng = np.random.default_rng(1)
    q = np.linspace(0.0, 0.4, 40)
    p = cs.SolventParams(c1=1.01, c2=0.8)
    structures = [_structure(120, 3, rng), _structure(200, 40, rng)]
    engines = [Engine(0), Engine(0)]
    _beside([lambda k=k: cs.debye_solvent_basis(structures[k], q, p, engine=engines[k]) for k in range(2)], 400)
    for e in engines:
        e.close()


def test_bins_of_two_threads_do_not_meet():
    """Weighted P(r) (over 64 weights, whole products: the sums are exact in any order), few bins beside many."""
    rng = np.random.default_rng(2)
    xyz, w = rng.uniform(-9.0, 9.0, size=(300, 3)), 1.0 + np.arange(300) % 100
    engines = [Engine(0), Engine(0)]
    bins = [16, 4000]
    _beside([lambda k=k: cs.pair_distance_histogram(xyz, w, bins[k], engine=engines[k])[1] for k in range(2)], 300)
    for e in engines:
        e.close()
