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


def test_class_counts_of_two_threads_do_not_meet():
    rng = np.random.default_rng(1)
    q = np.linspace(0.0, 0.4, 40)
    p = cs.SolventParams(c1=1.01, c2=0.8)
    structures = [_structure(120, 3, rng), _structure(200, 40, rng)]
    engines = [Engine(0), Engine(0)]
    alone = [cs.debye_solvent_basis(s, q, p, engine=e) for s, e in zip(structures, engines)]
    failed = []
    start = threading.Barrier(2)

    def work(k):
        try:
            start.wait()
            for _ in range(400):
                if not np.array_equal(cs.debye_solvent_basis(structures[k], q, p, engine=engines[k]), alone[k]):
                    raise AssertionError("another result beside the other thread")
        except Exception as e:  # noqa: BLE001
            failed.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for e in engines:
        e.close()
    assert not failed, failed
