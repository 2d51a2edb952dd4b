"""Contexts on several host threads whose eigensystems need different amounts of shared
memory in the same kernel at the same time (two orders in turn per thread, so that
every launch is a direct one).  A launch whose function attribute another thread has
lowered fails.  Tolerance: as a single thread, to the bit."""
import threading

import numpy as np
import pytest

from imcom_b200 import Solver

pytestmark = pytest.mark.gpu


def _eigen(s, n, out):
    x = np.arange(n, dtype=float)
    V = np.random.default_rng(n).standard_normal((n, n))
    s.set_inputs(x, x, np.ones(n, dtype=np.int32), x[:1], x[:1], None, None, 1.0, 1.0)
    s.load_A(np.asfortranarray(V @ V.T))
    out.append(s.eigen_A()[1].copy())


def test_orders_side_by_side():
    orders = [(40, 500), (70, 480), (530, 1000), (600, 900)]
    ref = {}
    with Solver(0) as s:
        for n in sum(orders, ()):
            got = []
            _eigen(s, n, got)
            ref[n] = got[0]
    errors = []

    def work(pair):
        try:
            with Solver(0) as s:
                for k in range(60):
                    n = pair[k % 2]
                    got = []
                    _eigen(s, n, got)
                    assert np.array_equal(got[0], ref[n])
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(p,)) for p in orders]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
