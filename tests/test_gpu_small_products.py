"""The GEMM's small tiles (csrc/dgemm_tile.cuh) at the edges of their 32 x 32 x 32,
on both sides of the rule that picks them, and on a share of the SMs (several
tiles per CTA).

Tolerance: a sum of n products differs from the exact one by n eps sum |q b| at
most (numpy's own sum as much again)."""
import numpy as np
import pytest

from imcom_b200 import Solver
from imcom_b200.api import OPT_SM_SHARE

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("n,m,share", [(1, 1, 0), (3, 5, 0), (31, 33, 0), (32, 32, 0), (33, 31, 0),
                                       (64, 65, 0), (97, 1, 0), (130, 257, 0), (255, 256, 0),
                                       (600, 400, 0), (900, 700, 0), (300, 500, 2)])
def test_small_products(n, m, share):
    rng = np.random.default_rng(n + m)
    Q, B = rng.standard_normal((n, n)), rng.standard_normal((n, m))
    x, X = np.arange(n, dtype=float), np.arange(m, dtype=float)
    with Solver(0) as s:
        s.set_option(OPT_SM_SHARE, share)
        s.set_inputs(x, x, np.ones(n, dtype=np.int32), X, X, None, None, 1.0, 1.0)
        s.load_QL(np.asfortranarray(Q), np.arange(n, 0, -1.0))
        s.load_B(np.asfortranarray(B))
        P = s.build_P()
    bound = 2 * n * EPS * (np.abs(Q).T @ np.abs(B))
    assert P.shape == (n, m)
    assert np.all(np.abs(P - Q.T @ B) <= bound)
