"""The panels of the tridiagonalisation (csrc/eigen_panel.cu) at the sizes where
they can go wrong: orders around the tiles' 128 rows and 8 columns and the
panel's 32 columns, odd orders (a row of padding), the first orders that need a
panel before the resident end, and shares of the SMs (several rounds of rows per
CTA, V and W or x too large for shared memory).

Tolerances: a backward-stable reduction gives eigenvalues within c n eps |A|_2
of LAPACK's and the same bound for the residual and the orthogonality; c = 10,
the threshold of LAPACK's own test ratios."""
import numpy as np
import pytest
import torch

from imcom_b200 import ImcomError, Solver
from imcom_b200.api import (OPT_EIGEN_MAXITER, OPT_SM_SHARE, OPT_STALL_TEST, OPT_TAIL_CTAS,
                            STALL_TRIDIAG)

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _matrix(n, seed):
    """Symmetric with an 8-decade spectrum of both signs."""
    rng = np.random.default_rng(seed)
    V = rng.standard_normal((n, min(n, 24)))
    d = rng.standard_normal(n) * 10.0 ** rng.uniform(-8, 0, n)
    A = V @ V.T / n + np.diag(d)
    return np.asfortranarray(0.5 * (A + A.T))


def _eigen(s, A):
    n = A.shape[0]
    x = np.arange(n, dtype=float)
    s.set_inputs(x, x, np.ones(n, dtype=np.int32), x[:1], x[:1], None, None, 1.0, 1.0)
    s.load_A(A)
    return s.eigen_A()


def _check(A, Q, L):
    n = A.shape[0]
    a, q, l = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (A, Q, L))
    w = torch.linalg.eigvalsh(a).flip(0)
    norm = float(w.abs().max())
    assert float((l - w).abs().max()) <= 10 * n * EPS * norm
    assert float(torch.linalg.norm(a @ q - q * l)) <= 10 * n * EPS * norm
    assert float(torch.linalg.norm(q.T @ q - torch.eye(n, device="cuda", dtype=a.dtype))) <= \
        10 * n * EPS


@pytest.mark.parametrize("n,share,tail", [
    (2, 0, -1), (3, 0, -1), (9, 0, -1), (33, 0, -1), (34, 0, -1), (127, 0, -1), (128, 0, -1),
    (129, 0, -1), (136, 0, -1), (137, 0, -1), (161, 0, -1), (257, 0, -1), (1000, 0, -1),
    (130, 1, -1), (301, 3, -1), (900, 1, -1), (1001, 3, -1), (700, 24, 8), (1301, 24, 0),
    (2049, 0, 0), (2083, 0, 0), (2112, 0, 0), (2305, 0, 0), (3001, 0, 0), (4800, 1, -1)])
def test_panel_tridiagonalisation(n, share, tail):
    A = _matrix(n, n)
    with Solver(0) as s:
        s.set_option(OPT_EIGEN_MAXITER, 4000000)
        s.set_option(OPT_SM_SHARE, share)
        s.set_option(OPT_TAIL_CTAS, tail)
        Q, L, _ = _eigen(s, A)
    _check(A, Q, L)


def test_panel_exchange_timeout_returns_eigen_error():
    A = _matrix(200, 1)
    with Solver(0) as s:
        s.set_option(OPT_TAIL_CTAS, -1)
        s.set_option(OPT_EIGEN_MAXITER, 2000)
        s.set_option(OPT_STALL_TEST, STALL_TRIDIAG)
        with pytest.raises(ImcomError) as ei:
            _eigen(s, A)
        assert ei.value.status == 5
        s.set_option(OPT_STALL_TEST, 0)
        s.set_option(OPT_EIGEN_MAXITER, 0)
        Q, L, _ = _eigen(s, A)
    _check(A, Q, L)
