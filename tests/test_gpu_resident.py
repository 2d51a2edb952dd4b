"""The resident end of the tridiagonalisation (csrc/eigen_res.cu) at the sizes
where it can go wrong: pairs of rows and 64-column groups with remainders, each
column-slot count, its largest order and the first order that needs a panel
before it, and on shares of the SMs (many rows per CTA).

Tolerances: a backward-stable reduction gives eigenvalues within c n eps |A|_2
of LAPACK's and the same bound for the residual and the orthogonality; c = 10,
the threshold of LAPACK's own test ratios."""
import numpy as np
import pytest

from imcom_b200 import ImcomError, Solver
from imcom_b200.api import (OPT_EIGEN_MAXITER, OPT_SM_SHARE, OPT_STALL_TEST, STALL_TRIDIAG)

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
    bound = 10 * n * EPS * np.linalg.norm(A, 2)
    assert np.abs(L - np.linalg.eigvalsh(A)[::-1]).max() <= bound
    assert np.linalg.norm(A @ Q - Q * L, 2) <= bound
    assert np.linalg.norm(Q.T @ Q - np.eye(n), 2) <= 10 * n * EPS


@pytest.mark.parametrize("n,share", [(2, 0), (3, 0), (5, 0), (63, 0), (64, 0), (65, 0), (129, 0),
                                     (296, 0), (297, 0), (512, 0), (513, 0), (1024, 0), (1025, 0),
                                     (1537, 0), (2048, 0), (2049, 0), (300, 8), (64, 1), (301, 3),
                                     (613, 24), (901, 24)])
def test_resident_tridiagonalisation(n, share):
    A = _matrix(n, n)
    with Solver(0) as s:
        s.set_option(OPT_SM_SHARE, share)
        Q, L, _ = _eigen(s, A)
    _check(A, Q, L)


def test_resident_diagonal_and_zero():
    """Columns whose reflector is the identity."""
    for A in (np.diag(np.arange(1.0, 71.0)), np.zeros((70, 70))):
        with Solver(0) as s:
            Q, L, _ = _eigen(s, np.asfortranarray(A))
        assert np.array_equal(np.sort(L), np.sort(np.diag(A)))
        assert np.abs(Q.T @ Q - np.eye(70)).max() <= 10 * 70 * EPS


def test_resident_exchange_timeout_returns_eigen_error():
    A = _matrix(200, 1)
    with Solver(0) as s:
        s.set_option(OPT_EIGEN_MAXITER, 2000)
        s.set_option(OPT_STALL_TEST, STALL_TRIDIAG)
        with pytest.raises(ImcomError) as ei:
            _eigen(s, A)
        assert ei.value.status == 5
        s.set_option(OPT_STALL_TEST, 0)
        s.set_option(OPT_EIGEN_MAXITER, 0)
        Q, L, _ = _eigen(s, A)
    _check(A, Q, L)
