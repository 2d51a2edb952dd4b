"""The ends of the divide and conquer (csrc/eigen_dc.cu): leaves of every size
(odd ones with a dummy player), splits, entries whose squares underflow, and the
triangular factors of the back-transformation around their 128 columns.

Tolerances: a backward-stable method gives eigenvalues, residual and
orthogonality within c n eps |A|_2; c = 10, the threshold of LAPACK's own test
ratios."""
import numpy as np
import pytest

from imcom_b200 import Solver

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _eigen(A):
    n = A.shape[0]
    x = np.arange(n, dtype=float)
    with Solver(0) as s:
        s.set_inputs(x, x, np.ones(n, dtype=np.int32), x[:1], x[:1], None, None, 1.0, 1.0)
        s.load_A(np.asfortranarray(A))
        Q, L, _ = s.eigen_A()
    return Q, L


def _check(A):
    n = A.shape[0]
    Q, L = _eigen(A)
    bound = 10 * n * EPS * np.linalg.norm(A, 2)
    assert np.abs(L - np.linalg.eigvalsh(A)[::-1]).max() <= bound
    assert np.linalg.norm(A @ Q - Q * L, 2) <= bound
    assert np.linalg.norm(Q.T @ Q - np.eye(n), 2) <= 10 * n * EPS


@pytest.mark.parametrize("n", [1, 2, 3, 4, 15, 16, 17, 31, 32, 33, 34, 63, 64, 65, 66, 127, 128, 129,
                               130, 256, 257, 258, 385, 700])
def test_leaves_and_blocks(n):
    rng = np.random.default_rng(n)
    V = rng.standard_normal((n, n)) * 10.0 ** rng.uniform(-4, 0, n)
    _check(V @ V.T)


@pytest.mark.parametrize("n", [20, 33])
@pytest.mark.parametrize("tiny", [1e-160, 1e-300, 0.0])
def test_tiny_and_zero_couplings(n, tiny):
    rng = np.random.default_rng(n)
    A = np.diag(np.where(np.arange(n) < n // 2, rng.uniform(1, 2, n), tiny * rng.uniform(1, 2, n)))
    e = tiny * rng.uniform(1, 2, n - 1)
    _check(A + np.diag(e, 1) + np.diag(e, -1))
