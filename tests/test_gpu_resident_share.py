"""The resident tridiagonalisation (csrc/eigen_res.cu) on shares of 8 SMs and more, where
it runs (a smaller share takes the cluster tail): the smallest share with orders around
what its shared memory holds, odd orders, one pair of rows per CTA, and CTAs that retire
in every column of the end.  A launch count shows that no panel and no cluster ran: the

Tolerance: a backward-stable method gives eigenvalues, residual and orthogonality within
c n eps |A|_2; c = 10, the threshold of LAPACK's own test ratios."""
import numpy as np
import pytest

from imcom_b200 import Solver
from imcom_b200.api import OPT_SM_SHARE

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("n,share", [(2, 8), (16, 8), (17, 8), (64, 8), (301, 8), (460, 8), (480, 9),
                                     (500, 8), (48, 24), (97, 48), (700, 24), (800, 24), (900, 24),
                                     (1151, 48)])
def test_resident_on_a_share(n, share):
    rng = np.random.default_rng(n)
    V = rng.standard_normal((n, min(n, 24)))
    A = V @ V.T / n + np.diag(rng.standard_normal(n) * 10.0 ** rng.uniform(-8, 0, n))
    A = np.asfortranarray(0.5 * (A + A.T))
    x = np.arange(n, dtype=float)
    with Solver(0) as s:
        s.set_inputs(x, x, np.ones(n, dtype=np.int32), x[:1], x[:1], None, None, 1.0, 1.0)
        s.set_option(OPT_SM_SHARE, share)
        s.load_A(A)
        Q, L, _ = s.eigen_A()
    bound = 10 * n * EPS * np.linalg.norm(A, 2)
    assert np.abs(L - np.linalg.eigvalsh(A)[::-1]).max() <= bound
    assert np.linalg.norm(A @ Q - Q * L, 2) <= bound
    assert np.linalg.norm(Q.T @ Q - np.eye(n), 2) <= 10 * n * EPS
