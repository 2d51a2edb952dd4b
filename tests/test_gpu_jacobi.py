"""The batched Jacobi kernel (csrc/eigen_jacobi.cu) at the edges of its layout:
eight lanes per pair and four pairs per warp, 32-row chunks, odd orders (an idle
player), more systems than SMs.

Tolerances: a backward-stable method gives eigenvalues, residual and
orthogonality within c n eps |A|_2; c = 10, the threshold of LAPACK's own test
ratios."""
import numpy as np
import pytest

from imcom_b200 import Solver

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("n,count", [(1, 2), (2, 3), (7, 2), (8, 2), (9, 2), (16, 150), (32, 2),
                                     (33, 2), (63, 2), (64, 2), (65, 2), (95, 2), (96, 2),
                                     (97, 2), (104, 2), (111, 2), (112, 2)])
def test_jacobi_kernel(n, count):
    rng = np.random.default_rng(n)
    V = rng.standard_normal((count, n, 2 * n)) * 10.0 ** rng.uniform(-3, 0, (count, n, 1))
    A = V @ V.transpose(0, 2, 1)
    A[-1] = np.diag(np.arange(float(n)))  # nothing to rotate, a zero column
    with Solver(0) as s:
        Q, L, sweeps = s.eigh_jacobi_batched(A)
    assert sweeps[-1] <= 1
    for a, q, w in zip(A, Q, L):
        bound = 10 * n * EPS * np.linalg.norm(a, 2)
        assert np.abs(w - np.linalg.eigvalsh(a)).max() <= bound
        assert np.linalg.norm(a @ q - q * w, 2) <= bound
        assert np.linalg.norm(q.T @ q - np.eye(n), 2) <= 10 * n * EPS
