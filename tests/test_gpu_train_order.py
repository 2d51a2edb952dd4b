"""Training and its gradient (csrc/kappa.cu) add up the tiles of a batch in a fixed
order, so the same call gives the same bits whatever the timing and the grid: one
tile, odd batches, several tiles per CTA, more tiles than rows of the workspace
(1024 tiles of 32 samples), shares of the SMs.  Tolerance: none."""
import numpy as np
import pytest

from imcom_b200 import Solver
from imcom_b200 import kappa_model as KM
from imcom_b200.api import OPT_SM_SHARE

pytestmark = pytest.mark.gpu


def _data(n):
    rng = np.random.default_rng(n)
    f = rng.standard_normal((12, n)).astype(np.float32)
    t = (f[0] - 0.5 * f[3] + 0.1 * rng.standard_normal(n)).astype(np.float32)
    return f, t


@pytest.mark.parametrize("n,batch,epochs", [(70, 1, 3), (900, 37, 8), (20000, 512, 2),
                                            (20000, 5000, 6), (40000, 35000, 3)])
def test_training_bits(n, batch, epochs):
    f, t = _data(n)
    p = KM.init_params(3)
    with Solver(0) as s:
        runs = []
        for share in (0, 0, 0, 24, 3):
            s.set_option(OPT_SM_SHARE, share)
            runs.append(s.mlp_train(f, t, p, epochs=epochs, batch=batch, lr=2e-3, seed=7))
    for q, loss in runs[1:]:
        assert np.array_equal(q, runs[0][0])
        assert np.array_equal(loss, runs[0][1])


@pytest.mark.parametrize("n", [33, 4737, 40000])
def test_gradient_bits(n):
    f, t = _data(n)
    p = KM.init_params(5)
    with Solver(0) as s:
        runs = []
        for share in (0, 0, 0, 24, 3):
            s.set_option(OPT_SM_SHARE, share)
            runs.append(s.mlp_gradient(f, t, p))
    for g, loss in runs[1:]:
        assert np.array_equal(g, runs[0][0])
        assert loss == runs[0][1]
