"""The training kernel (csrc/kappa.cu) at its edges: tiles of 32 samples, more
tiles than SMs, a short last batch (CTAs without a tile), batches of one, a
share of the SMs.

Tolerances.  Gradient: the sums agree to fp32 rounding except where a
pre-activation rounds to another bfloat16 (2^-8 of one term of thousands): 1e-4
of the largest entry, the bar of the gradient's own check.  Training: Adam moves
an entry by about lr per step whatever its gradient's size, so only entries with
a clear sign can be compared; with 1e-2 relative gradient error in each of s
steps they differ by 3e-2 s lr.  The epoch's mean loss: 5122 entries, each 1e-4
of the largest gradient (order one per sample) at most and 2 lr off, change it
by 4e-3 at lr = 2e-3."""
import numpy as np
import pytest

from imcom_b200 import Solver
from imcom_b200 import kappa_model as KM
from imcom_b200.api import OPT_SM_SHARE
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    f = rng.standard_normal((12, n)).astype(np.float32)
    t = (f[0] - 0.5 * f[3] + 0.1 * rng.standard_normal(n)).astype(np.float32)
    return f, t


@pytest.mark.parametrize("n,share", [(1, 0), (31, 0), (32, 0), (33, 0), (4736, 0), (4737, 0),
                                     (9999, 0), (300, 3)])
def test_gradient(n, share):
    f, t = _data(n, n)
    p = KM.init_params(5)
    with Solver(0) as s:
        s.set_option(OPT_SM_SHARE, share)
        g, loss = s.mlp_gradient(f, t, p)
    loss_ref, g_ref = M.loss_and_grad(p, f, t)
    assert abs(loss - loss_ref) < 1e-4 * abs(loss_ref)
    assert np.max(np.abs(g - g_ref)) < 1e-4 * np.max(np.abs(g_ref))


def _order(n, state):
    order = list(range(n))
    for q in range(n - 1, 0, -1):
        state ^= (state << 13) & 0xffffffff
        state ^= state >> 17
        state ^= (state << 5) & 0xffffffff
        j = state % (q + 1)
        order[q], order[j] = order[j], order[q]
    return np.array(order), state


@pytest.mark.parametrize("n,batch,epochs,share", [(5, 1, 1, 0), (37, 16, 2, 0), (600, 512, 2, 0),
                                                  (1300, 5000, 3, 0), (640, 512, 4, 3),
                                                  (10000, 5000, 2, 0)])
def test_training(n, batch, epochs, share):
    lr = 2e-3
    f, t = _data(n, n)
    p = KM.init_params(3).astype(np.float64)
    with Solver(0) as s:
        s.set_option(OPT_SM_SHARE, share)
        got, loss = s.mlp_train(f, t, p, epochs=epochs, batch=batch, lr=lr, seed=7)
    m1 = np.zeros_like(p)
    m2 = np.zeros_like(p)
    step, state = 0, 7
    for ep in range(epochs):
        order, state = _order(n, state)
        total = 0.0
        for b in range(0, n, batch):
            idx = order[b:b + batch]
            l, g = M.loss_and_grad(p.astype(np.float32), f[:, idx], t[idx])
            total += l
            g = g / len(idx)
            step += 1
            m1 = 0.9 * m1 + 0.1 * g
            m2 = 0.999 * m2 + 0.001 * g * g
            p = p - lr * (m1 / (1 - 0.9 ** step)) / (np.sqrt(m2 / (1 - 0.999 ** step)) + 1e-8)
        assert abs(loss[ep] - total / n) < 4e-3 * max(1.0, total / n)
    assert np.median(np.abs(got - p)) < 3e-2 * step * lr
