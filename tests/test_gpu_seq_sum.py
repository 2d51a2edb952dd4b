"""C's sequential sum by binades with predicted chunks (csrc/tables.cu) at its
edges: counts around the 4096-term chunk, spectra whose sum crosses many binades
early, late or all along, and terms too small for a binade.  The oracle adds the
GPU's own spectrum term by term; the sums are the same to the bit."""
import numpy as np
import pytest

from imcom_b200 import Solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _image(n, kind):
    x = np.arange(n) - n // 2
    r2 = x[:, None] ** 2 + x[None, :] ** 2
    if kind == "smooth":       # a spectrum peaked at the first and last rows
        return np.exp(-r2 / (2.0 * 4.0 ** 2))
    if kind == "noise":        # a flat one
        return np.random.default_rng(n).standard_normal((n, n))
    if kind == "wave":         # one that is peaked in the middle of the walk
        return np.exp(-r2 / (2.0 * 8.0 ** 2)) * np.cos(np.pi * x)[None, :]
    return 1e-160 * np.random.default_rng(n).standard_normal((n, n))  # squares near underflow


@pytest.mark.parametrize("n", [8, 63, 64, 65, 91, 128, 250, 362])
@pytest.mark.parametrize("kind", ["smooth", "noise", "wave", "tiny"])
def test_sequential_sum(n, kind):
    G = np.exp(-((np.arange(n) - n // 2)[:, None] ** 2 + (np.arange(n) - n // 2)[None, :] ** 2) / 8.0)
    with Solver(0) as s:
        s.set_psfs(np.asfortranarray(G), np.zeros(1), np.asfortranarray(_image(n, kind)), True)
        C, _, Gm = s.psf_spectra(spectra=True)
    assert C == O.calc_C(Gm)
