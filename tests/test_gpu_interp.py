"""A and B assembly (csrc/interp.cu) where its windows are special: arguments on
table nodes (seven-point windows, delta weights), windows clipped at the
table's edges, arguments outside it (zero), every interpolation order, tables
smaller than the eight gathered rows, and ragged tiles, against the oracle's
Neville interpolation of its own tables.  Bar: 1e-12 of the table scale, as
for A and B everywhere (rounding of the tables, amplified by the weights)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _setup(nps, npad, n, m, E, seed, mode):
    rng = np.random.default_rng(seed)
    psf = 0.5
    half = 0.5 * nps * psf  # table half width in pixels: offsets reach its edge
    if mode == "nodes":     # every difference a whole number of table steps
        step = psf / npad if npad in (1, 2, 4) else psf
        pos = lambda k: rng.integers(-3, 4, k) * step  # noqa: E731
    elif mode == "edges":   # differences around and beyond the table's edges
        pos = lambda k: rng.choice([-0.5, 0.5], k) * half + rng.uniform(-1, 1, k) * psf  # noqa: E731
    else:
        pos = lambda k: rng.uniform(-0.4, 0.4, k) * half  # noqa: E731
    x, y, X, Y = pos(n), pos(n), pos(m), pos(m)
    e = np.sort(rng.integers(1, E + 1, n)).astype(np.int32)
    G = rng.random((nps, nps, E))
    Gam = rng.random((nps, nps))
    return x, y, e, X, Y, np.asfortranarray(G), np.asfortranarray(Gam), psf


@pytest.mark.parametrize("nps,npad,n,m,mode,npoly", [
    (24, 3, 33, 31, "inside", 7), (24, 3, 70, 17, "edges", 7), (24, 4, 45, 40, "nodes", 7),
    (24, 1, 32, 32, "edges", 5), (24, 2, 16, 65, "nodes", 3), (24, 3, 40, 33, "edges", 1),
    (25, 3, 17, 15, "inside", 6), (24, 3, 9, 8, "edges", 8), (2, 1, 5, 7, "edges", 7),
    (3, 1, 6, 4, "inside", 7), (2, 3, 7, 9, "edges", 7), (7, 1, 34, 3, "edges", 7),
    (8, 1, 1, 1, "inside", 7)])
def test_lookup_windows(solver, nps, npad, n, m, mode, npoly):
    E = 3
    x, y, e, X, Y, G, Gam, psf = _setup(nps, npad, n, m, E, nps * 100 + n, mode)
    solver.set_inputs(x, y, e, X, Y, None, None, psf, psf)
    solver.set_psfs(G, np.zeros(E), Gam, 0)
    solver.psf_spectra()
    A = solver.build_A(npoly, npad)
    B = solver.build_B(npoly, npad)
    Gt = np.stack([O.ft_r2c(np.asfortranarray(G[:, :, k])) for k in range(E)], axis=2)
    Gmt = O.ft_r2c(Gam)
    At = O.build_Alookup(np.asfortranarray(Gt), npad)
    Bt = O.build_Blookup(np.asfortranarray(Gt), Gmt, npad)
    A_o = O.lookup_A(x, y, e, 0, nps, npad, psf, psf, At, npoly)
    B_o = O.lookup_B(x, y, e, X, Y, 0, nps, npad, psf, psf, Bt, npoly)
    assert np.abs(A - A_o).max() <= 1e-12 * np.abs(At).max()
    assert np.abs(B - B_o).max() <= 1e-12 * np.abs(Bt).max()
    assert np.array_equal(A, A.T)
    assert np.array_equal(A == 0.0, A_o == 0.0) and np.array_equal(B == 0.0, B_o == 0.0)
