"""The tensor-core kernel of imcom_gpu_build_images (csrc/stacks.cu) at the edges
of its tiles: 32 pixels, 64-deep stages, every stack width, split sums, and
stack columns that are not 16-byte aligned.

Tolerance: the n-term dot-product bound n u |T|^T |I| (any order of summation),
plus one rounding per partial sum of the reference's own sum."""
import numpy as np
import pytest
import torch

from imcom_b200 import Solver

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("n,m,S,odd", [
    (1, 1, 1, False), (2, 33, 2, True), (63, 31, 7, False), (64, 32, 8, True), (65, 64, 9, False),
    (257, 97, 16, True), (300, 40, 17, False), (511, 33, 24, True), (1000, 65, 25, False),
    (129, 200, 32, False), (333, 129, 33, True), (2500, 70, 40, False), (77, 95, 41, True),
    (1025, 96, 48, False), (640, 31, 49, False), (900, 33, 56, True), (128, 161, 57, False),
    (4100, 35, 64, False), (515, 66, 65, True), (301, 50, 129, False)])
def test_stacks_tensor_kernel(n, m, S, odd):
    rng = np.random.default_rng(n * 1000 + S)
    T = np.asfortranarray(rng.standard_normal((n, m)))
    I = rng.standard_normal((n, S)) * 10.0 ** rng.uniform(-3, 3, (n, 1))
    with Solver(0) as s:
        s.set_inputs(rng.random(n), rng.random(n), np.ones(n, dtype=np.int32), rng.random(m),
                     rng.random(m))
        s.load_T(T)
        # odd: columns of odd leading dimension from an address of 8 mod 16
        ld = n + 3 - (n % 2) * 2 if odd else n + (n % 2)
        buf = torch.zeros(S * ld + 2, dtype=torch.float64, device="cuda")
        dI = buf[1 if odd else 0:][:S * ld].view(S, ld)[:, :n]
        dI.copy_(torch.from_numpy(np.ascontiguousarray(I.T)))
        dH = torch.full((S, m), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        s.build_images_device(dI, dH)
        s.synchronize()
        H = dH.cpu().numpy().T
        H2 = s.build_images(I)
    ref = T.T @ I
    bound = (2 * n + 64) * U * (np.abs(T).T @ np.abs(I))
    assert np.all(np.abs(H - ref) <= bound)
    assert np.all(np.abs(H2 - ref) <= bound)
