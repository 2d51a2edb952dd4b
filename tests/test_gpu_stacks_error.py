"""Rounding of the automatic choice of imcom_gpu_build_images against the two kernels
that it stands in for (FMA up to 32 stacks, the GEMM above): its error against
extended-precision sums is no larger.  Errors are 2-norms over 512 pixels x 6 stacks
(3072 sums of n products of random sign, so the norms are known to a few per cent);
10% are left for that."""
import numpy as np
import pytest
import torch

from imcom_b200 import Solver
from imcom_b200.api import OPT_STACK_KERNEL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 4096, 8192])
@pytest.mark.parametrize("S", [1, 2, 8, 16, 24, 32, 40, 48, 56, 64])
def test_error_no_larger(n, S):
    m, q = 512, min(S, 6)
    rng = np.random.default_rng(n)
    T = rng.standard_normal((n, m)) * np.exp(rng.standard_normal((n, m)))
    I = 1.0 + rng.standard_normal((n, S))
    ref = np.stack([(T.astype(np.longdouble) * I[:, k:k + 1]).sum(axis=0) for k in range(q)])
    err = {}
    with Solver(0) as s:
        s.set_inputs(rng.random(n), rng.random(n), np.ones(n, dtype=np.int32), rng.random(m),
                     rng.random(m))
        s.load_T(np.asfortranarray(T))
        dI = torch.from_numpy(np.ascontiguousarray(I.T)).cuda()
        dH = torch.empty(S, m, dtype=torch.float64, device="cuda")
        for kernel in (2, 1 if S <= 32 else 0):
            s.set_option(OPT_STACK_KERNEL, kernel)
            torch.cuda.synchronize()
            s.build_images_device(dI, dH)
            s.synchronize()
            err[kernel] = float(np.linalg.norm((dH[:q].cpu().numpy() - ref).astype(np.float64)))
    assert err[2] <= 1.1 * err[1 if S <= 32 else 0]
