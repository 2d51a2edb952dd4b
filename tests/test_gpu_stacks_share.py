"""More than 32 image stacks on a share of the SMs (IMCOM_OPT_SM_SHARE): the same sums
as on the whole GPU, and the kernel keeps to the share.  The second is seen in the time: 256 tiles of
pixels on 4 of 148 SMs are 64 in turn where the whole GPU takes two, so at least 8 times
as long (a kernel that ignores the share takes the same time)."""
import numpy as np
import pytest
import torch

from imcom_b200 import Solver
from imcom_b200.api import OPT_SM_SHARE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [33, 40, 48, 56, 64, 100])
def test_share(S):
    n, m = (2048, 8192) if S <= 64 else (300, 8192)
    rng = np.random.default_rng(S)
    with Solver(0) as s:
        s.set_inputs(rng.random(n), rng.random(n), np.ones(n, dtype=np.int32), rng.random(m),
                     rng.random(m))
        s.load_T(np.asfortranarray(rng.standard_normal((n, m))))
        dI = torch.from_numpy(rng.standard_normal((S, n))).cuda()
        dH = torch.empty(S, m, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        out, time = [], []
        for share in (0, 4):
            s.set_option(OPT_SM_SHARE, share)
            best = 1e9
            for _ in range(5):
                s.build_images_device(dI, dH)
                s.synchronize()
                best = min(best, s.stage_times()["epilogue"])
            out.append(dH.cpu().numpy().copy())
            time.append(best)
    # two orders of one sum of random signs: sqrt(n) u each of the result
    assert np.linalg.norm(out[0] - out[1]) <= 2 * n ** 0.5 * 2.0 ** -53 * np.linalg.norm(out[0])
    assert time[1] > 8 * time[0]
