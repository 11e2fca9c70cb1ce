"""Long sums of equal terms in the walking 3-D spreading kernel: a sum of n equal FP32 terms rounds the same way at every
step and drifts by up to n / 4 eps (eps = 2^-24), so a warp puts its sums away after a run of visits.

4096 equal points are one subproblem. With runs of at most 64 visits and the rest of a list (at most 128) the drift is
(192 + 4096 / 64) / 4 eps = 3.8e-6 at worst, plus 0.5e-6 for taps and passes; one run of 4096 drifts by up to 6e-5."""
import numpy as np
import pytest

from helpers import crand, to_dev, to_np
from oracle import gridding

TOL = 4.3e-6


@pytest.mark.gpu
@pytest.mark.parametrize("w", [4, 6, 7])
@pytest.mark.parametrize("T", [1, 2, 4, 8, 16, 32])
def test_equal_points(cuda, T, w):
    import hastycucompute_b200 as hb
    rng = np.random.default_rng(10 * T + w)
    nmodes, M = (16, 12, 20), 4096
    worst = 0.0
    for _ in range(8):
        coords = [np.full(M, v, np.float32) for v in rng.uniform(-np.pi, np.pi, 3)]
        c = np.repeat(crand(rng, T, 1), M, axis=1)
        plan = hb.NufftPlan(hb.NufftType.TYPE_1, hb.NufftOpts(nmodes=nmodes, ntransf=T, kernel_width=w))
        plan.set_spread_tuning(4096)
        plan.setpts([to_dev(x, cuda) for x in coords])
        got, ref = to_np(plan(to_dev(c, cuda))), gridding.nufft1(coords, c, nmodes, w=w)
        worst = max(worst, max(np.linalg.norm(got[t] - ref[t]) / np.linalg.norm(ref[t]) for t in range(T)))
    assert worst <= TOL
