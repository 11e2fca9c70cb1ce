"""The bounded waits of the walking 3-D spreading kernel: with no tries at all every wait runs out at once, the
output is NaN, the error reaches the caller once (through check and through setpts), and the plan works again."""
import numpy as np
import pytest

from helpers import crand, rand_coords, relerr, to_dev, to_np
from oracle import gridding


def _plan(cuda, T, M=6000, nmodes=(20, 16, 12), maxp=None):
    import hastycucompute_b200 as hb
    rng = np.random.default_rng(T)
    coords, c = rand_coords(rng, 3, M), crand(rng, T, M)
    plan = hb.NufftPlan(hb.NufftType.TYPE_1, hb.NufftOpts(nmodes=nmodes, ntransf=T, kernel_width=6))
    if maxp:
        plan.set_spread_tuning(maxp)
    d = [to_dev(x, cuda) for x in coords]
    plan.setpts(d)
    return hb, plan, d, to_dev(c, cuda), gridding.nufft1(coords, c, nmodes, w=6)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [1, 3, 8, 17, 33])
@pytest.mark.parametrize("maxp", [None, 64])  # whole segments, and parts of them through the reduction
def test_wait_runs_out(cuda, T, maxp):
    hb, plan, d, c, ref = _plan(cuda, T, maxp=maxp)
    plan.set_spread_wait(0)
    assert np.isnan(to_np(plan(c))).all()
    with pytest.raises(hb.HastyError, match="HB_ERR_TIMEOUT"):
        plan.check()
    plan.check()  # reported once
    plan.set_spread_wait(1 << 20)
    assert relerr(to_np(plan(c)), ref) <= 1e-5
    plan.check()
    plan.set_spread_wait(0)
    plan(c)
    with pytest.raises(hb.HastyError, match="HB_ERR_TIMEOUT"):
        plan.setpts(d)
    plan.set_spread_wait(1 << 20)
    plan.setpts(d)
    assert relerr(to_np(plan(c)), ref) <= 1e-5


@pytest.mark.gpu
def test_wait_limit_is_checked(cuda):
    hb, plan, *_ = _plan(cuda, 2, M=10)
    for bad in (-1, (1 << 20) + 1):
        with pytest.raises(hb.HastyError, match="INVALID_ARG"):
            plan.set_spread_wait(bad)


def test_null_plan():
    from hastycucompute_b200 import _lib
    lib = _lib.load()
    assert lib.hb_nufft_check(None, None) == 1 and lib.hb_nufft_set_spread_wait(None, 1) == 1
