"""The walking 3-D spreading kernel (csrc/spread_walk.cuh) on the GPU where it can go wrong: the smallest
grids (a segment and the cells below it nearly wrap onto themselves), a last segment shorter than the others,
transform counts around the lane groups, every width it serves, all points in one cell, on the grid's edges or in
few planes (parts of dense segments), and no points at all, against the FP64 gridding oracle.

Tolerance 1e-5, the suite's parity bar: no FP32 sum runs over more than a subproblem's candidates
(<= 4096: sqrt(4096) * 6e-8 = 4e-6 at worst, for terms of equal sign)."""
import numpy as np
import pytest

from helpers import crand, rand_coords, relerr, to_dev, to_np
from oracle import gridding

PARITY = 1e-5


def _check(cuda, nmodes, coords, T, w, maxp=None, per_cta=0):
    import hastycucompute_b200 as hb
    rng = np.random.default_rng(T * 100 + w)
    c = crand(rng, T, coords[0].size)
    plan = hb.NufftPlan(hb.NufftType.TYPE_1, hb.NufftOpts(nmodes=nmodes, ntransf=T, kernel_width=w))
    if T >= 5:  # (fewer transforms walk with the cells on the lanes, the automatic choice)
        plan.set_spread_kernel("transforms", per_cta)
    if maxp:
        plan.set_spread_tuning(maxp)
    plan.setpts([to_dev(x, cuda) for x in coords])
    got = to_np(plan(to_dev(c, cuda)))
    if coords[0].size == 0:
        assert not got.any()
        return
    assert relerr(got, gridding.nufft1(coords, c, nmodes, w=w)) <= PARITY


@pytest.mark.gpu
@pytest.mark.parametrize("w", [4, 5, 6, 7])
@pytest.mark.parametrize("nmodes,T", [((8, 8, 8), 8), ((40, 9, 12), 5), ((9, 20, 8), 17), ((20, 12, 8), 33), ((12, 8, 8), 16), ((8, 8, 8), 1),
                                      ((40, 9, 12), 2), ((9, 20, 8), 3), ((20, 12, 8), 4)])
def test_shapes(cuda, nmodes, T, w):
    _check(cuda, nmodes, rand_coords(np.random.default_rng(w), 3, 2500), T, w)


@pytest.mark.gpu
@pytest.mark.parametrize("T,per_cta", [(9, 8), (9, 16), (9, 32), (1, 0), (2, 0), (3, 0)])
@pytest.mark.parametrize("where", ["one cell", "edges", "planes", "none", "line"])
def test_dense(cuda, where, T, per_cta):
    rng = np.random.default_rng(5)
    nmodes, M = (20, 16, 12), 3000
    if where == "one cell":
        coords = [np.full(M, 0.3 * a, np.float32) for a in (1, -2, 3)]
    elif where == "edges":
        coords = [rng.choice(np.array([-np.pi, np.pi * (1 - 1e-6), 0.0, -1e-7], np.float32), M) for _ in range(3)]
    elif where == "planes":
        coords = rand_coords(rng, 3, M)
        coords[0] = (0.05 * coords[0]).astype(np.float32)
    elif where == "line":
        coords = [np.linspace(-np.pi, np.pi, M, endpoint=False).astype(np.float32)] + [np.zeros(M, np.float32)] * 2
    else:
        coords = [np.zeros(0, np.float32)] * 3
    for maxp in (32, 100, 4096):
        _check(cuda, nmodes, coords, T, 6, maxp, per_cta)
