"""Gathering interpolation against the FP64 restatement: runs of one and several turns per CTA with a remainder, a
single point, transforms that fill the lane groups or not, footprints that wrap, and every row split of a plane.

Bound 1e-5: taps, products and a sum of w^d terms in float32 (about 1e-6 relative for w^3 <= 512 with random
signs), as for the other type-2 parity tests.
"""
import numpy as np
import pytest

from helpers import crand, rand_coords, relerr, to_dev, to_np
from oracle import gridding

CASES = [
    # dim, nmodes, M, ntransf, width
    (1, (37,), 257, 1, 6),
    (2, (24, 20), 2424837, 1, 4),       # two turns of 256 points and a last one of 5
    (2, (17, 30), 1031, 2, 7),
    (3, (16, 12, 20), 303109, 5, 5),    # two turns of 32, five transforms on eight lanes
    (3, (12, 14, 10), 151563, 32, 6),   # four turns of 8 and a last one of 3
    (3, (12, 12, 12), 1, 3, 6),
    (3, (14, 10, 12), 4099, 12, 4),
    (3, (10, 10, 10), 9, 40, 7),
    (3, (14, 10, 12), 4099, 4, 8),
    (3, (14, 12, 16), 1025, 16, 9),
]


@pytest.mark.gpu
@pytest.mark.parametrize("dim,nmodes,M,T,w", CASES)
def test_gather_matches_oracle(cuda, dim, nmodes, M, T, w):
    import hastycucompute_b200 as hb
    rng = np.random.default_rng(31 + M)
    coords = rand_coords(rng, dim, M)
    f = crand(rng, T, *nmodes)
    plan = hb.NufftPlan(hb.NufftType.TYPE_2, hb.NufftOpts(nmodes=nmodes, ntransf=T, kernel_width=w))
    plan.setpts([to_dev(x, cuda) for x in coords])
    got = to_np(plan(to_dev(f, cuda)))
    e = relerr(got, gridding.nufft2(coords, f, w=w))
    assert e <= 1e-5, f"type2 parity {e:.2e}"
