"""The column-pair FFT passes (csrc/fftp.cuh) on the GPU, at every radix, with odd and even column
counts, a row count that leaves the last block partly empty, and a workspace whose pairs are not
16-byte aligned, against the FP64 oracle.

Tolerance 1e-6: a forward and an inverse FP32 transform of two axes pass through about 36 butterfly
levels of 0.3 - 0.6 eps rounding each, sqrt(36) * 0.6 * 6e-8 = 2e-7 in the 2-norm, times a margin."""
import numpy as np
import pytest

from helpers import crand, rand_coords, relerr, to_dev, to_np
from oracle import gridding
from oracle import toeplitz as otp

TOL = 1e-6

# image edges N: 2N = P Q covers the radices 8 .. 26 in both places
SHAPES = [(36, 40), (44, 45), (48, 50), (52, 54), (55, 60), (63, 65), (66, 70), (72, 75), (77, 81), (84, 98), (99, 117),
          (105, 121), (112, 125), (130, 143), (147, 156), (165, 192), (200, 216), (220, 234), (250, 260), (312, 338),
          (36, 40, 33), (44, 33, 45)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("B", [1, 2, 5, 17])
def test_toeplitz_lengths(cuda, shape, B):
    import torch
    import hastycucompute_b200 as hb
    from hastycucompute_b200.toeplitz import make_workspace
    rng = np.random.default_rng(sum(shape) * 31 + B)
    S, x = crand(rng, B, *shape), crand(rng, *shape)
    K = crand(rng, *[2 * s for s in shape])
    Kt = hb.transform_toeplitz_kernel(to_dev(K, cuda))
    ref = otp.sense_normal(x, S, K.astype(np.complex128), fast=True)
    for off in (0, 1):  # pairs aligned to 16 bytes, and not
        ws = torch.empty(make_workspace(shape, B, cuda).numel() + 1, dtype=torch.complex64, device=cuda)[off:]
        got = hb.sense_normal(to_dev(x, cuda), to_dev(S, cuda), Kt, None, ws)
        assert relerr(to_np(got), ref) <= TOL
    inp = to_dev(S, cuda)
    out = torch.empty_like(inp)
    hb.toeplitz_multiplication(inp, out, Kt, None, to_dev(x, cuda))
    ref = otp.toeplitz_multiplication(S, np.zeros_like(S), K.astype(np.complex128), x)
    assert relerr(to_np(out), ref) <= TOL


# modes whose fine grids (twice the modes, rounded up) are 72 .. 600 points
@pytest.mark.gpu
@pytest.mark.parametrize("nmodes,T", [((36, 33, 40), 5), ((50, 45, 59), 8), ((61, 30, 72), 3), ((75, 100), 1), ((96, 190), 7),
                                      ((108, 199), 2), ((215, 288), 12), ((300, 180), 17)])
def test_nufft_lengths(cuda, nmodes, T):
    import hastycucompute_b200 as hb
    rng = np.random.default_rng(sum(nmodes) + T)
    M, w = 3001, 5
    coords = rand_coords(rng, len(nmodes), M)
    d = [to_dev(c, cuda) for c in coords]
    for sign in (-1, 1):
        c, f = crand(rng, T, M), crand(rng, T, *nmodes)
        p1 = hb.NufftPlan(hb.NufftType.TYPE_1, hb.NufftOpts(nmodes=nmodes, ntransf=T, kernel_width=w, sign=sign))
        p1.setpts(d)
        assert relerr(to_np(p1(to_dev(c, cuda))), gridding.nufft1(coords, c, nmodes, w=w, sign=sign)) <= TOL
        p2 = hb.NufftPlan(hb.NufftType.TYPE_2, hb.NufftOpts(nmodes=nmodes, ntransf=T, kernel_width=w, sign=sign))
        p2.setpts(d)
        assert relerr(to_np(p2(to_dev(f, cuda))), gridding.nufft2(coords, f, w=w, sign=sign)) <= TOL
