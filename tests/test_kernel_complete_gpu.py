"""A Toeplitz kernel build is complete when the call returns: its stream is idle, and another stream that does not
wait for it reads the finished kernel."""
import numpy as np
import pytest

from helpers import rand_coords, relerr, to_dev, to_np
from oracle import toeplitz as otp


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(96, 96, 96), (256, 240)])
@pytest.mark.parametrize("how", ["kernel", "build", "frames"])
def test_complete_on_return(cuda, shape, how):
    import torch
    import hastycucompute_b200 as hb
    coords = rand_coords(np.random.default_rng(1), len(shape), 200000)
    d = [to_dev(c, cuda) for c in coords]
    nd = torch.ones((1, 200000), dtype=torch.complex64, device=cuda)
    kernel = torch.empty(tuple(2 * n for n in shape), dtype=torch.complex64, device=cuda)
    frames = torch.empty((1, *kernel.shape), dtype=torch.complex64, device=cuda)
    side = torch.cuda.Stream(cuda)
    torch.cuda.synchronize()
    if how == "kernel":
        hb.toeplitz_kernel(d, kernel, nd, kernel_width=6)
    elif how == "build":
        kernel = hb.build_toeplitz_kernel(d, shape, kernel_width=6)
    else:
        hb.toeplitz_kernels_frames([d], frames, kernel_width=6)
        kernel = frames[0]
    idle = torch.cuda.current_stream().query()
    assert idle
    with torch.cuda.stream(side):
        got = kernel.clone()
    side.synchronize()
    assert torch.equal(got, kernel)
    if len(shape) == 2:
        assert relerr(to_np(got), otp.toeplitz_kernel(coords, shape, None, w=6)) <= 1e-5
