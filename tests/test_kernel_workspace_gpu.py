"""Toeplitz kernel builds in a caller's workspace, in one too small (what does not fit is allocated), and with the
library's own allocations give the same kernel up to the rounding of the point order."""
import ctypes as C

import numpy as np
import pytest

from helpers import rand_coords, relerr, to_dev, to_np
from oracle import toeplitz as otp


@pytest.mark.gpu
@pytest.mark.parametrize("shape,frames,w", [((16, 12, 10), 1, 6), ((16, 12, 10), 3, 4), ((24, 30), 2, 6), ((12, 12, 12), 2, 9)])
def test_workspace(cuda, shape, frames, w):
    import torch
    from hastycucompute_b200 import _lib
    from hastycucompute_b200._torch import ptr, stream_ptr
    rng = np.random.default_rng(sum(shape) + frames)
    dim, counts = len(shape), [1500 + 700 * f for f in range(frames)]
    coords = [rand_coords(rng, dim, m) for m in counts]
    cat = [to_dev(np.concatenate([c[i] for c in coords]), cuda) for i in range(dim)]
    cp = [ptr(c) for c in cat] + [C.c_void_p(None)] * (3 - dim)
    nd = torch.ones(sum(counts), dtype=torch.complex64, device=cuda)
    kshape = tuple(2 * n for n in shape)
    n = C.c_size_t()
    _lib.call("hb_toeplitz_kernels_workspace_size", dim, _lib.i64_array(kshape), frames, _lib.i64_array(counts), w, C.byref(n))
    ref = [otp.toeplitz_kernel(c, shape, None, w=w) for c in coords]
    for size in (int(n.value), 4096, 0, None):
        out = torch.full((frames, *kshape), float("nan"), dtype=torch.complex64, device=cuda)
        args = (dim, _lib.i64_array(kshape), frames, _lib.i64_array(counts), cp[0], cp[1], cp[2], ptr(nd), ptr(out), w)
        if size is None:
            _lib.call("hb_toeplitz_kernels_frames", *args, stream_ptr(cuda))
        else:
            ws = torch.empty(size + 8, dtype=torch.uint8, device=cuda)[8:]
            _lib.call("hb_toeplitz_kernels_frames_ws", *args, ptr(ws), size, stream_ptr(cuda))
        for f in range(frames):
            assert relerr(to_np(out[f]), ref[f]) <= 1e-5
