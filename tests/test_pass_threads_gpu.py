"""Host threads that launch the same pass instance with different amounts of shared memory (the run-time
radices serve every length they divide, with memory for that length): each call succeeds and gives its own result."""
import ctypes as C
import threading

import numpy as np
import pytest

from helpers import crand, relerr, to_dev, to_np
from oracle import toeplitz as otp


# Every pass of the larger shape needs more than the 48 KB that any kernel may have. 2N = 264 and 676: column pairs,
# radices above 20 (12 x 22, 26 x 26). 36 and 3072: no pair split, the shared-memory kernel.
@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [((132, 132), (338, 338)), ((18, 18), (1536, 18))])
def test_shapes_at_once(cuda, shapes):
    import torch
    import hastycucompute_b200 as hb
    from hastycucompute_b200 import _lib
    from hastycucompute_b200._torch import ptr
    from hastycucompute_b200.toeplitz import make_workspace
    rng = np.random.default_rng(shapes[1][0])
    lib = _lib.load()
    start, errors = threading.Barrier(len(shapes)), []

    def work(args, out, ref, stream):
        start.wait(60)
        for _ in range(10000):  # (the bare entry: a thread spends its time between setting up launches and launching)
            if lib.hb_sense_normal(*args):
                errors.append(lib.hb_last_error())
                break
        stream.synchronize()
        if relerr(to_np(out), ref) > 1e-6:
            errors.append("wrong result")

    threads, tensors = [], []
    for shape in shapes:
        S, x, K = crand(rng, 1, *shape), crand(rng, *shape), crand(rng, *[2 * s for s in shape])
        keep = [to_dev(x, cuda), to_dev(S, cuda), hb.transform_toeplitz_kernel(to_dev(K, cuda)),
                torch.empty(shape, dtype=torch.complex64, device=cuda), make_workspace(shape, 1, cuda)]
        stream = torch.cuda.Stream(cuda)
        args = (2, _lib.i64_array(shape), 1, *[ptr(t) for t in keep], keep[-1].numel() * 8, C.c_void_p(stream.cuda_stream))
        ref = otp.sense_normal(x, S, K.astype(np.complex128), fast=True)
        threads.append(threading.Thread(target=work, args=(args, keep[3], ref, stream)))
        tensors.append(keep)
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
