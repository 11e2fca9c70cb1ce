"""Host arithmetic of the kernel builds' workspace: it holds the partial planes of the dense segments in the worst
case."""
import ctypes as C

import pytest


def _size(shape, M, w):
    from hastycucompute_b200 import _lib
    n = C.c_size_t()
    st = _lib.load().hb_toeplitz_kernels_workspace_size(len(shape), _lib.i64_array([2 * s for s in shape]), 1, _lib.i64_array([M]), w,
                                                        C.byref(n))
    return st, n.value


@pytest.mark.parametrize("w", [4, 7])
@pytest.mark.parametrize("maxp", [512, 2048, 4096])
def test_workspace_holds_the_dense_parts(w, maxp):
    """Every point in a z plane that two segments of four tiles share and in reach of four columns, and every segment
    just above the subproblem limit: 8 M candidates in segments of maxp + 1, each of two parts (16 + 8 bytes) and
    31 + W + 2 W planes of 64 cells; next to them 11 arrays of 4 bytes a point."""
    M = 1184 * maxp  # setpts takes subproblems of maxp candidates from here on
    segments = 8 * M // (maxp + 1)
    need = segments * (2 * (16 + 8) + (32 + w - 1 + 2 * w) * 64 * 8) + 44 * M
    assert _size((64, 64, 64), M, w)[1] - _size((64, 64, 64), 0, w)[1] >= need


@pytest.mark.parametrize("shape,M", [((900, 900, 900), 10), ((1 << 20, 4), 10), ((16, 16), (1 << 31) - 1)])
def test_refuses_what_the_build_refuses(shape, M):
    """A fine grid of 2^32 cells, more than 2^20 modes and 2^31 points are argument errors of a build, so its caller
    must not be sent to allocate a workspace for them first."""
    assert _size(shape, M, 6)[0] == 1


@pytest.mark.parametrize("shape,M", [((400, 400, 400), 10), ((1 << 19, 4), 10), ((16, 16), (1 << 31) - 2)])
def test_takes_what_the_build_takes(shape, M):
    assert _size(shape, M, 6)[0] == 0
