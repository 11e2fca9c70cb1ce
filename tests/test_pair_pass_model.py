"""Model of the in-place step 1 of the column-pair FFT passes (csrc/fftp.cuh) with lanes that do not run in
lock-step: the lanes of a row (one t, eight column pairs) run in an order of their own, each up to the next barrier
of the kernel, and the pass still has to give the transform of every pair. Whether the kernel has the barrier is
read from its source."""
import re
from pathlib import Path

import numpy as np
import pytest

PAIRS = 8
SRC = (Path(__file__).resolve().parent.parent / "hastycucompute_b200" / "csrc" / "fftp.cuh").read_text()


def _step1_barrier() -> bool:
    """Is there a barrier of the row's lanes between the sample loads and the stores into the transpose?"""
    body = SRC[SRC.index("void pair_step1("):]
    body = body[: body.index("Y[pair_slot<Op>(k1 * Q + t, k1, cp)] = v[k1];")]
    after_loads = body[body.rindex("pair_inputs<P, HM>"):]
    return re.search(r"if constexpr \(kPairInPlace<Op, HM> && Op::kStoreLFast\) __syncwarp\(0xffu << \(threadIdx\.x & 24\)\);",
                     after_loads) is not None


def _slot(row, k1, cp, rotate):  # pair_slot
    return row, cp ^ (k1 & (PAIRS - 1)) if rotate else cp


def _run(P, Q, rotate, barrier, rng):
    """Steps 1 and 2 in one memory; returns the transforms and those of the samples."""
    L = P * Q
    x = rng.standard_normal((L, PAIRS)) + 1j * rng.standard_normal((L, PAIRS))
    mem = x.copy()
    dft = np.exp(-2j * np.pi * np.outer(np.arange(P), np.arange(P)) / P)
    for t in rng.permutation(Q):  # rows touch no slots of one another
        lanes = rng.permutation(PAIRS)
        loaded = {}
        if barrier:
            loaded = {cp: mem[t + Q * np.arange(P), cp].copy() for cp in lanes}
        for cp in lanes:
            v = loaded[cp] if barrier else mem[t + Q * np.arange(P), cp].copy()
            v = (dft @ v) * np.exp(-2j * np.pi * t * np.arange(P) / L)
            for k1 in range(P):
                mem[_slot(k1 * Q + t, k1, cp, rotate)] = v[k1]
    X = np.empty_like(x)
    for k1 in range(P):
        for cp in range(PAIRS):
            u = np.array([mem[_slot(k1 * Q + t, k1, cp, rotate)] for t in range(Q)])
            X[k1 + P * np.arange(Q), cp] = np.fft.fft(u)
    return X, np.fft.fft(x, axis=0)


@pytest.mark.parametrize("P,Q", [(8, 8), (8, 16), (16, 20), (9, 13), (26, 25)])
@pytest.mark.parametrize("rotate", [False, True])
def test_lanes_out_of_step(P, Q, rotate):
    """Rows are the slots {k1 Q + t}: those that step 1 reads ({t + Q j}) for every t, so rotated or not the eight
    lanes of a t meet only one another; eight threads t * 8 .. t * 8 + 7 lie in one warp."""
    assert {k1 * Q + 3 for k1 in range(P)} == {3 + Q * j for j in range(P)}
    X, ref = _run(P, Q, rotate, rotate and _step1_barrier(), np.random.default_rng(P * Q))
    assert np.abs(X - ref).max() <= 1e-9 * np.abs(ref).max()
