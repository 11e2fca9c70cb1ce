"""The spreading tuner and the 3-D walking kernel: plans of one to four transforms, which walk by default but refuse
the kernel name "transforms", have it timed as "auto"; choices that an older build cached are not reused."""
import numpy as np
import pytest
import torch

from hastycucompute_b200 import autotune
from helpers import rand_coords, to_dev


@pytest.mark.parametrize("T,kernel", [(1, "auto"), (4, "auto"), (5, "transforms")])
def test_walk_is_among_the_candidates(T, kernel):
    assert {k for k, _, _ in autotune.spread_candidates((64, 64, 64), T)} == {kernel, "cells"}
    assert {k for k, _, _ in autotune.spread_candidates((64, 64), T)} == {"transforms", "cells"}


def test_choices_of_older_kernels_are_not_reused(tmp_path, monkeypatch):
    monkeypatch.setenv("HASTY_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    c = [torch.from_numpy(x) for x in rand_coords(np.random.default_rng(0), 3, 5000)]
    key = autotune._key((16, 16, 16), 2, 6, c)
    old = key[key.index("d3|"):]  # a key without the revision of the kernels
    choice = {"kernel": "cells", "block": [4, 4, 2], "max_candidates": 2048, "ms": 0.5, "timings": []}
    autotune._store({old: choice, "interp|" + old: {"interp_group": 4, "ms": 0.1, "timings": []}})

    class Timed(Exception):
        pass

    def timed(*a, **k):
        raise Timed

    monkeypatch.setattr(autotune, "NufftPlan", timed)
    for tune in (autotune.tune_spread, autotune.tune_interp):
        with pytest.raises(Timed):
            tune((16, 16, 16), 2, c, 6)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [1, 2, 4])
def test_tuner_times_the_walk(cuda, tmp_path, monkeypatch, T):
    import hastycucompute_b200 as hb
    monkeypatch.setenv("HASTY_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    coords = [to_dev(x, cuda) for x in rand_coords(np.random.default_rng(T), 3, 300000)]
    best = autotune.tune_spread((64, 64, 64), T, coords, 6)
    timed = {(k, m) for _, k, _, m in best["timings"]}
    assert {("auto", m) for m in autotune.MAXP_TRANSFORMS} <= timed and any(k == "cells" for k, _ in timed)
    plan = hb.NufftPlan(hb.NufftType.TYPE_1, hb.NufftOpts(nmodes=(64, 64, 64), ntransf=T, kernel_width=6))
    autotune.apply(plan, best)
    plan.setpts(coords)
