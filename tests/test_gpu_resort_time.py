"""The page re-sort's time after few movers: the first step after winds start, which may move any
number of superdroplets, takes no more than twice the re-sort of a steady step with such movers."""
import ctypes as C

import numpy as np
import pytest

from cleo_b200 import abi, workloads as W
from cleo_b200.sdm import make_sdm

pytestmark = pytest.mark.gpu


def test_winds_that_start_after_still_steps():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    lib = abi.load_library()
    w = W.bubble3d(ndims=(64, 64, 48), seed=7)
    p = w["params"]
    p.condstep = p.collstep = abi.STEP_OFF
    p.motion_tv = abi.TV_NULL
    state = dict(w["state"])
    still = dict(state)
    for f in abi.STATE_FIELDS:
        if "vel_" in f:
            still[f] = np.zeros_like(state[f])
    s = make_sdm(w, lib=lib)
    assert lib.cleo_b200_set_resort_policy(s.ctx, abi.RESORT_PAGES) == 0
    assert lib.cleo_b200_set_profiling(s.ctx, 1) == 0
    ms, count, stats = (C.c_double * 5)(), (C.c_uint64 * 5)(), (C.c_uint64 * 4)()
    times, movers = [], []
    for k, st in enumerate([state, state, still, still, state, state, still, still, state, state]):
        s.upload_state(st)
        s.run_step(k * w["tstep"], (k + 1) * w["tstep"])
        assert lib.cleo_b200_stage_times(s.ctx, ms, count) == 0 and count[1] == 1
        assert lib.cleo_b200_resort_stats(s.ctx, stats) == 0
        times.append(ms[1])
        movers.append(stats[0])
    s.check()
    print("sort ms", [round(t, 3) for t in times], "movers", movers)
    assert min(movers[4], movers[5], movers[8], movers[9]) > 100_000 and movers[3] == movers[7] == 0
    assert min(times[4], times[8]) <= 2.0 * max(times[5], times[9]), times
