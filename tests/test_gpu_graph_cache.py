"""The captured steps a context keeps: eight patterns of sub-steps of a one-gridbox domain, whose
collision sub-steps alternate between two buffers, are replayed and not captured again."""
import time

import pytest

from cleo_b200 import abi, workloads as W
from cleo_b200.sdm import make_sdm

pytestmark = pytest.mark.gpu

SECONDS = [1, 2, 3, 4, 5, 6, 7, 9]  # an odd sum: every second cycle starts from the other buffer


def test_eight_patterns_of_a_box_are_replayed():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    lib = abi.load_library()
    w = W.box_golovin(n_sd=2048)
    calls = [[] for _ in SECONDS]  # per pattern, the calls' host times
    s = make_sdm(w, lib=lib)
    t = 0
    for cycle in range(10):
        for k, sec in enumerate(SECONDS):
            s.synchronize()
            t0 = time.perf_counter()
            s.run_step(t, t + 100 * sec)
            calls[k].append(time.perf_counter() - t0)
            t += 100 * sec
    s.check()
    s.close()
    for c in calls:  # the first two calls of a pattern capture it, from either buffer
        assert min(c[2:]) < 0.5 * min(c[:2]), [[round(1e6 * x) for x in c] for c in calls]
