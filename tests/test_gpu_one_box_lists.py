"""The one-gridbox collision step (cleo_b200/csrc/onebox.cuh) at the edges of its two forms: the
one-block front (up to 28,000 slots) and the separate kernels beyond, counts around a block's share
and odd ones, with multiplicities of a few so that nulls appear from the first steps, several
collision sub-steps to a step, bit for bit against the correctly rounded oracle."""
import numpy as np
import pytest

import checkers as K
from cleo_b200 import abi, workloads as W
from cleo_b200.config import realtime2step
from cleo_b200.sdm import make_sdm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 4097, 27935, 27936, 27937, 40001])
@pytest.mark.parametrize("nulls", [False, True], ids=["valid", "nulls"])
def test_one_box_equals_oracle(n, nulls):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    w = W.box_golovin(n_sd=n, seed=n, numconc=2 ** 23 if not nulls else 2 ** 23 * n / 8192)
    if nulls:  # few real droplets each, many collisions
        w["supers"]["xi"][:] = np.random.default_rng(n).integers(1, 4, n)
        w["supers"]["radius"] *= 60.0
    w["params"].collstep = realtime2step(0.5)  # two sub-steps to a step of 1 s
    w["params"].coll_delt = 0.5
    w["params"].exec_mode = abi.EXEC_BATCHED
    g = make_sdm(w, lib=abi.load_library())
    o = make_sdm(w, lib=K.oracle_lib(cr=True), prefix="oc")
    for k in range(4):
        for s in (g, o):
            s.run_step(k * w["tstep"], (k + 1) * w["tstep"])
    g.check()
    K.assert_identical_run(g, o, f"one box of {n}")
    g.close()
    o.close()
