"""The collision kernels' bound of a pair's probability (cleo_b200/csrc/pair_bound.h) as it is
compiled, for the host: a pair is never left alone where the oracle's probability exceeds the random
number, taken just below it; two multiplicities, and kernels that are negative or vanishingly small.
On the GPU, breakup with a negative kernel, which every path decides by the probability itself."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

import checkers as K
from cleo_b200 import abi, workloads as W
from cleo_b200.config import VOL0, make_params
from cleo_b200.sdm import make_sdm
from test_pair_bound import _radii

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "%s/cleo_b200/csrc/pair_bound.h"
extern "C" int apart(const cleo_b200_params* p, uint32_t n, double volume, double r1, uint64_t x1,
                     double r2, uint64_t x2, uint64_t u) {
  const float coef = cleo::pair_bound_coef(cleo::pair_bound_kernel(*p), n, volume);
  return cleo::pair_apart(*p, coef, (float)r1, (float)r2, cleo::pair_xi(x1, x2), cleo::pair_phi(u));
}
"""


@pytest.fixture(scope="module")
def apart(tmp_path_factory):
    d = tmp_path_factory.mktemp("bound")
    src, out = d / "bound.cpp", d / "libbound.so"
    src.write_text(SOURCE % ROOT)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o",
                    str(out), str(src)], check=True)
    f = C.CDLL(str(out)).apart
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_uint32, C.c_double, C.c_double, C.c_uint64, C.c_double,
                  C.c_uint64, C.c_uint64]
    return f


def _below(prob):
    """The largest random word whose number, its leading 53 bits, is below prob > 0."""
    return ((min(2 ** 53, math.ceil(prob * 2.0 ** 53)) - 1) << 11) | 0x7FF


def _prob(p, n, volume, r1, x1, r2, x2):
    one = K.oracle_lib().oc_pair_probability(C.byref(p), r1, x1, 1e-18, r2, x2, 1e-18,
                                             volume / VOL0)
    return n * (n - 1.0) / (2.0 * (n // 2)) * float(max(x1, x2)) * one


@pytest.mark.parametrize("prob", [abi.PROB_GOLOVIN, abi.PROB_LONG, abi.PROB_CONST])
def test_no_pair_that_collides_is_left_alone(apart, prob):
    rng = np.random.default_rng(100 + prob)
    left = close = 0
    for _ in range(40000):
        p = make_params(colltstep=float(rng.choice([0.1, 1.0, 10.0])), coll_prob=prob,
                        coaleff=float(rng.choice([1.0, 0.3])), const_kernel=1e-9)
        n = int(rng.integers(2, 3000))
        volume = 10.0 ** rng.uniform(-1, 7)
        r1, r2 = (float(r) for r in _radii(rng))
        x1, x2 = (int(10.0 ** rng.uniform(0, 18)) for _ in range(2))
        pr = _prob(p, n, volume, r1, x1, r2, x2)
        if pr > 0.0:
            assert not apart(C.byref(p), n, volume, r1, x1, r2, x2, _below(pr))
        if 0.0 < pr < 0.4:  # the bound is of use: twice the probability is mostly above it
            left += apart(C.byref(p), n, volume, r1, x1, r2, x2, _below(2.0 * pr))
            close += 1
    if prob != abi.PROB_LONG:
        assert left > 0.8 * close


@pytest.mark.parametrize("kernel", [-1e-9, -1e-3, 1e-35, 1e-44, 5e-324])
def test_kernels_without_a_bound(apart, kernel):
    """A random number of nothing, or any for a negative kernel: not left alone."""
    p = make_params(colltstep=1.0, coll_prob=abi.PROB_CONST, const_kernel=kernel)
    words = [0] if kernel > 0 else [0, 1 << 63, (1 << 64) - 1]
    for n, volume, x in ((2, 1e6, 1), (1000, 1e-1, 10 ** 18), (3, 1e12, 5)):
        for u in words:
            assert not apart(C.byref(p), n, volume, 1.0, x, 2.0, x, u)
    p = make_params(colltstep=1.0, coll_prob=abi.PROB_LONG, coaleff=-abs(kernel))
    assert not apart(C.byref(p), 100, 1e6, 30.0, 10 ** 6, 60.0, 10 ** 6, (1 << 64) - 1)


def test_no_collisions_at_all(apart):
    for p in (make_params(colltstep=1.0, coll_prob=abi.PROB_CONST, const_kernel=0.0),
              make_params(colltstep=1.0, coll_prob=abi.PROB_LONG, coaleff=0.0)):
        assert apart(C.byref(p), 100, 1e6, 30.0, 10 ** 6, 60.0, 10 ** 6, 1 << 62)


@pytest.mark.gpu
@pytest.mark.parametrize("ndims,median", [((1, 1, 1), 900.0), ((2, 2, 3), 40.0), ((2, 2, 3), 300.0)])
def test_breakup_with_a_negative_kernel(ndims, median):
    """prob - floor(prob) of a negative probability: a pair breaks up where the random number is
    below 1 - |prob|."""
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    w = W.uneven3d(ndims=ndims, seed=3, median=median)
    p = w["params"]
    p.condstep = p.motionstep = abi.STEP_OFF
    p.coll_prob, p.coll_enact = abi.PROB_CONST, abi.ENACT_BREAKUP
    w["supers"]["xi"][:] = 10 ** 6 + np.arange(len(w["supers"]["xi"]), dtype=np.uint64) % 7
    counts = np.bincount(w["supers"]["sdgbxindex"], minlength=w["grid"]["ngbxs"])
    volume = float(w["state"]["volume"].max()) * VOL0
    p.const_kernel = -0.7 * volume / (counts.max() * 1e6 * p.coll_delt)  # the largest: some -0.7
    runs = []
    for library, prefix, mode in ((abi.load_library(), "cleo_b200", abi.EXEC_BATCHED),
                                  (abi.load_library(), "cleo_b200", abi.EXEC_PLAIN),
                                  (K.oracle_lib(cr=True), "oc", abi.EXEC_PLAIN)):
        p.exec_mode = mode
        s = make_sdm(w, lib=library, prefix=prefix)
        for k in range(2):
            s.run_step(k * w["tstep"], (k + 1) * w["tstep"])
        s.check()
        runs.append(s)
    changed = runs[2].download_supers()["xi"].sum() > 1.2 * w["supers"]["xi"].sum()
    assert changed
    K.assert_identical_run(runs[0], runs[2], "batched")
    K.assert_identical_run(runs[1], runs[2], "plain")
