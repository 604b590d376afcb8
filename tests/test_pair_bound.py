"""The single-precision bound with which the collision kernels leave a pair alone without evaluating
its probability (cleo_b200/csrc/batched.cuh, pair_bound_coef and pair_apart), restated in numpy
float32, against the oracle's probability: never below it, over radii from haze to the largest
drops, around the branch points of Simmel's velocity and of the collection efficiency, equal radii,
and the range of multiplicities, counts and volumes."""
import ctypes as C

import numpy as np
import pytest

import checkers as K
from cleo_b200 import abi
from cleo_b200.config import R0, VOL0, make_params

F = np.float32


def _bound(p, n, volume, r1, r2, xi):
    """coef * xi * k of a gridbox of n superdroplets in volume (m^3)."""
    if p.coll_prob == abi.PROB_GOLOVIN:
        k0 = F(1.5e3 * R0 * R0 * R0 * 4.0 / 3.0 * np.pi)
    elif p.coll_prob == abi.PROB_LONG:
        k0 = F(np.pi * R0 * R0) * abs(F(p.coaleff))
    else:
        k0 = abs(F(p.const_kernel))
    coef = F(1.005) * (F(n) * (F(n) - F(1))) / (F(2) * F(n // 2))
    coef = coef * (k0 * F(p.coll_delt) / F(volume))
    a, b = F(r1), F(r2)
    k = F(1)
    if p.coll_prob == abi.PROB_LONG:
        rs, rb = min(a, b), max(a, b)
        eff = max(F(4.5e4 * R0 * R0 * 100 * 100) * (rb * rb)
                  * (F(1.00001) - F(3e-4 / R0 / 100) / rs), F(0.001))
        if not rb < F(49.9):
            eff = max(eff, F(1))
        k = eff * ((a + b) * (a + b)) * min(F(1.189e-4) * (rb * rb), F(9.18))
    elif p.coll_prob == abi.PROB_GOLOVIN:
        k = a * a * a + b * b * b
    return float(coef * np.nextafter(F(xi), F(np.inf)) * k)


def _radii(rng):
    kind = rng.integers(4)
    if kind == 0:
        return 10.0 ** rng.uniform(-2, 3.6, 2)
    edge = rng.choice([3.0, 50.0, 67.215, 755.82, 1738.92])
    if kind == 1:
        return edge * (1.0 + rng.normal() * 1e-6), 10.0 ** rng.uniform(-2, 3.6)
    if kind == 2:
        return edge * (1.0 + rng.normal() * 1e-3), edge * (1.0 + rng.normal() * 1e-3)
    r = 10.0 ** rng.uniform(-2, 3.6)
    return r, r * (1.0 + rng.normal() * 1e-4)


@pytest.mark.parametrize("prob", [abi.PROB_GOLOVIN, abi.PROB_LONG, abi.PROB_CONST])
def test_bound_is_never_below_the_probability(prob):
    lib = K.oracle_lib()
    rng = np.random.default_rng(prob)
    msol = 1e-18
    for _ in range(40000):
        p = make_params(colltstep=float(rng.choice([0.1, 1.0, 10.0])), coll_prob=prob,
                        coaleff=float(rng.choice([1.0, 0.3])), const_kernel=1e-9)
        n = int(rng.integers(2, 3000))
        volume = 10.0 ** rng.uniform(-1, 7)
        r1, r2 = (float(r) for r in _radii(rng))
        xi = int(10.0 ** rng.uniform(0, 18))
        one = lib.oc_pair_probability(C.byref(p), r1, xi, msol, r2, xi, msol, volume / VOL0)
        scale = n * (n - 1.0) / (2.0 * (n // 2))
        assert _bound(p, n, volume, r1, r2, xi) >= scale * xi * one, (n, volume, r1, r2, xi)
