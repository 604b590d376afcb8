"""Quotients and square roots from shared reciprocals (cleo_b200/csrc/ddmath.h: quot, recip_from,
sqrt_recip_from), built for the host, against the IEEE operators, bit for bit: random operands over
the window and the significands where rounding is hardest, each with first approximations off by
up to the 2^-19 that the functions allow (the device's come from its approximate instructions,
whose error is about 2^-20). A quotient lies within the method's error of a rounding boundary, 2^-51
ulp, once in 10^15 operands, so none of these may differ."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "%s/cleo_b200/csrc/ddmath.h"
using namespace cleo;
static double first(double exact, double off) {  // the approximation's high word, moved by off
  return bitsd(dbits(exact * (1.0 + off)) & 0xFFFFFFFF00000000ull);
}
extern "C" uint64_t quotients(const double* a, const double* b, uint64_t n, double off) {
  uint64_t bad = 0;
  for (uint64_t i = 0; i < n; ++i)
    bad += dbits(quot(a[i], b[i], recip_from(b[i], first(1.0 / b[i], off)))) != dbits(a[i] / b[i]);
  return bad;
}
// a / b by a polished reciprocal; the operator where the divisor is all ones, as in the solver
static double by(double a, double b, double y) { return all_ones(b) ? a / b : quot(a, b, y); }
extern "C" uint64_t roots(const double* z, const double* a, uint64_t n, double off) {
  uint64_t bad = 0;
  for (uint64_t i = 0; i < n; ++i) {
    double s, y;
    sqrt_recip_from(z[i], first(1.0 / std::sqrt(z[i]), off), s, y);
    const double r = std::sqrt(z[i]);
    // the root, quotients by it and by its cube (a polished product of reciprocals)
    const double r3 = r * r * r;
    bad += dbits(s) != dbits(r) || dbits(by(a[i], s, y)) != dbits(a[i] / r) ||
           dbits(by(a[i], r3, recip_polish(r3, y * y * y))) != dbits(a[i] / r3);
  }
  return bad;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("recip")
    src, out = d / "recip.cpp", d / "librecip.so"
    src.write_text(SOURCE % ROOT)
    subprocess.run(["g++", "-O2", "-std=c++17", "-march=native", "-ffp-contract=off", "-fPIC",
                    "-shared", "-o", str(out), str(src)], check=True)
    lib = C.CDLL(str(out))
    for f in (lib.quotients, lib.roots):
        f.argtypes = [C.c_void_p, C.c_void_p, C.c_uint64, C.c_double]
        f.restype = C.c_uint64
    return lib


def _operands(span, n, rng, hard):
    """n doubles of either sign-free exponent range; hard: significands near powers of two, of
    ones, and of squares (where quotients and roots come closest to rounding boundaries)."""
    e = np.exp2(np.floor(rng.uniform(-span, span, n)))
    m = 1.0 + rng.random(n)
    if hard:
        k = rng.integers(0, 6, n)
        tiny = rng.integers(0, 64, n) * 2.0 ** -52
        short = np.round(m * 2.0 ** 26) * 2.0 ** -26
        m = np.select([k == 0, k == 1, k == 2, k == 3, k == 4],
                      [1.0 + tiny, 2.0 - (tiny + 2.0 ** -52), short, short * short / 2.0,
                       1.0 / m], m)
    return np.ascontiguousarray(e * m)


OFFSETS = (0.0, 2.0 ** -20, -(2.0 ** -20), 2.0 ** -19, -(2.0 ** -21))  # the cut adds up to 2^-20


@pytest.mark.parametrize("hard", [False, True])
@pytest.mark.parametrize("span", [3, 140])
def test_quotients_equal_the_operator(host, span, hard):
    rng = np.random.default_rng(span + hard)
    n = 1_000_000
    a, b = _operands(span, n, rng, hard), _operands(span, n, rng, hard)
    b[::2] *= -1.0
    a[:1000] = 0.0
    b[:1000] = np.abs(b[:1000])  # (a zero's sign is not kept; its only user adds it to 1)
    for off in OFFSETS:
        assert host.quotients(a.ctypes.data, b.ctypes.data, n, off) == 0, off


def _midpoint_significands():
    """Doubles z whose root lies within 2^-51 ulp of a rounding midpoint: with z scaled to an
    integer Z of 2^104 .. 2^106, a multiple of 2^52 or 2^53, Z = M^2 + M + k for k = 0 and 2
    (M^2 + M is even, so k is); M from M^2 + M + k = 0 mod 2^52 or 2^53, lifted bit by bit."""
    out = []
    for bits in (52, 53):
        for k in (0, 2, -2, 4, -4, 6, 8):
            sols = {0, 1}
            sols = {x for x in sols if (x * x + x + k) % 2 == 0}
            for j in range(2, bits + 1):
                sols = {y for x in sols for y in (x, x + (1 << (j - 1)))
                        if (y * y + y + k) % (1 << j) == 0}
            for x in sols:
                for m in (x, x + (1 << bits)):
                    big = m * m + m + k
                    if (1 << 52) <= m < (1 << 53) and (1 << 104) <= big < (1 << 106):
                        if big % (1 << (53 if big >= (1 << 105) else 52)) == 0:
                            out.append(float(big) * 2.0 ** -104)
    return out


@pytest.mark.parametrize("hard", [False, True])
def test_roots_and_their_quotients_equal_the_operators(host, hard):
    rng = np.random.default_rng(5 + hard)
    n = 1_000_000
    z, a = _operands(70, n, rng, hard), _operands(100, n, rng, hard)
    special = _midpoint_significands()
    assert len(special) >= 4
    s = np.concatenate([np.asarray(special) * 4.0 ** j for j in (-30, 0, 1, 30)])
    z[:s.size] = s
    for off in OFFSETS:
        assert host.roots(z.ctypes.data, a.ctypes.data, n, off) == 0, off
