"""The kernels' division by a shared divisor (csrc/gi_dev.cuh div_step, div_shared), restated in C with fmaf and compiled here:
its quotients equal IEEE division bit for bit over whole binades of numerators, for divisors across the range it takes
(random mantissas, all-ones and one-bit mantissas), and at the ends of the numerators it takes."""
import ctypes as C
import os
import subprocess

import pytest

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
static float f(uint32_t u) { float x; memcpy(&x, &u, 4); return x; }
static uint32_t b(float x) { uint32_t u; memcpy(&u, &x, 4); return u; }
static float step(float x, float d, float r) {
  float q0 = x * r;
  float q1 = fmaf(fmaf(-q0, d, x), r, q0);
  return fmaf(fmaf(-q1, d, x), r, q1);
}
/* numerators: n consecutive floats from bits u0 (and, every third, its negative); returns how many quotients differ */
uint64_t shared_diff(float d, uint32_t u0, uint32_t n, uint32_t stride) {
  volatile float one = 1.0f;
  float r = one / d;
  uint64_t bad = 0;
  for (uint32_t i = 0; i < n; i++) {
    float x = f(u0 + i * stride);
    volatile float q = x / d;
    bad += b(step(x, d, r)) != b(q);
  }
  return bad;
}
float from_bits(uint32_t u) { return f(u); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    src = os.path.join(d, "division.c")
    with open(src, "w") as fh:
        fh.write(SRC)
    so = os.path.join(d, "division.so")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", so, src, "-lm"], check=True)
    h = C.CDLL(so)
    h.shared_diff.argtypes = [C.c_float, C.c_uint32, C.c_uint32, C.c_uint32]
    h.shared_diff.restype = C.c_uint64
    h.from_bits.argtypes = [C.c_uint32]
    h.from_bits.restype = C.c_float
    return h


# divisor mantissas: 1, the next ones, all ones, alternating bits, and a few arbitrary ones
MANTISSAS = [0x000000, 0x000001, 0x7fffff, 0x7ffffe, 0x555555, 0x2aaaaa, 0x400000, 0x3fffff, 0x4ccccd, 0x123456, 0x6dbb5a]


@pytest.mark.parametrize("exponent", [-30, -27, -13, -1, 0, 1, 3])   # weight sums lie in [1e-9, 8]
@pytest.mark.parametrize("m", MANTISSAS)
def test_shared_division_equals_ieee(lib, exponent, m):
    d = lib.from_bits(((exponent + 127) << 23) | m)
    assert lib.shared_diff(d, 127 << 23, 1 << 20, 8) == 0                 # a binade at every eighth numerator
    assert lib.shared_diff(d, 0x17800000, 1 << 16, 1) == 0                # the smallest numerators taken, 2^-80 ..
    assert lib.shared_diff(d, 0x5d800000 - (1 << 16), 1 << 16, 1) == 0    # the largest, .. 2^60
    assert lib.shared_diff(d, 0, 1, 1) == 0                               # +0


def test_shared_division_whole_binade(lib):
    d = lib.from_bits((127 << 23) | 0x4ccccd)
    assert lib.shared_diff(d, 130 << 23, 1 << 23, 1) == 0
