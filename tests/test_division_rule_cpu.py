"""div_shared of csrc/gi_dev.cuh itself (its text compiled for the host, with the device's built-ins as their C equivalents): the
quotients of three numerators by a shared divisor equal IEEE division bit for bit whichever way the guard sends them.  +0, -0,
negatives, subnormals, the numerators on both sides of 2^-80 and 2^60, infinities and NaN, alone and mixed in one vector; and
exactly the vectors of +0 and of numerators inside [2^-80, 2^60] go through the reciprocal."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <algorithm>
using std::min;
using std::max;
#define __device__
#define __forceinline__ inline
static inline uint32_t __float_as_uint(float x) { uint32_t u; memcpy(&u, &x, 4); return u; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
struct f3 { float x, y, z; };
static inline f3 mk(float x, float y, float z) { f3 r = {x, y, z}; return r; }
static uint64_t divided;
static inline f3 operator/(f3 a, float b) { divided++; return mk(a.x / b, a.y / b, a.z / b); }
"""
TAIL = r"""
extern "C" uint64_t rule(const float *x, uint64_t n, const float *b, uint64_t nb, uint64_t *through) {
  uint64_t bad = 0;
  divided = 0;
  for (uint64_t k = 0; k < nb; k++)
    for (uint64_t i = 0; i < n; i++) {
      volatile float one = 1.0f;
      const float d = b[k], r = one / d;
      const f3 q = div_shared(mk(x[3 * i], x[3 * i + 1], x[3 * i + 2]), d, r);
      const float got[3] = {q.x, q.y, q.z};
      for (int a = 0; a < 3; a++) {
        volatile float want = x[3 * i + a] / d;
        const float w = want;
        bad += !(__float_as_uint(got[a]) == __float_as_uint(w) || (got[a] != got[a] && w != w));
      }
    }
  *through = n * nb - divided;
  return bad;
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    text = open(os.path.join(ROOT, "real-time-gi-lab_b200", "csrc", "gi_dev.cuh")).read()
    a = text.index("__device__ __forceinline__ float div_step(")
    z = text.index("return x / b;", a)
    body = text[a:text.index("}\n", z) + 2]
    d = tmp_path_factory.mktemp("rule")
    src, so = os.path.join(d, "rule.cpp"), os.path.join(d, "rule.so")
    with open(src, "w") as fh:
        fh.write(HEAD + body + TAIL)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", so, src, "-lm"], check=True)
    lib = C.CDLL(so)
    lib.rule.restype = C.c_uint64

    def run(x, b):
        x, b = np.ascontiguousarray(x, np.float32), np.ascontiguousarray(b, np.float32)
        t = C.c_uint64()
        bad = lib.rule(x.ctypes.data_as(C.c_void_p), C.c_uint64(x.size // 3), b.ctypes.data_as(C.c_void_p), C.c_uint64(b.size), C.byref(t))
        return int(bad), int(t.value)
    return run


EDGES = np.array([0x00000000, 0x80000000, 0x00000001, 0x80000001, 0x007fffff, 0x00800000, 0x177fffff, 0x17800000, 0x17800001,
                  0x3f800000, 0xbf800000, 0x5d7fffff, 0x5d800000, 0x5d800001, 0x7f7fffff, 0xff7fffff, 0x7f800000, 0xff800000,
                  0x7fc00000, 0xffc00000], np.uint32).view(np.float32)


def _divisors(rng, n):
    e = rng.integers(-30, 4, n)   # weight sums lie in [1e-9, 8]
    m = rng.integers(0, 1 << 23, n)
    m[:4] = [0, 1, 0x7fffff, 0x7ffffe]
    return np.clip((((e + 127) << 23) | m).astype(np.uint32).view(np.float32), np.float32(1e-9), np.float32(8.0))


def test_edges_mixed(rule):
    x = np.stack(np.meshgrid(EDGES, EDGES, EDGES, indexing="ij"), -1).reshape(-1, 3)
    b = _divisors(np.random.default_rng(1), 40)
    u = x.view(np.uint32)
    taken = ((u == 0) | ((u >= 0x17800000) & (u <= 0x5d800000))).all(1).sum()
    bad, through = rule(x, b)
    assert bad == 0
    assert through == taken * b.size


@pytest.mark.parametrize("lo,hi", [(0x17800000 - 4096, 0x17800000 + 4096), (0x5d800000 - 4096, 0x5d800000 + 4096), (0x3f000000, 0x42000000)])
def test_ranges(rule, lo, hi):
    rng = np.random.default_rng(lo & 0xffff)
    x = rng.integers(lo, hi, (60000, 3)).astype(np.uint32)
    x[::3] |= np.uint32(0x80000000)                     # every third vector with its numerators negated
    x[1::7, 1] = 0                                      # and +0 beside others
    bad, through = rule(x.view(np.float32), _divisors(rng, 25))
    assert bad == 0
    assert through > 0


@pytest.mark.parametrize("m", [0x000000, 0x000001, 0x7fffff, 0x7ffffe, 0x555555, 0x4ccccd, 0x6dbb5a])
def test_binade(rule, m):
    """A whole binade of numerators (three in a vector) for one divisor: the hard cases of the last rounding are among them."""
    x = np.arange(0x3f800000, 0x40000000, dtype=np.uint32)[:(1 << 23) // 3 * 3]
    bad, through = rule(x.view(np.float32), np.array([(127 << 23) | m], np.uint32).view(np.float32))
    assert bad == 0
    assert through == x.size // 3
