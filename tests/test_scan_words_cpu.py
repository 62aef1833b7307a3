"""The chained scans' states lie in a buffer of scan_cap + 1 words: a rebuild whose scans would have more parts is refused before
anything is launched, and gi_vox_build_noalloc takes clipmaps up to 2^25 pointers, as its static scratch allows."""
import ctypes as C
import os
import subprocess

import pytest

from rtgi import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "real-time-gi-lab_b200", "csrc")

SRC = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstring>
#include "gi_dev.cuh"
#include "gi_internal.h"
// stands in for the launch: a rebuild that is not refused must not reach a device here
int main() {
  struct { unsigned levels, G, max_bricks, cap; } c[] = {
      {1, 16, 256, 15},        // 4,096 pointers, 256 a part: 16 parts
      {4, 16, 256, 15},        // 16,384 pointers, 1,024 a part: 16 parts
      {8, 128, 256, 4095},     // 16.8 M pointers, 4,096 a part: 4,096 parts
      {1, 4, 4097, 16},        // 4,097 bricks, 256 a part: 17 parts
  };
  for (auto &k : c) {
    gi::VoxDev v;
    gi::SceneDev s;
    memset((void *)&v, 0, sizeof v);
    memset((void *)&s, 0, sizeof s);
    v.levels = k.levels; v.G = k.G; v.max_bricks = k.max_bricks; v.scan_cap = k.cap; v.blocks = 8;
    printf("%d\n", (int)gi_launch_vox_build(v, s, 148u, 0));
  }
}
"""


def test_more_parts_than_words_are_refused(tmp_path):
    import torch
    if torch.cuda.is_available():
        pytest.skip("host-side check; a build without the refusal would launch on null buffers")
    lib = os.path.join(ROOT, "real-time-gi-lab_b200", "lib")
    src, exe = tmp_path / "parts.cu", tmp_path / "parts"
    src.write_text(SRC)
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", CSRC, "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe), "-L", lib, "-lgi_b200",
                    "-Xlinker", "-rpath=" + lib], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["1"] * 4, out   # cudaErrorInvalidValue


@pytest.mark.parametrize("levels,G,word", [(2, 256, b"16-byte aligned"), (3, 256, b"exceeds the static scratch"),
                                           (8, 160, b"16-byte aligned"), (8, 164, b"exceeds the static scratch")])
def test_noalloc_pointer_limit(levels, G, word):
    lib = _lib.load()
    p = _lib.GiVoxParams(0.1, levels, G, 4096, 1 << 20, 0, 0)
    eye = (C.c_double * 3)(0.0, 0.0, 0.0)
    ok, odd = C.c_void_p(16), C.c_void_p(20)   # never dereferenced: a buffer off its alignment is refused after the sizes
    st = lib.gi_vox_build_noalloc(C.byref(p), eye, odd, ok, 0, ok, 0, ok, 1, *([ok] * 8), None)
    assert st == _lib.GI_ERR_INVALID
    assert word in lib.gi_last_error()
