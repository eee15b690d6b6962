"""The coincidence kernels' split of a double into two floats by its bits
(ff_of in csrc/pa_coinc.cu), built for the host: high part (float)d, low part
(float)(d - high), for every exponent that the bits are used for and the ones
beside it, both signs, ties of both parts; no undefined arithmetic (the build
traps on it)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "polgraw-allsky_gb300", "csrc")

SHIM = r'''
#include <cstdio>
#include <cstring>
#define __device__
#define __noinline__
#define __forceinline__ inline
template <class T, class F> static T bits(F f) { T t; memcpy(&t, &f, sizeof t); return t; }
static long long __double_as_longlong(double d) { return bits<long long>(d); }
static float __int_as_float(int i) { return bits<float>(i); }
static float __uint_as_float(unsigned i) { return bits<float>(i); }
static int __float_as_int(float f) { return bits<int>(f); }
static unsigned __float_as_uint(float f) { return bits<unsigned>(f); }
'''

MAIN = r'''
int main() {
  double d;
  while (fread(&d, 8, 1, stdin) == 1) {
    const FF f = ff_of(d);
    fwrite(&f, 8, 1, stdout);
  }
}
'''


def test_split_by_bits(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    text = open(os.path.join(CSRC, "pa_coinc.cu")).read()
    i, j = text.index("// a number as the sum of two floats"), text.index("// Order key of a double")
    src, exe = tmp_path / "ff.cpp", tmp_path / "ff"
    src.write_text(SHIM + text[i:j] + MAIN)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-Wall", "-Werror", "-Wno-unused-function", "-fsanitize=undefined",
                    "-fsanitize-undefined-trap-on-error", str(src), "-o", str(exe)], check=True)
    rng = np.random.default_rng(1)
    m = np.concatenate([rng.integers(0, 2 ** 52, 200), [0, 1, 2 ** 28, 2 ** 28 - 1, 2 ** 28 + 1, 2 ** 29, 3 * 2 ** 28,
                                                        2 ** 52 - 1, 2 ** 52 - 2 ** 28, 2 ** 52 - 2 ** 28 - 1]]).astype(np.uint64)
    e = np.arange(940, 1152, dtype=np.uint64)
    d = ((e[:, None] << np.uint64(52)) | m[None, :]).ravel().view(np.float64)
    d = np.concatenate([d, -d, [0.0, -0.0, 5e-324]])
    out = subprocess.run([str(exe)], input=d.tobytes(), stdout=subprocess.PIPE, check=True).stdout
    got = np.frombuffer(out, np.float32).reshape(-1, 2)
    with np.errstate(over="ignore", invalid="ignore"):
        h = d.astype(np.float32)
        low = (d - h.astype(np.float64)).astype(np.float32)
    assert np.array_equal(got[:, 0], h)
    assert np.array_equal(got[:, 1], low, equal_nan=True)
