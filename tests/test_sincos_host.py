"""The FP64 forms' sine and cosine (sincos_fast in csrc/pa_sincos.cuh), built for
the host, against extended precision: every entry of its table, between them,
both signs, up to and across the 2^25 from which on the library's take over.

Tolerance: the last addition rounds to half a unit in the last place, 5.6e-17
below 1; its second term is below 0.0123 and rounds to 9e-19, and so do the two
fused operations that form it; the polynomials' and the reduction's parts are
smaller: 8e-17."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "polgraw-allsky_gb300", "csrc")

SHIM = r'''
#include <cmath>
#include <cstdio>
#include <cstring>
#define __device__
#define __noinline__
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))
struct double2 { double x, y; };
static const double2& __ldg(const double2* p) { return *p; }
static long long bits(double d) { long long b; memcpy(&b, &d, 8); return b; }
static int __double2hiint(double d) { return (int)(bits(d) >> 32); }
static int __double2loint(double d) { return (int)(unsigned)bits(d); }
'''

MAIN = r'''
int main() {
  double x, o[2];
  while (fread(&x, 8, 1, stdin) == 1) {
    pa::sincos_fast(x, &o[0], &o[1]);
    fwrite(o, 8, 2, stdout);
  }
}
'''


def test_against_extended_precision(tmp_path):
    cxx = shutil.which("g++")
    if not cxx or np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no host compiler, or no extended precision")
    text = re.sub(r"#(include|pragma)[^\n]*", "", open(os.path.join(CSRC, "pa_sincos.cuh")).read())
    src, exe = tmp_path / "sc.cpp", tmp_path / "sc"
    src.write_text(SHIM + text + MAIN)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-fno-strict-aliasing", "-fconstexpr-ops-limit=200000000",
                    str(src), "-o", str(exe)], check=True)
    rng = np.random.default_rng(2)
    step = 2 * np.pi / 256
    k = np.arange(-300, 301) * step
    x = np.concatenate([k, k + step / 2, np.nextafter(k + step / 2, 9), k + rng.uniform(-step / 2, step / 2, k.size),
                        rng.uniform(-50, 50, 20000), 2.0 ** rng.uniform(-60, 25, 20000) * rng.choice([-1, 1], 20000),
                        [0.0, 1e-310, np.nextafter(2.0 ** 25, 0), -np.nextafter(2.0 ** 25, 0), 2.0 ** 25, -2.0 ** 25 - 1,
                         1e15]])
    out = subprocess.run([str(exe)], input=x.tobytes(), stdout=subprocess.PIPE, check=True).stdout
    got = np.frombuffer(out).reshape(-1, 2)
    lx = x.astype(np.longdouble)
    for f, col in ((np.sin, 0), (np.cos, 1)):
        assert np.max(np.abs(got[:, col] - f(lx))) <= 8e-17
    special = np.array([np.inf, -np.inf, np.nan])
    out = subprocess.run([str(exe)], input=special.tobytes(), stdout=subprocess.PIPE, check=True).stdout
    assert np.isnan(np.frombuffer(out)).all()
