"""Rules that the compiler does not check.

* Every header that a translation unit includes is listed in build.py, so that
  a change of it recompiles what includes it.
* A kernel launched with the programmatic attribute (EngineT::launch) waits for
  the kernels before it, in every block and before anything that can return or
  touch what they write, and lets the next one come after that."""
import os
import re

import pytest

from polgraw_gb300 import build

CSRC = os.path.join(build.HERE, "csrc")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_headers_are_listed():
    want = set()
    for n in os.listdir(CSRC):
        if n.endswith((".cu", ".cuh", ".h")):
            want |= set(re.findall(r'#include "(pa_[\w.]+)"', _text(n)))
    assert {"pa_engine.cuh", "pa_sincos.cuh"} <= want
    assert want <= {os.path.basename(h) for h in build.HEADERS}


def _body(text, name):
    m = re.search(r"__global__[^;{]*?\b%s\(" % name, text)
    assert m, name
    i = text.index("{", text.index(")", m.end()))
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j]
    raise AssertionError(name)


@pytest.mark.parametrize("name,file", [("k_prelude_mod", "pa_engine.cuh"), ("k_pair_a", "pa_pair.cuh"),
                                       ("k_pair_b", "pa_pair.cuh"), ("k_resample", "pa_engine.cuh"),
                                       ("k_normthresh", "pa_engine.cuh")])
def test_dependent_kernels_wait_first(name, file):
    body = _body(_text(file), name)
    wait, go = body.index("pdl_wait()"), body.index("pdl_go()")
    before = body[:wait]
    assert wait < go and body.count("pdl_wait()") == 1
    assert "return" not in before and "for (;;)" not in before
    # nothing that a kernel writes (tables and inputs only), no stores
    assert not re.findall(r"\b(shftf|part|xin|odd|spec|yint|ybuf|xm|ph0|F|sums|sums_r|cand|ncand|counter)\s*\[", before)
    assert set(re.findall(r"ldg\w*\(&?(\w+)", before)) <= {"tw2"}


def test_dependent_kernels_are_these():
    launched = set(re.findall(r"\blaunch\((k_\w+|ka|kb)\b", _text("pa_engine.cuh")))
    assert launched == {"k_prelude_mod", "k_resample", "k_normthresh", "ka", "kb"}
