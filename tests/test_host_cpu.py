"""The widening of packed depths on the host, compiled with the vector
instructions of the host it is built on and without any (as on hosts that have
others): the same numbers, for each width, at every remainder of the vector
loops and from every start that a thread may have.  No source includes the
vector header but the one that has both branches."""
import ctypes as C
import glob
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "graph_analytics_applesilicon_b200", "csrc")


@pytest.fixture(scope="module", params=["as built", "no vectors"])
def widen(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("widen")
    (d / "w.cpp").write_text('#include "host_cpu.hpp"\n'
                             'extern "C" void widen(int f, const uint8_t* in, uint64_t lo, uint64_t hi, uint32_t* out)'
                             ' { gb::cpuPause(); gb::widenRange(f, in, lo, hi, out); }\n')
    so = str(d / "w.so")
    flags = [] if request.param == "as built" else ["-U__SSE2__"]
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + CSRC, str(d / "w.cpp"), "-o", so] + flags, check=True)
    f = C.CDLL(so).widen
    f.argtypes = [C.c_int, C.c_void_p, C.c_uint64, C.c_uint64, C.c_void_p]
    f.restype = None
    return f


@pytest.mark.parametrize("fmt", [0, 1, 2])
def test_widths_and_remainders(widen, fmt):
    rng = np.random.default_rng(fmt)
    top = (15, 255, 65535)[fmt]
    for n in list(range(1, 70)) + [1000, 4099]:
        d = rng.integers(0, top + 1, n)  # the largest is the sentinel
        d[rng.random(n) < 0.2] = top
        want = np.where(d == top, 0xFFFFFFFF, d).astype(np.uint32)
        if fmt == 0:
            e = np.append(d, 0) if n % 2 else d
            packed = (e[0::2] | e[1::2] << 4).astype(np.uint8)
        else:
            packed = d.astype((np.uint8, np.uint16)[fmt - 1])
        for lo in range(0, n, 32):
            out = np.full(n + 1, 7, np.uint32)
            widen(fmt, packed.ctypes.data, lo, n, out.ctypes.data)
            assert np.array_equal(out[lo:n], want[lo:]) and (out[:lo] == 7).all() and out[n] == 7


def test_vector_instructions_stay_behind_a_branch():
    for p in glob.glob(os.path.join(CSRC, "*")):
        if os.path.basename(p) != "host_cpu.hpp" and os.path.isfile(p):
            text = open(p).read()
            assert "mmintrin" not in text and "_mm_" not in text, p
