"""The error flags of the kernels: all of them are read and reset together, and a code names one wait."""
import ctypes as C
import os
import re
import subprocess

import fa_b200_capi as capi

SRC = os.path.join(os.path.dirname(capi.__file__), "csrc")
HARNESS = r"""
#include "error_flags.h"
static int state[4];
template <int I> static int flag(bool clear) { const int v = state[I]; if (clear) state[I] = 0; return v; }
extern "C" int run(int* io, int clear) {
    static int (*const flags[])(bool) = {flag<0>, flag<1>, flag<2>, flag<3>};
    for (int i = 0; i < 4; ++i) state[i] = io[i];
    const int code = fa::first_error(flags, 4, clear != 0);
    for (int i = 0; i < 4; ++i) io[i] = state[i];
    return code;
}
"""


def test_every_flag_is_reset_whatever_the_others_hold(tmp_path):
    src, so = tmp_path / "h.cpp", tmp_path / "h.so"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", SRC, str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    for mask in range(16):
        held = [7 * (i + 1) if mask >> i & 1 else 0 for i in range(4)]
        io = (C.c_int * 4)(*held)
        want = next((x for x in held if x), 0)
        assert lib.run(io, 0) == want and list(io) == held
        assert lib.run(io, 1) == want and list(io) == [0] * 4


def test_every_kernel_with_an_error_flag_is_asked():
    """A flag that the merge leaves out would never be reported or reset."""
    text = {f: open(os.path.join(SRC, f)).read() for f in os.listdir(SRC) if f.endswith(".cu")}
    readers = {m for t in text.values() for m in re.findall(r"int (\w+_error_flag)\(bool clear\) \{", t)} - {"any_error_flag"}
    asked = {m for t in text.values() for lst in re.findall(r"flags\[\]\)\(bool\) = \{([^}]*)\}", t) for m in re.findall(r"\w+_error_flag", lst)}
    assert readers == asked and len(readers) >= 7


def test_a_wait_code_belongs_to_one_kernel():
    """Kernels whose flags are reported through one function number their waits apart (the latent decode's, older, overlap the
    backward's)."""
    seen = {}
    for f in sorted(os.listdir(SRC)):
        if f.endswith(".cu") and f != "mla_sm100_pair.cu":
            for code in set(re.findall(r"err, (\d+)\)", open(os.path.join(SRC, f)).read())):
                assert seen.setdefault(code, f) == f, (code, f, seen[code])
    assert len(seen) >= 50
