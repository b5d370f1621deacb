"""Division of cell indices by the grid's fixed extents (DivBy in
torch_b200/csrc/trg_types.h) against the integer division: every small
divisor, divisors around powers of two, and the indices around multiples and
at the top of the 31-bit range, where a wrong multiplier shows."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest

import common

SRC = r"""
#include "%s"
extern "C" long wrong(unsigned d, const unsigned* n, long count) {
    const trg::DivBy by = trg::make_div_by(d);
    long w = 0;
    for (long i = 0; i < count; ++i) w += trg::div_by(n[i], by) != n[i] / d;
    return w;
}
""" % os.path.join(common.ROOT, "torch_b200", "csrc", "trg_types.h")


@pytest.fixture(scope="module")
def wrong():
    d = tempfile.mkdtemp(prefix="div_by_")
    src, so = os.path.join(d, "m.cpp"), os.path.join(d, "m.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so, src], check=True)
    fn = C.CDLL(so).wrong
    fn.restype, fn.argtypes = C.c_long, [C.c_uint, C.c_void_p, C.c_long]

    def count(d, n):
        a = np.ascontiguousarray(n, dtype=np.uint32)  # held over the call
        return fn(d, a.ctypes.data, len(a))

    return count


def indices(d, rng):
    top = (1 << 31) - 1
    q = np.concatenate([np.arange(0, 40), rng.integers(0, top // d + 1, 200), [top // d]]).astype(np.int64)
    n = np.concatenate([q * d - 1, q * d, q * d + 1, q * d + d - 1, [0, top - 1, top]])
    return n[(n >= 0) & (n <= top)]


@pytest.mark.parametrize("divisors", ["small", "powers"])
def test_div_by_equals_division(wrong, divisors):
    rng = np.random.default_rng(1)
    ds = range(1, 3000) if divisors == "small" else sorted(
        {d for k in range(31) for d in ((1 << k) - 1, 1 << k, (1 << k) + 1) if 1 <= d < (1 << 31)} | {(1 << 31) - 1})
    for d in ds:
        assert wrong(d, indices(d, rng)) == 0, d
