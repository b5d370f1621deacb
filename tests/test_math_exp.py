"""trg_exp's short evaluation (torch_b200/csrc/trg_math.h) returns what the
long one, trg_exp_dd, returns: over the arguments it serves, at the ends of
its range, next to zero and next to multiples of ln2/128, where the reduced
argument changes sign."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest

import common

HDR = os.path.join(common.ROOT, "torch_b200", "csrc", "trg_math.h")
SRC = r"""
#include "%s"
long differ(const double* x, long n) {
    long d = 0;
    for (long i = 0; i < n; ++i) {
        const double a = trg_exp(x[i]), b = trg_exp_dd(x[i], 0.0);
        d += !(a == b || (a != a && b != b));
    }
    return d;
}
""" % HDR


@pytest.fixture(scope="module")
def differ():
    d = tempfile.mkdtemp(prefix="trg_exp_")
    src, so = os.path.join(d, "m.c"), os.path.join(d, "m.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-o", so, src, "-lm"], check=True)
    fn = C.CDLL(so).differ
    fn.restype, fn.argtypes = C.c_long, [C.c_void_p, C.c_long]
    return lambda x: fn(np.ascontiguousarray(x, dtype=np.float64).ctypes.data, len(x))


@pytest.mark.parametrize("lo,hi", [(-746, 710), (-40, 0), (-1, 1), (-1e-3, 1e-3), (-708.01, -707.99), (708.9, 709.9)])
def test_short_exp_equals_the_long_one(differ, lo, hi):
    assert differ(np.random.default_rng(3).uniform(lo, hi, 400_000)) == 0


def test_short_exp_at_special_arguments(differ):
    k = np.arange(-130_000, 130_000) * (np.log(2.0) / 128)
    near = np.concatenate([k, np.nextafter(k, np.inf), np.nextafter(k, -np.inf), k + np.log(2.0) / 256])
    tiny = 10.0 ** np.random.default_rng(4).uniform(-320, -8, 100_000)
    special = [0.0, -0.0, np.inf, -np.inf, np.nan, -708.0, np.nextafter(-708.0, 0), 709.0, 709.79, -745.2, 5e-324]
    assert differ(near) == 0 and differ(tiny) == 0 and differ(-tiny) == 0 and differ(special) == 0
