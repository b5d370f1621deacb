"""Division through a shared reciprocal (Recip, over_gm1 in
torch_b200/csrc/trg_device.cuh) against the correctly rounded quotient, as
bits: random operands, quotients next to the midpoint of two doubles, divisors
whose significand is all ones or next to it, both ends of the exponents the
short form takes, subnormals, infinities, NaN and zeros of either sign.  The
host's division (IEEE 754) and the device's built-in one are the references."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu

CSRC = os.path.join(common.ROOT, "torch_b200", "csrc")
SRC = r"""
#include "trg_device.cuh"
using namespace trg;
__global__ void k_recip(const double* a, const double* b, long n, double* div, double* own) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    Recip r;
    r.set(b[i]);
    div[i] = r.div(a[i]);
    own[i] = a[i] / b[i];
}
__global__ void k_gm1(Params P, const double* a, long n, double* out) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i < n) out[i] = over_gm1(P, a[i]);
}
static double* up(const double* h, long n) {
    double* d = nullptr;
    cudaMalloc(&d, n * sizeof(double));
    if (h) cudaMemcpy(d, h, n * sizeof(double), cudaMemcpyHostToDevice);
    return d;
}
static void down(double* h, double* d, long n) {
    if (h) cudaMemcpy(h, d, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
}
extern "C" int recip(const double* a, const double* b, long n, double* div, double* own) {
    double *da = up(a, n), *db = up(b, n), *d0 = up(nullptr, n), *d1 = up(nullptr, n);
    k_recip<<<(unsigned)((n + 255) / 256), 256>>>(da, db, n, d0, d1);
    down(div, d0, n); down(own, d1, n);
    down(nullptr, da, n); down(nullptr, db, n);
    return (int)cudaGetLastError();
}
extern "C" int gm1(double gamma, const double* a, long n, double* out) {
    Params P{};
    P.gamma = gamma;
    P.gm1_rcp = 1.0 / (gamma - 1.0);
    double *da = up(a, n), *d0 = up(nullptr, n);
    k_gm1<<<(unsigned)((n + 255) / 256), 256>>>(P, da, n, d0);
    down(out, d0, n); down(nullptr, da, n);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module", params=["--fmad=false", "--fmad=true"])
def lib(request, tmp_path_factory):
    """The header compiled as each build of the kernels does."""
    d = tmp_path_factory.mktemp("recip")
    (d / "r.cu").write_text(SRC)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", request.param,
                    "-Xcompiler", "-fPIC,-ffp-contract=off", "-I", CSRC, "-shared", "-o", str(d / "r.so"),
                    str(d / "r.cu")], check=True)
    return C.CDLL(str(d / "r.so"))


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def same_bits(x, y):
    return (x.view(np.uint64) == y.view(np.uint64)) | (np.isnan(x) & np.isnan(y))


def check(lib, a, b):
    a, b = (np.ascontiguousarray(np.broadcast_to(v, np.broadcast(a, b).shape), dtype=np.float64).ravel() for v in (a, b))
    out = [np.empty_like(a) for _ in range(2)]
    assert lib.recip(ptr(a), ptr(b), C.c_long(a.size), *[ptr(o) for o in out]) == 0
    with np.errstate(all="ignore"):
        want = a / b
    for name, got in zip(("shared", "built-in"), out):
        bad = np.nonzero(~same_bits(got, want))[0]
        assert bad.size == 0, (name, bad.size, [(a[i].hex(), b[i].hex(), got[i].hex(), want[i].hex()) for i in bad[:4]])


def significands(rng, n):
    return 1.0 + rng.integers(0, 1 << 52, n) * 2.0 ** -52


def test_random_operands(lib):
    rng = np.random.default_rng(11)
    for _ in range(4):
        n = 1 << 21
        e = rng.integers(-490, 490, (2, n))
        sgn = rng.choice([-1.0, 1.0], (2, n))
        check(lib, np.ldexp(sgn[0] * significands(rng, n), e[0]), np.ldexp(sgn[1] * significands(rng, n), e[1]))


def test_quotients_next_to_midpoints(lib):
    """a the double next to (q + half an ulp) b, and its neighbours."""
    rng = np.random.default_rng(12)
    a, b = [], []
    for _ in range(120000):
        q = 2 * int(rng.integers(1 << 52, 1 << 53)) + 1  # 54 bits, odd: a midpoint
        d = int(rng.integers(1 << 52, 1 << 53)) | 1
        p = q * d
        s = p.bit_length() - 53
        for k in (-1, 0, 1):
            a.append(float((p >> s) + k) * 2.0 ** (s - 105))
            b.append(float(d) * 2.0 ** -52)
    check(lib, np.array(a), np.array(b))


def test_divisors_next_to_all_ones(lib):
    rng = np.random.default_rng(13)
    k = np.arange(64)
    near = np.concatenate([2.0 - (k + 1) * 2.0 ** -52, 1.0 + k * 2.0 ** -52,
                           1.0 + (rng.integers(0, 1 << 20, 64) * 2.0 ** 32 + (2.0 ** 32 - 1)) * 2.0 ** -52])
    for e in (-480, -3, 0, 7, 480):
        check(lib, significands(rng, 40000)[:, None][:4000], np.ldexp(near, e)[None, :])


def test_ends_of_the_exponents(lib):
    rng = np.random.default_rng(14)
    ends = np.concatenate([np.ldexp(significands(rng, 40), e) for e in
                           (-1074, -1030, -1022, -1000, -540, -502, -501, -500, -499, -1, 0, 1, 498, 499, 500, 501, 900, 1022,
                            1023)] + [np.ldexp([1.0, 2.0 - 2.0 ** -52], e) for e in (-501, -500, 499, 500)])
    ends = np.concatenate([ends, -ends])
    check(lib, ends[:, None], ends[None, :])


def test_zeros_infinities_and_nan(lib):
    v = np.array([0.0, -0.0, 1.0, -1.0, 3.0, -3.0, 5e-324, -5e-324, 1e-300, 1e300, np.inf, -np.inf, np.nan, 0.1, -0.7])
    check(lib, v[:, None], v[None, :])


@pytest.mark.parametrize("gamma", [1.67, 5.0 / 3.0, 1.4, 1.0001, 1.1, 2.0, 3.0, 1.0 + 2.0 ** -20])
def test_division_by_gamma_minus_one(lib, gamma):
    rng = np.random.default_rng(15)
    a = np.concatenate([np.ldexp(significands(rng, 100000), rng.integers(-480, 480, 100000)),
                        [0.0, -0.0, np.inf, np.nan, 1e-310, -1e-200]])
    out = np.empty_like(a)
    assert lib.gm1(C.c_double(gamma), ptr(a), C.c_long(a.size), ptr(out)) == 0
    assert np.all(same_bits(out, a / (gamma - 1.0)))
