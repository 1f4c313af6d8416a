"""csrc/ieee64.cuh on the GPU: div64 and sqrt64 have the bits of IEEE division
and square root (numpy on the host rounds correctly), for random operands, for
quotients and roots next to representable numbers and to midpoints between
them, and for everything the fast path leaves alone (zeros, infinities, NaN,
subnormals, the ends of the exponent range, powers of two)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "ieee64.cuh"
using namespace mafm;
__global__ void k(const double* a, const double* b, double* q, double* s, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        q[i] = div64(a[i], b[i]);
        s[i] = sqrt64(a[i]);
    }
}
extern "C" int run(const double* a, const double* b, double* q, double* s, int n) {
    double* d;
    const size_t bytes = (size_t)n * sizeof(double);
    if (cudaMalloc(&d, 4 * bytes) != cudaSuccess) return 1;
    cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
    k<<<304, 256>>>(d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, n);
    cudaMemcpy(q, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
    cudaMemcpy(s, d + 3 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
    const int e = cudaGetLastError() != cudaSuccess;
    cudaFree(d);
    return e;
}
"""


@pytest.fixture(scope="module")
def gpu(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    tmp = tmp_path_factory.mktemp("ieee64")
    (tmp / "k.cu").write_text(SOURCE)
    so = str(tmp / "libk.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-fmad=false", "-shared", "-Xcompiler",
                    "-fPIC", "-I", os.path.join(ROOT, "mechafm_gb300", "csrc"), str(tmp / "k.cu"), "-o", so], check=True)
    fn = C.CDLL(so).run
    p = C.POINTER(C.c_double)
    fn.argtypes = [p, p, p, p, C.c_int]

    def call(a, b):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        q, s = np.empty_like(a), np.empty_like(a)
        assert fn(*[x.ctypes.data_as(p) for x in (a, b, q, s)], len(a)) == 0
        return q, s
    return call


def nudge(x, by):
    return (x.view(np.int64) + by).view(np.float64)


def operands(kind, rng, n):
    unit = lambda: rng.integers(0, 1 << 52, n, dtype=np.uint64)  # noqa: E731
    mant = lambda u: (u | np.uint64(1023 << 52)).view(np.float64)  # noqa: E731
    if kind == "ordinary":
        return np.ldexp(mant(unit()), rng.integers(-60, 60, n)) * rng.choice([-1.0, 1.0], n), \
            np.ldexp(mant(unit()), rng.integers(-60, 60, n)) * rng.choice([-1.0, 1.0], n)
    if kind == "any bits":
        return tuple(rng.integers(0, 1 << 64, n, dtype=np.uint64).view(np.float64) for _ in range(2))
    if kind == "exponent limits":
        e = [-1074, -1023, -1022, -501, -500, -499, -1, 0, 1, 499, 500, 501, 1023]
        return np.ldexp(mant(unit()), rng.choice(e, n)), np.ldexp(mant(unit()), rng.choice(e, n))
    if kind == "near quotients":      # a next to b times a 27-bit number or a 28-bit one (a midpoint's neighbour)
        b = mant(unit() & np.uint64(0xffffffffff000000 & (2 ** 52 - 1)))
        return nudge(b * mant(unit() & np.uint64((2 ** 52 - 1) ^ (2 ** 25 - 1))), rng.integers(-2, 3, n)), b
    if kind == "near roots":          # a next to a square, b of few bits
        r = mant(unit() & np.uint64((2 ** 52 - 1) ^ (2 ** 26 - 1)))
        return nudge(r * r, rng.integers(-2, 3, n)), mant(rng.integers(0, 16, n, dtype=np.uint64))
    if kind == "all-ones mantissas":
        return np.ldexp(nudge(np.full(n, 2.0), -rng.integers(1, 9, n)), rng.integers(-9, 9, n)), \
            np.ldexp(nudge(np.full(n, 2.0), -rng.integers(1, 9, n)), rng.integers(-9, 9, n))
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308, 1.0, -1.0, 2.0,
                        4.0, 0.5, 3.0, 1.7976931348623157e308, nudge(np.array([4.0]), -1)[0]])
    a, b = np.meshgrid(special, special)
    return a.reshape(-1), b.reshape(-1)


@pytest.mark.parametrize("kind", ["ordinary", "any bits", "exponent limits", "near quotients", "near roots",
                                  "all-ones mantissas", "special"])
def test_bits_of_division_and_root(gpu, kind):
    a, b = operands(kind, np.random.default_rng(len(kind)), 1 << 21)
    q, s = gpu(a, b)
    with np.errstate(all="ignore"):
        for got, want in ((q, a / b), (s, np.sqrt(a))):
            both_nan = np.isnan(got) & np.isnan(want)
            np.testing.assert_array_equal(got.view(np.int64)[~both_nan], want.view(np.int64)[~both_nan])
