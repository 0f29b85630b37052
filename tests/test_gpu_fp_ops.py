"""The reciprocals, roots and quotients of the hot kernels on the device
(csrc/fp_ops.cuh, compiled here into a kernel of its own): recip, root and quot
against the IEEE 1/x, sqrt(fmax(0, x)) and x/d bit for bit, and root_inverse and
near_recip against what they stand for, CUDA's rsqrt and a reciprocal shared by
two quotients: no further from the exact value, by the largest, the mean and the
number of misrounded results over the same operands.  Over the whole range that
their comments give, and at its ends."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "how-mhd-kokkos_b200" / "csrc"
SRC = r"""
#include "fp_ops.cuh"
#include <cstddef>
__global__ void k(int op, size_t n, const double* x, const double* d, double* out) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    using namespace how;
    out[i] = op == 0 ? near_recip(x[i]) : op == 1 ? recip(x[i]) : op == 2 ? root_inverse(x[i])
           : op == 3 ? root(x[i]) : op == 4 ? quot(x[i], d[i], recip(d[i])) : op == 5 ? larger(x[i], d[i])
           : op == 6 ? (double)root((float)x[i]) : op == 7 ? rsqrt(x[i]) : d[i] * (1.0 / (x[i] * d[i]));
}
extern "C" int run(int op, size_t n, const double* x, const double* d, double* out) {
    double *gx = nullptr, *gd = nullptr, *go = nullptr;
    const size_t b = n * sizeof(double);
    cudaError_t e = cudaMalloc(&gx, b);
    if (!e) e = cudaMalloc(&gd, b);
    if (!e) e = cudaMalloc(&go, b);
    if (!e) e = cudaMemcpy(gx, x, b, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(gd, d, b, cudaMemcpyHostToDevice);
    if (!e) { k<<<(unsigned)((n + 255) / 256), 256>>>(op, n, gx, gd, go); e = cudaGetLastError(); }
    if (!e) e = cudaMemcpy(out, go, b, cudaMemcpyDeviceToHost);
    cudaFree(gx); cudaFree(gd); cudaFree(go);
    return (int)e;
}
"""
NEAR_RECIP, RECIP, ROOT_INVERSE, ROOT, QUOT, LARGER, ROOT32, RSQRT, SHARED_RECIP = range(9)


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not found")
    d = tmp_path_factory.mktemp("fp_ops")
    (d / "k.cu").write_text(SRC)
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false",
                    "-I", str(CSRC), "-shared", "-Xcompiler", "-fPIC", "-o", str(d / "k.so"), str(d / "k.cu")],
                   check=True)
    lib = ctypes.CDLL(str(d / "k.so"))
    P = ctypes.POINTER(ctypes.c_double)

    def call(op, x, y=None):
        x = np.ascontiguousarray(x, np.float64)
        y = np.ascontiguousarray(np.ones_like(x) if y is None else y, np.float64)
        out = np.empty_like(x)
        assert lib.run(ctypes.c_int(op), ctypes.c_size_t(x.size), *(a.ctypes.data_as(P) for a in (x, y, out))) == 0
        return out
    return call


def _normals(lo, hi, n=2_000_000, seed=1):
    """Positive, exponents lo..hi-1 evenly, a quarter of the significands next to one and two."""
    rng = np.random.default_rng(seed)
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    m[0::4] |= np.uint64(0xFFFFFFFFFFF00)
    m[1::4] &= np.uint64(0x00000000000FF)
    m[2::64] = np.uint64(0xFFFFFFFFFFFFF)
    m[3::64] = np.uint64(0)
    e = rng.integers(lo + 1023, hi + 1023, n, dtype=np.uint64)
    return ((e << np.uint64(52)) | m).view(np.float64)


def _ulps(got, want):
    """|got - want| in units of the last place of `want` (a long double)."""
    _, e = np.frexp(want)
    return np.abs((got.astype(np.longdouble) - want) * np.ldexp(np.longdouble(1), 53 - e))


def _no_further(a, b, want):
    a, b = _ulps(a, want), _ulps(b, want)
    assert a.max() <= b.max() and a.mean() <= b.mean() and (a > 0.5).sum() <= (b > 0.5).sum()


def _same(a, b):
    np.testing.assert_array_equal(a.view(np.uint64), b.view(np.uint64))


def test_reciprocals(run):
    x = _normals(-1022, 1022)
    x[::2] *= -1
    _same(run(RECIP, x), 1.0 / x)
    x, d = _normals(-300, 300, seed=6), _normals(-300, 300, seed=7)
    _no_further(run(NEAR_RECIP, x), run(SHARED_RECIP, x, d), 1 / x.astype(np.longdouble))


def test_roots(run):
    x = _normals(-960, 1024)     # (below, the remainder of the correction is subnormal)
    _same(run(ROOT, x), np.sqrt(x))
    x = _normals(-1022, 1024, seed=8)
    _no_further(run(ROOT_INVERSE, x), run(RSQRT, x), 1 / np.sqrt(x.astype(np.longdouble)))
    low = _normals(-1022, -960, 100_000)
    assert _ulps(run(ROOT, low), np.sqrt(low.astype(np.longdouble))).max() <= 1.0


def test_ends_of_the_roots(run):
    x = np.array([0.0, -0.0, -1.0, -5e-324, -np.inf, np.nan, -np.nan, np.inf, 5e-324, 1e-310,
                  np.finfo(np.float64).max, np.finfo(np.float64).tiny])
    want = np.array([0, 0, 0, 0, 0, 0, 0, np.inf, 0, 0, np.sqrt(np.finfo(np.float64).max),
                     np.sqrt(np.finfo(np.float64).tiny)])
    _same(run(ROOT, x), want)
    x32 = np.array([0.0, -0.0, -1.0, -np.inf, np.nan, np.inf, 4.0, 2.25])
    _same(run(ROOT32, x32), np.array([0, 0, 0, 0, 0, np.inf, 2.0, 1.5]))


def test_quotients(run):
    d = _normals(-300, 300, seed=2)
    x = _normals(-600, 600, seed=3)
    x[::2] *= -1
    x[::97] = 0.0
    _same(run(QUOT, x, d) + 0.0, x / d + 0.0)
    # a quotient that overflows is infinite; a tiny one is within a unit of 2^-1074 |y|
    assert (run(QUOT, np.array([1e300, -1e300]), np.array([1e-300, 1e-300])) == [np.inf, -np.inf]).all()
    d = _normals(0, 40, 100_000, seed=4)
    x = _normals(-1022, -940, 100_000, seed=5)
    y = (x.astype(np.longdouble) / d).astype(np.longdouble)
    assert (np.abs(run(QUOT, x, d) - y) <= np.maximum(np.abs(y) * 2.0 ** -52, np.longdouble(2.0) ** -1074 * 1.5)).all()


def test_larger_of_non_negative_values(run):
    a = np.array([0.0, 1.0, 2.0, np.inf, 1e-310, 3.0])
    b = np.array([0.0, 2.0, 1.0, 5.0, 0.0, np.inf])
    _same(run(LARGER, a, b), np.maximum(a, b))
