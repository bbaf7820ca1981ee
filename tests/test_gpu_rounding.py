"""The correctly rounded operations of csrc/fixed_point.cuh and the FP32 rounding of
csrc/pimc_device.cuh against IEEE arithmetic on the host, bit for bit."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "pi-qmc_gb300", "csrc")

PROGRAM = r"""
#include "pimc_device.cuh"
using namespace pimc;
__global__ void apply(int op, int n, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = op == 0 ? reciprocal(a[i]) : op == 1 ? divide(a[i], b[i])
         : op == 2 ? square_root(a[i]) : (double)f32_rn(a[i]);
}
extern "C" int run(int op, int n, const double* a, const double* b, double* out) {
  double *da = nullptr, *db = nullptr, *dout = nullptr;
  const size_t bytes = (size_t)n * sizeof(double);
  int bad = cudaMalloc(&da, bytes) || cudaMalloc(&db, bytes) || cudaMalloc(&dout, bytes);
  if (!bad) {
    cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
    apply<<<(n + 255) / 256, 256>>>(op, n, da, db, dout);
    bad = cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost) != cudaSuccess;
  }
  cudaFree(da);
  cudaFree(db);
  cudaFree(dout);
  return bad;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    import pimc_gb300.build as B
    d = tmp_path_factory.mktemp("rounding")
    src, lib = d / "rounding.cu", d / "rounding.so"
    src.write_text(PROGRAM)
    subprocess.run([B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", CSRC, "-o", str(lib), str(src)], check=True, capture_output=True)
    f = C.CDLL(str(lib)).run
    f.argtypes = [C.c_int, C.c_int] + 3 * [C.POINTER(C.c_double)]
    f.restype = C.c_int

    def call(op, a, b=None):
        a = np.ascontiguousarray(a, np.float64)
        b = np.ascontiguousarray(a if b is None else b, np.float64)
        out = np.empty_like(a)
        p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in (a, b, out)]
        assert f(op, len(a), *p) == 0
        return out
    return call


def _values(rng, n):
    """Any bit pattern, ordinary magnitudes, powers of two and their neighbours, the ends
    of the normal and subnormal ranges, zeros, infinities and NaN."""
    bits = rng.integers(0, 1 << 64, n, np.uint64).view(np.float64)
    mid = np.exp(rng.uniform(-40, 40, n)) * rng.choice([-1.0, 1.0], n)
    two = np.ldexp(1.0, np.arange(-1074, 1024))
    two = np.concatenate([two, np.nextafter(two, 0), np.nextafter(two, np.inf)])
    tiny = np.finfo(float).tiny
    ends = np.array([0.0, tiny, np.nextafter(tiny, 0), 5e-324, np.finfo(float).max, np.inf, np.nan,
                     np.finfo(np.float32).max, np.finfo(np.float32).tiny, 2.0 ** -149, 2.0 ** -150])
    ends = np.concatenate([ends, np.nextafter(ends[:-2], np.inf)])
    v = np.concatenate([bits, mid, two, -two, ends, -ends])
    return v[rng.permutation(len(v))]


def _same(got, want):
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2])
def test_correct_rounding(run, seed):
    rng = np.random.default_rng(seed)
    n = 1 << 20
    with np.errstate(all="ignore"):
        v, w = _values(rng, n), _values(rng, n)
        # results near their rounding boundaries: of a product or a square, and its neighbours
        x = np.ldexp(rng.integers(1 << 52, 1 << 53, n).astype(float), rng.integers(-80, 20, n))
        y = np.ldexp(rng.integers(1 << 52, 1 << 53, n).astype(float), rng.integers(-80, 20, n))
        step = rng.integers(-3, 4, n)
        prod = ((x * y).view(np.int64) + step).view(np.float64)
        square = ((x * x).view(np.int64) + step).view(np.float64)
        small = rng.integers(1, 1 << 26, n).astype(float)  # exact squares and quotients
        v = np.concatenate([v, x, small])
        _same(run(0, v), 1.0 / v)
        a = np.concatenate([_values(rng, n)[:len(w)], prod, small * np.floor(y / x * 64)])
        b = np.concatenate([w, x, small])
        _same(run(1, a, b), a / b)
        # quotients next to the middle of two doubles: (q + half a unit) b for small b
        q = rng.integers(1 << 52, 1 << 53, n)
        d = rng.integers(1, 1 << 9, n) * 2 + 1
        a = np.ldexp(((2 * (q >> 10) + 1) * d).astype(float), -1)
        _same(run(1, a, d.astype(float)), a / d)
        r = np.concatenate([_values(rng, n), square, small * small])
        _same(run(2, r), np.sqrt(r))
        f = np.concatenate([_values(rng, n),
                            # 24 bits and a half, and its neighbours
                            (np.ldexp(rng.integers(1 << 24, 1 << 25, n).astype(float) * 1.0,
                                      rng.integers(-170, 100, n)).view(np.int64) + step)
                            .view(np.float64)])
        _same(run(3, f), f.astype(np.float32).astype(np.float64))
