"""The quick form of the 3D Euler splits, in both precisions: its quotient against the division at
the edges of the ranges it is guarded by, and whole splits against the general form."""
import ctypes
import subprocess

import numpy as np
import pytest

import configs  # noqa: F401  (puts the repository on the path)
from amrclaw_b200.build import ARCH, CSRC, nvcc

pytestmark = pytest.mark.gpu

SRC = """
#include "riemann3d.cuh"
#include <cstdio>
using namespace amrb;
template <class T>
__global__ void quotients(const T* x, const T* a, T* q, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) q[t] = SplitRange<T>::a_ok(a[t]) ? split_quotient(x[t], a[t], split_recip(a[t])) : T(-1);
}
// d split at the interface of states l and r, both ways: out [n][2][10]; quick: taken there
template <class T>
__global__ void splits(T g1, const T* l, const T* r, const T* d, T* out, int* quick, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  T L[6], R[6], D[5];
  L[0] = R[0] = T(0);
  for (int m = 0; m < 5; ++m) { L[m + 1] = l[5 * t + m]; R[m + 1] = r[5 * t + m]; D[m] = d[5 * t + m]; }
  const Roe3T<T> o = roe3d(g1, L, R);
  const int ixyz = 1 + t % 3, icoor = 2 + (t / 3) % 2;
  quick[t] = euler3d_trans_sub(o, ixyz);
  T m[5], p[5];
  for (int k = 0; k < 2; ++k) {
    if (k == 0) euler3d_trans<false>(o, split_recip(o.a), ixyz, icoor, D, m, p);
    else euler3d_trans<true>(o, split_recip(o.a), ixyz, icoor, D, m, p);
    for (int c = 0; c < 5; ++c) { out[20 * t + 10 * k + c] = m[c]; out[20 * t + 10 * k + 5 + c] = p[c]; }
  }
}
template <class T>
static int run_q(const T* x, const T* a, T* q, int n) {
  try {
    T *dx, *da, *dq;
    AMR_CUDA(cudaMalloc((void**)&dx, sizeof(T) * n)); AMR_CUDA(cudaMalloc((void**)&da, sizeof(T) * n)); AMR_CUDA(cudaMalloc((void**)&dq, sizeof(T) * n));
    AMR_CUDA(cudaMemcpy(dx, x, sizeof(T) * n, cudaMemcpyHostToDevice)); AMR_CUDA(cudaMemcpy(da, a, sizeof(T) * n, cudaMemcpyHostToDevice));
    quotients<T><<<(n + 127) / 128, 128>>>(dx, da, dq, n);
    AMR_CUDA(cudaMemcpy(q, dq, sizeof(T) * n, cudaMemcpyDeviceToHost));
    cudaFree(dx); cudaFree(da); cudaFree(dq);
  } catch (std::exception& e) { std::fprintf(stderr, "%s\\n", e.what()); return 1; }
  return 0;
}
template <class T>
static int run_s(T g1, const T* l, const T* r, const T* d, T* out, int* quick, int n) {
  try {
    T* b; int* dk;
    AMR_CUDA(cudaMalloc((void**)&b, sizeof(T) * 35 * n)); AMR_CUDA(cudaMalloc((void**)&dk, sizeof(int) * n));
    AMR_CUDA(cudaMemcpy(b, l, sizeof(T) * 5 * n, cudaMemcpyHostToDevice));
    AMR_CUDA(cudaMemcpy(b + 5 * n, r, sizeof(T) * 5 * n, cudaMemcpyHostToDevice));
    AMR_CUDA(cudaMemcpy(b + 10 * n, d, sizeof(T) * 5 * n, cudaMemcpyHostToDevice));
    splits<T><<<(n + 127) / 128, 128>>>(g1, b, b + 5 * n, b + 10 * n, b + 15 * n, dk, n);
    AMR_CUDA(cudaMemcpy(out, b + 15 * n, sizeof(T) * 20 * n, cudaMemcpyDeviceToHost));
    AMR_CUDA(cudaMemcpy(quick, dk, sizeof(int) * n, cudaMemcpyDeviceToHost));
    cudaFree(b); cudaFree(dk);
  } catch (std::exception& e) { std::fprintf(stderr, "%s\\n", e.what()); return 1; }
  return 0;
}
extern "C" int q64(const double* x, const double* a, double* q, int n) { return run_q(x, a, q, n); }
extern "C" int q32(const float* x, const float* a, float* q, int n) { return run_q(x, a, q, n); }
extern "C" int s64(double g, const double* l, const double* r, const double* d, double* o, int* k, int n) { return run_s(g, l, r, d, o, k, n); }
extern "C" int s32(float g, const float* l, const float* r, const float* d, float* o, int* k, int n) { return run_s(g, l, r, d, o, k, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("splits"))
    with open(d + "/splits.cu", "w") as f:
        f.write(SRC)
    subprocess.run([nvcc(), "-std=c++17", "-O3", *ARCH, "--fmad=false", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, "-o",
                    d + "/splits.so", d + "/splits.cu"], check=True)
    return ctypes.CDLL(d + "/splits.so")


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


# the guarded exponents of x and of a, and the largest and smallest of the format
RANGES = {np.float64: ((-900, 900), (-40, 40), (-1074, 1023)), np.float32: ((-70, 90), (-10, 20), (-149, 127))}


@pytest.mark.parametrize("T", [np.float64, np.float32])
def test_quotients(lib, T):
    (x0, x1), (a0, a1), (f0, f1) = RANGES[T]
    rng = np.random.default_rng(7)
    n = 200000
    one = T(1)

    def values(exps, count):
        return np.ldexp((1 + rng.random(count)).astype(T), rng.choice(exps, count)).astype(T)

    a = np.concatenate([values(np.arange(a0, a1), n), values([a0, a0 + 1, a1 - 2, a1 - 1], n)])
    a[a >= np.ldexp(one, a1)] = np.ldexp(one, a1 - 1)
    a[:4] = np.ldexp(one, a0), np.nextafter(np.ldexp(one, a1), T(0)), np.nextafter(np.ldexp(one, a0), T(9)), one
    with np.errstate(under="ignore", over="ignore"):
        x = np.concatenate([values(np.arange(x0, x1), n), values([x0 - 2, x0 - 1, x0, x0 + 1, x1 - 2, x1 - 1, x1, f0, f0 + 9, f1], n)])
        # numerators close to a multiple of 2a: the quotients that are hardest to round
        near = (T(2) * a[::7] * values(np.arange(-3, 4), len(a[::7]))).astype(T)
        x[::7] = np.nextafter(near, np.where(rng.random(len(near)) < 0.5, T(-np.inf), T(np.inf)).astype(T))
        x *= np.where(rng.random(2 * n) < 0.5, T(-1), one)
        p = rng.permutation(2 * n)
        x = x[p]
        x[:8] = 0, -0.0, np.inf, -np.inf, np.nan, np.nextafter(T(0), one), np.ldexp(one, x0), np.nextafter(np.ldexp(one, x1), T(0))
        want = x / (T(2) * a)
    assert x.dtype == a.dtype == want.dtype == T
    q = np.zeros_like(x)
    assert (lib.q64 if T is np.float64 else lib.q32)(_p(x), _p(a), _p(q), len(x)) == 0
    finite = np.isfinite(x)
    assert np.array_equal(q[finite], want[finite])
    assert np.isnan(q[~finite]).all()


@pytest.mark.parametrize("T", [np.float64, np.float32])
def test_splits(lib, T):
    rng = np.random.default_rng(11)
    n = 100000

    def states():
        rho, pr = 10 ** rng.uniform(-2, 2, n), 10 ** rng.uniform(-2, 2, n)
        u = rng.uniform(-0.9, 0.9, (3, n)) * np.sqrt(1.4 * pr / rho)
        return np.stack([rho, *(rho * u), pr / 0.4 + 0.5 * rho * (u ** 2).sum(axis=0)], axis=1).astype(T)

    l = states()
    r = (l * (1 + 1e-2 * rng.uniform(-1, 1, (n, 1)))).astype(T)
    d = (rng.normal(size=(n, 5)) * 10 ** rng.uniform(-12, 3, (n, 1))).astype(T)
    d[rng.random((n, 5)) < 0.1] = 0
    d[:100] = 0
    out, quick = np.zeros((n, 2, 10), T), np.zeros(n, np.int32)
    g1 = (ctypes.c_double if T is np.float64 else ctypes.c_float)(0.4)
    assert (lib.s64 if T is np.float64 else lib.s32)(g1, _p(l), _p(r), _p(d), _p(out), _p(quick), n) == 0
    assert quick.sum() > 0.5 * n
    out = out[quick == 1]
    assert np.isfinite(out).all() and np.array_equal(out[:, 0], out[:, 1])
