"""The 2D step of plugins whose waves do not all fit in shared memory at once: five waves that
each carry two of ten components (in FP32 seven, of fourteen) give every pair of components what
a plugin with that one wave alone gives it, in the unsplit and the split step, order 1 and 2."""
import ctypes
import subprocess

import numpy as np
import pytest

import configs  # noqa: F401  (puts the repository on the path)
from amrclaw_b200.build import ARCH, CSRC, nvcc

pytestmark = pytest.mark.gpu

SRC = """
#include "kernels2d.cu"
#include <vector>
namespace amrb {
// components 2k and 2k+1 move with wave k, in x at speed c(k), in y at d(k); FIRST: the wave the
// plugin starts with
template <int NWV, int FIRST>
struct Pairs {
  static constexpr int MEQN = 2 * NWV, MWAVES = NWV, NAUX = 0;
  template <class R>
  __device__ static R speed(int ixy, int k) { k += FIRST; return ixy == 1 ? R(0.3) * R(k + 1) - R(0.7) : R(0.9) - R(0.4) * R(k); }
  template <class R>
  __device__ static void rpn(const ProbDev&, int ixy, const R* qL, const R* qR, const R*, const R*, R (&wave)[MWAVES][MEQN],
                             R (&s)[MWAVES], R (&amdq)[MEQN], R (&apdq)[MEQN]) {
    for (int k = 0; k < MWAVES; ++k) {
      s[k] = speed<R>(ixy, k);
      for (int m = 0; m < MEQN; ++m) wave[k][m] = m / 2 == k ? qR[m] - qL[m] : R(0);
    }
    for (int m = 0; m < MEQN; ++m) {
      amdq[m] = dmin(s[m / 2], R(0)) * wave[m / 2][m];
      apdq[m] = dmax(s[m / 2], R(0)) * wave[m / 2][m];
    }
  }
  template <class R>
  __device__ static void rpt(const ProbDev&, int ixy, int, const R*, const R*, const R*, const R*, const R*, const R* asdq,
                             R (&bm)[MEQN], R (&bp)[MEQN]) {
    for (int m = 0; m < MEQN; ++m) {
      const R v = speed<R>(3 - ixy, m / 2);
      bm[m] = dmin(v, R(0)) * asdq[m];
      bp[m] = dmax(v, R(0)) * asdq[m];
    }
  }
};
static_assert(Step2Layout<Pairs<7, 0>>::WG < 7 && Split2Layout<Pairs<5, 0>>::WG < 5, "these go through their waves in groups");
static_assert(Step2Layout<Pairs<1, 0>>::WG == 1, "");

template <class S, class R>
static int step(R* q, int mx, int my, int order, int trans, int split) {
  // one patch, its two buffers one after the other in the pool; q: [m][my+4][mx+4], in and out
  const long long plane = (long long)(mx + 4) * (my + 4), n = S::MEQN * plane;
  try {
    R* pool; PatchDev* patches; StepWork* work; unsigned long long* cfl;
    AMR_CUDA(cudaMalloc((void**)&pool, sizeof(R) * (2 * n + 64)));
    AMR_CUDA(cudaMalloc((void**)&patches, sizeof(PatchDev)));
    std::vector<StepWork> w;
    for (int j = 1; j <= my; j += TILE2) for (int i = 1; i <= mx; i += TILE2) w.push_back(StepWork{0, i, j, 0, 0, 0, 0});
    AMR_CUDA(cudaMalloc((void**)&work, sizeof(StepWork) * w.size()));
    AMR_CUDA(cudaMalloc((void**)&cfl, 8));
    AMR_CUDA(cudaMemset(cfl, 0, 8));
    const long long second = (n + 31) / 32 * 32;
    PatchDev P{};
    P.q[0] = 0; P.q[1] = second; P.ffl = P.aux = -1; P.ihi = mx - 1; P.jhi = my - 1; P.mitot = mx + 4; P.mjtot = my + 4; P.mktot = 1;
    P.level = 1;
    AMR_CUDA(cudaMemcpy(patches, &P, sizeof(P), cudaMemcpyHostToDevice));
    AMR_CUDA(cudaMemcpy(work, w.data(), sizeof(StepWork) * w.size(), cudaMemcpyHostToDevice));
    AMR_CUDA(cudaMemcpy(pool, q, sizeof(R) * n, cudaMemcpyHostToDevice));
    AMR_CUDA(cudaMemcpy(pool + second, q, sizeof(R) * n, cudaMemcpyHostToDevice));
    StepArgs a{};
    a.pool = pool; a.patches = patches; a.work = work; a.nwork = (int)w.size(); a.dt = 0.25; a.dx = 0.5; a.dy = 0.4; a.cflmax = cfl;
    for (int& l : a.sp.mthlim) l = 4;
    a.sp.order = order; a.sp.trans = trans; a.sp.split = split;
    launch_step2_t<S, R>(a, (int)w.size(), 0);
    AMR_CUDA(cudaDeviceSynchronize());
    AMR_CUDA(cudaMemcpy(q, pool + second, sizeof(R) * n, cudaMemcpyDeviceToHost));
    cudaFree(pool); cudaFree(patches); cudaFree(work); cudaFree(cfl);
  } catch (std::exception& e) { std::fprintf(stderr, "%s\\n", e.what()); return 1; }
  return 0;
}
template <int W, int N, class R>
static int one(R* q, int mx, int my, int order, int trans, int split, int k) {
  if (k == W) return step<Pairs<1, W>, R>(q, mx, my, order, trans, split);
  if constexpr (W + 1 < N) return one<W + 1, N>(q, mx, my, order, trans, split, k);
  return 2;
}
extern "C" int run_all64(double* q, int mx, int my, int order, int trans, int split) {
  return step<Pairs<5, 0>, double>(q, mx, my, order, trans, split);
}
extern "C" int run_one64(double* q, int mx, int my, int order, int trans, int split, int k) {
  return one<0, 5>(q, mx, my, order, trans, split, k);
}
extern "C" int run_all32(float* q, int mx, int my, int order, int trans, int split) {
  return step<Pairs<7, 0>, float>(q, mx, my, order, trans, split);
}
extern "C" int run_one32(float* q, int mx, int my, int order, int trans, int split, int k) {
  return one<0, 7>(q, mx, my, order, trans, split, k);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("waves"))
    with open(d + "/waves.cu", "w") as f:
        f.write(SRC)
    subprocess.run([nvcc(), "-std=c++17", "-O1", *ARCH, "--fmad=false", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, "-o",
                    d + "/waves.so", d + "/waves.cu"], check=True)
    return ctypes.CDLL(d + "/waves.so")


@pytest.mark.parametrize("bits,waves", [(64, 5), (32, 7)])
@pytest.mark.parametrize("mx,my", [(1, 1), (16, 16), (17, 15), (40, 37)])
@pytest.mark.parametrize("order,trans,split", [(2, 2, 0), (2, 1, 0), (1, 0, 0), (2, 0, 1), (1, 0, 1)])
def test_pairs_of_components(lib, mx, my, order, trans, split, bits, waves):
    run_all, run_one = (lib.run_all64, lib.run_one64) if bits == 64 else (lib.run_all32, lib.run_one32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    q = np.random.default_rng(mx + my).normal(size=(2 * waves, my + 4, mx + 4)).astype("f%d" % (bits // 8))
    together = q.copy()
    assert run_all(p(together), mx, my, order, trans, split) == 0
    inside = (slice(None), slice(2, my + 2), slice(2, mx + 2))
    assert not np.array_equal(together[inside], q[inside])
    for k in range(waves):
        pair = np.ascontiguousarray(q[2 * k:2 * k + 2])
        assert run_one(p(pair), mx, my, order, trans, split, k) == 0
        assert np.array_equal(pair[inside], together[2 * k:2 * k + 2][inside]), k
