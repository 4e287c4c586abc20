"""A plugin that has what include/amrgpu_riemann.cuh asks for, and nothing else, goes through the
step kernels' templates: the compiler's front end instantiates them on it."""
import os
import subprocess
import tempfile

import configs  # noqa: F401  (puts the repository on the path)
from amrclaw_b200.build import CSRC, nvcc

PLUGIN3 = """
#include "kernels3d.cu"
namespace amrb {
template <class R>
struct Contract3 {
  static constexpr int NV = 2, NW = 1;
  R un;
  template <int DIR>
  __device__ void load(const R*, const PatchDev&, long long, long long, long long, int e) { un = R(e); }
  template <int DIR>
  __device__ void rpn(const Step3Params&, const R* QL, const R* QR, R (&W)[NW][NV], R* S, R* AM, R* AP) {
    S[0] = un;
    for (int m = 0; m < NV; ++m) { W[0][m] = QR[m + 1] - QL[m + 1]; AM[m] = R(0); AP[m] = un * W[0][m]; }
  }
  template <int DIR>
  __device__ void rpt(int, int, const R* in, R* m, R* p) const { for (int k = 0; k < NV; ++k) { m[k] = R(0); p[k] = un * in[k]; } }
  template <int DIR>
  __device__ void rptt(int, int, int, const R* in, R* m, R* p) const { for (int k = 0; k < NV; ++k) { m[k] = R(0); p[k] = un * in[k]; } }
};
static_assert(amrgpu_plugin::Check3D<Contract3<double>, Step3Params, double>::value, "");
static_assert(amrgpu_plugin::Check3D<Contract3<float>, Step3Params, float>::value, "");
// a limiter for each wave of a larger plugin
static_assert(sizeof(Step3Params::mthlim) / sizeof(int) >= 8, "");
template int launch_step3_t<double, Contract3<double>>(const Step3Args&, const long long*, long long, long long, cudaStream_t);
template int launch_step3_t<float, Contract3<float>>(const Step3Args&, const long long*, long long, long long, cudaStream_t);
}
"""

PLUGIN2 = """
#include "kernels2d.cu"
namespace amrb {
template <int NE, int NWV>
struct Contract2 {
  static constexpr int MEQN = NE, MWAVES = NWV, NAUX = 0;
  template <class R>
  __device__ static void rpn(const ProbDev&, int, const R* qL, const R* qR, const R*, const R*, R (&wave)[MWAVES][MEQN],
                             R (&s)[MWAVES], R (&amdq)[MEQN], R (&apdq)[MEQN]) {
    for (int k = 0; k < MWAVES; ++k) { s[k] = R(1); for (int m = 0; m < MEQN; ++m) wave[k][m] = (qR[m] - qL[m]) / R(MWAVES); }
    for (int m = 0; m < MEQN; ++m) { amdq[m] = R(0); apdq[m] = qR[m] - qL[m]; }
  }
  template <class R>
  __device__ static void rpt(const ProbDev&, int, int, const R*, const R*, const R*, const R*, const R*, const R* asdq,
                             R (&bm)[MEQN], R (&bp)[MEQN]) {
    for (int m = 0; m < MEQN; ++m) { bm[m] = R(0); bp[m] = asdq[m]; }
  }
};
// a block's shared memory holds a tile of these, as it did with the tile's waves in chunks of rows
template <class S> constexpr bool unsplit_fits() { return Step2Layout<S>::TOTAL * 8 <= 232448 - 512; }
template <class S> constexpr bool split_fits() { return Split2Layout<S>::TOTAL * 8 <= 232448 - 512; }
static_assert(unsplit_fits<Contract2<8, 7>>() && unsplit_fits<Contract2<8, 5>>() && unsplit_fits<Contract2<10, 1>>(), "");
static_assert(split_fits<Contract2<7, 7>>() && split_fits<Contract2<8, 7>>() && split_fits<Contract2<10, 5>>(), "");
static_assert(split_fits<Contract2<11, 3>>() && split_fits<Contract2<12, 1>>(), "");
// the plugins of this library have all their waves there at once
static_assert(Step2Layout<Euler2>::WG == 4 && Split2Layout<Euler2>::WG == 4 && Split2Layout<Acoustics2>::WG == 2, "");
// a limiter for each wave of a larger plugin
static_assert(sizeof(StepParams::mthlim) / sizeof(int) >= 8, "");
static_assert(amrgpu_plugin::Check2D<Contract2<8, 5>, ProbDev, double>::value, "");
template void launch_step2_t<Contract2<8, 5>, double>(const StepArgs&, int, cudaStream_t);
template void launch_step2_t<Contract2<8, 5>, float>(const StepArgs&, int, cudaStream_t);
template void launch_step2_batch_t<Contract2<8, 5>, double>(const StepBatch&, int, cudaStream_t);
}
"""


def _front_end(src):
    """Compiles to intermediate code without optimising it (nothing is kept)."""
    with tempfile.TemporaryDirectory() as d:
        with open(d + "/plugin.cu", "w") as f:
            f.write(src)
        r = subprocess.run([nvcc(), "-std=c++17", "-arch=compute_100a", "-ptx", "-G", "--fmad=false", "-I", CSRC, "-o", os.devnull,
                            d + "/plugin.cu"], capture_output=True, text=True)
    return r.returncode, r.stderr


def test_3d_plugin_of_the_contract_alone():
    rc, err = _front_end(PLUGIN3.replace("const long long*", "const long long*"))
    assert rc == 0, err


def test_2d_plugin_of_the_contract_alone():
    rc, err = _front_end(PLUGIN2)
    assert rc == 0, err
