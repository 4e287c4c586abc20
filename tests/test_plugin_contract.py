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
template int launch_step3_t<double, Contract3<double>>(const Step3Args&, const long long*, long long, long long, cudaStream_t);
template int launch_step3_t<float, Contract3<float>>(const Step3Args&, const long long*, long long, long long, cudaStream_t);
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
