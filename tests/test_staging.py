"""The pinned staging chain on the host, against a counting stand-in for the four CUDA calls it
makes: pinned memory stays within the limit however uploads grow, except for the one chunk of
an upload that is larger itself; a chunk is reused or freed only after the stream was waited for."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import configs  # noqa: F401  (puts the repository on the path)
from amrclaw_b200.build import CSRC, nvcc

SRC = """
#include "hostutil.hpp"
#include <map>
using namespace amrb;
static std::map<char*, size_t> live;     // pinned blocks
static std::map<char*, size_t> pending;  // staged since the stream was last waited for
static long long syncs = 0, frees = 0, faults = 0;
static size_t held() { size_t s = 0; for (auto& b : live) s += b.second; return s; }
extern "C" cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::malloc(n); live[(char*)*p] = n; return cudaSuccess; }
extern "C" cudaError_t cudaFreeHost(void* p) {
  ++frees;
  char* c = (char*)p;
  for (auto& q : pending) if (q.first >= c && q.first < c + live[c]) ++faults;
  live.erase(c);
  std::free(p);
  return cudaSuccess;
}
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t) { ++syncs; pending.clear(); return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "error"; }
static Staging* stg = nullptr;
extern "C" void start(long long soon) { stg = new Staging; stg->soon = (size_t)soon; syncs = frees = faults = 0; pending.clear(); }
// stages n bytes; returns the pinned bytes
extern "C" long long stage(const char* src, long long n) {
  char* p = (char*)stg->put(src, (size_t)n, nullptr);
  bool inside = false;
  for (auto& b : live) inside = inside || (p >= b.first && p + n <= b.first + b.second);
  for (auto& q : pending) if (p < q.first + q.second && q.first < p + n) ++faults;  // still being copied
  if (!inside || (n > 0 && std::memcmp(p, src, (size_t)n) != 0)) ++faults;
  pending[p] = (size_t)n;
  return (long long)held();
}
extern "C" void wait() { cudaStreamSynchronize(nullptr); stg->reset(); }
extern "C" void stop(long long* out) { pending.clear(); stg->destroy(); delete stg; out[0] = syncs; out[1] = frees; out[2] = faults; out[3] = (long long)held(); }
"""
MB = 1 << 20
LIMIT = 256 * MB


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("staging"))
    with open(d + "/staging.cpp", "w") as f:
        f.write(SRC)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), "include")
    # (bound to the stand-ins here, also where the process has loaded a CUDA runtime)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", CSRC, "-I", cuda, "-o", d + "/staging.so",
                    d + "/staging.cpp"], check=True)
    lib = ctypes.CDLL(d + "/staging.so")
    lib.stage.restype = ctypes.c_longlong
    return lib


def run(lib, sizes, soon=8 * MB, wait_every=0):
    src = np.random.default_rng(1).integers(0, 256, max(sizes), dtype=np.uint8)
    lib.start(ctypes.c_longlong(soon))
    held = []
    for k, n in enumerate(sizes):
        held.append(lib.stage(src.ctypes.data_as(ctypes.c_char_p), ctypes.c_longlong(n)))
        if wait_every and k % wait_every == wait_every - 1:
            lib.wait()
    out = (ctypes.c_longlong * 4)()
    lib.stop(out)
    assert out[2] == 0 and out[3] == 0
    return held, out[0]


@pytest.mark.parametrize("wait_every", [0, 1, 3])
def test_growing_uploads_stay_within_the_limit(lib, wait_every):
    held, _ = run(lib, [k * MB + 17 for k in (3, 20, 33, 47, 60, 75, 90, 110, 130, 150, 180)], wait_every=wait_every)
    assert max(held) <= LIMIT


def test_an_upload_past_the_limit_is_alone(lib):
    held, _ = run(lib, [30 * MB, 100 * MB, 260 * MB, 5 * MB, 300 * MB, 1000, 250 * MB])
    assert held[2] == 260 * MB and held[4] == 300 * MB
    assert max(held) == 300 * MB


def test_small_uploads_grow_with_use(lib):
    held, syncs = run(lib, [300_000] * 2000, wait_every=10)
    assert max(held) <= 8 * MB and syncs == 200  # ten of them fit: only the caller waits
    held, syncs = run(lib, [3 * MB] * 400, soon=32 * MB)
    assert held[-1] <= LIMIT and syncs < 60
    assert held == sorted(held)
