// Host side of the one-launch bisection (bisect_kernel, flags3d.cu): its device buffers, the
// launch and the read-back of the tree, and the clusters in the reference's order.
#pragma once
#include "flags3d.cuh"
#include "hostutil.hpp"

namespace amrb {

struct DeviceBisect {
  // Limits of the device form; a bisection past them is done by waves on the host instead.
  static constexpr int MAX_NODES = 16384, MAX_HIST = 1 << 18, MAX_DIM = 1 << 20, MAX_PLANE = 1 << 19;
  static constexpr long long MAX_POINTS = 2 << 20;
  int max_nodes = MAX_NODES;                   // (a test asks for less of these two)
  long long max_wait = BISECT_MAX_WAIT;
  int launched = 0;                            // kernels of the last run
  DBuf<char> tree;                  // BisectHead, then the nodes
  DBuf<unsigned long long> pts;
  DBuf<int> node_of, hist;
  void free() { tree.free(); pts.free(); node_of.free(); hist.free(); }

  // Whether the device form takes a level of dims d; npts: the points of a 2D list (those of
  // a 3D level are counted on the device).
  static bool takes(int ndim, LvlDims d, size_t npts) {
    const int dims[3] = {d.is, d.js, ndim == 3 ? d.ks : 1};
    long long cells = 1, plane = 0, len = 0;
    for (int k = 0; k < ndim; ++k) { cells *= dims[k]; len += dims[k]; if (dims[k] >= MAX_DIM) return false; }
    for (int k = 0; k < ndim; ++k) plane = std::max(plane, cells / dims[k]);  // most points with one index
    return plane <= MAX_PLANE && len <= MAX_HIST && (ndim == 3 || (long long)npts <= MAX_POINTS);
  }
  // ndim 3: the flagged cells of level array f; ndim 2: list (bisect_point). False if the
  // limits do not hold or ran out, or the launch gave up waiting.
  bool run(int ndim, const int8_t* f, LvlDims d, const std::vector<unsigned long long>& list, double cutoff, cudaStream_t st,
           Staging& stg, std::vector<BisectNode>& T) {
    launched = 0;
    if (!takes(ndim, d, list.size())) return false;
    const int dims[3] = {d.is, d.js, ndim == 3 ? d.ks : 1};
    const long long cells = (long long)dims[0] * dims[1] * dims[2];
    const size_t np = ndim == 2 ? std::max<size_t>(list.size(), 1) : (size_t)std::min(cells, MAX_POINTS);
    tree.ensure(sizeof(BisectHead) + sizeof(BisectNode) * MAX_NODES);
    node_of.ensure(np);
    hist.ensure((size_t)2 * MAX_HIST);
    if (ndim == 2) pts.upload(list, st, stg);
    else pts.ensure(np);
    BisectArgs a{};
    a.head = reinterpret_cast<BisectHead*>(tree.d);
    a.nodes = reinterpret_cast<BisectNode*>(tree.d + sizeof(BisectHead));
    a.max_nodes = max_nodes;
    a.pts = pts.d; a.max_points = (unsigned)np;
    a.node_of = node_of.d; a.hist = hist.d; a.max_hist = MAX_HIST;
    for (int k = 0; k < 3; ++k) a.dims[k] = dims[k];
    a.cutoff = cutoff;
    a.max_wait = max_wait;
    launched = launch_bisect(ndim, a, f, d, (unsigned)list.size(), st);
    struct First { BisectHead head; BisectNode node[BISECT_FIRST]; };
    static_assert(sizeof(First) == sizeof(BisectHead) + sizeof(BisectNode) * BISECT_FIRST, "the tree is contiguous");
    std::vector<First> h(1);
    AMR_CUDA(cudaMemcpyAsync(h.data(), tree.d, sizeof(First), cudaMemcpyDeviceToHost, st));
    AMR_CUDA(cudaStreamSynchronize(st));
    stg.reset();
    if (h[0].head.stop != 0) return false;
    const int n = h[0].head.nodes;
    T.assign(h[0].node, h[0].node + std::min(n, BISECT_FIRST));
    if (n > BISECT_FIRST) {
      T.resize(n);
      AMR_CUDA(cudaMemcpyAsync(T.data() + BISECT_FIRST, a.nodes + BISECT_FIRST, sizeof(BisectNode) * (n - BISECT_FIRST),
                               cudaMemcpyDeviceToHost, st));
      AMR_CUDA(cudaStreamSynchronize(st));
    }
    return true;
  }

  // The leaves in the reference's depth-first order (the part at or above a cut first).
  static std::vector<int> leaves(const std::vector<BisectNode>& T) {
    std::vector<int> out, stack;
    if (!T.empty() && T[0].n > 0) stack.push_back(0);
    while (!stack.empty()) {
      const int id = stack.back();
      stack.pop_back();
      if (T[id].child < 0) { out.push_back(id); continue; }
      stack.push_back(T[id].child + 1);
      stack.push_back(T[id].child);
    }
    return out;
  }
};

}  // namespace amrb
