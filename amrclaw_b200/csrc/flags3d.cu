// Device kernels of the 3D level flag arrays (flglvl.f, domprep.f, domshrink.f,
// domup.f, spest.f, flag2refine.f, bufnst.f, projec.f, shiftset.f, colate.f).
// Every kernel is a grid-stride loop over int8 cells; the arrays of a 128^3 level
// are about 2 MB, so each pass is a few microseconds of HBM time.
#include "flags3d.cuh"
#include <algorithm>

namespace amrb {

namespace {

constexpr int NGF = 2;  // num_ghost of the patch storage

// std::max / Fortran max argument order (the CPU restatement's)
__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }

int blocks_for(long long n, int block) {
  return (int)std::max<long long>(1, std::min<long long>((n + block - 1) / block, 148LL * 32));
}

#define GRID_STRIDE(t, n) for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < (n); t += (long long)gridDim.x * blockDim.x)

__global__ void boxes_kernel(int8_t* a, LvlDims d, const LvlBox* boxes, int nbox, int mode) {
  const int b = blockIdx.y;
  if (b >= nbox) return;
  const LvlBox B = boxes[b];
  const int ni = B.i1 - B.i0 + 1, nj = B.j1 - B.j0 + 1, nk = B.k1 - B.k0 + 1;
  if (ni <= 0 || nj <= 0 || nk <= 0) return;
  const long long n = (long long)ni * nj * nk;
  GRID_STRIDE(t, n) {
    const int i = B.i0 + (int)(t % ni), j = B.j0 + (int)((t / ni) % nj), k = B.k0 + (int)(t / ((long long)ni * nj));
    int8_t& v = a[d.at(i, j, k)];
    if (mode == 0) v = 1;
    else if (v == 0) v = 3;
  }
}

// extend_borders: ring cells of the six faces (edges and corners excluded) copy a 1 of the adjacent interior cell
__global__ void extend_kernel(int8_t* a, LvlDims d) {
  const long long fx = (long long)d.js * d.ks, fy = (long long)d.is * d.ks, fz = (long long)d.is * d.js;
  GRID_STRIDE(t0, 2 * (fx + fy + fz)) {
    long long t = t0;
    int i, j, k, si, sj, sk;
    if (t < 2 * fx) {
      const bool hi = t >= fx; if (hi) t -= fx;
      j = 1 + (int)(t % d.js); k = 1 + (int)(t / d.js);
      i = hi ? d.is + 1 : 0; si = hi ? d.is : 1; sj = j; sk = k;
    } else if ((t -= 2 * fx) < 2 * fy) {
      const bool hi = t >= fy; if (hi) t -= fy;
      i = 1 + (int)(t % d.is); k = 1 + (int)(t / d.is);
      j = hi ? d.js + 1 : 0; sj = hi ? d.js : 1; si = i; sk = k;
    } else {
      t -= 2 * fy;
      const bool hi = t >= fz; if (hi) t -= fz;
      i = 1 + (int)(t % d.is); j = 1 + (int)(t / d.is);
      k = hi ? d.ks + 1 : 0; sk = hi ? d.ks : 1; si = i; sj = j;
    }
    if (a[d.at(si, sj, sk)] == 1) a[d.at(i, j, k)] = 1;
  }
}

// fill_edges_corners, edges: a ring edge cell becomes 1 where both face neighbours are 1
__global__ void edges_kernel(int8_t* a, LvlDims d) {
  const int is = d.is, js = d.js, ks = d.ks;
  GRID_STRIDE(t0, 4LL * (ks + is + js)) {
    long long t = t0;
    auto F = [&](int i, int j, int k) { return (int)a[d.at(i, j, k)]; };
    if (t < 4LL * ks) {
      const int k = 1 + (int)(t / 4), e = (int)(t % 4);
      if (e == 0 && F(0, 1, k) + F(1, 0, k) == 2) a[d.at(0, 0, k)] = 1;
      if (e == 1 && F(0, js, k) + F(1, js + 1, k) == 2) a[d.at(0, js + 1, k)] = 1;
      if (e == 2 && F(is, 0, k) + F(is + 1, 1, k) == 2) a[d.at(is + 1, 0, k)] = 1;
      if (e == 3 && F(is, js + 1, k) + F(is + 1, js, k) == 2) a[d.at(is + 1, js + 1, k)] = 1;
    } else if ((t -= 4LL * ks) < 4LL * is) {
      const int i = 1 + (int)(t / 4), e = (int)(t % 4);
      if (e == 0 && F(i, 0, 1) + F(i, 1, 0) == 2) a[d.at(i, 0, 0)] = 1;
      if (e == 1 && F(i, js, 0) + F(i, js + 1, 1) == 2) a[d.at(i, js + 1, 0)] = 1;
      if (e == 2 && F(i, 0, ks) + F(i, 1, ks + 1) == 2) a[d.at(i, 0, ks + 1)] = 1;
      if (e == 3 && F(i, js + 1, ks) + F(i, js, ks + 1) == 2) a[d.at(i, js + 1, ks + 1)] = 1;
    } else {
      t -= 4LL * is;
      const int j = 1 + (int)(t / 4), e = (int)(t % 4);
      if (e == 0 && F(0, j, 1) + F(1, j, 0) == 2) a[d.at(0, j, 0)] = 1;
      if (e == 1 && F(is, j, 0) + F(is + 1, j, 1) == 2) a[d.at(is + 1, j, 0)] = 1;
      if (e == 2 && F(0, j, ks) + F(1, j, ks + 1) == 2) a[d.at(0, j, ks + 1)] = 1;
      if (e == 3 && F(is + 1, j, ks) + F(is, j, ks + 1) == 2) a[d.at(is + 1, j, ks + 1)] = 1;
    }
  }
}

// fill_edges_corners, corners: one thread, after the edges
__global__ void corners_kernel(int8_t* a, LvlDims d) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  const int is = d.is, js = d.js, ks = d.ks;
  auto F = [&](int i, int j, int k) { return (int)a[d.at(i, j, k)]; };
  if (F(0, 0, 1) + F(0, 1, 0) + F(1, 0, 0) == 3) a[d.at(0, 0, 0)] = 1;
  if (F(is + 1, 0, 1) + F(is + 1, 1, 0) + F(is, 0, 0) == 3) a[d.at(is + 1, 0, 0)] = 1;
  if (F(0, js + 1, 1) + F(0, js, 0) + F(1, js + 1, 0) == 3) a[d.at(0, js + 1, 0)] = 1;
  if (F(is + 1, js + 1, 1) + F(is + 1, js, 0) + F(is, js + 1, 0) == 3) a[d.at(is + 1, js + 1, 0)] = 1;
  if (F(0, 0, ks) + F(0, 1, ks + 1) + F(1, 0, ks + 1) == 3) a[d.at(0, 0, ks + 1)] = 1;
  if (F(is + 1, 0, ks) + F(is + 1, 1, ks + 1) + F(is, 0, ks + 1) == 3) a[d.at(is + 1, 0, ks + 1)] = 1;
  if (F(0, js + 1, ks) + F(0, js, ks + 1) + F(1, js + 1, ks + 1) == 3) a[d.at(0, js + 1, ks + 1)] = 1;
  if (F(is + 1, js + 1, ks) + F(is + 1, js, ks + 1) + F(is, js + 1, ks + 1) == 3) a[d.at(is + 1, js + 1, ks + 1)] = 1;
}

__device__ __forceinline__ bool is_ring(const LvlDims& d, int i, int j, int k) {
  return i == 0 || j == 0 || k == 0 || i == d.is + 1 || j == d.js + 1 || k == d.ks + 1;
}

// every cell of `out`: 0 on the ring, interior kept where all 27 cells of `in` are positive
__global__ void shrink_kernel(const int8_t* in, int8_t* out, LvlDims d) {
  GRID_STRIDE(t, d.size()) {
    const int i = (int)(t % (d.is + 2)), j = (int)((t / (d.is + 2)) % (d.js + 2)), k = (int)(t / ((long long)(d.is + 2) * (d.js + 2)));
    int8_t v = 0;
    if (!is_ring(d, i, j, k)) {
      bool ok = true;
      for (int c = -1; c <= 1 && ok; ++c)
        for (int b = -1; b <= 1 && ok; ++b) {
          const int8_t* row = in + d.at(i - 1, j + b, k + c);
          if (row[0] <= 0 || row[1] <= 0 || row[2] <= 0) ok = false;
        }
      v = ok ? in[t] : (int8_t)0;
    }
    out[t] = v;
  }
}

// every cell of `fine`: 0 on the ring, the covering coarse cell's value inside
__global__ void up_kernel(const int8_t* c, LvlDims cd, int8_t* f, LvlDims fd, int rx, int ry, int rz) {
  GRID_STRIDE(t, fd.size()) {
    const int i = (int)(t % (fd.is + 2)), j = (int)((t / (fd.is + 2)) % (fd.js + 2)), k = (int)(t / ((long long)(fd.is + 2) * (fd.js + 2)));
    f[t] = is_ring(fd, i, j, k) ? (int8_t)0 : c[cd.at((i - 1) / rx + 1, (j - 1) / ry + 1, (k - 1) / rz + 1)];
  }
}

__global__ void zero_interior_kernel(int8_t* f, LvlDims d) {
  GRID_STRIDE(t, (long long)d.is * d.js * d.ks) {
    const int i = 1 + (int)(t % d.is), j = 1 + (int)((t / d.is) % d.js), k = 1 + (int)(t / ((long long)d.is * d.js));
    f[d.at(i, j, k)] = 0;
  }
}

__global__ void zero_ring_kernel(int8_t* f, LvlDims d) {
  GRID_STRIDE(t, d.size()) {
    const int i = (int)(t % (d.is + 2)), j = (int)((t / (d.is + 2)) % (d.js + 2)), k = (int)(t / ((long long)(d.is + 2) * (d.js + 2)));
    if (is_ring(d, i, j, k)) f[t] = 0;
  }
}

// Binary search of the patch that holds level cell t.
__device__ __forceinline__ int patch_of(const long long* pre, int np, long long t) {
  int lo = 0, hi = np - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// flag2refine.f pattern of the 3D Euler example: undivided pressure difference (or of every
// component) against tolsp; BADPT (2) / GOODPT (0) into the zeroed level array (setflags.f)
template <class T>
__global__ void flag_cells_kernel(const T* pool, const PatchDev* patches, const int* plist, const long long* cell0, int np,
                                  long long ncells, int flag_pressure, double gamma1, double tolsp, int nvar, int8_t* f, LvlDims d) {
  GRID_STRIDE(t, ncells) {
    const int pi = patch_of(cell0, np, t);
    const PatchDev& P = patches[plist[pi]];
    const int mx = P.ihi - P.ilo + 1, my = P.jhi - P.jlo + 1;
    const long long loc = t - cell0[pi];
    const int i = (int)(loc % mx) + 1, j = (int)((loc / mx) % my) + 1, k = (int)(loc / ((long long)mx * my)) + 1;
    const long long plane = (long long)P.mitot * P.mjtot * P.mktot;
    const T* q = pool + P.q[P.cur];
    auto Q = [&](int m, int ii, int jj, int kk) {
      return q[(m - 1) * plane + ((long long)(kk - 1 + NGF) * P.mjtot + (jj - 1 + NGF)) * P.mitot + (ii - 1 + NGF)];
    };
    double dq = 0.0;
    if (flag_pressure) {
      auto pres = [&](int a, int b, int c) {
        const double rho = Q(1, a, b, c), mu = Q(2, a, b, c), mv = Q(3, a, b, c), mw = Q(4, a, b, c);
        return gamma1 * (Q(5, a, b, c) - 0.5 * (mu * mu + mv * mv + mw * mw) / rho);
      };
      const double dpi = fabs(pres(i + 1, j, k) - pres(i - 1, j, k));
      const double dpj = fabs(pres(i, j + 1, k) - pres(i, j - 1, k));
      const double dpk = fabs(pres(i, j, k + 1) - pres(i, j, k - 1));
      dq = dmax(dmax(dmax(dq, dpi), dpj), dpk);
    } else {
      for (int m = 1; m <= nvar; ++m) {
        const double dqi = fabs(Q(m, i + 1, j, k) - Q(m, i - 1, j, k));
        const double dqj = fabs(Q(m, i, j + 1, k) - Q(m, i, j - 1, k));
        const double dqk = fabs(Q(m, i, j, k + 1) - Q(m, i, j, k - 1));
        dq = dmax(dmax(dmax(dq, dqi), dqj), dqk);
      }
    }
    f[d.at(P.ilo + i, P.jlo + j, P.klo + k)] = (dq > tolsp) ? (int8_t)2 : (int8_t)0;
  }
}

// shiftset.f: every positive flag, in (k, j, i) order, stamps its value on the box of
// half-width b around it; the value a cell ends with is that of the lexicographically
// last (k, j, i) source within b in every direction. Three separable passes:
// t1(i, j, k) = last source along i (rows j, k interior, i over the whole array width)
__global__ void shift_i_kernel(const int8_t* f, int8_t* t1, LvlDims d, int b) {
  GRID_STRIDE(t, (long long)(d.is + 2) * d.js * d.ks) {
    const int i = (int)(t % (d.is + 2)), j = 1 + (int)((t / (d.is + 2)) % d.js), k = 1 + (int)(t / ((long long)(d.is + 2) * d.js));
    int8_t v = 0;
    for (int s = min(i + b, d.is); s >= max(i - b, 1); --s) {
      const int8_t x = f[d.at(s, j, k)];
      if (x > 0) { v = x; break; }
    }
    t1[d.at(i, j, k)] = v;
  }
}
// t2(i, j, k) = t1 of the last row j' within b that holds a source (k interior)
__global__ void shift_j_kernel(const int8_t* t1, int8_t* t2, LvlDims d, int b) {
  GRID_STRIDE(t, (long long)(d.is + 2) * (d.js + 2) * d.ks) {
    const int i = (int)(t % (d.is + 2)), jj = (int)((t / (d.is + 2)) % (d.js + 2)), k = 1 + (int)(t / ((long long)(d.is + 2) * (d.js + 2)));
    int8_t v = 0;
    for (int j = min(jj + b, d.js); j >= max(jj - b, 1); --j) {
      const int8_t x = t1[d.at(i, j, k)];
      if (x > 0) { v = x; break; }
    }
    t2[d.at(i, jj, k)] = v;
  }
}
// f += t2 of the last plane k' within b that holds a source (interior cells only)
__global__ void shift_k_add_kernel(const int8_t* t2, int8_t* f, LvlDims d, int b) {
  GRID_STRIDE(t, (long long)d.is * d.js * d.ks) {
    const int i = 1 + (int)(t % d.is), j = 1 + (int)((t / d.is) % d.js), kk = 1 + (int)(t / ((long long)d.is * d.js));
    int8_t v = 0;
    for (int k = min(kk + b, d.ks); k >= max(kk - b, 1); --k) {
      const int8_t x = t2[d.at(i, j, k)];
      if (x > 0) { v = x; break; }
    }
    int8_t& o = f[d.at(i, j, kk)];
    o = (int8_t)(o + v);
  }
}

__global__ void colate_kernel(int8_t* f, const int8_t* dom, LvlDims d) {
  GRID_STRIDE(t, (long long)d.is * d.js * d.ks) {
    const int i = 1 + (int)(t % d.is), j = 1 + (int)((t / d.is) % d.js), k = 1 + (int)(t / ((long long)d.is * d.js));
    const long long a = d.at(i, j, k);
    f[a] = f[a] < dom[a] ? f[a] : dom[a];
  }
}

// extend_borders with periodic directions, one direction per launch in the order x, y, z
// (a later direction reads ring cells an earlier one wrote): a periodic direction copies
// the far interior layer over its whole ring face (0..n+1 in the other two indices); a
// non-periodic one extends a 1 of the adjacent interior cell (other indices interior only)
__global__ void border_dir_kernel(int8_t* a, LvlDims d, int dir, int periodic) {
  const int e = periodic ? 2 : 0, o = periodic ? 0 : 1;
  const long long na = (dir == 0 ? d.js : d.is) + e, nb = (dir == 2 ? d.js : d.ks) + e;
  GRID_STRIDE(t, 2 * na * nb) {
    const bool hi = t >= na * nb;
    const long long r = hi ? t - na * nb : t;
    const int u = (int)(r % na) + o, v = (int)(r / na) + o;
    const int n = dir == 0 ? d.is : dir == 1 ? d.js : d.ks;
    const int ring = hi ? n + 1 : 0;
    const int src = periodic ? (hi ? 1 : n) : (hi ? n : 1);
    long long at, from;
    if (dir == 0) { at = d.at(ring, u, v); from = d.at(src, u, v); }
    else if (dir == 1) { at = d.at(u, ring, v); from = d.at(u, src, v); }
    else { at = d.at(u, v, ring); from = d.at(u, v, src); }
    if (periodic) a[at] = a[from];
    else if (a[from] == 1) a[at] = 1;
  }
}

// per: bit 0, 1, 2 set for periodic x, y, z; skip: leave the ring of periodic directions as it is
void borders(int8_t* a, LvlDims d, bool edges, cudaStream_t s, int per = 0, bool skip = false) {
  if (per == 0) {
    const long long n = 2LL * ((long long)d.js * d.ks + (long long)d.is * d.ks + (long long)d.is * d.js);
    extend_kernel<<<blocks_for(n, 256), 256, 0, s>>>(a, d);
  } else {
    for (int dir = 0; dir < 3; ++dir) {
      const bool p = (per >> dir) & 1;
      if (p && skip) continue;
      const long long na = (dir == 0 ? d.js : d.is) + (p ? 2 : 0), nb = (dir == 2 ? d.js : d.ks) + (p ? 2 : 0);
      border_dir_kernel<<<blocks_for(2 * na * nb, 256), 256, 0, s>>>(a, d, dir, p ? 1 : 0);
    }
  }
  if (edges) {
    edges_kernel<<<blocks_for(4LL * (d.is + d.js + d.ks), 256), 256, 0, s>>>(a, d);
    corners_kernel<<<1, 32, 0, s>>>(a, d);
  }
}

}  // namespace

void launch_domprep(int8_t* a, LvlDims d, const LvlBox* boxes, int nbox, cudaStream_t s, int per) {
  AMR_CUDA(cudaMemsetAsync(a, 0, d.size(), s));
  for (int b0 = 0; b0 < nbox; b0 += 65535)
    boxes_kernel<<<dim3(8, std::min(65535, nbox - b0)), 256, 0, s>>>(a, d, boxes + b0, std::min(65535, nbox - b0), 0);
  borders(a, d, true, s, per);
  AMR_CUDA(cudaGetLastError());
}

void launch_domshrink(const int8_t* in, int8_t* out, LvlDims d, cudaStream_t s, int per) {
  shrink_kernel<<<blocks_for(d.size(), 256), 256, 0, s>>>(in, out, d);
  borders(out, d, false, s, per, true);
  AMR_CUDA(cudaGetLastError());
}

void launch_domup(const int8_t* crse, LvlDims cd, int8_t* fine, LvlDims fd, int rx, int ry, int rz, cudaStream_t s, int per) {
  up_kernel<<<blocks_for(fd.size(), 256), 256, 0, s>>>(crse, cd, fine, fd, rx, ry, rz);
  borders(fine, fd, true, s, per);
  AMR_CUDA(cudaGetLastError());
}

void launch_domcopy_borders(int8_t* a, LvlDims d, cudaStream_t s, int per) {
  borders(a, d, false, s, per);
  AMR_CUDA(cudaGetLastError());
}

void launch_zero_interior(int8_t* f, LvlDims d, cudaStream_t s) {
  zero_interior_kernel<<<blocks_for((long long)d.is * d.js * d.ks, 256), 256, 0, s>>>(f, d);
  AMR_CUDA(cudaGetLastError());
}

void launch_flag_cells3(const void* pool, const PatchDev* patches, const int* plist, const long long* cell0, int np,
                        long long ncells, int flag_pressure, double gamma1, double tolsp, int nvar, int8_t* f, LvlDims d,
                        cudaStream_t s, bool f32) {
  if (ncells <= 0) return;
  if (f32)
    flag_cells_kernel<<<blocks_for(ncells, 256), 256, 0, s>>>(static_cast<const float*>(pool), patches, plist, cell0, np, ncells,
                                                              flag_pressure, gamma1, tolsp, nvar, f, d);
  else
    flag_cells_kernel<<<blocks_for(ncells, 256), 256, 0, s>>>(static_cast<const double*>(pool), patches, plist, cell0, np, ncells,
                                                              flag_pressure, gamma1, tolsp, nvar, f, d);
  AMR_CUDA(cudaGetLastError());
}

void launch_bufnst3(int8_t* f, LvlDims d, const LvlBox* proj, int nproj, int ibuff, int8_t* t1, int8_t* t2, cudaStream_t s) {
  for (int b0 = 0; b0 < nproj; b0 += 65535)
    boxes_kernel<<<dim3(8, std::min(65535, nproj - b0)), 256, 0, s>>>(f, d, proj + b0, std::min(65535, nproj - b0), 1);
  zero_ring_kernel<<<blocks_for(d.size(), 256), 256, 0, s>>>(f, d);
  shift_i_kernel<<<blocks_for((long long)(d.is + 2) * d.js * d.ks, 256), 256, 0, s>>>(f, t1, d, ibuff);
  shift_j_kernel<<<blocks_for((long long)(d.is + 2) * (d.js + 2) * d.ks, 256), 256, 0, s>>>(t1, t2, d, ibuff);
  shift_k_add_kernel<<<blocks_for((long long)d.is * d.js * d.ks, 256), 256, 0, s>>>(t2, f, d, ibuff);
  AMR_CUDA(cudaGetLastError());
}

void launch_colate3(int8_t* f, const int8_t* dom, LvlDims d, cudaStream_t s) {
  colate_kernel<<<blocks_for((long long)d.is * d.js * d.ks, 256), 256, 0, s>>>(f, dom, d);
  AMR_CUDA(cudaGetLastError());
}

// ======================================================================= signatures (signs.f)
namespace {
// The row / column / plane counts of the flagged cells (f != 0) of each box: blockIdx.y is
// the box, each warp takes i-rows (fixed j, k) of it in turn, 32 cells of a row at a time
// (lane = i, coalesced reads). The i-counts go to shared memory one lane per bin; the j-
// and k-counts of a chunk are summed across the warp first and added once. Counts are
// integers, so the order of the adds does not matter. SH: a box's counts fit in shared memory
// (12288 of them); longer boxes are counted in place.
template <bool SH>
__global__ void signatures3_kernel(const int8_t* f, LvlDims d, const SigBox* boxes, const int* off, int* hist) {
  extern __shared__ int block_counts[];
  const SigBox B = boxes[blockIdx.y];
  const int ni = B.hi[0] - B.lo[0] + 1, nj = B.hi[1] - B.lo[1] + 1, nk = B.hi[2] - B.lo[2] + 1;
  const int nh = ni + nj + nk;
  int* const h = hist + off[blockIdx.y];
  int* const sh = SH ? block_counts : h;
  if (SH) {
    for (int t = threadIdx.x; t < nh; t += blockDim.x) sh[t] = 0;
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const long long rows = (long long)nj * nk;
  for (long long r = (long long)blockIdx.x * nwarps + warp; r < rows; r += (long long)gridDim.x * nwarps) {
    const int j = (int)(r % nj), k = (int)(r / nj);
    const int8_t* row = f + d.at(B.lo[0], B.lo[1] + j, B.lo[2] + k);
    int cnt = 0;
    for (int i0 = 0; i0 < ni; i0 += 32) {
      const int i = i0 + lane;
      const int flag = (i < ni && row[i] != 0) ? 1 : 0;
      if (flag) atomicAdd(&sh[i], 1);
      cnt += __popc(__ballot_sync(0xffffffffu, flag));
    }
    if (lane == 0 && cnt) {
      atomicAdd(&sh[ni + j], cnt);
      atomicAdd(&sh[ni + nj + k], cnt);
    }
  }
  if (!SH) return;
  __syncthreads();
  for (int t = threadIdx.x; t < nh; t += blockDim.x)
    if (sh[t]) atomicAdd(&h[t], sh[t]);
}
__global__ void scatter_points_kernel(const int* pts, int n, int8_t* f, LvlDims d) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    f[d.at(pts[2 * t] + 1, pts[2 * t + 1] + 1, 1)] = 1;
}
}  // namespace

void launch_scatter_points2(const int* pts, int n, int8_t* f, LvlDims d, cudaStream_t s) {
  AMR_CUDA(cudaMemsetAsync(f, 0, (size_t)d.size(), s));
  if (n > 0) scatter_points_kernel<<<blocks_for(n, 256), 256, 0, s>>>(pts, n, f, d);
  AMR_CUDA(cudaGetLastError());
}

void launch_signatures3(const int8_t* f, LvlDims d, const SigBox* boxes, int nbox, const int* off, int total, int maxlen,
                        long long maxrows, int* hist, cudaStream_t s) {
  if (nbox <= 0) return;
  AMR_CUDA(cudaMemsetAsync(hist, 0, sizeof(int) * (size_t)total, s));
  // blocks of 8 warps, a warp per i-row: enough blocks per box for its rows
  const int slabs = (int)std::max<long long>(1, std::min<long long>(64, (maxrows + 7) / 8));
  for (int base = 0; base < nbox; base += 65535) {
    const int cnt = std::min(65535, nbox - base);
    if (maxlen <= 12288) signatures3_kernel<true><<<dim3(slabs, cnt), 256, sizeof(int) * (size_t)maxlen, s>>>(f, d, boxes + base, off + base, hist);
    else signatures3_kernel<false><<<dim3(slabs, cnt), 256, 0, s>>>(f, d, boxes + base, off + base, hist);
  }
  AMR_CUDA(cudaGetLastError());
}

// ======================================================================= bisection
namespace {
constexpr int BIS_THREADS = 1024;
constexpr int BIS_BLOCKS = 32;
constexpr int BIS_Q = 4;     // points of a thread in flight
constexpr int BIS_SH = 320;  // counts of a node that its warp keeps in shared memory

__global__ void bisect_head_kernel(BisectHead* h, unsigned npts) {
  *h = BisectHead{};
  h->points = npts;
}
// the flagged cells of the interior, in any order (only their counts are used)
__global__ void __launch_bounds__(256) list_points_kernel(const int8_t* f, LvlDims d, unsigned long long* pts, unsigned max_points, BisectHead* h) {
  const long long row = (d.is + 31) / 32 * 32, n = row * d.js * d.ks;  // whole warps per i-row
  const int lane = threadIdx.x & 31;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t % row) + 1;
    const long long r = t / row;
    const int j = (int)(r % d.js) + 1, k = (int)(r / d.js) + 1;
    const bool on = i <= d.is && f[d.at(i, j, k)] != 0;
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (m == 0) continue;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&h->points, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    const unsigned at = base + __popc(m & ((1u << lane) - 1u));
    if (on && at < max_points) pts[at] = bisect_point(i, j, k);
  }
}

// All blocks of the launch (co-resident: it is a cooperative one). False when a block gave up
// waiting (max_wait); every block then leaves.
__device__ __forceinline__ bool bisect_barrier(BisectHead* h, unsigned& turn, long long max_wait) {
  if (gridDim.x == 1) { __syncthreads(); return true; }
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ++turn;
    __threadfence();
    atomicAdd(&h->arrived, 1u);
    const long long t0 = clock64();
    ok = 1;
    while (*(volatile unsigned*)&h->arrived < turn * gridDim.x) {
      if (clock64() - t0 > max_wait) { ok = 0; break; }
    }
    if (!ok) atomicExch(&h->stop, 2);
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// A warp's reduction of a key to its largest, on every lane.
__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v) {
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}

// moment.f and findcut.f for one node by one warp, from its counts h (per i, then j, then k).
// Returns whether it is cut. SH: the counts are in shared memory.
template <int ND, bool SH>
__device__ __forceinline__ bool bisect_node(BisectNode& N, const int* h, double cutoff) {
  const int lane = threadIdx.x & 31;
  auto at_ = [](const int* q) { return SH ? *q : __ldcg(q); };
  const int* hd[3];
  int n = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    hd[d] = h;
    if (d >= ND) { N.clo[d] = N.lo[d]; N.chi[d] = N.hi[d]; continue; }
    const int len = N.hi[d] - N.lo[d] + 1;
    int first = 0x7fffffff, last = -1, sum = 0;
#pragma unroll 4
    for (int t = lane; t < len; t += 32) {
      const int v = at_(h + t);
      if (v) { first = min(first, t); last = max(last, t); sum += v; }
    }
    first = __reduce_min_sync(0xffffffffu, first);
    last = __reduce_max_sync(0xffffffffu, last);
    if (d == 0) n = __reduce_add_sync(0xffffffffu, sum);
    N.clo[d] = last < 0 ? N.lo[d] : N.lo[d] + first;
    N.chi[d] = last < 0 ? N.hi[d] : N.lo[d] + last;
    h += len;
  }
  N.n = n;
  if (n == 0) return false;
  long long vol = 1;
#pragma unroll
  for (int d = 0; d < ND; ++d) vol *= N.chi[d] - N.clo[d] + 1;
  if ((double)n / (double)vol >= cutoff) return false;
  // a hole: the first zero of the first direction that has one
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    int z = 0x7fffffff;
#pragma unroll 4
    for (int t = N.clo[d] + lane; t <= N.chi[d]; t += 32)
      if (at_(hd[d] + (t - N.lo[d])) == 0) z = min(z, t);
    z = __reduce_min_sync(0xffffffffu, z);
    if (z != 0x7fffffff) { N.dir = d + 1; N.cut = z; return true; }
  }
  // the largest sign change of the Laplacian of each direction's counts, the one nearest to
  // the middle among equals, the first among those
  int best[3] = {0, 0, 0}, at[3] = {0, 0, 0}, mid[3] = {0, 0, 0};
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    const int lo = N.clo[d], hi = N.chi[d];
    mid[d] = (lo + hi) / 2;
    unsigned long long key = 0;
#pragma unroll 2
    for (int t = lo + 2 + lane; t <= hi - 1; t += 32) {
      const int* c = hd[d] + (t - N.lo[d]);
      const int c0 = at_(c - 2), c1 = at_(c - 1), c2 = at_(c), c3 = at_(c + 1);
      const int a = c2 - 2 * c1 + c0, b = c3 - 2 * c2 + c1;
      if ((a < 0 && b > 0) || (a > 0 && b < 0)) {  // (a product of two counts can pass 32 bits)
        const unsigned long long v = ((unsigned long long)abs(a - b) << 42) | ((unsigned long long)(0x1fffff - abs(t - mid[d])) << 21) |
                                     (unsigned long long)(0x1fffff - t);
        key = v > key ? v : key;
      }
    }
    key = warp_max64(key);
    if (key) { best[d] = (int)(key >> 42); at[d] = 0x1fffff - (int)(key & 0x1fffff); }
  }
  int index, side;
  if (ND == 2) {
    // src/2d/findcut.f: the larger change; of equal ones the one nearer to its middle
    const bool x = best[0] > best[1] || (best[0] == best[1] && abs(at[0] - mid[0]) < abs(at[1] - mid[1]));
    side = x ? 1 : 2;
    index = x ? at[0] : at[1];
    if ((x ? best[0] : best[1]) < 2) index = 0;
  } else {
    // src/3d/findcut.f: the directions ordered by their change, the leading equal ones again
    // by the distance from their middles
    int o[3] = {0, 1, 2};
    for (int a = 0; a < 2; ++a)
      for (int b = a + 1; b < 3; ++b)
        if (best[o[a]] < best[o[b]]) { const int t = o[a]; o[a] = o[b]; o[b] = t; }
    const int same = best[o[0]] > best[o[1]] ? 1 : best[o[1]] > best[o[2]] ? 2 : 3;
    if (same != 1)
      for (int a = 0; a < same - 1; ++a)
        for (int b = a + 1; b < same; ++b)
          if (abs(at[o[a]] - mid[o[a]]) > abs(at[o[b]] - mid[o[b]])) { const int t = o[a]; o[a] = o[b]; o[b] = t; }
    index = at[o[0]];
    side = o[0] + 1;
    if (best[o[0]] < 2) index = 0;
  }
  N.dir = side;
  N.cut = index;
  return index != 0;
}

// One launch for the whole bisection. A wave is the nodes [w0, w1) of one depth: every point
// moves to its part of the node that was cut above it and counts itself there, then a warp
// per node takes the decisions that the host took from the counts of a wave, and makes the
// two parts. Going back to the host between waves cost 24-33 us a wave (an upload, a clear, a
// launch, a copy and a wait): 205 us a bisection of a 100^2 quadrants run (140 bisections,
// about 6 waves each), where this launch takes 65 us and is bound by the latency of its waves'
// dependent L2 reads.
template <int ND>
__global__ void __launch_bounds__(BIS_THREADS) bisect_kernel(BisectArgs A) {
  __shared__ int counts[BIS_THREADS / 32 * BIS_SH];
  BisectHead* H = A.head;
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, nthr = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  const unsigned warp = tid >> 5, nwarps = nthr >> 5;
  unsigned turn = 0;
  const unsigned np = H->points;
  if (np > A.max_points) {
    if (tid == 0) H->stop = 1;
    return;
  }
  const int root_len = A.dims[0] + A.dims[1] + (ND == 3 ? A.dims[2] : 0);
  for (unsigned t = tid; t < (unsigned)root_len; t += nthr) A.hist[t] = 0;
  for (unsigned q = tid; q < np; q += nthr) A.node_of[q] = 0;
  if (tid == 0) {
    BisectNode R{};
    for (int d = 0; d < 3; ++d) { R.lo[d] = 1; R.hi[d] = d < ND ? A.dims[d] : 1; }
    R.child = -1;
    A.nodes[0] = R;
    H->nodes = 1;
  }
  if (!bisect_barrier(H, turn, A.max_wait)) return;
  int w0 = 0, w1 = 1, cur = 0;
  while (true) {
    if (tid == 0) H->hlen[cur ^ 1] = 0;
    int* hist = A.hist + (long long)cur * A.max_hist;
    // BIS_Q points of a thread at a time: their loads are in flight together
    for (unsigned q0 = tid; q0 < np; q0 += BIS_Q * nthr) {
      unsigned long long P[BIS_Q];
      int b[BIS_Q], ch[BIS_Q], dir[BIS_Q], cut[BIS_Q], at[BIS_Q], lo[BIS_Q][ND], hi[BIS_Q][ND];
#pragma unroll
      for (int u = 0; u < BIS_Q; ++u) {
        const unsigned q = q0 + u * nthr;
        b[u] = q < np ? A.node_of[q] : -1;
        P[u] = q < np ? A.pts[q] : 0;
      }
#pragma unroll
      for (int u = 0; u < BIS_Q; ++u) {
        ch[u] = -2;  // stays where it is
        if (b[u] < 0 || b[u] >= w0) continue;
        const BisectNode* N = A.nodes + b[u];
        ch[u] = __ldcg(&N->child); dir[u] = __ldcg(&N->dir); cut[u] = __ldcg(&N->cut);
      }
#pragma unroll
      for (int u = 0; u < BIS_Q; ++u) {
        if (ch[u] == -1) b[u] = -1;  // in a leaf
        if (ch[u] >= 0) {
          b[u] = (int)((P[u] >> (21 * (dir[u] - 1))) & 0x1fffff) >= cut[u] ? ch[u] : ch[u] + 1;
          A.node_of[q0 + u * nthr] = b[u];
        }
      }
#pragma unroll
      for (int u = 0; u < BIS_Q; ++u) {
        if (b[u] < 0) continue;
        const BisectNode* N = A.nodes + b[u];
        at[u] = __ldcg(&N->hoff);
#pragma unroll
        for (int d = 0; d < ND; ++d) { lo[u][d] = __ldcg(&N->lo[d]); hi[u][d] = __ldcg(&N->hi[d]); }
      }
#pragma unroll
      for (int u = 0; u < BIS_Q; ++u) {
        if (b[u] < 0) continue;
        int o = at[u];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          atomicAdd(hist + o + ((int)((P[u] >> (21 * d)) & 0x1fffff) - lo[u][d]), 1);
          o += hi[u][d] - lo[u][d] + 1;
        }
      }
    }
    if (!bisect_barrier(H, turn, A.max_wait)) return;
    int* next = A.hist + (long long)(cur ^ 1) * A.max_hist;
    for (int b = w0 + (int)warp; b < w1; b += (int)nwarps) {
      BisectNode N;
#pragma unroll
      for (int d = 0; d < 3; ++d) { N.lo[d] = __ldcg(&A.nodes[b].lo[d]); N.hi[d] = __ldcg(&A.nodes[b].hi[d]); }
      N.hoff = __ldcg(&A.nodes[b].hoff);
      N.child = -1; N.dir = 0; N.cut = 0; N.pad = 0;
      int len_all = 0;
#pragma unroll
      for (int d = 0; d < ND; ++d) len_all += N.hi[d] - N.lo[d] + 1;
      bool cutit;
      if (len_all <= BIS_SH) {
        int* own = counts + (threadIdx.x >> 5) * BIS_SH;
        __syncwarp();
#pragma unroll 4
        for (int t = lane; t < len_all; t += 32) own[t] = __ldcg(hist + N.hoff + t);
        __syncwarp();
        cutit = bisect_node<ND, true>(N, own, A.cutoff);
      } else {
        cutit = bisect_node<ND, false>(N, hist + N.hoff, A.cutoff);
      }
      int id = -1, off = 0, len[2] = {0, 0};
      if (cutit) {
        int all = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) all += N.chi[d] - N.clo[d] + 1;
        len[0] = all - (N.cut - N.clo[N.dir - 1]);
        len[1] = all - (N.chi[N.dir - 1] - N.cut + 1);
        if (lane == 0) {
          id = atomicAdd(&H->nodes, 2);
          off = atomicAdd(&H->hlen[cur ^ 1], len[0] + len[1]);
        }
        id = __shfl_sync(0xffffffffu, id, 0);
        off = __shfl_sync(0xffffffffu, off, 0);
        if (id + 2 > A.max_nodes || off + len[0] + len[1] > A.max_hist) {
          if (lane == 0) atomicExch(&H->stop, 1);
          id = -1;
        }
      }
      if (id >= 0) {
        for (int t = lane; t < len[0] + len[1]; t += 32) next[off + t] = 0;
        if (lane == 0) {
          N.child = id;
          BisectNode U{};
#pragma unroll
          for (int d = 0; d < 3; ++d) { U.lo[d] = N.clo[d]; U.hi[d] = N.chi[d]; }
          U.child = -1;
          BisectNode L = U;
          U.lo[N.dir - 1] = N.cut; U.hoff = off;
          L.hi[N.dir - 1] = N.cut - 1; L.hoff = off + len[0];
          A.nodes[id] = U;
          A.nodes[id + 1] = L;
        }
      }
      if (lane == 0) A.nodes[b] = N;
    }
    if (!bisect_barrier(H, turn, A.max_wait)) return;
    if (*(volatile int*)&H->stop) return;
    w0 = w1;
    w1 = *(volatile int*)&H->nodes;
    if (w0 == w1) return;
    cur ^= 1;
  }
}
}  // namespace

int launch_bisect(int ndim, const BisectArgs& a, const int8_t* f, LvlDims d, unsigned npts, cudaStream_t s) {
  bisect_head_kernel<<<1, 1, 0, s>>>(a.head, ndim == 3 ? 0u : npts);
  if (ndim == 3) {
    const long long cells = (long long)((d.is + 31) / 32 * 32) * d.js * d.ks;
    list_points_kernel<<<blocks_for(cells, 256), 256, 0, s>>>(f, d, a.pts, a.max_points, a.head);
  }
  AMR_CUDA(cudaGetLastError());
  // a list of up to a few thousand points is one block's work, with no grid barrier
  const unsigned blocks = ndim == 3 ? BIS_BLOCKS : std::max(1u, std::min((unsigned)BIS_BLOCKS, npts / 4096));
  if (blocks == 1) {
    bisect_kernel<2><<<1, BIS_THREADS, 0, s>>>(a);
    AMR_CUDA(cudaGetLastError());
    return 2;
  }
  void* args[1] = {const_cast<BisectArgs*>(&a)};
  AMR_CUDA(cudaLaunchCooperativeKernel(ndim == 3 ? (const void*)bisect_kernel<3> : (const void*)bisect_kernel<2>, dim3(blocks),
                                       dim3(BIS_THREADS), args, 0, s));
  return ndim == 3 ? 3 : 2;
}

// ======================================================================= Richardson estimation
namespace {
template <class T>
__global__ void coarsen3_kernel(T* pool, const Rect3* rects, const int* rect_of, const PatchDev* vp, int nvar) {
  const int k = blockIdx.y;
  const PatchDev P = vp[k];
  const Rect3 R = rects[rect_of[k]];
  const T* src = pool + R.off;
  T* dst = pool + P.q[0];
  const long long sj = R.ni, sk = (long long)R.ni * R.nj, splane = sk * R.nk;
  const long long n = (long long)P.mitot * P.mjtot * P.mktot;
  GRID_STRIDE(t, n * nvar) {
    const int m = (int)(t / n);
    const long long rem = t % n;
    const int i = (int)(rem % P.mitot), j = (int)((rem / P.mitot) % P.mjtot), kk = (int)(rem / ((long long)P.mitot * P.mjtot));
    const T* s0 = src + m * splane + (2 * kk) * sk + (2 * j) * sj + 2 * i;
    const double v = (((((((double)s0[0] + (double)s0[1]) + (double)s0[sj]) + (double)s0[sj + 1]) + (double)s0[sk]) + (double)s0[sk + 1]) +
                      (double)s0[sk + sj]) + (double)s0[sk + sj + 1];
    dst[m * n + rem] = (T)(v / 8.0);
  }
}
template <class T>
__global__ void errf3_kernel(const T* pool, const PatchDev* vp, int np, double order, double tol, int8_t* f, LvlDims d) {
  const int k = blockIdx.y;
  const PatchDev C = vp[k], F = vp[np + k];
  const int nxc = (F.ihi - F.ilo + 1) / 2, nyc = (F.jhi - F.jlo + 1) / 2, nzc = (F.khi - F.klo + 1) / 2;
  const T* fine = pool + F.q[1];
  const T* crse = pool + C.q[1];
  const long long fj = F.mitot, fk = (long long)F.mitot * F.mjtot;
  GRID_STRIDE(t, (long long)nxc * nyc * nzc) {
    const int ic = (int)(t % nxc), jc = (int)((t / nxc) % nyc), kc = (int)(t / ((long long)nxc * nyc));
    const T* f0 = fine + (2 * kc + NGF) * fk + (2 * jc + NGF) * fj + (2 * ic + NGF);
    // errf1.f: term1..term8 in the reference's order
    const double aval = ((((((((double)f0[0] + (double)f0[1]) + (double)f0[fj + 1]) + (double)f0[fj]) + (double)f0[fk]) + (double)f0[fk + 1]) +
                         (double)f0[fk + fj + 1]) + (double)f0[fk + fj]) / 8.0;
    const double c = (double)crse[((long long)(kc + NGF) * C.mjtot + (jc + NGF)) * C.mitot + (ic + NGF)];
    const double est = fabs((aval - c) / order);
    if (est >= tol) {
      const int gi = F.ilo + 2 * ic + 1, gj = F.jlo + 2 * jc + 1, gk = F.klo + 2 * kc + 1;  // array index = global + 1
      for (int dk = 0; dk <= 1; ++dk)
        for (int dj = 0; dj <= 1; ++dj)
          for (int di = 0; di <= 1; ++di) {
            int8_t& a = f[d.at(gi + di, gj + dj, gk + dk)];
            a = (int8_t)(a + 2);
          }
    }
  }
}
}  // namespace

void launch_coarsen3(void* pool, const Rect3* rects, const int* rect_of, const PatchDev* vp, int np, int nvar, cudaStream_t s,
                     bool f32) {
  for (int base = 0; base < np; base += 65535) {
    const int n = std::min(65535, np - base);
    if (f32) coarsen3_kernel<<<dim3(16, n), 256, 0, s>>>(static_cast<float*>(pool), rects, rect_of + base, vp + base, nvar);
    else coarsen3_kernel<<<dim3(16, n), 256, 0, s>>>(static_cast<double*>(pool), rects, rect_of + base, vp + base, nvar);
    AMR_CUDA(cudaGetLastError());
  }
}
void launch_errf3(const void* pool, const PatchDev* vp, int np, double order, double tol, int8_t* f, LvlDims d, cudaStream_t s,
                  bool f32) {
  for (int base = 0; base < np; base += 65535) {
    const int n = std::min(65535, np - base);
    // the partners of vp[base..] are np entries further on, from the shifted pointer too
    if (f32) errf3_kernel<<<dim3(8, n), 256, 0, s>>>(static_cast<const float*>(pool), vp + base, np, order, tol, f, d);
    else errf3_kernel<<<dim3(8, n), 256, 0, s>>>(static_cast<const double*>(pool), vp + base, np, order, tol, f, d);
    AMR_CUDA(cudaGetLastError());
  }
}

}  // namespace amrb
