// Cell-list neighbour list: TorchNeighborList.forward (nblist.py:304-445 with
// image padding, 472-490 without a box) and check_cutoff (nblist.py:620-660).
//
// With a box the reference asserts rc <= half the minimum box height, so each
// pair has at most one periodic image inside rc and the pair SET equals the
// minimum-image set: atoms are binned by wrapped fractional coordinates into
// cells at least rc high, and every candidate in the (deduplicated) 27
// neighbouring cells is tested with the minimum-image distance
// (spatial.py:15-36 convention, floor(f + 0.5)).  Rows are sorted by j so the
// output is deterministic and sorted by (i, j).
#include "admp_common.cuh"
#include "runtime.h"

namespace admp {

struct NbMeta {
  double b[9], bi[9];
  double lo[3], hi[3], cs[3];
  int nc[3];
  int ncells;
  // the single-precision test: box, accept below `lo` (and above `small`), reject above `hi`
  float bt[9];
  float lo32, hi32, small32;
  int ortho;
};

// What the host reads back per frame: geometry status, the device error word
// and the number of pairs.
struct NbResult {
  int status;
  int ecode;
  long long npairs;
};

// Neighbours per atom that the counting search keeps for the filling pass
// (512 B an atom, a quarter of the output at 90 neighbours); an atom with more
// is searched again, and up to kNbRow of them are ordered in registers, longer
// rows inside their own slice of the output.
constexpr int kNbKeep = 128;
constexpr int kNbRow = 256;
// Atoms a single block bins by itself (one launch instead of four).  A list of 1,536 / 2,100 / 3,000 / 6,007 atoms
// takes 60 / 68 / 71 / 100 us by one block and 66 / 66 / 66 / 84 by the four launches.
constexpr int kNbOneBlock = 2048;

// Device state of a build over nf frames of N atoms: per-atom arrays are
// [nf][N], per-cell arrays [nf][mc + 1].  cs32 / cs64 / sorted hold the
// atoms in cell order: wrapped fractional coordinates (with a box) or
// positions relative to the lower corner (without).
struct NbWS {
  NbMeta* meta;
  NbResult* res;
  double4* cs64;
  float4* cs32;
  int* cell;    // cell of an atom, -1 if it is not binned
  int* slot;    // its place within the cell
  int* count;
  int* start;
  int* sorted;
  int* scell;   // cells in cell order
  int* kept;    // [nf][N][kNbKeep] unordered neighbours of the atoms in cell order
  int* rowcnt;
  long long* rowptr;
};

__device__ __forceinline__ NbWS nb_frame(NbWS w, int f, int N, int mc) {
  const size_t a = (size_t)f * N, c = (size_t)f * (mc + 1);
  w.meta += f;
  w.res += f;
  w.cs64 += a;
  w.cs32 += a;
  w.cell += a;
  w.slot += a;
  w.count += c;
  w.start += c;
  w.sorted += a;
  w.scell += a;
  w.kept += a * kNbKeep;
  w.rowcnt += a;
  w.rowptr += (size_t)f * (N + 1);
  return w;
}

// Bounds of the positions (no box) by one block.
template <typename T>
__device__ void nb_bounds(int N, const T* __restrict__ pos, NbMeta* meta) {
  __shared__ double smin[3][32], smax[3][32];
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
  for (int i = threadIdx.x; i < N; i += blockDim.x)
    for (int e = 0; e < 3; ++e) {
      double v = pos[3 * (size_t)i + e];
      mn[e] = fmin(mn[e], v);
      mx[e] = fmax(mx[e], v);
    }
  for (int e = 0; e < 3; ++e)
    for (int o = 16; o > 0; o >>= 1) {
      mn[e] = fmin(mn[e], __shfl_xor_sync(0xffffffffu, mn[e], o));
      mx[e] = fmax(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], o));
    }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0)
    for (int e = 0; e < 3; ++e) {
      smin[e][w] = mn[e];
      smax[e][w] = mx[e];
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int e = 0; e < 3; ++e) {
      double a = 1e300, b = -1e300;
      for (int k = 0; k < nw; ++k) {
        a = fmin(a, smin[e][k]);
        b = fmax(b, smax[e][k]);
      }
      meta->lo[e] = a;
      meta->hi[e] = b;
    }
  }
}

// Geometry, validity and cell grid of one frame (one thread).
template <typename T>
__device__ void nb_setup(int pbc, const T* __restrict__ box, double rc, int maxcells, NbMeta* m, NbResult* r) {
  int status = 0;
  int nc[3];
  if (pbc) {
    load_box(box, m->b);
    double V = inv3(m->b, m->bi);
    const double* a = m->b;
    double h[3];
    for (int d = 0; d < 3; ++d) {
      const double* u = a + ((d + 1) % 3) * 3;
      const double* v = a + ((d + 2) % 3) * 3;
      double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2], cz = u[0] * v[1] - u[1] * v[0];
      h[d] = fabs(V) / sqrt(cx * cx + cy * cy + cz * cz);
    }
    double mh = fmin(h[0], fmin(h[1], h[2])) / 2.0;
    if (!(rc <= mh)) status = ADMP_ERR_CUTOFF_TOO_LARGE;
    if (!isfinite(V) || V == 0.0) status = ADMP_ERR_NONFINITE;
    for (int d = 0; d < 3; ++d) {
      double r = h[d] / rc;
      nc[d] = r >= 1.0 && r < 1e6 ? (int)floor(r) : 1;
    }
  } else {
    for (int d = 0; d < 3; ++d) {
      double ext = m->hi[d] - m->lo[d];
      if (!(ext >= 0.0) || !isfinite(ext)) {  // no finite coordinate on this axis leaves the bounds crossed
        status = ADMP_ERR_NONFINITE;
        ext = 0.0;
      }
      m->cs[d] = rc;
      double r = ext / rc;
      nc[d] = r < 1e6 ? (int)floor(r) + 1 : 1;
    }
  }
  // keep the grid at most `maxcells` cells (cells may grow beyond rc, never shrink)
  while ((long long)nc[0] * nc[1] * nc[2] > maxcells) {
    int d = nc[0] >= nc[1] && nc[0] >= nc[2] ? 0 : (nc[1] >= nc[2] ? 1 : 2);
    nc[d] = (nc[d] + 1) / 2;
  }
  for (int d = 0; d < 3; ++d) {
    m->nc[d] = nc[d];
    if (!pbc) m->cs[d] = fmax(rc, (m->hi[d] - m->lo[d]) / nc[d] * (1.0 + 1e-12) + 1e-300);
  }
  m->ncells = nc[0] * nc[1] * nc[2];
  double bsum = 0.0;
  m->ortho = 1;
  for (int k = 0; k < 9; ++k) {
    const double bk = pbc ? m->b[k] : (k % 4 == 0 ? 1.0 : 0.0);
    m->bt[k] = (float)bk;
    bsum += pbc ? fabs(bk) : (k % 4 == 0 ? m->hi[k / 4] - m->lo[k / 4] : 0.0);
    if (k % 4 && m->bt[k] != 0.f) m->ortho = 0;
  }
  // |r^2_float - r^2| <= 2 r |dr|, |dr| <= (a few ulp of a coordinate) * sum |B|
  const float mg = (float)(1e-3 * rc * rc + 1e-5 * rc * bsum);
  m->lo32 = (float)(rc * rc) - mg;
  m->hi32 = (float)(rc * rc) + mg;
  m->small32 = 1e-3f + mg;
  r->status = status;
  r->npairs = 0;
}

// Cell coordinates of atom i (wrapped fractional, or relative to the lower
// corner for the single-precision test); returns its cell, -1 for an atom
// that is not binned (invalid frame, non-finite position).
template <typename T>
__device__ __forceinline__ int nb_locate(int pbc, int i, const T* __restrict__ pos, const NbMeta* m, int status,
                                         double* v, DevError* err) {
  if (status) return -1;  // invalid box / cutoff: no atom is binned, later passes skip it
  double r[3] = {(double)pos[3 * (size_t)i], (double)pos[3 * (size_t)i + 1], (double)pos[3 * (size_t)i + 2]};
  if (!isfinite(r[0]) || !isfinite(r[1]) || !isfinite(r[2])) {
    report_error(err, ADMP_ERR_NONFINITE, 4, i);
    return -1;
  }
  int c[3];
  if (pbc) {
    for (int e = 0; e < 3; ++e) {
      double f = r[0] * m->bi[0 * 3 + e] + r[1] * m->bi[1 * 3 + e] + r[2] * m->bi[2 * 3 + e];
      f -= floor(f);
      c[e] = min((int)(f * m->nc[e]), m->nc[e] - 1);
      v[e] = f;
    }
  } else {
    for (int e = 0; e < 3; ++e) {
      c[e] = min(max((int)((r[e] - m->lo[e]) / m->cs[e]), 0), m->nc[e] - 1);
      v[e] = r[e];
    }
  }
  return (c[0] * m->nc[1] + c[1]) * m->nc[2] + c[2];
}

__device__ __forceinline__ void nb_place(int pbc, const NbWS& w, int i, int c, int at, const double* v) {
  w.sorted[at] = i;
  w.scell[at] = c;
  w.cs64[at] = make_double4(v[0], v[1], v[2], 0.0);
  const double* lo = w.meta->lo;
  w.cs32[at] = pbc ? make_float4((float)v[0], (float)v[1], (float)v[2], 0.f)
                   : make_float4((float)(v[0] - lo[0]), (float)(v[1] - lo[1]), (float)(v[2] - lo[2]), 0.f);
}

// Exclusive scan of n values by one block of 1024 threads -> out[0..n],
// out[n] = total: tiles of 4096 values, warp shuffles inside a tile.
template <typename TI, typename TO>
__device__ void nb_block_scan(const TI* __restrict__ in, TO* __restrict__ out, int n) {
  __shared__ TO wsum[33];
  __shared__ TO carry_sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  TO carry = 0;
  for (int t0 = 0; t0 < n; t0 += 4 * blockDim.x) {
    const int b = t0 + 4 * threadIdx.x;
    TO v[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = b + k < n ? (TO)in[b + k] : TO(0);
      s += v[k];
    }
    TO inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const TO up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += up;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      const TO x = lane < nw ? wsum[lane] : TO(0);
      TO y = x;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const TO up = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += up;
      }
      wsum[lane] = y - x;
      if (lane == 31) carry_sh = y;
    }
    __syncthreads();
    TO acc = carry + wsum[warp] + inc - s;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (b + k < n) out[b + k] = acc;
      acc += v[k];
    }
    carry += carry_sh;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry;
}

// Geometry of every frame (a block per frame) and, with BIN, the whole cell
// sort of it: bin, scan and placement by the one block.  Three launches cost
// more than 2 atoms a thread, so frames of up to kNbOneBlock atoms take this form.
template <typename T, bool BIN>
__global__ void __launch_bounds__(1024) nb_setup_kernel(int pbc, int N, int mc, const T* __restrict__ pos,
                                                        const T* __restrict__ box, double rc, NbWS w0,
                                                        DevError* err) {
  const int f = blockIdx.x;
  const NbWS w = nb_frame(w0, f, N, mc);
  pos += (size_t)f * N * 3;
  if (!pbc) nb_bounds<T>(N, pos, w.meta);
  if (threadIdx.x == 0) nb_setup<T>(pbc, pbc ? box + (size_t)f * 9 : nullptr, rc, mc, w.meta, w.res);
  __syncthreads();
  const int ncells = w.meta->ncells, status = w.res->status;
  for (int k = threadIdx.x; k < ncells; k += blockDim.x) w.count[k] = 0;
  if (!BIN) return;
  __syncthreads();
  double v[3];
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const int c = nb_locate<T>(pbc, i, pos, w.meta, status, v, err);
    w.cell[i] = c;
    w.rowcnt[i] = 0;
    if (c >= 0) w.slot[i] = atomicAdd(w.count + c, 1);
  }
  __syncthreads();
  nb_block_scan<int, int>(w.count, w.start, ncells);
  __syncthreads();
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const int c = w.cell[i];
    if (c < 0) continue;
    nb_locate<T>(pbc, i, pos, w.meta, status, v, err);
    nb_place(pbc, w, i, c, w.start[c] + w.slot[i], v);
  }
}

// Larger frames: the same three steps as launches over all atoms.
template <typename T>
__global__ void nb_bin_kernel(int pbc, int N, int mc, const T* __restrict__ pos, NbWS w0, DevError* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, f = blockIdx.y;
  if (i >= N) return;
  const NbWS w = nb_frame(w0, f, N, mc);
  double v[3];
  const int c = nb_locate<T>(pbc, i, pos + (size_t)f * N * 3, w.meta, w.res->status, v, err);
  w.cell[i] = c;
  w.rowcnt[i] = 0;
  if (c >= 0) w.slot[i] = atomicAdd(w.count + c, 1);
}

static __global__ void __launch_bounds__(1024) nb_cell_scan_kernel(int N, int mc, NbWS w0) {
  const NbWS w = nb_frame(w0, blockIdx.x, N, mc);
  nb_block_scan<int, int>(w.count, w.start, w.meta->ncells);
}

template <typename T>
__global__ void nb_scatter_kernel(int pbc, int N, int mc, const T* __restrict__ pos, NbWS w0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, f = blockIdx.y;
  if (i >= N) return;
  const NbWS w = nb_frame(w0, f, N, mc);
  const int c = w.cell[i];
  if (c < 0) return;
  double v[3];
  nb_locate<T>(pbc, i, pos + (size_t)f * N * 3, w.meta, 0, v, nullptr);
  nb_place(pbc, w, i, c, w.start[c] + w.slot[i], v);
}

// Row offsets and what the host reads back.
static __global__ void __launch_bounds__(1024) nb_row_scan_kernel(int N, int mc, NbWS w0, const DevError* err) {
  const NbWS w = nb_frame(w0, blockIdx.x, N, mc);
  nb_block_scan<int, long long>(w.rowcnt, w.rowptr, N);
  __syncthreads();
  if (threadIdx.x == 0) {
    w.res->npairs = w.rowptr[N];
    w.res->ecode = err->code;
  }
}

// Search of one warp for the neighbours of the atom at place `at` of the cell
// order: visit(in, j) is called by the whole warp for every 32 candidates, each
// lane with its candidate's place j in the cell order and whether it is one.
//
// The atoms of the up to 27 cells around the atom form a few contiguous runs
// of the cell order (cells adjacent along z follow each other); lane q holds
// neighbour cell q and the runs are walked 32 atoms at a time.  With three or
// more cells on every axis a candidate's image is fixed by its cell's wrap and
// goes into the home coordinate; otherwise it is rounded to.  A candidate is
// tested in single precision with a margin far above the rounding error of
// r^2, and in double only inside the margin around rc^2 and 0.01^2: the double
// test is the list's definition.
template <typename F>
__device__ __forceinline__ void nb_search(int pbc, double rc, const NbWS& w, int at, F&& visit) {
  const int lane = threadIdx.x & 31;
  const NbMeta* __restrict__ m = w.meta;
  const int nc0 = m->nc[0], nc1 = m->nc[1], nc2 = m->nc[2];
  const int ci = w.scell[at];
  const int n0 = pbc ? min(nc0, 3) : 3, n1 = pbc ? min(nc1, 3) : 3, n2 = pbc ? min(nc2, 3) : 3;
  const int nq = n0 * n1 * n2;
  const bool fixed = pbc && nq == 27;
  // lane q: neighbour cell q; code: its image along each axis, two bits each
  int begin = 0, len = 0, code = 0;
  if (lane < nq) {
    const int lq = lane / n2, q2 = lane - lq * n2, q0 = lq / n1, q1 = lq - q0 * n1;
    const int cq = ci / nc2, cx = cq / nc1;
    int c[3] = {cx + q0 - (n0 == 3), cq - cx * nc1 + q1 - (n1 == 3), ci - cq * nc2 + q2 - (n2 == 3)};
    const int nc[3] = {nc0, nc1, nc2};
    bool in = true;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      if (pbc) {
        const int s = c[e] < 0 ? -1 : (c[e] >= nc[e] ? 1 : 0);
        c[e] -= s * nc[e];
        code |= (s + 1) << (2 * e);
      } else {
        in = in && c[e] >= 0 && c[e] < nc[e];
      }
    }
    if (in) {
      const int cc = (c[0] * nc1 + c[1]) * nc2 + c[2];
      begin = w.start[cc];
      len = w.start[cc + 1] - begin;
    }
  }
  const int end = begin + len;
  const int pend = __shfl_up_sync(0xffffffffu, end, 1), pcode = __shfl_up_sync(0xffffffffu, code, 1);
  const bool opens = lane < nq && (lane == 0 || begin != pend || code != pcode);
  // lane q: first cell of the next run, and the end of q's own
  const unsigned later = (__ballot_sync(0xffffffffu, opens) >> lane) >> 1;
  const int next = later ? lane + __ffs(later) : nq;
  const int rend = __shfl_sync(0xffffffffu, end, next - 1);
  float bt[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) bt[k] = m->bt[k];
  const bool ortho = m->ortho != 0;
  const float lo = m->lo32, hi = m->hi32, small = m->small32;
  const float4 fi = w.cs32[at];
  constexpr float kRound = 12582912.f;  // 1.5 * 2^23: adding and taking it off rounds |x| < 2^22 to an integer
  for (int a = 0; a < nq;) {
    const int s = __shfl_sync(0xffffffffu, begin, a), e = __shfl_sync(0xffffffffu, rend, a);
    const int cd = __shfl_sync(0xffffffffu, code, a);
    a = __shfl_sync(0xffffffffu, next, a);
    float g0 = fi.x, g1 = fi.y, g2 = fi.z;
    if (fixed) {
      g0 += (cd & 1) ? 0.f : ((cd & 2) ? -1.f : 1.f);
      g1 += (cd & 4) ? 0.f : ((cd & 8) ? -1.f : 1.f);
      g2 += (cd & 16) ? 0.f : ((cd & 32) ? -1.f : 1.f);
    }
    for (int t0 = s; t0 < e; t0 += 32) {
      const int j = t0 + lane;
      bool in = false;
      if (j < e && j != at) {
        const float4 fj = w.cs32[j];
        float f0 = fj.x - g0, f1 = fj.y - g1, f2 = fj.z - g2;
        if (pbc && !fixed) {
          f0 -= (f0 + kRound) - kRound;
          f1 -= (f1 + kRound) - kRound;
          f2 -= (f2 + kRound) - kRound;
        }
        float r2;
        if (ortho) {
          const float v0 = f0 * bt[0], v1 = f1 * bt[4], v2 = f2 * bt[8];
          r2 = v0 * v0 + v1 * v1 + v2 * v2;
        } else {
          r2 = 0.f;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const float v = f0 * bt[k] + f1 * bt[3 + k] + f2 * bt[6 + k];
            r2 += v * v;
          }
        }
        if (r2 > hi) {
          in = false;
        } else if (r2 < lo && r2 > small) {
          in = true;
        } else {
          const double4 di = w.cs64[at], dj = w.cs64[j];
          double df[3] = {dj.x - di.x, dj.y - di.y, dj.z - di.z};
          double d2;
          if (pbc) {
            for (int k = 0; k < 3; ++k) df[k] -= floor(df[k] + 0.5);
            double dr[3];
            for (int k = 0; k < 3; ++k)
              dr[k] = df[0] * m->b[0 * 3 + k] + df[1] * m->b[1 * 3 + k] + df[2] * m->b[2 * 3 + k];
            d2 = dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2];
          } else {
            d2 = df[0] * df[0] + df[1] * df[1] + df[2] * df[2];
          }
          const double d = sqrt(d2);
          in = pbc ? (d < rc && d > 0.01) : (d < rc);
        }
      }
      visit(in, j);
    }
  }
}

// The neighbours of the atom at place `at` in no particular order: hit(k, j)
// is called by the lane that found the k-th one, j its atom index.
template <typename F>
__device__ __forceinline__ void nb_hits(int pbc, double rc, const NbWS& w, int at, F&& hit) {
  int cnt = 0;
  nb_search(pbc, rc, w, at, [&](bool in, int j) {
    const unsigned hits = __ballot_sync(0xffffffffu, in);
    if (in) hit(cnt + __popc(hits & ((1u << (threadIdx.x & 31)) - 1u)), w.sorted[j]);
    cnt += __popc(hits);
  });
}

// Counting pass: a warp per atom, in cell order (the warps of a block share
// candidate cells, so their loads hit L1).  Every lane collects its own hits,
// up to kNbLane, and one prefix sum at the end packs them.  The neighbours are
// kept for the filling pass if there are at most kNbKeep and none was dropped
// (kept[0] = -1 otherwise).
//
// The search was one thread per atom, run twice, with an insertion sort of the
// row in global memory.  20,000 atoms at 90 neighbours (FP32): counting 567 ->
// 60 us, filling 1937 -> 20 us; 1,536 atoms (FP64) 279 -> 14 and 1505 -> 5 us.
// It is bound by issue (70% of the cycles, ~2,300 instructions an atom, two
// thirds of them for the ~35 groups of 32 candidates).
constexpr int kNbLane = 12;

static __global__ void __launch_bounds__(256) nb_count_kernel(int pbc, int N, int mc, double rc, NbWS w0) {
  __shared__ int found[8][kNbLane][32];
  const NbWS w = nb_frame(w0, blockIdx.y, N, mc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int at = blockIdx.x * (blockDim.x >> 5) + warp;
  if (w.res->status || at >= w.start[w.meta->ncells]) return;
  int mine = 0;
  nb_search(pbc, rc, w, at, [&](bool in, int j) {
    if (in) {
      if (mine < kNbLane) found[warp][mine][lane] = j;
      ++mine;
    }
  });
  int upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += up;
  }
  const int cnt = __shfl_sync(0xffffffffu, upto, 31);
  const bool keep = __all_sync(0xffffffffu, mine <= kNbLane) && cnt <= kNbKeep;
  int* kept = w.kept + (size_t)at * kNbKeep;
  if (keep) {
    for (int k = 0; k < mine; ++k) kept[upto - mine + k] = w.sorted[found[warp][k][lane]];
  } else if (lane == 0) {
    kept[0] = -1;
  }
  if (lane == 0) w.rowcnt[w.sorted[at]] = cnt;
}

// Ascending bitonic sort of the 32 R values v[u] of a warp, element lane R + u.
template <int R>
__device__ __forceinline__ void nb_sort(int (&v)[R]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
    for (int s = k >> 1; s > 0; s >>= 1) {
      if (s < R) {  // both elements in this lane
#pragma unroll
        for (int u = 0; u < R; ++u) {
          if (u & s) continue;
          const bool up = k < R ? (u & k) == 0 : ((lane * R) & k) == 0;
          const int x = v[u], y = v[u + s];
          v[u] = up ? min(x, y) : max(x, y);
          v[u + s] = up ? max(x, y) : min(x, y);
        }
      } else {
        const bool low = (lane & (s / R)) == 0, up = ((lane * R) & k) == 0;
#pragma unroll
        for (int u = 0; u < R; ++u) {
          const int x = v[u], y = __shfl_xor_sync(0xffffffffu, x, s / R);
          v[u] = low == up ? min(x, y) : max(x, y);
        }
      }
    }
  }
}

// n <= 32 R values of `row` (shared or global) in ascending order into `out`
// (shared; values past n are not meaningful).
template <int R>
__device__ __forceinline__ void nb_order(const int* row, int n, int* out) {
  const int lane = threadIdx.x & 31;
  int v[R];
#pragma unroll
  for (int u = 0; u < R; ++u) v[u] = lane + 32 * u < n ? row[lane + 32 * u] : 0x7fffffff;
  nb_sort<R>(v);
  __syncwarp();
#pragma unroll
  for (int u = 0; u < R; ++u) out[lane * R + u] = v[u];
  __syncwarp();
}

// Output of the fill pass: frame f's rows start at pairs[f * stride].
struct NbOut {
  long long* pairs;
  long long* bscale;
  void* ds;            // distances in the positions' type, or null
  long long stride;    // rows of one frame's slice
  long long cap;       // rows that may be written in it
};

// Filling pass: a warp per atom orders its neighbours by index (bitonic sort
// in registers: about 260 instructions for 128 values, against 900 for ranking
// each value against all others) and writes the row, whole and coalesced, with
// the pair distances (admp_pair_distances) if they are asked for.  The rows of
// a frame's slice past its own pairs become (0, 0), distance 1, scale 0.
template <typename T>
__global__ void __launch_bounds__(256) nb_fill_kernel(int pbc, int N, int mc, double rc, NbWS w0,
                                                      const T* __restrict__ pos, NbOut o) {
  __shared__ __align__(16) int ord_sh[8][kNbRow];
  const int f = blockIdx.y;
  if (o.stride) {
    const NbResult* r = w0.res + f;
    for (long long k = r->npairs + blockIdx.x * (long long)blockDim.x + threadIdx.x; k < o.stride;
         k += (long long)gridDim.x * blockDim.x) {
      const size_t p = (size_t)f * o.stride + k;
      store_pair(o.pairs, p, 0, 0);
      if (o.bscale) o.bscale[p] = 0;
      if (o.ds) reinterpret_cast<T*>(o.ds)[p] = T(1);
    }
  }
  const NbWS w = nb_frame(w0, f, N, mc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int at = blockIdx.x * (blockDim.x >> 5) + warp;
  if (w.res->status || at >= w.start[w.meta->ncells]) return;
  const int i = w.sorted[at], n = w.rowcnt[i];
  const long long base = w.rowptr[i];
  if (n == 0 || base + n > o.cap) return;
  const size_t out = (size_t)f * o.stride + base;
  int* ord = ord_sh[warp];
  const NbMeta* __restrict__ m = w.meta;
  const T* ps = o.ds ? pos + (size_t)f * N * 3 : nullptr;
  double ri[3] = {0.0, 0.0, 0.0};
  if (o.ds)
    for (int e = 0; e < 3; ++e) ri[e] = (double)ps[3 * (size_t)i + e];
  auto emit = [&](int k, int j) {
    store_pair(o.pairs, out + k, i, j);
    if (o.bscale) o.bscale[out + k] = i < j ? 1 : 0;
    if (o.ds) {
      double dr[3], n[3];
      for (int e = 0; e < 3; ++e) dr[e] = ri[e] - (double)ps[3 * (size_t)j + e];
      if (pbc) min_image(m->b, m->bi, dr, n);
      reinterpret_cast<T*>(o.ds)[out + k] = (T)sqrt(dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2]);
    }
  };
  if (n <= kNbRow) {
    const int* row = w.kept + (size_t)at * kNbKeep;
    if (n > kNbKeep || row[0] < 0) {
      nb_hits(pbc, rc, w, at, [&](int k, int j) {
        if (k < kNbRow) ord[k] = j;
      });
      __syncwarp();
      row = ord;
    }
    if (n <= 32)
      nb_order<1>(row, n, ord);
    else if (n <= 64)
      nb_order<2>(row, n, ord);
    else if (n <= 128)
      nb_order<4>(row, n, ord);
    else
      nb_order<8>(row, n, ord);
    for (int k = lane; k < n; k += 32) emit(k, ord[k]);
  } else {
    // first column: unordered hits; second column: each at its rank; then the pairs
    nb_hits(pbc, rc, w, at, [&](int k, int j) {
      if (k < n) o.pairs[2 * (out + k)] = j;
    });
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
      const long long v = o.pairs[2 * (out + k)];
      int r = 0;
      for (int p = 0; p < n; ++p) r += o.pairs[2 * (out + p)] < v;
      o.pairs[2 * (out + r) + 1] = v;
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) emit(k, (int)o.pairs[2 * (out + k) + 1]);
  }
}

static int max_cells(int N) { return 2 * N + 128; }

static NbWS carve_nb(void* ws, size_t bytes, int nf, int N, size_t* need) {
  Carver c(ws, bytes);
  NbWS w;
  const size_t mc = (size_t)(max_cells(N) + 1) * nf, NT = (size_t)N * nf;
  w.meta = c.take<NbMeta>(nf);
  w.res = c.take<NbResult>(nf);
  w.cs64 = c.take<double4>(NT);
  w.cs32 = c.take<float4>(NT);
  w.cell = c.take<int>(NT);
  w.slot = c.take<int>(NT);
  w.count = c.take<int>(mc);
  w.start = c.take<int>(mc);
  w.sorted = c.take<int>(NT);
  w.scell = c.take<int>(NT);
  w.kept = c.take<int>(NT * kNbKeep);
  w.rowcnt = c.take<int>(NT);
  w.rowptr = c.take<long long>((size_t)(N + 1) * nf);
  *need = c.off;
  return w;
}

template <typename T>
static int nblist_count_impl(int pbc, int nf, int N, const T* pos, const T* box, double rc, void* ws, size_t bytes,
                             long long* npairs, cudaStream_t st) {
  size_t need;
  NbWS w = carve_nb(ws, bytes, nf, N, &need);
  if (need > bytes || !ws) return fail(ADMP_ERR_WORKSPACE, "nblist workspace: need %zu bytes, got %zu", need, bytes);
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  const int mc = max_cells(N);
  if (N <= kNbOneBlock) {
    nb_setup_kernel<T, true><<<nf, 1024, 0, st>>>(pbc, N, mc, pos, box, rc, w, err);
  } else {
    const dim3 grid((N + 255) / 256, nf);
    nb_setup_kernel<T, false><<<nf, 1024, 0, st>>>(pbc, N, mc, pos, box, rc, w, err);
    nb_bin_kernel<T><<<grid, 256, 0, st>>>(pbc, N, mc, pos, w, err);
    nb_cell_scan_kernel<<<nf, 1024, 0, st>>>(N, mc, w);
    nb_scatter_kernel<T><<<grid, 256, 0, st>>>(pbc, N, mc, pos, w);
  }
  nb_count_kernel<<<dim3((N + 7) / 8, nf), 256, 0, st>>>(pbc, N, mc, rc, w);
  nb_row_scan_kernel<<<nf, 1024, 0, st>>>(N, mc, w, err);
  ADMP_CUDA_TRY(cudaGetLastError());
  const NbResult* h = (const NbResult*)read_back(w.res, sizeof(NbResult) * nf, st);
  if (!h) return ADMP_ERR_CUDA;
  int ecode = 0;
  for (int f = 0; f < nf; ++f) {
    if (h[f].status == ADMP_ERR_CUTOFF_TOO_LARGE)
      return fail(ADMP_ERR_CUTOFF_TOO_LARGE, "Cutoff %g is larger than half the minimum height of the box.", rc);
    if (h[f].status) return fail(h[f].status, "neighbour list: invalid box or positions");
    ecode |= h[f].ecode;
    npairs[f] = h[f].npairs;
  }
  return ecode ? check_error(err, st) : ADMP_OK;
}

template <typename T>
static int nblist_fill_impl(int pbc, int nf, int N, double rc, const NbWS& w, const T* pos, const NbOut& o,
                            cudaStream_t st) {
  nb_fill_kernel<T><<<dim3((N + 7) / 8, nf), 256, 0, st>>>(pbc, N, max_cells(N), rc, w, pos, o);
  ADMP_CUDA_TRY(cudaGetLastError());
  return ADMP_OK;
}

}  // namespace admp

using namespace admp;

extern "C" size_t admp_nblist_workspace_size(int natoms) {
  size_t need;
  carve_nb(nullptr, 0, 1, natoms < 0 ? 0 : natoms, &need);
  return need;
}

extern "C" size_t admp_nblist_frames_workspace_size(int nframes, int natoms) {
  size_t need;
  carve_nb(nullptr, 0, nframes < 0 ? 0 : nframes, natoms < 0 ? 0 : natoms, &need);
  return need;
}

extern "C" int admp_nblist_frames_count(int dtype, int pbc, int nframes, int natoms, const void* pos, const void* box,
                                        double cutoff, void* workspace, size_t workspace_bytes, long long* npairs,
                                        void* stream) {
  if (!npairs) return fail(ADMP_ERR_BAD_ARG, "npairs is null");
  if (nframes < 0 || nframes > ADMP_NBLIST_MAX_FRAMES)
    return fail(ADMP_ERR_BAD_ARG, "admp_nblist_count: %d frames (0..%d)", nframes, ADMP_NBLIST_MAX_FRAMES);
  for (int f = 0; f < nframes; ++f) npairs[f] = 0;
  if (natoms == 0 || nframes == 0) return ADMP_OK;
  if (natoms < 0 || !pos || (pbc && !box) || !(cutoff > 0)) return fail(ADMP_ERR_BAD_ARG, "admp_nblist_count: args");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return nblist_count_impl<double>(pbc, nframes, natoms, (const double*)pos, (const double*)box, cutoff, workspace,
                                     workspace_bytes, npairs, st);
  if (dtype == ADMP_F32)
    return nblist_count_impl<float>(pbc, nframes, natoms, (const float*)pos, (const float*)box, cutoff, workspace,
                                    workspace_bytes, npairs, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_nblist_count(int dtype, int pbc, int natoms, const void* pos, const void* box, double cutoff,
                                 void* workspace, size_t workspace_bytes, long long* npairs, void* stream) {
  return admp_nblist_frames_count(dtype, pbc, 1, natoms, pos, box, cutoff, workspace, workspace_bytes, npairs, stream);
}

extern "C" int admp_nblist_frames_fill(int dtype, int pbc, int nframes, int natoms, const void* pos, double cutoff,
                                       void* workspace, size_t workspace_bytes, long long stride, long long* pairs,
                                       long long* buffer_scales, void* ds, void* stream) {
  if (nframes < 0 || nframes > ADMP_NBLIST_MAX_FRAMES || natoms < 0 || stride < 0)
    return fail(ADMP_ERR_BAD_ARG, "admp_nblist_frames_fill: args");
  if (natoms == 0 || nframes == 0 || stride == 0) return ADMP_OK;
  if (!pos || !pairs) return fail(ADMP_ERR_BAD_ARG, "admp_nblist_frames_fill: args");
  size_t need;
  const NbWS w = carve_nb(workspace, workspace_bytes, nframes, natoms, &need);
  if (need > workspace_bytes || !workspace) return fail(ADMP_ERR_WORKSPACE, "nblist workspace too small");
  const NbOut o{pairs, buffer_scales, ds, stride, stride};
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64) return nblist_fill_impl<double>(pbc, nframes, natoms, cutoff, w, (const double*)pos, o, st);
  if (dtype == ADMP_F32) return nblist_fill_impl<float>(pbc, nframes, natoms, cutoff, w, (const float*)pos, o, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_nblist_fill(int dtype, int pbc, int natoms, const void* pos, const void* box, double cutoff,
                                void* workspace, size_t workspace_bytes, long long* pairs, long long* buffer_scales,
                                long long capacity, void* stream) {
  (void)pos;
  (void)box;
  if (natoms == 0) return ADMP_OK;
  if (natoms < 0 || (capacity > 0 && !pairs)) return fail(ADMP_ERR_BAD_ARG, "admp_nblist_fill: args");
  if (dtype != ADMP_F64 && dtype != ADMP_F32) return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  cudaStream_t st = (cudaStream_t)stream;
  size_t need;
  NbWS w = carve_nb(workspace, workspace_bytes, 1, natoms, &need);
  if (need > workspace_bytes || !workspace) return fail(ADMP_ERR_WORKSPACE, "nblist workspace too small");
  const NbResult* h = (const NbResult*)read_back(w.res, sizeof(NbResult), st);
  if (!h) return ADMP_ERR_CUDA;
  const long long total = h->npairs;
  if (total > capacity)
    return fail(ADMP_ERR_CAPACITY, "neighbour list: %lld pairs exceed capacity %lld", total, capacity);
  if (total == 0) return ADMP_OK;
  return nblist_fill_impl<double>(pbc, 1, natoms, cutoff, w, nullptr, NbOut{pairs, buffer_scales, nullptr, 0, capacity},
                                  st);
}
