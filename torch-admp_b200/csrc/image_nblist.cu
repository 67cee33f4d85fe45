// Neighbour list over periodic images, for cutoffs above half the box
// (the pair set of dp_nblist, nblist.py:33-93 and make_local_pairs /
// make_ds, nblist.py:173-240): every periodic image j + n.B of atom j within
// rc of atom i gives one pair (i, j) with i < j (buffer scale 1), and every
// image i + n.B (n != 0) of atom i itself gives a pair (i, i) (scale 1/2);
// the pair distances are |r_j - r_i + n.B| with the image shift n stored per
// pair, so they are differentiable in the positions and the box.
//
// Atoms are wrapped into the cell for the search (fractional coordinates
// mod 1); the stored shift refers to the caller's unwrapped positions.  With
// wrapped coordinates |f_j - f_i| < 1, so images |n_d| <= ceil(rc / h_d) cover
// the cutoff (h_d = V / |b_e x b_f| the height of the cell along axis d).
// The search is O(N^2 x images), meant for the small cells that need it.
#include "admp_common.cuh"
#include "runtime.h"

namespace admp {

struct ImgGeom {
  double b[9], bi[9];
  int m[3];
  int pbc;
  int bad;  // more images than an atom's counts hold
};

// Open boundaries (pbc == 0, box unused): identity cell, no wrap, no images.
// A singular box, or a cutoff of more than 2^19 - 1 cells along an axis or 2^31
// images in all (the packed image vectors and the counts), has no image walked.
template <typename T>
__device__ __forceinline__ void img_geom(const T* box, int pbc, double rc, ImgGeom& g) {
  g.pbc = pbc;
  g.bad = 0;
  if (!pbc) {
    for (int k = 0; k < 9; ++k) g.b[k] = g.bi[k] = (k % 4 == 0) ? 1.0 : 0.0;
    g.m[0] = g.m[1] = g.m[2] = 0;
    return;
  }
  load_box(box, g.b);
  const double V = fabs(inv3(g.b, g.bi));
  double images = 1.0, most = 0.0;
  for (int d = 0; d < 3; ++d) {
    const double* u = g.b + ((d + 1) % 3) * 3;
    const double* v = g.b + ((d + 2) % 3) * 3;
    const double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2], cz = u[0] * v[1] - u[1] * v[0];
    const double h = V / sqrt(cx * cx + cy * cy + cz * cz);
    const double m = ceil(rc / h);
    g.m[d] = (int)m;
    images *= 2.0 * m + 1.0;
    most = fmax(most, m);
  }
  if (images > 2147483647.0 || most > (double)((1 << 19) - 1)) {
    g.bad = 1;
    g.m[0] = g.m[1] = g.m[2] = 0;
  }
}

// Wrapped fractional coordinates and integer cell offsets of every atom.
template <typename T>
__global__ void __launch_bounds__(256) img_frac_kernel(int N, const T* __restrict__ pos, const T* __restrict__ box,
                                                       int pbc, double rc, double* __restrict__ frac,
                                                       int* __restrict__ cell, int* __restrict__ ntrunc) {
  __shared__ ImgGeom g;
  if (threadIdx.x == 0) img_geom<T>(box, pbc, rc, g);
  if (blockIdx.x == 0 && threadIdx.x == 0) *ntrunc = g.bad ? -1 : 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double r0 = pos[3 * (size_t)i], r1 = pos[3 * (size_t)i + 1], r2 = pos[3 * (size_t)i + 2];
  for (int e = 0; e < 3; ++e) {
    const double x = r0 * g.bi[0 * 3 + e] + r1 * g.bi[1 * 3 + e] + r2 * g.bi[2 * 3 + e];
    const double fl = g.pbc ? floor(x) : 0.0;
    frac[3 * (size_t)i + e] = x - fl;
    cell[3 * (size_t)i + e] = (int)fl;
  }
}

// A block of kImgWarps warps per atom i.  The images (j, n) of an atom are one
// sequence, j-major; each warp takes a contiguous part of it, 32 at a time, so
// the hits of the parts follow each other in the output order.
constexpr int kImgWarps = 8;
constexpr int kImgKeep = 1536;   // r^2 of an atom's images kept in shared memory for the nnei cut
constexpr int kImgTable = 1024;  // image vectors tabulated in shared memory

struct ImgBlock {
  ImgGeom g;
  long long nimg;
  long long tab[kImgTable];  // packed image vectors of the first kImgTable images
};

// 20 bits a component, offset by 2^19
__device__ __forceinline__ long long img_pack(const ImgGeom& g, long long k) {
  const long long n2 = 2 * g.m[2] + 1, n1 = 2 * g.m[1] + 1, q = k / n2, o = 1 << 19;
  return ((q / n1 - g.m[0] + o) << 40) | ((q % n1 - g.m[1] + o) << 20) | (k - q * n2 - g.m[2] + o);
}

template <typename T>
__device__ __forceinline__ void img_block(ImgBlock& b, const T* box, int pbc, double rc) {
  if (threadIdx.x == 0) {
    img_geom<T>(box, pbc, rc, b.g);
    b.nimg = (2LL * b.g.m[0] + 1) * (2LL * b.g.m[1] + 1) * (2LL * b.g.m[2] + 1);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < min(b.nimg, (long long)kImgTable); k += blockDim.x) b.tab[k] = img_pack(b.g, k);
  __syncthreads();
}

// The calling warp visits positions [t0, t1) of atom i's image sequence:
// visit(in, j, na, nb, nc, r2) by all lanes for every 32, `in` for an image
// within sqrt(thr2) other than the atom itself.
template <typename F>
__device__ __forceinline__ void img_visit(const ImgBlock& b, const double* __restrict__ frac, int i, double thr2,
                                          long long t0, long long t1, F&& visit) {
  const int lane = threadIdx.x & 31;
  const double f0 = frac[3 * (size_t)i], f1 = frac[3 * (size_t)i + 1], f2 = frac[3 * (size_t)i + 2];
  const long long nimg = b.nimg, dk = 32 % nimg;
  const int dj = (int)(32 / nimg);
  int j = (int)((t0 + lane) / nimg);
  long long k = t0 + lane - (long long)j * nimg;
  for (long long t = t0; t < t1; t += 32) {
    bool in = false;
    int na = 0, nb = 0, nc = 0;
    double r2 = 0.0;
    if (t + lane < t1) {
      const long long code = k < kImgTable ? b.tab[k] : img_pack(b.g, k);
      na = (int)(code >> 40) - (1 << 19);
      nb = (int)((code >> 20) & 0xfffff) - (1 << 19);
      nc = (int)(code & 0xfffff) - (1 << 19);
      const double df[3] = {frac[3 * (size_t)j] - f0 + na, frac[3 * (size_t)j + 1] - f1 + nb,
                            frac[3 * (size_t)j + 2] - f2 + nc};
      for (int e = 0; e < 3; ++e) {
        const double v = df[0] * b.g.b[0 * 3 + e] + df[1] * b.g.b[1 * 3 + e] + df[2] * b.g.b[2 * 3 + e];
        r2 += v * v;
      }
      in = r2 <= thr2 && !(j == i && na == 0 && nb == 0 && nc == 0);
    }
    visit(in, j, na, nb, nc, r2);
    k += dk;
    j += dj;
    if (k >= nimg) {
      k -= nimg;
      ++j;
    }
  }
}

// part `w` of kImgWarps of [lo, hi), 32-aligned within it
__device__ __forceinline__ void img_part(long long lo, long long hi, int w, long long& t0, long long& t1) {
  const long long step = ((hi - lo + kImgWarps - 1) / kImgWarps + 31) / 32 * 32;
  t0 = min(lo + w * step, hi);
  t1 = min(t0 + step, hi);
}

__device__ __forceinline__ int img_block_sum(int v, int* red) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  int s = 0;
  for (int w = 0; w < kImgWarps; ++w) s += red[w];
  return s;
}

// Per atom: the squared radius that keeps its `nnei` nearest images (all of
// them when it has no more than nnei within rc).  The nnei-th smallest r^2 is
// found exactly by bisection over the bit patterns of non-negative doubles,
// which order like the values; the r^2 within rc are kept in shared memory for
// it (searched for again at every step past kImgKeep of them).  Then the
// (i, j >= i) pair counts of each part.
//
// One thread per atom took 1,148 us (count) and 717 us (fill) for 280 atoms at
// rc 9 A (27 images); a block per atom 24 and 17 us.
template <typename T>
__global__ void __launch_bounds__(32 * kImgWarps)
    img_count_kernel(int N, const double* __restrict__ frac, const T* __restrict__ box, int pbc, double rc, int nnei,
                     double* __restrict__ thr, int* __restrict__ cnt_ij, int* __restrict__ cnt_ii,
                     int* __restrict__ ntrunc) {
  __shared__ ImgBlock b;
  __shared__ double kept[kImgKeep];
  __shared__ int red[kImgWarps], nkept;
  if (threadIdx.x == 0) nkept = 0;
  img_block<T>(b, box, pbc, rc);
  const int i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (b.g.bad) {
    if (lane == 0) cnt_ij[i * kImgWarps + warp] = cnt_ii[i * kImgWarps + warp] = 0;
    if (threadIdx.x == 0) thr[i] = -1.0;
    return;
  }
  const double rc2 = rc * rc;
  const long long all = (long long)N * b.nimg;
  long long t0, t1;
  double t2 = rc2;
  if (nnei >= 0) {
    img_part(0, all, warp, t0, t1);
    auto count = [&](double within) {
      int n = 0;
      img_visit(b, frac, i, within, t0, t1, [&](bool in, int, int, int, int, double) { n += in; });
      return img_block_sum(n, red);
    };
    int mine = 0;
    img_visit(b, frac, i, rc2, t0, t1, [&](bool in, int, int, int, int, double r2) {
      if (in) {
        ++mine;
        const int k = atomicAdd(&nkept, 1);
        if (k < kImgKeep) kept[k] = r2;
      }
    });
    const int total = img_block_sum(mine, red);
    if (total > nnei) {  // block-uniform
      if (threadIdx.x == 0) atomicAdd(ntrunc, 1);
      if (nnei == 0) {
        t2 = -1.0;
      } else {
        unsigned long long lo = 0ull, hi = (unsigned long long)__double_as_longlong(rc2);
        while (lo < hi) {  // smallest bits with count(r2 <= value) >= nnei
          const unsigned long long mid = lo + (hi - lo) / 2;
          const double within = __longlong_as_double((long long)mid);
          int n;
          if (total <= kImgKeep) {
            n = 0;
            for (int k = threadIdx.x; k < total; k += blockDim.x) n += kept[k] <= within;
            n = img_block_sum(n, red);
          } else {
            n = count(within);
          }
          if (n >= nnei)
            hi = mid;
          else
            lo = mid + 1;
        }
        t2 = __longlong_as_double((long long)lo);
      }
    }
  }
  if (threadIdx.x == 0) thr[i] = t2;
  img_part((long long)i * b.nimg, all, warp, t0, t1);
  int nij = 0, nii = 0;
  img_visit(b, frac, i, t2, t0, t1, [&](bool in, int j, int, int, int, double) {
    nij += in && j != i;
    nii += in && j == i;
  });
  nij = warp_sum(nij);
  nii = warp_sum(nii);
  if (lane == 0) {
    cnt_ij[i * kImgWarps + warp] = nij;
    cnt_ii[i * kImgWarps + warp] = nii;
  }
}

template <typename T>
__global__ void __launch_bounds__(32 * kImgWarps)
    img_fill_kernel(int N, const double* __restrict__ frac, const int* __restrict__ cell, const T* __restrict__ box,
                    int pbc, double rc, const double* __restrict__ thr, const long long* __restrict__ off_ij,
                    const long long* __restrict__ off_ii, long long base_ii, long long* __restrict__ pairs,
                    int* __restrict__ shifts) {
  __shared__ ImgBlock b;
  img_block<T>(b, box, pbc, rc);
  const int i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  long long pij = off_ij[i * kImgWarps + warp], pii = base_ii + off_ii[i * kImgWarps + warp];
  const int k0 = cell[3 * (size_t)i], k1 = cell[3 * (size_t)i + 1], k2 = cell[3 * (size_t)i + 2];
  long long t0, t1;
  img_part((long long)i * b.nimg, (long long)N * b.nimg, warp, t0, t1);
  img_visit(b, frac, i, thr[i], t0, t1, [&](bool in, int j, int na, int nb, int nc, double) {
    const unsigned self = __ballot_sync(0xffffffffu, in && j == i), other = __ballot_sync(0xffffffffu, in && j != i);
    if (in) {
      const unsigned below = (1u << lane) - 1u;
      const long long p = j == i ? pii + __popc(self & below) : pij + __popc(other & below);
      store_pair(pairs, p, i, j);
      // relative to the caller's unwrapped positions: n + k_i - k_j
      shifts[3 * p] = na + k0 - cell[3 * (size_t)j];
      shifts[3 * p + 1] = nb + k1 - cell[3 * (size_t)j + 1];
      shifts[3 * p + 2] = nc + k2 - cell[3 * (size_t)j + 2];
    }
    pii += __popc(self);
    pij += __popc(other);
  });
}

// ds = |r_j - r_i + n.B|
template <typename T>
__global__ void __launch_bounds__(256) img_dist_kernel(int N, long long P, const long long* __restrict__ pairs,
                                                       const int* __restrict__ shifts, const T* __restrict__ pos,
                                                       const T* __restrict__ box, T* __restrict__ ds, DevError* err) {
  __shared__ double b[9];
  if (threadIdx.x < 9) b[threadIdx.x] = box ? (double)box[threadIdx.x] : 0.0;
  __syncthreads();
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const long long i = pairs[2 * p], j = pairs[2 * p + 1];
    if (i < 0 || i >= N || j < 0 || j >= N) {
      report_error(err, ADMP_ERR_BAD_INDEX, 4, p);
      ds[p] = T(0);
      continue;
    }
    double r2 = 0.0;
    for (int e = 0; e < 3; ++e) {
      const double v = (double)pos[3 * j + e] - (double)pos[3 * i + e] + shifts[3 * p] * b[e] +
                       shifts[3 * p + 1] * b[3 + e] + shifts[3 * p + 2] * b[6 + e];
      r2 += v * v;
    }
    ds[p] = (T)sqrt(r2);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) img_dist_bwd_kernel(int N, long long P, const long long* __restrict__ pairs,
                                                           const int* __restrict__ shifts, const T* __restrict__ pos,
                                                           const T* __restrict__ box, const T* __restrict__ g,
                                                           T* __restrict__ gpos, T* __restrict__ gbox, DevError* err) {
  __shared__ double b[9];
  __shared__ double red[9 * 32];
  if (threadIdx.x < 9) b[threadIdx.x] = box ? (double)box[threadIdx.x] : 0.0;
  __syncthreads();
  double vb[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const long long i = pairs[2 * p], j = pairs[2 * p + 1];
    if (i < 0 || i >= N || j < 0 || j >= N) {
      report_error(err, ADMP_ERR_BAD_INDEX, 5, p);
      continue;
    }
    const double gp = g[p];
    if (gp == 0.0) continue;
    const int n[3] = {shifts[3 * p], shifts[3 * p + 1], shifts[3 * p + 2]};
    double dr[3];
    for (int e = 0; e < 3; ++e)
      dr[e] = (double)pos[3 * j + e] - (double)pos[3 * i + e] + n[0] * b[e] + n[1] * b[3 + e] + n[2] * b[6 + e];
    const double d = sqrt(dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2]);
    if (d == 0.0) continue;
    const double s = gp / d;
    for (int e = 0; e < 3; ++e) {
      const double v = s * dr[e];
      if (gpos && i != j) {
        atomicAdd(gpos + 3 * j + e, (T)v);
        atomicAdd(gpos + 3 * i + e, (T)(-v));
      }
      for (int a = 0; a < 3; ++a) vb[a * 3 + e] += n[a] * v;
    }
  }
  if (gbox && box) {
    __shared__ double out[9];
    if (threadIdx.x < 9) out[threadIdx.x] = 0.0;
    __syncthreads();
    block_atomic_sum<9>(vb, out, red);
    if (threadIdx.x < 9 && out[threadIdx.x] != 0.0) atomicAdd(gbox + threadIdx.x, (T)out[threadIdx.x]);
  }
}

// What the host reads back.
struct ImgResult {
  long long n_ij, n_ii;
  int ntrunc, pad;
};

// Exclusive scans of the two part-count arrays into long long offsets (block
// 0: i < j pairs, block 1: self images), tiles of 1024 values.
static __global__ void __launch_bounds__(1024) img_scan_kernel(const int* __restrict__ cij, const int* __restrict__ cii,
                                                               long long* __restrict__ oij, long long* __restrict__ oii,
                                                               int n, const int* __restrict__ ntrunc, ImgResult* res) {
  __shared__ long long wsum[32], tile;
  const int* in = blockIdx.x ? cii : cij;
  long long* out = blockIdx.x ? oii : oij;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long carry = 0;
  for (int b = 0; b < n; b += 1024) {
    const int i = b + threadIdx.x;
    const long long v = i < n ? in[i] : 0;
    long long inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const long long up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += up;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      const long long x = wsum[lane];
      long long y = x;
      for (int o = 1; o < 32; o <<= 1) {
        const long long up = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += up;
      }
      wsum[lane] = y - x;
      if (lane == 31) tile = y;
    }
    __syncthreads();
    if (i < n) out[i] = carry + wsum[warp] + inc - v;
    carry += tile;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    (blockIdx.x ? res->n_ii : res->n_ij) = carry;
    if (blockIdx.x == 0) res->ntrunc = *ntrunc;
  }
}

// workspace: thr [N] double, wrapped coordinates, part counts and offsets
// [kImgWarps N], truncated-atom count, result record
struct ImgWS {
  double *thr, *frac;
  int *cell, *cij, *cii, *ntrunc;
  long long *oij, *oii;
  ImgResult* res;
};

static size_t img_carve(void* ws, int N, ImgWS* w) {
  Carver c(ws, 0);
  const size_t parts = (size_t)N * kImgWarps;
  w->thr = c.take<double>(N);
  w->frac = c.take<double>(3 * (size_t)N);
  w->cell = c.take<int>(3 * (size_t)N);
  w->cij = c.take<int>(parts);
  w->cii = c.take<int>(parts);
  w->oij = c.take<long long>(parts);
  w->oii = c.take<long long>(parts);
  w->ntrunc = c.take<int>(1);
  w->res = c.take<ImgResult>(1);
  return c.off;
}

template <typename T>
static int img_count_impl(int pbc, int N, const T* pos, const T* box, double rc, int nnei, void* ws, size_t bytes,
                          long long* n_ij, long long* n_ii, int* n_truncated, cudaStream_t st) {
  ImgWS w;
  const size_t need = img_carve(ws, N, &w);
  if (!ws || need > bytes) return fail(ADMP_ERR_WORKSPACE, "image neighbour list: workspace needs %zu bytes", need);
  img_frac_kernel<T><<<(N + 255) / 256, 256, 0, st>>>(N, pos, box, pbc, rc, w.frac, w.cell, w.ntrunc);
  img_count_kernel<T><<<N, 32 * kImgWarps, 0, st>>>(N, w.frac, box, pbc, rc, nnei, w.thr, w.cij, w.cii, w.ntrunc);
  img_scan_kernel<<<2, 1024, 0, st>>>(w.cij, w.cii, w.oij, w.oii, N * kImgWarps, w.ntrunc, w.res);
  count_launches(3);
  ADMP_CUDA_TRY(cudaGetLastError());
  const ImgResult* h = (const ImgResult*)read_back(w.res, sizeof(ImgResult), st);
  if (!h) return ADMP_ERR_CUDA;
  if (h->ntrunc < 0)
    return fail(ADMP_ERR_BAD_ARG, "image neighbour list: cutoff %g takes too many images of the box (or it is singular)", rc);
  *n_ij = h->n_ij;
  *n_ii = h->n_ii;
  if (n_truncated) *n_truncated = h->ntrunc;
  return ADMP_OK;
}

template <typename T>
static int img_fill_impl(int pbc, int N, const T* pos, const T* box, double rc, void* ws, size_t bytes,
                         long long* pairs, int* shifts, long long capacity, cudaStream_t st) {
  ImgWS w;
  const size_t need = img_carve(ws, N, &w);
  if (!ws || need > bytes) return fail(ADMP_ERR_WORKSPACE, "image neighbour list: workspace needs %zu bytes", need);
  const ImgResult* h = (const ImgResult*)read_back(w.res, sizeof(ImgResult), st);
  if (!h) return ADMP_ERR_CUDA;
  const long long n_ij = h->n_ij, total = h->n_ij + h->n_ii;
  if (total > capacity)
    return fail(ADMP_ERR_CAPACITY, "image neighbour list: %lld pairs, capacity %lld", total, capacity);
  if (total == 0) return ADMP_OK;
  img_fill_kernel<T><<<N, 32 * kImgWarps, 0, st>>>(N, w.frac, w.cell, box, pbc, rc, w.thr, w.oij, w.oii, n_ij, pairs,
                                                   shifts);
  count_launches(1);
  ADMP_CUDA_TRY(cudaGetLastError());
  return ADMP_OK;
}

}  // namespace admp

using namespace admp;

extern "C" size_t admp_image_nblist_workspace_size(int natoms) {
  ImgWS w;
  return img_carve(nullptr, natoms < 0 ? 0 : natoms, &w);
}

extern "C" int admp_image_nblist_count(int dtype, int pbc, int natoms, const void* pos, const void* box,
                                       double cutoff, int nnei, void* workspace, size_t workspace_bytes,
                                       long long* n_ij, long long* n_ii, int* n_truncated, void* stream) {
  if (!n_ij || !n_ii) return fail(ADMP_ERR_BAD_ARG, "admp_image_nblist_count: null outputs");
  *n_ij = 0;
  *n_ii = 0;
  if (n_truncated) *n_truncated = 0;
  if (!(cutoff > 0)) return fail(ADMP_ERR_BAD_ARG, "rcut must be positive, got %g", cutoff);
  if (natoms == 0) return ADMP_OK;
  if (natoms < 0 || !pos || (pbc && !box)) return fail(ADMP_ERR_BAD_ARG, "admp_image_nblist_count: args");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return img_count_impl<double>(pbc, natoms, (const double*)pos, (const double*)box, cutoff, nnei, workspace,
                                  workspace_bytes, n_ij, n_ii, n_truncated, st);
  if (dtype == ADMP_F32)
    return img_count_impl<float>(pbc, natoms, (const float*)pos, (const float*)box, cutoff, nnei, workspace,
                                 workspace_bytes, n_ij, n_ii, n_truncated, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_image_nblist_fill(int dtype, int pbc, int natoms, const void* pos, const void* box,
                                      double cutoff, void* workspace, size_t workspace_bytes, long long* pairs,
                                      int* shifts, long long capacity, void* stream) {
  if (natoms == 0) return ADMP_OK;
  if (natoms < 0 || !pos || (pbc && !box) || (capacity > 0 && (!pairs || !shifts)))
    return fail(ADMP_ERR_BAD_ARG, "admp_image_nblist_fill: args");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return img_fill_impl<double>(pbc, natoms, (const double*)pos, (const double*)box, cutoff, workspace,
                                 workspace_bytes, pairs, shifts, capacity, st);
  if (dtype == ADMP_F32)
    return img_fill_impl<float>(pbc, natoms, (const float*)pos, (const float*)box, cutoff, workspace,
                                workspace_bytes, pairs, shifts, capacity, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_image_pair_distances(int dtype, int natoms, long long npairs, const long long* pairs,
                                         const int* shifts, const void* pos, const void* box, void* ds, void* stream) {
  if (npairs == 0) return ADMP_OK;
  if (npairs < 0 || !pairs || !shifts || !pos || !ds)
    return fail(ADMP_ERR_BAD_ARG, "admp_image_pair_distances: args");
  cudaStream_t st = (cudaStream_t)stream;
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  long long blocks = (npairs + 255) / 256;
  if (blocks > 8192) blocks = 8192;
  if (dtype == ADMP_F64)
    img_dist_kernel<double><<<(unsigned)blocks, 256, 0, st>>>(natoms, npairs, pairs, shifts, (const double*)pos,
                                                              (const double*)box, (double*)ds, err);
  else if (dtype == ADMP_F32)
    img_dist_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(natoms, npairs, pairs, shifts, (const float*)pos,
                                                             (const float*)box, (float*)ds, err);
  else
    return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  count_launches(1);
  ADMP_CUDA_TRY(cudaGetLastError());
  return check_error(err, st);
}

extern "C" int admp_image_pair_distances_backward(int dtype, int natoms, long long npairs, const long long* pairs,
                                                  const int* shifts, const void* pos, const void* box,
                                                  const void* grad_ds, void* grad_pos, void* grad_box, void* stream) {
  if (npairs == 0) return ADMP_OK;
  if (npairs < 0 || !pairs || !shifts || !pos || !grad_ds)
    return fail(ADMP_ERR_BAD_ARG, "admp_image_pair_distances_backward: args");
  cudaStream_t st = (cudaStream_t)stream;
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  long long blocks = (npairs + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  if (dtype == ADMP_F64)
    img_dist_bwd_kernel<double><<<(unsigned)blocks, 256, 0, st>>>(natoms, npairs, pairs, shifts, (const double*)pos,
                                                                  (const double*)box, (const double*)grad_ds,
                                                                  (double*)grad_pos, (double*)grad_box, err);
  else if (dtype == ADMP_F32)
    img_dist_bwd_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(natoms, npairs, pairs, shifts, (const float*)pos,
                                                                 (const float*)box, (const float*)grad_ds,
                                                                 (float*)grad_pos, (float*)grad_box, err);
  else
    return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  count_launches(1);
  ADMP_CUDA_TRY(cudaGetLastError());
  return check_error(err, st);
}
