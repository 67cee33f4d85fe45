// Charges of a dense quadratic model with at most one linear constraint:
// H q + C^T lam = -chi, C q = b (qeq.py:1530-1617), H symmetric positive
// definite, in double precision.  One cooperative launch: Cholesky by tiles of
// 32 with -chi and C as further rows, so that the forward substitution comes
// with the factorisation, then the backward substitution and the Schur
// complement by one block.
//
// A few hundred atoms are bound by the chain of tile columns, not by
// arithmetic.  A block solves the two panel tiles that its trailing tile needs
// by itself, and the block of the next diagonal tile factorises it before it
// meets the others, so that a column costs one barrier over the grid.  201 / 429 /
// 1,024 unknowns: 130 / 225 / 575 us, where the library's Cholesky, its two
// triangular solves and the steps between took 326 / 520 / 1,020 (with as many
// unknowns as 1,536 and no constraint they were the faster: 1,024 and 940).
// Of the 11 us of a column the factor takes 3.5, panel and update 2.5, the
// barrier 1.6, loads 1, the backward substitution 2.3.
#include "pme_host.h"
#include "qeq_cg.cuh"

namespace admp {

constexpr int kSpdTile = 32;
constexpr int kSpdThreads = 512;

struct SpdArgs {
  int n, nt;  // unknowns, tile columns
  const double *H, *chi, *C, *b;
  double *A, *L;  // (nt + 1) x nt tiles, row-major; the last tile row holds the right-hand sides
  double* q;
  int* info;  // 0, or the column at which H is not positive definite + 1, or n + 1 for a zero Schur complement
  CgShared* sh;
};

typedef double SpdTile[kSpdTile][kSpdTile + 1];

// A thread's two values of a tile, taken to registers first: the loads of several tiles are then in flight together.
static_assert(kSpdThreads == kSpdTile * kSpdTile / 2, "two values a thread");
__device__ __forceinline__ double2 spd_fetch(const double* src, int ld) {
  const double* p = src + (size_t)(threadIdx.x >> 5) * ld + (threadIdx.x & 31);
  return make_double2(p[0], p[(size_t)(kSpdTile / 2) * ld]);
}
__device__ __forceinline__ void spd_put(SpdTile& t, double2 v) {
  t[threadIdx.x >> 5][threadIdx.x & 31] = v.x;
  t[(threadIdx.x >> 5) + kSpdTile / 2][threadIdx.x & 31] = v.y;
}

__device__ __forceinline__ void spd_store(double* dst, const SpdTile& t, int ld) {
  for (int e = threadIdx.x; e < kSpdTile * kSpdTile; e += kSpdThreads) dst[(size_t)(e >> 5) * ld + (e & 31)] = t[e >> 5][e & 31];
}

// Cholesky factor of a diagonal tile by one warp, lane = row; the diagonal becomes 1 / L_jj.  Returns the column at
// which a pivot was not positive, or 32.
__device__ __forceinline__ int spd_factor(SpdTile& t, int lane) {
  double a[kSpdTile];
#pragma unroll
  for (int c = 0; c < kSpdTile; ++c) a[c] = t[lane][c];
  int bad = kSpdTile;
  double d = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
  for (int j = 0; j < kSpdTile; ++j) {
    if (!(d > 0.0) && bad == kSpdTile) bad = j;
    const double inv = rsqrt(d);
    const double l = a[j] * inv;
    a[j] = lane == j ? inv : l;
    // the next pivot first: its lane has all it needs, and the rest of the column fills the wait
    if (j + 1 < kSpdTile) d = __shfl_sync(0xffffffffu, a[(j + 1) & 31] - l * l, j + 1);
#pragma unroll
    for (int c = j + 1; c < kSpdTile; ++c) a[c] -= l * __shfl_sync(0xffffffffu, l, c);
  }
#pragma unroll
  for (int c = 0; c < kSpdTile; ++c) t[lane][c] = a[c];
  return bad;
}

// t <- t L^-T by one warp, lane = row; LT: the factor's transpose
typedef double SpdFactorT[kSpdTile][kSpdTile + 2];
__device__ __forceinline__ void spd_panel(SpdTile& t, const SpdFactorT& LT, int lane) {
  double x[kSpdTile];
#pragma unroll
  for (int c = 0; c < kSpdTile; ++c) x[c] = t[lane][c];
#pragma unroll
  for (int m = 0; m < kSpdTile; ++m) {
    x[m] *= LT[m][m];
#pragma unroll
    for (int c = m & ~1; c < kSpdTile; c += 2) {
      const double2 l = *reinterpret_cast<const double2*>(&LT[m][c]);
      if (c > m) x[c] -= x[m] * l.x;
      if (c + 1 > m) x[c + 1] -= x[m] * l.y;
    }
  }
#pragma unroll
  for (int c = 0; c < kSpdTile; ++c) t[lane][c] = x[c];
}

static __global__ void __launch_bounds__(kSpdThreads) spd_kkt_kernel(SpdArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SpdTile Pi, Pj;
  __shared__ __align__(16) SpdFactorT LT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = a.n, nt = a.nt, ld = nt * kSpdTile;
  unsigned target = 0;
  auto meet = [&]() { return cg_barrier<kSyncBlock>(a.sh, target, kSpdThreads); };
  auto stop = [&]() {
    if (threadIdx.x == 0) atomicExch(a.info, -1);
  };
  auto at = [&](double* M, int i, int j) { return M + ((size_t)i * ld + j) * kSpdTile; };
  for (long long e = blockIdx.x * (long long)kSpdThreads + threadIdx.x; e < (long long)(ld + kSpdTile) * ld;
       e += (long long)gridDim.x * kSpdThreads) {
    const int r = (int)(e / ld), c = (int)(e - (long long)r * ld);
    double v = r == c ? 1.0 : 0.0;  // rows past n: the unit matrix
    if (c < n) {
      if (r < n)
        v = a.H[(size_t)r * n + c];
      else if (r == ld)
        v = -a.chi[c];
      else if (r == ld + 1 && a.C)
        v = a.C[c];
    }
    a.A[e] = v;
  }
  if (!meet()) return stop();
  // the block that finishes the next diagonal tile factorises it at once
  auto factor = [&](SpdTile& t, int k) {
    if (warp == 0) {
      const int bad = spd_factor(t, lane);
      if (lane == 0 && bad < kSpdTile) atomicExch(a.info, k * kSpdTile + bad + 1);
    }
    __syncthreads();
    spd_store(at(a.L, k, k), t, ld);
  };
  if (blockIdx.x == 0) {
    spd_put(Pi, spd_fetch(at(a.A, 0, 0), ld));
    __syncthreads();
    factor(Pi, 0);
  }
  if (!meet()) return stop();
  for (int k = 0; k < nt; ++k) {
    // a verdict on a later tile may be there already and is left for its own turn, so that all blocks leave together
    const int bad = *(volatile int*)a.info;
    if (bad && (bad - 1) / kSpdTile <= k) return;
    // trailing tiles by rows: row r of the np below the diagonal has r + 1, the right-hand sides' np - 1; the last
    // column has only its panel
    const int np = nt - k, tiles = np > 1 ? (np - 1) * (np + 2) / 2 : 1;
    double2 lk = make_double2(0.0, 0.0);
    if ((int)blockIdx.x < tiles) lk = spd_fetch(at(a.L, k, k), ld);
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      int r = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
      while (r * (r + 1) / 2 > t) --r;
      while ((r + 1) * (r + 2) / 2 <= t) ++r;
      const int c = t - r * (r + 1) / 2, i = k + 1 + r, j = k + 1 + c;
      const double2 pi = spd_fetch(at(a.A, i, k), ld);
      const double2 pj = i != j ? spd_fetch(at(a.A, j, k), ld) : pi;
      // half the threads, four values of the trailing tile each: rows r0, r0 + 16, columns c0, c0 + 16
      const bool upd = np > 1 && threadIdx.x < kSpdThreads / 2;
      const int r0 = (threadIdx.x >> 4) & 15, c0 = threadIdx.x & 15;
      double* D = at(a.A, i, j) + (size_t)r0 * ld + c0;
      const size_t half = (size_t)(kSpdTile / 2) * ld;
      double v[4] = {0.0, 0.0, 0.0, 0.0}, w[4] = {0.0, 0.0, 0.0, 0.0};
      if (upd) v[0] = D[0], v[1] = D[16], v[2] = D[half], v[3] = D[half + 16];
      if (t == (int)blockIdx.x) {
        LT[lane][warp] = lk.x;
        LT[lane][warp + kSpdTile / 2] = lk.y;
      }
      spd_put(Pi, pi);
      spd_put(Pj, pj);
      __syncthreads();
      if (warp == 0) spd_panel(Pi, LT, lane);
      if (warp == 1 && i != j) spd_panel(Pj, LT, lane);
      __syncthreads();
      if (c == 0) spd_store(at(a.L, i, k), Pi, ld);
      if (np > 1) {
        const SpdTile& Q = i == j ? Pi : Pj;
        if (upd) {
#pragma unroll 8
          for (int m = 0; m < kSpdTile; ++m) {
            const double p0 = Pi[r0][m], p1 = Pi[r0 + 16][m], q0 = Q[c0][m], q1 = Q[c0 + 16][m];
            w[0] += p0 * q0;
            w[1] += p0 * q1;
            w[2] += p1 * q0;
            w[3] += p1 * q1;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] -= w[e];
        }
        if (t == 0) {  // tile (k + 1, k + 1)
          if (upd) {
            Pj[r0][c0] = v[0], Pj[r0][c0 + 16] = v[1];
            Pj[r0 + 16][c0] = v[2], Pj[r0 + 16][c0 + 16] = v[3];
          }
          __syncthreads();
          factor(Pj, k + 1);
        } else if (upd) {
          D[0] = v[0], D[16] = v[1], D[half] = v[2], D[half + 16] = v[3];
        }
      }
      __syncthreads();
    }
    if (!meet()) return stop();
  }
  if (blockIdx.x != 0) return;
  // backward substitution: warp g sums rows g, g + 16, ... of the column, warps 0 and 1 solve the tile
  double* x = reinterpret_cast<double*>(smem_raw);  // [2][ld]
  __shared__ double part[kSpdThreads / 32][2][kSpdTile];
  for (int k = nt - 1; k >= 0; --k) {
    double s[2] = {0.0, 0.0};
    const double* col = a.L + (size_t)k * kSpdTile + lane;
    const double2 lk = spd_fetch(at(a.L, k, k), ld);
    double y = warp < 2 ? col[(size_t)(ld + warp) * ld] : 0.0;
#pragma unroll 8
    for (int r = (k + 1) * kSpdTile + warp; r < ld; r += kSpdThreads / 32) {
      const double l = col[(size_t)r * ld];
      s[0] += l * x[r];
      s[1] += l * x[ld + r];
    }
    part[warp][0][lane] = s[0];
    part[warp][1][lane] = s[1];
    spd_put(Pi, lk);
    __syncthreads();
    if (warp < 2) {
#pragma unroll
      for (int g = 0; g < kSpdThreads / 32; ++g) y -= part[g][warp][lane];
#pragma unroll
      for (int c = kSpdTile - 1; c >= 0; --c) {
        const double xc = __shfl_sync(0xffffffffu, y, c) * Pi[c][c];
        if (lane == c)
          y = xc;
        else if (lane < c)
          y -= Pi[c][lane] * xc;
      }
      x[warp * ld + k * kSpdTile + lane] = y;
    }
    __syncthreads();
  }
  // lam = (C x_0 - b) / (C x_1), q = x_0 - lam x_1
  double lam = 0.0;
  if (a.C) {
    __shared__ double red[2 * 32], sums[2];
    if (threadIdx.x < 2) sums[threadIdx.x] = 0.0;
    __syncthreads();
    double v[2] = {0.0, 0.0};
    for (int i = threadIdx.x; i < n; i += kSpdThreads) {
      v[0] += a.C[i] * x[i];
      v[1] += a.C[i] * x[ld + i];
    }
    block_atomic_sum<2>(v, sums, red);
    if (sums[1] == 0.0) {
      if (threadIdx.x == 0) *a.info = n + 1;
      return;
    }
    lam = (sums[0] - *a.b) / sums[1];
  }
  for (int i = threadIdx.x; i < n; i += kSpdThreads) a.q[i] = x[i] - lam * x[ld + i];
}

struct SpdWS {
  CgShared* sh;
  int* info;
  double *A, *L;
  size_t bytes;
};
static SpdWS spd_carve(void* ws, size_t bytes, int n) {
  const size_t nt = (n + kSpdTile - 1) / kSpdTile, elems = (nt + 1) * nt * kSpdTile * kSpdTile;
  Carver c(ws, bytes);
  SpdWS w;
  w.sh = c.take<CgShared>(1);
  w.info = c.take<int>(1);
  w.A = c.take<double>(elems);
  w.L = c.take<double>(elems);
  w.bytes = c.off;
  return w;
}

static int spd_kkt(int n, const double* H, const double* chi, const double* C, const double* b, double* q, int* info,
                   void* ws, size_t bytes, cudaStream_t st) {
  const SpdWS w = spd_carve(ws, bytes, n);
  if (!ws || w.bytes > bytes) return fail(ADMP_ERR_WORKSPACE, "dense solve: need %zu bytes, got %zu", w.bytes, bytes);
  int dev = 0, sms = 0, coop = 0, per_sm = 0;
  ADMP_CUDA_TRY(cudaGetDevice(&dev));
  ADMP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  ADMP_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  SpdArgs a{n, (n + kSpdTile - 1) / kSpdTile, H, chi, C, b, w.A, w.L, q, w.info, w.sh};
  const size_t smem = 2 * (size_t)a.nt * kSpdTile * sizeof(double);
  ADMP_CUDA_TRY(ensure_smem(spd_kkt_kernel, smem));
  ADMP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, spd_kkt_kernel, kSpdThreads, smem));
  if (!coop || per_sm < 1) return fail(ADMP_ERR_CUDA, "dense solve: no cooperative launch");
  const int tiles = (a.nt - 1) * (a.nt + 2) / 2, grid = tiles < 1 ? 1 : (tiles < sms ? tiles : sms);
  ADMP_CUDA_TRY(cudaMemsetAsync(w.sh, 0, sizeof(CgShared), st));
  ADMP_CUDA_TRY(cudaMemsetAsync(w.info, 0, sizeof(int), st));
  void* args[] = {&a};
  std::lock_guard<std::mutex> alone(grid_mutex(dev));
  ADMP_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)spd_kkt_kernel, dim3(grid), dim3(kSpdThreads), args, smem, st));
  count_launches(1);
  const void* p = read_back(w.info, sizeof(int), st);
  if (!p) return ADMP_ERR_CUDA;
  *info = *(const int*)p;
  return *info < 0 ? fail(ADMP_ERR_CUDA, "dense solve: a block waited too long for the others") : ADMP_OK;
}

}  // namespace admp

using namespace admp;

extern "C" size_t admp_qeq_dense_workspace_size(int natoms) {
  return natoms <= 0 || natoms > ADMP_QEQ_DENSE_MAX ? 0 : spd_carve(nullptr, 0, natoms).bytes;
}

extern "C" int admp_qeq_dense_solve(int natoms, const double* H, const double* chi, const double* constraint,
                                    const double* value, double* q, int* info, void* workspace,
                                    size_t workspace_bytes, void* stream) {
  if (natoms <= 0 || natoms > ADMP_QEQ_DENSE_MAX || !H || !chi || !q || !info || (constraint && !value))
    return fail(ADMP_ERR_BAD_ARG, "admp_qeq_dense_solve: args");
  return spd_kkt(natoms, H, chi, constraint, value, q, info, workspace, workspace_bytes, (cudaStream_t)stream);
}
