// The CG iterations of one system as one persistent launch.
//
// A solve of a few thousand atoms is bound by launches and by the latency of
// its kernels, not by work: one iteration of 3,000 atoms on a 48^3 mesh took
// thirteen launches of 10-50 blocks, 105 us, of which the arithmetic is under
// 10.  Here one block per SM stays for the whole solve; the phases of an
// iteration are separated by a barrier over the grid, every transform spreads
// its lines over all blocks, the twiddles and (while they fit) the atoms'
// stencils are built once per launch, and the host reads the result once.
// Now 36 us (3,000 atoms, 48^3, FP32), 52 (10,701, 64^3, FP64; 110 before) and
// 50 (2,304 electrode atoms, 64 x 64 x 160, FP32; 100 before): a barrier takes
// 1.8 of them, there are six (eight in the last case).
//
//   A   direction p = r + beta p of the group's atoms, spread
//   Z   z transform of the mesh lines,  Y  y transform
//   X   x transform, Green's function, inverse x transform
//   Y'  inverse y,  Z' inverse z
//       (Z with Y and Y' with Z' in one block's shared memory while the planes are small)
//       (a quarter of the warps multiply p by the pair matrix meanwhile)
//   E   gather, rest of the matvec, p.Hp and C.Hp
//   F   x += alpha p, r -= alpha P(Hp), |r|^2; zero Hp and the mesh
//
// Iteration -1 takes the initial charges in the direction's place and leaves
// r = -P(chi + H x) and p = r: a pass of these phases instead of seventeen
// launches (a solve of 3,000 atoms 1,660 -> 1,563 us, of 10,701 4,119 -> 4,013).
//
// Arithmetic, scalars and stopping rule are those of the kernels in
// qeq_kernels.cuh.  The scalars of iteration k live in slot k % 3, so that a
// slot is zeroed (phase F of the iteration before) two barriers after its last
// reader.  All blocks are resident (cooperative launch); a block that waits
// for the others longer than kCgSpin polls sets the status and leaves, as then
// do the others.
#pragma once

#include "qeq_kernels.cuh"

namespace admp {

constexpr int kCgThreads = 512;
constexpr int kCgWarps = kCgThreads / 32;  // cg_block_sum counts on 16
constexpr int kCgFft = 384;                // threads of the transforms; the others multiply by the pair matrix
constexpr long long kCgSpin = 1LL << 23;
constexpr int kCgMaxLines = kCgFft;      // lines of a block's y transform
constexpr int kCgLaunch = 128;           // iterations per launch
// Complex values of the largest x plane that one block transforms in z and y by itself: two barriers and a trip of
// the spectrum through L2 less in each direction, for fewer blocks at work.  19 iterations of 48^3 (FP32) 776 -> 690
// us, 58 of 64^3 (FP64) 3,090 -> 2,895; with 64 x 160 values a plane both ways take the same (1,732 and 1,738).
constexpr int kCgPlane = 4096;

struct CgSlot {
  double rr_new, pHp, Cv[kMaxConst], sp, spz, spz2;
};

// In global memory beside the vectors; zeroed before the first launch of a
// solve (the barrier counter before every launch).
struct CgShared {
  CgSlot slot[3];
  unsigned arrived;
};

template <typename T>
struct CgArgs {
  int N, K0, K1, K2;
  double kappa;
  QEqParams P;
  const T *pos, *box, *C, *green;
  const double *diag, *zc, *chi;
  T *mesh, *p, *Hp;
  Cplx<T>* spec;
  double *x, *r;
  PairList<T> list;
  int have_pairs;
  CGScal* sc;
  CgShared* sh;
  int k0, k1;        // iterations of this launch: k0 <= k < k1
  int init;          // iteration -1 first: r = -P(chi + H x), p = r
  int lz, ly, lx;    // lines (z: pairs of lines) a block transforms at a time
  int planes;        // a block transforms whole x planes in z and y
  int buf;           // complex values in each of the two line buffers
  int group;         // atoms of a warp's group (at most kPw)
  int kept;          // stencil groups a warp keeps, 0: built anew every time
};

// Barrier over the grid; false when it ran out of polls.  Called by the whole
// block, or (kSyncPart) by its first nthr threads.
template <int SYNC>
__device__ __forceinline__ bool cg_barrier(CgShared* sh, unsigned& target, int nthr) {
  __shared__ int ok;
  target += gridDim.x;
  group_sync<SYNC>(nthr);
  if (threadIdx.x == 0) {
    unsigned seen;
    __threadfence();
    atomicAdd(&sh->arrived, 1u);
    long long polls = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&sh->arrived) : "memory");
    } while (seen < target && ++polls < kCgSpin);
    ok = seen >= target;
    __threadfence();
  }
  group_sync<SYNC>(nthr);
  return ok != 0;
}

// Sums of NV <= 4 values over the block, added to out[0 .. NV): the warp sums
// are taken together and one warp adds the 16 warps' results.
template <int NV>
__device__ __forceinline__ void cg_block_sum(const double (&in)[NV], double* out, double (*sh)[kCgWarps]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = in[k];
  if (NV == 1) {
    v[0] = warp_sum(v[0]);
    if (lane == 0) sh[0][warp] = v[0];
  } else {
    const double s = warp_sum_each<4>(v, lane);  // lane l: value l / 8
    if ((lane & 7) == 0) sh[lane >> 3][warp] = s;
  }
  __syncthreads();
  if (warp == 0) {
    const int q = lane >> 3, w = lane & 7;
    double s = q < NV ? sh[q][w] + sh[q][w + 8] : 0.0;
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (w == 0 && q < NV && s != 0.0) atomicAdd(out + q, s);
  }
}

template <typename T>
struct CgFft {
  Cplx<T> *W0, *W1, *W2, *A, *B;
};

// forward (mesh -> half spectrum) or inverse z pass of this block's line pairs
template <typename T, bool INV>
__device__ void cg_z_pass(const CgArgs<T>& a, const CgFft<T>& f, const Radices& R) {
  const int K2 = a.K2, K2h = K2 / 2 + 1, L = a.K0 * a.K1, npair = (L + 1) / 2;
  const FastDiv fdK2 = fast_div(K2), fdK2h = fast_div(K2h);
  for (int p0 = blockIdx.x * a.lz; p0 < npair; p0 += gridDim.x * a.lz) {
    const int np = min(a.lz, npair - p0);
    for (int idx = threadIdx.x; idx < np * K2; idx += kCgFft) {
      const int p = fdiv(idx, fdK2), t = idx - p * K2;
      const size_t l0 = 2 * (size_t)(p0 + p);
      const bool two = l0 + 1 < (size_t)L;
      Cplx<T> z;
      if (!INV) {
        z.x = a.mesh[l0 * K2 + t];
        z.y = two ? a.mesh[(l0 + 1) * K2 + t] : T(0);
      } else {
        const bool lo = t < K2h;
        const int tt = lo ? t : K2 - t;
        Cplx<T> u = a.spec[l0 * K2h + tt], v;
        v.x = v.y = T(0);
        if (two) v = a.spec[(l0 + 1) * K2h + tt];
        if (!lo) {
          u.y = -u.y;
          v.y = -v.y;
        }
        z.x = u.x - v.y;
        z.y = u.y + v.x;
      }
      f.A[idx] = z;
    }
    group_sync<kSyncPart>(kCgFft);
    Cplx<T>* R2 = fft_run<T, false, kSyncPart, INV>(R, f.A, f.B, np, K2, K2, 1, f.W2, threadIdx.x, kCgFft);
    if (!INV) {
      for (int idx = threadIdx.x; idx < np * K2h; idx += kCgFft) {
        const int p = fdiv(idx, fdK2h), k = idx - p * K2h;
        const Cplx<T> Z = R2[p * K2 + k], Zm = R2[p * K2 + (k == 0 ? 0 : K2 - k)];
        const size_t l0 = 2 * (size_t)(p0 + p);
        Cplx<T> u, v;
        u.x = (Z.x + Zm.x) * T(0.5);
        u.y = (Z.y - Zm.y) * T(0.5);
        v.x = (Z.y + Zm.y) * T(0.5);
        v.y = (Zm.x - Z.x) * T(0.5);
        a.spec[l0 * K2h + k] = u;
        if (l0 + 1 < (size_t)L) a.spec[(l0 + 1) * K2h + k] = v;
      }
    } else {
      for (int idx = threadIdx.x; idx < np * K2; idx += kCgFft) {
        const int p = fdiv(idx, fdK2), t = idx - p * K2;
        const size_t l0 = 2 * (size_t)(p0 + p);
        const Cplx<T> z = R2[idx];
        a.mesh[l0 * K2 + t] = z.x;
        if (l0 + 1 < (size_t)L) a.mesh[(l0 + 1) * K2 + t] = z.y;
      }
    }
    group_sync<kSyncPart>(kCgFft);
  }
}

// y pass in place: line c = x K2h + kz, element y at (x K1 + y) K2h + kz
template <typename T, bool INV>
__device__ void cg_y_pass(const CgArgs<T>& a, const CgFft<T>& f, const Radices& R) {
  __shared__ long long off[kCgMaxLines];
  const int K1 = a.K1, K2h = a.K2 / 2 + 1, L = a.K0 * K2h;
  for (int c0 = blockIdx.x * a.ly; c0 < L; c0 += gridDim.x * a.ly) {
    const int n = min(a.ly, L - c0);
    const FastDiv fdn = fast_div(n);
    if (threadIdx.x < n) {
      const int c = c0 + threadIdx.x, xx = c / K2h;
      off[threadIdx.x] = (long long)xx * K1 * K2h + (c - xx * K2h);
    }
    group_sync<kSyncPart>(kCgFft);
    for (int idx = threadIdx.x; idx < K1 * n; idx += kCgFft) {
      const int y = fdiv(idx, fdn), c = idx - y * n;
      f.A[idx] = a.spec[off[c] + (long long)y * K2h];
    }
    group_sync<kSyncPart>(kCgFft);
    Cplx<T>* R1 = fft_run<T, true, kSyncPart, INV>(R, f.A, f.B, n, K1, 1, n, f.W1, threadIdx.x, kCgFft);
    for (int idx = threadIdx.x; idx < K1 * n; idx += kCgFft) {
      const int y = fdiv(idx, fdn), c = idx - y * n;
      a.spec[off[c] + (long long)y * K2h] = R1[idx];
    }
    group_sync<kSyncPart>(kCgFft);
  }
}

// z and y passes of whole x planes: the half spectrum of a plane goes from the one to the other in shared memory.
template <typename T>
__device__ void cg_plane_fwd(const CgArgs<T>& a, const CgFft<T>& f, const Radices& R1, const Radices& R2) {
  const int K1 = a.K1, K2 = a.K2, K2h = K2 / 2 + 1, np = (K1 + 1) / 2;
  const FastDiv fdK2 = fast_div(K2), fdK2h = fast_div(K2h);
  for (int x = blockIdx.x; x < a.K0; x += gridDim.x) {
    const T* Q = a.mesh + (size_t)x * K1 * K2;
    for (int idx = threadIdx.x; idx < np * K2; idx += kCgFft) {
      const int p = fdiv(idx, fdK2), t = idx - p * K2;
      Cplx<T> z;
      z.x = Q[2 * p * K2 + t];
      z.y = 2 * p + 1 < K1 ? Q[(2 * p + 1) * K2 + t] : T(0);
      f.A[idx] = z;
    }
    group_sync<kSyncPart>(kCgFft);
    Cplx<T>* Z = fft_run<T, false, kSyncPart, false>(R2, f.A, f.B, np, K2, K2, 1, f.W2, threadIdx.x, kCgFft);
    Cplx<T>* U = Z == f.A ? f.B : f.A;
    for (int idx = threadIdx.x; idx < np * K2h; idx += kCgFft) {
      const int p = fdiv(idx, fdK2h), k = idx - p * K2h;
      const Cplx<T> z = Z[p * K2 + k], zm = Z[p * K2 + (k == 0 ? 0 : K2 - k)];
      Cplx<T> u, v;
      u.x = (z.x + zm.x) * T(0.5);
      u.y = (z.y - zm.y) * T(0.5);
      v.x = (z.y + zm.y) * T(0.5);
      v.y = (zm.x - z.x) * T(0.5);
      U[2 * p * K2h + k] = u;
      if (2 * p + 1 < K1) U[(2 * p + 1) * K2h + k] = v;
    }
    group_sync<kSyncPart>(kCgFft);
    const Cplx<T>* V = fft_run<T, true, kSyncPart, false>(R1, U, Z, K2h, K1, 1, K2h, f.W1, threadIdx.x, kCgFft);
    Cplx<T>* H = a.spec + (size_t)x * K1 * K2h;
    for (int idx = threadIdx.x; idx < K1 * K2h; idx += kCgFft) H[idx] = V[idx];
    group_sync<kSyncPart>(kCgFft);
  }
}

template <typename T>
__device__ void cg_plane_inv(const CgArgs<T>& a, const CgFft<T>& f, const Radices& R1, const Radices& R2) {
  const int K1 = a.K1, K2 = a.K2, K2h = K2 / 2 + 1, np = (K1 + 1) / 2;
  const FastDiv fdK2 = fast_div(K2);
  for (int x = blockIdx.x; x < a.K0; x += gridDim.x) {
    const Cplx<T>* H = a.spec + (size_t)x * K1 * K2h;
    for (int idx = threadIdx.x; idx < K1 * K2h; idx += kCgFft) f.A[idx] = H[idx];
    group_sync<kSyncPart>(kCgFft);
    Cplx<T>* V = fft_run<T, true, kSyncPart, true>(R1, f.A, f.B, K2h, K1, 1, K2h, f.W1, threadIdx.x, kCgFft);
    Cplx<T>* Z = V == f.A ? f.B : f.A;
    for (int idx = threadIdx.x; idx < np * K2; idx += kCgFft) {
      const int p = fdiv(idx, fdK2), t = idx - p * K2;
      const bool lo = t < K2h;
      const int tt = lo ? t : K2 - t;
      Cplx<T> u = V[2 * p * K2h + tt], v;
      v.x = v.y = T(0);
      if (2 * p + 1 < K1) v = V[(2 * p + 1) * K2h + tt];
      if (!lo) {
        u.y = -u.y;
        v.y = -v.y;
      }
      Cplx<T> z;
      z.x = u.x - v.y;
      z.y = u.y + v.x;
      Z[idx] = z;
    }
    group_sync<kSyncPart>(kCgFft);
    const Cplx<T>* R = fft_run<T, false, kSyncPart, true>(R2, Z, V, np, K2, K2, 1, f.W2, threadIdx.x, kCgFft);
    T* Q = a.mesh + (size_t)x * K1 * K2;
    for (int idx = threadIdx.x; idx < np * K2; idx += kCgFft) {
      const int p = fdiv(idx, fdK2), t = idx - p * K2;
      const Cplx<T> z = R[idx];
      Q[2 * p * K2 + t] = z.x;
      if (2 * p + 1 < K1) Q[(2 * p + 1) * K2 + t] = z.y;
    }
    group_sync<kSyncPart>(kCgFft);
  }
}

// x pass: transform, cached 2 G_s, inverse transform
template <typename T>
__device__ void cg_x_pass(const CgArgs<T>& a, const CgFft<T>& f, const Radices& R) {
  const int K0 = a.K0, L = a.K1 * (a.K2 / 2 + 1);
  for (int c0 = blockIdx.x * a.lx; c0 < L; c0 += gridDim.x * a.lx) {
    const int n = min(a.lx, L - c0);
    const FastDiv fdn = fast_div(n);
    for (int idx = threadIdx.x; idx < K0 * n; idx += kCgFft) {
      const int x = fdiv(idx, fdn), c = c0 + idx - x * n;
      f.A[idx] = a.spec[(size_t)x * L + c];
    }
    group_sync<kSyncPart>(kCgFft);
    Cplx<T>* F = fft_run<T, true, kSyncPart, false>(R, f.A, f.B, n, K0, 1, n, f.W0, threadIdx.x, kCgFft);
    Cplx<T>* O = F == f.A ? f.B : f.A;
    for (int idx = threadIdx.x; idx < K0 * n; idx += kCgFft) {
      const int x = fdiv(idx, fdn), c = c0 + idx - x * n;
      const T g = a.green[(size_t)x * L + c];
      F[idx].x *= g;
      F[idx].y *= g;
    }
    group_sync<kSyncPart>(kCgFft);
    Cplx<T>* I = fft_run<T, true, kSyncPart, true>(R, F, O, n, K0, 1, n, f.W0, threadIdx.x, kCgFft);
    for (int idx = threadIdx.x; idx < K0 * n; idx += kCgFft) {
      const int x = fdiv(idx, fdn), c = c0 + idx - x * n;
      a.spec[(size_t)x * L + c] = I[idx];
    }
    group_sync<kSyncPart>(kCgFft);
  }
}

// Hp += real-space matrix times p by the block's threads t0, t0 + 1, ...: four
// entries a thread in flight, the first atom's share summed over its run.
template <typename T>
__device__ void cg_pairs(const CgArgs<T>& a, int t0, int nthr) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  const long long n = (long long)*a.list.n, step = (long long)gridDim.x * nthr;
  for (long long p0 = blockIdx.x * (long long)nthr + ((threadIdx.x - t0) & ~31); p0 < n; p0 += U * step) {
    int2 ij[U];
    T c[U], vi[U], vj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long p = p0 + u * step + lane;
      ij[u] = p < n ? a.list.ij[p] : make_int2(-1, -1);
      c[u] = p < n ? a.list.coef[p] : T(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool on = c[u] != T(0);
      vi[u] = on ? a.p[ij[u].x] : T(0);
      vj[u] = on ? a.p[ij[u].y] : T(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const WarpRuns runs(ij[u].x, lane);
      const T w = runs.sum(c[u] != T(0) ? c[u] * vj[u] : T(0));
      if (runs.opens && w != T(0)) atomicAdd(a.Hp + ij[u].x, w);
      if (c[u] != T(0)) atomicAdd(a.Hp + ij[u].y, c[u] * vi[u]);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kCgThreads) qeq_cg_kernel(CgArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ Geom g;
  __shared__ Radices R0, R1, R2;
  __shared__ double red[4][kCgWarps], red2[4][kCgWarps];
  __shared__ double Ginv[kMaxConst * kMaxConst];
  __shared__ int broken;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool kspace = (a.P.flags & ADMP_QEQ_KSPACE) != 0, slab = (a.P.flags & ADMP_QEQ_SLAB) != 0;
  CgFft<T> f;
  f.W0 = reinterpret_cast<Cplx<T>*>(smem_raw);
  f.W1 = f.W0 + a.K0;
  f.W2 = f.W1 + a.K1;
  f.A = f.W2 + a.K2;
  f.B = f.A + a.buf;
  unsigned char* st_base = reinterpret_cast<unsigned char*>(f.B + a.buf);
  constexpr size_t kStBytes = (WarpStencil<T, false>::bytes() + 15) / 16 * 16;
  const int nkeep = a.kept > 0 ? a.kept : 1;
  SysDesc d;
  d.atom_off = 0;
  d.natoms = a.N;
  d.K0 = a.K0;
  d.K1 = a.K1;
  d.K2 = a.K2;
  load_geom(a.box, 0, &g);
  if (threadIdx.x == 0) broken = 0;
  if (threadIdx.x < kMaxConst * kMaxConst) Ginv[threadIdx.x] = a.sc->Ginv[threadIdx.x];
  if (kspace) {
    make_twiddles(f.W0, a.K0);
    make_twiddles(f.W1, a.K1);
    make_twiddles(f.W2, a.K2);
    if (threadIdx.x == 32) factor_radices(a.K0, R0);
    if (threadIdx.x == 64) factor_radices(a.K1, R1);
    if (threadIdx.x == 96) factor_radices(a.K2, R2);
  }
  __syncthreads();
  // warp w of block b takes the groups of a.group atoms w G + b, + G kCgWarps, ...
  const int ng = (a.N + a.group - 1) / a.group, g0 = warp * gridDim.x + blockIdx.x, gstep = gridDim.x * kCgWarps;
  auto atoms = [&](int gi) { return min(a.group, a.N - gi * a.group); };
  auto stencil = [&](int u) {
    WarpStencil<T, false> ws;
    ws.carve(st_base + (size_t)(warp * nkeep + (a.kept ? u : 0)) * kStBytes);
    return ws;
  };
  auto build = [&](WarpStencil<T, false>& ws, int gi) {
    warp_build_stencil<T, false>(ws, d, g, a.pos, nullptr, nullptr, gi * a.group, gi * a.group + atoms(gi), lane);
  };
  if (kspace && a.kept) {
    int u = 0;
    for (int gi = g0; gi < ng; gi += gstep, ++u) {
      WarpStencil<T, false> ws = stencil(u);
      build(ws, gi);
    }
  }
  CGScal* sc = a.sc;
  if (sc->done) return;  // the same for every block: only phase A writes it, behind the first barrier
  double rr0 = sc->rr;
  const double nn = sc->nn, pre = sc->pre, Lz2 = sc->Lz2;
  const double few = a.P.tol > 0.0 ? a.P.tol * (double)a.N : 0.0, few2 = few * few;
  const int nc = sc->n_const;
  unsigned target = 0;
  auto stop = [&]() {
    if (threadIdx.x == 0) atomicExch(&sc->status, ADMP_ERR_CUDA);
  };
  auto meet = [&]() { return cg_barrier<kSyncBlock>(a.sh, target, kCgThreads); };
  for (int k = a.init ? -1 : a.k0;; ++k) {
    const bool init = k < 0;  // the matvec of the initial charges in the direction's place
    CgSlot& S = a.sh->slot[(k + 3) % 3];
    volatile CgSlot& S1 = a.sh->slot[(k + 2) % 3];  // iteration k - 1
    volatile CgSlot& S2 = a.sh->slot[(k + 4) % 3];  // iteration k - 2
    // ---- A: convergence of the last iterate, direction, spread (the first group's values are asked for before
    // the scalars are worked out)
    double rv = 0.0, zv = 0.0;
    T pv = T(0);
    if (g0 < ng && lane < atoms(g0)) {
      const int i = g0 * a.group + lane;
      rv = a.r[i];
      pv = a.p[i];
      zv = a.zc[i];
    }
    const double rr = k == 0 ? rr0 : S1.rr_new, rp = k == 0 ? 0.0 : (k == 1 ? rr0 : S2.rr_new);
    if (k > 0) {
      // sqrt(rr) / N < tol; the square root and the division only where rounding could decide
      bool conv = rr < few2 * (1.0 - 1e-9);
      if (!conv && rr <= few2 * (1.0 + 1e-9)) conv = sqrt(rr) / (double)a.N < a.P.tol;
      if (conv || k >= a.P.max_iter) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
          sc->rr_new = rr;
          sc->iter = k;
          sc->status = conv ? ADMP_OK : ADMP_ERR_NOT_CONVERGED;
          sc->done = 1;
        }
        return;
      }
    }
    if (k >= a.k1) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->rr_new = rr;
        sc->iter = k;
      }
      return;
    }
    {
      const double beta = rp != 0.0 ? rr / rp : 0.0;
      double acc[3] = {0, 0, 0};
      int u = 0;
      for (int gi = g0; gi < ng; gi += gstep, ++u) {
        WarpStencil<T, false> ws = stencil(u);
        const int na = atoms(gi);
        if (kspace && !a.kept) build(ws, gi);
        if (lane < na) {
          const int i = gi * a.group + lane;
          if (u > 0) {
            rv = a.r[i];
            pv = a.p[i];
            zv = a.zc[i];
          }
          double pn = rv;  // the first direction is the residual
          if (k != 0) {
            pn = init ? a.x[i] : rv + beta * (double)pv;
            pv = (T)pn;
            a.p[i] = pv;
          }
          if (kspace) ws.q[lane] = pv;
          acc[0] += pn;
          acc[1] += pn * zv;
          acc[2] += pn * zv * zv;
        }
        __syncwarp();
        if (kspace) spread_group<T>(ws, na, a.K1, a.K2, a.mesh, lane);
        __syncwarp();
      }
      cg_block_sum<3>(acc, &S.sp, red);
    }
    if (!meet()) return stop();
    // ---- Z .. Z': the mesh part by the first kCgFft threads; the pairs, which need only p and Hp, by the others
    if (threadIdx.x < kCgFft) {
      if (kspace) {
        unsigned t = target;
        bool ok = true;
        auto pass = [&]() { return cg_barrier<kSyncPart>(a.sh, t, kCgFft); };
        if (a.planes) {
          cg_plane_fwd<T>(a, f, R1, R2);
          if ((ok = pass())) cg_x_pass<T>(a, f, R0);
          if (ok && (ok = pass())) cg_plane_inv<T>(a, f, R1, R2);
        } else {
          cg_z_pass<T, false>(a, f, R2);
          if ((ok = pass())) cg_y_pass<T, false>(a, f, R1);
          if (ok && (ok = pass())) cg_x_pass<T>(a, f, R0);
          if (ok && (ok = pass())) cg_y_pass<T, true>(a, f, R1);
          if (ok && (ok = pass())) cg_z_pass<T, true>(a, f, R2);
        }
        if (!ok && threadIdx.x == 0) broken = 1;
      }
    } else if (a.have_pairs) {
      cg_pairs<T>(a, kCgFft, kCgThreads - kCgFft);
    }
    if (kspace) target += (a.planes ? 2 : 4) * gridDim.x;
    __syncthreads();
    if (broken) return stop();
    if (!meet()) return stop();
    // ---- E: potential, diagonal and rank-one terms, p.Hp and C.Hp
    {
      volatile CgSlot& V = S;
      const double sp = V.sp, spz = V.spz, spz2 = V.spz2;
      double acc[5] = {0, 0, 0, 0, 0};
      int u = 0;
      for (int gi = g0; gi < ng; gi += gstep, ++u) {
        const int na = atoms(gi), i = gi * a.group + (lane >> 2);
        const bool mine = (lane & 3) == 0 && (lane >> 2) < na;
        const double x = mine ? (double)a.p[i] : 0.0, dg = mine ? a.diag[i] : 0.0;
        const T hp = mine ? a.Hp[i] : T(0);
        T pot = T(0);
        if (kspace) {
          WarpStencil<T, false> ws = stencil(u);
          if (!a.kept) build(ws, gi);
          pot = gather_group<T, false>(ws, na, a.K1, a.K2, a.mesh, lane);
          __syncwarp();
        }
        if (mine) {
          double h = (double)(T)(hp + pot) + dg * x + nn * sp;
          if (slab) {
            const double z = a.zc[i];
            h += pre * (2.0 * z * spz - spz2 - z * z * sp - Lz2 / 6.0 * sp);
          }
          if (init)
            a.r[i] = h += a.chi[i];
          else
            a.Hp[i] = (T)h;
          acc[0] += x * h;
#pragma unroll
          for (int c = 0; c < kMaxConst; ++c)
            if (c < nc) acc[1 + c] += cval(a.C, c, (long long)a.N, i) * h;
        }
      }
      // p.Hp and the first three of C.Hp are next to each other in the slot
      const double a4[4] = {acc[0], acc[1], acc[2], acc[3]};
      cg_block_sum<4>(a4, &S.pHp, red2);
      if (nc == kMaxConst) {
        __syncthreads();
        const double a1[1] = {acc[4]};
        cg_block_sum<1>(a1, &S.Cv[kMaxConst - 1], red);
      }
    }
    if (!meet()) return stop();
    // ---- F: iterate and residual; zero what the next iteration accumulates into
    {
      const int tid = blockIdx.x * kCgThreads + threadIdx.x, nthr = gridDim.x * kCgThreads;
      T hv = T(0), pw = T(0);
      double xv = 0.0, rw = 0.0;
      if (tid < a.N) {
        hv = a.Hp[tid];
        pw = a.p[tid];
        xv = a.x[tid];
        rw = a.r[tid];
      }
      volatile CgSlot& V = S;
      const double pHp = V.pHp, alpha = pHp != 0.0 ? rr / pHp : 0.0;
      double lam[kMaxConst];
#pragma unroll
      for (int c = 0; c < kMaxConst; ++c) lam[c] = c < nc ? V.Cv[c] : 0.0;
      {
        double t[kMaxConst];
#pragma unroll
        for (int r0 = 0; r0 < kMaxConst; ++r0) {
          t[r0] = 0.0;
#pragma unroll
          for (int c = 0; c < kMaxConst; ++c)
            if (r0 < nc && c < nc) t[r0] += Ginv[r0 * kMaxConst + c] * lam[c];
        }
#pragma unroll
        for (int c = 0; c < kMaxConst; ++c) lam[c] = t[c];
      }
      double acc[1] = {0.0};
      for (int i = tid; i < a.N; i += nthr) {
        if (i != tid) {
          hv = a.Hp[i];
          pw = a.p[i];
          xv = a.x[i];
          rw = a.r[i];
        }
        double w = init ? rw : (double)hv;
        a.Hp[i] = T(0);
#pragma unroll
        for (int c = 0; c < kMaxConst; ++c)
          if (c < nc) w -= cval(a.C, c, (long long)a.N, i) * lam[c];
        const double rn = init ? -w : rw - alpha * w;
        if (init)
          a.p[i] = (T)rn;
        else
          a.x[i] = xv + alpha * (double)pw;
        a.r[i] = rn;
        acc[0] += rn * rn;
      }
      if (kspace) {
        const size_t M = (size_t)a.K0 * a.K1 * a.K2;
        for (size_t i = tid; i < M; i += nthr) a.mesh[i] = T(0);
      }
      if (blockIdx.x == 0 && threadIdx.x == 0) a.sh->slot[(k + 1) % 3] = CgSlot{};
      cg_block_sum<1>(acc, &S.rr_new, red);
    }
    if (!meet()) return stop();
    if (init) {
      volatile CgSlot& V = S;
      rr0 = V.rr_new;
      const bool conv = sqrt(rr0) / (double)a.N < a.P.tol, stay = !conv && a.P.max_iter > 0;
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->rr = sc->rr_new = rr0;
        if (!stay) {
          sc->status = conv ? ADMP_OK : ADMP_ERR_NOT_CONVERGED;
          sc->done = 1;
        }
      }
      if (!stay) return;
    }
  }
}

}  // namespace admp
