// The CG iterations of one system as one persistent launch.
//
// A solve of a few thousand atoms is bound by launches and by the latency of
// its kernels, not by work: one iteration of 3,000 atoms on a 48^3 mesh took
// thirteen launches of 10-50 blocks, 105 us, of which the arithmetic is under
// 10.  Here one block per SM stays for the whole solve; the phases of an
// iteration are separated by a barrier over the grid, every transform spreads
// its lines over all blocks, the twiddles and (while they fit) the atoms'
// stencils are built once per launch, and the host reads the result once.
//
//   A   direction p = r + beta p of the group's atoms, spread
//   Z   z transform of the mesh lines; real-space matrix times p
//   Y   y transform
//   X   x transform, Green's function, inverse x transform
//   Y'  inverse y,  Z' inverse z
//   E   gather, rest of the matvec, p.Hp and C.Hp
//   F   x += alpha p, r -= alpha P(Hp), |r|^2; zero Hp and the mesh
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

constexpr int kCgThreads = 256;
constexpr int kCgWarps = kCgThreads / 32;
constexpr long long kCgSpin = 1LL << 23;
constexpr int kCgMaxLines = kCgThreads;  // lines of a block's y transform
constexpr int kCgLaunch = 128;           // iterations per launch

struct CgSlot {
  double rr_new, pHp, Cv[kMaxConst], sp, spz, spz2;
};

// In global memory beside the vectors; zeroed before the first launch of a
// solve (the barrier counter before every launch).
struct CgShared {
  CgSlot slot[3];
  unsigned arrived;
  int failed;
};

template <typename T>
struct CgArgs {
  int N, K0, K1, K2;
  double kappa;
  QEqParams P;
  const T *pos, *box, *C, *green;
  const double *diag, *zc;
  T *mesh, *p, *Hp;
  Cplx<T>* spec;
  double *x, *r;
  PairList<T> list;
  int have_pairs;
  CGScal* sc;
  CgShared* sh;
  int k0, k1;        // iterations of this launch: k0 <= k < k1
  int lz, ly, lx;    // lines (z: pairs of lines) a block transforms at a time
  int buf;           // complex values in each of the two line buffers
  int kept;          // stencil groups a warp keeps, 0: built anew every time
};

// Barrier over the grid; false when it ran out of polls.
__device__ __forceinline__ bool cg_barrier(CgShared* sh, unsigned& target) {
  __shared__ int ok;
  target += gridDim.x;
  __syncthreads();
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
  __syncthreads();
  return ok != 0;
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
    for (int idx = threadIdx.x; idx < np * K2; idx += kCgThreads) {
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
    __syncthreads();
    Cplx<T>* R2 = fft_run<T, false, false, INV>(R, f.A, f.B, np, K2, K2, 1, f.W2, threadIdx.x, kCgThreads);
    if (!INV) {
      for (int idx = threadIdx.x; idx < np * K2h; idx += kCgThreads) {
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
      for (int idx = threadIdx.x; idx < np * K2; idx += kCgThreads) {
        const int p = fdiv(idx, fdK2), t = idx - p * K2;
        const size_t l0 = 2 * (size_t)(p0 + p);
        const Cplx<T> z = R2[idx];
        a.mesh[l0 * K2 + t] = z.x;
        if (l0 + 1 < (size_t)L) a.mesh[(l0 + 1) * K2 + t] = z.y;
      }
    }
    __syncthreads();
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
    __syncthreads();
    for (int idx = threadIdx.x; idx < K1 * n; idx += kCgThreads) {
      const int y = fdiv(idx, fdn), c = idx - y * n;
      f.A[idx] = a.spec[off[c] + (long long)y * K2h];
    }
    __syncthreads();
    Cplx<T>* R1 = fft_run<T, true, false, INV>(R, f.A, f.B, n, K1, 1, n, f.W1, threadIdx.x, kCgThreads);
    for (int idx = threadIdx.x; idx < K1 * n; idx += kCgThreads) {
      const int y = fdiv(idx, fdn), c = idx - y * n;
      a.spec[off[c] + (long long)y * K2h] = R1[idx];
    }
    __syncthreads();
  }
}

// x pass: transform, cached 2 G_s, inverse transform
template <typename T>
__device__ void cg_x_pass(const CgArgs<T>& a, const CgFft<T>& f, const Radices& R) {
  const int K0 = a.K0, L = a.K1 * (a.K2 / 2 + 1);
  for (int c0 = blockIdx.x * a.lx; c0 < L; c0 += gridDim.x * a.lx) {
    const int n = min(a.lx, L - c0);
    const FastDiv fdn = fast_div(n);
    for (int idx = threadIdx.x; idx < K0 * n; idx += kCgThreads) {
      const int x = fdiv(idx, fdn), c = c0 + idx - x * n;
      f.A[idx] = a.spec[(size_t)x * L + c];
    }
    __syncthreads();
    Cplx<T>* F = fft_run<T, true, false, false>(R, f.A, f.B, n, K0, 1, n, f.W0, threadIdx.x, kCgThreads);
    Cplx<T>* O = F == f.A ? f.B : f.A;
    for (int idx = threadIdx.x; idx < K0 * n; idx += kCgThreads) {
      const int x = fdiv(idx, fdn), c = c0 + idx - x * n;
      const T g = a.green[(size_t)x * L + c];
      F[idx].x *= g;
      F[idx].y *= g;
    }
    __syncthreads();
    Cplx<T>* I = fft_run<T, true, false, true>(R, F, O, n, K0, 1, n, f.W0, threadIdx.x, kCgThreads);
    for (int idx = threadIdx.x; idx < K0 * n; idx += kCgThreads) {
      const int x = fdiv(idx, fdn), c = c0 + idx - x * n;
      a.spec[(size_t)x * L + c] = I[idx];
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(kCgThreads) qeq_cg_kernel(CgArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ Geom g;
  __shared__ Radices R0, R1, R2;
  __shared__ double red[5 * 32];
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
  if (kspace) {
    make_twiddles(f.W0, a.K0);
    make_twiddles(f.W1, a.K1);
    make_twiddles(f.W2, a.K2);
    if (threadIdx.x == 32) factor_radices(a.K0, R0);
    if (threadIdx.x == 64) factor_radices(a.K1, R1);
    if (threadIdx.x == 96) factor_radices(a.K2, R2);
  }
  __syncthreads();
  // warp w of block b takes the groups of eight atoms w G + b, + G kCgWarps, ...
  const int ng = (a.N + kPw - 1) / kPw, g0 = warp * gridDim.x + blockIdx.x, gstep = gridDim.x * kCgWarps;
  auto stencil = [&](int u) {
    WarpStencil<T, false> ws;
    ws.carve(st_base + (size_t)(warp * nkeep + (a.kept ? u : 0)) * kStBytes);
    return ws;
  };
  if (kspace && a.kept) {
    int u = 0;
    for (int gi = g0; gi < ng; gi += gstep, ++u) {
      WarpStencil<T, false> ws = stencil(u);
      warp_build_stencil<T, false>(ws, d, g, a.pos, nullptr, nullptr, gi * kPw, a.N, lane);
    }
  }
  CGScal* sc = a.sc;
  if (sc->done) return;  // the same for every block: only phase A writes it, behind the first barrier
  const double rr0 = sc->rr;
  const int nc = sc->n_const;
  unsigned target = 0;
  auto stop = [&]() {
    if (threadIdx.x == 0) {
      atomicExch(&a.sh->failed, 1);
      atomicExch(&sc->status, ADMP_ERR_CUDA);
    }
  };
  for (int k = a.k0;; ++k) {
    CgSlot& S = a.sh->slot[k % 3];
    volatile CgSlot& S1 = a.sh->slot[(k + 2) % 3];  // iteration k - 1
    volatile CgSlot& S2 = a.sh->slot[(k + 1) % 3];  // iteration k - 2
    const double rr = k == 0 ? rr0 : S1.rr_new;
    // ---- A: convergence of the last iterate, direction, spread
    if (k > 0) {
      const bool conv = sqrt(rr) / (double)a.N < a.P.tol;
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
      const double rp = k == 0 ? 0.0 : (k == 1 ? rr0 : S2.rr_new);
      const double beta = rp != 0.0 ? rr / rp : 0.0;
      double acc[3] = {0, 0, 0};
      int u = 0;
      for (int gi = g0; gi < ng; gi += gstep, ++u) {
        WarpStencil<T, false> ws = stencil(u);
        const int na = min(kPw, a.N - gi * kPw);
        if (kspace && !a.kept) warp_build_stencil<T, false>(ws, d, g, a.pos, nullptr, nullptr, gi * kPw, a.N, lane);
        if (lane < na) {
          const int i = gi * kPw + lane;
          T pt = a.p[i];
          double pn = (double)pt;
          if (k > 0) {
            pn = a.r[i] + beta * pn;
            pt = (T)pn;
            a.p[i] = pt;
          } else {
            pn = a.r[i];  // the first direction is the residual
          }
          if (kspace) ws.q[lane] = pt;
          const double z = a.zc[i];
          acc[0] += pn;
          acc[1] += pn * z;
          acc[2] += pn * z * z;
        }
        __syncwarp();
        if (kspace) spread_group<T>(ws, na, a.K1, a.K2, a.mesh, lane);
        __syncwarp();
      }
      block_atomic_sum<3>(acc, &S.sp, red);
    }
    if (!cg_barrier(a.sh, target)) return stop();
    // ---- Z .. Z': the mesh part; the pairs need only p and Hp
    if (kspace) cg_z_pass<T, false>(a, f, R2);
    if (a.have_pairs) {
      const long long n = (long long)*a.list.n;
      for (long long p0 = blockIdx.x * (long long)kCgThreads + (threadIdx.x & ~31); p0 < n;
           p0 += (long long)gridDim.x * kCgThreads) {
        const long long p = p0 + lane;
        int2 ij = make_int2(-1, -1);
        T c = T(0);
        if (p < n) {
          ij = a.list.ij[p];
          c = a.list.coef[p];
        }
        const bool on = c != T(0);
        const WarpRuns runs(ij.x, lane);
        const T w = runs.sum(on ? c * a.p[ij.y] : T(0));
        if (runs.opens && w != T(0)) atomicAdd(a.Hp + ij.x, w);
        if (on) atomicAdd(a.Hp + ij.y, c * a.p[ij.x]);
      }
    }
    if (kspace) {
      if (!cg_barrier(a.sh, target)) return stop();
      cg_y_pass<T, false>(a, f, R1);
      if (!cg_barrier(a.sh, target)) return stop();
      cg_x_pass<T>(a, f, R0);
      if (!cg_barrier(a.sh, target)) return stop();
      cg_y_pass<T, true>(a, f, R1);
      if (!cg_barrier(a.sh, target)) return stop();
      cg_z_pass<T, true>(a, f, R2);
    }
    if (!cg_barrier(a.sh, target)) return stop();
    // ---- E: potential, diagonal and rank-one terms, p.Hp and C.Hp
    {
      volatile CgSlot& V = S;
      const double sp = V.sp, spz = V.spz, spz2 = V.spz2, nn = sc->nn, pre = sc->pre, Lz2 = sc->Lz2;
      double acc[5] = {0, 0, 0, 0, 0};
      int u = 0;
      for (int gi = g0; gi < ng; gi += gstep, ++u) {
        const int na = min(kPw, a.N - gi * kPw);
        T pot = T(0);
        if (kspace) {
          WarpStencil<T, false> ws = stencil(u);
          if (!a.kept) warp_build_stencil<T, false>(ws, d, g, a.pos, nullptr, nullptr, gi * kPw, a.N, lane);
          pot = gather_group<T, false>(ws, na, a.K1, a.K2, a.mesh, lane);
          __syncwarp();
        }
        if ((lane & 3) == 0 && (lane >> 2) < na) {
          const int i = gi * kPw + (lane >> 2);
          const double x = (double)a.p[i];
          double h = (double)(T)(a.Hp[i] + pot) + a.diag[i] * x + nn * sp;
          if (slab) {
            const double z = a.zc[i];
            h += pre * (2.0 * z * spz - spz2 - z * z * sp - Lz2 / 6.0 * sp);
          }
          a.Hp[i] = (T)h;
          acc[0] += x * h;
          for (int c = 0; c < nc; ++c) acc[1 + c] += cval(a.C, c, (long long)a.N, i) * h;
        }
      }
      double a1[1] = {acc[0]};
      block_atomic_sum<1>(a1, &S.pHp, red);
      if (nc > 0) {
        double a4[4] = {acc[1], acc[2], acc[3], acc[4]};
        block_atomic_sum<4>(a4, S.Cv, red);
      }
    }
    if (!cg_barrier(a.sh, target)) return stop();
    // ---- F: iterate and residual; zero what the next iteration accumulates into
    {
      volatile CgSlot& V = S;
      const double pHp = V.pHp, alpha = pHp != 0.0 ? rr / pHp : 0.0;
      double lam[kMaxConst] = {0, 0, 0, 0};
      for (int r0 = 0; r0 < nc; ++r0)
        for (int c = 0; c < nc; ++c) lam[r0] += sc->Ginv[r0 * kMaxConst + c] * V.Cv[c];
      double acc[1] = {0.0};
      const int tid = blockIdx.x * kCgThreads + threadIdx.x, nthr = gridDim.x * kCgThreads;
      for (int i = tid; i < a.N; i += nthr) {
        double w = (double)a.Hp[i];
        a.Hp[i] = T(0);
        for (int c = 0; c < nc; ++c) w -= cval(a.C, c, (long long)a.N, i) * lam[c];
        a.x[i] += alpha * (double)a.p[i];
        const double rn = a.r[i] - alpha * w;
        a.r[i] = rn;
        acc[0] += rn * rn;
      }
      block_atomic_sum<1>(acc, &S.rr_new, red);
      if (kspace) {
        const size_t M = (size_t)a.K0 * a.K1 * a.K2;
        for (size_t i = tid; i < M; i += nthr) a.mesh[i] = T(0);
      }
      if (blockIdx.x == 0 && threadIdx.x == 0) a.sh->slot[(k + 1) % 3] = CgSlot{};
    }
    if (!cg_barrier(a.sh, target)) return stop();
  }
}

}  // namespace admp
