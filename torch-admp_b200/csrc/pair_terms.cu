// Pair-list and per-atom terms of the drop-in path.
//   admp_pair_energy      pme.py:312-349 (Ewald real), pme.py:529-561 (OBC),
//                         qeq.py:104-119 (Gaussian damping pair part)
//   admp_atom_terms       pme.py:448-527 (self, non-neutral, slab),
//                         qeq.py:121-126 (damping self), qeq.py:159-209 (site)
//   admp_pair_distances   nblist.py:517-551 with spatial.py:15-36
#include "admp_common.cuh"
#include "pair_terms.h"

namespace admp {

template <typename T, int MODE>
__global__ void __launch_bounds__(256)
    pair_list_kernel(int N, long long P, const long long* __restrict__ pairs, const T* __restrict__ ds,
                     const void* __restrict__ scales, int int_scales, const T* __restrict__ q,
                     const T* __restrict__ eta, T kappa,
                     T ke, double* __restrict__ energy, int estride, int put, T* __restrict__ dE_dds,
                     T* __restrict__ dE_dq, T* __restrict__ dE_deta, DevError* err) {
  __shared__ double red[32];
  const int f = blockIdx.y;
  pairs += (size_t)f * P * 2;
  ds += (size_t)f * P;
  // buffer scales of the working type, or int64 as the neighbour list makes them
  const T* bs = int_scales ? nullptr : (const T*)scales + (size_t)f * P;
  const long long* ibs = int_scales ? (const long long*)scales + (size_t)f * P : nullptr;
  q += (size_t)f * N;
  if (eta) eta += (size_t)f * N;
  if (dE_dds) dE_dds += (size_t)f * P;
  if (dE_dq) dE_dq += (size_t)f * N;
  if (dE_deta) dE_deta += (size_t)f * N;
  const T two_over_sqrtpi = T(2.0 / kSqrtPi);
  const int lane = threadIdx.x & 31;
  double e = 0.0;
  for (long long p0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); p0 < P;
       p0 += (long long)gridDim.x * blockDim.x) {
    const long long p = p0 + lane;
    long long i = 0, j = 0;
    bool ok = p < P;
    if (ok) {
      const longlong2 ij = load_pair(pairs, p);
      i = ij.x;
      j = ij.y;
      if (i < 0 || i >= N || j < 0 || j >= N) {
        report_error(err, ADMP_ERR_BAD_INDEX, 1, p);
        if (put && dE_dds) dE_dds[p] = T(0);
        ok = false;
      }
    }
    const T d = ok ? ds[p] : T(1), s = ok ? (ibs ? (T)ibs[p] : bs[p]) : T(0);
    const T qi = ok ? q[i] : T(0), qj = ok ? q[j] : T(0);
    T ei = T(0), ej = T(0);
    if (MODE == ADMP_PAIR_DAMPING && ok) {
      ei = eta[i];
      ej = eta[j];
    }
    // a full list has scale 0 on half of its pairs: nothing to evaluate there unless a value is not finite
    const bool skip = !ok || (s == T(0) && isfinite(d + qi * qj + ei + ej));
    T ep = T(0), dd = T(0), c = T(0), gi = T(0), gj = T(0);
    if (!skip) {
      const T thr = MODE == ADMP_PAIR_OBC ? T(1e-8) : T(1e-4);
      const bool valid = fabs((double)d) > (double)thr;
      const T inv = valid ? T(1) / d : T(0);
      if (MODE == ADMP_PAIR_EWALD) {
        const T x = kappa * d;
        const T er = erfc_t(x);
        ep = er * qi * qj * inv * s * ke;
        dd = valid ? (-two_over_sqrtpi * kappa * exp_t(-x * x) * inv - er * inv * inv) * qi * qj * s * ke : T(0);
        c = er * inv * s * ke;
      } else if (MODE == ADMP_PAIR_OBC) {
        ep = qi * qj * ke * inv * s;
        dd = valid ? -qi * qj * ke * inv * inv * s : T(0);
        c = ke * inv * s;
      } else {
        const T eij = sqrt_t((ei * ei + ej * ej) / T(2));
        const bool zero = eij == T(0);
        const T eijs = zero ? T(1e-10) : eij;
        const T x = d / (T(2) * eijs);
        const T er = erfc_t(x);
        const T ge = two_over_sqrtpi * exp_t(-x * x);
        ep = -er * qi * qj * inv * s * ke;
        dd = valid ? (ge / (T(2) * eijs) * inv + er * inv * inv) * qi * qj * s * ke : T(0);
        c = -er * inv * s * ke;
        if (dE_deta && !zero) {
          const T deij = -ge * d / (T(2) * eijs * eijs) * qi * qj * inv * s * ke;
          gi = deij * ei / (T(2) * eijs);
          gj = deij * ej / (T(2) * eijs);
        }
      }
      e += (double)ep;
    }
    if (ok && dE_dds) dE_dds[p] = put ? dd : dE_dds[p] + dd;
    if ((dE_dq || (MODE == ADMP_PAIR_DAMPING && dE_deta)) && __any_sync(0xffffffffu, !skip)) {
      // one atomic per run of pairs with the same first atom, one per pair for the second
      const WarpRuns runs(ok ? (int)i : -1, lane);
      if (dE_dq) {
        const T a = runs.sum(c != T(0) ? c * qj : T(0));
        if (runs.opens && a != T(0)) atomicAdd(dE_dq + i, a);
        if (c != T(0)) atomicAdd(dE_dq + j, c * qi);
      }
      if (MODE == ADMP_PAIR_DAMPING && dE_deta) {
        const T a = runs.sum(gi);
        if (runs.opens && a != T(0)) atomicAdd(dE_deta + i, a);
        if (gj != T(0)) atomicAdd(dE_deta + j, gj);
      }
    }
  }
  double v[1] = {e};
  if (energy) block_atomic_sum<1>(v, energy + (size_t)f * estride, red);
}

template <typename T>
__global__ void __launch_bounds__(512)
    atom_terms_kernel(int flags, int N, const T* __restrict__ pos, const T* __restrict__ box,
                      const T* __restrict__ q, const T* __restrict__ eta, const T* __restrict__ chi,
                      const T* __restrict__ hard, double kappa, double ke, double* __restrict__ energy,
                      double* __restrict__ terms, T* __restrict__ dq, T* __restrict__ dpos,
                      T* __restrict__ dbox, T* __restrict__ deta, T* __restrict__ dchi,
                      T* __restrict__ dhard) {
  __shared__ double red[6 * 32];
  __shared__ double sums[6];
  __shared__ double geo[20];  // box 9, binv 9, V, Lz
  const int f = blockIdx.x;
  const int axis = (flags >> 8) & 3;
  q += (size_t)f * N;
  if (pos) pos += (size_t)f * N * 3;
  if (eta) eta += (size_t)f * N;
  if (chi) chi += (size_t)f * N;
  if (hard) hard += (size_t)f * N;
  if (threadIdx.x < 6) sums[threadIdx.x] = 0.0;
  if (threadIdx.x == 0 && box) {
    double b[9], bi[9];
    load_box(box + (size_t)f * 9, b);
    double V = inv3(b, bi);
    for (int k = 0; k < 9; ++k) {
      geo[k] = b[k];
      geo[9 + k] = bi[k];
    }
    geo[18] = V;
    geo[19] = sqrt(b[axis * 3] * b[axis * 3] + b[axis * 3 + 1] * b[axis * 3 + 1] + b[axis * 3 + 2] * b[axis * 3 + 2]);
  }
  __syncthreads();
  // pass 1: Q, sum q^2, Mz, sum q z^2, damping self, site
  double v[6] = {0, 0, 0, 0, 0, 0};
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const double qi = q[i];
    v[0] += qi;
    v[1] += qi * qi;
    if (flags & ADMP_TERM_SLAB) {
      const double z = pos[3 * (size_t)i + axis];
      v[2] += qi * z;
      v[3] += qi * z * z;
    }
    if (flags & ADMP_TERM_DAMP_SELF) {
      const double e = eta[i];
      const double einv = fabs(e) > 1e-4 ? 1.0 / e : 0.0;
      v[4] += einv / (2.0 * kSqrtPi) * qi * qi;
    }
    if (flags & ADMP_TERM_SITE) v[5] += (double)chi[i] * qi + (double)hard[i] * qi * qi;
  }
  block_atomic_sum<6>(v, sums, red);
  const double Q = sums[0], Sq2 = sums[1], Mz = sums[2], Sz2 = sums[3];
  double Eself = 0, Enn = 0, Eslab = 0, Eds = 0, Esite = 0, pre = 0, V = 0, Lz = 0;
  if (flags & ADMP_TERM_SELF) Eself = -ke * kappa / kSqrtPi * Sq2;
  if (box) {
    V = geo[18];
    Lz = geo[19];
  }
  if (flags & ADMP_TERM_NON_NEUTRAL) Enn = -kPi / (2.0 * V * kappa * kappa) * ke * Q * Q;
  if (flags & ADMP_TERM_SLAB) {
    pre = 2.0 * kPi / V * ke;
    Eslab = pre * (Mz * Mz - Q * Sz2 - Q * Q * Lz * Lz / 12.0);
  }
  if (flags & ADMP_TERM_DAMP_SELF) Eds = ke * sums[4];
  if (flags & ADMP_TERM_SITE) Esite = sums[5];
  if (threadIdx.x == 0) {
    if (energy) energy[f] += Eself + Enn + Eslab + Eds + Esite;
    if (terms) {
      terms[f * 5 + 0] += Eself;
      terms[f * 5 + 1] += Enn;
      terms[f * 5 + 2] += Eslab;
      terms[f * 5 + 3] += Eds;
      terms[f * 5 + 4] += Esite;
    }
    if (dbox) {
      double g[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      const double Ev = Enn + Eslab;  // both scale as 1/V: dE/dbox = -E B^T
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) g[i * 3 + j] = -Ev * geo[9 + j * 3 + i];
      if ((flags & ADMP_TERM_SLAB) && Lz > 0) {
        const double dLz = pre * (-Q * Q * 2.0 * Lz / 12.0);
        for (int j = 0; j < 3; ++j) g[axis * 3 + j] += dLz * geo[axis * 3 + j] / Lz;
      }
      for (int k = 0; k < 9; ++k) dbox[(size_t)f * 9 + k] += (T)g[k];
    }
  }
  // pass 2: per-atom gradients
  const double cself = (flags & ADMP_TERM_SELF) ? -2.0 * ke * kappa / kSqrtPi : 0.0;
  const double cnn = (flags & ADMP_TERM_NON_NEUTRAL) ? -kPi / (V * kappa * kappa) * ke * Q : 0.0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const double qi = q[i];
    double g = cself * qi + cnn;
    if (flags & ADMP_TERM_SLAB) {
      const double z = pos[3 * (size_t)i + axis];
      g += pre * (2.0 * Mz * z - Sz2 - Q * z * z - Q * Lz * Lz / 6.0);
      if (dpos) dpos[((size_t)f * N + i) * 3 + axis] += (T)(pre * (2.0 * Mz * qi - 2.0 * Q * qi * z));
    }
    if (flags & ADMP_TERM_DAMP_SELF) {
      const double e = eta[i];
      const bool ok = fabs(e) > 1e-4;
      const double einv = ok ? 1.0 / e : 0.0;
      g += ke * qi * einv / kSqrtPi;
      if (deta) deta[(size_t)f * N + i] += (T)(ok ? -ke * qi * qi / (2.0 * kSqrtPi) * einv * einv : 0.0);
    }
    if (flags & ADMP_TERM_SITE) {
      g += (double)chi[i] + 2.0 * (double)hard[i] * qi;
      if (dchi) dchi[(size_t)f * N + i] += (T)qi;
      if (dhard) dhard[(size_t)f * N + i] += (T)(qi * qi);
    }
    if (dq) dq[(size_t)f * N + i] += (T)g;
  }
}

// Damping self energies (DAMP: q, eta) or chemical site energies (q, chi,
// hardness) of every atom: gradients are written, energies summed into
// energy[frame].  A block per 256 atoms (one block a frame, two passes over the
// atoms, took 20 us at 20,000 atoms).
template <typename T, bool DAMP>
__global__ void __launch_bounds__(256)
    atom_energy_kernel(int N, const T* __restrict__ q, const T* __restrict__ u, const T* __restrict__ w, double ke,
                       double* __restrict__ energy, T* __restrict__ dq, T* __restrict__ du, T* __restrict__ dw) {
  __shared__ double red[32];
  const int f = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
  double v[1] = {0.0};
  if (i < N) {
    const size_t a = (size_t)f * N + i;
    const double qi = q[a];
    if (DAMP) {
      const double e = u[a];
      const bool ok = fabs(e) > 1e-4;
      const double einv = ok ? 1.0 / e : 0.0;
      v[0] = ke * einv / (2.0 * kSqrtPi) * qi * qi;
      if (dq) dq[a] = (T)(ke * qi * einv / kSqrtPi);
      if (du) du[a] = (T)(ok ? -ke * qi * qi / (2.0 * kSqrtPi) * einv * einv : 0.0);
    } else {
      const double chi = u[a], hard = w[a];
      v[0] = chi * qi + hard * qi * qi;
      if (dq) dq[a] = (T)(chi + 2.0 * hard * qi);
      if (du) du[a] = (T)qi;
      if (dw) dw[a] = (T)(qi * qi);
    }
  }
  block_atomic_sum<1>(v, energy + f, red);
}

template <typename T>
__global__ void __launch_bounds__(256)
    pair_dist_kernel(int pbc, int N, long long P, const long long* __restrict__ pairs,
                     const T* __restrict__ pos, const T* __restrict__ box, T* __restrict__ ds,
                     DevError* err) {
  __shared__ double geo[18];
  if (threadIdx.x == 0 && pbc) {
    load_box(box, geo);
    inv3(geo, geo + 9);
  }
  __syncthreads();
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
       p += (long long)gridDim.x * blockDim.x) {
    const long long i = pairs[2 * p], j = pairs[2 * p + 1];
    if (i < 0 || i >= N || j < 0 || j >= N) {
      report_error(err, ADMP_ERR_BAD_INDEX, 2, p);
      ds[p] = T(0);
      continue;
    }
    double dr[3], n[3];
    if (pbc) {
      for (int e = 0; e < 3; ++e) dr[e] = (double)pos[3 * i + e] - (double)pos[3 * j + e];
      min_image(geo, geo + 9, dr, n);
    } else {
      for (int e = 0; e < 3; ++e) dr[e] = (double)pos[3 * j + e] - (double)pos[3 * i + e];
    }
    ds[p] = (T)sqrt(dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2]);
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
    pair_dist_bwd_kernel(int pbc, int N, long long P, const long long* __restrict__ pairs,
                         const T* __restrict__ pos, const T* __restrict__ box, const T* __restrict__ g,
                         T* __restrict__ gpos, T* __restrict__ gbox, DevError* err) {
  __shared__ double geo[18];
  __shared__ double red[9 * 32];
  const int f = blockIdx.y;
  pairs += (size_t)f * P * 2;
  g += (size_t)f * P;
  pos += (size_t)f * N * 3;
  if (box) box += (size_t)f * 9;
  if (gpos) gpos += (size_t)f * N * 3;
  if (gbox) gbox += (size_t)f * 9;
  if (threadIdx.x == 0 && pbc) {
    load_box(box, geo);
    inv3(geo, geo + 9);
  }
  __syncthreads();
  double vb[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  const int lane = threadIdx.x & 31;
  for (long long p0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); p0 < P;
       p0 += (long long)gridDim.x * blockDim.x) {
    const long long p = p0 + lane;
    const double gp = p < P ? (double)g[p] : 0.0;
    if (!__any_sync(0xffffffffu, p < P && gp != 0.0)) {
      if (p >= P) continue;
      const longlong2 ij = load_pair(pairs, p);
      if (ij.x < 0 || ij.x >= N || ij.y < 0 || ij.y >= N) report_error(err, ADMP_ERR_BAD_INDEX, 3, p);
      continue;
    }
    long long i = 0, j = 0;
    bool ok = p < P;
    if (ok) {
      const longlong2 ij = load_pair(pairs, p);
      i = ij.x;
      j = ij.y;
      if (i < 0 || i >= N || j < 0 || j >= N) {
        report_error(err, ADMP_ERR_BAD_INDEX, 3, p);
        ok = false;
      }
    }
    const bool live = ok && gp != 0.0;
    double dr[3] = {0, 0, 0}, n[3] = {0, 0, 0}, s = 0.0;
    if (live) {
      if (pbc) {
        for (int e = 0; e < 3; ++e) dr[e] = (double)pos[3 * i + e] - (double)pos[3 * j + e];
        min_image(geo, geo + 9, dr, n);
      } else {
        for (int e = 0; e < 3; ++e) dr[e] = (double)pos[3 * j + e] - (double)pos[3 * i + e];
      }
      const double r2 = dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2];
      s = r2 == 0.0 ? 0.0 : gp * rsqrt(r2);
    }
    // dr points from j to i with a box and from i to j without: the first atom gets +v or -v; its share is summed
    // over the run of pairs that start with it
    const WarpRuns runs(ok ? (int)i : -1, lane);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const double v = s == 0.0 ? 0.0 : s * dr[e];
      if (gpos) {
        const T w = (T)(pbc ? v : -v), a = runs.sum(w);
        if (runs.opens && a != T(0)) atomicAdd(gpos + 3 * i + e, a);
        if (w != T(0)) atomicAdd(gpos + 3 * j + e, -w);
      }
      if (pbc && gbox)
        for (int k = 0; k < 3; ++k) vb[k * 3 + e] -= n[k] * v;
    }
  }
  if (pbc && gbox) {
    __shared__ double out[9];
    if (threadIdx.x < 9) out[threadIdx.x] = 0.0;
    __syncthreads();
    block_atomic_sum<9>(vb, out, red);
    if (threadIdx.x < 9 && out[threadIdx.x] != 0.0) atomicAdd(gbox + threadIdx.x, (T)out[threadIdx.x]);
  }
}

// out[f][k] = in[f][k] * w[f] for up to four arrays in one launch
struct ScaleArgs {
  const void* in[4];
  void* out[4];
  long long n[4];  // values per frame
};
template <typename T>
__global__ void __launch_bounds__(256) scale_frames_kernel(ScaleArgs a, const T* __restrict__ w, long long wstride) {
  const int f = blockIdx.y;
  const T x = w[f * wstride];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const T* in = (const T*)a.in[k] + (size_t)f * a.n[k];
    T* out = (T*)a.out[k] + (size_t)f * a.n[k];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.n[k];
         i += (long long)gridDim.x * blockDim.x)
      out[i] = in[i] * x;
  }
}

// ------------------------------------------------------------------ host side
// energy[f estride] += E of frame f; dE/dds is added to, or with `put` written.
template <typename T>
int launch_pair_energy(int mode, int nf, int N, long long P, const long long* pairs, const T* ds, const void* bs,
                       bool int_scales, const T* q, const T* eta, double kappa, double ke, double* energy, int estride,
                       bool put, T* dds, T* dq, T* deta, DevError* err, cudaStream_t st) {
  if (P == 0 || nf == 0) return ADMP_OK;
  long long blocks = (P + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  const dim3 grid((unsigned)blocks, (unsigned)nf);
  auto* k = mode == ADMP_PAIR_EWALD ? pair_list_kernel<T, ADMP_PAIR_EWALD>
            : mode == ADMP_PAIR_OBC ? pair_list_kernel<T, ADMP_PAIR_OBC>
                                    : pair_list_kernel<T, ADMP_PAIR_DAMPING>;
  k<<<grid, 256, 0, st>>>(N, P, pairs, ds, bs, int_scales ? 1 : 0, q, eta, (T)kappa, (T)ke, energy, estride,
                          put ? 1 : 0, dds, dq, deta, err);
  ADMP_CUDA_TRY(cudaGetLastError());
  return ADMP_OK;
}
template int launch_pair_energy<float>(int, int, int, long long, const long long*, const float*, const void*, bool,
                                       const float*, const float*, double, double, double*, int, bool, float*, float*,
                                       float*, DevError*, cudaStream_t);
template int launch_pair_energy<double>(int, int, int, long long, const long long*, const double*, const void*, bool,
                                        const double*, const double*, double, double, double*, int, bool, double*,
                                        double*, double*, DevError*, cudaStream_t);

template <typename T>
static int pair_energy_impl(int mode, int nf, int N, long long P, const long long* pairs, const void* ds,
                            const void* bs, const void* q, const void* eta, double kappa, double ke,
                            double* energy, void* dds, void* dq, void* deta, cudaStream_t st) {
  if (P == 0 || nf == 0) return ADMP_OK;
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  const int s = launch_pair_energy<T>(mode, nf, N, P, pairs, (const T*)ds, bs, false, (const T*)q, (const T*)eta,
                                      kappa, ke, energy, 1, false, (T*)dds, (T*)dq, (T*)deta, err, st);
  return s ? s : check_error(err, st);
}

}  // namespace admp

using namespace admp;

extern "C" int admp_pair_energy(int dtype, int mode, int nframes, int natoms, long long npairs,
                                const long long* pairs, const void* ds, const void* buffer_scales,
                                const void* q, const void* eta, double kappa, double ke, double* energy,
                                void* dE_dds, void* dE_dq, void* dE_deta, void* stream) {
  if (mode < 0 || mode > 2 || nframes < 0 || natoms < 0 || npairs < 0) return fail(ADMP_ERR_BAD_ARG, "admp_pair_energy: bad mode/sizes");
  if (npairs > 0 && (!pairs || !ds || !buffer_scales || !q)) return fail(ADMP_ERR_BAD_ARG, "admp_pair_energy: null input");
  if (mode == ADMP_PAIR_DAMPING && npairs > 0 && !eta) return fail(ADMP_ERR_BAD_ARG, "admp_pair_energy: damping needs eta");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return pair_energy_impl<double>(mode, nframes, natoms, npairs, pairs, ds, buffer_scales, q, eta, kappa, ke,
                                    energy, dE_dds, dE_dq, dE_deta, st);
  if (dtype == ADMP_F32)
    return pair_energy_impl<float>(mode, nframes, natoms, npairs, pairs, ds, buffer_scales, q, eta, kappa, ke,
                                   energy, dE_dds, dE_dq, dE_deta, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_atom_terms(int dtype, int flags, int nframes, int natoms, const void* pos, const void* box,
                               const void* q, const void* eta, const void* chi, const void* hardness,
                               double kappa, double ke, double* energy, double* terms, void* dE_dq,
                               void* dE_dpos, void* dE_dbox, void* dE_deta, void* dE_dchi, void* dE_dhard,
                               void* stream) {
  if (nframes <= 0 || natoms < 0) return nframes == 0 ? ADMP_OK : fail(ADMP_ERR_BAD_ARG, "admp_atom_terms: sizes");
  if (!q) return fail(ADMP_ERR_BAD_ARG, "admp_atom_terms: q is null");
  if ((flags & (ADMP_TERM_NON_NEUTRAL | ADMP_TERM_SLAB)) && !box) return fail(ADMP_ERR_BAD_ARG, "admp_atom_terms: box needed");
  if ((flags & ADMP_TERM_SLAB) && !pos) return fail(ADMP_ERR_BAD_ARG, "admp_atom_terms: pos needed");
  if ((flags & ADMP_TERM_DAMP_SELF) && !eta) return fail(ADMP_ERR_BAD_ARG, "admp_atom_terms: eta needed");
  if ((flags & ADMP_TERM_SITE) && (!chi || !hardness)) return fail(ADMP_ERR_BAD_ARG, "admp_atom_terms: chi/hardness needed");
  if (((flags >> 8) & 3) > 2) return fail(ADMP_ERR_BAD_ARG, "admp_atom_terms: slab axis");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64) {
    atom_terms_kernel<double><<<nframes, 512, 0, st>>>(flags, natoms, (const double*)pos, (const double*)box,
                                                       (const double*)q, (const double*)eta, (const double*)chi,
                                                       (const double*)hardness, kappa, ke, energy, terms,
                                                       (double*)dE_dq, (double*)dE_dpos, (double*)dE_dbox,
                                                       (double*)dE_deta, (double*)dE_dchi, (double*)dE_dhard);
  } else if (dtype == ADMP_F32) {
    atom_terms_kernel<float><<<nframes, 512, 0, st>>>(flags, natoms, (const float*)pos, (const float*)box,
                                                      (const float*)q, (const float*)eta, (const float*)chi,
                                                      (const float*)hardness, kappa, ke, energy, terms,
                                                      (float*)dE_dq, (float*)dE_dpos, (float*)dE_dbox,
                                                      (float*)dE_deta, (float*)dE_dchi, (float*)dE_dhard);
  } else {
    return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  }
  ADMP_CUDA_TRY(cudaGetLastError());
  return ADMP_OK;
}

extern "C" int admp_pair_distances(int dtype, int pbc, int natoms, long long npairs, const long long* pairs,
                                   const void* pos, const void* box, void* ds, void* stream) {
  if (npairs == 0) return ADMP_OK;
  if (npairs < 0 || !pairs || !pos || !ds || (pbc && !box)) return fail(ADMP_ERR_BAD_ARG, "admp_pair_distances: args");
  cudaStream_t st = (cudaStream_t)stream;
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  long long blocks = (npairs + 255) / 256;
  if (blocks > 8192) blocks = 8192;
  if (dtype == ADMP_F64)
    pair_dist_kernel<double><<<(unsigned)blocks, 256, 0, st>>>(pbc, natoms, npairs, pairs, (const double*)pos,
                                                               (const double*)box, (double*)ds, err);
  else if (dtype == ADMP_F32)
    pair_dist_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(pbc, natoms, npairs, pairs, (const float*)pos,
                                                              (const float*)box, (float*)ds, err);
  else
    return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  ADMP_CUDA_TRY(cudaGetLastError());
  return check_error(err, st);
}

static int pair_dist_bwd(int dtype, int pbc, int nf, int natoms, long long npairs, const long long* pairs,
                         const void* pos, const void* box, const void* grad_ds, void* grad_pos, void* grad_box,
                         DevError* err, cudaStream_t st) {
  long long blocks = (npairs + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  const dim3 grid((unsigned)blocks, (unsigned)nf);
  if (dtype == ADMP_F64)
    pair_dist_bwd_kernel<double><<<grid, 256, 0, st>>>(pbc, natoms, npairs, pairs, (const double*)pos,
                                                       (const double*)box, (const double*)grad_ds, (double*)grad_pos,
                                                       (double*)grad_box, err);
  else if (dtype == ADMP_F32)
    pair_dist_bwd_kernel<float><<<grid, 256, 0, st>>>(pbc, natoms, npairs, pairs, (const float*)pos, (const float*)box,
                                                      (const float*)grad_ds, (float*)grad_pos, (float*)grad_box, err);
  else
    return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  ADMP_CUDA_TRY(cudaGetLastError());
  return ADMP_OK;
}

extern "C" int admp_pair_distances_backward(int dtype, int pbc, int natoms, long long npairs,
                                            const long long* pairs, const void* pos, const void* box,
                                            const void* grad_ds, void* grad_pos, void* grad_box, void* stream) {
  if (npairs == 0) return ADMP_OK;
  if (npairs < 0 || !pairs || !pos || !grad_ds || (pbc && !box)) return fail(ADMP_ERR_BAD_ARG, "admp_pair_distances_backward: args");
  cudaStream_t st = (cudaStream_t)stream;
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  const int s = pair_dist_bwd(dtype, pbc, 1, natoms, npairs, pairs, pos, box, grad_ds, grad_pos, grad_box, err, st);
  return s ? s : check_error(err, st);
}

extern "C" int admp_pair_distances_frames_backward(int dtype, int pbc, int nframes, int natoms, long long npairs,
                                                   const long long* pairs, const void* pos, const void* box,
                                                   const void* grad_ds, void* grad_pos, void* grad_box, void* stream) {
  if (nframes < 0 || nframes > 65535 || natoms < 0 || npairs < 0 || (dtype != ADMP_F64 && dtype != ADMP_F32))
    return fail(ADMP_ERR_BAD_ARG, "admp_pair_distances_frames_backward: args");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t size = dtype == ADMP_F64 ? 8 : 4;
  if (grad_pos) ADMP_CUDA_TRY(cudaMemsetAsync(grad_pos, 0, size * 3 * natoms * nframes, st));
  if (grad_box) ADMP_CUDA_TRY(cudaMemsetAsync(grad_box, 0, size * 9 * nframes, st));
  if (npairs == 0 || nframes == 0) return ADMP_OK;
  if (!pairs || !pos || !grad_ds || (pbc && !box))
    return fail(ADMP_ERR_BAD_ARG, "admp_pair_distances_frames_backward: args");
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  return pair_dist_bwd(dtype, pbc, nframes, natoms, npairs, pairs, pos, box, grad_ds, grad_pos, grad_box, err, st);
}

// Frames are the y dimension of these grids; the entry points take more of them in several launches.
constexpr int kGridFrames = 65535;
static const void* frame_at(const void* p, long long elems, size_t size) { return p ? (const char*)p + elems * size : p; }
static void* frame_at(void* p, long long elems, size_t size) { return p ? (char*)p + elems * size : p; }

template <typename T>
static int damping_frames(bool ints, int nf, int N, long long P, const long long* pairs, const void* ds, const void* bs,
                          const void* q, const void* eta, double ke, double* energy, void* dds, void* dq, void* deta,
                          DevError* err, cudaStream_t st) {
  atom_energy_kernel<T, true><<<dim3((N + 255) / 256, nf), 256, 0, st>>>(N, (const T*)q, (const T*)eta, nullptr, ke,
                                                                         energy, (T*)dq, (T*)deta, nullptr);
  ADMP_CUDA_TRY(cudaGetLastError());
  return launch_pair_energy<T>(ADMP_PAIR_DAMPING, nf, N, P, pairs, (const T*)ds, bs, ints, (const T*)q, (const T*)eta,
                               0.0, ke, energy, 1, true, (T*)dds, (T*)dq, (T*)deta, err, st);
}

extern "C" int admp_damping_energy(int dtype, int flags, int nframes, int natoms, long long npairs, const long long* pairs,
                                   const void* ds, const void* buffer_scales, const void* q, const void* eta, double ke,
                                   double* energy, void* dE_dds, void* dE_dq, void* dE_deta, void* stream) {
  if (nframes <= 0 || natoms <= 0 || npairs < 0 || !q || !eta || !energy)
    return fail(ADMP_ERR_BAD_ARG, "admp_damping_energy: args");
  if (npairs > 0 && (!pairs || !ds || !buffer_scales)) return fail(ADMP_ERR_BAD_ARG, "admp_damping_energy: pairs");
  if (dtype != ADMP_F64 && dtype != ADMP_F32) return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  cudaStream_t st = (cudaStream_t)stream;
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  ADMP_CUDA_TRY(cudaMemsetAsync(energy, 0, sizeof(double) * nframes, st));
  const bool ints = (flags & ADMP_PAIR_INT64_SCALES) != 0;
  const size_t es = dtype == ADMP_F64 ? 8 : 4, ss = ints ? 8 : es;
  for (int f = 0; f < nframes; f += kGridFrames) {
    const int nf = nframes - f < kGridFrames ? nframes - f : kGridFrames;
    const long long a = (long long)f * natoms, p = f * npairs;
    auto* call = dtype == ADMP_F64 ? damping_frames<double> : damping_frames<float>;
    const int s = call(ints, nf, natoms, npairs, pairs + 2 * p, frame_at(ds, p, es), frame_at(buffer_scales, p, ss),
                       frame_at(q, a, es), frame_at(eta, a, es), ke, energy + f, frame_at(dE_dds, p, es),
                       frame_at(dE_dq, a, es), frame_at(dE_deta, a, es), err, st);
    if (s) return s;
  }
  return npairs == 0 ? ADMP_OK : check_error(err, st);
}

template <typename T>
static void site_frames(int nf, int N, const void* q, const void* chi, const void* hard, double* energy, void* dq,
                        void* dchi, void* dhard, cudaStream_t st) {
  atom_energy_kernel<T, false><<<dim3((N + 255) / 256, nf), 256, 0, st>>>(N, (const T*)q, (const T*)chi, (const T*)hard,
                                                                          0.0, energy, (T*)dq, (T*)dchi, (T*)dhard);
}

extern "C" int admp_site_energy(int dtype, int nframes, int natoms, const void* q, const void* chi,
                                const void* hardness, double* energy, void* dE_dq, void* dE_dchi, void* dE_dhard,
                                void* stream) {
  if (nframes <= 0 || natoms <= 0 || !q || !chi || !hardness || !energy)
    return fail(ADMP_ERR_BAD_ARG, "admp_site_energy: args");
  if (dtype != ADMP_F64 && dtype != ADMP_F32) return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  cudaStream_t st = (cudaStream_t)stream;
  ADMP_CUDA_TRY(cudaMemsetAsync(energy, 0, sizeof(double) * nframes, st));
  const size_t es = dtype == ADMP_F64 ? 8 : 4;
  for (int f = 0; f < nframes; f += kGridFrames) {
    const long long a = (long long)f * natoms;
    auto* call = dtype == ADMP_F64 ? site_frames<double> : site_frames<float>;
    call(nframes - f < kGridFrames ? nframes - f : kGridFrames, natoms, frame_at(q, a, es), frame_at(chi, a, es),
         frame_at(hardness, a, es), energy + f, frame_at(dE_dq, a, es), frame_at(dE_dchi, a, es),
         frame_at(dE_dhard, a, es), st);
    ADMP_CUDA_TRY(cudaGetLastError());
  }
  return ADMP_OK;
}

extern "C" int admp_scale_frames(int dtype, int nframes, int narrays, const void* const* in, void* const* out,
                                 const long long* per_frame, const void* w, long long w_stride, void* stream) {
  if (nframes <= 0 || narrays < 0 || narrays > 4 || !w)
    return nframes == 0 ? ADMP_OK : fail(ADMP_ERR_BAD_ARG, "admp_scale_frames: args");
  if (dtype != ADMP_F64 && dtype != ADMP_F32) return fail(ADMP_ERR_BAD_ARG, "bad dtype");
  const size_t es = dtype == ADMP_F64 ? 8 : 4;
  cudaStream_t st = (cudaStream_t)stream;
  for (int f = 0; f < nframes; f += kGridFrames) {
    ScaleArgs a{};
    long long most = 0;
    for (int k = 0; k < narrays; ++k) {
      a.in[k] = frame_at(in[k], f * per_frame[k], es);
      a.out[k] = frame_at(out[k], f * per_frame[k], es);
      a.n[k] = per_frame[k];
      most = most > per_frame[k] ? most : per_frame[k];
    }
    if (most == 0) return ADMP_OK;
    long long blocks = (most + 255) / 256;
    if (blocks > 2048) blocks = 2048;
    const dim3 grid((unsigned)blocks, nframes - f < kGridFrames ? nframes - f : kGridFrames);
    const void* wf = frame_at(w, f * w_stride, es);
    if (dtype == ADMP_F64)
      scale_frames_kernel<double><<<grid, 256, 0, st>>>(a, (const double*)wf, w_stride);
    else
      scale_frames_kernel<float><<<grid, 256, 0, st>>>(a, (const float*)wf, w_stride);
    ADMP_CUDA_TRY(cudaGetLastError());
  }
  return ADMP_OK;
}
