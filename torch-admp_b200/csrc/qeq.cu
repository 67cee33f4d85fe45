// admp_qeq_solve / admp_qeq_hvp: matrix-free projected CG for the QEq and
// electrode charges (replaces pgrad_optimize and the quadratic / LBFGS
// minimisers, qeq.py:1117-1527, electrode.py:456-560).
#include <vector>

#include "pme_host.h"
#include "qeq_cg.cuh"
#include "qeq_kernels.cuh"

namespace admp {

template <typename T>
struct QEqWS {
  RecipPlan<T> plan;
  SysDesc* table;
  T* mesh;
  Cplx<T>* spec;
  T* green;
  double* acc;
  double *x, *r, *diag, *zc, *chi_eff, *hx;
  T *p, *Hp;
  PairList<T> list;
  CGScal* sc;
  CgShared* cg;
  size_t bytes;
};

// nf frames of N atoms each (frame f: atoms [f N, (f+1) N), box f, mesh
// kmesh[3 f .. 3 f + 2]); every per-atom vector spans all frames.
template <typename T>
static int qeq_carve(QEqWS<T>& w, void* ws, size_t bytes, int nf, int N, long long P, const int* kmesh,
                     double kappa, int flags) {
  if (nf <= 0 || nf > kMaxBatch) return fail(ADMP_ERR_BAD_ARG, "qeq: %d frames per call (1..%d)", nf, kMaxBatch);
  SysSpec sys[kMaxBatch];
  for (int f = 0; f < nf; ++f) {
    sys[f].natoms = N;
    sys[f].atom_off = f * N;
    for (int d = 0; d < 3; ++d) sys[f].K[d] = (flags & ADMP_QEQ_KSPACE) ? kmesh[3 * f + d] : 1;
    sys[f].kappa = kappa > 0 ? kappa : 1.0;
    sys[f].box_idx = f;
  }
  int s = build_recip_plan<T>(sys, nf, w.plan);
  if (s) return s;
  const size_t NT = (size_t)nf * N;
  Carver c(ws, bytes);
  w.table = reinterpret_cast<SysDesc*>(c.take<unsigned char>(sys_table_bytes()));
  w.mesh = c.take<T>((flags & ADMP_QEQ_KSPACE) ? w.plan.mesh_elems : 0);
  w.spec = c.take<Cplx<T>>((flags & ADMP_QEQ_KSPACE) ? w.plan.spec_elems : 0);
  w.green = c.take<T>((flags & ADMP_QEQ_KSPACE) ? w.plan.spec_elems : 0);
  w.acc = c.take<double>((size_t)kAccStride * nf);
  w.x = c.take<double>(NT);
  w.r = c.take<double>(NT);
  w.diag = c.take<double>(NT);
  w.zc = c.take<double>(NT);
  w.chi_eff = c.take<double>(NT);
  w.hx = c.take<double>(NT);
  w.p = c.take<T>(NT);
  w.Hp = c.take<T>(NT);
  w.list.ij = c.take<int2>(P > 0 ? P : 0);
  w.list.coef = c.take<T>(P > 0 ? P : 0);
  w.list.n = c.take<unsigned long long>(1);
  w.sc = c.take<CGScal>(nf);
  w.cg = c.take<CgShared>(1);
  w.bytes = c.off;
  return ADMP_OK;
}

template <typename T>
struct QEqCtx {
  QEqWS<T> w;
  QEqParams P;
  int nf;
  int N;
  long long Pn;
  const long long* pairs;
  const T* pos;
  const T* box;
  const T* C;
  int nc;
  cudaStream_t st;
};

// Hv = H v (Hv zeroed, sums of v already in sc); optional double copy.
template <typename T>
static int qeq_matvec(QEqCtx<T>& c, const T* v, T* Hv, double* hv_out) {
  const Batch& b = c.w.plan.b;
  if (c.P.flags & ADMP_QEQ_KSPACE) {
    int s = launch_recip_potential<T>(c.w.plan, c.pos, c.box, v, c.w.mesh, c.w.spec, c.w.acc, c.P.ke, Hv, c.st,
                                      nullptr, c.w.green);
    if (s) return s;
  }
  if (c.Pn > 0 && (c.P.flags & (ADMP_QEQ_RSPACE | ADMP_QEQ_DAMPING))) {
    long long blocks = (c.Pn + 511) / 512;  // about half of a full list's pairs are kept
    if (blocks > 4096) blocks = 4096;
    qeq_coo_spmv_kernel<T><<<(unsigned)blocks, 256, 0, c.st>>>(c.w.list, v, Hv, c.w.sc, c.N, c.nf);
  }
  qeq_finish_kernel<T><<<b.nblk_atom, 256, 0, c.st>>>(b, c.P, v, Hv, c.w.diag, c.w.zc, c.C, (long long)c.N,
                                                     c.w.sc, hv_out);
  ADMP_CUDA_TRY(cudaGetLastError());
  return ADMP_OK;
}

// Set-up of the persistent solve (qeq_cg.cuh) of one system: false where its
// line buffers do not fit a block's shared memory, and where it is too large.
//
// One block an SM hides less latency than the kernels of the multi-launch loop,
// which pays off while launches and short kernels bound an iteration.  A solve
// (ms, this / the loop) of 10,701 atoms, 64^3: 1.3 / 3.0 (FP32), 2.0 / 3.5 (FP64);
// 42,000, 100^3: 3.4 / 4.4, 6.0 / 8.0; 90,000, 128^3: 7.7 / 8.4, 15.1 / 16.9;
// 120,000, 144^3: 11.5 / 11.3, 21.0 / 21.3, 142^3: 14.4 / 15.4, 29.3 / 29.7;
// 180,000, 160^3: 20.3 / 17.5, 33.6 / 31.5; 300,000, 192^3: 35.1 / 26.7, 61.4 / 53.5.
//
// The pairs are a quarter of the warps' work, at four entries a lane, and fall
// behind the mesh once their list outgrows the L2 (listed pairs; half of a full
// list has scale 0 and is dropped).  8.0 M, 10,701 atoms at 12 A: 2.8 / 3.1, 3.9 /
// 4.0; 9.1 M, 30,000 at 9 A: 4.4 / 4.6, 7.0 / 6.8; 12 M, 40,000 at 9 A: 5.9 / 5.2,
// 10.2 / 7.7; 29 M, 40,000 at 12 A: 14.4 / 6.7, 20.0 / 9.1.  Without a mesh, 20,000
// atoms 0.43 / 0.47, 0.53 / 0.50; 60,000 0.76 / 0.64, 0.95 / 0.70; 140,000 1.53 /
// 0.99, 2.37 / 1.18.
constexpr long long kCgMesh = 3000000, kCgPairs = 10000000;
constexpr int kCgAtoms = 150000, kCgAtomsNoMesh = 20000;
template <typename T>
static bool cg_plan(const QEqCtx<T>& c, int sms, CgArgs<T>& a, size_t& smem) {
  const SysDesc& d = c.w.plan.hs[0];
  const bool mesh = (c.P.flags & ADMP_QEQ_KSPACE) != 0;
  if (c.N > (mesh ? kCgAtoms : kCgAtomsNoMesh) || c.Pn > kCgPairs) return false;
  if (mesh && (long long)d.K0 * d.K1 * d.K2 > kCgMesh) return false;
  const size_t budget = 200 * 1024, cs = sizeof(Cplx<T>);
  const int cap = (int)(64 * 1024 / cs);  // complex values in a line buffer
  a.N = c.N;
  a.K0 = d.K0;
  a.K1 = d.K1;
  a.K2 = d.K2;
  a.buf = a.planes = 0;
  a.lz = a.ly = a.lx = 1;
  if (mesh) {
    auto lines = [&](long long total, int K) {
      int most = cap / K < kCgMaxLines ? cap / K : kCgMaxLines;
      most = most < 1 ? 1 : most;
      const long long rounds = (total + (long long)sms * most - 1) / ((long long)sms * most);
      return (int)((total + sms * rounds - 1) / (sms * rounds));
    };
    a.lz = lines(((long long)a.K0 * a.K1 + 1) / 2, a.K2);
    a.ly = lines((long long)a.K0 * d.K2h, a.K1);
    a.lx = lines((long long)a.K1 * d.K2h, a.K0);
    const int plane = slab_plane_elems(a.K1, a.K2);
    a.planes = a.K0 <= sms && plane <= kCgPlane;
    a.buf = a.lz * a.K2 > a.ly * a.K1 ? a.lz * a.K2 : a.ly * a.K1;
    if (a.planes) a.buf = plane;
    a.buf = a.buf > a.lx * a.K0 ? a.buf : a.lx * a.K0;
  }
  const size_t fft = ((size_t)a.K0 + a.K1 + a.K2 + 2 * (size_t)a.buf) * cs;
  const size_t st = (WarpStencil<T, false>::bytes() + 15) / 16 * 16 * kCgWarps;
  // the smallest group that still gives every warp one at most; eight atoms above that
  a.group = kPw;
  for (int s = 2; s < kPw; s <<= 1)
    if ((c.N + s - 1) / s <= sms * kCgWarps) {
      a.group = s;
      break;
    }
  const int groups = (c.N + a.group - 1) / a.group, per_warp = (groups + sms * kCgWarps - 1) / (sms * kCgWarps);
  a.kept = fft + st * per_warp <= budget ? per_warp : 0;
  smem = fft + st * (a.kept ? a.kept : 1);
  return smem <= budget;
}

// The CG iterations by the persistent kernel; `used` is false (and nothing
// launched) where the multi-kernel loop has to take the solve.
template <typename T>
static int cg_persistent(QEqCtx<T>& c, CGScal* h, bool& used) {
  used = false;
  if (c.nf != 1) return ADMP_OK;
  int dev = 0, sms = 0, coop = 0;
  ADMP_CUDA_TRY(cudaGetDevice(&dev));
  ADMP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  ADMP_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  CgArgs<T> a{};
  size_t smem = 0;
  if (!coop || !cg_plan<T>(c, sms, a, smem)) return ADMP_OK;
  ADMP_CUDA_TRY(ensure_smem(qeq_cg_kernel<T>, smem));
  int per_sm = 0;
  ADMP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, qeq_cg_kernel<T>, kCgThreads, smem));
  if (per_sm < 1) return ADMP_OK;
  a.kappa = c.w.plan.hs[0].kappa;
  a.P = c.P;
  a.pos = c.pos;
  a.box = c.box;
  a.C = c.C;
  a.green = c.w.green;
  a.diag = c.w.diag;
  a.zc = c.w.zc;
  a.chi = c.w.chi_eff;
  a.mesh = c.w.mesh;
  a.p = c.w.p;
  a.Hp = c.w.Hp;
  a.spec = c.w.spec;
  a.x = c.w.x;
  a.r = c.w.r;
  a.list = c.w.list;
  a.have_pairs = c.Pn > 0 && (c.P.flags & (ADMP_QEQ_RSPACE | ADMP_QEQ_DAMPING));
  a.sc = c.w.sc;
  a.sh = c.w.cg;
  used = true;
  if (c.P.flags & ADMP_QEQ_KSPACE)
    ADMP_CUDA_TRY(cudaMemsetAsync(c.w.mesh, 0, sizeof(T) * (size_t)a.K0 * a.K1 * a.K2, c.st));
  ADMP_CUDA_TRY(cudaMemsetAsync(c.w.cg, 0, sizeof(CgShared), c.st));
  for (a.k0 = 0;; a.k0 = h->iter) {
    a.k1 = a.k0 + kCgLaunch;
    a.init = a.k0 == 0;
    if (a.k0) ADMP_CUDA_TRY(cudaMemsetAsync(&c.w.cg->arrived, 0, sizeof(unsigned), c.st));
    void* args[] = {&a};
    std::lock_guard<std::mutex> alone(grid_mutex(dev));
    ADMP_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)qeq_cg_kernel<T>, dim3(sms), dim3(kCgThreads), args, smem,
                                              c.st));
    count_launches(1);
    const void* p = read_back(c.w.sc, sizeof(CGScal), c.st);
    if (!p) return ADMP_ERR_CUDA;
    *h = *(const CGScal*)p;
    // another status is not the end: a singular Gram matrix left one, and the solve's own verdict replaces it
    if (h->done || h->status == ADMP_ERR_CUDA || h->iter >= c.P.max_iter + kCgLaunch) return ADMP_OK;
  }
}

template <typename T>
static int qeq_prepare(QEqCtx<T>& c, const T* chi, const T* hard, const T* eta, const T* shift, const T* ds,
                       const T* bs, double kappa) {
  const Batch& b = c.w.plan.b;
  ADMP_CUDA_TRY(cudaMemsetAsync(c.w.sc, 0, sizeof(CGScal) * c.nf, c.st));
  ADMP_CUDA_TRY(cudaMemsetAsync(c.w.Hp, 0, sizeof(T) * c.N * (size_t)c.nf, c.st));
  qeq_setup_kernel<T><<<b.nblk_atom, 256, 0, c.st>>>(b, c.P, c.pos, c.box, chi, hard, eta, shift, c.w.diag, c.w.zc,
                                                    c.w.chi_eff, c.w.sc);
  if (c.P.flags & ADMP_QEQ_KSPACE) {
    int s = launch_green_build<T>(c.w.plan, c.box, c.w.green, c.P.ke, c.st);
    if (s) return s;
  }
  if (c.nc > 0) {
    qeq_gram_kernel<T><<<b.nblk_atom, 256, 0, c.st>>>(b, c.nc, c.C, (long long)c.N, c.w.sc);
    qeq_gram_invert_kernel<<<(c.nf + 31) / 32, 32, 0, c.st>>>(b, c.nc, c.w.sc);
  }
  if (c.Pn > 0 && (c.P.flags & (ADMP_QEQ_RSPACE | ADMP_QEQ_DAMPING))) {
    DevError* err = scratch_error(c.st);
    long long blocks = (c.Pn + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    ADMP_CUDA_TRY(cudaMemsetAsync(c.w.list.n, 0, sizeof(*c.w.list.n), c.st));
    qeq_pair_coef_kernel<T><<<(unsigned)blocks, 256, 0, c.st>>>(c.N * c.nf, c.Pn, c.P.flags, kappa, c.P.ke, c.pairs,
                                                                ds, bs, eta, c.w.list, err);
  }
  ADMP_CUDA_TRY(cudaGetLastError());
  return ADMP_OK;
}

template <typename T>
static int qeq_solve_impl(int flags, int nf, int N, const int* kmesh, const T* pos, const T* box, long long Pn,
                          const long long* pairs, const T* ds, const T* bs, const T* chi, const T* hard, const T* eta,
                          const T* shift, double kappa, double ke, int nc, const T* C, const double* bvals, T* q,
                          double tol, int max_iter, int* iters, double* resid, void* ws, size_t bytes,
                          cudaStream_t st) {
  QEqCtx<T> c;
  int s = qeq_carve<T>(c.w, ws, bytes, nf, N, Pn, kmesh, kappa, flags);
  if (s) return s;
  if (!ws || c.w.bytes > bytes) return fail(ADMP_ERR_WORKSPACE, "qeq workspace: need %zu bytes, got %zu", c.w.bytes, bytes);
  s = bind_plan<T>(c.w.plan, c.w.table, st);
  if (s) return s;
  c.P.flags = flags;
  c.P.axis = (flags >> 8) & 3;
  c.P.max_iter = max_iter;
  c.P.tol = tol;
  c.P.ke = ke;
  c.nf = nf;
  c.N = N;
  c.Pn = Pn;
  c.pairs = pairs;
  c.pos = pos;
  c.box = box;
  c.C = C;
  c.nc = nc;
  c.st = st;
  const Batch& b = c.w.plan.b;
  const long long NT = (long long)nf * N;
  const int sb = (nf + 63) / 64;
  s = qeq_prepare<T>(c, chi, hard, eta, shift, ds, bs, kappa);
  if (s) return s;
  double bv[4] = {0, 0, 0, 0};
  const bool dev_b = (flags & ADMP_QEQ_DEVICE_B) != 0;
  for (int k = 0; k < nc && !dev_b; ++k) bv[k] = bvals[k];
  qeq_set_b_kernel<<<sb, 64, 0, st>>>(nf, c.w.sc, nc, bv[0], bv[1], bv[2], bv[3], dev_b ? bvals : nullptr);
  // x0 (optionally projected onto C x = b)
  const int cb = (int)((NT + 255) / 256 < 2048 ? (NT + 255) / 256 : 2048);
  cast_kernel<T><<<cb > 0 ? cb : 1, 256, 0, st>>>(NT, q, c.w.x);
  if ((flags & ADMP_QEQ_PROJECT_Q0) && nc > 0) {
    qeq_sums_kernel<T, double><<<b.nblk_atom, 256, 0, st>>>(b, c.w.x, c.w.zc, C, (long long)N, nc, 1, c.w.sc, nullptr,
                                                            nullptr);
    qeq_project_kernel<T><<<b.nblk_atom, 256, 0, st>>>(b, c.w.x, C, (long long)N, c.w.sc);
    qeq_clear_acc_kernel<<<sb, 64, 0, st>>>(nf, c.w.sc);
  }
  std::vector<CGScal> h(nf);
  bool persistent = false;
  s = cg_persistent<T>(c, h.data(), persistent);
  if (s) return s;
  if (!persistent) {
    // H x0 -> hx (double); the p buffer carries x0 in T for the matvec
    qeq_sums_kernel<T, double><<<b.nblk_atom, 256, 0, st>>>(b, c.w.x, c.w.zc, C, (long long)N, nc, 0, c.w.sc, c.w.Hp,
                                                            c.w.p);
    s = qeq_matvec<T>(c, c.w.p, c.w.Hp, c.w.hx);
    if (s) return s;
    qeq_clear_acc_kernel<<<sb, 64, 0, st>>>(nf, c.w.sc);
    ADMP_CUDA_TRY(cudaMemsetAsync(c.w.Hp, 0, sizeof(T) * NT, st));
    qeq_resid_kernel<T><<<b.nblk_atom, 256, 0, st>>>(b, c.w.hx, c.w.chi_eff, C, (long long)N, c.w.zc, c.w.r, c.w.p,
                                                     c.w.sc, 0);
    qeq_resid_kernel<T><<<b.nblk_atom, 256, 0, st>>>(b, c.w.hx, c.w.chi_eff, C, (long long)N, c.w.zc, c.w.r, c.w.p,
                                                     c.w.sc, 1);
    qeq_init_done_kernel<<<(nf + 31) / 32, 32, 0, st>>>(b, c.P, c.w.sc);
    ADMP_CUDA_TRY(cudaGetLastError());
    // iterate; read the per-frame done flags every `chunk` iterations
    RecipPlan<T> pl = c.w.plan;
    pl.b.done = &c.w.sc->done;
    pl.b.done_stride = (int)(sizeof(CGScal) / sizeof(int));
    pl.b.status_off = (int)((offsetof(CGScal, status) - offsetof(CGScal, done)) / sizeof(int));
    c.w.plan = pl;
  }
  const int chunk = 8;
  int it = 0;
  while (!persistent) {
    for (int k = 0; k < chunk; ++k) {
      qeq_rotate_kernel<<<(nf + 31) / 32, 32, 0, st>>>(b, c.w.sc);
      s = qeq_matvec<T>(c, c.w.p, c.w.Hp, nullptr);
      if (s) return s;
      qeq_update_kernel<T><<<b.nblk_atom, 256, 0, st>>>(b, c.w.x, c.w.r, c.w.p, c.w.Hp, C, (long long)N, c.w.sc);
      qeq_direction_kernel<T><<<b.nblk_atom, 256, 0, st>>>(b, c.P, c.w.r, c.w.p, c.w.zc, c.w.sc);
    }
    ADMP_CUDA_TRY(cudaGetLastError());
    it += chunk;
    ADMP_CUDA_TRY(cudaMemcpyAsync(h.data(), c.w.sc, sizeof(CGScal) * nf, cudaMemcpyDeviceToHost, st));
    ADMP_CUDA_TRY(cudaStreamSynchronize(st));
    bool all = true;
    for (int f = 0; f < nf; ++f) all = all && h[f].done;
    if (all || it > max_iter + chunk) break;
  }
  cast_back_kernel<T><<<cb > 0 ? cb : 1, 256, 0, st>>>(NT, c.w.x, q);
  ADMP_CUDA_TRY(cudaGetLastError());
  int worst = ADMP_OK, worst_f = 0;
  for (int f = 0; f < nf; ++f) {
    if (iters) iters[f] = h[f].iter;
    if (resid) resid[f] = sqrt(h[f].rr_new > 0 ? h[f].rr_new : h[f].rr) / (N > 0 ? N : 1);
    const int stf = h[f].done || h[f].status == ADMP_ERR_CUDA ? h[f].status : ADMP_ERR_NOT_CONVERGED;
    if (stf && (worst == ADMP_OK || worst == ADMP_ERR_NOT_CONVERGED)) {
      worst = stf;
      worst_f = f;
    }
  }
  DevError* err = scratch_error(st);
  int e = err ? check_error(err, st) : ADMP_OK;
  if (e) return e;
  if (worst == ADMP_ERR_NOT_CONVERGED)
    return fail(ADMP_ERR_NOT_CONVERGED, "QEq CG did not converge in %d iterations (frame %d, residual %g)",
                h[worst_f].iter, worst_f, sqrt(h[worst_f].rr_new > 0 ? h[worst_f].rr_new : h[worst_f].rr) / N);
  if (worst) return fail(worst, "QEq solve failed (frame %d, status %d)", worst_f, worst);
  return ADMP_OK;
}

template <typename T>
static int qeq_hvp_impl(int flags, int nf, int N, const int* kmesh, const T* pos, const T* box, long long Pn,
                        const long long* pairs, const T* ds, const T* bs, const T* hard, const T* eta, double kappa,
                        double ke, const T* p, T* out, void* ws, size_t bytes, cudaStream_t st) {
  QEqCtx<T> c;
  int s = qeq_carve<T>(c.w, ws, bytes, nf, N, Pn, kmesh, kappa, flags);
  if (s) return s;
  if (!ws || c.w.bytes > bytes) return fail(ADMP_ERR_WORKSPACE, "qeq workspace: need %zu bytes, got %zu", c.w.bytes, bytes);
  s = bind_plan<T>(c.w.plan, c.w.table, st);
  if (s) return s;
  c.nf = nf;
  c.P.flags = flags;
  c.P.axis = (flags >> 8) & 3;
  c.P.max_iter = 0;
  c.P.tol = 0;
  c.P.ke = ke;
  c.N = N;
  c.Pn = Pn;
  c.pairs = pairs;
  c.pos = pos;
  c.box = box;
  c.C = nullptr;
  c.nc = 0;
  c.st = st;
  const Batch& b = c.w.plan.b;
  s = qeq_prepare<T>(c, nullptr, hard, eta, nullptr, ds, bs, kappa);
  if (s) return s;
  qeq_sums_kernel<T, T><<<b.nblk_atom, 256, 0, st>>>(b, p, c.w.zc, nullptr, (long long)N, 0, 0, c.w.sc, c.w.Hp,
                                                     nullptr);
  s = qeq_matvec<T>(c, p, c.w.Hp, nullptr);
  if (s) return s;
  ADMP_CUDA_TRY(cudaMemcpyAsync(out, c.w.Hp, sizeof(T) * N * (size_t)nf, cudaMemcpyDeviceToDevice, st));
  DevError* err = scratch_error(st);
  return err ? check_error(err, st) : ADMP_OK;
}

// ------------------------------------------------------------ dense Hessian
template <typename T>
struct HessWS {
  RecipPlan<T> one, unit, all;  // geometry, one atom per column, all atoms per column
  SysDesc *t_one, *t_unit, *t_all;
  T *mesh, *green, *rep, *ones;
  Cplx<T>* spec;
  double *acc, *diag, *zc, *chi;
  PairList<T> list;
  CGScal* sc;
  size_t bytes;
};

template <typename T>
static int hess_plan(RecipPlan<T>& p, int n, int natoms, int stride, const int* K, double kappa) {
  SysSpec sys[kMaxBatch];
  for (int c = 0; c < n; ++c) {
    sys[c].natoms = natoms;
    sys[c].atom_off = c * stride;
    for (int d = 0; d < 3; ++d) sys[c].K[d] = K[d];
    sys[c].kappa = kappa;
    sys[c].box_idx = 0;
    sys[c].green_off = 0;
  }
  return build_recip_plan<T>(sys, n, p);
}

template <typename T>
static int hess_carve(HessWS<T>& w, void* ws, size_t bytes, int N, long long P, const int* kmesh, double kappa,
                      int flags, int cols) {
  const int one[3] = {1, 1, 1};
  const int* K = (flags & ADMP_QEQ_KSPACE) ? kmesh : one;
  int s = hess_plan<T>(w.one, 1, N, 0, K, kappa);
  if (!s) s = hess_plan<T>(w.unit, cols, 1, 1, K, kappa);
  if (!s) s = hess_plan<T>(w.all, cols, N, N, K, kappa);
  if (s) return s;
  const bool ks = (flags & ADMP_QEQ_KSPACE) != 0;
  Carver c(ws, bytes);
  w.t_one = reinterpret_cast<SysDesc*>(c.take<unsigned char>(sys_table_bytes()));
  w.t_unit = reinterpret_cast<SysDesc*>(c.take<unsigned char>(sys_table_bytes()));
  w.t_all = reinterpret_cast<SysDesc*>(c.take<unsigned char>(sys_table_bytes()));
  w.mesh = c.take<T>(ks ? w.all.mesh_elems : 0);
  w.spec = c.take<Cplx<T>>(ks ? w.all.spec_elems : 0);
  w.green = c.take<T>(ks ? w.one.spec_elems : 0);
  w.rep = c.take<T>(ks ? 3 * (size_t)N * cols : 0);
  w.ones = c.take<T>(cols);
  w.acc = c.take<double>((size_t)kAccStride * cols);
  w.diag = c.take<double>(N);
  w.zc = c.take<double>(N);
  w.chi = c.take<double>(N);
  w.list.ij = c.take<int2>(P > 0 ? P : 0);
  w.list.coef = c.take<T>(P > 0 ? P : 0);
  w.list.n = c.take<unsigned long long>(1);
  w.sc = c.take<CGScal>(1);
  w.bytes = c.off;
  return ADMP_OK;
}

template <typename T>
static int qeq_hessian_impl(int flags, int N, const int* kmesh, const T* pos, const T* box, long long Pn,
                            const long long* pairs, const T* ds, const T* bs, const T* hard, const T* eta, double kappa,
                            double ke, int cols, T* H, void* ws, size_t bytes, cudaStream_t st) {
  HessWS<T> w;
  int s = hess_carve<T>(w, ws, bytes, N, Pn, kmesh, kappa > 0 ? kappa : 1.0, flags, cols);
  if (s) return s;
  if (!ws || w.bytes > bytes) return fail(ADMP_ERR_WORKSPACE, "Hessian workspace: need %zu bytes, got %zu", w.bytes, bytes);
  QEqParams P{flags, (flags >> 8) & 3, 0, 0.0, ke};
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  ADMP_CUDA_TRY(cudaMemsetAsync(w.sc, 0, sizeof(CGScal), st));
  ADMP_CUDA_TRY(cudaMemsetAsync(H, 0, sizeof(T) * (size_t)N * N, st));
  s = bind_plan<T>(w.one, w.t_one, st);
  if (s) return s;
  qeq_setup_kernel<T><<<w.one.b.nblk_atom, 256, 0, st>>>(w.one.b, P, pos, box, (const T*)nullptr, hard, eta,
                                                         (const T*)nullptr, w.diag, w.zc, w.chi, w.sc);
  const bool pair = Pn > 0 && (flags & (ADMP_QEQ_RSPACE | ADMP_QEQ_DAMPING));
  if (pair) {
    long long blocks = (Pn + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    ADMP_CUDA_TRY(cudaMemsetAsync(w.list.n, 0, sizeof(*w.list.n), st));
    qeq_pair_coef_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(N, Pn, flags, kappa, ke, pairs, ds, bs, eta, w.list, err);
    s = probe_error(err, st);
    if (s) return s;
  }
  if (flags & ADMP_QEQ_KSPACE) {
    s = launch_green_build<T>(w.one, box, w.green, ke, st);
    if (s) return s;
    const long long rep = 3LL * N * cols;
    hess_repeat_kernel<T><<<(unsigned)((rep + 255) / 256), 256, 0, st>>>(N, cols, pos, w.rep, w.ones);
    for (int c0 = 0; c0 < N; c0 += cols) {
      const int n = N - c0 < cols ? N - c0 : cols;
      if (c0 == 0 || n != cols) {
        if (n != cols) {  // the last columns
          s = hess_plan<T>(w.unit, n, 1, 1, kmesh, kappa);
          if (!s) s = hess_plan<T>(w.all, n, N, N, kmesh, kappa);
          if (s) return s;
        }
        s = bind_plan<T>(w.unit, w.t_unit, st);
        if (!s) s = bind_plan<T>(w.all, w.t_all, st);
        if (s) return s;
      }
      ADMP_CUDA_TRY(cudaMemsetAsync(w.mesh, 0, w.all.mesh_elems * sizeof(T), st));
      s = launch_spread<T>(w.unit, pos + 3 * (size_t)c0, box, w.ones, w.mesh, nullptr, st);
      if (!s) s = launch_fft_green<T>(w.all, w.mesh, w.spec, box, w.acc, ke, st, w.green);
      if (!s)
        s = launch_gather<T, false>(w.all, w.rep, box, w.ones, w.mesh, H + (size_t)c0 * N, nullptr, w.acc, nullptr, st);
      if (s) return s;
    }
  }
  if (pair) {
    long long blocks = (Pn + 511) / 512;
    if (blocks > 4096) blocks = 4096;
    hess_pairs_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(w.list, N, H);
  }
  const int tiles = (N + 15) / 16;
  hess_finish_kernel<T><<<dim3(tiles, tiles), 256, 0, st>>>(N, P, w.diag, w.zc, w.sc, H);
  ADMP_CUDA_TRY(cudaGetLastError());
  return pair ? probed_error(err, st) : ADMP_OK;
}

}  // namespace admp

using namespace admp;

static size_t qeq_ws_bytes(int dtype, int nframes, int natoms, long long npairs, const int* kmesh) {
  if (nframes <= 0 || nframes > kMaxBatch || natoms <= 0) return 0;
  std::vector<int> K(3 * (size_t)nframes, 1);
  if (kmesh)
    for (size_t k = 0; k < K.size(); ++k) K[k] = kmesh[k];
  const int fl = kmesh ? ADMP_QEQ_KSPACE : 0;
  if (dtype == ADMP_F32) {
    QEqWS<float> w;
    return qeq_carve<float>(w, nullptr, 0, nframes, natoms, npairs, K.data(), 1.0, fl) ? 0 : w.bytes;
  }
  QEqWS<double> w;
  return qeq_carve<double>(w, nullptr, 0, nframes, natoms, npairs, K.data(), 1.0, fl) ? 0 : w.bytes;
}

extern "C" size_t admp_qeq_workspace_size(int dtype, int natoms, long long npairs, const int* kmesh, int n_const) {
  (void)n_const;
  return qeq_ws_bytes(dtype, 1, natoms, npairs, kmesh);
}

extern "C" size_t admp_qeq_frames_workspace_size(int dtype, int nframes, int natoms, long long npairs,
                                                 const int* kmesh, int n_const) {
  (void)n_const;
  return qeq_ws_bytes(dtype, nframes, natoms, npairs, kmesh);
}

extern "C" int admp_qeq_solve_frames(int dtype, int flags, int nframes, int natoms, const int* kmesh, const void* pos,
                                     const void* box, long long npairs, const long long* pairs, const void* ds,
                                     const void* buffer_scales, const void* chi, const void* hardness,
                                     const void* eta, const void* rhs_shift, double kappa, double ke, int n_const,
                                     const void* C, const double* b, void* q, double tol, int max_iter, int* iters,
                                     double* resid, void* workspace, size_t workspace_bytes, void* stream) {
  if (nframes <= 0 || nframes > kMaxBatch)
    return fail(ADMP_ERR_BAD_ARG, "admp_qeq_solve: %d frames (1..%d)", nframes, kMaxBatch);
  if (natoms <= 0 || !pos || !box || !hardness || !q) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_solve: args");
  if (n_const < 0 || n_const > kMaxConst || (n_const > 0 && (!C || !b)))
    return fail(ADMP_ERR_BAD_ARG, "admp_qeq_solve: n_const must be in [0, %d] with C and b", kMaxConst);
  if ((flags & ADMP_QEQ_KSPACE) && (!kmesh || !(kappa > 0))) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_solve: kspace needs kmesh and kappa");
  if ((flags & ADMP_QEQ_DAMPING) && !eta) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_solve: damping needs eta");
  if (npairs > 0 && (!pairs || !ds || !buffer_scales)) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_solve: pairs");
  std::vector<int> K(3 * (size_t)nframes, 1);
  if (flags & ADMP_QEQ_KSPACE)
    for (size_t k = 0; k < K.size(); ++k) K[k] = kmesh[k];
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return qeq_solve_impl<double>(flags, nframes, natoms, K.data(), (const double*)pos, (const double*)box, npairs,
                                  pairs, (const double*)ds, (const double*)buffer_scales, (const double*)chi,
                                  (const double*)hardness, (const double*)eta, (const double*)rhs_shift, kappa, ke,
                                  n_const, (const double*)C, b, (double*)q, tol, max_iter, iters, resid, workspace,
                                  workspace_bytes, st);
  if (dtype == ADMP_F32)
    return qeq_solve_impl<float>(flags, nframes, natoms, K.data(), (const float*)pos, (const float*)box, npairs, pairs,
                                 (const float*)ds, (const float*)buffer_scales, (const float*)chi,
                                 (const float*)hardness, (const float*)eta, (const float*)rhs_shift, kappa, ke,
                                 n_const, (const float*)C, b, (float*)q, tol, max_iter, iters, resid, workspace,
                                 workspace_bytes, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_qeq_solve(int dtype, int flags, int natoms, const int* kmesh, const void* pos, const void* box,
                              long long npairs, const long long* pairs, const void* ds, const void* buffer_scales,
                              const void* chi, const void* hardness, const void* eta, const void* rhs_shift,
                              double kappa, double ke, int n_const, const void* C, const double* b, void* q,
                              double tol, int max_iter, int* iters, double* resid, void* workspace,
                              size_t workspace_bytes, void* stream) {
  return admp_qeq_solve_frames(dtype, flags, 1, natoms, kmesh, pos, box, npairs, pairs, ds, buffer_scales, chi,
                               hardness, eta, rhs_shift, kappa, ke, n_const, C, b, q, tol, max_iter, iters, resid,
                               workspace, workspace_bytes, stream);
}

extern "C" int admp_qeq_hvp_frames(int dtype, int flags, int nframes, int natoms, const int* kmesh, const void* pos,
                                   const void* box, long long npairs, const long long* pairs, const void* ds,
                                   const void* buffer_scales, const void* hardness, const void* eta, double kappa,
                                   double ke, const void* p, void* out, void* workspace, size_t workspace_bytes,
                                   void* stream) {
  if (nframes <= 0 || nframes > kMaxBatch)
    return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hvp: %d frames (1..%d)", nframes, kMaxBatch);
  if (natoms <= 0 || !pos || !box || !hardness || !p || !out) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hvp: args");
  if ((flags & ADMP_QEQ_KSPACE) && (!kmesh || !(kappa > 0))) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hvp: kspace needs kmesh and kappa");
  if ((flags & ADMP_QEQ_DAMPING) && !eta) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hvp: damping needs eta");
  if (npairs > 0 && (!pairs || !ds || !buffer_scales)) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hvp: pairs");
  std::vector<int> K(3 * (size_t)nframes, 1);
  if (flags & ADMP_QEQ_KSPACE)
    for (size_t k = 0; k < K.size(); ++k) K[k] = kmesh[k];
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return qeq_hvp_impl<double>(flags, nframes, natoms, K.data(), (const double*)pos, (const double*)box, npairs,
                                pairs, (const double*)ds, (const double*)buffer_scales, (const double*)hardness,
                                (const double*)eta, kappa, ke, (const double*)p, (double*)out, workspace,
                                workspace_bytes, st);
  if (dtype == ADMP_F32)
    return qeq_hvp_impl<float>(flags, nframes, natoms, K.data(), (const float*)pos, (const float*)box, npairs, pairs,
                               (const float*)ds, (const float*)buffer_scales, (const float*)hardness,
                               (const float*)eta, kappa, ke, (const float*)p, (float*)out, workspace, workspace_bytes,
                               st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_qeq_hvp(int dtype, int flags, int natoms, const int* kmesh, const void* pos, const void* box,
                            long long npairs, const long long* pairs, const void* ds, const void* buffer_scales,
                            const void* hardness, const void* eta, double kappa, double ke, const void* p, void* out,
                            void* workspace, size_t workspace_bytes, void* stream) {
  return admp_qeq_hvp_frames(dtype, flags, 1, natoms, kmesh, pos, box, npairs, pairs, ds, buffer_scales, hardness,
                             eta, kappa, ke, p, out, workspace, workspace_bytes, stream);
}

extern "C" size_t admp_qeq_hessian_workspace_size(int dtype, int natoms, long long npairs, const int* kmesh, int cols) {
  if (natoms <= 0 || cols <= 0 || cols > kMaxBatch) return 0;
  const int fl = kmesh ? ADMP_QEQ_KSPACE : 0;
  if (dtype == ADMP_F32) {
    HessWS<float> w;
    return hess_carve<float>(w, nullptr, 0, natoms, npairs, kmesh, 1.0, fl, cols) ? 0 : w.bytes;
  }
  HessWS<double> w;
  return hess_carve<double>(w, nullptr, 0, natoms, npairs, kmesh, 1.0, fl, cols) ? 0 : w.bytes;
}

extern "C" int admp_qeq_hessian(int dtype, int flags, int natoms, const int* kmesh, const void* pos, const void* box,
                                long long npairs, const long long* pairs, const void* ds, const void* buffer_scales,
                                const void* hardness, const void* eta, double kappa, double ke, int cols, void* H,
                                void* workspace, size_t workspace_bytes, void* stream) {
  if (natoms <= 0 || cols <= 0 || cols > kMaxBatch || !pos || !box || !hardness || !H)
    return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hessian: args");
  if ((flags & ADMP_QEQ_KSPACE) && (!kmesh || !(kappa > 0))) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hessian: kspace needs kmesh and kappa");
  if ((flags & ADMP_QEQ_DAMPING) && !eta) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hessian: damping needs eta");
  if (npairs > 0 && (!pairs || !ds || !buffer_scales)) return fail(ADMP_ERR_BAD_ARG, "admp_qeq_hessian: pairs");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return qeq_hessian_impl<double>(flags, natoms, kmesh, (const double*)pos, (const double*)box, npairs, pairs,
                                    (const double*)ds, (const double*)buffer_scales, (const double*)hardness,
                                    (const double*)eta, kappa, ke, cols, (double*)H, workspace, workspace_bytes, st);
  if (dtype == ADMP_F32)
    return qeq_hessian_impl<float>(flags, natoms, kmesh, (const float*)pos, (const float*)box, npairs, pairs,
                                   (const float*)ds, (const float*)buffer_scales, (const float*)hardness,
                                   (const float*)eta, kappa, ke, cols, (float*)H, workspace, workspace_bytes, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}
