// admp_pme_recip: reciprocal-space PME energy and gradients for nframes
// systems (CoulombForceModule._forward_pbc_reciprocal, pme.py:351-446, and
// the autograd backward through spread_charges / setup_kpts, recip.py).
#include <string.h>

#include "pair_terms.h"
#include "pme_host.h"

namespace admp {

template <typename T>
static int recip_chunk_plan(int c0, int nsys, int N, const int* kmesh, double kappa, RecipPlan<T>& p) {
  SysSpec sys[kMaxBatch];
  for (int s = 0; s < nsys; ++s) {
    sys[s].natoms = N;
    sys[s].atom_off = s * N;
    for (int d = 0; d < 3; ++d) sys[s].K[d] = kmesh[3 * (c0 + s) + d];
    sys[s].kappa = kappa;
    sys[s].box_idx = s;
  }
  return build_recip_plan<T>(sys, nsys, p);
}

template <typename T>
static size_t recip_ws_bytes(size_t mesh_elems, size_t spec_elems, int nsys) {
  Carver c(nullptr, 0);
  c.take<unsigned char>(sys_table_bytes());
  c.take<T>(mesh_elems);
  c.take<Cplx<T>>(spec_elems);
  c.take<double>((size_t)nsys * kAccStride);
  return c.off;
}

// Workspace of the largest chunk, from the mesh sizes alone (as build_recip_plan
// lays the meshes out; every mesh within its range fits the passes).
template <typename T>
static int recip_ws_size(int nf, const int* kmesh, size_t* out) {
  size_t best = 0;
  for (int c0 = 0; c0 < nf; c0 += kMaxBatch) {
    const int ns = nf - c0 < kMaxBatch ? nf - c0 : kMaxBatch;
    size_t mesh = 0, spec = 0;
    for (int s = 0; s < ns; ++s) {
      const int* K = kmesh + 3 * (c0 + s);
      for (int d = 0; d < 3; ++d)
        if (K[d] <= 0 || K[d] > kMaxMesh) return fail(ADMP_ERR_MESH, "mesh size %d out of range [1, %d]", K[d], kMaxMesh);
      mesh += mesh_elems_of(K);
      spec += spec_elems_of(K);
    }
    const size_t b = recip_ws_bytes<T>(mesh, spec, ns);
    best = b > best ? b : best;
  }
  *out = best;
  return ADMP_OK;
}

template <typename T>
static int pme_recip_impl(int nf, int N, const int* kmesh, const T* pos, const T* box, const T* q, double kappa,
                          double ke, double* energy, T* dpos, T* dq, T* dbox, void* ws, size_t bytes,
                          cudaStream_t st) {
  for (int c0 = 0; c0 < nf; c0 += kMaxBatch) {
    const int ns = nf - c0 < kMaxBatch ? nf - c0 : kMaxBatch;
    RecipPlan<T> p;
    int s = recip_chunk_plan<T>(c0, ns, N, kmesh, kappa, p);
    if (s) return s;
    Carver c(ws, bytes);
    SysDesc* table = reinterpret_cast<SysDesc*>(c.take<unsigned char>(sys_table_bytes()));
    T* mesh = c.take<T>(p.mesh_elems);
    Cplx<T>* spec = c.take<Cplx<T>>(p.spec_elems);
    double* acc = c.take<double>((size_t)ns * kAccStride);
    if (!c.ok() || !ws) return fail(ADMP_ERR_WORKSPACE, "pme_recip workspace: need %zu bytes, got %zu", c.off, bytes);
    s = bind_plan<T>(p, table, st);
    if (s) return s;
    ADMP_CUDA_TRY(cudaMemsetAsync(acc, 0, sizeof(double) * ns * kAccStride, st));
    const size_t ao = (size_t)c0 * N;
    s = launch_recip<T>(p, pos + ao * 3, box + (size_t)c0 * 9, q + ao, mesh, spec, acc, ke, dq ? dq + ao : nullptr,
                        dpos ? dpos + ao * 3 : nullptr, st, dbox != nullptr);
    if (s) return s;
    recip_finalize_kernel<T><<<(ns + 127) / 128, 128, 0, st>>>(p.b, box + (size_t)c0 * 9, acc,
                                                               energy ? energy + c0 : nullptr,
                                                               dbox ? dbox + (size_t)c0 * 9 : nullptr);
    ADMP_CUDA_TRY(cudaGetLastError());
  }
  return ADMP_OK;
}

// Real-space, reciprocal, self, non-neutral and slab energies and their
// gradients: table and zeroing, pairs, spread, three FFT passes, gather,
// finalize -- eight launches (ten where build_recip_plan splits the passes of
// few large planes in two, one more above eight systems).  Outputs are written, and the host waits only for
// the pair kernel's error word, after the rest has been launched.
template <typename T>
static int coulomb_impl(int flags, int nf, int N, const int* kmesh, const T* pos, const T* box, long long P,
                        const long long* pairs, const T* ds, const void* bs, const T* q, double kappa, double ke, T* energy,
                        double* comps, T* dpos, T* dq, T* dbox, T* dds, void* ws, size_t bytes, cudaStream_t st) {
  DevError* err = scratch_error(st);
  if (!err) return ADMP_ERR_CUDA;
  const bool pair = (flags & ADMP_QEQ_RSPACE) && P > 0;
  for (int c0 = 0; c0 < nf; c0 += kMaxBatch) {
    const int ns = nf - c0 < kMaxBatch ? nf - c0 : kMaxBatch;
    RecipPlan<T> p;
    int s = recip_chunk_plan<T>(c0, ns, N, kmesh, kappa, p);
    if (s) return s;
    Carver c(ws, bytes);
    SysDesc* table = reinterpret_cast<SysDesc*>(c.take<unsigned char>(sys_table_bytes()));
    T* mesh = c.take<T>(p.mesh_elems);
    Cplx<T>* spec = c.take<Cplx<T>>(p.spec_elems);
    double* acc = c.take<double>((size_t)ns * kAccStride);
    if (!c.ok() || !ws) return fail(ADMP_ERR_WORKSPACE, "coulomb workspace: need %zu bytes, got %zu", c.off, bytes);
    ZeroSpans z{};
    z.add(mesh, p.mesh_elems * sizeof(T));
    z.add(acc, sizeof(double) * ns * kAccStride);
    if (c0 == 0) {
      z.add(comps, sizeof(double) * 5 * nf);
      z.add(dpos, sizeof(T) * 3 * (size_t)nf * N);
      z.add(dq, sizeof(T) * (size_t)nf * N);
      if (!pair) z.add(dds, sizeof(T) * (size_t)nf * P);
    }
    s = prep_plan<T>(p, table, z, st);
    if (s) return s;
    if (c0 == 0 && pair) {
      s = launch_pair_energy<T>(ADMP_PAIR_EWALD, nf, N, P, pairs, ds, bs, (flags & ADMP_PAIR_INT64_SCALES) != 0, q,
                                nullptr, kappa, ke, comps, 5, true, dds, dq, nullptr, err, st);
      if (!s) s = probe_error(err, st);
      if (s) return s;
    }
    const size_t ao = (size_t)c0 * N;
    const TermArgs terms{kTermEwald | ((flags & ADMP_QEQ_SLAB) ? kTermSlab : 0), (flags >> 8) & 3, ke, acc};
    s = launch_recip<T>(p, pos + ao * 3, box + (size_t)c0 * 9, q + ao, mesh, spec, acc, ke, dq ? dq + ao : nullptr,
                        dpos ? dpos + ao * 3 : nullptr, st, dbox != nullptr, nullptr, terms);
    if (s) return s;
    coulomb_finalize_kernel<T><<<(ns + 127) / 128, 128, 0, st>>>(p.b, box + (size_t)c0 * 9, terms, comps + 5 * c0,
                                                                 energy + c0, dbox ? dbox + (size_t)c0 * 9 : nullptr);
    ADMP_CUDA_TRY(cudaGetLastError());
  }
  return pair ? probed_error(err, st) : ADMP_OK;
}

}  // namespace admp

using namespace admp;

extern "C" size_t admp_pme_recip_workspace_size(int dtype, int nframes, const int* kmesh) {
  if (nframes <= 0 || !kmesh) return 0;
  size_t out = 0;
  int s = dtype == ADMP_F32 ? recip_ws_size<float>(nframes, kmesh, &out) : recip_ws_size<double>(nframes, kmesh, &out);
  return s ? 0 : out;
}

extern "C" int admp_pme_recip(int dtype, int nframes, int natoms, const int* kmesh, const void* pos, const void* box,
                              const void* q, double kappa, double ke, double* energy, void* dE_dpos, void* dE_dq,
                              void* dE_dbox, void* workspace, size_t workspace_bytes, void* stream) {
  if (nframes == 0) return ADMP_OK;
  if (nframes < 0 || natoms < 0 || !kmesh || !box || !(kappa > 0)) return fail(ADMP_ERR_BAD_ARG, "admp_pme_recip: args");
  if (natoms > 0 && (!pos || !q)) return fail(ADMP_ERR_BAD_ARG, "admp_pme_recip: null pos/q");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return pme_recip_impl<double>(nframes, natoms, kmesh, (const double*)pos, (const double*)box, (const double*)q,
                                  kappa, ke, energy, (double*)dE_dpos, (double*)dE_dq, (double*)dE_dbox, workspace,
                                  workspace_bytes, st);
  if (dtype == ADMP_F32)
    return pme_recip_impl<float>(nframes, natoms, kmesh, (const float*)pos, (const float*)box, (const float*)q, kappa,
                                 ke, energy, (float*)dE_dpos, (float*)dE_dq, (float*)dE_dbox, workspace,
                                 workspace_bytes, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_coulomb_pbc(int dtype, int flags, int nframes, int natoms, const int* kmesh, const void* pos,
                                const void* box, long long npairs, const long long* pairs, const void* ds,
                                const void* buffer_scales, const void* q, double kappa, double ke, void* energy,
                                double* comps, void* dE_dpos, void* dE_dq, void* dE_dbox, void* dE_dds, void* workspace,
                                size_t workspace_bytes, void* stream) {
  if (nframes <= 0 || natoms <= 0 || npairs < 0 || !kmesh || !pos || !box || !q || !energy || !comps || !(kappa > 0))
    return fail(ADMP_ERR_BAD_ARG, "admp_coulomb_pbc: args");
  if (!(flags & ADMP_QEQ_KSPACE)) return fail(ADMP_ERR_BAD_ARG, "admp_coulomb_pbc: needs the reciprocal part");
  if (((flags >> 8) & 3) > 2) return fail(ADMP_ERR_BAD_ARG, "admp_coulomb_pbc: slab axis");
  if (npairs > 0 && (flags & ADMP_QEQ_RSPACE) && (!pairs || !ds || !buffer_scales))
    return fail(ADMP_ERR_BAD_ARG, "admp_coulomb_pbc: pairs");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == ADMP_F64)
    return coulomb_impl<double>(flags, nframes, natoms, kmesh, (const double*)pos, (const double*)box, npairs, pairs,
                                (const double*)ds, buffer_scales, (const double*)q, kappa, ke,
                                (double*)energy, comps, (double*)dE_dpos, (double*)dE_dq, (double*)dE_dbox,
                                (double*)dE_dds, workspace, workspace_bytes, st);
  if (dtype == ADMP_F32)
    return coulomb_impl<float>(flags, nframes, natoms, kmesh, (const float*)pos, (const float*)box, npairs, pairs,
                               (const float*)ds, buffer_scales, (const float*)q, kappa, ke,
                               (float*)energy, comps, (float*)dE_dpos, (float*)dE_dq, (float*)dE_dbox, (float*)dE_dds,
                               workspace, workspace_bytes, st);
  return fail(ADMP_ERR_BAD_ARG, "bad dtype");
}

extern "C" int admp_read_back(const void* dev, size_t bytes, void* host, void* stream) {
  const void* h = read_back(dev, bytes, (cudaStream_t)stream);
  if (!h) return ADMP_ERR_CUDA;
  memcpy(host, h, bytes);
  return ADMP_OK;
}
