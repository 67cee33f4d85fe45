// TorchScript-visible operators over the C ABI (torch.ops.admp_b200.*), with
// C++ autograd, so that CoulombForceModule, GaussianDampingForceModule,
// SiteForceModule and QEqForceModule can be compiled with torch.jit.script
// and saved as the reference's modules can (test_jit.py).  Every energy call
// produces the gradients the backward needs in the same launch sequence, as
// the Python autograd functions of admp_b200.ops do.
//
//   coulomb_pbc(pos, box, pairs, ds, bs, q, kappa, kmesh, spacing, ethresh,
//               ke, rspace, kspace, slab, axis) -> [E, comps, kmesh]
//                 pme.py:261-310 (real, reciprocal, self, non-neutral, slab)
//   neighbor_list(pos, box, cutoff, nframes) -> status, pairs, scales, ds
//                 nblist.py:304-445, 517-551
//   coulomb_obc(pairs, ds, bs, q, ke) -> E                     pme.py:529-561
//   damping(ds, q, eta, pairs, bs, ke) -> E                    qeq.py:60-129
//   site(q, chi, hardness) -> E                                qeq.py:159-209
//
// Inputs are in the standardised (nframes, ...) layout of BaseForceModule.
#include <ATen/cuda/CUDAContext.h>
#include <torch/library.h>
#include <torch/torch.h>

#include <cmath>
#include <vector>

#include "admp_b200.h"

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// Status -> the exception types of the Python layer (admp_b200._lib.check):
// bad arguments / mesh -> ValueError, bad index -> IndexError, else RuntimeError.
void check(int st, const char* what) {
  if (st == ADMP_OK) return;
  TORCH_CHECK_VALUE(st != ADMP_ERR_BAD_ARG && st != ADMP_ERR_MESH, what, ": ", admp_last_error_message());
  TORCH_CHECK_INDEX(st != ADMP_ERR_BAD_INDEX, what, ": ", admp_last_error_message());
  TORCH_CHECK(false, what, ": ", admp_last_error_message(), " [", admp_status_string(st), "]");
}

int dtype_code(const Tensor& t) {
  TORCH_CHECK(t.scalar_type() == torch::kDouble || t.scalar_type() == torch::kFloat,
              "admp_b200 ops take float64 or float32 tensors");
  return t.scalar_type() == torch::kDouble ? ADMP_F64 : ADMP_F32;
}

void* stream_of(const Tensor& t) {
  TORCH_CHECK(t.is_cuda(), "admp_b200 ops run on CUDA tensors (there is no CPU path)");
  return (void*)at::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

template <typename X>
X* ptr(const Tensor& t) {
  return t.defined() ? (X*)t.data_ptr() : nullptr;
}

// Buffer scales as a call takes them: int64 (as the neighbour list makes them) or the working type.
Tensor scales_of(const Tensor& bs, const Tensor& like) {
  return (bs.scalar_type() == torch::kLong ? bs : bs.to(like.scalar_type())).contiguous();
}
int scale_flag(const Tensor& bs) { return bs.scalar_type() == torch::kLong ? ADMP_PAIR_INT64_SCALES : 0; }

// Whether admp_scale_frames may take a tensor's pointer: batched and other wrapped tensors have no memory of their own,
// and a saved-tensor hook may return another layout.
bool plain(const Tensor& t, const Tensor& like) {
  return t.has_storage() && !t.unsafeGetTensorImpl()->key_set().has_any(c10::DispatchKeySet(
                                {c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                 c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                                 c10::DispatchKey::Negative})) &&
         t.device() == like.device() && t.scalar_type() == like.scalar_type();
}

// Saved gradients times the incoming dL/dE of each frame, all in one launch;
// by torch operators where the product itself is to be differentiated
// (create_graph with a dL/dE that needs a gradient) or a tensor is not plain
// (is_grads_batched: one dL/dE for each of a batch of backward passes).
variable_list scaled(const variable_list& saved, const Tensor& gE) {
  bool direct = !(at::GradMode::is_enabled() && gE.requires_grad()) && plain(gE, gE);
  for (const Tensor& t : saved) direct = direct && (!t.defined() || (plain(t, gE) && t.is_contiguous()));
  if (!direct) {
    variable_list r(saved.size());
    for (size_t i = 0; i < saved.size(); ++i)
      if (saved[i].defined()) {
        std::vector<int64_t> shape(saved[i].dim(), 1);
        shape[0] = gE.numel();
        r[i] = saved[i] * gE.reshape(shape);
      }
    return r;
  }
  const void* in[4];
  void* out[4];
  long long n[4];
  int k = 0;
  variable_list r(saved.size());
  const int64_t nf = gE.numel();
  for (size_t i = 0; i < saved.size(); ++i) {
    if (!saved[i].defined()) continue;
    r[i] = torch::empty_like(saved[i]);
    in[k] = saved[i].data_ptr();
    out[k] = r[i].data_ptr();
    n[k++] = nf > 0 ? saved[i].numel() / nf : 0;
  }
  if (k && nf > 0)
    check(admp_scale_frames(dtype_code(gE), (int)nf, k, in, out, n, gE.data_ptr(), nf > 1 ? gE.stride(0) : 0,
                            stream_of(gE)),
          "gradient scaling");
  return r;
}

Tensor f64(int64_t n, const Tensor& like) {
  return torch::zeros({n}, like.options().dtype(torch::kDouble));
}

// Mesh per frame: explicit kmesh, ceil(L / spacing) or ceil(2 kappa L / (3 ethresh^0.2))
// (pme.py:380-392), with the same double arithmetic as the Python modules.
std::vector<int> kmesh_per_frame(const Tensor& box, double kappa, const std::vector<int64_t>& kmesh,
                                 const std::vector<double>& spacing, double ethresh) {
  const int64_t nf = box.size(0);
  std::vector<int> km(3 * nf);
  Tensor diag;
  std::vector<double> L(3 * nf);
  if (kmesh.empty()) {
    // the raw boxes through page-locked staging: one copy, no conversion kernels
    const size_t bytes = (size_t)nf * 9 * box.element_size();
    if (bytes <= 64 * 1024) {
      std::vector<char> h(bytes);
      check(admp_read_back(box.data_ptr(), bytes, h.data(), stream_of(box)), "box");
      for (int64_t k = 0; k < 3 * nf; ++k) {
        const int64_t e = (k / 3) * 9 + (k % 3) * 4;
        L[k] = box.scalar_type() == torch::kDouble ? ((const double*)h.data())[e] : ((const float*)h.data())[e];
      }
    } else {
      diag = torch::diagonal(box.detach(), 0, 1, 2).to(torch::kCPU, torch::kDouble).contiguous();
      for (int64_t k = 0; k < 3 * nf; ++k) L[k] = diag.data_ptr<double>()[k];
    }
  }
  for (int64_t f = 0; f < nf; ++f)
    for (int d = 0; d < 3; ++d) {
      if (!kmesh.empty()) {
        km[3 * f + d] = (int)kmesh[d];
      } else {
        const double l = L[3 * f + d];
        km[3 * f + d] = spacing.empty() ? (int)std::ceil(2 * kappa * l / (3.0 * std::pow(ethresh, 1.0 / 5.0)))
                                        : (int)std::ceil(l / spacing[d]);
      }
    }
  return km;
}

class CoulombPBC : public torch::autograd::Function<CoulombPBC> {
 public:
  static variable_list forward(AutogradContext* ctx, Tensor pos, Tensor box, Tensor ds, Tensor q, Tensor pairs,
                               Tensor bs, double kappa, std::vector<int64_t> kmesh, std::vector<double> spacing,
                               double ethresh, double ke, bool rspace, bool kspace, bool slab, int64_t axis) {
    const int dt = dtype_code(pos);
    void* st = stream_of(pos);
    const int64_t nf = pos.size(0), N = pos.size(1), P = pairs.size(1);
    ctx->set_materialize_grads(false);
    // gradients of the inputs that need one, produced with the energy
    Tensor gpos, gbox, gds, gq;
    std::vector<int> km = kspace ? kmesh_per_frame(box, kappa, kmesh, spacing, ethresh)
                                 : std::vector<int>(3 * nf, 1);
    Tensor kmt = torch::empty({nf, 3}, torch::kLong);
    for (int64_t k = 0; k < 3 * nf; ++k) kmt.data_ptr<int64_t>()[k] = km[k];
    if (kspace && N > 0 && nf > 0) {
      if (pos.requires_grad()) gpos = torch::empty_like(pos);
      if (box.requires_grad()) gbox = torch::empty_like(box);
      if (ds.requires_grad()) gds = torch::empty_like(ds);
      if (q.requires_grad()) gq = torch::empty_like(q);
      Tensor E = torch::empty({nf}, pos.options());
      Tensor comps = torch::empty({nf, 5}, pos.options().dtype(torch::kDouble));
      const size_t nbytes = admp_pme_recip_workspace_size(dt, (int)nf, km.data());
      TORCH_CHECK(nbytes > 0, "reciprocal workspace: ", admp_last_error_message());
      Tensor ws = torch::empty({(int64_t)nbytes}, pos.options().dtype(torch::kUInt8));
      const int flags = ADMP_QEQ_KSPACE | (rspace ? ADMP_QEQ_RSPACE : 0) |
                        (slab ? ADMP_QEQ_SLAB | ((int)axis << 8) : 0) | scale_flag(bs);
      check(admp_coulomb_pbc(dt, flags, (int)nf, (int)N, km.data(), ptr<void>(pos), ptr<void>(box), P,
                             ptr<const long long>(pairs), ptr<void>(ds), ptr<void>(bs), ptr<void>(q), kappa, ke,
                             ptr<void>(E), ptr<double>(comps), ptr<void>(gpos), ptr<void>(gq), ptr<void>(gbox),
                             ptr<void>(gds), ptr<void>(ws), nbytes, st),
            "Coulomb energy");
      ctx->save_for_backward({gpos, gbox, gds, gq});
      ctx->mark_non_differentiable({comps, kmt});
      return {E, comps, kmt};
    }
    Tensor E_real = f64(nf, pos), E_recip = f64(nf, pos);
    Tensor terms = torch::zeros({nf, 5}, pos.options().dtype(torch::kDouble));
    if (pos.requires_grad()) gpos = torch::zeros_like(pos);
    if (box.requires_grad()) gbox = torch::zeros_like(box);
    if (ds.requires_grad()) gds = torch::zeros_like(ds);
    if (q.requires_grad()) gq = torch::zeros_like(q);
    const Tensor bst = bs.to(pos.scalar_type());
    if (rspace && P > 0)
      check(admp_pair_energy(dt, ADMP_PAIR_EWALD, (int)nf, (int)N, P, ptr<const long long>(pairs), ptr<void>(ds),
                             ptr<void>(bst), ptr<void>(q), nullptr, kappa, ke, ptr<double>(E_real), ptr<void>(gds),
                             ptr<void>(gq), nullptr, st),
            "real-space pair energy");
    if (slab && N > 0)
      check(admp_atom_terms(dt, ADMP_TERM_SLAB | ((int)axis << 8), (int)nf, (int)N, ptr<void>(pos), ptr<void>(box),
                            ptr<void>(q), nullptr, nullptr, nullptr, kappa, ke, nullptr, ptr<double>(terms),
                            ptr<void>(gq), ptr<void>(gpos), ptr<void>(gbox), nullptr, nullptr, nullptr, st),
            "slab term");
    Tensor comps = torch::stack({E_real, E_recip, terms.select(1, 0), terms.select(1, 1), terms.select(1, 2)}, 1);
    Tensor E = comps.sum(1).to(q.scalar_type());
    ctx->save_for_backward({gpos, gbox, gds, gq});
    ctx->mark_non_differentiable({comps, kmt});
    return {E, comps, kmt};
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    variable_list out(15);
    if (g[0].defined()) {
      const variable_list s = scaled(ctx->get_saved_variables(), g[0]);
      for (int k = 0; k < 4; ++k) out[k] = s[k];
    }
    return out;
  }
};

// Full pair list of nf frames of N atoms (nblist.py:304-445), rows of a frame
// padded to the longest frame's count, and its pair distances, differentiable
// in positions and box (nblist.py:517-551; an empty box: open boundaries).  The counts come from
// admp_nblist_frames_count on the same workspace.
class NeighborList : public torch::autograd::Function<NeighborList> {
 public:
  static variable_list forward(AutogradContext* ctx, Tensor pos, Tensor box, Tensor ws, double cutoff, int64_t nf,
                               int64_t N, int64_t P) {
    const auto lo = pos.options().dtype(torch::kLong);
    Tensor pairs = torch::empty({nf * P, 2}, lo), bs = torch::empty({nf * P}, lo);
    Tensor ds = torch::empty({nf * P}, pos.options());
    check(admp_nblist_frames_fill(dtype_code(pos), box.numel() ? 1 : 0, (int)nf, (int)N, ptr<void>(pos), cutoff,
                                  ptr<void>(ws), (size_t)ws.numel(), P, ptr<long long>(pairs), ptr<long long>(bs),
                                  ptr<void>(ds), stream_of(pos)),
          "neighbour list fill");
    ctx->save_for_backward({pos, box, pairs});
    ctx->saved_data["nf"] = nf;
    ctx->saved_data["N"] = N;
    ctx->mark_non_differentiable({pairs, bs});
    ctx->set_materialize_grads(false);  // else zeros as large as the pair list are made for them
    return {pairs, bs, ds};
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    Tensor gpos, gbox;
    if (g[2].defined()) {
      const Tensor &pos = s[0], &box = s[1];
      const int64_t nf = ctx->saved_data["nf"].toInt(), N = ctx->saved_data["N"].toInt();
      if (ctx->needs_input_grad(0)) gpos = torch::empty_like(pos);
      if (box.numel() && ctx->needs_input_grad(1)) gbox = torch::empty_like(box);
      const Tensor gds = g[2].contiguous();
      if (gpos.defined() || gbox.defined())
        check(admp_pair_distances_frames_backward(dtype_code(pos), box.numel() ? 1 : 0, (int)nf, (int)N,
                                                  nf > 0 ? s[2].size(0) / nf : 0, ptr<const long long>(s[2]),
                                                  ptr<void>(pos), box.numel() ? ptr<void>(box) : nullptr, ptr<void>(gds), ptr<void>(gpos),
                                                  ptr<void>(gbox), stream_of(pos)),
              "pair distances backward");
    }
    return {gpos, gbox, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

class CoulombOBC : public torch::autograd::Function<CoulombOBC> {
 public:
  static variable_list forward(AutogradContext* ctx, Tensor ds, Tensor q, Tensor pairs, Tensor bs, double ke) {
    const int dt = dtype_code(q);
    void* st = stream_of(q);
    const int64_t nf = q.size(0), N = q.size(1), P = pairs.size(1);
    const bool need = ds.requires_grad() || q.requires_grad();
    Tensor E = f64(nf, q), gds, gq;
    if (need) {
      gds = torch::zeros_like(ds);
      gq = torch::zeros_like(q);
    }
    if (P > 0)
      check(admp_pair_energy(dt, ADMP_PAIR_OBC, (int)nf, (int)N, P, ptr<const long long>(pairs), ptr<void>(ds),
                             ptr<void>(bs), ptr<void>(q), nullptr, 0.0, ke, ptr<double>(E), ptr<void>(gds),
                             ptr<void>(gq), nullptr, st),
            "open-boundary Coulomb");
    ctx->save_for_backward({gds, gq});
    return {E.to(q.scalar_type())};
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    Tensor out_ds, out_q;
    if (g[0].defined() && s[1].defined()) {
      const Tensor w = g[0].to(s[1].scalar_type()).view({-1, 1});
      out_ds = s[0] * w;
      out_q = s[1] * w;
    }
    return {out_ds, out_q, Tensor(), Tensor(), Tensor()};
  }
};

class Damping : public torch::autograd::Function<Damping> {
 public:
  static variable_list forward(AutogradContext* ctx, Tensor ds, Tensor q, Tensor eta, Tensor pairs, Tensor bs,
                               double ke) {
    const int dt = dtype_code(q);
    void* st = stream_of(q);
    const int64_t nf = q.size(0), N = q.size(1), P = pairs.size(1);
    Tensor gds, gq, geta;
    const bool any = nf > 0 && N > 0;
    // gradients of the inputs that need one; the call writes them
    auto grad = [&](const Tensor& x) {
      return !x.requires_grad() ? Tensor() : any ? torch::empty_like(x) : torch::zeros_like(x);
    };
    gds = grad(ds);
    gq = grad(q);
    geta = grad(eta);
    Tensor E = any ? torch::empty({nf}, q.options().dtype(torch::kDouble)) : f64(nf, q);
    if (any)
      check(admp_damping_energy(dt, scale_flag(bs), (int)nf, (int)N, P, ptr<const long long>(pairs), ptr<void>(ds), ptr<void>(bs),
                                ptr<void>(q), ptr<void>(eta), ke, ptr<double>(E), ptr<void>(gds), ptr<void>(gq),
                                ptr<void>(geta), st),
            "damping energy");
    ctx->save_for_backward({gds, gq, geta});
    return {E.to(q.scalar_type())};
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    variable_list out(6);
    if (g[0].defined()) {
      const variable_list r = scaled(s, g[0]);
      for (int k = 0; k < 3; ++k) out[k] = r[k];
    }
    return out;
  }
};

class Site : public torch::autograd::Function<Site> {
 public:
  static variable_list forward(AutogradContext* ctx, Tensor q, Tensor chi, Tensor hard) {
    const int dt = dtype_code(q);
    void* st = stream_of(q);
    const int64_t nf = q.size(0), N = q.size(1);
    const bool any = nf > 0 && N > 0;
    auto grad = [&](const Tensor& x) {
      return !x.requires_grad() ? Tensor() : any ? torch::empty_like(x) : torch::zeros_like(x);
    };
    Tensor gq = grad(q), gc = grad(chi), gh = grad(hard);
    Tensor E = any ? torch::empty({nf}, q.options().dtype(torch::kDouble)) : f64(nf, q);
    if (any)
      check(admp_site_energy(dt, (int)nf, (int)N, ptr<void>(q), ptr<void>(chi), ptr<void>(hard), ptr<double>(E),
                             ptr<void>(gq), ptr<void>(gc), ptr<void>(gh), st),
            "site energy");
    ctx->save_for_backward({gq, gc, gh});
    return {E.to(q.scalar_type())};
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    return g[0].defined() ? scaled(s, g[0]) : variable_list(3);
  }
};

// Status and (when it is 0) pairs [nf P, 2], scales [nf P], distances [nf P] of positions [nf N, 3].  The kernels
// index a box a frame and three coordinates an atom, so both counts are checked before a pointer is taken.
std::tuple<int64_t, Tensor, Tensor, Tensor> neighbor_list(Tensor pos, std::optional<Tensor> box, double cutoff,
                                                          int64_t nf) {
  TORCH_CHECK_VALUE(nf >= 0 && pos.dim() >= 1, "neighbour list: positions [frames x atoms, 3]");
  const int64_t rows = pos.size(0);
  TORCH_CHECK_INDEX((nf > 0 ? rows % nf == 0 : rows == 0) && pos.numel() >= 3 * rows, "neighbour list: positions ",
                    pos.sizes(), " for ", nf, " frame(s) of atoms with three coordinates");
  if (box.has_value()) {
    TORCH_CHECK_INDEX(nf == 1 ? box->numel() >= 9 : box->numel() == 9 * nf, "neighbour list: box ", box->sizes(), " for ", nf, " frame(s)");
    TORCH_CHECK_TYPE(box->scalar_type() == pos.scalar_type(), "neighbour list: box and positions of one type");
    TORCH_CHECK(box->device() == pos.device(), "neighbour list: box on ", box->device(), ", positions on ", pos.device());
  }
  Tensor p = pos.contiguous(), b = box.has_value() ? box->contiguous() : torch::empty({0}, p.options());
  const int dt = dtype_code(p);
  void* st = stream_of(p);
  const int64_t N = nf > 0 ? p.size(0) / nf : 0;
  const size_t nbytes = admp_nblist_frames_workspace_size((int)nf, (int)N);
  Tensor ws = torch::empty({(int64_t)nbytes}, p.options().dtype(torch::kUInt8));
  std::vector<long long> np(nf > 0 ? nf : 1, 0);
  const int status = admp_nblist_frames_count(dt, b.numel() ? 1 : 0, (int)nf, (int)N, ptr<void>(p), ptr<void>(b),
                                              cutoff, ptr<void>(ws), nbytes, np.data(), st);
  if (status != ADMP_OK) return {status, Tensor(), Tensor(), Tensor()};
  long long P = 0;
  for (long long n : np) P = n > P ? n : P;
  auto r = NeighborList::apply(p, b, ws, cutoff, nf, N, (int64_t)P);
  return {0, r[0], r[1], r[2]};
}

std::vector<Tensor> coulomb_pbc(Tensor pos, Tensor box, Tensor pairs, Tensor ds, Tensor bs, Tensor q, double kappa,
                                std::vector<int64_t> kmesh, std::vector<double> spacing, double ethresh, double ke,
                                bool rspace, bool kspace, bool slab, int64_t axis) {
  TORCH_CHECK(kmesh.empty() || kmesh.size() == 3, "kmesh: 3 values or none");
  TORCH_CHECK(spacing.empty() || spacing.size() == 3, "spacing: 3 values or none");
  auto r = CoulombPBC::apply(pos.contiguous(), box.contiguous(), ds.contiguous(), q.contiguous(),
                             pairs.to(torch::kLong).contiguous(), scales_of(bs, q), kappa, kmesh, spacing, ethresh, ke,
                             rspace, kspace, slab, axis);
  return {r[0], r[1], r[2]};
}

Tensor coulomb_obc(Tensor pairs, Tensor ds, Tensor bs, Tensor q, double ke) {
  return CoulombOBC::apply(ds.contiguous(), q.contiguous(), pairs.to(torch::kLong).contiguous(),
                           bs.to(q.scalar_type()).contiguous(), ke)[0];
}

Tensor damping(Tensor ds, Tensor q, Tensor eta, Tensor pairs, Tensor bs, double ke) {
  return Damping::apply(ds.contiguous(), q.contiguous(), eta.contiguous(), pairs.to(torch::kLong).contiguous(),
                        scales_of(bs, q), ke)[0];
}

Tensor site(Tensor q, Tensor chi, Tensor hard) {
  return Site::apply(q.contiguous(), chi.contiguous(), hard.contiguous())[0];
}

}  // namespace

TORCH_LIBRARY(admp_b200, m) {
  m.def("coulomb_pbc(Tensor pos, Tensor box, Tensor pairs, Tensor ds, Tensor bs, Tensor q, float kappa, "
        "int[] kmesh, float[] spacing, float ethresh, float ke, bool rspace, bool kspace, bool slab, int axis) "
        "-> Tensor[]",
        &coulomb_pbc);
  m.def("neighbor_list(Tensor pos, Tensor? box, float cutoff, int nframes) -> (int, Tensor, Tensor, Tensor)",
        &neighbor_list);
  m.def("coulomb_obc(Tensor pairs, Tensor ds, Tensor bs, Tensor q, float ke) -> Tensor", &coulomb_obc);
  m.def("damping(Tensor ds, Tensor q, Tensor eta, Tensor pairs, Tensor bs, float ke) -> Tensor", &damping);
  m.def("site(Tensor q, Tensor chi, Tensor hardness) -> Tensor", &site);
}
