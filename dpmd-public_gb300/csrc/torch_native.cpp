// Native part of the Python operators (ops.py): the torch.ops.deepmd calls of
// the operator form under a private namespace, with their autograd in C++.
// A small training batch spends its time on the host: through Python autograd
// functions and ctypes the tabulate chain up to the double backward took 520
// us for 75 us of kernels.  ops.py keeps the deepmd schemas and turns errors
// into its own exception type.
//
//   tab           tabulate_fusion_se_a (source/op/pt/
//                 tabulate_multi_device.cc:1498-1552)
//   prod_force    ProdForceSeA (source/op/tf/prod_force_multi_device.cc:6-14),
//                 differentiable wrt net_deriv (prod_force_grad_multi_device.cc)
//   prod_virial   ProdVirialSeA (source/op/tf/prod_virial_multi_device.cc:5-15)
//   env_mat       ProdEnvMatA, internal periodic mode
//                 (source/op/tf/prod_env_mat_multi_device.cc:11-28)
//   env_mat_nlist prod_env_mat_a from an external list (forward_lower)
#include <torch/csrc/Exceptions.h>

#include <memory>
#include <mutex>

#include "torch_tab.h"

namespace {

// Library errors reach Python as the operators' own exception type (GbdpError)
// from the backward passes too, where no Python frame of ops.py stands between
// the autograd engine and the caller.
PyObject* g_error_type = nullptr;

struct LibraryError : public torch::PyTorchError {
  explicit LibraryError(const std::string& m) : torch::PyTorchError(m) {}
  PyObject* python_type() override { return g_error_type ? g_error_type : PyExc_RuntimeError; }
};

void raise_library_error(const std::string& msg) { throw LibraryError(msg); }

gbdp_stream stream_of(const Tensor& t) { return cur_stream(t); }

bool is64(const Tensor& t) {
  TORCH_CHECK_TYPE(t.scalar_type() == torch::kFloat64 || t.scalar_type() == torch::kFloat32,
                   "unsupported dtype ", t.scalar_type(), "; float32 and float64 only");
  return t.scalar_type() == torch::kFloat64;
}

std::vector<int64_t> host_ints(const Tensor& t) {
  const Tensor h = t.detach().to(torch::kCPU, torch::kInt64).contiguous();
  return {h.data_ptr<int64_t>(), h.data_ptr<int64_t>() + h.numel()};
}

Tensor i32(const Tensor& t) { return t.to(torch::kInt32).contiguous(); }

Tensor bytes(size_t n, const Tensor& like) {
  return torch::empty({(int64_t)(n ? n : 1)}, like.options().dtype(torch::kUInt8));
}

template <typename T>
T* ptr(const Tensor& t) {
  return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr;
}

// ------------------------------------------------------- force, virial --
struct Dims {
  int nf, nloc, nall, nnei;
};
Dims dims_of(const Tensor& net, const Tensor& natoms, int64_t na, int64_t nr) {
  const auto n = host_ints(natoms);
  TORCH_CHECK(n.size() >= 2, "natoms must hold nloc and nall");
  return {(int)net.size(0), (int)n[0], (int)n[1], (int)(na + nr)};
}

Tensor force_call(const Tensor& net_in, const Tensor& der_in, const Tensor& nl_in, const Dims& d) {
  need_cuda(net_in);
  need_cuda(der_in);
  need_cuda(nl_in);
  const c10::cuda::OptionalCUDAGuard guard(net_in.device());
  const bool f64 = is64(net_in);
  const Tensor net = net_in.contiguous(), der = der_in.to(net.scalar_type()).contiguous(),
               nl = i32(nl_in);
  Tensor force = torch::empty({d.nf, (int64_t)d.nall * 3}, net.options());
  const size_t wsb = gbdp_prod_call_workspace_bytes(d.nf, d.nloc, d.nall, d.nnei, 0, f64, 0);
  const Tensor ws = bytes(wsb, net);
  int rc;
  if (f64)
    rc = gbdp_prod_force_a_f64(ptr<double>(force), ptr<double>(net), ptr<double>(der),
                               ptr<int>(nl), d.nloc, d.nall, d.nnei, d.nf, 0, ptr<void>(ws), wsb,
                               stream_of(net));
  else
    rc = gbdp_prod_force_a_f32(ptr<float>(force), ptr<float>(net), ptr<float>(der), ptr<int>(nl),
                               d.nloc, d.nall, d.nnei, d.nf, 0, ptr<void>(ws), wsb,
                               stream_of(net));
  check_rc(rc, "prod_force_se_a");
  return force;
}

std::vector<Tensor> virial_call(const Tensor& net_in, const Tensor& der_in, const Tensor& rij_in,
                                const Tensor& nl_in, const Dims& d) {
  need_cuda(net_in);
  need_cuda(der_in);
  need_cuda(rij_in);
  need_cuda(nl_in);
  const c10::cuda::OptionalCUDAGuard guard(net_in.device());
  const bool f64 = is64(net_in);
  const auto st = net_in.scalar_type();
  const Tensor net = net_in.contiguous(), der = der_in.to(st).contiguous(),
               rij = rij_in.to(st).contiguous(), nl = i32(nl_in);
  Tensor vir = torch::empty({d.nf, 9}, net.options());
  Tensor av = torch::empty({d.nf, (int64_t)d.nall * 9}, net.options());
  const size_t wsb = gbdp_prod_call_workspace_bytes(d.nf, d.nloc, d.nall, d.nnei, 0, f64, 1);
  const Tensor ws = bytes(wsb, net);
  int rc;
  if (f64)
    rc = gbdp_prod_virial_a_f64(ptr<double>(vir), ptr<double>(av), ptr<double>(net),
                                ptr<double>(der), ptr<double>(rij), ptr<int>(nl), d.nloc, d.nall,
                                d.nnei, d.nf, 0, ptr<void>(ws), wsb, stream_of(net));
  else
    rc = gbdp_prod_virial_a_f32(ptr<float>(vir), ptr<float>(av), ptr<float>(net), ptr<float>(der),
                                ptr<float>(rij), ptr<int>(nl), d.nloc, d.nall, d.nnei, d.nf, 0,
                                ptr<void>(ws), wsb, stream_of(net));
  check_rc(rc, "prod_virial_se_a");
  return {vir, av};
}

Tensor force_grad_call(const Tensor& g_in, const Tensor& der_in, const Tensor& nl_in, int nloc,
                       int nnei, int nf) {
  const c10::cuda::OptionalCUDAGuard guard(g_in.device());
  const bool f64 = is64(g_in);
  const Tensor g = g_in.contiguous(), der = der_in.to(g.scalar_type()).contiguous(),
               nl = i32(nl_in);
  Tensor out = torch::empty({nf, (int64_t)nloc * nnei * 4}, g.options());
  int rc;
  if (f64)
    rc = gbdp_prod_force_grad_a_f64(ptr<double>(out), ptr<double>(g), ptr<double>(der),
                                    ptr<int>(nl), nloc, nnei, nf, stream_of(g));
  else
    rc = gbdp_prod_force_grad_a_f32(ptr<float>(out), ptr<float>(g), ptr<float>(der), ptr<int>(nl),
                                    nloc, nnei, nf, stream_of(g));
  check_rc(rc, "prod_force_grad_a");
  return out;
}

Tensor virial_grad_call(const Tensor& g_in, const Tensor& der_in, const Tensor& rij_in,
                        const Tensor& nl_in, int nloc, int nnei, int nf) {
  const c10::cuda::OptionalCUDAGuard guard(g_in.device());
  const bool f64 = is64(g_in);
  const auto st = g_in.scalar_type();
  const Tensor g = g_in.contiguous(), der = der_in.to(st).contiguous(),
               rij = rij_in.to(st).contiguous(), nl = i32(nl_in);
  Tensor out = torch::empty({nf, (int64_t)nloc * nnei * 4}, g.options());
  int rc;
  if (f64)
    rc = gbdp_prod_virial_grad_a_f64(ptr<double>(out), ptr<double>(g), ptr<double>(der),
                                     ptr<double>(rij), ptr<int>(nl), nloc, nnei, nf, stream_of(g));
  else
    rc = gbdp_prod_virial_grad_a_f32(ptr<float>(out), ptr<float>(g), ptr<float>(der),
                                     ptr<float>(rij), ptr<int>(nl), nloc, nnei, nf, stream_of(g));
  check_rc(rc, "prod_virial_grad_a");
  return out;
}

struct ForceFn : public torch::autograd::Function<ForceFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& net, const Tensor& der,
                        const Tensor& nl, const Tensor& natoms, int64_t na, int64_t nr) {
    const Dims d = dims_of(net, natoms, na, nr);
    ctx->save_for_backward({der, nl});
    ctx->saved_data["nf"] = (int64_t)d.nf;
    ctx->saved_data["nloc"] = (int64_t)d.nloc;
    ctx->saved_data["nall"] = (int64_t)d.nall;
    ctx->saved_data["nnei"] = (int64_t)d.nnei;
    return force_call(net, der, nl, d);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const int64_t nf = ctx->saved_data["nf"].toInt(), nloc = ctx->saved_data["nloc"].toInt(),
                  nall = ctx->saved_data["nall"].toInt(), nnei = ctx->saved_data["nnei"].toInt();
    const Tensor gf = g[0].reshape({nf, nall, 3}).slice(1, 0, nloc).contiguous();
    Tensor out = force_grad_call(gf, s[0], s[1], (int)nloc, (int)nnei, (int)nf);
    return {out, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

struct VirialFn : public torch::autograd::Function<VirialFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& net, const Tensor& der,
                               const Tensor& rij, const Tensor& nl, const Tensor& natoms,
                               int64_t na, int64_t nr) {
    const Dims d = dims_of(net, natoms, na, nr);
    ctx->save_for_backward({der, rij, nl});
    ctx->saved_data["nf"] = (int64_t)d.nf;
    ctx->saved_data["nloc"] = (int64_t)d.nloc;
    ctx->saved_data["nnei"] = (int64_t)d.nnei;
    return virial_call(net, der, rij, nl, d);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const int64_t nf = ctx->saved_data["nf"].toInt();
    // the atom virial alone carries no gradient, as in the Python form
    const Tensor gv = g[0].defined() ? g[0].contiguous() : torch::zeros({nf, 9}, s[0].options());
    Tensor out = virial_grad_call(gv, s[0], s[1], s[2], (int)ctx->saved_data["nloc"].toInt(),
                                  (int)ctx->saved_data["nnei"].toInt(), (int)nf);
    return {out, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor tab(const Tensor& table, const Tensor& info, const Tensor& em_x, const Tensor& em,
           int64_t M) {
  need_cuda(table);
  is64(table);  // float32 and float64 only
  return TabFn::apply(table, info, em_x, em, M);
}
Tensor prod_force(const Tensor& net, const Tensor& der, const Tensor& nl, const Tensor& natoms,
                  int64_t na, int64_t nr) {
  return ForceFn::apply(net, der, nl, natoms, na, nr);
}
std::vector<Tensor> prod_virial(const Tensor& net, const Tensor& der, const Tensor& rij,
                                const Tensor& nl, const Tensor& natoms, int64_t na, int64_t nr) {
  return VirialFn::apply(net, der, rij, nl, natoms, na, nr);
}

// --------------------------------------------------------- env matrix --
// Host plan and device frame table of one set of equal frames.  Read only
// after it is made, except for the candidate capacity, which only grows; every
// call takes its own workspace, so calls on several streams or threads share
// nothing they write.
struct Plan {
  int nloc, dev;
  bool f64;
  double rcut;
  std::vector<double> boxes;
  gbdp_nbr_plan plan;
  Tensor frames_dev;
  size_t ws_bytes;
  std::mutex mu;  // guards plan.max_cand
};
constexpr int kMaxCandLimit = 4096;  // 4 warps x capacity x 9 B of shared memory

std::shared_ptr<Plan> plan_for(int nloc, const std::vector<double>& boxes, double rcut,
                               const Tensor& coord, bool f64) {
  static std::mutex mu;
  // never destroyed: at process exit the CUDA context may be gone first
  static auto& cache = *new std::vector<std::shared_ptr<Plan>>();
  const int dev = coord.device().index();
  std::lock_guard<std::mutex> lock(mu);
  for (const auto& p : cache)
    if (p->nloc == nloc && p->dev == dev && p->f64 == f64 && p->rcut == rcut && p->boxes == boxes)
      return p;
  auto p = std::make_shared<Plan>();
  p->nloc = nloc;
  p->dev = dev;
  p->f64 = f64;
  p->rcut = rcut;
  p->boxes = boxes;
  // float coordinates come with a float box: the reference builds its cell
  // grid and ghost shifts from that box converted to double
  // (source/lib/src/coord.cc:42-47)
  std::vector<double> bx = boxes;
  if (!f64)
    for (double& v : bx) v = (double)(float)v;
  const int nf = (int)(bx.size() / 9);
  std::vector<int> counts(nf, nloc);
  std::vector<gbdp_nbr_frame> frames(nf);
  check_rc(gbdp_nbr_plan_make(&p->plan, frames.data(), nf, counts.data(), bx.data(), (float)rcut, 0),
           "nbr_plan_make");
  p->frames_dev = torch::from_blob(frames.data(), {(int64_t)(sizeof(gbdp_nbr_frame) * nf)},
                                   torch::kUInt8)
                      .to(coord.device());
  p->ws_bytes = gbdp_env_workspace_bytes(&p->plan, f64 ? 1 : 0);
  if (cache.size() > 16) cache.clear();
  cache.push_back(p);
  return p;
}

const char* status_text(int st) {
  switch (st) {
    case 1: return "candidate overflow (raise max_cand)";
    case 2: return "extended-atom overflow";
    case 3: return "device wait timed out";
    case 4: return "index out of range";
  }
  return "?";
}

std::vector<int> sections(at::IntArrayRef sel) { return {sel.begin(), sel.end()}; }

std::vector<Tensor> env_mat(const Tensor& coord_in, const Tensor& type_in, const Tensor& natoms,
                            const Tensor& box, const Tensor& mesh, const Tensor& avg_in,
                            const Tensor& std_in, double rcut, double rcut_smth,
                            at::IntArrayRef sel_a, at::IntArrayRef sel_r) {
  need_cuda(coord_in);
  need_cuda(type_in);
  need_cuda(avg_in);
  need_cuda(std_in);
  for (const int64_t s : sel_r)
    TORCH_CHECK(s == 0, "Rotational free descriptor only support all-angular information: "
                        "sel_r should be all zero.");
  const auto nat = host_ints(natoms);
  TORCH_CHECK(nat.size() >= 2, "natoms must hold nloc and nall");
  const int nloc = (int)nat[0];
  TORCH_CHECK_NOT_IMPLEMENTED(mesh.numel() == 6,
                              "only the internal periodic mode (mesh of 6) is implemented on GB300");
  TORCH_CHECK(nat[0] == nat[1], "internal periodic mode requires nloc == nall");
  TORCH_CHECK(sel_a.size() == nat.size() - 2,
              "number of types should match the length of sel array");
  const c10::cuda::OptionalCUDAGuard guard(coord_in.device());
  const bool f64 = is64(coord_in);
  const auto st = coord_in.scalar_type();
  const int64_t nf = coord_in.size(0);
  const Tensor hb = box.detach().to(torch::kCPU, torch::kFloat64).reshape({nf, 9}).contiguous();
  const auto plan = plan_for(nloc, {hb.data_ptr<double>(), hb.data_ptr<double>() + hb.numel()},
                             rcut, coord_in, f64);
  const Tensor coord = coord_in.reshape({nf * nloc, 3}).contiguous();
  const Tensor type = i32(type_in.reshape({nf * nloc}));
  const Tensor avg = avg_in.to(st).contiguous(), sd = std_in.to(st).contiguous();
  const std::vector<int> sel = sections(sel_a);
  int64_t nnei = 0;
  for (const int s : sel) nnei += s;
  const int64_t n = nf * nloc, next = plan->plan.ext_total;
  const auto fo = coord.options(), io = fo.dtype(torch::kInt32);
  Tensor em = torch::empty({nf, (int64_t)nloc * nnei * 4}, fo);
  Tensor der = torch::empty({nf, (int64_t)nloc * nnei * 12}, fo);
  Tensor rij = torch::empty({nf, (int64_t)nloc * nnei * 3}, fo);
  Tensor nl = torch::empty({nf, (int64_t)nloc * nnei}, io);
  const Tensor xc = torch::empty({next, 3}, fo);
  const Tensor xi = torch::empty({2 * next + nf}, io);  // extended types, map; nall per frame
  const Tensor ws = bytes(plan->ws_bytes, coord);
  int* xi_p = ptr<int>(xi);
  gbdp_nbr_plan pl;
  {
    std::lock_guard<std::mutex> lock(plan->mu);
    pl = plan->plan;
  }
  TORCH_INTERNAL_ASSERT(pl.nloc_total == n);
  for (;;) {
    int rc;
    const gbdp_nbr_frame* fr = reinterpret_cast<const gbdp_nbr_frame*>(ptr<uint8_t>(plan->frames_dev));
    if (f64)
      rc = gbdp_prod_env_mat_a_f64(ptr<double>(em), ptr<double>(der), ptr<double>(rij),
                                   ptr<int>(nl), nullptr, ptr<double>(xc), xi_p, xi_p + next,
                                   xi_p + 2 * next, ptr<double>(coord), ptr<int>(type),
                                   ptr<double>(avg), ptr<double>(sd), &pl, fr, (float)rcut_smth,
                                   sel.data(), (int)sel.size(), ptr<void>(ws), plan->ws_bytes,
                                   stream_of(coord));
    else
      rc = gbdp_prod_env_mat_a_f32(ptr<float>(em), ptr<float>(der), ptr<float>(rij), ptr<int>(nl),
                                   nullptr, ptr<float>(xc), xi_p, xi_p + next, xi_p + 2 * next,
                                   ptr<float>(coord), ptr<int>(type), ptr<float>(avg),
                                   ptr<float>(sd), &pl, fr, (float)rcut_smth, sel.data(),
                                   (int)sel.size(), ptr<void>(ws), plan->ws_bytes,
                                   stream_of(coord));
    check_rc(rc, "prod_env_mat_a");
    const int status = gbdp_env_status(ptr<void>(ws), stream_of(coord));
    if (status == 0) break;
    // a centre with more candidates than the capacity: double it and run again
    // (source/op/tf/prod_env_mat_multi_device.cc:1583-1605); the plan keeps it
    if (status == GBDP_STATUS_CAND_OVERFLOW && pl.max_cand < kMaxCandLimit) {
      pl.max_cand = std::min(2 * pl.max_cand, kMaxCandLimit);
      std::lock_guard<std::mutex> lock(plan->mu);
      plan->plan.max_cand = std::max(plan->plan.max_cand, pl.max_cand);
      continue;
    }
    TORCH_CHECK(false, "prod_env_mat_a device status ", status, ": ", status_text(status),
                status == GBDP_STATUS_CAND_OVERFLOW
                    ? " at max_cand " + std::to_string(pl.max_cand)
                    : std::string());
  }
  return {em, der, rij, nl};
}

std::vector<Tensor> env_mat_nlist(const Tensor& coord_in, const Tensor& type_in,
                                  const Tensor& nl_in, const Tensor& avg_in, const Tensor& std_in,
                                  double rcut, double rcut_smth, at::IntArrayRef sel_in) {
  need_cuda(coord_in);
  need_cuda(type_in);
  need_cuda(nl_in);
  need_cuda(avg_in);
  need_cuda(std_in);
  const c10::cuda::OptionalCUDAGuard guard(coord_in.device());
  const bool f64 = is64(coord_in);
  const auto st = coord_in.scalar_type();
  TORCH_CHECK(nl_in.dim() == 3, "nlist must be [nframes, nloc, nnei]");
  const int64_t nf = nl_in.size(0), nloc = nl_in.size(1), width = nl_in.size(2);
  const int64_t nall = coord_in.reshape({nf, -1}).size(1) / 3;
  TORCH_CHECK(type_in.reshape({nf, -1}).size(1) == nall, "type must have nall entries per frame");
  const std::vector<int> sel = sections(sel_in);
  int64_t nnei = 0;
  for (const int s : sel) nnei += s;
  const Tensor coord = coord_in.contiguous(), type = i32(type_in), nlist = i32(nl_in),
               avg = avg_in.to(st).contiguous(), sd = std_in.to(st).contiguous();
  const auto fo = coord.options(), io = fo.dtype(torch::kInt32);
  Tensor em = torch::empty({nf, nloc * nnei * 4}, fo);
  Tensor der = torch::empty({nf, nloc * nnei * 12}, fo);
  Tensor rij = torch::empty({nf, nloc * nnei * 3}, fo);
  Tensor nl = torch::empty({nf, nloc * nnei}, io);
  const Tensor status = torch::zeros({1}, io);
  int rc;
  if (f64)
    rc = gbdp_prod_env_mat_a_nlist_f64(
        ptr<double>(em), ptr<double>(der), ptr<double>(rij), ptr<int>(nl), ptr<int>(status),
        ptr<double>(coord), ptr<int>(type), ptr<int>(nlist), ptr<double>(avg), ptr<double>(sd),
        (int)nf, (int)nloc, (int)nall, (int)width, (float)rcut, (float)rcut_smth, sel.data(),
        (int)sel.size(), stream_of(coord));
  else
    rc = gbdp_prod_env_mat_a_nlist_f32(
        ptr<float>(em), ptr<float>(der), ptr<float>(rij), ptr<int>(nl), ptr<int>(status),
        ptr<float>(coord), ptr<int>(type), ptr<int>(nlist), ptr<float>(avg), ptr<float>(sd),
        (int)nf, (int)nloc, (int)nall, (int)width, (float)rcut, (float)rcut_smth, sel.data(),
        (int)sel.size(), stream_of(coord));
  check_rc(rc, "prod_env_mat_a_nlist");
  const int s = status.item<int>();
  TORCH_CHECK(s == 0, "prod_env_mat_a_nlist device status ", s, ": ", status_text(s));
  return {em, der, rij, nl};
}

}  // namespace

// (called once at load, with the GIL held; the class is kept for good)
extern "C" void gbdp_native_set_error_type(PyObject* type) {
  Py_XINCREF(type);
  g_error_type = type;
}

TORCH_LIBRARY(gbdp_native, m) {
  m.def("tab(Tensor table, Tensor table_info, Tensor em_x, Tensor em, int last_layer_size) -> Tensor",
        tab);
  m.def("prod_force(Tensor net_deriv, Tensor in_deriv, Tensor nlist, Tensor natoms, int n_a_sel, "
        "int n_r_sel) -> Tensor",
        prod_force);
  m.def("prod_virial(Tensor net_deriv, Tensor in_deriv, Tensor rij, Tensor nlist, Tensor natoms, "
        "int n_a_sel, int n_r_sel) -> Tensor[]",
        prod_virial);
  m.def("env_mat(Tensor coord, Tensor type, Tensor natoms, Tensor box, Tensor mesh, Tensor davg, "
        "Tensor dstd, float rcut, float rcut_smth, int[] sel_a, int[] sel_r) -> Tensor[]",
        env_mat);
  m.def("env_mat_nlist(Tensor coord, Tensor type, Tensor nlist, Tensor davg, Tensor dstd, "
        "float rcut, float rcut_smth, int[] sel) -> Tensor[]",
        env_mat_nlist);
}
