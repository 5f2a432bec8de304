// tabulate_fusion_se_a on libtorch: calls into libgbdp.so on the current CUDA
// stream and the autograd chain forward -> grad -> grad-of-grad wrt dy
// (source/op/pt/tabulate_multi_device.cc:605-830), shared by the TorchScript
// shim (torch_ops.cpp) and the Python operators' native part
// (torch_native.cpp).
#pragma once

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/autograd.h>
#include <torch/library.h>
#include <torch/types.h>

#include <string>
#include <vector>

#include "gbdp.h"

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// raises the library's last error as the including side's exception
[[noreturn]] void raise_library_error(const std::string& msg);

void check_rc(int rc, const char* what) {
  if (rc != GBDP_OK)
    raise_library_error(std::string(what) + " failed (" + std::to_string(rc) +
                        "): " + gbdp_last_error());
}

void need_cuda(const Tensor& t) {
  TORCH_CHECK(t.is_cuda(),
              "the GB300 deepmd operators run on CUDA tensors only (got a CPU tensor); "
              "there is no CPU fallback");
}

gbdp_stream cur_stream(const Tensor& t) {
  return reinterpret_cast<gbdp_stream>(c10::cuda::getCurrentCUDAStream(t.device().index()).stream());
}

// table_info is read on the host, as the reference's kernels do (tabulate.cu
// reads it through a host pointer); check the table covers every row it
// addresses
template <typename T>
std::vector<T> host_info(const Tensor& info, const Tensor& table) {
  // (a host copy only where it is not a contiguous FP64 host tensor already)
  const Tensor h = info.detach().to(torch::kCPU, torch::kFloat64).contiguous();
  TORCH_CHECK(h.numel() >= 5, "table_info must hold at least 5 values");
  const double* v = h.data_ptr<double>();
  TORCH_CHECK(v[3] > 0 && v[4] > 0, "table strides must be positive");
  std::vector<T> out(v, v + h.numel());
  const T lo = (T)v[0], up = (T)v[1], mx = (T)v[2], s0 = (T)v[3], s1 = (T)v[4];
  const long last = (long)((T)(up - lo) / s0) + (long)((T)(mx - up) / s1) - 1;
  TORCH_CHECK(table.size(0) > last, "table has ", table.size(0),
              " rows but table_info addresses row ", last);
  return out;
}

Tensor tab_forward(const Tensor& table_in, const Tensor& info, const Tensor& em_x_in,
                   const Tensor& em_in, int64_t M) {
  need_cuda(table_in);
  need_cuda(em_x_in);
  need_cuda(em_in);
  TORCH_CHECK(table_in.dim() == 2, "Dim of table should be 2");
  TORCH_CHECK(em_x_in.dim() == 2, "Dim of input should be 2");
  TORCH_CHECK(em_in.dim() == 3, "Dim of input should be 3");
  const c10::cuda::OptionalCUDAGuard guard(table_in.device());
  const Tensor table = table_in.contiguous();
  const Tensor em_x = em_x_in.to(table.scalar_type()).contiguous();
  const Tensor em = em_in.to(table.scalar_type()).contiguous();
  const int nloc = (int)em.size(0), nnei = (int)em.size(1);
  Tensor out = torch::empty({nloc, 4, M}, table.options());
  int rc;
  if (table.scalar_type() == torch::kFloat64) {
    auto hi = host_info<double>(info, table);
    rc = gbdp_tabulate_fusion_se_a_f64(out.data_ptr<double>(), table.data_ptr<double>(), hi.data(),
                                       em_x.data_ptr<double>(), em.data_ptr<double>(), nloc, nnei,
                                       (int)M, 1, cur_stream(table));
  } else {
    TORCH_CHECK(table.scalar_type() == torch::kFloat32, "table must be float32 or float64");
    auto hi = host_info<float>(info, table);
    rc = gbdp_tabulate_fusion_se_a_f32(out.data_ptr<float>(), table.data_ptr<float>(), hi.data(),
                                       em_x.data_ptr<float>(), em.data_ptr<float>(), nloc, nnei,
                                       (int)M, 1, cur_stream(table));
  }
  check_rc(rc, "tabulate_fusion_se_a");
  return out;
}

std::vector<Tensor> tab_grad(const Tensor& table_in, const Tensor& info, const Tensor& em_x_in,
                             const Tensor& em_in, const Tensor& dy_in) {
  need_cuda(dy_in);
  TORCH_CHECK(dy_in.dim() == 3, "Dim of dy_tensor should be 3");
  const c10::cuda::OptionalCUDAGuard guard(table_in.device());
  const Tensor table = table_in.contiguous();
  const auto st = table.scalar_type();
  const Tensor em_x = em_x_in.to(st).contiguous();
  const Tensor em = em_in.to(st).contiguous();
  const Tensor dy = dy_in.to(st).contiguous();
  const int nloc = (int)em.size(0), nnei = (int)em.size(1), M = (int)dy.size(2);
  Tensor gx = torch::empty_like(em_x), gm = torch::empty_like(em);
  int rc;
  if (st == torch::kFloat64) {
    auto hi = host_info<double>(info, table);
    rc = gbdp_tabulate_fusion_se_a_grad_f64(gx.data_ptr<double>(), gm.data_ptr<double>(),
                                            table.data_ptr<double>(), hi.data(),
                                            em_x.data_ptr<double>(), em.data_ptr<double>(),
                                            dy.data_ptr<double>(), nloc, nnei, M, 1,
                                            cur_stream(table));
  } else {
    auto hi = host_info<float>(info, table);
    rc = gbdp_tabulate_fusion_se_a_grad_f32(gx.data_ptr<float>(), gm.data_ptr<float>(),
                                            table.data_ptr<float>(), hi.data(),
                                            em_x.data_ptr<float>(), em.data_ptr<float>(),
                                            dy.data_ptr<float>(), nloc, nnei, M, 1,
                                            cur_stream(table));
  }
  check_rc(rc, "tabulate_fusion_se_a_grad");
  return {gx, gm};
}

Tensor tab_grad_grad(const Tensor& table_in, const Tensor& info, const Tensor& em_x_in,
                     const Tensor& em_in, const Tensor& gx_in, const Tensor& gm_in, int64_t M) {
  const c10::cuda::OptionalCUDAGuard guard(table_in.device());
  const Tensor table = table_in.contiguous();
  const auto st = table.scalar_type();
  const Tensor em_x = em_x_in.to(st).contiguous();
  const Tensor em = em_in.to(st).contiguous();
  const Tensor gx = gx_in.to(st).contiguous();
  const Tensor gm = gm_in.to(st).contiguous();
  const int nloc = (int)em.size(0), nnei = (int)em.size(1);
  Tensor dz = torch::empty({nloc, 4, M}, table.options());
  int rc;
  if (st == torch::kFloat64) {
    auto hi = host_info<double>(info, table);
    rc = gbdp_tabulate_fusion_se_a_grad_grad_f64(
        dz.data_ptr<double>(), table.data_ptr<double>(), hi.data(), em_x.data_ptr<double>(),
        em.data_ptr<double>(), gx.data_ptr<double>(), gm.data_ptr<double>(), nloc, nnei, (int)M,
        1, cur_stream(table));
  } else {
    auto hi = host_info<float>(info, table);
    rc = gbdp_tabulate_fusion_se_a_grad_grad_f32(
        dz.data_ptr<float>(), table.data_ptr<float>(), hi.data(), em_x.data_ptr<float>(),
        em.data_ptr<float>(), gx.data_ptr<float>(), gm.data_ptr<float>(), nloc, nnei, (int)M, 1,
        cur_stream(table));
  }
  check_rc(rc, "tabulate_fusion_se_a_grad_grad");
  return dz;
}

// dy -> (dy_dem_x, dy_dem); differentiable wrt dy only (the grad-grad kernel)
struct TabGradFn : public torch::autograd::Function<TabGradFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& table, const Tensor& info,
                               const Tensor& em_x, const Tensor& em, const Tensor& dy) {
    ctx->save_for_backward({table, info, em_x, em});
    ctx->saved_data["M"] = dy.size(2);
    return tab_grad(table, info, em_x, em, dy);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    Tensor gx = g[0].defined() ? g[0] : torch::zeros_like(s[2]);
    Tensor gm = g[1].defined() ? g[1] : torch::zeros_like(s[3]);
    Tensor dz = tab_grad_grad(s[0], s[1], s[2], s[3], gx, gm, ctx->saved_data["M"].toInt());
    return {Tensor(), Tensor(), Tensor(), Tensor(), dz};
  }
};

struct TabFn : public torch::autograd::Function<TabFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& table, const Tensor& info,
                        const Tensor& em_x, const Tensor& em, int64_t M) {
    ctx->save_for_backward({table, info, em_x, em});
    return tab_forward(table, info, em_x, em, M);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    auto gg = TabGradFn::apply(s[0], s[1], s[2], s[3], g[0].contiguous());
    return {Tensor(), Tensor(), gg[0], gg[1], Tensor()};
  }
};

}  // namespace
