// libtorch registration of the deepmd operators on this path, for C++
// processes that run TorchScript models (DeepPotPT::compute,
// source/api_cc/src/DeepPotPT.cc:171-410, as LAMMPS does).  It stands in for
// the reference's libdeepmd_op_pt.so on the se_e2_a path: it owns
// TORCH_LIBRARY(deepmd) with enable_mpi (source/op/pt/print_summary.cc:14;
// deepmd/pt/cxx_op.py:22-60 skips loading the reference's library when it is
// present) and tabulate_fusion_se_a with the reference's schema and
// autograd (source/op/pt/tabulate_multi_device.cc:605-830,1498-1552):
// forward -> descriptor [nloc, 4, M]; backward -> grads for em_x and em;
// the grad op's backward -> the grad for dy only.  Every call goes to
// libgbdp.so on the current CUDA stream; CPU tensors raise.
#include "torch_tab.h"

namespace {

void raise_library_error(const std::string& msg) {
  TORCH_CHECK(false, msg);
  std::terminate();  // not reached
}

std::vector<Tensor> tabulate_fusion_se_a(const Tensor& table, const Tensor& table_info,
                                         const Tensor& em_x, const Tensor& em,
                                         int64_t last_layer_size) {
  return {TabFn::apply(table, table_info, em_x, em, last_layer_size)};
}

Tensor enable_mpi() { return torch::zeros({1}, torch::kBool); }

}  // namespace

TORCH_LIBRARY(deepmd, m) {
  m.def("enable_mpi", enable_mpi);
  m.def("tabulate_fusion_se_a", tabulate_fusion_se_a);
}
