// Python bindings of the host code.
#include "host.h"

namespace mb200_host {
namespace {

using NoGil = py::call_guard<py::gil_scoped_release>;

}  // namespace
}  // namespace mb200_host

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using namespace mb200_host;
  m.def("selective_scan", &selective_scan);
  m.def("pscan", &pscan, NoGil());
  m.def("conv1d_silu", &conv1d_silu, NoGil());
  m.def("rms_norm", &rms_norm, NoGil());
  m.def("add_rms_norm", &add_rms_norm, NoGil());
  m.def("add_residual", &add_residual, NoGil());
  m.def("ssm_step", &ssm_step, NoGil());
  m.def("conv_step", &conv_step, NoGil());
  m.def("block", &block, NoGil());
  m.def("reversible", &reversible);
  m.def("block_step", &block_step, NoGil());
  m.def("selftest_queue_conversions", &selftest_queue_conversions);
  m.def("selftest_block_step_give_up", &selftest_block_step_give_up);
}
