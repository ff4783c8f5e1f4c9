// Python bindings of the native library (pybind11): tensors cross the boundary as raw device pointers, streams as
// integer handles, so nothing here allocates.  The operators that take tensors are in tensor_calls.cpp, the one file
// that depends on libtorch.
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include <stdexcept>
#include <string>

#include "include/fm_api.h"
#include "include/fm_ops.h"
#include "include/fm_symm.h"

namespace py = pybind11;

// Value of a descriptor field.  The key is a string object made once per call site: looking seventy fields
// up by C string made a Python string for each, 6 us of every launch.
template <class T>
static T field(const py::dict& d, PyObject* key, T dflt) {
  PyObject* o = PyDict_GetItemWithError(d.ptr(), key);      // borrowed
  if (o == nullptr || o == Py_None) {
    if (PyErr_Occurred()) throw py::error_already_set();
    return dflt;
  }
  return py::reinterpret_borrow<py::object>(o).cast<T>();
}
#define FM_KEY(name) ([]() -> PyObject* { static PyObject* k = PyUnicode_InternFromString(name); return k; }())

static void check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string(what) + ": " + fm_last_error());
}

static FmGemmDesc gemm_descriptor(const py::dict& d) {
  FmGemmDesc g{};
  g.A = reinterpret_cast<const void*>(field<uintptr_t>(d, FM_KEY("A"), 0));
  g.B = reinterpret_cast<const void*>(field<uintptr_t>(d, FM_KEY("B"), 0));
  g.a_mn = field<int>(d, FM_KEY("a_mn"), 0);
  g.b_mn = field<int>(d, FM_KEY("b_mn"), 0);
  g.a_inner = field<long long>(d, FM_KEY("a_inner"), 0);
  g.a_outer = field<long long>(d, FM_KEY("a_outer"), 0);
  g.lda = field<long long>(d, FM_KEY("lda"), 0);
  g.b_inner = field<long long>(d, FM_KEY("b_inner"), 0);
  g.b_outer = field<long long>(d, FM_KEY("b_outer"), 0);
  g.ldb = field<long long>(d, FM_KEY("ldb"), 0);
  g.mode = field<int>(d, FM_KEY("mode"), 0);
  g.num_groups = field<int>(d, FM_KEY("num_groups"), 1);
  g.M = field<int>(d, FM_KEY("M"), 0);
  g.N = field<int>(d, FM_KEY("N"), 0);
  g.K = field<int>(d, FM_KEY("K"), 0);
  g.uniform_rows = field<int>(d, FM_KEY("uniform_rows"), 0);
  g.group_rows = reinterpret_cast<const int*>(field<uintptr_t>(d, FM_KEY("group_rows"), 0));
  g.group_offs = reinterpret_cast<const int*>(field<uintptr_t>(d, FM_KEY("group_offs"), 0));
  g.group_b = reinterpret_cast<const int*>(field<uintptr_t>(d, FM_KEY("group_b"), 0));
  g.b_group_stride = field<int>(d, FM_KEY("b_group_stride"), 0);
  g.gated = field<int>(d, FM_KEY("gated"), 0);
  g.n_half = field<int>(d, FM_KEY("n_half"), 0);
  g.bn = field<int>(d, FM_KEY("bn"), 256);
  g.swizzle_m = field<int>(d, FM_KEY("swizzle_m"), 0);
  g.cta_pair = field<int>(d, FM_KEY("cta_pair"), 0);
  g.epi = field<int>(d, FM_KEY("epi"), 0);
  g.C = reinterpret_cast<void*>(field<uintptr_t>(d, FM_KEY("C"), 0));
  g.ldc = field<long long>(d, FM_KEY("ldc"), 0);
  g.c_group_stride = field<long long>(d, FM_KEY("c_group_stride"), 0);
  g.out_fp32 = field<int>(d, FM_KEY("out_fp32"), 0);
  g.accumulate = field<int>(d, FM_KEY("accumulate"), 0);
  g.alpha = field<float>(d, FM_KEY("alpha"), 1.0f);
  g.alpha_dev = reinterpret_cast<const float*>(field<uintptr_t>(d, FM_KEY("alpha_dev"), 0));
  g.residual = reinterpret_cast<const void*>(field<uintptr_t>(d, FM_KEY("residual"), 0));
  g.ld_residual = field<long long>(d, FM_KEY("ld_residual"), 0);
  g.act_out = reinterpret_cast<void*>(field<uintptr_t>(d, FM_KEY("act_out"), 0));
  g.ld_act = field<long long>(d, FM_KEY("ld_act"), 0);
  g.pre_out = reinterpret_cast<void*>(field<uintptr_t>(d, FM_KEY("pre_out"), 0));
  g.ld_pre = field<long long>(d, FM_KEY("ld_pre"), 0);
  g.probs = reinterpret_cast<const float*>(field<uintptr_t>(d, FM_KEY("probs"), 0));
  g.act_kind = field<int>(d, FM_KEY("act_kind"), 0);
  g.pre_in = reinterpret_cast<const void*>(field<uintptr_t>(d, FM_KEY("pre_in"), 0));
  g.ld_pre_in = field<long long>(d, FM_KEY("ld_pre_in"), 0);
  g.dprobs = reinterpret_cast<float*>(field<uintptr_t>(d, FM_KEY("dprobs"), 0));
  g.dst_base = reinterpret_cast<void* const*>(field<uintptr_t>(d, FM_KEY("dst_base"), 0));
  g.dst_rank = reinterpret_cast<const int*>(field<uintptr_t>(d, FM_KEY("dst_rank"), 0));
  g.dst_row = reinterpret_cast<const int*>(field<uintptr_t>(d, FM_KEY("dst_row"), 0));
  g.ld_dst = field<long long>(d, FM_KEY("ld_dst"), 0);
  g.dst_flags = reinterpret_cast<int* const*>(field<uintptr_t>(d, FM_KEY("dst_flags"), 0));
  g.num_ranks = field<int>(d, FM_KEY("num_ranks"), 1);
  g.row_aux = reinterpret_cast<const float*>(field<uintptr_t>(d, FM_KEY("row_aux"), 0));
  g.row_aux_dst = reinterpret_cast<float* const*>(field<uintptr_t>(d, FM_KEY("row_aux_dst"), 0));
  g.gate_flags = reinterpret_cast<const int*>(field<uintptr_t>(d, FM_KEY("gate_flags"), 0));
  g.gate_group_base = reinterpret_cast<const int*>(field<uintptr_t>(d, FM_KEY("gate_group_base"), 0));
  g.gate_blocks_per_group = field<int>(d, FM_KEY("gate_blocks_per_group"), 0);
  g.gate_expected = field<int>(d, FM_KEY("gate_expected"), 0);
  g.gate_k_blocks_per_src = field<int>(d, FM_KEY("gate_k_blocks_per_src"), 0);
  g.n_rotate = field<int>(d, FM_KEY("n_rotate"), 0);
  g.k_rotate = field<int>(d, FM_KEY("k_rotate"), 0);
  g.cols_per_rank = field<int>(d, FM_KEY("cols_per_rank"), 0);
  g.dst_row_offset = field<long long>(d, FM_KEY("dst_row_offset"), 0);
  g.adam_p = reinterpret_cast<void*>(field<uintptr_t>(d, FM_KEY("adam_p"), 0));
  g.adam_m = reinterpret_cast<void*>(field<uintptr_t>(d, FM_KEY("adam_m"), 0));
  g.adam_v = reinterpret_cast<void*>(field<uintptr_t>(d, FM_KEY("adam_v"), 0));
  g.adam_lr = field<float>(d, FM_KEY("adam_lr"), 0.f);
  g.adam_beta1 = field<float>(d, FM_KEY("adam_beta1"), 0.f);
  g.adam_beta2 = field<float>(d, FM_KEY("adam_beta2"), 0.f);
  g.adam_eps = field<float>(d, FM_KEY("adam_eps"), 0.f);
  g.adam_wd = field<float>(d, FM_KEY("adam_wd"), 0.f);
  g.adam_rbc1 = field<float>(d, FM_KEY("adam_rbc1"), 1.f);
  g.adam_rbc2 = field<float>(d, FM_KEY("adam_rbc2"), 1.f);
  g.max_ctas = field<int>(d, FM_KEY("max_ctas"), 0);
  g.timeout_ns = field<unsigned long long>(d, FM_KEY("timeout_ns"), 0ull);
  g.wait_ns = reinterpret_cast<unsigned long long*>(field<uintptr_t>(d, FM_KEY("wait_ns"), 0));
  g.status = reinterpret_cast<int*>(field<uintptr_t>(d, FM_KEY("status"), 0));
  return g;
}
static void gemm_launch(const py::dict& d, uintptr_t stream) {
  const FmGemmDesc g = gemm_descriptor(d);
  check(fm_gemm_launch(&g, reinterpret_cast<cudaStream_t>(stream)), "fm_gemm_launch");
}
static long long gemm_workspace(const py::dict& d) {
  const FmGemmDesc g = gemm_descriptor(d);
  return fm_gemm_workspace(&g);
}

void bind_ops(py::module_& m);   // ops_bindings.cpp
void bind_symm(py::module_& m);  // symm_bindings.cpp

int fm_add_tensor_calls(PyObject* module);   // tensor_calls.cpp

PYBIND11_MODULE(_C, m) {
  m.doc() = "fluidmoe_b200 native kernels (sm_100a)";
  m.def("gemm_launch", &gemm_launch, py::arg("desc"), py::arg("stream"));
  m.def("gemm_workspace", &gemm_workspace, py::arg("desc"));
  m.def("last_error", []() { return std::string(fm_last_error()); });
  m.attr("EPI_STORE") = (int)FM_EPI_STORE;
  m.attr("EPI_ACT") = (int)FM_EPI_ACT;
  m.attr("EPI_SCATTER") = (int)FM_EPI_SCATTER;
  m.attr("EPI_DACT") = (int)FM_EPI_DACT;
  m.attr("EPI_COLSCATTER") = (int)FM_EPI_COLSCATTER;
  m.attr("EPI_ADAM") = (int)FM_EPI_ADAM;
  m.attr("ACT_GELU") = (int)FM_ACT_GELU;
  m.attr("ACT_SILU") = (int)FM_ACT_SILU;
  m.attr("ACT_NONE") = (int)FM_ACT_NONE;
  bind_ops(m);
  bind_symm(m);
  if (fm_add_tensor_calls(m.ptr()) != 0) throw py::error_already_set();
}
