// Python calls of the C ABI (include/b200_paged.h) without ctypes: every function of the table below takes tensors, None and plain
// numbers and passes data pointers, int and float values on; a call that leaves out the last argument, the stream, runs on the caller's
// current one.  A call's arguments are converted by the types of its prototype.  new(like, dtype, *shape) allocates beside a tensor.
// Host time of a wrapper in ops.py, measured with ctypes / here: rmsnorm 7.3 / 4.1 us, gemm 11.6 / 5.6 us, of which the launch is 2.5 - 3.5:
// decode steps of the hybrid decoders and short prompts, 130 - 160 launches each, were bound by it.
#include <Python.h>

#include <ATen/Functions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <limits>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/b200_paged.h"

namespace {

PyObject* g_error = nullptr;  // vllm_neuron_b200._cabi.B200Error

struct Raised {};  // a Python exception is set

struct Unlocked {  // other threads run Python meanwhile; taken back also where a C++ exception passes
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

template <typename T>
T arg(PyObject* o) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) return nullptr;
    if (THPVariable_Check(o)) {
      const at::Tensor& t = THPVariable_Unpack(o);
      if (!t.is_cuda()) {
        PyErr_SetString(g_error ? g_error : PyExc_RuntimeError, "b200 ops need CUDA tensors (no CPU fallback)");
        throw Raised{};
      }
      return (T)t.data_ptr();
    }
    void* p = PyLong_AsVoidPtr(o);
    if (!p && PyErr_Occurred()) throw Raised{};
    return (T)p;
  } else if constexpr (std::is_floating_point_v<T>) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Raised{};
    return (T)v;
  } else {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Raised{};
    if (sizeof(T) < sizeof(v) && (v < (long long)std::numeric_limits<T>::min() || v > (long long)std::numeric_limits<T>::max())) {
      PyErr_Format(PyExc_OverflowError, "%lld does not fit the argument's type", v);
      throw Raised{};
    }
    return (T)v;
  }
}

template <auto Fn>
struct Call;
template <typename R, typename... A, R (*Fn)(A...)>
struct Call<Fn> {
  static constexpr Py_ssize_t N = sizeof...(A);
  static constexpr bool streamed = std::is_same_v<std::tuple_element_t<N, std::tuple<int, A...>>, void*>;
  template <size_t... I>
  static R run(PyObject* const* args, Py_ssize_t n, std::index_sequence<I...>) {
    std::tuple<A...> v{(Py_ssize_t)I < n ? arg<A>(args[I]) : A{}...};
    if constexpr (streamed) {
      if (n == N - 1) std::get<N - 1>(v) = (void*)c10::cuda::getCurrentCUDAStream().stream();
    }
    Unlocked u;  // a full launch queue blocks here
    return std::apply(Fn, v);
  }
  static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != N && !(streamed && n == N - 1)) {
      PyErr_Format(PyExc_TypeError, "%zd arguments given, %zd expected", n, N);
      return nullptr;
    }
    try {
      const R r = run(args, n, std::index_sequence_for<A...>{});
      if constexpr (std::is_signed_v<R>) return PyLong_FromLongLong(r);
      else return PyLong_FromUnsignedLongLong(r);
    } catch (const Raised&) {
      return nullptr;
    }
    END_HANDLE_TH_ERRORS
  }
};

// new(like, dtype or None, *shape): an uninitialised contiguous tensor on like's device
PyObject* new_tensor(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 2 || n > 8 || !THPVariable_Check(args[0]) || !(args[1] == Py_None || THPDtype_Check(args[1]))) {
    PyErr_SetString(PyExc_TypeError, "new(like, dtype or None, *shape)");
    return nullptr;
  }
  const at::Tensor& like = THPVariable_Unpack(args[0]);
  int64_t shape[6];
  for (Py_ssize_t i = 2; i < n; ++i) {
    shape[i - 2] = PyLong_AsLongLong(args[i]);
    if (shape[i - 2] == -1 && PyErr_Occurred()) return nullptr;
  }
  const at::ScalarType type = args[1] == Py_None ? like.scalar_type() : reinterpret_cast<THPDtype*>(args[1])->scalar_type;
  const auto options = at::TensorOptions().dtype(type).device(like.device());
  at::Tensor made;
  {
    Unlocked u;  // an allocation that gives cached blocks back waits for the device
    made = at::empty(at::IntArrayRef(shape, n - 2), options);
  }
  return THPVariable_Wrap(std::move(made));
  END_HANDLE_TH_ERRORS
}

PyObject* set_error(PyObject*, PyObject* type) {
  Py_INCREF(type);
  Py_XSETREF(g_error, type);
  Py_RETURN_NONE;
}

#define FN(name) {#name, (PyCFunction)(void (*)(void))Call<&name>::call, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"new", (PyCFunction)(void (*)(void))new_tensor, METH_FASTCALL, nullptr},
    {"set_error", set_error, METH_O, nullptr},
    FN(b200_add_group_rmsnorm), FN(b200_advance_decode), FN(b200_argmax), FN(b200_batched_linear), FN(b200_bias_act),
    FN(b200_block_table_scatter), FN(b200_build_decode_meta), FN(b200_build_prefill_meta), FN(b200_causal_conv), FN(b200_clamped_glu),
    FN(b200_delta_prep), FN(b200_delta_scan), FN(b200_diff_head_norm_gate), FN(b200_dyt_norm), FN(b200_dyt_residual), FN(b200_embed_bigram),
    FN(b200_embed_rmsnorm), FN(b200_embed_scale), FN(b200_embedding), FN(b200_gated_group_rmsnorm), FN(b200_gated_scan),
    FN(b200_gated_scan_prep), FN(b200_gather_logprobs), FN(b200_gemm), FN(b200_gemm_rope_kv_write), FN(b200_gemm_silu_mul),
    FN(b200_gemm_silu_mul_quant), FN(b200_gemm_workspace_bytes), FN(b200_glu), FN(b200_grouped_linear), FN(b200_head_rmsnorm_gate),
    FN(b200_hyper_embed), FN(b200_hyper_residual), FN(b200_kv_pool_mean), FN(b200_kv_write), FN(b200_kv_write_vmix),
    FN(b200_latent_attn_decode), FN(b200_latent_attn_decode_split), FN(b200_latent_attn_prefill_tc), FN(b200_latent_attn_prefill_tc_supported), FN(b200_latent_kv_write), FN(b200_latent_q_prep), FN(b200_matrix_memory_gates), FN(b200_matrix_memory_out),
    FN(b200_matrix_memory_scan), FN(b200_moe_align), FN(b200_moe_gather_scale), FN(b200_moe_tile_rows), FN(b200_moe_topk),
    FN(b200_moe_topk_grouped), FN(b200_paged_attn_decode), FN(b200_paged_attn_decode_workspace_bytes), FN(b200_paged_attn_prefill),
    FN(b200_poly_norm), FN(b200_postln_residual), FN(b200_qk_norm_rope_kv_write), FN(b200_quantize_per_token), FN(b200_remask_spec_output),
    FN(b200_rms_residual), FN(b200_rmsnorm), FN(b200_rmsnorm_cols), FN(b200_rope_kv_write), FN(b200_row_lse), FN(b200_sample_candidates),
    FN(b200_scaled_add_rmsnorm2), FN(b200_selective_scan), FN(b200_silu_mul), FN(b200_ssd_scan_mma), FN(b200_ssd_step),
    FN(b200_swa_sink_attn), FN(b200_swa_sink_attn_decode_tc), FN(b200_swa_sink_attn_prefill), FN(b200_swa_attn_prefill_tc_sink),
    FN(b200_swa_sink_attn_prefill_tc_supported), FN(b200_topk_candidates),
    {nullptr, nullptr, 0, nullptr}};
#undef FN

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200_bind", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200_bind(void) {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "torch", B200_BIND_TORCH) < 0) Py_CLEAR(m);
  return m;
}
