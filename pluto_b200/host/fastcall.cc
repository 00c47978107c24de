// CPython binding of the C ABI for the per-call paths of pluto_b200.layers: one vectorcall function
// per entry point, arguments converted straight to the C types.  A ctypes call spends 1 to 5 us on
// the same (it grows with the number of arguments, and decode has 24); with launches at 3 to 4 us
// that is a large part of what a single-token call costs.
//
// Pointers come as integers (tensor.data_ptr()), None, or bytes objects (the cache descriptor that
// kv_cache() below packs).  The GIL is released around the call.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/pluto_b200.h"

namespace {

template <typename T>
bool convert(PyObject* o, T& value) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) {
      value = nullptr;
    } else if (PyBytes_Check(o)) {
      value = reinterpret_cast<T>(PyBytes_AS_STRING(o));
    } else {
      const unsigned long long bits = PyLong_AsUnsignedLongLong(o);
      if (bits == ~0ull && PyErr_Occurred()) return false;
      value = reinterpret_cast<T>(static_cast<uintptr_t>(bits));
    }
  } else if constexpr (std::is_floating_point_v<T>) {
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) return false;
    value = static_cast<T>(d);
  } else {
    const long long n = PyLong_AsLongLong(o);
    if (n == -1 && PyErr_Occurred()) return false;
    if constexpr (std::is_same_v<T, int>) {
      if (n < INT32_MIN || n > INT32_MAX) {
        PyErr_SetString(PyExc_OverflowError, "argument does not fit a C int");
        return false;
      }
    }
    value = static_cast<T>(n);
  }
  return true;
}

PyObject* to_python(int v) { return PyLong_FromLong(v); }
PyObject* to_python(size_t v) { return PyLong_FromSize_t(v); }

template <auto Function>
struct Entry;
template <typename R, typename... A, R (*Function)(A...)>
struct Entry<Function> {
  template <size_t... I>
  static PyObject* call(PyObject* const* args, std::index_sequence<I...>) {
    std::tuple<std::remove_const_t<A>...> values;
    if (!(convert(args[I], std::get<I>(values)) && ...)) return nullptr;
    R result;
    Py_BEGIN_ALLOW_THREADS
    result = Function(std::get<I>(values)...);
    Py_END_ALLOW_THREADS
    return to_python(result);
  }
  static PyObject* fastcall(PyObject*, PyObject* const* args, Py_ssize_t count) {
    if (count != static_cast<Py_ssize_t>(sizeof...(A))) {
      PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", static_cast<Py_ssize_t>(sizeof...(A)), count);
      return nullptr;
    }
    return call(args, std::index_sequence_for<A...>{});
  }
};

// kv_cache(k_base, v_base, block_table, max_blocks, page_size, page_stride, token_stride, dtype,
// num_pages) -> bytes: struct pluto_kv_cache of one pool.
PyObject* kv_cache(PyObject*, PyObject* const* args, Py_ssize_t count) {
  if (count != 9) {
    PyErr_SetString(PyExc_TypeError, "kv_cache takes 9 arguments");
    return nullptr;
  }
  pluto_kv_cache c = {};
  if (!convert(args[0], c.k_base) || !convert(args[1], c.v_base) || !convert(args[2], c.block_table) ||
      !convert(args[3], c.max_blocks) || !convert(args[4], c.page_size) || !convert(args[5], c.page_stride) ||
      !convert(args[6], c.token_stride) || !convert(args[7], c.dtype) || !convert(args[8], c.num_pages))
    return nullptr;
  return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&c), sizeof(c));
}

template <auto Function>
constexpr PyMethodDef entry(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Entry<Function>::fastcall)), METH_FASTCALL, nullptr};
}
#define ENTRY(name) entry<&name>(#name)

PyMethodDef methods[] = {
    ENTRY(pluto_attn_fwd),
    ENTRY(pluto_attn_bwd),
    ENTRY(pluto_attn_bwd_workspace_bytes),
    ENTRY(pluto_attn_probs),
    ENTRY(pluto_gqa_prefill_fwd),
    ENTRY(pluto_gqa_prefill_fwd_workspace_bytes),
    ENTRY(pluto_gqa_gate_bwd),
    ENTRY(pluto_gqa_prefill_bwd),
    ENTRY(pluto_gqa_prefill_bwd_workspace_bytes),
    ENTRY(pluto_qk_prepare_bwd),
    ENTRY(pluto_qk_prepare_bwd_workspace_bytes),
    ENTRY(pluto_qk_prepare),
    ENTRY(pluto_gqa_decode),
    ENTRY(pluto_gqa_decode_workspace_bytes),
    ENTRY(pluto_gqa_decode_noalloc),
    ENTRY(pluto_gqa_decode_probs),
    ENTRY(pluto_cached_attention_step),
    ENTRY(pluto_cached_attention_step_workspace_bytes),
    ENTRY(pluto_gdn_token_step),
    ENTRY(pluto_gdn_token_step_scratch_bytes),
    ENTRY(pluto_gdn_gates),
    ENTRY(pluto_gdn_conv_silu),
    ENTRY(pluto_gdn_prefill),
    ENTRY(pluto_gdn_prefill_workspace_bytes),
    ENTRY(pluto_gdn_step),
    ENTRY(pluto_gdn_out_norm_gate),
    ENTRY(pluto_gdn_out_norm_gate_bwd),
    ENTRY(pluto_gdn_out_norm_gate_bwd_workspace_bytes),
    ENTRY(pluto_gdn_recurrence_bwd),
    ENTRY(pluto_gdn_recurrence_bwd_workspace_bytes),
    ENTRY(pluto_gdn_conv_silu_bwd),
    ENTRY(pluto_linear_imported_fwd),
    ENTRY(pluto_dense_fwd),
    ENTRY(pluto_dense_bwd),
    ENTRY(pluto_dense_workspace_bytes),
    ENTRY(pluto_block_linear_fwd),
    ENTRY(pluto_block_linear_bwd),
    ENTRY(pluto_block_linear_workspace_bytes),
    ENTRY(pluto_dequantize_matrix),
    {"kv_cache", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&kv_cache)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&module); }
