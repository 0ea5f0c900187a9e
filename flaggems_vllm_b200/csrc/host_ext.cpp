// Native host path of the operators: argument checks, allocations and launches of the common cases in one C++ call
// each.  A decode-sized layer spends a few microseconds per kernel on the device; checked and launched from Python
// it cost the host 85 us, most of it interpreter time.
//
// Every function here serves the usual types, layouts and options and returns None for anything else (and for
// every error): the Python operator then goes its own way, which serves the rest and raises the errors.  Nothing
// is kept between calls.
#define PY_SSIZE_T_CLEAN
#include <ATen/ATen.h>
#include <Python.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <cstdlib>
#include <cstring>

#include "../../include/moe_sm100.h"

namespace {

std::atomic<int32_t*> g_status[64];        // status word of every device, registered by _lib.status_word

#define MOE_NONE Py_RETURN_NONE

bool is_tensor(PyObject* o) { return THPVariable_Check(o); }
const at::Tensor& tensor(PyObject* o) { return THPVariable_Unpack(o); }
bool truth(PyObject* o) { return o == Py_True; }
bool plain_bool(PyObject* o) { return o == Py_True || o == Py_False; }
bool as_int(PyObject* o, long long* v) {
  if (!PyLong_CheckExact(o)) return false;
  *v = PyLong_AsLongLong(o);
  if (*v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}
bool as_double(PyObject* o, double* v) {
  if (PyFloat_CheckExact(o)) { *v = PyFloat_AS_DOUBLE(o); return true; }
  long long i;
  if (!as_int(o, &i)) return false;
  *v = (double)i;
  return true;
}
// float32 -> MOE_F32 ..., -1 otherwise
int float_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return MOE_F32;
    case at::kHalf: return MOE_F16;
    case at::kBFloat16: return MOE_BF16;
    default: return -1;
  }
}
bool cuda_dense(const at::Tensor& t, int dev) { return t.is_cuda() && t.get_device() == dev && t.is_contiguous(); }
bool set_on(const char* name) { return std::getenv(name) != nullptr; }
at::Tensor bytes_on(int64_t n, const at::Tensor& like) { return at::empty({n}, like.options().dtype(at::kByte)); }

// a switch that pins one of the other kernels, or asks for a status check after the call
bool switched() {
  static const char* const names[] = {"FLAGGEMS_B200_GENERIC_GEMM", "FLAGGEMS_B200_TC_WIDE", "FLAGGEMS_B200_TC_PAIR",
                                      "FLAGGEMS_B200_TC_PAIR_WIDE", "FLAGGEMS_B200_PRESORT", "FLAGGEMS_B200_TMA_OUT",
                                      "FLAGGEMS_B200_SMALL_M", "FLAGGEMS_B200_W8_WIDEN", "FLAGGEMS_B200_CHECK_STATUS"};
  for (const char* n : names)
    if (set_on(n)) return true;
  return false;
}

PyObject* set_status(PyObject*, PyObject* const* a, Py_ssize_t n) {
  long long dev, ptr;
  if (n != 2 || !as_int(a[0], &dev) || !as_int(a[1], &ptr) || dev < 0 || dev >= 64) {
    PyErr_SetString(PyExc_ValueError, "set_status(device, pointer)");
    return nullptr;
  }
  g_status[dev].store(reinterpret_cast<int32_t*>(ptr));
  MOE_NONE;
}

// The interpreter lock is given back for as long as a function allocates and launches: cudaMalloc may wait for the
// device, and a launch waits when the stream's queue is full, while the work it waits for may need another thread
// of the process (another stream's, another rank's).  Nothing between the braces of its scope touches a Python object.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  Unlocked() = default;
  Unlocked(const Unlocked&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state); }
};

int32_t* status_of(int dev) { return dev >= 0 && dev < 64 ? g_status[dev].load(std::memory_order_relaxed) : nullptr; }

// fused_experts(hidden, w1, w2, topk_weights, topk_ids, inplace, activation, apply_router_weight_on_input, use_fp8_w8a8,
//   use_int8_w8a8, use_int8_w8a16, use_int4_w4a16, per_channel_quant, global_num_experts, expert_map, w1_scale, w2_scale,
//   a1_scale, a2_scale, block_shape)
PyObject* fused_experts(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 20) MOE_NONE;
  for (int i = 0; i < 5; ++i)
    if (!is_tensor(a[i])) MOE_NONE;
  for (int i : {5, 7, 8, 9, 10, 11, 12})
    if (!plain_bool(a[i])) MOE_NONE;
  const at::Tensor &x = tensor(a[0]), &w1 = tensor(a[1]), &w2 = tensor(a[2]), &tw = tensor(a[3]), &ti = tensor(a[4]);
  const char* act = PyUnicode_Check(a[6]) ? PyUnicode_AsUTF8(a[6]) : nullptr;
  if (!act || std::strcmp(act, "silu") != 0 || a[17] != Py_None || a[18] != Py_None) MOE_NONE;
  long long ng;
  if (!as_int(a[13], &ng)) MOE_NONE;
  if (!x.is_cuda() || x.dim() != 2 || w1.dim() != 3 || w2.dim() != 3 || ti.dim() != 2 || switched()) MOE_NONE;
  const int dev = x.get_device();
  const int code = float_code(x);
  if ((code != MOE_F16 && code != MOE_BF16) || !cuda_dense(x, dev) || !cuda_dense(w1, dev) || !cuda_dense(w2, dev) ||
      !cuda_dense(tw, dev) || !cuda_dense(ti, dev))
    MOE_NONE;
  const int64_t M = x.size(0), H = x.size(1), E = w1.size(0), N = w1.size(1), k = ti.size(1), I = N / 2;
  if (M <= 0 || M > 32768 || w1.size(2) != H || N % 2 != 0 || w2.size(0) != E || w2.size(1) != H || w2.size(2) != I ||
      ti.size(0) != M || !tw.sizes().equals(ti.sizes()) || tw.scalar_type() != at::kFloat)
    MOE_NONE;
  const bool ids64 = ti.scalar_type() == at::kLong;
  if (!ids64 && ti.scalar_type() != at::kInt) MOE_NONE;
  const bool fp8 = truth(a[8]), i8 = truth(a[9]), weight_only = truth(a[10]) || truth(a[11]), per_channel = truth(a[12]);
  const at::Tensor *s1 = nullptr, *s2 = nullptr;
  int mode = MOE_MODE_HALF, kind = 0;
  if (fp8 || i8 || weight_only) {
    if (!is_tensor(a[15]) || !is_tensor(a[16])) MOE_NONE;
    s1 = &tensor(a[15]);
    s2 = &tensor(a[16]);
    if (!cuda_dense(*s1, dev) || !cuda_dense(*s2, dev) || s1->scalar_type() != at::kFloat || s2->scalar_type() != at::kFloat) MOE_NONE;
    const at::ScalarType wt = fp8 ? at::kFloat8_e4m3fn : at::kChar;
    if (w1.scalar_type() != wt || w2.scalar_type() != wt) MOE_NONE;
    if (fp8 && a[19] != Py_None) {
      long long b0, b1;
      if (i8 || per_channel || !PyList_CheckExact(a[19]) || PyList_GET_SIZE(a[19]) != 2 || !as_int(PyList_GET_ITEM(a[19], 0), &b0) ||
          !as_int(PyList_GET_ITEM(a[19], 1), &b1) || b0 != 128 || b1 != 128 || H % 128 != 0 || I % 128 != 0)
        MOE_NONE;
      if (!s1->sizes().equals({E, N / 128, H / 128}) || !s2->sizes().equals({E, H / 128, I / 128})) MOE_NONE;
      mode = MOE_MODE_FP8_BLOCK;
    } else {
      if (a[19] != Py_None || s1->numel() != E * N || s2->numel() != E * H) MOE_NONE;
      if (fp8 || i8) {
        if (fp8 == i8 || !per_channel) MOE_NONE;  // per-tensor scales: the Python path
        mode = fp8 ? MOE_MODE_FP8_ROW : MOE_MODE_INT8_ROW;
        kind = fp8 ? 1 : 0;
      } else {
        mode = MOE_MODE_W8A16;
      }
    }
  } else if (w1.scalar_type() != x.scalar_type() || w2.scalar_type() != x.scalar_type()) {
    MOE_NONE;
  }
  const int32_t* emap = nullptr;
  const int64_t experts = ng == -1 ? E : ng;
  if (a[14] != Py_None) {
    if (!is_tensor(a[14])) MOE_NONE;
    const at::Tensor& m = tensor(a[14]);
    if (!cuda_dense(m, dev) || m.scalar_type() != at::kInt || m.numel() < experts) MOE_NONE;
    emap = m.const_data_ptr<int32_t>();
  }
  int32_t* status = status_of(dev);
  int64_t bytes[4];
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);  // what is served depends on the device
  if (status == nullptr || experts <= 0 || experts > (1 << 20) ||
      moe_layer_workspace(mode, code, M, (int)k, (int)experts, (int)E, (int)H, (int)I, MOE_ACT_SILU, bytes) != 0)
    MOE_NONE;
  const bool inplace = truth(a[5]), weight_on_input = truth(a[7]);
  at::Tensor out;
  int rc;
  {
    Unlocked unlocked;
    out = inplace ? x : at::empty_like(x);
    at::Tensor ws[4];
    for (int i = 0; i < 4; ++i) ws[i] = bytes_on(bytes[i], x);
    rc = moe_layer(mode, code, x.const_data_ptr(), M, (int)k, ti.const_data_ptr(), ids64, tw.const_data_ptr<float>(),
                   w1.const_data_ptr(), s1 ? s1->const_data_ptr<float>() : nullptr, w2.const_data_ptr(),
                   s2 ? s2->const_data_ptr<float>() : nullptr, out.mutable_data_ptr(), (int)experts, emap, (int)E, (int)H,
                   (int)I, weight_on_input, MOE_ACT_SILU, 0.0f, 0.0f, 0.0f, kind, nullptr, kind, nullptr, ws[0].mutable_data_ptr(),
                   ws[1].mutable_data_ptr(), ws[2].mutable_data_ptr(), ws[3].mutable_data_ptr(), 63, status,
                   c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
  }
  if (rc != 0) MOE_NONE;
  if (inplace) {
    Py_INCREF(a[0]);
    return a[0];
  }
  return THPVariable_Wrap(out);
}

// grouped_topk(scores, n_group, topk_group, topk, renormalize, scaling, bias, scoring_func) -> (weights, ids)
PyObject* grouped_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8 || !is_tensor(a[0]) || !is_tensor(a[6]) || !plain_bool(a[4])) MOE_NONE;
  const at::Tensor &s = tensor(a[0]), &b = tensor(a[6]);
  long long groups, keep, k, func;
  double scale;
  if (!as_int(a[1], &groups) || !as_int(a[2], &keep) || !as_int(a[3], &k) || !as_int(a[7], &func) || !as_double(a[5], &scale)) MOE_NONE;
  if (!s.is_cuda() || s.dim() != 2 || b.dim() != 1) MOE_NONE;
  const int dev = s.get_device();
  const int64_t M = s.size(0), E = s.size(1);
  const int sc = float_code(s), bc = float_code(b);
  if (sc < 0 || bc < 0 || !cuda_dense(b, dev) || b.numel() != E || M <= 0 || groups <= 0 || groups > 32 || E % groups != 0 || k <= 0 ||
      k > 32 || (func != 0 && func != 1))
    MOE_NONE;
  const bool renormalize = truth(a[4]);
  at::Tensor w, ids;
  int rc;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    w = at::empty({M, k}, s.options().dtype(at::kFloat));
    ids = at::empty({M, k}, s.options().dtype(at::kInt));
    rc = moe_grouped_topk(s.const_data_ptr(), sc, s.stride(0), s.stride(1), b.const_data_ptr(), bc, nullptr, M, (int)E, (int)groups,
                          (int)keep, (int)k, renormalize, (float)scale, (int)func, w.mutable_data_ptr<float>(),
                          ids.mutable_data_ptr<int32_t>(), c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
  }
  if (rc != 0) MOE_NONE;
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(w));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(ids));
  return r;
}

// topk_route(weights, ids, rows, gating, renormalize, bias, sigmoid, scale) -> True when done
PyObject* topk_route(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8 || !plain_bool(a[4]) || !plain_bool(a[6])) MOE_NONE;
  for (int i = 0; i < 4; ++i)
    if (!is_tensor(a[i])) MOE_NONE;
  const at::Tensor &w = tensor(a[0]), &ids = tensor(a[1]), &rows = tensor(a[2]), &g = tensor(a[3]);
  double scale;
  if (!as_double(a[7], &scale) || !g.is_cuda() || g.dim() != 2 || w.dim() != 2) MOE_NONE;
  const int dev = g.get_device();
  const int64_t M = g.size(0), E = g.size(1), k = w.size(1);
  const int gc = float_code(g);
  const int kind = ids.scalar_type() == at::kInt ? 0 : (ids.scalar_type() == at::kLong ? 1 : -1);
  if (gc < 0 || kind < 0 || !cuda_dense(g, dev) || !cuda_dense(w, dev) || !cuda_dense(ids, dev) || !cuda_dense(rows, dev) ||
      w.scalar_type() != at::kFloat || rows.scalar_type() != at::kInt || w.size(0) != M || !ids.sizes().equals(w.sizes()) ||
      !rows.sizes().equals(w.sizes()) || M <= 0 || k <= 0 || k > 32 || k > E || E > 1024)
    MOE_NONE;
  const float* bias = nullptr;
  if (a[5] != Py_None) {
    if (!is_tensor(a[5])) MOE_NONE;
    const at::Tensor& b = tensor(a[5]);
    if (!cuda_dense(b, dev) || b.scalar_type() != at::kFloat || b.dim() != 1 || b.numel() != E) MOE_NONE;
    bias = b.const_data_ptr<float>();
  }
  const bool sigmoid = truth(a[6]), renormalize = truth(a[4]);
  int rc;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    rc = moe_topk_route(g.const_data_ptr(), gc, bias, nullptr, M, (int)E, (int)k, sigmoid, renormalize, (float)scale,
                        w.mutable_data_ptr<float>(), ids.mutable_data_ptr(), kind, rows.mutable_data_ptr<int32_t>(),
                        c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
  }
  if (rc != 0) MOE_NONE;
  Py_RETURN_TRUE;
}

// router_gemm(x, weight) -> fp32 logits
PyObject* router_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !is_tensor(a[0]) || !is_tensor(a[1])) MOE_NONE;
  const at::Tensor &x = tensor(a[0]), &w = tensor(a[1]);
  if (!x.is_cuda() || x.dim() != 2 || w.dim() != 2) MOE_NONE;
  const int dev = x.get_device(), xc = float_code(x), wc = float_code(w);
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  int32_t* status = status_of(dev);
  if (xc < 0 || wc < 0 || !status || !cuda_dense(w, dev) || w.size(1) != K || M <= 0 || K % 8 != 0 || x.stride(1) != 1 ||
      x.stride(0) % 8 != 0 || ((uintptr_t)x.const_data_ptr() & 15) || N > (1 << 30) || K > (1 << 30))
    MOE_NONE;
  at::Tensor out;
  int rc;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    out = at::empty({M, N}, x.options().dtype(at::kFloat));
    rc = moe_router_gemm_ex(x.const_data_ptr(), xc, x.stride(0), w.const_data_ptr(), wc, M, (int)N, (int)K,
                            out.mutable_data_ptr<float>(), status, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
  }
  if (rc != 0) MOE_NONE;
  return THPVariable_Wrap(out);
}

// align(topk_ids, num_experts, block_size, capacity) -> (sorted_ids, expert_ids, num_tokens_post_pad)
PyObject* align(PyObject*, PyObject* const* a, Py_ssize_t n) {
  long long E, bs, cap;
  if (n != 4 || !is_tensor(a[0]) || !as_int(a[1], &E) || !as_int(a[2], &bs) || !as_int(a[3], &cap)) MOE_NONE;
  const at::Tensor& ids = tensor(a[0]);
  if (!ids.is_cuda() || !ids.is_contiguous() || E <= 0 || E > 4096 || bs <= 0 || bs > (1 << 20) || cap < 0) MOE_NONE;
  const int dev = ids.get_device();
  const bool ids64 = ids.scalar_type() == at::kLong;
  int32_t* status = status_of(dev);
  if ((!ids64 && ids.scalar_type() != at::kInt) || !status) MOE_NONE;
  const int64_t blocks = (cap + bs - 1) / bs;
  at::Tensor sorted, experts, npp;
  int rc;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    const auto opt = ids.options().dtype(at::kInt);
    sorted = at::empty({cap}, opt);
    experts = at::empty({blocks}, opt);
    npp = at::empty({1}, opt);
    rc = moe_align_block_size(ids.const_data_ptr(), ids64, ids.numel(), (int)E, (int)bs, sorted.mutable_data_ptr<int32_t>(), cap,
                              experts.mutable_data_ptr<int32_t>(), blocks, npp.mutable_data_ptr<int32_t>(), status,
                              c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
  }
  if (rc != 0) MOE_NONE;
  PyObject* r = PyTuple_New(3);
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(sorted));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(experts));
  PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(npp));
  return r;
}

// No C++ exception crosses into the interpreter (an allocation can throw): it becomes the Python path's problem.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  try {
    return F(self, a, n);
  } catch (const std::exception&) {
    MOE_NONE;
  }
}

#define MOE_FN(name) {#name, (PyCFunction)(void (*)(void))guarded<name>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {MOE_FN(set_status), MOE_FN(fused_experts), MOE_FN(grouped_topk), MOE_FN(topk_route),
                         MOE_FN(router_gemm), MOE_FN(align), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_ext", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ext(void) { return PyModule_Create(&module); }
