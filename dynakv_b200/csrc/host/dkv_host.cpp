// Native host side of the Python entry points: turns torch tensors into the C ABI's argument structs and launches.
//
// A decode step is two short kernels per layer; marshalling them through ctypes costs 25-45 us of Python per call, more
// than the kernels take on small caches.  The functions here do the same work in 3-5 us.  Each of them handles the plain
// case -- CUDA tensors of the documented shapes, types and layouts -- and returns None for anything else, without having
// launched or changed anything; the Python callers then take their own path, which copies what has to be copied and
// raises what has to be raised.  No state is kept between calls but the address of each device's status word.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>

#include "../../../include/dynakv_b200.h"

namespace {

constexpr int MAX_DEVICES = 64;
int32_t* g_status[MAX_DEVICES];

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return DKV_F32;
    case at::kHalf: return DKV_F16;
    case at::kBFloat16: return DKV_BF16;
    default: return -1;
  }
}

bool is_tensor(PyObject* o) { return THPVariable_Check(o); }
const at::Tensor& unpack(PyObject* o) { return THPVariable_Unpack(o); }
// a plain CUDA tensor on `dev` (no subclass that wants to see the call, no gradient to record)
bool plain(PyObject* o, int dev) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = unpack(o);
  return t.is_cuda() && t.get_device() == dev && !t.requires_grad();
}
void* stream_of(int dev) { return at::cuda::getCurrentCUDAStream(dev).stream(); }

// [rows, X] or [B, H, X] whose first two axes fold into one without a copy
bool fold(const at::Tensor& t, int64_t& rows, int64_t& cols, int64_t& stride_r, int64_t& stride_c) {
  if (t.dim() == 2) {
    rows = t.size(0); cols = t.size(1); stride_r = t.stride(0); stride_c = t.stride(1);
    return true;
  }
  if (t.dim() != 3 || (t.size(0) > 1 && t.stride(0) != t.size(1) * t.stride(1))) return false;
  rows = t.size(0) * t.size(1); cols = t.size(2); stride_r = t.stride(1); stride_c = t.stride(2);
  return true;
}

bool fill_side(dkv_side& s, const at::Tensor& flat, const at::Tensor& lens, const at::Tensor& offs, int64_t& rows, int64_t& tokens) {
  int64_t fr, fc, fs, fe, or_, oc, os, oe, ls, le;
  if (!fold(flat, fr, fc, fs, fe) || !fold(lens, rows, tokens, ls, le) || !fold(offs, or_, oc, os, oe)) return false;
  if (fe != 1 || fr != rows || or_ != rows || oc != tokens || lens.scalar_type() != at::kInt || offs.scalar_type() != at::kInt) return false;
  s.flat = flat.data_ptr();
  s.flat_stride = fs;
  s.lens = static_cast<int32_t*>(lens.data_ptr());
  s.lens_stride_a = ls;
  s.lens_stride_s = tokens > 1 ? le : 1;
  s.offs = static_cast<int32_t*>(offs.data_ptr());
  s.offs_stride_a = os;
  s.offs_stride_s = tokens > 1 ? oe : 1;
  s.ptr = nullptr;
  return true;
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dt, const at::Device& dev) {
  return at::Tensor(at::detail::empty_cuda(sizes, dt, dev, std::nullopt));
}

// A [rows, cols] view of int or data rows inside `base` (no autograd here: a tensor over the same storage is all a view has
// to be, and costs a tenth of what a dispatched narrow() does).
at::Tensor rows_view(const at::Tensor& base, int64_t offset, at::IntArrayRef sizes, at::IntArrayRef strides) {
  at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(base.storage()), base.key_set(), base.dtype());
  t.unsafeGetTensorImpl()->set_storage_offset(base.storage_offset() + offset);
  t.unsafeGetTensorImpl()->set_sizes_and_strides(sizes, strides);
  return t;
}

// a runtime call that failed here: raised once, and not found again by the launch check of the next call
PyObject* fail(const char* what, cudaError_t e) {
  cudaGetLastError();
  PyErr_Format(PyExc_RuntimeError, "%s failed: %s", what, cudaGetErrorString(e));
  return nullptr;
}
PyObject* fail(const char* what, int rc) {
  PyErr_Format(PyExc_RuntimeError, "%s failed (code %d): %s", what, rc, dkv_last_error());
  return nullptr;
}

// attend(q, k_flat, k_up, v_flat, v_up, l_k, o_k, l_v, o_v, theta, out|None, seq_lens|None, batch_index|None,
//        k_norm_weight|None, k_norm_eps, len_multiple, route_min, route_max, two_stage) -> out; an integer in place of the last
// is a switch point: every row through the kernel of its own length
PyObject* attend(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 19 || !is_tensor(v[0]) || !unpack(v[0]).is_cuda()) Py_RETURN_NONE;
  const int dev = unpack(v[0]).get_device();
  if (dev < 0 || dev >= MAX_DEVICES || g_status[dev] == nullptr) Py_RETURN_NONE;
  for (int i = 0; i < 9; ++i)
    if (!plain(v[i], dev)) Py_RETURN_NONE;
  for (int i = 10; i < 14; ++i)
    if (v[i] != Py_None && !plain(v[i], dev)) Py_RETURN_NONE;
  const at::Tensor &q = unpack(v[0]), &k_up = unpack(v[2]), &v_up = unpack(v[4]), &k_flat = unpack(v[1]), &v_flat = unpack(v[3]);
  const auto dt = q.scalar_type();
  dkv_attn_args a = {};
  a.dtype = dtype_code(dt);
  const bool q4 = q.dim() == 4;
  if (a.dtype < 0 || !(q.dim() == 3 || (q4 && q.size(2) == 1)) || q.stride(-1) != 1) Py_RETURN_NONE;
  if (k_up.dim() != 3 || v_up.sizes() != k_up.sizes() || !k_up.is_contiguous() || !v_up.is_contiguous()) Py_RETURN_NONE;
  if (k_flat.scalar_type() != dt || v_flat.scalar_type() != dt || k_up.scalar_type() != dt || v_up.scalar_type() != dt) Py_RETURN_NONE;
  const int64_t B = q.size(0), Hq = q.size(1), D = q.size(q4 ? 3 : 2);
  if (B == 0 || k_up.size(2) != D) Py_RETURN_NONE;
  int64_t rows_k, rows_v, S_k, S_v;
  if (!fill_side(a.k, k_flat, unpack(v[5]), unpack(v[6]), rows_k, S_k) || !fill_side(a.v, v_flat, unpack(v[7]), unpack(v[8]), rows_v, S_v)) Py_RETURN_NONE;
  if (rows_k != rows_v || S_k != S_v || rows_k % B != 0) Py_RETURN_NONE;
  a.n_q_heads = (int32_t)Hq;
  a.n_basis_groups = (int32_t)k_up.size(0);
  a.head_dim = (int32_t)D;
  a.rank = (int32_t)k_up.size(1);
  a.arenas_per_batch = (int32_t)(rows_k / B);
  a.seq_len = (int32_t)S_k;
  a.q = q.data_ptr();
  a.q_stride_b = q.stride(0);
  a.q_stride_h = q.stride(1);
  a.k_up = k_up.data_ptr();
  a.v_up = v_up.data_ptr();
  a.theta = (float)PyFloat_AsDouble(v[9]);
  a.batch = (int32_t)B;
  if (v[11] != Py_None) {
    const at::Tensor& t = unpack(v[11]);
    if (t.scalar_type() != at::kInt || t.numel() != B || !t.is_contiguous()) Py_RETURN_NONE;
    a.seq_lens = static_cast<const int32_t*>(t.data_ptr());
  }
  if (v[12] != Py_None) {
    const at::Tensor& t = unpack(v[12]);
    if (t.scalar_type() != at::kInt || !t.is_contiguous()) Py_RETURN_NONE;
    a.batch_index = static_cast<const int32_t*>(t.data_ptr());
    a.batch = (int32_t)t.numel();
  }
  if (v[13] != Py_None) {
    const at::Tensor& t = unpack(v[13]);
    if (t.scalar_type() != at::kFloat || !t.is_contiguous()) Py_RETURN_NONE;
    a.k_norm_weight = static_cast<const float*>(t.data_ptr());
  }
  a.k_norm_eps = (float)PyFloat_AsDouble(v[14]);
  a.len_multiple = (int32_t)PyLong_AsLong(v[15]);
  a.route_min_tokens = (int32_t)PyLong_AsLong(v[16]);
  a.route_max_tokens = (int32_t)PyLong_AsLong(v[17]);
  if (PyErr_Occurred()) return nullptr;
  if ((a.route_min_tokens || a.route_max_tokens) && a.seq_lens == nullptr) Py_RETURN_NONE;
  a.status = g_status[dev];
  a.stream = stream_of(dev);
  at::Tensor out;
  if (v[10] != Py_None) {
    out = unpack(v[10]);
    if (out.scalar_type() != dt || out.dim() != 3 || out.stride(2) != 1) Py_RETURN_NONE;
  } else {
    out = empty({B, Hq, D}, dt, q.device());
  }
  a.out = out.data_ptr();
  a.out_stride_b = out.stride(0);
  a.out_stride_h = out.stride(1);
  const bool two_stage = v[18] == Py_True, routed = !PyBool_Check(v[18]);
  const long switch_tokens = routed ? PyLong_AsLong(v[18]) : 0;
  if (PyErr_Occurred()) return nullptr;
  if (routed && a.seq_lens == nullptr) Py_RETURN_NONE;
  const size_t need = two_stage || routed ? dkv_split_workspace_bytes(&a) : dkv_fused_workspace_bytes(&a);
  at::Tensor ws;
  if (need) {
    ws = empty({(int64_t)need}, at::kByte, q.device());
    a.workspace = ws.data_ptr();
    a.workspace_bytes = need;
  }
  const int rc = routed ? dkv_routed_decode(&a, (int32_t)switch_tokens) : two_stage ? dkv_two_stage_decode(&a) : dkv_fused_decode(&a);
  if (rc) return fail(routed ? "dkv_routed_decode" : two_stage ? "dkv_two_stage_decode" : "dkv_fused_decode", rc);
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// The arguments that the two stage operators share: one side of the cache and its basis, [B, Hq] rows of type `like`.
bool operator_args(dkv_attn_args& a, const at::Tensor& like, dkv_side& side, PyObject* flat, PyObject* lens, PyObject* offs, const at::Tensor& up, int dev) {
  a.dtype = dtype_code(like.scalar_type());
  if (a.dtype < 0 || up.dim() != 3 || !up.is_contiguous() || up.scalar_type() != like.scalar_type() || unpack(flat).scalar_type() != like.scalar_type())
    return false;
  const int64_t B = like.size(0);
  int64_t rows, tokens;
  if (B == 0 || !fill_side(side, unpack(flat), unpack(lens), unpack(offs), rows, tokens) || rows % B != 0 || tokens == 0) return false;
  a.n_q_heads = (int32_t)like.size(1);
  a.n_basis_groups = (int32_t)up.size(0);
  a.rank = (int32_t)up.size(1);
  a.head_dim = (int32_t)up.size(2);
  a.arenas_per_batch = (int32_t)(rows / B);
  a.batch = (int32_t)B;
  a.seq_len = (int32_t)tokens;
  a.theta = 10000.f;
  a.len_multiple = 1;
  a.status = g_status[dev];
  a.stream = stream_of(dev);
  return true;
}
// whether the first argument is a CUDA tensor and all of them are plain tensors on its device, whose status word is known
int operator_device(PyObject* const* v, int n) {
  if (!is_tensor(v[0]) || !unpack(v[0]).is_cuda()) return -1;
  const int dev = unpack(v[0]).get_device();
  if (dev < 0 || dev >= MAX_DEVICES || g_status[dev] == nullptr) return -1;
  for (int i = 0; i < n; ++i)
    if (!plain(v[i], dev)) return -1;
  return dev;
}

// scores(q, k_up, k_flat, lens, offs, theta) -> scaled scores [B, Hq, S]
PyObject* scores(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = n == 6 ? operator_device(v, 5) : -1;
  if (dev < 0) Py_RETURN_NONE;
  const at::Tensor &q = unpack(v[0]), &up = unpack(v[1]);
  dkv_attn_args a = {};
  if (q.dim() != 3 || q.stride(2) != 1 || !operator_args(a, q, a.k, v[2], v[3], v[4], up, dev) || q.size(2) != up.size(2)) Py_RETURN_NONE;
  a.q = q.data_ptr();
  a.q_stride_b = q.stride(0);
  a.q_stride_h = q.stride(1);
  a.k_up = up.data_ptr();
  a.theta = (float)PyFloat_AsDouble(v[5]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor out = empty({q.size(0), q.size(1), a.seq_len}, q.scalar_type(), q.device());
  a.out = out.data_ptr();
  a.out_stride_b = out.stride(0);
  a.out_stride_h = out.stride(1);
  if (int rc = dkv_scores(&a)) return fail("dkv_scores", rc);
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// softmax_v(scores, v_flat, v_up, lens, offs) -> [B, Hq, D]
PyObject* softmax_v(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = n == 5 ? operator_device(v, 5) : -1;
  if (dev < 0) Py_RETURN_NONE;
  const at::Tensor &sc = unpack(v[0]), &up = unpack(v[2]);
  dkv_attn_args a = {};
  if (sc.dim() != 3 || sc.stride(2) != 1 || !operator_args(a, sc, a.v, v[1], v[3], v[4], up, dev)) Py_RETURN_NONE;
  a.v_up = up.data_ptr();
  const at::Tensor out = empty({sc.size(0), sc.size(1), up.size(2)}, sc.scalar_type(), sc.device());
  a.out = out.data_ptr();
  a.out_stride_b = out.stride(0);
  a.out_stride_h = out.stride(1);
  at::Tensor ws;
  if (const size_t need = dkv_softmax_v_workspace_bytes(&a)) {
    ws = empty({(int64_t)need}, at::kByte, sc.device());
    a.workspace = ws.data_ptr();
    a.workspace_bytes = need;
  }
  if (int rc = dkv_softmax_v(&a, sc.data_ptr(), sc.stride(0), sc.stride(1))) return fail("dkv_softmax_v", rc);
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

long long_max(PyObject* list) {
  long m = 0;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) m = std::max(m, PyLong_AsLong(PyList_GET_ITEM(list, i)));
  return m;
}

// append_token(k_state, v_state, key_states, key_len, value_states, value_len, arenas, width, len_multiple, row_counter|None)
//   -> (flat_k, flat_v, lens_k, lens_v, offs_k, offs_v) and the states advanced by one token, or None (nothing done) when
//   a buffer may have to grow
PyObject* append_token(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 10 || !PyList_Check(v[0]) || !PyList_Check(v[1]) || !is_tensor(v[2]) || !unpack(v[2]).is_cuda()) Py_RETURN_NONE;
  const int dev = unpack(v[2]).get_device();
  if (dev < 0 || dev >= MAX_DEVICES || g_status[dev] == nullptr) Py_RETURN_NONE;
  for (int i = 2; i < 6; ++i)
    if (!plain(v[i], dev)) Py_RETURN_NONE;
  const at::Tensor &ks = unpack(v[2]), &kl = unpack(v[3]), &vs = unpack(v[4]), &vl = unpack(v[5]);
  const long A = PyLong_AsLong(v[6]), width = PyLong_AsLong(v[7]), mult = PyLong_AsLong(v[8]);
  if (PyErr_Occurred()) return nullptr;
  if (ks.dim() != 3 || ks.size(1) != 1 || ks.size(2) % A != 0 || vs.sizes() != ks.sizes() || !ks.is_contiguous() || !vs.is_contiguous()) Py_RETURN_NONE;
  const int64_t B = ks.size(0), rows = B * A;
  for (const at::Tensor* t : {&kl, &vl})
    // (without an axis for the arenas: one per row, or refused by the general path)
    if (t->scalar_type() != at::kInt || t->numel() != rows || !t->is_contiguous() || !(t->dim() == 3 || (t->dim() == 2 && A == 1))) Py_RETURN_NONE;
  dkv_append_args a = {};
  a.dtype = dtype_code(ks.scalar_type());
  if (a.dtype < 0 || vs.scalar_type() != ks.scalar_type()) Py_RETURN_NONE;
  at::Tensor view[2][3];
  int64_t pos = 0;
  PyObject* bounds[2];
  for (int sd = 0; sd < 2; ++sd) {
    PyObject* st = v[sd];
    if (PyList_GET_SIZE(st) != 6) Py_RETURN_NONE;
    for (int i = 0; i < 4; ++i)
      if (!plain(PyList_GET_ITEM(st, i), dev)) Py_RETURN_NONE;
    const at::Tensor &flat = unpack(PyList_GET_ITEM(st, 0)), &lens = unpack(PyList_GET_ITEM(st, 1)), &offs = unpack(PyList_GET_ITEM(st, 2)),
                     &ptr = unpack(PyList_GET_ITEM(st, 3));
    bounds[sd] = PyList_GET_ITEM(st, 5);
    if (!PyLong_Check(PyList_GET_ITEM(st, 4)) || !PyList_Check(bounds[sd])) Py_RETURN_NONE;
    const int64_t seq = PyLong_AsLong(PyList_GET_ITEM(st, 4));
    if (sd == 0) pos = seq;
    dkv_side& s = sd ? a.v : a.k;
    int64_t r, cap;
    if (flat.scalar_type() != ks.scalar_type() || !fill_side(s, flat, lens, offs, r, cap) || r != rows || ptr.scalar_type() != at::kInt ||
        ptr.numel() != rows || !ptr.is_contiguous() || seq != pos || seq + 1 > cap || long_max(bounds[sd]) + width > flat.size(1))
      Py_RETURN_NONE;
    s.ptr = static_cast<int32_t*>(ptr.data_ptr());
    a.seq_capacity = (int32_t)(sd ? std::min<int64_t>(a.seq_capacity, cap) : cap);
    view[sd][0] = flat;
    if (lens.dim() == 2) {
      view[sd][1] = rows_view(lens, 0, {rows, seq + 1}, lens.strides());
      view[sd][2] = rows_view(offs, 0, {rows, seq + 1}, offs.strides());
    } else {
      view[sd][1] = lens.narrow(1, 0, seq + 1);
      view[sd][2] = offs.narrow(1, 0, seq + 1);
    }
  }
  if (v[9] != Py_None) {
    if (!plain(v[9], dev)) Py_RETURN_NONE;
    const at::Tensor& t = unpack(v[9]);
    if (t.scalar_type() != at::kInt || t.numel() != B || !t.is_contiguous()) Py_RETURN_NONE;
    a.seq_lens = static_cast<int32_t*>(t.data_ptr());
  }
  a.batch = (int32_t)B;
  a.arenas_per_batch = (int32_t)A;
  a.max_dim = (int32_t)(ks.size(2) / A);
  a.new_k = ks.data_ptr();
  a.new_v = vs.data_ptr();
  a.len_k = static_cast<const int32_t*>(kl.data_ptr());
  a.len_v = static_cast<const int32_t*>(vl.data_ptr());
  a.seq_pos = (int32_t)pos;
  a.len_multiple = (int32_t)mult;
  a.status = g_status[dev];
  a.stream = stream_of(dev);
  if (int rc = dkv_append_decode(&a)) return fail("dkv_append_decode", rc);
  for (int sd = 0; sd < 2; ++sd) {
    PyList_SetItem(v[sd], 4, PyLong_FromLongLong(pos + 1));
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(bounds[sd]); ++i)
      PyList_SetItem(bounds[sd], i, PyLong_FromLong(PyLong_AsLong(PyList_GET_ITEM(bounds[sd], i)) + width));
  }
  PyObject* r = PyTuple_New(6);
  for (int i = 0; i < 3; ++i)
    for (int sd = 0; sd < 2; ++sd) PyTuple_SET_ITEM(r, 2 * i + sd, THPVariable_Wrap(view[sd][i]));
  return r;
  END_HANDLE_TH_ERRORS
}

// new_state(flat [rows, capacity], seq_capacity) -> [flat, lens, offs, ptr, 0, [0] * rows], all zero: the three index buffers
// are views of one allocation, so that a new layer costs two fills and not four of each side
PyObject* new_state(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !is_tensor(v[0]) || !unpack(v[0]).is_cuda()) Py_RETURN_NONE;
  const at::Tensor& flat = unpack(v[0]);
  const int64_t seq = PyLong_AsLong(v[1]);
  if (PyErr_Occurred()) return nullptr;
  if (flat.dim() != 2 || !flat.is_contiguous() || flat.requires_grad() || seq < 0 || seq % 4) Py_RETURN_NONE;
  const int64_t rows = flat.size(0);
  c10::cuda::CUDAGuard guard(flat.device());
  cudaStream_t st = at::cuda::getCurrentCUDAStream(flat.get_device()).stream();
  const at::Tensor ints = empty({2 * rows * seq + rows}, at::kInt, flat.device());
  cudaError_t e = cudaMemsetAsync(flat.data_ptr(), 0, flat.nbytes(), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(ints.data_ptr(), 0, ints.nbytes(), st);
  if (e != cudaSuccess) return fail("zeroing a new cache layer", e);
  PyObject* zeros = PyList_New(rows);
  for (int64_t i = 0; i < rows; ++i) PyList_SET_ITEM(zeros, i, PyLong_FromLong(0));
  PyObject* r = PyList_New(6);
  Py_INCREF(v[0]);
  PyList_SET_ITEM(r, 0, v[0]);
  for (int i = 0; i < 2; ++i) PyList_SET_ITEM(r, 1 + i, THPVariable_Wrap(rows_view(ints, i * rows * seq, {rows, seq}, {seq, 1})));
  PyList_SET_ITEM(r, 3, THPVariable_Wrap(rows_view(ints, 2 * rows * seq, {rows}, {1})));
  PyList_SET_ITEM(r, 4, PyLong_FromLong(0));
  PyList_SET_ITEM(r, 5, zeros);
  return r;
  END_HANDLE_TH_ERRORS
}

// grow(buffer [rows, cols], new_cols) -> [rows, new_cols] that holds the old columns and zeros behind them
PyObject* grow(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !is_tensor(v[0]) || !unpack(v[0]).is_cuda()) Py_RETURN_NONE;
  const at::Tensor& t = unpack(v[0]);
  const int64_t cols = PyLong_AsLong(v[1]);
  if (PyErr_Occurred()) return nullptr;
  if (t.dim() != 2 || t.stride(1) != 1 || t.requires_grad() || cols < t.size(1) || t.numel() == 0) Py_RETURN_NONE;
  // what a two-dimensional copy cannot express: rows that overlap (one row may have any stride), pitches past 2^31 - 1 bytes
  constexpr int64_t MAX_PITCH = 2147483647;
  if (t.stride(0) < t.size(1) || (int64_t)t.element_size() * std::max(t.stride(0), cols) > MAX_PITCH) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(t.device());
  cudaStream_t st = at::cuda::getCurrentCUDAStream(t.get_device()).stream();
  const at::Tensor r = empty({t.size(0), cols}, t.scalar_type(), t.device());
  const size_t es = t.element_size(), had = t.size(1) * es, pitch = cols * es;
  cudaError_t e = cudaMemcpy2DAsync(r.data_ptr(), pitch, t.data_ptr(), t.stride(0) * es, had, t.size(0), cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess && pitch > had) e = cudaMemset2DAsync(static_cast<char*>(r.data_ptr()) + had, pitch, 0, pitch - had, t.size(0), st);
  if (e != cudaSuccess) return fail("growing a cache buffer", e);
  return THPVariable_Wrap(r);
  END_HANDLE_TH_ERRORS
}

// A cache layer's state list [flat, lens, offs, ptr, tokens, bounds] of plain tensors on `dev`, as a side of the C ABI.
bool state_side(PyObject* st, int dev, at::ScalarType dt, int64_t rows, dkv_side& s, int64_t& cap) {
  if (!PyList_Check(st) || PyList_GET_SIZE(st) != 6) return false;
  for (int i = 0; i < 4; ++i)
    if (!plain(PyList_GET_ITEM(st, i), dev)) return false;
  const at::Tensor& ptr = unpack(PyList_GET_ITEM(st, 3));
  int64_t r;
  const at::Tensor& flat = unpack(PyList_GET_ITEM(st, 0));
  if (flat.scalar_type() != dt || !fill_side(s, flat, unpack(PyList_GET_ITEM(st, 1)), unpack(PyList_GET_ITEM(st, 2)), r, cap) || r != rows ||
      ptr.scalar_type() != at::kInt || ptr.numel() != rows || !ptr.is_contiguous())
    return false;
  s.ptr = static_cast<int32_t*>(ptr.data_ptr());
  return true;
}

// The arguments that both block calls share: k_state|None, v_state|None, key_states, key_len, value_states, value_len, arenas,
// row width, len_multiple, first position, row counts|None, row counter|None.
constexpr Py_ssize_t BLOCK_ARGS = 12;
bool block_sides(PyObject* const* v, dkv_pack_args (&a)[2]) {
  if (!is_tensor(v[2]) || !unpack(v[2]).is_cuda()) return false;
  const int dev = unpack(v[2]).get_device();
  if (dev < 0 || dev >= MAX_DEVICES || g_status[dev] == nullptr) return false;
  const int64_t A = PyLong_AsLong(v[6]);
  for (int sd = 0; sd < 2; ++sd) {
    if (!plain(v[2 + 2 * sd], dev) || !plain(v[3 + 2 * sd], dev)) return false;
    const at::Tensor &x = unpack(v[2 + 2 * sd]), &l = unpack(v[3 + 2 * sd]);
    dkv_pack_args& p = a[sd];
    p = {};
    p.dtype = dtype_code(x.scalar_type());
    if (p.dtype < 0 || x.dim() != 3 || x.stride(2) != 1 || unpack(v[2]).dim() != 3 || x.size(0) != unpack(v[2]).size(0) || x.size(1) != unpack(v[2]).size(1) ||
        l.dim() != 2 || l.size(0) != x.size(0) * A || l.size(1) != x.size(1) || l.scalar_type() != at::kInt || !l.is_contiguous())
      return false;
    // the sides may differ in type and, within bounds, in width: the row width is the keys', values of a joint row may have fewer
    const int64_t row_dim = PyLong_AsLong(v[7]);
    if (A != 1 && x.size(2) < A * row_dim) return false;
    p.batch = (int32_t)x.size(0);
    p.arenas_per_batch = (int32_t)A;
    p.n_new = (int32_t)x.size(1);
    p.max_dim = (int32_t)(A == 1 ? std::min(row_dim, x.size(2)) : row_dim);
    p.states = x.data_ptr();
    p.stride_b = x.stride(0);
    p.stride_j = row_dim;
    p.stride_s = x.stride(1);
    p.new_lens = static_cast<const int32_t*>(l.data_ptr());
    p.len_multiple = (int32_t)PyLong_AsLong(v[8]);
    p.seq_pos = (int32_t)PyLong_AsLong(v[9]);
    if (v[10] != Py_None) p.row_counts = static_cast<const int32_t*>(unpack(v[10]).data_ptr());
    if (v[11] != Py_None) p.seq_lens = static_cast<const int32_t*>(unpack(v[11]).data_ptr());
    p.status = g_status[dev];
    p.stream = stream_of(dev);
    if (v[sd] != Py_None) {
      int64_t cap;
      if (!state_side(v[sd], dev, x.scalar_type(), l.size(0), p.side, cap)) return false;
      p.seq_capacity = (int32_t)cap;
    }
  }
  return true;
}
int pack_sides(const dkv_pack_args (&a)[2], long sides) {
  if (sides == 3 && a[0].dtype != a[1].dtype) {
    const int rc = dkv_pack_bulk(&a[0]);
    return rc ? rc : dkv_pack_bulk(&a[1]);
  }
  return sides == 3 ? dkv_pack_pair(&a[0], &a[1]) : sides == 1 ? dkv_pack_bulk(&a[0]) : sides == 2 ? dkv_pack_bulk(&a[1]) : 0;
}

// block_begin(...) -> per side (largest sum of lengths given, largest write pointer, largest end, write pointers, ends): the
// rows' totals on the host.  Sides that have a state are packed behind the copy (nothing flagged), before it is waited for.
PyObject* block_begin(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  dkv_pack_args a[2];
  if (n != BLOCK_ARGS || !block_sides(v, a)) Py_RETURN_NONE;
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor& x = unpack(v[2]);
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t rows = (int64_t)a[0].batch * a[0].arenas_per_batch;
  const at::Tensor totals = empty({2, rows, 4}, at::kInt, x.device());
  const at::Tensor host = at::empty({2, rows, 4}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
  cudaStream_t st = static_cast<cudaStream_t>(a[0].stream);
  if (int rc = dkv_row_totals(&a[0], &a[1], static_cast<int32_t*>(totals.data_ptr()))) return fail("dkv_row_totals", rc);
  cudaEvent_t here = nullptr;
  cudaError_t e = cudaMemcpyAsync(host.data_ptr(), totals.data_ptr(), host.nbytes(), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&here, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventRecord(here, st);
  int rc = 0;
  if (e == cudaSuccess) {
    for (dkv_pack_args& p : a) p.status = nullptr;
    rc = pack_sides(a, (v[0] != Py_None ? 1 : 0) | (v[1] != Py_None ? 2 : 0));
    Py_BEGIN_ALLOW_THREADS
    e = cudaEventSynchronize(here);
    Py_END_ALLOW_THREADS
  }
  if (here) cudaEventDestroy(here);
  if (rc) return fail("dkv_pack_bulk", rc);
  if (e != cudaSuccess) return fail("reading a block's totals", e);
  PyObject* r = PyTuple_New(2);
  for (int sd = 0; sd < 2; ++sd) {
    const int32_t* t = static_cast<const int32_t*>(host.data_ptr()) + sd * rows * 4;
    long raw = 0, now = 0, end = 0;
    PyObject *ptrs = PyList_New(rows), *ends = PyList_New(rows);
    for (int64_t i = 0; i < rows; ++i) {
      const long p = t[4 * i + 2], q = p + t[4 * i + 1];
      raw = std::max(raw, (long)t[4 * i]);
      now = std::max(now, p);
      end = std::max(end, q);
      PyList_SET_ITEM(ptrs, i, PyLong_FromLong(p));
      PyList_SET_ITEM(ends, i, PyLong_FromLong(q));
    }
    PyTuple_SET_ITEM(r, sd, Py_BuildValue("(lllNN)", raw, now, end, ptrs, ends));
  }
  return r;
  END_HANDLE_TH_ERRORS
}

// block_pack(..., sides): 1 = K, 2 = V, 3 = both
PyObject* block_pack(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  dkv_pack_args a[2];
  if (n != BLOCK_ARGS + 1 || !block_sides(v, a)) Py_RETURN_NONE;
  const long sides = PyLong_AsLong(v[BLOCK_ARGS]);
  if (PyErr_Occurred()) return nullptr;
  if (int rc = pack_sides(a, sides)) return fail("dkv_pack_bulk", rc);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// views(k_state, v_state) -> (flat_k, flat_v, lens_k, lens_v, offs_k, offs_v), metadata cut at the tokens stored
PyObject* views(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) Py_RETURN_NONE;
  at::Tensor t[6];
  for (int sd = 0; sd < 2; ++sd) {
    if (!PyList_Check(v[sd]) || PyList_GET_SIZE(v[sd]) != 6) Py_RETURN_NONE;
    const int64_t s = PyLong_AsLong(PyList_GET_ITEM(v[sd], 4));
    for (int i = 0; i < 3; ++i) {
      PyObject* o = PyList_GET_ITEM(v[sd], i);
      if (!THPVariable_CheckExact(o) || unpack(o).dim() != 2 || unpack(o).requires_grad() || (i && unpack(o).size(1) < s)) Py_RETURN_NONE;
      t[2 * i + sd] = i ? rows_view(unpack(o), 0, {unpack(o).size(0), s}, unpack(o).strides()) : unpack(o);
    }
  }
  if (PyErr_Occurred()) return nullptr;
  PyObject* r = PyTuple_New(6);
  for (int i = 0; i < 6; ++i) PyTuple_SET_ITEM(r, i, THPVariable_Wrap(t[i]));
  return r;
  END_HANDLE_TH_ERRORS
}

// expand(state, max_dim) -> dense zero-padded rows [rows, tokens stored, max_dim]
PyObject* expand(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !PyList_Check(v[0]) || PyList_GET_SIZE(v[0]) != 6 || !is_tensor(PyList_GET_ITEM(v[0], 0)) || !unpack(PyList_GET_ITEM(v[0], 0)).is_cuda()) Py_RETURN_NONE;
  const at::Tensor& flat = unpack(PyList_GET_ITEM(v[0], 0));
  const int64_t s = PyLong_AsLong(PyList_GET_ITEM(v[0], 4)), dim = PyLong_AsLong(v[1]), rows = flat.size(0);
  if (PyErr_Occurred()) return nullptr;
  dkv_side side = {};
  int64_t cap;
  if (dim < 1 || dtype_code(flat.scalar_type()) < 0 || !state_side(v[0], flat.get_device(), flat.scalar_type(), rows, side, cap) || s > cap) Py_RETURN_NONE;
  const at::Tensor dense = empty({rows, s, dim}, flat.scalar_type(), flat.device());
  if (int rc = dkv_decompress(dtype_code(flat.scalar_type()), (int32_t)rows, (int32_t)s, (int32_t)dim, &side, dense.data_ptr(), stream_of(flat.get_device())))
    return fail("dkv_decompress", rc);
  return THPVariable_Wrap(dense);
  END_HANDLE_TH_ERRORS
}

// One side of the gate: argument struct from tensors, outputs allocated; false for anything but the plain case.
struct GateSide {
  dkv_gate_args a = {};
  at::Tensor lengths, masked;
};
// scratch of one side or of both, in one allocation
at::Tensor gate_scratch(GateSide* g, int sides) {
  size_t at[3] = {0, 0, 0};
  for (int i = 0; i < sides; ++i) at[i + 1] = at[i] + std::max<size_t>((dkv_gate_workspace_bytes(&g[i].a) + 255) / 256 * 256, 256);
  const at::Tensor ws = empty({(int64_t)at[sides]}, at::kByte, g[0].lengths.device());
  for (int i = 0; i < sides; ++i) {
    g[i].a.workspace = static_cast<char*>(ws.data_ptr()) + at[i];
    g[i].a.workspace_bytes = at[i + 1] - at[i];
  }
  return ws;
}
bool gate_side(GateSide& g, PyObject* const* t, long low_rank, double threshold, bool want, long len_multiple, bool native) {
  if (!is_tensor(t[0]) || !unpack(t[0]).is_cuda()) return false;
  const int dev = unpack(t[0]).get_device();
  if (dev < 0 || dev >= MAX_DEVICES || g_status[dev] == nullptr) return false;
  for (int i = 0; i < 3; ++i)
    if (!plain(t[i], dev)) return false;
  const at::Tensor &x = unpack(t[0]), &w = unpack(t[1]), &b = unpack(t[2]);
  const auto dt = x.scalar_type();
  dkv_gate_args& a = g.a;
  a.dtype = dtype_code(dt);
  if (a.dtype < 0 || x.dim() < 1 || !x.is_contiguous() || !w.is_contiguous() || !b.is_contiguous() || w.scalar_type() != dt || b.scalar_type() != dt) return false;
  const int64_t d = x.size(-1);
  if (d == 0 || w.dim() != 2 || w.size(0) != d || w.size(1) != d || b.numel() != d) return false;
  a.n_rows = (int32_t)(x.numel() / d);
  a.dim = (int32_t)d;
  a.low_rank = (int32_t)low_rank;
  a.threshold = (float)threshold;
  a.len_multiple = (int32_t)len_multiple;
  a.native_rounding = native ? 1 : 0;
  a.status = g_status[dev];
  a.x = x.data_ptr();
  a.x_stride = d;
  a.w = w.data_ptr();
  a.b = b.data_ptr();
  g.lengths = empty(x.sizes().slice(0, x.dim() - 1), at::kInt, x.device());
  a.lengths = static_cast<int32_t*>(g.lengths.data_ptr());
  if (want) {
    g.masked = empty(x.sizes(), dt, x.device());
    a.masked = g.masked.data_ptr();
    a.masked_stride = d;
  }
  a.stream = stream_of(dev);
  return true;
}

// gate(states, weight, bias, low_rank, threshold, return_masked, len_multiple, native_rounding) -> (masked|None, lengths)
PyObject* gate(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8) Py_RETURN_NONE;
  const long low_rank = PyLong_AsLong(v[3]), len_multiple = PyLong_AsLong(v[6]);
  const double threshold = PyFloat_AsDouble(v[4]);
  if (PyErr_Occurred()) return nullptr;
  const bool want = v[5] == Py_True;
  GateSide g;
  if (!gate_side(g, v, low_rank, threshold, want, len_multiple, v[7] == Py_True)) Py_RETURN_NONE;
  const at::Tensor ws = gate_scratch(&g, 1);
  if (int rc = dkv_gate_lengths(&g.a)) return fail("dkv_gate_lengths", rc);
  PyObject* r = PyTuple_New(2);
  if (want) {
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(g.masked));
  } else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(r, 0, Py_None);
  }
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(g.lengths));
  return r;
  END_HANDLE_TH_ERRORS
}

// gate_both(k, Wk, bk, v, Wv, bv, low_rank, threshold, len_multiple) -> (masked k, masked v, lengths k, lengths v)
PyObject* gate_both(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 9) Py_RETURN_NONE;
  const long low_rank = PyLong_AsLong(v[6]), len_multiple = PyLong_AsLong(v[8]);
  const double threshold = PyFloat_AsDouble(v[7]);
  if (PyErr_Occurred()) return nullptr;
  GateSide g[2];
  for (int i = 0; i < 2; ++i)
    if (!gate_side(g[i], v + 3 * i, low_rank, threshold, true, len_multiple, true)) Py_RETURN_NONE;
  // (the sides may be on two devices, though no one launch takes both then)
  const bool one_device = g[0].lengths.device() == g[1].lengths.device();
  const at::Tensor ws = gate_scratch(g, one_device ? 2 : 1), ws2 = one_device ? at::Tensor() : gate_scratch(g + 1, 1);
  if (int rc = dkv_gate_lengths_both(&g[0].a, &g[1].a)) return fail("dkv_gate_lengths_both", rc);
  PyObject* r = PyTuple_New(4);
  for (int i = 0; i < 2; ++i) {
    PyTuple_SET_ITEM(r, i, THPVariable_Wrap(g[i].masked));
    PyTuple_SET_ITEM(r, 2 + i, THPVariable_Wrap(g[i].lengths));
  }
  return r;
  END_HANDLE_TH_ERRORS
}

// set_status(device index, address): where kernels on that device report their DKV_ST_* conditions
PyObject* set_status_word(PyObject*, PyObject* const* v, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "set_status(device, address)");
    return nullptr;
  }
  const long dev = PyLong_AsLong(v[0]);
  void* p = PyLong_AsVoidPtr(v[1]);
  if (PyErr_Occurred()) return nullptr;
  if (dev >= 0 && dev < MAX_DEVICES) g_status[dev] = static_cast<int32_t*>(p);
  Py_RETURN_NONE;
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL
PyMethodDef methods[] = {{"attend", FAST(attend), "decode attention"},
                         {"scores", FAST(scores), "scaled scores of a query"},
                         {"softmax_v", FAST(softmax_v), "softmax over scores applied to the values"},
                         {"append_token", FAST(append_token), "decode append"},
                         {"new_state", FAST(new_state), "buffers of a new cache layer"},
                         {"grow", FAST(grow), "a cache buffer with more columns"},
                         {"block_begin", FAST(block_begin), "totals of a block of tokens, first attempt at its pack"},
                         {"block_pack", FAST(block_pack), "pack of a block of tokens"},
                         {"views", FAST(views), "a layer's tensors, cut at the tokens stored"},
                         {"expand", FAST(expand), "dense rows of a layer's side"},
                         {"gate", FAST(gate), "cutoff gate of one side"},
                         {"gate_both", FAST(gate_both), "cutoff gate of both sides"},
                         {"set_status", FAST(set_status_word), "status word of a device"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "native host side of dynakv_b200", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
