// Tensor-level entry points over the C ABI as a CPython extension module (`calibquant_b200._native`).
//
// What bounds the small calls of this library is the host: a decode step on a short context takes ~10 us of GPU time,
// while argument checks, output allocation, pointer extraction and the ctypes call took 25 us in Python.  Here the
// same work costs ~3 us per call: fast-call argument vectors, tensors unpacked in place, the current stream read
// through c10.  No arithmetic lives here: every function checks its arguments, allocates its results and calls one
// entry point of libcalibquant_b200.so on torch's current stream.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/cuda/CUDAException.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <tuple>
#include <vector>

#include "../../include/calibquant_b200.h"

namespace {

using at::Tensor;

struct PyRaised {};      // a Python exception is already set

[[noreturn]] void raise(PyObject* type, const char* text) {
  PyErr_SetString(type, text);
  throw PyRaised();
}

#define CQ_BEGIN try { HANDLE_TH_ERRORS
#define CQ_END END_HANDLE_TH_ERRORS } catch (const PyRaised&) { return nullptr; }

// A negative status becomes the exception calibquant_b200._lib.check raises for it.
void check(int rc, const char* where) {
  if (rc == CQ_OK) return;
  PyObject* mod = PyImport_ImportModule("calibquant_b200._lib");
  PyObject* res = mod ? PyObject_CallMethod(mod, "check", "is", rc, where) : nullptr;
  Py_XDECREF(res);
  Py_XDECREF(mod);
  if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s: status %d", where, rc);
  throw PyRaised();
}

void want_args(Py_ssize_t got, Py_ssize_t want, const char* where) {
  if (got != want) { PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", where, want, got); throw PyRaised(); }
}

const Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch.Tensor");
  return THPVariable_Unpack(o);
}
Tensor opt_tensor(PyObject* o) { return o == Py_None ? Tensor() : tensor(o); }

int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    PyObject* idx = PyNumber_Index(o);
    if (!idx) throw PyRaised();
    const long long w = PyLong_AsLongLong(idx);
    Py_DECREF(idx);
    if (w == -1 && PyErr_Occurred()) throw PyRaised();
    return w;
  }
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyRaised();
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyRaised();
  return v != 0;
}

void need_cuda(const Tensor& t) {
  if (t.defined() && !t.is_cuda()) raise(PyExc_RuntimeError, "calibquant_b200 runs on CUDA tensors only (no CPU fallback)");
}
// a number that is divided by (an integer division by zero would end the process)
int64_t divisor(int64_t v, const char* what) {
  if (v == 0) { PyErr_Format(PyExc_ZeroDivisionError, "%s is zero", what); throw PyRaised(); }
  return v;
}
void want_dims(const Tensor& t, int64_t n, const char* what) {
  if (t.dim() == n) return;
  PyErr_Format(PyExc_ValueError, "%s must have %lld dimensions, got %lld", what, (long long)n, (long long)t.dim());
  throw PyRaised();
}
// one query row per (batch row, head)
void want_one_row(const Tensor& q, int64_t D) {
  if (q.numel() == q.size(0) * q.size(1) * D) return;
  PyErr_Format(PyExc_RuntimeError, "a decode step takes one query row per head, got %lld elements for %lld rows of %lld",
               (long long)q.numel(), (long long)(q.size(0) * q.size(1)), (long long)D);
  throw PyRaised();
}
int dtype_enum(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kHalf: return CQ_DTYPE_F16;
    case at::kBFloat16: return CQ_DTYPE_BF16;
    default: PyErr_Format(PyExc_TypeError, "unsupported dtype torch.%s; expected float16 or bfloat16", c10::toString(t.scalar_type()));
             throw PyRaised();
  }
}
Tensor contiguous(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }

// rows a kernel reads with 16-byte accesses: channels contiguous, the other strides multiples of 8 elements
bool rows_ok(const Tensor& t) {
  if (t.stride(3) != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) return false;
  return t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0;
}
Tensor with_rows(const Tensor& t) { return rows_ok(t) ? t : t.contiguous(); }

// Other Python threads run while a call of the library is under way: a launch waits where the stream's queue is full, and what
// it waits for may itself need the interpreter (a host function in the stream, another thread's launches).
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
// No Python object may be touched in `call`: its arguments are plain values and tensors' pointers.
template <typename F>
void launch(F&& call, const char* where) {
  int rc;
  { Unlocked u; rc = call(); }
  check(rc, where);
}

struct Call {            // device and stream of one call
  c10::cuda::OptionalCUDAGuard guard;
  cudaStream_t stream;
  explicit Call(const Tensor& t) {
    if (c10::cuda::current_device() != t.get_device()) guard.set_index(t.get_device());
    stream = c10::cuda::getCurrentCUDAStream(t.get_device()).stream();
  }
};

Tensor empty(at::IntArrayRef size, const Tensor& like) { return at::empty(size, like.options()); }
Tensor empty(at::IntArrayRef size, const Tensor& like, at::ScalarType dt) { return at::empty(size, like.options().dtype(dt)); }

PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* wrap2(Tensor a, Tensor b) {
  PyObject* tup = PyTuple_New(2);
  if (!tup) throw PyRaised();
  PyTuple_SET_ITEM(tup, 0, wrap(std::move(a)));
  PyTuple_SET_ITEM(tup, 1, wrap(std::move(b)));
  return tup;
}
PyObject* wrap3(Tensor a, Tensor b, Tensor c) {
  PyObject* tup = PyTuple_New(3);
  if (!tup) throw PyRaised();
  PyTuple_SET_ITEM(tup, 0, wrap(std::move(a)));
  PyTuple_SET_ITEM(tup, 1, wrap(std::move(b)));
  PyTuple_SET_ITEM(tup, 2, wrap(std::move(c)));
  return tup;
}

// ---- scratch -------------------------------------------------------------------------------------------------------
// Grow-only buffer per (device, stream), zeroed when created: its first word is the sticky device status the decode
// kernels set when a bounded wait runs out.  Guarded by the GIL; the map is never destroyed (at exit the CUDA context may be
// gone before it).
//   * A capture takes the buffer an eager warm-up call created, if it is large enough, and the graph's replays go on using it
//     for as long as the graph lives, which is not known here: such a buffer is never freed.  One that replaces it is at
//     least twice its size, so that all the retired ones together are smaller than the one in use.
//   * A buffer created during a capture lives in that graph's memory pool, like any intermediate of the graph: eager calls and
//     other captures never see it, and the reference kept here ends with the next capture.
struct Scratch {
  Tensor buf;
  unsigned long long capture = 0;      // the capture it was created in
  bool in_graph = false;               // an eager buffer that a capture has used
};
using WsKey = std::tuple<int, cudaStream_t, bool>;      // device, stream, created during a capture
std::map<WsKey, Scratch>& workspaces() { static auto* m = new std::map<WsKey, Scratch>(); return *m; }
std::vector<Tensor>& retired() { static auto* v = new std::vector<Tensor>(); return *v; }

bool capturing(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) (void)cudaGetLastError();      // the default stream beside a capture
  return status != cudaStreamCaptureStatusNone;
}

Tensor workspace(int64_t nbytes, int device, cudaStream_t stream) {
  Scratch& eager = workspaces()[WsKey(device, stream, false)];
  const bool enough = eager.buf.defined() && eager.buf.numel() >= nbytes, in_capture = capturing(stream);
  if (enough) {
    if (in_capture) eager.in_graph = true;
    return eager.buf;
  }
  c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
  const auto fresh = [&](int64_t n, const Tensor& before) {
    Tensor buf = at::zeros({std::max<int64_t>(n, 256)}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
    if (before.defined()) buf.narrow(0, 0, 4).copy_(before.narrow(0, 0, 4));      // a sticky status survives the regrowth
    return buf;
  };
  if (!in_capture) {
    Tensor buf = fresh(eager.in_graph ? std::max(nbytes, 2 * eager.buf.numel()) : nbytes, eager.buf);
    if (eager.in_graph) retired().push_back(eager.buf);
    eager = Scratch{buf, 0, false};
    return buf;
  }
  cudaStreamCaptureStatus status;
  unsigned long long id = 0;
  C10_CUDA_CHECK(cudaStreamGetCaptureInfo(stream, &status, &id));
  Scratch& own = workspaces()[WsKey(device, stream, true)];
  if (own.buf.defined() && own.capture == id && own.buf.numel() >= nbytes) return own.buf;
  own = Scratch{fresh(nbytes, own.capture == id ? own.buf : Tensor()), id, true};
  return own.buf;
}

PyObject* py_workspace(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 3, "workspace");      // nbytes, device index, stream handle
  return wrap(workspace(integer(a[0]), (int)integer(a[1]), reinterpret_cast<cudaStream_t>(integer(a[2]))));
  CQ_END
}
// the buffers that exist for (device, stream): eager, then capture-only
PyObject* py_workspaces_of(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 2, "workspaces_of");
  PyObject* list = PyList_New(0);
  for (const bool capturing : {false, true}) {
    auto it = workspaces().find(WsKey((int)integer(a[0]), reinterpret_cast<cudaStream_t>(integer(a[1])), capturing));
    if (it == workspaces().end() || !it->second.buf.defined()) continue;
    PyObject* t = wrap(it->second.buf);
    PyList_Append(list, t);
    Py_DECREF(t);
  }
  return list;
  CQ_END
}

// ---- quantize + pack -----------------------------------------------------------------------------------------------
PyObject* py_pack_last_dim(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 3, "pack_last_dim");      // data [B,nh,R,L], group_size, bits
  need_cuda(tensor(a[0]));
  const Tensor x = contiguous(tensor(a[0]));
  const int64_t g = divisor(integer(a[1]), "group_size"), bits = integer(a[2]), B = x.size(0), nh = x.size(1), R = x.size(2), L = x.size(3);
  Call call(x);
  Tensor code = empty({B, nh, R, L * bits / 32}, x, at::kInt), scale = empty({B, nh, R, L / g}, x), mn = empty({B, nh, R, L / g}, x);
  const int dt = dtype_enum(x);
  launch([&] { return cq_pack_last_dim(x.data_ptr(), B * nh * R, L, (int)g, (int)bits, dt, (int32_t*)code.data_ptr(),
                         scale.data_ptr(), mn.data_ptr(), call.stream); }, "cq_pack_last_dim");
  return wrap3(code, scale, mn);
  CQ_END
}

PyObject* py_pack_k_per_channel(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 3, "pack_k_per_channel");      // k [B,H,T,D], group_size, bits
  need_cuda(tensor(a[0]));
  const Tensor k = with_rows(tensor(a[0]));
  const int64_t g = divisor(integer(a[1]), "group_size"), bits = integer(a[2]), B = k.size(0), H = k.size(1), T = k.size(2), D = k.size(3);
  Call call(k);
  Tensor code = empty({B, H, D, T * bits / 32}, k, at::kInt), scale = empty({B, H, D, T / g}, k), mn = empty({B, H, D, T / g}, k);
  const int dt = dtype_enum(k);
  launch([&] { return cq_pack_k_per_channel(k.data_ptr(), (int)B, (int)H, T, (int)D, k.stride(0), k.stride(1), k.stride(2), (int)g, (int)bits,
                              dt, (int32_t*)code.data_ptr(), scale.data_ptr(), mn.data_ptr(), call.stream); }, "cq_pack_k_per_channel");
  return wrap3(code, scale, mn);
  CQ_END
}

PyObject* py_pack_v_per_token(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 3, "pack_v_per_token");      // v [B,H,T,D], group_size, bits
  need_cuda(tensor(a[0]));
  const Tensor v = with_rows(tensor(a[0]));
  const int64_t g = divisor(integer(a[1]), "group_size"), bits = integer(a[2]), B = v.size(0), H = v.size(1), T = v.size(2), D = v.size(3);
  Call call(v);
  Tensor code = empty({B, H, T, D * bits / 32}, v, at::kInt), scale = empty({B, H, T, D / g}, v), mn = empty({B, H, T, D / g}, v);
  const int dt = dtype_enum(v);
  launch([&] { return cq_pack_v_per_token(v.data_ptr(), (int)B, (int)H, T, (int)D, v.stride(0), v.stride(1), v.stride(2), (int)g, (int)bits,
                            dt, (int32_t*)code.data_ptr(), scale.data_ptr(), mn.data_ptr(), call.stream); }, "cq_pack_v_per_token");
  return wrap3(code, scale, mn);
  CQ_END
}

// ---- uint8 format: quantize + encode ---------------------------------------------------------------------------------
PyObject* py_quant_encode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 3, "quant_encode");      // x [B,T,H,D], bits, clip factor -> enc [B,H,T,D*bits/8], scale, zero point
  need_cuda(tensor(a[0]));
  want_dims(tensor(a[0]), 4, "x");
  const Tensor x = with_rows(tensor(a[0]));
  const int64_t bits = integer(a[1]), B = x.size(0), T = x.size(1), H = x.size(2), D = x.size(3);
  const float clip = (float)real(a[2]);
  const int64_t st[3] = {x.stride(0), x.stride(1), x.stride(2)};
  const int dt = dtype_enum(x);
  Call call(x);
  Tensor s = empty({B, 1, H, D}, x), zp = empty({B, 1, H, D}, x), enc = empty({B, H, T, D * bits / 8}, x, at::kByte);
  if (reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 && st[0] % 8 == 0 && st[1] % 8 == 0 && st[2] % 8 == 0) {
    launch([&] { return cq_calib_quant_encode(x.data_ptr(), (int)B, (int)T, (int)H, (int)D, st, (int)bits, clip, dt, s.data_ptr(), zp.data_ptr(),
                                (uint8_t*)enc.data_ptr(), call.stream); }, "cq_calib_quant_encode");
    return wrap3(enc, s, zp);
  }
  launch([&] { return cq_calib_minmax(x.data_ptr(), (int)B, (int)T, (int)H, (int)D, st, (int)bits, clip, dt, s.data_ptr(), zp.data_ptr(),
                        call.stream); }, "cq_calib_minmax");
  launch([&] { return cq_calib_quantize(x.data_ptr(), (int)B, (int)T, (int)H, (int)D, st, (int)bits, dt, s.data_ptr(), zp.data_ptr(), 0,
                          nullptr, (uint8_t*)enc.data_ptr(), call.stream); }, "cq_calib_quantize");
  return wrap3(enc, s, zp);
  CQ_END
}

// ---- the quantized product -------------------------------------------------------------------------------------------
PyObject* py_qbmm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 6, "qbmm");      // group_size, fA [B,Hq,1,K], qB, scales, zeros, bits
  for (int i = 1; i < 5; ++i) need_cuda(tensor(a[i]));
  const Tensor fA = contiguous(tensor(a[1])), qB = contiguous(tensor(a[2])), s = contiguous(tensor(a[3])), z = contiguous(tensor(a[4]));
  if (fA.dim() != 4 || qB.dim() != 4) raise(PyExc_AssertionError, "fA and qB must have four dimensions");
  const int64_t bits = divisor(integer(a[5]), "bits"), B = fA.size(0), Hq = fA.size(1), K = fA.size(3), Hkv = qB.size(1);
  if (fA.size(2) != 1) raise(PyExc_ValueError, "only M == 1 (one query row) is implemented");
  const int64_t N = qB.size(3) * (32 / bits);
  Call call(fA);
  Tensor out = empty({B, Hq, 1, N}, fA);
  Tensor ws = workspace((int64_t)cq_qbmm_workspace_bytes((int)B, (int)Hq, K, N), fA.get_device(), call.stream);
  const int group = (int)integer(a[0]), dt = dtype_enum(fA);
  launch([&] { return cq_qbmm(fA.data_ptr(), (const int32_t*)qB.data_ptr(), s.data_ptr(), z.data_ptr(), out.data_ptr(), (int)B, (int)Hq, (int)Hkv,
                K, N, group, (int)bits, dt, ws.data_ptr(), (size_t)ws.numel(), call.stream); }, "cq_qbmm");
  return wrap(out);
  CQ_END
}

// ---- decode step -----------------------------------------------------------------------------------------------------
// Tensors of a packed operand (code, scale, minimum), made contiguous; false when there is nothing packed.
bool unpack3(PyObject* o, Tensor (&t)[3]) {
  if (o == Py_None) return false;
  PyObject* seq = PySequence_Fast(o, "a packed operand is a (code, scale, mn) sequence");
  if (!seq) throw PyRaised();
  const bool ok = PySequence_Fast_GET_SIZE(seq) == 3;
  if (ok) {
    for (int i = 0; i < 3; ++i) {
      PyObject* e = PySequence_Fast_GET_ITEM(seq, i);
      if (!THPVariable_Check(e)) { Py_DECREF(seq); raise(PyExc_TypeError, "expected a torch.Tensor"); }
      t[i] = THPVariable_Unpack(e);
    }
  }
  Py_DECREF(seq);
  if (!ok) raise(PyExc_ValueError, "a packed operand is (code, scale, mn)");
  for (auto& x : t) { need_cuda(x); }
  return true;
}

void check_fp_rows(const Tensor& k, const Tensor& v, int64_t D) {
  for (const Tensor* t : {&k, &v})
    if (t->stride(3) != 1 || t->stride(2) != D)
      raise(PyExc_ValueError, "k_fp/v_fp token rows must be contiguous ([.., T, D] with stride D)");
  if (k.strides() != v.strides()) raise(PyExc_ValueError, "k_fp and v_fp must share strides");
}
void check_counter(const Tensor& t) {
  if (t.scalar_type() != at::kInt || !t.is_cuda()) raise(PyExc_AssertionError, "t_fp_dev must be an int32 CUDA tensor");
}

// q, k_pack, v_pack, k_fp, v_fp, t_sys, bits, group_size, calibrate, mask, out, t_fp, t_fp_dev
PyObject* py_decode_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 13, "decode_attention");
  const Tensor& q_in = tensor(a[0]);
  Tensor kp[3], vp[3];
  const bool has_k = unpack3(a[1], kp), has_v = unpack3(a[2], vp);
  const Tensor k_fp = opt_tensor(a[3]), v_fp = opt_tensor(a[4]);
  Tensor mask = opt_tensor(a[9]), out = opt_tensor(a[10]);
  const Tensor live = opt_tensor(a[12]);
  need_cuda(q_in); need_cuda(k_fp); need_cuda(v_fp); need_cuda(mask);
  if (!k_fp.defined() && !has_k) raise(PyExc_ValueError, "decode_attention needs packed or full-precision keys");
  const Tensor q = contiguous(q_in);
  want_one_row(q, q.size(-1));
  cq_decode_args d = {};
  d.batch = (int32_t)q.size(0); d.n_q_heads = (int32_t)q.size(1); d.head_dim = (int32_t)q.size(-1);
  d.n_kv_heads = (int32_t)(k_fp.defined() ? k_fp.size(1) : kp[0].size(1));
  d.bits = (int32_t)integer(a[6]); d.group_size = (int32_t)integer(a[7]); d.dtype = dtype_enum(q);
  d.calibrate = a[8] == Py_None ? d.bits <= 2 : truth(a[8]);
  d.q = q.data_ptr();
  if (has_k && kp[0].numel() > 0) {
    if (!has_v) raise(PyExc_TypeError, "v_pack is missing");
    for (auto& t : kp) t = contiguous(t);
    for (auto& t : vp) t = contiguous(t);
    d.t_vis = (int32_t)vp[0].size(2);
    d.k_code = (const int32_t*)kp[0].data_ptr(); d.k_scale = kp[1].data_ptr(); d.k_mn = kp[2].data_ptr();
    d.v_code = (const int32_t*)vp[0].data_ptr(); d.v_scale = vp[1].data_ptr(); d.v_mn = vp[2].data_ptr();
  }
  if (k_fp.defined() && k_fp.size(2) > 0) {
    if (!v_fp.defined()) raise(PyExc_TypeError, "v_fp is missing");
    check_fp_rows(k_fp, v_fp, d.head_dim);
    d.t_fp = (int32_t)(a[11] == Py_None ? k_fp.size(2) : integer(a[11]));
    d.k_fp = k_fp.data_ptr(); d.v_fp = v_fp.data_ptr();
    d.fp_stride_b = k_fp.stride(0); d.fp_stride_h = k_fp.stride(1);
  }
  d.t_sys = (int32_t)std::min<int64_t>(integer(a[5]), d.t_fp);
  if (live.defined()) { check_counter(live); d.t_fp_dev = (const int32_t*)live.data_ptr(); }
  if (mask.defined()) {
    mask = mask.reshape({d.batch, -1});
    if (mask.scalar_type() != q.scalar_type() || mask.stride(1) != 1) mask = mask.to(q.scalar_type()).contiguous();
    if (mask.size(1) != d.t_vis + d.t_fp) {
      PyErr_Format(PyExc_ValueError, "Attention mask should cover %d keys, but covers %lld", d.t_vis + d.t_fp, (long long)mask.size(1));
      throw PyRaised();
    }
    d.mask = mask.data_ptr(); d.mask_stride_b = mask.stride(0);
  }
  Call call(k_fp.defined() ? k_fp : kp[0]);
  const bool own_out = !out.defined();
  if (own_out) out = empty(q_in.sizes(), q);
  d.out = out.data_ptr();
  const size_t nbytes = cq_decode_attn_workspace_bytes(&d);
  if (nbytes == 0) {      // the size query refused the arguments: the call itself says why
    const int rc = cq_decode_attn(&d, nullptr, 0, call.stream);
    check(rc ? rc : CQ_ERR_WORKSPACE, "cq_decode_attn");
  }
  const Tensor ws = workspace((int64_t)nbytes, q.get_device(), call.stream);
  launch([&] { return cq_decode_attn(&d, ws.data_ptr(), (size_t)ws.numel(), call.stream); }, "cq_decode_attn");
  return wrap(own_out ? out : out.reshape(q_in.sizes()));
  CQ_END
}

// q, enc_k, enc_v, scale_key, zero_point_key, scale_value, zero_point_value, k_fp, v_fp, bits, sys_len, normalize, mask, t_fp_dev
PyObject* py_u8_decode_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 14, "u8_decode_attention");
  const Tensor& q_in = tensor(a[0]);
  const Tensor &k_fp = tensor(a[7]), &v_fp = tensor(a[8]);
  need_cuda(q_in); need_cuda(k_fp); need_cuda(v_fp);
  want_dims(q_in, 4, "q");
  want_one_row(q_in, q_in.size(3));
  const Tensor q = contiguous(q_in);
  cq_u8_decode_args d = {};
  const int64_t B = q.size(0), Hq = q.size(1), D = q.size(3), Hkv = k_fp.size(1), t_fp = k_fp.size(2);
  const Tensor enc_k = contiguous(tensor(a[1])), enc_v = contiguous(tensor(a[2]));
  need_cuda(enc_k); need_cuda(enc_v);
  d.bits = (int32_t)integer(a[9]);
  Tensor par[4];
  const int64_t hs = tensor(a[3]).numel() / divisor(B * D, "the number of query elements per head");
  for (int i = 0; i < 4; ++i) {
    const Tensor& p = tensor(a[3 + i]);
    if ((hs != Hq && hs != Hkv) || p.numel() != B * hs * D || p.scalar_type() != q.scalar_type())
      raise(PyExc_ValueError, "scale / zero point must hold one row of D values per query head or per KV head");
    need_cuda(p);
    par[i] = contiguous(p);
  }
  if (t_fp) {
    for (const Tensor* t : {&k_fp, &v_fp})
      if (t->stride(3) != 1 || t->stride(2) != D) raise(PyExc_ValueError, "k_fp / v_fp token rows must be contiguous");
  }
  Tensor mask = opt_tensor(a[12]);
  const int64_t t_vis = enc_k.size(2);
  if (mask.defined()) {
    mask = mask.reshape({B, -1}).to(q.scalar_type()).contiguous();
    if (mask.size(1) != t_vis + t_fp) {
      PyErr_Format(PyExc_ValueError, "mask must cover %lld keys, got %lld", (long long)(t_vis + t_fp), (long long)mask.size(1));
      throw PyRaised();
    }
    d.mask = mask.data_ptr(); d.mask_stride_b = mask.stride(0);
  }
  if (k_fp.strides() != v_fp.strides()) raise(PyExc_ValueError, "k_fp and v_fp must share strides");
  const Tensor live = opt_tensor(a[13]);
  Call call(q);
  Tensor out = empty({B, Hq, 1, D}, q, at::kBFloat16);
  d.batch = (int32_t)B; d.n_q_heads = (int32_t)Hq; d.n_kv_heads = (int32_t)Hkv; d.head_dim = (int32_t)D;
  d.t_vis = (int32_t)t_vis; d.t_fp = (int32_t)t_fp; d.t_sys = (int32_t)integer(a[10]);
  d.dtype = dtype_enum(q); d.n_scale_heads = (int32_t)hs;
  d.calibrate = a[11] == Py_None ? d.bits <= 2 : truth(a[11]);
  d.q = q.data_ptr(); d.enc_k = (const uint8_t*)enc_k.data_ptr(); d.enc_v = (const uint8_t*)enc_v.data_ptr();
  d.scale_key = par[0].data_ptr(); d.zero_point_key = par[1].data_ptr();
  d.scale_value = par[2].data_ptr(); d.zero_point_value = par[3].data_ptr();
  if (t_fp) { d.k_fp = k_fp.data_ptr(); d.v_fp = v_fp.data_ptr(); }
  d.fp_stride_b = k_fp.stride(0); d.fp_stride_h = k_fp.stride(1);
  d.out = out.data_ptr();
  if (live.defined()) {      // the low word of an int64 counter serves as well
    if (live.scalar_type() != at::kLong || !live.is_cuda()) check_counter(live);
    d.t_fp_dev = (const int32_t*)live.data_ptr();
  }
  const size_t nbytes = cq_u8_decode_attn_workspace_bytes(&d);
  if (nbytes == 0)
    raise(PyExc_ValueError, "cq_u8_decode_attn rejects this request (sizes, head counts or more than 51200 keys)");
  const Tensor ws = workspace((int64_t)nbytes, q.get_device(), call.stream);
  launch([&] { return cq_u8_decode_attn(&d, ws.data_ptr(), (size_t)ws.numel(), call.stream); }, "cq_u8_decode_attn");
  return wrap(out);
  CQ_END
}

// ---- refused positions ------------------------------------------------------------------------------------------------
// A word of page-locked memory per (device, stream) that a launch sets when it refuses a position: as with any asynchronous
// error, a later call on the stream raises.  None while a capture runs that no call on the stream has gone before.
using FlagKey = std::pair<int, cudaStream_t>;
struct Flag {
  Tensor word;
  int32_t* device = nullptr;
};
std::map<FlagKey, Flag>& refusals() { static auto* m = new std::map<FlagKey, Flag>(); return *m; }
int32_t* refusal_flag(cudaStream_t stream, int device) {
  Flag& f = refusals()[FlagKey(device, stream)];
  if (!f.word.defined()) {
    if (capturing(stream)) return nullptr;
    Tensor word = at::zeros({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    void* dev = nullptr;
    C10_CUDA_CHECK(cudaHostGetDevicePointer(&dev, word.data_ptr(), 0));
    f = Flag{word, static_cast<int32_t*>(dev)};
  }
  volatile int32_t* word = f.word.data_ptr<int32_t>();
  if (*word != 0) {
    *word = 0;
    raise(PyExc_RuntimeError, "position_ids of an earlier decode step on this stream lie outside the rotary table");
  }
  return f.device;
}
// the word's value (0 where there is none); the caller has synchronised
PyObject* py_refused(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 2, "refused");      // device index, stream handle
  auto it = refusals().find(FlagKey((int)integer(a[0]), reinterpret_cast<cudaStream_t>(integer(a[1]))));
  if (it == refusals().end() || !it->second.word.defined()) return PyLong_FromLong(0);
  return PyLong_FromLong(*static_cast<volatile int32_t*>(it->second.word.data_ptr<int32_t>()));
  CQ_END
}

// ---- the launches around the attention -------------------------------------------------------------------------------
// qkv, cos, sin, position_ids, n_kv_heads, n_rep, k_cache, v_cache, append_index, t_fp_dev, weight | None (given: qkv is the input
// of the projection, x [B,1,K], and the matrix product is made here), strict: positions outside the table are refused
PyObject* py_rope_split_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 12, "rope_split_append");
  Tensor qkv_in = tensor(a[0]);
  if (a[10] != Py_None) {
    need_cuda(qkv_in);
    need_cuda(tensor(a[10]));
    const Tensor weight = tensor(a[10]);
    Unlocked u;
    qkv_in = at::mm(qkv_in.view({-1, qkv_in.size(-1)}), weight.t());
  }
  const Tensor &k_cache = tensor(a[6]), &v_cache = tensor(a[7]);
  for (int i : {0, 1, 2, 3, 6, 7}) need_cuda(i == 0 ? qkv_in : tensor(a[i]));
  const Tensor cos = contiguous(tensor(a[1])), sin = contiguous(tensor(a[2])), pos = contiguous(tensor(a[3]));
  const int64_t hkv = integer(a[4]), n_rep = integer(a[5]), B = qkv_in.size(0), D = cos.size(-1);
  const int64_t per_row = qkv_in.numel() / std::max<int64_t>(B, 1);
  if (per_row != hkv * (n_rep + 2) * D) {
    PyErr_Format(PyExc_ValueError, "qkv rows must hold %lld elements, got %lld", (long long)(hkv * (n_rep + 2) * D), (long long)per_row);
    throw PyRaised();
  }
  const Tensor qkv = contiguous(qkv_in);
  if (cos.scalar_type() != qkv.scalar_type() || sin.scalar_type() != qkv.scalar_type() || k_cache.scalar_type() != qkv.scalar_type())
    raise(PyExc_TypeError, "qkv, rotary tables and caches must share one dtype");
  if (pos.scalar_type() != at::kLong || pos.numel() != B)
    raise(PyExc_ValueError, "position_ids must be int64 with one position per batch row");
  for (const Tensor* t : {&k_cache, &v_cache})
    if (t->stride(3) != 1 || t->stride(2) != D)
      raise(PyExc_ValueError, "cache token rows must be contiguous ([.., T, D] with stride D)");
  if (k_cache.strides() != v_cache.strides()) raise(PyExc_ValueError, "k_cache and v_cache must share strides");
  for (const Tensor* t : {&k_cache, &v_cache})
    if (t->size(0) < B || t->size(1) < hkv || t->size(2) < k_cache.size(2)) {
      PyErr_Format(PyExc_ValueError, "a cache of %lld rows and %lld heads does not hold %lld rows and %lld heads", (long long)t->size(0),
                   (long long)t->size(1), (long long)B, (long long)hkv);
      throw PyRaised();
    }
  if ((a[8] == Py_None) == (a[9] == Py_None)) raise(PyExc_ValueError, "give exactly one of append_index and t_fp_dev");
  const Tensor live = opt_tensor(a[9]);
  if (live.defined()) check_counter(live);
  Call call(qkv);
  Tensor q = empty({B, hkv * n_rep, 1, D}, qkv);
  const void* table[2] = {cos.data_ptr(), sin.data_ptr()};
  const int at = a[8] == Py_None ? 0 : (int)integer(a[8]), dt = dtype_enum(qkv);
  const int32_t* count = live.defined() ? (const int32_t*)live.data_ptr() : nullptr;
  if (truth(a[11])) {
    int32_t* refused = refusal_flag(call.stream, qkv.get_device());
    launch([&] { return cq_rope_split_append_strict(qkv.data_ptr(), per_row, table[0], table[1], (int)cos.size(0), (const int64_t*)pos.data_ptr(), (int)B,
                                      (int)hkv, (int)n_rep, (int)D, q.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(),
                                      k_cache.stride(0), k_cache.stride(1), (int)k_cache.size(2), at, count, dt, refused,
                                      call.stream); }, "cq_rope_split_append_strict");
  } else {
    launch([&] { return cq_rope_split_append(qkv.data_ptr(), per_row, table[0], table[1], (int)cos.size(0), (const int64_t*)pos.data_ptr(), (int)B,
                               (int)hkv, (int)n_rep, (int)D, q.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), k_cache.stride(0),
                               k_cache.stride(1), (int)k_cache.size(2), at, count, dt, call.stream); }, "cq_rope_split_append");
  }
  return wrap(q);
  CQ_END
}

// x, weight -> whether the launches of few rows can take them (layouts, types, devices; the caller has counted the rows)
PyObject* py_small_ok(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 2, "small_ok");
  const Tensor &x = tensor(a[0]), &w = tensor(a[1]);
  const bool ok = w.is_cuda() && x.is_cuda() && w.device() == x.device() && w.scalar_type() == x.scalar_type() &&
                  (x.scalar_type() == at::kHalf || x.scalar_type() == at::kBFloat16) && w.dim() == 2 && w.is_contiguous() && x.is_contiguous() &&
                  x.size(-1) == w.size(1) && w.size(1) % 8 == 0 && reinterpret_cast<uintptr_t>(w.data_ptr()) % 16 == 0 &&
                  reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0;
  return PyBool_FromLong(ok);
  CQ_END
}

// a, b, dim, length -> the first `length` of both along dim, as views
PyObject* py_heads_of(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 4, "heads_of");
  const int64_t dim = integer(a[2]), len = integer(a[3]);
  return wrap2(tensor(a[0]).narrow(dim, 0, len), tensor(a[1]).narrow(dim, 0, len));
  CQ_END
}

// x [.., K] of up to four rows, weight [N, K] -> [.., N]
PyObject* py_linear_small(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 2, "linear_small");
  for (int i : {0, 1}) need_cuda(tensor(a[i]));
  const Tensor x = contiguous(tensor(a[0])), &w = tensor(a[1]);
  const int64_t K = x.size(-1), rows = K ? x.numel() / K : 0;
  if (w.dim() != 2 || !w.is_contiguous() || w.size(1) != K || w.scalar_type() != x.scalar_type())
    raise(PyExc_ValueError, "weight must be contiguous [N, K] of x's dtype");
  Call call(x);
  std::vector<int64_t> shape = x.sizes().vec();
  shape.back() = w.size(0);
  // Rows longer than 4096 go to the matrix product (us, GEMV / product: 1 x 4096 -> 4096 8.5 / 14.6, four rows 13.4 / 13.4; 2 x 6144 ->
  // 6144 15.8 / 12.6, four rows 24.9 / 12.4; 1 x 14336 -> 4096 31.8 / 26.5)
  if (K > 4096 && rows <= 4) {
    Tensor product;
    { Unlocked u; product = at::mm(x.view({rows, K}), w.t()).view(shape); }
    return wrap(product);
  }
  Tensor out = empty(shape, x);
  const int dt = dtype_enum(x);
  launch([&] { return cq_linear_small(x.data_ptr(), w.data_ptr(), out.data_ptr(), (int)rows, (int)w.size(0), (int)K, dt, call.stream); }, "cq_linear_small");
  return wrap(out);
  CQ_END
}

// qkv [B,T,Hkv*(n_rep+2)*D], cos, sin, position_ids | None, n_kv_heads, n_rep, k_cache | None, v_cache | None, vis_start, vis_len
PyObject* py_prefill_rope_split(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 10, "prefill_rope_split");
  for (int i : {0, 1, 2}) need_cuda(tensor(a[i]));
  Tensor qkv = tensor(a[0]);
  const Tensor cos = contiguous(tensor(a[1])), sin = contiguous(tensor(a[2]));
  const int64_t hkv = integer(a[4]), n_rep = integer(a[5]), D = cos.size(-1), per_tok = hkv * (n_rep + 2) * D;
  if (qkv.dim() != 3 || qkv.size(2) != per_tok) {
    PyErr_Format(PyExc_ValueError, "qkv must be [B,T,%lld]", (long long)per_tok);
    throw PyRaised();
  }
  const int64_t B = qkv.size(0), T = qkv.size(1);
  if (qkv.stride(2) != 1 || qkv.stride(0) % 8 || qkv.stride(1) % 8 || reinterpret_cast<uintptr_t>(qkv.data_ptr()) % 16)
    qkv = qkv.contiguous();
  if (cos.scalar_type() != qkv.scalar_type() || sin.scalar_type() != qkv.scalar_type())
    raise(PyExc_TypeError, "qkv and rotary tables must share one dtype");
  Tensor pos = opt_tensor(a[3]);
  if (pos.defined()) {
    need_cuda(pos);
    pos = pos.reshape({-1, T});
    if (pos.size(0) == 1 && B > 1) pos = pos.expand({B, T});
    if (pos.scalar_type() != at::kLong || pos.size(0) != B) raise(PyExc_ValueError, "position_ids must be int64 [B,T]");
    pos = pos.contiguous();
  }
  const Tensor kc = opt_tensor(a[6]), vc = opt_tensor(a[7]);
  const int64_t vis_start = integer(a[8]), vis_len = integer(a[9]);
  if (kc.defined() != vc.defined()) raise(PyExc_ValueError, "give both caches or neither");
  int64_t cap = 0, sb = 0, sh = 0;
  if (kc.defined()) {
    for (const Tensor* t : {&kc, &vc})
      if (t->scalar_type() != qkv.scalar_type() || t->stride(3) != 1 || t->stride(2) != D)
        raise(PyExc_ValueError, "caches must be [B,Hkv,capacity,D] of the data dtype with contiguous token rows");
    if (kc.strides() != vc.strides()) raise(PyExc_ValueError, "k_cache and v_cache must share strides");
    cap = kc.size(2); sb = kc.stride(0); sh = kc.stride(1);
    if (T - vis_len > cap) {
      PyErr_Format(PyExc_ValueError, "%lld full-precision tokens do not fit a cache of %lld", (long long)(T - vis_len), (long long)cap);
      throw PyRaised();
    }
  }
  Call call(qkv);
  Tensor q = empty({B, T, hkv * n_rep, D}, qkv), k = empty({B, T, hkv, D}, qkv);
  const int dt = dtype_enum(qkv);
  launch([&] { return cq_prefill_rope_split(qkv.data_ptr(), qkv.stride(0), qkv.stride(1), cos.data_ptr(), sin.data_ptr(), (int)cos.size(0),
                              pos.defined() ? (const int64_t*)pos.data_ptr() : nullptr, (int)B, (int)T, (int)hkv, (int)n_rep, (int)D,
                              q.data_ptr(), k.data_ptr(), kc.defined() ? kc.data_ptr() : nullptr, vc.defined() ? vc.data_ptr() : nullptr,
                              sb, sh, (int)cap, (int)vis_start, (int)vis_len, dt, call.stream); }, "cq_prefill_rope_split");
  // the values stay where the projection put them: a strided view of [B,T,Hkv,n_rep+2,D]
  Tensor v = qkv.view({B, T, hkv, n_rep + 2, D}).select(3, n_rep + 1);
  return wrap3(q, k, v);
  CQ_END
}

PyObject* py_prefill_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 4, "prefill_attention");      // q [B,T,Hq,D], k, v [B,T,Hkv,D], out | None
  for (int i = 0; i < 3; ++i) need_cuda(tensor(a[i]));
  for (int i = 0; i < 3; ++i) want_dims(tensor(a[i]), 4, "q, k and v");
  const Tensor q = with_rows(tensor(a[0])), k = with_rows(tensor(a[1])), v = with_rows(tensor(a[2]));
  Tensor out = opt_tensor(a[3]);
  Call call(q);
  if (!out.defined()) out = empty({q.size(0), q.size(1), q.size(2), q.size(3)}, q);
  int64_t st[4][3];
  const Tensor* all[4] = {&q, &k, &v, &out};
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 3; ++j) st[i][j] = all[i]->stride(j);
  const int dt = dtype_enum(q);
  launch([&] { return cq_prefill_attn(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), (int)q.size(0), (int)q.size(1), (int)q.size(2),
                        (int)k.size(2), (int)q.size(3), st[0], st[1], st[2], st[3], dt, call.stream); }, "cq_prefill_attn");
  return wrap(out);
  CQ_END
}

// ---- QJL sign sketches -------------------------------------------------------------------------------------------------
int proj_enum(const Tensor& proj, const Tensor& data) {
  if (proj.scalar_type() == at::kFloat) return CQ_DTYPE_F32;
  if (proj.scalar_type() == data.scalar_type()) return dtype_enum(data);
  raise(PyExc_TypeError, "Unsupported data types for QJL: the projection must be float32 or match the keys");
}

// key_states [B,H,n,G,128], outlier_indices uint8 [B,H,n,oc], rand_prj [sketch,128], outlier_sketch_dim
PyObject* py_qjl_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 4, "qjl_quant");
  for (int i = 0; i < 3; ++i) need_cuda(tensor(a[i]));
  want_dims(tensor(a[0]), 5, "key_states");
  const Tensor k = contiguous(tensor(a[0])), idx = contiguous(tensor(a[1])), proj = contiguous(tensor(a[2]));
  const int dt = dtype_enum(k), pdt = proj_enum(proj, k);
  const int64_t B = k.size(0), H = k.size(1), N = k.size(2), G = k.size(3), D = k.size(4), s = proj.size(0), os = integer(a[3]);
  if (idx.scalar_type() != at::kByte || idx.size(0) != B || idx.size(1) != H || idx.size(2) != N)
    raise(PyExc_ValueError, "outlier_indices must be uint8 [B,H,n,outlier_count]");
  Call call(k);
  Tensor kq = empty({B, H, N, G, s / 8}, k, at::kByte), koq = empty({B, H, N, G, os / 8}, k, at::kByte), norms = empty({B, H, N, G}, k);
  launch([&] { return cq_qjl_quant(k.data_ptr(), (const uint8_t*)idx.data_ptr(), proj.data_ptr(), pdt, B * H * N, (int)G, (int)D, (int)s, (int)os,
                     (int)idx.size(3), dt, (uint8_t*)kq.data_ptr(), (uint8_t*)koq.data_ptr(), norms.data_ptr(), call.stream); }, "cq_qjl_quant");
  return wrap3(kq, koq, norms);
  CQ_END
}

// keys [B,H,T,128] (strided), rand_prj [256,128], outlier_sketch_dim, outlier_count -> (idx, kq, koq, outlier norms, key norms)
PyObject* py_qjl_build(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 4, "qjl_build");
  need_cuda(tensor(a[0])); need_cuda(tensor(a[1]));
  const Tensor k = with_rows(tensor(a[0])), proj = contiguous(tensor(a[1]));
  const int64_t B = k.size(0), H = k.size(1), N = k.size(2) / 32, os = integer(a[2]), oc = integer(a[3]), s = proj.size(0);
  const int64_t st[3] = {k.stride(0), k.stride(1), k.stride(2)};
  Call call(k);
  Tensor idx = empty({B, H, N, oc}, k, at::kByte), kq = empty({B, H, N, 32, s / 8}, k, at::kByte);
  Tensor koq = empty({B, H, N, 32, os / 8}, k, at::kByte), onorm = empty({B, H, N, 32}, k), knorm = empty({B, H, N, 32}, k);
  const int dt = dtype_enum(k), pdt = proj_enum(proj, k);
  launch([&] { return cq_qjl_build(k.data_ptr(), (int)B, (int)H, (int)N, 32, (int)k.size(3), st, proj.data_ptr(), pdt, (int)s, (int)os,
                     (int)oc, dt, (uint8_t*)idx.data_ptr(), (uint8_t*)kq.data_ptr(), (uint8_t*)koq.data_ptr(),
                     knorm.data_ptr(), onorm.data_ptr(), call.stream); }, "cq_qjl_build");
  PyObject* tup = PyTuple_New(5);
  if (!tup) throw PyRaised();
  const Tensor all[5] = {idx, kq, koq, onorm, knorm};
  for (int i = 0; i < 5; ++i) PyTuple_SET_ITEM(tup, i, wrap(all[i]));
  return tup;
  CQ_END
}

// key_quant, key_outlier_quant, key_norm, key_outlier_norm, outlier_indices, query_sketch | None, query [B,Hq,1,128], rand_prj
PyObject* py_qjl_gqa_score(PyObject*, PyObject* const* a, Py_ssize_t n) {
  CQ_BEGIN
  want_args(n, 8, "qjl_gqa_score");
  for (int i = 0; i < 8; ++i)
    if (a[i] != Py_None) need_cuda(tensor(a[i]));
  want_dims(tensor(a[0]), 5, "key_quant");
  const Tensor kq = contiguous(tensor(a[0])), koq = contiguous(tensor(a[1])), kn = contiguous(tensor(a[2])), on = contiguous(tensor(a[3]));
  const Tensor idx = contiguous(tensor(a[4])), q = contiguous(tensor(a[6])), proj = contiguous(tensor(a[7]));
  Tensor qs = opt_tensor(a[5]);
  if (qs.defined()) qs = (qs.scalar_type() == at::kFloat ? qs : qs.to(at::kFloat)).contiguous();
  const int64_t B = kq.size(0), Hkv = kq.size(1), N = kq.size(2), G = kq.size(3), Hq = q.size(1), D = q.size(-1);
  const int dt = dtype_enum(q), pdt = proj_enum(proj, q);
  if (kn.scalar_type() != q.scalar_type() || on.scalar_type() != q.scalar_type())
    raise(PyExc_TypeError, "key norms must have the query dtype");
  if (Hq % divisor(Hkv, "the number of key heads")) raise(PyExc_ValueError, "query heads must be a multiple of key heads");
  Call call(q);
  Tensor scores = empty({B, Hq, N * G, 1}, q, at::kFloat);
  launch([&] { return cq_qjl_gqa_score((const uint8_t*)kq.data_ptr(), (const uint8_t*)koq.data_ptr(), kn.data_ptr(), on.data_ptr(),
                         (const uint8_t*)idx.data_ptr(), qs.defined() ? (const float*)qs.data_ptr() : nullptr, q.data_ptr(),
                         proj.data_ptr(), pdt, (int)B, (int)Hkv, (int)(Hq / Hkv), (int)N, (int)G, (int)D, (int)kq.size(4) * 8,
                         (int)koq.size(4) * 8, (int)idx.size(3), dt, (float*)scores.data_ptr(), call.stream); }, "cq_qjl_gqa_score");
  return wrap(scores);
  CQ_END
}

#define CQ_FN(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    CQ_FN(workspace), CQ_FN(workspaces_of), CQ_FN(refused), CQ_FN(pack_last_dim), CQ_FN(pack_k_per_channel), CQ_FN(pack_v_per_token),
    CQ_FN(quant_encode), CQ_FN(qbmm), CQ_FN(decode_attention), CQ_FN(u8_decode_attention), CQ_FN(rope_split_append), CQ_FN(linear_small), CQ_FN(small_ok), CQ_FN(heads_of),
    CQ_FN(prefill_rope_split), CQ_FN(prefill_attention),
    CQ_FN(qjl_quant), CQ_FN(qjl_build), CQ_FN(qjl_gqa_score), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Tensor-level entry points over libcalibquant_b200.so.", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
