// python_calls.cpp - the host path between Python and the C ABI of include/darkforest_kernels.h.
//
// A decode step or a short sequence keeps the GPU busy for a few microseconds per call, less than an interpreted wrapper
// takes to read a dozen tensors' pointers and to convert the arguments of a ctypes call (7 to 12 us). This module does that
// work - checks, default outputs, the current stream, the call itself with the interpreter lock released - in native code,
// about a microsecond per call before the launch. Behaviour is that of the Python functions in __init__.py, which document
// the arguments and pass them here in order.
//
// The module links no kernel library: bind() receives the addresses of the C functions from the library that the Python
// side loaded, and the exception class that a failed call raises.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>

#include "../../include/darkforest_kernels.h"

namespace {

// ---------------------------------------------------------------- the bound C functions
#define DF_FUNCTIONS(X)                                                                                                     \
  X(df_attn_forward_block) X(df_attn_forward_bf16) X(df_attn_backward) X(df_attn_backward_bf16) X(df_attn_backward_block)    \
  X(df_attn_backward_block_bf16) X(df_attn_backward_static_scratch) X(df_attn_delta) X(df_attn_delta_bf16) X(df_attn_decode) \
  X(df_attn_merge_partials) X(df_attn_accumulate) X(df_linear_qkv_forward) X(df_linear_forward) X(df_linear_gelu_forward)    \
  X(df_chunked_logit_ce) X(df_layernorm_forward) X(df_layernorm_backward) X(df_gelu_forward) X(df_gelu_backward)             \
  X(df_adamw_update) X(df_adamw_update_multi) X(launch_fused_attention) X(launch_fused_mha_forward)                          \
  X(launch_attention_backward) X(launch_fused_mha_backward) X(df_attn_last_status) X(df_attn_status_string)

struct Functions {
#define X(name) decltype(&::name) name = nullptr;
  DF_FUNCTIONS(X)
#undef X
} fn;
PyObject *attention_error = nullptr;  // AttentionError of the package

struct PythonError {};  // a Python exception is set

[[noreturn]] void raise(PyObject *type, const char *text) {
  PyErr_SetString(type, text);
  throw PythonError();
}

// ---------------------------------------------------------------- arguments
const at::Tensor &tensor(PyObject *o) {
  if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch tensor");
  return THPVariable_Unpack(o);
}

// Device address of a tensor argument; None is a null pointer.
template <typename T = float>
T *ptr(PyObject *o) {
  if (o == Py_None) return nullptr;
  const at::Tensor &t = tensor(o);
  if (!t.is_cuda()) raise(attention_error, "attention tensors must live on a CUDA device (no CPU path)");
  if (!t.is_contiguous()) raise(attention_error, "attention tensors must be contiguous");
  return static_cast<T *>(t.data_ptr());
}

uint64_t whole(PyObject *o) {
  if (PyLong_CheckExact(o)) {
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
    if (v == ~0ull && PyErr_Occurred()) throw PythonError();
    return v;
  }
  PyObject *n = PyNumber_Long(o);
  if (!n) throw PythonError();
  const unsigned long long v = PyLong_AsUnsignedLongLongMask(n);
  Py_DECREF(n);
  return v;
}
uint32_t u32(PyObject *o) { return static_cast<uint32_t>(whole(o)); }
float real(PyObject *o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PythonError();
  return static_cast<float>(v);
}
uint32_t truth(PyObject *o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PythonError();
  return static_cast<uint32_t>(v);
}

void *stream(PyObject *o) {
  if (o == Py_None) return static_cast<void *>(c10::cuda::getCurrentCUDAStream().stream());
  PyObject *v = PyObject_GetAttrString(o, "cuda_stream");
  if (!v) throw PythonError();
  const uint64_t s = whole(v);
  Py_DECREF(v);
  return reinterpret_cast<void *>(s);
}

struct Shape3 { uint32_t batch, seq, width; };
Shape3 shape3(PyObject *o) {
  const at::Tensor &t = tensor(o);
  if (t.dim() != 3) raise(PyExc_ValueError, "expected a [batch, seq, heads * d_head] tensor");
  return {static_cast<uint32_t>(t.size(0)), static_cast<uint32_t>(t.size(1)), static_cast<uint32_t>(t.size(2))};
}
struct Shape2 { uint32_t rows, cols; };
Shape2 shape2(PyObject *o) {
  const at::Tensor &t = tensor(o);
  if (t.dim() != 2) raise(PyExc_ValueError, "expected a two-dimensional tensor");
  return {static_cast<uint32_t>(t.size(0)), static_cast<uint32_t>(t.size(1))};
}
uint32_t head_dim(uint64_t width, uint32_t heads) {
  if (heads == 0) raise(PyExc_ZeroDivisionError, "n_heads is zero");
  return static_cast<uint32_t>(width / heads);
}

// ---------------------------------------------------------------- outputs
// Holds the object that a call returns or writes: the caller's, or a new tensor wrapped for Python.
class Out {
 public:
  Out() = default;
  Out(const Out &) = delete;
  Out &operator=(const Out &) = delete;
  ~Out() { Py_XDECREF(o_); }
  void keep(PyObject *o) { Py_INCREF(o); o_ = o; }
  void wrap(at::Tensor t) {
    o_ = THPVariable_Wrap(std::move(t));
    if (!o_) throw PythonError();
  }
  PyObject *get() const { return o_; }
  PyObject *release() { PyObject *o = o_; o_ = nullptr; return o; }

 private:
  PyObject *o_ = nullptr;
};

void given_or_like(Out &out, PyObject *given, PyObject *model) {
  if (given != Py_None) out.keep(given);
  else out.wrap(at::empty_like(tensor(model)));
}
void given_or_empty(Out &out, PyObject *given, PyObject *model, at::IntArrayRef sizes, at::ScalarType type = at::kFloat) {
  if (given != Py_None) out.keep(given);
  else out.wrap(at::empty(sizes, at::TensorOptions().dtype(type).device(tensor(model).device())));
}
void given_or_typed(Out &out, PyObject *given, PyObject *model, at::ScalarType type) {
  given_or_empty(out, given, model, tensor(model).sizes(), type);
}

PyObject *tuple_of(std::initializer_list<Out *> outs) {
  PyObject *t = PyTuple_New(static_cast<Py_ssize_t>(outs.size()));
  if (!t) throw PythonError();
  Py_ssize_t i = 0;
  for (Out *o : outs) PyTuple_SET_ITEM(t, i++, o->release());
  return t;
}

void check(int status) {
  if (status == DF_OK) return;
  const std::string text = std::string("attention call failed: ") + fn.df_attn_status_string(status) + " (" + std::to_string(status) + ")";
  raise(attention_error, text.c_str());
}

// Runs a C function on a stream (its last argument) with the interpreter lock released and checks its status.
template <typename F, typename... A>
void call(F *f, PyObject *stream_arg, A... args) {
  void *s = stream(stream_arg);
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = f(args..., s);
  Py_END_ALLOW_THREADS
  check(status);
}

using Args = PyObject *const *;

// ---------------------------------------------------------------- attention
PyObject *forward(Args a) {  // q k v n_heads scale causal out lse causal_shift stream
  const Shape3 q = shape3(a[0]);
  const uint32_t seq_k = static_cast<uint32_t>(tensor(a[1]).size(1)), heads = u32(a[3]), d = head_dim(q.width, heads);
  Out out, lse;
  given_or_like(out, a[6], a[0]);
  given_or_empty(lse, a[7], a[0], {q.batch, heads, q.seq});
  call(fn.df_attn_forward_block, a[9], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(out.get()), ptr(lse.get()), q.batch, heads, q.seq, seq_k, d, real(a[4]),
       truth(a[5]), static_cast<int64_t>(whole(a[8])));
  return tuple_of({&out, &lse});
}

PyObject *forward_bf16(Args a) {  // q k v n_heads scale causal out lse causal_shift out_fp32 stream
  if (tensor(a[0]).scalar_type() != at::kBFloat16) raise(attention_error, "forward_bf16 needs bfloat16 tensors");
  const Shape3 q = shape3(a[0]);
  const uint32_t seq_k = static_cast<uint32_t>(tensor(a[1]).size(1)), heads = u32(a[3]), d = head_dim(q.width, heads);
  const uint32_t out_fp32 = truth(a[9]);
  const at::ScalarType type = out_fp32 ? at::kFloat : at::kBFloat16;
  Out out, lse;
  given_or_typed(out, a[6], a[0], type);
  if (tensor(out.get()).scalar_type() != type) raise(attention_error, "forward_bf16: out dtype does not match out_fp32");
  given_or_empty(lse, a[7], a[0], {q.batch, heads, q.seq});
  call(fn.df_attn_forward_bf16, a[10], ptr<void>(a[0]), ptr<void>(a[1]), ptr<void>(a[2]), ptr<void>(out.get()), ptr(lse.get()), q.batch, heads, q.seq,
       seq_k, d, real(a[4]), truth(a[5]), static_cast<int64_t>(whole(a[8])), out_fp32);
  return tuple_of({&out, &lse});
}

PyObject *backward(Args a) {  // q k v out d_out lse n_heads scale causal d_q d_k d_v delta_buf stream
  const Shape3 q = shape3(a[0]);
  const uint32_t heads = u32(a[6]), d = head_dim(q.width, heads);
  Out dq, dk, dv, delta;
  given_or_like(dq, a[9], a[0]);
  given_or_like(dk, a[10], a[1]);
  given_or_like(dv, a[11], a[2]);
  given_or_empty(delta, a[12], a[0], {q.batch, heads, q.seq});
  call(fn.df_attn_backward, a[13], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(a[3]), ptr(a[4]), ptr(a[5]), ptr(dq.get()), ptr(dk.get()), ptr(dv.get()),
       ptr(delta.get()), q.batch, heads, q.seq, d, real(a[7]), truth(a[8]));
  return tuple_of({&dq, &dk, &dv});
}

PyObject *backward_bf16(Args a) {  // as backward
  const Shape3 q = shape3(a[0]);
  const uint32_t heads = u32(a[6]), d = head_dim(q.width, heads);
  Out dq, dk, dv, delta;
  given_or_like(dq, a[9], a[0]);
  given_or_like(dk, a[10], a[1]);
  given_or_like(dv, a[11], a[2]);
  given_or_empty(delta, a[12], a[0], {q.batch, heads, q.seq});
  call(fn.df_attn_backward_bf16, a[13], ptr<void>(a[0]), ptr<void>(a[1]), ptr<void>(a[2]), ptr<void>(a[3]), ptr<void>(a[4]), ptr(a[5]),
       ptr<void>(dq.get()), ptr<void>(dk.get()), ptr<void>(dv.get()), ptr(delta.get()), q.batch, heads, q.seq, d, real(a[7]), truth(a[8]));
  return tuple_of({&dq, &dk, &dv});
}

PyObject *backward_static_scratch(Args a) {  // q k v out d_out lse n_heads scale causal d_q d_k d_v stream
  const Shape3 q = shape3(a[0]);
  const uint32_t heads = u32(a[6]), d = head_dim(q.width, heads);
  Out dq, dk, dv;
  given_or_like(dq, a[9], a[0]);
  given_or_like(dk, a[10], a[1]);
  given_or_like(dv, a[11], a[2]);
  call(fn.df_attn_backward_static_scratch, a[12], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(a[3]), ptr(a[4]), ptr(a[5]), ptr(dq.get()), ptr(dk.get()),
       ptr(dv.get()), q.batch, heads, q.seq, d, real(a[7]), truth(a[8]));
  return tuple_of({&dq, &dk, &dv});
}

PyObject *backward_block(Args a) {  // q k v d_out lse delta_buf n_heads scale causal causal_shift d_q d_k d_v stream
  const Shape3 q = shape3(a[0]);
  const uint32_t seq_k = static_cast<uint32_t>(tensor(a[1]).size(1)), heads = u32(a[6]), d = head_dim(q.width, heads);
  Out dq, dk, dv;
  given_or_like(dq, a[10], a[0]);
  given_or_like(dk, a[11], a[1]);
  given_or_like(dv, a[12], a[2]);
  call(fn.df_attn_backward_block, a[13], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(a[3]), ptr(a[4]), ptr(a[5]), ptr(dq.get()), ptr(dk.get()), ptr(dv.get()),
       q.batch, heads, q.seq, seq_k, d, real(a[7]), truth(a[8]), static_cast<int64_t>(whole(a[9])));
  return tuple_of({&dq, &dk, &dv});
}

PyObject *backward_block_bf16(Args a) {  // as backward_block, with out_fp32 before stream
  const Shape3 q = shape3(a[0]);
  const uint32_t seq_k = static_cast<uint32_t>(tensor(a[1]).size(1)), heads = u32(a[6]), d = head_dim(q.width, heads);
  const uint32_t out_fp32 = truth(a[13]);
  const at::ScalarType type = out_fp32 ? at::kFloat : at::kBFloat16;
  Out dq, dk, dv;
  given_or_typed(dq, a[10], a[0], type);
  given_or_typed(dk, a[11], a[1], type);
  given_or_typed(dv, a[12], a[2], type);
  call(fn.df_attn_backward_block_bf16, a[14], ptr<void>(a[0]), ptr<void>(a[1]), ptr<void>(a[2]), ptr<void>(a[3]), ptr(a[4]), ptr(a[5]),
       ptr<void>(dq.get()), ptr<void>(dk.get()), ptr<void>(dv.get()), q.batch, heads, q.seq, seq_k, d, real(a[7]), truth(a[8]),
       static_cast<int64_t>(whole(a[9])), out_fp32);
  return tuple_of({&dq, &dk, &dv});
}

PyObject *delta(Args a) {  // out d_out n_heads delta_buf stream
  const Shape3 o = shape3(a[0]);
  const uint32_t heads = u32(a[2]), d = head_dim(o.width, heads);
  Out buf;
  given_or_empty(buf, a[3], a[0], {o.batch, heads, o.seq});
  call(fn.df_attn_delta, a[4], ptr(a[0]), ptr(a[1]), ptr(buf.get()), o.batch, heads, o.seq, d);
  return buf.release();
}

PyObject *delta_bf16(Args a) {  // as delta
  const Shape3 o = shape3(a[0]);
  const uint32_t heads = u32(a[2]), d = head_dim(o.width, heads);
  Out buf;
  given_or_empty(buf, a[3], a[0], {o.batch, heads, o.seq});
  call(fn.df_attn_delta_bf16, a[4], ptr<void>(a[0]), ptr<void>(a[1]), ptr(buf.get()), o.batch, heads, o.seq, d);
  return buf.release();
}

PyObject *decode(Args a) {  // q k v n_heads cur_seq_len scale block_table page_size partials max_chunks out stream
  const uint32_t heads = u32(a[3]), d = head_dim(static_cast<uint64_t>(tensor(a[0]).numel()), heads);
  Out out;
  given_or_like(out, a[10], a[0]);
  float *part[3] = {nullptr, nullptr, nullptr};
  if (a[8] != Py_None) {
    PyObject *seq = PySequence_Fast(a[8], "partials is a sequence of three tensors");
    if (!seq) throw PythonError();
    const bool three = PySequence_Fast_GET_SIZE(seq) == 3;
    try {
      for (int i = 0; three && i < 3; ++i) part[i] = ptr(PySequence_Fast_GET_ITEM(seq, i));
    } catch (...) {
      Py_DECREF(seq);
      throw;
    }
    Py_DECREF(seq);
    if (!three) raise(PyExc_ValueError, "partials is a sequence of three tensors");
  }
  call(fn.df_attn_decode, a[11], ptr(a[0]), ptr<void>(a[1]), ptr<void>(a[2]), ptr<int32_t>(a[6]), ptr(out.get()), part[0], part[1], part[2], u32(a[9]), heads,
       u32(a[4]), d, real(a[5]), u32(a[7]), tensor(a[1]).scalar_type() == at::kBFloat16 ? 1u : 0u);
  return out.release();
}

PyObject *merge_partials(Args a) {  // o_a lse_a o_b lse_b n_heads stream
  const Shape3 o = shape3(a[0]);
  const uint32_t heads = u32(a[4]), d = head_dim(o.width, heads);
  call(fn.df_attn_merge_partials, a[5], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(a[3]), o.batch, heads, o.seq, d);
  return PyTuple_Pack(2, a[0], a[1]);
}

PyObject *accumulate(Args a) {  // dst src stream
  call(fn.df_attn_accumulate, a[2], ptr(a[0]), ptr(a[1]), static_cast<uint64_t>(tensor(a[0]).numel()));
  Py_INCREF(a[0]);
  return a[0];
}

// ---------------------------------------------------------------- projections, loss head
PyObject *linear_qkv(Args a) {  // x wq wk wv bq bk bv q k v stream
  const Shape2 x = shape2(a[0]);
  const uint32_t n = static_cast<uint32_t>(tensor(a[1]).size(0));
  Out q, k, v;
  given_or_empty(q, a[7], a[0], {x.rows, n});
  given_or_empty(k, a[8], a[0], {x.rows, n});
  given_or_empty(v, a[9], a[0], {x.rows, n});
  call(fn.df_linear_qkv_forward, a[10], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(a[3]), ptr(a[4]), ptr(a[5]), ptr(a[6]), ptr(q.get()), ptr(k.get()), ptr(v.get()),
       x.rows, x.cols, n);
  return tuple_of({&q, &k, &v});
}

PyObject *linear(Args a) {  // x w bias residual out stream
  const Shape2 x = shape2(a[0]);
  const uint32_t n = static_cast<uint32_t>(tensor(a[1]).size(0));
  Out out;
  given_or_empty(out, a[4], a[0], {x.rows, n});
  call(fn.df_linear_forward, a[5], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(a[3]), ptr(out.get()), x.rows, x.cols, n);
  return out.release();
}

PyObject *linear_gelu(Args a) {  // x w bias pre_activation out keep_pre_activation stream
  const Shape2 x = shape2(a[0]);
  const uint32_t n = static_cast<uint32_t>(tensor(a[1]).size(0));
  Out out, pre;
  given_or_empty(out, a[4], a[0], {x.rows, n});
  if (a[3] == Py_None && !truth(a[5])) pre.keep(Py_None);
  else given_or_empty(pre, a[3], a[0], {x.rows, n});
  call(fn.df_linear_gelu_forward, a[6], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(pre.get()), ptr(out.get()), x.rows, x.cols, n);
  return tuple_of({&pre, &out});
}

PyObject *chunked_logit_ce(Args a) {  // logits targets loss total_rows grad_logits stream
  const Shape2 z = shape2(a[0]);
  call(fn.df_chunked_logit_ce, a[5], ptr(a[0]), ptr<uint32_t>(a[1]), ptr(a[4]), ptr(a[2]), z.rows, z.cols, u32(a[3]));
  Py_INCREF(a[2]);
  return a[2];
}

// ---------------------------------------------------------------- LayerNorm, GELU, AdamW
PyObject *layernorm(Args a) {  // x gamma beta out means rstds stream
  const Shape2 x = shape2(a[0]);
  Out out, means, rstds;
  given_or_like(out, a[3], a[0]);
  given_or_empty(means, a[4], a[0], {x.rows});
  given_or_empty(rstds, a[5], a[0], {x.rows});
  call(fn.df_layernorm_forward, a[6], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(out.get()), ptr(means.get()), ptr(rstds.get()), x.rows, x.cols);
  return tuple_of({&out, &means, &rstds});
}

PyObject *layernorm_backward(Args a) {  // grad_out x gamma means rstds grad_x grad_gamma grad_beta stream
  const Shape2 x = shape2(a[1]);
  Out gx;
  given_or_like(gx, a[5], a[1]);
  call(fn.df_layernorm_backward, a[8], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(a[3]), ptr(a[4]), ptr(gx.get()), ptr(a[6]), ptr(a[7]), x.rows, x.cols);
  return gx.release();
}

PyObject *gelu(Args a) {  // x out stream
  Out out;
  given_or_like(out, a[1], a[0]);
  call(fn.df_gelu_forward, a[2], ptr(a[0]), ptr(out.get()), static_cast<uint64_t>(tensor(a[0]).numel()));
  return out.release();
}

PyObject *gelu_backward(Args a) {  // grad_out x grad_x stream
  Out gx;
  given_or_like(gx, a[2], a[1]);
  call(fn.df_gelu_backward, a[3], ptr(a[0]), ptr(a[1]), ptr(gx.get()), static_cast<uint64_t>(tensor(a[1]).numel()));
  return gx.release();
}

PyObject *adamw_update(Args a) {  // p m v g lr beta1 beta2 eps weight_decay bc1 bc2 stream
  call(fn.df_adamw_update, a[11], ptr(a[0]), ptr(a[1]), ptr(a[2]), ptr(a[3]), static_cast<uint64_t>(tensor(a[0]).numel()), real(a[4]), real(a[5]), real(a[6]),
       real(a[7]), real(a[8]), real(a[9]), real(a[10]));
  Py_RETURN_NONE;
}

PyObject *adamw_step(Args a) {  // table n_tensors total_chunks lr beta1 beta2 eps weight_decay bc1 bc2 stream
  call(fn.df_adamw_update_multi, a[10], ptr<df_adamw_tensor_t>(a[0]), u32(a[1]), whole(a[2]), real(a[3]), real(a[4]), real(a[5]), real(a[6]), real(a[7]),
       real(a[8]), real(a[9]));
  Py_RETURN_NONE;
}

// ---------------------------------------------------------------- AttentionContext (legacy symbols, legacy stream)
void expect_shape(PyObject *o, uint32_t rows, uint64_t cols, const char *what) {
  const at::Tensor &t = tensor(o);
  if (t.dim() == 2 && t.size(0) == static_cast<int64_t>(rows) && t.size(1) == static_cast<int64_t>(cols)) return;
  const std::string text = std::string("attention ") + what + " shape mismatch";
  raise(attention_error, text.c_str());
}

// The legacy symbols run on the legacy default stream: work that the caller queued on another stream has to be finished,
// work on the default stream itself is in order already.
void finish_other_stream() {
  const c10::cuda::CUDAStream s = c10::cuda::getCurrentCUDAStream();
  if (s.stream() == nullptr || s.stream() == cudaStreamLegacy) return;
  Py_BEGIN_ALLOW_THREADS
  s.synchronize();
  Py_END_ALLOW_THREADS
}

PyObject *context_forward(Args a) {  // n_heads seq_len d_head q k v scale causal out
  const uint32_t heads = u32(a[0]), seq = u32(a[1]), d = u32(a[2]);
  expect_shape(a[8], seq, static_cast<uint64_t>(heads) * d, "output");
  float *q = ptr(a[3]), *k = ptr(a[4]), *v = ptr(a[5]), *out = ptr(a[8]);
  const float scale = real(a[6]);
  const uint32_t causal = truth(a[7]);
  finish_other_stream();
  Py_BEGIN_ALLOW_THREADS
  if (heads == 1) fn.launch_fused_attention(q, k, v, out, seq, d, scale, causal);  // lib.rs:2055-2065
  else fn.launch_fused_mha_forward(q, k, v, out, heads, seq, d, scale, causal);
  Py_END_ALLOW_THREADS
  check(fn.df_attn_last_status());
  Py_RETURN_NONE;
}

PyObject *context_backward(Args a) {  // n_heads seq_len d_head q k v d_out scale causal d_q d_k d_v probabilities
  const uint32_t heads = u32(a[0]), seq = u32(a[1]), d = u32(a[2]);
  const char *names[3] = {"d_q", "d_k", "d_v"};
  for (int i = 0; i < 3; ++i) expect_shape(a[9 + i], seq, static_cast<uint64_t>(heads) * d, names[i]);
  float *q = ptr(a[3]), *k = ptr(a[4]), *v = ptr(a[5]), *g = ptr(a[6]), *dq = ptr(a[9]), *dk = ptr(a[10]), *dv = ptr(a[11]), *prob = ptr(a[12]);
  const float scale = real(a[7]);
  const uint32_t causal = truth(a[8]);
  finish_other_stream();
  Py_BEGIN_ALLOW_THREADS
  if (heads == 1) fn.launch_attention_backward(q, k, v, g, dq, dk, dv, prob, seq, d, scale, causal);  // lib.rs:2260-2274
  else fn.launch_fused_mha_backward(q, k, v, g, dq, dk, dv, prob, heads, seq, d, scale, causal);
  Py_END_ALLOW_THREADS
  check(fn.df_attn_last_status());
  Py_RETURN_NONE;
}

// ---------------------------------------------------------------- module
PyObject *bind(PyObject *, PyObject *args) {  // ({name: address}, error class)
  PyObject *table, *error;
  if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &table, &error)) return nullptr;
#define X(name)                                                                                       \
  {                                                                                                   \
    PyObject *v = PyDict_GetItemString(table, #name);                                                 \
    void *p = v ? PyLong_AsVoidPtr(v) : nullptr;                                                      \
    if (!p) {                                                                                         \
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "no address given for " #name);      \
      return nullptr;                                                                                 \
    }                                                                                                 \
    fn.name = reinterpret_cast<decltype(fn.name)>(p);                                                 \
  }
  DF_FUNCTIONS(X)
#undef X
  Py_INCREF(error);
  Py_XSETREF(attention_error, error);
  Py_RETURN_NONE;
}

template <PyObject *(*F)(Args), int N>
PyObject *entry(PyObject *, Args args, Py_ssize_t n) {
  if (n != N || !attention_error) {
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments, or bind() was not called");
    return nullptr;
  }
  try {
    return F(args);
  } catch (const PythonError &) {
  } catch (const std::exception &e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}
#define ENTRY(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&entry<name, n>)), METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    ENTRY(forward, 10), ENTRY(forward_bf16, 11), ENTRY(backward, 14), ENTRY(backward_bf16, 14), ENTRY(backward_static_scratch, 13),
    ENTRY(backward_block, 14), ENTRY(backward_block_bf16, 15), ENTRY(delta, 5), ENTRY(delta_bf16, 5), ENTRY(decode, 12),
    ENTRY(merge_partials, 6), ENTRY(accumulate, 3), ENTRY(linear_qkv, 11), ENTRY(linear, 6), ENTRY(linear_gelu, 7), ENTRY(chunked_logit_ce, 6),
    ENTRY(layernorm, 7), ENTRY(layernorm_backward, 9), ENTRY(gelu, 3), ENTRY(gelu_backward, 4), ENTRY(adamw_update, 12), ENTRY(adamw_step, 11),
    ENTRY(context_forward, 9), ENTRY(context_backward, 13), {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "df_python_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_df_python_calls(void) { return PyModule_Create(&module); }
