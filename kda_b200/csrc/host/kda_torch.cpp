// The operators' host path on torch tensors: argument checks, conversions, output and workspace allocation, autograd and
// the calls into libkda_b200.so.  Reached from kda_b200/ops.py through plain CPython functions (METH_FASTCALL).
//
// Why native: a decode step of one sequence keeps the GPU busy for 5 us, while the same steps in Python (attribute
// look-ups, a ctypes structure, torch.empty, the device context manager) took 23 us of host time, and a training call 300 to
// 500 us through three Python autograd functions.  Here a decode call costs about 6 us and a whole forward + backward about 50 us.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>
#include <optional>
#include <sstream>
#include <string>

#include "kda_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

PyObject* g_kda_error = nullptr;        // kda_b200._lib.KdaError
PyObject* g_raise_status = nullptr;     // kda_b200._lib.raise_chunk_status(value, what)

// ---- errors: the Python exception types of the operators' contract ---------------------------------------------------
struct PyFailure {
  PyObject* type;
  std::string text;
};
template <class... A>
std::string cat(const A&... a) {
  std::ostringstream s;
  (s << ... << a);
  return s.str();
}
template <class... A>
[[noreturn]] void fail(PyObject* type, const A&... a) {
  throw PyFailure{type, cat(a...)};
}
#define KDA_REQUIRE(cond, type, ...) \
  do {                               \
    if (!(cond)) fail(type, __VA_ARGS__); \
  } while (0)

struct GilRelease {
  PyThreadState* st = PyEval_SaveThread();
  ~GilRelease() { PyEval_RestoreThread(st); }
};
struct GilAcquire {
  PyGILState_STATE st = PyGILState_Ensure();
  ~GilAcquire() { PyGILState_Release(st); }
};

// A code of the library other than 0: KdaError.  Also thrown on autograd's own threads, hence as a python_error that
// carries the Python exception across them.
[[noreturn]] void throw_current_python_error() {
  python_error e;
  e.persist();
  throw e;      // NOLINT
}
void check_rc(int rc, const char* what) {
  if (rc == 0) return;
  GilAcquire gil;
  PyErr_SetString(g_kda_error ? g_kda_error : PyExc_RuntimeError, cat(what, " failed with code ", rc, ": ", kda_b200_strerror(rc)).c_str());
  throw_current_python_error();
}
bool checked_mode() {
  const char* e = std::getenv("KDA_B200_CHECK");
  return e && *e && std::strcmp(e, "0") != 0;
}
void check_chunk_status(const Tensor& ws, const char* what) {
  uint32_t v = 0;
  check_rc(kda_chunk_status(ws.data_ptr(), &v), "kda_chunk_status");
  if (!v) return;
  GilAcquire gil;
  PyObject* r = PyObject_CallFunction(g_raise_status, "Is", static_cast<unsigned>(v), what);
  if (r) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, "kda_b200: device status set");
  }
  throw_current_python_error();
}

// ---- small helpers ---------------------------------------------------------------------------------------------------
int dtype_code(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? KDA_BF16 : KDA_FP32; }
bool known_dtype(const Tensor& t) { return t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kFloat; }
template <class T = void>
T* ptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }
Tensor dense(const Tensor& t) { return t.defined() ? t.contiguous() : t; }
Tensor f32(const Tensor& t) {
  if (!t.defined()) return t;
  const Tensor c = t.contiguous();
  return c.scalar_type() == at::kFloat ? c : c.to(at::kFloat);
}
// The kernels need 16-byte aligned rows.  Heads narrower than theirs are read in place but may start anywhere (they used to be padded into new
// tensors); full-width tensors at odd addresses are refused by the library.
Tensor aligned(const Tensor& t, bool narrow) {
  return narrow && t.defined() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 ? t.clone() : t;
}
Tensor i32(const Tensor& t, const at::Device& dev) {
  if (!t.defined()) return t;
  if (t.scalar_type() == at::kInt && t.device() == dev) return t.contiguous();
  return t.to(at::TensorOptions().device(dev).dtype(at::kInt)).contiguous();
}
Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const at::Device& dev) {
  return at::detail::empty_cuda(shape, dt, dev, std::nullopt);      // straight to the allocator: 0.5 us less than through the dispatcher
}
Tensor bytes(size_t n, const at::Device& dev) { return empty({static_cast<int64_t>(n)}, at::kByte, dev); }
cudaStream_t stream_of(const at::Device& dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

struct Sizes {
  int64_t B, T, HQ, H, K, V;      // H counts value heads; q and k have HQ
};
// The operators' common argument checks (types and texts as documented in kda_b200/ops.py).
Sizes check_common(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& h0, const Tensor& cu) {
  KDA_REQUIRE(q.is_cuda(), PyExc_RuntimeError, "kda_b200 runs on CUDA (sm_100a) tensors only; there is no CPU path");
  KDA_REQUIRE(q.dim() == 4 && v.dim() == 4, PyExc_ValueError, "q, k, v must be [B, T, H, D], got q=", q.sizes(), " v=", v.sizes());
  const Sizes s{q.size(0), q.size(1), q.size(2), v.size(2), q.size(3), v.size(3)};
  KDA_REQUIRE(q.sizes() == k.sizes(), PyExc_AssertionError, "q and k must have the same shape, got q=", q.sizes(), " vs k=", k.sizes());
  KDA_REQUIRE(s.HQ > 0 && s.H % s.HQ == 0, PyExc_AssertionError, "For GVA, num_v_heads (HV=", s.H, ") must be evenly divisible by num_qk_heads (H=", s.HQ,
              "), but got HV % H = ", s.HQ > 0 ? s.H % s.HQ : 0);
  KDA_REQUIRE(s.K <= 256, PyExc_AssertionError, "Currently we only support key headdim <=256 for KDA, got ", s.K, ".");
  KDA_REQUIRE(v.size(0) == s.B && v.size(1) == s.T, PyExc_AssertionError, "v must have shape [B, T, HV, V], got ", v.sizes());
  KDA_REQUIRE((g.sizes() == at::IntArrayRef{s.B, s.T, s.H, s.K}), PyExc_AssertionError, "g must have shape [B, T, HV, K]=[", s.B, ", ", s.T, ", ", s.H, ", ", s.K,
              "], got ", g.sizes());
  KDA_REQUIRE((beta.sizes() == at::IntArrayRef{s.B, s.T, s.H}), PyExc_AssertionError, "beta must have shape [B, T, HV]=[", s.B, ", ", s.T, ", ", s.H, "], got ",
              beta.sizes());
  if (cu.defined()) {
    KDA_REQUIRE(s.B == 1, PyExc_ValueError, "The batch size is expected to be 1 rather than ", s.B,
                " when using `cu_seqlens`.Please flatten variable-length inputs before processing.");
    KDA_REQUIRE(!h0.defined() || h0.size(0) == cu.size(0) - 1, PyExc_ValueError,
                "The number of initial states is expected to be equal to the number of input sequences, i.e., ", cu.size(0) - 1, " rather than ",
                h0.defined() ? h0.size(0) : 0, ".");
  }
  KDA_REQUIRE(!h0.defined() || h0.scalar_type() == at::kFloat, PyExc_AssertionError, "initial_state must be in float32.");
  KDA_REQUIRE(known_dtype(q) && k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(), PyExc_NotImplementedError,
              "kda_b200: q, k, v must share dtype bfloat16 or float32, got ", q.scalar_type());
  return s;
}

// ======================================================================================================================
// token-recurrent forward (decode)
// ======================================================================================================================
struct RecurrentCall {
  Tensor q, k, v, g, beta, A_log, dt_bias, h0, cu, slots, accepted, out;
  std::optional<double> scale, lower_bound;
  bool output_final = false, inplace = false, l2norm = false, gate = false, beta_sigmoid = false, transposed = false;
  bool training = false;      // float32 with gradients: the forward that the backward belongs to,
  Tensor saved;               // and what it leaves for it (undefined: nothing)
};

std::pair<Tensor, Tensor> recurrent_fwd(RecurrentCall& c) {
  const Sizes s = check_common(c.q, c.k, c.v, c.g, c.beta, Tensor(), c.cu);
  KDA_REQUIRE(!c.transposed || s.K == 64 || s.K == 128, PyExc_NotImplementedError, "kda_b200: transpose_state_layout needs K = 64 or 128, got ", s.K);
  const at::Device dev = c.q.device();
  const c10::cuda::CUDAGuard guard(dev);
  kda_recurrent_args a{};
  // the gate activation and the beta sigmoid run inside the recurrent kernels (no separate pass over g and beta)
  Tensor g, beta, A32, b32;
  if (c.gate) {
    KDA_REQUIRE(c.A_log.defined(), PyExc_AssertionError, "A_log must be provided when use_gate_in_kernel=True.");
    g = known_dtype(c.g) ? dense(c.g) : f32(c.g);
    A32 = f32(c.A_log.device() == dev ? c.A_log : c.A_log.to(dev));
    b32 = c.dt_bias.defined() ? f32(c.dt_bias.device() == dev ? c.dt_bias : c.dt_bias.to(dev)) : Tensor();
    KDA_REQUIRE(A32.numel() == s.H && (!b32.defined() || b32.numel() == s.H * s.K), PyExc_ValueError, "A_log must have ", s.H, " elements and dt_bias ", s.H * s.K);
    a.A_log = ptr<float>(A32);
    a.dt_bias = ptr<float>(b32);
    a.g_raw_dtype = dtype_code(g);
    a.lower_bound = static_cast<float>(c.lower_bound.value_or(0.0));
    a.use_lower_bound = c.lower_bound.has_value();
  } else {
    g = f32(c.g);
  }
  if (c.beta_sigmoid) {
    beta = known_dtype(c.beta) ? dense(c.beta) : f32(c.beta);
    a.beta_sigmoid = 1;
    a.beta_raw_dtype = dtype_code(beta);
  } else {
    beta = f32(c.beta);
  }
  const Tensor q = dense(c.q), k = dense(c.k), v = dense(c.v);
  const Tensor cu = i32(c.cu, dev);
  const int64_t N = cu.defined() ? cu.numel() - 1 : s.B;
  const Tensor h0 = dense(c.h0);
  Tensor ht;
  if (c.inplace) {
    KDA_REQUIRE(c.h0.defined(), PyExc_AssertionError, "inplace_final_state needs an initial_state");
    KDA_REQUIRE(h0.data_ptr() == c.h0.data_ptr() && h0.scalar_type() == at::kFloat, PyExc_ValueError, "inplace_final_state needs a contiguous fp32 initial_state");
    ht = h0;
  } else if (c.output_final) {
    ht = empty({N, s.H, c.transposed ? s.V : s.K, c.transposed ? s.K : s.V}, at::kFloat, dev);
  }
  Tensor idx, acc;
  if (c.slots.defined()) {
    KDA_REQUIRE(c.inplace, PyExc_ValueError, "ssm_state_indices requires inplace_final_state=True");
    idx = i32(c.slots, dev);
    a.state_indices_stride = idx.dim() == 1 ? 1 : static_cast<int32_t>(idx.stride(0));
    KDA_REQUIRE(idx.dim() != 1 || cu.defined() || s.T <= 1, PyExc_ValueError, "ssm_state_indices must be [N, T] when a sequence has more than one token");
    acc = i32(c.accepted, dev);
  } else {
    KDA_REQUIRE(!c.accepted.defined(), PyExc_ValueError, "num_accepted_tokens requires ssm_state_indices");
  }
  Tensor o;
  if (c.out.defined()) {
    KDA_REQUIRE(c.out.sizes() == c.v.sizes(), PyExc_AssertionError, "`out` must have v's shape");
    KDA_REQUIRE(c.out.is_contiguous() && c.out.scalar_type() == c.v.scalar_type(), PyExc_ValueError, "`out` must be contiguous and of v's dtype");
    o = c.out;
  } else {
    o = empty(v.sizes(), v.scalar_type(), dev);
  }
  a.q = ptr(q); a.k = ptr(k); a.v = ptr(v); a.g = static_cast<const float*>(ptr(g)); a.beta = static_cast<const float*>(ptr(beta));
  a.h0 = ptr<float>(h0); a.ht = ptr<float>(ht); a.o = ptr(o);
  a.cu_seqlens = ptr<int32_t>(cu); a.state_indices = ptr<int32_t>(idx); a.num_accepted_tokens = ptr<int32_t>(acc);
  a.tokens = s.B * s.T; a.N = static_cast<int32_t>(N); a.T = static_cast<int32_t>(s.T); a.H = static_cast<int32_t>(s.H);
  a.K = static_cast<int32_t>(s.K); a.V = static_cast<int32_t>(s.V); a.HQ = static_cast<int32_t>(s.HQ);
  a.io_dtype = dtype_code(q); a.use_qk_l2norm = c.l2norm; a.transpose_state = c.transposed;
  a.scale = static_cast<float>(c.scale ? *c.scale : 1.0 / std::sqrt(static_cast<double>(s.K)));
  if (c.training) {
    if (c.saved.defined()) check_rc(kda_recurrent_train_fwd(&a, c.saved.data_ptr(), static_cast<size_t>(c.saved.numel()), stream_of(dev)), "kda_recurrent_train_fwd");
    else check_rc(kda_recurrent_walk_fwd(&a, stream_of(dev)), "kda_recurrent_walk_fwd");
    return {o, ht};
  }
  check_rc(kda_recurrent_fwd(&a, stream_of(dev)), "kda_recurrent_fwd");
  if (checked_mode()) {
    uint32_t st = 0;
    check_rc(kda_recurrent_status(&st), "kda_recurrent_status");
    if (st) fail(g_kda_error, "kda_recurrent_fwd: device status ", st, " (a bounded wait gave up); the outputs are incomplete");
  }
  // in place: the caller's own tensor object comes back
  return {o, c.inplace ? c.h0 : ht};
}

// ======================================================================================================================
// chunked forward / backward (bf16, K = V = 128 inside the kernels)
// ======================================================================================================================
struct ChunkOpts {
  double scale = 1.0, lower_bound = 0.0;
  bool has_lower_bound = false, output_final = false, l2norm = false, gate = false, beta_sigmoid = false, safe_gate = false;
  int slices = 0;
};

// What the forward leaves for the backward.
struct ChunkSaved {
  Tensor q, k, v, g, beta, h0, cu, ws, g_raw, A32, b32, beta_raw;
};

int64_t sequences(const ChunkSaved& s) { return s.cu.defined() ? s.cu.numel() - 1 : s.q.size(0); }      // no cu_seqlens: the batch rows

kda_gate_args gate_args(const ChunkSaved& s, const ChunkOpts& o, int64_t tokens, int64_t H, int64_t K) {
  kda_gate_args a{};
  a.g_raw = ptr(s.g_raw); a.A_log = ptr<float>(s.A32); a.dt_bias = ptr<float>(s.b32); a.beta_raw = ptr(s.beta_raw);
  a.tokens = tokens; a.H = static_cast<int32_t>(H); a.K = static_cast<int32_t>(s.g_raw.defined() ? K : 8);
  a.g_dtype = s.g_raw.defined() ? dtype_code(s.g_raw) : KDA_FP32;
  a.beta_dtype = s.beta_raw.defined() ? dtype_code(s.beta_raw) : KDA_FP32;
  a.use_lower_bound = o.has_lower_bound; a.lower_bound = static_cast<float>(o.lower_bound);
  return a;
}

kda_chunk_args chunk_args(const ChunkSaved& s, const ChunkOpts& o, int save) {
  kda_chunk_args a{};
  a.q = ptr(s.q); a.k = ptr(s.k); a.v = ptr(s.v); a.g = ptr<float>(s.g); a.beta = ptr<float>(s.beta); a.h0 = ptr<float>(s.h0);
  a.cu_seqlens = ptr<int32_t>(s.cu); a.workspace = ptr(s.ws); a.workspace_bytes = static_cast<size_t>(s.ws.numel());
  a.tokens = s.q.size(0) * s.q.size(1);
  a.N = static_cast<int32_t>(sequences(s)); a.H = static_cast<int32_t>(s.v.size(2)); a.HQ = static_cast<int32_t>(s.q.size(2));
  a.K = a.V = 128; a.k_cols = static_cast<int32_t>(s.q.size(3)); a.v_cols = static_cast<int32_t>(s.v.size(3)); a.io_dtype = dtype_code(s.q); a.use_qk_l2norm = o.l2norm;
  a.save_for_backward = save; a.scale = static_cast<float>(o.scale); a.scan_slices = o.slices; a.safe_gate = o.safe_gate;
  return a;
}
int save_bits(const ChunkOpts& o) { return 1 | (o.l2norm ? 2 : 0); }      // bit 1: the forward keeps the normalised q, k

// o (and the final state) of the chunked forward; `s` receives the tensors the kernels read.
std::pair<Tensor, Tensor> chunk_forward(ChunkSaved& s, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& h0,
                                        const Tensor& A_log, const Tensor& dt_bias, const Tensor& cu, const ChunkOpts& o, bool need_grad) {
  const at::Device dev = q.device();
  const c10::cuda::CUDAGuard guard(dev);
  const cudaStream_t st = stream_of(dev);
  const int64_t B = q.size(0), T = q.size(1), H = v.size(2), K = q.size(3), V = v.size(3), tokens = B * T;
  const bool narrow = K < 128 || V < 128;
  s.q = aligned(dense(q), narrow); s.k = aligned(dense(k), narrow); s.v = aligned(dense(v), narrow); s.h0 = aligned(dense(h0), narrow);
  // the forward kernel activates g and beta itself; the activated values are written only for a backward
  if (o.gate) {
    s.g_raw = dense(g);
    s.A32 = f32(A_log);
    s.b32 = f32(dt_bias);
    if (need_grad) s.g = empty(g.sizes(), at::kFloat, dev);
  } else {
    s.g = aligned(f32(g), narrow);
  }
  if (o.beta_sigmoid) {
    s.beta_raw = dense(beta);
    if (need_grad) s.beta = empty(beta.sizes(), at::kFloat, dev);
  } else {
    s.beta = f32(beta);
  }
  s.cu = cu;
  const int64_t N = sequences(s);
  const int save = need_grad ? save_bits(o) : 0;
  s.ws = bytes(kda_chunk_workspace_bytes(tokens, static_cast<int32_t>(N), static_cast<int32_t>(H), static_cast<int32_t>(K), static_cast<int32_t>(V), save), dev);
  const Tensor out = empty(v.sizes(), v.scalar_type(), dev);
  const Tensor ht = o.output_final ? empty({N, H, K, V}, at::kFloat, dev) : Tensor();
  kda_chunk_args a = chunk_args(s, o, save);
  a.o = ptr(out);
  a.ht = ptr<float>(ht);
  if (o.gate) {
    a.g_raw = ptr(s.g_raw); a.g_raw_dtype = dtype_code(s.g_raw); a.A_log = ptr<float>(s.A32); a.dt_bias = ptr<float>(s.b32);
    a.use_lower_bound = o.has_lower_bound; a.lower_bound = static_cast<float>(o.lower_bound);
  }
  if (o.beta_sigmoid) {
    a.beta_raw = ptr(s.beta_raw); a.beta_raw_dtype = dtype_code(s.beta_raw);
  }
  check_rc(kda_chunk_fwd(&a, st), "kda_chunk_fwd");
  if (checked_mode()) check_chunk_status(s.ws, "kda_chunk_fwd");
  return {out, ht};
}

class ChunkFunction : public torch::autograd::Function<ChunkFunction> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                               const std::optional<Tensor>& h0, const std::optional<Tensor>& A_log, const std::optional<Tensor>& dt_bias,
                               const std::optional<Tensor>& cu, const ChunkOpts& o) {
    ChunkSaved s;
    auto [out, ht] = chunk_forward(s, q, k, v, g, beta, h0.value_or(Tensor()), A_log.value_or(Tensor()), dt_bias.value_or(Tensor()),
                                   cu.value_or(Tensor()), o, true);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({s.q, s.k, s.v, s.g, s.beta, s.h0, s.cu, s.ws, s.g_raw, s.A32, s.b32, s.beta_raw});
    // of the parameters themselves only shape and type: they may be updated before the backward (which reads the float32 copies)
    for (const auto& [name, t] : {std::pair{"A_log", A_log}, std::pair{"dt_bias", dt_bias}}) {
      if (!t) continue;
      ctx->saved_data[std::string(name) + "_sizes"] = t->sizes().vec();
      ctx->saved_data[std::string(name) + "_dtype"] = static_cast<int64_t>(t->scalar_type());
    }
    ctx->saved_data["flags"] = static_cast<int64_t>(o.has_lower_bound | o.output_final << 1 | o.l2norm << 2 | o.gate << 3 | o.beta_sigmoid << 4 | o.safe_gate << 5 |
                                                    static_cast<int64_t>(o.slices) << 8);
    ctx->saved_data["scale"] = o.scale;
    ctx->saved_data["lower_bound"] = o.lower_bound;
    ctx->saved_data["g_dtype"] = static_cast<int64_t>(g.scalar_type());
    ctx->saved_data["beta_dtype"] = static_cast<int64_t>(beta.scalar_type());
    if (o.output_final) return {out, ht};
    return {out};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list t = ctx->get_saved_variables();
    ChunkSaved s{t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], t[10], t[11]};
    ChunkOpts o;
    const int64_t f = ctx->saved_data["flags"].toInt();
    o.has_lower_bound = f & 1; o.output_final = f & 2; o.l2norm = f & 4; o.gate = f & 8; o.beta_sigmoid = f & 16; o.safe_gate = f & 32;
    o.slices = static_cast<int>(f >> 8);
    o.scale = ctx->saved_data["scale"].toDouble();
    o.lower_bound = ctx->saved_data["lower_bound"].toDouble();
    const at::Device dev = s.q.device();
    const c10::cuda::CUDAGuard guard(dev);
    const cudaStream_t st = stream_of(dev);
    const int64_t tokens = s.q.size(0) * s.q.size(1), H = s.v.size(2), K = s.q.size(3), V = s.v.size(3), N = sequences(s);
    const bool narrow = K < 128 || V < 128;
    const Tensor d_o = grads[0].defined() ? aligned(dense(grads[0].scalar_type() == s.v.scalar_type() ? grads[0] : grads[0].to(s.v.scalar_type())), narrow) : at::zeros_like(s.v);
    const Tensor d_ht = grads.size() > 1 ? aligned(f32(grads[1]), narrow) : Tensor();
    const Tensor dq = empty(s.q.sizes(), s.q.scalar_type(), dev), dk = empty(s.k.sizes(), s.k.scalar_type(), dev), dv = empty(s.v.sizes(), s.v.scalar_type(), dev);
    Tensor dg = empty(s.g.sizes(), at::kFloat, dev), dbeta = empty(s.beta.sizes(), at::kFloat, dev);
    const Tensor dh0 = s.h0.defined() ? empty(s.h0.sizes(), at::kFloat, dev) : Tensor();
    const int flags = (o.l2norm ? 1 | 4 : 0) | (s.q.size(2) != H ? 2 : 0);
    const Tensor bws = bytes(
        kda_chunk_bwd_workspace_bytes(tokens, static_cast<int32_t>(N), static_cast<int32_t>(H), static_cast<int32_t>(K), static_cast<int32_t>(V), flags), dev);
    kda_chunk_args a = chunk_args(s, o, save_bits(o));
    a.d_o = ptr(d_o); a.d_ht = ptr<float>(d_ht); a.dq = ptr(dq); a.dk = ptr(dk); a.dv = ptr(dv); a.dg = ptr<float>(dg); a.dbeta = ptr<float>(dbeta);
    a.dh0 = ptr<float>(dh0); a.bwd_workspace = ptr(bws); a.bwd_workspace_bytes = static_cast<size_t>(bws.numel());
    check_rc(kda_chunk_bwd(&a, st), "kda_chunk_bwd");
    if (checked_mode()) check_chunk_status(s.ws, "kda_chunk_bwd");
    Tensor dA, db;
    if (o.gate || o.beta_sigmoid) {
      kda_gate_args ga = gate_args(s, o, tokens, H, K);
      Tensor dg_raw, dbeta_raw, gws;
      if (o.gate) {
        dg_raw = empty(s.g_raw.sizes(), s.g_raw.scalar_type(), dev);
        dA = empty({H}, at::kFloat, dev);
        if (s.b32.defined()) db = empty({H * K}, at::kFloat, dev);
        gws = bytes(kda_gate_bwd_workspace_bytes(tokens, static_cast<int32_t>(H), static_cast<int32_t>(K)), dev);
        ga.dg = ptr<float>(dg); ga.dg_raw = ptr(dg_raw); ga.dA_log = ptr<float>(dA); ga.ddt_bias = ptr<float>(db);
        ga.workspace = ptr(gws); ga.workspace_bytes = static_cast<size_t>(gws.numel());
      }
      if (o.beta_sigmoid) {
        dbeta_raw = empty(s.beta_raw.sizes(), s.beta_raw.scalar_type(), dev);
        ga.dbeta = ptr<float>(dbeta); ga.dbeta_raw = ptr(dbeta_raw);
      }
      check_rc(kda_gate_bwd(&ga, st), "kda_gate_bwd");
      if (o.gate) dg = dg_raw;
      if (o.beta_sigmoid) dbeta = dbeta_raw;
    }
    const auto g_dtype = static_cast<at::ScalarType>(ctx->saved_data["g_dtype"].toInt());
    const auto beta_dtype = static_cast<at::ScalarType>(ctx->saved_data["beta_dtype"].toInt());
    if (dg.scalar_type() != g_dtype) dg = dg.to(g_dtype);
    if (dbeta.scalar_type() != beta_dtype) dbeta = dbeta.to(beta_dtype);
    auto as = [&](const Tensor& d, const std::string& name) {
      return d.view(ctx->saved_data[name + "_sizes"].toIntVector()).to(static_cast<at::ScalarType>(ctx->saved_data[name + "_dtype"].toInt()));
    };
    if (dA.defined()) dA = as(dA, "A_log");
    if (db.defined()) db = as(db, "dt_bias");
    return {dq, dk, dv, dg, dbeta, dh0, dA, db, Tensor(), Tensor()};
  }
};

struct ChunkCall {
  Tensor q, k, v, g, beta, A_log, dt_bias, h0, cu;
  std::optional<double> scale, lower_bound;
  bool output_final = false, l2norm = false, gate = false, beta_sigmoid = false, safe_gate = false, transposed = false;
  int slices = 0;
};

// Forward-mode tangents: there is no forward-mode derivative, and a call without gradients passes autograd by, which would drop them.
bool has_tangent(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->defined() && t->_fw_grad(0).defined()) return true;
  return false;
}

bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// bf16, heads up to 128.  Returns false for a call that takes another path: float32 (token-recurrent kernels), larger heads, and the narrow
// ones that the kernels do not read in place (no multiple of eight columns; gradients with grouped value heads).
bool chunk_kda(ChunkCall& c, Tensor& o, Tensor& ht) {
  const Sizes s = check_common(c.q, c.k, c.v, c.g, c.beta, c.h0, c.cu);
  const bool grads = wants_grad({&c.q, &c.k, &c.v, &c.g, &c.beta, &c.h0, &c.A_log, &c.dt_bias});
  if (c.q.scalar_type() != at::kBFloat16 || s.K > 128 || s.V > 128 || s.K % 8 || s.V % 8) return false;
  if ((s.K < 128 || s.V < 128) && grads && s.HQ != s.H) return false;
  KDA_REQUIRE(!has_tangent({&c.q, &c.k, &c.v, &c.g, &c.beta, &c.h0, &c.A_log, &c.dt_bias}), PyExc_NotImplementedError,
              "kda_b200: chunk_kda has no forward-mode derivative (jvp)");
  ChunkOpts opt;
  opt.scale = c.scale ? *c.scale : 1.0 / std::sqrt(static_cast<double>(s.K));
  opt.output_final = c.output_final; opt.l2norm = c.l2norm; opt.gate = c.gate; opt.beta_sigmoid = c.beta_sigmoid; opt.safe_gate = c.safe_gate;
  opt.slices = c.slices;
  if (c.gate) {
    KDA_REQUIRE(c.A_log.defined(), PyExc_AssertionError, "A_log must be provided when use_gate_in_kernel=True.");
    if (c.safe_gate) {
      KDA_REQUIRE(c.lower_bound, PyExc_ValueError, "`lower_bound` must be specified when `safe_gate=True` and `use_gate_in_kernel=True`.");
      KDA_REQUIRE(*c.lower_bound >= -5 && *c.lower_bound < 0, PyExc_ValueError, "`lower_bound` must be in the safe range [-5, 0), got ", *c.lower_bound, ".");
    }
    KDA_REQUIRE(s.K % 8 == 0, PyExc_NotImplementedError, "kda_b200: the gate kernels need K to be a multiple of 8, got ", s.K);
    KDA_REQUIRE(known_dtype(c.g), PyExc_NotImplementedError, "kda_b200: raw gate / beta inputs must be bfloat16 or float32");
    KDA_REQUIRE(c.A_log.numel() == s.H, PyExc_AssertionError, "A_log must have H=", s.H, " elements, got ", c.A_log.numel());
    KDA_REQUIRE(!c.dt_bias.defined() || c.dt_bias.numel() == s.H * s.K, PyExc_AssertionError, "dt_bias must have H*K=", s.H * s.K, " elements");
    opt.has_lower_bound = c.lower_bound.has_value();
    opt.lower_bound = c.lower_bound.value_or(0.0);
  } else {
    c.A_log = c.dt_bias = Tensor();
  }
  KDA_REQUIRE(!c.beta_sigmoid || known_dtype(c.beta), PyExc_NotImplementedError, "kda_b200: raw beta must be bfloat16 or float32");
  const at::Device dev = c.q.device();
  if (c.transposed && c.h0.defined()) c.h0 = c.h0.transpose(-1, -2);
  const Tensor cu = i32(c.cu, dev);
  if (grads) {
    auto some = [](const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; };
    const variable_list r = ChunkFunction::apply(c.q, c.k, c.v, c.g, c.beta, some(c.h0), some(c.A_log), some(c.dt_bias), some(cu), opt);
    o = r[0];
    if (r.size() > 1) ht = r[1];
  } else {
    ChunkSaved saved;
    std::tie(o, ht) = chunk_forward(saved, c.q, c.k, c.v, c.g, c.beta, c.h0, c.A_log, c.dt_bias, cu, opt, false);
  }
  if (c.transposed && ht.defined()) ht = ht.transpose(-1, -2).contiguous();
  return true;
}

// ======================================================================================================================
// CPython functions
// ======================================================================================================================
Tensor tensor_arg(PyObject* o, const char* name) {
  if (o == Py_None) return Tensor();
  KDA_REQUIRE(THPVariable_Check(o), PyExc_TypeError, "kda_b200: `", name, "` must be a tensor");
  return THPVariable_Unpack(o);
}
Tensor need_arg(PyObject* o, const char* name) {
  KDA_REQUIRE(o != Py_None, PyExc_TypeError, "kda_b200: `", name, "` must be a tensor, got None");
  return tensor_arg(o, name);
}
bool bool_arg(PyObject* o) {
  if (o == Py_True) return true;
  if (o == Py_False || o == Py_None) return false;
  const int r = PyObject_IsTrue(o);
  if (r < 0) throw python_error();
  return r != 0;
}
std::optional<double> double_arg(PyObject* o) {
  if (o == Py_None) return std::nullopt;
  const double d = PyFloat_AsDouble(o);
  if (d == -1.0 && PyErr_Occurred()) throw python_error();
  return d;
}
PyObject* pair(PyObject* a, PyObject* b) {
  PyObject* t = PyTuple_Pack(2, a, b);
  Py_DECREF(a);
  Py_DECREF(b);
  return t;
}
PyObject* wrap(const Tensor& t) {
  if (t.defined()) return THPVariable_Wrap(t);
  Py_RETURN_NONE;
}
#define KDA_BEGIN \
  HANDLE_TH_ERRORS try {
#define KDA_END                                     \
  }                                                 \
  catch (const PyFailure& e) {                      \
    PyErr_SetString(e.type, e.text.c_str());        \
    return nullptr;                                 \
  }                                                 \
  END_HANDLE_TH_ERRORS

PyObject* py_recurrent_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  KDA_BEGIN
  KDA_REQUIRE(n == 20 || n == 21, PyExc_TypeError, "recurrent_fwd takes 20 or 21 arguments");
  RecurrentCall c;
  c.q = need_arg(a[0], "q"); c.k = need_arg(a[1], "k"); c.v = need_arg(a[2], "v"); c.g = need_arg(a[3], "g"); c.beta = need_arg(a[4], "beta");
  c.A_log = tensor_arg(a[5], "A_log"); c.dt_bias = tensor_arg(a[6], "dt_bias"); c.h0 = tensor_arg(a[7], "initial_state");
  c.scale = double_arg(a[8]); c.output_final = bool_arg(a[9]); c.inplace = bool_arg(a[10]); c.cu = tensor_arg(a[11], "cu_seqlens");
  c.slots = tensor_arg(a[12], "ssm_state_indices"); c.accepted = tensor_arg(a[13], "num_accepted_tokens"); c.l2norm = bool_arg(a[14]);
  c.gate = bool_arg(a[15]); c.beta_sigmoid = bool_arg(a[16]); c.lower_bound = double_arg(a[17]); c.out = tensor_arg(a[18], "out");
  c.transposed = bool_arg(a[19]);
  c.training = n == 21;
  if (c.training) c.saved = tensor_arg(a[20], "saved");
  std::pair<Tensor, Tensor> r;
  {
    GilRelease nogil;
    const at::NoGradGuard no_grad;
    r = recurrent_fwd(c);
  }
  return pair(wrap(r.first), wrap(r.second));
  KDA_END
}

PyObject* py_chunk_kda(PyObject*, PyObject* const* a, Py_ssize_t n) {
  KDA_BEGIN
  KDA_REQUIRE(n == 18, PyExc_TypeError, "chunk_kda takes 18 arguments");
  ChunkCall c;
  c.q = need_arg(a[0], "q"); c.k = need_arg(a[1], "k"); c.v = need_arg(a[2], "v"); c.g = need_arg(a[3], "g"); c.beta = need_arg(a[4], "beta");
  c.A_log = tensor_arg(a[5], "A_log"); c.dt_bias = tensor_arg(a[6], "dt_bias"); c.h0 = tensor_arg(a[7], "initial_state");
  c.scale = double_arg(a[8]); c.output_final = bool_arg(a[9]); c.cu = tensor_arg(a[10], "cu_seqlens"); c.l2norm = bool_arg(a[11]);
  c.gate = bool_arg(a[12]); c.beta_sigmoid = bool_arg(a[13]); c.lower_bound = double_arg(a[14]); c.safe_gate = bool_arg(a[15]);
  c.transposed = bool_arg(a[16]); c.slices = static_cast<int>(double_arg(a[17]).value_or(0));
  Tensor o, ht;
  bool done;
  {
    GilRelease nogil;
    done = chunk_kda(c, o, ht);
  }
  if (!done) Py_RETURN_NONE;
  return pair(wrap(o), wrap(ht));
  KDA_END
}

PyObject* py_set_errors(PyObject*, PyObject* args) {
  PyObject *err, *raiser;
  if (!PyArg_ParseTuple(args, "OO", &err, &raiser)) return nullptr;
  Py_INCREF(err);
  Py_INCREF(raiser);
  g_kda_error = err;
  g_raise_status = raiser;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"recurrent_fwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_recurrent_fwd)), METH_FASTCALL, "decode / token-recurrent forward"},
    {"chunk_kda", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_chunk_kda)), METH_FASTCALL, "chunked forward with autograd; None: not this path"},
    {"set_errors", py_set_errors, METH_VARARGS, "exception type and status reporter of kda_b200._lib"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_kda_torch", "host path of the kda_b200 operators", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__kda_torch() { return PyModule_Create(&module_def); }
