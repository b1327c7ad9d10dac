// The operators as PyTorch sees them: schema, CUDA implementations and autograd, in native
// code.  Checks arguments, allocates outputs and workspaces from the caching allocator and
// calls the C ABI (include/trifast_b200.h); no kernel lives here.
//
// What bounds the small problems is this layer: the device needs 15 us for an n = 64 bf16 forward
// and 31 us for an n = 32 fp32 training step (replayed as a graph), a pass through these
// operators takes 15 and 93 us, and with Python operators, Python autograd and ctypes calls it took
// 98 and 413 us.
//
// Mirrors the reference's operator boundary (src/trifast/torch.py:17-65 forward, :68-182
// backward, :185-217 autograd).

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <atomic>
#include <cctype>
#include <cstdlib>
#include <cstring>

#include "../../include/trifast_b200.h"

namespace {

using at::Tensor;

// ------------------------------------------------------------------ arguments
struct Problem {
  int64_t batch, heads, rows, n, d;
};

Problem check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b,
                     const Tensor& mask) {
  TORCH_CHECK_VALUE(q.dim() == 5, "q must be (batch, heads, rows, n, d); got ", q.sizes());
  const Problem p{q.size(0), q.size(1), q.size(2), q.size(3), q.size(4)};
  TORCH_CHECK_VALUE(k.sizes() == q.sizes() && v.sizes() == q.sizes(),
                    "q, k and v must have the same shape");
  const int64_t want_b[4] = {p.batch, p.heads, p.n, p.n};
  TORCH_CHECK_VALUE(b.sizes() == at::IntArrayRef(want_b, 4), "bias must be ",
                    at::IntArrayRef(want_b, 4), "; got ", b.sizes());
  const int64_t want_m[3] = {p.batch, p.rows, p.n};
  TORCH_CHECK_VALUE(mask.sizes() == at::IntArrayRef(want_m, 3), "mask must be ",
                    at::IntArrayRef(want_m, 3), "; got ", mask.sizes());
  const auto dt = q.scalar_type();
  TORCH_CHECK_TYPE(k.scalar_type() == dt && v.scalar_type() == dt && b.scalar_type() == dt,
                   "q, k, v and bias must share one dtype");
  TORCH_CHECK_TYPE(mask.scalar_type() == at::kBool,
                   "mask must be a bool tensor (True = key masked out)");
  const auto check_device = [&](const char* name, const Tensor& t) {
    TORCH_CHECK_VALUE(t.device() == q.device(), name, " is on ", t.device(), " but q is on ",
                      q.device(), ": every tensor must live on the same CUDA device");
  };
  check_device("k", k);
  check_device("v", v);
  check_device("bias", b);
  check_device("mask", mask);
  TORCH_CHECK(q.is_cuda(), "trifast_b200 runs on CUDA devices only (there is no CPU path)");
  return p;
}

int32_t dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return TRIFAST_F32;
    case at::kBFloat16: return TRIFAST_BF16;
    case at::kHalf: return TRIFAST_F16;
    default:
      TORCH_CHECK_TYPE(false, "unsupported dtype ", t, "; expected float32, bfloat16 or float16");
  }
}

// A contiguous tensor with the canonical strides: contiguous() alone keeps whatever strides
// extent-1 dimensions came with (PyTorch ignores them), but the library reads every stride.
Tensor dense(const Tensor& t) {
  Tensor c = t.contiguous();
  const int64_t nd = c.dim();
  int64_t want[8], acc = 1;
  bool same = true;
  for (int64_t a = nd - 1; a >= 0; --a) {
    want[a] = acc;
    same &= c.stride(a) == acc;
    acc *= std::max<int64_t>(c.size(a), 1);
  }
  return same ? c : c.as_strided(c.sizes(), at::IntArrayRef(want, nd));
}

// (b, h, i, j, d): d contiguous, every other stride a positive multiple of 16 bytes (TMA
// cannot describe an expanded dimension), base 16-byte aligned; anything else is copied.
Tensor prep5(const Tensor& t) {
  const int64_t es = t.element_size();
  bool ok = t.stride(4) == 1 && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0 &&
            t.stride(3) >= t.size(4);
  for (int a = 0; a < 4 && ok; ++a)
    ok = (t.stride(a) > 0 || t.size(a) == 1) && t.stride(a) * es % 16 == 0;
  return ok ? t : dense(t);
}

// Whether the kernels can take the bias and the mask as they lie: innermost stride 1, and, for
// the 16-bit kernels where no copies are prepared anyway (n a multiple of 8), rows that TMA and
// 4-byte reads can address.  Anything else (a projection's permuted output, a transposed map,
// an expanded view) goes in with TRIFAST_FLAG_STRIDED, and the call's prepare kernel makes the
// copies it needs: no separate copies here.
bool as_they_lie(const Tensor& b, const Tensor& m, int64_t n) {
  if (b.stride(3) != 1 || b.stride(2) < n || m.stride(2) != 1 || m.stride(1) < n) return false;
  if (b.scalar_type() == at::kFloat || n % 8 != 0) return true;
  bool ok = reinterpret_cast<uintptr_t>(b.const_data_ptr()) % 16 == 0 &&
            reinterpret_cast<uintptr_t>(m.const_data_ptr()) % 4 == 0;
  for (int a = 0; a < 3 && ok; ++a) ok = (b.stride(a) > 0 && b.stride(a) % 8 == 0) || b.size(a) == 1;
  for (int a = 0; a < 2 && ok; ++a) ok = m.stride(a) % 4 == 0 || m.size(a) == 1;
  return ok;
}

trifast_t5 view5(const Tensor& t) {
  return {const_cast<void*>(t.const_data_ptr()), {t.stride(0), t.stride(1), t.stride(2), t.stride(3)}};
}
trifast_t4_strided view4(const Tensor& t) {
  return {const_cast<void*>(t.const_data_ptr()), {t.stride(0), t.stride(1), t.stride(2), t.stride(3)}};
}
trifast_mask_strided view_mask(const Tensor& m) {
  return {static_cast<const uint8_t*>(m.const_data_ptr()), {m.stride(0), m.stride(1), m.stride(2)}};
}
// (the longer descriptors start with the shorter ones)
const trifast_t4* ptr(const trifast_t4_strided& v) { return reinterpret_cast<const trifast_t4*>(&v); }
const trifast_mask* ptr(const trifast_mask_strided& v) { return reinterpret_cast<const trifast_mask*>(&v); }

// Debug overrides of the tile heuristic, read per call like the rest of the binding does.
trifast_shape make_shape(const Problem& p, const Tensor& b, const Tensor& mask) {
  int32_t kernel = TRIFAST_KERNEL_AUTO;
  if (const char* e = std::getenv("TRIFAST_B200_KERNEL"); e && *e) {
    if (!strcasecmp(e, "simt"))
      kernel = TRIFAST_KERNEL_SIMT;
    else if (!strcasecmp(e, "tcgen05"))
      kernel = TRIFAST_KERNEL_TCGEN05;
    else
      TORCH_CHECK_VALUE(!strcasecmp(e, "auto"), "TRIFAST_B200_KERNEL=", e);
  }
  int32_t flags = 0;
  if (const char* f = std::getenv("TRIFAST_B200_FLAGS"); f && *f) {
    char* end = nullptr;
    flags = (int32_t)std::strtol(f, &end, 10);
    bool ok = end != f;
    while (std::isspace((unsigned char)*end)) ++end;
    ok = ok && !*end;
    TORCH_CHECK_VALUE(ok, "TRIFAST_B200_FLAGS=", f, " is not a decimal integer");
  }
  if (!as_they_lie(b, mask, p.n)) flags |= TRIFAST_FLAG_STRIDED;
  return {(int32_t)p.batch, (int32_t)p.heads, (int32_t)p.n, (int32_t)p.rows, (int32_t)p.d,
          dtype_code(b.scalar_type()), kernel, flags};
}

void check_rc(int rc, const char* what) {
  if (rc == TRIFAST_OK) return;
  TORCH_CHECK(false, what, ": ", trifast_status_str(rc), " (status ", rc,
              rc == TRIFAST_ERR_LAUNCH ? std::string(", ") + trifast_last_cuda_error() : std::string(),
              ")");
}

// First thing in every call: if an earlier kernel on this device gave up on one of its
// bounded waits, its outputs (and those of every launch since) were never written.  Costs one
// read of host memory when nothing is wrong.
void raise_if_device_gave_up(c10::DeviceIndex dev, cudaStream_t stream) {
  static std::atomic<volatile uint32_t*> words[64];
  TORCH_CHECK(dev >= 0 && dev < 64, "device index ", (int)dev);
  volatile uint32_t* w = words[dev].load(std::memory_order_acquire);
  if (!w) {
    uint32_t* p = nullptr;
    check_rc(trifast_host_status_word(&p), "trifast_host_status_word");
    w = p;
    words[dev].store(w, std::memory_order_release);
  }
  if (*w == 0) return;
  // (while the stream is being captured the status cannot be read: the word stays set, and the
  // next call outside the capture clears both)
  const bool cleared = trifast_check_device_status(stream) != TRIFAST_ERR_LAUNCH;
  if (cleared) *w = 0;
  TORCH_CHECK(false, "trifast_b200: ", trifast_status_str(TRIFAST_ERR_DEVICE_TIMEOUT),
              " in an earlier call on this device; the results of that call and of the calls "
              "after it are invalid ",
              cleared ? "(status cleared, retry is possible)"
                      : "(the status could not be cleared here, as during a graph capture)");
}

// ------------------------------------------------------------------ CUDA implementations
std::tuple<Tensor, Tensor> forward_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_,
                                        const Tensor& b, const Tensor& mask) {
  const Problem p = check_inputs(q_, k_, v_, b, mask);
  const trifast_shape shp = make_shape(p, b, mask);
  const c10::cuda::CUDAGuard guard(q_.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  raise_if_device_gave_up(q_.device().index(), stream);
  const Tensor q = prep5(q_), k = prep5(k_), v = prep5(v_);
  Tensor o = at::empty({p.batch, p.heads, p.rows, p.n, p.d}, q.options());
  Tensor lse = at::empty({p.batch, p.heads, p.rows, p.n}, q.options().dtype(at::kFloat));
  const size_t ws_bytes = trifast_forward_workspace_bytes(&shp);  // 0 on the CUDA-core plan
  Tensor ws;
  if (ws_bytes) ws = at::empty({(int64_t)ws_bytes}, q.options().dtype(at::kByte));
  const trifast_t5 tq = view5(q), tk = view5(k), tv = view5(v), to = view5(o);
  const trifast_t4_strided tb = view4(b);
  const trifast_mask_strided tm = view_mask(mask);
  check_rc(trifast_forward(&shp, &tq, &tk, &tv, ptr(tb), ptr(tm), &to, lse.mutable_data_ptr<float>(),
                           ws_bytes ? ws.mutable_data_ptr() : nullptr, ws_bytes, stream),
           "trifast_forward");
  return {o, lse};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> grads_cuda(const Tensor& do_, const Tensor& q_,
                                                      const Tensor& k_, const Tensor& v_,
                                                      const Tensor& b, const Tensor& o_,
                                                      const Tensor& lse_, const Tensor& mask) {
  const Problem p = check_inputs(q_, k_, v_, b, mask);
  const auto like_q = [&](const char* name, const Tensor& t) {
    TORCH_CHECK_VALUE(t.sizes() == q_.sizes() && t.scalar_type() == q_.scalar_type(), name,
                      " must be ", q_.sizes(), " ", q_.scalar_type(), "; got ", t.sizes(), " ",
                      t.scalar_type());
    TORCH_CHECK_VALUE(t.device() == q_.device(), name, " is on ", t.device(), " but q is on ",
                      q_.device());
  };
  like_q("do", do_);
  like_q("o", o_);
  const int64_t want_l[4] = {p.batch, p.heads, p.rows, p.n};
  TORCH_CHECK_VALUE(lse_.sizes() == at::IntArrayRef(want_l, 4) && lse_.scalar_type() == at::kFloat,
                    "lse must be float32 ", at::IntArrayRef(want_l, 4), "; got ",
                    lse_.scalar_type(), " ", lse_.sizes());
  TORCH_CHECK_VALUE(lse_.device() == q_.device(), "lse is on ", lse_.device(), " but q is on ",
                    q_.device());
  const trifast_shape shp = make_shape(p, b, mask);
  const c10::cuda::CUDAGuard guard(q_.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  raise_if_device_gave_up(q_.device().index(), stream);
  const Tensor d_o = prep5(do_), q = prep5(q_), k = prep5(k_), v = prep5(v_), o = prep5(o_),
               lse = lse_.contiguous();
  const at::IntArrayRef s5 = q_.sizes();
  Tensor dq = at::empty(s5, q.options()), dk = at::empty(s5, q.options()),
         dv = at::empty(s5, q.options());
  Tensor db = at::empty({p.batch, p.heads, p.n, p.n}, q.options());
  const size_t ws_bytes = trifast_backward_workspace_bytes(&shp);
  Tensor ws = at::empty({(int64_t)ws_bytes}, q.options().dtype(at::kByte));
  const trifast_t5 tdo = view5(d_o), tq = view5(q), tk = view5(k), tv = view5(v), to = view5(o),
                   tdq = view5(dq), tdk = view5(dk), tdv = view5(dv);
  const trifast_t4_strided tb = view4(b), tdb = view4(db);
  const trifast_mask_strided tm = view_mask(mask);
  check_rc(trifast_backward(&shp, &tdo, &tq, &tk, &tv, ptr(tb), ptr(tm), &to,
                            lse.const_data_ptr<float>(), &tdq, &tdk, &tdv, ptr(tdb), ws.mutable_data_ptr(), ws_bytes, stream),
           "trifast_backward");
  return {dq, dk, dv, db};
}

// The reference's signature: a zero gradient for the mask as well (torch.py:102,182).
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> backward_cuda(
    const Tensor& d_o, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b,
    const Tensor& o, const Tensor& lse, const Tensor& mask) {
  auto [dq, dk, dv, db] = grads_cuda(d_o, q, k, v, b, o, lse, mask);
  return {dq, dk, dv, db, at::zeros_like(mask)};
}

// ------------------------------------------------------------------ autograd
// (Nested calls go through the dispatcher, so that tracing sees operators, not pointers.)
using ForwardSig = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&,
                                              const Tensor&, const Tensor&);
using GradsSig = std::tuple<Tensor, Tensor, Tensor, Tensor>(
    const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
    const Tensor&, const Tensor&);
using BackwardSig = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>(
    const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
    const Tensor&, const Tensor&);

template <typename Sig>
c10::TypedOperatorHandle<Sig> find_op(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}
std::tuple<Tensor, Tensor> call_forward(const Tensor& q, const Tensor& k, const Tensor& v,
                                        const Tensor& b, const Tensor& mask) {
  static auto op = find_op<ForwardSig>("trifast_b200::triangle_attention");
  return op.call(q, k, v, b, mask);
}

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

class TriangleAttention : public torch::autograd::Function<TriangleAttention> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k,
                               const Tensor& v, const Tensor& b, const Tensor& mask) {
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->set_materialize_grads(false);
    auto [o, lse] = call_forward(q, k, v, b, mask);
    ctx->save_for_backward({q, k, v, b, mask, o, lse});
    return {o, lse};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    static auto op = find_op<GradsSig>("trifast_b200::triangle_attention_grads");
    const auto s = ctx->get_saved_variables();
    // (the gradient of lse is ignored, as in the reference)
    const Tensor d_o = grads[0].defined() ? grads[0] : at::zeros_like(s[5]);
    auto [dq, dk, dv, db] = op.call(d_o, s[0], s[1], s[2], s[3], s[5], s[6], s[4]);
    return {dq, dk, dv, db, Tensor()};
  }
};

bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!c10::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->requires_grad()) return true;
  return false;
}

std::tuple<Tensor, Tensor> forward_autograd(const Tensor& q, const Tensor& k, const Tensor& v,
                                            const Tensor& b, const Tensor& mask) {
  if (!wants_grad({&q, &k, &v, &b})) {
    at::AutoDispatchBelowADInplaceOrView below;
    return call_forward(q, k, v, b, mask);
  }
  const variable_list r = TriangleAttention::apply(q, k, v, b, mask);
  return {r[0], r[1]};
}

// The gradients have no gradient of their own: asking for one is an error when it is reached.
class Once : public torch::autograd::Function<Once> {
 public:
  static variable_list forward(AutogradContext*, const Tensor& d_o, const Tensor& q,
                               const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& o,
                               const Tensor& lse, const Tensor& mask) {
    static auto op = find_op<GradsSig>("trifast_b200::triangle_attention_grads");
    at::AutoDispatchBelowADInplaceOrView below;
    auto [dq, dk, dv, db] = op.call(d_o, q, k, v, b, o, lse, mask);
    return {dq, dk, dv, db};
  }
  static variable_list backward(AutogradContext*, variable_list) {
    TORCH_CHECK(false, "trifast_b200::triangle_attention_backward has no gradient formula: "
                "triangle attention can be differentiated once");
  }
};

std::tuple<Tensor, Tensor, Tensor, Tensor> grads_autograd(const Tensor& d_o, const Tensor& q,
                                                          const Tensor& k, const Tensor& v,
                                                          const Tensor& b, const Tensor& o,
                                                          const Tensor& lse, const Tensor& mask) {
  if (wants_grad({&d_o, &q, &k, &v, &b, &o, &lse})) {
    const variable_list r = Once::apply(d_o, q, k, v, b, o, lse, mask);
    return {r[0], r[1], r[2], r[3]};
  }
  static auto op = find_op<GradsSig>("trifast_b200::triangle_attention_grads");
  at::AutoDispatchBelowADInplaceOrView below;
  return op.call(d_o, q, k, v, b, o, lse, mask);
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> backward_autograd(
    const Tensor& d_o, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b,
    const Tensor& o, const Tensor& lse, const Tensor& mask) {
  if (wants_grad({&d_o, &q, &k, &v, &b, &o, &lse})) {
    const variable_list r = Once::apply(d_o, q, k, v, b, o, lse, mask);
    return {r[0], r[1], r[2], r[3], at::zeros_like(mask)};
  }
  static auto op = find_op<BackwardSig>("trifast_b200::triangle_attention_backward");
  at::AutoDispatchBelowADInplaceOrView below;
  return op.call(d_o, q, k, v, b, o, lse, mask);
}

}  // namespace

TORCH_LIBRARY(trifast_b200, m) {
  m.def("triangle_attention(Tensor q, Tensor k, Tensor v, Tensor b, Tensor mask) -> (Tensor, Tensor)",
        {at::Tag::pt2_compliant_tag});
  m.def(
      "triangle_attention_backward(Tensor do, Tensor q, Tensor k, Tensor v, Tensor b, Tensor o, "
      "Tensor l, Tensor mask) -> (Tensor, Tensor, Tensor, Tensor, Tensor)",
      {at::Tag::pt2_compliant_tag});
  // the same without the mask's zero gradient, which autograd does not need
  m.def(
      "triangle_attention_grads(Tensor do, Tensor q, Tensor k, Tensor v, Tensor b, Tensor o, "
      "Tensor l, Tensor mask) -> (Tensor, Tensor, Tensor, Tensor)",
      {at::Tag::pt2_compliant_tag});
}
TORCH_LIBRARY_IMPL(trifast_b200, CUDA, m) {
  m.impl("triangle_attention", &forward_cuda);
  m.impl("triangle_attention_backward", &backward_cuda);
  m.impl("triangle_attention_grads", &grads_cuda);
}
TORCH_LIBRARY_IMPL(trifast_b200, Autograd, m) {
  m.impl("triangle_attention", &forward_autograd);
  m.impl("triangle_attention_backward", &backward_autograd);
  m.impl("triangle_attention_grads", &grads_autograd);
}
