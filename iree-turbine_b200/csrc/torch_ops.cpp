// CUDA implementations of torch.ops.b200k.*: the whole host side of a call in native code.
//
// The schemas and the Meta implementations stay in Python (ops.py); this file registers what the
// dispatcher runs for CUDA tensors, and for `linear` and `sdpa` what it runs under autograd.
//
// Why native: a small call is bound by the host.  A decode-step GEMM or a 4-sequence decode takes
// 6 to 13 us on the device, while the Python implementation of the op (trampoline, argument
// structure, ctypes) took 17 to 22 us per call.  Here an op costs the dispatcher, one allocation from
// torch's caching allocator per output and the launch: 4 to 6 us.
//
// The kernels are reached through the C ABI (include/b200k.h) of libb200kern.so, opened on first use
// next to this file (or at $B200K_LIB), so importing the package needs neither a GPU nor the kernel
// library, and a call without the library fails loudly.
#include <dlfcn.h>

#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty_like.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/library.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <string>

#include "../../include/b200k.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using OptType = std::optional<at::ScalarType>;

// ---------------------------------------------------------------------------------------------
// the kernel library
// ---------------------------------------------------------------------------------------------
struct Api {
#define B200K_FN(name) decltype(&::name) name
  B200K_FN(b200k_abi_version);
  B200K_FN(b200k_gemm_nt);
  B200K_FN(b200k_attention_fwd);
  B200K_FN(b200k_attention_bwd_workspace_bytes);
  B200K_FN(b200k_attention_bwd);
  B200K_FN(b200k_paged_attention_fwd);
  B200K_FN(b200k_decode_workspace_bytes);
  B200K_FN(b200k_decode_attention);
  B200K_FN(b200k_paged_gather);
  B200K_FN(b200k_kv_append);
  B200K_FN(b200k_quantize_e4m3_ws);
  B200K_FN(b200k_col_sum);
#undef B200K_FN
};

std::string library_path() {
  if (const char* env = std::getenv("B200K_LIB")) return env;
  Dl_info info;
  TORCH_CHECK(dladdr(reinterpret_cast<void*>(&library_path), &info) != 0 && info.dli_fname, "b200k: dladdr failed");
  const std::string self = info.dli_fname;
  const size_t slash = self.rfind('/');
  return (slash == std::string::npos ? std::string(".") : self.substr(0, slash)) + "/libb200kern.so";
}

Api load_api() {
  const std::string path = library_path();
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(h, path, " cannot be loaded: the CUDA kernel library has not been built (", dlerror(),
              "). There is no CPU fallback.");
  Api a;
#define B200K_FN(name)                                         \
  a.name = reinterpret_cast<decltype(a.name)>(dlsym(h, #name)); \
  TORCH_CHECK(a.name, path, " does not export " #name)
  B200K_FN(b200k_abi_version);
  B200K_FN(b200k_gemm_nt);
  B200K_FN(b200k_attention_fwd);
  B200K_FN(b200k_attention_bwd_workspace_bytes);
  B200K_FN(b200k_attention_bwd);
  B200K_FN(b200k_paged_attention_fwd);
  B200K_FN(b200k_decode_workspace_bytes);
  B200K_FN(b200k_decode_attention);
  B200K_FN(b200k_paged_gather);
  B200K_FN(b200k_kv_append);
  B200K_FN(b200k_quantize_e4m3_ws);
  B200K_FN(b200k_col_sum);
#undef B200K_FN
  TORCH_CHECK(a.b200k_abi_version() == B200K_ABI_VERSION, path, ": ABI version ", a.b200k_abi_version(),
              ", this library expects ", B200K_ABI_VERSION);
  return a;
}

const Api& api() {
  static const Api a = load_api();  // a failed load throws and is tried again by the next call
  return a;
}

// Raises what the ctypes binding raises for this status (ValueError for a bad argument, B200kError
// otherwise).  Off the hot path: only the failing call takes the GIL.
void check(int status) {
  if (status == B200K_OK) return;
  pybind11::gil_scoped_acquire gil;
  pybind11::module_::import("iree_turbine_b200._launcher").attr("check")(status);
}

// ---------------------------------------------------------------------------------------------
// per-device state and small helpers
// ---------------------------------------------------------------------------------------------
constexpr int kMaxDevices = 64;

// One int32 status word per device: kernels OR a code into it when a bounded wait gives up.  Created
// on the device's first use and kept for the life of the process.
Tensor status_tensor(int64_t device) {
  static std::mutex mu;
  static Tensor* words[kMaxDevices] = {};  // never destroyed: kernels may outlive static destructors
  TORCH_CHECK(device >= 0 && device < kMaxDevices, "b200k: device ordinal ", device, " out of range");
  std::lock_guard<std::mutex> lock(mu);
  if (!words[device]) {
    // outside any dispatch mode or inference mode of the caller: this tensor outlives the call
    at::AutoDispatchBelowAutograd below;
    c10::InferenceMode plain(false);
    words[device] = new Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device)));
  }
  return *words[device];
}

int32_t* status_ptr(c10::DeviceIndex device) {
  static std::atomic<int32_t*> cached[kMaxDevices] = {};
  TORCH_CHECK(device >= 0 && device < kMaxDevices, "b200k: device ordinal ", int(device), " out of range");
  int32_t* p = cached[device].load(std::memory_order_acquire);
  if (!p) {
    p = status_tensor(device).data_ptr<int32_t>();
    cached[device].store(p, std::memory_order_release);
  }
  return p;
}

// Which attention forward kernel the ops ask for (ops.ATTENTION_KERNEL): a tuning and testing knob.
std::atomic<int32_t> g_attention_kernel{B200K_ATTN_AUTO};

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf:
      return B200K_F16;
    case at::kBFloat16:
      return B200K_BF16;
    case at::kFloat:
      return B200K_F32;
    case at::kFloat8_e4m3fn:
      return B200K_E4M3;
    default:
      TORCH_CHECK_VALUE(false, "b200k: dtype ", t, " is not supported");
  }
}

bool is_half(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }

// Every tensor argument must live on the device of the first one: the dispatcher takes this path as
// soon as one argument is a CUDA tensor, and a kernel must never get a host pointer or another GPU's.
void one_device(const char* op, at::Device dev, std::initializer_list<const Tensor*> rest) {
  for (const Tensor* t : rest)
    if (t->defined())
      TORCH_CHECK(t->device() == dev, "b200k.", op, ": all tensor arguments must be on one device, got ", dev, " and ",
                  t->device());
}

// Current device = the tensors' device for the duration of a call, and its current stream.
struct OnDevice {
  explicit OnDevice(at::Device dev) : guard(dev), index(dev.index()) {}
  void* stream() const { return c10::cuda::getCurrentCUDAStream(index).stream(); }
  c10::cuda::CUDAGuard guard;
  c10::DeviceIndex index;
};

Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, at::Device dev) {
  return Tensor(at::detail::empty_cuda(sizes, dtype, dev, std::nullopt));
}

// Scratch of one call, from torch's caching allocator on the current stream.
struct Scratch {
  Scratch(size_t bytes) : data(c10::cuda::CUDACachingAllocator::get()->allocate(bytes > 16 ? bytes : 16)) {}
  void* get() const { return data.get(); }
  c10::DataPtr data;
};

const Tensor& defined_or_none(const OptTensor& t) {
  static const Tensor none;
  return t.has_value() ? *t : none;
}

bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

// ---------------------------------------------------------------------------------------------
// GEMM
// ---------------------------------------------------------------------------------------------
at::ScalarType gemm_out_dtype(at::ScalarType in, OptType out) {
  if (is_half(in)) {
    const at::ScalarType od = out.value_or(at::kFloat);
    TORCH_CHECK(od == at::kFloat || od == in, "gemm_nt: out_dtype must be float32 or ", in);
    return od;
  }
  const at::ScalarType od = out.value_or(at::kBFloat16);
  TORCH_CHECK(od == at::kBFloat16 || od == at::kFloat, "gemm_fp8_nt: out_dtype must be bfloat16 or float32");
  return od;
}

// A 2-D view whose last dim is contiguous and whose row stride is a multiple of 16 bytes.
Tensor row_major_2d(const Tensor& t) {
  if (t.stride(1) != 1 || (t.stride(0) * t.element_size()) % 16 != 0 || !aligned16(t)) return t.contiguous();
  return t;
}

int activation_code(c10::string_view name) {
  if (name == "none") return B200K_ACT_NONE;
  if (name == "relu") return B200K_ACT_RELU;
  if (name == "gelu") return B200K_ACT_GELU;
  if (name == "silu") return B200K_ACT_SILU;
  TORCH_CHECK_VALUE(false, "unknown activation '", name, "'; expected one of ['gelu', 'none', 'relu', 'silu']");
}

// a is stored [M, K] ([K, M] with a_km), b [N, K] ([K, N] with b_kn).
Tensor run_gemm(const Tensor& a_in, const Tensor& b_in, OptType out_dtype, bool a_km, bool b_kn, const Tensor& scale_a,
                const Tensor& scale_b, const Tensor& bias_in, int activation) {
  OnDevice on(a_in.device());
  const Tensor a = row_major_2d(a_in), b = row_major_2d(b_in);
  b200k_gemm_args g = {};
  g.m = a.size(a_km ? 1 : 0);
  g.k = a.size(a_km ? 0 : 1);
  g.n = b.size(b_kn ? 1 : 0);
  TORCH_CHECK(b.size(b_kn ? 0 : 1) == g.k && a.scalar_type() == b.scalar_type(),
              "gemm: operands do not match: ", a.sizes(), " ", a.scalar_type(), " and ", b.sizes(), " ", b.scalar_type());
  Tensor out = empty({g.m, g.n}, gemm_out_dtype(a.scalar_type(), out_dtype), a.device());
  g.a = a.data_ptr();
  g.b = b.data_ptr();
  g.c = out.data_ptr();
  g.lda = a.stride(0);
  g.ldb = b.stride(0);
  g.ldc = g.n;
  g.a_km = a_km;
  g.b_kn = b_kn;
  g.in_dtype = dtype_code(a.scalar_type());
  g.out_dtype = dtype_code(out.scalar_type());
  if (scale_a.defined()) g.scale_a = static_cast<const float*>(scale_a.data_ptr());
  if (scale_b.defined()) g.scale_b = static_cast<const float*>(scale_b.data_ptr());
  g.status = status_ptr(on.index);
  g.activation = activation;
  Tensor bias;
  if (bias_in.defined()) {
    TORCH_CHECK(bias_in.numel() >= g.n, "linear_act: bias must be [N]");
    bias = bias_in.contiguous();
    g.bias = bias.data_ptr();
    g.bias_dtype = dtype_code(bias.scalar_type());
  }
  check(api().b200k_gemm_nt(&g, on.stream()));
  return out;
}

Tensor gemm_nt(const Tensor& a, const Tensor& b, OptType out_dtype) {
  one_device("gemm_nt", a.device(), {&b});
  return run_gemm(a, b, out_dtype, false, false, {}, {}, {}, B200K_ACT_NONE);
}

Tensor gemm(const Tensor& a, const Tensor& b, bool trans_a, bool trans_b, OptType out_dtype) {
  one_device("gemm", a.device(), {&b});
  return run_gemm(a, b, out_dtype, trans_a, !trans_b, {}, {}, {}, B200K_ACT_NONE);
}

Tensor linear_act(const Tensor& a, const Tensor& w, const OptTensor& bias, c10::string_view activation,
                  OptType out_dtype) {
  const Tensor& b = defined_or_none(bias);
  one_device("linear_act", a.device(), {&w, &b});
  return run_gemm(a, w, out_dtype, false, false, {}, {}, b, activation_code(activation));
}

Tensor gemm_fp8_nt(const Tensor& a, const Tensor& b, const Tensor& scale_a, const Tensor& scale_b, OptType out_dtype) {
  one_device("gemm_fp8_nt", a.device(), {&b, &scale_a, &scale_b});
  TORCH_CHECK(scale_a.numel() == 1 && scale_b.numel() == 1 && scale_a.scalar_type() == at::kFloat &&
                  scale_b.scalar_type() == at::kFloat,
              "gemm_fp8_nt: scales must be one-element float32 tensors");
  return run_gemm(a, b, out_dtype, false, false, scale_a, scale_b, {}, B200K_ACT_NONE);
}

// A [B, R, C] operand as the kernel can read it without a copy: either the last dim is contiguous or
// the middle one is (the matrix is stored transposed); otherwise a contiguous copy.
std::pair<Tensor, bool> batched_operand(const Tensor& t) {
  const int64_t es = t.element_size();
  auto ok = [es](const Tensor& x) {
    return x.stride(2) == 1 && (x.stride(1) * es) % 16 == 0 && (x.stride(0) * es) % 16 == 0 && x.stride(1) >= x.size(2) &&
           aligned16(x) && x.size(2) % 8 == 0;
  };
  if (ok(t)) return {t, false};
  Tensor tt = t.transpose(1, 2);
  if (ok(tt)) return {tt, true};
  return {t.contiguous(), false};
}

Tensor bmm(const Tensor& a, const Tensor& b, OptType out_dtype) {
  one_device("bmm", a.device(), {&b});
  OnDevice on(a.device());
  b200k_gemm_args g = {};
  g.batch = a.size(0);
  g.m = a.size(1);
  g.k = a.size(2);
  g.n = b.size(2);
  TORCH_CHECK(b.size(0) == g.batch && b.size(1) == g.k && a.scalar_type() == b.scalar_type(), "bmm: operands do not match: ",
              a.sizes(), " ", a.scalar_type(), " and ", b.sizes(), " ", b.scalar_type());
  Tensor out = empty({g.batch, g.m, g.n}, gemm_out_dtype(a.scalar_type(), out_dtype), a.device());
  if (g.batch == 0 || g.m == 0 || g.n == 0) return out;
  const auto [as, at_] = batched_operand(a);  // at_: stored [B, K, M]
  const auto [bs, bt] = batched_operand(b);   // bt: stored [B, N, K] (the kernel's native form)
  g.a = as.data_ptr();
  g.b = bs.data_ptr();
  g.c = out.data_ptr();
  g.a_km = at_;
  g.b_kn = !bt;
  g.lda = as.stride(1);
  g.ldb = bs.stride(1);
  g.ldc = g.n;
  g.a_batch_stride = as.stride(0);
  g.b_batch_stride = bs.stride(0);
  g.c_batch_stride = g.m * g.n;
  g.in_dtype = dtype_code(a.scalar_type());
  g.out_dtype = dtype_code(out.scalar_type());
  g.status = status_ptr(on.index);
  check(api().b200k_gemm_nt(&g, on.stream()));
  return out;
}

std::tuple<Tensor, Tensor> quantize_e4m3(const Tensor& x_in) {
  OnDevice on(x_in.device());
  TORCH_CHECK(x_in.scalar_type() == at::kFloat, "quantize_e4m3: x must be float32");
  const Tensor x = x_in.contiguous();
  Tensor y = empty(x.sizes(), at::kFloat8_e4m3fn, x.device());
  Tensor scale = empty({1}, at::kFloat, x.device());
  Scratch ws(B200K_QUANTIZE_WORKSPACE_BYTES);
  check(api().b200k_quantize_e4m3_ws(static_cast<const float*>(x.data_ptr()), y.data_ptr(),
                                     static_cast<float*>(scale.data_ptr()), ws.get(), B200K_QUANTIZE_WORKSPACE_BYTES,
                                     x.numel(), on.stream()));
  return {y, scale};
}

Tensor col_sum(const Tensor& x) {
  OnDevice on(x.device());
  TORCH_CHECK(x.dim() == 2 && is_half(x.scalar_type()), "col_sum: x must be a float16 or bfloat16 matrix");
  if (x.stride(1) != 1 || x.size(0) == 0 || x.size(1) % 8 != 0 || x.stride(0) % 8 != 0 || !aligned16(x))
    return x.to(at::kFloat).sum(0).to(x.scalar_type());  // rows that 16-byte loads cannot cover
  Tensor out = empty({x.size(1)}, x.scalar_type(), x.device());
  check(api().b200k_col_sum(x.data_ptr(), out.data_ptr(), x.size(0), x.size(1), x.stride(0), dtype_code(x.scalar_type()),
                            on.stream()));
  return out;
}

// ---------------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------------
Tensor bhsd(const Tensor& t) {
  TORCH_CHECK(t.dim() == 4, "attention: tensors must be 4-D [B,H,S,D]");
  const auto s = t.strides();
  const bool ok =
      s[3] == 1 && s[0] > 0 && s[1] > 0 && s[2] > 0 && ((s[0] | s[1] | s[2]) & 7) == 0 && aligned16(t);
  return ok ? t : t.contiguous();
}

// The output takes q's memory layout when q's rows are contiguous (as aten's operator does).
Tensor attention_out_like(const Tensor& q) {
  if (q.is_contiguous() || q.dim() != 4 || q.stride(-1) != 1) return empty(q.sizes(), q.scalar_type(), q.device());
  return at::empty_like(q);
}

template <typename Args>
void set_kernel_and_status(Args& a, c10::DeviceIndex dev) {
  a.kernel = a.head_dim == 128 ? g_attention_kernel.load(std::memory_order_relaxed) : B200K_ATTN_AUTO;
  a.status = status_ptr(dev);
}

void check_attention(const Tensor& q, const Tensor& k, const Tensor& v) {
  TORCH_CHECK(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(),
              "attention: q, k, v must share a dtype");
  TORCH_CHECK(k.sizes() == v.sizes(), "attention: k and v must have the same shape");
  TORCH_CHECK(q.size(0) <= k.size(0) && q.size(3) == k.size(3), "attention: q and k do not match");
}

Tensor run_attention(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, double scale, bool causal, float* lse,
                     const OnDevice& on) {
  const Tensor q = bhsd(q_in), k = bhsd(k_in), v = bhsd(v_in);
  check_attention(q, k, v);
  Tensor o = attention_out_like(q_in);
  b200k_attention_args a = {};
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.o = o.data_ptr();
  a.batch = q.size(0);
  a.q_heads = q.size(1);
  a.seq_q = q.size(2);
  a.head_dim = q.size(3);
  a.kv_heads = k.size(1);
  a.seq_kv = k.size(2);
#define B200K_STRIDES(name, t)      \
  a.name##_stride_b = (t).stride(0); \
  a.name##_stride_h = (t).stride(1); \
  a.name##_stride_s = (t).stride(2)
  B200K_STRIDES(q, q);
  B200K_STRIDES(k, k);
  B200K_STRIDES(v, v);
  B200K_STRIDES(o, o);
  a.dtype = dtype_code(q.scalar_type());
  a.causal = causal;
  a.scale = static_cast<float>(scale);
  a.lse = lse;
  set_kernel_and_status(a, on.index);
  check(api().b200k_attention_fwd(&a, on.stream()));
  return o;
}

Tensor attention(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool causal) {
  one_device("attention", q.device(), {&k, &v});
  OnDevice on(q.device());
  return run_attention(q, k, v, scale, causal, nullptr, on);
}

std::tuple<Tensor, Tensor> attention_lse(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool causal) {
  one_device("attention_lse", q.device(), {&k, &v});
  OnDevice on(q.device());
  Tensor lse = empty(q.sizes().slice(0, 3), at::kFloat, q.device());
  Tensor o = run_attention(q, k, v, scale, causal, static_cast<float*>(lse.data_ptr()), on);
  return {o, lse};
}

std::tuple<Tensor, Tensor, Tensor> attention_bwd(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in,
                                                 const Tensor& o_in, const Tensor& do_in, double scale, bool causal,
                                                 const OptTensor& lse_in) {
  Tensor lse = defined_or_none(lse_in);
  one_device("attention_bwd", q_in.device(), {&k_in, &v_in, &o_in, &do_in, &lse});
  OnDevice on(q_in.device());
  if (lse.defined())
    TORCH_CHECK(lse.scalar_type() == at::kFloat && lse.sizes() == q_in.sizes().slice(0, 3),
                "attention_bwd: lse must be float32 [B, Hq, Sq]");
  for (const Tensor* t : {&q_in, &k_in, &v_in, &o_in, &do_in}) {
    TORCH_CHECK(t->dim() == 4 && (t->size(3) == 64 || t->size(3) == 128) && t->size(3) == q_in.size(3),
                "attention_bwd: tensors must be [B,H,S,D] with D = 128 or 64, the same for all");
    TORCH_CHECK(t->scalar_type() == q_in.scalar_type(), "attention_bwd: all tensors must share a dtype");
  }
  TORCH_CHECK(is_half(q_in.scalar_type()), "attention_bwd: dtype must be float16 or bfloat16, got ", q_in.scalar_type());
  TORCH_CHECK(k_in.sizes() == v_in.sizes(), "attention_bwd: k and v must have the same shape");
  TORCH_CHECK(o_in.sizes() == q_in.sizes() && do_in.sizes() == q_in.sizes(),
              "attention_bwd: o and d_o must have q's shape");
  TORCH_CHECK(q_in.size(0) == k_in.size(0), "attention_bwd: batch mismatch");
  TORCH_CHECK(k_in.size(1) > 0 && q_in.size(1) % k_in.size(1) == 0,
              "attention_bwd: query heads must be a multiple of kv heads");
  if (lse.defined()) lse = lse.contiguous();
  const Tensor q = bhsd(q_in), k = bhsd(k_in), v = bhsd(v_in), o = bhsd(o_in), d_o = bhsd(do_in);
  Tensor d_q = empty(q.sizes(), q.scalar_type(), q.device());
  Tensor d_k = empty(k.sizes(), q.scalar_type(), q.device());
  Tensor d_v = empty(v.sizes(), q.scalar_type(), q.device());
  b200k_attention_bwd_args a = {};
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.o = o.data_ptr();
  a.d_o = d_o.data_ptr();
  a.d_q = d_q.data_ptr();
  a.d_k = d_k.data_ptr();
  a.d_v = d_v.data_ptr();
  B200K_STRIDES(q, q);
  B200K_STRIDES(k, k);
  B200K_STRIDES(v, v);
  B200K_STRIDES(o, o);
  B200K_STRIDES(do, d_o);
  B200K_STRIDES(dq, d_q);
  B200K_STRIDES(dk, d_k);
  B200K_STRIDES(dv, d_v);
#undef B200K_STRIDES
  a.batch = q.size(0);
  a.q_heads = q.size(1);
  a.seq_q = q.size(2);
  a.head_dim = q.size(3);
  a.kv_heads = k.size(1);
  a.seq_kv = k.size(2);
  a.dtype = dtype_code(q.scalar_type());
  a.causal = causal;
  a.scale = static_cast<float>(scale);
  a.status = status_ptr(on.index);
  a.lse = lse.defined() ? static_cast<const float*>(lse.data_ptr()) : nullptr;
  a.workspace_bytes = std::max<uint64_t>(api().b200k_attention_bwd_workspace_bytes(&a), 16);
  Scratch ws(a.workspace_bytes);
  a.workspace = ws.get();
  check(api().b200k_attention_bwd(&a, on.stream()));
  return {d_q, d_k, d_v};
}

// ---------------------------------------------------------------------------------------------
// decode and the paged cache
// ---------------------------------------------------------------------------------------------
void launch_decode(b200k_decode_args& a, const OnDevice& on) {
  a.status = status_ptr(on.index);
  a.workspace_bytes = api().b200k_decode_workspace_bytes(&a);
  Scratch ws(a.workspace_bytes);
  a.workspace = ws.get();
  check(api().b200k_decode_attention(&a, on.stream()));
}

// Block tables, lengths and positions are read by the kernels as int32 with one row (entry) per sequence; a table of
// int64, torch's own default, would be taken apart into low and high words.  Those kept for more sequences than
// the call has are fine: the first ones are used.
void check_table(const char* op, const Tensor& t, int64_t sequences) {
  TORCH_CHECK(t.scalar_type() == at::kInt && t.dim() == 2 && t.size(0) >= sequences, op,
              ": block_table must be int32 [num_seqs, max_pages] for ", sequences, " sequences, got ", t.scalar_type(), " ",
              t.sizes());
}

void check_per_sequence(const char* op, const char* name, const Tensor& t, int64_t sequences) {
  const auto sizes = t.sizes();
  const bool vector = std::count_if(sizes.begin(), sizes.end(), [](int64_t n) { return n != 1; }) <= 1;
  TORCH_CHECK(t.scalar_type() == at::kInt && vector && t.numel() >= sequences, op, ": ", name,
              " must be int32 [num_seqs] for ", sequences, " sequences, got ", t.scalar_type(), " ", sizes);
}

void check_decode(const char* op, const Tensor& q, const Tensor& kc, const Tensor& vc, const Tensor& lens) {
  TORCH_CHECK(q.dim() == 3 && kc.dim() == 4, op, ": q must be 3-D and the K/V caches 4-D");
  TORCH_CHECK(q.scalar_type() == kc.scalar_type() && q.scalar_type() == vc.scalar_type(), op,
              ": q and the KV cache must share a dtype");
  TORCH_CHECK(kc.sizes() == vc.sizes() && kc.size(3) == q.size(2), op, ": cache shapes do not match");
  check_per_sequence(op, "seq_lens", lens, q.size(0));
}

Tensor decode_attention(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& lens_in, double scale,
                        int64_t chunk_tokens) {
  one_device("decode_attention", q_in.device(), {&k_in, &v_in, &lens_in});
  OnDevice on(q_in.device());
  check_decode("decode_attention", q_in, k_in, v_in, lens_in);
  TORCH_CHECK(k_in.size(0) >= q_in.size(0), "decode_attention: k must have one history per sequence");
  const Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous(), lens = lens_in.contiguous();
  Tensor o = empty(q.sizes(), q.scalar_type(), q.device());
  b200k_decode_args a = {};
  a.q = q.data_ptr();
  a.k_cache = k.data_ptr();
  a.v_cache = v.data_ptr();
  a.o = o.data_ptr();
  a.seq_lens = static_cast<const int32_t*>(lens.data_ptr());
  a.num_seqs = q.size(0);
  a.q_heads = q.size(1);
  a.head_dim = q.size(2);
  a.kv_heads = k.size(1);
  a.max_seq_len = k.size(2);
  a.kv_batch_stride = k.stride(0);
  a.kv_head_stride = k.stride(1);
  a.dtype = dtype_code(q.scalar_type());
  a.chunk_tokens = static_cast<int32_t>(chunk_tokens);
  a.scale = static_cast<float>(scale);
  launch_decode(a, on);
  return o;
}

Tensor paged_decode_attention(const Tensor& q_in, const Tensor& kc_in, const Tensor& vc_in, const Tensor& bt_in,
                              const Tensor& lens_in, double scale, int64_t chunk_tokens) {
  one_device("paged_decode_attention", q_in.device(), {&kc_in, &vc_in, &bt_in, &lens_in});
  OnDevice on(q_in.device());
  check_decode("paged_decode_attention", q_in, kc_in, vc_in, lens_in);
  check_table("paged_decode_attention", bt_in, q_in.size(0));
  const Tensor q = q_in.contiguous(), kc = kc_in.contiguous(), vc = vc_in.contiguous(), bt = bt_in.contiguous(),
               lens = lens_in.contiguous();
  Tensor o = empty(q.sizes(), q.scalar_type(), q.device());
  b200k_decode_args a = {};
  a.q = q.data_ptr();
  a.k_cache = kc.data_ptr();
  a.v_cache = vc.data_ptr();
  a.o = o.data_ptr();
  a.block_table = static_cast<const int32_t*>(bt.data_ptr());
  a.seq_lens = static_cast<const int32_t*>(lens.data_ptr());
  a.num_seqs = q.size(0);
  a.q_heads = q.size(1);
  a.head_dim = q.size(2);
  a.kv_heads = kc.size(1);
  a.page_size = kc.size(2);
  a.num_pages = kc.size(0);
  a.block_table_stride = bt.stride(0);
  a.max_seq_len = bt.size(1) * kc.size(2);
  a.kv_page_stride = kc.stride(0);
  a.kv_head_stride = kc.stride(1);
  a.dtype = dtype_code(q.scalar_type());
  a.chunk_tokens = static_cast<int32_t>(chunk_tokens);
  a.scale = static_cast<float>(scale);
  launch_decode(a, on);
  return o;
}

Tensor paged_gather(const Tensor& cache_in, const Tensor& bt_in, const Tensor& lens_in, int64_t max_seq_len) {
  one_device("paged_gather", cache_in.device(), {&bt_in, &lens_in});
  OnDevice on(cache_in.device());
  TORCH_CHECK(cache_in.dim() == 4, "paged_gather: cache must be [num_pages, heads, page_size, head_dim]");
  check_table("paged_gather", bt_in, 0);
  check_per_sequence("paged_gather", "seq_lens", lens_in, bt_in.size(0));
  const Tensor cache = cache_in.contiguous(), bt = bt_in.contiguous(), lens = lens_in.contiguous();
  Tensor out = at::zeros({bt.size(0), cache.size(1), max_seq_len, cache.size(3)}, cache.options());
  check(api().b200k_paged_gather(cache.data_ptr(), static_cast<const int32_t*>(bt.data_ptr()),
                                 static_cast<const int32_t*>(lens.data_ptr()), out.data_ptr(), bt.size(0), cache.size(1),
                                 cache.size(3), cache.size(2), cache.size(0), bt.stride(0), max_seq_len, cache.stride(0),
                                 cache.stride(1), cache.element_size(), on.stream()));
  return out;
}

void kv_append(const Tensor& kn_in, const Tensor& vn_in, Tensor kc, Tensor vc, const Tensor& bt_in,
               const Tensor& pos_in) {
  one_device("kv_append", kn_in.device(), {&vn_in, &kc, &vc, &bt_in, &pos_in});
  OnDevice on(kn_in.device());
  TORCH_CHECK_VALUE(kc.is_contiguous() && vc.is_contiguous(),
                    "kv_append: the caches are written in place and must be contiguous");
  TORCH_CHECK(kn_in.dim() == 4 && kn_in.sizes() == vn_in.sizes() && kc.dim() == 4 && kc.sizes() == vc.sizes() &&
                  kn_in.size(2) == kc.size(1) && kn_in.size(3) == kc.size(3) && kn_in.scalar_type() == kc.scalar_type() &&
                  vn_in.scalar_type() == kc.scalar_type() && vc.scalar_type() == kc.scalar_type(),
              "kv_append: heads, head_dim and dtypes of new rows and caches must match");
  check_table("kv_append", bt_in, kn_in.size(0));
  check_per_sequence("kv_append", "positions", pos_in, kn_in.size(0));
  const Tensor kn = kn_in.contiguous(), vn = vn_in.contiguous(), bt = bt_in.contiguous(), pos = pos_in.contiguous();
  check(api().b200k_kv_append(kn.data_ptr(), vn.data_ptr(), kc.data_ptr(), vc.data_ptr(),
                              static_cast<const int32_t*>(bt.data_ptr()), static_cast<const int32_t*>(pos.data_ptr()),
                              kn.size(0), kn.size(1), kn.size(2), kn.size(3), kc.size(2), kc.size(0), bt.stride(0),
                              kc.stride(0), kc.stride(1), kc.element_size(), status_ptr(on.index), on.stream()));
}

Tensor paged_attention(const Tensor& q_in, const Tensor& kc_in, const Tensor& vc_in, const Tensor& bt_in,
                       const Tensor& lens_in, double scale, bool causal) {
  one_device("paged_attention", q_in.device(), {&kc_in, &vc_in, &bt_in, &lens_in});
  OnDevice on(q_in.device());
  const Tensor q = bhsd(q_in);
  TORCH_CHECK(kc_in.dim() == 4 && kc_in.sizes() == vc_in.sizes() && kc_in.size(3) == q.size(3) &&
                  kc_in.scalar_type() == q.scalar_type() && vc_in.scalar_type() == q.scalar_type(),
              "paged_attention: caches do not match q");
  check_table("paged_attention", bt_in, q.size(0));
  check_per_sequence("paged_attention", "seq_lens", lens_in, q.size(0));
  const Tensor kc = kc_in.contiguous(), vc = vc_in.contiguous(), bt = bt_in.contiguous(), lens = lens_in.contiguous();
  Tensor o = attention_out_like(q_in);
  b200k_paged_attention_args a = {};
  a.q = q.data_ptr();
  a.k_cache = kc.data_ptr();
  a.v_cache = vc.data_ptr();
  a.o = o.data_ptr();
  a.block_table = static_cast<const int32_t*>(bt.data_ptr());
  a.seq_lens = static_cast<const int32_t*>(lens.data_ptr());
  a.batch = q.size(0);
  a.q_heads = q.size(1);
  a.kv_heads = kc.size(1);
  a.seq_q = q.size(2);
  a.page_size = kc.size(2);
  a.num_pages = kc.size(0);
  a.block_table_stride = bt.stride(0);
  a.max_seq_kv = bt.size(1) * kc.size(2);
  a.head_dim = q.size(3);
  a.q_stride_b = q.stride(0);
  a.q_stride_h = q.stride(1);
  a.q_stride_s = q.stride(2);
  a.o_stride_b = o.stride(0);
  a.o_stride_h = o.stride(1);
  a.o_stride_s = o.stride(2);
  a.kv_page_stride = kc.stride(0);
  a.kv_head_stride = kc.stride(1);
  a.dtype = dtype_code(q.scalar_type());
  a.causal = causal;
  a.scale = static_cast<float>(scale);
  set_kernel_and_status(a, on.index);
  check(api().b200k_paged_attention_fwd(&a, on.stream()));
  return o;
}

// ---------------------------------------------------------------------------------------------
// autograd: the differentiable ops call the ops above through the dispatcher, so a fake or traced
// tensor takes its own path.
// ---------------------------------------------------------------------------------------------
template <typename Fn>
auto typed_op(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Fn>();
}

Tensor call_linear_act(const Tensor& x, const Tensor& w, const OptTensor& bias) {
  static const auto op =
      typed_op<Tensor(const Tensor&, const Tensor&, const OptTensor&, c10::string_view, OptType)>("b200k::linear_act");
  return op.call(x, w, bias, "none", x.scalar_type());
}

Tensor call_gemm(const Tensor& a, const Tensor& b, bool ta, bool tb, at::ScalarType out) {
  static const auto op = typed_op<Tensor(const Tensor&, const Tensor&, bool, bool, OptType)>("b200k::gemm");
  return op.call(a, b, ta, tb, out);
}

Tensor call_col_sum(const Tensor& x) {
  static const auto op = typed_op<Tensor(const Tensor&)>("b200k::col_sum");
  return op.call(x);
}

struct LinearFunction : torch::autograd::Function<LinearFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& bias) {
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->save_for_backward({x, w});
    ctx->saved_data["bias"] = bias.has_value() && bias->defined();
    return call_linear_act(x, w, bias);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    const Tensor dy = grads[0].contiguous();
    Tensor dx, dw, db;
    if (ctx->needs_input_grad(0)) dx = call_gemm(dy, w, false, false, x.scalar_type());  // [M, N] @ [N, K]
    if (ctx->needs_input_grad(1)) dw = call_gemm(dy, x, true, false, w.scalar_type());   // [M, N]^T @ [M, K]
    // an absent bias is not among the inputs that needs_input_grad counts
    if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2)) {
      // col_sum has no derivative: where this sum is differentiated itself, torch's operators compute it
      const bool differentiated = (at::GradMode::is_enabled() && dy.requires_grad()) || dy._fw_grad(0).defined();
      db = differentiated ? dy.to(at::kFloat).sum(0).to(dy.scalar_type()) : call_col_sum(dy);
    }
    return {dx, dw, db};
  }
};

Tensor linear_autograd(const Tensor& x, const Tensor& w, const OptTensor& bias) {
  return LinearFunction::apply(x, w, bias);
}

std::tuple<Tensor, Tensor> call_attention_lse(const Tensor& q, const Tensor& k, const Tensor& v, double scale,
                                              bool causal) {
  static const auto op =
      typed_op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, double, bool)>(
          "b200k::attention_lse");
  return op.call(q, k, v, scale, causal);
}

struct SdpaFunction : torch::autograd::Function<SdpaFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                        double scale, bool causal) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [o, lse] = call_attention_lse(q, k, v, scale, causal);
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["causal"] = causal;
    return o;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    static const auto op =
        typed_op<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                                    const Tensor&, double, bool, const OptTensor&)>(
            "b200k::attention_bwd");
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dv] = op.call(s[0], s[1], s[2], s[3], grads[0], ctx->saved_data["scale"].toDouble(),
                                ctx->saved_data["causal"].toBool(), s[4]);
    return {dq, dk, dv, Tensor(), Tensor()};
  }
};

Tensor sdpa_autograd(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool causal) {
  return SdpaFunction::apply(q, k, v, scale, causal);
}

Tensor linear_cuda(const Tensor& x, const Tensor& w, const OptTensor& bias) { return call_linear_act(x, w, bias); }

Tensor sdpa_cuda(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool causal) {
  return attention(q, k, v, scale, causal);
}

TORCH_LIBRARY_IMPL(b200k, CUDA, m) {
  m.impl("gemm_nt", gemm_nt);
  m.impl("gemm", gemm);
  m.impl("bmm", bmm);
  m.impl("linear_act", linear_act);
  m.impl("linear", linear_cuda);
  m.impl("gemm_fp8_nt", gemm_fp8_nt);
  m.impl("quantize_e4m3", quantize_e4m3);
  m.impl("col_sum", col_sum);
  m.impl("attention", attention);
  m.impl("attention_lse", attention_lse);
  m.impl("attention_bwd", attention_bwd);
  m.impl("sdpa", sdpa_cuda);
  m.impl("decode_attention", decode_attention);
  m.impl("paged_decode_attention", paged_decode_attention);
  m.impl("paged_gather", paged_gather);
  m.impl("kv_append", kv_append);
  m.impl("paged_attention", paged_attention);
}

TORCH_LIBRARY_IMPL(b200k, Autograd, m) {
  m.impl("linear", linear_autograd);
  m.impl("sdpa", sdpa_autograd);
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  m.def("status_word", &status_tensor, "The device's status word (an int32 tensor of one element).");
  m.def("attention_kernel", [] { return g_attention_kernel.load(std::memory_order_relaxed); });
  m.def("set_attention_kernel", [](int32_t k) { g_attention_kernel.store(k, std::memory_order_relaxed); });
}
