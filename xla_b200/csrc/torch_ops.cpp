// The operators' CUDA kernels: argument checks, output allocation and one call into the C ABI (include/qmm_b200.h).
//
// A decode linear runs for 3 to 15 us on the GPU; the same steps in Python (dispatcher re-entry, validation, ctypes
// marshalling) took 17 to 19 us per call and bounded every small call.  Only well-formed calls are handled here.
// Anything else (a shape or dtype the validators reject, a strided operand, the N-minor blockwise layout) goes to the
// Python form of the operator registered beside each one ("..._any"), which raises the reference's errors or converts.
//
// Semantics: torch_xla/experimental/xla_quantized_matmul.py:76-183, torch_xla/experimental/custom_kernel.py:1066-1106.
#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/library.h>

#include <list>
#include <mutex>

#include "../../include/qmm_b200.h"

namespace {

using at::Tensor;
using std::optional;

// Per-thread settings (xla_b200.force_variant, xla_b200.set_activation_saturation).
thread_local int tl_variant = QMM_VARIANT_AUTO;
thread_local int tl_saturate = 1;

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return QMM_F32;
    case at::kBFloat16: return QMM_BF16;
    case at::kHalf: return QMM_F16;
    default: return -1;
  }
}

// ---- scratch ----------------------------------------------------------------------------------------------------------
// One buffer per (device, stream), zero-filled when created (the kernels keep its flag words zero) and grown on demand.
// The buffers come from torch's allocator on their own stream, so giving one back is ordered with the work that used
// it.  At most kMaxBuffers are kept, the least recently used goes first; a buffer that a stream capture has seen is
// kept for good, because the captured graph holds its address.  A capture never allocates: it gets the stream's buffer
// or none.  `lock` is held while the kernels that share a buffer are enqueued, so that two threads on one stream
// cannot interleave theirs.
constexpr size_t kMaxBuffers = 64;
struct Scratch {
  int device;
  cudaStream_t stream;
  Tensor buf;
  bool captured = false;
};
std::mutex g_scratch_lock;
std::list<Scratch> g_scratch;       // most recently used first
std::list<Tensor> g_captured;       // outgrown buffers whose address a graph may hold

void scratch(int device, cudaStream_t stream, size_t need, void** ptr, size_t* bytes) {
  *ptr = nullptr;
  *bytes = 0;
  if (need == 0) return;
  auto it = g_scratch.begin();
  while (it != g_scratch.end() && !(it->device == device && it->stream == stream)) ++it;
  if (it == g_scratch.end() || (size_t)it->buf.numel() < need) {
    const bool capturing = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
    if (capturing && it == g_scratch.end()) return;
    if (!capturing) {
      size_t size = std::max<size_t>(need, 16u << 20);
      if (it == g_scratch.end()) {
        if (g_scratch.size() >= kMaxBuffers) {
          if (g_scratch.back().captured) g_captured.push_back(g_scratch.back().buf);
          g_scratch.pop_back();
        }
        g_scratch.push_front(Scratch{device, stream, Tensor()});
        it = g_scratch.begin();
      } else {
        size = std::max<size_t>(need, 2 * (size_t)it->buf.numel());
        if (it->captured) g_captured.push_back(it->buf);
        it->captured = false;
      }
      it->buf = at::zeros({(int64_t)size}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
    } else {
      it->captured = true;
    }
  } else if (!it->captured && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
    it->captured = true;
  }
  if (it != g_scratch.begin()) g_scratch.splice(g_scratch.begin(), g_scratch, it);
  *ptr = g_scratch.front().buf.data_ptr();
  *bytes = (size_t)g_scratch.front().buf.numel();
}

// ---- helpers ----------------------------------------------------------------------------------------------------------
bool on(const Tensor& t, const at::Device& d) { return t.is_cuda() && t.device() == d; }
bool on(const optional<Tensor>& t, const at::Device& d) { return !t.has_value() || on(*t, d); }

// `t` as the contiguous fp32 tensor the kernels read, without a copy where it is one
Tensor as_f32(const Tensor& t) { return t.scalar_type() == at::kFloat ? t.contiguous() : t.to(at::kFloat).contiguous(); }

at::ScalarType promote(const Tensor& x, const Tensor& scale, const optional<Tensor>& zp) {
  at::ScalarType dt = c10::promoteTypes(x.scalar_type(), scale.scalar_type());
  return zp.has_value() ? c10::promoteTypes(dt, zp->scalar_type()) : dt;
}

Tensor output(const Tensor& x, int64_t N, at::ScalarType dt) {
  if (x.dim() == 2) return at::empty({x.size(0), N}, x.options().dtype(dt));
  auto shape = x.sizes().vec();
  shape.back() = N;
  return at::empty(shape, x.options().dtype(dt));
}

// The few shapes whose zero points are applied after the kernel (in the Python form).
bool zero_point_outside(const Tensor& x, int64_t N, int wbits, int64_t block, const optional<Tensor>& zp) {
  return zp.has_value() && tl_variant == QMM_VARIANT_AUTO && x.scalar_type() != at::kFloat &&
         !qmm_zero_point_in_kernel(wbits, x.numel() / x.size(-1), N, x.size(-1), block, dtype_code(x.scalar_type()));
}

struct Call {
  const Tensor& x;
  const Tensor& w;
  Tensor scale, zp;
  int wbits;
  int64_t M, N, K, block;  // block 0: per channel

  // Scales (and zero points) in the one type that the kernels read besides fp32, or fp32
  void scales_to_f32() {
    scale = as_f32(scale);
    if (zp.defined()) zp = as_f32(zp);
  }
  bool scales_f32() const { return scale.scalar_type() == at::kFloat; }
  const void* zp_ptr() const { return zp.defined() ? zp.data_ptr() : nullptr; }
};

// Scales in 16 bits go to the kernel as they are; where the one that this shape takes reads fp32 only, they are converted.
template <typename F>
bool with_scales(Call& c, F run) {
  int rc = run();
  if (rc == QMM_ERR_UNSUPPORTED && !c.scales_f32()) {
    c.scales_to_f32();
    rc = run();
  }
  return rc == QMM_OK;
}

// Runs one linear; false when the library refused it (the Python form repeats the call and raises its error).
bool weight_only(Call& c, Tensor& out) {
  const int dev = c.x.get_device();
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev).stream();
  std::lock_guard<std::mutex> hold(g_scratch_lock);
  void* ws;
  size_t ws_bytes;
  scratch(dev, st, qmm_weight_only_workspace_size_for(c.wbits, c.M, c.N, c.K), &ws, &ws_bytes);
  return with_scales(c, [&] {
    return qmm_weight_only_typed(c.wbits, c.x.data_ptr(), dtype_code(c.x.scalar_type()), c.w.data_ptr(), c.scale.data_ptr(), c.zp_ptr(),
                                 dtype_code(c.scale.scalar_type()), out.data_ptr(), dtype_code(out.scalar_type()), c.M, c.N, c.K,
                                 c.block, tl_variant, ws, ws_bytes, st);
  });
}

bool w8a8(Call& c, Tensor& out) {
  const int dev = c.x.get_device();
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev).stream();
  std::lock_guard<std::mutex> hold(g_scratch_lock);
  constexpr size_t kFlags = 2048;  // the other kernels' flag words stay zero
  const size_t need = qmm_workspace_size(QMM_OP_W8A8_PERCHANNEL, c.M, c.N, c.K);
  void* ws;
  size_t ws_bytes;
  scratch(dev, st, need + kFlags, &ws, &ws_bytes);
  Tensor own;  // a stream capture that began before the stream had scratch (or enough of it)
  if (ws_bytes < need + kFlags) {
    own = at::empty({(int64_t)need}, c.x.options().dtype(at::kByte));
    ws = own.data_ptr();
  } else {
    ws = static_cast<uint8_t*>(ws) + kFlags;
  }
  return with_scales(c, [&] {
    return qmm_w8a8_perchannel_typed(c.x.data_ptr(), dtype_code(c.x.scalar_type()), (const int8_t*)c.w.data_ptr(), c.scale.data_ptr(),
                                     c.zp_ptr(), dtype_code(c.scale.scalar_type()), out.data_ptr(), dtype_code(out.scalar_type()), c.M,
                                     c.N, c.K, tl_saturate, tl_variant, ws, need, st);
  });
}

// The shapes and layouts the kernels take as they are: contiguous activations, a contiguous K-minor weight, scales (and
// zero points) of its row count, or of K / block rows of it.
bool plain(const Tensor& x, const Tensor& w, const Tensor& scale, const optional<Tensor>& zp, int64_t block, bool packed) {
  if (x.dim() < 1 || w.dim() != 2 || x.numel() == 0 || w.numel() == 0) return false;
  if (dtype_code(x.scalar_type()) < 0 || !x.is_contiguous() || !w.is_contiguous()) return false;
  if (w.scalar_type() != (packed ? at::kByte : at::kChar)) return false;
  const int64_t N = w.size(0), K = x.size(-1);
  if (w.size(1) * (packed ? 2 : 1) != K) return false;
  if (block != -1 && (block <= 0 || K % block != 0)) return false;
  auto fits = [&](const Tensor& t) {
    if (!t.is_floating_point()) return false;
    return block == -1 ? t.dim() == 1 && t.size(0) == N : t.dim() == 2 && t.size(0) == K / block && t.size(1) == N;
  };
  const at::Device d = x.device();
  return on(w, d) && on(scale, d) && on(zp, d) && fits(scale) && (!zp.has_value() || fits(*zp));
}

Call make_call(const Tensor& x, const Tensor& w, const Tensor& scale, const optional<Tensor>& zp, int64_t block, bool packed) {
  const int64_t K = x.size(-1);
  Call c{x, w, scale, zp.has_value() ? *zp : Tensor(), packed ? 4 : 8, x.numel() / K, w.size(0), K, block == -1 ? 0 : block};
  const bool as_they_are = dtype_code(scale.scalar_type()) >= 0 && scale.is_contiguous() &&
                           (!zp.has_value() || (zp->scalar_type() == scale.scalar_type() && zp->is_contiguous()));
  if (!as_they_are) c.scales_to_f32();
  return c;
}

template <typename Sig, typename... A>
Tensor python_form(const char* name, A&&... args) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>().call(std::forward<A>(args)...);
}

// ---- the operators ----------------------------------------------------------------------------------------------------
Tensor quantized_matmul(const Tensor& x, const Tensor& w, const Tensor& scale, const optional<Tensor>& zp, optional<int64_t> block_size,
                        optional<bool> int4_weight, optional<bool> quantize_activation) {
  if (block_size.value_or(-1) == -1 && plain(x, w, scale, zp, -1, false)) {
    c10::cuda::OptionalCUDAGuard guard(x.device());
    const bool qact = quantize_activation.value_or(false);
    const at::ScalarType dt = promote(x, scale, zp);
    if (dtype_code(dt) >= 0 && (qact || !zero_point_outside(x, w.size(0), 8, -1, zp))) {
      Call c = make_call(x, w, scale, zp, -1, false);
      Tensor out = output(x, c.N, dt);
      if (qact ? w8a8(c, out) : weight_only(c, out)) return out;
    }
  }
  return python_form<decltype(quantized_matmul)>("xla_b200::quantized_matmul_any", x, w, scale, zp, block_size, int4_weight,
                                                 quantize_activation);
}

Tensor quantized_matmul_int8(const Tensor& x, const Tensor& w, const Tensor& scalar, const optional<Tensor>& zp,
                             const optional<Tensor>& quant_block_size, bool quantize_activation, optional<int64_t> batch_block_size,
                             optional<int64_t> out_block_size, optional<int64_t> in_block_size) {
  if (!zp.has_value() && !quant_block_size.has_value() && x.dim() == 2 && plain(x, w, scalar, zp, -1, false)) {
    c10::cuda::OptionalCUDAGuard guard(x.device());
    Call c = make_call(x, w, scalar, zp, -1, false);
    Tensor out = output(x, c.N, x.scalar_type());
    if (quantize_activation ? w8a8(c, out) : weight_only(c, out)) return out;
  }
  return python_form<decltype(quantized_matmul_int8)>("xla_b200::quantized_matmul_int8_any", x, w, scalar, zp, quant_block_size,
                                                      quantize_activation, batch_block_size, out_block_size, in_block_size);
}

Tensor quantized_matmul_packed(const Tensor& x, const Tensor& w, const Tensor& scale, const optional<Tensor>& zp, int64_t block_size,
                               bool int4_weight, bool weight_is_packed, bool quantize_activation, optional<at::ScalarType> out_dtype) {
  if (!(quantize_activation && (weight_is_packed || block_size != -1)) && plain(x, w, scale, zp, block_size, weight_is_packed)) {
    c10::cuda::OptionalCUDAGuard guard(x.device());
    const at::ScalarType dt = out_dtype.has_value() ? *out_dtype : promote(x, scale, zp);
    if (dtype_code(dt) >= 0 && (quantize_activation || !zero_point_outside(x, w.size(0), weight_is_packed ? 4 : 8, block_size, zp))) {
      Call c = make_call(x, w, scale, zp, block_size, weight_is_packed);
      Tensor out = output(x, c.N, dt);
      if (quantize_activation ? w8a8(c, out) : weight_only(c, out)) return out;
    }
  }
  return python_form<decltype(quantized_matmul_packed)>("xla_b200::quantized_matmul_packed_any", x, w, scale, zp, block_size, int4_weight,
                                                        weight_is_packed, quantize_activation, out_dtype);
}

Tensor quantized_gate_up(const Tensor& x, const Tensor& w, const Tensor& scale, int64_t block_size, bool int4_weight,
                         bool weight_is_packed, optional<at::ScalarType> out_dtype) {
  if (plain(x, w, scale, {}, block_size, weight_is_packed) && w.size(0) % 16 == 0) {
    const int64_t K = x.size(-1), M = x.numel() / K;
    const int wbits = weight_is_packed ? 4 : 8;
    const bool half = x.scalar_type() != at::kFloat;
    const at::ScalarType dt = out_dtype.has_value() ? *out_dtype : promote(x, scale, {});
    const bool tc = M > 32 || (tl_variant == QMM_VARIANT_AUTO && half && dtype_code(dt) >= 0 &&
                               qmm_gate_up_on_tensor_cores(wbits, dtype_code(x.scalar_type()), dtype_code(dt), M, w.size(0), K,
                                                           block_size == -1 ? 0 : block_size));
    // (up to 32 tokens `tc` has asked for the shape, scale blocks of any multiple of 128 among them)
    const bool decode = !tc && half && K % (512 / wbits) == 0 && (block_size == -1 || block_size % (512 / wbits) == 0) &&
                        (tl_variant == QMM_VARIANT_AUTO || tl_variant == QMM_VARIANT_MMA);
    const bool batch = tc && K >= 128 && K % (128 / wbits) == 0 &&
                       (M <= 32 || block_size == -1 || block_size == 128 || block_size % 256 == 0) &&
                       (tl_variant == QMM_VARIANT_AUTO || tl_variant == QMM_VARIANT_I8TC);
    if (dtype_code(dt) >= 0 && (decode || batch)) {
      c10::cuda::OptionalCUDAGuard guard(x.device());
      Call c = make_call(x, w, scale, {}, block_size, weight_is_packed);
      c.scales_to_f32();
      const int dev = x.get_device();
      const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev).stream();
      Tensor out = output(x, c.N / 2, dt);
      int rc;
      if (decode) {
        rc = qmm_gate_up_decode(wbits, x.data_ptr(), dtype_code(x.scalar_type()), w.data_ptr(), (const float*)c.scale.data_ptr(),
                                out.data_ptr(), dtype_code(dt), M, c.N, K, c.block, st);
      } else {
        std::lock_guard<std::mutex> hold(g_scratch_lock);
        void* ws;
        size_t ws_bytes;
        scratch(dev, st, qmm_weight_only_workspace_size(M, K), &ws, &ws_bytes);
        // (short of scratch, the Python form takes the decode kernel up to 32 tokens)
        rc = qmm_gate_up(wbits, x.data_ptr(), dtype_code(x.scalar_type()), w.data_ptr(), (const float*)c.scale.data_ptr(),
                         out.data_ptr(), dtype_code(dt), M, c.N, K, c.block, ws, ws_bytes, st);
      }
      if (rc == QMM_OK) return out;
    }
  }
  return python_form<decltype(quantized_gate_up)>("xla_b200::quantized_gate_up_any", x, w, scale, block_size, int4_weight,
                                                  weight_is_packed, out_dtype);
}

}  // namespace

TORCH_LIBRARY_IMPL(xla, CUDA, m) {
  m.impl("quantized_matmul", &quantized_matmul);
  m.impl("quantized_matmul_int8", &quantized_matmul_int8);
}

TORCH_LIBRARY_IMPL(xla_b200, CUDA, m) {
  m.impl("quantized_matmul_packed", &quantized_matmul_packed);
  m.impl("quantized_gate_up", &quantized_gate_up);
}

extern "C" {
// The calling thread's kernel family and activation saturation.
__attribute__((visibility("default"))) void qmmt_set_thread_state(int variant, int saturate) {
  tl_variant = variant;
  tl_saturate = saturate;
}
// The scratch of `stream` on `device` for callers above the C ABI; NULL / 0 when there is none to be had.
__attribute__((visibility("default"))) void qmmt_scratch(int device, void* stream, size_t need, void** ptr, size_t* bytes) {
  std::lock_guard<std::mutex> hold(g_scratch_lock);
  scratch(device, static_cast<cudaStream_t>(stream), need, ptr, bytes);
}
}
