// The operators of the forward path (quantize*, projection*, run of GEMM and plan, and the fused
// projections) bound natively: argument checks, output and scratch allocation and the C-ABI call in one C++
// function behind the torch dispatcher.  The schemas and fake kernels are registered in Python (backend.py);
// this file adds the CUDA implementations of the names the reference binds from its own extension
// (csrc/dualscale_sm80.cu:400-412, csrc/projection_sm80.cu:154-182, csrc/graph_projection.cuh:178-203).
//
// Why native: the same checks, two torch.empty and a ctypes call took 33-40 us of host time per call in
// Python, more than the GPU needs for most projections of fewer than 2048 rows (7-35 us).
//
// Compiled by the host compiler into a library of its own, so that libslidesparse_b200.so keeps a plain C
// interface with no torch types.  Nothing here touches the GPU when it is loaded.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/library.h>
#include <cstring>

#include "../../include/slidesparse_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

void check(int rc) {
  if (rc == SS_OK) return;
  const std::string message = ss_last_error();
  TORCH_CHECK_VALUE(rc != SS_E_ARG && rc != SS_E_FORMAT && rc != SS_E_LIMIT, message);
  TORCH_CHECK(false, message);
}

int group_of(int64_t group) {
  TORCH_CHECK_VALUE(group == 4 || group == 6 || group == 8, "unknown sparsity mode ", group, ": expected 2:4, 4:6 or 6:8");
  return static_cast<int>(group);
}

void check_config(int64_t config) {
  // the reference's SM80 tile identifiers: 0-6 and 11-17
  TORCH_CHECK_VALUE((config >= 0 && config <= 6) || (config >= 11 && config <= 17), "invalid config");
}

int64_t ceil_to(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

int64_t lifted(int64_t k, int group) {
  TORCH_CHECK_VALUE(k > 0, "K must be positive");
  return ceil_to((k + group - 1) / group * (group / 2 - 1) * 4, 128);
}

void* ptr(const Tensor& t) { return t.numel() ? t.data_ptr() : nullptr; }

void check_input(const Tensor& x) {
  TORCH_CHECK_VALUE(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() >= 1, "BF16 CUDA input required");
}

// The input as a matrix with unit column stride: where it is one already (any row stride), in place.
struct Rows {
  Tensor held;             // keeps a copy or a view alive
  const void* data;
  int64_t m, k, stride;
  Rows(const Tensor& x, int64_t width) : k(width) {
    if (x.is_contiguous()) {
      m = k ? x.numel() / k : 0;
      stride = k;
      data = ptr(x);
      return;
    }
    held = x.dim() == 2 ? x : x.reshape({-1, k});
    if (held.stride(-1) != 1) held = held.contiguous();
    m = held.size(0);
    stride = held.stride(0);
    data = ptr(held);
  }
};

Tensor new_output(const Tensor& x, int64_t n) {
  c10::SmallVector<int64_t, 5> sizes(x.sizes().begin(), x.sizes().end());
  sizes.back() = n;
  return at::detail::empty_cuda(sizes, at::kBFloat16, x.device(), std::nullopt);
}

// q [pm, pk] and sa [pm] of one call, carved from one block of the caching allocator (sa first: 4 * pm is
// a multiple of 128 bytes, so q stays 16-byte aligned); it goes back when the call returns, in stream order.
struct Scratch {
  c10::DataPtr block;
  int8_t* q;
  float* sa;
  Scratch(int64_t pm, int64_t pk) : block(c10::cuda::CUDACachingAllocator::get()->allocate(4 * pm + pm * pk)) {
    sa = static_cast<float*>(block.get());
    q = static_cast<int8_t*>(block.get()) + 4 * pm;
  }
};

void* current_stream(const Tensor& x) { return c10::cuda::getCurrentCUDAStream(x.get_device()).stream(); }

void check_weights(const at::Device& device, const Tensor& packed, const Tensor& metadata, const Tensor& sw,
                   const Tensor& bias, int64_t pk) {
  for (const Tensor* t : {&packed, &metadata, &sw, &bias})
    TORCH_CHECK_VALUE(t->device() == device && t->is_contiguous(), "buffer device/layout mismatch");
  TORCH_CHECK_VALUE(packed.scalar_type() == at::kChar && packed.dim() == 2 && metadata.scalar_type() == at::kInt, "packed types");
  TORCH_CHECK_VALUE(sw.scalar_type() == at::kFloat && bias.scalar_type() == at::kFloat, "scale/bias must be FP32");
  TORCH_CHECK_VALUE(packed.size(0) % 32 == 0 && packed.size(1) * 2 == pk, "padding mismatch");
  TORCH_CHECK_VALUE(metadata.numel() == packed.size(0) * pk / 32, "metadata/token scales size");
}

void check_channels(const Tensor& packed, const Tensor& sw, const Tensor& bias, int64_t n) {
  TORCH_CHECK_VALUE(n > 0 && n <= packed.size(0) && sw.numel() >= n && (bias.numel() == 0 || bias.numel() >= n),
                    "original dimensions/channels");
}

struct Addend {
  Tensor held;
  const void* data = nullptr;
  int64_t stride = 0;
  Addend(const OptTensor& addend, const at::Device& device, int64_t m, int64_t n, bool flatten) {
    if (!addend.has_value()) return;
    held = flatten ? addend->reshape({-1, n}) : *addend;
    TORCH_CHECK_VALUE(held.is_cuda() && held.device() == device && held.scalar_type() == at::kBFloat16 && held.dim() == 2 &&
                          held.size(0) == m && held.size(1) == n && held.stride(1) == 1,
                      "addend must be BF16 [M,N] with unit column stride");
    data = ptr(held);
    stride = held.stride(0);
  }
};

std::tuple<Tensor, Tensor> quantize(const Tensor& input, int64_t group_id) {
  check_input(input);
  const int group = group_of(group_id);
  const Rows x(input, input.size(-1));
  TORCH_CHECK_VALUE(x.m > 0, "empty input unsupported by native frontend");
  const int64_t pk = lifted(x.k, group), pm = ceil_to(x.m, 32);
  const c10::cuda::CUDAGuard guard(input.device());
  Tensor q = at::detail::empty_cuda({pm, pk}, at::kChar, input.device(), std::nullopt);
  Tensor sa = at::detail::empty_cuda({pm}, at::kFloat, input.device(), std::nullopt);
  check(ss_quantize_lift(x.data, x.stride, x.m, x.k, group, static_cast<int8_t*>(q.data_ptr()),
                         static_cast<float*>(sa.data_ptr()), current_stream(input)));
  return {q, sa};
}
std::tuple<Tensor, Tensor> quantize_scalar(const Tensor& input) { return quantize(input, 4); }

Tensor projection(const Tensor& input, const Tensor& packed, const Tensor& metadata, const Tensor& scales, const Tensor& bias,
                  int64_t group_id, int64_t n, int64_t config, const OptTensor& output_addend) {
  check_input(input);
  const int group = group_of(group_id);
  check_config(config);
  const Rows x(input, input.size(-1));
  TORCH_CHECK_VALUE(x.m > 0, "empty input unsupported by native frontend");
  const int64_t pk = lifted(x.k, group), pm = ceil_to(x.m, 32);
  check_weights(input.device(), packed, metadata, scales, bias, pk);
  check_channels(packed, scales, bias, n);
  const Addend addend(output_addend, input.device(), x.m, n, true);
  const c10::cuda::CUDAGuard guard(input.device());
  const Scratch scratch(pm, pk);
  Tensor out = new_output(input, n);
  check(ss_projection(x.data, x.stride, x.m, x.k, group, packed.const_data_ptr<int8_t>(), metadata.const_data_ptr<int32_t>(),
                      scales.const_data_ptr<float>(), static_cast<const float*>(ptr(bias)), addend.data, addend.stride, n,
                      packed.size(0), scratch.q, scratch.sa, out.data_ptr(), n, current_stream(input)));
  return out;
}

Tensor gemm_run(const Tensor& q, const Tensor& packed, const Tensor& metadata, const Tensor& sa, const Tensor& sw,
                const Tensor& bias, int64_t m, int64_t n, int64_t config, const OptTensor& output_addend) {
  TORCH_CHECK_VALUE(q.is_cuda() && q.scalar_type() == at::kChar && q.dim() == 2 && q.is_contiguous(), "q must be row-major CUDA int8");
  const int64_t pm = q.size(0), pk = q.size(1);
  TORCH_CHECK_VALUE(pk % 128 == 0 && pm % 32 == 0, "padding mismatch");
  check_weights(q.device(), packed, metadata, sw, bias, pk);
  TORCH_CHECK_VALUE(sa.scalar_type() == at::kFloat && sa.numel() == pm && sa.device() == q.device(), "metadata/token scales size");
  TORCH_CHECK_VALUE(m > 0 && m <= pm, "original dimensions/channels");
  check_channels(packed, sw, bias, n);
  check_config(config);
  const Addend addend(output_addend, q.device(), m, n, false);
  const c10::cuda::CUDAGuard guard(q.device());
  Tensor out = at::detail::empty_cuda({m, n}, at::kBFloat16, q.device(), std::nullopt);
  check(ss_gemm_run(q.const_data_ptr<int8_t>(), packed.const_data_ptr<int8_t>(), metadata.const_data_ptr<int32_t>(),
                    static_cast<const float*>(ptr(sa)), sw.const_data_ptr<float>(), static_cast<const float*>(ptr(bias)),
                    addend.data, addend.stride, out.data_ptr(), n, m, n, pm, packed.size(0), pk, current_stream(q)));
  return out;
}

Tensor prepared_run(const Tensor& input, int64_t handle, int64_t n) {
  int64_t shape[6];
  TORCH_CHECK(ss_plan_shape(handle, shape, 6) == SS_OK, "prepared graph handle absent");
  const int64_t device = shape[0], m = shape[1], k = shape[2], pm = shape[4], pk = shape[5];
  TORCH_CHECK_VALUE(input.is_cuda() && input.get_device() == device && input.scalar_type() == at::kBFloat16 && input.dim() >= 1 &&
                        input.size(-1) == k, "prepared input identity");
  TORCH_CHECK_VALUE(input.numel() == m * k && n == shape[3], "prepared shape changed");
  const Rows x(input, k);
  const c10::cuda::CUDAGuard guard(input.device());
  Tensor out = new_output(input, n);
  void* stream = current_stream(input);
  int rc = ss_plan_run(handle, x.data, x.stride, nullptr, nullptr, out.data_ptr(), n, stream);
  if (rc == SS_E_ARG && std::strstr(ss_last_error(), "caller scratch")) {
    // another stream, or an outer graph capture: independent scratch from torch's allocator
    const Scratch scratch(pm, pk);
    rc = ss_plan_run(handle, x.data, x.stride, scratch.q, scratch.sa, out.data_ptr(), n, stream);
  }
  check(rc);
  return out;
}

// ---- projections with element-wise neighbours in their kernels -------------------------------------------

constexpr int64_t kNone = 0, kNormModulate = 1, kGelu = 2;

// A BF16 [batch, width] tensor of per-batch values as (pointer, row stride).
struct PerBatch {
  Tensor shift, scale;
  int64_t stride = 0, rows = 1;
  PerBatch(const Tensor& x, int64_t prologue, const OptTensor& shift_in, const OptTensor& scale_in) {
    TORCH_CHECK_VALUE(prologue == kNone || prologue == kNormModulate || prologue == kGelu, "unknown prologue");
    const int64_t k = x.size(-1);
    if (x.dim() == 3) rows = x.size(1);
    if (prologue != kNormModulate) return;
    TORCH_CHECK_VALUE(x.dim() == 3, "norm_modulate needs [batch, rows, k] input");
    const int64_t batch = x.size(0);
    for (const OptTensor* t : {&shift_in, &scale_in})
      TORCH_CHECK_VALUE(t->has_value() && (*t)->scalar_type() == at::kBFloat16 && (*t)->device() == x.device() && (*t)->dim() == 2 &&
                            (*t)->size(0) == batch && (*t)->size(1) == k,
                        "shift / scale must be BF16 [batch, k] on the input's device");
    shift = *shift_in;
    scale = *scale_in;
    auto usable = [&](const Tensor& t) {
      return t.stride(1) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && t.stride(0) % 8 == 0 && t.stride(0) >= k;
    };
    if (!usable(shift) || !usable(scale) || (batch > 1 && shift.stride(0) != scale.stride(0))) {
      shift = shift.contiguous();
      scale = scale.contiguous();
    }
    stride = batch > 1 ? shift.stride(0) : k;
  }
};

// input -> out (new, or the residual that is accumulated into)
void projection_fused_into(const Tensor& input, int64_t prologue, const OptTensor& shift, const OptTensor& scale, double eps,
                           const Tensor& packed, const Tensor& metadata, const Tensor& scales, const Tensor& bias,
                           int64_t group_id, int64_t n, const OptTensor& output_addend, const Tensor* gate, Tensor& out) {
  const int group = group_of(group_id);
  const PerBatch per_batch(input, prologue, shift, scale);
  Rows x(input, input.size(-1));
  if (prologue != kNone && (reinterpret_cast<uintptr_t>(x.data) % 16 || x.stride % 8 || x.k % 8)) {
    x.held = input.reshape({-1, x.k}).contiguous();
    x.data = ptr(x.held);
    x.stride = x.k;
    TORCH_CHECK_VALUE(reinterpret_cast<uintptr_t>(x.data) % 16 == 0 && x.k % 8 == 0, "a prologue needs k % 8 == 0");
  }
  TORCH_CHECK_VALUE(x.m > 0, "empty input unsupported by native frontend");
  const int64_t pk = lifted(x.k, group), pm = ceil_to(x.m, 32);
  check_weights(input.device(), packed, metadata, scales, bias, pk);
  check_channels(packed, scales, bias, n);
  const Addend addend(output_addend, input.device(), x.m, n, true);
  const void* gate_data = nullptr;
  int64_t gate_stride = 0;
  if (gate) {
    TORCH_CHECK_VALUE(input.dim() == 3, "gated accumulation needs [batch, rows, k] input, a residual and no addend");
    const int64_t batch = input.size(0), rows = input.size(1);
    TORCH_CHECK_VALUE(out.scalar_type() == at::kBFloat16 && out.device() == input.device() && out.is_contiguous() && out.dim() == 3 &&
                          out.size(0) == batch && out.size(1) == rows && out.size(2) == n &&
                          reinterpret_cast<uintptr_t>(out.data_ptr()) % 16 == 0 && n % 8 == 0,
                      "residual must be contiguous, 16-byte aligned BF16 [batch, rows, n] with n % 8 == 0");
    TORCH_CHECK_VALUE(gate->scalar_type() == at::kBFloat16 && gate->device() == input.device() && gate->dim() == 2 &&
                          gate->size(0) == batch && gate->size(1) == n && gate->stride(1) == 1,
                      "gate must be BF16 [batch, n] with unit column stride");
    TORCH_CHECK_VALUE(rows % 32 == 0, "gated accumulation needs rows per batch to be a multiple of 32");
    gate_data = gate->data_ptr();
    gate_stride = batch > 1 ? gate->stride(0) : n;
  }
  const c10::cuda::CUDAGuard guard(input.device());
  const Scratch scratch(pm, pk);
  if (!gate) out = new_output(input, n);
  const bool norm = prologue == kNormModulate;
  check(ss_projection_fused(x.data, x.stride, x.m, x.k, group, static_cast<int>(prologue),
                            norm ? per_batch.shift.data_ptr() : nullptr, norm ? per_batch.scale.data_ptr() : nullptr,
                            per_batch.stride, per_batch.rows, norm ? static_cast<float>(eps) : 0.f,
                            packed.const_data_ptr<int8_t>(), metadata.const_data_ptr<int32_t>(), scales.const_data_ptr<float>(),
                            static_cast<const float*>(ptr(bias)), addend.data, addend.stride, gate_data, gate_stride, n,
                            packed.size(0), scratch.q, scratch.sa, out.data_ptr(), n, current_stream(input)));
}

Tensor projection_fused(const Tensor& input, int64_t prologue, const OptTensor& shift, const OptTensor& scale, double eps,
                        const Tensor& packed, const Tensor& metadata, const Tensor& scales, const Tensor& bias,
                        int64_t group, int64_t n, const OptTensor& output_addend) {
  check_input(input);
  Tensor out;
  projection_fused_into(input, prologue, shift, scale, eps, packed, metadata, scales, bias, group, n, output_addend, nullptr, out);
  return out;
}

void projection_fused_accumulate(const Tensor& residual, const Tensor& input, int64_t prologue, const OptTensor& shift,
                                 const OptTensor& scale, double eps, const Tensor& packed, const Tensor& metadata,
                                 const Tensor& scales, const Tensor& bias, int64_t group, int64_t n, const Tensor& gate) {
  check_input(input);
  Tensor out = residual;
  projection_fused_into(input, prologue, shift, scale, eps, packed, metadata, scales, bias, group, n, std::nullopt, &gate, out);
}

// x + gate[:, None] * y in torch's own operators, which have every derivative and batching rule
Tensor gate_add_torch(const Tensor& x, const Tensor& gate, const Tensor& y) { return at::addcmul(x, gate.unsqueeze(1), y); }

// Where a gradient or a forward-mode tangent hangs on an operand (a dual tensor does not require gradients),
// torch's operators; the kernel knows neither.
Tensor gate_add_autograd(const Tensor& x, const Tensor& gate, const Tensor& y) {
  for (const Tensor* t : {&x, &gate, &y})
    if ((at::GradMode::is_enabled() && t->requires_grad()) || t->_fw_grad(/*level=*/0).defined()) return gate_add_torch(x, gate, y);
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("slidesparse_b200::gate_add", "")
                             .typed<Tensor(const Tensor&, const Tensor&, const Tensor&)>();
  const at::AutoDispatchBelowADInplaceOrView below;
  return op.call(x, gate, y);
}

// x + gate[:, None] * y: one pass of this library's kernel where the rows allow it, torch's otherwise
Tensor gate_add(const Tensor& x, const Tensor& gate, const Tensor& y) {
  auto aligned = [](const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; };
  const bool usable = x.dim() == 3 && x.numel() > 0 && y.sizes() == x.sizes() && gate.dim() == 2 && gate.size(0) == x.size(0) &&
                      gate.size(1) == x.size(2) && x.scalar_type() == at::kBFloat16 && y.scalar_type() == at::kBFloat16 &&
                      gate.scalar_type() == at::kBFloat16 && x.is_cuda() && y.device() == x.device() && gate.device() == x.device() &&
                      x.is_contiguous() && y.is_contiguous() && x.size(2) % 8 == 0 && gate.stride(1) == 1 &&
                      (gate.size(0) == 1 || (gate.stride(0) % 8 == 0 && gate.stride(0) >= gate.size(1))) &&
                      aligned(x) && aligned(y) && aligned(gate) && x.size(0) * x.size(1) < (1ll << 31) && x.size(2) < (1ll << 31);
  if (!usable) return gate_add_torch(x, gate, y);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor out = new_output(x, x.size(2));
  check(ss_gate_add(x.data_ptr(), gate.data_ptr(), gate.size(0) > 1 ? gate.stride(0) : gate.size(1), y.data_ptr(), out.data_ptr(),
                    x.size(0) * x.size(1), x.size(1), x.size(2), current_stream(x)));
  return out;
}

}  // namespace

TORCH_LIBRARY_IMPL(sdacc_dualscale_sm80, CUDA, m) { m.impl("run", TORCH_FN(gemm_run)); }

TORCH_LIBRARY_IMPL(sdacc_mild_projection_sm80, CUDA, m) {
  // one front-end serves all three variants: they produce identical bits
  m.impl("quantize", TORCH_FN(quantize));
  m.impl("quantize_packed16", TORCH_FN(quantize));
  m.impl("quantize_scalar", TORCH_FN(quantize_scalar));
  m.impl("projection", TORCH_FN(projection));
  m.impl("projection_packed16", TORCH_FN(projection));
  m.impl("projection_scalar", TORCH_FN(projection));
}

TORCH_LIBRARY_IMPL(sdacc_prepared_projection_sm80, CUDA, m) { m.impl("run", TORCH_FN(prepared_run)); }

TORCH_LIBRARY_IMPL(slidesparse_b200, CUDA, m) {
  m.impl("projection_fused", TORCH_FN(projection_fused));
  m.impl("projection_fused_accumulate_", TORCH_FN(projection_fused_accumulate));
  m.impl("gate_add", TORCH_FN(gate_add));
}

TORCH_LIBRARY_IMPL(slidesparse_b200, Autograd, m) { m.impl("gate_add", TORCH_FN(gate_add_autograd)); }

TORCH_LIBRARY_IMPL(slidesparse_b200, FuncTorchBatched, m) { m.impl("gate_add", TORCH_FN(gate_add_torch)); }
