// Shared host/device helpers of the gewell_b200 kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <string>

#include "../../include/gewell_b200.h"
#include "../../include/gewell_b200_test.h"

namespace gw {

// ---------------------------------------------------------------------------
// host: status + error message plumbing
// ---------------------------------------------------------------------------
gw_status fail(gw_status code, const std::string& message);
void clear_error();

#define GW_CUDA_CHECK(expr, what)                                                          \
  do {                                                                                     \
    cudaError_t gw_cuda_status_ = (expr);                                                  \
    if (gw_cuda_status_ != cudaSuccess)                                                    \
      return ::gw::fail(GW_CUDA_ERROR, std::string(what) + ": " + cudaGetErrorString(gw_cuda_status_)); \
  } while (0)

inline size_t align_up(size_t value, size_t alignment) {
  return (value + alignment - 1) / alignment * alignment;
}

inline cudaStream_t as_stream(void* stream) { return static_cast<cudaStream_t>(stream); }

// Per-GPU state (keyed by the device that is current at the call).
constexpr int kMaxDeviceSlots = 64;
int current_device_slot();
// Error word written by bounded waits (0 = no error): lazily allocated, one per GPU.
uint32_t* device_error_word();
// Set-up of device memory, complete when these return.  cudaMemset and a cudaMemcpy to the device may return earlier, and the
// streams that use the memory need not be ordered behind the default stream they run on.
cudaError_t zero_now(void* device, size_t bytes);
cudaError_t upload_now(void* device, const void* host, size_t bytes);
int sm_count();
// Counts the kernels this library launches (read by gw_debug_launch_count); every launch site calls it.
void note_launch(unsigned kernels = 1);
// Error word of the allocation-free linear (static_scratch.cu) on the current GPU, cleared on read;
// 0 when that entry point has not run on this GPU.
uint32_t take_static_scratch_error();

constexpr size_t scale_storage_bytes(size_t rows, size_t width) {
  return ((rows + 127) / 128) * ((width + 63) / 64) * 512;
}

// ---------------------------------------------------------------------------
// device: number formats
// ---------------------------------------------------------------------------
using bf16 = __nv_bfloat16;

__host__ __device__ __forceinline__ size_t scale_offset(size_t row, size_t block, size_t width) {
  return ((row / 128) * (width / 64) + block / 4) * 512 + (row % 32) * 16 + ((row % 128) / 32) * 4 +
         block % 4;
}

// Division by a launch constant (dividends below 2^31): a multiplication instead of the 20 to 100 instructions of an
// integer division.
struct Divisor {
  uint32_t value, multiplier, shift;
  static Divisor of(uint32_t d) {
    uint32_t s = 0;
    while ((1ull << s) < d) ++s;                         // 2^(s-1) < d <= 2^s
    return Divisor{d, uint32_t(((1ull << (31 + s)) + d - 1) / d), s};
  }
  // multiplier = ceil(2^(31 + s) / d) < 2^32, exact for n < 2^31
#ifdef __CUDACC__
  __device__ __forceinline__ uint32_t quotient(uint32_t n) const { return shift == 0 ? n : __umulhi(n, multiplier) >> (shift - 1); }
#endif
};

#ifdef __CUDACC__
// Programmatic dependent launch.  A kernel launched with the programmatic-
// serialisation attribute may start while its predecessor in the stream still
// runs; griddep_wait() blocks until that predecessor has completed and its
// writes are visible (no-op for a normal launch).  griddep_enter() waits and
// then lets the successor start being scheduled: so when a kernel starts,
// everything before its direct predecessor is complete and visible, and only
// what that one predecessor writes is not.  The activation quantisers alone
// let the successor start first (griddep_enter_first): they are short, and the
// GEMM behind them gets its weights under way at the end of the kernel in
// front of them.  Before its wait a kernel may
//   - read the launch's parameters and what the host wrote before the launch,
//   - read what an earlier launch than its direct predecessor wrote, if that
//     one is none of those quantisers: so the grouped MoE GEMMs read the
//     expert offsets, with the routing and the rows' own launch before them,
//   - bring weights into L2 (ptx::tma_prefetch_*), whoever writes them,
//   - read weights that are settled: in front of the launch, or of the
//     quantiser before it, the same call launched another kernel, which is no
//     quantiser and writes no weights (weights_settled in StreamProblem and
//     DenseProblem).  Of what runs in front of a public entry point's first
//     launch nothing is known; it may have produced the weights.
// Everything else in global memory is touched after the wait.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void griddep_enter() {
  griddep_wait();
  griddep_launch();
}
__device__ __forceinline__ void griddep_enter_first() {
  griddep_launch();
  griddep_wait();
}

#endif  // __CUDACC__

// Launch with the programmatic-serialisation attribute: the kernel may be scheduled while
// its predecessor in the stream drains, and keeps to the rule above.
template <typename... Params, typename... Args>
inline cudaError_t launch_pdl_shared(void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared_bytes, cudaStream_t stream,
                                     Args&&... args) {
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = shared_bytes;
  config.stream = stream;
  cudaLaunchAttribute attribute{};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  note_launch();
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}
template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, cudaStream_t stream, Args&&... args) {
  return launch_pdl_shared(kernel, grid, block, 0, stream, static_cast<Args&&>(args)...);
}

#ifdef __CUDACC__
__device__ __forceinline__ float rcp_approx_ftz(float value) {
  float result;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(result) : "f"(value));
  return result;
}

__device__ __forceinline__ float e4m3_to_float(uint8_t code) {
  return __half2float(__half(__nv_cvt_fp8_to_halfraw(code, __NV_E4M3)));
}

__device__ __forceinline__ uint8_t float_to_e4m3(float value) {
  return __nv_cvt_float_to_fp8(value, __NV_SATFINITE, __NV_E4M3);
}

__device__ __forceinline__ float2 e2m1x2_to_float2(uint8_t packed) {
  return __half22float2(__half2(__nv_cvt_fp4x2_to_halfraw2(packed, __NV_E2M1)));
}

__device__ __forceinline__ uint8_t float2_to_e2m1x2(float lo, float hi) {
  return __nv_cvt_float2_to_fp4x2(make_float2(lo, hi), __NV_E2M1, cudaRoundNearest);
}

// GeGLU with both BF16 rounding boundaries kept: FP32 operation order of the
// reference's gelu_tanh_multiply_bf16 (src/bf16_activation.cuh:10-16).
__device__ __forceinline__ float gelu_tanh_multiply_bf16(float gate, float up) {
  const float cube = gate * gate * gate;
  const float inner = 0.7978845608028654F * (gate + 0.044715F * cube);
  const float activated = 0.5F * gate * (1.0F + tanhf(inner));
  const bf16 rounded = __float2bfloat16_rn(activated);
  return __bfloat162float(__float2bfloat16_rn(__bfloat162float(rounded) * up));
}

__device__ __forceinline__ float bf16_bits_to_float(uint32_t bits16) {
  return __uint_as_float(bits16 << 16);
}
#endif  // __CUDACC__

}  // namespace gw
