// Shared runtime pieces of the GB300 embedding library: error state, device arena,
// launch helpers and warp/block reductions. Everything here is host/device plumbing
// for the kernels in this directory; no torch types appear anywhere.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <vector>

namespace fe {

// ---------------------------------------------------------------- errors
// The C ABI reports failures the way the reference does
// (src/embedding_cuda_kernels.cpp:65-82): return 1 and keep a thread-local message.
void set_error(const std::string& msg);
void clear_error();
const char* last_error();

struct Error : std::runtime_error {
  explicit Error(const std::string& m) : std::runtime_error(m) {}
};

inline void cuda_check(cudaError_t code, const char* what) {
  if (code != cudaSuccess) throw Error(std::string(what) + ": " + cudaGetErrorString(code));
}
#define FE_CUDA(call) ::fe::cuda_check((call), #call)
#define FE_LAUNCH(what) ::fe::cuda_check(cudaGetLastError(), what)

// Run `body` and convert exceptions into the reference's 0/1 status convention.
template <typename F>
int guarded(F&& body) {
  clear_error();
  try {
    body();
    return 0;
  } catch (const std::exception& e) {
    set_error(e.what());
    cudaGetLastError();
    return 1;
  }
}

// ---------------------------------------------------------------- memory
inline std::size_t align256(std::size_t b) { return (b + 255u) & ~std::size_t(255u); }

// Free-memory preflight with the reference's 5% reserve (src/embedding_cuda_kernels.cpp:234-251).
void check_memory_available(std::size_t required, const char* where);

// One cudaMalloc per call, carved into 256-byte aligned pieces (the reference's
// CudaWorkspace arena, src/embedding_cuda_kernels.cpp:88-127). Sizes are collected first so
// that the preflight sees the whole request.
class Arena {
 public:
  Arena() = default;
  Arena(const Arena&) = delete;
  Arena& operator=(const Arena&) = delete;
  ~Arena() { release(); }
  template <typename T>
  void reserve(T** slot, std::size_t count) {
    plan_.push_back({reinterpret_cast<void**>(slot), align256(count * sizeof(T))});
  }
  void commit(const char* where);
  void release();
  std::size_t bytes() const { return total_; }

 private:
  struct Item {
    void** slot;
    std::size_t bytes;
  };
  std::vector<Item> plan_;
  void* base_ = nullptr;
  std::size_t total_ = 0;
};

struct Stream {
  cudaStream_t s = nullptr;
  Stream() { FE_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)); }
  ~Stream() {
    if (s) cudaStreamDestroy(s);
  }
  Stream(const Stream&) = delete;
  Stream& operator=(const Stream&) = delete;
};

inline int ceil_div(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }

// Entry points that read caller-owned device buffers run on their own non-blocking stream,
// which does not wait for the legacy default stream. Order `s` after everything enqueued so far
// on the legacy stream (and, through it, on every blocking stream) so that the caller's last
// writes to those buffers are complete.
void order_after_legacy_stream(cudaStream_t s);
int sm_count();
// Lets `kernel` be launched with `bytes` of dynamic shared memory. Beyond 48 KB in all, its static share included (up to
// 25 KB here), a kernel has to be allowed more; it is then allowed `most`, the most that any call uses: the limit is a state
// of the whole process, and set to what one call needs, a smaller call on another thread would lower it before the larger
// one's launch.
void allow_dynamic_shared(const void* kernel, std::size_t bytes, std::size_t most);

// ---------------------------------------------------------------- host uploads
// Host -> device copy of caller memory (pageable or not), ordered on stream s. Copies of at
// least kStagedUploadMin bytes go through a process-wide pair of pinned staging buffers: host
// threads fill one buffer while the copy engine drains the other, so large inputs move at
// pinned-copy speed rather than through the driver's pageable path. The source may be reused
// when the call returns. Smaller copies, and copies from pinned memory, are plain
// cudaMemcpyAsync calls.
constexpr std::size_t kStagedUploadMin = std::size_t(1) << 20;
void upload(void* dst, const void* src, std::size_t bytes, cudaStream_t s);

// ---------------------------------------------------------------- device helpers
// Unevaluated sum hi + lo of two floats (about 48 bits), for sums that FP32 is too short for. This
// part's FP64 pipe issues one warp instruction every 19 cycles of an SM (measured: 3.5 FP64
// multiply-adds per ns and SM against 250 in FP32), so ten FP32 instructions are many times cheaper
// than one FP64 addition. The rounding intrinsics keep the compiler from contracting the sums.
struct Float2Sum {
  float hi, lo;
};
__device__ __forceinline__ Float2Sum two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return Float2Sum{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ Float2Sum add(Float2Sum a, Float2Sum b) {
  const Float2Sum s = two_sum(a.hi, b.hi);
  // an infinite sum keeps no low part (its residual would be NaN)
  const float lo = isfinite(s.hi) ? __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)) : 0.0f;
  const float hi = __fadd_rn(s.hi, lo);  // |lo| is far below |s.hi|: renormalise
  return Float2Sum{hi, __fsub_rn(lo, __fsub_rn(hi, s.hi))};
}
__device__ __forceinline__ Float2Sum add(Float2Sum a, float b) { return add(a, Float2Sum{b, 0.0f}); }
__device__ __forceinline__ Float2Sum mul(Float2Sum a, float b) {
  const float p = __fmul_rn(a.hi, b);
  return Float2Sum{p, __fmaf_rn(a.lo, b, __fmaf_rn(a.hi, b, -p))};
}
__device__ __forceinline__ Float2Sum mul(Float2Sum a, Float2Sum b) {
  const float p = __fmul_rn(a.hi, b.hi);
  return Float2Sum{p, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.hi, -p)))};
}
__device__ __forceinline__ Float2Sum split(double v) {
  const float h = (float)v;
  return Float2Sum{h, (float)(v - (double)h)};
}
// a / b for normal b of moderate size: one Newton step on the quotient of the high parts.
__device__ __forceinline__ Float2Sum divide(Float2Sum a, Float2Sum b) {
  const float r = __frcp_rn(b.hi), q = __fmul_rn(a.hi, r);
  const float res = __fadd_rn(__fmaf_rn(-q, b.hi, a.hi), __fmaf_rn(-q, b.lo, a.lo));
  const float c = __fmul_rn(res, r), h = __fadd_rn(q, c);
  return Float2Sum{h, __fadd_rn(c, __fsub_rn(q, h))};
}
// Correctly rounded 1 / x for x in [1, 2^126): one Newton step by fused multiply-add on an approximation
// within one unit in the last place (Markstein 1990, whose theorem leaves out significands of all ones; with this
// part's approximation the step rounds correctly for them too: compared for all 2^23 significands). Larger x, where the
// result is below 1.2e-38, give 0, and NaN gives NaN. Free of the branch to a slow path, so that several pairs are in flight.
__device__ __forceinline__ float reciprocal(float x) {
  float r, c;
  asm("min.NaN.f32 %0, %1, 0f7F7FC99E;" : "=f"(c) : "f"(x));  // 3.4e38: an infinite x must not make the step NaN
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(c));
  return __fmaf_rn(r, __fmaf_rn(-c, r, 1.0f), r);
}
// hi is rounded to nearest, so lo is at most half a unit of hi's last place
__device__ __forceinline__ double value(Float2Sum a) { return (double)a.hi + (double)a.lo; }
__device__ __forceinline__ Float2Sum warp_sum(Float2Sum v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = add(v, Float2Sum{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace fe
