// Normal draws of the std::mt19937 stream on the GPU (see mt_normal.cuh).
//
// The engine is serial on the host: 1.2 ms for the 160,000 draws of a spectral start of 20,000 points, twice the graph
// build it runs beside. A state of 624 words can be stepped in three parallel parts (word i needs words i, i + 1 and
// i + 397 of the old state, or i - 227 of the new one), so one block makes the words at the pace of its three barriers
// per state; the polar method's points are then tested, compacted in order and finished by all SMs: 172 + 8 + 23 us,
// and the call 5.0 -> 4.1 ms.
#include <climits>

#include "../../include/fastembedr_cuda.h"
#include "mt_normal.cuh"

namespace fe {
namespace {

constexpr int kState = 624, kShift = 397;
constexpr int kWordThreads = 256;
constexpr int kPointThreads = 256, kPerThread = 4;  // candidate points of four words each
constexpr int kPerBlock = kPointThreads * kPerThread;

__global__ void __launch_bounds__(kWordThreads)
mt_words_kernel(std::uint32_t seed, int states, std::uint32_t* __restrict__ words) {
  __shared__ std::uint32_t s_mt[2][kState];
  if (threadIdx.x == 0) {
    std::uint32_t x = seed;
    s_mt[0][0] = x;
    for (int i = 1; i < kState; ++i) {
      x = 1812433253u * (x ^ (x >> 30)) + (std::uint32_t)i;
      s_mt[0][i] = x;
    }
  }
  __syncthreads();
  for (int t = 0; t < states; ++t) {
    const std::uint32_t* from = s_mt[t & 1];
    std::uint32_t* to = s_mt[(t & 1) ^ 1];
    std::uint32_t* out = words + (long long)t * kState;
    auto step = [&](int i, std::uint32_t far, std::uint32_t next) {
      const std::uint32_t y = (from[i] & 0x80000000u) | (next & 0x7fffffffu);
      std::uint32_t z = far ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
      to[i] = z;
      z ^= z >> 11;
      z ^= (z << 7) & 0x9d2c5680u;
      z ^= (z << 15) & 0xefc60000u;
      out[i] = z ^ (z >> 18);
    };
    const int a = threadIdx.x;
    if (a < kState - kShift) step(a, from[a + kShift], from[a + 1]);
    __syncthreads();
    const int b = a + (kState - kShift);
    if (a < kState - kShift) step(b, to[b - (kState - kShift)], from[b + 1]);
    __syncthreads();
    const int c = a + 2 * (kState - kShift);
    if (c < kState) step(c, to[c - (kState - kShift)], c + 1 < kState ? from[c + 1] : to[0]);
    __syncthreads();
  }
}

struct PolarPoint {
  double x, y, r2;
  bool accepted;
};

__device__ __forceinline__ double canonical(std::uint32_t lo, std::uint32_t hi) {
  const double r = ((double)lo + (double)hi * 4294967296.0) * 5.421010862427522170037e-20;  // 2^-64
  return r >= 1.0 ? 0.99999999999999988897769753748 : r;
}

// The square of the radius is rounded as the host rounds it, or a point next to the unit circle could be accepted by one
// and not by the other, which would shift every later draw, and its logarithm, of 1 - r2, would be off by far more than r2.
using Radius = NormalStream::Radius;
__device__ __forceinline__ PolarPoint polar_point(uint4 w, Radius radius) {
  PolarPoint p;
  p.x = 2.0 * canonical(w.x, w.y) - 1.0;
  p.y = 2.0 * canonical(w.z, w.w) - 1.0;
  const double xx = __dmul_rn(p.x, p.x), yy = __dmul_rn(p.y, p.y);
  p.r2 = radius == Radius::kFusedX ? __fma_rn(p.x, p.x, yy)
                                   : radius == Radius::kFusedY ? __fma_rn(p.y, p.y, xx) : __dadd_rn(xx, yy);
  p.accepted = p.r2 <= 1.0 && p.r2 != 0.0;
  return p;
}

// Sum over the block of one int per thread, and the sum over the threads before this one.
__device__ __forceinline__ int block_prefix(int v, int& total) {
  __shared__ int s_w[kPointThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  __syncthreads();
  if (lane == 31) s_w[warp] = x;
  __syncthreads();
  int before = 0;
  total = 0;
  for (int w = 0; w < kPointThreads / 32; ++w) {
    if (w < warp) before += s_w[w];
    total += s_w[w];
  }
  return before + x - v;
}

__global__ void __launch_bounds__(kPointThreads)
polar_count_kernel(const uint4* __restrict__ words, int candidates, Radius radius, int* __restrict__ counts) {
  const int first = blockIdx.x * kPerBlock + threadIdx.x * kPerThread;
  int mine = 0;
  for (int u = 0; u < kPerThread; ++u)
    if (first + u < candidates) mine += polar_point(words[first + u], radius).accepted;
  int total = 0;
  block_prefix(mine, total);
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kPointThreads)
polar_fill_kernel(const uint4* __restrict__ words, int candidates, Radius radius, const int* __restrict__ counts,
                  long long pairs, double sd, double scale, double2* __restrict__ out, int* __restrict__ enough) {
  int before = 0, unused = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += kPointThreads) before += counts[b];
  block_prefix(before, before);
  const int first = blockIdx.x * kPerBlock + threadIdx.x * kPerThread;
  PolarPoint p[kPerThread];
  int mine = 0;
#pragma unroll
  for (int u = 0; u < kPerThread; ++u) {
    p[u].accepted = false;
    if (first + u < candidates) p[u] = polar_point(words[first + u], radius);
    mine += p[u].accepted;
  }
  long long at = before + block_prefix(mine, unused);
#pragma unroll
  for (int u = 0; u < kPerThread; ++u) {
    if (!p[u].accepted) continue;
    if (at < pairs) {
      const double m = sqrt(-2.0 * log(p[u].r2) / p[u].r2);
      out[at] = make_double2(p[u].y * m * sd * scale, p[u].x * m * sd * scale);
    }
    if (++at == pairs) *enough = 1;
  }
}

}  // namespace

MtNormalBlock::MtNormalBlock(std::uint32_t seed, std::size_t count, double sd, double scale, long long max_points)
    : count_(count) {
  const long long pairs = (long long)(count / 2);
  // pi / 4 of the points are accepted, with a standard deviation of half the root of their number: 2% and 4,096 more
  const long long enough = (long long)((double)pairs * 1.2733 * 1.02) + 4096;
  const long long points = max_points > 0 ? std::min(enough, max_points) : enough;
  const long long states = (points * 4 + kState - 1) / kState;
  if (states * (kState / 4) > INT_MAX / 2) throw Error("too many draws for one block");
  const int candidates = (int)(states * (kState / 4)), blocks = ceil_div(candidates, kPerBlock);
  std::uint32_t* words = nullptr;
  int* counts = nullptr;
  arena_.reserve(&words, (std::size_t)candidates * 4);
  arena_.reserve(&counts, blocks);
  arena_.reserve(&out_, count);
  arena_.reserve(&enough_, 1);
  arena_.commit("normal draws");
  cudaStream_t s = stream_.s;
  FE_CUDA(cudaMemsetAsync(enough_, 0, sizeof(int), s));
  mt_words_kernel<<<1, kWordThreads, 0, s>>>(seed, (int)states, words);
  FE_LAUNCH("mt_words_kernel");
  const uint4* quads = reinterpret_cast<const uint4*>(words);
  const Radius radius = NormalStream::radius_rounding();
  polar_count_kernel<<<blocks, kPointThreads, 0, s>>>(quads, candidates, radius, counts);
  FE_LAUNCH("polar_count_kernel");
  polar_fill_kernel<<<blocks, kPointThreads, 0, s>>>(quads, candidates, radius, counts, pairs, sd, scale,
                                                     reinterpret_cast<double2*>(out_), enough_);
  FE_LAUNCH("polar_fill_kernel");
}

MtNormalBlock::~MtNormalBlock() { cudaStreamSynchronize(stream_.s); }

bool MtNormalBlock::copy_to(double* dst, cudaStream_t s) {
  int enough = 0;
  FE_CUDA(cudaMemcpyAsync(&enough, enough_, sizeof(int), cudaMemcpyDeviceToHost, stream_.s));
  FE_CUDA(cudaStreamSynchronize(stream_.s));
  if (!enough) return false;
  FE_CUDA(cudaMemcpyAsync(dst, out_, sizeof(double) * count_, cudaMemcpyDeviceToDevice, s));
  return true;
}

}  // namespace fe

extern "C" int fastembedr_cuda_normal_draws(unsigned int seed, long long count, long long max_points, double* device,
                                            double* host, int* enough) {
  return fe::guarded([&] {
    if (!device || !host || !enough) throw fe::Error("null output of the normal draws");
    if (count < 2 || count % 2 != 0) throw fe::Error("the normal draws come in pairs");
    std::mt19937 rng(seed);
    fe::NormalStream stream(0.0, 1e-4);
    stream.fill(rng, host, (std::size_t)count, 10000.0);
    fe::Stream st;
    fe::Arena a;
    double* d = nullptr;
    a.reserve(&d, (std::size_t)count);
    a.commit("normal draws");
    fe::MtNormalBlock block(seed, (std::size_t)count, 1e-4, 10000.0, max_points);
    *enough = block.copy_to(d, st.s) ? 1 : 0;
    if (*enough) FE_CUDA(cudaMemcpyAsync(device, d, sizeof(double) * count, cudaMemcpyDeviceToHost, st.s));
    FE_CUDA(cudaStreamSynchronize(st.s));
  });
}
