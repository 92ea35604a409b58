// The least squares of UMAP's curve 1 / (1 + a x^(2b)) over the reference's grid of (a, b): 443,000 terms. On the
// host, with a power each, they take 5 ms, longer than building the graph of 100,000 points and running its
// epochs; here a block per (b, seven values of a) computes the powers of its b once: 47 us, beside the uploads
// and the graph build, bound by the FP64 pipe.
#include <cmath>

#include "umap_curve.cuh"

namespace fe {
namespace {

constexpr int kThreads = 320;
constexpr int kPerBlock = 7;  // values of a per block, one per warp

// The grid's values as the reference accumulates them.
__device__ __forceinline__ double stepped(double first, double step, int i) {
  for (int t = 0; t < i; ++t) first = __dadd_rn(first, step);
  return first;
}

__device__ __forceinline__ void curve_point(double spread, double min_dist, int i, double& x, double& y) {
  x = __ddiv_rn(__dmul_rn(__dmul_rn(spread, 3.0), (double)i), 299.0);
  y = x < min_dist ? 1.0 : exp(-(x - min_dist) / spread);
}

__global__ void __launch_bounds__(kThreads)
umap_curve_grid_kernel(double spread, double min_dist, double* __restrict__ loss) {
  __shared__ double s_p[kCurvePoints], s_y[kCurvePoints];
  const int ib = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kCurvePoints) {
    double x, y;
    curve_point(spread, min_dist, threadIdx.x, x, y);
    s_p[threadIdx.x] = pow(x, 2.0 * stepped(0.25, 0.05, ib));
    s_y[threadIdx.x] = y;
  }
  __syncthreads();
  const int ia = blockIdx.y * kPerBlock + warp;
  if (warp >= kPerBlock || ia >= kCurveLogA) return;
  const double a = exp(stepped(-4.0, 0.2, ia));
  double sum = 0.0;
  for (int i = lane; i < kCurvePoints; i += 32) {
    const double e = 1.0 / (1.0 + a * s_p[i]) - s_y[i];
    sum += e * e;
  }
  sum = warp_sum(sum);
  if (lane == 0) loss[ia * kCurveB + ib] = sum;
}

}  // namespace

void curve_grid_losses(double spread, double min_dist, double* loss, cudaStream_t s) {
  umap_curve_grid_kernel<<<dim3(kCurveB, ceil_div(kCurveLogA, kPerBlock)), kThreads, 0, s>>>(spread, min_dist, loss);
  FE_LAUNCH("umap_curve_grid_kernel");
}

}  // namespace fe
