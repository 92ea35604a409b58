// Exact O(n^2) t-SNE quantities on the GPU: repulsive forces with the all-pairs Z, and the
// KL divergence of evaluate_kl_f (fastEmbedR src/tsne_neighbors.cpp:1034-1059, :1338-1365).
// Pair terms are FP32; the forces accumulate tiles of 1024 partners in FP32 and fold them into FP64, the
// normaliser folds 128 partners into two-float sums, so the n^2 sums at N = 1M (5e11 pairs) carry no more
// than the FP32 error of a tile.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "tsne_exact.cuh"
#include "twofloat.cuh"

namespace fe {

constexpr int kPairTile = 1024;

// rep_i = -sum_j q_ij^2 (y_i - y_j) (unnormalised) and zrow_i = sum_{j != i} q_ij.
__global__ void __launch_bounds__(256)
exact_pairs_kernel(const float2* __restrict__ y, int n, double* __restrict__ rep, double* __restrict__ zrow) {
  __shared__ float2 tile[kPairTile];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const float2 yi = i < n ? y[i] : make_float2(0.0f, 0.0f);
  double gx = 0.0, gy = 0.0, z = 0.0;
  for (int t0 = 0; t0 < n; t0 += kPairTile) {
    const int cnt = min(kPairTile, n - t0);
    __syncthreads();
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) tile[t] = y[t0 + t];
    __syncthreads();
    float fx = 0.0f, fy = 0.0f, fz = 0.0f;
    for (int t = 0; t < cnt; ++t) {
      const float2 yj = tile[t];
      const float dx = yi.x - yj.x, dy = yi.y - yj.y;
      const float q = 1.0f / (1.0f + (dx * dx + dy * dy));
      const float w = (t0 + t == i) ? 0.0f : 1.0f;
      fz += w * q;
      fx += w * q * q * dx;
      fy += w * q * q * dy;
    }
    gx += fx;
    gy += fy;
    z += fz;
  }
  if (i < n) {
    rep[2 * (long long)i] = -gx;
    rep[2 * (long long)i + 1] = -gy;
    zrow[i] = z;
  }
}

// All-pairs sum of q without the pairs (i, i), Z: tiles of kPairTile x kPairTile points on and above the diagonal (an
// off-diagonal tile counts twice), dealt to the blocks in turn; part[block] receives the block's sum.
// One reciprocal per pair bounds the pass (16 a clock and SM: 1.1 ms for the 5e9 pairs of 100,000
// points; evaluating both (i, j) and (j, i) with IEEE division took 7.2 ms). It is correctly rounded: the sum averages
// rounding errors out, but not the 3.5e-9 of itself by which __fdividef (within 2 ulp) exceeds the quotient on
// average; here 2e-10 are left (20,000 points). The whole KL of 100,000 points takes 1.63 ms, 1.86 with __fdividef. Each thread sums 128
// partners of a row in FP32 and adds that to a two-float sum.
constexpr int kPairRows = 4;  // rows per thread
constexpr int kPairFold = 128;
static_assert(kPairTile == 256 * kPairRows && kPairTile % kPairFold == 0, "tile");

__device__ __forceinline__ float pair_q(float2 a, float2 b) {
  const float dx = a.x - b.x, dy = a.y - b.y;
  return reciprocal(fmaf(dy, dy, fmaf(dx, dx, 1.0f)));
}

__global__ void __launch_bounds__(256)
sum_q_tiles_kernel(const float2* __restrict__ y, int n, int tiles, double* __restrict__ part) {
  __shared__ float2 tile[kPairTile];
  __shared__ double s_w[8];
  const long long pairs = (long long)tiles * (tiles + 1) / 2;
  double total = 0.0;
  for (long long q = blockIdx.x; q < pairs; q += gridDim.x) {
    // q = b (b + 1) / 2 + a, a <= b
    int b = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
    while ((long long)b * (b + 1) / 2 > q) --b;
    while ((long long)(b + 1) * (b + 2) / 2 <= q) ++b;
    const int a = (int)(q - (long long)b * (b + 1) / 2);
    const int i0 = a * kPairTile, j0 = b * kPairTile, cnt = min(kPairTile, n - j0);
    __syncthreads();
    for (int t = threadIdx.x; t < cnt; t += 256) tile[t] = y[j0 + t];
    __syncthreads();
    float2 yi[kPairRows];
#pragma unroll
    for (int r = 0; r < kPairRows; ++r) yi[r] = y[min(n - 1, i0 + (int)threadIdx.x + r * 256)];
    Float2Sum acc[kPairRows];
#pragma unroll
    for (int r = 0; r < kPairRows; ++r) acc[r] = Float2Sum{0.0f, 0.0f};
    for (int t0 = 0; t0 < cnt; t0 += kPairFold) {
      float f[kPairRows] = {0.0f, 0.0f, 0.0f, 0.0f};
      const int t1 = min(cnt, t0 + kPairFold);
      if (a != b) {
#pragma unroll 4
        for (int t = t0; t < t1; ++t) {
          const float2 yj = tile[t];
#pragma unroll
          for (int r = 0; r < kPairRows; ++r) f[r] += pair_q(yi[r], yj);
        }
      } else {  // leaving the terms of 1 out, not subtracting them, keeps a small Z exact
#pragma unroll 4
        for (int t = t0; t < t1; ++t) {
          const float2 yj = tile[t];
#pragma unroll
          for (int r = 0; r < kPairRows; ++r) f[r] += t == (int)threadIdx.x + r * 256 ? 0.0f : pair_q(yi[r], yj);
        }
      }
#pragma unroll
      for (int r = 0; r < kPairRows; ++r) acc[r] = add(acc[r], f[r]);
    }
    Float2Sum v{0.0f, 0.0f};
#pragma unroll
    for (int r = 0; r < kPairRows; ++r)
      if (i0 + (int)threadIdx.x + r * 256 < n) v = add(v, acc[r]);
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) total += (a == b ? 1.0 : 2.0) * value(v);
  }
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = total;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += s_w[w];
    part[blockIdx.x] = t;
  }
}

// Exact repulsion of selected points against every point, partners split into gridDim.y slices:
// part[(slice * 3 + c) * n_rows + r] holds slice sums of -q^2 dx, -q^2 dy and q (c = 0, 1, 2) for
// the point y[inv[rows[r]]], excluding the point itself. FP32 pair terms, FP64 tile sums.
__global__ void __launch_bounds__(256)
exact_rows_kernel(const float2* __restrict__ y, int n, const int* __restrict__ rows, const int* __restrict__ inv,
                  int n_rows, int slice, double* __restrict__ part) {
  __shared__ float2 tile[kPairTile];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int si = r < n_rows ? inv[rows[r]] : -1;
  const float2 yi = si >= 0 ? y[si] : make_float2(0.0f, 0.0f);
  const int j0 = blockIdx.y * slice, j1 = min(n, j0 + slice);
  double gx = 0.0, gy = 0.0, z = 0.0;
  for (int t0 = j0; t0 < j1; t0 += kPairTile) {
    const int cnt = min(kPairTile, j1 - t0);
    __syncthreads();
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) tile[t] = y[t0 + t];
    __syncthreads();
    float fx = 0.0f, fy = 0.0f, fz = 0.0f;
    for (int t = 0; t < cnt; ++t) {
      const float2 yj = tile[t];
      const float dx = yi.x - yj.x, dy = yi.y - yj.y;
      const float q = 1.0f / (1.0f + (dx * dx + dy * dy));
      const float w = (t0 + t == si) ? 0.0f : 1.0f;
      fz += w * q;
      fx += w * q * q * dx;
      fy += w * q * q * dy;
    }
    gx += fx;
    gy += fy;
    z += fz;
  }
  if (r < n_rows) {
    const long long b = (long long)blockIdx.y * 3 * n_rows;
    part[b + r] = -gx;
    part[b + n_rows + r] = -gy;
    part[b + 2LL * n_rows + r] = z;
  }
}

// out[c * n_rows + r] = sum over slices (in slice order) of part.
__global__ void sum_slices_kernel(const double* __restrict__ part, int n_rows, int slices, double* __restrict__ out) {
  const long long m = 3LL * n_rows;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < m; t += (long long)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int sl = 0; sl < slices; ++sl) acc += part[sl * m + t];
    out[t] = acc;
  }
}

// out = sum of v, in a fixed order (one block).
__global__ void reduce_double_kernel(const double* __restrict__ v, int n, double* out) {
  __shared__ double part[1024];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += v[i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = part[0];
}

// KL = sum_CSR p log((p + 1e-9) / (q / Z + 1e-9)); Z rounded to float as the reference keeps it.
// Row i of P belongs to the point at y[inv[i]] (inv = nullptr: y is in row order); columns index y.
// Warp per row, entries in two floats (the FP64 divisions and logarithms of an entry took 150 FP64
// instructions at 19 cycles each: 2.1 ms for 100,000 rows); part[block] receives the block's sum.
__global__ void __launch_bounds__(256)
kl_rows_kernel(const int* __restrict__ row_ptr, const int* __restrict__ col, const float* __restrict__ val,
               const float2* __restrict__ y, const float2* __restrict__ y_rows, const int* __restrict__ inv, int n,
               const double* __restrict__ zsum, double* __restrict__ part) {
  __shared__ float4 table[kLogEntries];
  __shared__ double s_w[8];
  fill_log_table(table);
  __syncthreads();
  const int lane = threadIdx.x & 31, warps = gridDim.x * 8;
  const double over_z = 1.0 / (double)(float)fmax(*zsum, (double)FLT_MIN);
  const Float2Sum inv_z = split(over_z);
  const Float2Sum tiny = split(1e-9);
  Float2Sum acc{0.0f, 0.0f};
  for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < n; i += warps) {
    const float2 yi = inv ? y[inv[i]] : y_rows[i];
    const unsigned end = row_ptr[i + 1];  // unsigned: the step past a row that ends near 2^31 goes beyond it
    for (unsigned p = row_ptr[i] + lane; p < end; p += 32) {
      const float2 yj = y[col[p]];
      const float pv = val[p];
      const float dx = yi.x - yj.x, dy = yi.y - yj.y;
      const float d2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
      Float2Sum den;
      if (!(d2 > 1.0e30f)) den = add(mul(divide(Float2Sum{1.0f, 0.0f}, two_sum(1.0f, d2)), inv_z), tiny);
      else den = split(1.0 / (1.0 + (double)d2) * over_z + 1e-9);  // q is small, but Z may be as well
      const Float2Sum l = log_two(divide(add(tiny, pv), den), table);
      acc = add(acc, mul(l, pv));
    }
  }
  acc = warp_sum(acc);
  if (lane == 0) s_w[threadIdx.x >> 5] = value(acc);
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += s_w[w];
    part[blockIdx.x] = t;
  }
}

namespace {
// Z; part: scratch of n doubles.
void total_q(const float2* y, int n, double* part, double* out, cudaStream_t s) {
  const int tiles = ceil_div(n, kPairTile);
  const int blocks = (int)std::min<long long>((long long)tiles * (tiles + 1) / 2, std::min(n, sm_count() * 8));
  sum_q_tiles_kernel<<<blocks, 256, 0, s>>>(y, n, tiles, part);
  FE_LAUNCH("sum_q_tiles_kernel");
  reduce_double_kernel<<<1, 1024, 0, s>>>(part, blocks, out);
  FE_LAUNCH("reduce_double_kernel");
}
}  // namespace

void exact_repulsion(const float* d_y, int n, double* d_rep, double* d_zrow, double* d_ztotal, cudaStream_t s) {
  exact_pairs_kernel<<<ceil_div(n, 256), 256, 0, s>>>(reinterpret_cast<const float2*>(d_y), n, d_rep, d_zrow);
  FE_LAUNCH("exact_pairs_kernel");
  reduce_double_kernel<<<1, 1024, 0, s>>>(d_zrow, n, d_ztotal);
  FE_LAUNCH("reduce_double_kernel");
}

int exact_rows_slices(int n, int n_rows) {
  const int row_blocks = ceil_div(n_rows, 256);
  const int want = std::max(1, ceil_div(8 * sm_count(), row_blocks));
  return std::min(want, std::max(1, ceil_div(n, kPairTile)));
}

void exact_repulsion_rows(const float* d_y, int n, const int* d_rows, const int* d_inv, int n_rows, double* d_part,
                          double* d_out, double* d_zrow, double* d_ztotal, cudaStream_t s) {
  const float2* y = reinterpret_cast<const float2*>(d_y);
  const int slices = exact_rows_slices(n, n_rows);
  const int slice = ceil_div(n, slices);
  exact_rows_kernel<<<dim3(ceil_div(n_rows, 256), slices), 256, 0, s>>>(y, n, d_rows, d_inv, n_rows, slice, d_part);
  FE_LAUNCH("exact_rows_kernel");
  sum_slices_kernel<<<std::max(1, std::min(ceil_div(3 * n_rows, 256), sm_count() * 4)), 256, 0, s>>>(
      d_part, n_rows, slices, d_out);
  FE_LAUNCH("sum_slices_kernel");
  total_q(y, n, d_zrow, d_ztotal, s);
}

void exact_kl(const DeviceCsr& P, const float* d_y, const int* d_inv, double* d_zrow, double* d_work,
              double* d_scalars, cudaStream_t s) {
  exact_kl_range(P.row_ptr, P.col, P.val, P.n, d_y, d_inv, 0, d_zrow, d_work, d_scalars, s);
}

void exact_kl_range(const int* row_ptr, const int* col, const float* val, int n, const float* d_y, const int* d_inv,
                    int y_begin, double* d_zrow, double* d_work, double* d_scalars, cudaStream_t s) {
  const float2* y = reinterpret_cast<const float2*>(d_y);
  total_q(y + y_begin, n, d_zrow, d_scalars, s);
  const int blocks = std::max(1, std::min(ceil_div(n, 8), sm_count() * 8));
  kl_rows_kernel<<<blocks, 256, 0, s>>>(row_ptr, col, val, y, y + y_begin, d_inv, n, d_scalars, d_work);
  FE_LAUNCH("kl_rows_kernel");
  reduce_double_kernel<<<1, 1024, 0, s>>>(d_work, blocks, d_scalars + 1);
  FE_LAUNCH("reduce_double_kernel");
}

}  // namespace fe
