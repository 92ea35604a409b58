// PCA start of t-SNE on the GPU.
//
// The reference's device PCA initialisation (opentsne_fft_from_knn_impl,
// src/embedding_cuda_kernels.cpp:5860-5893) centres the columns of the data on the host
// (raft_tsvd_scores_to_device, :3379-3437: column means in double, float data minus float mean),
// calls RAPIDS RAFT's tsvd_fit_transform with the COV_EIG_DQ solver and sign flipping based on
// the scores (:3495-3525; RAFT is not vendored and the reference pins no version), then centres
// the two score columns and scales both by 1e-4 / the larger standard deviation
// (tsvd_scores_to_rowmajor_init_kernel :1337, finalize_tsne_pca_init_stats_kernel :1352,
// scale_tsne_pca_init_kernel :1411). The published algorithm of that solver: the Gram matrix
// C = Xc^T Xc, its symmetric eigendecomposition, components = eigenvectors of the largest
// eigenvalues, scores = Xc V, and each score column's sign chosen so that its entry of largest
// magnitude is positive.
//
// Here every step runs on the GPU: column means; C from exact products in two-float sums (tiles of C x
// row slices, partials summed in a fixed order in FP64); a cyclic Jacobi eigendecomposition on one
// block in two-float arithmetic (round-robin ordering: the p/2 disjoint rotations of a step are applied
// together) and one FP64 refinement of the two leading eigenvectors; scores in two-float; the sign rule; and the reference's scaling. The centred data
// are scaled by the power of two that brings their largest magnitude near 1, so that no product leaves the float range.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "pca.cuh"

namespace fe {
namespace {

constexpr int kGramTile = 16;
constexpr int kGramRows = 64;
constexpr int kGramSlices = 128;
constexpr int kMeanSlices = 32;
constexpr int kJacobiThreads = 1024;
constexpr int kJacobiSweeps = 30;
constexpr int kPcaMaxFeatures = 1024;
constexpr float kCloseGap = 1.0e-4f;
constexpr int kJacobiSharedFeatures = 152;  // 152 x 152 two-float values: 185 KB of shared memory

// Exponent of the power of two the centred data are divided by (`bits`: their largest magnitude's).
__device__ __forceinline__ int data_exponent(int bits) {
  const float top = __int_as_float(bits);
  return top > 0.0f ? min(max(ilogbf(top), -100), 126) : 0;
}

// part[column][slice] = sum of the slice's rows of the column, range[column][slice] = their smallest and largest
// value, status[0] set on a non-finite value. 200,000 x 50: one FP64 sum per block of a column took 389 us,
// 19 us now.
__global__ void __launch_bounds__(256)
pca_sum_kernel(const float* __restrict__ X, int n, double* __restrict__ part, float2* __restrict__ range,
               int* __restrict__ status) {
  __shared__ double s_sum[8];
  __shared__ float2 s_range[8];
  const float* col = X + (long long)blockIdx.x * n;
  const int first = blockIdx.y * 256 + threadIdx.x, stride = gridDim.y * 256;
  Float2Sum s{0.0f, 0.0f};
  float lo = FLT_MAX, hi = -FLT_MAX;
  bool finite = true;
#pragma unroll 4
  for (int i = first; i < n; i += stride) {
    const float v = col[i];
    finite &= isfinite(v);
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
    s = add(s, v);
  }
  double t = value(s);
  if (!isfinite(s.hi)) {  // finite values whose sum leaves the float range
    t = 0.0;
    for (int i = first; i < n; i += stride) t += (double)col[i];
  }
  if (!finite) atomicExch(status, 1);
  t = warp_sum(t);
  lo = warp_min(lo);
  hi = warp_max(hi);
  if ((threadIdx.x & 31) == 0) {
    s_sum[threadIdx.x >> 5] = t;
    s_range[threadIdx.x >> 5] = make_float2(lo, hi);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    t = 0.0;
    for (int w = 0; w < 8; ++w) {
      t += s_sum[w];
      lo = fminf(lo, s_range[w].x);
      hi = fmaxf(hi, s_range[w].y);
    }
    part[blockIdx.x * gridDim.y + blockIdx.y] = t;
    range[blockIdx.x * gridDim.y + blockIdx.y] = make_float2(lo, hi);
  }
}

// The columns' means; status[1] = bits of the largest magnitude of the centred data. (Of the data themselves it would
// be a constant column's: one of 1e23 beside columns of spread 1 would leave these no bits.)
__global__ void pca_mean_kernel(const double* __restrict__ part, const float2* __restrict__ range, int p, int slices,
                                int n, float* __restrict__ mean, int* __restrict__ status) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= p) return;
  double t = 0.0;
  float lo = FLT_MAX, hi = -FLT_MAX;
  for (int y = 0; y < slices; ++y) {
    t += part[c * slices + y];
    lo = fminf(lo, range[c * slices + y].x);
    hi = fmaxf(hi, range[c * slices + y].y);
  }
  const float m = (float)(t / (double)n);
  mean[c] = m;
  atomicMax(status + 1, __float_as_int(fmaxf(fabsf(lo - m), fabsf(hi - m))));
}

// partial[slice][a][b] = sum over the slice's rows of u_a u_b, u = (X - mean) / 2^e, for the block's 16 x 16
// tile of C on or above the diagonal (blockIdx.x = tile, blockIdx.y = row slice). A product is exact as
// float + residual, so each adds ten FP32 instructions where FP64 took one multiply-add at a warp
// instruction in 19 cycles per SM; four rows are read from shared memory at a time (rows 68 floats apart:
// no bank conflicts). 200,000 x 50: 4513 us with FP64 sums over all tiles, 201 us now, bound by FP32 issue.
__global__ void __launch_bounds__(kGramTile * kGramTile)
pca_gram_kernel(const float* __restrict__ X, const float* __restrict__ mean, const int* __restrict__ status, int n,
                int p, double* __restrict__ partial) {
  __shared__ __align__(16) float sa[kGramTile][kGramRows + 4];
  __shared__ __align__(16) float sb[kGramTile][kGramRows + 4];
  int tb = 0;  // blockIdx.x = tb (tb + 1) / 2 + ta, ta <= tb
  while ((tb + 1) * (tb + 2) / 2 <= (int)blockIdx.x) ++tb;
  const int ta = (int)blockIdx.x - tb * (tb + 1) / 2;
  const int la = threadIdx.x / kGramTile, lb = threadIdx.x % kGramTile;
  const int a = ta * kGramTile + la, b = tb * kGramTile + lb;
  const float unit = scalbnf(1.0f, -data_exponent(status[1]));
  Float2Sum acc{0.0f, 0.0f};
  auto product = [&](float u, float v) {
    const float q = __fmul_rn(u, v);
    const Float2Sum t = two_sum(acc.hi, q);
    acc = Float2Sum{t.hi, __fadd_rn(acc.lo, __fadd_rn(t.lo, __fmaf_rn(u, v, -q)))};
  };
  // thread t loads rows t % 64 of columns t / 64 + 4 j; the next chunk's loads are in flight over this one's products
  constexpr int kLoads = kGramTile * kGramRows / (kGramTile * kGramTile);
  const int row = threadIdx.x % kGramRows, col = threadIdx.x / kGramRows;
  const long long chunks = (n + kGramRows - 1) / kGramRows;
  float ra[kLoads], rb[kLoads], ma[kLoads], mb[kLoads];
  auto fetch = [&](long long ch) {
    const long long r = ch * kGramRows + row;
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      const int ca = ta * kGramTile + col + j * (kGramTile / kLoads), cb = tb * kGramTile + col + j * (kGramTile / kLoads);
      ra[j] = (r < n && ca < p) ? X[(long long)ca * n + r] : ma[j];
      rb[j] = (r < n && cb < p) ? X[(long long)cb * n + r] : mb[j];
    }
  };
#pragma unroll
  for (int j = 0; j < kLoads; ++j) {
    const int ca = ta * kGramTile + col + j * (kGramTile / kLoads), cb = tb * kGramTile + col + j * (kGramTile / kLoads);
    ma[j] = ca < p ? mean[ca] : 0.0f;
    mb[j] = cb < p ? mean[cb] : 0.0f;
  }
  fetch(blockIdx.y);
  for (long long ch = blockIdx.y; ch < chunks; ch += gridDim.y) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      sa[col + j * (kGramTile / kLoads)][row] = (ra[j] - ma[j]) * unit;
      sb[col + j * (kGramTile / kLoads)][row] = (rb[j] - mb[j]) * unit;
    }
    __syncthreads();
    fetch(ch + gridDim.y);
#pragma unroll 4
    for (int r = 0; r < kGramRows; r += 4) {
      const float4 u = *(const float4*)&sa[la][r], v = *(const float4*)&sb[lb][r];
      product(u.x, v.x);
      product(u.y, v.y);
      product(u.z, v.z);
      product(u.w, v.w);
    }
    acc = two_sum(acc.hi, acc.lo);
  }
  if (a < p && b < p) {
    const double v = value(acc);
    partial[((long long)blockIdx.y * p + a) * p + b] = v;
    partial[((long long)blockIdx.y * p + b) * p + a] = v;
  }
}

// C = sum of the partials: eight warps share the slices of 32 entries.
__global__ void __launch_bounds__(256)
pca_gram_sum_kernel(const double* __restrict__ partial, int p, int slices, double* __restrict__ C) {
  __shared__ double s_sum[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = blockIdx.x * 32 + lane;
  double sum = 0.0;
  if (t < p * p) {
#pragma unroll 4
    for (int y = warp; y < slices; y += 8) sum += partial[(long long)y * p * p + t];
  }
  s_sum[warp][lane] = sum;
  __syncthreads();
  if (warp == 0 && t < p * p) {
    for (int w = 1; w < 8; ++w) sum += s_sum[w][lane];
    C[t] = sum;
  }
}

// The members i < j of pair k at a step of the round-robin ordering over m (even) indices.
__device__ __forceinline__ int2 jacobi_pair(int k, int step, int m) {
  int u = k + step, w = m - 1 - k + step;  // positions k and m - 1 - k around the circle 1 .. m - 1
  if (u >= m) u -= m - 1;
  if (w >= m) w -= m - 1;
  if (k == 0) u = 0;
  return make_int2(min(u, w), max(u, w));
}

// Cosine and sine of the rotation with tangent t (|t| <= 1), orthonormal to two-float precision: one Newton
// step c0 + c0 (1 - (1 + t^2) c0^2) / 2 and its second-order term on the float reciprocal root.
__device__ __forceinline__ void jacobi_angle(float t, Float2Sum& c, Float2Sum& s) {
  const float tt = __fmul_rn(t, t), c0 = rsqrtf(1.0f + tt);
  const Float2Sum r = mul(mul(add(Float2Sum{tt, __fmaf_rn(t, t, -tt)}, 1.0f), c0), c0);
  const float e = add(Float2Sum{-r.hi, -r.lo}, 1.0f).hi;
  c = two_sum(c0, __fmul_rn(c0, __fmaf_rn(0.375f * e, e, 0.5f * e)));
  s = mul(c, t);
}

// (x, y) <- (c x - s y, s x + c y)
__device__ __forceinline__ void jacobi_rotate(Float2Sum& x, Float2Sum& y, Float2Sum c, Float2Sum s) {
  auto combine = [](Float2Sum a, Float2Sum v, Float2Sum b, Float2Sum w) {  // a v + b w
    const float q = __fmul_rn(a.hi, v.hi), r = __fmul_rn(b.hi, w.hi);
    const Float2Sum t = two_sum(q, r);
    const float lo = __fmaf_rn(a.hi, v.lo, __fmaf_rn(a.lo, v.hi, __fmaf_rn(a.hi, v.hi, -q)));
    const float l2 = __fmaf_rn(b.hi, w.lo, __fmaf_rn(b.lo, w.hi, __fmaf_rn(b.hi, w.hi, -r)));
    const float l = __fadd_rn(t.lo, __fadd_rn(lo, l2)), hi = __fadd_rn(t.hi, l);
    return Float2Sum{hi, __fsub_rn(l, __fsub_rn(hi, t.hi))};
  };
  const Float2Sum u = combine(c, x, Float2Sum{-s.hi, -s.lo}, y);
  y = combine(s, x, c, y);
  x = u;
}

// The eigenvalues of the symmetric p x p matrix C by cyclic Jacobi, one block, and the rotations. Only the upper
// triangle of A is kept (m x m, m = p rounded up to even; in shared memory, or in `work` beyond
// kJacobiSharedFeatures). Round-robin ordering: step t pairs position 0 with position m - 1 and the others
// around a circle; a step's m/2 disjoint rotations are applied together, J^T A J as one update of the 2 x 2
// blocks of (pair, pair). The eigenvectors are the product of all rotations, whose tangents are kept
// (`tangents`, kJacobiSweeps (m - 1) m / 2 floats) for the kernel below, instead of carrying all of V along. A tangent
// is FP32: an angle a little off leaves a little of the entry to the next sweep. Stops when the off-diagonal mass is
// below 1e-26 of the diagonal mass (entries below 2^-43 of the spectrum), or after kJacobiSweeps sweeps.
// lambda: the eigenvalues; info: the indices of the two largest, the number of steps, and whether an eigenvalue lies within
// kCloseGap of one of the two (of the largest).
//
// p = 50 (200,000 rows): 1916 us with A and V in FP64 in global memory, 194 us now and 41 for the vectors, bound by the
// latency of the two dependent phases of a step; the whole start of 5,000 x 150: 90.8 ms, 6.2 now; x 300, with A in
// global memory: 1,516 ms, 131 now.
template <bool kShared>
__global__ void __launch_bounds__(kJacobiThreads)
pca_jacobi_kernel(const double* __restrict__ C, int p, Float2Sum* __restrict__ work, float* __restrict__ tangents,
                  double* __restrict__ lambda, int* __restrict__ info) {
  extern __shared__ Float2Sum s_a[];
  __shared__ int2 s_pair[kJacobiThreads];
  __shared__ float4 s_rot[kJacobiThreads];  // c, s
  __shared__ float s_red[2][kJacobiThreads / 32];
  __shared__ bool s_done;
  __shared__ int s_lead[2];
  Float2Sum* A = kShared ? s_a : work;
  const int m = p + (p & 1), half = m / 2;
  double top = 0.0;  // scaled by a power of two to a largest diagonal entry near 1
  for (int t = 0; t < p; ++t) top = fmax(top, C[(long long)t * p + t]);
  const double unit = top > 0.0 && isfinite(top) ? scalbn(1.0, -ilogb(top)) : 1.0;
  for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
    const int r = t / m, c = t % m;
    A[t] = r < p && c < p ? split(C[(long long)r * p + c] * unit) : Float2Sum{0.0f, 0.0f};
  }
  __syncthreads();
  auto at = [&](int i, int j) -> Float2Sum& { return A[min(i, j) * m + max(i, j)]; };
  // The triangle of blocks (k1 <= k2), folded into rows of half + 1: row r, then row half - 1 - r (the
  // middle row of an odd number stands alone).
  const int items = (half + 1) / 2 * (half + 1);
  auto block_of = [&](int t) {
    const int r = t / (half + 1), c = t % (half + 1);
    if (c < half - r) return make_int2(r, r + c);
    return 2 * r == half - 1 ? make_int2(-1, -1) : make_int2(half - 1 - r, c - 1);
  };
  const int2 first = block_of(threadIdx.x);  // most threads have one block: found once
  int steps = 0;  // taken so far
  for (int sweep = 0; sweep < kJacobiSweeps; ++sweep) {
    float off = 0.0f, dia = 0.0f;
    for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
      const int r = t / m, c = t % m;
      const float v = A[t].hi;
      if (r == c) dia += v * v;
      else if (r < c) off += 2.0f * v * v;
    }
    off = warp_sum(off);
    dia = warp_sum(dia);
    if ((threadIdx.x & 31) == 0) {
      s_red[0][threadIdx.x >> 5] = off;
      s_red[1][threadIdx.x >> 5] = dia;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      float o = 0.0f, d = 0.0f;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        o += s_red[0][w];
        d += s_red[1][w];
      }
      s_done = !(o > 1e-26f * d);
    }
    __syncthreads();
    if (s_done) break;
    for (int step = 0; step < m - 1; ++step, ++steps) {
      for (int k = threadIdx.x; k < half; k += blockDim.x) {
        const int2 q = jacobi_pair(k, step, m);
        const Float2Sum aij = A[q.x * m + q.y], aii = A[q.x * m + q.x], ajj = A[q.y * m + q.y];
        float t = 0.0f;
        Float2Sum c{1.0f, 0.0f}, s{0.0f, 0.0f};
        if (aij.hi != 0.0f) {
          // a tau beyond the float range rotates by nothing
          const float tau = __fdividef((ajj.hi - aii.hi) + (ajj.lo - aii.lo), 2.0f * aij.hi);
          const float q = fmaf(tau, tau, 1.0f);
          const float size = __fdividef(1.0f, fabsf(tau) + q * rsqrtf(q));
          t = size > 0.0f ? copysignf(fminf(size, 1.0f), tau) : 0.0f;
          if (t != 0.0f) jacobi_angle(t, c, s);
        }
        tangents[(long long)steps * half + k] = t;
        s_pair[k] = q;
        s_rot[k] = make_float4(c.hi, c.lo, s.hi, s.lo);
      }
      __syncthreads();
      for (int t = threadIdx.x; t < items; t += blockDim.x) {
        const int2 ks = t == (int)threadIdx.x ? first : block_of(t);
        const int k1 = ks.x, k2 = ks.y;
        if (k1 < 0) continue;
        const int2 u = s_pair[k1], v = s_pair[k2];
        const float4 ru = s_rot[k1], rv = s_rot[k2];
        if (ru.z == 0.0f && rv.z == 0.0f) continue;
        const Float2Sum cu{ru.x, ru.y}, su{ru.z, ru.w}, cv{rv.x, rv.y}, sv{rv.z, rv.w};
        Float2Sum a = at(u.x, v.x), b = at(u.x, v.y), d = at(u.y, v.x), e = at(u.y, v.y);
        jacobi_rotate(a, b, cv, sv);
        jacobi_rotate(d, e, cv, sv);
        jacobi_rotate(a, d, cu, su);
        jacobi_rotate(b, e, cu, su);
        at(u.x, v.x) = a;
        at(u.x, v.y) = b;
        if (k1 != k2) at(u.y, v.x) = d;
        at(u.y, v.y) = e;
      }
      __syncthreads();
    }
  }
  if (threadIdx.x == 0) {
    auto above = [&](int a, int b) {
      const Float2Sum x = A[a * m + a], y = A[b * m + b];
      return x.hi > y.hi || (x.hi == y.hi && x.lo > y.lo);
    };
    int b0 = 0, b1 = -1;
    for (int i = 1; i < p; ++i)
      if (above(i, b0)) b0 = i;
    for (int i = 0; i < p; ++i)
      if (i != b0 && (b1 < 0 || above(i, b1))) b1 = i;
    info[0] = b0;
    info[1] = b1;
    info[2] = steps;
    s_lead[0] = b0;
    s_lead[1] = b1;
  }
  __syncthreads();
  const float l0 = A[s_lead[0] * m + s_lead[0]].hi, l1 = A[s_lead[1] * m + s_lead[1]].hi, near = kCloseGap * l0;
  bool close = l0 - l1 < near;
  for (int i = threadIdx.x; i < p; i += blockDim.x)
    if (i != s_lead[0] && i != s_lead[1]) close |= l1 - A[i * m + i].hi < near;
  close = __syncthreads_or(close);
  if (threadIdx.x == 0) info[3] = close;
  for (int i = threadIdx.x; i < p; i += blockDim.x) lambda[i] = value(A[i * m + i]) / unit;
}

// All eigenvectors, vectors[v * p + i]: the rotations applied in reverse to the unit vectors, a warp for each of a
// block's two. x <- J x for each step's J, (x_i, x_j) <- (c x_i + s x_j, -s x_i + c x_j); the block computes the
// rotations of as many steps as it has threads for. Where they are to be refined, the block of a leading vector x_c also
// computes y[c * p + r] = (C x_c)_r. 50 vectors: 41 us, little more than the two leading ones alone took (36).
__global__ void __launch_bounds__(kJacobiThreads)
pca_vectors_kernel(const float* __restrict__ tangents, int p, const int* __restrict__ info,
                   const double* __restrict__ C, Float2Sum* __restrict__ vectors, double* __restrict__ y) {
  __shared__ int2 s_pair[kJacobiThreads];
  __shared__ float4 s_rot[kJacobiThreads];
  __shared__ Float2Sum s_vec[2][kPcaMaxFeatures];
  const int m = p + (p & 1), half = m / 2, first = 2 * (int)blockIdx.x;
  const int comp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (comp < 2)
    for (int i = lane; i < m; i += 32) s_vec[comp][i] = Float2Sum{i == first + comp ? 1.0f : 0.0f, 0.0f};
  const int batch = kJacobiThreads / half;
  for (int last = info[2]; last > 0; last -= batch) {
    const int count = min(batch, last), g = threadIdx.x / half, k = threadIdx.x - g * half;
    if (g < count) {
      const int done = last - 1 - g;
      const float t = tangents[(long long)done * half + k];
      Float2Sum c{1.0f, 0.0f}, s{0.0f, 0.0f};
      if (t != 0.0f) jacobi_angle(-t, c, s);
      s_pair[threadIdx.x] = jacobi_pair(k, done % (m - 1), m);
      s_rot[threadIdx.x] = make_float4(c.hi, c.lo, s.hi, s.lo);
    }
    __syncthreads();
    if (comp < 2) {
      Float2Sum* vec = s_vec[comp];
      for (int q = 0; q < count; ++q) {
        for (int j = q * half + lane; j < (q + 1) * half; j += 32) {
          const float4 r = s_rot[j];
          if (r.z == 0.0f) continue;
          const int2 u = s_pair[j];
          jacobi_rotate(vec[u.x], vec[u.y], Float2Sum{r.x, r.y}, Float2Sum{r.z, r.w});
        }
        __syncwarp();
      }
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < 2 * p; i += blockDim.x) {
    const int v = i / p;
    if (first + v < p) vectors[(long long)(first + v) * p + i % p] = s_vec[v][i % p];
  }
  if (!info[3]) return;
  for (int c = 0; c < 2; ++c) {
    const int v = info[c] - first;
    if (v < 0 || v > 1) continue;
    for (int r = comp; r < p; r += kJacobiThreads / 32) {
      double t = 0.0;
      for (int i = lane; i < p; i += 32) t += C[(long long)r * p + i] * value(s_vec[v][i]);
      t = warp_sum(t);
      if (lane == 0) y[c * p + r] = t;
    }
  }
}

// One step of Ogita and Aishima's refinement (2018) for the two leading eigenvectors x_c: with S = X^T C X and
// R = I - X^T X in FP64, x_c gains sum over i of e_ic x_i, e_ic = (S_ic + lambda_c R_ic) / (lambda_c - lambda_i), or
// R_ic / 2 for an eigenvalue that cannot be told from lambda_c. It squares the error, which in two floats is some 1e-13
// over the gap of the eigenvalues: with a gap of 1e-7 of the largest, a start of 151 features was off by 5e-7 of its
// largest coordinate, 7e-8 now (6e-8 is the rounding to float). Where no eigenvalue is that close (info[3]) the vectors
// are good to 1e-9 as they are. vectors[c * p + i] = component c; a block takes 32 coordinates, for which its warps form
// every e_ic and share the sums.
__global__ void __launch_bounds__(kJacobiThreads)
pca_refine_kernel(const Float2Sum* __restrict__ X, const double* __restrict__ y, int p,
                  const double* __restrict__ lambda, const int* __restrict__ info, Float2Sum* __restrict__ vectors) {
  constexpr int kWarps = kJacobiThreads / 32;
  __shared__ double s_e[2][kPcaMaxFeatures], s_sum[kWarps][2][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, at = blockIdx.x * 32 + lane;
  const int lead[2] = {info[0], info[1]};
  double t[2] = {0.0, 0.0};
  if (info[3]) {
    for (int q = warp; q < 2 * p; q += kWarps) {
      const int c = q / p, i = q - c * p;
      const Float2Sum *x = X + (long long)i * p, *xc = X + (long long)lead[c] * p;
      double s = 0.0, r = 0.0;
      for (int j = lane; j < p; j += 32) {
        const double v = value(x[j]);
        s += v * y[c * p + j];
        r += v * value(xc[j]);
      }
      s = warp_sum(s);
      r = (i == lead[c] ? 1.0 : 0.0) - warp_sum(r);
      const double gap = lambda[lead[c]] - lambda[i];
      if (lane == 0)
        s_e[c][i] = fabs(gap) > 1e-12 * fabs(lambda[lead[0]]) ? (s + lambda[lead[c]] * r) / gap : 0.5 * r;
    }
    __syncthreads();
    if (at < p)
      for (int j = warp; j < p; j += kWarps) {
        const double v = value(X[(long long)j * p + at]);
        t[0] += s_e[0][j] * v;
        t[1] += s_e[1][j] * v;
      }
  }
  s_sum[warp][0][lane] = t[0];
  s_sum[warp][1][lane] = t[1];
  __syncthreads();
  if (warp >= 2 || at >= p) return;
  double sum = 0.0;
  for (int w = 0; w < kWarps; ++w) sum += s_sum[w][warp][lane];
  vectors[warp * p + at] = split(value(X[(long long)lead[warp] * p + at]) + sum);
}

struct ArgMax {
  double v;
  long long i;
};

// Scores (two-float sums over the features of the scaled data) and block partial argmax |score| per
// component. 200,000 x 50: 77 us with FP64 sums, 29 us now.
__global__ void __launch_bounds__(256)
pca_scores_kernel(const float* __restrict__ X, const float* __restrict__ mean, const int* __restrict__ status, int n,
                  int p, const Float2Sum* __restrict__ V, double2* __restrict__ sc, ArgMax* __restrict__ part) {
  __shared__ ArgMax s_m[2][32];
  __shared__ float4 s_v[kPcaMaxFeatures];  // component 0 high, low, component 1 high, low
  __shared__ float s_mean[kPcaMaxFeatures];
  for (int a = threadIdx.x; a < p; a += blockDim.x) {
    s_v[a] = make_float4(V[a].hi, V[a].lo, V[p + a].hi, V[p + a].lo);
    s_mean[a] = mean[a];
  }
  const int ex = data_exponent(status[1]);
  const float unit = scalbnf(1.0f, -ex);
  const double back = scalbn(1.0, ex);
  __syncthreads();
  ArgMax m0{-1.0, 0}, m1{-1.0, 0};
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    Float2Sum fx{0.0f, 0.0f}, fy{0.0f, 0.0f};
#pragma unroll 4
    for (int a = 0; a < p; ++a) {
      const float v = (X[(long long)a * n + r] - s_mean[a]) * unit;
      const float4 w = s_v[a];
      fx = add(fx, mul(Float2Sum{w.x, w.y}, v));
      fy = add(fy, mul(Float2Sum{w.z, w.w}, v));
    }
    const double x = value(fx) * back, y = value(fy) * back;
    sc[r] = make_double2(x, y);
    if (fabs(x) > m0.v) m0 = ArgMax{fabs(x), r};
    if (fabs(y) > m1.v) m1 = ArgMax{fabs(y), r};
  }
  // first index among equal maxima: compare (value desc, index asc)
  for (int o = 16; o > 0; o >>= 1) {
    const double v0 = __shfl_down_sync(0xffffffffu, m0.v, o), v1 = __shfl_down_sync(0xffffffffu, m1.v, o);
    const long long i0 = __shfl_down_sync(0xffffffffu, m0.i, o), i1 = __shfl_down_sync(0xffffffffu, m1.i, o);
    if (v0 > m0.v || (v0 == m0.v && i0 < m0.i)) m0 = ArgMax{v0, i0};
    if (v1 > m1.v || (v1 == m1.v && i1 < m1.i)) m1 = ArgMax{v1, i1};
  }
  if ((threadIdx.x & 31) == 0) {
    s_m[0][threadIdx.x >> 5] = m0;
    s_m[1][threadIdx.x >> 5] = m1;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    ArgMax best{-1.0, 0};
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      const ArgMax q = s_m[threadIdx.x][w];
      if (q.v > best.v || (q.v == best.v && q.i < best.i)) best = q;
    }
    part[blockIdx.x * 2 + threadIdx.x] = best;
  }
}

// Signed float scores (each component's largest in magnitude positive; non-finite -> 0) and the blocks' partial moments (sums of x, y, x^2, y^2 of the
// scores over the data's power of two). One block of FP64 sums and the scaling took 1144 us for 200,000
// rows; the two kernels take 26 us.
__global__ void __launch_bounds__(256)
pca_moments_kernel(const double2* __restrict__ sc, const int* __restrict__ status, int n,
                   const ArgMax* __restrict__ largest, int nlargest, float2* __restrict__ init,
                   double* __restrict__ part) {
  __shared__ Float2Sum s_red[4][8];
  __shared__ float s_sign[2];
  if (threadIdx.x < 64) {  // a warp per component
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
    ArgMax best{-1.0, 0};
    for (int b = lane; b < nlargest; b += 32) {
      const ArgMax q = largest[b * 2 + c];
      if (q.v > best.v || (q.v == best.v && q.i < best.i)) best = q;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double v = __shfl_xor_sync(0xffffffffu, best.v, o);
      const long long i = __shfl_xor_sync(0xffffffffu, best.i, o);
      if (v > best.v || (v == best.v && i < best.i)) best = ArgMax{v, i};
    }
    if (lane == 0) s_sign[c] = (c == 0 ? sc[best.i].x : sc[best.i].y) < 0.0 ? -1.0f : 1.0f;
  }
  __syncthreads();
  const float sx = s_sign[0], sy = s_sign[1];
  const float unit = scalbnf(1.0f, -data_exponent(status[1]));
  Float2Sum m[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) m[c] = Float2Sum{0.0f, 0.0f};
  for (int r = blockIdx.x * 256 + threadIdx.x; r < n; r += gridDim.x * 256) {
    const double2 v = sc[r];
    float x = sx * (float)v.x, y = sy * (float)v.y;
    if (!isfinite(x)) x = 0.0f;
    if (!isfinite(y)) y = 0.0f;
    init[r] = make_float2(x, y);
    x *= unit;
    y *= unit;
    const float xx = __fmul_rn(x, x), yy = __fmul_rn(y, y);
    m[0] = add(m[0], x);
    m[1] = add(m[1], y);
    m[2] = add(m[2], Float2Sum{xx, __fmaf_rn(x, x, -xx)});
    m[3] = add(m[3], Float2Sum{yy, __fmaf_rn(y, y, -yy)});
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const Float2Sum v = warp_sum(m[c]);
    if ((threadIdx.x & 31) == 0) s_red[c][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    Float2Sum t = s_red[threadIdx.x][0];
    for (int w = 1; w < 8; ++w) t = add(t, s_red[threadIdx.x][w]);
    part[blockIdx.x * 4 + threadIdx.x] = value(t);
  }
}

// The reference's t-SNE scaling: (v - mean) * 1e-4 / max sd.
__global__ void __launch_bounds__(256)
pca_scale_kernel(float2* __restrict__ init, const int* __restrict__ status, int n, const double* __restrict__ part,
                 int nparts) {
  __shared__ double s_t[4];
  __shared__ double s_stat[3];
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (c < 4) {
    double t = 0.0;
    for (int b = lane; b < nparts; b += 32) t += part[b * 4 + c];
    t = warp_sum(t);
    const int ex = data_exponent(status[1]);
    if (lane == 0) s_t[c] = scalbn(t, c < 2 ? ex : 2 * ex);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double dn = (double)max(n, 1), den = (double)max(n - 1, 1);
    const double ssx = fmax(s_t[2] - s_t[0] * s_t[0] / dn, 0.0), ssy = fmax(s_t[3] - s_t[1] * s_t[1] / dn, 0.0);
    const double sd = fmax(sqrt(ssx / den), sqrt(ssy / den));
    s_stat[0] = s_t[0] / dn;
    s_stat[1] = s_t[1] / dn;
    s_stat[2] = (isfinite(sd) && sd > 0.0) ? 1.0e-4 / sd : 1.0;
  }
  __syncthreads();
  for (int r = blockIdx.x * 256 + threadIdx.x; r < n; r += gridDim.x * 256) {
    const float2 v = init[r];
    init[r] = make_float2((float)(((double)v.x - s_stat[0]) * s_stat[2]), (float)(((double)v.y - s_stat[1]) * s_stat[2]));
  }
}

}  // namespace

void pca_tsne_start(const float* X, int n, int p, float2* init, cudaStream_t s) {
  if (n < 2 || p < 2) throw Error("invalid dimensions in device PCA initialization");
  if (p > kPcaMaxFeatures)
    throw Error("device PCA initialization supports at most 1024 features; reduce the dimension first");
  const int tiles = ceil_div(p, kGramTile);
  const int tri = tiles * (tiles + 1) / 2;
  const int slices = std::max(1, std::min({kGramSlices, ceil_div(n, kGramRows), sm_count() * 4 / tri}));
  const int sblocks = std::max(1, std::min(ceil_div(n, 256), sm_count() * 4));
  const int mblocks = std::max(1, std::min(ceil_div(n, 1024), sm_count() * 2));
  const int mslices = std::max(1, std::min(kMeanSlices, ceil_div(n, 1024)));
  const std::size_t m = p + (p & 1);
  const bool shared = p <= kJacobiSharedFeatures;
  double *sums = nullptr, *partial = nullptr, *C = nullptr, *moments = nullptr;
  double *lambda = nullptr, *y = nullptr;
  float *mean = nullptr, *tangents = nullptr;
  float2* range = nullptr;
  Float2Sum *work = nullptr, *all = nullptr, *V = nullptr;
  double2* sc = nullptr;
  ArgMax* am = nullptr;
  int* info = nullptr;
  int* status = nullptr;  // non-finite data, bits of the largest centred magnitude
  Arena w;
  w.reserve(&sums, (std::size_t)p * mslices);
  w.reserve(&range, (std::size_t)p * mslices);
  w.reserve(&mean, p);
  w.reserve(&partial, (std::size_t)slices * p * p);
  w.reserve(&C, (std::size_t)p * p);
  w.reserve(&work, shared ? 1 : m * m);
  w.reserve(&tangents, kJacobiSweeps * (m - 1) * (m / 2));
  w.reserve(&lambda, p);
  w.reserve(&info, 4);
  w.reserve(&all, (std::size_t)p * p);
  w.reserve(&y, 2 * (std::size_t)p);
  w.reserve(&V, 2 * (std::size_t)p);
  w.reserve(&sc, n);
  w.reserve(&am, 2 * (std::size_t)sblocks);
  w.reserve(&status, 2);
  w.reserve(&moments, 4 * (std::size_t)mblocks);
  w.commit("device PCA initialization");
  FE_CUDA(cudaMemsetAsync(status, 0, 2 * sizeof(int), s));
  pca_sum_kernel<<<dim3(p, mslices), 256, 0, s>>>(X, n, sums, range, status);
  FE_LAUNCH("pca_sum_kernel");
  pca_mean_kernel<<<ceil_div(p, 128), 128, 0, s>>>(sums, range, p, mslices, n, mean, status);
  FE_LAUNCH("pca_mean_kernel");
  int h_bad = 0;
  FE_CUDA(cudaMemcpyAsync(&h_bad, status, sizeof(int), cudaMemcpyDeviceToHost, s));
  FE_CUDA(cudaStreamSynchronize(s));
  if (h_bad) throw Error("PCA input must contain only finite values");
  pca_gram_kernel<<<dim3(tri, slices), kGramTile * kGramTile, 0, s>>>(X, mean, status, n, p,
                                                                                         partial);
  FE_LAUNCH("pca_gram_kernel");
  pca_gram_sum_kernel<<<ceil_div(p * p, 32), 256, 0, s>>>(partial, p, slices, C);
  FE_LAUNCH("pca_gram_sum_kernel");
  if (shared) {
    const int smem = (int)(m * m * sizeof(Float2Sum));
    allow_dynamic_shared((const void*)pca_jacobi_kernel<true>, smem,
                         kJacobiSharedFeatures * kJacobiSharedFeatures * sizeof(Float2Sum));
    pca_jacobi_kernel<true><<<1, kJacobiThreads, smem, s>>>(C, p, work, tangents, lambda, info);
  } else {
    pca_jacobi_kernel<false><<<1, kJacobiThreads, 0, s>>>(C, p, work, tangents, lambda, info);
  }
  FE_LAUNCH("pca_jacobi_kernel");
  pca_vectors_kernel<<<ceil_div(p, 2), kJacobiThreads, 0, s>>>(tangents, p, info, C, all, y);
  FE_LAUNCH("pca_vectors_kernel");
  pca_refine_kernel<<<ceil_div(p, 32), kJacobiThreads, 0, s>>>(all, y, p, lambda, info, V);
  FE_LAUNCH("pca_refine_kernel");
  pca_scores_kernel<<<sblocks, 256, 0, s>>>(X, mean, status, n, p, V, sc, am);
  FE_LAUNCH("pca_scores_kernel");
  pca_moments_kernel<<<mblocks, 256, 0, s>>>(sc, status, n, am, sblocks, init, moments);
  FE_LAUNCH("pca_moments_kernel");
  pca_scale_kernel<<<mblocks, 256, 0, s>>>(init, status, n, moments, mblocks);
  FE_LAUNCH("pca_scale_kernel");
  FE_CUDA(cudaStreamSynchronize(s));
}

}  // namespace fe
