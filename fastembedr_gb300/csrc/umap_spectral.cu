// Spectral start of UMAP on the GPU.
//
// Restates initialize_layout_csr (src/fast_knn_umap.cpp:2231-2528), as optimize_layout_csr
// (:3088-3205) calls it for spectral_knn_init(backend = "cpu") / umap_init: the symmetric
// normalised adjacency D^-1/2 W D^-1/2 of the fuzzy graph, a block of 8 vectors drawn from the
// reference's std::mt19937 / normal(0, 1e-4) x 1e4 stream, spectral_n_iter rounds of
// multiply + modified Gram-Schmidt against the trivial eigenvector sqrt(deg) / |sqrt(deg)| and
// the earlier columns, a Rayleigh-Ritz step (the 8 x 8 projected matrix, diagonalised by the
// reference's largest-off-diagonal Jacobi rotations), the two leading Ritz vectors centred,
// scaled to max |y| = 10 and jittered by the stream's normal(0, 1e-4) draws
// (scale_embedding_max_abs_and_jitter, :2705-2730), then the optional scale_embedding_sdev
// (:2681-2703).
//
// The random draws are made in the reference's order (on the host, or the start block of a large layout on
// the GPU; the column redraw of a vanishing Gram-Schmidt column included); every arithmetic step runs on the GPU in
// FP64, in a fixed order, so that results are deterministic; they differ from the CPU's by rounding. Degrees, the
// normalisation and the steps after the rounds follow the reference's operations without contraction (__d*_rn) but for
// sums over points, which go by blocks. The rounds do not: a row's products are fused into its sum and split over lanes, a
// pass orthonormalises by Cholesky QR (Gram-Schmidt where a column vanishes, with its products not fused), and a Ritz
// rotation takes its angle with one division and a reciprocal root. Against a restatement in long double on graphs of 600
// and 1,500 points (well mixed, clustered, with eigenvalues next to 1) the start is as close as with Gram-Schmidt in the
// reference's order, 1e-13 to 1e-6 of a layout of 10 for either.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <future>
#include <random>
#include <vector>

#include "umap_spectral.cuh"

namespace fe {
namespace {

constexpr int kSpThreads = 256;
constexpr int kSpMaxBlocks = 1024;
constexpr int kSpBlock = 8;                           // block size of the reference for 2 components
constexpr int kSpPairs = kSpBlock * (kSpBlock + 1) / 2;  // upper triangle of the projected matrix

int sp_blocks(int n) { return std::max(1, std::min(ceil_div(n, kSpThreads), kSpMaxBlocks)); }

// Fixed-order sum of `count` partials, valid in every thread of the block (all threads call). The
// loads go to L2: the partials may come from other blocks of the same launch.
__device__ double sum_partials(const double* __restrict__ part, int count) {
  __shared__ double s_total;
  if (threadIdx.x < 32) {
    double s = 0.0;
    int b = threadIdx.x;
    // the lane's partials in order; eight loads are issued before their adds
    for (; b + 7 * 32 < count; b += 8 * 32) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldcg(part + b + u * 32);
#pragma unroll
      for (int u = 0; u < 8; ++u) s = __dadd_rn(s, v[u]);
    }
    for (; b < count; b += 32) s = __dadd_rn(s, __ldcg(part + b));
    s = warp_sum(s);
    if (threadIdx.x == 0) s_total = s;
  }
  __syncthreads();
  const double r = s_total;
  __syncthreads();
  return r;
}

// Block sum of v into *dst (fixed order: warp trees, then warps in order).
__device__ void block_partial_at(double v, double* __restrict__ dst) {
  __shared__ double s_w[kSpThreads / 32];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = __dadd_rn(t, s_w[w]);
    *dst = t;
  }
}

__device__ void block_partial(double v, double* __restrict__ part) { block_partial_at(v, part + blockIdx.x); }

// deg[r] = float(sum of row r's weights in double)
__global__ void sp_degree_kernel(const int* __restrict__ offsets, const float* __restrict__ w, int n,
                                 float* __restrict__ deg) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int p = offsets[r]; p < offsets[r + 1]; ++p) s = __dadd_rn(s, (double)w[p]);
    deg[r] = (float)s;
  }
}

// nw[p] = float(w / sqrt(max(deg_r deg_j, 1e-24))): one warp per row, lanes over its entries. (Entries are numbered
// unsigned where a step may go beyond a row that ends near 2^31.)
__global__ void __launch_bounds__(kSpThreads)
sp_adjacency_kernel(const int* __restrict__ offsets, const int* __restrict__ nb, const float* __restrict__ w,
                    const float* __restrict__ deg, int n, float* __restrict__ nw) {
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps) {
    const double dr = (double)deg[r];
    for (unsigned p = offsets[r] + lane, end = offsets[r + 1]; p < end; p += 32) {
      const double den = __dsqrt_rn(fmax(__dmul_rn(dr, (double)deg[nb[p]]), 1e-24));
      nw[p] = (float)__ddiv_rn((double)w[p], den);
    }
  }
}

// triv[r] = sqrt(max(deg_r, 0)); block partials of sum triv^2 (one thread per row, grid-stride
// with a fixed row-to-block assignment).
__global__ void __launch_bounds__(kSpThreads)
sp_trivial_kernel(const float* __restrict__ deg, int n, double* __restrict__ triv, double* __restrict__ part) {
  double acc = 0.0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const double t = __dsqrt_rn(fmax((double)deg[r], 0.0));
    triv[r] = t;
    acc = __dadd_rn(acc, __dmul_rn(t, t));
  }
  block_partial(acc, part);
}

__global__ void sp_normalise_trivial_kernel(double* __restrict__ triv, int n, const double* __restrict__ part,
                                            int nparts) {
  const double nrm = __dsqrt_rn(fmax(sum_partials(part, nparts), 1e-12));
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    triv[r] = __ddiv_rn(triv[r], nrm);
}

// ---------------------------------------------------------------- subspace iteration
//
// The block subspace iteration runs as one cooperative launch: all rounds of multiply and
// orthonormalisation. Block vb of `nparts` owns the rows (k nparts + vb) points + t, t < points, of every tile k: it
// multiplies them and keeps their B values in shared memory through the pass (as long as kSpSharedRows hold
// them; in the global buffers beyond). Blocks exchange sums without a barrier: a partial is published with the
// exchange's number in the same words, and whoever needs the sum polls for all partials and adds them in
// block order. `points` and `nparts` follow from n and the number of SMs, so the sums do not depend on the launch.
// Columns written during the launch are read through L2 (__ldcg): another block may have written them, and L1
// is not coherent.
//
// A pass forms all 44 products of the columns with each other and with the trivial vector at once, eliminates
// the 8 x 8 matrix in every block and applies the triangular factor (Cholesky QR: the same columns as the
// reference's modified Gram-Schmidt up to rounding, times the square of the columns' condition). Where
// a column keeps less than a tenth of its norm, or nearly vanishes, the pass runs as modified Gram-Schmidt in the
// reference's steps instead, which also decides on redraws.
//
// What bounds a round is the FP64 pipe (a warp instruction in 19 cycles of an SM) and the latency of the exchanges.
// 20,000 points, 30 rounds: 6.45 ms as 18 grid barriers a round around Gram-Schmidt steps on 79 blocks that
// re-read their columns through L2; 4.76 ms with the rows in shared memory on 126 blocks and 17 exchanges a
// round; 1.46 ms now.

constexpr long long kSpWaitCycles = 4000000000LL;  // about 2 s at the SM clock
constexpr int kSpRoundThreads = 512;
constexpr int kSpParts = 152;         // blocks, at most (one per SM, or as many as there are SMs)
constexpr int kSpSharedRows = 3456;   // rows of a block in shared memory: 64 bytes each, 216 KB

// Tiles of a block and rows per tile for at most `blocks` blocks: each has its share, of a warp's width at least.
int sp_tiles(int n, int blocks) { return ceil_div(n, (long long)blocks * kSpRoundThreads); }
int sp_points(int n, int blocks) { return std::max(32, ceil_div(n, (long long)blocks * sp_tiles(n, blocks))); }

struct SpGrid {
  int error;   // 1: a wait gave up
  int status;  // -1, or 16 * (round + 1) + column of a vanished Gram-Schmidt column
};

// A published partial: the low and high half of the double, each beside the exchange's number. A 64-bit store is
// seen whole, so a reader that finds the number in both words has the value.
struct SpSlot {
  unsigned long long lo, hi;
};

__device__ __forceinline__ void sp_publish(SpSlot* slot, double v, unsigned gen) {
  const unsigned long long tag = (unsigned long long)gen << 32;
  *(volatile unsigned long long*)&slot->lo = tag | (unsigned)__double2loint(v);
  *(volatile unsigned long long*)&slot->hi = tag | (unsigned)__double2hiint(v);
}

// Waits for exchange `gen` in the slot; false after kSpWaitCycles, or when another block gave up.
__device__ __forceinline__ bool sp_collect(const SpSlot* slot, unsigned gen, SpGrid* grid, double& v) {
  const long long t0 = clock64();
  for (int spins = 0;; ++spins) {
    const unsigned long long lo = *(const volatile unsigned long long*)&slot->lo;
    const unsigned long long hi = *(const volatile unsigned long long*)&slot->hi;
    if ((unsigned)(lo >> 32) == gen && (unsigned)(hi >> 32) == gen) {
      v = __hiloint2double((int)(unsigned)hi, (int)(unsigned)lo);
      return true;
    }
    if ((spins & 255) == 255 && (*(volatile int*)&grid->error != 0 || clock64() - t0 > kSpWaitCycles)) {
      atomicExch(&grid->error, 1);
      return false;
    }
  }
}

// Shared state of a block.
constexpr int kSpProducts = kSpBlock + kSpPairs;  // trivial x column, then the upper triangle column x column
struct SpShared {
  double red[kSpProducts + 4][kSpRoundThreads / 32];  // the warps' partials of each sum
  double gram[kSpProducts];
  double w[kSpBlock][kSpBlock];  // the triangular factor: new column c = sum over a <= c of w[a][c] x_a + wt[c] triv
  double wt[kSpBlock];
  int usable;
  double total[kSpBlock];                      // the columns' sums over all rows
  double norm, inverse;                        // of the column that becomes final
  int failed;
};

// Exchange number `gen` (1, 2, ...): publishes the block's partials of the columns in `mask` and leaves their
// sums over all blocks in sh.total, the root of column `pending`'s and its reciprocal in sh.norm and sh.inverse.
// Two sets of slots in turn: a block publishes exchange gen + 2 only after it has read every block's gen + 1,
// which follows that block's reading of gen. With `barrier` (and mask 1) it also orders the memory
// accesses of all blocks before it with those after it. False when a wait gave up.
__device__ bool sp_exchange(SpShared& sh, SpSlot* slots, unsigned gen, unsigned mask, int warps, int nparts,
                            int pending, bool barrier, SpGrid* grid) {
  __syncthreads();
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (c < kSpBlock && ((mask >> c) & 1u)) {
    SpSlot* col = slots + ((gen & 1u) * kSpBlock + c) * kSpParts;
    double v = lane < warps ? sh.red[c][lane] : 0.0;
#pragma unroll
    for (int o = kSpRoundThreads / 64; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) {
      if (barrier) __threadfence();
      sp_publish(col + blockIdx.x, v, gen);
    }
    double t = 0.0;
    bool ok = true;
    for (int b = lane; ok && b < nparts; b += 32) {
      double u = 0.0;
      ok = sp_collect(col + b, gen, grid, u);
      t = __dadd_rn(t, u);
    }
    if (!ok) sh.failed = 1;
    if (barrier) __threadfence();
    t = warp_sum(t);
    if (lane == 0) {
      sh.total[c] = t;
      if (c == pending) {
        const double nrm = __dsqrt_rn(t);
        sh.norm = nrm;
        sh.inverse = __drcp_rn(nrm);
      }
    }
  }
  __syncthreads();
  return sh.failed == 0;
}

// The warp's sums of eight columns: each halving exchange passes half of the columns on, so 4 + 2 + 1 + 1 + 1
// additions do what a tree per column does in 40. Column c's sum ends in lane 4 c.
__device__ __forceinline__ void sp_warp_columns(const double (&acc)[kSpBlock], SpShared& sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double a[4], b[2];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const bool up = (lane & 16) != 0;
    const double give = up ? acc[c] : acc[c + 4], keep = up ? acc[c + 4] : acc[c];
    a[c] = __dadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, 16));
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const bool up = (lane & 8) != 0;
    const double give = up ? a[c] : a[c + 2], keep = up ? a[c + 2] : a[c];
    b[c] = __dadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, 8));
  }
  const bool up = (lane & 4) != 0;
  double v = __dadd_rn(up ? b[1] : b[0], __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4));
  v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
  v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
  if ((lane & 3) == 0) sh.red[lane >> 2][w] = v;
}

// The warp's sums of 48 values: value v < 32 ends in lane v, value 32 + u in lane 2 u.
__device__ __forceinline__ void sp_warp_products(double (&v)[kSpProducts + 4], SpShared& sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int c = 0; c < o; ++c)
      v[c] = __dadd_rn(up ? v[c + o] : v[c], __shfl_xor_sync(0xffffffffu, up ? v[c] : v[c + o], o));
    if (o > 1) {
#pragma unroll
      for (int c = 32; c < 32 + o / 2; ++c)
        v[c] = __dadd_rn(up ? v[c + o / 2] : v[c], __shfl_xor_sync(0xffffffffu, up ? v[c] : v[c + o / 2], o));
    }
  }
  v[32] = __dadd_rn(v[32], __shfl_xor_sync(0xffffffffu, v[32], 1));
  sh.red[lane][w] = v[0];
  if ((lane & 1) == 0) sh.red[32 + (lane >> 1)][w] = v[32];
}

// Sums the products over all blocks into sh.gram, in two hops: the partials of product v are added by warp
// v / nparts of block v % nparts, which publishes the total. (Every block adding all 44 x nparts partials itself
// would cost more on the FP64 pipe than the second hop.) False when a wait gave up.
__device__ bool sp_exchange_products(SpShared& sh, SpSlot* partials, SpSlot* totals, unsigned gen, int warps,
                                     int nparts, SpGrid* grid) {
  __syncthreads();
  const int t = threadIdx.x, lane = t & 31;
  if (t < kSpProducts) {
    double v = sh.red[t][0];
    for (int w = 1; w < warps; ++w) v = __dadd_rn(v, sh.red[t][w]);
    sp_publish(partials + t * kSpParts + blockIdx.x, v, gen);
  }
  __syncwarp();
  for (int v = blockIdx.x + (t >> 5) * nparts; v < kSpProducts; v += (kSpRoundThreads / 32) * nparts) {
    double sum = 0.0;
    bool ok = true;
    for (int b = lane; ok && b < nparts; b += 32) {
      double u = 0.0;
      ok = sp_collect(partials + v * kSpParts + b, gen, grid, u);
      sum = __dadd_rn(sum, u);
    }
    if (!ok) sh.failed = 1;
    sum = warp_sum(sum);
    if (lane == 0) sp_publish(totals + v, sum, gen);
  }
  if (t < kSpProducts) {
    double u = 0.0;
    if (!sp_collect(totals + t, gen, grid, u)) sh.failed = 1;
    sh.gram[t] = u;
  }
  __syncthreads();
  return sh.failed == 0;
}

// The triangular factor from the products, by one warp: elimination of [G | I], G = X^T X less the trivial
// vector's part, without pivoting; lane j < 16 holds column j. Leaves L^-1 in the right half: w = L^-T D^-1/2.
// sh.usable says whether every column keeps a tenth of its norm and 1e-8 (the pass falls back otherwise).
__device__ void sp_factor(SpShared& sh) {
  const int lane = threadIdx.x, j = lane & 15, b = j & (kSpBlock - 1);
  double m[kSpBlock];
#pragma unroll
  for (int i = 0; i < kSpBlock; ++i) {
    const int lo = min(i, b), hi = max(i, b);
    const double g = sh.gram[kSpBlock + lo * kSpBlock - lo * (lo - 1) / 2 + hi - lo];
    m[i] = j < kSpBlock ? __fma_rn(-sh.gram[lo], sh.gram[hi], g) : (i == b ? 1.0 : 0.0);
  }
  const double own = sh.gram[kSpBlock + b * kSpBlock - b * (b - 1) / 2];
  double pivot = 0.0;  // lane c: D_c
#pragma unroll
  for (int c = 0; c < kSpBlock; ++c) {
    const double d = __shfl_sync(0xffffffffu, m[c], c);
    if (j == c) pivot = d;
    const double r = __drcp_rn(d);
#pragma unroll
    for (int i = c + 1; i < kSpBlock; ++i) {
      const double f = __dmul_rn(__shfl_sync(0xffffffffu, m[i], c), r);
      m[i] = __fma_rn(-f, m[c], m[i]);
    }
  }
  const bool good = j >= kSpBlock || (pivot >= 0.01 * own && pivot > 1e-16 && pivot < 1e300);
  const bool usable = __all_sync(0xffffffffu, good);
  const double scale = __drcp_rn(__dsqrt_rn(j < kSpBlock ? pivot : 1.0));
#pragma unroll
  for (int c = 0; c < kSpBlock; ++c) {
    const double v = __dmul_rn(m[c], __shfl_sync(0xffffffffu, scale, c));
    if (lane >= kSpBlock && lane < 2 * kSpBlock) sh.w[b][c] = v;
  }
  __syncwarp();
  if (lane < kSpBlock) {
    double v = 0.0;
    for (int a = 0; a <= lane; ++a) v = __fma_rn(-sh.gram[a], sh.w[a][lane], v);
    sh.wt[lane] = v;
  }
  if (lane == 0) sh.usable = usable;
}

// One column's sum over entries first .. end - 1 of a row by eight lanes (lane & 7 = column): per group of 8
// entries the lanes load the entries' neighbours and weights (one each, the next group's ahead), pass them
// round by shuffles, and every lane gathers its column's 8 values, the next group's before it adds this one's.
// `step` entries apart.
__device__ __forceinline__ double sp_row_sum(const int* __restrict__ nb, const float* __restrict__ nw,
                                             const double* xc, unsigned first, unsigned end, unsigned step,
                                             unsigned gmask) {
  const int c = threadIdx.x & 7;
  auto entry = [&](unsigned p, int& j, double& w) {
    j = p < end ? nb[p] : 0;
    w = p < end ? (double)nw[p] : 0.0;
  };
  auto gather = [&](unsigned base, int j, double (&v)[8]) {
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int jt = __shfl_sync(gmask, j, t, 8);
      v[t] = base + t < end ? __ldcg(xc + jt) : 0.0;
    }
  };
  double acc = 0.0, w, v[8];
  int j;
  entry(first + c, j, w);
  gather(first, j, v);
  for (unsigned base = first; base < end; base += step) {
    int jn;
    double wn, vn[8];
    entry(base + step + c, jn, wn);
    gather(base + step, jn, vn);
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const double wt = __shfl_sync(gmask, w, t, 8);
      if (base + t < end) acc = __fma_rn(wt, v[t], acc);
      v[t] = vn[t];
    }
    w = wn;
  }
  return acc;
}

// y[:, c] = A x[:, c] for the B columns. A warp works on four rows at once, eight lanes per row
// (lane = 8 * slot + column), so that all 32 lanes of a warp instruction on the FP64 pipe carry work; entries
// beyond a row's first kSpRowEntries are shared by the four slots, or the longest rows of a graph (a few hundred
// entries) would hold up a whole block's pass.
constexpr int kSpRowEntries = 32;
template <typename RowOf, typename Store>
__device__ void sp_multiply_rows(const int* __restrict__ offsets, const int* __restrict__ nb,
                                 const float* __restrict__ nw, int n, int B, const double* x, int begin, int end,
                                 int stride, RowOf row_of, Store store) {
  const int lane = threadIdx.x & 31, slot = lane >> 3, c = lane & 7;
  const double* xc = x + (long long)(c < B ? c : 0) * n;
  for (int g0 = begin + (threadIdx.x >> 5) * 4; g0 < end; g0 += stride) {
    const int g = g0 + slot, r = g < end ? row_of(g) : n;
    const unsigned p0 = r < n ? offsets[r] : 0, p1 = r < n ? offsets[r + 1] : 0;
    double acc = sp_row_sum(nb, nw, xc, p0, min(p1, p0 + kSpRowEntries), 8, 0xffu << (slot * 8));
    unsigned longer = __ballot_sync(0xffffffffu, p1 - p0 > kSpRowEntries);
    while (longer) {
      const int who = __ffs(longer) - 1;  // the first lane of a slot
      longer &= ~(0xffu << who);
      const unsigned q0 = __shfl_sync(0xffffffffu, p0, who) + kSpRowEntries, q1 = __shfl_sync(0xffffffffu, p1, who);
      double more = sp_row_sum(nb, nw, xc, q0 + slot * 8, q1, 32, 0xffu << (slot * 8));
      more = __dadd_rn(more, __shfl_xor_sync(0xffffffffu, more, 8));
      more = __dadd_rn(more, __shfl_xor_sync(0xffffffffu, more, 16));
      if (slot == who >> 3) acc = __dadd_rn(acc, more);
    }
    if (r < n && c < B) store(c, g, r, acc);
  }
}

__global__ void __launch_bounds__(kSpThreads)
sp_multiply_kernel(const int* __restrict__ offsets, const int* __restrict__ nb, const float* __restrict__ nw,
                   int n, int B, const double* __restrict__ x, double* __restrict__ y) {
  const int rows = (blockDim.x >> 5) * 4;  // of a block at once
  sp_multiply_rows(
      offsets, nb, nw, n, B, x, blockIdx.x * rows, n, gridDim.x * rows, [](int g) { return g; },
      [&](int c, int, int r, double v) { y[(long long)c * n + r] = v; });
}

// A block's rows of the B columns: in shared memory, or in the global buffer m.
template <bool kShared>
struct SpRows {
  double* s;  // kShared: column-major, `cap` rows
  double* m;
  int n, cap, points, nparts, tiles;
  __device__ int row(int tile, int t) const {  // n: no row
    return t < points ? (tile * nparts + (int)blockIdx.x) * points + t : n;
  }
  __device__ int warps() const { return (points + 31) / 32; }
  __device__ double get(int c, int tile, int i) const {
    return kShared ? s[c * cap + tile * points + threadIdx.x] : __ldcg(m + (long long)c * n + i);
  }
  __device__ void set(int c, int tile, int i, double v) const {
    if (kShared) s[c * cap + tile * points + threadIdx.x] = v;
    else m[(long long)c * n + i] = v;
  }
};

// Cholesky QR of the block's eight columns against each other and the trivial vector; the new columns are
// written to m. 1: done; 0: not usable (the columns are as before); -1: a wait gave up.
template <bool kShared>
__device__ int sp_orthonormalise_at_once(const SpRows<kShared>& rows, const double* __restrict__ triv, SpShared& sh,
                                         SpSlot* slots, SpGrid* grid, unsigned& gen) {
  const int n = rows.n, warps = rows.warps();
  const bool mine = (int)threadIdx.x < 32 * warps;
  if (mine) {
    double acc[kSpProducts + 4];
#pragma unroll
    for (int v = 0; v < kSpProducts + 4; ++v) acc[v] = 0.0;
    for (int k = 0; k < rows.tiles; ++k) {
      const int i = rows.row(k, threadIdx.x);
      if (i >= n) continue;
      const double t = triv[i];
      double x[kSpBlock];
#pragma unroll
      for (int c = 0; c < kSpBlock; ++c) x[c] = rows.get(c, k, i);
      int v = kSpBlock;
#pragma unroll
      for (int a = 0; a < kSpBlock; ++a) {
        acc[a] = __fma_rn(t, x[a], acc[a]);
#pragma unroll
        for (int b = a; b < kSpBlock; ++b, ++v) acc[v] = __fma_rn(x[a], x[b], acc[v]);
      }
    }
    sp_warp_products(acc, sh);
  }
  SpSlot* partials = slots + 2 * kSpBlock * kSpParts;
  if (!sp_exchange_products(sh, partials, partials + kSpProducts * kSpParts, ++gen, warps, rows.nparts, grid))
    return -1;
  if (threadIdx.x < 32) sp_factor(sh);
  __syncthreads();
  if (!sh.usable) return 0;
  if (mine) {
    for (int k = 0; k < rows.tiles; ++k) {
      const int i = rows.row(k, threadIdx.x);
      if (i >= n) continue;
      const double t = triv[i];
      double x[kSpBlock];
#pragma unroll
      for (int c = 0; c < kSpBlock; ++c) x[c] = rows.get(c, k, i);
#pragma unroll
      for (int c = 0; c < kSpBlock; ++c) {
        double v = __dmul_rn(sh.wt[c], t);
#pragma unroll
        for (int a = 0; a <= c; ++a) v = __fma_rn(sh.w[a][c], x[a], v);
        rows.m[(long long)c * n + i] = v;
      }
    }
  }
  return sp_exchange(sh, slots, ++gen, 1u, warps, rows.nparts, -1, true, grid) ? 1 : -1;
}

// Modified Gram-Schmidt of the columns from..B-1 of a block's rows against the trivial vector and the
// columns before them (columns below `from` are final), as a wavefront. Column c's step j (j = 0..c)
// subtracts its last dot times u_j (u_0 = triv, u_j = q_{j-1}) and forms the partials of its dot
// with v_j = q_j, or of its squared norm when j = c; a column is divided by its norm at the start
// of the step after its norm step, and written to m. Step j needs q_j final, so every column whose next
// step has its v final advances in the same step: the pass takes 2 (B - from) + 1 exchanges instead
// of one per projection, and each column sees exactly the operations of the column-by-column
// order. The columns' post-multiply values survive for a redraw: in m (kShared), or copied to `backup`.
// Returns 0 when done, 1 + c when column c vanished, -1 when a wait gave up.
template <bool kShared>
__device__ int sp_orthonormalise(const SpRows<kShared>& rows, double* backup, const double* __restrict__ triv, int B,
                                 int from, SpShared& sh, SpSlot* slots, SpGrid* grid, unsigned& gen) {
  // the first projection of every column, which the earlier columns do not change
  const unsigned all = ((1u << B) - 1u) & ~((1u << from) - 1u);
  const int warps = rows.warps(), n = rows.n;
  const bool mine = (int)threadIdx.x < 32 * warps;
  if (mine) {
    double acc[kSpBlock];
#pragma unroll
    for (int c = 0; c < kSpBlock; ++c) acc[c] = 0.0;
    for (int k = 0; k < rows.tiles; ++k) {
      const int i = rows.row(k, threadIdx.x);
      if (i >= n) continue;
      const double t = triv[i];
#pragma unroll
      for (int c = 0; c < kSpBlock; ++c)
        if ((all >> c) & 1u) {
          const double x = rows.get(c, k, i);
          if (!kShared) backup[(long long)c * n + i] = x;
          acc[c] = __dadd_rn(acc[c], __dmul_rn(x, t));
        }
    }
    sp_warp_columns(acc, sh);
  }
  if (!sp_exchange(sh, slots, ++gen, all, warps, rows.nparts, -1, false, grid)) return -1;
  int jn[kSpBlock];  // next step of each column (block-uniform)
#pragma unroll
  for (int c = 0; c < kSpBlock; ++c) jn[c] = 0;
  int nfinal = from, pending = -1;
  while (nfinal < B) {
    double nrm = 0.0, inv = 0.0;
    const int fin = pending;
    if (fin >= 0) {
      nrm = sh.norm;
      inv = sh.inverse;
      if (nrm < 1e-10) return 1 + fin;
      nfinal = fin + 1;
    }
    // ready columns: not final, next step's v final (or the norm step); all share one step j
    int j = kSpBlock;
#pragma unroll
    for (int c = 0; c < kSpBlock; ++c)
      if (c >= nfinal && c < B && (jn[c] == c || jn[c] < nfinal)) j = min(j, jn[c]);
    unsigned ready = 0u;
#pragma unroll
    for (int c = 0; c < kSpBlock; ++c)
      if (c >= nfinal && c < B && jn[c] == j && (j == c || j < nfinal)) ready |= 1u << c;
    if (mine) {
      double d[kSpBlock], acc[kSpBlock];
#pragma unroll
      for (int c = 0; c < kSpBlock; ++c) {
        d[c] = ((ready >> c) & 1u) ? sh.total[c] : 0.0;
        acc[c] = 0.0;
      }
      for (int k = 0; k < rows.tiles; ++k) {
        const int i = rows.row(k, threadIdx.x);
        if (i >= n) continue;
        double xf = 0.0;
        if (fin >= 0) {
          const double x = rows.get(fin, k, i), q = __dmul_rn(x, inv);
          xf = __fma_rn(__fma_rn(-q, nrm, x), inv, q);  // x / nrm
          rows.m[(long long)fin * n + i] = xf;
          if (kShared) rows.set(fin, k, i, xf);
        }
        if (ready) {
          const double ui = j == 0 ? triv[i] : rows.get(j - 1, k, i);
          const double vi = j == fin ? xf : rows.get(j, k, i);
#pragma unroll
          for (int c = 0; c < kSpBlock; ++c)
            if ((ready >> c) & 1u) {
              const double x = __dsub_rn(rows.get(c, k, i), __dmul_rn(d[c], ui));
              rows.set(c, k, i, x);
              acc[c] = __dadd_rn(acc[c], __dmul_rn(x, j < c ? vi : x));
            }
        }
      }
      if (ready) sp_warp_columns(acc, sh);
    }
    pending = -1;
#pragma unroll
    for (int c = 0; c < kSpBlock; ++c)
      if ((ready >> c) & 1u) {
        if (jn[c] == c) pending = c;
        jn[c] += 1;
      }
    // the step that finished the last column has nothing to sum: a barrier before the next multiply
    if (!sp_exchange(sh, slots, ++gen, ready ? ready : 1u, warps, rows.nparts, pending, !ready, grid)) return -1;
  }
  return 0;
}

// Rounds round_begin..round_end-1 of the subspace iteration over the two blocks buf0 / buf1 (n x B
// column-major): round r multiplies buf[r % 2] into buf[(r + 1) % 2] and orthonormalises the
// result (round -1: orthonormalise buf0 only). Unless kShared, buf[r % 2] then holds the post-multiply
// copy. The first round starts at column first_from and multiplies only when first_multiply is set. A
// column whose norm vanishes stops every block at the same step (they all compute the same norm);
// block 0 records round and column in grid->status for the host's redraw. `slots`: kSpSlots, zeroed.
constexpr int kSpSlots = 2 * kSpBlock * kSpParts + kSpProducts * (kSpParts + 1);
template <bool kShared>
__global__ void __launch_bounds__(kSpRoundThreads, 1)
sp_rounds_kernel(const int* __restrict__ offsets, const int* __restrict__ nbr, const float* __restrict__ nw,
                 const double* __restrict__ triv, int n, int B, int points, int tiles, double* buf0, double* buf1,
                 SpSlot* slots, int round_begin, int round_end, int first_from, int first_multiply, SpGrid* grid) {
  extern __shared__ double s_rows[];
  __shared__ SpShared sh;
  if (threadIdx.x == 0) sh.failed = 0;
  __syncthreads();
  unsigned gen = 0;
  SpRows<kShared> rows{s_rows, nullptr, n, tiles * points, points, (int)gridDim.x, tiles};
  for (int r = round_begin; r < round_end; ++r) {
    rows.m = ((r + 1) & 1) ? buf1 : buf0;
    double* other = (r & 1) ? buf1 : buf0;
    const bool first = r == round_begin;
    if (!first || first_multiply) {
      sp_multiply_rows(
          offsets, nbr, nw, n, B, other, 0, tiles * points, kSpRoundThreads / 32 * 4,
          [&](int g) { return rows.row(g / points, g % points); },
          [&](int c, int g, int i, double v) {
            rows.m[(long long)c * n + i] = v;
            if (kShared) s_rows[c * rows.cap + g] = v;
          });
    } else if (kShared && (int)threadIdx.x < points) {
      for (int k = 0; k < tiles; ++k) {
        const int i = rows.row(k, threadIdx.x);
        if (i >= n) continue;
        for (int c = 0; c < B; ++c) rows.set(c, k, i, __ldcg(rows.m + (long long)c * n + i));
      }
    }
    __syncthreads();
    // Both write to buffers that other blocks' multiplies have read: after an exchange, so after those.
    if (B == kSpBlock && (!first || first_from == 0)) {
      const int done = sp_orthonormalise_at_once(rows, triv, sh, slots, grid, gen);
      if (done < 0) return;
      if (done) continue;
    } else if (!kShared && !sp_exchange(sh, slots, ++gen, 1u, rows.warps(), (int)gridDim.x, -1, true, grid)) {
      return;
    }
    const int st = sp_orthonormalise<kShared>(rows, other, triv, B, first ? first_from : 0, sh, slots, grid, gen);
    if (st > 0) {
      if (blockIdx.x == 0 && threadIdx.x == 0) grid->status = 16 * (r + 1) + (st - 1);
      return;
    }
    if (st < 0) return;
  }
}

// Block partials of q[:, a] . z[:, b] for a <= b (pair index in row-major upper-triangle order).
__global__ void __launch_bounds__(kSpThreads)
sp_project_kernel(const double* __restrict__ q, const double* __restrict__ z, int n, int B,
                  double* __restrict__ part) {
  __shared__ double s_w[kSpThreads / 32][kSpPairs];
  double acc[kSpPairs];
#pragma unroll
  for (int t = 0; t < kSpPairs; ++t) acc[t] = 0.0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    int t = 0;
#pragma unroll
    for (int a = 0; a < kSpBlock; ++a) {
      const double qv = a < B ? q[(long long)a * n + r] : 0.0;
#pragma unroll
      for (int b = a; b < kSpBlock; ++b, ++t)
        if (b < B) acc[t] = __dadd_rn(acc[t], __dmul_rn(qv, z[(long long)b * n + r]));
    }
  }
#pragma unroll
  for (int t = 0; t < kSpPairs; ++t) {
    const double v = warp_sum(acc[t]);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5][t] = v;
  }
  __syncthreads();
  if ((int)threadIdx.x < kSpPairs) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s = __dadd_rn(s, s_w[w][threadIdx.x]);
    part[(long long)blockIdx.x * kSpPairs + threadIdx.x] = s;
  }
}

// One warp: the projected matrix from the partials, the reference's Jacobi rotations (at most
// 80, each on the largest off-diagonal entry, the first in row order among equals), Ritz values sorted
// descending; coef[c * 8 + b] = component c's coefficients on the basis. The lanes share the entries of the search
// and the rows of a rotation; matrices in shared memory. 753 us by one thread, 186 us now, bound by the chain of
// divisions and roots of an angle.
__global__ void sp_ritz_kernel(const double* __restrict__ part, int nparts, int B, double* __restrict__ coef) {
  __shared__ double s_pair[kSpPairs];
  __shared__ double P[kSpBlock][kSpBlock + 1], V[kSpBlock][kSpBlock + 1];
  if (blockIdx.x != 0) return;
  if ((int)threadIdx.x < kSpPairs) {
    // entry t of the upper triangle: its block partials in block order, loads issued ahead
    const int t = threadIdx.x;
    double s = 0.0;
    int k = 0;
    for (; k + 7 < nparts; k += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = part[(long long)(k + u) * kSpPairs + t];
#pragma unroll
      for (int u = 0; u < 8; ++u) s = __dadd_rn(s, v[u]);
    }
    for (; k < nparts; ++k) s = __dadd_rn(s, part[(long long)k * kSpPairs + t]);
    s_pair[t] = s;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x, row = lane & (kSpBlock - 1);
  // lane t < 28: the t-th entry i < j in row order
  int pi = 0, pj = lane + 1;
  while (pj >= kSpBlock && pi < kSpBlock - 1) {
    ++pi;
    pj += pi + 1 - kSpBlock;
  }
  const bool entry = lane < kSpBlock * (kSpBlock - 1) / 2 && pj < B;
  if (lane < kSpBlock) {
    for (int b = 0; b < kSpBlock; ++b) {
      const int lo = min(lane, b), hi = max(lane, b);
      P[lane][b] = s_pair[lo * kSpBlock - lo * (lo - 1) / 2 + hi - lo];
      V[lane][b] = lane == b ? 1.0 : 0.0;
    }
  }
  __syncwarp();
  for (int sweep = 0; sweep < 80; ++sweep) {
    // the largest: the bits of positive doubles are in their order, high words first
    double mx = entry ? fabs(P[pi][pj]) : 0.0;
    if (!(mx > 0.0)) mx = 0.0;  // NaN exceeds nothing
    const unsigned hi = (unsigned)__double2hiint(mx), top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = hi == top ? (unsigned)__double2loint(mx) : 0u, low = __reduce_max_sync(0xffffffffu, lo);
    const int at = __ffs(__ballot_sync(0xffffffffu, hi == top && lo == low)) - 1;
    if (__hiloint2double((int)top, (int)low) < 1e-10) break;
    const int p = __shfl_sync(0xffffffffu, pi, at), q = __shfl_sync(0xffffffffu, pj, at);
    const double app = P[p][p], aqq = P[q][q], apq = P[p][q];
    const double akp = P[row][p], akq = P[row][q], vp = V[row][p], vq = V[row][q];
    __syncwarp();
    // tau = d / g; sign(tau) / (|tau| + sqrt(1 + tau^2)) with one division (|g| is at least 2e-10)
    const double d = __dsub_rn(aqq, app), g = __dmul_rn(2.0, apq);
    const double size = __ddiv_rn(fabs(g), __dadd_rn(fabs(d), __dsqrt_rn(__fma_rn(d, d, __dmul_rn(g, g)))));
    const double tt = d == 0.0 || (d > 0.0) == (g > 0.0) ? size : -size;
    const double cs = rsqrt(__fma_rn(tt, tt, 1.0));
    const double sn = __dmul_rn(tt, cs);
    if (lane < B) {
      if (row != p && row != q) {
        const double x = __dsub_rn(__dmul_rn(cs, akp), __dmul_rn(sn, akq));
        const double y = __dadd_rn(__dmul_rn(sn, akp), __dmul_rn(cs, akq));
        P[row][p] = x;
        P[p][row] = x;
        P[row][q] = y;
        P[q][row] = y;
      }
      V[row][p] = __dsub_rn(__dmul_rn(cs, vp), __dmul_rn(sn, vq));
      V[row][q] = __dadd_rn(__dmul_rn(sn, vp), __dmul_rn(cs, vq));
    }
    if (lane == 0) {
      const double cc = __dmul_rn(cs, cs), ss = __dmul_rn(sn, sn);
      const double cross = __dmul_rn(__dmul_rn(__dmul_rn(2.0, sn), cs), apq);
      P[p][p] = __dadd_rn(__dsub_rn(__dmul_rn(cc, app), cross), __dmul_rn(ss, aqq));
      P[q][q] = __dadd_rn(__dadd_rn(__dmul_rn(ss, app), cross), __dmul_rn(cc, aqq));
      P[p][q] = 0.0;
      P[q][p] = 0.0;
    }
    __syncwarp();
  }
  if (lane != 0) return;
  int order[kSpBlock];
  for (int i = 0; i < B; ++i) {
    int j = i;
    while (j > 0 && P[i][i] > P[order[j - 1]][order[j - 1]]) {
      order[j] = order[j - 1];
      --j;
    }
    order[j] = i;
  }
  for (int c = 0; c < 2; ++c)
    for (int b = 0; b < kSpBlock; ++b) coef[c * kSpBlock + b] = b < B ? V[b][order[c]] : 0.0;
}

// emb[:, c] = q coef_c (basis order), with block partials of each column's sum.
__global__ void __launch_bounds__(kSpThreads)
sp_embed_kernel(const double* __restrict__ q, const double* __restrict__ coef, int n, int B,
                double* __restrict__ emb, double* __restrict__ part) {
  double acc0 = 0.0, acc1 = 0.0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    double v0 = 0.0, v1 = 0.0;
    for (int b = 0; b < B; ++b) {
      const double x = q[(long long)b * n + r];
      v0 = __dadd_rn(v0, __dmul_rn(x, coef[b]));
      v1 = __dadd_rn(v1, __dmul_rn(x, coef[kSpBlock + b]));
    }
    emb[r] = v0;
    emb[(long long)n + r] = v1;
    acc0 = __dadd_rn(acc0, v0);
    acc1 = __dadd_rn(acc1, v1);
  }
  block_partial(acc0, part);
  __syncthreads();
  block_partial(acc1, part + gridDim.x);
}

// emb[:, c] -= mean_c (sums in part[c * nparts ...]); block maxima of |emb| into pmax.
__global__ void __launch_bounds__(kSpThreads)
sp_centre_kernel(double* __restrict__ emb, int n, const double* __restrict__ part, int nparts,
                 double* __restrict__ pmax) {
  __shared__ double s_w[kSpThreads / 32];
  const double m0 = __ddiv_rn(sum_partials(part, nparts), (double)n);
  const double m1 = __ddiv_rn(sum_partials(part + nparts, nparts), (double)n);
  double mx = 0.0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const double a = __dsub_rn(emb[r], m0), b = __dsub_rn(emb[(long long)n + r], m1);
    emb[r] = a;
    emb[(long long)n + r] = b;
    if (isfinite(a)) mx = fmax(mx, fabs(a));
    if (isfinite(b)) mx = fmax(mx, fabs(b));
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = fmax(t, s_w[w]);
    pmax[blockIdx.x] = t;
  }
}

// emb = emb * (10 / max|emb|) + jitter, unless the maximum is zero or not finite.
__global__ void sp_expand_kernel(double* __restrict__ emb, int n, const double* __restrict__ pmax, int nparts,
                                 const double* __restrict__ jitter) {
  __shared__ double s_mx;
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int b = 0; b < nparts; ++b) t = fmax(t, pmax[b]);
    s_mx = t;
  }
  __syncthreads();
  const double mx = s_mx;
  if (!isfinite(mx) || mx <= 0.0) return;
  const double ex = __ddiv_rn(10.0, mx);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 2LL * n;
       t += (long long)gridDim.x * blockDim.x)
    emb[t] = __dadd_rn(__dmul_rn(emb[t], ex), jitter[t]);
}

// scale_embedding_sdev: column c -> (x - mean) * (target / sd), sd over n - 1.
__global__ void __launch_bounds__(kSpThreads)
sp_column_sum_kernel(const double* __restrict__ col, int n, const double* __restrict__ mean_part, int nparts,
                     double* __restrict__ part) {
  const double mean = mean_part ? __ddiv_rn(sum_partials(mean_part, nparts), (double)n) : 0.0;
  double acc = 0.0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    if (mean_part) {
      const double d = __dsub_rn(col[r], mean);
      acc = __dadd_rn(acc, __dmul_rn(d, d));
    } else {
      acc = __dadd_rn(acc, col[r]);
    }
  }
  block_partial(acc, part);
}

__global__ void sp_rescale_kernel(double* __restrict__ col, int n, const double* __restrict__ mean_part,
                                  const double* __restrict__ ss_part, int nparts, double target) {
  const double mean = __ddiv_rn(sum_partials(mean_part, nparts), (double)n);
  const double sd = __dsqrt_rn(__ddiv_rn(sum_partials(ss_part, nparts), (double)(n - 1)));
  if (!isfinite(sd) || sd <= 0.0) return;
  const double sc = __ddiv_rn(target, sd);
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    col[r] = __dmul_rn(__dsub_rn(col[r], mean), sc);
}

}  // namespace

SpectralDraws spectral_draws(int n, int seed, int device, bool on_host) {
  SpectralDraws d;
  d.n = n;
  const int B = std::min(n - 1, kSpBlock);
  if (B < 2) return d;
  const std::size_t count = (std::size_t)n * B;
  std::mt19937 rng((std::uint32_t)seed);
  // (an odd count leaves a value in the host stream; a polar path that is not the library's has no twin)
  const bool on_device = !on_host && n >= kSpectralDeviceDraws && count % 2 == 0 && MtNormalBlock::fits(count) &&
                         NormalStream::polar_path() && NormalStream::radius_rounding() != NormalStream::Radius::kOther;
  if (on_device) {
    FE_CUDA(cudaSetDevice(device));
    try {
      d.device = std::make_shared<MtNormalBlock>((std::uint32_t)seed, count, 1e-4, 10000.0);
    } catch (const Error&) {
      cudaGetLastError();  // no memory for the words: drawn on the host, which needs none
    }
  }
  if (!d.device) {
    d.block.resize(count);
    d.normal.fill(rng, d.block.data(), count, 10000.0);
  }
  d.tail = std::async(std::launch::async, [rng, n, skip = d.device ? count / 2 : 0]() mutable {
             NormalStream::skip(rng, skip);
             SpectralTail t{rng, std::vector<double>(2 * (std::size_t)n)};
             NormalStream jitter(0.0, 1e-4);
             jitter.fill(rng, t.jitter.data(), t.jitter.size(), 1.0);
             return t;
           }).share();
  return d;
}

void umap_spectral_start(const int* offsets, const int* neighbors, const float* weights, int n, long long nnz,
                         int spectral_n_iter, double init_scale, int seed, double* out, cudaStream_t s,
                         SpectralDraws* pre, int max_blocks) {
  if (n < 1 || spectral_n_iter < 1) throw Error("invalid spectral initialization parameters");
  std::mt19937 rng((std::uint32_t)seed);
  std::uniform_real_distribution<double> uniform(-10.0, 10.0);
  const int B = std::min(n - 1, kSpBlock);
  const int nb = sp_blocks(n);
  const int gb = std::max(1, std::min(ceil_div(n, kSpThreads), sm_count() * 8));
  const int gw = std::max(1, std::min(ceil_div(n, kSpThreads / 32), sm_count() * 8));  // warp per row
  const int gm = std::max(1, std::min(ceil_div(n, kSpThreads / 8), sm_count() * 8));   // 8 lanes per row
  std::vector<double> host;
  if (nnz < 1 || B < 2) {
    // the reference's fallback: uniform(-10, 10) coordinates, column after column
    host.resize(2 * (std::size_t)n);
    for (double& v : host) v = uniform(rng);
    FE_CUDA(cudaMemcpyAsync(out, host.data(), sizeof(double) * host.size(), cudaMemcpyHostToDevice, s));
  } else {
    float *deg = nullptr, *nw = nullptr;
    double *triv = nullptr, *q = nullptr, *z = nullptr, *pa = nullptr, *pb = nullptr, *pc = nullptr;
    double *coef = nullptr, *jit = nullptr;
    SpGrid* grid = nullptr;
    SpSlot* slots = nullptr;
    Arena w;
    w.reserve(&deg, n);
    w.reserve(&nw, (std::size_t)nnz);
    w.reserve(&triv, n);
    w.reserve(&q, (std::size_t)n * B);
    w.reserve(&z, (std::size_t)n * B);
    w.reserve(&pa, kSpMaxBlocks * kSpPairs);
    w.reserve(&pb, kSpMaxBlocks * 2);
    w.reserve(&pc, kSpMaxBlocks * 2);
    w.reserve(&coef, 2 * kSpBlock);
    w.reserve(&jit, 2 * (std::size_t)n);
    w.reserve(&grid, 1);
    w.reserve(&slots, kSpSlots);
    w.commit("UMAP spectral start");
    sp_degree_kernel<<<gb, kSpThreads, 0, s>>>(offsets, weights, n, deg);
    FE_LAUNCH("sp_degree_kernel");
    sp_adjacency_kernel<<<gw, kSpThreads, 0, s>>>(offsets, neighbors, weights, deg, n, nw);
    FE_LAUNCH("sp_adjacency_kernel");
    sp_trivial_kernel<<<nb, kSpThreads, 0, s>>>(deg, n, triv, pa);
    FE_LAUNCH("sp_trivial_kernel");
    sp_normalise_trivial_kernel<<<gb, kSpThreads, 0, s>>>(triv, n, pa, nb);
    FE_LAUNCH("sp_normalise_trivial_kernel");
    SpGrid g0{0, -1};
    FE_CUDA(cudaMemcpyAsync(grid, &g0, sizeof(SpGrid), cudaMemcpyHostToDevice, s));
    SpectralDraws local;
    SpectralDraws* dr = pre;
    int dev = 0, coop = 0;
    FE_CUDA(cudaGetDevice(&dev));
    if (!dr || dr->n != n) {
      local = spectral_draws(n, seed, dev);
      dr = &local;
    }
    if (dr->device && !dr->device->copy_to(q, s)) {
      local = spectral_draws(n, seed, dev, true);
      dr = &local;
    }
    std::mt19937 live;  // the stream after the block, from the first redraw on
    bool redrawn = false;

    // The subspace iteration as cooperative launches: the initial orthonormalisation (round -1) and
    // spectral_n_iter rounds. A launch that stops at a vanished column is resumed from it after the host redraws
    // the column from the stream, as the reference redraws and repeats it.
    int blocks = std::min(kSpParts, sm_count());
    if (max_blocks > 0) blocks = std::min(blocks, max_blocks);
    int points = sp_points(n, blocks), tiles = sp_tiles(n, blocks);
    const int parts = ceil_div(n, (long long)points * tiles);
    const bool shared = (long long)tiles * points <= kSpSharedRows;
    const int smem = shared ? kSpBlock * tiles * points * (int)sizeof(double) : 0;
    const void* rounds = shared ? (const void*)sp_rounds_kernel<true> : (const void*)sp_rounds_kernel<false>;
    allow_dynamic_shared(rounds, smem, kSpBlock * kSpSharedRows * sizeof(double));
    int per_sm = 0;
    FE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rounds, kSpRoundThreads, smem));
    if (per_sm * sm_count() < parts) throw Error("the spectral start's subspace iteration cannot be made resident");
    FE_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) throw Error("the device does not support cooperative launches");
    if (!dr->device)
      FE_CUDA(cudaMemcpyAsync(q, dr->block.data(), sizeof(double) * dr->block.size(), cudaMemcpyHostToDevice, s));
    int r0 = -1, from = 0, mult = 0;
    for (;;) {
      int r_end = spectral_n_iter;
      FE_CUDA(cudaMemsetAsync(slots, 0, kSpSlots * sizeof(SpSlot), s));
      void* args[] = {(void*)&offsets, (void*)&neighbors, (void*)&nw, (void*)&triv, (void*)&n, (void*)&B,
                      (void*)&points, (void*)&tiles, (void*)&q, (void*)&z, (void*)&slots, (void*)&r0, (void*)&r_end,
                      (void*)&from, (void*)&mult, (void*)&grid};
      FE_CUDA(cudaLaunchCooperativeKernel(rounds, dim3(parts), dim3(kSpRoundThreads), args, smem, s));
      FE_LAUNCH("sp_rounds_kernel");
      SpGrid g1;
      FE_CUDA(cudaMemcpyAsync(&g1, grid, sizeof(SpGrid), cudaMemcpyDeviceToHost, s));
      FE_CUDA(cudaStreamSynchronize(s));
      if (g1.error) throw Error("spectral start: an exchange of the subspace iteration timed out");
      if (g1.status < 0) break;
      const int rr = g1.status / 16 - 1, f = g1.status % 16;
      if (rr < -1 || rr >= spectral_n_iter || f < 0 || f >= B) throw Error("spectral start: invalid redraw status");
      if (!redrawn) live = dr->tail.get().rng;
      redrawn = true;
      host.resize(n);
      dr->normal.fill(live, host.data(), host.size(), 10000.0);
      // the later columns back to their post-multiply values where the pass had started on them, then
      // the redrawn column
      double* m = ((rr + 1) & 1) ? z : q;
      const double* bk = (rr & 1) ? z : q;
      if (!shared && f + 1 < B)
        FE_CUDA(cudaMemcpyAsync(m + (std::size_t)(f + 1) * n, bk + (std::size_t)(f + 1) * n,
                                sizeof(double) * (std::size_t)(B - f - 1) * n, cudaMemcpyDeviceToDevice, s));
      FE_CUDA(cudaMemcpyAsync(m + (std::size_t)f * n, host.data(), sizeof(double) * n, cudaMemcpyHostToDevice, s));
      FE_CUDA(cudaMemcpyAsync(grid, &g0, sizeof(SpGrid), cudaMemcpyHostToDevice, s));
      r0 = rr;
      from = f;
      mult = 0;
    }
    // after round r the block is in buf[(r + 1) % 2]: the last round leaves it in buf[n_iter % 2]
    if (spectral_n_iter & 1) std::swap(q, z);
    sp_multiply_kernel<<<gm, kSpThreads, 0, s>>>(offsets, neighbors, nw, n, B, q, z);
    FE_LAUNCH("sp_multiply_kernel");
    sp_project_kernel<<<nb, kSpThreads, 0, s>>>(q, z, n, B, pa);
    FE_LAUNCH("sp_project_kernel");
    sp_ritz_kernel<<<1, 64, 0, s>>>(pa, nb, B, coef);
    FE_LAUNCH("sp_ritz_kernel");
    sp_embed_kernel<<<nb, kSpThreads, 0, s>>>(q, coef, n, B, out, pb);
    FE_LAUNCH("sp_embed_kernel");
    sp_centre_kernel<<<nb, kSpThreads, 0, s>>>(out, n, pb, nb, pc);
    FE_LAUNCH("sp_centre_kernel");
    // jitter: a fresh normal(0, 1e-4) distribution on the same stream, column after column (drawn
    // ahead unless a redraw moved the stream on)
    std::vector<double> fresh;
    if (redrawn) {
      NormalStream jitter(0.0, 1e-4);
      fresh.resize(2 * (std::size_t)n);
      jitter.fill(live, fresh.data(), fresh.size(), 1.0);
    }
    const std::vector<double>& jv = redrawn ? fresh : dr->tail.get().jitter;
    FE_CUDA(cudaMemcpyAsync(jit, jv.data(), sizeof(double) * jv.size(), cudaMemcpyHostToDevice, s));
    sp_expand_kernel<<<gb, kSpThreads, 0, s>>>(out, n, pc, nb, jit);
    FE_LAUNCH("sp_expand_kernel");
    FE_CUDA(cudaStreamSynchronize(s));
  }
  if (std::isfinite(init_scale) && init_scale > 0.0 && n >= 2) {
    double *pm = nullptr, *ps = nullptr;
    Arena w;
    w.reserve(&pm, kSpMaxBlocks);
    w.reserve(&ps, kSpMaxBlocks);
    w.commit("UMAP start rescale");
    for (int c = 0; c < 2; ++c) {
      double* col = out + (std::size_t)c * n;
      sp_column_sum_kernel<<<nb, kSpThreads, 0, s>>>(col, n, nullptr, nb, pm);
      FE_LAUNCH("sp_column_sum_kernel");
      sp_column_sum_kernel<<<nb, kSpThreads, 0, s>>>(col, n, pm, nb, ps);
      FE_LAUNCH("sp_column_sum_kernel");
      sp_rescale_kernel<<<gb, kSpThreads, 0, s>>>(col, n, pm, ps, nb, init_scale);
      FE_LAUNCH("sp_rescale_kernel");
    }
    FE_CUDA(cudaStreamSynchronize(s));
  }
}

}  // namespace fe
