// Per-iteration kernels of the t-SNE gradient loop on the GPU.
//
// Reference algorithm (fastEmbedR src/tsne_neighbors.cpp:1152-1260 on the CPU,
// src/embedding_cuda_kernels.cpp:2472-2886 on CUDA): bound the layout by a square,
// interpolate charges {1, x, y} onto a uniform grid, convolve with the kernels
// q = 1/(1 + d^2) and q^2 by FFT on the zero-padded 2G x 2G torus, interpolate the potentials
// back, combine with the sparse attractive term and apply the gains/momentum update.
//
// GB300 layout of one iteration (6 launches, two streams, captured in a CUDA graph):
//   side stream:  attractive_kernel        warp per CSR row, rows in storage (spatial) order, one
//                                          queue of rows per SM
//   main stream:  scatter_kernel           points -> 64-bit fixed-point charges (deterministic)
//                 row FFTs, column FFTs with the products, inverse row FFTs (tsne_fft.cu)
//   join:         update_kernel            potential gather + gains/momentum/step clip +
//                                          recentring; epilogue reduces the new bounding box and
//                                          mean into the next iteration's grid
// Interpolation: the reference bilinear splat on G shared nodes (default), or 3 equispaced
// Lagrange nodes per box over floor(G / 3) boxes, as in FIt-SNE-style interpolation.
#include <cfloat>
#include <climits>
#include <cmath>
#include <algorithm>
#include <vector>

#include "tsne_grid.cuh"

namespace fe {

constexpr int kStepThreads = 256;

// ---------------------------------------------------------------- stencils
template <int TAPS>
struct Stencil {
  int base;
  float w[TAPS];
};

// Bilinear (TAPS = 2): bilinear_grid_value_t / the scatter of src/tsne_neighbors.cpp:1194-1213.
// Lagrange (TAPS = 3): nodes at x0 + (3b + j + 0.5) h, j = 0..2, of box b.
template <int TAPS>
__device__ __forceinline__ Stencil<TAPS> make_stencil(float x, float x0, float inv_h, float inv_box, int nodes) {
  Stencil<TAPS> s;
  if constexpr (TAPS == 2) {
    const float raw = (x - x0) * inv_h;
    const float c = fmaxf(0.0f, fminf((float)(nodes - 1), raw));
    int u0 = (int)floorf(c);
    u0 = max(0, min(nodes - 2, u0));
    const float f = c - (float)u0;
    s.base = u0;
    s.w[0] = 1.0f - f;
    s.w[1] = f;
  } else {
    const int nbox = nodes / 3;
    int b = (int)floorf((x - x0) * inv_box);
    b = max(0, min(nbox - 1, b));
    const float t = (x - x0) * inv_h - (float)(3 * b) - 0.5f;
    s.base = 3 * b;
    s.w[0] = 0.5f * (t - 1.0f) * (t - 2.0f);
    s.w[1] = t * (2.0f - t);
    s.w[2] = 0.5f * t * (t - 1.0f);
  }
  return s;
}

// (instance, first slot) of this point block. A single instance needs no table (null): its blocks
// follow one another, and the kernels that a small layout waits for have one load less in their chain.
__device__ __forceinline__ int2 point_block(const int2* __restrict__ blocks) {
  return blocks ? blocks[blockIdx.x] : make_int2(0, (int)blockIdx.x * kPointBlock);
}

// ---------------------------------------------------------------- layout statistics
// Fixed-order reduction of the per-block partials into the grid of the next iteration
// (the bounding-square rule of src/tsne_neighbors.cpp:1168-1184).
__device__ void finish_layout_stats(const StepPartial* __restrict__ part, int nblocks, int n, int grid, int mode,
                                    GridState* __restrict__ next) {
  __shared__ StepPartial s_stat[kStepThreads / 32];
  float mnx = FLT_MAX, mxx = -FLT_MAX, mny = FLT_MAX, mxy = -FLT_MAX;
  double sx = 0.0, sy = 0.0;
  // partials written by the other blocks of this launch: read through L2, eight loads in flight
#pragma unroll 8
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
    const float4 mm = __ldcg(reinterpret_cast<const float4*>(part + b));
    const double2 ss = __ldcg(reinterpret_cast<const double2*>(part + b) + 1);
    mnx = fminf(mnx, mm.x);
    mxx = fmaxf(mxx, mm.y);
    mny = fminf(mny, mm.z);
    mxy = fmaxf(mxy, mm.w);
    sx += ss.x;
    sy += ss.y;
  }
  mnx = warp_min(mnx);
  mxx = warp_max(mxx);
  mny = warp_min(mny);
  mxy = warp_max(mxy);
  // (warps without a partial stay off the FP64 pipe: a warp's two sums hold it for 190 cycles)
  if (nblocks > 1 && (int)(threadIdx.x & ~31u) < nblocks) {
    sx = warp_sum(sx);
    sy = warp_sum(sy);
  }
  if ((threadIdx.x & 31) == 0) s_stat[threadIdx.x >> 5] = StepPartial{mnx, mxx, mny, mxy, sx, sy};
  __syncthreads();
  // warps without a partial hold the neutral values
  const int warps = min((int)(blockDim.x / 32), (nblocks + 31) / 32);
  if (threadIdx.x == 32 || threadIdx.x == 64) {  // the means, beside the box
    const bool is_x = threadIdx.x == 32;
    double sum = is_x ? s_stat[0].sum_x : s_stat[0].sum_y;
    for (int w = 1; w < warps; ++w) sum += is_x ? s_stat[w].sum_x : s_stat[w].sum_y;
    (is_x ? next->mean_x : next->mean_y) = sum / (double)n;
  }
  if (threadIdx.x == 0) {
    StepPartial p = s_stat[0];
    for (int w = 1; w < warps; ++w) {
      p.min_x = fminf(p.min_x, s_stat[w].min_x);
      p.max_x = fmaxf(p.max_x, s_stat[w].max_x);
      p.min_y = fminf(p.min_y, s_stat[w].min_y);
      p.max_y = fmaxf(p.max_y, s_stat[w].max_y);
    }
    const float min_x = p.min_x, max_x = p.max_x, min_y = p.min_y, max_y = p.max_y;
    GridState g;
    g.cx = 0.5f * (min_x + max_x);
    g.cy = 0.5f * (min_y + max_y);
    float span = fmaxf(max_x - min_x, max_y - min_y);
    if (!isfinite(span) || span <= 0.0f) span = 1.0f;
    const float half = 0.55f * span + 1.0e-3f;
    g.x0 = g.cx - half;
    g.y0 = g.cy - half;
    if (mode == kInterpBilinear) {
      g.nodes = grid;
      g.h = (2.0f * half) / (float)(grid - 1);
      g.box = g.h;
    } else {
      const int nbox = grid / 3;
      g.nodes = 3 * nbox;
      g.box = (2.0f * half) / (float)nbox;
      g.h = g.box / 3.0f;
    }
    g.inv_h = 1.0f / g.h;
    g.inv_box = 1.0f / g.box;
    // |mass| and |mass * d| summed over any subset of points stay below 1.5625 n max(half, 1)
    // (stencil weights sum to 1 in absolute value for bilinear, 1.5625 for Lagrange; |d| <= half):
    // scale so that bound stays below 2^62.
    float bound = 2.0f * (float)n * fmaxf(half, 1.0f);
    if (!(bound < 1.0e30f)) bound = 1.0e30f;
    int e = 0;
    frexpf(bound, &e);  // bound < 2^e
    g.qscale = ldexpf(1.0f, 62 - e);
    g.inv_qscale = ldexpf(1.0f, e - 62);
    // the same bound over the points of one block (at most kPointBlock), below 2^30
    float tbound = 2.0f * (float)min(n, kPointBlock) * fmaxf(half, 1.0f);
    if (!(tbound < 1.0e30f)) tbound = 1.0e30f;
    int et = 0;
    frexpf(tbound, &et);
    g.tile_shift = (62 - e) - (30 - et);  // >= 0: et <= e
    g.tscale = ldexpf(1.0f, 30 - et);
    next->x0 = g.x0;
    next->y0 = g.y0;
    next->h = g.h;
    next->inv_h = g.inv_h;
    next->box = g.box;
    next->inv_box = g.inv_box;
    next->cx = g.cx;
    next->cy = g.cy;
    next->z = 0.0;
    next->inv_z = 0.0f;
    next->nodes = g.nodes;
    next->qscale = g.qscale;
    next->inv_qscale = g.inv_qscale;
    next->tscale = g.tscale;
    next->tile_shift = g.tile_shift;
  }
}

// Statistics of the block's points (one per thread). The coordinate sums are kept in two floats, within
// 2^-47 of the sum of magnitudes (256 floats of similar size add up exactly), and go on in FP64
// from the partials; with FP64 warp sums the update took 52 us at 1M points.
__device__ __forceinline__ void block_partial(float mnx, float mxx, float mny, float mxy, float sx, float sy,
                                              StepPartial* out) {
  __shared__ float4 s_box[kStepThreads / 32];
  __shared__ Float2Sum s_sum[kStepThreads / 32][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  mnx = warp_min(mnx);
  mxx = warp_max(mxx);
  mny = warp_min(mny);
  mxy = warp_max(mxy);
  const Float2Sum wx = warp_sum(Float2Sum{sx, 0.0f}), wy = warp_sum(Float2Sum{sy, 0.0f});
  if (lane == 0) {
    s_box[warp] = make_float4(mnx, mxx, mny, mxy);
    s_sum[warp][0] = wx;
    s_sum[warp][1] = wy;
  }
  __syncthreads();
  if (warp == 0) {
    constexpr int W = kStepThreads / 32;
    const float4 b = s_box[lane & (W - 1)];
    float4 r = b;
    Float2Sum x = s_sum[lane & (W - 1)][0], y = s_sum[lane & (W - 1)][1];
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
      r.x = fminf(r.x, __shfl_xor_sync(0xffffffffu, r.x, o));
      r.y = fmaxf(r.y, __shfl_xor_sync(0xffffffffu, r.y, o));
      r.z = fminf(r.z, __shfl_xor_sync(0xffffffffu, r.z, o));
      r.w = fmaxf(r.w, __shfl_xor_sync(0xffffffffu, r.w, o));
      x = add(x, Float2Sum{__shfl_xor_sync(0xffffffffu, x.hi, o), __shfl_xor_sync(0xffffffffu, x.lo, o)});
      y = add(y, Float2Sum{__shfl_xor_sync(0xffffffffu, y.hi, o), __shfl_xor_sync(0xffffffffu, y.lo, o)});
    }
    if (lane == 0) *out = StepPartial{r.x, r.y, r.z, r.w, value(x), value(y)};
  }
}

// Returns true in exactly one of the `blocks` blocks sharing `counter`: the last one to finish
// (counter reset for reuse).
__device__ __forceinline__ bool last_block_done(unsigned* counter, int blocks) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned prev = atomicAdd(counter, 1u);
    s_last = prev == (unsigned)blocks - 1u;
    if (s_last) *counter = 0u;
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

// Initial statistics of ynew (setup, and after an external layout write). One point per thread;
// each instance's last block finishes that instance's grid.
__global__ void __launch_bounds__(kStepThreads)
layout_stats_kernel(const float2* __restrict__ ynew, const TsneInstance* __restrict__ inst,
                    const int2* __restrict__ blocks, int mode, StepPartial* __restrict__ part,
                    unsigned* __restrict__ counter, GridState* __restrict__ next) {
  const int2 bl = blocks[blockIdx.x];
  const TsneInstance I = inst[bl.x];
  const int i = bl.y + threadIdx.x;
  float mnx = FLT_MAX, mxx = -FLT_MAX, mny = FLT_MAX, mxy = -FLT_MAX, sx = 0.0f, sy = 0.0f;
  if (i < I.pt_begin + I.n) {
    const float2 p = ynew[i];
    mnx = mxx = p.x;
    mny = mxy = p.y;
    sx = p.x;
    sy = p.y;
  }
  block_partial(mnx, mxx, mny, mxy, sx, sy, part + blockIdx.x);
  if (last_block_done(counter + bl.x, I.blocks))
    finish_layout_stats(part + I.block_begin, I.blocks, I.n, I.grid, mode, next + bl.x);
}

// ---------------------------------------------------------------- scatter
// Each point adds (w, w*(x - cx), w*(y - cy)) to its TAPS x TAPS stencil nodes of its instance's
// grid; the first block of every instance also promotes the grid computed by the previous update
// (`next`) to `cur`.
// Points are stored in spatial (Morton) order and every block takes 256 consecutive points of one
// instance, so a block covers a compact patch of the grid even when clusters collapse onto a few
// cells:
//   1. runs of equal stencil anchors inside a warp are summed by a segmented shuffle reduction
//      (a fixed tree: the same inputs give the same float sums);
//   2. run heads accumulate into a kTile x kTile node tile in shared memory anchored at the block's
//      lowest anchor, in 32-bit fixed point (the run sums rounded to a multiple of 1 / tscale,
//      about 2^-30 of the largest sum a block can make; native 32-bit shared atomics); heads
//      outside the tile add to the grid directly in 64-bit fixed point (x qscale), four lanes a node, so that its
//      three sums leave the SM as one request (a lane per head kept the few SMs of a small layout busy with
//      12 requests a point: twenty iterations at 2,000 points 785 -> 673 us, at 100,000 3.22 -> 3.14 ms);
//   3. the tile is flushed with one 64-bit integer atomic per touched node and value, the tile sum
//      shifted up to the grid's scale (exact: both scales are powers of two).
// Integer sums do not depend on the order in which atomics arrive, so the charges (and the
// whole iteration) are deterministic.
constexpr int kScatterTile = 32;

__device__ __forceinline__ void red_add_i64(long long* p, long long v) {
  atomicAdd(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(v));
}

template <int TAPS>
__global__ void __launch_bounds__(256)
scatter_kernel(const float2* __restrict__ y, const TsneInstance* __restrict__ inst, const int2* __restrict__ blocks,
               GridState* __restrict__ cur, const GridState* __restrict__ next, int n) {
  constexpr int NV = TAPS * TAPS * 3;
  __shared__ __align__(16) int tile[kScatterTile * kScatterTile * 3];
  __shared__ int s_box[4];
  __shared__ float4 s_beyond[kPointBlock / 32][32];
  const int2 bl = point_block(blocks);
  const int i = bl.y + threadIdx.x;
  // the point is requested beside the instance and grid records (clamped as in the update)
  const float2 own = y[min(i, n - 1)];
  const TsneInstance I = inst[bl.x];
  const int grid = I.grid;
  long long* __restrict__ charges = I.charges;
  const GridState g = next[bl.x];
  const int lane = threadIdx.x & 31;
  for (int t = threadIdx.x; t < kScatterTile * kScatterTile * 3 / 4; t += blockDim.x)
    reinterpret_cast<int4*>(tile)[t] = make_int4(0, 0, 0, 0);
  if (threadIdx.x == 0) {
    s_box[0] = INT_MAX;
    s_box[1] = INT_MAX;
    s_box[2] = -1;
    s_box[3] = -1;
  }
  if (bl.y == I.pt_begin && threadIdx.x == 0) cur[bl.x] = g;
  const bool valid = i < I.pt_begin + I.n;
  const float2 p = valid ? own : make_float2(g.cx, g.cy);
  const Stencil<TAPS> sx = make_stencil<TAPS>(p.x, g.x0, g.inv_h, g.inv_box, g.nodes);
  const Stencil<TAPS> sy = make_stencil<TAPS>(p.y, g.y0, g.inv_h, g.inv_box, g.nodes);
  const float dx = p.x - g.cx, dy = p.y - g.cy;
  float v[NV];
#pragma unroll
  for (int a = 0; a < TAPS; ++a)
#pragma unroll
    for (int b = 0; b < TAPS; ++b) {
      const float w = valid ? sy.w[a] * sx.w[b] : 0.0f;
      v[(a * TAPS + b) * 3 + 0] = w;
      v[(a * TAPS + b) * 3 + 1] = w * dx;
      v[(a * TAPS + b) * 3 + 2] = w * dy;
    }
  const int key = valid ? sy.base * grid + sx.base : -1 - lane;
  const int prev = __shfl_up_sync(0xffffffffu, key, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != key);
  if (heads != 0xffffffffu) {
    // suffix sums restricted to contiguous runs [lane, next head)
    const unsigned above = heads & ~((2u << lane) - 1u);
    const int run_end = above ? __ffs(above) - 1 : 32;
    // no further than the longest run (the levels beyond add nothing)
    const int longest = __reduce_max_sync(0xffffffffu, run_end - lane);
    for (int off = 1; off < longest; off <<= 1) {
      const bool take = lane + off < run_end;
#pragma unroll
      for (int c = 0; c < NV; ++c) {
        const float o = __shfl_down_sync(0xffffffffu, v[c], off);
        if (take) v[c] += o;
      }
    }
  }
  const bool head = valid && ((heads >> lane) & 1u);
  __syncthreads();
  // the block's anchors: a reduction per warp first (32 lanes on one address would take turns)
  const int x_lo = __reduce_min_sync(0xffffffffu, head ? sx.base : INT_MAX);
  const int y_lo = __reduce_min_sync(0xffffffffu, head ? sy.base : INT_MAX);
  const int x_hi = __reduce_max_sync(0xffffffffu, head ? sx.base : -1);
  const int y_hi = __reduce_max_sync(0xffffffffu, head ? sy.base : -1);
  if (lane == 0 && x_hi >= 0) {
    atomicMin(&s_box[0], x_lo);
    atomicMin(&s_box[1], y_lo);
    atomicMax(&s_box[2], x_hi);
    atomicMax(&s_box[3], y_hi);
  }
  __syncthreads();
  const int ox = s_box[0], oy = s_box[1];
  const int tx = sx.base - ox, ty = sy.base - oy;
  const bool in_tile = tx + TAPS <= kScatterTile && ty + TAPS <= kScatterTile;
  if (head && in_tile) {
#pragma unroll
    for (int a = 0; a < TAPS; ++a)
#pragma unroll
      for (int b = 0; b < TAPS; ++b) {
        int* t = tile + ((ty + a) * kScatterTile + tx + b) * 3;
        const int c = (a * TAPS + b) * 3;
        atomicAdd(t, __float2int_rn(v[c] * g.tscale));
        atomicAdd(t + 1, __float2int_rn(v[c + 1] * g.tscale));
        atomicAdd(t + 2, __float2int_rn(v[c + 2] * g.tscale));
      }
  }
  // Heads beyond the tile, node by node: four lanes take one node's three sums, which lie in one 32-byte
  // sector and leave the SM as one request (a lane per head sent three).
  const unsigned beyond = __ballot_sync(0xffffffffu, head && !in_tile);
  if (beyond) {
    float4* mine = s_beyond[threadIdx.x >> 5];
    const int rank = __popc(beyond & ((1u << lane) - 1u)), count = 4 * __popc(beyond);
#pragma unroll
    for (int a = 0; a < TAPS; ++a)
#pragma unroll
      for (int b = 0; b < TAPS; ++b) {
        const int c = (a * TAPS + b) * 3;
        if (head && !in_tile)
          mine[rank] = make_float4(v[c], v[c + 1], v[c + 2],
                                   __int_as_float(((sy.base + a) * grid + sx.base + b) * kChargeStride));
        __syncwarp();
        for (int t = lane; t < count; t += 32) {
          const float* e = reinterpret_cast<const float*>(mine + (t >> 2));
          const int u = t & 3;
          if (u < 3) red_add_i64(charges + __float_as_int(e[3]) + u, __float2ll_rn(e[u] * g.qscale));
        }
        __syncwarp();
      }
  }
  __syncthreads();
  if (s_box[2] < 0) return;  // no valid point in this block
  const int wu = min(kScatterTile, s_box[2] - ox + TAPS);
  const int hu = min(kScatterTile, s_box[3] - oy + TAPS);
  for (int t = threadIdx.x; t < wu * hu; t += blockDim.x) {
    const int r = t / wu, c = t - r * wu;
    const int* src = tile + (r * kScatterTile + c) * 3;
    const int a0 = src[0], a1 = src[1], a2 = src[2];
    if (a0 != 0 || a1 != 0 || a2 != 0) {
      long long* dst = charges + ((long long)(oy + r) * grid + ox + c) * kChargeStride;
      const int sh = g.tile_shift;
      red_add_i64(dst, (long long)((unsigned long long)(long long)a0 << sh));
      red_add_i64(dst + 1, (long long)((unsigned long long)(long long)a1 << sh));
      red_add_i64(dst + 2, (long long)((unsigned long long)(long long)a2 << sh));
    }
  }
}

// ---------------------------------------------------------------- attractive pass
// a_i = exag * sum_j p_ij q_ij (y_i - y_j), q = 1 / (1 + d^2)
// (add_sparse_attractive_gradient_f, src/tsne_neighbors.cpp:1061-1088).
// Rows are taken in storage (spatial) order: slot_rows[s] = (begin, end) of the CSR row of the
// point in slot s (rebuilt at every reorder), so a row is one contiguous segment of P and
// neighbouring slots belong to neighbouring points, whose neighbour sets overlap.
//
// What bounds the pass is the rate at which 32-byte sectors reach the SMs from L2: a y gather that
// misses L1 costs a whole sector, and the SMs take about one sector per clock each (measured: 2.07
// random 8-byte gathers per ns and SM from L2, 6.1 from L1). So the slots are divided into one
// contiguous range of chunks per SM and every warp takes its chunks from the counter of the SM it
// runs on (%smid): the gathers of an SM then stay within one neighbourhood of the layout, which its
// L1 holds, where one counter for all SMs spread every neighbourhood over all of them. The stream
// of columns and values bypasses L1. A warp whose SM has no chunk left takes chunks from the
// SM with the most left, so uneven row lengths, or an SM shared with the grid stage, cost nothing.
//
// How many gathers L1 serves depends on the layout: 75 to 77 % where neighbours in the data lie close together in the
// layout (discs drawn from the data's own coordinates), and the pass is then bound by instruction issue (75 % of the
// issue slots at 400,000 points); 54 % on an optimised layout of 30 large clusters, where it is half issue, half
// waiting (50 % of the slots at 200,000 points). So the rest of the kernel is about instructions. A row is read
// in rounds of 128 entries from c0, its first entry rounded down to a multiple of 4, with 128-bit
// loads (lane l takes entries 4 l .. + 3); entries outside the row are masked only in the rounds that
// can hold some. Two rows share one reduction, and the two rows after them are prefetched into L2
// (cp.async.bulk.prefetch), a lane each. Each lane sums its entries in a fixed order, rounds are
// added with Kahan compensation, and the warp sum is a fixed butterfly: the force depends only on
// the row and its entries' positions modulo 4, not on the schedule. The chunk size and the number
// of resident blocks are launch parameters chosen at run time by timing (tsne_tune_attractive); the
// result does not depend on them.
constexpr int kAttrThreads = 256;
constexpr int kAttrWarps = kAttrThreads / 32;
__device__ __forceinline__ void prefetch_l2_range(const void* base, long long first, long long last, int elem) {
  // [first, last) elements of a 4-byte array, widened to 16-byte boundaries (the arena pads
  // every buffer to 256 bytes, so the widened range stays inside the allocation)
  if (last <= first) return;
  const unsigned long long a = (unsigned long long)base + (unsigned long long)(first * elem);
  const unsigned long long e = (unsigned long long)base + (unsigned long long)(last * elem);
  const unsigned long long a16 = a & ~15ull, e16 = (e + 15ull) & ~15ull;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a16), "r"((unsigned)(e16 - a16)) : "memory");
}

// Butterfly of the lane partials of two rows, (x0, y0) and (x1, y1): lanes 0-7 end with the warp's x0
// sum, 8-15 with x1, 16-23 with y0, 24-31 with y1. A row's sum is the same in either place.
__device__ __forceinline__ float butterfly_rows(float x0, float y0, float x1, float y1, int lane) {
  const bool h16 = lane & 16, h8 = lane & 8;
  float k0 = h16 ? y0 : x0, k1 = h16 ? y1 : x1;
  k0 += __shfl_xor_sync(0xffffffffu, h16 ? x0 : y0, 16);
  k1 += __shfl_xor_sync(0xffffffffu, h16 ? x1 : y1, 16);
  float k = h8 ? k1 : k0;
  k += __shfl_xor_sync(0xffffffffu, h8 ? k0 : k1, 8);
  k += __shfl_xor_sync(0xffffffffu, k, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 2);
  k += __shfl_xor_sync(0xffffffffu, k, 1);
  return k;
}

__device__ __forceinline__ void prefetch_row(const int* col, const float* val, int2 se) {
  prefetch_l2_range(col, se.x, se.y, 4);
  prefetch_l2_range(val, se.x, se.y, 4);
}

// P is read once per pass: its columns and values must not displace the layout in L1.
__device__ __forceinline__ void ld_stream(const int* pc, const float* pv, int (&c)[4], float (&v)[4]) {
  asm volatile("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
               : "l"(pc));
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "l"(pv));
}

// Lane partials of row [b, e) of the point yi in slot s. Entries of a round outside the row count as
// the point s itself with value 0, whose term is exactly zero. (Positions are unsigned: the round after a row that ends
// near 2^31 begins beyond it.)
__device__ __forceinline__ float2 attr_row(const int* __restrict__ col, const float* __restrict__ val,
                                           const float2* __restrict__ y, unsigned b, unsigned e, int s, float2 yi, int lane) {
  float ax = 0.0f, ay = 0.0f, kx = 0.0f, ky = 0.0f;
  for (unsigned c0 = b & ~3u; c0 < e; c0 += 128u) {
    const unsigned p = c0 + 4u * lane;
    int c[4] = {s, s, s, s};
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (p < e) ld_stream(col + p, val + p, c, v);
    if (c0 < b || e - c0 < 128) {  // a round that can hold entries of other rows
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (p + u < b || p + u >= e) {
          c[u] = s;
          v[u] = 0.0f;
        }
    }
    float rx = 0.0f, ry = 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float2 yj = __ldg(y + c[u]);
      const float dx = yi.x - yj.x, dy = yi.y - yj.y;
      // fast reciprocal (within 2 ulp; 1 + d^2 >= 1 is never denormal or huge); the rounding of
      // d^2 is fixed so that a change of the surrounding code cannot change the force's bits
      const float q = __fdividef(1.0f, __fadd_rn(1.0f, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))));
      const float cq = v[u] * q;
      rx += cq * dx;
      ry += cq * dy;
    }
    const float tx = rx - kx, ty = ry - ky;
    const float nx = ax + tx, ny = ay + ty;
    kx = (nx - ax) - tx;
    ky = (ny - ay) - ty;
    ax = nx;
    ay = ny;
  }
  return make_float2(ax, ay);
}

// Chunk queues of the attractive pass: queue q's count of chunks taken, at ctr[(1 + q) *
// kAttrCtrStride] (a 32-byte sector each); ctr[0] counts finished blocks. All zero between launches.
constexpr int kAttrCtrStride = 8;
// A warp whose queue is empty looks at kAttrProbes others and helps one that has more than kAttrLeave
// chunks left (an SM with long rows, or none of this launch's blocks). No more than that: the last
// chunks of a queue are taken within microseconds by its own 40 to 48 warps, while thousands of idle
// warps reading every counter and chasing the last chunks cost 18 us a launch.
constexpr unsigned kAttrLeave = 16;
constexpr int kAttrProbes = 2;

// The chunks of queue q of nq: [begin, begin + size) of 0 .. nchunks - 1.
struct AttrQueue {
  unsigned begin, size;
};
__device__ __forceinline__ AttrQueue attr_queue(unsigned q, unsigned nq, unsigned nchunks) {
  const unsigned per = nchunks / nq, extra = nchunks - per * nq;
  return AttrQueue{q * per + min(q, extra), per + (q < extra ? 1u : 0u)};
}

// The next chunk of queue q, or nchunks when it is empty.
__device__ __forceinline__ unsigned attr_take(unsigned* __restrict__ ctr, unsigned q, unsigned nq, unsigned nchunks,
                                              int lane) {
  const AttrQueue Q = attr_queue(q, nq, nchunks);
  unsigned t = 0;
  if (lane == 0) t = atomicAdd(ctr + (1 + q) * kAttrCtrStride, 1u);
  t = __shfl_sync(0xffffffffu, t, 0);
  return t < Q.size ? Q.begin + t : nchunks;
}

// The next chunk of the warp's queue q; once that is empty, of another queue that needs help, which
// becomes the warp's; nchunks when it found none.
__device__ __forceinline__ unsigned attr_pop(unsigned* __restrict__ ctr, unsigned& q, unsigned nq, unsigned nchunks,
                                             unsigned& rnd, int lane) {
  unsigned c = attr_take(ctr, q, nq, nchunks, lane);
  for (int probe = 0; c >= nchunks && probe < kAttrProbes; ++probe) {
    rnd = rnd * 1664525u + 1013904223u;
    const unsigned v = __umulhi(rnd, nq);
    const unsigned taken = __ldcg(ctr + (1 + v) * kAttrCtrStride), size = attr_queue(v, nq, nchunks).size;
    if (size > taken && size - taken > kAttrLeave) {
      q = v;
      c = attr_take(ctr, q, nq, nchunks, lane);
    }
  }
  return c;
}

// A chunk of any queue that has one left, or nchunks (the counters are read by all lanes at once).
__device__ __forceinline__ unsigned attr_left(unsigned* __restrict__ ctr, unsigned nq, unsigned nchunks, int lane) {
  for (unsigned v0 = 0; v0 < nq; v0 += 32) {
    const unsigned v = v0 + lane;
    const unsigned taken = v < nq ? __ldcg(ctr + (1 + v) * kAttrCtrStride) : 0u;
    unsigned some = __ballot_sync(0xffffffffu, v < nq && taken < attr_queue(v, nq, nchunks).size);
    for (; some; some &= some - 1u) {
      const unsigned c = attr_take(ctr, v0 + __ffs(some) - 1, nq, nchunks, lane);
      if (c < nchunks) return c;
    }
  }
  return nchunks;
}

// Per iteration on discs (see above) of 1M points (143 M entries, 90 neighbours): 0.508 -> 0.326 ms; 200,000: 98 -> 80
// us. The queues took the L1 hit rate from 27 to 77 % there and the time to 0.35 ms; the rest came from the
// masks, the shared reductions and the prefetch. On an optimised layout of 1M points in 30 clusters: 0.582 -> 0.495 ms
// (hits 22 -> 54 % at 200,000 points). Six blocks per SM with a few spilled registers are
// faster than five without (0.360 ms at 1M). Rounds narrower than 128 entries at a row's end would
// save instructions but sum a row in another order; they measured 0.317 ms and are not used.
__global__ void __launch_bounds__(kAttrThreads, 6)
attractive_kernel(const int2* __restrict__ slot_rows, const int* __restrict__ col, const float* __restrict__ val,
                  const float2* __restrict__ y, int n, float exag, float2* __restrict__ attr,
                  unsigned* __restrict__ ctr, int chunk, unsigned nq) {
  const int lane = threadIdx.x & 31;
  const unsigned nchunks = (unsigned)((n + chunk - 1) / chunk);
  // with a warp for every chunk, warp w takes chunk w and no counter is touched
  const bool queued = nchunks > gridDim.x * kAttrWarps;
  unsigned q = 0, c = blockIdx.x * kAttrWarps + (threadIdx.x >> 5), next = nchunks;
  unsigned rnd = c * 2654435761u;
  bool sweep = false;
  auto pop = [&]() -> unsigned {
    if (!queued) return nchunks;
    if (!sweep) return attr_pop(ctr, q, nq, nchunks, rnd, lane);
    return attr_left(ctr, nq, nchunks, lane);
  };
  if (queued) {
    asm("mov.u32 %0, %%smid;" : "=r"(q));
    q %= nq;
    // a block's first two chunks per warp come with one atomic
    __shared__ unsigned s_first;
    if (threadIdx.x == 0) s_first = atomicAdd(ctr + (1 + q) * kAttrCtrStride, 2u * kAttrWarps);
    __syncthreads();
    const AttrQueue Q = attr_queue(q, nq, nchunks);
    const unsigned t0 = s_first + (threadIdx.x >> 5), t1 = t0 + kAttrWarps;
    c = t0 < Q.size ? Q.begin + t0 : pop();
    if (c < nchunks) next = t1 < Q.size ? Q.begin + t1 : pop();
  }
  // lane l holds the bounds of row l of the chunk (chunk <= 32) and its point, so a row's bounds cost
  // no load; the next chunk's are loaded while this one is processed
  auto rows_of = [&](unsigned ch, int2& se, float2& yl) {
    const long long s = (long long)ch * chunk + lane;
    se = make_int2(0, 0);
    yl = make_float2(0.0f, 0.0f);
    if (ch < nchunks && lane < chunk && s < n) {
      se = __ldg(slot_rows + s);
      yl = __ldg(y + s);
    }
  };
  int2 se;
  float2 yl;
  for (;;) {
    rows_of(c, se, yl);
    if (lane < 2) prefetch_row(col, val, se);
    while (c < nchunks) {
      int2 sn;
      float2 yn;
      rows_of(next, sn, yn);
      const int s0 = (int)c * chunk, rows = min(chunk, n - s0);
      for (int t = 0; t < rows; t += 2) {
        // L2 prefetch of the two rows after these, in this chunk or the next: further ahead the
        // rows in flight of all warps no longer fit L2 (8 rows: 0.42 ms at 1M)
        const bool inside = t + 2 < chunk;
        if (inside ? (lane >> 1) == (t >> 1) + 1 : lane < 2) prefetch_row(col, val, inside ? se : sn);
        float2 a[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          // a missing second row has bounds (0, 0) in its lane, or repeats nothing past lane 31
          const int src = min(t + u, 31);
          const int b = __shfl_sync(0xffffffffu, se.x, src), e = __shfl_sync(0xffffffffu, se.y, src);
          const float2 yi = make_float2(__shfl_sync(0xffffffffu, yl.x, src), __shfl_sync(0xffffffffu, yl.y, src));
          a[u] = attr_row(col, val, y, b, t + u < rows ? e : b, s0 + t + u, yi, lane);
        }
        const float sum = exag * butterfly_rows(a[0].x, a[0].y, a[1].x, a[1].y, lane);
        // lanes 0, 8, 16, 24 hold x0, x1, y0, y1
        const int u = (lane >> 3) & 1;
        if ((lane & 7) == 0 && t + u < rows) reinterpret_cast<float*>(attr + s0 + t + u)[lane >> 4] = sum;
      }
      c = next;
      se = sn;
      yl = yn;
      if (c < nchunks) next = pop();
    }
    if (!queued || sweep) break;
    // the last block to finish takes whatever is left (chunks of an SM that ran no block of this
    // launch and that no probe met), then clears the counters for the next launch
    if (!last_block_done(ctr, gridDim.x)) return;
    sweep = true;
    q = 0;
    c = pop();
    next = c < nchunks ? pop() : nchunks;
  }
  if (sweep) {
    __syncthreads();
    for (unsigned v = threadIdx.x; v < nq; v += blockDim.x) ctr[(1 + v) * kAttrCtrStride] = 0u;
  }
}

// slot_rows[t] = CSR segment of the point stored in slot t.
__global__ void bind_rows_kernel(const int* __restrict__ perm, const int* __restrict__ row_ptr, int n,
                                 int2* __restrict__ slot_rows) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int o = perm[t];
    slot_rows[t] = make_int2(row_ptr[o], row_ptr[o + 1]);
  }
}

// ---------------------------------------------------------------- update
template <int TAPS>
__device__ __forceinline__ float pick(const float (&w)[TAPS], int a) {
  float v = w[0];
#pragma unroll
  for (int t = 1; t < TAPS; ++t) v = a == t ? w[t] : v;
  return v;
}

__device__ __forceinline__ int sign3(float v) { return (v > 0.0f) - (v < 0.0f); }

// One thread per point: interpolate the potentials, form the gradient
//   g_i = a_i - ((y_i - c) phi_q2 - phi_xy) / Z     (src/tsne_neighbors.cpp:1247-1259)
// and apply gains / momentum / step clip (apply_open_tsne_update_f, :1297-1336) with the
// recentring of zero_mean_f (:1280-1291) folded in by subtracting the previous mean. The
// epilogue reduces bounding box and mean of the new layout into `next`. DIAG writes the
// repulsive force instead of updating.
template <int TAPS, bool DIAG>
__global__ void __launch_bounds__(kStepThreads)
update_kernel(float2* __restrict__ y, const float2* __restrict__ attr, float2* __restrict__ gains,
              float2* __restrict__ update, const TsneInstance* __restrict__ inst, const int2* __restrict__ blocks,
              const GridState* __restrict__ cur, GridState* __restrict__ next, StepPartial* __restrict__ part,
              unsigned* __restrict__ counter, int n, int mode, float lr, float mom, float min_gain, float max_step,
              float2* __restrict__ out_rep) {
  const int2 bl = point_block(blocks);
  const int i = bl.y + threadIdx.x;
  // the point's state is requested beside the instance and grid records (clamped: the last block of
  // the last instance may reach past the end)
  const int ic = min(i, n - 1);
  const float2 p = y[ic];
  float2 a = make_float2(0.0f, 0.0f), ga = a, up = a;
  if constexpr (!DIAG) {
    a = attr[ic];
    ga = gains[ic];
    up = update[ic];
  }
  const TsneInstance I = inst[bl.x];
  const GridState g = cur[bl.x];
  const float4* __restrict__ pot = I.potential;
  const int grid = I.grid;
  const float lr_i = lr * I.lr_mult;
  const bool clip = isfinite(max_step) && max_step > 0.0f;
  const float max2 = max_step * max_step;
  float mnx = FLT_MAX, mxx = -FLT_MAX, mny = FLT_MAX, mxy = -FLT_MAX, sx = 0.0f, sy = 0.0f;
  if (i < I.pt_begin + I.n) {
    const Stencil<TAPS> stx = make_stencil<TAPS>(p.x, g.x0, g.inv_h, g.inv_box, g.nodes);
    const Stencil<TAPS> sty = make_stencil<TAPS>(p.y, g.y0, g.inv_h, g.inv_box, g.nodes);
    float r0 = 0.0f, r1 = 0.0f, r2 = 0.0f;
#pragma unroll
    for (int v = 0; v < TAPS; ++v) {
      const float4* row = pot + (long long)(sty.base + v) * grid + stx.base;
#pragma unroll
      for (int b = 0; b < TAPS; ++b) {
        const float w = sty.w[v] * stx.w[b];
        const float4 f = __ldg(row + b);
        r0 += w * f.x;
        r1 += w * f.y;
        r2 += w * f.z;
      }
    }
    const float repx = -((p.x - g.cx) * r0 - r1) * g.inv_z;
    const float repy = -((p.y - g.cy) * r0 - r2) * g.inv_z;
    if constexpr (DIAG) {
      out_rep[i] = make_float2(repx, repy);
    } else {
      const float gx = repx + a.x, gy = repy + a.y;
      float gnx = sign3(up.x) != sign3(gx) ? ga.x + 0.2f : ga.x * 0.8f + min_gain;
      float gny = sign3(up.y) != sign3(gy) ? ga.y + 0.2f : ga.y * 0.8f + min_gain;
      if (gnx < min_gain) gnx = min_gain;
      if (gny < min_gain) gny = min_gain;
      float ux = mom * up.x - lr_i * gnx * gx;
      float uy = mom * up.y - lr_i * gny * gy;
      const float s2 = ux * ux + uy * uy;
      if (clip && s2 > max2) {
        const float sc = max_step / sqrtf(fmaxf(s2, FLT_MIN));
        ux *= sc;
        uy *= sc;
      }
      const float nx = (p.x - (float)g.mean_x) + ux;
      const float ny = (p.y - (float)g.mean_y) + uy;
      gains[i] = make_float2(gnx, gny);
      update[i] = make_float2(ux, uy);
      y[i] = make_float2(nx, ny);
      mnx = mxx = nx;
      mny = mxy = ny;
      sx = nx;
      sy = ny;
    }
  }
  if constexpr (!DIAG) {
    block_partial(mnx, mxx, mny, mxy, sx, sy, part + blockIdx.x);
    if (last_block_done(counter + bl.x, I.blocks))
      finish_layout_stats(part + I.block_begin, I.blocks, I.n, I.grid, mode, next + bl.x);
  }
}

__global__ void fill_state_kernel(float2* __restrict__ gains, float2* __restrict__ update, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    gains[i] = make_float2(1.0f, 1.0f);
    update[i] = make_float2(0.0f, 0.0f);
  }
}

__global__ void finalize_kernel(const float2* __restrict__ y, const TsneInstance* __restrict__ inst,
                                const int2* __restrict__ blocks, const GridState* __restrict__ next,
                                const int* __restrict__ perm, float2* __restrict__ out) {
  const int2 bl = blocks[blockIdx.x];
  const TsneInstance& I = inst[bl.x];
  const float mx = (float)next[bl.x].mean_x, my = (float)next[bl.x].mean_y;
  const int i = bl.y + threadIdx.x;
  if (i < I.pt_begin + I.n) {
    const float2 p = y[i];
    out[perm ? perm[i] : i] = make_float2(p.x - mx, p.y - my);
  }
}

// ---------------------------------------------------------------- spatial reorder
__device__ __forceinline__ unsigned spread_bits(unsigned v) {
  v &= 0xffffu;
  v = (v | (v << 8)) & 0x00ff00ffu;
  v = (v | (v << 4)) & 0x0f0f0f0fu;
  v = (v | (v << 2)) & 0x33333333u;
  v = (v | (v << 1)) & 0x55555555u;
  return v;
}

// Sort key: instance index above the Morton code of the stencil anchor, so a stable sort keeps
// every instance inside its slot range.
template <int TAPS>
__global__ void anchor_keys_kernel(const float2* __restrict__ y, const TsneInstance* __restrict__ inst,
                                   const int2* __restrict__ blocks, const GridState* __restrict__ next,
                                   int morton_bits, unsigned* __restrict__ keys, int* __restrict__ order) {
  const int2 bl = blocks[blockIdx.x];
  const TsneInstance& I = inst[bl.x];
  const GridState g = next[bl.x];
  const int i = bl.y + threadIdx.x;
  if (i < I.pt_begin + I.n) {
    const float2 p = y[i];
    const int bx = make_stencil<TAPS>(p.x, g.x0, g.inv_h, g.inv_box, g.nodes).base;
    const int by = make_stencil<TAPS>(p.y, g.y0, g.inv_h, g.inv_box, g.nodes).base;
    keys[i] = ((unsigned)bl.x << morton_bits) | spread_bits((unsigned)bx) | (spread_bits((unsigned)by) << 1);
    order[i] = i;
  }
}

__global__ void gather_points_kernel(const int* __restrict__ order, int n, const float2* __restrict__ y,
                                     const float2* __restrict__ gains, const float2* __restrict__ update,
                                     const int* __restrict__ perm, float2* __restrict__ scratch,
                                     int* __restrict__ perm_tmp, int* __restrict__ delta) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int o = order[r];
    scratch[r] = y[o];
    scratch[n + r] = gains[o];
    scratch[2 * (long long)n + r] = update[o];
    perm_tmp[r] = perm[o];
    delta[o] = r;
  }
}

__global__ void scatter_points_kernel(const float2* __restrict__ scratch, const int* __restrict__ perm_tmp, int n,
                                      const int* __restrict__ row_ptr, float2* __restrict__ y,
                                      float2* __restrict__ gains, float2* __restrict__ update, int* __restrict__ perm,
                                      int* __restrict__ inv, int2* __restrict__ slot_rows) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    y[r] = scratch[r];
    gains[r] = scratch[n + r];
    update[r] = scratch[2 * (long long)n + r];
    const int o = perm_tmp[r];
    perm[r] = o;
    inv[o] = r;
    slot_rows[r] = make_int2(row_ptr[o], row_ptr[o + 1]);
  }
}

// col[t] = delta[col[t]] for every entry, row by row in storage order. A block takes consecutive slots, whose
// rows name points near one another: most gathers then hit L1, where a pass over the entries in the order of the CSR (rows in
// the caller's order) is bound by the rate of random sectors from L2. Two rows of a warp are in flight, 128
// entries each. 1M points x 90 neighbours (115M entries): 575 -> 326 us on discs, 484 on an optimised
// layout (540 the first time, out of the caller's order), of 135 for moving the columns once. Shares of some 70 rows even out the row lengths: with 8 blocks
// per SM the pass took 425 us (discs), a third of it waiting for the longest shares.
// (positions are unsigned, as in attr_row)
__device__ __forceinline__ int4 relabel_load(const int* __restrict__ col, uint2 se, unsigned i) {
  int4 v = make_int4(0, 0, 0, 0);
  if (i >= se.x && i + 4 <= se.y) return __ldcs(reinterpret_cast<const int4*>(col + i));
  if (i >= se.x && i < se.y) v.x = col[i];
  if (i + 1 >= se.x && i + 1 < se.y) v.y = col[i + 1];
  if (i + 2 >= se.x && i + 2 < se.y) v.z = col[i + 2];
  if (i + 3 >= se.x && i + 3 < se.y) v.w = col[i + 3];
  return v;
}
__device__ __forceinline__ void relabel_store(int* __restrict__ col, uint2 se, unsigned i, int4 v) {
  if (i >= se.x && i + 4 <= se.y) {
    __stcs(reinterpret_cast<int4*>(col + i), v);
    return;
  }
  if (i >= se.x && i < se.y) col[i] = v.x;
  if (i + 1 >= se.x && i + 1 < se.y) col[i + 1] = v.y;
  if (i + 2 >= se.x && i + 2 < se.y) col[i + 2] = v.z;
  if (i + 3 >= se.x && i + 3 < se.y) col[i + 3] = v.w;
}
__global__ void __launch_bounds__(256)
relabel_rows_kernel(int* __restrict__ col, const int2* __restrict__ slot_rows, int n, const int* __restrict__ delta) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (n + (int)gridDim.x - 1) / (int)gridDim.x;
  const int first = (int)blockIdx.x * per, last = min(n, first + per);
  auto bounds = [&](int r) {
    const int2 se = r < last ? slot_rows[r] : make_int2(0, 0);
    return make_uint2(se.x, se.y);
  };
  uint2 a = bounds(first + warp), b = bounds(first + warp + 8);
  for (int r = first + warp; r < last; r += 16) {
    const uint2 an = bounds(r + 16), bn = bounds(r + 24);
    unsigned ia = (a.x & ~3u) + lane * 4, ib = (b.x & ~3u) + lane * 4;
    while (__any_sync(0xffffffffu, ia < a.y || ib < b.y)) {
      int4 va = relabel_load(col, a, ia), vb = relabel_load(col, b, ib);
      va = make_int4(delta[va.x], delta[va.y], delta[va.z], delta[va.w]);
      vb = make_int4(delta[vb.x], delta[vb.y], delta[vb.z], delta[vb.w]);
      relabel_store(col, a, ia, va);
      relabel_store(col, b, ib, vb);
      ia += 128;
      ib += 128;
    }
    a = an;
    b = bn;
  }
}

__global__ void identity_kernel(int* __restrict__ perm, int* __restrict__ inv, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    perm[i] = i;
    inv[i] = i;
  }
}

// ---------------------------------------------------------------- host side
namespace {
int point_blocks(int n) { return std::max(1, std::min(ceil_div(n, 256), sm_count() * 8)); }

template <typename K>
int persistent_blocks(K kernel, int threads, long long warps_needed) {
  int per_sm = 0;
  FE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0));
  per_sm = std::max(1, per_sm);
  return std::max(1, (int)std::min<long long>((long long)per_sm * sm_count(), (warps_needed + threads / 32 - 1) /
                                                                                   (threads / 32)));
}

int log2_ceil(int v) {
  int b = 0;
  while ((1 << b) < v) ++b;
  return b;
}
}  // namespace

TsneDevice::~TsneDevice() {
  if (fork) cudaEventDestroy(fork);
  if (join) cudaEventDestroy(join);
  if (side) cudaStreamDestroy(side);
}

int default_grid_size(int n, int /*mode*/) { return cuda_fft_grid_size(n); }

void tsne_device_alloc(TsneDevice& d, int n, int grid, int mode, cudaStream_t s) {
  tsne_batch_alloc(d, std::vector<int>{n}, std::vector<int>{grid}, std::vector<float>{1.0f}, mode, s);
}

namespace {
// Group instances by grid size, allocate the class workspaces in d.grid_arena and point the
// instance table at them (host copy; the caller uploads it). The set-up runs on s and waits for s alone: waiting for the
// device, or on the legacy stream, while another thread captures its graph is not allowed (the driver crashed there).
void build_grid_classes(TsneDevice& d, const std::vector<int>& grids, cudaStream_t s) {
  const int ninst = (int)d.inst.size();
  std::vector<int> distinct(grids.begin(), grids.end());
  std::sort(distinct.begin(), distinct.end());
  distinct.erase(std::unique(distinct.begin(), distinct.end()), distinct.end());
  d.classes.assign(distinct.size(), GridClass{});
  std::vector<std::vector<int>> members(distinct.size());
  for (int b = 0; b < ninst; ++b) {
    const int g = grids[b];
    if (g < 8 || g > 2048 || (g & (g - 1)) != 0) throw Error("`grid_size` must be a power of two between 8 and 2048.");
    const int c = (int)(std::lower_bound(distinct.begin(), distinct.end(), g) - distinct.begin());
    members[c].push_back(b);
  }
  d.grid_arena.release();
  int* d_members = nullptr;
  d.grid_arena.reserve(&d_members, ninst);
  for (std::size_t c = 0; c < distinct.size(); ++c) {
    GridClass& k = d.classes[c];
    k.grid = distinct[c];
    k.nodes = d.mode == kInterpBilinear ? k.grid : 3 * (k.grid / 3);
    k.fft = 2 * k.grid;
    k.log_fft = log2_ceil(k.fft);
    k.count = (int)members[c].size();
    k.first = members[c][0];
    fft_class_layout(k);
    const std::size_t m = k.fft, ld = k.ld;
    d.grid_arena.reserve(&k.charges, (std::size_t)k.count * k.grid * k.grid * kChargeStride);
    d.grid_arena.reserve(&k.potential, (std::size_t)k.count * k.grid * k.grid);
    d.grid_arena.reserve(&k.arow, (std::size_t)k.count * ld * m);
    d.grid_arena.reserve(&k.brow, (std::size_t)k.count * ld * (m / 2 + 1));
    d.grid_arena.reserve(&k.krow, (std::size_t)k.count * ld * (m / 2 + 1));
    d.grid_arena.reserve(&k.twiddle, k.twiddles);
    d.grid_arena.reserve(&k.zpart, (std::size_t)k.count * k.col_blocks);
  }
  d.grid_arena.commit("t-SNE grid workspaces");
  std::vector<int> flat;
  std::vector<std::vector<float2>> tables(distinct.size());
  int max_grid = 0;
  for (std::size_t c = 0; c < distinct.size(); ++c) {
    GridClass& k = d.classes[c];
    k.members = d_members + flat.size();
    max_grid = std::max(max_grid, k.grid);
    for (int j = 0; j < k.count; ++j) {
      const int b = members[c][j];
      flat.push_back(b);
      TsneInstance& I = d.inst[b];
      I.grid = k.grid;
      I.nodes = k.nodes;
      I.charges = k.charges + (std::size_t)j * k.grid * k.grid * kChargeStride;
      I.potential = k.potential + (std::size_t)j * k.grid * k.grid;
    }
    const std::vector<float2>& tw = tables[c] = fft_class_twiddles(k);
    FE_CUDA(cudaMemcpyAsync(k.twiddle, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice, s));
    FE_CUDA(cudaMemsetAsync(k.charges, 0, sizeof(long long) * kChargeStride * (std::size_t)k.count * k.grid * k.grid, s));
    FE_CUDA(cudaMemsetAsync(k.potential, 0, sizeof(float4) * (std::size_t)k.count * k.grid * k.grid, s));
  }
  FE_CUDA(cudaMemcpyAsync(d_members, flat.data(), sizeof(int) * ninst, cudaMemcpyHostToDevice, s));
  d.grid = d.inst[0].grid;
  d.nodes = d.inst[0].nodes;
  d.key_bits = 2 * log2_ceil(max_grid);
  d.sort_bits = d.key_bits + log2_ceil(ninst);
  if (d.sort_bits > 32) throw Error("t-SNE batch: too many instances for the spatial sort key");
  FE_CUDA(cudaStreamSynchronize(s));  // the tables go out of scope
}
}  // namespace

void tsne_batch_alloc(TsneDevice& d, const std::vector<int>& sizes, const std::vector<int>& grids,
                      const std::vector<float>& lr_mult, int mode, cudaStream_t s) {
  const int ninst = (int)sizes.size();
  if (ninst < 1 || grids.size() != sizes.size() || lr_mult.size() != sizes.size())
    throw Error("t-SNE batch: one size, grid and learning-rate multiplier per instance");
  d.mode = mode;
  d.inst.assign(ninst, TsneInstance{});
  long long total = 0;
  int nblocks = 0;
  for (int b = 0; b < ninst; ++b) {
    if (sizes[b] < 2) throw Error("t-SNE batch: every instance needs at least two points");
    TsneInstance& I = d.inst[b];
    I.pt_begin = (int)total;
    I.n = sizes[b];
    I.block_begin = nblocks;
    I.blocks = ceil_div(sizes[b], kPointBlock);
    I.lr_mult = lr_mult[b];
    total += sizes[b];
    nblocks += I.blocks;
  }
  if (total > INT_MAX / 2) throw Error("t-SNE batch: too many points");
  const int n = (int)total;
  d.n = n;
  d.nblocks = nblocks;
  d.attr_queues = sm_count();
  d.attr_blocks = persistent_blocks(attractive_kernel, kAttrThreads, n);
  // Up to 8 rows for each resident warp: one chunk a warp, without counters (20,000 points: 14 us
  // against 18 from the queues; 50,000: 24 against 29). More: queues of 4-row chunks (200,000
  // points: 79 us; 8 rows 84, 2 rows 80), of 8 rows where a warp takes many (1M: 326 against 331).
  const int warps = d.attr_blocks * kAttrWarps;
  d.attr_chunk = n <= 8 * warps ? std::max(1, ceil_div(n, warps)) : n <= 64 * warps ? 4 : 8;
  d.arena.release();
  d.arena.reserve(&d.d_inst, ninst);
  d.arena.reserve(&d.blocks, nblocks);
  d.arena.reserve(&d.y, n);
  d.arena.reserve(&d.attr, n);
  d.arena.reserve(&d.gains, n);
  d.arena.reserve(&d.update, n);
  d.arena.reserve(&d.cur, ninst);
  d.arena.reserve(&d.next, ninst);
  d.arena.reserve(&d.partial, nblocks);
  d.arena.reserve(&d.counter, ninst);
  const int nb = radix_sort_blocks(n);
  d.arena.reserve(&d.perm, n);
  d.arena.reserve(&d.inv, n);
  d.arena.reserve(&d.slot_rows, n);
  d.arena.reserve(&d.attr_ctr, (1 + (std::size_t)d.attr_queues) * kAttrCtrStride);
  d.arena.reserve(&d.keys, n);
  d.arena.reserve(&d.keys_tmp, n);
  d.arena.reserve(&d.order, n);
  d.arena.reserve(&d.order_tmp, n);
  d.arena.reserve(&d.delta, n);
  d.arena.reserve(&d.perm_tmp, n);
  d.arena.reserve(&d.scratch, 3 * (std::size_t)n);
  d.arena.reserve(&d.radix.hist, 256 * (std::size_t)nb);
  d.arena.reserve(&d.radix.offs, 256 * (std::size_t)nb + 1);
  d.arena.reserve(&d.radix.scan_tmp, ceil_div(256LL * nb, 1024));
  d.arena.commit("t-SNE optimizer state");
  d.reordered = false;
  build_grid_classes(d, grids, s);
  std::vector<int2> blk(nblocks);
  for (int b = 0; b < ninst; ++b)
    for (int t = 0; t < d.inst[b].blocks; ++t)
      blk[d.inst[b].block_begin + t] = make_int2(b, d.inst[b].pt_begin + t * kPointBlock);
  FE_CUDA(cudaMemcpyAsync(d.d_inst, d.inst.data(), sizeof(TsneInstance) * ninst, cudaMemcpyHostToDevice, s));
  FE_CUDA(cudaMemcpyAsync(d.blocks, blk.data(), sizeof(int2) * nblocks, cudaMemcpyHostToDevice, s));
  FE_CUDA(cudaMemsetAsync(d.counter, 0, sizeof(unsigned) * ninst, s));
  FE_CUDA(cudaMemsetAsync(d.attr_ctr, 0, sizeof(unsigned) * (1 + (std::size_t)d.attr_queues) * kAttrCtrStride, s));
  FE_CUDA(cudaMemsetAsync(d.cur, 0, sizeof(GridState) * ninst, s));
  if (!d.side) FE_CUDA(cudaStreamCreateWithFlags(&d.side, cudaStreamNonBlocking));
  if (!d.fork) FE_CUDA(cudaEventCreateWithFlags(&d.fork, cudaEventDisableTiming));
  if (!d.join) FE_CUDA(cudaEventCreateWithFlags(&d.join, cudaEventDisableTiming));
  FE_CUDA(cudaStreamSynchronize(s));  // blk goes out of scope
}

void tsne_regrid(TsneDevice& d, const std::vector<int>& grids, cudaStream_t s) {
  if (grids.size() != d.inst.size()) throw Error("t-SNE regrid: one grid size per instance");
  FE_CUDA(cudaStreamSynchronize(s));
  build_grid_classes(d, grids, s);
  FE_CUDA(cudaMemcpyAsync(d.d_inst, d.inst.data(), sizeof(TsneInstance) * d.inst.size(), cudaMemcpyHostToDevice, s));
  // `next` of every instance was laid out for its old grid: recompute it from the layout
  layout_stats_kernel<<<d.nblocks, kStepThreads, 0, s>>>(d.y, d.d_inst, d.blocks, d.mode, d.partial, d.counter,
                                                          d.next);
  FE_LAUNCH("layout_stats_kernel");
}

std::vector<float> tsne_grid_extents(TsneDevice& d, cudaStream_t s) {
  std::vector<GridState> g(d.inst.size());
  FE_CUDA(cudaMemcpyAsync(g.data(), d.next, sizeof(GridState) * g.size(), cudaMemcpyDeviceToHost, s));
  FE_CUDA(cudaStreamSynchronize(s));
  std::vector<float> ext(g.size());
  for (std::size_t b = 0; b < g.size(); ++b) ext[b] = g[b].h * (float)(g[b].nodes - 1);
  return ext;
}

void tsne_device_init(TsneDevice& d, const float* d_init, cudaStream_t s) {
  FE_CUDA(cudaMemcpyAsync(d.y, d_init, sizeof(float2) * d.n, cudaMemcpyDeviceToDevice, s));
  identity_kernel<<<point_blocks(d.n), 256, 0, s>>>(d.perm, d.inv, d.n);
  FE_LAUNCH("identity_kernel");
  fill_state_kernel<<<point_blocks(d.n), 256, 0, s>>>(d.gains, d.update, d.n);
  FE_LAUNCH("fill_state_kernel");
  layout_stats_kernel<<<d.nblocks, kStepThreads, 0, s>>>(d.y, d.d_inst, d.blocks, d.mode, d.partial, d.counter,
                                                          d.next);
  FE_LAUNCH("layout_stats_kernel");
}

static const int2* block_table(const TsneDevice& d) { return d.inst.size() == 1 ? nullptr : d.blocks; }

void tsne_grid_stage(TsneDevice& d, cudaStream_t s) {
  if (d.mode == kInterpBilinear)
    scatter_kernel<2><<<d.nblocks, kPointBlock, 0, s>>>(d.y, d.d_inst, block_table(d), d.cur, d.next, d.n);
  else
    scatter_kernel<3><<<d.nblocks, kPointBlock, 0, s>>>(d.y, d.d_inst, block_table(d), d.cur, d.next, d.n);
  FE_LAUNCH("scatter_kernel");
  fft_convolve(d, s);
}

void tsne_bind_rows(TsneDevice& d, const DeviceCsr& P, cudaStream_t s) {
  if (P.n != d.n) throw Error("t-SNE: P and the optimizer state have different sizes");
  bind_rows_kernel<<<point_blocks(d.n), 256, 0, s>>>(d.perm, P.row_ptr, d.n, d.slot_rows);
  FE_LAUNCH("bind_rows_kernel");
}

void tsne_attractive_stage(TsneDevice& d, const DeviceCsr& P, float exag, cudaStream_t s) {
  attractive_kernel<<<d.attr_blocks, kAttrThreads, 0, s>>>(d.slot_rows, P.col, P.val, d.y, d.n, exag, d.attr,
                                                           d.attr_ctr, d.attr_chunk, (unsigned)d.attr_queues);
  FE_LAUNCH("attractive_kernel");
}

// Run-time tuning of the attractive pass's launch: every (chunk, resident blocks per SM)
// candidate is launched once as warm-up and timed over `reps` launches with CUDA events on s, on
// the current layout (the pass only writes the attractive force, which the next iteration
// overwrites, so the optimizer state is untouched); the fastest is kept. Returns true when the
// choice changed (captured graphs hold the old launch).
bool tsne_tune_attractive(TsneDevice& d, const DeviceCsr& P, float exag, cudaStream_t s) {
  int per_sm = 0;
  FE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, attractive_kernel, kAttrThreads, 0));
  per_sm = std::max(1, per_sm);
  const int chunks[] = {2, 4, 8};
  const int old_chunk = d.attr_chunk, old_blocks = d.attr_blocks;
  cudaEvent_t e0, e1;
  FE_CUDA(cudaEventCreate(&e0));
  FE_CUDA(cudaEventCreate(&e1));
  constexpr int reps = 2;
  float best = -1.0f;
  int best_chunk = old_chunk, best_blocks = old_blocks;
  d.tuning.clear();
  for (int per = per_sm; per >= std::max(1, per_sm - 1); --per) {
    const int blocks = std::max(1, std::min(per * sm_count(), ceil_div(d.n, kAttrThreads / 32)));
    for (int chunk : chunks) {
      d.attr_chunk = chunk;
      d.attr_blocks = blocks;
      tsne_attractive_stage(d, P, exag, s);
      FE_CUDA(cudaEventRecord(e0, s));
      for (int r = 0; r < reps; ++r) tsne_attractive_stage(d, P, exag, s);
      FE_CUDA(cudaEventRecord(e1, s));
      FE_CUDA(cudaEventSynchronize(e1));
      float ms = 0.0f;
      FE_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      ms /= reps;
      d.tuning.push_back({chunk, blocks, ms});
      if (best < 0.0f || ms < best) {
        best = ms;
        best_chunk = chunk;
        best_blocks = blocks;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  d.attr_chunk = best_chunk;
  d.attr_blocks = best_blocks;
  d.tuned = true;
  return best_chunk != old_chunk || best_blocks != old_blocks;
}

void tsne_update_stage(TsneDevice& d, float lr, float mom, float min_gain, float max_step, cudaStream_t s) {
  if (d.mode == kInterpBilinear)
    update_kernel<2, false><<<d.nblocks, kStepThreads, 0, s>>>(d.y, d.attr, d.gains, d.update, d.d_inst, block_table(d),
                                                                d.cur, d.next, d.partial, d.counter, d.n, d.mode, lr, mom,
                                                                min_gain, max_step, nullptr);
  else
    update_kernel<3, false><<<d.nblocks, kStepThreads, 0, s>>>(d.y, d.attr, d.gains, d.update, d.d_inst, block_table(d),
                                                                d.cur, d.next, d.partial, d.counter, d.n, d.mode, lr, mom,
                                                                min_gain, max_step, nullptr);
  FE_LAUNCH("update_kernel");
}

void tsne_iteration(TsneDevice& d, const DeviceCsr& P, float exag, float lr, float mom, float min_gain,
                    float max_step, cudaStream_t s) {
  FE_CUDA(cudaEventRecord(d.fork, s));
  FE_CUDA(cudaStreamWaitEvent(d.side, d.fork, 0));
  tsne_attractive_stage(d, P, exag, d.side);
  FE_CUDA(cudaEventRecord(d.join, d.side));
  tsne_grid_stage(d, s);
  FE_CUDA(cudaStreamWaitEvent(s, d.join, 0));
  tsne_update_stage(d, lr, mom, min_gain, max_step, s);
}

void tsne_forces(TsneDevice& d, const DeviceCsr& P, float exag, float* d_attr, float* d_rep, cudaStream_t s) {
  tsne_attractive_stage(d, P, exag, s);
  tsne_grid_stage(d, s);
  FE_CUDA(cudaMemcpyAsync(d_attr, d.attr, sizeof(float2) * d.n, cudaMemcpyDeviceToDevice, s));
  float2* r = reinterpret_cast<float2*>(d_rep);
  if (d.mode == kInterpBilinear)
    update_kernel<2, true><<<d.nblocks, kStepThreads, 0, s>>>(d.y, d.attr, d.gains, d.update, d.d_inst, block_table(d),
                                                               d.cur, d.next, d.partial, d.counter, d.n, d.mode, 0.0f,
                                                               0.0f, 0.0f, 0.0f, r);
  else
    update_kernel<3, true><<<d.nblocks, kStepThreads, 0, s>>>(d.y, d.attr, d.gains, d.update, d.d_inst, block_table(d),
                                                               d.cur, d.next, d.partial, d.counter, d.n, d.mode, 0.0f,
                                                               0.0f, 0.0f, 0.0f, r);
  FE_LAUNCH("update_kernel(diagnostic)");
}

void tsne_finalize(TsneDevice& d, float* d_out, cudaStream_t s) {
  finalize_kernel<<<d.nblocks, kPointBlock, 0, s>>>(d.y, d.d_inst, d.blocks, d.next, d.perm,
                                                     reinterpret_cast<float2*>(d_out));
  FE_LAUNCH("finalize_kernel");
}

void tsne_reorder(TsneDevice& d, DeviceCsr& P, cudaStream_t s) {
  const int n = d.n;
  if (d.mode == kInterpBilinear)
    anchor_keys_kernel<2><<<d.nblocks, kPointBlock, 0, s>>>(d.y, d.d_inst, d.blocks, d.next, d.key_bits, d.keys,
                                                            d.order);
  else
    anchor_keys_kernel<3><<<d.nblocks, kPointBlock, 0, s>>>(d.y, d.d_inst, d.blocks, d.next, d.key_bits, d.keys,
                                                            d.order);
  FE_LAUNCH("anchor_keys_kernel");
  radix_sort_pairs(d.keys, d.order, d.keys_tmp, d.order_tmp, n, d.sort_bits, d.radix, s);
  gather_points_kernel<<<point_blocks(n), 256, 0, s>>>(d.order, n, d.y, d.gains, d.update, d.perm, d.scratch,
                                                       d.perm_tmp, d.delta);
  FE_LAUNCH("gather_points_kernel");
  scatter_points_kernel<<<point_blocks(n), 256, 0, s>>>(d.scratch, d.perm_tmp, n, P.row_ptr, d.y, d.gains, d.update,
                                                        d.perm, d.inv, d.slot_rows);
  FE_LAUNCH("scatter_points_kernel");
  relabel_rows_kernel<<<std::max(1, std::min(ceil_div(n, 16), sm_count() * 96)), 256, 0, s>>>(P.col, d.slot_rows, n,
                                                                                            d.delta);
  FE_LAUNCH("relabel_rows_kernel");
  d.reordered = true;
}

int tsne_reorder_launches(const TsneDevice& d) {
  // keys, radix passes x (histogram + 3-kernel scan + scatter), gather, scatter, relabel
  return 1 + ceil_div(d.sort_bits, 8) * 5 + 3;
}

int tsne_launches_per_iteration(const TsneDevice& d) { return 3 + 3 * (int)d.classes.size(); }

}  // namespace fe
