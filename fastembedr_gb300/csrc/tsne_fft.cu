// FFT convolution of the grid charges with the t-SNE kernels q = 1 / (1 + d^2) and q^2 on the
// zero-padded M x M torus (M = 2 G): the reference's grid stage (fastEmbedR
// src/tsne_neighbors.cpp:1214-1246, src/embedding_cuda_kernels.cpp:2472-2886).
//
// Real-input savings (the three charge planes and the kernel are real):
//   * the x and y charges travel as one complex plane A = x-charge + i y-charge (all M columns);
//   * the mass plane B is real, so its row spectra are Hermitian: B^[r][M - f] = conj(B^[r][f]),
//     and only f = 0 .. M/2 is kept. Rows are transformed in pairs: one complex FFT of m_r + i m_r'
//     gives both half spectra;
//   * the kernel rows q + i q^2 are real and even in x: their spectra Kq + i Kq2 have real parts,
//     and K^[dy][M - f] = K^[dy][f], so f = 0 .. M/2 is kept;
//   * the column pass takes frequency columns in conjugate pairs (c, M - c): A_c, A_(M-c), B_c and
//     one kernel column (K_(M-c) = K_c) are transformed, B_(M-c) being conj(B_c) row by row;
//     the Parseval sum of the pair is twice that of column c (once for c = 0 and c = M/2);
//   * the inverse row pass rebuilds each pair of B rows' full spectra from their halves, packed as
//     X1 + i X2 (real parts: the first row, imaginary parts: the second).
//
// Every transform lives in registers (fft.cuh), one group of T = M / E threads per sequence and the
// sequences of a block in step, with two exchanges through shared memory per transform; zero halves
// are skipped. What bounds the passes is the number of memory wavefronts and instructions, not DRAM
// (the grid is L2-resident), so the spectra lie column by column: the column pass, which touches every
// value four times, reads and writes consecutive addresses, 16 bytes a thread, and the row passes
// move 16 bytes for a pair of rows. The previous kernels (one work item at a time through shared
// memory, run-time lengths, row-major spectra read 8 bytes per 32-byte sector, strided twiddles,
// Parseval in FP64) computed the same bits; grid stage at G = 1024, 1M points: 0.260 -> 0.143 ms,
// G = 512: 77 -> 51 us, 32 instances of G = 256: 0.57 -> 0.23 ms.
#include <cfloat>
#include <cmath>
#include <vector>

#include "fft.cuh"
#include "tsne_grid.cuh"

namespace fe {
namespace {

// Row pairs, or column pairs, per block: blocks of at least 192 threads, so that short transforms fill
// warps.
template <int LOGM>
struct Blocks {
  static constexpr int T = FftPlan<LOGM>::T;
  static constexpr int PAIRS = T >= 64 ? 1 : 64 / T;  // row passes: 3 x PAIRS x T threads
  static constexpr int COLS = T >= 64 ? 1 : 64 / T;   // column pass: 4 x COLS x T threads
  static constexpr int KROWS = 3 * PAIRS;             // kernel rows of a block of the row pass
  // Blocks per SM that the registers must leave room for. Up to M = 512 the eight values of a thread fit 64 registers
  // and twice the warps hide the barriers and exchanges (32 instances of G = 256, ten iterations: 3.72 -> 3.40 ms; one
  // instance is bound by latency and runs the same). M = 1024 spills at 64 (one instance: 0.7% slower), 2048 needs two
  // blocks of 512 threads to fill an SM.
  static constexpr int ROW_BLOCKS = LOGM == 11 ? 2 : LOGM <= 9 ? 5 : 1;
  static constexpr int COL_BLOCKS = LOGM == 11 ? 2 : LOGM <= 9 ? 4 : 1;
};

// Kernel rows dy of one block: forward FFTs of (q, q^2) at columns c (offset c or c - M, zero beyond
// +-(nodes - 1)), frequencies 0 .. M/2 kept.
template <int LOGM>
__device__ __forceinline__ void kernel_rows(float2* sbuf, int row0, int nodes, int ld, const float2* __restrict__ tw,
                                            float h, float2* __restrict__ krow) {
  using P = FftPlan<LOGM>;
  constexpr int M = P::M, HM = M / 2, KR = Blocks<LOGM>::KROWS;
  const int g = threadIdx.x / P::T, tid = threadIdx.x % P::T;
  const float yo = (float)(row0 + g) * h;
  float2* buf = sbuf + g * P::M;
  float2 v[P::E];
#pragma unroll
  for (int e = 0; e < P::E; ++e) {
    const int c = tid + e * P::T;
    const int dx = c < HM ? c : c - M;
    const float xo = (float)dx * h;
    const float q = 1.0f / __fadd_rn(1.0f, __fmaf_rn(xo, xo, __fmul_rn(yo, yo)));
    const bool in = dx <= nodes - 1 && dx >= -(nodes - 1);
    v[e] = in ? make_float2(q, q * q) : make_float2(0.0f, 0.0f);
  }
  fft_top<LOGM, false>(v, tid, tw);
  fft_forward<LOGM>(v, buf, tid, tw);
  __syncthreads();
  fft_move_last<LOGM, true>(v, buf, tid);
  __syncthreads();
  for (int t = threadIdx.x; t < KR * (HM + 1); t += KR * P::T) {
    // in the order of the positions of a spectrum (p = bitrev f: even positions, and 1 for f = M/2)
    const int r = t % KR, u = t / KR, p = u == HM ? 1 : 2 * u;
    if (row0 + r < nodes)
      krow[(long long)bitrev(p, LOGM) * ld + row0 + r] = sbuf[r * P::M + P::slot(p)];
  }
}

// Row pass. Blocks from charge_blocks on take kernel rows (see above). The others take charge rows in
// pairs (p, p + npairs), npairs = ld / 2: forward FFTs of A of both rows and of m + i m'; the rows are
// cleared for the next scatter. A spectra to arow, separated B half spectra to brow, the rows of a
// pair side by side (places 2 p and 2 p + 1 of a column). blockIdx.y: member of the grid class
// (`first` is member 0, so that a single instance waits for one load less).
template <int LOGM>
__global__ void __launch_bounds__(3 * Blocks<LOGM>::PAIRS* FftPlan<LOGM>::T, Blocks<LOGM>::ROW_BLOCKS)
rows_forward_kernel(long long* __restrict__ charges, const int* __restrict__ members, int first, int grid, int nodes,
                    int ld, const float2* __restrict__ tw, const GridState* __restrict__ cur, int charge_blocks,
                    float2* __restrict__ arow, float2* __restrict__ brow, float2* __restrict__ krow) {
  using P = FftPlan<LOGM>;
  constexpr int M = P::M, HM = M / 2, NP = Blocks<LOGM>::PAIRS, THREADS = 3 * NP * P::T;
  extern __shared__ float2 sbuf[];
  const int b = blockIdx.y == 0 ? first : members[blockIdx.y];
  if ((int)blockIdx.x >= charge_blocks) {
    kernel_rows<LOGM>(sbuf, ((int)blockIdx.x - charge_blocks) * Blocks<LOGM>::KROWS, nodes, ld, tw, cur[b].h,
                      krow + (long long)blockIdx.y * (HM + 1) * ld);
    return;
  }
  const int g = threadIdx.x / P::T, tid = threadIdx.x % P::T;
  const int npairs = ld / 2, pair0 = blockIdx.x * NP, s = g % 3, r1 = pair0 + g / 3, r2 = r1 + npairs;
  charges += (long long)blockIdx.y * grid * grid * kChargeStride;
  arow += (long long)blockIdx.y * M * ld;
  brow += (long long)blockIdx.y * (HM + 1) * ld;
  const float inv_q = cur[b].inv_qscale;
  float2* buf = sbuf + g * P::M;
  float2 v[P::E];
  // groups 0 and 1: (x, y) charges of row r1 + s; group 2: masses of both rows
  const int ra = s == 1 ? r2 : r1, rb = s == 2 ? r2 : ra;
  const bool has_a = r1 < npairs && ra < nodes, has_b = r1 < npairs && rb < nodes;
  const long long* ca = charges + (long long)ra * grid * kChargeStride + (s == 2 ? 0 : 1);
  const long long* cb = charges + (long long)rb * grid * kChargeStride + (s == 2 ? 0 : 2);
#pragma unroll
  for (int e = 0; e < P::E / 2; ++e) {
    const int c = tid + e * P::T;
    const long long x = c < nodes && has_a ? ca[(long long)c * kChargeStride] : 0ll;
    const long long y = c < nodes && has_b ? cb[(long long)c * kChargeStride] : 0ll;
    v[e] = make_float2((float)x * inv_q, (float)y * inv_q);
  }
  fft_top<LOGM, true>(v, tid, tw);
  fft_forward<LOGM>(v, buf, tid, tw);
  __syncthreads();
  // every charge of the block has been read: clear them (32 bytes a node)
  for (int t = threadIdx.x; t < 2 * NP * nodes * 2; t += THREADS) {
    const int lr = t / (2 * nodes), w = t - lr * 2 * nodes;
    const int pair = pair0 + (lr >> 1), row = pair + (lr & 1) * npairs;
    if (pair < npairs && row < nodes)
      reinterpret_cast<longlong2*>(charges + (long long)row * grid * kChargeStride)[w] = make_longlong2(0, 0);
  }
  fft_move_last<LOGM, true>(v, buf, tid);
  __syncthreads();
  for (int t = threadIdx.x; t < NP * M; t += THREADS) {
    const int q = t % NP, p = t / NP, f = bitrev(p, LOGM);
    if (pair0 + q >= npairs) continue;
    const float2* S = sbuf + 3 * q * M;
    const float2 a1 = S[P::slot(p)], a2 = S[M + P::slot(p)];
    const long long at = (long long)f * ld + 2 * (pair0 + q);
    *reinterpret_cast<float4*>(arow + at) = make_float4(a1.x, a1.y, a2.x, a2.y);
    if (f <= HM) {  // the half spectra of the two mass rows from f and its conjugate partner M - f
      const float2 z = S[2 * M + P::slot(p)];
      const float2 y = S[2 * M + P::slot(bitrev((M - f) & (M - 1), LOGM))];
      *reinterpret_cast<float4*>(brow + at) =
          make_float4(0.5f * (z.x + y.x), 0.5f * (z.y - y.y), 0.5f * (z.y + y.y), -0.5f * (z.x - y.x));
    }
  }
}

// Column pass for the conjugate pairs (c, M - c), c = 0 .. M/2: groups 0 .. 3 of a pair transform A_c,
// A_(M-c), B_c and the kernel column; the products and the Parseval sum of |B^|^2 Kq over both
// columns (Z + n up to the 1 / M^2 scale) are formed on the values in registers and the first
// three transformed back in place. The sum is kept in two floats (48 bits).
template <int LOGM>
__global__ void __launch_bounds__(4 * Blocks<LOGM>::COLS* FftPlan<LOGM>::T, Blocks<LOGM>::COL_BLOCKS)
columns_convolve_kernel(float2* __restrict__ arow, float2* __restrict__ brow, const float2* __restrict__ krow,
                        int nodes, int ld, const float2* __restrict__ tw, double* __restrict__ zpart) {
  using P = FftPlan<LOGM>;
  constexpr int M = P::M, HM = M / 2, NC = Blocks<LOGM>::COLS, WARPS = 4 * NC * P::T / 32;
  extern __shared__ float2 sbuf[];
  __shared__ double s_z[WARPS];
  const int g = threadIdx.x / P::T, tid = threadIdx.x % P::T;
  const int s = g & 3, c = blockIdx.x * NC + g / 4, c2 = (M - c) & (M - 1);
  const int npairs = ld / 2;
  const bool valid = c <= HM;
  arow += (long long)blockIdx.y * M * ld;
  brow += (long long)blockIdx.y * (HM + 1) * ld;
  krow += (long long)blockIdx.y * (HM + 1) * ld;
  float2* buf = sbuf + g * P::M;
  float2* col = s == 2 ? brow + (long long)c * ld : arow + (long long)(s == 0 ? c : c2) * ld;
  float2 v[P::E];
  if (s == 3) {
    const float2* kc = krow + (long long)c * ld;
#pragma unroll
    for (int e = 0; e < P::E; ++e) {
      const int r = tid + e * P::T, dy = r < HM ? r : M - r;
      v[e] = valid && dy < nodes ? __ldg(kc + dy) : make_float2(0.0f, 0.0f);
    }
    fft_top<LOGM, false>(v, tid, tw);
  } else {
    // rows r and r + npairs lie side by side: both belong to this thread when nodes = M / 2
    if (nodes == HM) {
#pragma unroll
      for (int e = 0; e < P::E / 4; ++e) {
        const float4 x = valid ? reinterpret_cast<const float4*>(col)[tid + e * P::T] : make_float4(0.f, 0.f, 0.f, 0.f);
        v[e] = make_float2(x.x, x.y);
        v[e + P::E / 4] = make_float2(x.z, x.w);
      }
    } else {
#pragma unroll
      for (int e = 0; e < P::E / 2; ++e) {
        const int r = tid + e * P::T;
        v[e] = valid && r < nodes ? col[r < npairs ? 2 * r : 2 * (r - npairs) + 1] : make_float2(0.0f, 0.0f);
      }
    }
    fft_top<LOGM, true>(v, tid, tw);
  }
  fft_forward<LOGM>(v, buf, tid, tw);
  __syncthreads();
  float2* kv = sbuf + (g | 3) * P::M + tid;
  if (s == 3) {
#pragma unroll
    for (int e = 0; e < P::E; ++e) kv[e * P::T] = v[e];
  }
  __syncthreads();
  Float2Sum z{0.0f, 0.0f};
  if (s == 2) {
#pragma unroll
    for (int e = 0; e < P::E; ++e) {
      const float k = kv[e * P::T].x;
      const float xx = __fmul_rn(v[e].x, v[e].x), yy = __fmul_rn(v[e].y, v[e].y);
      const Float2Sum q = two_sum(xx, yy);
      const float lo = q.lo + (__fmaf_rn(v[e].x, v[e].x, -xx) + __fmaf_rn(v[e].y, v[e].y, -yy));
      const float p = __fmul_rn(q.hi, k);
      z = add(z, Float2Sum{p, __fmaf_rn(lo, k, __fmaf_rn(q.hi, k, -p))});
    }
  }
  if (s != 3) fft_scale_first<LOGM>(v, tw, [&](int e) { return kv[e * P::T].y; });
  fft_inverse_half<LOGM, 2>(v, buf, tid, tw, s != 3);
  if (s != 3 && valid && !(s == 1 && c2 == c)) {
    if (nodes == HM) {
#pragma unroll
      for (int e = 0; e < P::E / 4; ++e)
        reinterpret_cast<float4*>(col)[tid + e * P::T] =
            make_float4(v[e].x, v[e].y, v[e + P::E / 4].x, v[e + P::E / 4].y);
    } else {
#pragma unroll
      for (int e = 0; e < P::E / 2; ++e) {
        const int r = tid + e * P::T;
        if (r < nodes) col[r < npairs ? 2 * r : 2 * (r - npairs) + 1] = v[e];
      }
    }
  }
  if (c2 != c) {
    z.hi *= 2.0f;
    z.lo *= 2.0f;
  }
  z = warp_sum(z);
  if ((threadIdx.x & 31) == 0) s_z[threadIdx.x >> 5] = value(z);
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < WARPS; ++w) t += s_z[w];
    zpart[(long long)blockIdx.y * gridDim.x + blockIdx.x] = t;
  }
}

// Inverse row pass for the row pairs -> potentials (phi_q2, phi_x, phi_y) per node. The last block of
// an instance instead finalises Z = sum_k |F_mass|^2 Kq / M^2 - n (the reference's
// sum_i q_grid(y_i) - n).
template <int LOGM>
__global__ void __launch_bounds__(3 * Blocks<LOGM>::PAIRS* FftPlan<LOGM>::T, Blocks<LOGM>::ROW_BLOCKS)
rows_inverse_kernel(const float2* __restrict__ arow, const float2* __restrict__ brow,
                    float4* __restrict__ potential, const TsneInstance* __restrict__ inst,
                    const int* __restrict__ members, int first, int grid, int nodes, int ld,
                    const float2* __restrict__ tw, const double* __restrict__ zpart, int zblocks,
                    GridState* __restrict__ cur) {
  using P = FftPlan<LOGM>;
  constexpr int M = P::M, HM = M / 2, NP = Blocks<LOGM>::PAIRS, THREADS = 3 * NP * P::T;
  extern __shared__ float2 sbuf[];
  if (blockIdx.x == gridDim.x - 1) {
    const int b = blockIdx.y == 0 ? first : members[blockIdx.y];
    __shared__ double s_z[THREADS / 32];
    double z = 0.0;
    for (int t = threadIdx.x; t < zblocks; t += THREADS) z += zpart[(long long)blockIdx.y * zblocks + t];
    z = warp_sum(z);
    if ((threadIdx.x & 31) == 0) s_z[threadIdx.x >> 5] = z;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < THREADS / 32; ++w) t += s_z[w];
      const double zz = t / ((double)M * (double)M) - (double)inst[b].n;
      cur[b].z = zz;
      cur[b].inv_z = (float)(1.0 / fmax(zz, (double)FLT_MIN));
    }
    return;
  }
  const int g = threadIdx.x / P::T, tid = threadIdx.x % P::T, npairs = ld / 2, pair0 = blockIdx.x * NP;
  potential += (long long)blockIdx.y * grid * grid;
  arow += (long long)blockIdx.y * M * ld;
  brow += (long long)blockIdx.y * (HM + 1) * ld;
  // in batches whose loads are all in flight before the first is stored
  constexpr int U = 4;
  for (int t0 = threadIdx.x; t0 < NP * M; t0 += U * THREADS) {
    float4 a[U], x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * THREADS, q = t % NP, f = bitrev(t / NP, LOGM);
      if (t >= NP * M || pair0 + q >= npairs) continue;
      const long long at = (long long)f * ld + 2 * (pair0 + q);
      a[u] = __ldg(reinterpret_cast<const float4*>(arow + at));
      if (f <= HM) x[u] = __ldg(reinterpret_cast<const float4*>(brow + at));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * THREADS, q = t % NP, p = t / NP, f = bitrev(p, LOGM);
      if (t >= NP * M || pair0 + q >= npairs) continue;
      const bool two = pair0 + q + npairs < nodes;  // the column pass writes `nodes` rows
      float2* S = sbuf + 3 * q * M;
      S[P::slot(p)] = make_float2(a[u].x, a[u].y);
      S[M + P::slot(p)] = two ? make_float2(a[u].z, a[u].w) : make_float2(0.0f, 0.0f);
      if (f <= HM) {
        if (!two) x[u].z = x[u].w = 0.0f;
        S[2 * M + P::slot(p)] = make_float2(x[u].x - x[u].w, x[u].y + x[u].z);
        if (f > 0 && f < HM) S[2 * M + P::slot(bitrev(M - f, LOGM))] = make_float2(x[u].x + x[u].w, x[u].z - x[u].y);
      }
    }
  }
  __syncthreads();
  float2* buf = sbuf + g * P::M;
  float2 v[P::E];
  fft_move_last<LOGM, false>(v, buf, tid);
  __syncthreads();
  fft_inverse_half<LOGM>(v, buf, tid, tw, true);
  __syncthreads();
#pragma unroll
  for (int e = 0; e < P::E / 2; ++e) buf[P::slot(tid + e * P::T)] = v[e];
  __syncthreads();
  const float scale = 1.0f / ((float)M * (float)M);
  for (int t = threadIdx.x; t < 2 * NP * nodes; t += THREADS) {
    const int lr = t / nodes, c = t - lr * nodes, pair = pair0 + (lr >> 1), row = pair + (lr & 1) * npairs;
    if (pair >= npairs || row >= nodes) continue;
    const float2* S = sbuf + 3 * (lr >> 1) * M + P::slot(c);
    const float2 m = S[2 * M], a = S[(lr & 1) * M];
    potential[(long long)row * grid + c] =
        make_float4(((lr & 1) ? m.y : m.x) * scale, a.x * scale, a.y * scale, 0.0f);
  }
}

template <typename K>
void allow_shared(K kernel, int bytes) {
  FE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

template <int LOGM>
struct Pass {
  using P = FftPlan<LOGM>;
  using B = Blocks<LOGM>;
  static constexpr int kSeq = P::M * (int)sizeof(float2);

  static void layout(GridClass& k) {
    k.col_blocks = (P::M / 2 + 1 + B::COLS - 1) / B::COLS;
    k.twiddles = P::TWIDDLES;
    allow_shared(rows_forward_kernel<LOGM>, 3 * B::PAIRS * kSeq);
    allow_shared(columns_convolve_kernel<LOGM>, 4 * B::COLS * kSeq);
    allow_shared(rows_inverse_kernel<LOGM>, 3 * B::PAIRS * kSeq);
  }
  static std::vector<float2> twiddles() {
    // entry (span - 1 + k) of a pass with stride h: exp(-2 pi i (j + k h) / (2 span h)), j < h
    std::vector<float2> t;
    auto table = [&](int r, int h) {
      for (int span = 1; span < r; span <<= 1)
        for (int k = 0; k < span; ++k)
          for (int j = 0; j < h; ++j) {
            const double ang = -2.0 * M_PI * (double)((j + k * h) * (P::M / (2 * span * h))) / (double)P::M;
            t.push_back(make_float2((float)std::cos(ang), (float)std::sin(ang)));
          }
    };
    table(P::R1, P::T);
    table(P::R2, P::R3);
    if (P::R3 > 1) table(P::R3, 1);
    t.resize(P::TWIDDLES);
    return t;
  }
  static void rows_forward(const TsneDevice& d, const GridClass& c, cudaStream_t s) {
    const int charge = ceil_div(c.ld / 2, B::PAIRS);
    rows_forward_kernel<LOGM><<<dim3(charge + ceil_div(c.nodes, B::KROWS), c.count), 3 * B::PAIRS * P::T,
                                3 * B::PAIRS * kSeq, s>>>(c.charges, c.members, c.first, c.grid, c.nodes, c.ld,
                                                          c.twiddle, d.cur, charge, c.arow, c.brow, c.krow);
    FE_LAUNCH("rows_forward_kernel");
  }
  static void columns(const TsneDevice&, const GridClass& c, cudaStream_t s) {
    columns_convolve_kernel<LOGM><<<dim3(c.col_blocks, c.count), 4 * B::COLS * P::T, 4 * B::COLS * kSeq, s>>>(
        c.arow, c.brow, c.krow, c.nodes, c.ld, c.twiddle, c.zpart);
    FE_LAUNCH("columns_convolve_kernel");
  }
  static void rows_inverse(const TsneDevice& d, const GridClass& c, cudaStream_t s) {
    rows_inverse_kernel<LOGM><<<dim3(ceil_div(c.ld / 2, B::PAIRS) + 1, c.count), 3 * B::PAIRS * P::T,
                                3 * B::PAIRS * kSeq, s>>>(c.arow, c.brow, c.potential, d.d_inst, c.members, c.first,
                                                          c.grid, c.nodes, c.ld, c.twiddle, c.zpart, c.col_blocks,
                                                          d.cur);
    FE_LAUNCH("rows_inverse_kernel");
  }
};

// f(Pass<LOGM>()) for the class's transform length (G = 8 .. 2048).
template <typename F>
void for_length(const GridClass& k, F&& f) {
  switch (k.log_fft) {
    case 4: return f(Pass<4>());
    case 5: return f(Pass<5>());
    case 6: return f(Pass<6>());
    case 7: return f(Pass<7>());
    case 8: return f(Pass<8>());
    case 9: return f(Pass<9>());
    case 10: return f(Pass<10>());
    case 11: return f(Pass<11>());
    case 12: return f(Pass<12>());
    default: throw Error("t-SNE grid: no transform of this length");
  }
}
}  // namespace

void fft_class_layout(GridClass& k) {
  k.ld = (k.nodes + 1) & ~1;
  for_length(k, [&](auto p) { p.layout(k); });
}
std::vector<float2> fft_class_twiddles(const GridClass& k) {
  std::vector<float2> t;
  for_length(k, [&](auto p) { t = p.twiddles(); });
  return t;
}
void fft_convolve(TsneDevice& d, cudaStream_t s) {
  for (const GridClass& c : d.classes)
    for_length(c, [&](auto p) {
      p.rows_forward(d, c, s);
      p.columns(d, c, s);
      p.rows_inverse(d, c, s);
    });
}

}  // namespace fe
