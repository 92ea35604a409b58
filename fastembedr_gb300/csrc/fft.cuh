// Complex FFTs of length M = 16 .. 4096 held in the registers of T = M / E threads, E values each
// (4, 8 or 16), with an exchange through shared memory between register passes.
//
// Radix-2 butterflies throughout: forward transforms are decimation in frequency (natural order in,
// bit-reversed order out), inverse transforms decimation in time (bit-reversed in, natural out). The
// stages are done two to four at a time in registers, in passes of R1, R2 and R3 values:
//   pass 1 (top stages): v[e] = value tid + e T, so global memory is read and written in
//          consecutive addresses on the natural-order side;
//   pass 2: v[i R2 + e] = value (q / R3) R3 R2 + q % R3 + e R3, q = tid + i T;
//   pass 3 (last stages): v[i R3 + e] = value q R3 + e, q = tid + i T.
// A thread ends a forward transform with exactly the values its inverse transform begins with, so a
// convolution multiplies in registers. Twiddles come from one table per pass, [entry][j] with j
// consecutive across threads (a stride of M / 2^stage in a single table of M / 2 cost as many
// cache wavefronts as the data). Transforms whose upper half of inputs is zero, or whose upper
// half of outputs is not needed, leave that half of the top stage out.
#pragma once

#include <cuda_runtime.h>

namespace fe {

constexpr int fft_log2(int v) { return v <= 1 ? 0 : 1 + fft_log2(v / 2); }

template <int LOGM>
struct FftPlan {
  static constexpr int M = 1 << LOGM;
  static constexpr int E = LOGM >= 10 ? 16 : LOGM >= 5 ? 8 : 4;  // values per thread
  static constexpr int T = M / E;
  static constexpr int R1 = E;
  static constexpr int R2 = LOGM == 4 || LOGM == 5 || LOGM == 7 ? 4 : LOGM >= 11 ? 16 : 8;
  static constexpr int R3 = M / (R1 * R2);      // 1: two passes
  static constexpr int RL = R3 == 1 ? R2 : R3;  // values of the last pass
  static_assert(R1 * R2 * R3 == M && E % R2 == 0 && E % R3 == 0, "passes");
  // twiddle tables: pass 1, pass 2, pass 3
  static constexpr int TW2 = (R1 - 1) * (M / R1), TW3 = TW2 + (R2 - 1) * R3, TWIDDLES = TW3 + (R3 - 1);
  // Shared-memory slot of value i: the low bits are exchanged with higher ones so that every pass of
  // M >= 256 is free of bank conflicts (64-bit accesses; the map is linear in the bits of i).
  static __host__ __device__ constexpr int slot(int i) {
    return LOGM >= 11 ? i ^ ((i >> 4) & 15)
           : LOGM >= 9 ? i ^ ((i >> 4) & 7) ^ ((i >> 3) & 8)
           : LOGM == 8 ? i ^ ((i >> 4) & 3) ^ ((i >> 3) & 12)
                       : i ^ ((i >> 4) & 7);
  }
};

// Complex products of the forward and the inverse butterflies. Which product of a sum is rounded and
// which is fused is written out, so that the transforms' bits do not depend on the compiler's choice
// (layouts are reproducible bit for bit across changes of the code around them).
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 cmul_inverse(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)));
}
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ int bitrev(int f, int logm) { return (int)(__brev((unsigned)f) >> (32 - logm)); }

// The log2 R stages of one pass on R values at stride h, table entry (span - 1 + k) of stage span.
// HALF: v[R / 2 ..] is zero on entry.
template <int R, int H, bool HALF = false, int E>
__device__ __forceinline__ void dif_stages(float2 (&v)[E], int at, int j, const float2* __restrict__ tw) {
#pragma unroll
  for (int span = R / 2; span >= 1; span >>= 1)
#pragma unroll
    for (int e = 0; e < R; ++e) {
      if (e & span) continue;
      const float2 w = __ldg(tw + (span - 1 + (e & (span - 1))) * H + j);
      const float2 u = v[at + e];
      if (HALF && span == R / 2) {
        v[at + e + span] = cmul(u, w);
        continue;
      }
      const float2 x = v[at + e + span];
      v[at + e] = make_float2(__fadd_rn(u.x, x.x), __fadd_rn(u.y, x.y));
      v[at + e + span] = cmul(make_float2(__fsub_rn(u.x, x.x), __fsub_rn(u.y, x.y)), w);
    }
}
// HALF: v[R / 2 ..] is not needed on return. FIRST: the span of the first stage still to be done.
template <int R, int H, bool HALF = false, int FIRST = 1, int E>
__device__ __forceinline__ void dit_stages(float2 (&v)[E], int at, int j, const float2* __restrict__ tw) {
#pragma unroll
  for (int span = FIRST; span < R; span <<= 1)
#pragma unroll
    for (int e = 0; e < R; ++e) {
      if (e & span) continue;
      const float2 w = conjf2(__ldg(tw + (span - 1 + (e & (span - 1))) * H + j));
      const float2 x = cmul_inverse(v[at + e + span], w);
      const float2 u = v[at + e];
      v[at + e] = make_float2(__fadd_rn(u.x, x.x), __fadd_rn(u.y, x.y));
      if (!(HALF && span == R / 2)) v[at + e + span] = make_float2(__fsub_rn(u.x, x.x), __fsub_rn(u.y, x.y));
    }
}

// Shared memory <-> registers in the order of pass 1, 2 or 3.
template <int LOGM, int PASS, bool STORE>
__device__ __forceinline__ void fft_move(float2 (&v)[FftPlan<LOGM>::E], float2* __restrict__ buf, int tid) {
  using P = FftPlan<LOGM>;
  constexpr int R = PASS == 1 ? P::R1 : PASS == 2 ? P::R2 : P::R3;
  constexpr int H = PASS == 1 ? P::T : PASS == 2 ? P::R3 : 1;
#pragma unroll
  for (int i = 0; i < P::E / R; ++i) {
    const int q = tid + i * P::T;
    const int base = P::slot((q / H) * (H * R) + q % H);
#pragma unroll
    for (int e = 0; e < R; ++e) {
      float2& s = buf[base ^ P::slot(e * H)];
      if (STORE) s = v[i * R + e];
      else v[i * R + e] = s;
    }
  }
}
// The last pass's order: pass 3, or pass 2 of a two-pass length.
template <int LOGM, bool STORE>
__device__ __forceinline__ void fft_move_last(float2 (&v)[FftPlan<LOGM>::E], float2* __restrict__ buf, int tid) {
  fft_move<LOGM, FftPlan<LOGM>::R3 == 1 ? 2 : 3, STORE>(v, buf, tid);
}

// Pass 1 of a forward transform, on the values tid + e T in v.
template <int LOGM, bool HALF>
__device__ __forceinline__ void fft_top(float2 (&v)[FftPlan<LOGM>::E], int tid, const float2* __restrict__ tw) {
  dif_stages<FftPlan<LOGM>::R1, FftPlan<LOGM>::T, HALF>(v, 0, tid, tw);
}

// The passes after fft_top, exchanged through buf (M slots, free on entry); v ends in the last pass's
// order. Every thread of the block calls it (block barriers); buf is free again after the caller's
// next barrier.
template <int LOGM>
__device__ __forceinline__ void fft_forward(float2 (&v)[FftPlan<LOGM>::E], float2* __restrict__ buf, int tid,
                                            const float2* __restrict__ tw) {
  using P = FftPlan<LOGM>;
  fft_move<LOGM, 1, true>(v, buf, tid);
  __syncthreads();
  fft_move<LOGM, 2, false>(v, buf, tid);
#pragma unroll
  for (int i = 0; i < P::E / P::R2; ++i)
    dif_stages<P::R2, P::R3>(v, i * P::R2, (tid + i * P::T) % P::R3, tw + P::TW2);
  if constexpr (P::R3 > 1) {
    fft_move<LOGM, 2, true>(v, buf, tid);  // the slots this thread read
    __syncthreads();
    fft_move<LOGM, 3, false>(v, buf, tid);
#pragma unroll
    for (int i = 0; i < P::E / P::R3; ++i) dif_stages<P::R3, 1>(v, i * P::R3, 0, tw + P::TW3);
  }
}

// The first inverse stage on a spectrum in the last pass's order, value e multiplied by k(e): the
// products of the sums' first terms are fused into the sums.
template <int LOGM, typename K>
__device__ __forceinline__ void fft_scale_first(float2 (&v)[FftPlan<LOGM>::E], const float2* __restrict__ tw, K k) {
  using P = FftPlan<LOGM>;
  const float2 w = conjf2(__ldg(tw + (P::R3 == 1 ? P::TW2 : P::TW3)));
#pragma unroll
  for (int e = 0; e < P::E; e += 2) {
    const float k0 = k(e), k1 = k(e + 1);
    const float2 u = v[e], x = cmul_inverse(make_float2(__fmul_rn(v[e + 1].x, k1), __fmul_rn(v[e + 1].y, k1)), w);
    v[e] = make_float2(__fmaf_rn(u.x, k0, x.x), __fmaf_rn(u.y, k0, x.y));
    v[e + 1] = make_float2(__fmaf_rn(u.x, k0, -x.x), __fmaf_rn(u.y, k0, -x.y));
  }
}

// Inverse transform (no scaling) of a spectrum in the last pass's order; on return v[e], e < E / 2, is
// value tid + e T, the lower half. buf is free on entry, and again after the caller's next barrier.
// Every thread of the block calls it; groups that are not `active` only keep the barriers. FIRST = 2:
// the first stage has been done (fft_scale_first).
template <int LOGM, int FIRST = 1>
__device__ __forceinline__ void fft_inverse_half(float2 (&v)[FftPlan<LOGM>::E], float2* __restrict__ buf, int tid,
                                                 const float2* __restrict__ tw, bool active) {
  using P = FftPlan<LOGM>;
  if constexpr (P::R3 > 1) {
    if (active) {
#pragma unroll
      for (int i = 0; i < P::E / P::R3; ++i) dit_stages<P::R3, 1, false, FIRST>(v, i * P::R3, 0, tw + P::TW3);
      fft_move<LOGM, 3, true>(v, buf, tid);
    }
    __syncthreads();
    if (active) fft_move<LOGM, 2, false>(v, buf, tid);
  }
  if (active) {
#pragma unroll
    for (int i = 0; i < P::E / P::R2; ++i)
      dit_stages<P::R2, P::R3, false, P::R3 == 1 ? FIRST : 1>(v, i * P::R2, (tid + i * P::T) % P::R3, tw + P::TW2);
    fft_move<LOGM, 2, true>(v, buf, tid);
  }
  __syncthreads();
  if (active) {
    fft_move<LOGM, 1, false>(v, buf, tid);
    dit_stages<P::R1, P::T, true>(v, 0, tid, tw);
  }
}

}  // namespace fe
