// Exponential and logarithm in two floats (exp x: within 3e-12 of itself where its low part is a normal float; log x:
// within 1e-12 (1 + |log2 x|)), for the per-row searches
// and sums whose decisions FP32 is too short for: the FP64 pipe of this part issues one warp
// instruction every 19 cycles of an SM, and an FP64 exp or log takes 40 to 50 of them (about 900
// cycles) where these take 35 to 45 FP32 instructions (about 10).
//
// Both use the table method of Tang (1989, 1990). The tables live in shared memory, filled by the
// kernel that uses them.
#pragma once

#include "common.cuh"

namespace fe {

// exp x = 2^(m / 64) exp(t), t = x - m log(2) / 64: entry j = 2^(j / 64), two floats.
constexpr int kExpEntries = 64;
__device__ __forceinline__ void fill_exp_table(float2* t) {
  for (int i = threadIdx.x; i < kExpEntries; i += blockDim.x) {
    const Float2Sum v = split(exp2((double)i / 64.0));
    t[i] = make_float2(v.hi, v.lo);
  }
}
// x <= 0 (or slightly above); results below the float range are rounded to it.
__device__ __forceinline__ Float2Sum exp_two(Float2Sum x, const float2* __restrict__ table) {
  // log(2) / 64 in three parts, the first of 11 bits so that m times it is exact for |m| < 8192
  constexpr double kStep = 0.010830424696249145265;
  constexpr float c1 = 0.010826110839843750f;  // 1419 / 131072
  constexpr float c2 = (float)(kStep - (double)c1), c3 = (float)(kStep - (double)c1 - (double)c2);
  if (!(x.hi > -174.0f)) return Float2Sum{x.hi < 0.0f ? 0.0f : x.hi, 0.0f};  // underflows (NaN stays)
  const float m = rintf(x.hi * 92.332482616893656877f);
  const int im = (int)m;
  const float pm = __fmul_rn(m, c2);
  const Float2Sum t0 = two_sum(__fmaf_rn(-m, c1, x.hi), -pm);
  const Float2Sum t = two_sum(t0.hi, t0.lo + (x.lo - __fmaf_rn(m, c2, -pm) - m * c3));
  const float h = t.hi, tl = t.lo;
  const float q = h * h * fmaf(h, fmaf(h, fmaf(h, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f), 0.5f);
  const Float2Sum e = two_sum(h, tl + q);
  const float2 T = table[im & (kExpEntries - 1)];
  const Float2Sum p = mul(Float2Sum{T.x, T.y}, e);
  const Float2Sum s = two_sum(T.x, p.hi);
  const float lo = s.lo + (T.y + p.lo);
  // two factors: the exponent may be below the smallest normal's
  const int k = im >> 6, k1 = max(k, -100);
  const float f1 = __int_as_float((127 + k1) << 23), f2 = __int_as_float((127 + max(k - k1, -126)) << 23);
  const float hi = __fadd_rn(s.hi, lo), lo2 = __fsub_rn(lo, __fsub_rn(hi, s.hi));
  return Float2Sum{hi * f1 * f2, lo2 * f1 * f2};
}

// log x = e log 2 - log r + log1p(m r - 1): x = 2^e m, m in [2/3, 4/3), r a tabulated reciprocal of m's
// neighbourhood, |m r - 1| < 0.006. The entry for m = (kLogFirst + i) / 128 is (r, -log r high, low, 0).
constexpr int kLogFirst = 85, kLogEntries = 87;
__device__ __forceinline__ void fill_log_table(float4* t) {
  for (int i = threadIdx.x; i < kLogEntries; i += blockDim.x) {
    const float r = 128.0f / (float)(kLogFirst + i);
    const Float2Sum l = split(-log((double)r));
    t[i] = make_float4(r, l.hi, l.lo, 0.0f);
  }
}
__device__ __forceinline__ Float2Sum log_two(Float2Sum x, const float4* __restrict__ table) {
  const int bits = __float_as_int(x.hi);
  const int e = (bits - 0x3f2aaaab) >> 23;  // x.hi = 2^e m, m in [2/3, 4/3)
  const float scale = __int_as_float((127 - e) << 23);
  const float m = x.hi * scale, ml = x.lo * scale;
  // (clamped: a NaN must not index outside the table)
  const float4 t = table[min(max(__float2int_rn(m * 128.0f) - kLogFirst, 0), kLogEntries - 1)];
  const float p = __fmul_rn(m, t.x);
  const float z = __fsub_rn(p, 1.0f);  // exact
  const float zl = __fadd_rn(__fmaf_rn(m, t.x, -p), __fmul_rn(ml, t.x));
  // log1p(z + zl) = z + zl - z^2 / 2 - z zl + z^3 / 3 + z^2 zl - ...
  const float w = __fmul_rn(z, z), wl = __fmaf_rn(z, z, -w);
  const float poly = __fmul_rn(__fmul_rn(w, z), __fmaf_rn(z, __fmaf_rn(z, __fmaf_rn(z, -1.0f / 6.0f, 0.2f), -0.25f),
                                                          1.0f / 3.0f));
  // log 2 = 0.693145751953125 (16 bits: e times it is exact) + 1.42860682030941723e-6
  const Float2Sum s = two_sum((float)e * 0.693145751953125f, t.y);
  const Float2Sum u = two_sum(s.hi, z), v = two_sum(u.hi, -0.5f * w);
  const float zz = __fmul_rn(z, zl), cross = __fmaf_rn(-z, zz, zz);
  const float lo = s.lo + u.lo + v.lo + t.z + zl - 0.5f * wl - cross + poly + (float)e * 1.42860682030941723e-6f;
  return two_sum(v.hi, lo);
}

}  // namespace fe
