// stats.cuh -- per-variable statistics shared by the Pearson paths.
//
// GB300's FP64 pipe runs at a small fraction of its FP32 pipe, so the sums
// over observations are compensated float pairs (Knuth's TwoSum, squares with
// their exact FMA residual), about 2^-47 relative, and so are the few
// operations that finish a variable's statistics: every lane of its warp makes
// them, and the 60 or so that they took in FP64 (16 cycles of the SM's FP64 pipe
// each) were most of the batched prologue (300 problems, 220000 variables:
// 683 us, now 450; 348 with the lighter passes below).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "kernels.cuh"

namespace gt {

// Compensated float accumulator: hi + lo carries the sum of the added values.
struct FloatPairSum {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float v) {
    const float t = hi + v;
    const float bp = t - hi;
    lo += (hi - (t - bp)) + (v - bp);
    hi = t;
  }
};

// Sum of the lanes' (hi, lo) pairs, left in every lane.  TwoSum is exact in
// either operand order, so every lane ends with the same pair.
__device__ __forceinline__ void warp_pair_sum(float &hi, float &lo) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
    const float t = hi + oh, bp = t - hi;
    lo = (lo + ol) + ((hi - (t - bp)) + (oh - bp));
    hi = t;
  }
}

// Visits x[0..n) across the warp: float4 loads when x is 16-byte aligned.
template <class F>
__device__ __forceinline__ void warp_for_each(const float *__restrict__ x, int64_t n, F &&f) {
  const int lane = threadIdx.x & 31;
  const int64_t n4 = (reinterpret_cast<uintptr_t>(x) & 15u) == 0 ? (n >> 2) : 0;
  const float4 *x4 = reinterpret_cast<const float4 *>(x);
  for (int64_t k = lane; k < n4; k += 32) {
    const float4 t = x4[k];
    f(t.x);
    f(t.y);
    f(t.z);
    f(t.w);
  }
  for (int64_t k = 4 * n4 + lane; k < n; k += 32) f(x[k]);
}

// The same, four values at a time while there are four: f4(float4), then f.
template <class F4, class F>
__device__ __forceinline__ void warp_for_each4(const float *__restrict__ x, int64_t n, F4 &&f4,
                                               F &&f) {
  const int lane = threadIdx.x & 31;
  int64_t done;
  if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) {
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    for (int64_t k = lane; k < (n >> 2); k += 32) f4(x4[k]);
    done = n & ~int64_t(3);
  } else {
    done = n & ~int64_t(127);
    for (int64_t k = lane; k < done; k += 128)
      f4(make_float4(x[k], x[k + 32], x[k + 64], x[k + 96]));
  }
  for (int64_t k = done + lane; k < n; k += 32) f(x[k]);
}

// Sum of x[0..n) as a float pair in every lane, with the count of non-NaN
// values, of NaN values, and the largest finite magnitude; values are
// multiplied by the power of two `sc` first.
struct WarpSums {
  float hi, lo;
  int cnt, nan;
  float amax;
};
__device__ __forceinline__ WarpSums warp_sums(const float *__restrict__ x, int64_t n, float sc) {
  const unsigned FULL = 0xffffffffu;
  FloatPairSum s;
  int cnt = 0, nan = 0;
  float amax = 0.f;
  warp_for_each(x, n, [&](float v) {
    if (v != v) {
      nan++;
    } else {
      s.add(v * sc);
      cnt++;
      const float a = fabsf(v);
      if (a <= 3.4e38f) amax = fmaxf(amax, a);
    }
  });
  WarpSums r;
  r.hi = s.hi;
  r.lo = s.lo;
  warp_pair_sum(r.hi, r.lo);
  r.cnt = __reduce_add_sync(FULL, cnt);
  r.nan = __reduce_add_sync(FULL, nan);
  r.amax = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(amax)));
  return r;
}

// The statistics from the scaled mean m + mlo and sum of squares q + qlo (values
// times 2^-e).
__device__ __forceinline__ ColStats colstats_finish(float m, float mlo, float q, float qlo, int e,
                                                    int flags) {
  ColStats st;
  st.mhi = m;
  st.mlo = mlo;
  st.flags = flags;
  st.e = e;
  if (flags & 2) {
    st.ihi = st.ilo = 0.f;
  } else {
    // 1/sqrt(q + qlo): an estimate y, then y (1 - r)^(-1/2) with r = 1 - (q + qlo) y^2
    const float y = rsqrtf(q), y2 = y * y, y2l = fmaf(y, y, -y2);
    const float r = fmaf(-qlo, y2, fmaf(-q, y2l, fmaf(-q, y2, 1.f)));
    const float d = y * r * fmaf(0.375f, r, 0.5f);
    st.ihi = y + d;
    st.ilo = d - (st.ihi - y);
  }
  return st;
}

// Scale exponent e with the largest magnitude in [2^e, 2^(e+1)).
__device__ __forceinline__ int binade(float amax) {
  int e = 0;
  if (amax > 0.f) e = int((__float_as_uint(amax) >> 23) & 255u) - 127;
  return e < -126 ? -126 : (e > 126 ? 126 : e);
}

// One warp's statistics of a variable x[0..n): the mean, refined by the mean
// residual (the corrected two-pass algorithm), and the inverse norm of the
// centred values.  use 0: every value counts and any NaN flags the variable;
// use 1: NaN values are skipped.  Every lane returns the same result.
// The centred pass runs on the values times 2^-e (2^e the binade of the
// largest magnitude), so its squares neither overflow nor underflow whatever
// the data's scale; the first pass is redone scaled only if its plain sum
// overflowed.  A constant variable gets a mean equal to its value (its pair
// sum is exact and the quotient is corrected), so its centred values are
// exactly 0 and it is flagged.
static __device__ __noinline__ ColStats colstats_warp_any(const float *__restrict__ x, int64_t n,
                                                   int use) {
  WarpSums w = warp_sums(x, n, 1.f);
  const int e = binade(w.amax);
  const float sc = __uint_as_float(uint32_t(127 - e) << 23);
  const float t = w.hi + w.lo;
  float shi = w.hi * sc, slo = w.lo * sc;
  if (!(t - t == 0.f) && w.amax != 0.f) {  // the plain sum overflowed
    const WarpSums ws = warp_sums(x, n, sc);
    shi = ws.hi;
    slo = ws.lo;
  }
  const int cnt = w.cnt;
  // the scaled mean as a pair: a quotient, corrected by its residual, then the
  // residual of the corrected one (exactly 0 for a constant variable)
  const float N = float(cnt), dN = float(cnt - int(N));  // dN: from 2^24 on
  const float invN = cnt > 0 ? 1.f / N : 0.f;
  auto residual = [&](float m) { return fmaf(-m, N, shi) + fmaf(-m, dN, slo); };
  const float m0 = shi * invN;
  float mhi = fmaf(residual(m0), invN, m0);
  float mlo = residual(mhi) * invN;
  FloatPairSum c, ss;
  float sse = 0.f;
  warp_for_each(x, n, [&](float v) {
    if (v != v) return;
    const float d = (v * sc - mhi) - mlo;
    c.add(d);
    const float q = d * d;
    sse += fmaf(d, d, -q);
    ss.add(q);
  });
  float chi = c.hi, clo = c.lo, qhi = ss.hi, qlo = ss.lo + sse;
  warp_pair_sum(chi, clo);
  warp_pair_sum(qhi, qlo);
  const float C = chi + clo, cm = C * invN;
  mlo += cm;
  qlo = fmaf(-C, cm, qlo);
  const float m = mhi + mlo, q = qhi + qlo;
  mlo -= m - mhi;
  qlo -= q - qhi;
  int flags = use == 0 && w.nan > 0 ? 1 : 0;
  if (!(q > 0.f) || cnt < 2) flags |= 2;
  return colstats_finish(m, mlo, q, qlo, e, flags);
}

// colstats_warp_any with fewer instructions a value (18 in the two passes, not
// 33) for the common variable: every value finite and counted, the plain sum
// too, fewer than 2^24 values.  The first pass is plain, with the extremes (equal:
// a constant variable, whose mean is its value).  The centred pass sums the
// residuals four at a time and the squares, with the products' exact residuals, one
// by one into float pairs: the sum of the squares is good to about 2^-47, beside
// the rounding of each centred value itself (2^-24 of it, as in colstats_warp_any).
// It is repeated with the corrected mean where the correction is not small (its
// square beyond 2^-14 of the variance: a mean far above the spread); a mean that
// three passes have not settled goes to colstats_warp_any.
__device__ __forceinline__ ColStats colstats_warp(const float *__restrict__ x, int64_t n,
                                                  int use) {
  const unsigned FULL = 0xffffffffu;
  if (use != 0 || n < 2 || n >= (int64_t(1) << 24)) return colstats_warp_any(x, n, use);
  float s = 0.f, mn = __int_as_float(0x7f800000), mx = -mn;
  warp_for_each(x, n, [&](float v) {
    s += v;
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(FULL, s, o);
    mn = fminf(mn, __shfl_xor_sync(FULL, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, o));
  }
  if (!(s - s == 0.f)) return colstats_warp_any(x, n, use);  // a NaN, an infinity, an overflow
  const int e = binade(fmaxf(fabsf(mn), fabsf(mx)));
  const float sc = __uint_as_float(uint32_t(127 - e) << 23);
  if (mn == mx) return colstats_finish(mn * sc, 0.f, 0.f, 0.f, e, 2);
  const float N = float(int(n)), invN = 1.f / N;
  float m = (s * sc) * invN, mlo = 0.f, q = 0.f, qlo = 0.f;
#pragma unroll 1
  for (int pass = 0; pass < 3; pass++) {
    FloatPairSum c, ss;
    auto centred = [&](float v) {  // its square goes to ss
      const float d = fmaf(v, sc, -m) - mlo;
      const float p = d * d;
      ss.add(p);
      ss.lo += fmaf(d, d, -p);
      return d;
    };
    warp_for_each4(
        x, n,
        [&](float4 v) {
          c.add((centred(v.x) + centred(v.y)) + (centred(v.z) + centred(v.w)));
        },
        [&](float v) { c.add(centred(v)); });
    q = ss.hi;
    qlo = ss.lo;
    warp_pair_sum(c.hi, c.lo);
    warp_pair_sum(q, qlo);
    const float C = c.hi + c.lo, cm = C * invN;  // cm: the mean's correction
    mlo += cm;
    const float mean = m + mlo;
    mlo -= mean - m;
    m = mean;
    const float cc = C * cm;
    qlo -= cc;
    if (cc <= 0x1p-14f * q) {  // (the sums follow the mean of this pass)
      const float sum = q + qlo;
      qlo -= sum - q;
      return colstats_finish(m, mlo, sum, qlo, e, sum > 0.f ? 0 : 2);
    }
  }
  return colstats_warp_any(x, n, use);
}

// z = (x - mean) * inv_norm in float arithmetic with the mean as a float
// pair: the float rounding of the exact value to within a couple of ulp.
struct Centerer {
  float mhi, mlo, inv, sc;  // of the values times sc, a power of two
  __device__ __forceinline__ explicit Centerer(const ColStats &s)
      : mhi(s.mhi), mlo(s.mlo), inv(s.ihi), sc(s.scale()) {}
  __device__ __forceinline__ float operator()(float x) const {
    return (fmaf(x, sc, -mhi) - mlo) * inv;
  }
};

}  // namespace gt
