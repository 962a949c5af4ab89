// distance.cu -- gpuDist's six metrics on CUDA cores.
//
// Reference: src/distance.cpp:209-316 (distance, distance_device) launching
// the `*_kernel_same` kernels of inst/cuda/distance.cu (euclidean :40-78,
// maximum :116-154, manhattan :192-232, canberra :273-316, binary :366-415,
// minkowski :453-493).  Those kernels use one 32-thread block per (x, y) with
// a shared-memory tree reduction; here every metric runs on the tiled engine
// of allpairs_simt.cuh, computing each unordered pair once.
//
// Semantics follow R's stats::dist (the reference's documented model):
//  * canberra omits terms whose numerator and denominator are both zero
//    (a = b = 0) and scales the sum by dim / terms-used; a term with a zero
//    denominator only (a = -b != 0) is +Inf.  The reference kernel instead
//    skips every zero-denominator term and never rescales
//    (inst/cuda/distance.cu:294), so the two differ only when zeros occur.
//  * minkowski evaluates |a-b|^p exactly for p = 1, 2, 3 and as
//    2^(p log2 |a-b|) otherwise (the reference uses the low-accuracy __powf,
//    :471, :487); the final root is FP32 (cbrtf for p = 3, else 2^(log2(s) / p)).
#include "common.cuh"
#include "allpairs_simt.cuh"
#include "kernels.cuh"

#include <cmath>

namespace gt {

namespace {

struct OpEuclid {
  static constexpr int kUnrollK = 1;  // measured fastest (up to 10 % over a full unroll)
  static constexpr int NACC = 1;
  __device__ static float pad() { return 0.f; }
  __device__ void init(float (&c)[1]) const { c[0] = 0.f; }
  __device__ void step(float (&c)[1], float a, float b) const {
    const float d = a - b;
    c[0] = fmaf(d, d, c[0]);
  }
  __device__ float finish(const float (&c)[1], int64_t) const { return sqrtf(c[0]); }
};

struct OpManhattan {
  static constexpr int kUnrollK = 1;  // measured fastest (up to 10 % over a full unroll)
  static constexpr int NACC = 1;
  __device__ static float pad() { return 0.f; }
  __device__ void init(float (&c)[1]) const { c[0] = 0.f; }
  __device__ void step(float (&c)[1], float a, float b) const { c[0] += fabsf(a - b); }
  __device__ float finish(const float (&c)[1], int64_t) const { return c[0]; }
};

struct OpMaximum {
  static constexpr int kUnrollK = 1;  // measured fastest (up to 10 % over a full unroll)
  static constexpr int NACC = 1;
  __device__ static float pad() { return 0.f; }
  __device__ void init(float (&c)[1]) const { c[0] = 0.f; }
  __device__ void step(float (&c)[1], float a, float b) const { c[0] = fmaxf(c[0], fabsf(a - b)); }
  __device__ float finish(const float (&c)[1], int64_t) const { return c[0]; }
};

// Binary on bit-packed points (bit k of word w: coordinate 32 w + k is
// nonzero); the engine carries the words as float bit patterns and the two
// counts (bits on in exactly one point, bits on in either) as integers in
// the accumulator slots.  The reference counts per coordinate in float
// (inst/cuda/distance.cu:366-415); the counts, and so the results, are the same.
struct OpBinaryBits {
  static constexpr int NACC = 2;  // bits on in exactly one, bits on in either
  static constexpr bool kSkipPad = true;
  __device__ static float pad() { return 0.f; }
  __device__ void init(float (&c)[2]) const { c[0] = __int_as_float(0); c[1] = __int_as_float(0); }
  __device__ void step(float (&c)[2], float a, float b) const {
    const unsigned x = __float_as_uint(a), y = __float_as_uint(b);
    c[0] = __int_as_float(__float_as_int(c[0]) + __popc(x ^ y));
    c[1] = __int_as_float(__float_as_int(c[1]) + __popc(x | y));
  }
  __device__ float finish(const float (&c)[2], int64_t) const {
    const float d = float(__float_as_int(c[1]));
    return d != 0.f ? float(__float_as_int(c[0])) / d : 0.f;
  }
};

// The same counts packed in one 32-bit accumulator (bits on in either << 16 |
// bits on in exactly one), for fewer than 65536 coordinates, where neither
// count can carry out of its half: a single-accumulator operation, so large
// problems take the 128 x 128 tiles (the binary kernel spends its time per
// tile, not on its two words of arithmetic per pair).
struct OpBinaryPacked {
  static constexpr int NACC = 1;
  static constexpr bool kSkipPad = true;
  static constexpr int kUnrollK = 1;  // a few words per point: the slab's loop stops early
  __device__ static float pad() { return 0.f; }
  __device__ void init(float (&c)[1]) const { c[0] = __uint_as_float(0u); }
  __device__ void step(float (&c)[1], float a, float b) const {
    const unsigned x = __float_as_uint(a), y = __float_as_uint(b);
    c[0] = __uint_as_float(__float_as_uint(c[0]) + __popc(x ^ y) +
                           (unsigned(__popc(x | y)) << 16));
  }
  __device__ float finish(const float (&c)[1], int64_t) const {
    const unsigned v = __float_as_uint(c[0]);
    const float d = float(int(v >> 16));
    return d != 0.f ? float(int(v & 0xffffu)) / d : 0.f;
  }
};

// One warp per point: word w of point i holds the nonzero pattern of
// coordinates 32 w .. 32 w + 31 (NaN counts as nonzero, as in OpBinary).
__global__ void __launch_bounds__(256)
pack_nonzero_kernel(const float *__restrict__ P, int64_t n, int64_t dim, int64_t words,
                    unsigned *__restrict__ bits) {
  const int64_t i = (int64_t(blockIdx.x) * 256 + threadIdx.x) >> 5;
  if (i >= n) return;  // whole warps
  const int lane = threadIdx.x & 31;
  for (int64_t w = 0; w < words; w++) {
    const int64_t k = 32 * w + lane;
    const unsigned b = __ballot_sync(0xffffffffu, k < dim && P[i * dim + k] != 0.f);
    if (lane == 0) bits[i * words + w] = b;
  }
}

struct OpMink3 {
  static constexpr int kUnrollK = 1;  // measured fastest (up to 10 % over a full unroll)
  static constexpr int NACC = 1;
  __device__ static float pad() { return 0.f; }
  __device__ void init(float (&c)[1]) const { c[0] = 0.f; }
  __device__ void step(float (&c)[1], float a, float b) const {
    const float d = fabsf(a - b);
    c[0] = fmaf(d * d, d, c[0]);
  }
  // FP32 root: one FP64 root per entry would cost GB300 more than the entry's
  // whole sum (its FP64 rate is ~1/64 of FP32); cbrtf is within 1 ulp
  __device__ float finish(const float (&c)[1], int64_t) const { return cbrtf(c[0]); }
};

struct OpMinkP {
  static constexpr int kUnrollK = 1;  // measured fastest (up to 10 % over a full unroll)
  static constexpr int NACC = 1;
  float p;
  __device__ static float pad() { return 0.f; }
  __device__ void init(float (&c)[1]) const { c[0] = 0.f; }
  // |a - b|^p as 2^(p log2 |a - b|) (0, Inf and NaN come out as from powf;
  // relative error about 2 |p log2 |a - b|| ulp, against powf's 1 ulp, at less
  // than half of powf's instructions)
  __device__ void step(float (&c)[1], float a, float b) const {
    c[0] += exp2f(p * log2f(fabsf(a - b)));
  }
  // s^(1/p) in FP32 as 2^(log2(s) / p): relative error about |log2 s| ulp
  __device__ float finish(const float (&c)[1], int64_t) const {
    return c[0] > 0.f ? exp2f(__fdiv_rn(log2f(c[0]), p)) : c[0];
  }
};

// Writes one distance in the full square layout (d[y*n + x], both halves)
// or R's dist layout (strict lower triangle by columns).
template <class Op>
struct OutDist {
  Op op;
  float *out;
  int64_t n, K;
  int layout;
  // the full layout's mirror goes through shared memory (coalesced stores)
  static constexpr bool kStagedMirror = true;
  __device__ bool staged(bool mirror) const { return mirror && layout == GT_LAYOUT_FULL; }
  __device__ float value(int64_t r, int64_t c, const float (&acc)[Op::NACC]) const {
    return (r == c) ? 0.f : op.finish(acc, K);
  }
  __device__ void store(int64_t r, int64_t c, float v) const { out[r * n + c] = v; }
  __device__ void operator()(int64_t r, int64_t c, const float (&acc)[Op::NACC], bool mirror) const {
    if (layout == GT_LAYOUT_FULL) {
      const float v = (r == c) ? 0.f : op.finish(acc, K);
      out[r * n + c] = v;
      if (mirror) out[c * n + r] = v;
    } else {
      if (c <= r) return;  // each unordered pair once; (r, c) with c > r
      const int64_t i = c, j = r;
      out[n * j - j * (j + 1) / 2 + i - j - 1] = op.finish(acc, K);
    }
  }
};

// An entry whose value the kernel has already formed.
struct OpValue {
  static constexpr int NACC = 1;
  __device__ float finish(const float (&c)[1], int64_t) const { return c[0]; }
};

// Canberra.  A term |a - b| / |a + b| by IEEE division is about 19
// instructions (and, where both values are zero, its slow path).  While a
// tile's values are all zero or of magnitude 2^-30 to 2^60, two terms are added
// with one reciprocal,
//   n0 / d0 + n1 / d1 = (n0 d1 + n1 d0) / (d0 d1),
// for two columns at a time in packed FP32 (f32x2): 12 instructions for four
// terms, with half as many rounded additions to the sum and the reciprocal
// at 1 ulp.  Zeros are stored as 2^-60: next to a value of the range that
// changes neither a - b nor a + b, and a pair of zeros adds 0 / 2^-59 = 0, so
// the loop tests nothing; nonzero products lie in [2^-118, 2^122].  Opposite
// values make a zero product, whose reciprocal gives the term's +Inf, or NaN
// where both terms are infinite (0 times Inf): nothing else makes a NaN there,
// so it is read as +Inf.  Coordinates where both points are zero are counted
// at the end from the points' nonzero bits, 32 to a popcount, which the slabs leave in
// shared memory (a buffer in the workspace, filled by a launch of its own, made calls on
// two streams share it).  From the
// first slab with a huge, tiny or non-finite value on (voted by the barrier
// that ends the slab before it) a tile takes the divisions, on the values
// themselves.  Fewer than 8 coordinates (FEW), whose additions do not make up for the
// roundings of a shared denominator, take a reciprocal a term and correct the quotient
// by its residual (about half an ulp, as the division).
// Bound by issue (68 % of the slots): 16000 x 64, a tenth zeros, dist layout: 1.55 ms
// (9.54 before, 4.4 of them the two FP64 divisions of each rescaled entry); by divisions,
// signed values of 1e-12, 4.6 (5.1).
constexpr float kCanZero = 0x1p-60f, kCanLo = 0x1p-30f, kCanHi = 0x1p60f;
constexpr int kCanMinK = 8;
constexpr int kCanSlabs = 32;  // slabs whose bits the shared memory holds

// sum * dim / used with one rounding (the product's and the quotient's
// residuals are added back) where the product cannot overflow.
__device__ __forceinline__ float canberra_finish(float sum, int zeros, int64_t K) {
  const float k = float(K), used = float(K - zeros);
  if (used == 0.f) return __int_as_float(0x7fc00000);
  if (zeros == 0) return sum;
  if (!(sum < 0x1p90f)) return sum * __fdiv_rn(k, used);
  const float p = sum * k, pe = fmaf(sum, k, -p);
  const float q = __fdiv_rn(p, used);
  return q + __fdividef(fmaf(-q, used, p) + pe, used);
}

// The nonzero bits of a chunk.
__device__ __forceinline__ unsigned canberra_bits(const float4 &v) {
  return unsigned(v.x != 0.f) | unsigned(v.y != 0.f) << 1 | unsigned(v.z != 0.f) << 2 |
         unsigned(v.w != 0.f) << 3;
}

// Replaces a chunk's zeros; whether a value is out of the range.
__device__ __forceinline__ bool canberra_prepare(float4 &v) {
  bool bad = false;
  float *e = &v.x;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const bool zero = e[i] == 0.f;
    bad |= !(zero || (fabsf(e[i]) >= kCanLo && fabsf(e[i]) <= kCanHi));
    if (zero) e[i] = kCanZero;
  }
  return bad;
}

// 64 x 64 tiles, three blocks an SM: 128 x 128 tiles with two blocks or one
// measured 1.51 and 1.87 ms where these took 1.49, and 215 / 236 us against 185
// at 4000 x 100 (full).
template <bool FEW>
__global__ void __launch_bounds__(kSimtThreads, 3)
canberra_kernel(SimtArgs a, OutDist<OpValue> out) {
  constexpr int TM = 4, TN = 4, BM = 16 * TM, BN = 16 * TN;
  constexpr int LDA = simt_ld<BM>(), LDB = simt_ld<BN>();
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (ti > tj) return;
  const int64_t row0 = int64_t(ti) * BM, col0 = int64_t(tj) * BN;
  __shared__ __align__(16) float sA[2][kSimtBK * LDA];
  __shared__ __align__(16) float sB[2][kSimtBK * LDB];
  // nonzero bits of rows and columns, 16 coordinates each (one slab); rows an odd number
  // of words apart
  __shared__ __align__(4) uint16_t nz[2][64][kCanSlabs + 2];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;

  float2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN / 2; j++) acc[i][j] = make_float2(0.f, 0.f);
  float4 ra[BM * 4 / kSimtThreads], rb[BN * 4 / kSimtThreads];
  simt_load<BM, OpEuclid>(ra, a.R, a.ldr, a.nr, row0, 0, a.K, a.vec_ok);
  simt_load<BN, OpEuclid>(rb, a.C, a.ldc, a.nc, col0, 0, a.K, a.vec_ok);
  static_assert(BM * 4 == kSimtThreads && BN * 4 == kSimtThreads, "a chunk a thread");
  auto note = [&](int kb) {  // the bits of slab kb, in ra and rb: four threads' chunks a row
    const int q = threadIdx.x & 3;
    unsigned m = (canberra_bits(ra[0]) | canberra_bits(rb[0]) << 16) << (4 * q);
    m |= __shfl_xor_sync(0xffffffffu, m, 1);
    m |= __shfl_xor_sync(0xffffffffu, m, 2);
    if (q < 2 && kb < kCanSlabs) nz[q][threadIdx.x >> 2][kb] = uint16_t(q ? m >> 16 : m);
    return m;
  };
  // Slab kb in ra, rb to its buffer, zeros replaced; true if a value is out of the range
  // (uniform): then the slab is stored as it is.
  auto store = [&](int kb) {
    const int b = kb & 1, q = 4 * (threadIdx.x & 3);
    const unsigned m = note(kb);
    bool bad = canberra_prepare(ra[0]);
    bad |= canberra_prepare(rb[0]);
    simt_store<BM, false>(sA[b], ra);
    simt_store<BN, true>(sB[b], rb);
    if (!__syncthreads_or(bad)) return false;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (!((m >> (q + i)) & 1u)) (&ra[0].x)[i] = 0.f;
      if (!((m >> (q + i + 16)) & 1u)) (&rb[0].x)[i] = 0.f;
    }
    simt_store<BM, false>(sA[b], ra);
    simt_store<BN, true>(sB[b], rb);
    __syncthreads();
    return true;
  };
  bool divide = store(0);
  const int nk = int((a.K + kSimtBK - 1) / kSimtBK);
  int kb = 0;
  for (; kb < nk && !divide; kb++) {
    const int buf = kb & 1;
    const bool more = kb + 1 < nk;
    if (more) {
      simt_load<BM, OpEuclid>(ra, a.R, a.ldr, a.nr, row0, int64_t(kb + 1) * kSimtBK, a.K, a.vec_ok);
      simt_load<BN, OpEuclid>(rb, a.C, a.ldc, a.nc, col0, int64_t(kb + 1) * kSimtBK, a.K, a.vec_ok);
    }
    const float *pa = sA[buf] + 4 * ty, *pb = sB[buf] + 4 * tx;
    if constexpr (FEW) {
      const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll 2
      for (int kk = 0; kk < int(a.K); kk++) {
        const float4 u = *reinterpret_cast<const float4 *>(pa + kk * LDA);
        const float4 v = *reinterpret_cast<const float4 *>(pb + kk * LDB);
        const float2 y[2] = {make_float2(v.x, v.y), make_float2(v.z, v.w)};
#pragma unroll
        for (int i = 0; i < TM; i++) {
          const float2 x = make_float2((&u.x)[i], (&u.x)[i]);
#pragma unroll
          for (int j = 0; j < TN / 2; j++) {
            float2 d = __fadd2_rn(x, y[j]), n = __ffma2_rn(y[j], minus, x);
            n = make_float2(fabsf(n.x), fabsf(n.y));
            d = make_float2(-fabsf(d.x), -fabsf(d.y));
            float2 inv;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.x) : "f"(-d.x));
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.y) : "f"(-d.y));
            const float2 q = __fmul2_rn(n, inv);
            acc[i][j] = __fadd2_rn(acc[i][j], __ffma2_rn(__ffma2_rn(q, d, n), inv, q));
          }
        }
      }
    } else {
      const float2 minus = make_float2(-1.f, -1.f);
      const int left = int(a.K - int64_t(kb) * kSimtBK), kend = left < kSimtBK ? left : kSimtBK;
#pragma unroll 2
      for (int kk = 0; kk < kend; kk += 2) {  // an odd last term pairs with padding, 0 / 2^-59
        float2 y0[TN / 2], y1[TN / 2];
#pragma unroll
        for (int g = 0; g < TN / 4; g++) {
          const float4 u = *reinterpret_cast<const float4 *>(pb + kk * LDB + 64 * g);
          const float4 v = *reinterpret_cast<const float4 *>(pb + (kk + 1) * LDB + 64 * g);
          y0[2 * g] = make_float2(u.x, u.y);
          y0[2 * g + 1] = make_float2(u.z, u.w);
          y1[2 * g] = make_float2(v.x, v.y);
          y1[2 * g + 1] = make_float2(v.z, v.w);
        }
#pragma unroll
        for (int g = 0; g < TM / 4; g++) {
          const float4 u = *reinterpret_cast<const float4 *>(pa + kk * LDA + 64 * g);
          const float4 v = *reinterpret_cast<const float4 *>(pa + (kk + 1) * LDA + 64 * g);
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float2 x0 = make_float2((&u.x)[e], (&u.x)[e]);
            const float2 x1 = make_float2((&v.x)[e], (&v.x)[e]);
#pragma unroll
            for (int j = 0; j < TN / 2; j++) {
              const float2 d0 = __fadd2_rn(x0, y0[j]), d1 = __fadd2_rn(x1, y1[j]);
              const float2 p0 = __fmul2_rn(__ffma2_rn(y0[j], minus, x0), d1);
              const float2 p1 = __fmul2_rn(__ffma2_rn(y1[j], minus, x1), d0);
              const float2 n = make_float2(fabsf(p0.x) + fabsf(p1.x), fabsf(p0.y) + fabsf(p1.y));
              const float2 d = __fmul2_rn(d0, d1);
              float2 inv;
              asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.x) : "f"(fabsf(d.x)));
              asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.y) : "f"(fabsf(d.y)));
              acc[4 * g + e][j] = __ffma2_rn(n, inv, acc[4 * g + e][j]);
            }
          }
        }
      }
    }
    if (more) divide = store(kb + 1);
    else __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; i++)  // the slabs without divisions end
#pragma unroll
    for (int j = 0; j < TN / 2; j++) {
      if (acc[i][j].x != acc[i][j].x) acc[i][j].x = __int_as_float(0x7f800000);
      if (acc[i][j].y != acc[i][j].y) acc[i][j].y = __int_as_float(0x7f800000);
    }
  for (; kb < nk; kb++) {
    const int buf = kb & 1;
    const bool more = kb + 1 < nk;
    if (more) {
      simt_load<BM, OpEuclid>(ra, a.R, a.ldr, a.nr, row0, int64_t(kb + 1) * kSimtBK, a.K, a.vec_ok);
      simt_load<BN, OpEuclid>(rb, a.C, a.ldc, a.nc, col0, int64_t(kb + 1) * kSimtBK, a.K, a.vec_ok);
    }
    const float *pa = sA[buf] + 4 * ty, *pb = sB[buf] + 4 * tx;
    const int left = int(a.K - int64_t(kb) * kSimtBK), kend = left < kSimtBK ? left : kSimtBK;
#pragma unroll 2
    for (int kk = 0; kk < kend; kk++) {
      const float4 u = *reinterpret_cast<const float4 *>(pa + kk * LDA);
      const float4 v = *reinterpret_cast<const float4 *>(pb + kk * LDB);
#pragma unroll
      for (int i = 0; i < TM; i++) {
#pragma unroll
        for (int j = 0; j < TN; j++) {
          const float x = (&u.x)[i], y = (&v.x)[j];
          const float num = fabsf(x - y), den = fabsf(x + y);
          // equal values add 0, zeros among them (a division of 0 takes its slow path)
          const bool same = num == 0.f;
          const float t = __fdiv_rn(same ? 1.f : num, same ? 1.f : den);
          float &sum = j & 1 ? acc[i][j / 2].y : acc[i][j / 2].x;
          sum += same ? 0.f : t;
        }
      }
    }
    if (more) {
      note(kb + 1);
      simt_store<BM, false>(sA[buf ^ 1], ra);
      simt_store<BN, true>(sB[buf ^ 1], rb);
    }
    __syncthreads();
  }

  // coordinates where both points are zero: all but those nonzero in either (the bits
  // past dim are zero in both)
  float val[TM][TN][1];
  int used[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) used[i][j] = 0;
  for (int64_t k0 = 0;;) {  // slabs k0 / 16 .. in nz
    const int64_t left = (a.K - k0 + kSimtBK - 1) / kSimtBK;
    const int slabs = left < kCanSlabs ? int(left) : kCanSlabs;
    for (int t = 0; t < slabs; t += 2) {
      const unsigned in = t + 1 < slabs ? 0xffffffffu : 0xffffu;
      unsigned zb[TN];
#pragma unroll
      for (int j = 0; j < TN; j++)
        zb[j] = *reinterpret_cast<const unsigned *>(&nz[1][tx + 16 * j][t]) & in;
#pragma unroll
      for (int i = 0; i < TM; i++) {
        const unsigned za = *reinterpret_cast<const unsigned *>(&nz[0][simt_row(i, ty)][t]) & in;
#pragma unroll
        for (int j = 0; j < TN; j++) used[i][j] += __popc(za | zb[j]);
      }
    }
    k0 += kCanSlabs * kSimtBK;
    if (k0 >= a.K) break;
    // further coordinates: from the points again
    __syncthreads();
#pragma unroll 1
    for (int q = threadIdx.x >> 5; q < 128 * kCanSlabs / 2; q += kSimtThreads / 32) {
      const int side = q >> 10, row = (q >> 4) & 63, t = 2 * (q & 15);
      static_assert(kCanSlabs == 32, "sixteen words a row");
      const int64_t i = (side ? col0 : row0) + row, k = k0 + 16 * t + (threadIdx.x & 31);
      const bool on = i < a.nr && k < a.K && __ldg(a.R + i * a.ldr + k) != 0.f;
      const unsigned w = __ballot_sync(0xffffffffu, on);
      if ((threadIdx.x & 31) == 0) *reinterpret_cast<unsigned *>(&nz[side][row][t]) = w;
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++)
      val[i][j][0] = canberra_finish(j & 1 ? acc[i][j / 2].y : acc[i][j / 2].x,
                                     int(a.K - used[i][j]), a.K);
  simt_write_tile<OutDist<OpValue>, TM, TN, 1>(a, out, a.symmetric && ti != tj, tx, ty, row0, col0,
                                               &sA[0][0], val);
}

SimtArgs dist_args(const float *pts, int64_t n, int64_t dim) {
  SimtArgs a;
  a.R = a.C = pts;
  a.ldr = a.ldc = dim;
  a.nr = a.nc = n;
  a.K = dim;
  a.symmetric = 1;
  a.vec_ok = (dim % 4 == 0) && aligned16(pts);
  return a;
}

cudaError_t run_canberra(const float *pts, int64_t n, int64_t dim, float *out, int layout,
                         cudaStream_t st) {
  ProfScope prof("dist", st);
  const SimtArgs a = dist_args(pts, n, dim);
  const OutDist<OpValue> o{OpValue{}, out, n, dim, layout};
  const unsigned g = unsigned(cdiv(n, 64));
  auto kern = dim < kCanMinK ? canberra_kernel<true> : canberra_kernel<false>;
  kern<<<dim3(g, g), kSimtThreads, 0, st>>>(a, o);
  count_launch();
  return cudaGetLastError();
}

template <class Op>
cudaError_t run_metric(const Op &op, const float *pts, int64_t n, int64_t dim, float *out,
                       int layout, cudaStream_t st) {
  const SimtArgs a = dist_args(pts, n, dim);
  OutDist<Op> o{op, out, n, dim, layout};
  ProfScope prof("dist", st);
  const int64_t t128 = cdiv(n, 128);
  if (Op::NACC == 1 && t128 * (t128 + 1) / 2 >= 2 * sm_count())
    return launch_allpairs_simt<Op, OutDist<Op>, 8, 8>(a, op, o, st);
  return launch_allpairs_simt<Op, OutDist<Op>, 4, 4>(a, op, o, st);
}

}  // namespace

int dist_check_args(int64_t n, int64_t dim, int method, int layout) {
  if (n < 0 || dim < 0) return fail(GT_EINVAL, "negative size (n=%lld, dim=%lld)",
                                    (long long)n, (long long)dim);
  if (method < GT_EUCLIDEAN || method > GT_MINKOWSKI)
    return fail(GT_EINVAL, "unknown distance method %d", method);
  if (layout != GT_LAYOUT_FULL && layout != GT_LAYOUT_DIST)
    return fail(GT_EINVAL, "unknown output layout %d", layout);
  if (cdiv(n, 64) > 65535) return fail(GT_EINVAL, "too many points (%lld)", (long long)n);
  return GT_OK;
}

// Euclidean distances on the FP32 CUDA-core path; used directly for
// GT_GRAM_FP32 and as the reference point of the tensor-core path.
int dist_simt(const float *d_pts, int64_t n, int64_t dim, float *d_out, int layout, int method,
              float p, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  switch (method) {
  case GT_EUCLIDEAN: e = run_metric(OpEuclid{}, d_pts, n, dim, d_out, layout, st); break;
  case GT_MAXIMUM: e = run_metric(OpMaximum{}, d_pts, n, dim, d_out, layout, st); break;
  case GT_MANHATTAN: e = run_metric(OpManhattan{}, d_pts, n, dim, d_out, layout, st); break;
  case GT_CANBERRA: e = run_canberra(d_pts, n, dim, d_out, layout, st); break;
  case GT_BINARY: {
    const int64_t words = cdiv(dim, 32);
    void *pb = nullptr;
    GT_TRY(ws_get(WS_SCRATCH0, size_t(n) * size_t(words) * 4, &pb));
    pack_nonzero_kernel<<<unsigned(cdiv(n, 8)), 256, 0, st>>>(d_pts, n, dim, words,
                                                             static_cast<unsigned *>(pb));
    count_launch();
    e = cudaGetLastError();
    if (e == cudaSuccess) {
      const float *bits = static_cast<const float *>(pb);
      e = dim < 65536 ? run_metric(OpBinaryPacked{}, bits, n, words, d_out, layout, st)
                      : run_metric(OpBinaryBits{}, bits, n, words, d_out, layout, st);
    }
    break;
  }
  case GT_MINKOWSKI:
    if (p == 1.f) e = run_metric(OpManhattan{}, d_pts, n, dim, d_out, layout, st);
    else if (p == 2.f) e = run_metric(OpEuclid{}, d_pts, n, dim, d_out, layout, st);
    else if (p == 3.f) e = run_metric(OpMink3{}, d_pts, n, dim, d_out, layout, st);
    else e = run_metric(OpMinkP{p}, d_pts, n, dim, d_out, layout, st);
    break;
  default: return fail(GT_EINVAL, "unknown distance method %d", method);
  }
  if (e != cudaSuccess) return fail(GT_ECUDA, "distance kernel launch: %s", cudaGetErrorString(e));
  return GT_OK;
}

}  // namespace gt

extern "C" int gt_distances_device(const float *d_points, int64_t n, int64_t dim, float *d_out,
                                   int layout, int method, float p, void *stream) {
  gt::clear_error();
  GT_TRY(gt::dist_check_args(n, dim, method, layout));
  if (n == 0) return GT_OK;
  if (!d_points || !d_out) return gt::fail(GT_EINVAL, "null device pointer");
  if (method == GT_MINKOWSKI && !(p > 0.f))
    return gt::fail(GT_EINVAL, "minkowski power must be positive (p=%g)", double(p));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (method == GT_EUCLIDEAN && gt_get_gram_path() != GT_GRAM_FP32)
    return gt::euclid_tc(d_points, n, dim, d_out, layout, st);
  return gt::dist_simt(d_points, n, dim, d_out, layout, method, p, st);
}

extern "C" int gt_distances(const float *points, int64_t n, int64_t dim, float *out, int method,
                            float p) {
  gt::clear_error();
  GT_TRY(gt::dist_check_args(n, dim, method, GT_LAYOUT_FULL));
  if (n == 0) return GT_OK;
  if (!points || !out) return gt::fail(GT_EINVAL, "null host pointer");
  cudaStream_t st = gt::lib_stream();
  gt::StreamSyncGuard guard(st);
  void *dp = nullptr, *dout = nullptr;
  GT_TRY(gt::ws_get(gt::WS_IN_A, size_t(n) * size_t(dim) * 4, &dp));
  void *direct = gt::host_output_ptr(out, size_t(n) * size_t(n) * 4);
  if (!(dout = direct)) GT_TRY(gt::ws_get(gt::WS_OUT0, size_t(n) * size_t(n) * 4, &dout));
  GT_CUDA(cudaMemcpyAsync(dp, points, size_t(n) * size_t(dim) * 4, cudaMemcpyHostToDevice, st));
  GT_TRY(gt_distances_device(static_cast<float *>(dp), n, dim, static_cast<float *>(dout),
                             GT_LAYOUT_FULL, method, p, st));
  if (!direct)
    GT_CUDA(cudaMemcpyAsync(out, dout, size_t(n) * size_t(n) * 4, cudaMemcpyDeviceToHost, st));
  GT_CUDA(cudaStreamSynchronize(st));
  bool failed = false;
  GT_TRY(gt::device_error_check(st, &failed));
  if (failed) return gt::fail(GT_ETIMEOUT, "a tensor-core kernel wait timed out");
  return GT_OK;
}
