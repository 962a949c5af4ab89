// backward.cu -- adjoints of gpuCor (pearson) and gpuDist (euclidean), and
// the MDS stress gradient.  No counterpart in the reference (gputools has no
// differentiation); the forward quantities follow inst/cuda/correlation.cu:
// 152-292 and inst/cuda/distance.cu:40-78.
//
// Pearson.  With c_j = x_j - mean, s_j = |c_j|, z_j = c_j / s_j and
// C_ij = z_i . z_j, an upstream G = dL/dC gives
//   W = S Z  (S = G + G^T, Z the p x n matrix of the z_j),
//   dL/dx_j = (w_j - z_j (z_j . w_j)) / s_j,
// i.e. one GEMM plus a rank-1 correction per variable.  Means and norms are
// recomputed (not stored by the forward pass) with compensated float sums;
// the centring, z_j . w_j and the correction run in float arithmetic with the
// mean as a float pair and the dot product compensated (GB300's FP64 pipe is
// a small fraction of its FP32 pipe).  S and Z^T are split
// into bf16 planes and W runs on the tcgen05 chunked-accumulation kernel
// (gram_tc.cu), or on the CUDA-core engine for GT_GRAM_FP32.
//
// Distances.  dL/dx_i = sum_j W_ij (x_i - x_j) = x_i rowsum(W)_i - (W X)_i with
// W_ij = (G_ij + G_ji) / D_ij (0 where D_ij = 0), or for MDS stress
// W_ij = 2 (D_ij - delta_ij) / D_ij.  Up to 32 dimensions (64 outside 8192 ..
// 32768 points) a fused CUDA-core kernel recomputes D_ij from the points and
// never materialises W.  Otherwise the adjoint is GEMMs plus a rank-1 correction: D comes from the tcgen05
// Euclidean path (exact near-zero recomputation included), one pass over D
// and G writes W as split-bf16 planes with its row sums, W X runs on the
// tcgen05 GEMM, and dX = X diag(rowsum W) - W X is formed on the points
// centred by their column means (the gradient does not change under a
// translation, and centring keeps the two terms from cancelling).
#include "common.cuh"
#include "allpairs_simt.cuh"
#include "kernels.cuh"
#include "stats.cuh"
#include "tc_ptx.cuh"

#include <cuda_bf16.h>

namespace gt {

namespace {

constexpr int64_t kKPadB = 64;

template <class T>
__device__ __forceinline__ void put_parts(T *dst, int64_t plane, int64_t idx, float v, int ns);

template <>
__device__ __forceinline__ void put_parts<float>(float *dst, int64_t, int64_t idx, float v, int) {
  dst[idx] = v;
}

template <>
__device__ __forceinline__ void put_parts<__nv_bfloat16>(__nv_bfloat16 *dst, int64_t plane,
                                                         int64_t idx, float v, int ns) {
  uint16_t p[3];
  if (ns == 3) tc::split_parts<tc::KIND_BF16X6>(v, p);
  else tc::split_parts<tc::KIND_BF16X3>(v, p);
  for (int q = 0; q < ns; q++) dst[q * plane + idx] = __ushort_as_bfloat16(p[q]);
}

// S = G + G^T as rows j, columns i (ld kp >= p, zero padded), float or bf16
// planes.  64 x 64 tiles: the transposed operand goes through shared memory,
// loads and stores in pairs along the rows when p is even.
template <class T>
__global__ void __launch_bounds__(256)
sym_operand_kernel(const float *__restrict__ G, int64_t p, int64_t kp, int ns, T *__restrict__ S) {
  __shared__ float tile[64][65];
  const int64_t i0 = int64_t(blockIdx.x) * 64, j0 = int64_t(blockIdx.y) * 64;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const bool pairs = (p & 1) == 0 && (reinterpret_cast<uintptr_t>(G) & 7u) == 0;
  // tile[a][b] = G[i0 + a][j0 + b]
#pragma unroll 4
  for (int r = 0; r < 8; r++) {
    const int a = ty + 8 * r;
    const int64_t i = i0 + a, j = j0 + 2 * tx;
    float2 v = make_float2(0.f, 0.f);
    if (i < p) {
      if (pairs && j + 1 < p) {
        v = *reinterpret_cast<const float2 *>(G + i * p + j);
      } else {
        if (j < p) v.x = G[i * p + j];
        if (j + 1 < p) v.y = G[i * p + j + 1];
      }
    }
    tile[a][2 * tx] = v.x;
    tile[a][2 * tx + 1] = v.y;
  }
  __syncthreads();
  const int64_t plane = p * kp;
#pragma unroll 4
  for (int r = 0; r < 8; r++) {
    const int b = ty + 8 * r;
    const int64_t j = j0 + b, i = i0 + 2 * tx;
    if (j >= p || i >= kp) continue;
    float2 g = make_float2(0.f, 0.f);
    if (pairs && i + 1 < p) {
      g = *reinterpret_cast<const float2 *>(G + j * p + i);
    } else {
      if (i < p) g.x = G[j * p + i];
      if (i + 1 < p) g.y = G[j * p + i + 1];
    }
    const float s0 = i < p ? g.x + tile[2 * tx][b] : 0.f;
    const float s1 = i + 1 < p ? g.y + tile[2 * tx + 1][b] : 0.f;
    if constexpr (std::is_same<T, float>::value) {
      *reinterpret_cast<float2 *>(S + j * kp + i) = make_float2(s0, s1);  // kp is even
    } else {
      put_parts<T>(S, plane, j * kp + i, s0, ns);
      put_parts<T>(S, plane, j * kp + i + 1, s1, ns);
    }
  }
}

// The f16x3 operands of the Pearson adjoint without float intermediates.
// S = G + G^T is taken in 64 x 64 tile pairs: the block of (I, J), I <= J,
// loads G[I][J] and G[J][I] once and has both S[I][J] and S[J][I] = S[I][J]^T.
// Pass 1 (sym_rowmax_kernel) folds every row's largest finite |S| into
// rowmax (float bits, atomicMax); pass 2 (sym_split_kernel) scales each row
// by the power of two that brings that maximum into [2^14, 2^15) and writes
// the two f16 planes ([2][p][kp], zero padded) and the factors that undo the
// scales.  G is read twice in all, S never stored in float.
// A thread holds four neighbours of four rows of either tile in registers
// (16-byte loads where the rows allow them, all in flight together) and meets
// the other tile's transpose in shared memory: 16 lanes a row.  Bound by memory:
// 4096 variables 29 -> 16.5 us (pass 1) and 34 -> 28 us (pass 2) with scalar loads
// through shared memory before.
__device__ __forceinline__ void sym_load(const float *__restrict__ G, int64_t p, int64_t i0,
                                         int64_t j, bool vec, float4 (&v)[4]) {
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int64_t i = i0 + 16 * r;
    v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i >= p) continue;
    const float *q = G + i * p + j;
    if (vec) {
      if (j < p) v[r] = *reinterpret_cast<const float4 *>(q);
    } else {
      if (j < p) v[r].x = q[0];
      if (j + 1 < p) v[r].y = q[1];
      if (j + 2 < p) v[r].z = q[2];
      if (j + 3 < p) v[r].w = q[3];
    }
  }
}
__device__ __forceinline__ void sym_stage(float (&t)[64][65], int ty, int tx, const float4 (&v)[4]) {
#pragma unroll
  for (int r = 0; r < 4; r++) {
    float *q = &t[ty + 16 * r][4 * tx];
    q[0] = v[r].x;
    q[1] = v[r].y;
    q[2] = v[r].z;
    q[3] = v[r].w;
  }
}
// Row a, columns 4 tx .. of S: the tile's values plus the transposed tile's.
__device__ __forceinline__ float4 sym_sum(float4 v, const float (&t)[64][65], int a, int tx) {
  return make_float4(v.x + t[4 * tx][a], v.y + t[4 * tx + 1][a], v.z + t[4 * tx + 2][a],
                     v.w + t[4 * tx + 3][a]);
}

__device__ __forceinline__ float finite_abs(float v) {
  const float a = fabsf(v);
  return a == a ? a : 0.f;  // NaN does not count, as fmaxf would skip it
}

__global__ void __launch_bounds__(256)
sym_rowmax_kernel(const float *__restrict__ G, int64_t p, int vec, unsigned *__restrict__ rowmax) {
  if (blockIdx.y > blockIdx.x) return;  // the pair (J, I) is done by block (I, J)
  __shared__ float tb[64][65];
  __shared__ float cm[8][64];
  const int64_t I0 = int64_t(blockIdx.y) * 64, J0 = int64_t(blockIdx.x) * 64;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  float4 va[4], vb[4];
  sym_load(G, p, I0 + ty, J0 + 4 * tx, vec, va);
  sym_load(G, p, J0 + ty, I0 + 4 * tx, vec, vb);
  sym_stage(tb, ty, tx, vb);
  __syncthreads();
  float c[4] = {0.f, 0.f, 0.f, 0.f};  // columns 4 tx .. (rows J0 + 4 tx .. of S)
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int a = ty + 16 * r;
    const float4 v = sym_sum(va[r], tb, a, tx);
    const float e[4] = {finite_abs(v.x), finite_abs(v.y), finite_abs(v.z), finite_abs(v.w)};
    float m = 0.f;  // row I0 + a of S
#pragma unroll
    for (int q = 0; q < 4; q++) {
      c[q] = fmaxf(c[q], e[q]);
      m = fmaxf(m, e[q]);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (tx == 0 && I0 + a < p) atomicMax(rowmax + I0 + a, __float_as_uint(m));
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    c[q] = fmaxf(c[q], __shfl_xor_sync(0xffffffffu, c[q], 16));
    if ((t & 16) == 0) cm[t >> 5][4 * tx + q] = c[q];
  }
  __syncthreads();
  if (t < 64 && J0 + t < p) {
    float m = cm[0][t];
#pragma unroll
    for (int q = 1; q < 8; q++) m = fmaxf(m, cm[q][t]);
    atomicMax(rowmax + J0 + t, __float_as_uint(m));
  }
}

__global__ void __launch_bounds__(256)
sym_split_kernel(const float *__restrict__ G, int64_t p, int64_t kp, int vec,
                 const unsigned *__restrict__ rowmax, uint16_t *__restrict__ planes,
                 float *__restrict__ scale) {
  if (blockIdx.y > blockIdx.x) return;
  __shared__ float ta[64][65], tb[64][65];
  const int64_t I0 = int64_t(blockIdx.y) * 64, J0 = int64_t(blockIdx.x) * 64;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  float4 va[4], vb[4];
  sym_load(G, p, I0 + ty, J0 + 4 * tx, vec, va);
  sym_load(G, p, J0 + ty, I0 + 4 * tx, vec, vb);
  sym_stage(ta, ty, tx, va);
  sym_stage(tb, ty, tx, vb);
  __syncthreads();
  // rows `row`, columns `col` .. of both planes
  auto put = [&](int64_t row, int64_t col, float4 v, int e) {
    const float sc = tc::exp2i(e), x[4] = {v.x * sc, v.y * sc, v.z * sc, v.w * sc};
    uint32_t w[2][2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      uint16_t h0[3], h1[3];
      tc::split_parts<tc::KIND_F16X3>(x[2 * q], h0);
      tc::split_parts<tc::KIND_F16X3>(x[2 * q + 1], h1);
      w[0][q] = uint32_t(h0[0]) | (uint32_t(h1[0]) << 16);
      w[1][q] = uint32_t(h0[1]) | (uint32_t(h1[1]) << 16);
    }
    uint16_t *o = planes + row * kp + col;
    *reinterpret_cast<uint2 *>(o) = make_uint2(w[0][0], w[0][1]);
    *reinterpret_cast<uint2 *>(o + p * kp) = make_uint2(w[1][0], w[1][1]);
  };
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int a = ty + 16 * r;
    if (I0 + a < p) {
      const int e = tc::f16_scale_exp(__uint_as_float(rowmax[I0 + a]));
      put(I0 + a, J0 + 4 * tx, sym_sum(va[r], tb, a, tx), e);
      if (tx == 0 && I0 == J0) scale[I0 + a] = tc::exp2i(-e);
    }
    if (I0 != J0 && J0 + a < p)
      put(J0 + a, I0 + 4 * tx, sym_sum(vb[r], ta, a, tx),
          tc::f16_scale_exp(__uint_as_float(rowmax[J0 + a])));
  }
}

// Z^T as f16x3 planes ([2][n][kp], zero padded): rows k (observations),
// columns i (variables), z = (x - mean) * inv_norm.  |z| <= 1 (the centred
// variable has unit norm), so one scale, 2^14, serves every row; scale[k] =
// 2^-14 undoes it.
// A block transposes 32 observations of 64 variables, its loads in flight together
// and two variables a store, so that a store fills a line of a row (4096
// variables of 1024 observations 16.5 -> 11.6 us; 32 x 32 with 2-byte stores before).
__global__ void __launch_bounds__(256)
zt_split_kernel(const float *__restrict__ X, int64_t p, int64_t n, int64_t kp,
                const ColStats *__restrict__ st, uint16_t *__restrict__ planes,
                float *__restrict__ scale) {
  __shared__ float tile[64][33];
  const int64_t k0 = int64_t(blockIdx.x) * 32, i0 = int64_t(blockIdx.y) * 64;
  const int tx = threadIdx.x, ty0 = threadIdx.y;
  if (ty0 == 0 && blockIdx.y == 0 && k0 + tx < n) scale[k0 + tx] = 1.f / 16384.f;
  float x[8];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const int64_t i = i0 + ty0 + 8 * r, k = k0 + tx;
    x[r] = i < p && k < n ? X[i * n + k] : 0.f;
  }
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const int64_t i = i0 + ty0 + 8 * r;
    float z = 0.f;
    if (i < p && k0 + tx < n) {
      const ColStats s = st[i];
      if (!s.flags) z = Centerer(s)(x[r]);
    }
    tile[ty0 + 8 * r][tx] = z;  // rows i
  }
  __syncthreads();
  const int64_t plane = n * kp, i = i0 + 2 * tx;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int ty = ty0 + 8 * r;
    const int64_t k = k0 + ty;
    if (k >= n) continue;
    uint16_t h0[3], h1[3];
    tc::split_parts<tc::KIND_F16X3>(tile[2 * tx][ty] * 16384.f, h0);
    tc::split_parts<tc::KIND_F16X3>(tile[2 * tx + 1][ty] * 16384.f, h1);
    uint32_t *o = reinterpret_cast<uint32_t *>(planes + k * kp + i);
    o[0] = uint32_t(h0[0]) | (uint32_t(h1[0]) << 16);
    o[plane / 2] = uint32_t(h0[1]) | (uint32_t(h1[1]) << 16);
  }
}

// Z^T: rows k (observations), columns i (variables, ld kp), zero padded.
template <class T>
__global__ void zt_operand_kernel(const float *__restrict__ X, int64_t p, int64_t n, int64_t kp,
                                  const ColStats *__restrict__ st, int ns, T *__restrict__ Zt) {
  __shared__ float tile[32][33];
  __shared__ float cen[32][5];  // the block's 32 variables: mean pair, inverse norm, scale, flag
  const int64_t k0 = int64_t(blockIdx.x) * 32, i0 = int64_t(blockIdx.y) * 32;
  const int tx = threadIdx.x, ty0 = threadIdx.y;
  if (ty0 == 0) {
    const int64_t i = i0 + tx;
    if (i < p) {
      const ColStats s = st[i];
      const Centerer c(s);
      cen[tx][0] = c.mhi;
      cen[tx][1] = c.mlo;
      cen[tx][2] = c.inv;
      cen[tx][3] = c.sc;
      cen[tx][4] = s.flags ? 1.f : 0.f;
    }
  }
  __syncthreads();
  for (int ty = ty0; ty < 32; ty += 8) {
    const int64_t i = i0 + ty, k = k0 + tx;
    float z = 0.f;
    if (i < p && k < n && cen[ty][4] == 0.f)
      z = (fmaf(X[i * n + k], cen[ty][3], -cen[ty][0]) - cen[ty][1]) * cen[ty][2];
    tile[ty][tx] = z;  // rows i
  }
  __syncthreads();
  const int64_t plane = n * kp;
  for (int ty = ty0; ty < 32; ty += 8) {
    const int64_t k = k0 + ty, i = i0 + tx;
    if (k >= n || i >= kp) continue;
    put_parts<T>(Zt, plane, k * kp + i, tile[tx][ty], ns);
  }
}

constexpr int kFinThreads = 256;

// Sum of the lanes' (hi, lo) float pairs, left in every lane (TwoSum).
__device__ __forceinline__ void warp_pair_sum_f(float &hi, float &lo) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
    const float t = hi + oh, bp = t - hi;
    lo = (lo + ol) + ((hi - (t - bp)) + (oh - bp));
    hi = t;
  }
}

__device__ __forceinline__ double block_sum_d(double v, double *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = (l < kFinThreads / 32) ? sh[l] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (l == 0) sh[0] = t;
  }
  __syncthreads();
  return sh[0];
}

// dX_j = (w_j - z_j (z_j . w_j)) * inv_norm_j, one warp per variable: the
// dot product as a compensated float pair (each product's exact residual by
// FMA, the sums by TwoSum), the correction in float.
__global__ void __launch_bounds__(kFinThreads)
cor_backward_finish_kernel(const float *__restrict__ X, int64_t p, int64_t n,
                           const ColStats *__restrict__ st, const float *__restrict__ W,
                           float *__restrict__ dX) {
  const int64_t j = (int64_t(blockIdx.x) * kFinThreads + threadIdx.x) >> 5;
  if (j >= p) return;  // whole warps
  const int lane = threadIdx.x & 31;
  const ColStats s = st[j];
  const float *x = X + j * n;
  const float *w = W + j * n;
  float *o = dX + j * n;
  if (s.flags) {
    for (int64_t k = lane; k < n; k += 32) o[k] = 0.f;
    return;
  }
  const Centerer cen(s);
  const float inv = cen.inv * cen.sc;
  float hi = 0.f, lo = 0.f;
  auto acc = [&](float xv, float wv) {
    const float z = cen(xv);
    const float pr = z * wv;
    const float pe = fmaf(z, wv, -pr);
    const float t = hi + pr, bp = t - hi;
    lo += ((hi - (t - bp)) + (pr - bp)) + pe;
    hi = t;
  };
  const bool v4 = (n & 3) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) |
                                    reinterpret_cast<uintptr_t>(o)) & 15u) == 0;
  if (v4) {
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
    for (int64_t k = lane; k < (n >> 2); k += 32) {
      const float4 a = x4[k], b = w4[k];
      acc(a.x, b.x);
      acc(a.y, b.y);
      acc(a.z, b.z);
      acc(a.w, b.w);
    }
  } else {
    for (int64_t k = lane; k < n; k += 32) acc(x[k], w[k]);
  }
  warp_pair_sum(hi, lo);
  const float d = hi + lo;
  if (v4) {
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
    float4 *o4 = reinterpret_cast<float4 *>(o);
    for (int64_t k = lane; k < (n >> 2); k += 32) {
      const float4 a = x4[k], b = w4[k];
      float4 r;
      r.x = fmaf(-cen(a.x), d, b.x) * inv;
      r.y = fmaf(-cen(a.y), d, b.y) * inv;
      r.z = fmaf(-cen(a.z), d, b.z) * inv;
      r.w = fmaf(-cen(a.w), d, b.w) * inv;
      o4[k] = r;
    }
  } else {
    for (int64_t k = lane; k < n; k += 32) o[k] = fmaf(-cen(x[k]), d, w[k]) * inv;
  }
}

struct OpDotB {
  static constexpr int NACC = 1;
  __device__ static float pad() { return 0.f; }
  __device__ void init(float (&c)[1]) const { c[0] = 0.f; }
  __device__ void step(float (&c)[1], float a, float b) const { c[0] = fmaf(a, b, c[0]); }
};

struct OutStore {
  float *out;
  int64_t ld;
  __device__ void operator()(int64_t r, int64_t c, const float (&acc)[1], bool) const {
    out[r * ld + c] = acc[0];
  }
};

// ------------------------------------------------------------ distances
constexpr int kDbRows = 128;   // rows i per CTA (one per thread)
constexpr int kDbCols = 32;    // points j per shared tile
static_assert(kDbRows / 32 == 4, "the coefficient copies step rows by four warps");

// Asynchronous 4-byte copy global -> shared (cp.async); bytes = 0 fills zero.
__device__ __forceinline__ void cp_async4(float *dst, const float *src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tc::smem_u32(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
// The same for 16 bytes (both addresses 16-byte aligned).
__device__ __forceinline__ void cp_async16(float *dst, const float *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Shared memory of dist_backward_kernel (floats, two buffers of each tile):
// the point tile [kDbCols][DMAX], the coefficients [kDbRows][kDbCols + 1]
// (G_ij, or delta_ij from either side of the diagonal) and, for mode 0, the
// transposed coefficients [kDbCols][kDbRows + 1] (G_ji).
template <int DMAX, int MODE>
struct DbSmem {
  static constexpr int XJ = kDbCols * DMAX;
  static constexpr int CFA = kDbRows * (kDbCols + 1);
  static constexpr int CFB = MODE == 0 ? kDbCols * (kDbRows + 1) : 0;
  static constexpr int FLOATS = 2 * (XJ + CFA + CFB);  // even: the doubles after it align
  static constexpr int BYTES = FLOATS * 4 + (kDbRows / 32) * 8;
};

// mode 0: W_ij = (G_ij + G_ji) / D_ij ; mode 1: MDS, W_ij = 2 (D_ij - delta_ij) / D_ij
// CTA (ib, js): rows i of block ib against points j of split js.  Writes the
// split's partial sums sum_j W_ij x_j (pacc) and sum_j W_ij (pw), and its
// partial loss; a second kernel reduces the splits in a fixed order.
// The tiles of 32 points and their coefficients are double-buffered: the
// copies of the next tile (cp.async) run while the current one is used.
// Every thread reads the same point j at a time (a broadcast), so the point
// tile needs no padding and is read 16 bytes at a time; 1 / D_ij comes from
// the hardware reciprocal square root (D_ij = D_ij^2 / D_ij), and the stress
// sums as a compensated float pair.
template <int DMAX, int MODE>
__global__ void __launch_bounds__(kDbRows)
dist_backward_kernel(const float *__restrict__ X, int64_t n, int64_t dim,
                     const float *__restrict__ aux, int64_t jchunk, float *__restrict__ pacc,
                     float *__restrict__ pw, double *__restrict__ ploss) {
  using L = DbSmem<DMAX, MODE>;
  extern __shared__ __align__(16) float dsm[];
  float *xj = dsm;                      // [2][kDbCols][DMAX]
  float *cfa = xj + 2 * L::XJ;          // [2][kDbRows][kDbCols + 1]
  float *cfb = cfa + 2 * L::CFA;        // [2][kDbCols][kDbRows + 1] (mode 0)
  double *sh = reinterpret_cast<double *>(dsm + L::FLOATS);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t i0 = int64_t(blockIdx.x) * kDbRows;
  const int64_t i = i0 + tid;
  const int64_t js = blockIdx.y;
  const int64_t jbeg = js * jchunk;
  const int64_t jend = (jbeg + jchunk < n) ? jbeg + jchunk : n;
  // points in 16-byte copies when every row starts on a 16-byte boundary
  const bool vec = (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  // copies of the tile of points jt .. jt + 31 into buffer b (one commit group);
  // the indices step from row to row (no products per copy)
  auto issue = [&](int b, int64_t jt) {
    float *xb = xj + b * L::XJ;
    if (vec) {
      for (int e = tid; e < kDbCols * DMAX / 4; e += kDbRows) {
        const int jj = e / (DMAX / 4), k = 4 * (e - jj * (DMAX / 4));
        const int64_t j = jt + jj;
        const bool ok = j < jend && k < dim;
        cp_async16(xb + 4 * e, ok ? X + j * dim + k : X, ok ? 16 : 0);
      }
    } else {
      for (int e = tid; e < kDbCols * DMAX; e += kDbRows) {
        const int jj = e / DMAX, k = e - jj * DMAX;
        const int64_t j = jt + jj;
        const bool ok = j < jend && k < dim;
        cp_async4(xb + e, ok ? X + j * dim + k : X, ok ? 4 : 0);
      }
    }
    float *ca = cfa + b * L::CFA;
    if (MODE == 0) {
      float *cb = cfb + b * L::CFB;
      const int64_t gj = jt + lane;
      int64_t gi = i0 + warp, off = gi * n + gj;  // G[gi][gj]
      for (int ii = warp; ii < kDbRows; ii += kDbRows / 32) {
        const bool ok = gi < n && gj < jend;
        cp_async4(ca + ii * (kDbCols + 1) + lane, ok ? aux + off : aux, ok ? 4 : 0);
        gi += kDbRows / 32;
        off += (kDbRows / 32) * n;
      }
      int64_t gj2 = jt, off2 = jt * n + i;  // G[gj2][i]
      for (int jj = 0; jj < kDbCols; jj++) {
        const bool ok = gj2 < jend && i < n;
        cp_async4(cb + jj * (kDbRows + 1) + tid, ok ? aux + off2 : aux, ok ? 4 : 0);
        gj2++;
        off2 += n;
      }
    } else {
      // delta in R dist layout: (a > b) at B(b) + a with B(b) = n b - b (b + 1) / 2 - b - 1;
      // each cell comes from exactly one side of the diagonal (the diagonal and
      // the cells past the tile are never read), and a side the tile does not
      // reach is skipped whole
      if (jt + kDbCols - 1 > i0) {  // cells with gj > gi: row gi, consecutive gj
        const int64_t gj = jt + lane;
        int64_t gi = i0 + warp, base = n * gi - gi * (gi + 1) / 2 - gi - 1;
        for (int ii = warp; ii < kDbRows; ii += kDbRows / 32) {
          if (gi < n && gj < jend && gj > gi)
            cp_async4(ca + ii * (kDbCols + 1) + lane, aux + (base + gj), 4);
          base += 4 * n - 4 * gi - 14;  // B(gi + 4) - B(gi)
          gi += 4;
        }
      }
      if (i0 + kDbRows - 1 > jt) {  // cells with i > gj: row gj, this thread's i
        int64_t gj = jt, base = n * gj - gj * (gj + 1) / 2 - gj - 1;
        for (int jj = 0; jj < kDbCols; jj++) {
          if (gj < jend && i < n && i > gj)
            cp_async4(ca + tid * (kDbCols + 1) + jj, aux + (base + i), 4);
          base += n - gj - 2;  // B(gj + 1) - B(gj)
          gj++;
        }
      }
    }
    cp_async_commit();
  };
  float xi[DMAX], acc[DMAX];
#pragma unroll
  for (int k = 0; k < DMAX; k++) {
    xi[k] = (i < n && k < dim) ? X[i * dim + k] : 0.f;
    acc[k] = 0.f;
  }
  float wsum = 0.f;
  FloatPairSum lsum;
  if (jbeg < jend) issue(0, jbeg);
  int b = 0;
  for (int64_t j0 = jbeg; j0 < jend; j0 += kDbCols, b ^= 1) {
    if (j0 + kDbCols < jend) {
      issue(b ^ 1, j0 + kDbCols);  // the other buffer: its last readers passed the barrier below
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();  // tile b complete and visible
    const float *xb = xj + b * L::XJ;
    const float *ca = cfa + b * L::CFA;
    const float *cb = cfb + b * L::CFB;
    if (i < n) {
      const int jmax = (jend - j0 < kDbCols) ? int(jend - j0) : kDbCols;
      for (int jj = 0; jj < jmax; jj++) {
        const int64_t j = j0 + jj;
        const float4 *x4 = reinterpret_cast<const float4 *>(xb + jj * DMAX);
        // four partial sums: four short dependency chains instead of one
        float q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f;
#pragma unroll
        for (int k = 0; k < DMAX / 4; k++) {
          const float4 v = x4[k];
          const float t0 = xi[4 * k] - v.x, t1 = xi[4 * k + 1] - v.y;
          const float t2 = xi[4 * k + 2] - v.z, t3 = xi[4 * k + 3] - v.w;
          q0 = fmaf(t0, t0, q0);
          q1 = fmaf(t1, t1, q1);
          q2 = fmaf(t2, t2, q2);
          q3 = fmaf(t3, t3, q3);
        }
        const float d2 = (q0 + q1) + (q2 + q3);
        if (j == i) continue;
        // 1 / d: the reciprocal square root estimate above the normal range's
        // floor, IEEE operations below it
        float inv_d = 0.f, d = 0.f;
        if (d2 >= 1e-30f) {
          inv_d = rsqrtf(d2);
          d = d2 * inv_d;
        } else if (d2 > 0.f) {
          d = sqrtf(d2);
          inv_d = 1.f / d;
        }
        const float c = MODE == 0 ? ca[tid * (kDbCols + 1) + jj] + cb[jj * (kDbRows + 1) + tid]
                                  : ca[tid * (kDbCols + 1) + jj];
        // coincident points add to the stress but not to the gradient
        if (MODE == 1 && j > i) {
          const float e = d - c;
          const float q = e * e;
          lsum.add(q);
          lsum.lo += fmaf(e, e, -q);
        }
        if (!(d2 > 0.f)) continue;
        const float w = MODE == 0 ? c * inv_d : 2.f * (d - c) * inv_d;
        wsum += w;
#pragma unroll
        for (int k = 0; k < DMAX / 4; k++) {
          const float4 v = x4[k];
          acc[4 * k] = fmaf(w, v.x, acc[4 * k]);
          acc[4 * k + 1] = fmaf(w, v.y, acc[4 * k + 1]);
          acc[4 * k + 2] = fmaf(w, v.z, acc[4 * k + 2]);
          acc[4 * k + 3] = fmaf(w, v.w, acc[4 * k + 3]);
        }
      }
    }
    __syncthreads();  // every thread is done with tile b before it is refilled
  }
  if (i < n) {
    float *pa = pacc + (js * n + i) * dim;
#pragma unroll
    for (int k = 0; k < DMAX; k++)
      if (k < dim) pa[k] = acc[k];
    pw[js * n + i] = wsum;
  }
  if (MODE == 1) {
    float lh = lsum.hi, ll = lsum.lo;
    warp_pair_sum(lh, ll);
    if (lane == 0) sh[warp] = double(lh) + double(ll);
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int w = 0; w < kDbRows / 32; w++) t += sh[w];
      ploss[blockIdx.y * gridDim.x + blockIdx.x] = t;
    }
  }
}

// dX_i = x_i * sum_s pw[s][i] - sum_s pacc[s][i]; splits added in order.
__global__ void dist_backward_reduce_kernel(const float *__restrict__ X, int64_t n, int64_t dim,
                                            int64_t nsplit, const float *__restrict__ pacc,
                                            const float *__restrict__ pw,
                                            float *__restrict__ dX) {
  const int64_t total = n * dim;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total;
       e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = e / dim;
    float w = 0.f, a = 0.f;
    for (int64_t s = 0; s < nsplit; s++) {
      w += pw[s * n + i];
      a += pacc[s * n * dim + e];
    }
    dX[e] = fmaf(X[e], w, -a);
  }
}

// ---- each unordered pair once
// The adjoint of the distances in 64 x 64 tiles of point pairs i < j: the
// distance, 1 / D and W_ij are formed once per unordered pair and used for both
// points (the kernel above forms them for (i, j) and for (j, i)).
//   phase 1: thread (ty, tx) takes the pairs of rows ty + 16 a and columns tx +
//            16 b; the squares sum in the same four chains over k mod 4 as above,
//            two chains to a packed FP32 operation, so D is the same number;
//            W goes to shared memory in both orientations;
//   phase 2: warps 0..3 add sum_j W_ij x_j to the row block's running sums, warps
//            4..7 form sum_i W_ij x_i of the column block, 4 rows x DMAX / 8
//            dimensions a thread.
// A block walks `len` consecutive tiles of the row-major list (I, J >= I).  The
// column sums of every tile, and the row sums whenever the row block or the
// segment ends, go to partial buffers that a second kernel adds in a fixed order.
// Bound by issue and latency at 16 warps an SM (61 % of the issue slots): 185
// instructions a pair, where the ordered kernel makes 380.  8192 x 32 (MDS stress):
// 299 us per call, 455 with ordered pairs; the gradient's error 0.8e-7 (1.2e-7).
constexpr int kPtT = 64, kPtThreads = 256;

template <int DMAX>
struct PtSmem {
  static constexpr int LD = DMAX + 4;   // rows 4 banks apart (mod 32)
  // W rows 8 banks apart, W^T rows 4: a warp's 4 x 8 stores meet no conflicts
  static constexpr int LW = kPtT + 8, LT = kPtT + 4;
  static constexpr int X = kPtT * LD, W = kPtT * LW, WT = kPtT * LT;
  static constexpr int SUMS = kPtT * DMAX;  // the row block's running sums
  static constexpr int BYTES = (3 * X + W + WT + SUMS) * 4;
};

// The partial buffers: column sums of tile (I, J) at J (J + 1) / 2 + I, row sums
// of row block I in segment q at q + I (both lists of [64][dim] blocks, with
// [64] sums of W beside them).
struct PtPartials {
  float *col, *colw, *row, *roww;
  double *loss;  // one per segment
};

// W of a pair with a NaN coordinate: the pair adds nothing to the gradient (a NaN
// that no operation makes).
constexpr int kPtNone = 0x7fc0abcd;

__host__ __device__ inline int64_t pt_first(int64_t I, int64_t nb) { return I * nb - I * (I - 1) / 2; }

template <int DMAX, int MODE>
__global__ void __launch_bounds__(kPtThreads, 2)
dist_pairs_kernel(const float *__restrict__ X, int64_t n, int64_t dim,
                  const float *__restrict__ aux, int64_t nb, int64_t len, PtPartials out) {
  using L = PtSmem<DMAX>;
  constexpr int DPT = DMAX / 8;  // dimensions per thread in phase 2
  extern __shared__ __align__(16) float dsm[];
  float *xi = dsm, *xj = dsm + L::X;  // [64][LD]; xj double-buffered
  float *ws = xj + 2 * L::X, *wt = ws + L::W;  // W_ij at ws[i][j] and wt[j][i]
  float *rsum = wt + L::WT;                    // [128 threads][4][DPT]
  __shared__ float wred[2][4][kPtT];           // sums of W: columns; rows (running)
  __shared__ double lred[kPtThreads / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ty = 4 * (warp >> 1) + (lane >> 3), tx = 8 * (warp & 1) + (lane & 7);
  const int side = warp >> 2, w4 = warp & 3;           // phase 2: row or column sums
  const int rg = lane >> 1, dg = 2 * w4 + (lane & 1);  // ... of rows 4 rg .., dimensions DPT dg ..
  const bool vec = (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;

  auto load = [&](float *dst, int64_t p0) {  // points p0 .. p0 + 63, zero past the end
    if (vec) {
      for (int e = tid; e < kPtT * DMAX / 4; e += kPtThreads) {
        const int r = e / (DMAX / 4), k = 4 * (e - r * (DMAX / 4));
        const bool ok = p0 + r < n && k < dim;
        cp_async16(dst + r * L::LD + k, ok ? X + (p0 + r) * dim + k : X, ok ? 16 : 0);
      }
    } else {
      for (int e = tid; e < kPtT * DMAX; e += kPtThreads) {
        const int r = e / DMAX, k = e - r * DMAX;
        const bool ok = p0 + r < n && k < dim;
        cp_async4(dst + r * L::LD + k, ok ? X + (p0 + r) * dim + k : X, ok ? 4 : 0);
      }
    }
    cp_async_commit();
  };

  // the segment's first tile (I, J)
  const int64_t total = nb * (nb + 1) / 2, t0 = int64_t(blockIdx.x) * len;
  const int64_t t1 = t0 + len < total ? t0 + len : total;
  int64_t I = 0;
  {
    int64_t lo = 0, hi = nb;  // largest I with pt_first(I) <= t0
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) / 2;
      if (pt_first(mid, nb) <= t0) lo = mid;
      else hi = mid;
    }
    I = lo;
  }
  int64_t J = I + (t0 - pt_first(I, nb));

  float acc[4][DPT], wsum[4];
  // acc to block `slot` of a partial list
  auto flush = [&](float *sums, int64_t slot) {
#pragma unroll
    for (int r = 0; r < 4; r++) {
      float *p = sums + (slot * kPtT + 4 * rg + r) * dim + DPT * dg;
#pragma unroll
      for (int k = 0; k < DPT; k++)
        if (DPT * dg + k < dim) p[k] = acc[r][k];
    }
  };
  // The row sums of each tile are formed from zero and then added to the running
  // ones (in shared memory): shorter chains of roundings.
  float *own = rsum + (tid & 127);  // element e at own[128 e]
  auto zero_rows = [&] {
    if (side == 0) {
#pragma unroll
      for (int e = 0; e < 4 * DPT; e++) own[128 * e] = 0.f;
      if ((lane & 1) == 0)
#pragma unroll
        for (int r = 0; r < 4; r++) wred[1][w4][4 * rg + r] = 0.f;
    }
  };
  zero_rows();
  FloatPairSum lsum;
  load(xi, I * kPtT);
  load(xj, J * kPtT);
  int b = 0;
  for (int64_t t = t0; t < t1; t++) {
    cp_async_wait<0>();
    __syncthreads();  // xi, xj[b] are in; the other xj and W have been read
    const bool row_ends = J + 1 == nb;
    const int64_t i0 = I * kPtT, j0 = J * kPtT;
    if (t + 1 < t1) load(xj + (b ^ 1) * L::X, (row_ends ? I + 1 : J + 1) * kPtT);
    const float *xb = xj + b * L::X;
    // ------------------------------------------------ phase 1, two columns at a time
    bool none = false;
    auto phase1 = [&](auto inner) {
      constexpr bool INNER = decltype(inner)::value;  // every pair i < j < n
#pragma unroll 1
      for (int h = 0; h < 2; h++) {
        const int64_t gj0 = j0 + tx + 32 * h;
        float cf[4][2];
#pragma unroll
        for (int a = 0; a < 4; a++) {
          const int64_t gi = i0 + ty + 16 * a;
          const float *row = aux + (MODE == 0 ? gi * n : n * gi - gi * (gi + 1) / 2 - gi - 1) + gj0;
#pragma unroll
          for (int c = 0; c < 2; c++) {
            const int64_t gj = gj0 + 16 * c;
            const bool ok = INNER || (gi < gj && gj < n);
            cf[a][c] = ok ? row[16 * c] : 0.f;
            if (MODE == 0 && ok) cf[a][c] += aux[gj * n + gi];
          }
        }
        float2 q0[4][2], q1[4][2];  // chains k mod 4 = 0, 1 and 2, 3
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
          for (int c = 0; c < 2; c++) q0[a][c] = q1[a][c] = make_float2(0.f, 0.f);
        const float *pi = xi + ty * L::LD, *pj = xb + (tx + 32 * h) * L::LD;
        const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll 2  // fully unrolled, its loads are hoisted past the registers
        for (int k = 0; k < DMAX; k += 4) {
          float4 u[4], v[2];
#pragma unroll
          for (int a = 0; a < 4; a++)
            u[a] = *reinterpret_cast<const float4 *>(pi + 16 * a * L::LD + k);
#pragma unroll
          for (int c = 0; c < 2; c++)
            v[c] = *reinterpret_cast<const float4 *>(pj + 16 * c * L::LD + k);
#pragma unroll
          for (int a = 0; a < 4; a++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
              const float2 d0 = __ffma2_rn(make_float2(v[c].x, v[c].y), minus,
                                           make_float2(u[a].x, u[a].y));
              const float2 d1 = __ffma2_rn(make_float2(v[c].z, v[c].w), minus,
                                           make_float2(u[a].z, u[a].w));
              q0[a][c] = __ffma2_rn(d0, d0, q0[a][c]);
              q1[a][c] = __ffma2_rn(d1, d1, q1[a][c]);
            }
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
          for (int c = 0; c < 2; c++) {
            const int il = ty + 16 * a, jl = tx + 16 * (2 * h + c);
            const float d2 = (q0[a][c].x + q0[a][c].y) + (q1[a][c].x + q1[a][c].y);
            float w = 0.f;
            if (INNER || (i0 + il < j0 + jl && j0 + jl < n)) {
              float inv_d = 0.f, d = 0.f;
              if (d2 >= 1e-30f) {
                inv_d = tc::rsqrt_approx(d2);
                d = d2 * inv_d;
              } else if (d2 > 0.f) {
                d = sqrtf(d2);
                inv_d = 1.f / d;
              }
              if (MODE == 1) {
                const float e = d - cf[a][c], q = e * e;
                lsum.add(q);
                lsum.lo += fmaf(e, e, -q);
              }
              // coincident points add to the stress but not to the gradient
              if (d2 > 0.f) w = MODE == 0 ? cf[a][c] * inv_d : 2.f * (d - cf[a][c]) * inv_d;
              if (d2 != d2) {
                w = __int_as_float(kPtNone);
                none = true;
              }
            }
            ws[il * L::LW + jl] = w;
            wt[jl * L::LT + il] = w;
          }
      }
    };
    if (I < J && j0 + kPtT <= n) phase1(std::true_type{});
    else phase1(std::false_type{});
    const bool skips = __syncthreads_or(none);
    // ------------------------------------------------ phase 2
#pragma unroll
    for (int r = 0; r < 4; r++) {
      wsum[r] = 0.f;
#pragma unroll
      for (int k = 0; k < DPT; k++) acc[r][k] = 0.f;
    }
    const float *pw = (side ? ws : wt) + 4 * rg, *px = (side ? xi : xb) + DPT * dg;
    const int lw = side ? L::LW : L::LT;
    auto rows16 = [&](int m0, auto sum_w) {
#pragma unroll 8
      for (int m = m0; m < m0 + kPtT / 4; m++) {
        const float4 w = *reinterpret_cast<const float4 *>(pw + m * lw);
        const float wr[4] = {w.x, w.y, w.z, w.w};
        __align__(16) float v[DPT];
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {  // DPT even: 8-byte reads at least
          if (DPT % 4 == 0 && k % 4 == 0)
            *reinterpret_cast<float4 *>(v + k) =
                *reinterpret_cast<const float4 *>(px + m * L::LD + k);
          else if (DPT % 4 != 0)
            *reinterpret_cast<float2 *>(v + k) =
                *reinterpret_cast<const float2 *>(px + m * L::LD + k);
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
#pragma unroll
          for (int k = 0; k < DPT; k++) acc[r][k] = fmaf(wr[r], v[k], acc[r][k]);
          if constexpr (decltype(sum_w)::value) wsum[r] += wr[r];
        }
      }
    };
    if (!skips) {
#pragma unroll 1
      for (int q = 0; q < 4; q++) {  // a quarter of the sums of W in each warp
        if (q == w4) rows16(16 * q, std::true_type{});
        else rows16(16 * q, std::false_type{});
      }
    } else {  // a NaN coordinate in the tile: only the pairs that count (0 * NaN would not be 0)
#pragma unroll 1
      for (int m = 0; m < kPtT; m++) {
#pragma unroll 1
        for (int r = 0; r < 4; r++) {
          const float w = pw[m * lw + r];
          const int64_t i = i0 + (side ? m : 4 * rg + r), j = j0 + (side ? 4 * rg + r : m);
          if (i >= j || j >= n || __float_as_int(w) == kPtNone) continue;
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (q != r) continue;
#pragma unroll
            for (int k = 0; k < DPT; k++) acc[q][k] = fmaf(w, px[m * L::LD + k], acc[q][k]);
            if (m >> 4 == w4) wsum[q] += w;
          }
        }
      }
    }
    const bool flush_row = row_ends || t + 1 == t1;  // uniform
    if (side == 1) {
      flush(out.col, J * (J + 1) / 2 + I);
    } else {
#pragma unroll
      for (int r = 0; r < 4; r++)
#pragma unroll
        for (int k = 0; k < DPT; k++) {
          acc[r][k] += own[128 * (r * DPT + k)];
          own[128 * (r * DPT + k)] = flush_row ? 0.f : acc[r][k];
        }
      if (flush_row) flush(out.row, int64_t(blockIdx.x) + I);
    }
    // the four warps' shares of the sums of W: the columns', the rows' running ones
    if ((lane & 1) == 0) {
#pragma unroll
      for (int r = 0; r < 4; r++) {
        float *p = &wred[side ? 0 : 1][w4][4 * rg + r];
        *p = side ? wsum[r] : *p + wsum[r];
      }
    }
    __syncthreads();
    if (tid < 2 * kPtT && (tid < kPtT || flush_row)) {
      const int sd = tid >> 6, r = tid & 63;  // columns: the first 64 threads, rows: the next
      const float sum = (wred[sd][0][r] + wred[sd][1][r]) + (wred[sd][2][r] + wred[sd][3][r]);
      if (sd) {
        out.roww[(int64_t(blockIdx.x) + I) * kPtT + r] = sum;
#pragma unroll
        for (int q = 0; q < 4; q++) wred[1][q][r] = 0.f;
      } else {
        out.colw[(J * (J + 1) / 2 + I) * kPtT + r] = sum;
      }
    }
    if (row_ends) {
      I++;
      J = I;
      if (t + 1 < t1) load(xi, I * kPtT);  // (the barrier above: its readers are done)
    } else {
      J++;
    }
    b ^= 1;
  }
  if (MODE == 1) {
    float lh = lsum.hi, ll = lsum.lo;
    warp_pair_sum(lh, ll);
    if (lane == 0) lred[warp] = double(lh) + double(ll);
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
      for (int q = 0; q < kPtThreads / 32; q++) s += lred[q];
      out.loss[blockIdx.x] = s;
    }
  }
}

// dX_i = x_i * sum of W - sum of the partial sums, in a fixed order: the row
// block's segments, then the tiles above it.  A block takes 8 points: a warp
// sums each one's W, then a thread each (point, dimension), in four chains.
constexpr int kPtRedRows = 8;
__global__ void __launch_bounds__(256)
dist_pairs_reduce_kernel(const float *__restrict__ X, int64_t n, int64_t dim, int64_t nb,
                         int64_t len, PtPartials in, float *__restrict__ dX) {
  __shared__ float w[kPtRedRows];
  const int64_t i0 = int64_t(blockIdx.x) * kPtRedRows, B = i0 / kPtT, r0 = i0 - B * kPtT;
  const int64_t q0 = pt_first(B, nb) / len, nq = (pt_first(B + 1, nb) - 1) / len - q0 + 1;
  const int64_t c0 = B * (B + 1) / 2;
  {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float s = 0.f;
    for (int64_t q = lane; q < nq; q += 32) s += in.roww[(q0 + q + B) * kPtT + r0 + warp];
    for (int64_t q = lane; q <= B; q += 32) s += in.colw[(c0 + q) * kPtT + r0 + warp];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) w[warp] = s;
  }
  __syncthreads();
  const int64_t rows = n - i0 < kPtRedRows ? n - i0 : kPtRedRows, step = kPtT * dim;
  for (int64_t e = threadIdx.x; e < rows * dim; e += 256) {
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    const float *p = in.row + (q0 + B) * step + r0 * dim + e;
    for (int64_t q = 0; q < nq; q++) a[0] += p[q * step];
    p = in.col + c0 * step + r0 * dim + e;
    int64_t q = 0;
    for (; q + 8 <= B + 1; q += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = p[(q + u) * step];
#pragma unroll
      for (int u = 0; u < 8; u++) a[u & 3] += v[u];
    }
    for (; q <= B; q++) a[0] += p[q * step];
    dX[i0 * dim + e] = fmaf(X[i0 * dim + e], w[e / dim], -((a[0] + a[1]) + (a[2] + a[3])));
  }
}

// The partial losses summed by one CTA in a fixed order (thread t takes
// t, t + 1024, ...; then a butterfly in each warp and across the warps), so
// the result does not depend on timing.
constexpr int kLossThreads = 1024;
__global__ void __launch_bounds__(kLossThreads)
loss_reduce_kernel(const double *__restrict__ ploss, int64_t count, double *__restrict__ loss) {
  __shared__ double sh[kLossThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double t = 0.0;
  for (int64_t i = threadIdx.x; i < count; i += kLossThreads) t += ploss[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) sh[warp] = t;
  __syncthreads();
  if (warp == 0) {
    t = sh[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) *loss = t;
  }
}

// ---------------------------------------------- distances on the tensor cores
// Column means of the points as FP64 (compensated float sums per thread, a
// fixed-order block reduction): one CTA per dimension.
__global__ void __launch_bounds__(kFinThreads)
adj_colmean_kernel(const float *__restrict__ X, int64_t n, int64_t dim, double *__restrict__ mean) {
  __shared__ double sh[32];
  const int64_t c = blockIdx.x;
  double v = 0.0;
  float hi = 0.f, lo = 0.f;
  for (int64_t i = threadIdx.x; i < n; i += kFinThreads) {
    const float x = X[i * dim + c];
    const float t = hi + x, bp = t - hi;
    lo += (hi - (t - bp)) + (x - bp);
    hi = t;
  }
  v = double(hi) + double(lo);
  v = block_sum_d(v, sh);
  if (threadIdx.x == 0) mean[c] = v / double(n);
}

// Centred points Xc (n x dim) and the GEMM's B operand: rows c (dimensions),
// columns j (points, ld kp, zero padded), three bf16 planes; 32 x 32 tiles
// transposed through shared memory.
__global__ void adj_points_kernel(const float *__restrict__ X, int64_t n, int64_t dim,
                                  int64_t kp, const double *__restrict__ mean,
                                  float *__restrict__ Xc, __nv_bfloat16 *__restrict__ Bt) {
  __shared__ float tile[32][33];
  const int64_t j0 = int64_t(blockIdx.x) * 32, c0 = int64_t(blockIdx.y) * 32;
  const int tx = threadIdx.x, ty0 = threadIdx.y;
  for (int ty = ty0; ty < 32; ty += 8) {
    const int64_t j = j0 + ty, c = c0 + tx;
    float v = 0.f;
    if (j < n && c < dim) {
      v = float(double(X[j * dim + c]) - mean[c]);
      Xc[j * dim + c] = v;
    }
    tile[ty][tx] = v;  // rows j
  }
  __syncthreads();
  const int64_t plane = dim * kp;
  for (int ty = ty0; ty < 32; ty += 8) {
    const int64_t c = c0 + ty, j = j0 + tx;
    if (c >= dim || j >= kp) continue;
    put_parts<__nv_bfloat16>(Bt, plane, c * kp + j, tile[tx][ty], 3);
  }
}

// W as the GEMM's A operand (rows i, columns j, ld kp, three bf16 planes),
// from the full distance matrix D and G (MODE 0: W = (G + G^T) / D) or the
// targets delta in R's dist layout (MODE 1: W = 2 (D - delta) / D); W_ii and
// W_ij with D_ij = 0 are 0.  Per 32 x 64 tile (two columns per thread, so the
// plane stores are 4 bytes): the rows' partial sums of W (rsum[i * nbj + jb])
// and, for MODE 1, the tile's part of the stress sum_{i<j} (D - delta)^2
// (lpart[ib * nbj + jb]); both are reduced in a fixed order afterwards.  G^T,
// and delta below the diagonal (stored by column there), go through shared
// memory so that every global read is coalesced; the stress sums as
// compensated float pairs.
constexpr int kAwRows = 32, kAwCols = 64;
template <int MODE>
__global__ void __launch_bounds__(256)
adj_weight_kernel(const float *__restrict__ D, const float *__restrict__ aux, int64_t n,
                  int64_t kp, __nv_bfloat16 *__restrict__ Wp, float *__restrict__ rsum,
                  double *__restrict__ lpart) {
  // MODE 0: tt[jj][ii] = G[j][i] (64 x 32); MODE 1: tt[ii][jj] = delta(i, j), i != j (32 x 64)
  __shared__ float tt[MODE == 0 ? kAwCols : kAwRows][MODE == 0 ? kAwRows + 1 : kAwCols + 1];
  __shared__ double lsh[8];
  const int64_t i0 = int64_t(blockIdx.y) * kAwRows, j0 = int64_t(blockIdx.x) * kAwCols;
  const int tx = threadIdx.x, ty0 = threadIdx.y;
  const int64_t nbj = gridDim.x;
  if (MODE == 0) {
    for (int jj = ty0; jj < kAwCols; jj += 8) {
      const int64_t j = j0 + jj, i = i0 + tx;
      tt[jj][tx] = (j < n && i < n) ? aux[j * n + i] : 0.f;
    }
  } else {
    // above the diagonal: row i of the dist layout, consecutive j
    for (int ii = ty0; ii < kAwRows; ii += 8) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int jj = tx + 32 * h;
        const int64_t i = i0 + ii, j = j0 + jj;
        if (i < n && j < n && i < j) tt[ii][jj] = aux[n * i - i * (i + 1) / 2 + j - i - 1];
      }
    }
    // below: delta(i, j) = delta(j, i), row j of the dist layout, consecutive i
    for (int jj = ty0; jj < kAwCols; jj += 8) {
      const int64_t i = i0 + tx, j = j0 + jj;
      if (i < n && j < n && i > j) tt[tx][jj] = aux[n * j - j * (j + 1) / 2 + i - j - 1];
    }
  }
  __syncthreads();
  const int64_t plane = n * kp;
  FloatPairSum lsum;
  for (int ii = ty0; ii < kAwRows; ii += 8) {
    const int64_t i = i0 + ii;
    float w[2] = {0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int jj = 2 * tx + h;
      const int64_t j = j0 + jj;
      if (i < n && j < n && i != j) {
        const float d = D[i * n + j];
        if (MODE == 0) {
          if (d > 0.f) w[h] = __fdividef(aux[i * n + j] + tt[jj][ii], d);
        } else {
          const float del = tt[ii][jj];
          const float e = d > 0.f ? d - del : -del;  // coincident points: in the stress only
          if (d > 0.f) w[h] = __fdividef(2.f * e, d);
          if (i < j) {
            const float q = e * e;
            lsum.add(q);
            lsum.lo += fmaf(e, e, -q);
          }
        }
      }
    }
    const int64_t j = j0 + 2 * tx;  // even, and kp is a multiple of 64
    if (i < n && j < kp) {
      uint16_t a[3], b[3];
      tc::split_parts<tc::KIND_BF16X6>(w[0], a);
      tc::split_parts<tc::KIND_BF16X6>(w[1], b);
      uint32_t *dst = reinterpret_cast<uint32_t *>(Wp + i * kp + j);
#pragma unroll
      for (int q = 0; q < 3; q++)
        dst[q * (plane / 2)] = uint32_t(a[q]) | (uint32_t(b[q]) << 16);
    }
    // row sum of the tile: the 32 lanes of a row, two columns each
    float r = w[0] + w[1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (tx == 0 && i < n) rsum[i * nbj + blockIdx.x] = r;
  }
  if (MODE == 1) {
    float lh = lsum.hi, ll = lsum.lo;
    warp_pair_sum(lh, ll);
    if (tx == 0) lsh[ty0] = double(lh) + double(ll);
    __syncthreads();
    if (tx == 0 && ty0 == 0) {
      double t = 0.0;
      for (int w = 0; w < 8; w++) t += lsh[w];
      lpart[int64_t(blockIdx.y) * nbj + blockIdx.x] = t;
    }
  }
}

// dX_i = xc_i * sum_b rsum[i][b] - C_i (C = W Xc, the sum of `parts` pieces
// of n x dim), the row's partials added in order (compensated), one warp per
// point.
__global__ void adj_finish_kernel(const float *__restrict__ Xc, const float *__restrict__ C,
                                  int parts, const float *__restrict__ rsum, int64_t n,
                                  int64_t dim, int64_t nbj, float *__restrict__ dX) {
  const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  float hi = 0.f, lo = 0.f;
  for (int64_t b = lane; b < nbj; b += 32) {
    const float x = rsum[i * nbj + b];
    const float t = hi + x, bp = t - hi;
    lo += (hi - (t - bp)) + (x - bp);
    hi = t;
  }
  warp_pair_sum_f(hi, lo);
  const float r = hi + lo;
  for (int64_t c = lane; c < dim; c += 32) {
    float w = C[i * dim + c];
    for (int q = 1; q < parts; q++) w += C[int64_t(q) * n * dim + i * dim + c];
    dX[i * dim + c] = fmaf(Xc[i * dim + c], r, -w);
  }
}

template <int MODE>
int dist_backward_tc(const float *X, int64_t n, int64_t dim, const float *aux, float *dX,
                     double *loss, cudaStream_t s) {
  const int64_t kp = cdiv(n, kKPadB) * kKPadB;
  // weight tiles: rows of 32, columns of 64 covering the padded k
  const int64_t nbj = kp / kAwCols, nbi = cdiv(n, int64_t(kAwRows));
  void *pD = nullptr, *pW = nullptr, *pM = nullptr;
  // the full distance matrix (tcgen05 Gram, near-zero pairs recomputed exactly)
  GT_TRY(ws_get(WS_ADJ0, size_t(n) * size_t(n) * 4, &pD));
  float *D = static_cast<float *>(pD);
  GT_TRY(euclid_tc(X, n, dim, D, GT_LAYOUT_FULL, s));
  GT_TRY(ws_get(WS_ADJ1, size_t(3) * size_t(n) * size_t(kp) * 2, &pW));
  auto *Wp = static_cast<__nv_bfloat16 *>(pW);
  // W Xc in K pieces when its output tiles alone would leave most SMs idle
  const int64_t out_tiles = cdiv(n, int64_t(128)) * cdiv(dim, int64_t(256));
  int parts = 1;
  while (parts < 4 && out_tiles * (parts + 1) <= int64_t(sm_count())) parts++;
  // misc: means | Xc | B planes | C (parts pieces) | rsum | loss parts
  const size_t b_mean = size_t(dim) * 8, b_xc = size_t(n) * size_t(dim) * 4;
  const size_t b_bt = size_t(3) * size_t(dim) * size_t(kp) * 2, b_c = size_t(parts) * b_xc;
  const size_t b_rs = size_t(n) * size_t(nbj) * 4, b_lp = size_t(nbi) * size_t(nbj) * 8;
  auto r256 = [](size_t b) { return (b + 255) & ~size_t(255); };
  GT_TRY(ws_get(WS_ADJ2, r256(b_mean) + r256(b_xc) + r256(b_bt) + r256(b_c) + r256(b_rs) + b_lp,
                &pM));
  char *m = static_cast<char *>(pM);
  auto *mean = reinterpret_cast<double *>(m);
  auto *Xc = reinterpret_cast<float *>(m + r256(b_mean));
  auto *Bt = reinterpret_cast<__nv_bfloat16 *>(m + r256(b_mean) + r256(b_xc));
  auto *C = reinterpret_cast<float *>(m + r256(b_mean) + r256(b_xc) + r256(b_bt));
  auto *rsum = reinterpret_cast<float *>(m + r256(b_mean) + r256(b_xc) + r256(b_bt) + r256(b_c));
  auto *lp = reinterpret_cast<double *>(m + r256(b_mean) + r256(b_xc) + r256(b_bt) + r256(b_c) +
                                        r256(b_rs));
  if (nbi > 65535 || cdiv(dim, 32) > 65535) return fail(GT_EINVAL, "too many points (%lld)", (long long)n);
  const dim3 blk(32, 8);
  adj_colmean_kernel<<<unsigned(dim), kFinThreads, 0, s>>>(X, n, dim, mean);
  adj_points_kernel<<<dim3(unsigned(kp / 32), unsigned(cdiv(dim, 32))), blk, 0, s>>>(
      X, n, dim, kp, mean, Xc, Bt);
  adj_weight_kernel<MODE><<<dim3(unsigned(nbj), unsigned(nbi)), blk, 0, s>>>(
      D, aux, n, kp, Wp, rsum, lp);
  count_launch(3);
  GT_CUDA(cudaGetLastError());
  // C = W Xc on the tensor cores (rows i, columns c)
  if (parts > 1)
    GT_TRY(gemm_tc_store_ksplit(Wp, n, Bt, dim, kp, parts, &parts, C, dim, s));
  else
    GT_TRY(gemm_tc_store(Wp, n, Bt, dim, kp, 3, C, dim, s));
  adj_finish_kernel<<<unsigned(cdiv(n * 32, 256)), 256, 0, s>>>(Xc, C, parts, rsum, n, dim, nbj,
                                                                  dX);
  count_launch();
  if (MODE == 1 && loss) {
    loss_reduce_kernel<<<1, kLossThreads, 0, s>>>(lp, nbi * nbj, loss);
    count_launch();
  }
  GT_CUDA(cudaGetLastError());
  return GT_OK;
}

// Bytes of the pair kernel's column sums.
int64_t dist_pairs_bytes(int64_t n, int64_t dim) {
  const int64_t nb = cdiv(n, kPtT);
  return nb * (nb + 1) / 2 * kPtT * (dim + 1) * 4;
}

// False, with nothing done, where its scratch cannot be had.
template <int DMAX, int MODE>
bool dist_backward_pairs(const float *X, int64_t n, int64_t dim, const float *aux, float *dX,
                         double *loss, cudaStream_t s, int *status) {
  using L = PtSmem<DMAX>;
  void *pc = nullptr;
  // the largest buffer first: the ordered kernel's fits where it does not
  if (!ws_try(WS_SCRATCH0, size_t(dist_pairs_bytes(n, dim)), s, &pc)) return false;
  const int64_t nb = cdiv(n, kPtT), total = nb * (nb + 1) / 2;
  auto kern = dist_pairs_kernel<DMAX, MODE>;
  int per = 0;
  *status = [&]() -> int {
    GT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES));
    GT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kPtThreads, L::BYTES));
    return GT_OK;
  }();
  if (*status != GT_OK) return true;
  const int64_t slots = int64_t(sm_count()) * (per < 1 ? 1 : per);
  const int64_t len = cdiv(total, slots), segs = cdiv(total, len);
  void *pr = nullptr, *pl = nullptr;
  if (!ws_try(WS_SCRATCH1, size_t(segs + nb) * kPtT * size_t(dim + 1) * 4, s, &pr) ||
      !ws_try(WS_SCRATCH2, size_t(segs) * 8, s, &pl))
    return false;
  PtPartials pp;
  pp.col = static_cast<float *>(pc);
  pp.colw = pp.col + total * kPtT * dim;
  pp.row = static_cast<float *>(pr);
  pp.roww = pp.row + (segs + nb) * kPtT * dim;
  pp.loss = static_cast<double *>(pl);
  kern<<<unsigned(segs), kPtThreads, L::BYTES, s>>>(X, n, dim, aux, nb, len, pp);
  dist_pairs_reduce_kernel<<<unsigned(cdiv(n, kPtRedRows)), 256, 0, s>>>(X, n, dim, nb, len, pp,
                                                                       dX);
  count_launch(2);
  if (MODE == 1 && loss) {
    loss_reduce_kernel<<<1, kLossThreads, 0, s>>>(pp.loss, segs, loss);
    count_launch();
  }
  *status = [&]() -> int {
    GT_CUDA(cudaGetLastError());
    return GT_OK;
  }();
  return true;
}

template <int MODE>
int launch_dist_backward(const float *X, int64_t n, int64_t dim, const float *aux, float *dX,
                         double *loss, cudaStream_t s) {
  // Up to 64 dimensions each unordered pair once, while the partial sums take at
  // most 1 GB (about 33000 points at 32 dimensions, 23000 at 64).  Measured (MDS
  // stress, us, pairs / ordered pairs / tensor cores): 1000 x 32 24 / 34 / -,
  // 4096 x 64 150 / 236 / 235, 8192 x 16 203 / 309 / -, 8192 x 32 299 / 455 / 670,
  // 8192 x 48 507 / 790 / 671, 10000 x 40 720 / - / 1090.  Past that the ordered
  // kernel holds no n^2 workspace; above 32 dimensions and up to 32768 points
  // (11 GB there) the tensor-core form is 10-15 % faster than it, and above 64
  // dimensions it is the only one.  They also take the problems whose partial sums
  // the device has no room for.
  if (dim <= 64 && dist_pairs_bytes(n, dim) <= (int64_t(1) << 30)) {
    int status = GT_OK;
    if (dim <= 16   ? dist_backward_pairs<16, MODE>(X, n, dim, aux, dX, loss, s, &status)
        : dim <= 32 ? dist_backward_pairs<32, MODE>(X, n, dim, aux, dX, loss, s, &status)
                    : dist_backward_pairs<64, MODE>(X, n, dim, aux, dX, loss, s, &status))
      return status;
  }
  if (dim > 64 || (dim > 32 && n >= 8192 && n <= 32768))
    return dist_backward_tc<MODE>(X, n, dim, aux, dX, loss, s);
  const int64_t ib = cdiv(n, kDbRows);
  // the kernel for the dimension, its shared memory, and the CTAs per SM
  auto pick = [&](auto kern, int bytes) -> int {
    int per = 0;
    if (bytes > 48 * 1024)
      GT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    GT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kDbRows, bytes));
    return per;
  };
  int per_sm = 0;
  if (dim <= 16) per_sm = pick(dist_backward_kernel<16, MODE>, DbSmem<16, MODE>::BYTES);
  else if (dim <= 32) per_sm = pick(dist_backward_kernel<32, MODE>, DbSmem<32, MODE>::BYTES);
  else per_sm = pick(dist_backward_kernel<64, MODE>, DbSmem<64, MODE>::BYTES);
  if (per_sm < 1) per_sm = 1;
  // the split count whose CTAs fill whole waves best (up to four waves; more
  // splits only when they fill clearly better)
  const int64_t slots = int64_t(sm_count()) * per_sm;
  int64_t nsplit = 1;
  double best_fill = 0.0;
  for (int64_t w = 1; w <= 4; w++) {
    const int64_t ns = w * slots / ib;
    if (ns < 1) continue;
    const double fill = double(ns * ib) / double(w * slots);
    if (fill > best_fill + 0.02) {
      best_fill = fill;
      nsplit = ns;
    }
  }
  const int64_t max_split = cdiv(n, kDbCols);
  if (nsplit > max_split) nsplit = max_split;
  if (nsplit < 1) nsplit = 1;
  if (nsplit > 65535) nsplit = 65535;
  const int64_t jchunk = cdiv(cdiv(n, nsplit), kDbCols) * kDbCols;
  nsplit = cdiv(n, jchunk);
  void *pa = nullptr, *pw = nullptr, *pl = nullptr;
  GT_TRY(ws_get(WS_SCRATCH0, size_t(nsplit) * size_t(n) * size_t(dim) * 4, &pa));
  GT_TRY(ws_get(WS_SCRATCH1, size_t(nsplit) * size_t(n) * 4, &pw));
  GT_TRY(ws_get(WS_SCRATCH2, size_t(nsplit) * size_t(ib) * 8, &pl));
  const dim3 grid(unsigned(ib), unsigned(nsplit), 1u);
  float *fa = static_cast<float *>(pa), *fw = static_cast<float *>(pw);
  double *dl = static_cast<double *>(pl);
  if (dim <= 16)
    dist_backward_kernel<16, MODE><<<grid, kDbRows, DbSmem<16, MODE>::BYTES, s>>>(
        X, n, dim, aux, jchunk, fa, fw, dl);
  else if (dim <= 32)
    dist_backward_kernel<32, MODE><<<grid, kDbRows, DbSmem<32, MODE>::BYTES, s>>>(
        X, n, dim, aux, jchunk, fa, fw, dl);
  else
    dist_backward_kernel<64, MODE><<<grid, kDbRows, DbSmem<64, MODE>::BYTES, s>>>(
        X, n, dim, aux, jchunk, fa, fw, dl);
  int64_t g = cdiv(n * dim, 256);
  if (g > int64_t(sm_count()) * 8) g = int64_t(sm_count()) * 8;
  dist_backward_reduce_kernel<<<unsigned(g), 256, 0, s>>>(X, n, dim, nsplit, fa, fw, dX);
  count_launch(2);
  if (MODE == 1 && loss) {
    loss_reduce_kernel<<<1, kLossThreads, 0, s>>>(dl, ib * nsplit, loss);
    count_launch();
  }
  GT_CUDA(cudaGetLastError());
  return GT_OK;
}

}  // namespace

int cor_backward_impl(const float *dX, int64_t p, int64_t n, const float *dG, float *d_dX,
                      cudaStream_t s) {
  if (p == 0 || n == 0) return GT_OK;
  const int path = gt_get_gram_path();
  const int64_t kp = cdiv(p, kKPadB) * kKPadB;
  void *pst = nullptr, *pS = nullptr, *pZ = nullptr, *pW = nullptr;
  GT_TRY(ws_get(WS_SCRATCH3, size_t(p) * sizeof(ColStats), &pst));
  ColStats *st = static_cast<ColStats *>(pst);
  ProfScope prof("cor_backward", s);
  GT_TRY(launch_colstats(dX, p, n, GT_EVERYTHING, st, s));
  GT_TRY(ws_get(WS_SCRATCH4 + 0, 256, &pW));  // keep the small slot allocated
  GT_TRY(ws_get(WS_OUT2, size_t(p) * size_t(n) * 4, &pW));
  float *W = static_cast<float *>(pW);
  const dim3 blk(32, 8);
  if (path == GT_GRAM_FP32) {
    GT_TRY(ws_get(WS_SCRATCH0, size_t(p) * size_t(kp) * 4, &pS));
    GT_TRY(ws_get(WS_SCRATCH1, size_t(n) * size_t(kp) * 4, &pZ));
    sym_operand_kernel<float><<<dim3(unsigned(kp / 64), unsigned(cdiv(p, 64))), blk, 0, s>>>(
        dG, p, kp, 1, static_cast<float *>(pS));
    zt_operand_kernel<float><<<dim3(unsigned(cdiv(n, 32)), unsigned(kp / 32)), blk, 0, s>>>(
        dX, p, n, kp, st, 1, static_cast<float *>(pZ));
    count_launch(2);
    SimtArgs a;
    a.R = static_cast<float *>(pS); a.C = static_cast<float *>(pZ);
    a.ldr = a.ldc = kp;
    a.nr = p; a.nc = n; a.K = kp;
    a.symmetric = 0; a.vec_ok = 1;
    cudaError_t e = launch_allpairs_simt<OpDotB, OutStore, 8, 8>(a, OpDotB{}, OutStore{W, n}, s);
    if (e != cudaSuccess) return fail(GT_ECUDA, "adjoint GEMM launch: %s", cudaGetErrorString(e));
  } else if (path == GT_GRAM_TC_F16X3 || path == GT_GRAM_TC_F16X6) {
    // f16x3 with every operand row scaled by a power of two (G + G^T is not
    // unit-scaled; z^T is bounded by 1 and takes one scale): three products,
    // the scales undone in the store
    void *prm = nullptr, *psc = nullptr;
    GT_TRY(ws_get(WS_ADJ0, size_t(p) * 4, &prm));
    GT_TRY(ws_get(WS_ADJ2, size_t(p + n) * 4, &psc));
    GT_TRY(ws_get(WS_SCRATCH0, size_t(2) * size_t(p) * size_t(kp) * 2, &pS));
    GT_TRY(ws_get(WS_SCRATCH1, size_t(2) * size_t(n) * size_t(kp) * 2, &pZ));
    auto *rowmax = static_cast<unsigned *>(prm);
    auto *scS = static_cast<float *>(psc), *scZ = scS + p;
    GT_CUDA(cudaMemsetAsync(rowmax, 0, size_t(p) * 4, s));
    const dim3 pairs(unsigned(kp / 64), unsigned(kp / 64));
    const int vec = p % 4 == 0 && (reinterpret_cast<uintptr_t>(dG) & 15) == 0;
    sym_rowmax_kernel<<<pairs, 256, 0, s>>>(dG, p, vec, rowmax);
    sym_split_kernel<<<pairs, 256, 0, s>>>(dG, p, kp, vec, rowmax, static_cast<uint16_t *>(pS), scS);
    zt_split_kernel<<<dim3(unsigned(cdiv(n, 32)), unsigned(kp / 64)), blk, 0, s>>>(
        dX, p, n, kp, st, static_cast<uint16_t *>(pZ), scZ);
    count_launch(3);
    GT_CUDA(cudaGetLastError());
    GT_TRY(gemm_tc_store_scaled(pS, p, pZ, n, kp, scS, scZ, W, n, s));
  } else {
    const int ns = path == GT_GRAM_TC_BF16X3 ? 2 : 3;
    GT_TRY(ws_get(WS_SCRATCH0, size_t(ns) * size_t(p) * size_t(kp) * 2, &pS));
    GT_TRY(ws_get(WS_SCRATCH1, size_t(ns) * size_t(n) * size_t(kp) * 2, &pZ));
    sym_operand_kernel<__nv_bfloat16>
        <<<dim3(unsigned(kp / 64), unsigned(cdiv(p, 64))), blk, 0, s>>>(
            dG, p, kp, ns, static_cast<__nv_bfloat16 *>(pS));
    zt_operand_kernel<__nv_bfloat16><<<dim3(unsigned(cdiv(n, 32)), unsigned(kp / 32)), blk, 0, s>>>(
        dX, p, n, kp, st, ns, static_cast<__nv_bfloat16 *>(pZ));
    count_launch(2);
    GT_CUDA(cudaGetLastError());
    GT_TRY(gemm_tc_store(pS, p, pZ, n, kp, ns, W, n, s));
  }
  cor_backward_finish_kernel<<<unsigned(cdiv(p, kFinThreads / 32)), kFinThreads, 0, s>>>(
      dX, p, n, st, W, d_dX);
  count_launch();
  GT_CUDA(cudaGetLastError());
  return GT_OK;
}

}  // namespace gt

extern "C" int gt_cor_backward_device(const float *d_X, int64_t p, int64_t n, const float *d_G,
                                      float *d_dX, void *stream) {
  gt::clear_error();
  if (p < 0 || n < 0) return gt::fail(GT_EINVAL, "negative size");
  if (p > 2147483647LL) return gt::fail(GT_EINVAL, "too many variables");
  if (p > 0 && n > 0 && (!d_X || !d_G || !d_dX)) return gt::fail(GT_EINVAL, "null device pointer");
  return gt::cor_backward_impl(d_X, p, n, d_G, d_dX, static_cast<cudaStream_t>(stream));
}

extern "C" int gt_dist_backward_device(const float *d_X, int64_t n, int64_t dim, const float *d_G,
                                       float *d_dX, void *stream) {
  gt::clear_error();
  if (n < 0 || dim < 0) return gt::fail(GT_EINVAL, "negative size");
  if (n == 0 || dim == 0) return GT_OK;
  if (!d_X || !d_G || !d_dX) return gt::fail(GT_EINVAL, "null device pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  gt::ProfScope prof("dist_backward", s);
  return gt::launch_dist_backward<0>(d_X, n, dim, d_G, d_dX, nullptr, s);
}

extern "C" int gt_mds_stress_device(const float *d_X, int64_t n, int64_t dim,
                                    const float *d_delta, float *d_dX, double *d_loss,
                                    void *stream) {
  gt::clear_error();
  if (n < 0 || dim < 0) return gt::fail(GT_EINVAL, "negative size");
  if (n == 0 || dim == 0) return GT_OK;
  if (!d_X || !d_delta || !d_dX) return gt::fail(GT_EINVAL, "null device pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  gt::ProfScope prof("mds_stress", s);
  return gt::launch_dist_backward<1>(d_X, n, dim, d_delta, d_dX, d_loss, s);
}
