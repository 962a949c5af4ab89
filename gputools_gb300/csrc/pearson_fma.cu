// pearson_fma.cu -- "everything" Pearson of small problems on CUDA cores.
//
// Reference: the three per-pair kernels of src/correlation.cpp:66-161
// (inst/cuda/correlation.cu:7-292).
//
// The tensor-core Gram (gram_tc.cu) computes 128 x 256 tiles, one CTA each:
// a problem of a few tiles leaves most SMs idle while a handful of warps write
// the outputs (40 observations x 100 variables: one CTA, 30 us).  Here two
// launches, statistics with the normalised rows in float, and the products in
// 32 x 32 tiles, spread the same work over the chip.  The products are FP32
// multiply-adds, summed in runs of 32 that are added to second sums, so the error stays below that of the f16x3 Gram, whose path
// (GT_GRAM_TC_F16X3) alone comes here.
#include "common.cuh"
#include "gram_core.cuh"
#include "kernels.cuh"
#include "stats.cuh"

namespace gt {

namespace {

constexpr int kFmaThreads = 256;
constexpr int kFmaK = 32;  // observations per slab

// One warp per variable: z = (x - mean) / ||x - mean|| in rows of ldz floats,
// zero past n; NaN for a variable with a NaN or without variance.  Rows nA ..
// of the output are the second operand's.
__global__ void __launch_bounds__(kFmaThreads)
pearson_norm_kernel(const float *__restrict__ A, int64_t nA, const float *__restrict__ B,
                    int64_t nvar, int64_t n, int64_t ldz, float *__restrict__ Z) {
  const int64_t v = (int64_t(blockIdx.x) * kFmaThreads + threadIdx.x) >> 5;
  if (v >= nvar) return;  // whole warps
  const float *x = v < nA ? A + v * n : B + (v - nA) * n;
  const ColStats st = colstats_warp(x, n, GT_EVERYTHING);
  const Centerer cen(st);
  float *z = Z + v * ldz;
  for (int64_t k = threadIdx.x & 31; k < ldz; k += 32)
    z[k] = k >= n ? 0.f : (st.flags ? __int_as_float(0x7fc00000) : cen(x[k]));
}

// One 32 x 32 tile of r, t and pairs per CTA.  Four groups of 64 threads take a
// quarter of the observations each, 4 x 4 entries a thread: with so few warps a
// SM the products' latency counts, and this makes 64 of them from 8 shared
// reads.  Slabs of 32 observations come in through a ring of four
// (cp.async).  Symmetric problems run the tiles on and above the diagonal and
// write both orientations from the tile staged in shared memory, each store 32
// consecutive floats.
constexpr int kFmaTile = 32, kFmaLd = kFmaK + 4;  // rows 4 banks apart: no conflicts
constexpr int kFmaStages = 4, kFmaSlab = kFmaTile * kFmaLd;

__device__ __forceinline__ void cp_async16(float *dst, const float *src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src),
               "r"(live ? 16 : 0)  // bytes read; the rest of the 16 is zero
               : "memory");
}

__global__ void __launch_bounds__(kFmaThreads)
pearson_fma_kernel(const float *__restrict__ ZA, const float *__restrict__ ZB, int64_t ldz,
                   const PearsonFinish fin) {
  const int tcols = int((fin.nc + kFmaTile - 1) / kFmaTile);
  const int ti = int(blockIdx.x) / tcols, tj = int(blockIdx.x) - ti * tcols;
  if (fin.symmetric && ti > tj) return;
  __shared__ __align__(16) float smem[kFmaStages * 2 * kFmaSlab];
  const int64_t row0 = int64_t(ti) * kFmaTile, col0 = int64_t(tj) * kFmaTile;
  const int group = threadIdx.x >> 6, tx = threadIdx.x & 7, ty = (threadIdx.x >> 3) & 7;

  // this thread's 16 bytes of each operand's slab
  const int lrow = threadIdx.x >> 3, lk = 4 * (threadIdx.x & 7);
  const bool liveA = row0 + lrow < fin.nr, liveB = col0 + lrow < fin.nc;
  const float *srcA = ZA + (liveA ? row0 + lrow : 0) * ldz + lk;
  const float *srcB = ZB + (liveB ? col0 + lrow : 0) * ldz + lk;
  const int nk = int(ldz / kFmaK);
  auto load = [&](int kb) {
    if (kb < nk) {
      float *d = smem + (kb % kFmaStages) * 2 * kFmaSlab + lrow * kFmaLd + lk;
      cp_async16(d, srcA + int64_t(kb) * kFmaK, liveA);
      cp_async16(d + kFmaSlab, srcB + int64_t(kb) * kFmaK, liveB);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < kFmaStages - 1; s++) load(s);

  float sum[4][4], acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) sum[i][j] = acc[i][j] = 0.f;
  for (int kb = 0; kb < nk; kb++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kFmaStages - 2) : "memory");
    __syncthreads();  // slab kb is in, and slab kb - 1 has been read
    load(kb + kFmaStages - 1);
    const float *pa = smem + (kb % kFmaStages) * 2 * kFmaSlab + ty * kFmaLd + 8 * group;
    const float *pb = pa + kFmaSlab + (tx - ty) * kFmaLd;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        a[i] = *reinterpret_cast<const float4 *>(pa + 8 * i * kFmaLd + h);
        b[i] = *reinterpret_cast<const float4 *>(pb + 8 * i * kFmaLd + h);
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
    if ((kb & 3) == 3 || kb + 1 == nk) {  // a run of up to 32 products ends
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          sum[i][j] += acc[i][j];
          acc[i][j] = 0.f;
        }
    }
  }

  // the groups' sums, then the tile, in shared memory
  constexpr int LD = kFmaTile + 1, PART = kFmaTile * LD;
  static_assert(5 * PART <= kFmaStages * 2 * kFmaSlab, "the sums and the tile fit the slabs");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
      smem[(1 + group) * PART + (ty + 8 * i) * LD + tx + 8 * j] = sum[i][j];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int rl = warp; rl < kFmaTile; rl += kFmaThreads / 32) {
    const float *p = smem + PART + rl * LD + lane;
    float v = clamp_r((p[0] + p[PART]) + (p[2 * PART] + p[3 * PART]));
    if (fin.symmetric && ti == tj && rl == lane && v == v) v = 1.f;
    smem[rl * LD + lane] = v;
  }
  __syncthreads();
  const bool mirror = fin.symmetric && ti != tj;
#pragma unroll 1
  for (int side = 0; side < (mirror ? 2 : 1); side++) {
    const int64_t r0 = side ? col0 : row0, c = (side ? row0 : col0) + lane;
    const int64_t nr = side ? fin.nc : fin.nr, nc = side ? fin.nr : fin.nc;
#pragma unroll
    for (int rl = warp; rl < kFmaTile; rl += kFmaThreads / 32) {
      if (r0 + rl >= nr || c >= nc) continue;
      const int64_t o = (r0 + rl) * fin.ld + c;
      fin.put(fin.corr + o, fin.ts + o, fin.pairs + o,
              side ? smem[lane * LD + rl] : smem[rl * LD + lane]);
    }
  }
}

}  // namespace

// Whether pearson_fma takes the problem.  Measured against the tensor-core Gram with
// its observations in pieces (us a call, here / there): 40 obs x 100 variables 23 /
// 31 (23 is the host's share), 700 x 400 25 / 32, 1000 x 300 23 / 31, 1500 x 250 31 /
// 31, 250 x 900 23 / 31, 100 x 1500 27 / 31, 2000 obs x 200 and 500 variables 37 / 43,
// 1500 x 20 and 4000 42 / 44; past the limits 1000 x 500 33 / 30, 400 x 1000 31 / 29,
// 4000 x 200 73 / 37 (a tile walks all observations), 100 x 1700 33 / 31 (outputs),
// 2500 x 50 and 2000 55 / 49.
// The relative error of r falls from 1.2e-7 .. 1.1e-6 to 0.2e-7 .. 1.5e-7.
bool pearson_fma_wins(int64_t nA, int64_t nB, int64_t n, int symmetric) {
  const double entries = double(nA) * double(nB);
  return n <= (symmetric ? 1500 : 2000) && entries <= 2.5e6 && entries * double(n) <= 2.4e8;
}

bool pearson_fma(const float *dA, int64_t nA, const float *dB, int64_t nB, int64_t n,
                 const PearsonOut &out, cudaStream_t s, int *status) {
  const int64_t ldz = cdiv(n, kFmaK) * kFmaK, nvar = nA + (out.symmetric ? 0 : nB);
  void *pz = nullptr;
  if (!ws_try(WS_SCRATCH0, size_t(nvar) * size_t(ldz) * 4, s, &pz)) return false;
  auto *Z = static_cast<float *>(pz);
  {
    ProfScope prof("pearson_prologue", s);
    pearson_norm_kernel<<<unsigned(cdiv(nvar, kFmaThreads / 32)), kFmaThreads, 0, s>>>(
        dA, nA, dB, nvar, n, ldz, Z);
    count_launch();
  }
  const PearsonFinish fin{out.corr, out.ts, out.pairs, out.ld, nA, nB, out.npairs,
                          std::sqrt(out.npairs - 2.f), 1.f, out.symmetric};
  const float *ZB = out.symmetric ? Z : Z + nA * ldz;
  ProfScope prof("pearson_gram", s);
  pearson_fma_kernel<<<unsigned(cdiv(nB, kFmaTile) * cdiv(nA, kFmaTile)), kFmaThreads, 0, s>>>(
      Z, ZB, ldz, fin);
  count_launch();
  *status = [&]() -> int {
    GT_CUDA(cudaGetLastError());
    return GT_OK;
  }();
  return true;
}

}  // namespace gt
