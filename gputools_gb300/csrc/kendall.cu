// kendall.cu -- gpuCor(method = "kendall"): tau-b from exact integer counts.
//
// Reference: src/kendall.cpp:13-55 masterKendall() launches
// inst/cuda/kendall.cu:4-47 gpuKendall, one 16x16 block per variable pair
// that loops over all observation pairs with float counters (exact only below
// 2^24) and reports (C - (T - C)) / T with joint ties counted as concordant,
// which is not R's cor(method = "kendall").
//
// Here the observation pairs are enumerated as (i, (i + d) mod n), d = 1 ..
// floor(n/2), i = 0 .. n-1 (for even n the row d = n/2 keeps only i < n/2),
// every unordered pair exactly once in rows of n.  With the pair's sign
//   s_v[p] = +1 where x_v[j] > x_v[i], -1 where they differ otherwise, 0 in a tie,
//   concordant - discordant = sum_p s_x[p] s_y[p],   untied = sum_p |s_x[p]|,
// so all counts are one Gram matrix of the sign rows.  One problem runs it on
// the tensor cores in FP8 (e4m3 holds -1, 0, 1 exactly, and FP32 sums of
// integers below 2^24 are exact); a batch counts on bit masks (below).
// tau-b = S / (sqrt(Tx) * sqrt(Ty)) is then evaluated in IEEE double with
// explicit round-to-nearest operations in R's order, clamped to [-1, 1]; NaN
// when either variable is constant; exactly 1 on the diagonal of cor(x).
#include "common.cuh"
#include "gram_core.cuh"
#include "kernels.cuh"
#include "tc_ptx.cuh"

#include <cmath>

namespace gt {

namespace {

constexpr int kKT = 256;        // threads per count CTA
constexpr int kKBK = 16;        // words per shared slab
constexpr int kKLd = 18;        // padded shared row, in words (uint2)

// Counts of one 64 x 64 tile of variable pairs over words [kbeg, kend):
// both[i][j] = popc(m), disc[i][j] = popc(m & (Gr ^ Gc)) with m = Ur & Uc,
// for rows row0 + ty + 16 i of MR and columns col0 + tx + 16 j of MC.
__device__ __forceinline__ void tile_counts(const uint2 *__restrict__ MR, int64_t nr,
                                            const uint2 *__restrict__ MC, int64_t nc, int64_t K,
                                            int64_t row0, int64_t col0, int64_t kbeg,
                                            int64_t kend, uint2 *sR, uint2 *sC,
                                            unsigned (&both)[4][4], unsigned (&disc)[4][4]) {
  constexpr int TM = 4, TN = 4;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) both[i][j] = disc[i][j] = 0u;
  for (int64_t k0 = kbeg; k0 < kend; k0 += kKBK) {
    // 64 rows x 16 words = 512 uint4 (two words each) per operand.
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const int q = threadIdx.x + s * kKT;
      const int row = q >> 3, c2 = q & 7;
      const int64_t gk = k0 + 2 * c2;
      uint4 vr = make_uint4(0u, 0u, 0u, 0u), vc = make_uint4(0u, 0u, 0u, 0u);
      const int64_t gr = row0 + row, gc = col0 + row;
      if (gr < nr) {
        if (gk < kend) { const uint2 w = MR[gr * K + gk]; vr.x = w.x; vr.y = w.y; }
        if (gk + 1 < kend) { const uint2 w = MR[gr * K + gk + 1]; vr.z = w.x; vr.w = w.y; }
      }
      if (gc < nc) {
        if (gk < kend) { const uint2 w = MC[gc * K + gk]; vc.x = w.x; vc.y = w.y; }
        if (gk + 1 < kend) { const uint2 w = MC[gc * K + gk + 1]; vc.z = w.x; vc.w = w.y; }
      }
      *reinterpret_cast<uint4 *>(&sR[row * kKLd + 2 * c2]) = vr;
      *reinterpret_cast<uint4 *>(&sC[row * kKLd + 2 * c2]) = vc;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kKBK / 2; kk++) {
      uint4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; i++)
        a[i] = *reinterpret_cast<const uint4 *>(&sR[(ty + 16 * i) * kKLd + 2 * kk]);
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const uint4 b = *reinterpret_cast<const uint4 *>(&sC[(tx + 16 * j) * kKLd + 2 * kk]);
#pragma unroll
        for (int i = 0; i < TM; i++) {
          const unsigned m0 = a[i].x & b.x, m1 = a[i].z & b.z;
          both[i][j] += __popc(m0) + __popc(m1);
          disc[i][j] += __popc(m0 & (a[i].y ^ b.y)) + __popc(m1 & (a[i].w ^ b.w));
        }
      }
    }
    __syncthreads();
  }
}

// tau-b = S / (sqrt(Tx) * sqrt(Ty)) in IEEE double, R's evaluation order,
// clamped to [-1, 1]; NaN when either variable is constant.  rx = sqrt(Tx)
// and ry = sqrt(Ty) (__dsqrt_rn) are taken once per variable.
// The zero tests and the clamp work on the bit patterns: FP64 instructions
// run at 1/64 of the integer rate and bound the pass that calls this.
__device__ __forceinline__ double taub(long long S, double rx, double ry) {
  constexpr long long kOne = 0x3ff0000000000000LL;
  if (__double_as_longlong(rx) == 0 || __double_as_longlong(ry) == 0)
    return __longlong_as_double(0x7ff8000000000000LL);
  const long long b = __double_as_longlong(__ddiv_rn(double(S), __dmul_rn(rx, ry)));
  const long long m = b & 0x7fffffffffffffffLL;
  return __longlong_as_double(m > kOne ? (b ^ m) | kOne : b);
}

constexpr int kSgThreads = 256;
constexpr int kSgRows = 32;  // pair rows a thread walks

// The launch shape of the sign pass.  A row of n observations is n4 bytes (n
// rounded up to 4), 4 per thread: `lanes` threads share a row segment (of
// `segs`), and `groups` of them take different pair rows, `dper` each.
struct SignPlan {
  int64_t n, n4, kpad, rows;  // rows of n4 bytes that cover kpad
  int lanes, segs, groups, dper;
  int64_t dblocks;
};

SignPlan make_sign_plan(int64_t n, int64_t drows) {
  SignPlan p;
  p.n = n;
  p.n4 = cdiv(n, 4) * 4;
  p.kpad = cdiv(drows * p.n4, 128) * 128;
  p.rows = cdiv(p.kpad, p.n4);
  const int64_t L = p.n4 / 4;
  p.lanes = int(L < kSgThreads ? L : kSgThreads);
  p.segs = int(cdiv(L, p.lanes));
  int64_t g = kSgThreads / p.lanes;
  p.groups = int(g > 32 ? 32 : g);
  const int64_t per = cdiv(cdiv(p.rows, p.groups), 4) * 4;
  p.dper = int(per < kSgRows ? per : kSgRows);
  p.dblocks = cdiv(p.rows, int64_t(p.groups) * p.dper);
  return p;
}

size_t sign_smem(const SignPlan &p) {
  return (size_t(p.lanes) + size_t(p.groups) * size_t(p.dper) / 4 + 2) * 16;
}

// The sign rows of pair rows d0 + 1 .. d0 + drows: variable v's row d holds
// n4 bytes (e4m3 +1 = 0x38, -1 = 0xb8, 0) at P[v * kpad + (d - d0 - 1) * n4],
// zero up to kpad; untied counts are added to T.  A block takes one variable,
// one row segment and groups * dper pair rows.  Each thread keeps its four
// x[i] in registers and slides a window of four x[i + d] along: one shared
// read per four signs, conflict-free because the window is stored by its
// index modulo 4.  Bound by the compares and selects of the ALU pipe (87 %
// busy); 500 x 1000: 61 us for 125 MB of signs.
__global__ void __launch_bounds__(kSgThreads)
kendall_signs_kernel(const float *__restrict__ X, int64_t nx, const float *__restrict__ Y,
                     SignPlan p, int64_t d0, int64_t drows, uint8_t *__restrict__ P,
                     unsigned *__restrict__ T) {
  extern __shared__ float win[];  // [4][quads]
  const int64_t units = int64_t(p.segs) * p.dblocks;
  const int64_t v = int64_t(blockIdx.x) / units;
  const int64_t u = int64_t(blockIdx.x) - v * units;
  const int64_t db = u / p.segs;
  const int64_t i0 = (u - db * p.segs) * (4 * int64_t(p.lanes));
  const int64_t rlo = db * (int64_t(p.groups) * p.dper);
  const float *x = v < nx ? X + v * p.n : Y + (v - nx) * p.n;
  const int quads = p.lanes + p.groups * p.dper / 4 + 2;
  for (int o = threadIdx.x; o < 4 * quads; o += kSgThreads) {
    int64_t j = i0 + d0 + rlo + 1 + o;  // the window starts at x[i0 + first d]
    if (j >= p.n) j -= p.n;
    win[(o & 3) * quads + (o >> 2)] = j < p.n ? x[j] : 0.f;
  }
  const int g = threadIdx.x / p.lanes, l = threadIdx.x - g * p.lanes;
  const int64_t i = i0 + 4 * int64_t(l);
  float xi[4];
  uint32_t full = 0, half = 0;  // bytes with i + e < n and, for d = n / 2, i + e < n / 2
#pragma unroll
  for (int e = 0; e < 4; e++) {
    xi[e] = i + e < p.n ? x[i + e] : 0.f;
    if (i + e < p.n) full |= 0xffu << (8 * e);
    if (i + e < p.n / 2) half |= 0xffu << (8 * e);
  }
  __syncthreads();
  unsigned untied = 0;
  if (g < p.groups && i < p.n4) {
    const int r0 = g * p.dper;  // multiple of 4
    const float *q = win + l + r0 / 4;
    float w[4] = {q[0], q[quads], q[2 * quads], q[3 * quads]};
    const int64_t row = rlo + r0, d = d0 + row + 1;  // the thread's first row
    uint8_t *dst = P + v * p.kpad + row * p.n4 + i;
    // four signs of the row k steps on, then the window's next value
    auto signs = [&](int k, const float *qn) {
      uint32_t word = 0;
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float xj = w[(k + e) & 3];
        if (xj != xi[e]) word |= 0xb8u << (8 * e);
        if (xj > xi[e]) word ^= 0x80u << (8 * e);
      }
      w[k] = qn[k * quads];
      return word;
    };
    const int step = int(p.n4);
    // rows that all lie inside the pass, below d = n / 2 and below kpad (an
    // unmasked byte past n is masked by `full`)
    if (row + p.dper <= drows && 2 * (d + p.dper - 1) < p.n) {
#pragma unroll 1
      for (int rr = 0; rr < p.dper; rr += 4) {
        q++;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t word = signs(k, q) & full;
          untied += __popc(word & 0x08080808u);
          *reinterpret_cast<uint32_t *>(dst) = word;
          dst += step;
        }
      }
    } else {
      const int64_t left = p.kpad - row * p.n4 - i;  // bytes to the end of the row buffer
#pragma unroll 1
      for (int rr = 0; rr < p.dper; rr += 4) {
        q++;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t word =
              signs(k, q) & (row + rr + k >= drows ? 0u : (2 * (d + rr + k) < p.n ? full : half));
          untied += __popc(word & 0x08080808u);
          if (int64_t(rr + k) * step < left) *reinterpret_cast<uint32_t *>(dst) = word;
          dst += step;
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) untied += __shfl_xor_sync(0xffffffffu, untied, o);
  if ((threadIdx.x & 31) == 0 && untied) atomicAdd(&T[v], untied);
}

// S += the Gram matrix of the sign rows (r of MA, c of MB) over pieces of
// 128-byte k-blocks, on tcgen05 (kind::f8f6f4).  A block computes one 128 x
// 256 tile over one piece of K: warp 0 loads (TMA, 128-byte swizzle), warp 1
// issues the MMAs (M = 128, N = 256, K = 32), warps 2..5 add the exact sums
// to S as integers, S[c * nr + r] so that a warp's 32 rows are one line.  Two
// stages of 48 KB and 256 TMEM columns a block: two blocks share an SM, one's
// fill and drain run under the other's MMAs, and no block stays resident.
// Every wait is bounded; a block that gives up sets the device error word,
// drains its copies and MMAs, and frees its TMEM.
// Bound by shared memory (an MMA reads 12 KB and its stage writes 12 KB per 128
// tensor-core cycles).  500 x 1000: 59 us, 2.8 PFLOP/s; the popcounts on
// CUDA cores that it replaced took 1.10 ms, their masks 0.21 ms.
constexpr int kSgBK = 128;                  // signs per stage
constexpr int kSgStages = 2;
constexpr int kSgATile = kBM * kSgBK, kSgBTile = kBN * kSgBK;
constexpr int kSgStage = kSgATile + kSgBTile;
constexpr int kSgGramThreads = 192;
constexpr int kSgGramSmem = kSgStages * kSgStage + 1024 + 256;
// FP32 holds every integer up to 2^24: at most so many signs per sum.
constexpr int64_t kSgMaxBlocks = (int64_t(1) << 24) / kSgBK;

__global__ void __launch_bounds__(kSgGramThreads, 2)
kendall_gram_kernel(const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                    TileSpace ts, int64_t kblocks, int64_t per, int64_t nr, int64_t nc,
                    int *__restrict__ S, const tc::WaitCfg wc) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~uintptr_t(1023));
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + kSgStages * kSgStage);
  uint64_t *empty = full + kSgStages;
  uint64_t *done = empty + kSgStages;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSgStages; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(done, 1);
    *abort_flag = 0;
    tc::fence_barrier_init();
    tc::prefetch_tensormap(&ma);
    tc::prefetch_tensormap(&mb);
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, kBN);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // piece-major: blocks that run together share a stretch of every operand row
  const int64_t piece = int64_t(blockIdx.x) / ts.ntiles;
  int64_t ti, tj;
  tile_coords(ts, int64_t(blockIdx.x) - piece * ts.ntiles, ti, tj);
  const int64_t row0 = ti * kBM, col0 = tj * kBN;
  const int64_t kb0 = piece * per;
  const int nk = int(kblocks - kb0 < per ? kblocks - kb0 : per);

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (; it < nk; it++) {
        const int s = it % kSgStages;
        if (!tc::mbar_wait(&empty[s], uint32_t((it / kSgStages) & 1) ^ 1u, abort_flag, wc)) {
          *abort_flag = 1;
          break;
        }
        uint8_t *st = smem + s * kSgStage;
        tc::mbar_arrive_expect_tx(&full[s], kSgStage);
        const int32_t k = int32_t((kb0 + it) * kSgBK);
        tc::tma_load_3d(st, &ma, &full[s], k, int32_t(row0), 0);
        tc::tma_load_3d(st + kSgATile, &mb, &full[s], k, int32_t(col0), 0);
      }
      // no bulk copy may still be writing shared memory at exit, should another warp
      // give up later
      for (int s = 0; s < kSgStages; s++) {
        const int fills = it / kSgStages + (s < it % kSgStages ? 1 : 0);
        if (fills > 0) tc::mbar_wait_bounded(&full[s], uint32_t((fills - 1) & 1), kDrainLimitNs);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the whole warp walks the loop (descriptors in uniform registers), one lane issues
    constexpr uint32_t idesc = tc::idesc_e4m3_f32acc(kBM, kBN);
    const bool lead = tc::elect_one();
    bool ok = true;
    for (int it = 0; it < nk; it++) {
      const int s = it % kSgStages;
      ok = __all_sync(0xffffffffu, tc::mbar_wait(&full[s], uint32_t((it / kSgStages) & 1),
                                                 abort_flag, wc));
      if (!ok) break;
      tc::tc_fence_after();
      const uint32_t sa = tc::smem_u32(smem + s * kSgStage), sb = sa + kSgATile;
      if (lead) {
#pragma unroll
        for (int k = 0; k < kSgBK / 32; k++)
          tc::umma_f8(tmem, tc::smem_desc_kmajor(sa + k * 32, 128),
                      tc::smem_desc_kmajor(sb + k * 32, 128), idesc, it == 0 && k == 0 ? 0u : 1u);
        tc::umma_commit(&empty[s]);
      }
      __syncwarp();
    }
    if (!ok) *abort_flag = 1;
    // every MMA issued above has finished before the sums are read and TMEM is released
    // (waited for here too: an epilogue warp may have given up while this one had not)
    if (lead) {
      tc::umma_commit(done);
      tc::mbar_wait_bounded(done, 0u, kDrainLimitNs);
    }
    __syncwarp();
  } else {
    const int q = warp & 3;  // TMEM lane quarter
    const int64_t r = row0 + q * 32 + lane;
    const bool got = tc::mbar_wait(done, 0u, abort_flag, wc);
    if (!got) *abort_flag = 1;
    if (__all_sync(0xffffffffu, got) && !*abort_flag) {
      tc::tc_fence_after();
      for (int c8 = 0; c8 < kBN / 32; c8++) {
        const int64_t c0 = col0 + 32 * c8;
        if (c0 >= nc || (ts.symmetric == kUpper && c0 + 31 < row0 + q * 32)) continue;
        float g[32];
        tc::tmem_ld32(tmem + uint32_t(32 * c8) + (uint32_t(q * 32) << 16), g);
        int *dst = S + c0 * nr + r;
#pragma unroll
        for (int j = 0; j < 32; j++)
          if (r < nr && c0 + j < nc) atomicAdd(dst + j * nr, __float2int_rn(g[j]));
      }
    }
    tc::tc_fence_before();
  }
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) atomicOr(wc.err, 1);
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, kBN);
  }
}

// out[r * nx + c] = tau-b of (Y_r, X_c) from S[c * ny + r], 32 x 32 entries a
// block; a symmetric problem (S valid for r <= c) takes the blocks on and
// above the diagonal and writes both entries, so each FP64 division is made
// once (they bound this pass).
__global__ void __launch_bounds__(256)
kendall_finish_kernel(const int *__restrict__ S, const unsigned *__restrict__ TX,
                      const unsigned *__restrict__ TY, int64_t nx, int64_t ny, int same,
                      double *__restrict__ out) {
  __shared__ double tile[32][33];  // [c][r]
  __shared__ double rx[32], ry[32];
  const int64_t c0 = int64_t(blockIdx.x) * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int64_t br = blockIdx.y; br * 32 < ny; br += gridDim.y) {
    const int64_t r0 = br * 32;
    if (same && r0 > c0) return;
    if (ty == 0 && c0 + tx < nx) rx[tx] = __dsqrt_rn(double(TX[c0 + tx]));
    if (ty == 1 && r0 + tx < ny) ry[tx] = __dsqrt_rn(double(TY[r0 + tx]));
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int cl = ty + 8 * k;
      const int64_t r = r0 + tx, c = c0 + cl;
      if (r >= ny || c >= nx || (same && r > c)) continue;
      const double t = (same && r == c) ? 1.0 : taub(S[c * ny + r], rx[cl], ry[tx]);
      tile[cl][tx] = t;
      if (same && r0 != c0) out[c * nx + r] = t;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int rl = ty + 8 * k;
      const int64_t r = r0 + rl, c = c0 + tx;
      if (r < ny && c < nx) out[r * nx + c] = same && r > c ? tile[rl][tx] : tile[tx][rl];
    }
    __syncthreads();
  }
}

// Tensor map of the sign rows: [variable][kpad] bytes, box 128 bytes x rows.
int sign_map(CUtensorMap *map, const uint8_t *base, int64_t nvar, int64_t kpad, int box_rows) {
  const cuuint64_t dims[3] = {cuuint64_t(kpad), cuuint64_t(nvar), 1};
  const cuuint64_t strides[2] = {cuuint64_t(kpad), cuuint64_t(kpad) * cuuint64_t(nvar)};
  const cuuint32_t box[3] = {kSgBK, cuuint32_t(box_rows), 1};
  return tc_map_3d(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, base, dims, strides, box,
                   CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace

int kendall_impl(const float *dX, int64_t nx, const float *dY, int64_t ny, int64_t n, int same,
                 double *d_out, cudaStream_t s) {
  if (nx == 0 || ny == 0) return GT_OK;
  const int64_t Dr = n / 2;  // pair rows
  const int64_t nvar = same ? nx : nx + ny;
  if (cdiv(ny, 64) > 65535 || cdiv(nx, 64) > 2147483647LL)
    return fail(GT_EINVAL, "too many variables");
  // pair rows per pass: at most 2 GB of signs
  const int64_t per_row = nvar * cdiv(n, 4) * 4;
  int64_t rows_chunk = per_row > 0 ? (int64_t(2) << 30) / per_row : Dr;
  if (rows_chunk < 1) rows_chunk = 1;
  if (rows_chunk > Dr) rows_chunk = Dr;

  // the integer sums, then the untied counts
  void *pS = nullptr;
  const size_t bytes = (size_t(nx) * size_t(ny) + size_t(nvar)) * 4;
  GT_TRY(ws_get(WS_SCRATCH0, bytes, &pS));
  int *S = static_cast<int *>(pS);
  auto *TX = reinterpret_cast<unsigned *>(S + nx * ny);
  unsigned *TY = same ? TX : TX + nx;
  GT_CUDA(cudaMemsetAsync(S, 0, bytes, s));

  if (Dr > 0) {
    // ... or as many as the device has room for (four times the bytes of the bit masks
    // that batches count)
    void *pP = nullptr;
    while (rows_chunk > 1 &&
           !ws_try(WS_SCRATCH2, size_t(nvar) * size_t(make_sign_plan(n, rows_chunk).kpad), s, &pP))
      rows_chunk = cdiv(rows_chunk, 2);
    if (!pP) GT_TRY(ws_get(WS_SCRATCH2, size_t(nvar) * size_t(make_sign_plan(n, 1).kpad), &pP));
    auto *P = static_cast<uint8_t *>(pP);
    tc::WaitCfg wc;
    GT_TRY(make_wait_cfg(&wc));
    GT_CUDA(cudaFuncSetAttribute(kendall_gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kSgGramSmem));
    for (int64_t d0 = 0; d0 < Dr; d0 += rows_chunk) {
      const int64_t dr = Dr - d0 < rows_chunk ? Dr - d0 : rows_chunk;
      const SignPlan sp = make_sign_plan(n, dr);
      const int64_t sblocks = nvar * sp.segs * sp.dblocks;
      if (sblocks > 2147483647LL) return fail(GT_EINVAL, "too many variables");
      kendall_signs_kernel<<<unsigned(sblocks), kSgThreads, sign_smem(sp), s>>>(dX, nx, dY, sp, d0,
                                                                               dr, P, TX);
      CUtensorMap ma, mb;
      GT_TRY(sign_map(&ma, same ? P : P + nx * sp.kpad, ny, sp.kpad, kBM));
      GT_TRY(sign_map(&mb, P, nx, sp.kpad, kBN));
      const int64_t kblocks = sp.kpad / kSgBK;
      TileSpace ts = make_tiles(ny, nx, same ? kUpper : kFull, 8);
      // pieces of K: enough blocks for two per SM, each piece at least 8
      // k-blocks (a block's start and its sums cost about as much) and short
      // enough for exact sums
      int64_t pieces = 2 * int64_t(sm_count()) / ts.ntiles;
      if (pieces > kblocks / 8) pieces = kblocks / 8;
      if (pieces < 1) pieces = 1;
      int64_t per = cdiv(kblocks, pieces);
      if (per > kSgMaxBlocks) per = kSgMaxBlocks;
      pieces = cdiv(kblocks, per);
      if (ts.ntiles * pieces > 2147483647LL) return fail(GT_EINVAL, "too many variables");
      ProfScope prof("kendall_count", s);
      kendall_gram_kernel<<<unsigned(ts.ntiles * pieces), kSgGramThreads, kSgGramSmem, s>>>(
          ma, mb, ts, kblocks, per, ny, nx, S, wc);
      count_launch(2);
      GT_CUDA(cudaGetLastError());
    }
  }
  const int64_t gy = cdiv(ny, 32);
  kendall_finish_kernel<<<dim3(unsigned(cdiv(nx, 32)), unsigned(gy < 65535 ? gy : 65535)), 256, 0,
                          s>>>(S, TX, TY, nx, ny, same, d_out);
  count_launch();
  GT_CUDA(cudaGetLastError());
  return GT_OK;
}

// ---------------------------------------------------------------- batches
// Many independent Kendall problems in one pass: one CTA per variable builds
// its pair masks and untied count; one count launch walks per-CTA lists of
// 64 x 64 tiles (balanced on the host) across all problems and writes tau-b
// directly (each tile covers its problem's full pair dimension).

namespace {

constexpr int kKbMaskThreads = 128;
constexpr int kKbStage = 4096;  // observations staged in shared memory (16 KB)

// One CTA per variable of the batch: warps take chunks of 32 consecutive
// words (lane e keeps word e, one coalesced store per chunk), reading the
// observations from shared memory when they fit; the untied count is the
// CTA's sum.  The same words and counts either way.
__global__ void __launch_bounds__(kKbMaskThreads)
kendall_batch_masks_kernel(const KendallBatchProblem *__restrict__ P,
                           const int64_t *__restrict__ var_prefix, int64_t nprob,
                           uint2 *__restrict__ M, unsigned long long *__restrict__ T,
                           double *__restrict__ root) {
  __shared__ unsigned long long part[kKbMaskThreads / 32];
  __shared__ float xs[kKbStage];
  const int64_t gv = blockIdx.x;
  const int64_t pi = find_segment(var_prefix, nprob, gv);
  const KendallBatchProblem pr = P[pi];
  const int64_t v = gv - var_prefix[pi];
  const float *x = pr.X + v * pr.n;
  uint2 *mv = M + pr.mask_off + v * pr.K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool staged = pr.n <= kKbStage;  // CTA-uniform
  if (staged) {
    for (int64_t k = threadIdx.x; k < pr.n; k += kKbMaskThreads) xs[k] = x[k];
    __syncthreads();
  }
  const int64_t n = pr.n, Wn = pr.Wn, K = pr.K;
  unsigned long long cnt = 0;
  auto words = [&](auto rd) {
    for (int64_t base = 32 * int64_t(warp); base < K; base += 32 * (kKbMaskThreads / 32)) {
      const int m = K - base < 32 ? int(K - base) : 32;
      int64_t dr = base / Wn, w = base - dr * Wn;
      uint2 mine = make_uint2(0u, 0u);
      for (int e = 0; e < m; e++) {  // warp-uniform
        const int64_t d = dr + 1, i = 32 * w + lane;
        bool untied = false, greater = false;
        if (i < n && (2 * d < n || i < n / 2)) {
          int64_t j = i + d;
          if (j >= n) j -= n;
          const float xi = rd(i), xj = rd(j);
          untied = xj != xi;
          greater = xj > xi;
        }
        const unsigned u = __ballot_sync(0xffffffffu, untied);
        const unsigned g = __ballot_sync(0xffffffffu, greater);
        if (lane == e) mine = make_uint2(u, g);
        cnt += __popc(u);
        if (++w == Wn) {
          w = 0;
          dr++;
        }
      }
      if (lane < m) mv[base + lane] = mine;
    }
  };
  if (staged) words([&](int64_t k) { return xs[k]; });
  else words([&](int64_t k) { return x[k]; });
  if (lane == 0) part[warp] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tot = 0;
    for (int q = 0; q < kKbMaskThreads / 32; q++) tot += part[q];
    T[pr.var_off + v] = tot;
    root[pr.var_off + v] = __dsqrt_rn(double(tot));
  }
}

__global__ void __launch_bounds__(kKT)
kendall_batch_count_kernel(const KendallBatchProblem *__restrict__ P,
                           const int64_t *__restrict__ tile_prefix, int64_t nprob,
                           const int64_t *__restrict__ cta_tiles,
                           const int64_t *__restrict__ cta_off, const uint2 *__restrict__ M,
                           const double *__restrict__ root) {
  __shared__ __align__(16) uint2 sR[64 * kKLd];
  __shared__ __align__(16) uint2 sC[64 * kKLd];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int64_t idx = cta_off[blockIdx.x]; idx < cta_off[blockIdx.x + 1]; idx++) {
    const int64_t gtile = cta_tiles[idx];
    const int64_t pi = find_segment(tile_prefix, nprob, gtile);
    const KendallBatchProblem pr = P[pi];
    const int64_t lt = gtile - tile_prefix[pi];
    int64_t tj = int64_t((sqrt(8.0 * double(lt) + 1.0) - 1.0) * 0.5);
    while ((tj + 1) * (tj + 2) / 2 <= lt) tj++;
    while (tj * (tj + 1) / 2 > lt) tj--;
    const int64_t ti = lt - tj * (tj + 1) / 2;  // ti <= tj
    const uint2 *Mp = M + pr.mask_off;
    unsigned both[4][4], disc[4][4];
    const int64_t row0 = ti * 64, col0 = tj * 64;
    tile_counts(Mp, pr.p, Mp, pr.p, pr.K, row0, col0, 0, pr.K, sR, sC, both, disc);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int64_t r = row0 + ty + 16 * i;
      if (r >= pr.p) continue;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int64_t c = col0 + tx + 16 * j;
        if (c >= pr.p) continue;
        const long long sv = (long long)both[i][j] - 2LL * (long long)disc[i][j];
        const double tau =
            (r == c) ? 1.0 : taub(sv, root[pr.var_off + c], root[pr.var_off + r]);
        pr.out[r * pr.p + c] = tau;
        if (ti != tj) pr.out[c * pr.p + r] = tau;
      }
    }
  }
}

}  // namespace

int kendall_batch_launch(const KendallBatchProblem *d_probs, const int64_t *d_var_prefix,
                         int64_t nprob, int64_t total_vars, const int64_t *d_tile_prefix,
                         const int64_t *d_cta_tiles, const int64_t *d_cta_off, int64_t ncta,
                         uint2 *d_masks, unsigned long long *d_T, cudaStream_t s) {
  // d_T holds the untied counts of all variables, then their square roots
  double *root = reinterpret_cast<double *>(d_T + total_vars);
  if (total_vars > 0) {
    kendall_batch_masks_kernel<<<unsigned(total_vars), kKbMaskThreads, 0, s>>>(
        d_probs, d_var_prefix, nprob, d_masks, d_T, root);
    count_launch();
  }
  if (ncta > 0) {
    kendall_batch_count_kernel<<<unsigned(ncta), kKT, 0, s>>>(d_probs, d_tile_prefix, nprob,
                                                             d_cta_tiles, d_cta_off, d_masks, root);
    count_launch();
  }
  GT_CUDA(cudaGetLastError());
  return GT_OK;
}

int kendall_check(int64_t nx, int64_t ny, int64_t n) {
  if (nx < 0 || ny < 0 || n < 0) return fail(GT_EINVAL, "negative size");
  if (n > 65536) return fail(GT_EINVAL, "kendall supports at most 65536 observations (n=%lld)",
                             (long long)n);
  return GT_OK;
}

int same_contents(const float *a, const float *b, int64_t count, bool *same, cudaStream_t s);

}  // namespace gt

extern "C" int gt_kendall_device(const float *d_X, int64_t nx, const float *d_Y, int64_t ny,
                                 int64_t n, double *d_out, void *stream) {
  gt::clear_error();
  GT_TRY(gt::kendall_check(nx, ny, n));
  if ((nx > 0 && !d_X) || (ny > 0 && !d_Y) || (nx * ny > 0 && !d_out))
    return gt::fail(GT_EINVAL, "null device pointer");
  const int same = (d_X == d_Y && nx == ny) ? 1 : 0;
  return gt::kendall_impl(d_X, nx, d_Y, ny, n, same, d_out, static_cast<cudaStream_t>(stream));
}

extern "C" int gt_kendall(const float *X, int64_t nx, const float *Y, int64_t ny, int64_t n,
                          double *out) {
  gt::clear_error();
  GT_TRY(gt::kendall_check(nx, ny, n));
  if (nx == 0 || ny == 0) return GT_OK;
  if (!X || !Y || !out) return gt::fail(GT_EINVAL, "null host pointer");
  cudaStream_t s = gt::lib_stream();
  gt::StreamSyncGuard guard(s);
  const size_t bx = size_t(nx) * size_t(n) * 4, by = size_t(ny) * size_t(n) * 4;
  void *dX = nullptr, *dY = nullptr, *dO = nullptr;
  GT_TRY(gt::ws_get(gt::WS_IN_A, bx, &dX));
  GT_CUDA(cudaMemcpyAsync(dX, X, bx, cudaMemcpyHostToDevice, s));
  bool same = (X == Y && nx == ny);
  if (!same) {
    GT_TRY(gt::ws_get(gt::WS_IN_B, by, &dY));
    GT_CUDA(cudaMemcpyAsync(dY, Y, by, cudaMemcpyHostToDevice, s));
    if (nx == ny)
      GT_TRY(gt::same_contents(static_cast<float *>(dX), static_cast<float *>(dY), nx * n, &same, s));
  }
  if (same) dY = dX;
  void *direct = gt::host_output_ptr(out, size_t(nx) * size_t(ny) * 8);
  if (!(dO = direct)) GT_TRY(gt::ws_get(gt::WS_OUT0, size_t(nx) * size_t(ny) * 8, &dO));
  GT_TRY(gt::kendall_impl(static_cast<float *>(dX), nx, static_cast<float *>(dY), ny, n,
                          same ? 1 : 0, static_cast<double *>(dO), s));
  if (!direct)
    GT_CUDA(cudaMemcpyAsync(out, dO, size_t(nx) * size_t(ny) * 8, cudaMemcpyDeviceToHost, s));
  GT_CUDA(cudaStreamSynchronize(s));
  bool failed = false;
  GT_TRY(gt::device_error_check(s, &failed));
  if (failed) return gt::fail(GT_ETIMEOUT, "a tensor-core kernel wait timed out");
  return GT_OK;
}
