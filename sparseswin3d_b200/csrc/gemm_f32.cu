// fp32 GEMM of the Linear layers: out[M, N] = a[M, K] w[N, K]^T (+ bias), on the fifth-generation tensor cores
// with the operands split into three bf16 terms each.
//
// x = h + m + l with h = bf16(x), m = bf16(x - h), l = bf16(x - h - m) holds all 24 bits of x (below about 2^-109 the last
// of them fall under the smallest bf16).  Six of the nine
// products are formed (h h, h m, m h, m m, h l, l h); the three left out are below 2^-25 of a term.  The tensor
// cores add up in fp32 but cut off instead of rounding, so the sums are kept short: the h h products of 64 steps
// of K go into a tensor-memory accumulator of their own, which the epilogue threads add up in registers, rounding
// to nearest; the five small products (2^-8 and below) share one accumulator for the whole of K.
// Against 64 bits (2-norm, normal operands): 7e-8 at K = 96, 8e-8 at 192, 1.0e-7 at 768, where the library's fp32 GEMM is
// at 1.8e-7, 2.5e-7 and 5.0e-7; all-positive operands 8.2e-8, 9.5e-8, 1.0e-7 against 1.5e-7, 2.1e-7, 4.1e-7.  Weight
// gradients of 150 000 rows: 2.0e-7 against 1.3e-6, all-positive 6e-8 against 2.1e-7 (with 64 steps a chunk 2.0e-7 against
// the library's 1.5e-7 at 96 x 96, hence one stage a chunk there).
//
// Weight gradients, out[N, K] = g[M, N]^T x[M, K] (TN): the operands' rows are then the steps of the sum, and the sum over M is split
// over blocks (partial results, added up in order by k_gemm_reduce).
//
// An Inf operand has no finite remainder (Inf - Inf), so a result that is not finite is formed again from the
// operands as they are, by plain fp32 multiply-adds, up to the first NaN; of a weight gradient only the row ranges whose partial
// result is not finite.  150 000 x 288 x 96, single calls: finite 82 us, one row of Inf 94, of NaN 91, all NaN 927 (library 461); its weight gradient
// 103, with one row (number 777) of Inf 479, of NaN 202, all NaN 98 (371).  Of the earlier form of the kernel: walked to the end 6060, over all rows by
// one thread 19 300.
//
// out = a w^T: persistent, one block per SM, 21 warps: eight bring fp32 pieces in three stages (32 of K) ahead, split them and store the terms
// of a in tensor memory (a thread is a row there) and those of w as 64-byte-swizzled tiles in shared memory; one issues the MMAs; twelve drain
// accumulators (a warp may read the 32 tensor-memory lanes warp_id % 4 selects; three warps share them, 32 columns each).  Up to K = 192 a block keeps
// to one tile of columns, whose w it splits once.  What bounds it: the latency of a producer warp's chain per stage (copies, split,
// stores: 0.95 us a stage, 40 % of the issue slots).  Steps, us at 150 000 x 288 x 96 with bias: 102; MMAs from uniform registers (see the issuer)
// 96; w kept 91 (shared memory was 84 % busy, a third of it the tensor cores' reads of a); a in tensor memory 79; twelve drain warps for
// eight 72; loads before the split 71.  The same sizes: 150 000 x 96 x 288 76 -> 70, 150 000 x 96 x 96 41 -> 31, 10 000 x 768 x 192 39 -> 31,
// 10 000 x 192 x 768 49 -> 39, 10 000 x 192 x 192 20 -> 16, 128 x 576 x 192 14 -> 10; the library's fp32 GEMM 447, 271, 153, 99, 81, 34, 15.
//
// Weight gradients the same way (a producer thread is a column of g; see k_gemm_f32_tn), 20 warps, with the partial results added up 150 000 rows 288 x 96
// 91 us (library 358), 96 x 96 56 (208), 10 000 rows 576 x 192 32 (111), 192 x 768 42.  With both operands in shared memory, split by eight warps,
// 138, 65, 44 and 58.
#include <math.h>

#include "attn_common.cuh"
#include "tcgen05.cuh"

namespace ssw {

constexpr int kGM = 128;                 // rows of a tile
constexpr int kGNMax = 96;              // columns of a tile at most (tensor memory holds four accumulators and the stages of a)
constexpr int kGK = 32;                  // K of a stage
constexpr int kGRowB = kGK * 2;          // bytes of an operand row: one 64-byte swizzle row
// Stages whose h h products share an accumulator: two, and one for the long sums of a weight gradient.
template <bool TN>
struct GemmChunk { static constexpr int kStages = TN ? 1 : 2; };
constexpr int kGProd = 8, kGEpi = 8;     // warps
constexpr int kGOpWB = kGNMax * kGRowB;  // ... of w
constexpr int kGTmemLow = 2 * kGNMax;    // two h h accumulators, then two of small products
constexpr int kGBiasOff = 1024, kGBiasB = kGEpi * (kGNMax / 2) * 4, kGFirst = 3072;   // the first operand tile: 1024-byte aligned
static_assert(kGBiasOff + kGBiasB <= kGFirst, "");

// out = a w^T: a in tensor memory, behind the accumulators, in two stages (h, m, l: 16 columns each); raw pieces of a warp and stage 2 KB.
constexpr int kNEpi = 12, kNThreads = 32 * (kGProd + 1 + kNEpi);
constexpr int kNRing = 2, kNTmemA = 4 * kGNMax, kNStageCols = 48;
constexpr int kNRaws = 4, kNRawWarp = 32 * 64, kNRawStage = kGProd * kNRawWarp, kNRawW = 3 * 4096;
static_assert(kNTmemA + kNRing * kNStageCols <= 512 && kGNMax <= 96, "");
// Weight gradients: eight warps for g, three for x (its 96 columns by fours and 32 rows by eights; 20 warps in all leave 96 registers a thread).
constexpr int kTProd = kGProd + 3, kTThreads = 32 * (kTProd + 1 + kGEpi);
constexpr int kTRawRow = 96 * 16, kTRawX = 8 * kTRawRow, kTRawOff = kGFirst + 4 * 3 * kGOpWB, kTSmem = kTRawOff + kNRaws * (kNRawStage + kTRawX) + 1024;
static_assert(kTSmem <= 227 * 1024, "");
struct GemmBars { uint64_t *hh_full, *hh_empty, *lo_full, *lo_empty; };

struct GemmParams {
  const float *a, *w, *bias;
  float* out;
  int gelu;               // the results go through GELU (erf form)
  int wide;               // rows of out start on 32-byte boundaries
  int64_t M;
  int N, K;
  int bn, n_tiles;        // columns of a tile (a multiple of 16), tiles across N
  int tiles;
  // TN: a is g [rows, M], w is x [rows, N]; out holds `splits` partial results [M, N] of rows_per_split rows each
  int64_t rows;
  int rows_per_split, mn_tiles;
  int raw_off;            // out = a w^T: where the raw stages lie
  int give_up;           // for tests: as if the first wait had run out (asked at each wait, it costs 2 %)
  int32_t* error;        // SSW_DEV_TIMEOUT goes here, or null
};

__device__ __forceinline__ float2 bf16x2_to_f32(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
// four fp32 values -> their three bf16 terms, packed
__device__ __forceinline__ void split4(const float4& x, uint2& h, uint2& m, uint2& l) {
  const float2 neg = make_float2(-1.f, -1.f);
  float2 p = make_float2(x.x, x.y), q = make_float2(x.z, x.w);
  h = make_uint2(pack2<__nv_bfloat16>(p.x, p.y), pack2<__nv_bfloat16>(q.x, q.y));
  p = __ffma2_rn(bf16x2_to_f32(h.x), neg, p);
  q = __ffma2_rn(bf16x2_to_f32(h.y), neg, q);
  m = make_uint2(pack2<__nv_bfloat16>(p.x, p.y), pack2<__nv_bfloat16>(q.x, q.y));
  p = __ffma2_rn(bf16x2_to_f32(m.x), neg, p);
  q = __ffma2_rn(bf16x2_to_f32(m.y), neg, q);
  l = make_uint2(pack2<__nv_bfloat16>(p.x, p.y), pack2<__nv_bfloat16>(q.x, q.y));
}
// x[0..7] -> the three terms of each, eight bf16 per 16 bytes
__device__ __forceinline__ void split8(const float (&x)[8], uint4& h, uint4& m, uint4& l) {
  uint2 h0, m0, l0, h1, m1, l1;
  split4(make_float4(x[0], x[1], x[2], x[3]), h0, m0, l0);
  split4(make_float4(x[4], x[5], x[6], x[7]), h1, m1, l1);
  h = make_uint4(h0.x, h0.y, h1.x, h1.y);
  m = make_uint4(m0.x, m0.y, m1.x, m1.y);
  l = make_uint4(l0.x, l0.y, l1.x, l1.y);
}
__device__ __forceinline__ void sts_u4(uint32_t a, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void stg_v8(float* dst, const float2 (&v)[4]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(__float_as_uint(v[0].x)), "r"(__float_as_uint(v[0].y)),
               "r"(__float_as_uint(v[1].x)), "r"(__float_as_uint(v[1].y)), "r"(__float_as_uint(v[2].x)), "r"(__float_as_uint(v[2].y)),
               "r"(__float_as_uint(v[3].x)), "r"(__float_as_uint(v[3].y))
               : "memory");
}
__device__ __forceinline__ float gelu_erf(float x) { return x * 0.5f * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) <= 3.402823466e38f); }
__device__ __forceinline__ void sts_v2(uint32_t a, uint2 v) {
  asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(a), "r"(v.x), "r"(v.y) : "memory");
}

// The warps that drain accumulators: number `ew`, tensor-memory lanes 32 `sub` and up, part number `ew` / 4 of a tile's columns; LOW accumulators of small products.  This is work in
// step with the MMAs (a read of the accumulator for every 64 of K, then the stores): with eight warps of half a tile each, 4700 clocks a tile of 96
// columns at K = 96, it was what 150 000 x 288 x 96 took 79 us for.
template <bool TN, int PARTS, int LOW>
__device__ __forceinline__ void gemm_drain(const GemmParams& p, unsigned char* smem, uint32_t tmem, int ew, int sub, int n_stages, const GemmBars& b,
                                           bool& timed_out) {
  constexpr int kChunk = GemmChunk<TN>::kStages, kCols = kGNMax / PARTS;
  const int lane = threadIdx.x & 31, bn = p.bn, part = ew >> 2;
  // this thread's columns [c0, c0 + hc) of a tile: 32 of them or what is left (none, where a tile is narrow); TN: half of them
  const int c0 = PARTS == 3 ? part * kCols : part * (bn / 2), hc = PARTS == 3 ? min(kCols, bn - c0) : bn / 2;
  const uint32_t t_acc = tmem + ((uint32_t)(sub * 32) << 16) + c0;
  const int n_chunks = (n_stages + kChunk - 1) / kChunk;
  float* const bias = reinterpret_cast<float*>(smem + kGBiasOff) + ew * kCols;   // of this warp's columns
  uint32_t ch = 0, tn = 0;
  // (after a time-out every tile that is left is stored as NaN: never a plausible result)
  for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++tn) {
    float2 acc[kCols / 2];
#pragma unroll
    for (int e = 0; e < kCols / 2; ++e) acc[e] = make_float2(0.f, 0.f);
    const int sp = TN ? t / p.mn_tiles : 0, mn = t - sp * (TN ? p.mn_tiles : 0), mt = mn / p.n_tiles;
    const int n0 = (mn - mt * p.n_tiles) * bn + c0, cols = min(hc, p.N - n0);   // (cols a multiple of four)
    if (!TN && p.bias) {   // on its way while the products are formed
      __syncwarp();
      for (int e = lane; e < cols; e += 32) bias[e] = __ldg(p.bias + n0 + e);
      __syncwarp();
    }
    auto add_columns = [&](uint32_t col) {   // (columns beyond hc of the last sixteen: read, not used)
      constexpr int kLoads = PARTS == 3 ? 2 : 1;   // at a time
#pragma unroll
      for (int e0 = 0; e0 < kCols; e0 += 16 * kLoads) {
        if (e0 >= hc) continue;
        uint32_t r[kLoads][16];
#pragma unroll
        for (int x = 0; x < kLoads; ++x) tmem_ldn(t_acc + col + e0 + 16 * x, r[x]);
        tmem_ld_wait();
#pragma unroll
        for (int x = 0; x < 16 * kLoads; x += 2)
          acc[(e0 + x) / 2] = __fadd2_rn(acc[(e0 + x) / 2], make_float2(__uint_as_float(r[x / 16][x % 16]), __uint_as_float(r[x / 16][x % 16 + 1])));
      }
    };
    for (int c = 0; c < n_chunks && !timed_out; ++c, ++ch) {
      const uint32_t hb = ch & 1;
      if (!mbar_wait_bounded(b.hh_full + hb, (ch >> 1) & 1)) { timed_out = true; break; }
      tc_fence_after();
      add_columns(hb * kGNMax);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(b.hh_empty + hb);
    }
    const uint32_t lb = tn % LOW;
    if (!timed_out && !mbar_wait_bounded(b.lo_full + lb, (tn / LOW) & 1)) timed_out = true;
    if (!timed_out) {
      tc_fence_after();
      add_columns(kGTmemLow + lb * kGNMax);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(b.lo_empty + lb);
    }
    // A thread stores its own row's columns, 32 bytes (a whole sector) at a time where they start on such a boundary.
    const int64_t m = (int64_t)mt * kGM + sub * 32 + lane;
    float* row = p.out + (TN ? (int64_t)sp * p.M * p.N : 0) + m * p.N + n0;
    const bool wide = p.wide && (n0 & 7) == 0;
    float2 check = make_float2(0.f, 0.f);
#pragma unroll
    for (int e = 0; e < kCols; e += 8) {
      if (e >= cols) continue;
      const bool two = e + 4 < cols;
      float2 v[4] = {acc[e / 2], acc[e / 2 + 1], acc[e / 2 + 2], acc[e / 2 + 3]};
      if (!TN && p.bias) {
        const float4 b0 = *reinterpret_cast<const float4*>(bias + e), b1 = *reinterpret_cast<const float4*>(bias + e + 4);
        v[0] = __fadd2_rn(v[0], make_float2(b0.x, b0.y));
        v[1] = __fadd2_rn(v[1], make_float2(b0.z, b0.w));
        v[2] = __fadd2_rn(v[2], make_float2(b1.x, b1.y));
        v[3] = __fadd2_rn(v[3], make_float2(b1.z, b1.w));
      }
      if (timed_out) v[0] = v[1] = v[2] = v[3] = make_float2(NAN, NAN);
      check = __fadd2_rn(check, __fadd2_rn(v[0], v[1]));
      if (two) check = __fadd2_rn(check, __fadd2_rn(v[2], v[3]));
      if (!TN && p.gelu) {
#pragma unroll
        for (int x = 0; x < 4; ++x) v[x] = make_float2(gelu_erf(v[x].x), gelu_erf(v[x].y));
      }
      if (m < p.M) {
        if (two && wide) {
          stg_v8(row + e, v);
        } else {
          *reinterpret_cast<float4*>(row + e) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
          if (two) *reinterpret_cast<float4*>(row + e + 4) = make_float4(v[2].x, v[2].y, v[3].x, v[3].y);
        }
      }
    }
    // a result that is not finite (or a sum of them that is not: looked at once more in vain): once more, from the operands
    if (!TN && !timed_out && m < p.M && not_finite(check.x + check.y)) {
      for (int e = 0; e < cols; ++e) {
        if (!not_finite(row[e])) continue;
        float v = 0.f;
        for (int k = 0; k < p.K && v == v; ++k) v = fmaf(__ldg(p.a + m * p.K + k), __ldg(p.w + (int64_t)(n0 + e) * p.K + k), v);
        if (p.bias) v += __ldg(p.bias + n0 + e);
        row[e] = p.gelu ? gelu_erf(v) : v;
      }
    }
  }
}

// out[M, N] = a[M, K] w[N, K]^T.  The rows of a go to tensor memory, where the tensor cores read them beside w in shared memory: a producer thread
// looks after sixteen columns of one row of a stage, brings them in with its warp through a private piece of shared memory, splits them
// and stores the three terms with tcgen05.st.  KEPT: a block's columns of w are split once, for all its row tiles.
template <bool KEPT>
__global__ void __launch_bounds__(kNThreads, 1) k_gemm_f32(GemmParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  uint64_t* full = bars;                     // [kNRing] operands of a stage are in place
  uint64_t* empty = full + kNRing;           // [kNRing] the stage's MMAs are done
  uint64_t* hh_full = empty + kNRing;        // [2] a chunk's h h accumulator is complete
  uint64_t* hh_empty = hh_full + 2;          // [2] ... has been read
  uint64_t* lo_full = hh_empty + 2;          // [2] a tile's small-product accumulator is complete
  uint64_t* lo_empty = lo_full + 2;          // [2]
  uint64_t* drain_bar = lo_empty + 2;        // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kNRing; ++s) {
      mbar_init(full + s, kGProd);
      mbar_init(empty + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(hh_full + b, 1);
      mbar_init(hh_empty + b, kNEpi);
      mbar_init(lo_full + b, 1);
      mbar_init(lo_empty + b, kNEpi);
    }
    mbar_init(drain_bar, 1);
    mbar_fence_init();
  }
  if (warp == kGProd) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_dependency_wait();
  const int n_stages = (p.K + kGK - 1) / kGK;       // of one tile
  const int bn = p.bn;
  constexpr int kChunk = GemmChunk<false>::kStages;
  bool timed_out = p.give_up != 0;
  const uint32_t w_smem = smem_u32(smem + kGFirst);   // [stage][3][bn rows of 64 bytes]: all of K, or the ring's stages

  if (warp < kGProd) {
    // =========================================== producers ====================================
    // A warp brings in 32 rows (the tensor-memory lanes warp % 4 selects) of 16 columns: 64 bytes a row by four lanes, into 2 KB of its own
    // for each stage under way, chunks swapped so that a thread then reads its row without bank conflicts.
    const int sub = warp & 3, kh = warp >> 2, lc = lane & 3, lr = lane >> 2;
    const uint32_t mine = smem_u32(smem + p.raw_off) + (uint32_t)warp * kNRawWarp;
    const int my_tiles = p.tiles > (int)blockIdx.x ? (p.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const int total = my_tiles * n_stages;   // (operands that fit the device keep this far below 2^31)
    int lt = blockIdx.x, ls = 0;             // tile and stage the next load belongs to
    const float *pa, *pw = nullptr;
    int rows_a, rows_w = 0;
    // w (KEPT: of the first tile): piece f4 of rows wr, wr + 32 and wr + 64 of a stage, each read by the thread that asked for it
    const int f4 = threadIdx.x & 7, wr = threadIdx.x >> 3;
    const uint32_t w_mine = smem_u32(smem + p.raw_off) + kNRaws * kNRawStage + threadIdx.x * 16u;
    auto open_tile = [&]() {
      const int mt = lt / p.n_tiles, n0 = (lt - mt * p.n_tiles) * bn;
      const int64_t m0 = (int64_t)mt * kGM + sub * 32;
      rows_a = (int)max((int64_t)0, min((int64_t)32, p.M - m0));
      pa = p.a + (m0 + lr) * p.K + kh * 16 + lc * 4;
      rows_w = min(bn, p.N - n0) - wr;
      pw = p.w + (int64_t)(n0 + wr) * p.K + f4 * 4;
    };
    open_tile();
    const int64_t k8 = (int64_t)p.K * 8, k32 = (int64_t)p.K * 32;
    int lslot = 0, loaded = 0;
    auto load = [&]() {   // one commit group per stage, empty beyond the last one
      if (loaded < total) {
        const bool kin = ls * kGK + kh * 16 + lc * 4 < p.K;   // K is a multiple of four
        const uint32_t dst = mine + (uint32_t)lslot * kNRawStage;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = lr + 8 * i;
          const bool on = kin && r < rows_a;
          cp_async16_or_zero(dst + r * 64 + ((lc ^ ((r >> 1) & 3)) << 4), on ? pa + i * k8 : p.a, on);
        }
        pa += kGK;
        if (!KEPT || loaded < n_stages) {
          const bool win = ls * kGK + f4 * 4 < p.K;
          const uint32_t wd = w_mine + (uint32_t)lslot * kNRawW;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const bool on = win && 32 * i < rows_w;
            cp_async16_or_zero(wd + i * 4096u, on ? pw + i * k32 : p.a, on);
          }
          pw += kGK;
        }
        lslot = lslot + 1 == kNRaws ? 0 : lslot + 1;
        ++loaded;
        if (++ls == n_stages) {
          ls = 0;
          lt += gridDim.x;
          if (lt < p.tiles) open_tile();
        }
      }
      cp_async_commit();
    };
    for (int x = 0; x < kNRaws - 1; ++x) load();
    auto store_w = [&](uint32_t stage, int r, int f, const float4& v) {
      uint2 h, m, l;
      split4(v, h, m, l);
      const uint32_t d = stage + (uint32_t)(r * kGRowB + (((f >> 1) ^ ((r >> 1) & 3)) << 4) + (f & 1) * 8);
      sts_v2(d, h);
      sts_v2(d + kGOpWB, m);
      sts_v2(d + 2 * kGOpWB, l);
    };
    int slot = 0;
    uint32_t s = 0, spar = 1;   // stage, parity of the use of it before this one
    for (int i = 0; i < total && !timed_out; ++i) {
      // this stage's pieces have landed, those of the warp's other lanes as well
      cp_async_wait<kNRaws - 2>();
      __syncwarp();
      const uint32_t src = mine + (uint32_t)slot * kNRawStage + lane * 64;
      int4 raw4[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) raw4[x] = lds_v4(src + ((x ^ ((lane >> 1) & 3)) << 4));
      load();   // into the slot of the stage before, which all lanes have read
      uint32_t h[8], m[8], l[8];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int4 u = raw4[x];
        uint2 h2, m2, l2;
        split4(make_float4(__int_as_float(u.x), __int_as_float(u.y), __int_as_float(u.z), __int_as_float(u.w)), h2, m2, l2);
        h[2 * x] = h2.x; h[2 * x + 1] = h2.y;
        m[2 * x] = m2.x; m[2 * x + 1] = m2.y;
        l[2 * x] = l2.x; l[2 * x + 1] = l2.y;
      }
      if (i >= kNRing && !mbar_wait_bounded(empty + s, spar)) {
        timed_out = true;
        break;
      }
      tc_fence_after();   // the MMAs that read the stage before come before the stores below
      const uint32_t ta = tmem + ((uint32_t)(sub * 32) << 16) + kNTmemA + s * kNStageCols + kh * 8;
      tmem_stn(ta, h);
      tmem_stn(ta + 16, m);
      tmem_stn(ta + 32, l);
      if (!KEPT || i < n_stages) {   // (kept: with the first tile)
        const uint32_t wsrc = w_mine + (uint32_t)slot * kNRawW;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          if (wr + 32 * x >= bn) continue;
          const int4 u = lds_v4(wsrc + x * 4096u);
          store_w(w_smem + (KEPT ? (uint32_t)i : s) * 3 * kGOpWB, wr + 32 * x, f4,
                  make_float4(__int_as_float(u.x), __int_as_float(u.y), __int_as_float(u.z), __int_as_float(u.w)));
        }
        fence_async_smem();  // the tensor cores read shared memory through the async proxy
      }
      slot = slot + 1 == kNRaws ? 0 : slot + 1;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + s);
      if (++s == kNRing) {
        s = 0;
        spar ^= 1;
      }
    }
    cp_async_wait<0>();   // nothing of this block's may still be on its way into shared memory
  } else if (warp == kGProd) {
    // =========================================== MMA issuer ===================================
    // All lanes walk along and one issues, on operands that the compiler can see are the same in each: an MMA takes them from
    // uniform registers, and from a branch of one lane each is first looked for among the lanes (some hundred instructions an
    // MMA: 150 000 x 288 x 96 102 us for 96, 10 000 x 192 x 768 49 for 41).
    const uint32_t idesc = instr_desc(1, 1, 0, bn), tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t w0 = smem_desc(w_smem, 512, 4);
    const bool leader = elect_one();
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      timed_out = !__all_sync(0xffffffffu, mbar_wait_bounded(bar, parity));
      return !timed_out;
    };
    timed_out = __any_sync(0xffffffffu, timed_out);
    uint32_t s = 0, spar = 0, ch = 0, tn = 0;   // stage and parity of its use, chunks, tiles so far
    for (int t = blockIdx.x; t < p.tiles && !timed_out; t += gridDim.x, ++tn) {
      const uint32_t lb = tn & 1;
      if (tn >= 2 && !wait(lo_empty + lb, ((tn >> 1) - 1) & 1)) break;
      for (int ks = 0; ks < n_stages; ++ks) {
        const uint32_t hb = ch & 1;
        const bool first = ks % kChunk == 0, last = ks % kChunk == kChunk - 1 || ks == n_stages - 1;
        if (first && ch >= 2 && !wait(hh_empty + hb, ((ch >> 1) - 1) & 1)) break;
        if (!wait(full + s, spar)) break;
        tc_fence_after();
        const uint32_t ta = tm + kNTmemA + s * kNStageCols, hh = tm + hb * kGNMax, lo = tm + kGTmemLow + lb * kGNMax;
        const uint64_t db = w0 + (KEPT ? ks : (int)s) * (3 * kGOpWB >> 4);
        if (leader) {
          constexpr int ob = kGOpWB >> 4;
#pragma unroll
          for (int k16 = 0; k16 < kGK / 16; ++k16) {
            const uint32_t a = ta + k16 * 8;
            const uint64_t b = db + k16 * 2;
            umma_ts(hh, a, b, idesc, !(first && k16 == 0));
            umma_ts(lo, a, b + 2 * ob, idesc, ks > 0 || k16 > 0);   // smallest first
            umma_ts(lo, a + 32, b, idesc, 1);
            umma_ts(lo, a + 16, b + ob, idesc, 1);
            umma_ts(lo, a, b + ob, idesc, 1);
            umma_ts(lo, a + 16, b, idesc, 1);
          }
          umma_commit(empty + s);
          if (last) umma_commit(hh_full + hb);
          if (ks == n_stages - 1) umma_commit(lo_full + lb);
        }
        __syncwarp();
        if (last) ++ch;
        if (++s == kNRing) {
          s = 0;
          spar ^= 1;
        }
      }
    }
    // let the tensor cores finish whatever was issued before the tensor memory is given back
    if (leader) umma_commit(drain_bar);
    __syncwarp();
    mbar_wait_bounded(drain_bar, 0);
  } else {
    gemm_drain<false, 3, 2>(p, smem, tmem, warp - kGProd - 1, warp & 3, n_stages, {hh_full, hh_empty, lo_full, lo_empty}, timed_out);
  }
  if (timed_out && p.error) atomicOr(reinterpret_cast<unsigned*>(p.error), SSW_DEV_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == kGProd) tmem_dealloc(tmem, 512);
}

// out[N, K] = g[M, N]^T x[M, K] over a range of rows (p.M and p.N are the N and K of it, the rows the steps of the sum): the columns of g go to tensor memory, where a
// producer thread is a column.  Its warp brings in 16 rows of 32 columns, 128 bytes a row, and the thread reads its column down them.  x goes to
// shared memory: a thread of three more warps takes four columns of eight consecutive rows and turns them in registers.
__global__ void __launch_bounds__(kTThreads, 1) k_gemm_f32_tn(GemmParams p) {
  constexpr int kRing = 4, kTmemA = 3 * kGNMax;   // one accumulator of small products: the sums are long
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  uint64_t* full = bars;                     // [kRing] operands of a stage are in place
  uint64_t* empty = full + kRing;            // [kRing] the stage's MMAs are done
  uint64_t* hh_full = empty + kRing;         // [2] a chunk's h h accumulator is complete
  uint64_t* hh_empty = hh_full + 2;          // [2] ... has been read
  uint64_t* lo_full = hh_empty + 2;          // [2] a tile's small-product accumulator is complete
  uint64_t* lo_empty = lo_full + 2;          // [2]
  uint64_t* drain_bar = lo_empty + 2;        // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRing; ++s) {
      mbar_init(full + s, kTProd);
      mbar_init(empty + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(hh_full + b, 1);
      mbar_init(hh_empty + b, kGEpi);
      mbar_init(lo_full + b, 1);
      mbar_init(lo_empty + b, kGEpi);
    }
    mbar_init(drain_bar, 1);
    mbar_fence_init();
  }
  if (warp == kTProd) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_dependency_wait();
  const int n_stages = (p.rows_per_split + kGK - 1) / kGK;       // of one tile
  const int bn = p.bn;
  bool timed_out = p.give_up != 0;
  const uint32_t x_smem = smem_u32(smem + kGFirst);   // [kRing][3][bn rows of 64 bytes]

  if (warp < kTProd) {
    // =========================================== producers ====================================
    const int my_tiles = p.tiles > (int)blockIdx.x ? (p.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const int total = my_tiles * n_stages;   // (operands that fit the device keep this far below 2^31)
    int lt = blockIdx.x, ls = 0;             // tile and stage the next load belongs to
    const bool is_x = warp >= kGProd;
    const int sub = warp & 3, kh = warp >> 2, lc = lane & 7, lr = lane >> 3;   // g
    const int tx = threadIdx.x - kGProd * 32, oct = tx & 3, quad = tx >> 2;    // x
    const uint32_t raw = smem_u32(smem + kTRawOff) + (is_x ? kNRaws * kNRawStage + tx * 16u : warp * kNRawWarp);
    const uint32_t raw_b = is_x ? kTRawX : kNRawStage;
    const int ld = is_x ? p.N : (int)p.M;
    const float* src = nullptr;
    int rows = 0;   // of the split, from this thread's first row of a stage on; 0 where its columns do not exist
    auto open_tile = [&]() {
      const int sp = lt / p.mn_tiles, mn = lt - sp * p.mn_tiles, mt = mn / p.n_tiles;
      const int at = is_x ? quad * 4 : sub * 32 + lc * 4, col = (is_x ? (mn - mt * p.n_tiles) * bn : mt * kGM) + at, r0 = is_x ? oct * 8 : kh * 16 + lr;
      const int64_t k0 = (int64_t)sp * p.rows_per_split + r0;
      rows = (int)max((int64_t)0, min((int64_t)p.rows_per_split - r0, p.rows - k0));
      if (col >= ld || (is_x && at >= bn)) rows = 0;   // M and N are multiples of four
      src = (is_x ? p.w : p.a) + k0 * ld + col;
    };
    open_tile();
    int lslot = 0, loaded = 0;
    auto load = [&]() {   // one commit group per stage, empty beyond the last one
      if (loaded < total) {
        const uint32_t dst = raw + (uint32_t)lslot * raw_b;
        if (is_x) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const bool on = ls * kGK + i < rows;
            cp_async16_or_zero(dst + i * kTRawRow, on ? src + (int64_t)i * ld : p.a, on);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const bool on = ls * kGK + 4 * i < rows;
            cp_async16_or_zero(dst + (lr + 4 * i) * 128 + lc * 16, on ? src + (int64_t)(4 * i) * ld : p.a, on);
          }
        }
        src += (int64_t)kGK * ld;
        lslot = lslot + 1 == kNRaws ? 0 : lslot + 1;
        ++loaded;
        if (++ls == n_stages) {
          ls = 0;
          lt += gridDim.x;
          if (lt < p.tiles) open_tile();
        }
      }
      cp_async_commit();
    };
    for (int x = 0; x < kNRaws - 1; ++x) load();
    int slot = 0;
    uint32_t s = 0, spar = 1;   // stage, parity of the use of it before this one
    for (int i = 0; i < total && !timed_out; ++i) {
      // this stage's pieces have landed, those of the warp's other lanes as well
      cp_async_wait<kNRaws - 2>();
      __syncwarp();
      const uint32_t at = raw + (uint32_t)slot * raw_b;
      slot = slot + 1 == kNRaws ? 0 : slot + 1;
      if (is_x) {
        float4 v[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const int4 u = lds_v4(at + x * kTRawRow);
          v[x] = make_float4(__int_as_float(u.x), __int_as_float(u.y), __int_as_float(u.z), __int_as_float(u.w));
        }
        load();   // into the slot of the stage before, which all lanes have read
        if (i >= kRing && !mbar_wait_bounded(empty + s, spar)) {
          timed_out = true;
          break;
        }
        if (quad * 4 < bn) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float x[8];
#pragma unroll
            for (int i8 = 0; i8 < 8; ++i8) x[i8] = j == 0 ? v[i8].x : j == 1 ? v[i8].y : j == 2 ? v[i8].z : v[i8].w;
            uint4 h, m, l;
            split8(x, h, m, l);
            const int row = quad * 4 + j;
            const uint32_t d = x_smem + s * 3 * kGOpWB + (uint32_t)(row * kGRowB + ((oct ^ ((row >> 1) & 3)) << 4));
            sts_u4(d, h);
            sts_u4(d + kGOpWB, m);
            sts_u4(d + 2 * kGOpWB, l);
          }
        }
        fence_async_smem();  // the tensor cores read shared memory through the async proxy
      } else {
        float x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) x[r] = lds_f32(at + r * 128 + lane * 4);
        load();
        uint32_t h[8], m[8], l[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint2 h2, m2, l2;
          split4(make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]), h2, m2, l2);
          h[2 * q] = h2.x; h[2 * q + 1] = h2.y;
          m[2 * q] = m2.x; m[2 * q + 1] = m2.y;
          l[2 * q] = l2.x; l[2 * q + 1] = l2.y;
        }
        if (i >= kRing && !mbar_wait_bounded(empty + s, spar)) {
          timed_out = true;
          break;
        }
        tc_fence_after();   // the MMAs that read the stage before come before the stores below
        const uint32_t ta = tmem + ((uint32_t)(sub * 32) << 16) + kTmemA + s * kNStageCols + kh * 8;
        tmem_stn(ta, h);
        tmem_stn(ta + 16, m);
        tmem_stn(ta + 32, l);
        tmem_st_wait();
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(full + s);
      if (++s == kRing) {
        s = 0;
        spar ^= 1;
      }
    }
    cp_async_wait<0>();   // nothing of this block's may still be on its way into shared memory
  } else if (warp == kTProd) {
    // =========================================== MMA issuer ===================================
    // (all lanes walk along: see k_gemm_f32)
    const uint32_t idesc = instr_desc(1, 1, 0, bn), tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t x0 = smem_desc(x_smem, 512, 4);
    const bool leader = elect_one();
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      timed_out = !__all_sync(0xffffffffu, mbar_wait_bounded(bar, parity));
      return !timed_out;
    };
    timed_out = __any_sync(0xffffffffu, timed_out);
    static_assert(GemmChunk<true>::kStages == 1, "");
    uint32_t s = 0, spar = 0, ch = 0, tn = 0;   // stage and parity of its use, chunks (stages), tiles so far
    for (int t = blockIdx.x; t < p.tiles && !timed_out; t += gridDim.x, ++tn) {
      if (tn >= 1 && !wait(lo_empty, (tn - 1) & 1)) break;
      for (int ks = 0; ks < n_stages; ++ks, ++ch) {
        const uint32_t hb = ch & 1;
        if (ch >= 2 && !wait(hh_empty + hb, ((ch >> 1) - 1) & 1)) break;
        if (!wait(full + s, spar)) break;
        tc_fence_after();
        const uint32_t ta = tm + kTmemA + s * kNStageCols, hh = tm + hb * kGNMax, lo = tm + kGTmemLow;
        const uint64_t db = x0 + s * (3 * kGOpWB >> 4);
        if (leader) {
          constexpr int ob = kGOpWB >> 4;
#pragma unroll
          for (int k16 = 0; k16 < kGK / 16; ++k16) {
            const uint32_t a = ta + k16 * 8;
            const uint64_t b = db + k16 * 2;
            umma_ts(hh, a, b, idesc, k16 > 0);
            umma_ts(lo, a, b + 2 * ob, idesc, ks > 0 || k16 > 0);   // smallest first
            umma_ts(lo, a + 32, b, idesc, 1);
            umma_ts(lo, a + 16, b + ob, idesc, 1);
            umma_ts(lo, a, b + ob, idesc, 1);
            umma_ts(lo, a + 16, b, idesc, 1);
          }
          umma_commit(empty + s);
          umma_commit(hh_full + hb);
          if (ks == n_stages - 1) umma_commit(lo_full);
        }
        __syncwarp();
        if (++s == kRing) {
          s = 0;
          spar ^= 1;
        }
      }
    }
    // let the tensor cores finish whatever was issued before the tensor memory is given back
    if (leader) umma_commit(drain_bar);
    __syncwarp();
    mbar_wait_bounded(drain_bar, 0);
  } else {
    gemm_drain<true, 2, 1>(p, smem, tmem, warp - kTProd - 1, warp & 3, n_stages, {hh_full, hh_empty, lo_full, lo_empty}, timed_out);
  }
  if (timed_out && p.error) atomicOr(reinterpret_cast<unsigned*>(p.error), SSW_DEV_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == kTProd) tmem_dealloc(tmem, 512);
}

// Partial results of a weight gradient added up in order.  If that is not finite, the partial results that are not are
// formed again from their rows of g and x, eight rows in flight and no further than the first NaN.
__global__ void __launch_bounds__(256) k_gemm_reduce(const float* __restrict__ partial, int splits, int rows_per_split, const float* __restrict__ g,
                                                     const float* __restrict__ x, int64_t rows, int N, int K, float* __restrict__ out) {
  grid_dependency_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, width = (int64_t)N * K;
  if (i >= width) return;
  float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
  for (int k = 0; k < splits; k += 4)
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (k + x < splits) s4[x] += __ldcg(partial + (k + x) * width + i);
  float s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
  if (not_finite(s)) {
    const int n = (int)(i / K), c = (int)(i - (int64_t)n * K);
    s = 0.f;
    for (int k = 0; k < splits && s == s; ++k) {
      float v = __ldcg(partial + k * width + i);
      if (not_finite(v)) {
        v = 0.f;
        const int64_t m0 = (int64_t)k * rows_per_split, m1 = min(rows, m0 + rows_per_split);
        for (int64_t m = m0; m < m1 && v == v; m += 8) {
          float gv[8], xv[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const bool on = m + e < m1;
            gv[e] = on ? __ldg(g + (m + e) * N + n) : 0.f;
            xv[e] = on ? __ldg(x + (m + e) * K + c) : 0.f;
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) v = fmaf(gv[e], xv[e], v);
        }
      }
      s += v;
    }
  }
  out[i] = s;
}

// gemm_gelu.cu
int gemm_gelu(const void* a, const void* w, const void* bias, int dtype, void* out, int64_t M, int32_t N, int32_t K, int32_t* error,
              int give_up, void* stream);

}  // namespace ssw

using namespace ssw;

// Columns of a tile: the split of N into equal tiles whose waves over the SMs cost least, a tile's cost being
// its columns plus the rows of A it splits (in the same units: both are rows of operands).  Where w is kept its columns are split once a block, and they
// are what the drain takes its time for all the same.  Against every other width, 22 shapes from 1000 x 768 x 3072 to 150 000 x 384 x 96: the fastest of all
// in each (10 000 x 192 x 192 64 columns 11.0 us, 48 13.4, 96 12.4; 2500 x 1536 x 384 80 columns 28.8, 64 34.9, 96 30.9; 3000 x 96 x 96 16 columns 4.5, 96 6.0).
static int gemm_columns(int64_t m_tiles, int N, int sms, int* n_tiles) {
  int best = 0;
  int64_t best_cost = 0;
  for (int nt = (N + kGNMax - 1) / kGNMax; nt <= (N + 15) / 16; ++nt) {
    const int bn = ((N + nt - 1) / nt + 15) / 16 * 16;
    const int used = (N + bn - 1) / bn;
    const int64_t cost = ((m_tiles * used + sms - 1) / sms) * (bn + kGM);
    if (!best || cost < best_cost) {
      best = bn;
      best_cost = cost;
      *n_tiles = used;
    }
  }
  return best;
}

// K up to which a block's columns of w are kept: six stages of 18 KB beside four of 28 KB of raw rows.
constexpr int kGKeptK = 6 * kGK;
static_assert(kGFirst + kGKeptK / kGK * 3 * kGOpWB + kNRaws * (kNRawStage + kNRawW) + 1024 <= 227 * 1024, "");

static int gemm_nt(const float* a, const float* w, const float* bias, float* out, int64_t M, int32_t N, int32_t K, int gelu, int32_t* error,
            int give_up, void* stream_) {
  if (M < 0 || N <= 0 || K <= 0) return SSW_E_INVALID;
  if (M == 0) return SSW_OK;
  if (!a || !w || !out) return SSW_E_INVALID;
  if ((N | K) & 3) return SSW_E_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(bias) |
       reinterpret_cast<uintptr_t>(out)) & 15)
    return SSW_E_INVALID;
  int dev = 0, sms = 0;
  SSW_CUDA_TRY(cudaGetDevice(&dev));
  SSW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  GemmParams p = {};
  p.a = a; p.w = w; p.bias = bias; p.out = out; p.M = M; p.N = N; p.K = K; p.gelu = gelu;
  p.error = error; p.give_up = give_up;
  p.wide = N % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 31) == 0;
  const int64_t m_tiles = ceil_div64(M, kGM);
  p.bn = gemm_columns(m_tiles, N, sms, &p.n_tiles);
  if (m_tiles * p.n_tiles >= ((int64_t)1 << 30)) return SSW_E_RANGE;
  p.tiles = (int)(m_tiles * p.n_tiles);
  const int n_stages = (K + kGK - 1) / kGK, groups = sms / p.n_tiles;   // blocks a column tile
  const bool kept = K <= kGKeptK && groups * p.n_tiles * 16 >= sms * 15;
  p.raw_off = kGFirst + (kept ? n_stages : kNRing) * 3 * kGOpWB;
  const int smem = p.raw_off + kNRaws * (kNRawStage + kNRawW) + 1024;
  auto kern = kept ? k_gemm_f32<true> : k_gemm_f32<false>;
  // kept: tile t, t + grid, ... of a block are of the same columns
  const int64_t grid = kept ? (m_tiles < groups ? m_tiles : groups) * p.n_tiles : p.tiles < sms ? p.tiles : sms;
  SSW_CUDA_TRY(allow_smem(kern));
  SSW_CUDA_TRY(launch_chained(kern, dim3((unsigned)grid), dim3(kNThreads), (size_t)smem, (cudaStream_t)stream_, p));
  SSW_LAUNCH_CHECK("k_gemm_f32");
  return SSW_OK;
}

extern "C" int ssw_gemm_f32(const float* a, const float* w, const float* bias, float* out, int64_t M, int32_t N, int32_t K,
                            int32_t* error, void* stream) {
  return gemm_nt(a, w, bias, out, M, N, K, 0, error, 0, stream);
}
extern "C" int ssw_gemm_f32_gelu(const float* a, const float* w, const float* bias, float* out, int64_t M, int32_t N, int32_t K,
                                 int32_t* error, void* stream) {
  return gemm_nt(a, w, bias, out, M, N, K, 1, error, 0, stream);
}

// Weight gradient [N, K] of M rows: equal splits of M, as many as give every SM a tile, of four stages (128 rows) at least.
// With more tiles than SMs, as many of up to eight as fill the waves best (3072 x 768, 192 tiles, 16 384 rows: one split is two
// waves for 1.3 of work, 1381 us where the library takes 1169; three splits take 930).
static void wgrad_shape(int64_t M, int32_t N, int32_t K, int sms, GemmParams& p, int& splits) {
  p.n_tiles = (K + kGNMax - 1) / kGNMax;
  p.bn = ((K + p.n_tiles - 1) / p.n_tiles + 15) / 16 * 16;
  p.n_tiles = (K + p.bn - 1) / p.bn;
  p.mn_tiles = (int)ceil_div64(N, kGM) * p.n_tiles;
  const int unit = 4 * kGK;
  int64_t want = sms / p.mn_tiles;
  if (want == 0) {
    want = 1;
    auto waves = [&](int64_t s) { return ceil_div64(p.mn_tiles * s, sms); };
    for (int64_t s = 2; s <= 8; ++s)
      if (waves(s) * want < waves(want) * s) want = s;
  }
  const int64_t per = ceil_div64(ceil_div64(M, want), unit) * unit;
  p.rows_per_split = (int)(per < (1 << 30) ? per : (1 << 30));
  splits = (int)ceil_div64(M, p.rows_per_split);
}
static int wgrad_sms(int* sms) {
  int dev = 0;
  SSW_CUDA_TRY(cudaGetDevice(&dev));
  SSW_CUDA_TRY(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
  return SSW_OK;
}

extern "C" int64_t ssw_gemm_f32_tn_workspace_floats(int64_t M, int32_t N, int32_t K) {
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  GemmParams p = {};
  int sms = 0, splits = 0;
  if (wgrad_sms(&sms) != SSW_OK) return -1;
  wgrad_shape(M, N, K, sms, p, splits);
  return (int64_t)splits * N * K;
}

static int gemm_tn(const float* g, const float* x, float* out, int64_t M, int32_t N, int32_t K, float* workspace, int32_t* error,
            int give_up, void* stream_) {
  if (M <= 0 || N <= 0 || K <= 0 || !g || !x || !out || !workspace) return SSW_E_INVALID;
  if ((N | K) & 3) return SSW_E_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) |
       reinterpret_cast<uintptr_t>(workspace)) & 15)
    return SSW_E_INVALID;
  GemmParams p = {};
  int sms = 0, splits = 0;
  const int rc = wgrad_sms(&sms);
  if (rc != SSW_OK) return rc;
  wgrad_shape(M, N, K, sms, p, splits);
  p.a = g; p.w = x; p.out = workspace; p.M = N; p.N = K; p.rows = M;
  p.wide = K % 8 == 0 && (reinterpret_cast<uintptr_t>(workspace) & 31) == 0;
  p.error = error; p.give_up = give_up;
  if ((int64_t)p.mn_tiles * splits >= ((int64_t)1 << 30)) return SSW_E_RANGE;
  p.tiles = p.mn_tiles * splits;
  SSW_CUDA_TRY(allow_smem(k_gemm_f32_tn));
  SSW_CUDA_TRY(launch_chained(k_gemm_f32_tn, dim3((unsigned)(p.tiles < sms ? p.tiles : sms)), dim3(kTThreads), kTSmem,
                              (cudaStream_t)stream_, p));
  SSW_CUDA_TRY(launch_chained(k_gemm_reduce, dim3((unsigned)ceil_div64((int64_t)N * K, 256)), dim3(256), 0, (cudaStream_t)stream_,
                              (const float*)workspace, splits, p.rows_per_split, g, x, M, (int)N, (int)K, out));
  return SSW_OK;
}

extern "C" int ssw_gemm_f32_tn(const float* g, const float* x, float* out, int64_t M, int32_t N, int32_t K, float* workspace,
                               int32_t* error, void* stream) {
  return gemm_tn(g, x, out, M, N, K, workspace, error, 0, stream);
}

// The three GEMMs, giving up at the first wait if asked to (for tests).
extern "C" int ssw_debug_gemm(int kind, const void* a, const void* w, int dtype, void* out, int64_t M, int32_t N, int32_t K, float* workspace,
                              int32_t* error, int give_up, void* stream) {
  const float *af = reinterpret_cast<const float*>(a), *wf = reinterpret_cast<const float*>(w);
  if (kind == 0) return gemm_nt(af, wf, nullptr, reinterpret_cast<float*>(out), M, N, K, 0, error, give_up, stream);
  if (kind == 1) return gemm_tn(af, wf, reinterpret_cast<float*>(out), M, N, K, workspace, error, give_up, stream);
  if (kind == 2) return gemm_gelu(a, w, nullptr, dtype, out, M, N, K, error, give_up, stream);
  return SSW_E_INVALID;
}
