// The first half of a Swin block's MLP in 16-bit inference: out = gelu(a[M, K] w[N, K]^T + bias), one kernel
// (swin3d_base.py:1109-1149: Linear, then the erf form of GELU).  As a library GEMM and an element-wise pass the
// hidden rows (4 C wide) cross memory three times instead of once, and the pass itself is bound by the
// instructions of erf.
//
// Persistent, one block per SM, 21 warps: four bring operand tiles in (16-byte asynchronous copies into the
// 64-byte-swizzled layout, two stages ahead), one issues the MMAs (128 x bn x 32 per stage, bn <= 128, accumulators
// double buffered in tensor memory), sixteen drain them: bias, GELU, rounding, and out through a staging piece so that
// four lanes store 64 bytes of one row.
// What bounds it is the drain (11 instructions and two special-function operations per element, two elements at a
// time), hence its sixteen warps.  bf16, against the library's GEMM and torch's GELU: 150 000 x 384 x 96 98 -> 71 us,
// 40 000 x 768 x 192 56 -> 46, 10 000 x 768 x 192 25 -> 20; 10 000 x 1536 x 384 35 -> 41, so the caller keeps to K <= 256.
// Relative error against 64 bits 1.7e-3 (one rounding) where the two passes have 2.7e-3 (two).
#include <math.h>

#include "attn_common.cuh"
#include "tcgen05.cuh"

namespace ssw {

int gemm_gelu(const void* a, const void* w, const void* bias, int dtype, void* out, int64_t M, int32_t N, int32_t K, int32_t* error,
              int give_up, void* stream);

constexpr int kHM = 128, kHN = 128, kHK = 32, kHRowB = kHK * 2;
constexpr int kHStages = 4, kHAhead = 2;
constexpr int kHProd = 4, kHEpi = 16;
constexpr int kHThreads = 32 * (kHProd + 1 + kHEpi);
constexpr int kHOpB = kHM * kHRowB, kHStageB = 2 * kHOpB;
constexpr int kHPitch = 80;                                     // bytes between rows of a staging piece: 64 and a skew
constexpr int kHPiece = 1024 + kHStages * kHStageB;
constexpr int kHSmem = kHPiece + kHEpi * 32 * kHPitch + 1024;

struct HalfGemmParams {
  const void *a, *w, *bias;
  void* out;
  int64_t M;
  int N, K, bn, n_tiles, tiles;
  int give_up;           // for tests: as if the first wait had run out
  int32_t* error;        // SSW_DEV_TIMEOUT goes here, or null
};

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// x Phi(x) for two values, as max(x, 0) - |x| erfc(|x| / sqrt 2) / 2.  erfc is the Chebyshev fit of Press et al.,
// Numerical Recipes, "erfcc" (relative error below 1.2e-7 for every argument), with log2 e and the factor 1/2 folded
// into the exponent; the arithmetic around it leaves a relative error of a few 1e-6 in the tails, where 16-bit
// results are rounded at 4.9e-4 (fp16) and 3.9e-3 (bf16).
__device__ __forceinline__ float2 gelu2(float2 x) {
  const float2 ax = make_float2(fabsf(x.x), fabsf(x.y));
  const float2 d = __ffma2_rn(ax, make_float2(0.35355339f, 0.35355339f), make_float2(1.f, 1.f));  // 1 + |x| / (2 sqrt 2)
  const float2 t = make_float2(rcp_approx(d.x), rcp_approx(d.y));
  constexpr double L = 1.4426950408889634;
  constexpr float c[10] = {(float)(-1.26551223 * L - 1.0), (float)(1.00002368 * L), (float)(0.37409196 * L), (float)(0.09678418 * L),
                           (float)(-0.18628806 * L), (float)(0.27886807 * L), (float)(-1.13520398 * L), (float)(1.48851587 * L),
                           (float)(-0.82215223 * L), (float)(0.17087277 * L)};
  float2 p = make_float2(c[9], c[9]);
#pragma unroll
  for (int i = 8; i >= 0; --i) p = __ffma2_rn(p, t, make_float2(c[i], c[i]));
  const float2 sq = __fmul2_rn(ax, make_float2((float)(-0.5 * L), (float)(-0.5 * L)));
  p = __ffma2_rn(sq, ax, p);
  const float2 h = __fmul2_rn(t, make_float2(fast_exp2(p.x), fast_exp2(p.y)));
  return __ffma2_rn(make_float2(-ax.x, -ax.y), h, make_float2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f)));
}

template <typename T>
__device__ __forceinline__ float elem_to_float(const T* p);
template <>
__device__ __forceinline__ float elem_to_float(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <>
__device__ __forceinline__ float elem_to_float(const __half* p) { return __half2float(*p); }

template <typename T>
__global__ void __launch_bounds__(kHThreads, 1) k_gemm_gelu(HalfGemmParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  uint64_t* full = bars;                  // [kHStages]
  uint64_t* empty = full + kHStages;      // [kHStages]
  uint64_t* acc_full = empty + kHStages;  // [2]
  uint64_t* acc_empty = acc_full + 2;     // [2]
  uint64_t* drain_bar = acc_empty + 2;    // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  const uint32_t stage0 = smem_u32(smem + 1024);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kHStages; ++s) {
      mbar_init(full + s, kHProd);
      mbar_init(empty + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + b, 1);
      mbar_init(acc_empty + b, kHEpi);
    }
    mbar_init(drain_bar, 1);
    mbar_fence_init();
  }
  if (warp == kHProd) tmem_alloc(tmem_slot, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_dependency_wait();
  const int n_stages = (p.K + kHK - 1) / kHK, bn = p.bn;
  bool timed_out = p.give_up != 0;

  if (warp < kHProd) {
    // ---- producers: 16-byte chunk ch of rows r0, r0 + 32, ... of both operands
    const int ch = threadIdx.x & 3, r0 = threadIdx.x >> 2;
    const int my_tiles = p.tiles > (int)blockIdx.x ? (p.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const int64_t total = (int64_t)my_tiles * n_stages;
    int lt = blockIdx.x, ls = 0, rows_a = 0, rows_w = 0;
    const T *pa = nullptr, *pw = nullptr;
    auto open_tile = [&]() {
      const int mt = lt / p.n_tiles, n0 = (lt - mt * p.n_tiles) * bn;
      const int64_t m0 = (int64_t)mt * kHM;
      rows_a = (int)min((int64_t)kHM, p.M - m0) - r0;
      rows_w = min(bn, p.N - n0) - r0;
      pa = reinterpret_cast<const T*>(p.a) + (m0 + r0) * p.K + ch * 8;
      pw = reinterpret_cast<const T*>(p.w) + (int64_t)(n0 + r0) * p.K + ch * 8;
    };
    if (total > 0) open_tile();
    const int64_t k32 = (int64_t)p.K * 32;
    const uint32_t off = (uint32_t)(r0 * kHRowB + ((ch ^ ((r0 >> 1) & 3)) << 4));
    for (int64_t i = 0; i < total + kHAhead && !timed_out; ++i) {
      if (i < total) {
        const int s = (int)(i % kHStages);
        const int64_t use = i / kHStages;
        if (use > 0 && !mbar_wait_bounded(empty + s, (uint32_t)(use - 1) & 1)) {
          timed_out = true;
          break;
        }
        const uint32_t dst = stage0 + (uint32_t)s * kHStageB + off;
        const bool kin = ls * kHK + ch * 8 < p.K;   // K is a multiple of eight
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const bool ona = kin && 32 * x < rows_a, onw = kin && 32 * x < rows_w;
          cp_async16_or_zero(dst + x * (32u * kHRowB), ona ? (const void*)(pa + x * k32) : p.a, ona);
          cp_async16_or_zero(dst + kHOpB + x * (32u * kHRowB), onw ? (const void*)(pw + x * k32) : p.a, onw);
        }
        pa += kHK;
        pw += kHK;
        if (++ls == n_stages) {
          ls = 0;
          lt += gridDim.x;
          if (lt < p.tiles) open_tile();
        }
      }
      cp_async_commit();
      if (i >= kHAhead) {
        cp_async_wait<kHAhead>();   // the stage asked for kHAhead steps ago has landed
        fence_async_smem();         // the tensor cores read shared memory through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(full + (int)((i - kHAhead) % kHStages));
      }
    }
    cp_async_wait<0>();
  } else if (warp == kHProd) {
    const int fmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    // (operands in uniform registers: see the issuer of gemm_f32.cu)
    const uint32_t idesc = instr_desc(fmt, fmt, 0, bn), tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t d0 = smem_desc(stage0, 512, 4);
    const bool leader = elect_one();
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      timed_out = !__all_sync(0xffffffffu, mbar_wait_bounded(bar, parity));
      return !timed_out;
    };
    timed_out = __any_sync(0xffffffffu, timed_out);
    uint32_t s = 0, spar = 0, tn = 0;
    for (int t = blockIdx.x; t < p.tiles && !timed_out; t += gridDim.x, ++tn) {
      const uint32_t ab = tn & 1;
      if (tn >= 2 && !wait(acc_empty + ab, ((tn >> 1) - 1) & 1)) break;
      for (int ks = 0; ks < n_stages; ++ks) {
        if (!wait(full + s, spar)) break;
        tc_fence_after();
        const uint64_t da = d0 + s * (kHStageB >> 4), db = da + (kHOpB >> 4);
        if (leader) {
#pragma unroll
          for (int k16 = 0; k16 < kHK / 16; ++k16) umma_ss(tm + ab * kHN, da + k16 * 2, db + k16 * 2, idesc, ks > 0 || k16 > 0);
          umma_commit(empty + s);
          if (ks == n_stages - 1) umma_commit(acc_full + ab);
        }
        __syncwarp();
        if (++s == kHStages) {
          s = 0;
          spar ^= 1;
        }
      }
    }
    if (leader) umma_commit(drain_bar);
    __syncwarp();
    mbar_wait_bounded(drain_bar, 0);
  } else {
    // ---- drain: 32 columns of 32 rows per warp
    const int ew = warp - kHProd - 1, sub = warp & 3, c0 = (ew >> 2) * 32;
    const uint32_t t_lane = (uint32_t)(sub * 32) << 16;
    unsigned char* piece = smem + kHPiece + ew * 32 * kHPitch;
    const int pr = lane >> 2, pc = lane & 3;
    uint32_t tn = 0;
    // (after a time-out every tile that is left is stored as NaN: never a plausible result)
    for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++tn) {
      const uint32_t ab = tn & 1;
      const int mt = t / p.n_tiles, n0 = (t - mt * p.n_tiles) * bn + c0;
      const int64_t m0 = (int64_t)mt * kHM + sub * 32;
      // bias of the warp's columns, one per lane
      float bias = 0.f;
      if (p.bias && c0 + lane < bn && n0 + lane < p.N) bias = elem_to_float(reinterpret_cast<const T*>(p.bias) + n0 + lane);
      timed_out = timed_out || !mbar_wait_bounded(acc_full + ab, (tn >> 1) & 1);
      uint32_t r[32];
      if (!timed_out) {
        tc_fence_after();
        tmem_ld32(tmem + t_lane + ab * kHN + c0, r);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty + ab);
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) r[e] = 0x7fffffffu;
      }
      bool odd = false;
      uint32_t o[16];
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        const float2 b2 = make_float2(__shfl_sync(0xffffffffu, bias, e), __shfl_sync(0xffffffffu, bias, e + 1));
        const float2 x = __fadd2_rn(make_float2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), b2);
        const float2 y = gelu2(x);
        odd = odd || !(fabsf(x.x) + fabsf(x.y) <= 3.0e38f);
        o[e / 2] = pack2<T>(y.x, y.y);
      }
      if (__any_sync(0xffffffffu, odd)) {  // infinities: x Phi(x) as it stands (Inf, and NaN for -Inf)
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float2 x = make_float2(__uint_as_float(r[e]) + __shfl_sync(0xffffffffu, bias, e),
                                 __uint_as_float(r[e + 1]) + __shfl_sync(0xffffffffu, bias, e + 1));
          if (!(fabsf(x.x) + fabsf(x.y) <= 3.0e38f)) o[e / 2] = pack2<T>(x.x * normcdff(x.x), x.y * normcdff(x.y));
        }
      }
      __syncwarp();
#pragma unroll
      for (int x = 0; x < 4; ++x)
        *reinterpret_cast<uint4*>(piece + lane * kHPitch + x * 16) = make_uint4(o[4 * x], o[4 * x + 1], o[4 * x + 2], o[4 * x + 3]);
      __syncwarp();
      const int n = n0 + pc * 8;
      const bool on = c0 + pc * 8 < bn && n < p.N;   // bn and N are multiples of eight
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int64_t m = m0 + pr + 8 * x;
        const uint4 v = *reinterpret_cast<const uint4*>(piece + (pr + 8 * x) * kHPitch + pc * 16);
        if (on && m < p.M) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out) + m * p.N + n) = v;
      }
    }
  }
  if (timed_out && p.error) atomicOr(reinterpret_cast<unsigned*>(p.error), SSW_DEV_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == kHProd) tmem_dealloc(tmem, 256);
}

}  // namespace ssw

using namespace ssw;

int ssw::gemm_gelu(const void* a, const void* w, const void* bias, int dtype, void* out, int64_t M, int32_t N, int32_t K, int32_t* error,
                   int give_up, void* stream_) {
  if (M < 0 || N <= 0 || K <= 0 || (dtype != SSW_BF16 && dtype != SSW_F16)) return SSW_E_INVALID;
  if (M == 0) return SSW_OK;
  if (!a || !w || !out) return SSW_E_INVALID;
  if ((N | K) & 7) return SSW_E_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) return SSW_E_INVALID;
  int dev = 0, sms = 0;
  SSW_CUDA_TRY(cudaGetDevice(&dev));
  SSW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  HalfGemmParams p = {};
  p.a = a; p.w = w; p.bias = bias; p.out = out; p.M = M; p.N = N; p.K = K;
  p.error = error; p.give_up = give_up;
  const int64_t m_tiles = ceil_div64(M, kHM);
  const int nt = (N + kHN - 1) / kHN;
  p.bn = ((N + nt - 1) / nt + 15) / 16 * 16;
  p.n_tiles = (N + p.bn - 1) / p.bn;
  if (m_tiles * p.n_tiles >= ((int64_t)1 << 30)) return SSW_E_RANGE;
  p.tiles = (int)(m_tiles * p.n_tiles);
  auto kern = dtype == SSW_BF16 ? k_gemm_gelu<__nv_bfloat16> : k_gemm_gelu<__half>;
  SSW_CUDA_TRY(allow_smem(kern));
  SSW_CUDA_TRY(launch_chained(kern, dim3((unsigned)(p.tiles < sms ? p.tiles : sms)), dim3(kHThreads), kHSmem, (cudaStream_t)stream_, p));
  return SSW_OK;
}

extern "C" int ssw_gemm_gelu(const void* a, const void* w, const void* bias, int dtype, void* out, int64_t M, int32_t N, int32_t K,
                             int32_t* error, void* stream) {
  return gemm_gelu(a, w, bias, dtype, out, M, N, K, error, 0, stream);
}
