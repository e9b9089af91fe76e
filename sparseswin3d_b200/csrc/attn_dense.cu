// Fused window attention for windows that hold more voxels than one pack (c > tile), 16-bit inputs,
// head_dim 32: the dense contraction of the path, on the fifth-generation tensor cores (tcgen05,
// accumulators in tensor memory).
//
// Upstream computes such a window like every other: one thread per output element of the c x c
// score block and of the c x hd output block (ops.cu:344-418).  Here a unit of work is one
// (window, head).  Its k and v slices (c x 64 bytes each) are gathered once into shared memory in
// the tensor cores' operand layout and stay there while the window's query rows pass in tiles of
// 128:
//
//   S[128 x 96]  = Q_tile K_tile^T       tcgen05.mma, operands from shared memory, S in tensor memory
//   P            = exp2(S*scale + bias + mask - m)   two threads per query row (tcgen05.ld gives a
//                  thread its part of the row of S), running maximum from 0 and +1e-8 as upstream (ops.cu:137,
//                  164); P goes back to tensor memory in the input type, as the A operand of the next product.
//                  16 bits keep 8 or 11 of a probability, and a row that averages hundreds of keys loses more than the
//                  rounding of the output with that, so the rounding residual is stored beside P and
//                  multiplied with the same V tile (A and B of an MMA must have the same 16-bit
//                  type: an fp16 P against a bf16 V is an illegal instruction)
//   O[128 x 32] += P V_tile              tcgen05.mma, over the key tiles of a query tile; with a running maximum, over one key
//                  tile, and the row's threads add it to the others' sums
//
// Two forms of the softmax.  A tile's scores are bounded by |q| |k| scale + bias, the largest of each over the tile (the
// producers find them while they gather).  While that bound lies below kLimit the exponentials need no maximum:
// upstream's own starts at 0, so with 0 as the reference (fp16: kRef, see there) nothing overflows, the
// result is the same quotient (the denominator relative to 0 is at least 1 wherever a maximum above 0 would have been
// subtracted, and there 1e-8 is below its rounding), no row statistics pass between threads.  The P V products
// of all key tiles (up to 1024 keys, 128 MMAs) add up in one tensor-memory accumulator; the tensor cores cut off where an fp32
// add rounds, some 1e-6 of the sum, two hundred times less than the rounding of the output.  From the first key tile beyond the bound on, the query tile
// goes on with the running maximum, which takes a pass over the scores of its own, and a key tile's sums are drained and added to those before
// in fp32, rounding to nearest.  (Values of either sign a hundred times the sum can meet there.  Two full windows of 9^3, one bias beyond the bound, fp16:
// 0.19 % of the results differ from the exact ones rounded; 0.72 % with one accumulator, scaled where a maximum grows.)  A million voxels, half of
// the 9^3 windows full, six heads of bf16, scores of four times the size: 3.86 ms with that one accumulator, 3.97 so; within the bound 2.28 and 2.30.
//
// Two query tiles are in flight, each a stream of its own: its own issuing warp, scores, P, sums and eight softmax warps, over key tiles that
// both share.  While one stream waits for a hand-over the other has the SM.  Nothing but key tiles and the units' headers
// ties them to one another.  A million voxels, half of the 9^3 windows full, six heads of bf16, in ms: 4.53 with one stream, 128-key tiles and
// MMAs issued from a branch of one lane (there every operand is looked for among the lanes: see the issuer); 2.99 two streams of four
// softmax warps; 2.82 eight softmax warps each (two threads a row); 2.30 MMAs issued from uniform registers; 2.27 the residual
// of P in one mixed-precision instruction; 2.26 the bias slice padded (see there) and staged by the softmax warps (10 000 voxels, 3 heads: 13.6 us
// by the producers ahead of the first rows, 11.5 so).  Bound by issue slots and their latencies: 66 % of them used (13 warp instructions a key, 7.5 of them
// the look-up of the bias, the exponential and the split of P), exponential unit 46 %, shared memory 35 to 60 %; without exponentials
// the time is the same within 3 %.  Floor of the exponential unit: 0.97 ms.
//
// Warp roles (768 threads, one CTA per SM): warps 0-1 issue the MMAs of a stream (one elected lane); warps 2-7 gather rows (plain 16-byte loads by
// voxel id, stored with the 64-byte swizzle the operand descriptors name); warps 8-23 are the softmax rows, eight warps a stream: a
// warp may touch the 32 tensor-memory lanes warp_id % 4 selects, so two warps share each quarter of the query rows and take
// sixteens of keys in turn (they exchange row maxima per key tile beyond the bound and row sums per query tile through shared memory).
// P takes the place of the scores it comes from: of sixteen columns of scores the first eight become P and the others its residual.
// Everything is handed over through mbarriers with bounded waits; on expiry the kernel sets SSW_DEV_TIMEOUT, lets the tensor
// cores drain and frees its tensor memory before it returns.
#include <math.h>

#include "attn_common.cuh"
#include "tcgen05.cuh"

namespace ssw {

template <typename T>
__device__ __forceinline__ float residual(float p, uint32_t h) {   // p less a 16-bit value
  float r;
  if constexpr (std::is_same<T, __nv_bfloat16>::value)
    asm("fma.rn.f32.bf16 %0, %1, %2, %3;" : "=f"(r) : "h"((uint16_t)h), "h"((uint16_t)0xbf80), "f"(p));
  else
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(r) : "h"((uint16_t)h), "h"((uint16_t)0xbc00), "f"(p));
  return r;
}

constexpr int kDQ = 128;       // query rows per tile = MMA M
constexpr int kDK = 96;        // keys per tile
constexpr int kDHD = 32;       // head_dim
constexpr int kDRowB = 64;     // bytes of one q / k / v head slice (32 x 16 bit)
constexpr int kDTileB = kDK * kDRowB;
constexpr int kDMaxKT = 11;    // key tiles in shared memory at most (1024 keys)
constexpr int kDStreams = 2;   // query tiles in flight, each with its own softmax warps, scores and sums
constexpr int kDProd = 6;      // producer warps (with four groups of eight rows each they gather the k and v of a key tile at once)
constexpr int kDParts = 2;     // softmax threads per query row, in different warps: sixteens of a tile's keys in turn
constexpr int kDSoftWarps = 4 * kDParts;  // softmax warps of a stream
constexpr int kDFirstSoft = kDStreams + kDProd;   // a multiple of 4: warp % 4 selects the tensor-memory lanes
constexpr int kDThreads = 32 * (kDFirstSoft + kDStreams * kDSoftWarps);
constexpr int kDSub = 16;      // keys a softmax thread takes at a time = K of an MMA
constexpr int kTmemCols = 512; // per stream: two tiles of scores, which P takes over, the sums O, and what was drained from O
constexpr int kTmemStream = 256, kTmemO = 2 * kDK, kTmemSum = kTmemO + kDHD;
static_assert(kDK % (2 * kDSub) == 0 && kTmemSum + kDHD <= kTmemStream && kDFirstSoft % 4 == 0 && kDTileB % 1024 == 0 &&
                  kDProd * 4 * 8 >= 2 * kDK,
              "");
// Scores (log2 domain, less kRef) up to which probabilities are formed without a maximum: exp2 of it times 1024 keys times
// a v below 2^60 stays far inside fp32, and inside the 16-bit type of P.  The bias slices of the units are stored less
// kRef.  fp16: with q and k of unit variance and 32 channels the bound of a tile is 16 or 17, above 15; where no score of a row
// is above 0, its largest P is then 2^-5 and holds 19 bits with its residual.
template <typename T>
struct DenseFast;
template <>
struct DenseFast<__nv_bfloat16> {
  static constexpr float kLimit = 40.f, kRef = 0.f, kExpMinusRef = 1.f;
  static constexpr uint32_t kMaxV = (127u + 60u) << 7;
};
template <>
struct DenseFast<__half> {
  static constexpr float kLimit = 15.f, kRef = 5.f, kExpMinusRef = 0.03125f;
  static constexpr uint32_t kMaxV = 0x7c00u;
};

// The bias slice in shared memory.  A warp's lanes are consecutive rows of a window, in a full one consecutive positions, and a look-up of the
// warp reads the slice at their codes.  With rows of x a multiple of 32 plus Wx words apart, and planes of y plus Wx Wy,
// consecutive positions lie in consecutive banks; with the table's own strides nearly every look-up takes two passes (51.8 M shared-memory wavefronts
// against 33.6 M over 172 full windows of 9^3 and six heads).  The padded slice takes the room of two plain ones, so it is staged for one head
// (see the units).  A million voxels, half of the 9^3 windows full, six heads of bf16, plain / padded: 2.27 / 2.26 ms (144 blocks for 148),
// the same shifted by four 2.18 / 2.02.  Where the padded slice does not fit, the table's strides stay.
struct BiasShape {
  int wy2, wx2;        // 2 Wy - 1, 2 Wx - 1: the table's own strides are wx2 and wx2 wy2
  int py, pz;          // words between rows of x / planes of y
  int off;             // padded code of the last position
  int floats;
};
inline BiasShape bias_shape(const int32_t w[3], bool padded) {
  BiasShape b;
  b.wy2 = 2 * w[1] - 1;
  b.wx2 = 2 * w[2] - 1;
  b.py = b.wx2 + (padded ? ((w[2] - b.wx2) % 32 + 32) % 32 : 0);
  b.pz = b.wy2 * b.py;
  if (padded) b.pz += ((w[1] * w[2] - b.pz) % 32 + 32) % 32;
  b.off = (w[0] - 1) * b.pz + (w[1] - 1) * b.py + (w[2] - 1);
  b.floats = (2 * b.off + 4) & ~3;
  return b;
}

struct DenseParams {
  const void* qkv;
  OutSet outs;
  int32_t* header;
  const int32_t* bins;        // per-occupancy tables of the plan
  const int32_t* pack_win;
  const int32_t* win_start;
  const int32_t* win_pstart;
  const int32_t* pack_perm;
  const int32_t* pack_meta;
  const float* table;
  int rel_off, H, C, tile, n_per_window, table_rows;
  int n_vox, w_cap;
  int c_cap;                  // rows the shared-memory buffers are sized for (a multiple of kDK)
  int kv_slots, q_bufs;       // key tiles in shared memory; query tiles per stream
  BiasShape bias;
  float scale;
  int use_mask;
};

// Shared memory (byte offsets from a 1024-byte aligned base):
//   [0, 2048)        mbarriers, the tensor-memory address, largest norms of the tiles
//   [2048, 8192)     partial row maxima / sums the softmax threads of a row exchange
//   K, V  kv_slots x 96 x 64 each   (64-byte swizzle), a ring over the key tiles of all units: the next unit's come in
//                    while this one's are in use
//   Q  2 streams x q_bufs x 128 x 64  (64-byte swizzle)
//   the bias slice of the head, pre-multiplied by log2 e
//   per unit (double buffered), per row of its window: the voxel id, 4 x padded relative-position code, region
struct DenseSmem {
  uint32_t k, v, q, bias, vox, rel4, reg, total;
};
__host__ __device__ inline DenseSmem dense_smem(int c_cap, int bias_floats, int kv_slots, int q_bufs) {
  DenseSmem s;
  uint32_t o = 8192u;
  s.k = o; o += (uint32_t)kv_slots * kDTileB;
  s.v = o; o += (uint32_t)kv_slots * kDTileB;
  s.q = o; o += (uint32_t)(kDStreams * q_bufs) * kDQ * kDRowB;
  s.bias = o; o += (uint32_t)bias_floats * 4u;
  s.vox = o; o += 2u * (uint32_t)c_cap * 4u;
  s.rel4 = o; o += 2u * (uint32_t)c_cap * 4u;
  s.reg = o; o += 2u * (uint32_t)c_cap * 4u;
  s.total = o;
  return s;
}
// Key tiles and query buffers to keep in shared memory: twice a full window's key tiles (at most 8) where they fit, at least one
// window's; two query tiles a stream where they fit, else one; the padded bias slice where it fits.  False: nothing fits.
inline bool dense_buffers(int n_per_window, const int32_t w[3], int& c_cap, int& kv_slots, int& q_bufs, BiasShape& bias) {
  const int need = (n_per_window + kDK - 1) / kDK;
  c_cap = need * kDK;
  if (need > kDMaxKT) return false;
  for (q_bufs = 2; q_bufs > 0; --q_bufs)
    for (int padded = 1; padded >= 0; --padded) {
      bias = bias_shape(w, padded != 0);
      for (kv_slots = 2 * need > 8 ? (need > 8 ? need : 8) : 2 * need; kv_slots >= need; --kv_slots)
        if ((size_t)dense_smem(c_cap, bias.floats, kv_slots, q_bufs).total + 1024 <= 227 * 1024) return true;
    }
  return false;
}

template <typename T, bool kMask>
__global__ void __launch_bounds__(kDThreads, 1) k_attn_dense(DenseParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // the operand layouts want 1024-byte aligned tiles: align the base by hand
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const DenseSmem L = dense_smem(p.c_cap, p.bias.floats, p.kv_slots, p.q_bufs);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  uint64_t* kv_full = bars;                    // [kDMaxKT] a key tile is in shared memory
  uint64_t* kv_empty = kv_full + kDMaxKT;      // [kDMaxKT] both streams are done with it
  uint64_t* meta_full = kv_empty + kDMaxKT;    // [2] a unit's header: voxel ids, metadata, bias slice of its head
  uint64_t* meta_empty = meta_full + 2;        // [2]
  uint64_t* drain_bar = meta_empty + 2;        // [1]
  uint64_t* q_full = drain_bar + 1;            // [stream][2]
  uint64_t* q_empty = q_full + 4;              // [stream][2]
  uint64_t* s_full = q_empty + 4;              // [stream][2] scores of a tile in tensor memory
  uint64_t* p_full = s_full + 4;               // [stream][2] P in their place
  uint64_t* pv_done = p_full + 4;              // [stream][2] P V of the tile done: added to O, the tile's columns free
  uint64_t* o_empty = pv_done + 4;             // [stream] a query tile's O has been read (one phase per query tile)
  uint64_t* xbar = o_empty + kDStreams;        // [stream][4] both threads of a quarter's rows have posted their maximum
  uint64_t* lbar = xbar + 4 * kDStreams;       // [stream][4] a query tile's partial row sums have been posted
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(lbar + 4 * kDStreams);
  int* unit_c = reinterpret_cast<int*>(tmem_slot + 1);      // [2] voxels of the unit's window, with its metadata
  // largest squared norms of a tile's rows, one word per producer warp (two of the eight unused)
  float* k_norm = reinterpret_cast<float*>(smem + 768);     // [kDMaxKT][8]; infinite where a v is too large for O
  float* q_norm = k_norm + kDMaxKT * 8;                     // [stream][4][8] by query tile of the stream
  float* b_max = q_norm + kDStreams * 4 * 8;                // [16] largest entry (or 0) of the bias slice, by the warps that staged it
  float* xmax = reinterpret_cast<float*>(smem + 2048);      // [stream][2][kDParts][128] partial row maxima
  float* xsum = xmax + kDStreams * 2 * kDParts * 128;       // [stream][2][128] partial row sums
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int H = p.H, C = p.C;

  // Whether there is any window beyond a pack is a device-side count: a launch that finds none
  // (the usual case on surface-sparse scenes) leaves before it sets anything up.
  grid_dependency_wait();
  // the windows beyond a pack, heaviest first: window slots [ws0, W) of the plan's pack order
  BinTables bins(const_cast<int32_t*>(p.bins), p.n_per_window);
  const int W = min(max(p.header[SSW_H_W], 0), p.w_cap);
  const int ws0 = p.tile + 1 <= p.n_per_window + 1 ? min(max(bins.wstart[p.tile + 1], 0), W) : W;
  const int n_units = (W - ws0) * H;
  // A block's units are u = blockIdx.x, + step, + 2 step, ..., window by window, and the bias slice in shared memory is that of one head: a
  // multiple of the heads of blocks, where that leaves out one block in sixteen at most, never changes heads.  (Head by head over all
  // blocks: 2.39 ms against 2.33 on a million voxels of full windows, six heads; a window's heads then find its rows in L2 no more.)
  const int odd = (int)gridDim.x % H, step = odd * 16 <= (int)gridDim.x ? gridDim.x - odd : gridDim.x;
  if ((int)blockIdx.x >= min(n_units, step)) return;
  if (threadIdx.x == 0) {
    for (int j = 0; j < kDMaxKT; ++j) {
      mbar_init(kv_full + j, kDProd);
      mbar_init(kv_empty + j, kDStreams);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(meta_full + b, kDProd);
      mbar_init(meta_empty + b, kDStreams * (kDSoftWarps + 1));
    }
    for (int b = 0; b < 2 * kDStreams; ++b) {
      mbar_init(q_full + b, kDProd);
      mbar_init(q_empty + b, 1);
      mbar_init(s_full + b, 1);
      mbar_init(p_full + b, kDSoftWarps);
      mbar_init(pv_done + b, 1);
    }
    for (int s = 0; s < kDStreams; ++s) mbar_init(o_empty + s, 4);
    for (int x = 0; x < 4 * kDStreams; ++x) {
      mbar_init(xbar + x, kDParts);
      mbar_init(lbar + x, 1);
    }
    mbar_init(drain_bar, kDStreams);
    mbar_fence_init();
  }
  if (threadIdx.x < kDStreams * kDSoftWarps) b_max[threadIdx.x] = 0.f;
  if (warp == 0) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // A head's bias slice (rows of the table are [code][head]) by `n` threads, eight loads in flight; the largest entry (or 0) of a warp's share.
  const int wyx2 = p.bias.wy2 * p.bias.wx2;
  const bool one_head = step % H == 0;   // the softmax warps stage it before their first unit; else the producers, unit by unit
  auto stage_bias = [&](int h, int t, int n) -> float {
    float* const bs = reinterpret_cast<float*>(smem + L.bias);
    float bm = 0.f;
    for (int i0 = t; i0 < p.table_rows; i0 += n * 8) {
      float v[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const int i = i0 + x * n;
        v[x] = i < p.table_rows ? __ldg(p.table + (int64_t)i * H + h) * kLog2e : 0.f;
      }
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const int i = i0 + x * n, z = i / wyx2, y = (i - z * wyx2) / p.bias.wx2;
        if (i < p.table_rows) bs[z * p.bias.pz + y * p.bias.py + (i - z * wyx2 - y * p.bias.wx2)] = v[x] - DenseFast<T>::kRef;
        bm = v[x] <= 3.0e38f ? fmaxf(bm, v[x]) : INFINITY;
      }
    }
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(bm)));
  };
  bool timed_out = false;
  constexpr float kRef = DenseFast<T>::kRef;
  const int a_fmt_qk = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
  // Every role walks the same units; a unit's query tiles go to the two streams in
  // turn, counted over all units, so a unit of one tile leaves one stream without work in it.

  if (warp < kDStreams) {
    // =========================================== MMA issuer of a stream =======================
    // One lane, two positions in the same sequence of key tiles: `sp`, the next tile whose scores are formed, runs up to
    // two tiles ahead of `pp`, the next one whose P V is (also across query tiles and units).  Within a unit the two go in turn and
    // a wait may suspend the thread.  Scores of the next unit may have to wait for key tiles that come in only after the P V behind
    // them: there the lane takes whichever can go, and sleeps in between (asking without a pause took half of all issue slots
    // of two schedulers, and the softmax warps there were what the others waited for).
    // All lanes walk along, on values that the compiler can see are the same in each (vote and shuffle results, parameters),
    // and one issues: an MMA takes its operands from uniform registers, and from a branch of one lane every operand is first
    // looked for among the lanes, some hundred instructions an MMA.
    const int s = warp;
    const bool leader = elect_one();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0) + s * kTmemStream;
    const int units = __shfl_sync(0xffffffffu, n_units, 0), stride = __shfl_sync(0xffffffffu, step, 0);
    struct Pos {
      uint32_t g, qn;              // key tiles / query tiles of the stream before it
      uint32_t slot, par;          // ring slot of the unit's first key tile, parity of that slot's use
      int u, un, qodd;             // unit, units before it, query tiles of all units before it modulo 2
      int t, j, c;                 // query tile, key tile, the window's voxels (0: not yet read)
    };
    auto ring = [&](uint32_t& slot, uint32_t& par, int n) {
      slot += n;
      if (slot >= (uint32_t)p.kv_slots) {
        slot -= p.kv_slots;
        par ^= 1;
      }
    };
    auto next_unit = [&](Pos& x) {
      ring(x.slot, x.par, (x.c + kDK - 1) / kDK);
      x.qodd ^= ((x.c + kDQ - 1) / kDQ) & 1;
      x.c = 0;
      ++x.un;
      x.u += stride;
    };
    auto advance = [&](Pos& x) {  // true: the unit's last tile of this stream
      ++x.g;
      if (++x.j * kDK < x.c) return false;
      x.j = 0;
      ++x.qn;
      x.t += kDStreams;
      return x.t * kDQ >= x.c;
    };
    auto ready = [&](uint64_t* bar, uint32_t parity, bool wait) -> bool {
      const bool ok = __all_sync(0xffffffffu, wait ? mbar_wait_bounded(bar, parity) : mbar_test(bar, parity));
      timed_out = timed_out || (wait && !ok);
      return ok;
    };
    auto window_of = [&](int un) { return __shfl_sync(0xffffffffu, *reinterpret_cast<volatile int*>(unit_c + (un & 1)), 0); };
    const uint64_t q_desc = smem_desc(smem_u32(smem + L.q) + (uint32_t)(s * p.q_bufs) * (kDQ * kDRowB), 512, 4);
    const uint64_t k_desc = smem_desc(smem_u32(smem + L.k), 512, 4), v_desc = smem_desc(smem_u32(smem + L.v), 512, 4);
    const uint32_t idesc_s = instr_desc(a_fmt_qk, a_fmt_qk, 0, 0);     // (N is added: a window's last key tile has fewer keys)
    const uint32_t idesc_o = instr_desc(a_fmt_qk, a_fmt_qk, 1, kDHD);  // A = P, B = V (MN-major)
    Pos sp = {0, 0, 0, 0, (int)blockIdx.x, 0, 0, 0, 0, 0}, pp = sp;
    uint32_t idle = 0;
    while (pp.u < units && !timed_out) {
      bool moved = false;
      const uint32_t ahead = sp.g - pp.g;
      const bool in_turn = sp.un == pp.un;
      // ---- scores of the next tile
      if (sp.u < units && ahead < 2) {
        if (sp.c == 0 && ready(meta_full + (sp.un & 1), (sp.un >> 1) & 1, in_turn)) {
          sp.c = window_of(sp.un);
          sp.t = (s - sp.qodd) & 1;
          if (sp.t * kDQ >= sp.c) next_unit(sp);   // nothing here for this stream
          moved = true;
        }
        if (sp.c > 0) {
          const uint32_t b = sp.g & 1, qb = p.q_bufs == 2 ? sp.qn & 1 : 0, qpar = p.q_bufs == 2 ? (sp.qn >> 1) & 1 : sp.qn & 1;
          uint32_t slot = sp.slot, par = sp.par;
          ring(slot, par, sp.j);
          // the scores go where the tile two before had its P
          if ((sp.j > 0 || ready(q_full + 2 * s + qb, qpar, in_turn)) && (sp.t >= kDStreams || ready(kv_full + slot, par, in_turn)) &&
              (sp.g < 2 || ready(pv_done + 2 * s + b, ((sp.g >> 1) - 1) & 1, in_turn))) {
            tc_fence_after();
            const int nk16 = (min(kDK, sp.c - sp.j * kDK) + 15) & ~15;
            const uint32_t idesc = idesc_s + ((uint32_t)(nk16 >> 3) << 17);
            const uint64_t qd = q_desc + qb * (kDQ * kDRowB >> 4), kd = k_desc + slot * (kDTileB >> 4);
            const bool q_end = (sp.j + 1) * kDK >= sp.c;  // every S of this query tile has been issued
            if (leader) {
#pragma unroll
              for (int ks = 0; ks < kDHD / 16; ++ks) umma_ss(tm + b * kDK, qd + ks * 2, kd + ks * 2, idesc, ks > 0);
              umma_commit(s_full + 2 * s + b);
              if (q_end) umma_commit(q_empty + 2 * s + qb);
            }
            __syncwarp();
            if (advance(sp)) next_unit(sp);
            moved = true;
          }
        }
      }
      // ---- P V of the oldest tile whose scores have been formed; a unit without tiles of this stream is left behind
      if (pp.un != sp.un || pp.g != sp.g) {
        if (pp.c == 0) {
          pp.c = window_of(pp.un);  // (sp has seen its meta_full)
          pp.t = (s - pp.qodd) & 1;
          pp.j = 0;
        }
        uint32_t slot = pp.slot, par = pp.par;
        ring(slot, par, pp.j);
        if (pp.t * kDQ >= pp.c) {
          // (each phase of kv_empty wants one arrival of each stream: the phase before has completed once the tile is full)
          if (ready(kv_full + slot, par, false)) {
            if (leader) mbar_arrive(kv_empty + slot);
            if (++pp.j * kDK >= pp.c) {
              pp.j = 0;
              if (leader) mbar_arrive(meta_empty + (pp.un & 1));
              next_unit(pp);
            }
            moved = true;
          }
        } else if (pp.g != sp.g) {
          const uint32_t b = pp.g & 1;
          // nothing else can go while the scores are two tiles ahead; O starts over with the query tile
          if (ready(p_full + 2 * s + b, (pp.g >> 1) & 1, ahead >= 2) &&
              (pp.j > 0 || pp.qn == 0 || ready(o_empty + s, (pp.qn - 1) & 1, ahead >= 2))) {
            tc_fence_after();
            const int n16 = (min(kDK, pp.c - pp.j * kDK) + 15) >> 4;
            const uint32_t a = tm + b * kDK;
            const uint64_t vd = v_desc + slot * (kDTileB >> 4);
            const bool kv_end = (pp.t + kDStreams) * kDQ >= pp.c;  // this stream's last use of the key tile
            if (leader) {
#pragma unroll
              for (int ks = 0; ks < kDK / 16; ++ks) {   // P, and its rounding residual beside it
                if (ks < n16) {
                  umma_ts(tm + kTmemO, a + ks * kDSub, vd + ks * (16 * kDRowB >> 4), idesc_o, ks > 0 || pp.j > 0);
                  umma_ts(tm + kTmemO, a + ks * kDSub + kDSub / 2, vd + ks * (16 * kDRowB >> 4), idesc_o, 1);
                }
              }
              umma_commit(pv_done + 2 * s + b);
              if (kv_end) umma_commit(kv_empty + slot);
            }
            __syncwarp();
            if (advance(pp)) {
              if (leader) mbar_arrive(meta_empty + (pp.un & 1));
              next_unit(pp);
            }
            moved = true;
          }
        }
      }
      if (!moved) __nanosleep(100);
      idle = moved ? 0 : idle + 1;
      if (idle > (1u << 20)) timed_out = true;
    }
    // let the tensor cores finish whatever was issued before the tensor memory is given back
    if (leader) umma_commit(drain_bar);
    __syncwarp();
    mbar_wait_bounded(drain_bar, 0);
  } else if (warp < kDFirstSoft) {
    // =========================================== producers ====================================
    const int pw = warp - kDStreams;
    const int chunk = lane & 3, rsub = lane >> 2;
    const T* qkv = reinterpret_cast<const T*>(p.qkv);
    // Four groups of eight 64-byte row pieces at a time: group g is rows [8 g, 8 g + 8) of `part` (0 q, 1 k, 2 v) from row r0 of the
    // window on, zero from row c on, stored with the 64-byte swizzle.  Returns the largest squared norm of this warp's rows (q, k; infinite
    // if one is not finite), or 0 / infinity (v: within kMaxV or not).
    auto gather = [&](const int* wvox, int c, int h, int n_groups, auto place) -> float {
      float top = 0.f;
      uint4 val[4];
      for (int g0 = pw; g0 < n_groups; g0 += kDProd * 4) {
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int gi = g0 + x * kDProd;
          int part, r0, rl;
          unsigned char* dst;
          val[x] = make_uint4(0, 0, 0, 0);
          if (gi < n_groups) {
            place(gi, part, r0, rl, dst);
            const int r = r0 + rl + rsub;
            if (r < c) val[x] = __ldg(reinterpret_cast<const uint4*>(qkv + (int64_t)wvox[r] * 3 * C + part * C + h * kDHD) + chunk);
          }
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int gi = g0 + x * kDProd;
          int part, r0, rl;
          unsigned char* dst;
          if (gi < n_groups) {
            place(gi, part, r0, rl, dst);
            rl += rsub;
            *reinterpret_cast<uint4*>(dst + (size_t)rl * kDRowB + ((chunk ^ ((rl >> 1) & 3)) << 4)) = val[x];
            if (part == 2) {
              const uint32_t vm = __vmaxu2(__vmaxu2(val[x].x & 0x7fff7fffu, val[x].y & 0x7fff7fffu),
                                           __vmaxu2(val[x].z & 0x7fff7fffu, val[x].w & 0x7fff7fffu));
              if (max(vm & 0xffffu, vm >> 16) >= DenseFast<T>::kMaxV) top = INFINITY;
            } else {
              float4 a, b;
              widen8<T>(val[x], a, b);
              float n2 = fmaf(a.x, a.x, fmaf(a.y, a.y, fmaf(a.z, a.z, a.w * a.w))) + fmaf(b.x, b.x, fmaf(b.y, b.y, fmaf(b.z, b.z, b.w * b.w)));
              n2 += __shfl_xor_sync(0xffffffffu, n2, 1);  // the four lanes of a row
              n2 += __shfl_xor_sync(0xffffffffu, n2, 2);
              top = n2 <= 3.0e38f ? fmaxf(top, n2) : INFINITY;  // (NaN as well)
            }
          }
        }
      }
      return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(top)));  // not negative: ordered as integers
    };
    // the window of a unit: a few dependent loads, asked for one unit ahead
    auto unit_window = [&](int u, int& first, int& c) {
      const int ws = W - 1 - u / H;
      const int k = min(max(__ldg(p.pack_win + ws), 0), p.w_cap - 1);
      first = __ldg(p.win_pstart + k);
      c = __ldg(p.win_start + k + 1) - __ldg(p.win_start + k);
    };
    uint32_t qn[kDStreams] = {0, 0};   // query tiles handed to each stream
    uint32_t slot = 0, use = 0;        // ring slot of the next key tile, how often the ring has been gone through
    int un = 0, qodd = 0, first_n = 0, c_n = 0, h_staged = -1;

    unit_window(blockIdx.x, first_n, c_n);
    for (int u = blockIdx.x; u < n_units && !timed_out; u += step, ++un) {
      int first = first_n, c = c_n;
      const int h = u % H;
      if (!(c > p.tile && c <= p.c_cap && first >= 0 && first <= p.n_vox - c)) {
        atomicOr(reinterpret_cast<unsigned*>(p.header + SSW_H_ERROR), SSW_DEV_BAD_PLAN);
        first = 0;   // a one-row window instead: the result is flagged, and every role still finds work
        c = 1;
      }
      if (u + step < n_units) unit_window(u + step, first_n, c_n);
      const int nkt = (c + kDK - 1) / kDK, nqt = (c + kDQ - 1) / kDQ;
      const int mb = un & 1;
      int* wvox = reinterpret_cast<int*>(smem + L.vox) + mb * p.c_cap;
      int* wrel4 = reinterpret_cast<int*>(smem + L.rel4) + mb * p.c_cap;
      int* wreg = reinterpret_cast<int*>(smem + L.reg) + mb * p.c_cap;
      // ---- the window's voxel ids and metadata
      if (un >= 2 && !mbar_wait_asleep(meta_empty + mb, ((un >> 1) - 1) & 1)) { timed_out = true; break; }
      if (pw == 0 && lane == 0) unit_c[mb] = c;
      for (int r = pw * 32 + lane; r < nkt * kDK; r += kDProd * 32) {  // (rows from c on: neutral entries)
        int vx = 0, m = 0;
        if (r < c) {
          vx = __ldg(p.pack_perm + first + r);
          m = __ldg(p.pack_meta + first + r);
        }
        const int code = meta_rel(m), z = code / wyx2, y = (code - z * wyx2) / p.bias.wx2;
        const int at = z * p.bias.pz + y * p.bias.py + (code - z * wyx2 - y * p.bias.wx2);
        const bool ok = (unsigned)vx < (unsigned)p.n_vox && code <= p.rel_off && at <= p.bias.off;
        if (!ok) atomicOr(reinterpret_cast<unsigned*>(p.header + SSW_H_ERROR), SSW_DEV_BAD_PLAN);
        wvox[r] = ok ? vx : 0;
        wrel4[r] = ok ? at * 4 : 0;
        wreg[r] = ok ? meta_region(m) : 0;
      }
      // ---- the head's bias slice (rows of the table are [code][head]), eight loads in flight
      if (!one_head && h != h_staged) {
        // (the unit before is of another head: both streams must be done with it)
        if (un >= 1 && !mbar_wait_asleep(meta_empty + (mb ^ 1), ((un - 1) >> 1) & 1)) { timed_out = true; break; }
        h_staged = h;
        const float top = stage_bias(h, pw * 32 + lane, kDProd * 32);
        if (lane == 0) b_max[pw] = top;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(meta_full + mb);
      // the other producer warps' ids are needed for the gathers below
      if (!mbar_wait_asleep(meta_full + mb, (un >> 1) & 1)) { timed_out = true; break; }
      // ---- key tiles; the first query tile of each stream after the first of them so that the MMAs can start early, the
      // others once all keys are in.  Whatever a wait here is for is work whose tiles have all been handed out before.
      auto query_tile = [&](int t) {
        const int s = (qodd + t) & 1;
        const uint32_t qi = qn[s]++, nb = (uint32_t)p.q_bufs, qb = nb == 2 ? qi & 1 : 0, uses = nb == 2 ? qi >> 1 : qi;
        if (uses >= 1 && !mbar_wait_asleep(q_empty + 2 * s + qb, (uses - 1) & 1)) {
          timed_out = true;
          return;
        }
        unsigned char* dq = smem + L.q + (size_t)(s * p.q_bufs + qb) * (kDQ * kDRowB);
        const float qm = gather(wvox, c, h, kDQ / 8, [&](int gi, int& part, int& r0, int& rl, unsigned char*& dst) {
          part = 0;
          r0 = t * kDQ;
          rl = gi * 8;
          dst = dq;
        });
        if (lane == 0) q_norm[(s * 4 + (qi & 3)) * 8 + pw] = qm;
        fence_async_smem();  // the tensor cores read shared memory through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(q_full + 2 * s + qb);
      };
      for (int j = 0; j < nkt && !timed_out; ++j) {
        if (use > 0 && !mbar_wait_asleep(kv_empty + slot, (use - 1) & 1)) { timed_out = true; break; }
        const int ng = ((min(kDK, c - j * kDK) + 15) & ~15) >> 3;
        unsigned char *dk = smem + L.k + (size_t)slot * kDTileB, *dv = smem + L.v + (size_t)slot * kDTileB;
        const float kn = gather(wvox, c, h, 2 * ng, [&](int gi, int& part, int& r0, int& rl, unsigned char*& dst) {
          part = gi < ng ? 1 : 2;
          r0 = j * kDK;
          rl = (gi < ng ? gi : gi - ng) * 8;
          dst = gi < ng ? dk : dv;
        });
        if (lane == 0) k_norm[slot * 8 + pw] = kn;
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(kv_full + slot);
        if (++slot == (uint32_t)p.kv_slots) {
          slot = 0;
          ++use;
        }
        if (j == 0) {
          for (int t = 0; t < min(nqt, kDStreams) && !timed_out; ++t) query_tile(t);
        }
      }
      for (int t = kDStreams; t < nqt && !timed_out; ++t) query_tile(t);
      qodd ^= nqt & 1;
    }
  } else {
    // =========================================== softmax rows =================================
    const int s = (warp - kDFirstSoft) / kDSoftWarps;
    const int part = ((warp - kDFirstSoft) >> 2) & (kDParts - 1);
    const int sw = warp & 3;                   // tensor-memory lanes [32 sw, 32 sw + 32)
    const int row_in_tile = sw * 32 + lane;
    const uint32_t tm = tmem + ((uint32_t)(sw * 32) << 16) + s * kTmemStream;
    const float qscale = p.scale * kLog2e;
    uint32_t g = 0;    // key tiles of the stream so far
    uint32_t qt = 0;   // query tiles of the stream begun
    uint32_t xn = 0;   // exchanges of maxima so far
    uint32_t slot0 = 0;  // ring slot of the unit's first key tile
    int un = 0, qodd = 0;
    if (one_head) {
      const float top = stage_bias(blockIdx.x % H, threadIdx.x - kDFirstSoft * 32, kDStreams * kDSoftWarps * 32);
      if (lane == 0) b_max[warp - kDFirstSoft] = top;
      asm volatile("bar.sync 1, %0;" ::"n"(kDStreams * kDSoftWarps * 32) : "memory");   // the softmax warps
    }
    for (int u = blockIdx.x; u < n_units && !timed_out; u += step, ++un) {
      const int mb = un & 1;
      if (!mbar_wait_bounded(meta_full + mb, (un >> 1) & 1)) { timed_out = true; break; }
      const int c = *reinterpret_cast<volatile int*>(unit_c + mb), h = u % H;
      const int nkt = (c + kDK - 1) / kDK, nqt = (c + kDQ - 1) / kDQ;
      const int* wvox = reinterpret_cast<const int*>(smem + L.vox) + mb * p.c_cap;
      const int* wrel4 = reinterpret_cast<const int*>(smem + L.rel4) + mb * p.c_cap;
      const int* wreg = reinterpret_cast<const int*>(smem + L.reg) + mb * p.c_cap;
      const uint32_t bias_a = smem_u32(smem + L.bias);
      const uint32_t rel4_a = smem_u32(wrel4), reg_a = smem_u32(wreg);
      float k_max = 0.f;   // largest squared key norm of the unit, known after the stream's first query tile in it
      for (int t = (s - qodd) & 1; t < nqt && !timed_out; t += kDStreams) {
        const int qrow = t * kDQ + row_in_tile;
        const bool live = qrow < c;
        // bias of (me, key j) = slice[(code_me + off) - code_j] in padded codes: my row's base, minus 4 * code_j
        const uint32_t my_bias = bias_a + (uint32_t)(live ? wrel4[qrow] : 0) + (uint32_t)p.bias.off * 4u;
        const int my_region = live ? wreg[qrow] : 0;
        float m = 0.f, l = 0.f;  // scores less kRef: the maximum starts from -kRef (0: ops.cu:137)
        bool fast = true;        // every key tile so far was within the bound
        float k_limit = 0.f;     // largest squared key norm the bound allows for this query tile
        uint32_t slot = slot0;
        for (int j = 0; j < nkt; ++j, ++g) {
          const uint32_t b = g & 1, src = tm + b * kDK;
          const int nk = min(kDK, c - j * kDK);  // valid keys
          if (!mbar_wait_bounded(s_full + 2 * s + b, (g >> 1) & 1)) { timed_out = true; break; }
          tc_fence_after();
          if (j == 0) {
            const float4 q4 = *reinterpret_cast<const float4*>(q_norm + (s * 4 + (qt & 3)) * 8);
            const float2 q2 = *reinterpret_cast<const float2*>(q_norm + (s * 4 + (qt & 3)) * 8 + 4);
            float top = b_max[lane & 15];   // (all of them: a warp's lanes hold every entry twice)
            top = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(top)));
            const float qq = fmaxf(fmaxf(fmaxf(q4.x, q4.y), fmaxf(q4.z, q4.w)), fmaxf(q2.x, q2.y));
            const float lim = (DenseFast<T>::kLimit + kRef - top) / fabsf(qscale);
            k_limit = lim > 0.f && qq <= 3.0e38f ? lim * lim / fmaxf(qq, 1e-30f) : -1.f;
          }
          const bool was_fast = fast;
          if (t < kDStreams) {
            const float4 k4 = *reinterpret_cast<const float4*>(k_norm + slot * 8);
            const float2 k2 = *reinterpret_cast<const float2*>(k_norm + slot * 8 + 4);
            const float top = fmaxf(fmaxf(fmaxf(k4.x, k4.y), fmaxf(k4.z, k4.w)), fmaxf(k2.x, k2.y));
            k_max = fmaxf(k_max, top);
            fast = fast && top <= k_limit;  // the same in every softmax thread
          } else if (j == 0) {
            fast = k_max <= k_limit;
          }
          if (++slot == (uint32_t)p.kv_slots) slot = 0;
          // scores of four keys in the log2 domain: bias from the head's slice, -100 across regions
          auto score4 = [&](const uint32_t* sr, uint32_t key4, float2& lo2, float2& hi2) {
            const int4 kr = lds_v4(rel4_a + key4);
            float2 b0 = make_float2(lds_f32(my_bias - (uint32_t)kr.x), lds_f32(my_bias - (uint32_t)kr.y));
            float2 b1 = make_float2(lds_f32(my_bias - (uint32_t)kr.z), lds_f32(my_bias - (uint32_t)kr.w));
            if constexpr (kMask) {
              const int4 kg = lds_v4(reg_a + key4);
              if (kg.x != my_region) b0.x += -100.0f * kLog2e;
              if (kg.y != my_region) b0.y += -100.0f * kLog2e;
              if (kg.z != my_region) b1.x += -100.0f * kLog2e;
              if (kg.w != my_region) b1.y += -100.0f * kLog2e;
            }
            const float2 qs2 = make_float2(qscale, qscale);
            lo2 = __ffma2_rn(make_float2(__uint_as_float(sr[0]), __uint_as_float(sr[1])), qs2, b0);
            hi2 = __ffma2_rn(make_float2(__uint_as_float(sr[2]), __uint_as_float(sr[3])), qs2, b1);
          };
          float corr = 1.f;
          if (!fast) {
            if (j == 0) m = -kRef;
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
            for (int k = part * kDSub; k < nk; k += kDParts * kDSub) {
              uint32_t sr[kDSub];
              tmem_ldn(src + k, sr);
              tmem_ld_wait();
#pragma unroll
              for (int q4 = 0; q4 < kDSub / 4; ++q4) {
                float2 v0, v1;
                score4(sr + q4 * 4, (uint32_t)(j * kDK + k + q4 * 4) * 4u, v0, v1);
                if (k + q4 * 4 < nk) mx[0] = fmaxf(mx[0], v0.x);   // nothing beyond the window's last voxel
                if (k + q4 * 4 + 1 < nk) mx[1] = fmaxf(mx[1], v0.y);
                if (k + q4 * 4 + 2 < nk) mx[2] = fmaxf(mx[2], v1.x);
                if (k + q4 * 4 + 3 < nk) mx[3] = fmaxf(mx[3], v1.y);
              }
            }
            float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            float* slots = xmax + (s * 2 + (xn & 1)) * (kDParts * 128) + row_in_tile;
            const float corr_sum = slots[part * 128];   // (of the tile before: see below)
            slots[part * 128] = mine;
            __syncwarp();
            if (lane == 0) mbar_arrive(xbar + s * 4 + sw);
            if (!mbar_wait_bounded(xbar + s * 4 + sw, xn & 1)) { timed_out = true; break; }
            ++xn;
            const float m_new = fmaxf(m, fmaxf(mine, slots[(part ^ 1) * 128]));
            corr = fast_exp2(m - m_new);
            m = m_new;
            // The tensor cores cut off where an fp32 add rounds: what they have added up is drained and added to the sums of the
            // tiles before, rounding to nearest, and this tile's product starts from zeros.
            xmax[(s * 2 + (xn & 1)) * (kDParts * 128) + part * 128 + row_in_tile] = corr;   // (the other thread has read what was posted there)
            if (j > 0) {
              if (!mbar_wait_bounded(pv_done + 2 * s + (b ^ 1), ((g - 1) >> 1) & 1)) { timed_out = true; break; }
              tc_fence_after();
              uint32_t part_o[kDHD / kDParts];
              tmem_ldn(tm + kTmemO + part * (kDHD / kDParts), part_o);
              tmem_ld_wait();
              if (j > 1 && !was_fast) {
                uint32_t sum[kDHD / kDParts];
                tmem_ldn(tm + kTmemSum + part * (kDHD / kDParts), sum);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < kDHD / kDParts; ++e)
                  part_o[e] = __float_as_uint(fmaf(__uint_as_float(sum[e]), corr_sum, __uint_as_float(part_o[e])));
              }
              tmem_stn(tm + kTmemSum + part * (kDHD / kDParts), part_o);
#pragma unroll
              for (int e = 0; e < kDHD / kDParts; ++e) part_o[e] = 0;
              tmem_stn(tm + kTmemO + part * (kDHD / kDParts), part_o);
            }
          }
          // P = exp2(s - m) and its rounding residual, written over the scores they come from; packed arithmetic, two keys at a time
          float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
          const float2 neg_m = make_float2(-m, -m);
          auto probabilities = [&](const uint32_t (&sr)[kDSub], int k, auto less_m, auto last) {
            uint32_t hi[kDSub / 2], lo[kDSub / 2];
#pragma unroll
            for (int q4 = 0; q4 < kDSub / 4; ++q4) {
              float2 v2[2];
              score4(sr + q4 * 4, (uint32_t)(j * kDK + k + q4 * 4) * 4u, v2[0], v2[1]);
#pragma unroll
              for (int x = 0; x < 2; ++x) {
                const int jj = q4 * 4 + x * 2;
                const float2 v = decltype(less_m)::value ? __fadd2_rn(v2[x], neg_m) : v2[x];
                float2 pv = make_float2(fast_exp2(v.x), fast_exp2(v.y));
                if (decltype(last)::value) {  // nothing beyond the window's last voxel
                  if (k + jj >= nk) pv.x = 0.f;
                  if (k + jj + 1 >= nk) pv.y = 0.f;
                }
                sum2[x] = __fadd2_rn(sum2[x], pv);
                hi[jj / 2] = pack2<T>(pv.x, pv.y);
                lo[jj / 2] = pack2<T>(residual<T>(pv.x, hi[jj / 2] & 0xffffu), residual<T>(pv.y, hi[jj / 2] >> 16));
              }
            }
            tmem_stn(src + k, hi);
            tmem_stn(src + k + kDSub / 2, lo);
          };
          auto tile = [&](auto less_m) {
#pragma unroll 1
            for (int k = part * kDSub; k < nk; k += kDParts * kDSub) {
              uint32_t sr[kDSub];
              tmem_ldn(src + k, sr);
              tmem_ld_wait();
              if (k + kDSub <= nk) probabilities(sr, k, less_m, std::false_type{});
              else probabilities(sr, k, less_m, std::true_type{});
            }
          };
          if (fast) tile(std::false_type{});
          else tile(std::true_type{});
          l = fmaf(l, corr, (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y));
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full + 2 * s + b);
        }
        if (timed_out) break;
        // ---- the query tile's output, by the one of a row's threads whose turn it is (so that the posted sums of two tiles before have
        // been read: the other thread's own tile lies in between)
        float* sums = xsum + (s * 2 + (qt & 1)) * 128;
        if ((int)(qt & 1) != part) {
          sums[row_in_tile] = l;
          __syncwarp();
          if (lane == 0) mbar_arrive(lbar + s * 4 + sw);
          ++qt;
          continue;
        }
        if (!mbar_wait_bounded(lbar + s * 4 + sw, qt & 1)) { timed_out = true; break; }
        l += sums[row_in_tile];
        uint32_t o[kDHD];
        if (!mbar_wait_bounded(pv_done + 2 * s + ((g - 1) & 1), ((g - 1) >> 1) & 1)) { timed_out = true; break; }
        tc_fence_after();
        tmem_ldn(tm + kTmemO, o);
        tmem_ld_wait();
        if (!fast && nkt > 1) {   // the last key tile's alone: the sums of those before
          const float corr_sum = xmax[(s * 2 + (xn & 1)) * (kDParts * 128) + part * 128 + row_in_tile];
#pragma unroll
          for (int e0 = 0; e0 < kDHD; e0 += 16) {
            uint32_t sum[16];
            tmem_ldn(tm + kTmemSum + e0, sum);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e0 + e] = __float_as_uint(fmaf(__uint_as_float(sum[e]), corr_sum, __uint_as_float(o[e0 + e])));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(o_empty + s);
        // + 1e-8 beside a sum relative to the maximum or 0 (ops.cu:164); one begun within the bound is relative to kRef
        const float eps = m < 0.f ? 1e-8f : 1e-8f * DenseFast<T>::kExpMinusRef;
        const float inv = __frcp_rn(l + eps);
        // A thread holds the four 16-byte pieces of its own row's head slice.  The four lanes of a group trade pieces, so that each store
        // instruction writes whole 64-byte segments, a row's slice from four lanes side by side: on a peer GPU every segment
        // crosses NVLink as a packet of its own.
        uint32_t w[4][4];
#pragma unroll
        for (int e = 0; e < kDHD / 2; ++e)
          w[e >> 2][e & 3] = pack2<T>(__uint_as_float(o[2 * e]) * inv, __uint_as_float(o[2 * e + 1]) * inv);
#pragma unroll
        for (int bit = 1; bit <= 2; bit <<= 1) {
          const bool up = (lane & bit) != 0;
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            if (x & bit) continue;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? w[x][e] : w[x | bit][e], bit);
              if (up) w[x][e] = got;
              else w[x | bit][e] = got;
            }
          }
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int r = t * kDQ + (row_in_tile & ~3) + x;
          if (r < c) {
            const int64_t off = (int64_t)wvox[r] * C + h * kDHD + (lane & 3) * 8;
            for (int d = 0; d < p.outs.n; ++d)
              *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.outs.base[d]) + off) = make_uint4(w[x][0], w[x][1], w[x][2], w[x][3]);
          }
        }
        ++qt;
      }
      slot0 = (slot0 + nkt) % (uint32_t)p.kv_slots;
      qodd ^= nqt & 1;
      __syncwarp();
      if (lane == 0) mbar_arrive(meta_empty + mb);
    }
  }
  if (timed_out) atomicOr(reinterpret_cast<unsigned*>(p.header + SSW_H_ERROR), SSW_DEV_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

int run_attn_dense(const AttnParams& a, const int32_t* bins, const int32_t* win_start, const int32_t* win_pstart,
                   int n_per_window, int dtype, const int32_t rpb_window[3], cudaStream_t stream) {
  DenseParams p = {};
  p.qkv = a.qkv;
  p.outs = a.outs;
  p.header = a.header;
  p.bins = bins;
  p.pack_win = a.pack_win;
  p.win_start = win_start;
  p.win_pstart = win_pstart;
  p.pack_perm = a.pack_perm;
  p.pack_meta = a.pack_meta;
  p.table = a.table;
  p.rel_off = a.rel_off;
  p.H = a.H;
  p.C = a.C;
  p.tile = a.tile;
  p.n_per_window = n_per_window;
  p.table_rows = (2 * rpb_window[0] - 1) * (2 * rpb_window[1] - 1) * (2 * rpb_window[2] - 1);
  p.n_vox = a.n_vox;
  p.w_cap = a.w_cap;
  p.scale = a.scale;
  p.use_mask = a.use_mask;
  if (!dense_buffers(n_per_window, rpb_window, p.c_cap, p.kv_slots, p.q_bufs, p.bias)) return SSW_E_UNSUPPORTED;
  const DenseSmem L = dense_smem(p.c_cap, p.bias.floats, p.kv_slots, p.q_bufs);
  const size_t smem = (size_t)L.total + 1024;  // slack for the 1024-byte alignment of the base
  int dev = 0, sms = 0;
  SSW_CUDA_TRY(cudaGetDevice(&dev));
  SSW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  void (*kern)(DenseParams) =
      dtype == SSW_BF16 ? (p.use_mask ? k_attn_dense<__nv_bfloat16, true> : k_attn_dense<__nv_bfloat16, false>)
                        : (p.use_mask ? k_attn_dense<__half, true> : k_attn_dense<__half, false>);
  SSW_CUDA_TRY(allow_smem(kern));
  SSW_CUDA_TRY(launch_chained(kern, dim3(sms), dim3(kDThreads), smem, stream, p));
  SSW_LAUNCH_CHECK("k_attn_dense");
  return SSW_OK;
}

// Whether run_attn_dense serves this configuration (otherwise the windows beyond a pack stay with
// the second phase of the mma.sync kernel).
bool attn_dense_supported(int head_dim, int n_per_window, const int32_t rpb_window[3]) {
  if (head_dim != kDHD) return false;
  int c_cap, kv_slots, q_bufs;
  BiasShape bias;
  return dense_buffers(n_per_window, rpb_window, c_cap, kv_slots, q_bufs, bias);
}

}  // namespace ssw
