// Fused window attention in fp32 for windows that hold more voxels than one pack (c > tile): a unit of work is
// (window, head, up to 64 of its query rows).
//
// k_attn_fused stages whole rows (q, k, v of all heads, 3 C floats), so from six heads of 32 channels on a pack is 24 rows or fewer and most windows of
// the deeper stages are beyond it: each query tile of 24 rows then takes a block's time alone, walks the window in key tiles of
// 24 rows, and waits at a barrier of the whole block twice for each.  Here a block of four warps stages the k and v slices of one
// head, 64 rows at a time (34 KB in two stages, 16-byte asynchronous copies, the next tile or the next unit's first on its way), and four such
// blocks share an SM, so that one gathers while others work.  Two adjacent lanes hold two query rows, half of the channels each,
// so that what a lane reads of a key serves two rows; warps 0-1 take every second four keys of 64 rows, warps 2-3 the others, and add up
// at the end.  Running maximum from 0 and +1e-8 as upstream (ops.cu:137, 164).
//
// us, with k_attn_fused alone / this kernel and k_attn_fused for the packs (room scenes, windows of 7^3): 10 000 voxels of 34-49 a window, 6 heads 86 /
// 41 + 12; 2 500, 12 heads 74 / 35 + 7; 40 000, 6 heads 180 / 99 + 36; 40 000, 3 heads 93 / 36 + 30; 150 000, 3 heads 225 / 66 + 94; full 9^3 windows,
// 45 700 voxels, 6 heads 1731 / 924 + 13.  Bound by the latency of a row's chain (dot product, maximum, exponential, sum) at 15 warps an
// SM (128 registers; 32 channels spill 40 bytes a thread): issue slots 51 %, shared memory 54 %.  One row on two lanes, 18 warps: 41 and 1096 us (shared memory 77 %: a 16-byte load returns
// 512 bytes a warp however few addresses it names); one row a thread: 55 and 1289; two rows, keys shared among four lanes: 42 and 1073.
#include "attn_common.cuh"

namespace ssw {

constexpr int kTRows = 64;       // query rows of a unit at most, keys of a stage
constexpr int kTThreads = 2 * kTRows;
constexpr int kTBlocks = 4;      // blocks per SM the registers are kept to
constexpr int kTLevels = 16;     // units per (window, head): up to 1023 rows
constexpr int kTSmemMost = 113 * 1024;   // two blocks an SM at least

struct TileParams {
  const float* qkv;
  OutSet outs;
  int32_t* header;
  const int32_t *bins, *pack_win, *win_start, *win_pstart, *pack_perm, *pack_meta;
  const float* table;
  int rel_off, H, C, tile, n_per_window, beyond_rows, table_rows, n_vox, w_cap;
  float scale;
  int use_mask;
};

// Two query rows of a head on two adjacent lanes, half of its channels each.  Lane x forms the probabilities of row x and hands them to its
// neighbour; both add up their channels of both rows.
template <int HH>
struct RowPair {
  float2 q[2][HH / 2], acc[2][HH / 2];
  float m, l;   // of row x
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int e = 0; e < HH / 2; ++e) acc[0][e] = acc[1][e] = q[0][e] = q[1][e] = make_float2(0.f, 0.f);
    m = 0.f;  // upstream's row maximum starts from 0 (ops.cu:137)
    l = 0.f;
  }
  __device__ __forceinline__ void scale(float f0, float f1) {
    const float2 a = make_float2(f0, f0), b = make_float2(f1, f1);
#pragma unroll
    for (int e = 0; e < HH / 2; ++e) {
      acc[0][e] = __fmul2_rn(acc[0][e], a);
      acc[1][e] = __fmul2_rn(acc[1][e], b);
    }
  }
};
// Four keys, `valid` of which exist: `kp` is the lane's half of the first one's k; v sits HD floats further, the metadata at meta_off.
template <int HH, bool kMask, bool kLast>
__device__ __forceinline__ void attend_four(RowPair<HH>& st, const unsigned char* kp, int row_bytes, int meta_off, const unsigned char* table_h, int my_region,
                                            int x, int valid) {
  float s[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float4* kr = reinterpret_cast<const float4*>(kp + u * row_bytes);
    float2 a0 = make_float2(0.f, 0.f), b0 = a0, a1 = a0, b1 = a0;
#pragma unroll
    for (int e = 0; e < HH / 4; ++e) {
      const float4 k = kr[e];
      a0 = __ffma2_rn(st.q[0][2 * e], make_float2(k.x, k.y), a0);
      b0 = __ffma2_rn(st.q[0][2 * e + 1], make_float2(k.z, k.w), b0);
      a1 = __ffma2_rn(st.q[1][2 * e], make_float2(k.x, k.y), a1);
      b1 = __ffma2_rn(st.q[1][2 * e + 1], make_float2(k.z, k.w), b1);
    }
    a0 = __fadd2_rn(a0, b0);
    a1 = __fadd2_rn(a1, b1);
    const float s0 = a0.x + a0.y, s1 = a1.x + a1.y;
    s[u] = (x ? s1 : s0) + __shfl_xor_sync(0xffffffffu, x ? s0 : s1, 1);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int2 km = *reinterpret_cast<const int2*>(kp + u * row_bytes + meta_off);
    s[u] += *reinterpret_cast<const float*>(table_h - km.x);
    if (kMask && my_region != km.y) s[u] += -100.0f * kLog2e;
    if (kLast && u >= valid) s[u] = -INFINITY;
  }
  const float mc = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
  if (__any_sync(0xffffffffu, mc > st.m)) {
    const float m_new = fmaxf(st.m, mc), mine = fast_exp2(st.m - m_new), other = __shfl_xor_sync(0xffffffffu, mine, 1);
    st.m = m_new;
    st.l *= mine;
    st.scale(x ? other : mine, x ? mine : other);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float mine = fast_exp2(s[u] - st.m), other = __shfl_xor_sync(0xffffffffu, mine, 1);
    st.l += mine;
    const float p0 = x ? other : mine, p1 = x ? mine : other;
    const float2 p0_2 = make_float2(p0, p0), p1_2 = make_float2(p1, p1);
    const float4* vr = reinterpret_cast<const float4*>(kp + u * row_bytes + 2 * HH * 4);
#pragma unroll
    for (int e = 0; e < HH / 4; ++e) {
      const float4 v = vr[e];
      st.acc[0][2 * e] = __ffma2_rn(p0_2, make_float2(v.x, v.y), st.acc[0][2 * e]);
      st.acc[0][2 * e + 1] = __ffma2_rn(p0_2, make_float2(v.z, v.w), st.acc[0][2 * e + 1]);
      st.acc[1][2 * e] = __ffma2_rn(p1_2, make_float2(v.x, v.y), st.acc[1][2 * e]);
      st.acc[1][2 * e + 1] = __ffma2_rn(p1_2, make_float2(v.z, v.w), st.acc[1][2 * e + 1]);
    }
  }
}
// Every second four of a stage's keys, from number `kh` on.
template <int HH, bool kMask>
__device__ __forceinline__ void attend_tile(RowPair<HH>& st, const unsigned char* kp, int row_bytes, int meta_off, const unsigned char* table_h, int my_region,
                                            int x, int kh, int keys) {
  for (int k = 4 * kh; k < keys; k += 8) {
    if (k + 4 <= keys) attend_four<HH, kMask, false>(st, kp + k * row_bytes, row_bytes, meta_off, table_h, my_region, x, 4);
    else attend_four<HH, kMask, true>(st, kp + k * row_bytes, row_bytes, meta_off, table_h, my_region, x, keys - k);
  }
}

template <int HD>
struct TileRow { static constexpr int kBytes = 2 * HD * 4 + 16; };   // k | v | metadata; 16 bytes skew the rows across the banks

template <int HD>
__global__ void __launch_bounds__(kTThreads, kTBlocks) k_attn_tiles(TileParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int HH = HD / 2, RB = TileRow<HD>::kBytes, CH = HD / 4, DATA = 2 * HD * 4;
  __shared__ int level_units[kTLevels];
  float* bias = reinterpret_cast<float*>(smem + 2 * kTRows * RB);
  const int H = p.H, C = p.C, tid = threadIdx.x, x = tid & 1, kh = tid / kTRows;   // half of the channels, which of the keys
  if (!tiles_take(p)) return;
  const int r0 = (tid & 32) + (tid >> 1 & 15);   // this thread's query rows of the unit: r0 and r0 + 16
  const float qscale = p.scale * kLog2e;
  // Windows come in pack order by occupancy, so those with more than 64 k rows are the last ones.  Level k holds the units of their query rows
  // number k; the highest level, with the largest windows, comes first, and in each the largest window.
  BinTables bins(const_cast<int32_t*>(p.bins), p.n_per_window);
  const int W = min(max(p.header[SSW_H_W], 0), p.w_cap);
  if (tid < kTLevels) {
    const int more = max(kTRows * (kTLevels - 1 - tid), p.tile) + 1;
    level_units[tid] = more <= p.n_per_window ? (W - min(max(bins.wstart[more], 0), W)) * H : 0;
  }
  __syncthreads();
  int n_units = 0;
  for (int k = 0; k < kTLevels; ++k) n_units += level_units[k];
  // The unit's window: a few dependent loads, asked for one unit ahead, and its first keys while the last ones of the unit before are used.
  struct Unit { int first, c, h, qb; };
  auto find = [&](int u) {
    Unit n;
    int in = u, k = 0;
    while (in >= level_units[k]) in -= level_units[k++];
    n.qb = kTLevels - 1 - k;
    n.h = in % H;
    const int kwin = min(max(__ldg(p.pack_win + (W - 1 - in / H)), 0), p.w_cap - 1);
    n.first = __ldg(p.win_pstart + kwin);
    n.c = __ldg(p.win_start + kwin + 1) - __ldg(p.win_start + kwin);
    return n;
  };
  auto check = [&](Unit& n) {
    if (n.c > p.tile && n.c > kTRows * n.qb && n.c <= p.n_per_window && n.first >= 0 && n.first <= p.n_vox - n.c) return;
    flag_bad_plan(p);
    n.first = 0;
    n.c = 1;
    n.qb = 1;   // a window of one key and no query row
  };
  auto load_tile = [&](const Unit& n, int j, unsigned char* rows) {   // keys 64 j and on
    const int at = n.first + j * kTRows, keys = min(kTRows, n.c - j * kTRows);
    if (tid < ((keys + 3) & ~3)) {
      const int m = tid < keys ? checked_meta(__ldg(p.pack_meta + at + tid), p) : 0;
      *reinterpret_cast<int2*>(rows + tid * RB + DATA) = make_int2(meta_rel(m) * 4, meta_region(m));
    }
#pragma unroll
    for (int i = tid; i < kTRows * 2 * CH; i += kTThreads) {
      const int row = i / (2 * CH), ch = i % (2 * CH), part = 1 + ch / CH;   // 1: k, 2: v
      if (row < ((keys + 3) & ~3)) {   // (zeros up to a whole four: 0 times anything else there could be NaN)
        const int v = row < keys ? checked_voxel(__ldg(p.pack_perm + at + row), p) : 0;
        cp_async16_or_zero(smem_u32(rows + row * RB + ch * 16), p.qkv + (int64_t)v * 3 * C + part * C + n.h * HD + (ch % CH) * 4, row < keys);
      }
    }
  };
  if ((int)blockIdx.x >= n_units) return;
  int h_staged = -1, stage = 0;
  Unit next = find(blockIdx.x);
  check(next);
  load_tile(next, 0, smem);
  cp_async_commit();
  for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
    const Unit cur = next;
    const int c = cur.c, h = cur.h;
    const bool more = u + (int)gridDim.x < n_units;
    if (more) next = find(u + gridDim.x);
    const int nb = (c + kTRows - 1) / kTRows;   // key tiles
    const int q0 = cur.qb * kTRows, q_rows = min(kTRows, c - q0);
    const bool active = (tid & 32) < q_rows;   // of the warp
    RowPair<HH> st;
    st.reset();
    int vox[2] = {-1, -1}, my_region = 0;
    const unsigned char* table_h = reinterpret_cast<const unsigned char*>(bias + p.rel_off);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = r0 + 16 * i;
      if (r >= q_rows) continue;
      vox[i] = checked_voxel(__ldg(p.pack_perm + cur.first + q0 + r), p);
      const int m = checked_meta(__ldg(p.pack_meta + cur.first + q0 + r), p);
      if (i == x) {
        table_h += meta_rel(m) * 4;
        my_region = meta_region(m);
      }
      const float4* src = reinterpret_cast<const float4*>(p.qkv + (int64_t)vox[i] * 3 * C + h * HD + x * HH);
#pragma unroll
      for (int e = 0; e < HH / 4; ++e) {
        const float4 v = __ldg(src + e);
        st.q[i][2 * e] = make_float2(v.x * qscale, v.y * qscale);
        st.q[i][2 * e + 1] = make_float2(v.z * qscale, v.w * qscale);
      }
    }
    if (h != h_staged) {   // (the grid is a multiple of the heads where it can be: a block then stays with one)
      h_staged = h;
#pragma unroll 8
      for (int i = tid; i < p.table_rows; i += kTThreads) bias[i] = __ldg(p.table + (int64_t)i * H + h) * kLog2e;
    }
    for (int j = 0; j < nb; ++j, stage ^= 1) {
      unsigned char* other = smem + (stage ^ 1) * (kTRows * RB);
      if (j + 1 < nb) {
        load_tile(cur, j + 1, other);
      } else if (more) {
        check(next);
        load_tile(next, 0, other);
      }
      cp_async_commit();
      cp_async_wait<1>();
      __syncthreads();
      if (active) {
        const unsigned char* kp = smem + stage * (kTRows * RB) + x * HH * 4;
        const int n = min(kTRows, c - j * kTRows), meta_off = DATA - x * HH * 4;
        if (p.use_mask) attend_tile<HH, true>(st, kp, RB, meta_off, table_h, my_region, x, kh, n);
        else attend_tile<HH, false>(st, kp, RB, meta_off, table_h, 0, x, kh, n);
      }
      __syncthreads();   // the stage may be filled again
    }
    // the two warps of a row put their sums together, through the stage used last
    float* sums = reinterpret_cast<float*>(smem + (stage ^ 1) * (kTRows * RB));   // [HD + 2][kTRows]
    if (kh == 1 && active) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < HH; ++e) sums[(x * HH + e) * kTRows + r0 + 16 * i] = e & 1 ? st.acc[i][e / 2].y : st.acc[i][e / 2].x;
      sums[HD * kTRows + r0 + 16 * x] = st.m;
      sums[(HD + 1) * kTRows + r0 + 16 * x] = st.l;
    }
    __syncthreads();
    if (kh == 0 && active) {
      const float m2 = sums[HD * kTRows + r0 + 16 * x], m_all = fmaxf(st.m, m2);
      float f = fast_exp2(st.m - m_all), f2 = fast_exp2(m2 - m_all);
      const float inv_l = 1.0f / (fmaf(st.l, f, sums[(HD + 1) * kTRows + r0 + 16 * x] * f2) + 1e-8f);  // ops.cu:164
      f *= inv_l;
      f2 *= inv_l;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float g = __shfl_xor_sync(0xffffffffu, f, 1), g2 = __shfl_xor_sync(0xffffffffu, f2, 1);
        const float fi = i == x ? f : g, fi2 = i == x ? f2 : g2;
        float o[HH];
#pragma unroll
        for (int e = 0; e < HH; ++e)
          o[e] = fmaf(e & 1 ? st.acc[i][e / 2].y : st.acc[i][e / 2].x, fi, sums[(x * HH + e) * kTRows + r0 + 16 * i] * fi2);
        if (vox[i] < 0) continue;
        const int64_t off = (int64_t)vox[i] * C + h * HD + x * HH;
        for (int d = 0; d < p.outs.n; ++d)  // the caller's rows, and the same on peer GPUs
#pragma unroll
          for (int e = 0; e < HH / 4; ++e)
            reinterpret_cast<float4*>(reinterpret_cast<float*>(p.outs.base[d]) + off)[e] = make_float4(o[4 * e], o[4 * e + 1], o[4 * e + 2], o[4 * e + 3]);
      }
    }
    __syncthreads();   // (read before the next keys come into that stage)
  }
}

template <int HD>
static size_t tiles_smem(int table_rows) { return 2 * kTRows * TileRow<HD>::kBytes + (((size_t)table_rows * 4 + 15) & ~(size_t)15); }
static int tiles_table(const int32_t w[3]) { return (2 * w[0] - 1) * (2 * w[1] - 1) * (2 * w[2] - 1); }

// Whether a launch of its own for the windows beyond a pack pays.  The host knows how many voxels there are for each window of the dense grid, not how
// many windows are beyond a pack: a launch that finds none costs 2 us.  us, k_attn_fused alone / both kernels, by voxels for each window (7^3, room
// scenes where nothing is said):
// packs of 48 rows (3 heads of 32): 40 000 voxels at 4.0 37 / 37, at 8.4 41 / 43; 150 000 at 4.6 112 / 101, at 10 230 / 162; 10 000 at 7.4 26 / 24; cells drawn
//   evenly, no window beyond a pack, 20 000 at 20 20 / 22, 100 000 at 15 49 / 51;
// 32 (6 of 32): 2000 at 2.0 8.3 / 10.2, 10 000 at 2.6 28 / 24, 40 000 at 4.0 63 / 67, 150 000 at 2.0 161 / 165, at 4.6 308 / 267;
// 24 (8 of 32): 2000 at 2.0 8.0 / 9.4, 10 000 at 2.6 30 / 27, 40 000 at 4.0 94 / 88, 150 000 at 0.7 150 / 152, at 2.0 242 / 233;
// 16 (24 of 16): 2000 at 2.0 22 / 16, 10 000 at 1.0 20 / 22, 40 000 at 4.0 217 / 226, at 8.4 396 / 347, 150 000 at 4.6 1257 / 1322.
// Few voxels leave SMs idle in k_attn_fused's second phase, so the line lies lower there.  With packs of 16 rows, many windows of little more than
// that are better left to the second phase, whose tiles are as small: a unit of 64 rows does a third of its work on 20 (cells drawn evenly, 100 000
// voxels, windows beyond a pack of 19.7 rows on average: 636 / 748; rooms, 23.2 rows 217 / 226, 26.7 396 / 347; both kernels ask the plan: see tiles_take).
bool attn_tiles_pays(const AttnParams& a, int64_t n_windows, int head_dim, const int32_t rpb_window[3], int* beyond_rows) {
  *beyond_rows = 0;
  if (a.n_per_window <= a.tile || (head_dim != 16 && head_dim != 32)) return false;
  if (tiles_smem<32>(tiles_table(rpb_window)) > kTSmemMost) return false;
  const bool few = a.n_vox <= 16384;
  if (a.tile < 24 && !few) *beyond_rows = 26;
  // voxels for four windows
  const int line = a.tile >= 48 ? 24 : a.tile >= 32 ? (few ? 10 : 17) : a.tile >= 24 ? (few ? 10 : 16) : few ? 8 : 28;
  return 4 * (int64_t)a.n_vox >= line * n_windows;
}

template <int HD>
static int launch_tiles(const TileParams& p, cudaStream_t stream) {
  int dev = 0, sms = 0;
  SSW_CUDA_TRY(cudaGetDevice(&dev));
  SSW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const size_t smem = tiles_smem<HD>(p.table_rows);
  int per_sm = (int)((227 * 1024) / (smem + 1024 + 64));
  if (per_sm > kTBlocks) per_sm = kTBlocks;
  const int all = sms * per_sm, grid = all >= p.H ? all / p.H * p.H : all;
  SSW_CUDA_TRY(allow_smem(k_attn_tiles<HD>, kTSmemMost));
  k_attn_tiles<HD><<<grid, kTThreads, smem, stream>>>(p);
  SSW_LAUNCH_CHECK("k_attn_tiles");
  return SSW_OK;
}

int run_attn_tiles(const AttnParams& a, const int32_t* win_start, const int32_t* win_pstart, int head_dim, const int32_t rpb_window[3],
                   cudaStream_t stream) {
  TileParams p = {};
  p.qkv = reinterpret_cast<const float*>(a.qkv);
  p.outs = a.outs;
  p.header = a.header;
  p.bins = a.bins;
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
  p.n_per_window = a.n_per_window;
  p.beyond_rows = a.beyond_rows;
  p.table_rows = tiles_table(rpb_window);
  p.n_vox = a.n_vox;
  p.w_cap = a.w_cap;
  p.scale = a.scale;
  p.use_mask = a.use_mask;
  return head_dim == 16 ? launch_tiles<16>(p, stream) : launch_tiles<32>(p, stream);
}

}  // namespace ssw
