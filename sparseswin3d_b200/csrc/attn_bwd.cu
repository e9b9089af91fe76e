// Backward of the fused window attention: gradients of qkv and of the relative-position bias
// table from the gradient of the output, without materialising the attention matrix.
//
// Upstream differentiates the unfused chain (swin3d_base.py:106-138, 177-188; ops.cu:169-194,
// 422-557): d(softmax) = out * (g - sum_row(out * g)) on the stored COO values, then the blocked
// products rc_cr / rr_rc / cr_rr.  Here the probabilities are recomputed from q and k instead of
// stored (the forward keeps nothing but its output), with the forward's exact definition:
//   s_ij = scale * q_i.k_j + bias[rel_i - rel_j] (- 100 if the regions differ)
//   m_i = max(0, max_j s_ij),  p_ij = exp(s_ij - m_i) / (sum_j exp(s_ij - m_i) + 1e-8)
//   dP_ij = dO_i.v_j,  D_i = sum_j p_ij dP_ij,  dS_ij = p_ij (dP_ij - D_i)
//   dq_i = scale * sum_j dS_ij k_j,  dk_j = scale * sum_i dS_ij q_i,  dv_j = sum_i p_ij dO_i,
//   dbias[rel_i - rel_j, h] += dS_ij
//
// A unit of work is (up to 64 rows, head): the q, k, v and dO slices of its rows are staged in shared
// memory as fp32 and the c x c matrices s and dP are formed there once, so that every product of the
// backward reads shared memory only:
//   scores    : W x parts threads (W = 32 or 64 rows, the row's keys dealt to the parts): s_ij, dP_ij, and the
//               part's own maximum, denominator and sum e dP, combined over the parts once
//   elementwise: P and dS in place; dbias into a shared-memory copy of the head's table column
//   products  : dq (dS, k), dk (dS^T, q), dv (P^T, dO), 16-byte channel chunks dealt to four quarters of the block
// All of it is packed fp32 FMAs (fma.rn.f32x2); probabilities and gradients are never rounded to 16 bits.
//   k_attn_bwd_pack: windows of up to 64 voxels, as many of one occupancy as fit, all of the above in one pass
//   k_attn_bwd_q   : up to 64 query rows of a larger window against all its key tiles with an online maximum:
//                    dq as (A - D B) / (l + 1e-8) with A = sum e dP k, B = sum e k; leaves
//                    (m_i, 1 / (l_i + 1e-8), D_i) per (row, head) for
//   k_attn_bwd_kv  : up to 64 key rows of a larger window against all its query tiles: dk, dv, dbias.
// The units are this file's own, from the plan's bin tables: the plan's tile is what the forward can stage of all heads at once,
// and with 12 heads of 32 channels, 16 rows, three quarters of a block had nothing to do.  The same pairs and channels as 12 heads
// of 500 windows and as 3 heads of 2000, 20 voxels each, fp32: 664 and 117 us in the plan's tiles, 98 and 101 in units; 200 voxels
// each (50 and 200 windows): 1932 and 750, 676 and 660.
// No atomics on the row gradients; the bias gradient of a block is flushed with global atomics at its end.
//
// What bounds it: instruction issue (about 160 fp32 multiply-adds per (query, key, head) in 80 packed ones, and
// 40 16-byte shared-memory reads that broadcast within a window).  Reading the rows from global memory per
// (query, key), one thread per row, it was bound by the latency of those reads at a tenth of the issue rate.
// 150 000 voxels x 3 heads of fp32 (10 voxels a window): 585 -> 310 us; 40 000 x 3 of bf16 (33 to 46 a window, one in
// five beyond a pack): 483 -> 229 us a block.  Measured on the former: 36 % of the issue slots, eight warps a scheduler
// pair; the 70 KB of rows and matrices leave room for two blocks per SM.  Two blocks of 256 threads leave 128 registers a
// thread: with 32 channels of 16 bits k_attn_bwd_q and k_attn_bwd_kv spill 33 and 19 of them, the pack kernel 5.
//
// The plan may be stale (the backward runs long after the forward that built it, possibly after
// the caller rebuilt another plan in the same buffer): item counts, descriptors, voxel ids and
// relative-position codes are held to their bounds exactly as in the forward kernels; a violation
// sets SSW_DEV_BAD_PLAN and is replaced by a harmless value.
#include <math.h>

#include "attn_common.cuh"

namespace ssw {

struct BwdParams {
  const void* qkv;
  const void* grad_out;
  void* dqkv;
  float* dtable;
  float* stats;  // [N * H * 4]: m (log2 domain), 1/(l + 1e-8), D, unused
  int32_t* header;
  const int32_t* bins;          // per-occupancy tables of the plan
  const int4* pack_desc;
  const int32_t* pack_perm;
  const int32_t* pack_meta;
  const float* table;
  int rel_off, H, C, tile;
  int n_per_window;
  int n_vox, pack_cap;  // bounds the kernels hold the plan's voxel ids and item counts to
  float scale;
  int use_mask;
  int table_rows;
  int table_smem;  // the head's column of the table and of its gradient fit in shared memory
};

constexpr int kBwdThreads = 256;
constexpr int kBwdRows = 64;             // rows of a tile at most
constexpr int kBwdMat = kBwdRows + 1;    // pitch of the score matrices: odd, so rows and columns are conflict free
// a staged row: q | k | v | dO, then {relative-position code, region}, 8 B unused: an odd number of 16-byte
// units, so the same chunk of consecutive rows lies in different banks
template <int HD>
constexpr int kBwdPitch = 4 * HD + 4;
constexpr int kBwdPlan = 2 * kBwdRows;       // voxel ids, metadata

// Units of k_attn_bwd_pack: up to kBwdRows rows of whole windows of one occupancy, from the plan's bin tables, whatever the
// plan's tile is (with wide rows the forward's holds 32, 16 or 8 rows, which would leave most of a block idle).
struct BwdUnits {
  int *cnt, *unit, *row;   // by occupancy: windows, units before the first of them, first row
  int n;                   // units in all
  __device__ explicit BwdUnits(int* base) : cnt(base), unit(base + kBwdRows + 4), row(base + 2 * (kBwdRows + 4)), n(0) {}
};

// Units of the kernels for larger windows: (window, kBwdRows rows of it), from the bin tables as well.  The plan's own items,
// every second, fourth or eighth of which would have to be picked out, leave blocks without work where their step and
// a window's number of items have a factor in common (windows of 200, 6 heads: 1166 us against 726).
struct BwdLarge {
  int* unit;   // by occupancy from kBwdRows + 1: units before the first window
  int n, bins; // units, occupancies
};
constexpr int kBwdSmall = 3 * (kBwdRows + 4);   // words of BwdUnits
__host__ __device__ inline int unit_ints(int n_per_window) {
  const int large = (n_per_window - kBwdRows + 4) & ~3;
  return large > kBwdSmall ? large : kBwdSmall;
}

template <int HD>
struct BwdSmem {
  static constexpr int kRows = 0;
  static constexpr int kS = kRows + kBwdRows * kBwdPitch<HD>;
  static constexpr int kDP = kS + kBwdRows * kBwdMat;
  static constexpr int kRed = kDP + kBwdRows * kBwdMat;       // [3][kBwdThreads]
  static constexpr int kPlan = kRed + 3 * kBwdThreads;        // [2][kBwdPlan], double buffered
  static constexpr int kUnits = kPlan + 2 * kBwdPlan;         // BwdUnits or BwdLarge: unit_ints() words
  static __host__ __device__ int table(int n_per_window) { return kUnits + unit_ints(n_per_window); }  // head's bias column, then its gradient
};

// One 16-byte piece of a 16-bit row -> eight floats in shared memory.
template <typename T>
__device__ __forceinline__ void store_wide(float* dst, const uint4& u) {
  float4 a, b;
  widen8<T>(u, a, b);
  reinterpret_cast<float4*>(dst)[0] = a;
  reinterpret_cast<float4*>(dst)[1] = b;
}

// Slices [slot0, slot0 + NS) (0 q, 1 k, 2 v, 3 dO) of `n` rows into the staged rows; vox: their voxel ids
// (shared memory).  fp32 goes by asynchronous copies, 16 bits through registers, four loads in flight.
template <typename T, int HD>
__device__ __forceinline__ void stage_slices(float* rows, const BwdParams& p, int h, const int* vox, int n, int mask) {
  constexpr int E = 16 / (int)sizeof(T), CH = HD / E;
  const T* qkv = reinterpret_cast<const T*>(p.qkv);
  const T* go = reinterpret_cast<const T*>(p.grad_out);
  const int total = n * 4 * CH;
  auto source = [&](int idx, int& row, int& slot, int& ch) -> const uint4* {
    row = idx / (4 * CH);
    const int rem = idx - row * 4 * CH;
    slot = rem / CH;
    ch = rem - slot * CH;
    const int64_t v = vox[row];
    const T* src = slot == 3 ? go + v * p.C + h * HD : qkv + (v * 3 + slot) * p.C + h * HD;
    return reinterpret_cast<const uint4*>(src) + ch;
  };
  if constexpr (sizeof(T) == 4) {
    for (int idx = threadIdx.x; idx < total; idx += kBwdThreads) {
      int row, slot, ch;
      const uint4* src = source(idx, row, slot, ch);
      if (mask >> slot & 1) cp_async16(rows + row * kBwdPitch<HD> + slot * HD + ch * E, src);
    }
    cp_async_commit();
    cp_async_wait<0>();
  } else {
    for (int base = threadIdx.x; base < total; base += 4 * kBwdThreads) {
      uint4 u[4];
      int off[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int idx = base + x * kBwdThreads;
        off[x] = -1;
        if (idx < total) {
          int row, slot, ch;
          const uint4* src = source(idx, row, slot, ch);
          if (mask >> slot & 1) {
            off[x] = row * kBwdPitch<HD> + slot * HD + ch * E;
            u[x] = __ldg(src);
          }
        }
      }
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (off[x] >= 0) store_wide<T>(rows + off[x], u[x]);
    }
  }
}

// Row metadata of the staged rows, from plan metadata words in shared memory.
template <int HD>
__device__ __forceinline__ void stage_meta(float* rows, const int* meta, int n) {
  for (int r = threadIdx.x; r < n; r += kBwdThreads) {
    const int m = meta[r];
    *reinterpret_cast<int2*>(rows + r * kBwdPitch<HD> + 4 * HD) = make_int2(meta_rel(m), meta_region(m));
  }
}

template <int HD>
__device__ __forceinline__ void load_regs(const float* src, float2 (&x)[HD / 2]) {
#pragma unroll
  for (int e = 0; e < HD / 4; ++e) {
    const float4 v = reinterpret_cast<const float4*>(src)[e];
    x[2 * e] = make_float2(v.x, v.y);
    x[2 * e + 1] = make_float2(v.z, v.w);
  }
}
template <int HD>
__device__ __forceinline__ float dot_smem(const float2 (&x)[HD / 2], const float* y) {
  float2 a = make_float2(0.f, 0.f), b = make_float2(0.f, 0.f);
#pragma unroll
  for (int e = 0; e < HD / 4; ++e) {
    const float4 v = reinterpret_cast<const float4*>(y)[e];
    a = __ffma2_rn(x[2 * e], make_float2(v.x, v.y), a);
    b = __ffma2_rn(x[2 * e + 1], make_float2(v.z, v.w), b);
  }
  return (a.x + b.x) + (a.y + b.y);
}

// acc[k] += sum over x in [0, n) of w[x * w_step] * (chunk c0 + k of row x at `src`)
template <int NCH>
__device__ __forceinline__ void weighted_sum(float4 (&acc)[NCH], const float* w, int w_step, const float* src, int pitch, int n) {
  float2 a[2 * NCH];
#pragma unroll
  for (int k = 0; k < NCH; ++k) {
    a[2 * k] = make_float2(acc[k].x, acc[k].y);
    a[2 * k + 1] = make_float2(acc[k].z, acc[k].w);
  }
#pragma unroll 4
  for (int x = 0; x < n; ++x) {
    const float f = w[x * w_step];
    const float2 f2 = make_float2(f, f);
    const float4* r = reinterpret_cast<const float4*>(src + x * pitch);
#pragma unroll
    for (int k = 0; k < NCH; ++k) {
      const float4 v = r[k];
      a[2 * k] = __ffma2_rn(f2, make_float2(v.x, v.y), a[2 * k]);
      a[2 * k + 1] = __ffma2_rn(f2, make_float2(v.z, v.w), a[2 * k + 1]);
    }
  }
#pragma unroll
  for (int k = 0; k < NCH; ++k) acc[k] = make_float4(a[2 * k].x, a[2 * k].y, a[2 * k + 1].x, a[2 * k + 1].y);
}
template <int NCH>
__device__ __forceinline__ void put_chunks(float* dst, const float4 (&v)[NCH], float f) {
#pragma unroll
  for (int k = 0; k < NCH; ++k)
    reinterpret_cast<float4*>(dst)[k] = make_float4(v[k].x * f, v[k].y * f, v[k].z * f, v[k].w * f);
}

// Slices of the staged rows out to dqkv: slot s of a row is part s of its q | k | v gradient.
template <typename T, int HD>
__device__ __forceinline__ void flush_slices(const float* rows, const BwdParams& p, int h, const int* vox, int n, int slot0, int n_slots) {
  constexpr int E = 16 / (int)sizeof(T), CH = HD / E;
  for (int idx = threadIdx.x; idx < n * n_slots * CH; idx += kBwdThreads) {
    const int row = idx / (n_slots * CH), rem = idx - row * n_slots * CH;
    const int slot = slot0 + rem / CH, ch = rem % CH;
    const float* src = rows + row * kBwdPitch<HD> + slot * HD + ch * E;
    T* dst = reinterpret_cast<T*>(p.dqkv) + ((int64_t)vox[row] * 3 + slot) * p.C + h * HD + ch * E;
    const float4 a = reinterpret_cast<const float4*>(src)[0];
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(dst) = a;
    } else {
      const float4 b = reinterpret_cast<const float4*>(src)[1];
      *reinterpret_cast<uint4*>(dst) = make_uint4(pack2<T>(a.x, a.y), pack2<T>(a.z, a.w), pack2<T>(b.x, b.y), pack2<T>(b.z, b.w));
    }
  }
}

// Voxel ids and metadata of `n` plan rows from `row0`, bounds checked, as {ids, metadata} at dst.
__device__ __forceinline__ void stage_plan(int* dst, const BwdParams& p, int row0, int n) {
  for (int r = threadIdx.x; r < n; r += kBwdThreads) {
    dst[r] = checked_voxel(__ldg(p.pack_perm + row0 + r), p);
    dst[kBwdRows + r] = checked_meta(__ldg(p.pack_meta + row0 + r), p);
  }
}

// Fills the table, by one warp (the caller synchronises the block and reads the number of units from cnt[0]).
__device__ __forceinline__ void fill_units(const BwdUnits& t, const BwdParams& p, bool any) {
  const BinTables bins(const_cast<int32_t*>(p.bins), p.n_per_window);
  const int lane = threadIdx.x & 31;
  int before = 0;
  long long rows = 0;
  bool bad = false;
  for (int c0 = 1; c0 <= kBwdRows; c0 += 32) {
    const int c = c0 + lane, wpp = kBwdRows / c;
    int m = any && c <= p.n_per_window ? __ldg(bins.cnt + c) : 0;
    if ((unsigned)m > (unsigned)(p.n_vox / c)) {
      bad = true;
      m = 0;
    }
    const int u = (m + wpp - 1) / wpp;
    const int inc = warp_incl_scan(u);
    t.cnt[c] = m;
    t.unit[c] = before + inc - u;
    t.row[c] = m ? __ldg(bins.rowstart + c) : 0;
    bad = bad || (m > 0 && ((unsigned)t.row[c] >= (unsigned)p.n_vox || m * c > p.n_vox - t.row[c]));
    rows += (long long)m * c;
    before += __shfl_sync(0xffffffffu, inc, 31);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rows += __shfl_xor_sync(0xffffffffu, rows, o);
  if (__any_sync(0xffffffffu, bad) || rows > p.n_vox) {
    if (lane == 0) flag_bad_plan(p);
    before = 0;
  }
  if (lane == 0) t.cnt[0] = before;
}

// Unit u, in descending occupancy: {first row, c, windows, -}
__device__ __forceinline__ int4 unit_desc(int u, const BwdUnits& t) {
  const int v = t.n - 1 - u;
  int lo = 1, hi = kBwdRows;   // largest c whose first unit is not beyond v
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.unit[mid] <= v) lo = mid; else hi = mid - 1;
  }
  const int wpp = kBwdRows / lo, first = (v - t.unit[lo]) * wpp;
  return make_int4(t.row[lo] + first * lo, lo, min(wpp, t.cnt[lo] - first), 0);
}

// The head's bias column (pre-multiplied by log2 e) and a cleared gradient column, or pointers to the tables
// in global memory.
struct BwdTable {
  const float* bias;
  float* grad;
  int step;
  float mul;
};
__device__ __forceinline__ BwdTable open_table(float* t, const BwdParams& p, int h) {
  if (!p.table_smem) return BwdTable{p.table + h, p.dtable + h, p.H, kLog2e};
  for (int i = threadIdx.x; i < p.table_rows; i += kBwdThreads) {
    t[i] = __ldg(p.table + (int64_t)i * p.H + h) * kLog2e;
    t[p.table_rows + i] = 0.f;
  }
  return BwdTable{t, t + p.table_rows, 1, 1.0f};
}
__device__ __forceinline__ void close_table(const BwdTable& t, const BwdParams& p, int h) {
  if (!p.table_smem) return;
  __syncthreads();
  for (int i = threadIdx.x; i < p.table_rows; i += kBwdThreads) {
    const float g = t.grad[i];
    if (g != 0.f) atomicAdd(p.dtable + (int64_t)i * p.H + h, g);
  }
}

// log2-domain score of a (query, key) pair from its raw dot product
__device__ __forceinline__ float pair_score(float qk, float qs, const BwdTable& t, int rel_i_off, int region_i, int2 mj, bool use_mask) {
  float s = fmaf(qk, qs, t.bias[(rel_i_off - mj.x) * t.step] * t.mul);
  if (use_mask && region_i != mj.y) s += -100.0f * kLog2e;
  return s;
}

// Scores of query row r (staged, q and dO in registers) against staged key rows [j0, j1) of the window that
// starts at row `first`: s and dP to the matrices (column = key - col0), returns their maximum.
template <int HD>
__device__ __forceinline__ float score_keys(const float* rows, float* S, float* DP, int r, int first, int j0, int j1, const float2 (&q)[HD / 2],
                                            const float2 (&go)[HD / 2], int2 mi, float qs, int rel_off, const BwdTable& tab, bool use_mask) {
  float mx = -INFINITY;
#pragma unroll 2
  for (int j = j0; j < j1; ++j) {
    const float* kr = rows + (first + j) * kBwdPitch<HD>;
    const int2 mj = *reinterpret_cast<const int2*>(kr + 4 * HD);
    const float s = pair_score(dot_smem<HD>(q, kr + HD), qs, tab, mi.x + rel_off, mi.y, mj, use_mask);
    S[r * kBwdMat + j] = s;
    DP[r * kBwdMat + j] = dot_smem<HD>(go, kr + 2 * HD);
    mx = fmaxf(mx, s);
  }
  return mx;
}

template <typename T, int HD>
__global__ void __launch_bounds__(kBwdThreads, 2) k_attn_bwd_pack(BwdParams p) {
  extern __shared__ __align__(16) float sm[];
  using L = BwdSmem<HD>;
  float *rows = sm + L::kRows, *S = sm + L::kS, *DP = sm + L::kDP, *red = sm + L::kRed;
  int* plan = reinterpret_cast<int*>(sm + L::kPlan);
  grid_dependency_wait();
  const int n_items = checked_count(p.header[SSW_H_PACKS], p);
  const int n_small = min(checked_count(p.header[SSW_H_PACKS_SMALL], p), n_items);
  const int h = (int)blockIdx.x % p.H, g = (int)blockIdx.x / p.H, step = (int)gridDim.x / p.H;
  // the work list is not followed here, but a plan whose list does not hold together is not sound
  for (int x = blockIdx.x * kBwdThreads + threadIdx.x; x < n_items; x += gridDim.x * kBwdThreads)
    checked_desc(__ldg(p.pack_desc + x), p, x < n_small);
  BwdUnits units(reinterpret_cast<int*>(sm + L::kUnits));
  if (threadIdx.x < 32) fill_units(units, p, n_items > 0);
  __syncthreads();
  units.n = units.cnt[0];
  if (g >= units.n) return;
  const BwdTable tab = open_table(sm + L::table(p.n_per_window), p, h);
  const float qs = p.scale * kLog2e;
  const bool use_mask = p.use_mask != 0;
  // heavy units first
  int4 d = unit_desc(g, units);
  stage_plan(plan, p, d.x, d.z * d.y);
  int buf = 0;
  for (int k = g; k < units.n; k += step, buf ^= 1) {
    const int* vox = plan + buf * kBwdPlan;
    const int c = d.y, n = d.z * c;
    __syncthreads();  // ids and metadata are in shared memory; the rows of the unit before have left it
    stage_slices<T, HD>(rows, p, h, vox, n, 15);
    stage_meta<HD>(rows, vox + kBwdRows, n);
    __syncthreads();
    // ids of the next unit, while this one is computed
    if (k + step < units.n) {
      d = unit_desc(k + step, units);
      stage_plan(plan + (buf ^ 1) * kBwdPlan, p, d.x, d.z * d.y);
    }
    const int W = n <= 32 ? 32 : 64, parts = kBwdThreads / W;
    const int r = threadIdx.x & (W - 1), part = threadIdx.x / W;
    const bool on = r < n;
    const int first = on ? r / c * c : 0;
    const int per = (c + parts - 1) >> (W == 32 ? 3 : 2), j0 = min(part * per, c), j1 = min(j0 + per, c);
    float m = 0.f, l = 0.f, dn = 0.f;  // this part's maximum (from 0), denominator, sum of e dP
    const int2 mi = *reinterpret_cast<const int2*>(rows + (on ? r : 0) * kBwdPitch<HD> + 4 * HD);
    if (on) {
      float2 q[HD / 2], go[HD / 2];
      load_regs<HD>(rows + r * kBwdPitch<HD>, q);
      load_regs<HD>(rows + r * kBwdPitch<HD> + 3 * HD, go);
      m = fmaxf(m, score_keys<HD>(rows, S, DP, r, first, j0, j1, q, go, mi, qs, p.rel_off, tab, use_mask));
      for (int j = j0; j < j1; ++j) {
        const float e = fast_exp2(S[r * kBwdMat + j] - m);
        S[r * kBwdMat + j] = e;
        l += e;
        dn = fmaf(e, DP[r * kBwdMat + j], dn);
      }
    }
    red[threadIdx.x] = m;
    red[kBwdThreads + threadIdx.x] = l;
    red[2 * kBwdThreads + threadIdx.x] = dn;
    __syncthreads();
    if (on) {
      float mt = 0.f, lt = 0.f, dt = 0.f;
      for (int x = 0; x < parts; ++x) mt = fmaxf(mt, red[x * W + r]);
      for (int x = 0; x < parts; ++x) {
        const float f = fast_exp2(red[x * W + r] - mt);
        lt = fmaf(f, red[kBwdThreads + x * W + r], lt);
        dt = fmaf(f, red[2 * kBwdThreads + x * W + r], dt);
      }
      const float inv = 1.0f / (lt + 1e-8f);
      const float D = dt * inv, f = fast_exp2(m - mt) * inv;
      for (int j = j0; j < j1; ++j) {
        const float pij = S[r * kBwdMat + j] * f;
        const float ds = pij * (DP[r * kBwdMat + j] - D);
        S[r * kBwdMat + j] = pij;
        DP[r * kBwdMat + j] = ds;
        const int relj = *reinterpret_cast<const int*>(rows + (first + j) * kBwdPitch<HD> + 4 * HD);
        atomicAdd(tab.grad + (mi.x + p.rel_off - relj) * tab.step, ds);
      }
    }
    __syncthreads();
    // three products of HD / 4 chunks each, dealt to four quarters (with W = 32 the upper half of the block is idle)
    constexpr int Q = HD / 4, NA = 3 * Q / 4, NB = Q - NA, NC = Q / 2;
    const float* ds_row = DP + r * kBwdMat;                          // dS[r][j]
    const float* ds_col = DP + first * kBwdMat + (r - first);        // dS[first + i][r]
    const float* p_col = S + first * kBwdMat + (r - first);
    const float* win = rows + first * kBwdPitch<HD>;
    float4 big[NA] = {}, half_[NC] = {}, small[NB] = {};
    const int P = kBwdPitch<HD>;
    if (on) {
      if (part == 0) {
        weighted_sum<NA>(big, ds_row, 1, win + HD, P, c);
      } else if (part == 1) {
        weighted_sum<NB>(small, ds_row, 1, win + HD + 4 * NA, P, c);
        weighted_sum<NC>(half_, ds_col, kBwdMat, win, P, c);
      } else if (part == 2) {
        weighted_sum<NC>(half_, ds_col, kBwdMat, win + 4 * NC, P, c);
        weighted_sum<NB>(small, p_col, kBwdMat, win + 3 * HD, P, c);
      } else if (part == 3) {
        weighted_sum<NA>(big, p_col, kBwdMat, win + 3 * HD + 4 * NB, P, c);
      }
    }
    __syncthreads();
    // results take the place of the rows they were made from: q <- dq, k <- dk, v <- dv
    if (on) {
      float* o = rows + r * P;
      if (part == 0) {
        put_chunks<NA>(o, big, p.scale);
      } else if (part == 1) {
        put_chunks<NB>(o + 4 * NA, small, p.scale);
        put_chunks<NC>(o + HD, half_, p.scale);
      } else if (part == 2) {
        put_chunks<NC>(o + HD + 4 * NC, half_, p.scale);
        put_chunks<NB>(o + 2 * HD, small, 1.0f);
      } else if (part == 3) {
        put_chunks<NA>(o + 2 * HD + 4 * NB, big, 1.0f);
      }
    }
    __syncthreads();
    flush_slices<T, HD>(rows, p, h, vox, n, 0, 3);
  }
  close_table(tab, p, h);
}

// Fills the table; the whole block calls it.  `scratch`: 24 words.
__device__ __forceinline__ BwdLarge fill_large(int* unit, int* scratch, const BwdParams& p, bool any) {
  const BinTables bins(const_cast<int32_t*>(p.bins), p.n_per_window);
  constexpr int kPer = (kMaxPerWindow - kBwdRows + kBwdThreads - 1) / kBwdThreads;
  const int nb = p.n_per_window - kBwdRows, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int u[kPer], sum = 0;
  long long rows = 0;
  bool bad = false;
#pragma unroll
  for (int x = 0; x < kPer; ++x) {
    const int i = threadIdx.x * kPer + x, c = kBwdRows + 1 + i;
    int m = any && i < nb ? __ldg(bins.cnt + c) : 0;
    if ((unsigned)m > (unsigned)(p.n_vox / c)) {
      bad = true;
      m = 0;
    }
    u[x] = m * ((c + kBwdRows - 1) / kBwdRows);
    sum += u[x];
    rows += (long long)m * c;
  }
  const int inc = warp_incl_scan(sum);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rows += __shfl_xor_sync(0xffffffffu, rows, o);
  long long* row_sum = reinterpret_cast<long long*>(scratch);
  int* unit_sum = scratch + 2 * (kBwdThreads / 32);
  if (lane == 31) {
    row_sum[warp] = rows;
    unit_sum[warp] = inc;
  }
  bad = __syncthreads_or(bad);
  int at = inc - sum, n = 0;
  rows = 0;
#pragma unroll
  for (int w = 0; w < kBwdThreads / 32; ++w) {
    if (w < warp) at += unit_sum[w];
    n += unit_sum[w];
    rows += row_sum[w];
  }
#pragma unroll
  for (int x = 0; x < kPer; ++x) {
    const int i = threadIdx.x * kPer + x;
    if (i < nb) unit[i] = at;
    at += u[x];
  }
  if (bad || rows > p.n_vox) {
    if (threadIdx.x == 0) flag_bad_plan(p);
    n = 0;
  }
  __syncthreads();
  return BwdLarge{unit, n, nb};
}

// Unit u, in descending occupancy: {first row of the window, its voxels, first row of the unit within it, -}
__device__ __forceinline__ int4 large_desc(int u, const BwdLarge& t, const BwdParams& p) {
  const BinTables bins(const_cast<int32_t*>(p.bins), p.n_per_window);
  const int v = t.n - 1 - u;
  int lo = 0, hi = t.bins - 1;   // last occupancy whose first unit is not beyond v
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.unit[mid] <= v) lo = mid; else hi = mid - 1;
  }
  const int c = kBwdRows + 1 + lo, tiles = (c + kBwdRows - 1) / kBwdRows, q = v - t.unit[lo], w = q / tiles;
  const int first = __ldg(bins.rowstart + c);
  if (first >= 0 && first <= p.n_vox - c && w * c <= p.n_vox - c - first) return make_int4(first + w * c, c, (q - w * tiles) * kBwdRows, 0);
  flag_bad_plan(p);
  return make_int4(0, 1, 0, 0);   // a one-row window
}

// Query tiles of windows of more than kBwdRows voxels.
template <typename T, int HD>
__global__ void __launch_bounds__(kBwdThreads, 2) k_attn_bwd_q(BwdParams p) {
  extern __shared__ __align__(16) float sm[];
  using L = BwdSmem<HD>;
  float *rows = sm + L::kRows, *S = sm + L::kS, *DP = sm + L::kDP, *red = sm + L::kRed;
  int* plan = reinterpret_cast<int*>(sm + L::kPlan);
  grid_dependency_wait();
  const int n_items = checked_count(p.header[SSW_H_PACKS], p);
  const int h = (int)blockIdx.x % p.H, g = (int)blockIdx.x / p.H, step = (int)gridDim.x / p.H;
  const BwdLarge large = fill_large(reinterpret_cast<int*>(sm + L::kUnits), reinterpret_cast<int*>(red), p, n_items > 0);
  if (g >= large.n) return;
  const BwdTable tab = open_table(sm + L::table(p.n_per_window), p, h);
  const float qs = p.scale * kLog2e;
  const bool use_mask = p.use_mask != 0;
  const int P = kBwdPitch<HD>;
  constexpr int NC = HD / 8;
  for (int k = g; k < large.n; k += step) {
    const int4 d = large_desc(k, large, p);
    const int c = d.y, r0 = d.z, n = min(kBwdRows, c - r0);
    const int r = threadIdx.x & 63, part = threadIdx.x >> 6;
    const bool on = r < n;
    __syncthreads();
    stage_plan(plan, p, d.x + r0, n);
    __syncthreads();
    stage_slices<T, HD>(rows, p, h, plan, n, 1 | 8);
    stage_meta<HD>(rows, plan + kBwdRows, n);
    __syncthreads();
    const int2 mi = *reinterpret_cast<const int2*>(rows + (on ? r : 0) * P + 4 * HD);
    float2 q[HD / 2], go[HD / 2];
    load_regs<HD>(rows + (on ? r : 0) * P, q);
    load_regs<HD>(rows + (on ? r : 0) * P + 3 * HD, go);
    float m = 0.f, l = 0.f, dn = 0.f;  // of the whole row, kept by all its threads
    float4 acc[NC] = {};               // parts 0, 1: chunks of A; 2, 3: chunks of B
    for (int k0 = 0; k0 < c; k0 += kBwdRows) {
      const int nk = min(kBwdRows, c - k0);
      __syncthreads();  // everyone is done with the key tile before
      stage_plan(plan + kBwdPlan, p, d.x + k0, nk);
      __syncthreads();
      stage_slices<T, HD>(rows, p, h, plan + kBwdPlan, nk, 2 | 4);
      stage_meta<HD>(rows, plan + kBwdPlan + kBwdRows, nk);
      __syncthreads();
      const int per = (nk + 3) / 4, j0 = min(part * per, nk), j1 = min(j0 + per, nk);
      float mx = m;
      if (on) mx = fmaxf(mx, score_keys<HD>(rows, S, DP, r, 0, j0, j1, q, go, mi, qs, p.rel_off, tab, use_mask));
      red[threadIdx.x] = mx;
      __syncthreads();
      const float m_new = fmaxf(fmaxf(red[r], red[64 + r]), fmaxf(red[128 + r], red[192 + r]));
      const float corr = fast_exp2(m - m_new);
      float lp = 0.f, dp = 0.f;
      if (on) {
        for (int j = j0; j < j1; ++j) {
          const float e = fast_exp2(S[r * kBwdMat + j] - m_new);
          const float edp = e * DP[r * kBwdMat + j];
          S[r * kBwdMat + j] = e;
          DP[r * kBwdMat + j] = edp;
          lp += e;
          dp += edp;
        }
      }
      red[kBwdThreads + threadIdx.x] = lp;
      red[2 * kBwdThreads + threadIdx.x] = dp;
      __syncthreads();
      const float *rl = red + kBwdThreads + r, *rd = red + 2 * kBwdThreads + r;
      l = fmaf(l, corr, (rl[0] + rl[64]) + (rl[128] + rl[192]));
      dn = fmaf(dn, corr, (rd[0] + rd[64]) + (rd[128] + rd[192]));
      m = m_new;
#pragma unroll
      for (int x = 0; x < NC; ++x) acc[x] = make_float4(acc[x].x * corr, acc[x].y * corr, acc[x].z * corr, acc[x].w * corr);
      if (on) weighted_sum<NC>(acc, (part < 2 ? DP : S) + r * kBwdMat, 1, rows + HD + (part & 1) * 4 * NC, P, nk);
    }
    const float inv = 1.0f / (l + 1e-8f), D = dn * inv;
    // dq = (A - D B) / (l + 1e-8): B through the k slot, the result in the q slot
    __syncthreads();
    if (on && part >= 2) put_chunks<NC>(rows + r * P + HD + (part & 1) * 4 * NC, acc, D);
    __syncthreads();
    if (on && part < 2) {
      const float* db = rows + r * P + HD + part * 4 * NC;
#pragma unroll
      for (int x = 0; x < NC; ++x) {
        const float4 v = reinterpret_cast<const float4*>(db)[x];
        acc[x] = make_float4(acc[x].x - v.x, acc[x].y - v.y, acc[x].z - v.z, acc[x].w - v.w);
      }
      put_chunks<NC>(rows + r * P + part * 4 * NC, acc, inv * p.scale);
      if (part == 0) reinterpret_cast<float4*>(p.stats)[(int64_t)(d.x + r0 + r) * p.H + h] = make_float4(m, inv, D, 0.f);
    }
    __syncthreads();
    flush_slices<T, HD>(rows, p, h, plan, n, 0, 1);
  }
}

// Key tiles of windows of more than kBwdRows voxels.
template <typename T, int HD>
__global__ void __launch_bounds__(kBwdThreads, 2) k_attn_bwd_kv(BwdParams p) {
  extern __shared__ __align__(16) float sm[];
  using L = BwdSmem<HD>;
  float *rows = sm + L::kRows, *S = sm + L::kS, *DP = sm + L::kDP, *red = sm + L::kRed;
  int* plan = reinterpret_cast<int*>(sm + L::kPlan);
  grid_dependency_wait();  // the row statistics come from the kernel this one is chained behind
  const int n_items = checked_count(p.header[SSW_H_PACKS], p);
  const int h = (int)blockIdx.x % p.H, g = (int)blockIdx.x / p.H, step = (int)gridDim.x / p.H;
  const BwdLarge large = fill_large(reinterpret_cast<int*>(sm + L::kUnits), reinterpret_cast<int*>(red), p, n_items > 0);
  if (g >= large.n) return;
  const BwdTable tab = open_table(sm + L::table(p.n_per_window), p, h);
  const float qs = p.scale * kLog2e;
  const bool use_mask = p.use_mask != 0;
  const int P = kBwdPitch<HD>;
  constexpr int NC = HD / 8;
  for (int k = g; k < large.n; k += step) {
    const int4 d = large_desc(k, large, p);
    const int c = d.y, r0 = d.z, n = min(kBwdRows, c - r0);
    const int r = threadIdx.x & 63, part = threadIdx.x >> 6;
    const bool on = r < n;
    __syncthreads();
    stage_plan(plan, p, d.x + r0, n);
    __syncthreads();
    stage_slices<T, HD>(rows, p, h, plan, n, 2 | 4);
    stage_meta<HD>(rows, plan + kBwdRows, n);
    __syncthreads();
    const int2 mj = *reinterpret_cast<const int2*>(rows + (on ? r : 0) * P + 4 * HD);
    float2 kr[HD / 2], vr[HD / 2];
    load_regs<HD>(rows + (on ? r : 0) * P + HD, kr);
    load_regs<HD>(rows + (on ? r : 0) * P + 2 * HD, vr);
    float4 acc[NC] = {};  // parts 0, 1: chunks of dk; 2, 3: chunks of dv
    for (int q0 = 0; q0 < c; q0 += kBwdRows) {
      const int nq = min(kBwdRows, c - q0);
      __syncthreads();  // everyone is done with the query tile before
      stage_plan(plan + kBwdPlan, p, d.x + q0, nq);
      float4* st = reinterpret_cast<float4*>(red);  // [64] row statistics
      if (threadIdx.x < nq) st[threadIdx.x] = reinterpret_cast<const float4*>(p.stats)[(int64_t)(d.x + q0 + threadIdx.x) * p.H + h];
      __syncthreads();
      stage_slices<T, HD>(rows, p, h, plan + kBwdPlan, nq, 1 | 8);
      stage_meta<HD>(rows, plan + kBwdPlan + kBwdRows, nq);
      __syncthreads();
      const int per = (nq + 3) / 4, i0 = min(part * per, nq), i1 = min(i0 + per, nq);
      if (on) {
#pragma unroll 2
        for (int i = i0; i < i1; ++i) {
          const float* qr = rows + i * P;
          const int2 mi = *reinterpret_cast<const int2*>(qr + 4 * HD);
          const float4 t = st[i];
          const float s = pair_score(dot_smem<HD>(kr, qr), qs, tab, mi.x + p.rel_off, mi.y, mj, use_mask);
          const float pij = fast_exp2(s - t.x) * t.y;
          const float ds = pij * (dot_smem<HD>(vr, qr + 3 * HD) - t.z);
          S[i * kBwdMat + r] = pij;
          DP[i * kBwdMat + r] = ds;
          atomicAdd(tab.grad + (mi.x + p.rel_off - mj.x) * tab.step, ds);
        }
      }
      __syncthreads();
      if (on) weighted_sum<NC>(acc, (part < 2 ? DP : S) + r, kBwdMat, rows + (part < 2 ? 0 : 3 * HD) + (part & 1) * 4 * NC, P, nq);
    }
    __syncthreads();
    if (on) put_chunks<NC>(rows + r * P + (part < 2 ? HD : 2 * HD) + (part & 1) * 4 * NC, acc, part < 2 ? p.scale : 1.0f);
    __syncthreads();
    flush_slices<T, HD>(rows, p, h, plan, n, 1, 2);
  }
  close_table(tab, p, h);
}

template <typename T, int HD>
static int launch_bwd(const BwdParams& p, cudaStream_t stream) {
  int dev = 0, sms = 0;
  SSW_CUDA_TRY(cudaGetDevice(&dev));
  SSW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const size_t smem = sizeof(float) * ((size_t)BwdSmem<HD>::table(p.n_per_window) + (p.table_smem ? 2 * (size_t)p.table_rows : 0));
  void (*kerns[3])(BwdParams) = {k_attn_bwd_pack<T, HD>, k_attn_bwd_q<T, HD>, k_attn_bwd_kv<T, HD>};
  // two blocks per SM, every block on one head throughout (it keeps that head's table column)
  const unsigned grid = (unsigned)(p.H * (2 * sms > p.H ? 2 * sms / p.H : 1));
  for (int k = 0; k < (p.n_per_window > kBwdRows ? 3 : 1); ++k) {
    SSW_CUDA_TRY(allow_smem(kerns[k]));
    SSW_CUDA_TRY(launch_chained(kerns[k], dim3(grid), dim3(kBwdThreads), smem, stream, p));
  }
  return SSW_OK;
}

}  // namespace ssw

using namespace ssw;

extern "C" int64_t ssw_attn_fused_bwd_workspace_floats(int64_t n_vox, int32_t heads) { return n_vox * heads * 4; }

extern "C" int ssw_attn_fused_bwd(const void* qkv, const void* grad_out, int dtype, int32_t heads, int32_t head_dim,
                                  const ssw_plan_layout* L, const int32_t* plan, const float* table,
                                  const int32_t rpb_window[3], float scale, int use_mask, void* dqkv, float* dtable,
                                  float* workspace, void* stream_) {
  if (!L || !plan || !table || !rpb_window || heads <= 0 || head_dim <= 0) return SSW_E_INVALID;
  if (L->n_vox == 0) return SSW_OK;
  if (!qkv || !grad_out || !dqkv || !dtable || !workspace) return SSW_E_INVALID;
  const int elt = dtype == SSW_F32 ? 4 : (dtype == SSW_BF16 || dtype == SSW_F16) ? 2 : 0;
  if (!elt) return SSW_E_INVALID;
  if ((head_dim * elt) % 16) return SSW_E_UNSUPPORTED;
  const uintptr_t align = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(grad_out) |
                          reinterpret_cast<uintptr_t>(dqkv) | reinterpret_cast<uintptr_t>(workspace);
  if (align & 15) return SSW_E_INVALID;
  BwdParams p;
  p.qkv = qkv;
  p.grad_out = grad_out;
  p.dqkv = dqkv;
  p.dtable = dtable;
  p.stats = workspace;
  p.header = const_cast<int32_t*>(plan + L->off_header);
  p.n_vox = (int)L->n_vox;
  p.pack_cap = (int)L->pack_cap;
  p.bins = plan + L->off_bins;
  p.pack_desc = reinterpret_cast<const int4*>(plan + L->off_pack_desc);
  p.pack_perm = plan + L->off_pack_perm;
  p.pack_meta = plan + L->off_pack_meta;
  p.table = table;
  p.rel_off = ((rpb_window[0] - 1) * (2 * rpb_window[1] - 1) + (rpb_window[1] - 1)) * (2 * rpb_window[2] - 1) +
              (rpb_window[2] - 1);
  p.H = heads;
  p.C = heads * head_dim;
  p.tile = L->tile_rows;
  p.scale = scale;
  p.use_mask = use_mask;
  p.n_per_window = L->n_per_window;
  p.table_rows = (2 * rpb_window[0] - 1) * (2 * rpb_window[1] - 1) * (2 * rpb_window[2] - 1);
  // two blocks per SM with both columns: 113 KB a block, 70 of them rows and matrices
  p.table_smem = p.table_rows <= 5000;
  if (p.tile > kBwdRows) return SSW_E_INVALID;
  cudaStream_t stream = (cudaStream_t)stream_;
  if (dtype == SSW_F32) {
    if (head_dim == 16) return launch_bwd<float, 16>(p, stream);
    if (head_dim == 32) return launch_bwd<float, 32>(p, stream);
  } else if (dtype == SSW_BF16) {
    if (head_dim == 16) return launch_bwd<__nv_bfloat16, 16>(p, stream);
    if (head_dim == 32) return launch_bwd<__nv_bfloat16, 32>(p, stream);
  } else {
    if (head_dim == 16) return launch_bwd<__half, 16>(p, stream);
    if (head_dim == 32) return launch_bwd<__half, 32>(p, stream);
  }
  return SSW_E_UNSUPPORTED;
}
