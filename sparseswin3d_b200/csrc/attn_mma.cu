// Fused window attention for 16-bit inputs (bf16 / fp16) on packs of sparse windows (mma.sync): a unit of work is 16 row slots of a pack, by one
// warp and in its registers.  (With 32 channels a head not quite: 20 warps leave 96, and 80 to 120 bytes a thread are spilled, 170 with windows beyond
// a pack; with 16 none.)
//
// The plan is *padded*: inside a pack every window gets a run of row slots rounded up to 1, 2, 4, 8, 16, 32, 48 or 64, so 16 slots hold whole windows
// (several when c < 16) or a 16-row slice of one window.  Softmax keeps upstream's semantics: the maximum starts at 0, the denominator gets
// +1e-8 (ops.cu:137, 164); bias from a copy of the table in shared memory (pre-multiplied by log2 e), -100 shift mask.  Values that are not finite:
// upstream confines them to their own window; here a k or v row that holds Inf or NaN also spoils the other windows that share its 16
// slots (the mask is added to the score, p is multiplied with v, and neither Inf - Inf nor 0 * Inf is 0).  Windows beyond a pack come here as well where the tcgen05 kernel does not serve them
// (16 channels a head, or a bias table too large): 16 query rows and a head at a time, key blocks in turn.
//
// The queries of 16 slots against their own window's keys, 16 at a time, are m16n8k16 products, and the fragments are loaded from the voxel
// rows themselves.  Lane t of a row's four takes channels [4 t, 4 t + 4) and [16 + 4 t, 16 + 4 t + 4) of the head for both operands of Q K^T,
// 8 bytes each, where the instruction's own order would have it read 4 bytes in four places: a product sums sixteen consecutive channels all the
// same, whichever of them a lane brings.  (16 bytes a lane, channels [8 t, 8 t + 8), would put other channels into the two sums, and with that
// other roundings: the 16-bit output of a stage of two blocks moves by 2e-4.  It is no
// faster: 47.5 us at 150 000 voxels, 3 heads, 43.8 shifted, for 47.6 and 43.5.)  A row of v is loaded 16 bytes a lane (8 for
// 16 channels) and becomes the other operand of P V by transposing its 8 x 8 blocks (movmatrix), which
// leaves a lane with the same eight channels of the output: one 16-byte store a row, four lanes side by side.
//
// us, with whole rows copied to shared memory by one bulk copy each and read from there by ldmatrix / so (rooms, windows of 7^3, shifted): 150 000 voxels,
// 3 heads of 32 bf16 48.8 / 45.5, 6 heads 82.7 / 65.8, 12 heads of 16 143 / 97, 3 of 16 40 / 35; 150 000 voxels of 23 a window 71 / 66; 4 x 33 333, 6 heads
// of 16 fp16 with the windows beyond a pack 37 / 32; 2 000 10.3 / 8.3; 100 000, windows of 5^3, fp16 30.6 / 26.  Windows beyond a pack alone, 79 000
// voxels in half-full 9^3 windows, heads of 16, bf16: 6 heads 675 / 553, 12 1373 / 1287, shifted 919 / 726; not so 3 heads 289 / 300 and 12 of fp16 1170 / 1257,
// where the rows of a window that all warps read from shared memory at a time had been the better form (with the next keys' rows asked for ahead 296 and
// 1229, but 12 heads shifted 774; with a window's query rows on neighbouring warps 309 and 1298).  Bound by instructions and their
// latencies: 18 M warp instructions at 150 000 x 3 heads (22.4 M before), 44 % of the issue slots with 20 warps an SM.  16 warps of 128 registers
// 46 us (4 x 33 333: 44), 24 of 80 49 us; the rows of the next head asked for ahead in registers 45, the next unit's rows brought into L2 46.
#include "attn_common.cuh"
#include "tcgen05.cuh"

namespace ssw {

constexpr int kTableMost = 160 * 1024;   // bytes of a bias table in shared memory
constexpr int kPackThreads = 640;        // one block per SM: 96 registers a thread, one copy of the bias table
constexpr int kPackWindow = 127;         // window number of unused slots (bits 5..11 of a slot's word)
constexpr int kPackWindowBits = 127 << 5;

template <typename T>
__device__ __forceinline__ void pack_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}
// The same, starting from zeros.
template <typename T>
__device__ __forceinline__ void pack_mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  }
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}

__device__ __forceinline__ float less_bf16(float p, uint32_t h) {   // p less a bf16 value
  float r;
  asm("fma.rn.f32.bf16 %0, %1, %2, %3;" : "=f"(r) : "h"((uint16_t)h), "h"((uint16_t)0xbf80), "f"(p));
  return r;
}

// A lane's part of a row's head slice: HD / 4 elements.
template <int HD>
struct RowPart { uint32_t x[HD / 8]; };
template <typename T, int HD>
__device__ __forceinline__ RowPart<HD> load_part(const T* row) {
  RowPart<HD> r;
  if constexpr (HD == 32) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(row));
    r.x[0] = v.x; r.x[1] = v.y; r.x[2] = v.z; r.x[3] = v.w;
  } else {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(row));
    r.x[0] = v.x; r.x[1] = v.y;
  }
  return r;
}

// The same of q or k: a product of sixteen channels takes consecutive ones, four from each lane of a row.
template <typename T, int HD>
__device__ __forceinline__ RowPart<HD> load_operand(const T* row) {
  RowPart<HD> r;
#pragma unroll
  for (int ks = 0; ks < HD / 16; ++ks) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(row + 16 * ks));
    r.x[2 * ks] = v.x; r.x[2 * ks + 1] = v.y;
  }
  return r;
}

// Sixteen query rows of a head: rows lane / 4 ("lo") and lane / 4 + 8 ("hi") and their running softmax.
template <int HD>
struct PackRows {
  RowPart<HD> q_lo, q_hi;
  float o[HD / 8][4];
  float m_lo, m_hi, l_lo, l_hi;
};

// One block of sixteen keys: rows lane / 4 of k_lo, v_lo and lane / 4 + 8 of k_hi, v_hi.  add_lo, add_hi: bias and masks of the lo / hi row against
// this lane's four score columns, log2 domain.  kOnly: there is no other block.
template <typename T, int HD, bool kOnly>
__device__ __forceinline__ void pack_block(PackRows<HD>& u, const RowPart<HD>& k_lo, const RowPart<HD>& k_hi, const RowPart<HD>& v_lo,
                                           const RowPart<HD>& v_hi, const float (&add_lo)[4], const float (&add_hi)[4], float qscale) {
  float s0[4], s1[4];
  pack_mma0<T>(s0, u.q_lo.x[0], u.q_hi.x[0], u.q_lo.x[1], u.q_hi.x[1], k_lo.x[0], k_lo.x[1]);
  pack_mma0<T>(s1, u.q_lo.x[0], u.q_hi.x[0], u.q_lo.x[1], u.q_hi.x[1], k_hi.x[0], k_hi.x[1]);
#pragma unroll
  for (int ks = 1; ks < HD / 16; ++ks) {
    pack_mma<T>(s0, u.q_lo.x[2 * ks], u.q_hi.x[2 * ks], u.q_lo.x[2 * ks + 1], u.q_hi.x[2 * ks + 1], k_lo.x[2 * ks], k_lo.x[2 * ks + 1]);
    pack_mma<T>(s1, u.q_lo.x[2 * ks], u.q_hi.x[2 * ks], u.q_lo.x[2 * ks + 1], u.q_hi.x[2 * ks + 1], k_hi.x[2 * ks], k_hi.x[2 * ks + 1]);
  }
  float a[4], b[4];   // scores of the lo / hi row
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a[j] = fmaf(j < 2 ? s0[j] : s1[j - 2], qscale, add_lo[j]);
    b[j] = fmaf(j < 2 ? s0[j + 2] : s1[j], qscale, add_hi[j]);
  }
  // the row maximum starts from 0 (ops.cu:137)
  float mx_lo = fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3])), mx_hi = fmaxf(fmaxf(b[0], b[1]), fmaxf(b[2], b[3]));
  mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 1));
  mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 1));
  mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 2));
  mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 2));
  if constexpr (kOnly) {
    u.m_lo = fmaxf(mx_lo, 0.f);
    u.m_hi = fmaxf(mx_hi, 0.f);
    u.l_lo = u.l_hi = 0.f;
  } else {
    const float n_lo = fmaxf(u.m_lo, mx_lo), n_hi = fmaxf(u.m_hi, mx_hi);
    if (__any_sync(0xffffffffu, n_lo != u.m_lo || n_hi != u.m_hi)) {
      const float c_lo = fast_exp2(u.m_lo - n_lo), c_hi = fast_exp2(u.m_hi - n_hi);
      u.l_lo *= c_lo;
      u.l_hi *= c_hi;
#pragma unroll
      for (int n = 0; n < HD / 8; ++n) {
        u.o[n][0] *= c_lo; u.o[n][1] *= c_lo;
        u.o[n][2] *= c_hi; u.o[n][3] *= c_hi;
      }
      u.m_lo = n_lo;
      u.m_hi = n_hi;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a[j] = fast_exp2(a[j] - u.m_lo);
    b[j] = fast_exp2(b[j] - u.m_hi);
  }
  u.l_lo += (a[0] + a[1]) + (a[2] + a[3]);
  u.l_hi += (b[0] + b[1]) + (b[2] + b[3]);
  const uint32_t p0 = pack2<T>(a[0], a[1]), p1 = pack2<T>(b[0], b[1]), p2 = pack2<T>(a[2], a[3]), p3 = pack2<T>(b[2], b[3]);
  // bf16 keeps 8 bits of a probability, and a row that averages many keys loses more than the rounding of its output with that: the
  // rounding residual goes through a second product
  constexpr bool kSplitP = std::is_same<T, __nv_bfloat16>::value;
  uint32_t r0 = 0, r1 = 0, r2 = 0, r3 = 0;
  if constexpr (kSplitP) {
    r0 = pack2<T>(less_bf16(a[0], p0 & 0xffffu), less_bf16(a[1], p0 >> 16));
    r1 = pack2<T>(less_bf16(b[0], p1 & 0xffffu), less_bf16(b[1], p1 >> 16));
    r2 = pack2<T>(less_bf16(a[2], p2 & 0xffffu), less_bf16(a[3], p2 >> 16));
    r3 = pack2<T>(less_bf16(b[2], p3 & 0xffffu), less_bf16(b[3], p3 >> 16));
  }
#pragma unroll
  for (int n = 0; n < HD / 8; ++n) {
    const uint32_t b0 = transpose8x8(v_lo.x[n]), b1 = transpose8x8(v_hi.x[n]);
    if constexpr (kOnly) pack_mma0<T>(u.o[n], p0, p1, p2, p3, b0, b1);
    else pack_mma<T>(u.o[n], p0, p1, p2, p3, b0, b1);
    if constexpr (kSplitP) pack_mma<T>(u.o[n], r0, r1, r2, r3, b0, b1);
  }
}

// Additive mask of a (query, key) pair of slots: -inf across windows, -100 across shift-mask regions, else 0.
template <bool kMask>
__device__ __forceinline__ float pack_mask(int a, int b) {
  const int x = a ^ b;
  return (x & kPackWindowBits) ? -INFINITY : kMask && (x & 31) ? -100.0f * kLog2e : 0.f;
}

// kBig: windows beyond a pack as well (as a branch of one kernel they cost the packs 10 %: registers).
template <typename T, int HD, bool kTableSmem, bool kMask, bool kBig>
__global__ void __launch_bounds__(kPackThreads, 1) k_attn_mma(AttnParams p) {
  extern __shared__ __align__(16) float table_s[];
  __shared__ uint64_t tbar;
  const int tile = p.tile, C = p.C, H = p.H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qr = lane >> 2, qt = lane & 3;
  const float qscale = p.scale * kLog2e;
  const T* qkv = reinterpret_cast<const T*>(p.qkv) + qt * 4;
  const int v_off = 2 * C + qt * (HD / 4 - 4);   // from a lane's first channels of q to those of v
  if (threadIdx.x == 0) {
    mbar_init(&tbar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  grid_dependency_wait();
  const int n_items = checked_count(p.header[SSW_H_PACKS], p);
  const int n_small = min(checked_count(p.header[SSW_H_PACKS_SMALL], p), n_items);
  // Units 16-slot tile by tile, the largest windows first (the work list ascends), dealt out across the SMs; where there are fewer than
  // warps, the heads of a tile are dealt out as well.
  const int per_item = tile >> 4, n_warps = (int)gridDim.x * (kPackThreads / 32);
  const int parts = min(H, max(1, n_warps / max(n_small * per_item, 1)));
  const int n_units = n_small * per_item * parts;
  struct Unit {
    int slot0, h0;       // first slot of the tile, first head
    int4 d;
    int vox[2], info[2]; // slots lane and lane + 32 of the pack: voxel (-1: none), and region | window << 5 | relative-position code << 16
  };
  auto unit_of = [&](int u, int& item, int& slot0, int& h0) {
    const int t = parts == 1 ? u : u / parts;
    h0 = u - t * parts;
    item = per_item == 4 ? t >> 2 : t / per_item;
    slot0 = (t - item * per_item) * 16;
  };
  auto fetch_desc = [&](int u) {   // of unit u, which exists
    int item, slot0, h0;
    unit_of(u, item, slot0, h0);
    return __ldg(p.pack_desc + (n_small - 1 - item));
  };
  // slot -> window of the pack and row of it (more than 32 slots a window: a pack of one)
  auto split_slot = [&](int slot, int cpad, int& wl, int& ii) {
    wl = cpad > 32 ? 0 : slot >> (31 - __clz(cpad));
    ii = slot - wl * cpad;
  };
  auto fetch = [&](int u, const int4& desc) {
    Unit n;
    int item;
    unit_of(u, item, n.slot0, n.h0);
    n.d = checked_desc(desc, p, true);
    const int c = n.d.y, cpad = slots_of_window(c, 1);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int slot = lane + 32 * k;
      int wl, ii;
      split_slot(slot, cpad, wl, ii);
      n.vox[k] = -1;
      n.info[k] = 0;
      if (slot < tile && wl < n.d.z && ii < c) {
        const int row = n.d.x + wl * c + ii;
        n.vox[k] = __ldg(p.pack_perm + row);
        n.info[k] = __ldg(p.pack_meta + row);
      }
    }
    return n;
  };
  auto settle = [&](Unit& n) {   // what was fetched, held to its bounds
    const int c = n.d.y, cpad = slots_of_window(c, 1);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int slot = lane + 32 * k;
      int wl, ii;
      split_slot(slot, cpad, wl, ii);
      const bool on = slot < tile && wl < n.d.z && ii < c;
      n.vox[k] = on ? checked_voxel(n.vox[k], p) : -1;
      const int m = on ? checked_meta(n.info[k], p) : 0;
      n.info[k] = on ? meta_region(m) | (wl << 5) | (meta_rel(m) << 16) : kPackWindow << 5;
    }
  };
  auto of_slot = [&](const int (&r)[2], int block, int x) { return __shfl_sync(0xffffffffu, (block & 32) ? r[1] : r[0], (block & 16) + x); };
  auto store = [&](const PackRows<HD>& r, int q_lo, int q_hi, int h) {
    float ll = r.l_lo, lh = r.l_hi;   // in four lanes each
    ll += __shfl_xor_sync(0xffffffffu, ll, 1);
    lh += __shfl_xor_sync(0xffffffffu, lh, 1);
    ll += __shfl_xor_sync(0xffffffffu, ll, 2);
    lh += __shfl_xor_sync(0xffffffffu, lh, 2);
    const float inv_lo = __frcp_rn(ll + 1e-8f), inv_hi = __frcp_rn(lh + 1e-8f);  // ops.cu:164
    uint32_t lo[HD / 8], hi[HD / 8];
#pragma unroll
    for (int n = 0; n < HD / 8; ++n) {
      lo[n] = pack2<T>(r.o[n][0] * inv_lo, r.o[n][1] * inv_lo);
      hi[n] = pack2<T>(r.o[n][2] * inv_hi, r.o[n][3] * inv_hi);
    }
    const int64_t o_lo = (int64_t)q_lo * C + h * HD + qt * (HD / 4), o_hi = (int64_t)q_hi * C + h * HD + qt * (HD / 4);
    for (int x = 0; x < p.outs.n; ++x) {  // the caller's rows, and the same on peer GPUs
      T* out = reinterpret_cast<T*>(p.outs.base[x]);
      if constexpr (HD == 32) {
        if (q_lo >= 0) *reinterpret_cast<uint4*>(out + o_lo) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        if (q_hi >= 0) *reinterpret_cast<uint4*>(out + o_hi) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      } else {
        if (q_lo >= 0) *reinterpret_cast<uint2*>(out + o_lo) = make_uint2(lo[0], lo[1]);
        if (q_hi >= 0) *reinterpret_cast<uint2*>(out + o_hi) = make_uint2(hi[0], hi[1]);
      }
    }
  };
  auto begin = [&](PackRows<HD>& r) {
#pragma unroll
    for (int n = 0; n < HD / 8; ++n) r.o[n][0] = r.o[n][1] = r.o[n][2] = r.o[n][3] = 0.f;
    r.m_lo = r.m_hi = r.l_lo = r.l_hi = 0.f;
  };

  // Under way ahead of their use: the descriptor two units ahead, voxel ids and metadata one.
  const int first_u = warp * (int)gridDim.x + (int)blockIdx.x;
  int u = first_u;
  int4 desc = make_int4(0, 1, 0, 0);
  if (u < n_units) desc = fetch_desc(u);
  Unit next = {};
  if (u < n_units) next = fetch(u, desc);
  if (u + n_warps < n_units) desc = fetch_desc(u + n_warps);
  if constexpr (kTableSmem) {
    const bool ok = stage_table(table_s, p.table, p.table_floats, threadIdx.x, kPackThreads, &tbar);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) {
        atomicOr(reinterpret_cast<unsigned*>(p.header + SSW_H_ERROR), SSW_DEV_TIMEOUT);
        mbar_wait_bounded(&tbar, 0);   // the copy must not outlive the block
      }
      return;
    }
  }
  const uint32_t table_a = kTableSmem ? smem_u32(table_s) : 0u;
  const int row_b = H * 4;   // bytes between rows of the table
  auto bias = [&](int at) {  // by byte offset
    if constexpr (kTableSmem) return lds_f32(table_a + (uint32_t)at);
    else return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(p.table) + at)) * kLog2e;
  };
  // ---- windows beyond a pack, unless the tcgen05 kernel takes them: 16 query rows and a head, the largest windows first; their keys' voxel ids and
  // metadata come in one block ahead
  const int n_big = kBig ? (n_items - n_small) * per_item * H : 0;
  for (int v = first_u; v < n_big; v += n_warps) {
    const int t = v / H, h = v - t * H, item = t / per_item, sub = t - item * per_item;
    const int4 d = checked_desc(__ldg(p.pack_desc + (n_items - 1 - item)), p, false);
    const int c = d.y, q0 = (-d.z - 1) * tile + sub * 16, q_end = min((-d.z - 1) * tile + tile, c);
    if (q0 >= q_end) continue;
    auto row_of = [&](int r, bool on, int& vox, int& info) {   // lanes 0..15
      vox = -1;
      info = kPackWindow << 5;
      if (lane < 16 && on) {
        vox = checked_voxel(__ldg(p.pack_perm + d.x + r), p);
        const int m = checked_meta(__ldg(p.pack_meta + d.x + r), p);
        info = meta_region(m) | (meta_rel(m) << 16);
      }
    };
    int q_vox, q_info, k_vox, k_info;
    row_of(q0 + lane, q0 + lane < q_end, q_vox, q_info);
    row_of(lane, lane < c, k_vox, k_info);
    const int me_lo = __shfl_sync(0xffffffffu, q_info, qr), me_hi = __shfl_sync(0xffffffffu, q_info, qr + 8);
    const int q_lo = __shfl_sync(0xffffffffu, q_vox, qr), q_hi = __shfl_sync(0xffffffffu, q_vox, qr + 8), some = __shfl_sync(0xffffffffu, q_vox, 0);
    const int row_lo = ((me_lo >> 16) + p.rel_off) * row_b + h * 4, row_hi = ((me_hi >> 16) + p.rel_off) * row_b + h * 4;
    const int64_t row_e = (int64_t)3 * C;
    PackRows<HD> r;
    r.q_lo = load_operand<T, HD>(qkv + (q_lo < 0 ? some : q_lo) * row_e + h * HD);
    r.q_hi = load_operand<T, HD>(qkv + (q_hi < 0 ? some : q_hi) * row_e + h * HD);
    begin(r);
    for (int k0 = 0; k0 < c; k0 += 16) {
      const int vox = k_vox, info = k_info;
      row_of(k0 + 16 + lane, k0 + 16 + lane < c, k_vox, k_info);
      const int n_lo = __shfl_sync(0xffffffffu, vox, qr), n_hi = __shfl_sync(0xffffffffu, vox, qr + 8);
      const T *klo = qkv + (n_lo < 0 ? some : n_lo) * row_e + h * HD, *khi = qkv + (n_hi < 0 ? some : n_hi) * row_e + h * HD;
      const RowPart<HD> k_lo = load_operand<T, HD>(klo + C), k_hi = load_operand<T, HD>(khi + C);
      const RowPart<HD> v_lo = load_part<T, HD>(klo + v_off), v_hi = load_part<T, HD>(khi + v_off);
      float add_lo[4], add_hi[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int km = __shfl_sync(0xffffffffu, info, (j >> 1) * 8 + qt * 2 + (j & 1)), off = (km >> 16) * row_b;
        add_lo[j] = bias(row_lo - off) + pack_mask<kMask>(km, me_lo);
        add_hi[j] = bias(row_hi - off) + pack_mask<kMask>(km, me_hi);
      }
      pack_block<T, HD, false>(r, k_lo, k_hi, v_lo, v_hi, add_lo, add_hi, qscale);
    }
    store(r, q_lo, q_hi, h);
  }
  // ---- packs
  for (; u < n_units; u += n_warps) {
    Unit cur = next;
    settle(cur);
    if (u + n_warps < n_units) next = fetch(u + n_warps, desc);
    if (u + 2 * n_warps < n_units) desc = fetch_desc(u + 2 * n_warps);
    const int c = cur.d.y, cpad = slots_of_window(c, 1), slot0 = cur.slot0;
    if (slot0 >= cur.d.z * cpad) continue;
    const int me_lo = of_slot(cur.info, slot0, qr), me_hi = of_slot(cur.info, slot0, qr + 8);
    const int q_lo = of_slot(cur.vox, slot0, qr), q_hi = of_slot(cur.vox, slot0, qr + 8);
    const int row_lo = ((me_lo >> 16) + p.rel_off) * row_b, row_hi = ((me_hi >> 16) + p.rel_off) * row_b;
    // An unused slot reads the rows of the tile's first one, which is never unused: its probability is 0 beside values of a window of the tile, and
    // as a query it is not stored.
    const int some = of_slot(cur.vox, slot0, 0);
    const int64_t row_e = (int64_t)3 * C;
    const T *lo = qkv + (q_lo < 0 ? some : q_lo) * row_e + cur.h0 * HD, *hi = qkv + (q_hi < 0 ? some : q_hi) * row_e + cur.h0 * HD;
    if (cpad <= 16) {   // the tile's slots are its keys: offsets and masks are the same for every head
      int at_lo[4], at_hi[4];
      float mask_lo[4], mask_hi[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int km = of_slot(cur.info, slot0, (j >> 1) * 8 + qt * 2 + (j & 1)), off = (km >> 16) * row_b - cur.h0 * 4;
        at_lo[j] = row_lo - off;
        at_hi[j] = row_hi - off;
        mask_lo[j] = pack_mask<kMask>(km, me_lo);
        mask_hi[j] = pack_mask<kMask>(km, me_hi);
      }
      for (int h = cur.h0; h < H; h += parts, lo += parts * HD, hi += parts * HD) {
        PackRows<HD> r;
        r.q_lo = load_operand<T, HD>(lo);
        r.q_hi = load_operand<T, HD>(hi);
        const RowPart<HD> k_lo = load_operand<T, HD>(lo + C), k_hi = load_operand<T, HD>(hi + C);
        const RowPart<HD> v_lo = load_part<T, HD>(lo + v_off), v_hi = load_part<T, HD>(hi + v_off);
        float add_lo[4], add_hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          add_lo[j] = bias(at_lo[j]) + mask_lo[j];
          add_hi[j] = bias(at_hi[j]) + mask_hi[j];
          at_lo[j] += parts * 4;
          at_hi[j] += parts * 4;
        }
        pack_block<T, HD, true>(r, k_lo, k_hi, v_lo, v_hi, add_lo, add_hi, qscale);
        store(r, q_lo, q_hi, h);
      }
    } else {
      const int kbase = slot0 / cpad * cpad, blocks = cpad >> 4;
      for (int h = cur.h0; h < H; h += parts, lo += parts * HD, hi += parts * HD) {
        PackRows<HD> r;
        r.q_lo = load_operand<T, HD>(lo);
        r.q_hi = load_operand<T, HD>(hi);
        begin(r);
        for (int kb = 0; kb < blocks; ++kb) {
          const int block = kbase + kb * 16, n_lo = of_slot(cur.vox, block, qr), n_hi = of_slot(cur.vox, block, qr + 8);
          const T *klo = qkv + (n_lo < 0 ? some : n_lo) * row_e + h * HD, *khi = qkv + (n_hi < 0 ? some : n_hi) * row_e + h * HD;
          const RowPart<HD> k_lo = load_operand<T, HD>(klo + C), k_hi = load_operand<T, HD>(khi + C);
          const RowPart<HD> v_lo = load_part<T, HD>(klo + v_off), v_hi = load_part<T, HD>(khi + v_off);
          float add_lo[4], add_hi[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int km = of_slot(cur.info, block, (j >> 1) * 8 + qt * 2 + (j & 1)), off = (km >> 16) * row_b - h * 4;
            add_lo[j] = bias(row_lo - off) + pack_mask<kMask>(km, me_lo);
            add_hi[j] = bias(row_hi - off) + pack_mask<kMask>(km, me_hi);
          }
          pack_block<T, HD, false>(r, k_lo, k_hi, v_lo, v_hi, add_lo, add_hi, qscale);
        }
        store(r, q_lo, q_hi, h);
      }
    }
  }
}

template <typename T, int HD>
static int launch_packs(AttnParams p, bool big, const int32_t rpb_window[3], cudaStream_t stream) {
  int dev = 0, sms = 0;
  SSW_CUDA_TRY(cudaGetDevice(&dev));
  SSW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t entries = (int64_t)(2 * rpb_window[0] - 1) * (2 * rpb_window[1] - 1) * (2 * rpb_window[2] - 1) * p.H;
  const bool in_smem = entries * 4 <= kTableMost;   // the rest of the SM's 256 KB is L1, for the rows
  p.table_floats = in_smem ? (int)entries : 0;
  const size_t smem = in_smem ? ((size_t)entries * 4 + 15) & ~(size_t)15 : 0;
  void (*kern)(AttnParams);
  auto pick = [&](auto table_smem, auto mask, auto big) {
    kern = k_attn_mma<T, HD, decltype(table_smem)::value, decltype(mask)::value, decltype(big)::value>;
  };
  auto pick2 = [&](auto table_smem, auto mask) { big ? pick(table_smem, mask, std::true_type{}) : pick(table_smem, mask, std::false_type{}); };
  auto pick1 = [&](auto table_smem) { p.use_mask ? pick2(table_smem, std::true_type{}) : pick2(table_smem, std::false_type{}); };
  in_smem ? pick1(std::true_type{}) : pick1(std::false_type{});
  SSW_CUDA_TRY(allow_smem(kern, kTableMost));
  SSW_CUDA_TRY(launch_chained(kern, dim3(sms), dim3(kPackThreads), smem, stream, p));
  SSW_LAUNCH_CHECK("k_attn_mma");
  return SSW_OK;
}

// What the default tile and the widest rows follow: the room that five, or three, stages of whole rows would take in one SM's shared memory
// beside the bias table.  No kernel keeps rows there any more, and nothing else asks for the smaller tile of wide rows (32 slots at 12 heads of 32): it stays
// because plans are built, sized and saved with it, and which windows are beyond a pack follows from it.  Rows wider than that have always been refused.
static int row_stages(int tile, int heads, int head_dim, const int32_t rpb_window[3]) {
  const int64_t stride = (int64_t)3 * heads * head_dim * 2 + 16;
  const int64_t per_stage = 16 + kMaxTile * 4 + tile * stride + producer_scratch_bytes(tile);
  const int64_t entries = (int64_t)(2 * rpb_window[0] - 1) * (2 * rpb_window[1] - 1) * (2 * rpb_window[2] - 1) * heads;
  const int64_t budget = 226 * 1024, base = 256 + stride, table = (entries * 4 + 15) & ~(int64_t)15;
  const int64_t fixed = base + (base + table + 4 * per_stage <= budget ? table : 0);
  return budget > fixed ? (int)((budget - fixed) / per_stage) : 0;
}

// The largest tile of 64/32/16 slots that leaves at least four such stages.
int mma_default_tile(int heads, int head_dim, const int32_t rpb_window[3]) {
  static const int kTiles[] = {64, 32, 16};
  for (int tile : kTiles)
    if (row_stages(tile, heads, head_dim, rpb_window) >= 4) return tile;
  return 16;
}

// Padded plan, 16-bit inputs: packs and larger windows.  `p` arrives with the plan pointers,
// qkv/out/table, H, C, tile, scale, use_mask and rel_off filled in.
int run_attn_dense(const AttnParams& a, const int32_t* bins, const int32_t* win_start, const int32_t* win_pstart,
                   int n_per_window, int dtype, const int32_t rpb_window[3], cudaStream_t stream);
bool attn_dense_supported(int head_dim, int n_per_window, const int32_t rpb_window[3]);

int run_attn_mma(AttnParams p, int dtype, int head_dim, const int32_t rpb_window[3], const int32_t* bins,
                 const int32_t* win_start, const int32_t* win_pstart, int n_per_window, cudaStream_t stream) {
  // Windows beyond a pack: the tcgen05 kernel where it serves the shape (and the window size allows
  // such windows at all), else this one.
  const bool dense = n_per_window > p.tile && attn_dense_supported(head_dim, n_per_window, rpb_window);
  if (row_stages(p.tile, p.H, head_dim, rpb_window) < 3) return SSW_E_UNSUPPORTED;
  if (p.tile & 15) return SSW_E_INVALID;
  const bool big = n_per_window > p.tile && !dense;
  int st = SSW_E_UNSUPPORTED;
  if (dtype == SSW_BF16) {
    if (head_dim == 16) st = launch_packs<__nv_bfloat16, 16>(p, big, rpb_window, stream);
    if (head_dim == 32) st = launch_packs<__nv_bfloat16, 32>(p, big, rpb_window, stream);
  } else if (dtype == SSW_F16) {
    if (head_dim == 16) st = launch_packs<__half, 16>(p, big, rpb_window, stream);
    if (head_dim == 32) st = launch_packs<__half, 32>(p, big, rpb_window, stream);
  }
  if (st != SSW_OK || !dense) return st;
  return run_attn_dense(p, bins, win_start, win_pstart, n_per_window, dtype, rpb_window, stream);
}

}  // namespace ssw
