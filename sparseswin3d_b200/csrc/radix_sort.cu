// Stable argsort of int32 keys (upstream's sort_indices, ops.cu:276-289, a thrust sort_by_key
// over a 0..n-1 sequence): least-significant-digit radix sort, 8 bits per pass, signed order.
//
// Per pass: k_radix_hist counts the digit of every key per tile of 1024 or 2048 keys into a digit-major
// table, a device-wide exclusive scan turns the table into global offsets, and k_radix_scatter
// re-reads the tile, ranks equal digits in key order (warp match + per-warp
// counters, so the pass is stable) and scatters (key, index) pairs.
#include "scan.cuh"
#include "ssw_common.cuh"

namespace ssw {

constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kSortThreads = 256;
constexpr int kManyRounds = 8, kFewRounds = 4;
constexpr int64_t kManyKeys = (int64_t)3 * 148 * kManyRounds * kSortThreads;
// Keys a thread takes: a larger tile has longer runs to write and a smaller table to scan, a smaller one has its blocks done sooner.
// The whole sort with 4 / 8 / 16 keys: 82 / 94 / 111 us for 100 000, 113 / 119 / - for 700 000, 141 / 135 / 158 for 1.3 M,
// 232 / 221 / 223 for 3.4 M, 448 / 387 / 446 for 8 M; the line lies at three tiles of 2048 for each of a B200's 148
// multiprocessors.  (A constant, not the present device's count: the size of a workspace is asked for without a device.)
static int sort_rounds(int64_t n) { return n >= kManyKeys ? kManyRounds : kFewRounds; }

__device__ __forceinline__ uint32_t digit_of(int32_t key, int shift) {
  return (((uint32_t)key ^ 0x80000000u) >> shift) & (kRadix - 1);
}

template <int kSortRounds>
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const int32_t* __restrict__ keys, int64_t n, int shift,
                                                             int32_t* __restrict__ hist, int n_tiles) {
  __shared__ int cnt[kRadix];
  cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * (kSortThreads * kSortRounds);
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r) {
    const int64_t e = base + r * kSortThreads + threadIdx.x;
    if (e < n) atomicAdd(&cnt[digit_of(keys[e], shift)], 1);
  }
  __syncthreads();
  hist[(int64_t)threadIdx.x * n_tiles + blockIdx.x] = cnt[threadIdx.x];
}

// Bound by its scattered writes and, in small sorts, by the chain of barriers and shared-memory round trips of a tile.  A warp counts
// 32 consecutive keys a round for itself, without waiting for the others; the counts of the eight warps then give every key its place in
// the tile, which is put in order in shared memory and written from there, neighbouring lanes to neighbouring slots.  The whole sort:
// 94 -> 76 us for 3000 keys, 104 -> 82 for 100 000, 154 -> 137 for 1.3 M, 283 -> 221 for 3.4 M and 560 -> 387 for 8 M against all warps side by side
// in rounds of 256 keys, four barriers a round, each thread writing its own keys.  (Eight keys a thread: 48 registers, 16 bytes spilled.)
template <int kSortRounds>
__global__ void __launch_bounds__(kSortThreads) k_radix_scatter(const int32_t* __restrict__ keys_in,
                                                                const int32_t* __restrict__ vals_in, int64_t n,
                                                                int shift, const int32_t* __restrict__ offsets,
                                                                int n_tiles, int32_t* __restrict__ keys_out,
                                                                int32_t* __restrict__ vals_out, int first_pass) {
  constexpr int kWarps = kSortThreads / 32;
  constexpr int kSortTile = kSortThreads * kSortRounds;
  static_assert(kSortThreads == kRadix, "a thread per digit");
  __shared__ int cnt[kWarps][kRadix];   // keys of a digit in the warp's run so far, then the tile's place of the first of them
  __shared__ int base[kRadix];          // slot in the output less place in the tile
  __shared__ int sums[kWarps];
  __shared__ int2 tile[kSortTile];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int i = lane; i < kRadix; i += 32) cnt[wid][i] = 0;
  const int slot = offsets[(int64_t)threadIdx.x * n_tiles + blockIdx.x];   // of the digit threadIdx.x
  const int64_t t0 = (int64_t)blockIdx.x * kSortTile;
  const int here = (int)min(n - t0, (int64_t)kSortTile);
  const int e0 = wid * (32 * kSortRounds) + lane;
  int32_t key[kSortRounds], val[kSortRounds];
  int rank[kSortRounds];
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r) {
    const int e = e0 + r * 32;
    key[r] = e < here ? keys_in[t0 + e] : 0;
    val[r] = first_pass ? (int32_t)(t0 + e) : e < here ? vals_in[t0 + e] : 0;
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r) {
    const bool live = e0 + r * 32 < here;
    const uint32_t d = digit_of(key[r], shift);
    // lanes with the same digit, in lane (= key) order
    const unsigned peers = __match_any_sync(0xffffffffu, live ? d : 0xffffffffu);
    const int before = __popc(peers & ((1u << lane) - 1u));
    const int had = live ? cnt[wid][d] : 0;
    __syncwarp();
    if (live && before == 0) cnt[wid][d] = had + __popc(peers);
    __syncwarp();
    rank[r] = had + before;
  }
  __syncthreads();
  int all = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const int c = cnt[w][threadIdx.x];
    cnt[w][threadIdx.x] = all;
    all += c;
  }
  int upto = all;   // and of the digits before, exclusive below
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += x;
  }
  if (lane == 31) sums[wid] = upto;
  __syncthreads();
  int place = upto - all;
  for (int w = 0; w < wid; ++w) place += sums[w];
#pragma unroll
  for (int w = 0; w < kWarps; ++w) cnt[w][threadIdx.x] += place;
  base[threadIdx.x] = slot - place;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r)
    if (e0 + r * 32 < here) tile[cnt[wid][digit_of(key[r], shift)] + rank[r]] = make_int2(key[r], val[r]);
  __syncthreads();
#pragma unroll 4
  for (int i = threadIdx.x; i < here; i += kSortThreads) {
    const int2 kv = tile[i];
    const int dst = base[digit_of(kv.x, shift)] + i;
    keys_out[dst] = kv.x;
    vals_out[dst] = kv.y;
  }
}

}  // namespace ssw

using namespace ssw;

// Two key buffers, one value buffer, digit table, scan workspace.
static int64_t sort_bytes(int64_t n, int rounds) {
  const int64_t table = (int64_t)kRadix * ceil_div64(n, kSortThreads * rounds);
  return 4 * (3 * n + table) + 8 * scan_workspace_i64(table) + 64;
}
// Small tiles want a larger table: at the line and for some 4 % beyond it, what the largest sort with small tiles wants, so that a workspace for
// n keys serves fewer as well as they can be served.
extern "C" int64_t ssw_argsort_workspace_bytes(int64_t n) {
  if (n <= 0) return 64;
  const int64_t here = sort_bytes(n, sort_rounds(n)), below = sort_bytes(kManyKeys - 1, kFewRounds);
  return n >= kManyKeys && here < below ? below : here;
}

extern "C" int ssw_argsort_i32(const int32_t* keys, int64_t n, int32_t* perm_out, void* workspace,
                               int64_t workspace_bytes, void* stream) {
  if (n < 0) return SSW_E_INVALID;
  if (n == 0) return SSW_OK;
  if (n >= (int64_t(1) << 31)) return SSW_E_RANGE;
  if (!keys || !perm_out || !workspace) return SSW_E_INVALID;
  if (workspace_bytes < sort_bytes(n, kManyRounds)) return SSW_E_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  // a workspace that holds the table of large tiles alone gets these: the same order, in a little more time
  const bool many = sort_rounds(n) == kManyRounds || workspace_bytes < sort_bytes(n, kFewRounds);
  const int tiles = (int)ceil_div64(n, kSortThreads * (many ? kManyRounds : kFewRounds));
  const int64_t table = (int64_t)kRadix * tiles;
  long long* ws = (long long*)workspace;
  const int64_t ws_i64 = scan_workspace_i64(table);
  int32_t* kbuf0 = reinterpret_cast<int32_t*>(ws + ws_i64);
  int32_t* kbuf1 = kbuf0 + n;
  int32_t* vbuf = kbuf1 + n;
  int32_t* hist = vbuf + n;
  SSW_CUDA_TRY(cudaMemsetAsync(ws, 0, 16, st));
  const int32_t* kin = keys;
  const int32_t* vin = nullptr;
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = pass * kRadixBits;
    // values ping-pong between vbuf and perm_out so that the last pass lands in perm_out
    int32_t* kout = (pass & 1) ? kbuf1 : kbuf0;
    int32_t* vout = (pass & 1) ? perm_out : vbuf;
    (many ? k_radix_hist<kManyRounds> : k_radix_hist<kFewRounds>)<<<tiles, kSortThreads, 0, st>>>(kin, n, shift, hist, tiles);
    SSW_LAUNCH_CHECK("k_radix_hist");
    auto f = [hist] __device__(int64_t i) -> int { return hist[i]; };
    auto g = [hist] __device__(int64_t i, int, long long ex) { hist[i] = (int32_t)ex; };
    int rc = device_scan(f, g, table, ws, st);
    if (rc) return rc;
    (many ? k_radix_scatter<kManyRounds> : k_radix_scatter<kFewRounds>)<<<tiles, kSortThreads, 0, st>>>(kin, vin, n, shift, hist, tiles, kout, vout, pass == 0);
    SSW_LAUNCH_CHECK("k_radix_scatter");
    kin = kout;
    vin = vout;
  }
  return SSW_OK;
}
