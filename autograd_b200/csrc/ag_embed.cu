// Token-embedding gather and its deterministic scatter-add backward.
//
// Forward: out[i,:] = table[ids[i],:], a pure copy (bit-exact).  One warp per token row,
// all 16-byte loads of a row chunk issued before the stores.
//
// Backward: dtable[ids[i],:] += dout[i,:] with a summation order that does not depend on
// scheduling.  No float atomics are used anywhere.  Very few ids take one launch without a sort
// (scatter_few_kernel); otherwise:
//   1. stable LSD radix sort of (id, position) pairs, 9 bits per pass, so that equal ids end
//      up adjacent and in ascending position order (up to 262144 ids: one histogram launch and
//      one launch per pass; beyond that a histogram, a scan and a scatter launch per pass);
//      up to 4096 ids one CTA makes all passes in shared memory instead;
//   2. the sorted list is cut into groups of 8 to 64 consecutive entries (see scatter_group).  A CTA, or a part of one, walks
//      one group, every
//      thread keeping a ring of 8 row requests in flight, summing each run of equal ids in list order.  A run
//      that is a complete segment (its id neither continues from the previous group nor
//      into the next one) starts from the current dtable row and is written back directly:
//      for such rows the result is bit-identical to numpy's sequential np.add.at.  A run cut
//      by a group boundary is written to a per-group partial slot instead;
//   3. a combine kernel finds the segments that span several groups and adds their partial slots
//      in group order onto the dtable row.
// Ids outside [0,V) are dropped and flagged in the status word.
#include <atomic>

#include "ag_common.cuh"

namespace {

// ------------------------------------------------------------------------------ gather
constexpr int GATHER_THREADS = 256;

// VW floats of a row moved as one access: 4, 2 or 1, the widest that the row length and the pointers allow.
template <int VW>
struct RowVec;
template <>
struct RowVec<4> { using Type = float4; };
template <>
struct RowVec<2> { using Type = float2; };
template <>
struct RowVec<1> { using Type = float; };

// LANES threads (a power of two up to 32) share a row, so that narrow rows leave few lanes of a warp idle.
template <int VW, int LANES>
__global__ void __launch_bounds__(GATHER_THREADS)
gather_forward_kernel(const int32_t* __restrict__ ids, const float* __restrict__ table, float* __restrict__ out,
                      int64_t n_ids, int C, int V, int* status) {
  using Vec = typename RowVec<VW>::Type;
  ag_pdl_wait();
  const int lane = threadIdx.x & (LANES - 1);
  const int64_t first = ((int64_t)blockIdx.x * GATHER_THREADS + threadIdx.x) / LANES;
  const int64_t step = (int64_t)gridDim.x * GATHER_THREADS / LANES;
  const int cp = C / VW;
  for (int64_t i = first; i < n_ids; i += step) {
    const int id = ids[i];
    const bool ok = id >= 0 && id < V;
    if (!ok && lane == 0) atomicOr(status, AG_STATUS_BAD_INDEX);
    const Vec* src = reinterpret_cast<const Vec*>(table + (int64_t)(ok ? id : 0) * C);
    Vec* dst = reinterpret_cast<Vec*>(out + i * C);
    for (int p = lane; p < cp; p += LANES * 4) {
      Vec v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (p + u * LANES < cp) v[u] = ok ? __ldg(src + p + u * LANES) : Vec{};
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (p + u * LANES < cp) __stcs(dst + p + u * LANES, v[u]);
    }
  }
}

// ------------------------------------------------------------------------------ radix sort
constexpr int SORT_BITS = 9;
constexpr int SORT_DIGITS = 1 << SORT_BITS;  // 512
constexpr int SORT_TILE = 1024;              // keys per CTA, one per thread
constexpr int SORT_WARPS = SORT_TILE / 32;

// Out-of-range ids get the key V (sorted behind every valid id, dropped later).
__global__ void __launch_bounds__(SORT_TILE)
sort_init_kernel(const int32_t* __restrict__ ids, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                 uint32_t* __restrict__ head_count, int64_t n, int V, int* status) {
  ag_pdl_wait();
  if (gridDim.x * gridDim.y <= 148) ag_pdl_trigger();  // single-wave grids let the next kernel be scheduled early
  if (blockIdx.x == 0 && threadIdx.x == 0) *head_count = 0u;  // the list of head groups starts empty
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int id = ids[i];
  const bool ok = id >= 0 && id < V;
  if (!ok) atomicOr(status, AG_STATUS_BAD_INDEX);
  keys[i] = ok ? (uint32_t)id : (uint32_t)V;
  vals[i] = (uint32_t)i;
}

// Per-tile digit histogram: hist[digit * n_tiles + tile].
__global__ void __launch_bounds__(SORT_TILE)
sort_hist_kernel(const uint32_t* __restrict__ keys, uint32_t* __restrict__ hist, int64_t n, int shift, int n_tiles) {
  ag_pdl_wait();
  if (gridDim.x * gridDim.y <= 148) ag_pdl_trigger();  // single-wave grids let the next kernel be scheduled early
  __shared__ uint32_t s_cnt[SORT_DIGITS];
  for (int d = threadIdx.x; d < SORT_DIGITS; d += SORT_TILE) s_cnt[d] = 0;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * SORT_TILE + threadIdx.x;
  if (i < n) atomicAdd(&s_cnt[(keys[i] >> shift) & (SORT_DIGITS - 1)], 1u);  // integer: order-free
  __syncthreads();
  for (int d = threadIdx.x; d < SORT_DIGITS; d += SORT_TILE) hist[(int64_t)d * n_tiles + blockIdx.x] = s_cnt[d];
}

// Exclusive scan of hist (digit-major, SORT_DIGITS*n_tiles entries) by a single CTA.  Blocks of
// 32768 entries: warp w owns entries [1024 w, 1024 w + 1024) of the block, loads them all at once
// (32 coalesced loads per lane in flight), scans them in registers with a running carry, then the 32
// warp totals are scanned and every warp writes its segment with its offset.
__global__ void __launch_bounds__(1024) sort_scan_kernel(uint32_t* __restrict__ hist, int64_t total) {
  ag_pdl_wait();
  ag_pdl_trigger();
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t base = 0; base < total; base += 32768) {
    const int64_t seg = base + (int64_t)warp * 1024 + lane;
    uint32_t v[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int64_t i = seg + k * 32;
      v[k] = i < total ? hist[i] : 0u;
    }
    uint32_t run = 0;  // sum of the warp's entries before row k
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const uint32_t x = v[k];
      uint32_t inc = x;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      v[k] = run + inc - x;  // exclusive prefix inside the warp's segment
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_warp[warp] = run;
    __syncthreads();
    const uint32_t carry = s_carry;
    uint32_t before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {  // 32 shared-memory broadcasts; same values for every thread
      const uint32_t t = s_warp[w];
      if (w < warp) before += t;
      all += t;
    }
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int64_t i = seg + k * 32;
      if (i < total) hist[i] = carry + before + v[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) s_carry = carry + all;
    __syncthreads();
  }
}

// Stable scatter of one tile: rank inside the tile = (#equal digits in earlier warps) +
// (#equal digits in lower lanes of the own warp).
__global__ void __launch_bounds__(SORT_TILE)
sort_scatter_kernel(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                    const uint32_t* __restrict__ hist, int64_t n, int shift, int n_tiles) {
  ag_pdl_wait();
  if (gridDim.x * gridDim.y <= 148) ag_pdl_trigger();  // single-wave grids let the next kernel be scheduled early
  __shared__ uint16_t s_cnt[SORT_WARPS][SORT_DIGITS];  // 32 KB
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = lane; d < SORT_DIGITS; d += 32) s_cnt[warp][d] = 0;
  __syncwarp();
  const int64_t i = (int64_t)blockIdx.x * SORT_TILE + threadIdx.x;
  const bool live = i < n;
  uint32_t key = 0, val = 0;
  int digit = 0;
  if (live) {
    key = keys_in[i];
    val = vals_in[i];
    digit = (key >> shift) & (SORT_DIGITS - 1);
  }
  // peers: live lanes of this warp holding the same digit
  const uint32_t live_mask = __ballot_sync(0xffffffffu, live);
  uint32_t peers = 0;
  if (live) peers = __match_any_sync(live_mask, digit);
  const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
  if (live && rank_in_warp == 0) s_cnt[warp][digit] = (uint16_t)__popc(peers);
  __syncthreads();
  if (live) {
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += s_cnt[w][digit];
    const uint32_t dst = hist[(int64_t)digit * n_tiles + blockIdx.x] + before + rank_in_warp;
    keys_out[dst] = key;
    vals_out[dst] = val;
  }
}

// ------------------------------------------------------------------------------ radix sort, few launches
// For up to SORT_FUSED_MAX_TILES tiles (262144 ids) a pass needs no scan launch and no separate
// histogram launch after the first one:
//   * sort_hist_ids_kernel reads the ids themselves (key = id, or V for an id outside the table;
//     value = position), writes the per-tile histogram of the first digit and zeroes the
//     histograms of the later passes;
//   * sort_scatter_fused_kernel derives its tile's digit offsets from the whole histogram
//     (n_tiles x SORT_DIGITS counters, tile-major, a few hundred KB in L2: thread d walks digit d
//     down the tiles with coalesced loads, then the CTA scans the 512 digit totals), places its
//     keys stably, and counts the next pass's per-tile histogram as it goes - integer atomics on
//     counters, aggregated per warp, whose final values do not depend on the order of the additions.
// The order of the sorted list is the one the unfused kernels produce: stable by digit, tile, rank.
constexpr int SORT_FUSED_MAX_TILES = 256;
constexpr int SORT_MAX_PASSES = 4;

__device__ __forceinline__ uint32_t sort_key_of(int id, int V) { return (id >= 0 && id < V) ? (uint32_t)id : (uint32_t)V; }

// hist0 and hist_later are tile-major: counter of (tile, digit) at [tile * SORT_DIGITS + digit].
__global__ void __launch_bounds__(SORT_TILE)
sort_hist_ids_kernel(const int32_t* __restrict__ ids, uint32_t* __restrict__ hist0, uint32_t* __restrict__ hist_later,
                     int64_t later_entries, uint32_t* __restrict__ head_count, int64_t n, int V, int* status) {
  ag_pdl_wait();
  if (gridDim.x <= 148) ag_pdl_trigger();
  if (blockIdx.x == 0 && threadIdx.x == 0) *head_count = 0u;  // the list of head groups starts empty
  __shared__ uint32_t s_cnt[SORT_DIGITS];
  for (int d = threadIdx.x; d < SORT_DIGITS; d += SORT_TILE) s_cnt[d] = 0;
  // the histograms of the later passes start at zero: this CTA clears its share
  for (int64_t e = (int64_t)blockIdx.x * SORT_TILE + threadIdx.x; e < later_entries; e += (int64_t)gridDim.x * SORT_TILE)
    hist_later[e] = 0u;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * SORT_TILE + threadIdx.x;
  if (i < n) {
    const int id = ids[i];
    if (id < 0 || id >= V) atomicOr(status, AG_STATUS_BAD_INDEX);
    atomicAdd(&s_cnt[sort_key_of(id, V) & (SORT_DIGITS - 1)], 1u);  // integer: order-free
  }
  __syncthreads();
  for (int d = threadIdx.x; d < SORT_DIGITS; d += SORT_TILE) hist0[(int64_t)blockIdx.x * SORT_DIGITS + d] = s_cnt[d];
}

// FIRST: keys and values come from the ids (pass 0); otherwise from keys_in / vals_in.
// hist: this pass's per-tile histogram; hist_next: the next pass's (NULL on the last pass), counted
// per tile of the OUTPUT positions.  Both tile-major.
template <bool FIRST>
__global__ void __launch_bounds__(SORT_TILE)
sort_scatter_fused_kernel(const int32_t* __restrict__ ids, const uint32_t* __restrict__ keys_in,
                          const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out,
                          uint32_t* __restrict__ vals_out, const uint32_t* __restrict__ hist,
                          uint32_t* __restrict__ hist_next, int64_t n, int V, int shift, int n_tiles) {
  ag_pdl_wait();
  if (gridDim.x <= 148) ag_pdl_trigger();
  __shared__ uint16_t s_cnt[SORT_WARPS][SORT_DIGITS];  // 32 KB
  __shared__ uint32_t s_tot[2][SORT_DIGITS], s_bef[2][SORT_DIGITS];
  __shared__ uint32_t s_base[SORT_DIGITS];             // first output position of (digit, this tile)
  __shared__ uint32_t s_wsum[SORT_DIGITS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = lane; d < SORT_DIGITS; d += 32) s_cnt[warp][d] = 0;
  // the tile's own key and position are requested first; they arrive while the offsets are computed
  const int64_t i = (int64_t)blockIdx.x * SORT_TILE + threadIdx.x;
  const bool live = i < n;
  uint32_t key = 0, val = 0;
  int digit = 0;
  if (live) {
    if (FIRST) {
      key = sort_key_of(ids[i], V);
      val = (uint32_t)i;
    } else {
      key = keys_in[i];
      val = vals_in[i];
    }
    digit = (key >> shift) & (SORT_DIGITS - 1);
  }

  // ---- offsets: total[d] = count of digit d over all tiles, before[d] = over the tiles before this one.
  // Thread (half, d) walks digit d down one half of the tiles; a warp's loads are 32 consecutive counters.
  {
    const int d = threadIdx.x & (SORT_DIGITS - 1), half = threadIdx.x >> 9;
    const int t0 = half ? (n_tiles + 1) / 2 : 0, t1 = half ? n_tiles : (n_tiles + 1) / 2;
    uint32_t total = 0, before = 0;
    for (int t = t0; t < t1; t += 8) {
      uint32_t v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = (t + u < t1) ? hist[(int64_t)(t + u) * SORT_DIGITS + d] : 0u;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        total += v[u];
        if (t + u < (int)blockIdx.x) before += v[u];
      }
    }
    s_tot[half][d] = total;
    s_bef[half][d] = before;
  }
  __syncthreads();
  if (threadIdx.x < SORT_DIGITS) {
    // exclusive scan of the 512 digit totals: 16 warps of 32 digits
    const int d = threadIdx.x;
    const uint32_t total = s_tot[0][d] + s_tot[1][d];
    uint32_t inc = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_wsum[warp] = inc;
    s_base[d] = inc - total + s_bef[0][d] + s_bef[1][d];  // the warps' offsets are added below
  }
  __syncthreads();
  if (threadIdx.x < SORT_DIGITS) {
    uint32_t wbase = 0;
    for (int w = 0; w < warp; ++w) wbase += s_wsum[w];
    s_base[threadIdx.x] += wbase;
  }

  const uint32_t live_mask = __ballot_sync(0xffffffffu, live);
  uint32_t peers = 0;
  if (live) peers = __match_any_sync(live_mask, digit);
  const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
  if (live && rank_in_warp == 0) s_cnt[warp][digit] = (uint16_t)__popc(peers);
  __syncthreads();
  if (live) {
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += s_cnt[w][digit];
    const uint32_t dst = s_base[digit] + before + rank_in_warp;
    keys_out[dst] = key;
    vals_out[dst] = val;
    if (hist_next) {
      // one atomic per distinct counter and warp (a hot id fills whole warps with the same counter)
      const uint32_t counter = (dst >> 10) * SORT_DIGITS + ((key >> (shift + SORT_BITS)) & (SORT_DIGITS - 1));
      const uint32_t same = __match_any_sync(live_mask, counter);
      if ((same & ((1u << lane) - 1u)) == 0) atomicAdd(&hist_next[counter], (uint32_t)__popc(same));  // order-free
    }
  }
}

// ------------------------------------------------------------------------------ scatter-add
// Up to SORT_SMALL_MAX ids: the same passes by one CTA, in one launch.  A warp owns 32 * ITEMS consecutive entries, in
// registers; what it has of every digit so far is a word of its row of counters, so that an entry's rank in the warp is that
// word and the entries of its own 32 before it.  The rows are scanned digit by digit, the digits' totals as above, and the
// entries change places through shared memory.  One SM takes 1.5 us more per 1000 entries, so that the launches win from some
// 5000 on (whole scatter-adds into a table of 30000, us, one CTA / launches: 1500 x 384 13.0 / 17.3, 4000 x 64 17.3 / 18.6, x 384
// 18.4 / 18.7, 6000 x 384 23.7 / 21.2).  A bitonic network over the next power of two took 42-50 us for 4000 x 64-1536.
constexpr int SORT_SMALL_MAX = 4096;
constexpr size_t sort_small_smem(int items) { return (size_t)SORT_WARPS * SORT_DIGITS * 2 + (size_t)SORT_TILE * items * 8; }

template <int ITEMS>
__global__ void __launch_bounds__(SORT_TILE)
sort_small_kernel(const int32_t* __restrict__ ids, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                  uint32_t* __restrict__ head_count, int n, int bits, int V, int* status) {
  ag_pdl_wait();
  ag_pdl_trigger();
  extern __shared__ __align__(16) unsigned char sort_smem[];
  uint16_t(*s_cnt)[SORT_DIGITS] = reinterpret_cast<uint16_t(*)[SORT_DIGITS]>(sort_smem);
  uint32_t* s_key = reinterpret_cast<uint32_t*>(sort_smem + SORT_WARPS * SORT_DIGITS * 2);
  uint32_t* s_val = s_key + SORT_TILE * ITEMS;
  __shared__ uint32_t s_base[SORT_DIGITS];
  __shared__ uint32_t s_wsum[SORT_DIGITS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = warp * 32 * ITEMS + lane;  // entry j is first + 32 j
  if (threadIdx.x == 0) *head_count = 0u;
  uint32_t key[ITEMS], val[ITEMS];
  bool bad = false;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = first + 32 * j;
    key[j] = (uint32_t)V;
    val[j] = (uint32_t)i;
    if (i < n) {
      key[j] = sort_key_of(ids[i], V);
      bad |= key[j] == (uint32_t)V;
    }
  }
  if (bad) atomicOr(status, AG_STATUS_BAD_INDEX);
  for (int shift = 0; shift < bits; shift += SORT_BITS) {
    uint4* row = reinterpret_cast<uint4*>(s_cnt[warp]);
    row[lane] = row[lane + 32] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    uint32_t rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (warp * 32 * ITEMS + 32 * j >= n) break;  // none of the warp's
      const bool live = first + 32 * j < n;
      const int digit = live ? (key[j] >> shift) & (SORT_DIGITS - 1) : 0;
      // entries of the same digit: a ballot per bit (match_any takes a turn per distinct digit)
      uint32_t peers = __ballot_sync(0xffffffffu, live);
      if (!live) peers = ~peers;
#pragma unroll
      for (int b = 0; b < SORT_BITS; ++b) {
        const bool bit = (digit >> b) & 1;
        const uint32_t set = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? set : ~set;
      }
      const uint32_t below = peers & ((1u << lane) - 1u);
      const uint32_t before = live ? s_cnt[warp][digit] : 0u;
      rank[j] = before + __popc(below);
      __syncwarp();
      if (live && below == 0) s_cnt[warp][digit] = (uint16_t)(before + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    uint32_t total = 0, inc = 0;
    if (threadIdx.x < SORT_DIGITS) {
#pragma unroll 8
      for (int w = 0; w < SORT_WARPS; ++w) {
        const uint32_t c = s_cnt[w][threadIdx.x];
        s_cnt[w][threadIdx.x] = (uint16_t)total;
        total += c;
      }
      inc = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (lane == 31) s_wsum[warp] = inc;
    }
    __syncthreads();
    if (threadIdx.x < SORT_DIGITS) {
      uint32_t base = inc - total;
#pragma unroll
      for (int w = 0; w < SORT_DIGITS / 32; ++w) base += w < warp ? s_wsum[w] : 0u;
      s_base[threadIdx.x] = base;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (first + 32 * j >= n) break;
      const int digit = (key[j] >> shift) & (SORT_DIGITS - 1);
      const uint32_t dst = s_base[digit] + s_cnt[warp][digit] + rank[j];
      s_key[dst] = key[j];
      s_val[dst] = val[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (first + 32 * j >= n) break;
      key[j] = s_key[first + 32 * j];
      val[j] = s_val[first + 32 * j];
    }
  }
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    if (first + 32 * j >= n) break;
    keys[first + 32 * j] = key[j];
    vals[first + 32 * j] = val[j];
  }
}

constexpr int SEG_THREADS = 128;    // threads of a CTA of the segmented sum: 32, 64 or 128 per group

template <int VW>
struct alignas(VW * 4) Cols {  // VW columns of a row
  float v[VW];
  __device__ __forceinline__ Cols& operator+=(const Cols& o) {
#pragma unroll
    for (int e = 0; e < VW; ++e) v[e] += o.v[e];
    return *this;
  }
};

// Table-gradient rows are fp32, or bf16 bit patterns (TT = uint16_t: the reference's bf16
// parameter-gradient storage, metal_ops.metal:12395-12446: the sum of a row's contributions is
// formed in fp32 from zero, and the row becomes bf16(old + sum), rounded once, to nearest even).
__device__ __forceinline__ uint32_t seg_bf16_rne(float value) {
  const uint32_t bits = __float_as_uint(value);
  if ((bits & 0x7f800000u) == 0x7f800000u) return ((bits >> 16) | ((bits & 0x007fffffu) ? 0x0040u : 0u)) & 0xffffu;
  return ((bits + 0x7fffu + ((bits >> 16) & 1u)) >> 16) & 0xffffu;
}
template <int VW>
__device__ __forceinline__ Cols<VW> seg_load(const float* p) {
  Cols<VW> r;
  *reinterpret_cast<typename RowVec<VW>::Type*>(r.v) = *reinterpret_cast<const typename RowVec<VW>::Type*>(p);
  return r;
}
template <int VW>
__device__ __forceinline__ Cols<VW> seg_load_once(const float* p) {
  Cols<VW> r;
  *reinterpret_cast<typename RowVec<VW>::Type*>(r.v) = __ldcs(reinterpret_cast<const typename RowVec<VW>::Type*>(p));
  return r;
}
template <int VW>
__device__ __forceinline__ Cols<VW> seg_load(const uint16_t* p) {
  Cols<VW> r;
  if constexpr (VW == 1) {
    r.v[0] = __uint_as_float((uint32_t)*p << 16);
  } else {
#pragma unroll
    for (int e = 0; e < VW; e += 2) {
      const uint32_t w = reinterpret_cast<const uint32_t*>(p)[e / 2];
      r.v[e] = __uint_as_float(w << 16);
      r.v[e + 1] = __uint_as_float(w & 0xffff0000u);
    }
  }
  return r;
}
template <int VW>
__device__ __forceinline__ void seg_store(float* p, const Cols<VW>& c) {
  *reinterpret_cast<typename RowVec<VW>::Type*>(p) = *reinterpret_cast<const typename RowVec<VW>::Type*>(c.v);
}
template <int VW>
__device__ __forceinline__ void seg_store(uint16_t* p, const Cols<VW>& c) {
  if constexpr (VW == 1) {
    *p = (uint16_t)seg_bf16_rne(c.v[0]);
  } else if constexpr (VW == 2) {
    *reinterpret_cast<uint32_t*>(p) = seg_bf16_rne(c.v[0]) | (seg_bf16_rne(c.v[1]) << 16);
  } else {
    *reinterpret_cast<uint2*>(p) = make_uint2(seg_bf16_rne(c.v[0]) | (seg_bf16_rne(c.v[1]) << 16),
                                              seg_bf16_rne(c.v[2]) | (seg_bf16_rne(c.v[3]) << 16));
  }
}

// ---- very few ids: one launch, no sort.  A block per position looks for the other occurrences of its id.  Three dependent
// launches (sort, segmented sum, combine) are all latency at this size.
// The columns of a row lie in pieces of 32 accesses.  The blocks of an id's positions share them, in the order of the positions
// and a piece each at least, so that a frequent id has as many blocks as its row has pieces.  Up to FEW_ORDERED occurrences are
// added by one warp per piece, in position order onto the table row; of more, the warps that a block has to spare for a piece
// (all eight where it has one piece) take consecutive shares, added in order.
// Up to 1024 ids of rows of up to 512 columns (four pieces of 128), or 256 ids.  Us, three launches / one, for ids that are
// distinct, Zipf of 32768, half of them one id, all of them one id (in brackets with all of an id's rows added by one block):
//   192 x 128 10.1 / 3.5, 12.6 / 3.6, 12.6 / 3.8 (3.7), 13.0 / 4.3 (4.3)    256 x 1280 10.4 / 3.5, 12.8 / 3.8 (9.5), 13.2 / 5.0
//   (27), 13.8 / 7.0 (51)    1024 x 128 16.3 / 5.4, 17.4 / 4.3, 18.0 / 7.5 (7.2), 18.0 / 10.6 (10.5)    1024 x 384 15.6 / 5.6,
//   17.8 / 5.0 (9.0), 18.1 / 11.0 (30), 18.3 / 16.7 (54)
constexpr int FEW_IDS_MAX = 1024, FEW_IDS_WIDE = 256, FEW_PIECES = 4;
constexpr int FEW_THREADS = 256;
constexpr int FEW_ORDERED = 16;  // occurrences that one warp adds
constexpr int FEW_BATCH = 8;     // rows requested together (16: 1024 distinct ids 5.6 -> 7.2 us, with fewer blocks per SM)

template <int VW, typename TT>
__global__ void __launch_bounds__(FEW_THREADS)
scatter_few_kernel(const int32_t* __restrict__ ids, const float* __restrict__ dout, TT* __restrict__ dtable, int n, int C, int V,
                   int* status) {
  __shared__ uint32_t s_mask[FEW_IDS_MAX / 32];
  __shared__ uint16_t s_at[FEW_IDS_MAX];
  __shared__ Cols<VW> s_part[FEW_THREADS / 32][32];
  constexpr bool F32 = sizeof(TT) == 4;
  constexpr int WARPS = FEW_THREADS / 32;
  static_assert(FEW_IDS_MAX == 32 * 32, "a lane per word of the mask");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ag_pdl_wait();
  ag_pdl_trigger();
  const int id = ids[blockIdx.x];
#pragma unroll
  for (int t = 0; t < FEW_IDS_MAX / FEW_THREADS; ++t) {
    const int j = t * FEW_THREADS + threadIdx.x;
    const uint32_t m = __ballot_sync(0xffffffffu, j < n && ids[j < n ? j : 0] == id);
    if (lane == 0) s_mask[t * WARPS + warp] = m;
  }
  if (id < 0 || id >= V) {
    if (threadIdx.x == 0) atomicOr(status, AG_STATUS_BAD_INDEX);
    return;
  }
  __syncthreads();
  const uint32_t mask = s_mask[lane];
  int before = __popc(mask);
  for (int o = 1; o < 32; o *= 2) {
    const int x = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += x;
  }
  const int count = __shfl_sync(0xffffffffu, before, 31);
  before -= __popc(mask);
  // this block's place among those of its id, and the pieces that fall to it
  const int word = blockIdx.x >> 5;
  const int rank = __shfl_sync(0xffffffffu, before, word) + __popc(s_mask[word] & ((1u << (blockIdx.x & 31)) - 1u));
  const int packets = C / VW, all = (packets + 31) / 32, blocks = count < all ? count : all;
  const int per_block = (all + blocks - 1) / blocks, begin = rank * per_block;
  if (begin >= all) return;  // the whole block
  const int pieces = all - begin < per_block ? all - begin : per_block;
  if (warp == 0)
    for (uint32_t m = mask; m; m &= m - 1) s_at[before++] = (uint16_t)(lane * 32 + __ffs(m) - 1);
  __syncthreads();

  const int share = count <= FEW_ORDERED || pieces >= 5 ? 1 : pieces >= 3 ? 2 : pieces == 2 ? 4 : 8;  // warps per piece
  const int sub = warp % share, per = (count + share - 1) / share;
  const int first = sub * per, last = first + per < count ? first + per : count;
  TT* row = dtable + (int64_t)id * C;
  for (int piece = warp / share; piece < (pieces + WARPS / share - 1) / (WARPS / share) * (WARPS / share); piece += WARPS / share) {
    const int packet = (begin + piece) * 32 + lane, at = packet * VW;
    const bool in = piece < pieces && packet < packets;
    Cols<VW> acc = {}, old = {};
    if (in) {
      if (sub == 0) old = seg_load<VW>(row + at);
      if (F32) acc = old;
      for (int k = first; k < last; k += FEW_BATCH) {
        Cols<VW> v[FEW_BATCH];
#pragma unroll
        for (int u = 0; u < FEW_BATCH; ++u)
          if (k + u < last) v[u] = seg_load_once<VW>(dout + (int64_t)s_at[k + u] * C + at);
#pragma unroll
        for (int u = 0; u < FEW_BATCH; ++u)
          if (k + u < last) acc += v[u];
      }
    }
    if (share > 1) {
      __syncthreads();  // what the round before left has been read
      s_part[warp][lane] = acc;
      __syncthreads();
      if (sub) continue;
      for (int w = 1; w < share; ++w) acc += s_part[warp + w][lane];
    }
    if (!in) continue;
    if (!F32) {
#pragma unroll
      for (int e = 0; e < VW; ++e) acc.v[e] = old.v[e] + acc.v[e];
    }
    seg_store<VW>(row + at, acc);
  }
}

// Block (TX, SEG_THREADS / TX): TX threads of VW columns each (128, or 32 so that a narrow row does not leave most of
// a CTA idle) per group, a group per thread row.  Grid = (groups / thread rows, ceil(C / (TX * VW))).
// VW: 4, 2 or 1 floats per access.
// partials: [n_groups][2][C] floats; slot 0 = the group's first run when it continues from
// the previous group or is the cut part of a longer segment, slot 1 = its last run when
// that run started inside this group and continues into the next one.
// Per-entry run information of a group, computed once per CTA.
constexpr uint32_t RUN_BEGIN = 1u, RUN_END = 2u, RUN_COMPLETE = 4u, RUN_SLOT1 = 8u, RUN_VALID = 16u;
constexpr int SEG_BATCH = 8;  // sorted entries whose rows are requested together

template <int VW, typename TT, int SEG_GROUP, int TX>
__global__ void __launch_bounds__(SEG_THREADS)
scatter_groups_kernel(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ pos,
                      const float* __restrict__ dout, TT* dtable, float* __restrict__ partials,
                      long long* __restrict__ heads, uint32_t* __restrict__ head_count,
                      uint32_t* __restrict__ head_list, int n_groups, int64_t n, int C, int V) {
  constexpr bool BF = sizeof(TT) == 2;  // rounded storage: sum from zero, add the old row last
  ag_pdl_wait();
  constexpr int TY = SEG_THREADS / TX;
  const int ty = TY == 1 ? 0 : threadIdx.y;
  // [0] = key before the group, [1..G] group, [G+1] = key after
  __shared__ uint32_t sh_key[TY][SEG_GROUP + 2];
  __shared__ uint32_t sh_pos[TY][SEG_GROUP];
  __shared__ uint32_t sh_info[TY][SEG_GROUP];
  uint32_t *s_key = sh_key[ty], *s_pos = sh_pos[ty], *s_info = sh_info[ty];
  const int64_t grp = (int64_t)blockIdx.x * TY + ty;
  const int64_t g0 = grp * SEG_GROUP;
  const int cnt = g0 >= n ? 0 : (int)((n - g0) < SEG_GROUP ? (n - g0) : SEG_GROUP);
  for (int t = threadIdx.x; t < SEG_GROUP + 2; t += TX) {
    const int64_t j = g0 - 1 + t;
    // sentinel 0xffffffff never equals a key (keys are <= V)
    s_key[t] = (j >= 0 && j < n && t <= cnt + 1) ? keys[j] : 0xffffffffu;
  }
  for (int t = threadIdx.x; t < SEG_GROUP; t += TX) s_pos[t] = t < cnt ? pos[g0 + t] : 0u;
  __syncthreads();
  for (int j = threadIdx.x; j < cnt; j += TX) {
    // the run (equal keys) around entry j: where it begins and ends inside the group, whether it is cut
    // by the group boundary on either side
    const uint32_t key = s_key[j + 1];
    int rb = j, re = j;
    while (rb > 0 && s_key[rb] == key) --rb;
    while (re + 1 < cnt && s_key[re + 2] == key) ++re;
    const bool from_prev = rb == 0 && s_key[0] == key;
    const bool into_next = re == cnt - 1 && s_key[cnt + 1] == key;
    uint32_t info = 0;
    if (j == rb) info |= RUN_BEGIN;
    if (j == re) info |= RUN_END;
    if (!from_prev && !into_next) info |= RUN_COMPLETE;
    if (!(from_prev || rb == 0)) info |= RUN_SLOT1;
    if (key < (uint32_t)V) info |= RUN_VALID;
    s_info[j] = info;
  }
  __syncthreads();

  const int col = (blockIdx.y * TX + threadIdx.x) * VW;
  if (col < C) {
    // A ring of SEG_BATCH row requests per thread: the row of entry j + SEG_BATCH (and the dtable row of
    // a complete run that begins there) is requested as soon as entry j has been added, so that a
    // thread always has SEG_BATCH - 1 or SEG_BATCH rows in flight.  The adds run in sorted (= position)
    // order, each complete run starting from its dtable row: the same sequence of additions as an
    // unbuffered add-at.
    Cols<VW> acc = {}, old = {};
    Cols<VW> v[SEG_BATCH], d[SEG_BATCH];
    auto request = [&](int u, int j) {
      v[u] = d[u] = Cols<VW>{};
      if (j < cnt) {
        const uint32_t info = s_info[j];
        if (info & RUN_VALID) {
          v[u] = seg_load_once<VW>(dout + (int64_t)s_pos[j] * C + col);
          if ((info & (RUN_BEGIN | RUN_COMPLETE)) == (RUN_BEGIN | RUN_COMPLETE))
            d[u] = seg_load<VW>(dtable + (int64_t)s_key[j + 1] * C + col);
        }
      }
    };
#pragma unroll
    for (int u = 0; u < SEG_BATCH; ++u) request(u, u);
    for (int j0 = 0; j0 < cnt; j0 += SEG_BATCH) {
#pragma unroll
      for (int u = 0; u < SEG_BATCH; ++u) {
        const int j = j0 + u;
        if (j < cnt) {
          const uint32_t info = s_info[j];
          if (info & RUN_VALID) {
            if (info & RUN_BEGIN) {
              if (BF) { old = d[u]; acc = Cols<VW>{}; }
              else acc = d[u];  // zero for a cut run
            }
            acc += v[u];
            if (info & RUN_END) {
              if (info & RUN_COMPLETE) {
                Cols<VW> sum = acc;
                if (BF) { sum = old; sum += acc; }
                seg_store<VW>(dtable + (int64_t)s_key[j + 1] * C + col, sum);
              } else {
                seg_store<VW>(partials + (grp * 2 + ((info & RUN_SLOT1) ? 1 : 0)) * C + col, acc);
              }
            }
          }
        }
        request(u, j + SEG_BATCH);
      }
    }
  }

  // The first warp of the group's first column slice leaves the group's head record for the combine
  // kernel (after its own share of the sums, so that it costs the CTA nothing): 2 * (last group holding entries of the segment) + (partial slot of the head run) when the
  // group's LAST run opens a segment that continues into following groups and starts in this group,
  // else -1.  The decision comes from the keys already in shared memory; only a head group (rare)
  // probes the first keys of the following groups, 32 per ballot.
  if (blockIdx.y == 0 && threadIdx.x < 32 && cnt > 0) {
    const int lane = threadIdx.x;
    long long rec = -1;
    if (g0 + cnt < n) {
      const uint32_t k_last = s_key[cnt];
      int rb = cnt - 1;
      while (rb > 0 && s_key[rb] == k_last) --rb;
      const bool from_prev = rb == 0 && s_key[0] == k_last;
      if (s_key[cnt + 1] == k_last && k_last < (uint32_t)V && !from_prev) {  // warp-uniform
        long long g_end = grp;
        for (long long gb = (long long)grp + 1;; gb += 32) {
          const long long gq = gb + lane;
          const bool same = gq < n_groups && keys[gq * SEG_GROUP] == k_last;
          const int m = __popc(__ballot_sync(0xffffffffu, same));
          g_end = gb + m - 1;
          if (m < 32) break;
        }
        rec = g_end * 2 + (rb == 0 ? 0 : 1);
      }
    }
    if (lane == 0) {
      heads[grp] = rec;
      // head groups are also listed, so that the combine kernel visits nothing else; the order of the
      // list varies from run to run, the work done per entry and its result do not
      if (rec >= 0) head_list[atomicAdd(head_count, 1u)] = (uint32_t)grp;
    }
  }
}

constexpr int SEG_SPLIT = 4;  // sub-ranges of a segment's groups summed side by side in the combine kernel

// Block (tx, SEG_SPLIT), grid (about one resident wave, column slices): a CTA takes entries
// blockIdx.x, blockIdx.x + gridDim.x, ... of the list of head groups (the heads of segments that span
// several groups; few) for its column slice.  For a head group, the
// partial slots of the segment's following groups are split into SEG_SPLIT consecutive sub-ranges; thread
// row y adds its sub-range in group order (8 loads in flight), then row 0 adds
// dtable row + head partial + sub-sum 0 + ... + sub-sum 3 and writes the dtable row.  Fixed order; a
// table row is written by exactly one CTA.
template <int VW, typename TT, int SEG_GROUP>
__global__ void __launch_bounds__(SEG_THREADS * SEG_SPLIT, 2)
scatter_combine_kernel(const uint32_t* __restrict__ keys, const long long* __restrict__ heads,
                       const uint32_t* __restrict__ head_count, const uint32_t* __restrict__ head_list, TT* dtable,
                       const float* __restrict__ partials, int64_t n, int C) {
  constexpr bool BF = sizeof(TT) == 2;
  ag_pdl_wait();
  __shared__ Cols<VW> s_sub[SEG_SPLIT][SEG_THREADS];
  const int col = (blockIdx.y * blockDim.x + threadIdx.x) * VW;
  const int y = threadIdx.y;
  const uint32_t n_heads = *head_count;
  for (uint32_t hi = blockIdx.x; hi < n_heads; hi += gridDim.x) {
    const int64_t grp = head_list[hi];
    const long long rec = heads[grp];
    const int64_t g_end = rec >> 1;
    const int head_slot = (int)(rec & 1);
    const int64_t g0 = grp * SEG_GROUP;
    const int cnt = (int)((n - g0) < SEG_GROUP ? (n - g0) : SEG_GROUP);
    const uint32_t key = keys[g0 + cnt - 1];
    TT* drow = dtable + (int64_t)key * C;
    const int64_t chunk = (g_end - grp + SEG_SPLIT - 1) / SEG_SPLIT;
    Cols<VW> sub = {};
    if (col < C) {
      int64_t g = grp + 1 + y * chunk;
      int64_t ge = g + chunk;
      if (ge > g_end + 1) ge = g_end + 1;
      for (; g + 8 <= ge; g += 8) {
        Cols<VW> v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = seg_load_once<VW>(partials + ((g + k) * 2 + 0) * C + col);
#pragma unroll
        for (int k = 0; k < 8; ++k) sub += v[k];
      }
      for (; g < ge; ++g) sub += seg_load<VW>(partials + (g * 2 + 0) * C + col);
    }
    __syncthreads();  // the previous head's sub-sums have been read
    s_sub[y][threadIdx.x] = sub;
    __syncthreads();
    if (y == 0 && col < C) {
      Cols<VW> old = seg_load<VW>(drow + col);
      const Cols<VW> head = seg_load<VW>(partials + (grp * 2 + head_slot) * C + col);
      Cols<VW> acc = head;
      if (!BF) { acc = old; acc += head; }
#pragma unroll
      for (int q = 0; q < SEG_SPLIT; ++q) acc += s_sub[q][threadIdx.x];
      if (BF) { old += acc; acc = old; }
      seg_store<VW>(drow + col, acc);
    }
  }
}

struct ScatterPlan {
  int64_t n_tiles, n_groups;
  size_t off_keys[2], off_vals[2], off_hist, off_heads, off_partials, total;
};

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Sorted entries per group.  Small groups request all their rows at once and leave more CTAs to share them; a long segment
// leaves half as many partial rows for the combine kernel where they are twice as long.  Whole scatter-adds, us, in groups of
// 8 / 16 / 32 / 64 (table of 30000, Zipf-distributed): 5000 x 64 19.0 / 20.0 / 24.9 / 35.6, x 384 19.4 / 20.6 / 25.7 / 32.1, 8000 x 64
// 20.4 / 21.4 / 24.9 / 36.4, x 384 23.1 / 21.8 / 24.9 / 32.7, 16000 x 64 24.6 / 22.8 / 27.0 / 37.6, x 384 31.0 / 27.9 / 28.0 / 34.2,
// x 1536 55.1 / 48.3 / 44.9 / 48.3, 32000 x 64 32.0 / 28.4 / 31.1 / 39.8, x 384 48.4 / 40.7 / 39.0 / 38.6, x 1536 97 / 81 / 73 / 72,
// 64000 x 64 47.6 / 39.5 / 37.0 / 45.6, x 1536 195 / 155 / 133 / 124; uniform ids alike.  The line goes by elements, so that the
// longest lists of the narrowest rows take 16 where 32 are 6 % ahead.
inline int scatter_group(int64_t n, int C) {
  const int64_t elems = n * C;
  if (n >= 24576 && elems >= 8000000) return 64;
  if (elems <= 800000 || (n <= 6144 && elems <= 2500000)) return 8;
  return elems <= 4500000 ? 16 : 32;
}

// group 0: the size that the scratch is made for, that of the smallest group that the call may take
inline ScatterPlan scatter_plan(int64_t n, int C, int group = 0) {
  if (!group) {
    group = scatter_group(n, C);
    if (group > 32) group = 32;  // AG_B200_SCATTER_GROUP may ask for 32
  }
  ScatterPlan p;
  p.n_tiles = (n + SORT_TILE - 1) / SORT_TILE;
  p.n_groups = (n + group - 1) / group;
  size_t off = 0;
  for (int b = 0; b < 2; ++b) {
    p.off_keys[b] = off; off += align256((size_t)n * 4);
    p.off_vals[b] = off; off += align256((size_t)n * 4);
  }
  p.off_hist = off;  // one histogram per pass when the passes are fused (few tiles), else one in all
  off += align256((size_t)SORT_DIGITS * p.n_tiles * 4 * (p.n_tiles <= SORT_FUSED_MAX_TILES ? SORT_MAX_PASSES : 1));
  // head records: a counter (256 bytes), the record of every group, the list of head groups
  p.off_heads = off; off += 256 + align256((size_t)p.n_groups * 8) + align256((size_t)p.n_groups * 4);
  p.off_partials = off; off += align256((size_t)p.n_groups * 2 * C * 4);
  p.total = off;
  return p;
}

}  // namespace

// =========================================================================================
extern "C" int ag_gather_forward(ag_ctx* ctx, const int32_t* ids, const float* table, float* out, int64_t n_ids,
                                 int C, int V) {
  if (!ctx) return AG_ERR_INVALID;
  if (n_ids == 0) return AG_OK;
  AG_REQUIRE(ctx, ids && table && out, "ag_gather_forward: null pointer");
  AG_REQUIRE(ctx, n_ids > 0 && C > 0 && V > 0, "ag_gather_forward: bad shape n=%lld C=%d V=%d", (long long)n_ids, C, V);
  const uintptr_t bits = reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(out) | (uintptr_t)((int64_t)C * 4);
  const int vw = (bits & 15u) == 0 ? 4 : ((bits & 7u) == 0 ? 2 : 1);
  int lanes = 32;
  while (lanes > 4 && lanes / 2 >= C / vw) lanes /= 2;
  // one row per warp (or part of one) up to 32 CTAs per SM: many short CTAs keep the load/store queues fuller than a
  // resident grid whose warps loop (65536 x 1536, Zipf ids: 80.0 us against 87.4 us with 8 CTAs per SM; 16: 82.2, 64: 79.9)
  int64_t want = (n_ids * lanes + GATHER_THREADS - 1) / GATHER_THREADS;
  const int64_t cap = (int64_t)ctx->sm_count * 32;
  const int grid = (int)(want < cap ? want : cap);
#define AG_GATHER(VW, LANES)                                                                                            \
  AG_LAUNCH_PDL(ctx, "gather_forward_kernel", (gather_forward_kernel<VW, LANES>), grid, GATHER_THREADS, 0, ids, table,  \
                out, n_ids, C, V, ctx->d_status)
#define AG_GATHER_LANES(VW)                   \
  switch (lanes) {                            \
    case 4: AG_GATHER(VW, 4); break;          \
    case 8: AG_GATHER(VW, 8); break;          \
    case 16: AG_GATHER(VW, 16); break;        \
    default: AG_GATHER(VW, 32); break;        \
  }
  if (vw == 4) {
    AG_GATHER_LANES(4)
  } else if (vw == 2) {
    AG_GATHER_LANES(2)
  } else {
    AG_GATHER_LANES(1)
  }
#undef AG_GATHER_LANES
#undef AG_GATHER
  return AG_OK;
}

extern "C" size_t ag_scatter_add_scratch_bytes(int64_t n_ids, int C, int V) {
  (void)V;
  if (n_ids <= 0 || C <= 0) return 0;
  return scatter_plan(n_ids, C).total;
}

namespace {
// The segmented sum over groups of G sorted entries and the combine over the listed head groups.
template <typename TT, int G, int VW>
int launch_groups_combine(ag_ctx* ctx, const ScatterPlan& p, const uint32_t* keys, const uint32_t* pos, const float* dout,
                           TT* dtable, float* partials, long long* heads, uint32_t* head_count, uint32_t* head_list,
                           int64_t n_ids, int C, int V) {
  const int tx = 32 * VW >= C ? 32 : SEG_THREADS;
  const int ty = SEG_THREADS / tx;
  dim3 grid((unsigned)((p.n_groups + ty - 1) / ty), (unsigned)((C + tx * VW - 1) / (tx * VW)));
  // combine: one resident wave of 512-thread CTAs (two per SM, with registers for eight partial rows in flight) over
  // all column slices
  int64_t cx = (int64_t)ctx->sm_count * 2 / grid.y;
  cx = cx < 1 ? 1 : (cx > p.n_groups ? p.n_groups : cx);
  dim3 cgrid((unsigned)cx, grid.y);
  auto groups = tx == 32 ? scatter_groups_kernel<VW, TT, G, 32> : scatter_groups_kernel<VW, TT, G, SEG_THREADS>;
  auto combine = scatter_combine_kernel<VW, TT, G>;
  AG_LAUNCH_PDL(ctx, "scatter_groups_kernel", groups, grid, dim3(tx, ty), 0, keys, pos, dout, dtable, partials, heads,
                head_count, head_list, (int)p.n_groups, n_ids, C, V);
  AG_LAUNCH_PDL(ctx, "scatter_combine_kernel", combine, cgrid, dim3(tx, SEG_SPLIT), 0, keys, (const long long*)heads,
                (const uint32_t*)head_count, (const uint32_t*)head_list, dtable, (const float*)partials, n_ids, C);
  return AG_OK;
}

template <typename TT>
int gather_backward_t(ag_ctx* ctx, const int32_t* ids, const float* dout, TT* dtable, void* scratch,
                      size_t scratch_bytes, int64_t n_ids, int C, int V) {
  if (!ctx) return AG_ERR_INVALID;
  if (n_ids == 0) return AG_OK;
  AG_REQUIRE(ctx, ids && dout && dtable, "ag_gather_backward: null pointer");
  AG_REQUIRE(ctx, n_ids > 0 && C > 0 && V > 0, "ag_gather_backward: bad shape n=%lld C=%d V=%d", (long long)n_ids, C, V);
  AG_REQUIRE(ctx, n_ids < (1ll << 31) && (int64_t)V < (1ll << 31) - 1, "ag_gather_backward: sizes exceed 32-bit keys");
  const bool small = n_ids <= SORT_SMALL_MAX;
  int group = ctx->scatter_group ? ctx->scatter_group : scatter_group(n_ids, C);
  ScatterPlan p = scatter_plan(n_ids, C, group);
  // larger groups leave fewer partial rows: a scratch made for them serves
  while (!ctx->scatter_group && scratch_bytes < p.total && group < (n_ids <= SORT_SMALL_MAX ? 8 : n_ids < 49152 ? 32 : 64))
    p = scatter_plan(n_ids, C, group *= 2);
  if (!scratch || scratch_bytes < p.total)
    AG_FAIL(ctx, AG_ERR_SCRATCH, "ag_gather_backward: scratch has %zu bytes, needs %zu", scratch_bytes, p.total);
  AG_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "ag_gather_backward: scratch not 256-byte aligned");
  AG_REQUIRE(ctx, (int64_t)SORT_DIGITS * p.n_tiles < (1ll << 31) && p.n_groups < (1ll << 31) - 1,
             "ag_gather_backward: too many ids");
  // widest access that the row length and both arrays allow
  const uintptr_t dbits = reinterpret_cast<uintptr_t>(dout) | (uintptr_t)((int64_t)C * 4);
  const uintptr_t tbits = reinterpret_cast<uintptr_t>(dtable);
  const int vw = (dbits & 15u) == 0 && (tbits & 15u) == 0 ? 4 : ((dbits & 7u) == 0 && (tbits & 7u) == 0 ? 2 : 1);
  if (n_ids <= (C <= FEW_PIECES * 32 * vw ? FEW_IDS_MAX : FEW_IDS_WIDE) && !ctx->scatter_group) {
    auto few = vw == 4 ? scatter_few_kernel<4, TT> : (vw == 2 ? scatter_few_kernel<2, TT> : scatter_few_kernel<1, TT>);
    AG_LAUNCH_PDL(ctx, "scatter_few_kernel", few, (int)n_ids, FEW_THREADS, 0, ids, dout, dtable, (int)n_ids, C, V, ctx->d_status);
    return AG_OK;
  }
  unsigned char* base = static_cast<unsigned char*>(scratch);
  uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(base + p.off_keys[0]), reinterpret_cast<uint32_t*>(base + p.off_keys[1])};
  uint32_t* vals[2] = {reinterpret_cast<uint32_t*>(base + p.off_vals[0]), reinterpret_cast<uint32_t*>(base + p.off_vals[1])};
  uint32_t* hist = reinterpret_cast<uint32_t*>(base + p.off_hist);
  float* partials = reinterpret_cast<float*>(base + p.off_partials);
  uint32_t* head_count = reinterpret_cast<uint32_t*>(base + p.off_heads);
  long long* heads = reinterpret_cast<long long*>(base + p.off_heads + 256);
  uint32_t* head_list = reinterpret_cast<uint32_t*>(base + p.off_heads + 256 + align256((size_t)p.n_groups * 8));
  const int n_tiles = (int)p.n_tiles;
  // keys are in [0, V]: sort just enough 9-bit digits to cover V
  int bits = 1;
  while (((int64_t)1 << bits) <= (int64_t)V) ++bits;
  const int passes = (bits + SORT_BITS - 1) / SORT_BITS;
  int cur = 0;
  if (small) {
#define AG_SORT_SMALL(ITEMS)                                                                                                    \
  {                                                                                                                            \
    auto kern = sort_small_kernel<ITEMS>;                                                                                      \
    static std::atomic<bool> attr_done[AG_MAX_DEVICES];                                                                        \
    if (!attr_done[ag_dev_slot(ctx)].load(std::memory_order_relaxed)) { /* the same for every caller: may be done twice */     \
      AG_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_small_smem(ITEMS)));      \
      attr_done[ag_dev_slot(ctx)].store(true, std::memory_order_relaxed);                                                      \
    }                                                                                                                          \
    AG_LAUNCH_PDL(ctx, "sort_small_kernel", kern, 1, SORT_TILE, sort_small_smem(ITEMS), ids, keys[0], vals[0], head_count,     \
                  (int)n_ids, bits, V, ctx->d_status);                                                                         \
  }
    if (n_ids <= SORT_TILE) AG_SORT_SMALL(1)
    else if (n_ids <= 2 * SORT_TILE) AG_SORT_SMALL(2)
    else AG_SORT_SMALL(4)
#undef AG_SORT_SMALL
  } else if (n_tiles <= SORT_FUSED_MAX_TILES) {
    // passes + 1 launches: no key/position initialisation, no scan, no histogram launch after the first
    const int64_t hist_entries = (int64_t)SORT_DIGITS * n_tiles;
    AG_LAUNCH_PDL(ctx, "sort_hist_ids_kernel", sort_hist_ids_kernel, n_tiles, SORT_TILE, 0, ids, hist, hist + hist_entries,
                  hist_entries * (passes - 1), head_count, n_ids, V, ctx->d_status);
    for (int pass = 0; pass < passes; ++pass) {
      uint32_t* h = hist + hist_entries * pass;
      uint32_t* h_next = pass + 1 < passes ? h + hist_entries : nullptr;
      if (pass == 0) {
        AG_LAUNCH_PDL(ctx, "sort_scatter_fused_kernel", sort_scatter_fused_kernel<true>, n_tiles, SORT_TILE, 0, ids,
                      (const uint32_t*)nullptr, (const uint32_t*)nullptr, keys[1], vals[1], (const uint32_t*)h, h_next,
                      n_ids, V, 0, n_tiles);
        cur = 1;
      } else {
        AG_LAUNCH_PDL(ctx, "sort_scatter_fused_kernel", sort_scatter_fused_kernel<false>, n_tiles, SORT_TILE, 0,
                      (const int32_t*)nullptr, (const uint32_t*)keys[cur], (const uint32_t*)vals[cur], keys[cur ^ 1],
                      vals[cur ^ 1], (const uint32_t*)h, h_next, n_ids, V, pass * SORT_BITS, n_tiles);
        cur ^= 1;
      }
    }
  } else {
    AG_LAUNCH_PDL(ctx, "sort_init_kernel", sort_init_kernel, n_tiles, SORT_TILE, 0, ids, keys[0], vals[0], head_count,
                  n_ids, V, ctx->d_status);
    for (int shift = 0; shift < bits; shift += SORT_BITS) {
      AG_LAUNCH_PDL(ctx, "sort_hist_kernel", sort_hist_kernel, n_tiles, SORT_TILE, 0, (const uint32_t*)keys[cur], hist,
                    n_ids, shift, n_tiles);
      AG_LAUNCH_PDL(ctx, "sort_scan_kernel", sort_scan_kernel, 1, 1024, 0, hist, (int64_t)SORT_DIGITS * n_tiles);
      AG_LAUNCH_PDL(ctx, "sort_scatter_kernel", sort_scatter_kernel, n_tiles, SORT_TILE, 0, (const uint32_t*)keys[cur],
                    (const uint32_t*)vals[cur], keys[cur ^ 1], vals[cur ^ 1], (const uint32_t*)hist, n_ids, shift, n_tiles);
      cur ^= 1;
    }
  }
#define AG_GROUPS(G)                                                                                                       \
  {                                                                                                                        \
    auto fn = vw == 4 ? launch_groups_combine<TT, G, 4> : (vw == 2 ? launch_groups_combine<TT, G, 2> : launch_groups_combine<TT, G, 1>); \
    return fn(ctx, p, keys[cur], vals[cur], dout, dtable, partials, heads, head_count, head_list, n_ids, C, V);            \
  }
  switch (group) {
    case 128: AG_GROUPS(128)
    case 64: AG_GROUPS(64)
    case 16: AG_GROUPS(16)
    case 32: AG_GROUPS(32)
    default: AG_GROUPS(8)
  }
#undef AG_GROUPS
}
}  // namespace

extern "C" int ag_gather_backward(ag_ctx* ctx, const int32_t* ids, const float* dout, float* dtable, void* scratch,
                                  size_t scratch_bytes, int64_t n_ids, int C, int V) {
  return gather_backward_t<float>(ctx, ids, dout, dtable, scratch, scratch_bytes, n_ids, C, V);
}

extern "C" int ag_gather_backward_bf16(ag_ctx* ctx, const int32_t* ids, const float* dout, uint16_t* dtable,
                                       void* scratch, size_t scratch_bytes, int64_t n_ids, int C, int V) {
  return gather_backward_t<uint16_t>(ctx, ids, dout, dtable, scratch, scratch_bytes, n_ids, C, V);
}
