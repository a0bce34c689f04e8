// tcgen05 tensor-core panels of the fused linear + cross-entropy head and of the projection.
//
// One persistent GEMM kernel, D[M,N] (+)= A[M,K] . B[N,K]^T, each operand read from memory either
// K-major ([MN][K], K contiguous) or MN-major ([K][MN], MN contiguous):
//   warp 0      : TMA producer  - cp.async.bulk.tensor tiles (128-byte swizzle) into a ring of
//                 shared-memory stages, completion on mbarriers;
//   warp 1      : allocates TMEM, then one elected lane issues tcgen05.mma (M = 128, N = BN with
//                 cta_group::1; M = 256 over a pair of CTAs with cta_group::2) from shared-memory
//                 descriptors into one of two TMEM accumulators; tcgen05.commit releases stages and
//                 publishes accumulators;
//   warps 4..11 : epilogue - tcgen05.ld of the finished accumulator (one TMEM lane = one output
//                 row per thread) into registers, then store / accumulate to global memory, while the
//                 MMA warp already works in the other accumulator.
// A launch carries one or two problems (see TcLaunch), so that two independent GEMMs fill each other's
// last round over the SMs.
//
// Bound: the tensor pipe at the power cap (94-96 % active at 1.5 GHz for the logits and dlogits panels of
// 16384 x 4096 x 1280, 0.29 and 0.30 ms); plain bf16 and the column-bound pass, whose MMAs are a third, by
// the operand bytes from L2 (about 40 per clock and SM).  Against tf32 pairs (0.55 logits, 0.59 dlogits, 0.65 dX,
// 0.58 dW) the same panel now takes 0.29, 0.30, 0.69 for both products, and 0.15 for the column bounds of dl.
//
// Operand modes:
//   F16X3  : every fp32 operand is split once into fp16 (hi, lo) after scaling by a power of two per row
//            (or column, where the contraction index is the row index), each k-step issues
//            hi*lo + lo*hi + hi*hi into the same fp32 accumulator, and the epilogue takes the scales out.
//            fp16 has the 11-bit significand of tf32, so a pair holds the same 22 bits and more; the scale
//            puts the largest element of the row at 2^14, so that elements down to 2^-17 of it keep all of
//            them and smaller ones err by at most 2^-40 of the largest.  Operands that are wide along the
//            contraction are balanced first (see TcBalance), so that this is measured by products that the
//            output contains and not by a large element that meets a small one.  The weight gradient of
//            the head is not: its rows err by 2^-40 of (the column's bound of dl) x (the sum of the column
//            of X, each row with its loss scale).  Twice the MMA rate of tf32 on half the operand bytes.
//   BF16   : operands rounded to bf16 once, a single MMA per k-step.
//   BF16X3 : hi = bf16(x), lo = bf16(x - hi), three MMAs at the bf16 rate (products to ~2^-17).
// Accumulation inside the tensor core truncates, with a bias that grows with the length of the chain
// (dW over 16384 rows in tf32: 2.7e-4 of the rms with one chain, 3.6e-5 with 8).  Every mode therefore ends a
// chain after `chain` k-steps, at most 768 elements in the split modes and 8192 in the others: the epilogue warps add
// the finished accumulator to the tile in their registers, round-to-nearest, while the MMA warp continues in the other
// accumulator (128 fp32 values per warp lane; 0.3 us of TMEM reads and adds against 3-4 us of MMAs per chain).
// The three GEMMs of the head read X, W and dl as stored; no transposed copy exists:
//   logits  = X   . W^T       A = X  [rows,C] K-major     B = W [vc,C]   K-major
//   dX     += dl  . W         A = dl [rows,vc] K-major    B = W [vc,C]   MN-major (contraction over vc)
//   dW     += dl^T. X         A = dl [rows,vc] MN-major   B = X [rows,C] MN-major (contraction over rows)
// An MN-major tile is fetched as one 3-d TMA box {128 bytes of MN, 64 k-rows, MN groups} (one 2-d box per
// group when the MN extent is ragged) and described to the MMA with the transposing descriptor forms
// (see TcDesc).
// Every output tile has exactly one writer, so accumulation order is fixed.
// Every mbarrier wait is bounded; on expiry the CTA raises AG_STATUS_WAIT_EXPIRED, all roles
// leave their loops, TMEM is released and the kernel returns.  Larger problems run on clusters
// of two CTAs (see tc_gemm_kernel); every CTA loads its own tiles with plain (single-destination) TMA
// loads.
#include <cuda.h>
#include <cuda_fp16.h>

#include <atomic>

#include "ag_flce.cuh"
#include "ag_tc.cuh"

namespace {

// Warps 0-3: TMA producer, MMA issuer, two idle (registers move between warp groups of four); 4-11: epilogue.
// The 168 registers a thread that the block starts with are shared out again as 4 x 32 x 56 and 8 x 32 x 224
// (64512 both ways): an epilogue thread holds 128 sums while it adds up chains.
constexpr int TC_EPI_WARPS = 8;
constexpr int TC_EPI_SLICES = TC_EPI_WARPS / 4;  // column slices of a tile; the four warps of a slice share its rows
constexpr int TC_ACC = 8 / TC_EPI_SLICES;        // 32-column chunks of a 256-column tile per warp, at most
constexpr int TC_THREADS = 128 + 32 * TC_EPI_WARPS;
// Longest chain of single products, in elements of K.  Terms of one sign lose 3.0e-5 of their sum in it, 7.6e-5 with
// 16384 elements and 7.9e-4 with 131072 (dW over 2 million rows).
constexpr int TC_CHAIN_SINGLE = 8192;
constexpr int TC_MAX_STAGES = 6;
constexpr int TC_SMEM_LIMIT = 227 * 1024;
constexpr int TC_WARP_STAGING = 3072;  // per epilogue warp: 32 rows of 64 bytes on their way to memory, 1 KB of column factors
constexpr int TC_STAGING = TC_EPI_WARPS * TC_WARP_STAGING;
constexpr int TC_SMEM_FIXED = 1024 + TC_STAGING + 256;  // alignment slack, staging, barriers

// operand modes (AgTcMode of ag_flce.cuh)
enum { TC_BF16 = AG_TC_BF16, TC_BF16X3 = AG_TC_BF16X3, TC_F16X3 = AG_TC_F16X3, TC_F16HI };  // F16HI: hi parts only
constexpr bool tc_mode_split(int mode) { return mode == TC_BF16X3 || mode == TC_F16X3; }
constexpr bool tc_mode_f16(int mode) { return mode == TC_F16X3 || mode == TC_F16HI; }

// STORE_FEW: see the kernel; STATS_KEEP: EPI_STATS that also writes the logits
enum { EPI_STORE = 0, EPI_STATS = 1, EPI_DLOGITS = 2, EPI_COLMAX = 3, EPI_STORE_FEW = 4, EPI_STATS_KEEP = 5 };
constexpr bool tc_epi_stats(int epi) { return epi == EPI_STATS || epi == EPI_STATS_KEEP; }

// One GEMM of a launch.
struct TcProblem {
  int M, N, K;
  int BN;              // tile width, multiple of 32, <= 256
  int split;           // operands come as (hi, lo) pairs and 3 MMAs are issued per k-step
  int tiles_m, tiles_n, k_iters;
  int splits;          // split-K: each output tile is computed by `splits` CTAs over disjoint k ranges
  int k_per_split;     // k iterations per split (the last one may be shorter)
  int chain;           // k iterations accumulated in TMEM before the sum moves to registers
  int64_t split_stride;  // elements between the partial outputs of consecutive splits
  int a_mn, b_mn;      // operand is MN-major in memory ([K][MN], MN contiguous) instead of K-major ([MN][K])
  int a_3d, b_3d;      // MN-major operand fetched as one 3-d box {MN group, TC_BK, groups} instead of one box per group
  int n_fastest;       // tile order: column tiles vary first ...
  int group_n;         // ... within groups of this many (the B rows of a group stay in L2)
  uint32_t idesc;
  uint32_t b_bytes;    // bytes of one B tile in a stage (an A tile has 128 x 128)
  float* D;
  int64_t ldd;
  int accumulate;
  const float* row_mul;  // scales of an F16X3 product: acc * row_mul[row] * col_mul[col] (null: 1)
  const float* col_mul;
  // EPI_STORE extras of the linear+bias+residual op: out = acc + bias[col] + resid[row][col]
  const float* bias;
  const float* resid;
  int64_t ld_resid;
};

// Fields of the fused cross-entropy epilogues; row-indexed arrays start at A's row 0.
struct TcHead {
  const int32_t* targets;
  int v0;                  // vocabulary index of column 0 of this panel
  int V;
  float2* part;            // EPI_STATS: per (column tile, slice, row) partial (max, sum exp), [2 tiles_n][part_ld]
  int64_t part_ld;
  float* tgt_logit;        // EPI_STATS: logit of the target column, written by the tile that holds it
  uint32_t* ticket;        // EPI_STATS: cleared for the kernel that follows
  float* logits;           // EPI_STATS_KEEP: row-indexed as A, column 0 is vocabulary index 0
  int64_t ld_logits;       // a multiple of 32
  const float* lse;        // EPI_DLOGITS
  const float* row_scale;
  const float* dloss;
  const float* denom;
  int ignore_mode;
  int dl_form;             // EPI_DLOGITS: operand mode of dl
  void* dl_hi;             // EPI_DLOGITS output: dl [M][ld_dl]; F16X3: (p - onehot) * 2^col_exp[col], without the row's scale
  void* dl_lo;
  int64_t ld_dl;
  const float* col_exp;    // F16X3: 14 + the exponent by which column v0 + col is scaled up (see EPI_COLMAX)
  // EPI_COLMAX: col_dist[v] = min over rows of a lower bound on lse - logit, i.e. e^-col_dist bounds |p - onehot|
  // of the column from above.  One product of the hi parts is enough; row_slack[row] * w_norm[col] bounds its error.
  uint32_t* col_dist;      // bits of a non-negative float
  const float* row_slack;
  const float* w_norm;     // norm of the row of W behind every column
  // The columns of dl are scaled up by 2^s, the rows of W that dX takes down: w_cap = max over rows of their largest
  // element (w_top) times 2^-s, so that an unlikely token's row, however large, does not set the scale of the others.
  const float* w_top;
  uint32_t* w_cap;         // bits of a non-negative float
};

// Which output tiles a unit (a CTA, or a pair of CTAs) computes: the n0 tiles of problem 0, which are the
// more expensive ones, are dealt round-robin; units that got one fewer (those from `heavy` on) first take
// `extra` tiles of problem 1 each; what remains of problem 1 is dealt round-robin again.
struct TcSchedule {
  int n0, n1, heavy, extra;
};

struct TcLaunch {
  CUtensorMap a_hi[2], a_lo[2], b_hi[2], b_lo[2];
  TcProblem pr[2];
  TcHead head;
  TcSchedule sched;
  int stages;
  uint32_t stage_bytes;
  int* status;
};

// ---------------------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ void tc_tma_load_2d(const CUtensorMap* tm, void* smem_dst, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          ag_smem_u32(smem_dst)),
      "l"(tm), "r"(ag_smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

__device__ __forceinline__ void tc_tma_load_3d(const CUtensorMap* tm, void* smem_dst, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          ag_smem_u32(smem_dst)),
      "l"(tm), "r"(ag_smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// ---- CTA pair (thread-block cluster of 2) helpers
__device__ __forceinline__ uint32_t tc_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t tc_map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void tc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// commit whose mbarrier may live in either CTA of the pair
__device__ __forceinline__ void tc_commit_pair(uint32_t cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_addr) : "memory");
}
// tile loads of a CTA of the pair: destination in the own shared memory, completion bytes counted on
// the mbarrier at `mbar_cluster_addr`, which is the leader's
__device__ __forceinline__ void tc_tma_load_2d_pair(const CUtensorMap* tm, void* smem_dst, uint32_t mbar_cluster_addr,
                                                    int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
          "r"(ag_smem_u32(smem_dst)),
      "l"(tm), "r"(mbar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tc_tma_load_3d_pair(const CUtensorMap* tm, void* smem_dst, uint32_t mbar_cluster_addr,
                                                    int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];" ::"r"(ag_smem_u32(smem_dst)),
      "l"(tm), "r"(mbar_cluster_addr), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// ---------------------------------------------------------------------------- tile schedule
struct TcItem {
  int prob, tm, tn, k_begin, k_end, split;
};

// The `step`-th piece of work of this unit; false when there is none left.
__device__ __forceinline__ bool tc_item(const TcLaunch& L, int unit, int units, int step, TcItem& it) {
  const TcSchedule& s = L.sched;
  const int mine0 = unit < s.n0 ? (s.n0 - 1 - unit) / units + 1 : 0;
  int tile;
  if (step < mine0) {
    it.prob = 0;
    tile = unit + step * units;
  } else {
    it.prob = 1;
    step -= mine0;
    const int light = units - s.heavy;
    if (unit >= s.heavy) {
      tile = step < s.extra ? step * light + (unit - s.heavy) : s.extra * light + (step - s.extra) * units + unit;
    } else {
      tile = s.extra * light + step * units + unit;
    }
    if (tile >= s.n1) return false;
  }
  const TcProblem& p = L.pr[it.prob];
  const int per_split = p.tiles_m * p.tiles_n;
  it.split = tile / per_split;
  tile -= it.split * per_split;
  it.k_begin = it.split * p.k_per_split;
  it.k_end = it.k_begin + p.k_per_split < p.k_iters ? it.k_begin + p.k_per_split : p.k_iters;
  if (p.n_fastest) {  // column tiles of a group first, then the row tiles, then the next group
    const int grp = tile / (p.tiles_m * p.group_n);
    tile -= grp * p.tiles_m * p.group_n;
    const int first = grp * p.group_n, width = p.tiles_n - first < p.group_n ? p.tiles_n - first : p.group_n;
    it.tm = tile / width;
    it.tn = first + tile - it.tm * width;
  } else {
    it.tn = tile / p.tiles_m;
    it.tm = tile - it.tn * p.tiles_m;
  }
  return true;
}

// two floats -> (hi, lo) fp16 pairs, packed two to a word
__device__ __forceinline__ void split_f16x2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void split_bf16x2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const float2 f = __bfloat1622float2(h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(x - f.x, y - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ void tc_st_global_v8(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// 32 columns of the lane's row of dl as fp16 or bf16 pairs (dst_lo null: hi only), `cols` of them inside the padded
// row (a multiple of 16).  A lane's 32 bytes are a whole sector, so nothing is gained by passing shared memory, whose
// bandwidth the MMAs need (panel of 16384 x 4096 x 384: 189 us this way, 212 us in 64-byte rows through shared memory).
template <bool BF16>
__device__ __forceinline__ void tc_store_pair16(const float (&v)[32], uint16_t* dst_hi, uint16_t* dst_lo, int cols) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (j * 16 >= cols) continue;
    uint32_t hi[8], lo[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (BF16) split_bf16x2(v[16 * j + 2 * k], v[16 * j + 2 * k + 1], hi[k], lo[k]);
      else split_f16x2(v[16 * j + 2 * k], v[16 * j + 2 * k + 1], hi[k], lo[k]);
    }
    tc_st_global_v8(dst_hi + 16 * j, hi);
    if (dst_lo) tc_st_global_v8(dst_lo + 16 * j, lo);
  }
}

// f[col .. col + 3]; f is a vector of the output's columns, 16-byte aligned where the output's rows are
__device__ __forceinline__ float4 tc_load_cols(const float* f, int col, int n) {
  if (col + 4 <= n && (reinterpret_cast<uintptr_t>(f + col) & 15u) == 0) return *reinterpret_cast<const float4*>(f + col);
  return make_float4(col < n ? f[col] : 0.f, col + 1 < n ? f[col + 1] : 0.f, col + 2 < n ? f[col + 2] : 0.f,
                     col + 3 < n ? f[col + 3] : 0.f);
}

// All MMAs of one stage: 4 steps of 32 bytes along K, three products each for (hi, lo) operands.
template <bool SPLIT, bool PAIR>
__device__ __forceinline__ void tc_stage_mmas(uint32_t tacc, uint32_t ah, uint32_t al, uint32_t a_step,
                                              uint32_t bh, uint32_t bl, uint32_t b_step, uint32_t idesc,
                                              uint32_t not_first) {
  constexpr uint32_t a_hi = TcDesc::hi, b_hi = TcDesc::hi;
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    const uint32_t ao = (uint32_t)kk * a_step, bo = (uint32_t)kk * b_step;
    if (SPLIT) {
      if (kk == 0)
        tc_mma<2, PAIR>(tacc, ah + ao, a_hi, bl + bo, b_hi, idesc, not_first);
      else
        tc_mma<1, PAIR>(tacc, ah + ao, a_hi, bl + bo, b_hi, idesc, 1u);
      tc_mma<1, PAIR>(tacc, al + ao, a_hi, bh + bo, b_hi, idesc, 1u);
      tc_mma<1, PAIR>(tacc, ah + ao, a_hi, bh + bo, b_hi, idesc, 1u);
    } else {
      if (kk == 0)
        tc_mma<2, PAIR>(tacc, ah + ao, a_hi, bh + bo, b_hi, idesc, not_first);
      else
        tc_mma<1, PAIR>(tacc, ah + ao, a_hi, bh + bo, b_hi, idesc, 1u);
    }
  }
}

// How far (in powers of two) a column of dl whose elements are at most e^-dist is scaled up: the exponent of TcHead::col_exp
__device__ __forceinline__ float tc_dist_shift(float dist) { return floorf(fminf(dist * kLog2e, 100.0f)); }
__device__ __forceinline__ float tc_pow2(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

// ---------------------------------------------------------------------------- the kernel
// PAIR: launched as clusters of two CTAs that share every 256-row output tile (see tc_mma): CTA `rank`
// owns rows [128 rank, 128 rank + 128) of the tile and loads its own A rows and half of the B columns,
// so a pair pulls a third less operand data through shared memory than two single CTAs.  All stage
// barriers that the MMA waits on live in the leader (rank 0); the leader's commits arrive on the
// barriers of both CTAs.
template <int EPI, bool PAIR>
__global__ void __launch_bounds__(TC_THREADS, 1) tc_gemm_kernel(const __grid_constant__ TcLaunch L) {
  constexpr bool STORE = EPI == EPI_STORE || EPI == EPI_STORE_FEW;
  extern __shared__ unsigned char tc_smem_raw[];
  // tiles need 1024-byte alignment for the 128-byte swizzle pattern
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t stage_bytes = L.stage_bytes;
  unsigned char* staging = tiles + (size_t)L.stages * stage_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + TC_STAGING);
  uint64_t* full = bars;
  uint64_t* empty = bars + TC_MAX_STAGES;
  uint64_t* acc_full = bars + 2 * TC_MAX_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? tc_cluster_rank() : 0u;
  // this CTA's (pair's) position in the stream of output tiles, and the number of positions
  const int unit = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int units = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int row_off = PAIR ? (int)rank * TC_BM : 0;        // first row of this CTA inside the tile
  const int bm_tile = PAIR ? 2 * TC_BM : TC_BM;            // rows of an output tile
  constexpr uint32_t A_BYTES = TC_BM * 128;

  if (threadIdx.x == 0) {
    for (int s = 0; s < L.stages; ++s) {
      ag_mbar_init(&full[s], 1);
      ag_mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ag_mbar_init(&acc_full[b], 1);
      ag_mbar_init(&acc_empty[b], PAIR ? 2 * TC_EPI_WARPS : TC_EPI_WARPS);  // one arrival per epilogue warp (of both CTAs)
    }
    *abort_flag = 0;
    ag_fence_mbar_init();
  }
  if (PAIR) tc_cluster_sync(); else __syncthreads();  // the peer's barriers exist before anything arrives on them
  if (warp == 1) {
    // 512 columns: two accumulators of up to 256 fp32 columns each (this kernel owns the SM)
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ag_smem_u32(tmem_slot)),
                   "r"(512u)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ag_smem_u32(tmem_slot)),
                   "r"(512u)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool expired = false;
  // Everything above touched no global memory and may overlap the tail of the previous kernel of the
  // stream; from here on its results are read.  No trigger for the next kernel: beside 227 KB of shared memory none of its CTAs
  // finds room anyway, and where they move in one by one as these leave, an SM is never empty and its L1 stays what is left beside
  // so much shared memory.  Norms that trigger early hand that on from kernel to kernel: the backward pass of 20 layers after the
  // head took 16.2 ms instead of 13.2.  Nor does a trigger pay beside products of 10 to 100 us (forward + backward, us, with / without):
  // heads 1000 x 768 x 8000 228 / 220, 2048 x 1024 x 8192 415 / 407, 4096 x 384 x 8192 418 / 419, bf16x3 4096 x 256 x 2048 126 / 117;
  // projections 2048 x 1536 x 1536 176.1 / 175.4, 1024 x 2048 x 2048 150 / 149, 16384 x 512 x 768 295 / 288, bf16 4096 x 1024 x 1024
  // 103 / 100.
  ag_pdl_wait();
  if (tc_epi_stats(EPI) && blockIdx.x == 0 && threadIdx.x == 0) *L.head.ticket = 0u;

  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      TcItem it;
      for (int step = 0; !expired && tc_item(L, unit, units, step, it); ++step) {
        const TcProblem& p = L.pr[it.prob];
        const CUtensorMap *ta_hi = &L.a_hi[it.prob], *ta_lo = &L.a_lo[it.prob], *tb_hi = &L.b_hi[it.prob],
                          *tb_lo = &L.b_lo[it.prob];
        const int bn_cta = PAIR ? p.BN / 2 : p.BN;               // B columns this CTA loads
        const int split = p.split;
        const int a_mn = p.a_mn, b_mn = p.b_mn, a_3d = p.a_3d, b_3d = p.b_3d;
        const uint32_t b_bytes = p.b_bytes;
        const uint32_t item_bytes = (A_BYTES + b_bytes) * (split ? 2u : 1u);
        const int m0 = it.tm * bm_tile + row_off, n0 = it.tn * p.BN + (PAIR ? (int)rank * bn_cta : 0);
        for (int k = it.k_begin; k < it.k_end; ++k) {
          if (!tc_wait(&empty[stage], phase ^ 1u, abort_flag)) {
            expired = true;
            break;
          }
          unsigned char* s = tiles + (size_t)stage * stage_bytes;
          // pair: the leader's barrier counts the bytes of both CTAs' loads; a completion that arrives
          // before the leader has posted its expectation only makes the pending count negative for a while
          uint32_t full_addr = ag_smem_u32(&full[stage]);
          if (PAIR) {
            if (rank == 0) ag_mbar_expect_tx(&full[stage], 2u * item_bytes);
            full_addr = tc_map_to_cta(full_addr, 0u);
          } else {
            ag_mbar_expect_tx(&full[stage], item_bytes);
          }
          const int kx = k * TC_BK;
          // K-major operand: one box {TC_BK, rows}.  MN-major operand: one box {128 bytes of MN, TC_BK rows} per
          // MN group, stored group after group.
          constexpr uint32_t gbytes = (uint32_t)TC_BK * 128u;
          auto load_operand = [&](const CUtensorMap* tm, unsigned char* dst, int mn0, int mn_rows, int mn_major, int is3d) {
            if (PAIR) {
              if (!mn_major) {
                tc_tma_load_2d_pair(tm, dst, full_addr, kx, mn0);
              } else if (is3d) {
                tc_tma_load_3d_pair(tm, dst, full_addr, 0, kx, mn0 / TC_MN_GROUP);
              } else {
                for (int g = 0; g * TC_MN_GROUP < mn_rows; ++g)
                  tc_tma_load_2d_pair(tm, dst + (size_t)g * gbytes, full_addr, mn0 + g * TC_MN_GROUP, kx);
              }
            } else if (!mn_major) {
              tc_tma_load_2d(tm, dst, &full[stage], kx, mn0);
            } else if (is3d) {
              tc_tma_load_3d(tm, dst, &full[stage], 0, kx, mn0 / TC_MN_GROUP);
            } else {
              for (int g = 0; g * TC_MN_GROUP < mn_rows; ++g)
                tc_tma_load_2d(tm, dst + (size_t)g * gbytes, &full[stage], mn0 + g * TC_MN_GROUP, kx);
            }
          };
          load_operand(ta_hi, s, m0, TC_BM, a_mn, a_3d);
          if (split) {
            load_operand(ta_lo, s + A_BYTES, m0, TC_BM, a_mn, a_3d);
            load_operand(tb_hi, s + 2 * A_BYTES, n0, bn_cta, b_mn, b_3d);
            load_operand(tb_lo, s + 2 * A_BYTES + b_bytes, n0, bn_cta, b_mn, b_3d);
          } else {
            load_operand(tb_hi, s + A_BYTES, n0, bn_cta, b_mn, b_3d);
          }
          if (++stage == (uint32_t)L.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (pair: the leader only)
    if (lane == 0 && rank == 0) {
      uint32_t stage = 0, phase = 0;
      uint32_t acc_par = 0;  // phase bits of the two accumulators' "free" barriers
      int buf = 0;
      const uint32_t stage_units = stage_bytes >> 4;
      const uint32_t tiles_u = ag_smem_u32(tiles) >> 4;
      TcItem it;
      for (int step = 0; !expired && tc_item(L, unit, units, step, it); ++step) {
        // Everything an MMA needs beyond two additions is prepared outside the k loop: this one thread
        // issues 12 (split operands) or 4 MMAs per stage and its instruction stream is on the critical path.
        const TcProblem& p = L.pr[it.prob];
        TcDesc dA, dB;
        dA.init(p.a_mn);
        dB.init(p.b_mn);
        const int split = p.split, chain = p.chain;
        const uint32_t b_lo_off = p.b_bytes >> 4, idesc = p.idesc;
        const uint32_t b_off = (split ? 2u * A_BYTES : A_BYTES) >> 4;
        uint32_t tacc = 0;
        int left = 0;  // k-steps left in the current accumulation chain
        for (int k = it.k_begin; k < it.k_end; ++k) {
          uint32_t not_first = 1u;
          if (left == 0) {
            if (!tc_wait(&acc_empty[buf], ((acc_par >> buf) & 1u) ^ 1u, abort_flag)) {
              expired = true;
              break;
            }
            acc_par ^= 1u << buf;
            tacc = tmem_base + (uint32_t)buf * 256u;
            left = it.k_end - k < chain ? it.k_end - k : chain;
            not_first = 0u;
          }
          if (!tc_wait(&full[stage], phase, abort_flag)) {
            expired = true;
            break;
          }
          tc_fence_after();
          const uint32_t su = tiles_u + stage * stage_units;
          const uint32_t ah = su + dA.lo_const, al = ah + (A_BYTES >> 4);  // A hi / lo tiles
          const uint32_t bh = su + b_off + dB.lo_const, bl = bh + b_lo_off;
          if (split)
            tc_stage_mmas<true, PAIR>(tacc, ah, al, dA.step, bh, bl, dB.step, idesc, not_first);
          else
            tc_stage_mmas<false, PAIR>(tacc, ah, al, dA.step, bh, bl, dB.step, idesc, not_first);
          // stage reusable once these MMAs have read it (pair: in both CTAs)
          if (PAIR) {
            const uint32_t e = ag_smem_u32(&empty[stage]);
            tc_commit_pair(tc_map_to_cta(e, 0u));
            tc_commit_pair(tc_map_to_cta(e, 1u));
          } else {
            tc_commit(&empty[stage]);
          }
          if (++stage == (uint32_t)L.stages) {
            stage = 0;
            phase ^= 1u;
          }
          if (--left == 0) {  // accumulator complete (pair: each CTA's epilogue waits on its own barrier)
            if (PAIR) {
              const uint32_t f = ag_smem_u32(&acc_full[buf]);
              tc_commit_pair(tc_map_to_cta(f, 0u));
              tc_commit_pair(tc_map_to_cta(f, 1u));
            } else {
              tc_commit(&acc_full[buf]);
            }
            buf ^= 1;
          }
        }
      }
    }
  }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 4..11)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    // Two warps share each TMEM lane quarter, one for each slice of the tile's columns.
    const int quarter = warp & 3;  // TMEM lanes [32*quarter, 32*quarter+32) are this warp's
    const int slice = (warp - 4) >> 2;
    unsigned char* stg = staging + (warp - 4) * TC_WARP_STAGING;
    uint32_t full_par = 0;
    int buf = 0;
    float cap = 0.0f;  // EPI_COLMAX: the lane's part of w_cap; the smallest distance of a column gives its largest value
    TcItem it = {};
    auto tile_epilogue = [&](const TcProblem& p) {
      const int n_chunks = p.BN >> 5;
      const int more = n_chunks % TC_EPI_SLICES, each = n_chunks / TC_EPI_SLICES;
      const int c_first = slice * each + (slice < more ? slice : more);  // first 32-column chunk of this warp
      const int n_mine = each + (slice < more ? 1 : 0);                  // and how many it has (at most TC_ACC)
      const int row0 = it.tm * bm_tile + row_off + quarter * 32;  // first row of the warp's block
      const int row = row0 + lane;
      const int col0 = it.tn * p.BN + c_first * 32;
      const int rows = p.M - row0 < 32 ? p.M - row0 : 32;         // rows of the block inside the output
      // What belongs to the tile's rows and columns is requested before the accumulator is waited for: beside 227 KB
      // of shared memory there is next to no L1, and the latency of L2 after the wait cost more than the arithmetic.
      const TcHead& h = L.head;
      const bool row_in = row < p.M;
      const float fac = p.row_mul && row_in ? p.row_mul[row] : 1.0f;
      const int target = !STORE && row_in ? h.targets[row] : -1;
      float e = 0.0f, sc = 0.0f, slack = 0.0f;
      if (EPI == EPI_DLOGITS && row_in) {
        e = h.lse[row];
        sc = h.row_scale ? h.dloss[0] * h.row_scale[row] : h.dloss[0] / h.denom[0];
      }
      if (EPI == EPI_COLMAX && row_in) {
        e = h.lse[row];
        slack = h.row_slack[row];
      }
      float4 cols0 = make_float4(1.f, 1.f, 1.f, 1.f), cols1 = make_float4(0.f, 0.f, 0.f, 0.f);  // of columns col0 + 4 lane ..
      if (lane < n_mine * 8) {
        if (p.col_mul) cols0 = tc_load_cols(p.col_mul, col0 + 4 * lane, p.N);
        if (EPI == EPI_DLOGITS && h.col_exp) cols1 = tc_load_cols(h.col_exp, col0 + 4 * lane, p.N);
        if (EPI == EPI_COLMAX) cols1 = tc_load_cols(h.w_norm, col0 + 4 * lane, p.N);
      }
      auto wait_full = [&]() {
        if (!tc_wait(&acc_full[buf], (full_par >> buf) & 1u, abort_flag)) {
          expired = true;
          return false;
        }
        full_par ^= 1u << buf;
        tc_fence_after();
        return true;
      };
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR)
            tc_mbar_arrive_cluster(tc_map_to_cta(ag_smem_u32(&acc_empty[buf]), 0u));  // the leader's MMA thread waits
          else
            ag_mbar_arrive(&acc_empty[buf]);
        }
        buf ^= 1;
      };
      const uint32_t toff = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c_first * 32u;
      // the columns' factors reach every lane through shared memory
      const float4* colf = reinterpret_cast<const float4*>(stg + 2048);
      if (p.col_mul) {
        __syncwarp();
        reinterpret_cast<float4*>(stg + 2048)[lane] = cols0;
        if (EPI == EPI_DLOGITS) reinterpret_cast<float4*>(stg + 2048)[32 + lane] = cols1;
        __syncwarp();
      }
      const bool valid = !STORE && target >= 0 && target < h.V;
      int tcol = STORE ? -1 : target - h.v0 - col0;  // target column relative to the warp's first
      if (EPI == EPI_DLOGITS || EPI == EPI_COLMAX) tcol = row_in && valid ? tcol : -1;
      // EPI_STATS: running (max, sum exp) of the row over the warp's columns
      float mx = -INFINITY, sum = 0.0f, tl = 0.0f;
      bool found = false;
      // EPI_DLOGITS
      const bool scaled = h.dl_form == TC_F16X3;
      if (EPI == EPI_DLOGITS && !valid && h.ignore_mode == AG_CE_IGNORE_MASKED) sc = 0.0f;
      const bool live = sc != 0.0f;
      const bool all_live = EPI == EPI_DLOGITS && __all_sync(0xffffffffu, live);
      // EPI_COLMAX
      float base = 3.0e38f;
      if (EPI == EPI_COLMAX) {
        const float wn = fmaxf(fmaxf(cols1.x, cols1.y), fmaxf(cols1.z, cols1.w));
        const float w_max = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(wn)));  // norms: not negative
        if (row_in && (valid || h.ignore_mode != AG_CE_IGNORE_MASKED)) base = fmaf(slack, -w_max, e);
      }
      // EPI_STORE
      const bool vec = STORE && ((p.ldd & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.D) & 15u) == 0) &&
                       ((p.split_stride & 3) == 0) &&
                       (!p.resid || (((p.ld_resid & 3) == 0) && (reinterpret_cast<uintptr_t>(p.resid) & 15u) == 0));
      float* D = p.D + (int64_t)it.split * p.split_stride + (int64_t)row0 * p.ldd;

      auto chunk = [&](const int c, float(&v)[32]) {
        const int col = col0 + c * 32;
        if (p.col_mul) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 x = colf[c * 8 + (j >> 2)];
            v[j] *= x.x; v[j + 1] *= x.y; v[j + 2] *= x.z; v[j + 3] *= x.w;
          }
        }
        const int hit = tcol - c * 32;
        if (STORE) {
          if (p.row_mul) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] *= fac;
          }
          if (rows > 0) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const int cc = col + half * 16;
              if (cc < p.N)
                tc_store_cols16(stg, lane, v + half * 16, D + cc, p.ldd, rows, p.N - cc, vec, p.accumulate,
                                p.bias ? p.bias + cc : nullptr,
                                p.resid ? p.resid + (int64_t)row0 * p.ld_resid + cc : nullptr, p.ld_resid);
            }
          }
        } else if (tc_epi_stats(EPI)) {
          // logit = v * fac with fac > 0, so the maximum is taken of the sums, and logit - max is one fused
          // multiply-add without the logit being rounded first
          const int n_valid = p.N - col;
          if (n_valid < 32) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j >= n_valid) v[j] = -INFINITY;  // contributes nothing below
          }
          if (EPI == EPI_STATS_KEEP && row_in && n_valid > 0) {  // whole 32-byte sectors; fac is a power of two: exact
            float* dst = h.logits + (int64_t)row * h.ld_logits + h.v0 + col;
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint32_t o[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) o[k] = __float_as_uint(v[j + k] * fac);
              tc_st_global_v8(dst + j, o);
            }
          }
          if (hit >= 0 && hit < 32 && hit < n_valid) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j == hit) tl = v[j];
            found = true;
          }
          float top = v[0];
#pragma unroll
          for (int j = 1; j < 32; ++j) top = fmaxf(top, v[j]);
          if (top > mx) {
            sum *= tc_exp2((mx - top) * fac * kLog2e);  // 0 the first time
            mx = top;
          }
          const float shift = mx == -INFINITY ? 0.0f : mx * fac;
          float part = 0.0f;
#pragma unroll
          for (int j = 0; j < 32; ++j) part += tc_exp2(fmaf(v[j], fac, -shift) * kLog2e);
          sum += part;
        } else if (EPI == EPI_DLOGITS) {
          if (scaled) {
            // q = (p - onehot) 2^col_exp, the row's scale is applied by the products
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 x = colf[32 + c * 8 + (j >> 2)];
              v[j] = tc_exp2(fmaf(fmaf(v[j], fac, -e), kLog2e, x.x));
              v[j + 1] = tc_exp2(fmaf(fmaf(v[j + 1], fac, -e), kLog2e, x.y));
              v[j + 2] = tc_exp2(fmaf(fmaf(v[j + 2], fac, -e), kLog2e, x.z));
              v[j + 3] = tc_exp2(fmaf(fmaf(v[j + 3], fac, -e), kLog2e, x.w));
            }
            if (hit >= 0 && hit < 32) {
              const float one = tc_exp2(reinterpret_cast<const float*>(colf + 32)[tcol]);
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (j == hit) v[j] -= one;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = tc_exp2((v[j] - e) * kLog2e);
            if (hit >= 0 && hit < 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (j == hit) v[j] -= 1.0f;
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] *= sc;
          }
          if (!all_live) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = live ? v[j] : 0.0f;
          }
          if (row_in && col < p.N) {
            const int64_t at = (int64_t)row * h.ld_dl + col;
            const int cols = (int)(h.ld_dl - col < 32 ? h.ld_dl - col : 32);  // the padded row's columns may be written
            uint16_t *hi = static_cast<uint16_t*>(h.dl_hi) + at, *lo = static_cast<uint16_t*>(h.dl_lo) + at;
            if (scaled)
              tc_store_pair16<false>(v, hi, lo, cols);
            else
              tc_store_pair16<true>(v, hi, h.dl_form == TC_BF16X3 ? lo : nullptr, cols);
          }
        } else {
          // distance of every column's largest logit from the row's lse, at most (see TcHead); at the target |p - 1|
          // may be as large as 1: distance 0
          uint32_t mine = 0;
          const float w_top = col + lane < p.N ? h.w_top[col + lane] : 0.0f;
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = fmaxf(fmaf(v[j], -fac, base), 0.0f);
          if (hit >= 0 && hit < 32) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j == hit) v[j] = 0.0f;
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const uint32_t m = __reduce_min_sync(0xffffffffu, __float_as_uint(v[j]));
            mine = lane == j ? m : mine;
          }
          if (col + lane < p.N) atomicMin(h.col_dist + col + lane, mine);
          cap = fmaxf(cap, w_top * tc_pow2(-(int)tc_dist_shift(__uint_as_float(mine))));
        }
      };
      if (!STORE && it.k_end - it.k_begin <= p.chain) {
        // One chain: straight from tensor memory, by one copy of the code for all chunks.  Where K is this short the
        // epilogue sets the time of a tile, and unrolled code that every tile runs through once is fetched anew each
        // time (16384 x 4096 x 384: 81 us instead of 66 for the column bounds, 205 instead of 162 for dlogits).
        if (!wait_full()) return;
#pragma unroll 1
        for (int c = 0; c < n_mine; ++c) {
          float v[32];
          tc_tmem_ld32(toff + (uint32_t)buf * 256u + (uint32_t)c * 32u, reinterpret_cast<uint32_t(&)[32]>(v));
          tc_tmem_ld_wait();
          chunk(c, v);
        }
        release();
      } else {
        // Several: added up in registers, in k order, so that the last accumulator is free before the stores
        float acc[TC_ACC][32];
        for (int k = it.k_begin; k < it.k_end; k += p.chain) {
          if (!wait_full()) return;
          const uint32_t t = toff + (uint32_t)buf * 256u;
          if (k == it.k_begin) {
#pragma unroll
            for (int c = 0; c < TC_ACC; ++c)
              if (c < n_mine) tc_tmem_ld32(t + (uint32_t)c * 32u, reinterpret_cast<uint32_t(&)[32]>(acc[c]));
            tc_tmem_ld_wait();
          } else {
#pragma unroll
            for (int c = 0; c < TC_ACC; ++c) {
              if (c < n_mine) {
                uint32_t r[32];
                tc_tmem_ld32(t + (uint32_t)c * 32u, r);
                tc_tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[c][j] += __uint_as_float(r[j]);
              }
            }
          }
          release();
        }
        if (EPI == EPI_STORE_FEW) {
          // A launch with a tile or two per unit is a chain of latencies, of which fetching code is one: a single copy
          // of it, the chunks move up to acc[0] one after the other (333 x 5003 x 392: 38 -> 33 us).  Otherwise the
          // moves cost energy that the tensor pipe at its power cap wants (16384 x 4096 x 1280: 720 against 696 us).
#pragma unroll 1
          for (int c = 0; c < n_mine; ++c) {
            chunk(c, acc[0]);
#pragma unroll
            for (int k = 1; k < TC_ACC; ++k)
#pragma unroll
              for (int j = 0; j < 32; ++j) acc[k - 1][j] = acc[k][j];
          }
        } else {
#pragma unroll
          for (int c = 0; c < TC_ACC; ++c)
            if (c < n_mine) chunk(c, acc[c]);
        }
      }
      if (tc_epi_stats(EPI) && row_in) {
        // a slice that saw no valid column (narrow last tile) contributes (max -inf, sum 0)
        h.part[(int64_t)(it.tn * TC_EPI_SLICES + slice) * h.part_ld + row] = make_float2(mx * fac, sum);
        if (found) h.tgt_logit[row] = tl * fac;
      }
    };
    for (int step = 0; !expired && tc_item(L, unit, units, step, it); ++step) {
      tile_epilogue(L.pr[STORE ? it.prob : 0]);
    }
    if (EPI == EPI_COLMAX) {
      const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(cap));
      if (lane == 0) atomicMax(L.head.w_cap, top);
    }
  }
  if (expired && lane == 0) atomicOr(L.status, AG_STATUS_WAIT_EXPIRED);
  tc_fence_before();
  // pair: neither CTA may leave, or free its tensor memory, while the other can still read its shared
  // memory or arrive on its barriers
  if (PAIR) tc_cluster_sync(); else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// ---------------------------------------------------------------------------- host side
// The driver API is reached through the runtime (cudaGetDriverEntryPoint) so that the library has
// no link-time dependency on libcuda and still loads on a machine without a driver.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn tc_encode_fn(ag_ctx* ctx) {
  static std::atomic<EncodeTiledFn> known{nullptr};
  EncodeTiledFn fn = known.load(std::memory_order_relaxed);
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !p) {
      snprintf(ctx->err, sizeof ctx->err, "cuTensorMapEncodeTiled is not available from this driver: %s",
               cudaGetErrorString(e));
      return nullptr;
    }
    fn = reinterpret_cast<EncodeTiledFn>(p);
    known.store(fn, std::memory_order_relaxed);
  }
  return fn;
}

// Tensor map of one operand array.  K-major [mn][K]: box {TC_BK, rows}.  MN-major [K][mn]: seen as
// {group, K, groups}, one box {group, TC_BK, groups of the tile} lands in shared memory as [group][k row][128 bytes];
// a ragged MN extent takes one box {group, TC_BK} per group instead.
int tc_encode(ag_ctx* ctx, CUtensorMap* tm, int mode, const void* ptr, int mn_major, int64_t mn, int64_t K, int64_t ld,
              int tile_rows) {
  EncodeTiledFn encode = tc_encode_fn(ctx);
  if (!encode) return AG_ERR_CUDA;
  constexpr int bk = TC_BK, group = TC_MN_GROUP;
  const bool is3d = mn_major && mn % group == 0;
  cuuint64_t dims[3], strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)group * 2};
  cuuint32_t box[3], estr[3] = {1, 1, 1};
  if (!mn_major) {
    dims[0] = (cuuint64_t)K; dims[1] = (cuuint64_t)mn;
    box[0] = (cuuint32_t)bk; box[1] = (cuuint32_t)tile_rows;
  } else if (is3d) {
    dims[0] = (cuuint64_t)group; dims[1] = (cuuint64_t)K; dims[2] = (cuuint64_t)(mn / group);
    box[0] = (cuuint32_t)group; box[1] = (cuuint32_t)bk; box[2] = (cuuint32_t)(tile_rows / group);
  } else {
    dims[0] = (cuuint64_t)mn; dims[1] = (cuuint64_t)K;
    box[0] = (cuuint32_t)group; box[1] = (cuuint32_t)bk;
  }
  const CUtensorMapDataType type = tc_mode_f16(mode) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUresult r = encode(tm, type, is3d ? 3 : 2, const_cast<void*>(ptr), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    AG_FAIL(ctx, AG_ERR_CUDA, "cuTensorMapEncodeTiled failed: CUresult %d (ptr %p, mn %lld, K %lld, ld %lld, box %ux%u)", (int)r,
            ptr, (long long)mn, (long long)K, (long long)ld, box[0], box[1]);
  return AG_OK;
}

// D[m][n] (+)= sum over splits, in split order, of the partial outputs P[s][m][n].
// VEC: N, ldd multiples of 4 and 16-byte aligned pointers: one 16-byte packet per thread and split,
// all splits' packets requested before the first add.
template <bool VEC>
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* __restrict__ P, int splits, int M, int N, float* D, int64_t ldd, int accumulate) {
  ag_pdl_wait();
  const int64_t total = (int64_t)M * N;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if (VEC) {
    const int n4 = N >> 2;
    const int64_t packets = (int64_t)M * n4;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < packets; i += stride) {
      const int m = (int)(i / n4), n = (int)(i - (int64_t)m * n4) << 2;
      float4* d = reinterpret_cast<float4*>(D + (int64_t)m * ldd + n);
      const float* src = P + (int64_t)m * N + n;
      float4 acc = accumulate ? *d : make_float4(0.f, 0.f, 0.f, 0.f);
      int sp = 0;
      for (; sp + 4 <= splits; sp += 4) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = __ldcs(reinterpret_cast<const float4*>(src + (int64_t)(sp + u) * total));
#pragma unroll
        for (int u = 0; u < 4; ++u) { acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w; }
      }
      for (; sp < splits; ++sp) {
        const float4 v = __ldcs(reinterpret_cast<const float4*>(src + (int64_t)sp * total));
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
      *d = acc;
    }
  } else {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
      const int m = (int)(i / N), n = (int)(i - (int64_t)m * N);
      float* d = D + (int64_t)m * ldd + n;
      float acc = accumulate ? *d : 0.0f;
      for (int sp = 0; sp < splits; ++sp) acc += P[(int64_t)sp * total + i];
      *d = acc;
    }
  }
}

// Largest number of CTA pairs (clusters of 2) of the kernel that are resident at once; 0 on error.
int tc_max_pairs(ag_ctx* ctx) {
  static std::atomic<int> known[AG_MAX_DEVICES];  // 1 + the answer
  std::atomic<int>& c = known[ag_dev_slot(ctx)];
  if (const int k = c.load(std::memory_order_relaxed)) return k - 1;
  auto kern = tc_gemm_kernel<EPI_STORE, true>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_LIMIT) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * ctx->sm_count);
  cfg.blockDim = dim3(TC_THREADS);
  cfg.dynamicSmemBytes = TC_SMEM_LIMIT;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    n = 0;
  }
  c.store(1 + n, std::memory_order_relaxed);
  return n;
}

template <int EPI, bool PAIR>
int tc_launch(ag_ctx* ctx, int grid, size_t smem, const TcLaunch& L) {
  static std::atomic<bool> attr_done[AG_MAX_DEVICES];
  auto kern = tc_gemm_kernel<EPI, PAIR>;
  if (!attr_done[ag_dev_slot(ctx)].load(std::memory_order_relaxed)) {  // the same for every caller: may be done twice
    AG_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_LIMIT));
    attr_done[ag_dev_slot(ctx)].store(true, std::memory_order_relaxed);
  }
  int rc_ev;
  if (ctx->tc_timing && (rc_ev = ag_event_record(ctx, ctx->tc_timing_base + 2 * ctx->tc_timing_count))) return rc_ev;
  {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[2];
    int n_at = 0;
    if (PAIR) {
      at[n_at].id = cudaLaunchAttributeClusterDimension;
      at[n_at].val.clusterDim.x = 2;
      at[n_at].val.clusterDim.y = 1;
      at[n_at].val.clusterDim.z = 1;
      ++n_at;
    }
    if (ctx->pdl) {
      at[n_at].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[n_at].val.programmaticStreamSerializationAllowed = 1;
      ++n_at;
    }
    cfg.attrs = at;
    cfg.numAttrs = n_at;
    AG_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, L));
    ctx->launches++;
    ag_enqueued(ctx);
  }
  if (ctx->tc_timing) {
    if ((rc_ev = ag_event_record(ctx, ctx->tc_timing_base + 2 * ctx->tc_timing_count + 1))) return rc_ev;
    ctx->tc_timing_count++;
  }
  return AG_OK;
}

struct TcOperand {
  const void* hi;
  const void* lo;   // null in bf16 mode
  int64_t ld;       // elements between consecutive rows of the array as stored
  int mn_major;     // 0: stored [MN][K] (K contiguous); 1: stored [K][MN] (MN contiguous)
};

struct TcGemm {
  int mode = TC_BF16;
  TcOperand A = {}, B = {};
  int M = 0, N = 0, K = 0;
  float* D = nullptr;
  int64_t ldd = 0;
  bool accumulate = false;
  const float *row_mul = nullptr, *col_mul = nullptr, *bias = nullptr, *resid = nullptr;
  int64_t ld_resid = 0;
  float* ws = nullptr;      // split-K partial outputs
  size_t ws_bytes = 0;
  int chain_elems = 0;      // longest accumulation chain in elements of K; 0: the default of the mode
};

// ---- the shape of a launch.  Costs in SM clocks, fitted to measurements:
//   a k-step takes the longer of its MMAs (4096 multiply-adds per clock) and of the
//   operand bytes that the CTA pulls from L2 (about 40 per clock: 128 A rows and the B rows it loads, BN or
//   BN / 2 as one CTA of a pair);
//   the epilogue of a tile overlaps the next tile's main loop, the last one of a unit does not;
//   units (CTAs or pairs) work in rounds over the SMs, so the number of tiles left over by a round counts.
struct TcShape {
  int bn, splits, k_per;
  int64_t tiles;      // over all splits
  double tile_cost;
};

double tc_kstep_cost(int mode, int bn, int bn_cta) {
  const int parts = tc_mode_split(mode) ? 2 : 1;
  const double mma = (parts == 2 ? 6.0 : 2.0) * bn, load = (128.0 + bn_cta) * 128.0 * parts / 40.0;
  return (mma > load ? mma : load) + 16.0;
}

// Clocks per column of the epilogues alone.  With 64 for dlogits the model took tiles of 128 columns where K is short,
// whose main loop then set the time (16384 x 4096 x 384: 162 us, with pairs and 256 columns 133).
// Stores of a result of 2^21 elements and more, partial ones counted, are bound by memory, all units at it at once: with
// the cost of a store on its own the model cut the contraction of the small dX finely and dealt units both products,
// where dW of a short batch (K = its rows) is nothing but stores (64 rows x 768 x 50000: 274 -> 165 us for both
// products, 256 x 1024 x 50000 318 -> 240, 100 x 512 x 20000 62 -> 50).
double tc_epilogue_cost(int epi, bool accumulate, int bn, int64_t elems) {
  if (epi == EPI_DLOGITS) return 300.0 + bn * 52.0;
  if (epi == EPI_STATS) return 300.0 + bn * 40.0;
  if (epi == EPI_STATS_KEEP) return 300.0 + bn * 52.0;
  if (epi == EPI_COLMAX) return 300.0 + bn * 30.0;
  return 300.0 + bn * (elems >= (1 << 21) ? (accumulate ? 70.0 : 35.0) : (accumulate ? 16.0 : 8.0));
}

TcShape tc_shape(const TcGemm& g, bool pair, int bn, int splits, int epi) {
  TcShape s;
  const int k_iters = (g.K + TC_BK - 1) / TC_BK;
  s.bn = bn;
  s.k_per = (k_iters + splits - 1) / splits;
  s.splits = (k_iters + s.k_per - 1) / s.k_per;
  const int bm = pair ? 2 * TC_BM : TC_BM;
  s.tiles = (int64_t)((g.M + bm - 1) / bm) * ((g.N + bn - 1) / bn) * s.splits;
  const double main = s.k_per * tc_kstep_cost(g.mode, bn, pair ? bn / 2 : bn);
  const double e = tc_epilogue_cost(epi, g.accumulate && s.splits == 1, bn, (int64_t)g.M * g.N * s.splits);
  s.tile_cost = (main > e ? main : e) + 100.0;
  return s;
}

// Clocks that the ordered reduction of the partial outputs adds: a launch, and its traffic at about 3500 bytes a clock.
double tc_reduce_cost(const TcGemm& g, int splits) {
  return splits > 1 ? 3000.0 + (double)g.M * g.N * 4.0 * (2 * splits + 2) / 3500.0 : 0.0;
}

int tc_max_splits(const TcGemm& g) {
  if (!g.ws) return 1;
  int64_t fit = (int64_t)(g.ws_bytes / ((size_t)g.M * g.N * sizeof(float)));
  const int k_iters = (g.K + TC_BK - 1) / TC_BK;
  if (fit > 16) fit = 16;
  if (fit > k_iters / 2) fit = k_iters / 2;
  return fit < 1 ? 1 : (int)fit;
}

// Longest path over the units when s0's tiles (the costlier ones) are dealt first (see TcSchedule).
double tc_makespan(const TcShape& s0, const TcShape* s1, int units, TcSchedule* out) {
  const int64_t base = s0.tiles / units;
  const int heavy = (int)(s0.tiles % units), light = units - heavy;
  TcSchedule sc = {(int)s0.tiles, s1 ? (int)s1->tiles : 0, heavy, 0};
  double best;
  if (!s1) {
    best = (double)(base + (heavy ? 1 : 0)) * s0.tile_cost;
  } else {
    best = 1e300;
    const int64_t lim = s1->tiles / units + 2;
    for (int64_t q = 0; q <= lim; ++q) {  // tiles of problem 1 on the units that have one tile of problem 0 more
      int64_t left = s1->tiles - q * heavy;
      if (left < 0) left = 0;
      int64_t ql = (left + light - 1) / light;
      if (ql < q) ql = q;
      double span = (double)base * s0.tile_cost + (double)ql * s1->tile_cost;
      if (heavy) {
        const double h = (double)(base + 1) * s0.tile_cost + (double)q * s1->tile_cost;
        if (h > span) span = h;
      }
      if (span < best) {
        best = span;
        sc.extra = (int)(ql - q);
      }
      if (!heavy) break;
    }
  }
  if (out) *out = sc;
  return best;
}

constexpr int kTcWidths[] = {256, 192, 128, 96, 64, 32};
constexpr int kTcSplits[] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 16};

bool tc_width_fits(const TcGemm& g, bool pair, int bn, int min_bn) {
  const int bn_cta = pair ? bn / 2 : bn;
  if (bn < min_bn) return false;
  if (pair && bn % 32 != 0) return false;
  return !(g.B.mn_major && bn_cta % TC_MN_GROUP != 0);
}

struct TcPlanned {
  TcShape shape[2];
  TcSchedule sched;
  bool pair;
};

void tc_choose(ag_ctx* ctx, const TcGemm* g, int n, int epi, int min_bn, TcPlanned* out) {
  double best = 1e300;
  const int n_pairs = ctx->tc_pair ? tc_max_pairs(ctx) : 0;
  for (int pair = 0; pair <= 1; ++pair) {
    if (pair && (n_pairs < 1 || (g[0].M <= TC_BM && (n < 2 || g[1].M <= TC_BM)))) continue;
    const int units = pair ? n_pairs : ctx->sm_count;
    // two problems: the width of each is chosen by its own cost, then the splits jointly
    int widths[2][6], n_widths[2] = {0, 0};
    for (int i = 0; i < n; ++i) {
      double w_best = 1e300;
      for (int bn : kTcWidths) {
        if (!tc_width_fits(g[i], pair, bn, min_bn)) continue;
        if (n == 1) {
          widths[i][n_widths[i]++] = bn;
          continue;
        }
        const TcShape s = tc_shape(g[i], pair, bn, 1, epi);
        const double c = (double)s.tiles * s.tile_cost;
        if (c < w_best) {
          w_best = c;
          widths[i][0] = bn;
          n_widths[i] = 1;
        }
      }
    }
    if (!n_widths[0] || (n == 2 && !n_widths[1])) continue;
    const int max0 = tc_max_splits(g[0]), max1 = n == 2 ? tc_max_splits(g[1]) : 1;
    for (int w = 0; w < n_widths[0]; ++w) {
      for (int s0 : kTcSplits) {
        if (s0 > max0) break;
        const TcShape a = tc_shape(g[0], pair, widths[0][w], s0, epi);
        if (n == 1) {
          TcSchedule sc;
          const double c = tc_makespan(a, nullptr, units, &sc) +
                           tc_epilogue_cost(epi, false, a.bn, (int64_t)g[0].M * g[0].N * a.splits) + tc_reduce_cost(g[0], a.splits);
          if (c < best) {
            best = c;
            *out = TcPlanned{{a, a}, sc, pair != 0};
          }
          continue;
        }
        for (int s1 : kTcSplits) {
          if (s1 > max1) break;
          const TcShape b = tc_shape(g[1], pair, widths[1][0], s1, epi);
          const bool swap = b.tile_cost > a.tile_cost;
          TcSchedule sc;
          const double c = tc_makespan(swap ? b : a, swap ? &a : &b, units, &sc) + tc_reduce_cost(g[0], a.splits) +
                           tc_reduce_cost(g[1], b.splits);
          if (c < best) {
            best = c;
            *out = TcPlanned{{a, b}, sc, pair != 0};
          }
        }
      }
    }
  }
}

int tc_fill_problem(ag_ctx* ctx, const TcGemm& g, const TcShape& s, bool pair, int units, int epi, TcLaunch& L, int i) {
  TcProblem& p = L.pr[i];
  const int bm = pair ? 2 * TC_BM : TC_BM, bn_cta = pair ? s.bn / 2 : s.bn;
  p.M = g.M; p.N = g.N; p.K = g.K;
  p.BN = s.bn;
  p.split = tc_mode_split(g.mode) ? 1 : 0;
  p.tiles_m = (g.M + bm - 1) / bm;
  p.tiles_n = (g.N + s.bn - 1) / s.bn;
  p.k_iters = (g.K + TC_BK - 1) / TC_BK;
  p.splits = s.splits;
  p.k_per_split = s.k_per;
  // Chains of equal length, of at most 768 elements: with 256 instead the gradients err half as much (9e-7 against
  // 2e-6 of the rms; unlimited tf32 chains had 2.4e-5) and their two products take 5 % longer.  Single products (2e-2)
  // run on to TC_CHAIN_SINGLE: what the accumulator cuts off grows with the chain whatever the operands are rounded to.
  const int most = g.chain_elems ? (g.chain_elems + TC_BK - 1) / TC_BK : (p.split ? 12 : TC_CHAIN_SINGLE / TC_BK);
  const int parts = (p.k_per_split + most - 1) / most;
  p.chain = (p.k_per_split + parts - 1) / parts;
  p.split_stride = 0;
  p.a_mn = g.A.mn_major ? 1 : 0;
  p.b_mn = g.B.mn_major ? 1 : 0;
  p.a_3d = (p.a_mn && g.M % TC_MN_GROUP == 0) ? 1 : 0;
  p.b_3d = (p.b_mn && g.N % TC_MN_GROUP == 0) ? 1 : 0;
  p.b_bytes = (uint32_t)bn_cta * 128u;
  // the tile order keeps the re-read operand of a round in L2
  const int64_t ab = (int64_t)bm * 128, bb = (int64_t)s.bn * 128;
  const int64_t fp_m_fast = (p.tiles_m < units ? p.tiles_m : units) * ab + ((units + p.tiles_m - 1) / p.tiles_m) * bb;
  const int64_t fp_n_fast = (p.tiles_n < units ? p.tiles_n : units) * bb + ((units + p.tiles_n - 1) / p.tiles_n) * ab;
  p.n_fastest = fp_n_fast <= fp_m_fast ? 1 : 0;
  // columns in groups whose B operand takes a third of L2: it is read from memory once, A once per group
  const int64_t b_tile = (int64_t)s.bn * g.K * 2 * (p.split ? 2 : 1);
  int64_t group = (int64_t)(ctx->l2_bytes / 3) / (b_tile > 0 ? b_tile : 1);
  if (group < 4) group = 4;
  p.group_n = group < p.tiles_n ? (int)group : p.tiles_n;
  // instruction descriptor: D fp32, A/B type (fp16 0, bf16 1), operand majors, N>>3 at bit 17, M>>4 at bit 24 (M = 256
  // for the instruction that spans a CTA pair)
  const uint32_t fmt = tc_mode_f16(g.mode) ? 0u : 1u;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)p.a_mn << 15) | ((uint32_t)p.b_mn << 16) |
            ((uint32_t)(p.BN >> 3) << 17) | ((uint32_t)(bm >> 4) << 24);
  p.D = g.D; p.ldd = g.ldd; p.accumulate = g.accumulate ? 1 : 0;
  p.row_mul = g.row_mul; p.col_mul = g.col_mul;
  p.bias = g.bias; p.resid = g.resid; p.ld_resid = g.ld_resid;
  if (p.splits > 1) {  // partial outputs [splits][M][N] in the workspace, summed in order afterwards
    p.D = g.ws;
    p.ldd = g.N;
    p.accumulate = 0;
    p.split_stride = (int64_t)g.M * g.N;
  }
  int rc;
  if ((rc = tc_encode(ctx, &L.a_hi[i], g.mode, g.A.hi, p.a_mn, g.M, g.K, g.A.ld, TC_BM))) return rc;
  if ((rc = tc_encode(ctx, &L.b_hi[i], g.mode, g.B.hi, p.b_mn, g.N, g.K, g.B.ld, bn_cta))) return rc;
  L.a_lo[i] = L.a_hi[i];
  L.b_lo[i] = L.b_hi[i];
  if (p.split) {
    if ((rc = tc_encode(ctx, &L.a_lo[i], g.mode, g.A.lo, p.a_mn, g.M, g.K, g.A.ld, TC_BM))) return rc;
    if ((rc = tc_encode(ctx, &L.b_lo[i], g.mode, g.B.lo, p.b_mn, g.N, g.K, g.B.ld, bn_cta))) return rc;
  }
  const uint32_t stage = (TC_BM * 128u + p.b_bytes) * (p.split ? 2u : 1u);
  if (stage > L.stage_bytes) L.stage_bytes = stage;
  return AG_OK;
}

// One launch of one or two independent GEMMs (two: plain stores only).  `head` carries the fields of the fused
// cross-entropy epilogues; min_bn bounds the tile width from below (the partial statistics have a fixed place).
int tc_gemm(ag_ctx* ctx, const TcGemm* g, int n, int epi = EPI_STORE, const TcHead* head = nullptr, int min_bn = 32,
            int* tiles_n_out = nullptr) {
  TcPlanned pl;
  tc_choose(ctx, g, n, epi, min_bn, &pl);
  const int units = pl.pair ? tc_max_pairs(ctx) : ctx->sm_count;
  TcLaunch L = {};
  if (head) L.head = *head;
  L.sched = pl.sched;
  L.status = ctx->d_status;
  const int order[2] = {n == 2 && pl.shape[1].tile_cost > pl.shape[0].tile_cost ? 1 : 0, 0};
  int64_t total = 0;
  for (int i = 0; i < n; ++i) {
    const int from = i == 0 ? order[0] : 1 - order[0];
    int rc = tc_fill_problem(ctx, g[from], pl.shape[from], pl.pair, units, epi, L, i);
    if (rc) return rc;
    total += pl.shape[from].tiles;
  }
  if (tiles_n_out) *tiles_n_out = L.pr[0].tiles_n;
  int stages = (TC_SMEM_LIMIT - TC_SMEM_FIXED) / (int)L.stage_bytes;
  if (stages > TC_MAX_STAGES) stages = TC_MAX_STAGES;
  AG_REQUIRE(ctx, stages >= 2, "tc_gemm: tile does not fit shared memory");
  L.stages = stages;
  const size_t smem = TC_SMEM_FIXED + (size_t)stages * L.stage_bytes;
  // the schedule deals tiles to `grid` units: with two problems every unit exists, with one a unit without a
  // tile is not launched
  int grid = units;
  if (n == 1 && total < units) {
    grid = (int)total;
    L.sched.heavy = 0;
  }
  if (pl.pair) grid *= 2;
  int rc;
  if (epi == EPI_STATS)
    rc = pl.pair ? tc_launch<EPI_STATS, true>(ctx, grid, smem, L) : tc_launch<EPI_STATS, false>(ctx, grid, smem, L);
  else if (epi == EPI_STATS_KEEP)
    rc = pl.pair ? tc_launch<EPI_STATS_KEEP, true>(ctx, grid, smem, L) : tc_launch<EPI_STATS_KEEP, false>(ctx, grid, smem, L);
  else if (epi == EPI_COLMAX)
    rc = pl.pair ? tc_launch<EPI_COLMAX, true>(ctx, grid, smem, L) : tc_launch<EPI_COLMAX, false>(ctx, grid, smem, L);
  else if (epi == EPI_DLOGITS)
    rc = pl.pair ? tc_launch<EPI_DLOGITS, true>(ctx, grid, smem, L) : tc_launch<EPI_DLOGITS, false>(ctx, grid, smem, L);
  else if (total <= 2 * (int64_t)units)
    rc = pl.pair ? tc_launch<EPI_STORE_FEW, true>(ctx, grid, smem, L) : tc_launch<EPI_STORE_FEW, false>(ctx, grid, smem, L);
  else
    rc = pl.pair ? tc_launch<EPI_STORE, true>(ctx, grid, smem, L) : tc_launch<EPI_STORE, false>(ctx, grid, smem, L);
  if (rc) return rc;
  for (int i = 0; i < n; ++i) {
    const int splits = pl.shape[i].splits;
    if (splits == 1) continue;
    const TcGemm& q = g[i];
    const int64_t n4 = ((int64_t)q.M * q.N + 3) / 4;
    int64_t want = (n4 + 255) / 256;
    if (want > (int64_t)ctx->sm_count * 8) want = (int64_t)ctx->sm_count * 8;
    const bool vec = (q.N % 4 == 0) && (q.ldd % 4 == 0) && ag_aligned16(q.D) && ag_aligned16(q.ws);
    if (vec)
      AG_LAUNCH_PDL(ctx, "splitk_reduce_kernel", splitk_reduce_kernel<true>, (int)want, 256, 0, (const float*)q.ws, splits,
                    q.M, q.N, q.D, q.ldd, q.accumulate ? 1 : 0);
    else
      AG_LAUNCH_PDL(ctx, "splitk_reduce_kernel", splitk_reduce_kernel<false>, (int)want, 256, 0, (const float*)q.ws, splits,
                    q.M, q.N, q.D, q.ldd, q.accumulate ? 1 : 0);
  }
  return AG_OK;
}

// ---------------------------------------------------------------------------- operand preparation
// src[R][Cc] (row stride lds) -> bf16 operand form [R][Cc] (row stride ldo): (hi, lo) pairs, or values in `hi`.
// Cc, lds and ldo are multiples of 4; one thread converts 4 consecutive elements.
template <bool PAIR>
__global__ void __launch_bounds__(256)
split_bf16_kernel(const float* __restrict__ src, int64_t lds, uint16_t* __restrict__ hi, uint16_t* __restrict__ lo, int64_t ldo,
                  int R, int Cc) {
  ag_pdl_wait();
  const int c4 = Cc >> 2;
  const int64_t total = (int64_t)R * c4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int64_t r = i / c4;
    const int c = (int)(i - r * c4) << 2;
    const float4 x = *reinterpret_cast<const float4*>(src + r * lds + c);
    uint2 h, l;
    split_bf16x2(x.x, x.y, h.x, l.x);
    split_bf16x2(x.z, x.w, h.y, l.y);
    *reinterpret_cast<uint2*>(hi + r * ldo + c) = h;
    if (PAIR) *reinterpret_cast<uint2*>(lo + r * ldo + c) = l;
  }
}

// Scale of an F16X3 row or column whose largest finite |element| has the bits `maxbits`: the power of two that
// puts it into [2^14, 2^15), and its inverse.  Maxima below 2^-112 (and all-zero rows) are scaled as 2^-112 would be.
__device__ __forceinline__ void tc_scale(uint32_t maxbits, float& mul, float& inv) {
  int e = (int)(maxbits >> 23) - 127;
  if (e < -112) e = -112;
  mul = __uint_as_float((uint32_t)(127 + 14 - e) << 23);
  inv = __uint_as_float((uint32_t)(127 - 14 + e) << 23);
}
__device__ __forceinline__ void tc_put_f16x4(const float4& v, __half* hi, __half* lo) {
  uint2 h, l;
  split_f16x2(v.x, v.y, h.x, l.x);
  split_f16x2(v.z, v.w, h.y, l.y);
  *reinterpret_cast<uint2*>(hi) = h;
  *reinterpret_cast<uint2*>(lo) = l;
}

// One scale per row or column makes the smallest elements of a long vector err by 2^-40 of its largest one.  That is far
// below fp32 unless the other operand is small just where this one is large (an outlier channel with small weights).  So
// the contraction index is balanced first: the operand whose maxima at every index are known is brought to the same
// maximum everywhere (`up`), the other one takes the inverse factors, and their products stay.  With equal maxima, what
// an element loses is at most 2^-39 of (largest of its row) x (largest of its column) after balancing, a product that
// the output contains.  Powers of two: exact.  An index at 2^-d of the largest maximum is multiplied by 2^d and 2^-d; d
// stops at 126.  Maxima within 2^TC_BALANCED of each other (most operands) are left as they are: 2^-31 at worst.
constexpr int TC_BALANCED = 8;
struct TcBalance {
  const uint32_t* max;     // bits of the largest |element| at every index; null: no balancing
  const uint32_t* bounds;  // the largest of them, and the largest complement (the smallest one) of those that are not
                           // zero; null: every block looks them all up itself
  int up;
};
struct TcBalanceNow {  // what a block knows of it
  uint32_t top;
  bool apply;
};
__device__ __forceinline__ float tc_balance(uint32_t max, const TcBalanceNow& b, int up) {
  const int d = min((int)(b.top >> 23) - (int)(max >> 23), 126);
  return tc_pow2(up ? d : -d);
}
// The bounds over n maxima; called by all 256 threads
__device__ __forceinline__ TcBalanceNow tc_balance_now(const TcBalance& b, int n, uint2 (&s_bounds)[8]) {
  if (!b.max) return {0u, false};
  uint32_t top = 0u, below = 0u;
  if (b.bounds) {
    top = b.bounds[0];
    below = b.bounds[1];
  } else {
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += 256) {
      const uint32_t m = b.max[i];
      top = max(top, m);
      if (m) below = max(below, ~m);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    below = __reduce_max_sync(0xffffffffu, below);
    if ((threadIdx.x & 31) == 0) s_bounds[threadIdx.x >> 5] = make_uint2(top, below);
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      top = max(top, s_bounds[w].x);
      below = max(below, s_bounds[w].y);
    }
  }
  return {top, (int)(top >> 23) - (int)(~below >> 23) > TC_BALANCED};
}

// A conversion to scaled fp16 pairs, or a part of one; several independent ones share a launch.
//   ROWS    pair scaled per row, inv[r] takes the scale out; norm[r] (may be null) = norm_mul * the row's
//           norm as it is converted; max[r] (may be null) the row's largest |element| before balancing.  `bal` goes by
//           column.
//   ROWMAX  bits of the largest |element| of every row; the bounds of them (see TcBalance) by integer atomic maxima, where
//           `bounds` (zero at first) is given.
//   COLMAX  bits of the largest |element| of every column, by integer atomic maxima (order-free) that start at zero.
//   COLMAX1 the same by one block per 32 columns: for up to TC_FEW_ROWS rows, needs no cleared words.
//   COLS    pair scaled per column from known maxima, which *cap (may be null) bounds too; inv[c] takes the scale out.
//           `again`: found once more, 32 columns per block, if the rows have to be balanced.
//   COLS1   COLMAX and COLS by one block per 128 columns: for up to TC_COLS1_ROWS rows.
//           The column kinds may weigh rows: by row_fac[r]; by the balance of the row; or (COLS) by 2^-s with
//           s = tc_dist_shift of col_dist[r], because the other operand's columns are scaled up by as much:
//           row_exp[r] = 14 + s, row_inv[r] = 2^-s.
//   COLSUM  partial column sums, gy of them.
//   FILL    fill_n words of `fill` set to fill_word.
// Row lengths are multiples of 4.  The column kinds work in blocks of 32 packets x 8 rows (COLMAX1: 8 x 32).
struct TcJob {
  enum Kind { ROWS, ROWMAX, COLMAX, COLMAX1, COLS, COLS1, COLSUM, FILL } kind;
  const float* src;
  int64_t lds;
  int R, Cc;
  __half *hi, *lo;
  int64_t ldo;
  float* inv;
  float* norm;
  float norm_mul;
  TcBalance bal;
  const float* row_fac;
  uint32_t *max, *bounds;  // of rows or columns
  int again;               // COLS: `max` are those of rows without a balance
  const uint32_t* cap;
  const uint32_t* col_dist;
  float *row_exp, *row_inv;
  float* sums;
  uint32_t* fill;
  uint32_t fill_word;
  int64_t fill_n;
  int gx, gy;  // blocks: columns, rows
  int team;    // ROWS: warps that share a row and keep it in registers, 0: one that reads it twice
};
constexpr int TC_MAX_JOBS = 5;
// Up to this many rows COLS may find balanced maxima again: a projection 2048 x 1536 x 1536 takes 175 us both ways (207 where
// rows have to be balanced) against 183 (190) with a launch for the balanced maxima, 1000 rows 121 (143) against 131.
constexpr int TC_AGAIN_ROWS = 2048;
struct TcJobs {
  TcJob job[TC_MAX_JOBS];
  int n;
};

// A packet of row r with the row's weight
__device__ __forceinline__ float4 tc_load_row4(const TcJob& j, const TcBalanceNow& bal, int r, int c) {
  float4 v = *reinterpret_cast<const float4*>(j.src + (int64_t)r * j.lds + c);
  if (j.row_fac || bal.apply) {  // not both
    const float f = j.row_fac ? j.row_fac[r] : tc_balance(j.bal.max[r], bal, j.bal.up);
    v.x *= f; v.y *= f; v.z *= f; v.w *= f;
  }
  return v;
}

__device__ __forceinline__ void tc_job_rowmax(const TcJob& j, int block, uint2 (&s_bounds)[8]) {
  const int lane = threadIdx.x & 31, c4 = j.Cc >> 2;
  uint32_t top = 0u, below = 0u;
  for (int r = block * 8 + (threadIdx.x >> 5); r < j.R; r += j.gy * 8) {
    const float4* s = reinterpret_cast<const float4*>(j.src + (int64_t)r * j.lds);
    uint4 m4 = make_uint4(0, 0, 0, 0);
#pragma unroll 8
    for (int i = lane; i < c4; i += 32) m4 = tc_max4(m4, tc_absbits4(s[i]));
    const uint32_t m = __reduce_max_sync(0xffffffffu, max(max(m4.x, m4.y), max(m4.z, m4.w)));
    if (lane == 0) j.max[r] = m;
    top = max(top, m);
    if (m) below = max(below, ~m);
  }
  if (!j.bounds) return;
  if (lane == 0) s_bounds[threadIdx.x >> 5] = make_uint2(top, below);
  __syncthreads();
  if (threadIdx.x) return;
#pragma unroll
  for (int w = 1; w < 8; ++w) {
    top = max(top, s_bounds[w].x);
    below = max(below, s_bounds[w].y);
  }
  if (top > __ldcg(j.bounds)) atomicMax(j.bounds, top);  // all blocks meet here: look first
  if (below > __ldcg(j.bounds + 1)) atomicMax(j.bounds + 1, below);
}

// A row's packets stay in the registers of a team of W warps between the search for the maximum and the conversion, up to
// TC_ROW_PACKETS of a lane; longer rows are read again (W 0: a warp per row).  Every team of a block takes as many turns.
// With a warp per row that read it twice, 20 KB rows came from L2 again: 16384 x 5120 174 us, now 106 (6.3 TB/s).
constexpr int TC_ROW_PACKETS = 5;
template <bool BALANCED, int W>
__device__ __forceinline__ void tc_job_rows(const TcJob& j, const TcBalanceNow& bal, int block, uint32_t (&s_red)[2][2][8]) {
  constexpr int TEAM = W ? W : 1, TEAMS = 8 / TEAM, KEEP = W ? TC_ROW_PACKETS : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c4 = j.Cc >> 2;
  const int at = (warp % TEAM) * 32 + lane, step = TEAM * 32;
  const uint4* b = reinterpret_cast<const uint4*>(j.bal.max);
  const int up = j.bal.up;
  auto balanced = [&](float4 v, int i) {
    if (BALANCED) {
      const uint4 m = b[i];
      v.x *= tc_balance(m.x, bal, up); v.y *= tc_balance(m.y, bal, up);
      v.z *= tc_balance(m.z, bal, up); v.w *= tc_balance(m.w, bal, up);
    }
    return v;
  };
  auto largest = [](const uint4& m) { return __reduce_max_sync(0xffffffffu, max(max(m.x, m.y), max(m.z, m.w))); };
  int turn = 0;
  for (int r0 = block * TEAMS; r0 < j.R; r0 += j.gy * TEAMS, turn ^= 1) {
    const int r = r0 + warp / TEAM;
    const bool in = r < j.R;
    const float4* s = reinterpret_cast<const float4*>(j.src + (int64_t)(in ? r : r0) * j.lds);
    uint4 m4 = make_uint4(0, 0, 0, 0), raw4 = m4;
    float4 kept[KEEP];
    if (W) {
#pragma unroll
      for (int i = 0; i < KEEP; ++i) {
        kept[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (at + i * step < c4) kept[i] = s[at + i * step];
      }
#pragma unroll
      for (int i = 0; i < KEEP; ++i) {
        if (BALANCED) {
          raw4 = tc_max4(raw4, tc_absbits4(kept[i]));
          if (at + i * step < c4) kept[i] = balanced(kept[i], at + i * step);
        }
        m4 = tc_max4(m4, tc_absbits4(kept[i]));
      }
    } else {
#pragma unroll 4
      for (int i = at; i < c4; i += step) {
        const float4 v = s[i];
        m4 = tc_max4(m4, tc_absbits4(balanced(v, i)));
        if (BALANCED) raw4 = tc_max4(raw4, tc_absbits4(v));
      }
    }
    uint32_t top = largest(m4), raw = BALANCED && j.max ? largest(raw4) : top;
    if (TEAM > 1) {
      if (lane == 0) {
        s_red[turn][0][warp] = top;
        s_red[turn][1][warp] = raw;
      }
      __syncthreads();
#pragma unroll
      for (int w = 0; w < TEAM; ++w) {
        top = max(top, s_red[turn][0][warp / TEAM * TEAM + w]);
        raw = max(raw, s_red[turn][1][warp / TEAM * TEAM + w]);
      }
    }
    float m, iv;
    tc_scale(top, m, iv);
    float ss = 0.0f;  // of the scaled elements: neither overflows nor vanishes
    auto put = [&](float4 v, int i) {
      v.x *= m; v.y *= m; v.z *= m; v.w *= m;
      tc_put_f16x4(v, j.hi + (int64_t)r * j.ldo + 4 * i, j.lo + (int64_t)r * j.ldo + 4 * i);
      ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    };
    if (W) {
#pragma unroll
      for (int i = 0; i < KEEP; ++i)
        if (in && at + i * step < c4) put(kept[i], at + i * step);
    } else if (in) {
#pragma unroll 4
      for (int i = at; i < c4; i += step) put(balanced(s[i], i), i);
    }
    if (j.norm) {
      ss = ag_warp_sum(ss);
      if (TEAM > 1) {
        __syncthreads();  // the maxima have been read
        if (lane == 0) s_red[turn][0][warp] = __float_as_uint(ss);
        __syncthreads();
        ss = 0.0f;
#pragma unroll
        for (int w = 0; w < TEAM; ++w) ss += __uint_as_float(s_red[turn][0][warp / TEAM * TEAM + w]);
      }
    }
    if (in && at == 0) {
      j.inv[r] = iv;
      if (j.max) j.max[r] = raw;
      if (j.norm) j.norm[r] = sqrtf(ss) * iv * j.norm_mul;
    }
  }
}
template <bool BALANCED>
__device__ __forceinline__ void tc_job_rows(const TcJob& j, const TcBalanceNow& bal, int block, uint32_t (&s_red)[2][2][8]) {
  switch (j.team) {
    case 1: tc_job_rows<BALANCED, 1>(j, bal, block, s_red); break;
    case 2: tc_job_rows<BALANCED, 2>(j, bal, block, s_red); break;
    case 4: tc_job_rows<BALANCED, 4>(j, bal, block, s_red); break;
    case 8: tc_job_rows<BALANCED, 8>(j, bal, block, s_red); break;
    default: tc_job_rows<BALANCED, 0>(j, bal, block, s_red); break;
  }
}

// Largest |elements| of a column packet over the thread's rows
__device__ __forceinline__ uint4 tc_thread_colmax(const TcJob& j, const TcBalanceNow& bal, int c, int first_row, int row_step) {
  uint4 m = make_uint4(0, 0, 0, 0);
  if (c < j.Cc) {
#pragma unroll 8
    for (int r = first_row; r < j.R; r += row_step) m = tc_max4(m, tc_absbits4(tc_load_row4(j, bal, r, c)));
  }
  return m;
}

// A block's atomics are one line per warp, and only where they would change anything: hundreds of row blocks meet at the
// same few words (16384 x 384 by itself: 23.8 us with four words per lane and no look, 12.8 us).
__device__ __forceinline__ void tc_job_colmax(const TcJob& j, const TcBalanceNow& bal, int block, uint4 (&s_max)[8][32]) {
  const int bx = block % j.gx, by = block / j.gx;
  s_max[threadIdx.x >> 5][threadIdx.x & 31] = tc_thread_colmax(
      j, bal, (bx * 32 + (threadIdx.x & 31)) * 4, by * 8 + (threadIdx.x >> 5), j.gy * 8);
  __syncthreads();
  const int c = bx * 128 + threadIdx.x;
  if (threadIdx.x >= 128 || c >= j.Cc) return;
  const uint32_t* words = reinterpret_cast<const uint32_t*>(s_max);
  uint32_t m = words[threadIdx.x];
#pragma unroll
  for (int y = 1; y < 8; ++y) m = max(m, words[y * 128 + threadIdx.x]);
  if (m > __ldcg(j.max + c)) atomicMax(j.max + c, m);
}

// Blocks of PX packets x 256 / PX rows.  FIND: the block looks for the maxima of its columns itself.
template <int PX, bool FIND>
__device__ __forceinline__ void tc_job_cols(const TcJob& j, const TcBalanceNow& bal, int block, int gx, int gy, uint4* s_max) {
  constexpr int PY = 256 / PX;
  const int bx = block % gx, by = block / gx, tx = threadIdx.x % PX, ty = threadIdx.x / PX;
  if (by >= gy) return;
  const int c = (bx * PX + tx) * 4;
  uint4 b = make_uint4(0, 0, 0, 0);
  if (FIND) {
    s_max[threadIdx.x] = tc_thread_colmax(j, bal, c, ty, PY);
    __syncthreads();
#pragma unroll
    for (int y = 0; y < PY; ++y) b = tc_max4(b, s_max[y * PX + tx]);
  } else if (c < j.Cc) {
    b = *reinterpret_cast<const uint4*>(j.max + c);
  }
  if (c >= j.Cc) return;
  if (j.cap) {
    const uint32_t cap = *j.cap;
    b = make_uint4(min(b.x, cap), min(b.y, cap), min(b.z, cap), min(b.w, cap));
  }
  float4 m, iv;
  tc_scale(b.x, m.x, iv.x); tc_scale(b.y, m.y, iv.y); tc_scale(b.z, m.z, iv.z); tc_scale(b.w, m.w, iv.w);
  if (by == 0 && ty == 0) *reinterpret_cast<float4*>(j.inv + c) = iv;
#pragma unroll 4
  for (int r = by * PY + ty; r < j.R; r += gy * PY) {
    float4 v = tc_load_row4(j, bal, r, c);
    if (j.col_dist) {
      const float s = tc_dist_shift(__uint_as_float(j.col_dist[r])), down = tc_pow2(-(int)s);
      v.x *= down; v.y *= down; v.z *= down; v.w *= down;
      if (c == 0) {
        j.row_exp[r] = 14.0f + s;
        j.row_inv[r] = down;
      }
    }
    v.x *= m.x; v.y *= m.y; v.z *= m.z; v.w *= m.w;
    tc_put_f16x4(v, j.hi + (int64_t)r * j.ldo + c, j.lo + (int64_t)r * j.ldo + c);
  }
}

// Five blocks per SM: with four, 668 blocks (a head 333 x 392 x 5003) are two rounds instead of one.
__global__ void __launch_bounds__(256, 5) tc_convert_kernel(const __grid_constant__ TcJobs jobs) {
  ag_pdl_wait();
  __shared__ uint4 s_max[8][32];
  __shared__ uint2 s_bounds[8];
  __shared__ uint32_t s_red[2][2][8];
  int block = blockIdx.x;
  for (int i = 0; i < jobs.n; ++i) {
    const TcJob& j = jobs.job[i];
    const int blocks = j.gx * j.gy;
    if (block < blocks) {
      const TcBalanceNow bal = tc_balance_now(j.bal, j.kind == TcJob::ROWS ? j.Cc : j.R, s_bounds);
      switch (j.kind) {
        case TcJob::ROWS:
          if (bal.apply) tc_job_rows<true>(j, bal, block, s_red);
          else tc_job_rows<false>(j, bal, block, s_red);
          break;
        case TcJob::ROWMAX: tc_job_rowmax(j, block, s_bounds); break;
        case TcJob::COLMAX: tc_job_colmax(j, bal, block, s_max); break;
        case TcJob::COLMAX1: ag_colmax_few<256>(j.src, j.lds, j.R, j.Cc, block, j.max, &s_max[0][0]); break;
        case TcJob::COLSUM:
          ag_colsum_partial(j.src, j.R, j.Cc, block % j.gx * 256 + threadIdx.x, block / j.gx, j.gy, j.sums);
          break;
        case TcJob::FILL:
          for (int64_t k = (int64_t)block * 256 + threadIdx.x; k < j.fill_n; k += (int64_t)blocks * 256) j.fill[k] = j.fill_word;
          break;
        case TcJob::COLS1: tc_job_cols<32, true>(j, bal, block, j.gx, 1, &s_max[0][0]); break;
        default:
          if (j.again && bal.apply) {  // narrow blocks, which read all rows in a few rounds; two per SM at most
            const int gx = (j.Cc + 31) / 32, gy = max(1, min(blocks, 296) / gx);
            for (int at = block; at < gx * gy; at += blocks) {
              tc_job_cols<8, true>(j, bal, at, gx, gy, &s_max[0][0]);
              __syncthreads();
            }
          } else {
            tc_job_cols<32, false>(j, bal, block, j.gx, j.gy, &s_max[0][0]);
          }
          break;
      }
      return;
    }
    block -= blocks;
  }
}

int tc_check_rows(ag_ctx* ctx, const void* src, int64_t lds, int64_t R, int Cc) {
  AG_REQUIRE(ctx, Cc % 4 == 0 && lds % 4 == 0 && R < (1ll << 31) && ag_aligned16(src),
             "tc_convert: rows must be whole 16-byte packets");
  return AG_OK;
}

int tc_split_bf16(ag_ctx* ctx, bool pair, const float* src, int64_t lds, void* hi, void* lo, int64_t ldo, int64_t R, int Cc) {
  if (int rc = tc_check_rows(ctx, src, lds, R, Cc)) return rc;
  int64_t want = (R * (Cc / 4) + 255) / 256;
  if (want > (int64_t)ctx->sm_count * 16) want = (int64_t)ctx->sm_count * 16;
  if (want < 1) want = 1;
  if (pair)
    AG_LAUNCH_PDL(ctx, "split_bf16_kernel", split_bf16_kernel<true>, (int)want, 256, 0, src, lds, (uint16_t*)hi, (uint16_t*)lo,
                  ldo, (int)R, Cc);
  else
    AG_LAUNCH_PDL(ctx, "split_bf16_kernel", split_bf16_kernel<false>, (int)want, 256, 0, src, lds, (uint16_t*)hi, (uint16_t*)lo,
                  ldo, (int)R, Cc);
  return AG_OK;
}

// Collects conversions and launches them together.
struct TcConvert {
  ag_ctx* ctx;
  TcJobs jobs = {};

  TcJob& add(TcJob::Kind kind, const float* src, int64_t lds, int64_t R, int Cc) {
    TcJob& j = jobs.job[jobs.n++];
    j = TcJob{};
    j.kind = kind;
    j.src = src; j.lds = lds; j.R = (int)R; j.Cc = Cc;
    const int64_t cap = (int64_t)ctx->sm_count * 8;
    if (kind == TcJob::ROWS || kind == TcJob::ROWMAX) {
      j.gx = 1;
      const int64_t gy = (R + 7) / 8;
      j.gy = (int)(gy < cap ? gy : cap);
    } else if (kind == TcJob::COLMAX1) {
      j.gx = (Cc + 31) / 32;
      j.gy = 1;
    } else {  // 128 columns per block; four rows per thread at least, about eight blocks per SM at most
      j.gx = (Cc + 127) / 128;
      const int64_t gy = (R + 31) / 32, lim = (cap + j.gx - 1) / j.gx;
      j.gy = kind == TcJob::COLS1 ? 1 : (int)(gy < lim ? gy : lim);
    }
    return j;
  }
  TcJob& rows(const float* src, int64_t lds, const TcBalance& bal, void* hi, void* lo, int64_t ldo, float* inv, int64_t R,
              int Cc) {
    TcJob& j = add(TcJob::ROWS, src, lds, R, Cc);
    j.bal = bal;
    j.hi = (__half*)hi; j.lo = (__half*)lo; j.ldo = ldo; j.inv = inv;
    j.norm_mul = 1.0f;
    const int lanes = (Cc / 4 + TC_ROW_PACKETS - 1) / TC_ROW_PACKETS;
    for (j.team = 1; j.team < 8 && j.team * 32 < lanes; j.team *= 2) {}
    if (j.team * 32 < lanes) j.team = 0;
    const int64_t cap = (int64_t)ctx->sm_count * 8, gy = (R * (j.team ? j.team : 1) + 7) / 8;
    j.gy = (int)(gy < cap ? gy : cap);
    return j;
  }
  TcJob& maxima(TcJob::Kind kind, const float* src, int64_t lds, uint32_t* max, int64_t R, int Cc) {
    TcJob& j = add(kind, src, lds, R, Cc);
    j.max = max;
    return j;
  }
  // max null: found here by one block per 128 columns
  TcJob& cols(const float* src, int64_t lds, uint32_t* max, void* hi, void* lo, int64_t ldo, float* inv, int64_t R, int Cc) {
    TcJob& j = add(max ? TcJob::COLS : TcJob::COLS1, src, lds, R, Cc);
    j.max = max;
    j.hi = (__half*)hi; j.lo = (__half*)lo; j.ldo = ldo; j.inv = inv;
    return j;
  }
  void colsum(const AgTcColsum& q) {
    TcJob& j = jobs.job[jobs.n++];
    j = TcJob{};
    j.kind = TcJob::COLSUM;
    j.src = q.g; j.R = (int)q.R; j.Cc = q.Cc; j.sums = q.partial;
    j.gx = (q.Cc + 255) / 256;
    j.gy = q.parts;
  }
  void fill(uint32_t* p, uint32_t word, int64_t n) {
    TcJob& j = jobs.job[jobs.n++];
    j = TcJob{};
    j.kind = TcJob::FILL;
    j.fill = p; j.fill_word = word; j.fill_n = n;
    j.gx = 1;
    j.gy = (int)(n < 1024 ? 1 : (n / 1024 < ctx->sm_count ? n / 1024 : ctx->sm_count));
  }
  int launch() {
    int blocks = 0;
    for (int i = 0; i < jobs.n; ++i) {
      const TcJob& j = jobs.job[i];
      if (j.kind != TcJob::FILL && j.kind != TcJob::COLSUM)
        if (int rc = tc_check_rows(ctx, j.src, j.lds, j.R, j.Cc)) return rc;
      blocks += j.gx * j.gy;
    }
    if (blocks) AG_LAUNCH_PDL(ctx, "tc_convert_kernel", tc_convert_kernel, blocks, 256, 0, jobs);
    jobs.n = 0;
    return AG_OK;
  }
};

// ---------------------------------------------------------------------------- dlogits from kept logits
// A panel of kept logits, rows 0.. of `logits` (row stride ld, a multiple of 32 floats) and columns v0 ..
struct TcKept {
  const float* logits;
  int64_t ld;
  int rows, cols, v0, V;
  const int32_t* targets;
  const float* lse;
  int ignore_mode;
  // distances (see TcHead::col_dist), of columns v0 ..
  uint32_t* col_dist;
  const float* w_top;
  uint32_t* w_cap;
  // dlogits, in operand form
  const float *row_scale, *dloss, *denom, *col_exp;
  uint16_t *hi, *lo;
  int64_t ld_dl;
  int row_threads;  // threads side by side on one row, a power of two; the others of a block take further rows
};

// What a row says about its logits: the target's column relative to `col`, and whether the row takes part
__device__ __forceinline__ int tc_kept_hit(const TcKept& a, int target, int col, bool& live) {
  const bool valid = target >= 0 && target < a.V;
  live = valid || a.ignore_mode != AG_CE_IGNORE_MASKED;
  return valid ? target - a.v0 - col : -1;
}

// Distance of every column's largest logit from the lse of its row.  Logits are read once and nothing else is done: what
// counts is the bytes in flight, KEPT_ROWS packets of a thread, all requested before the first is used.  A thread owns four
// columns, so the minima are registers and a block ends with one atomic per column, and only where it changes something.
constexpr int KEPT_ROWS = 8;
__global__ void __launch_bounds__(256) tc_kept_dist_kernel(const __grid_constant__ TcKept a) {
  ag_pdl_wait();
  const int col = (blockIdx.x * a.row_threads + (threadIdx.x & (a.row_threads - 1))) * 4;
  const int rows = 256 / a.row_threads, step = gridDim.y * rows;
  float cap = 0.0f;
  if (col < a.cols) {
    float d[4] = {3.0e38f, 3.0e38f, 3.0e38f, 3.0e38f};
    const float* at = a.logits + a.v0 + col;
    for (int r0 = blockIdx.y * rows + threadIdx.x / a.row_threads; r0 < a.rows; r0 += step * KEPT_ROWS) {
      float4 l[KEPT_ROWS];
      float e[KEPT_ROWS];
      int t[KEPT_ROWS];
#pragma unroll
      for (int i = 0; i < KEPT_ROWS; ++i) {
        const int r = min(r0 + i * step, a.rows - 1);  // the last row again: the minimum does not mind
        l[i] = __ldcs(reinterpret_cast<const float4*>(at + (int64_t)r * a.ld));
        e[i] = a.lse[r];
        t[i] = a.targets[r];
      }
#pragma unroll
      for (int i = 0; i < KEPT_ROWS; ++i) {
        bool live;
        const int hit = tc_kept_hit(a, t[i], col, live);
        const float base = live ? e[i] : 3.0e38f;
        const float q[4] = {base - l[i].x, base - l[i].y, base - l[i].z, base - l[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) d[j] = fminf(d[j], j == hit ? 0.0f : fmaxf(q[j], 0.0f));  // |p - 1| is 1 at most
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (col + j >= a.cols) break;
      const uint32_t mine = __float_as_uint(d[j]);
      if (mine < __ldcg(a.col_dist + col + j)) atomicMin(a.col_dist + col + j, mine);
      cap = fmaxf(cap, a.w_top[col + j] * tc_pow2(-(int)tc_dist_shift(d[j])));  // the smallest distance gives the largest
    }
  }
  const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(cap));
  if ((threadIdx.x & 31) == 0 && top > __ldcg(a.w_cap)) atomicMax(a.w_cap, top);
}

// dlogits of a panel, as EPI_DLOGITS writes them.  A thread owns eight columns, whose factors stay in registers, and
// requests four rows before it uses the first.
constexpr int KEPT_DL_ROWS = 4;
template <int FORM>
__global__ void __launch_bounds__(256) tc_kept_dlogits_kernel(const __grid_constant__ TcKept a) {
  ag_pdl_wait();
  const int col = (blockIdx.x * a.row_threads + (threadIdx.x & (a.row_threads - 1))) * 8;
  if (col >= a.cols) return;
  const int rows = 256 / a.row_threads, step = gridDim.y * rows;
  float exps[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) exps[j] = FORM == TC_F16X3 && col + j < a.cols ? a.col_exp[col + j] : 0.0f;
  const float dloss = a.dloss[0], mean = a.row_scale ? 0.0f : dloss / a.denom[0];
  const float* at = a.logits + a.v0 + col;
  for (int r0 = blockIdx.y * rows + threadIdx.x / a.row_threads; r0 < a.rows; r0 += step * KEPT_DL_ROWS) {
    float4 l[KEPT_DL_ROWS][2];
    float e[KEPT_DL_ROWS], s[KEPT_DL_ROWS];
    int t[KEPT_DL_ROWS];
#pragma unroll
    for (int i = 0; i < KEPT_DL_ROWS; ++i) {
      const int r = min(r0 + i * step, a.rows - 1);
      const float4* p = reinterpret_cast<const float4*>(at + (int64_t)r * a.ld);
      l[i][0] = __ldcs(p);
      l[i][1] = __ldcs(p + 1);
      e[i] = a.lse[r];
      t[i] = a.targets[r];
      s[i] = a.row_scale ? a.row_scale[r] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < KEPT_DL_ROWS; ++i) {
      const int r = r0 + i * step;
      if (r >= a.rows) break;
      float v[8] = {l[i][0].x, l[i][0].y, l[i][0].z, l[i][0].w, l[i][1].x, l[i][1].y, l[i][1].z, l[i][1].w};
      bool live;
      const int hit = tc_kept_hit(a, t[i], col, live);
      const float sc = a.row_scale ? dloss * s[i] : mean;
      live = live && sc != 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (FORM == TC_F16X3) {  // the row's scale is applied by the products
          v[j] = tc_exp2(fmaf(v[j] - e[i], kLog2e, exps[j]));
          if (j == hit) v[j] -= tc_exp2(exps[j]);
        } else {
          v[j] = tc_exp2((v[j] - e[i]) * kLog2e);
          if (j == hit) v[j] -= 1.0f;
          v[j] *= sc;
        }
        v[j] = live ? v[j] : 0.0f;
      }
      uint4 hi, lo;
      if (FORM == TC_F16X3) {
        split_f16x2(v[0], v[1], hi.x, lo.x); split_f16x2(v[2], v[3], hi.y, lo.y);
        split_f16x2(v[4], v[5], hi.z, lo.z); split_f16x2(v[6], v[7], hi.w, lo.w);
      } else {
        split_bf16x2(v[0], v[1], hi.x, lo.x); split_bf16x2(v[2], v[3], hi.y, lo.y);
        split_bf16x2(v[4], v[5], hi.z, lo.z); split_bf16x2(v[6], v[7], hi.w, lo.w);
      }
      *reinterpret_cast<uint4*>(a.hi + (int64_t)r * a.ld_dl + col) = hi;
      if (FORM != TC_BF16) *reinterpret_cast<uint4*>(a.lo + (int64_t)r * a.ld_dl + col) = lo;
    }
  }
}

// Blocks of these kernels: as many threads side by side as a row has packets, and rows for about `per_sm` blocks per SM
dim3 tc_kept_grid(ag_ctx* ctx, TcKept& a, int packet, int rows_ahead, int per_sm) {
  a.row_threads = 32;
  while (a.row_threads < 256 && a.row_threads * packet < a.cols) a.row_threads *= 2;
  const int gx = (a.cols + a.row_threads * packet - 1) / (a.row_threads * packet), rows = 256 / a.row_threads * rows_ahead;
  int gy = (ctx->sm_count * per_sm + gx - 1) / gx;
  if (gy > (a.rows + rows - 1) / rows) gy = (a.rows + rows - 1) / rows;
  return dim3(gx, gy);
}

// ---------------------------------------------------------------------------- workspace plan
inline size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }
inline int64_t up8(int64_t x) { return (x + 7) & ~(int64_t)7; }
inline int64_t up16(int64_t x) { return (x + 15) & ~(int64_t)15; }  // dl rows: whole 32-byte sectors in 16-bit types too

inline int tc_mode_of(int precision) {
  return precision == AG_CE_BF16 ? TC_BF16 : (precision == AG_CE_BF16X3 ? TC_BF16X3 : TC_F16X3);
}

struct TcPlan {
  int64_t rows_tile, vc;  // rows and columns of a dl panel
  bool f16;
  int64_t ldo;            // row length of the 16-bit operands of X and W
  size_t X_hi, X_lo, W_hi, W_lo;
  // F16X3 only.  XC, WC: X (times the loss scale of its row) and W scaled by column, for dW and dX; the scales and
  // what they are made from; row_fac: 2^-14 times the row's loss scale; max: words of maxima (see TcMaxima)
  size_t XC_hi, XC_lo, WC_hi, WC_lo;
  size_t X_inv, X_slack, W_inv, W_norm, W_top, max, wc_inv, xc_inv, row_fac, col_dist, col_exp, v_inv;
  size_t dl_hi, dl_lo, part, part_bytes, splitk, splitk_bytes, total;
  int64_t ldc;            // row length of a dl panel
};

TcPlan tc_plan(const ag_flce_desc* d) {
  TcPlan p = {};
  const int mode = tc_mode_of(d->precision);
  const bool pair16 = mode != TC_BF16;
  p.f16 = mode == TC_F16X3;
  p.rows_tile = d->N < AG_FLCE_ROWS_TILE ? d->N : AG_FLCE_ROWS_TILE;
  // A panel has the size of vocab_chunk columns of a full row tile: with fewer rows it is wider, so that short
  // batches are not cut into many small launches.
  int64_t vc = d->vocab_chunk;
  const int64_t wide = vc * AG_FLCE_ROWS_TILE / p.rows_tile / 256 * 256;
  if (wide > vc) vc = wide;
  p.vc = vc < d->V ? vc : d->V;
  p.ldc = up16(p.vc);
  p.ldo = p.f16 ? up8(d->C) : d->C;
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t o = off; off += up256(bytes); return o; };
  const size_t x16 = (size_t)d->N * p.ldo * 2, w16 = (size_t)d->V * p.ldo * 2;
  p.X_hi = take(x16);
  p.X_lo = pair16 ? take(x16) : p.X_hi;
  p.W_hi = take(w16);
  p.W_lo = pair16 ? take(w16) : p.W_hi;
  if (p.f16) {
    p.XC_hi = take(x16);
    p.XC_lo = take(x16);
    p.WC_hi = take(w16);
    p.WC_lo = take(w16);
    p.X_inv = take((size_t)d->N * 4);
    p.X_slack = take((size_t)d->N * 4);
    const size_t per_v = (size_t)d->V * 4;
    p.W_inv = take(per_v);
    p.W_norm = take(per_v);
    p.W_top = take(per_v);
    p.max = take((4 + (size_t)d->C * 3) * 4);
    p.wc_inv = take((size_t)d->C * 4);
    p.xc_inv = take((size_t)d->C * 4);
    p.row_fac = take((size_t)d->N * 4);
    p.col_dist = take((size_t)d->V * 4);
    p.col_exp = take(per_v);
    p.v_inv = take((size_t)d->V * 4);
  }
  const size_t dl_elems = (size_t)p.rows_tile * p.ldc;
  const size_t dl0 = off;
  p.dl_hi = take(dl_elems * 2);
  p.dl_lo = pair16 ? take(dl_elems * 2) : p.dl_hi;
  // forward: the partial softmax statistics take the place of the dl panel
  const size_t part_min = (size_t)TC_EPI_SLICES * 8 * d->N * sizeof(float2);  // eight column tiles at least
  if (off - dl0 < part_min) off = dl0 + up256(part_min);
  p.part = dl0;
  p.part_bytes = off - dl0;
  // split-K partial outputs of dX and dW: up to 16 splits of a 4096-column panel of dW
  p.splitk_bytes = up256((size_t)16 * (p.vc < 4096 ? p.vc : 4096) * d->C * sizeof(float));
  p.splitk = take(p.splitk_bytes);
  p.total = off;
  return p;
}

}  // namespace

// ---- entry points for other translation units (ag_flce.cuh) ---------------------------------
int ag_tc_gemm(ag_ctx* ctx, const AgTcGemm* gs, int n) {
  TcGemm g[2];
  for (int i = 0; i < n; ++i) {
    const AgTcGemm& s = gs[i];
    g[i].mode = s.mode;
    g[i].A = TcOperand{s.A.hi, s.A.lo, s.A.ld, s.A.mn_major};
    g[i].B = TcOperand{s.B.hi, s.B.lo, s.B.ld, s.B.mn_major};
    g[i].M = s.M; g[i].N = s.N; g[i].K = s.K;
    g[i].D = s.D; g[i].ldd = s.ldd; g[i].accumulate = s.accumulate;
    g[i].row_mul = s.row_mul; g[i].col_mul = s.col_mul;
    g[i].bias = s.bias; g[i].resid = s.resid; g[i].ld_resid = s.ld_resid;
    g[i].ws = s.ws; g[i].ws_bytes = s.ws_bytes;
    g[i].chain_elems = s.chain_elems;
  }
  return tc_gemm(ctx, g, n);
}

int ag_tc_split_bf16(ag_ctx* ctx, const float* src, int64_t lds, void* dst, int64_t ldo, int64_t R, int Cc) {
  return tc_split_bf16(ctx, false, src, lds, dst, nullptr, ldo, R, Cc);
}

int ag_tc_convert(ag_ctx* ctx, const AgTcConvert* c, int n, const AgTcMaxima* m, int n_maxima, uint32_t* colmax,
                  size_t colmax_words, const AgTcColsum* sums) {
  TcConvert maxima{ctx}, first{ctx}, second{ctx};
  if (sums) maxima.colsum(*sums);
  for (int i = 0; i < n_maxima; ++i) {
    const AgTcMaxima& q = m[i];
    const TcJob::Kind kind = !q.by_column ? TcJob::ROWMAX : q.R <= TC_FEW_ROWS ? TcJob::COLMAX1 : TcJob::COLMAX;
    maxima.maxima(kind, q.src, q.lds, q.max, q.R, q.Cc).bounds = q.bounds;
  }
  size_t used = 0;
  for (int i = 0; i < n; ++i) {
    const AgTcConvert& q = c[i];
    const TcBalance bal = {q.bal_max, q.bal_bounds, q.bal_up ? 1 : 0};
    if (!q.by_column) {
      first.rows(q.src, q.lds, bal, q.hi, q.lo, q.ldo, q.inv, q.R, q.Cc);
    } else if (q.R <= TC_COLS1_ROWS) {
      first.cols(q.src, q.lds, nullptr, q.hi, q.lo, q.ldo, q.inv, q.R, q.Cc).bal = bal;
    } else {
      uint32_t* cm = colmax + used;
      used += (size_t)((q.Cc + 3) / 4 * 4);
      AG_REQUIRE(ctx, used <= colmax_words, "tc_convert: too few words for column maxima");
      // Up to TC_AGAIN_ROWS the maxima are those of the rows as they are, found beside the ones that the balance goes by;
      // where the rows have to be balanced, every block finds its columns' again.
      const bool again = q.R <= TC_AGAIN_ROWS;
      TcJob& j = (again ? maxima : first).maxima(TcJob::COLMAX, q.src, q.lds, cm, q.R, q.Cc);
      if (!again) j.bal = bal;
      TcJob& k = (again ? first : second).cols(q.src, q.lds, cm, q.hi, q.lo, q.ldo, q.inv, q.R, q.Cc);
      k.bal = bal;
      k.again = again ? 1 : 0;
    }
  }
  if (int rc = maxima.launch()) return rc;
  if (int rc = first.launch()) return rc;
  return second.launch();
}

// =========================================================================================
bool ag_flce_tc_supported(const ag_flce_desc* d) {
  if (d->precision != AG_CE_3XTF32 && d->precision != AG_CE_BF16 && d->precision != AG_CE_BF16X3) return false;
  // TMA needs 16-byte aligned row starts: rows of X / W are C elements long
  const int q = d->precision == AG_CE_3XTF32 ? 4 : 8;
  if (d->C % q != 0) return false;
  if (d->vocab_chunk % 8 != 0 && d->vocab_chunk < d->V) return false;
  if (d->C < 32 || d->V < 32 || d->N < 1) return false;
  return true;
}

size_t ag_flce_tc_scratch_bytes(const ag_flce_desc* d) { return tc_plan(d).total; }

int64_t ag_flce_logits_ld(const ag_flce_desc* d) { return ((int64_t)d->V + 31) / 32 * 32; }

namespace {
// The logits product of rows r0.. and vocabulary v0.. (operands already converted)
TcGemm tc_logits(const ag_flce_desc* d, const TcPlan& p, unsigned char* b, int64_t r0, int rows, int64_t v0, int cols) {
  TcGemm g;
  g.mode = tc_mode_of(d->precision);
  g.A = TcOperand{b + p.X_hi + (size_t)(r0 * p.ldo) * 2, b + p.X_lo + (size_t)(r0 * p.ldo) * 2, p.ldo, 0};
  g.B = TcOperand{b + p.W_hi + (size_t)(v0 * p.ldo) * 2, b + p.W_lo + (size_t)(v0 * p.ldo) * 2, p.ldo, 0};
  g.M = rows; g.N = cols; g.K = d->C;
  if (p.f16) {
    g.row_mul = reinterpret_cast<const float*>(b + p.X_inv) + r0;
    g.col_mul = reinterpret_cast<const float*>(b + p.W_inv) + v0;
  }
  return g;
}

// Words of maxima: of W as dX takes it (see TcHead::w_cap); of the columns of W; of the columns of X times the row's loss
// scale; of the columns of X, which the channels are balanced by.
struct TcMaxima {
  uint32_t *w_cap, *w, *xc, *x;  // they lie in this order, w_cap with three words of padding
};
TcMaxima tc_maxima(const ag_flce_desc* d, const TcPlan& p, unsigned char* b) {
  uint32_t* m = reinterpret_cast<uint32_t*>(b + p.max);
  return {m, m + 4, m + 4 + d->C, m + 4 + 2 * (int64_t)d->C};
}
}  // namespace

int ag_flce_tc_forward(ag_ctx* ctx, const ag_flce_desc* d, const float* X, const float* W, void* tc_scratch,
                       const int32_t* targets, const float* row_scale, float* run_max, float* run_sum, float* tgt_logit,
                       uint32_t* ticket, float* lse, float* loss, float* logits) {
  const TcPlan p = tc_plan(d);
  unsigned char* b = static_cast<unsigned char*>(tc_scratch);
  const int mode = tc_mode_of(d->precision);
  int rc;
  if (p.f16) {
    const TcMaxima m = tc_maxima(d, p, b);
    const bool few = d->N <= TC_FEW_ROWS;
    if (!few) {
      AG_CUDA(ctx, cudaMemsetAsync(m.x, 0, (size_t)d->C * 4, ctx->stream));
      ag_enqueued(ctx);
    }
    TcConvert cv{ctx};
    cv.maxima(few ? TcJob::COLMAX1 : TcJob::COLMAX, X, d->C, m.x, d->N, d->C);
    if ((rc = cv.launch())) return rc;
    cv.rows(X, d->C, TcBalance{m.x, nullptr, 1}, b + p.X_hi, b + p.X_lo, p.ldo, (float*)(b + p.X_inv), d->N, d->C);
    cv.rows(W, d->C, TcBalance{m.x, nullptr, 0}, b + p.W_hi, b + p.W_lo, p.ldo, (float*)(b + p.W_inv), d->V, d->C);
    if ((rc = cv.launch())) return rc;
  } else if ((rc = tc_split_bf16(ctx, mode == TC_BF16X3, X, d->C, b + p.X_hi, b + p.X_lo, p.ldo, d->N, d->C)) ||
             (rc = tc_split_bf16(ctx, mode == TC_BF16X3, W, d->C, b + p.W_hi, b + p.W_lo, p.ldo, d->V, d->C))) {
    return rc;
  }
  // The logits stay in registers, so a launch takes as many columns as the partial statistics have room for
  // (16 bytes per row and column tile): for any usual vocabulary one launch, whose last round over the SMs is
  // one of hundreds.
  const int64_t part_ld = d->N;
  const int64_t tiles_fit = (int64_t)(p.part_bytes / ((size_t)TC_EPI_SLICES * part_ld * sizeof(float2)));
  const int min_bn = (d->V + 31) / 32 <= tiles_fit ? 32 : 256;
  const int64_t step = min_bn == 32 ? (int64_t)d->V : tiles_fit * 256;
  for (int64_t v0 = 0; v0 < d->V; v0 += step) {
    const int cols = (int)(d->V - v0 < step ? d->V - v0 : step);
    TcHead h = {};
    h.targets = targets;
    h.v0 = (int)v0;
    h.V = d->V;
    h.part = reinterpret_cast<float2*>(b + p.part);
    h.part_ld = part_ld;
    h.tgt_logit = tgt_logit;
    h.ticket = ticket;
    h.logits = logits;
    h.ld_logits = ag_flce_logits_ld(d);
    const TcGemm g = tc_logits(d, p, b, 0, (int)d->N, v0, cols);
    int tiles_n = 0;
    if ((rc = tc_gemm(ctx, &g, 1, logits ? EPI_STATS_KEEP : EPI_STATS, &h, min_bn, &tiles_n))) return rc;
    if ((rc = ag_flce_finish(ctx, d, h.part, tiles_n * TC_EPI_SLICES, targets, row_scale, run_max, run_sum, tgt_logit, ticket, lse,
                             loss, v0 == 0, v0 + step >= d->V)))
      return rc;
  }
  return AG_OK;
}

AgFlceTcInit ag_flce_tc_init(const ag_flce_desc* d, void* tc_scratch, bool kept) {
  const TcPlan p = tc_plan(d);
  if (!p.f16) return {};
  unsigned char* b = static_cast<unsigned char*>(tc_scratch);
  const TcMaxima m = tc_maxima(d, p, b);
  const bool few = d->N <= TC_FEW_ROWS;
  return {reinterpret_cast<float*>(b + p.row_fac), m.w_cap, 4 + (few || kept ? 2 : 3) * d->C, few && !kept ? m.x : nullptr};
}

int ag_flce_tc_backward(ag_ctx* ctx, const ag_flce_desc* d, const float* X, const float* W, void* tc_scratch,
                        const int32_t* targets, const float* lse, const float* row_scale, const float* dloss,
                        const float* denom, float* dX, float* dW, const float* logits) {
  const TcPlan p = tc_plan(d);
  unsigned char* b = static_cast<unsigned char*>(tc_scratch);
  const int mode = tc_mode_of(d->precision);
  const int C = d->C;
  int rc;
  const int64_t ld_logits = ag_flce_logits_ld(d);
  auto kept = [&](int64_t r0, int64_t rows, int64_t v0, int cols) {
    TcKept k = {};
    k.logits = logits + r0 * ld_logits;
    k.ld = ld_logits;
    k.rows = (int)rows;
    k.cols = cols;
    k.v0 = (int)v0;
    k.V = d->V;
    k.targets = targets + r0;
    k.lse = lse + r0;
    k.ignore_mode = d->ignore_mode;
    return k;
  };
  if (p.f16) {
    uint32_t* dist = (uint32_t*)(b + p.col_dist);
    const float* row_fac = (const float*)(b + p.row_fac);
    const TcMaxima m = tc_maxima(d, p, b);
    TcConvert cv{ctx};
    if (logits) {
      cv.maxima(TcJob::ROWMAX, W, C, (uint32_t*)(b + p.W_top), d->V, C);
    } else if (d->N > TC_FEW_ROWS) {  // of few rows the kernel before has found them
      cv.maxima(TcJob::COLMAX, X, C, m.x, d->N, C);
      if ((rc = cv.launch())) return rc;
    }
    if (!logits) {
      TcJob& x = cv.rows(X, C, TcBalance{m.x, nullptr, 1}, b + p.X_hi, b + p.X_lo, p.ldo, (float*)(b + p.X_inv), d->N, C);
      x.norm = (float*)(b + p.X_slack);
      x.norm_mul = 1.0f / 1024.0f;
      TcJob& w = cv.rows(W, C, TcBalance{m.x, nullptr, 0}, b + p.W_hi, b + p.W_lo, p.ldo, (float*)(b + p.W_inv), d->V, C);
      w.norm = (float*)(b + p.W_norm);
      w.max = (uint32_t*)(b + p.W_top);
    }
    cv.maxima(TcJob::COLMAX, W, C, m.w, d->V, C);
    if (dW) cv.maxima(TcJob::COLMAX, X, C, m.xc, d->N, C).row_fac = row_fac;
    cv.fill(dist, 0x7f7f7f7fu, d->V);  // 3.4e38 each
    if ((rc = cv.launch())) return rc;
    // How small every column of dl is, so that its fp16 pair keeps all its bits there too (dW of a token that no row
    // predicts).  Kept logits say it; otherwise one product of the hi parts bounds it, a third of the work of a full product.
    if (logits) {
      TcKept k = kept(0, d->N, 0, d->V);
      k.col_dist = dist;
      k.w_top = (const float*)(b + p.W_top);
      k.w_cap = m.w_cap;
      const dim3 grid = tc_kept_grid(ctx, k, 4, KEPT_ROWS, 8);
      AG_LAUNCH_PDL(ctx, "tc_kept_dist_kernel", tc_kept_dist_kernel, grid, 256, 0, k);
    } else {
      TcHead h = {};
      h.targets = targets;
      h.V = d->V;
      h.lse = lse;
      h.ignore_mode = d->ignore_mode;
      h.col_dist = dist;
      h.row_slack = (const float*)(b + p.X_slack);
      h.w_norm = (const float*)(b + p.W_norm);
      h.w_top = (const float*)(b + p.W_top);
      h.w_cap = m.w_cap;
      TcGemm g = tc_logits(d, p, b, 0, (int)d->N, 0, d->V);
      g.mode = TC_F16HI;
      if ((rc = tc_gemm(ctx, &g, 1, EPI_COLMAX, &h))) return rc;
    }
    // W by column for dX, its rows scaled down as the columns of dl are scaled up
    TcJob& wc = cv.cols(W, C, m.w, b + p.WC_hi, b + p.WC_lo, p.ldo, (float*)(b + p.wc_inv), d->V, C);
    wc.cap = m.w_cap;
    wc.col_dist = dist;
    wc.row_exp = (float*)(b + p.col_exp);
    wc.row_inv = (float*)(b + p.v_inv);
    if (dW) cv.cols(X, C, m.xc, b + p.XC_hi, b + p.XC_lo, p.ldo, (float*)(b + p.xc_inv), d->N, C).row_fac = row_fac;
    if ((rc = cv.launch())) return rc;
  } else {  // the recomputed logits need both, dW of kept ones X, dX W
    const bool pair = mode == TC_BF16X3;
    if ((!logits || dW) && (rc = tc_split_bf16(ctx, pair, X, C, b + p.X_hi, b + p.X_lo, p.ldo, d->N, C))) return rc;
    if ((!logits || dX) && (rc = tc_split_bf16(ctx, pair, W, C, b + p.W_hi, b + p.W_lo, p.ldo, d->V, C))) return rc;
  }
  for (int64_t r0 = 0; r0 < d->N; r0 += p.rows_tile) {
    const int rows = (int)(d->N - r0 < p.rows_tile ? d->N - r0 : p.rows_tile);
    for (int64_t v0 = 0; v0 < d->V; v0 += p.vc) {
      const int vc = (int)(d->V - v0 < p.vc ? d->V - v0 : p.vc);
      if (logits) {
        TcKept k = kept(r0, rows, v0, vc);
        k.row_scale = row_scale ? row_scale + r0 : nullptr;
        k.dloss = dloss;
        k.denom = denom;
        if (p.f16) k.col_exp = (const float*)(b + p.col_exp) + v0;
        k.hi = (uint16_t*)(b + p.dl_hi);
        k.lo = (uint16_t*)(b + p.dl_lo);
        k.ld_dl = p.ldc;
        const dim3 grid = tc_kept_grid(ctx, k, 8, KEPT_DL_ROWS, 3);
        if (mode == TC_F16X3)
          AG_LAUNCH_PDL(ctx, "tc_kept_dlogits_kernel", tc_kept_dlogits_kernel<TC_F16X3>, grid, 256, 0, k);
        else if (mode == TC_BF16X3)
          AG_LAUNCH_PDL(ctx, "tc_kept_dlogits_kernel", tc_kept_dlogits_kernel<TC_BF16X3>, grid, 256, 0, k);
        else
          AG_LAUNCH_PDL(ctx, "tc_kept_dlogits_kernel", tc_kept_dlogits_kernel<TC_BF16>, grid, 256, 0, k);
      } else {
        // logits panel recomputed on the tensor cores; its epilogue writes dlogits in operand form
        TcHead h = {};
        h.targets = targets + r0;
        h.v0 = (int)v0;
        h.V = d->V;
        h.lse = lse + r0;
        h.row_scale = row_scale ? row_scale + r0 : nullptr;
        h.dloss = dloss;
        h.denom = denom;
        h.ignore_mode = d->ignore_mode;
        h.dl_form = mode;
        h.dl_hi = b + p.dl_hi;
        h.dl_lo = b + p.dl_lo;
        if (p.f16) h.col_exp = (const float*)(b + p.col_exp) + v0;
        h.ld_dl = p.ldc;
        const TcGemm g = tc_logits(d, p, b, r0, rows, v0, vc);
        if ((rc = tc_gemm(ctx, &g, 1, EPI_DLOGITS, &h))) return rc;
      }
      // The two products of the panel are independent: one launch deals the tiles of both.
      TcGemm g[2];
      int n = 0;
      if (dW) {
        // dW[v0:v0+vc, :] += dl^T . X[r0:r0+rows, :]; the contraction index (row) is the row index of
        // both dl and X as stored: both operands MN-major
        TcGemm& q = g[n++];
        q.mode = mode;
        q.A = TcOperand{b + p.dl_hi, b + p.dl_lo, p.ldc, 1};
        const size_t x_hi = p.f16 ? p.XC_hi : p.X_hi, x_lo = p.f16 ? p.XC_lo : p.X_lo, at = (size_t)(r0 * p.ldo) * 2;
        q.B = TcOperand{b + x_hi + at, b + x_lo + at, p.ldo, 1};
        if (p.f16) {
          q.row_mul = (const float*)(b + p.v_inv) + v0;
          q.col_mul = (const float*)(b + p.xc_inv);
        }
        q.M = vc; q.N = C; q.K = rows;
        q.D = dW + v0 * C;
        q.ldd = C;
        q.accumulate = true;
        q.ws = reinterpret_cast<float*>(b + p.splitk);
        q.ws_bytes = dX ? p.splitk_bytes / 2 / 256 * 256 : p.splitk_bytes;
      }
      if (dX) {
        // dX[r0:r0+rows, :] += dl [rows, vc] . W[v0:v0+vc, :]; W as stored has the contraction index
        // (vocabulary) as its row index, i.e. it is the MN-major form of the B operand
        TcGemm& q = g[n++];
        q.mode = mode;
        q.A = TcOperand{b + p.dl_hi, b + p.dl_lo, p.ldc, 0};
        const size_t w_hi = p.f16 ? p.WC_hi : p.W_hi, w_lo = p.f16 ? p.WC_lo : p.W_lo, at = (size_t)(v0 * p.ldo) * 2;
        q.B = TcOperand{b + w_hi + at, b + w_lo + at, p.ldo, 1};
        q.M = rows; q.N = C; q.K = vc;
        q.D = dX + r0 * C;
        q.ldd = C;
        q.accumulate = true;
        if (p.f16) {
          q.row_mul = reinterpret_cast<const float*>(b + p.row_fac) + r0;
          q.col_mul = reinterpret_cast<const float*>(b + p.wc_inv);
        }
        const size_t used = dW ? p.splitk_bytes / 2 / 256 * 256 : 0;
        q.ws = reinterpret_cast<float*>(b + p.splitk + used);
        q.ws_bytes = p.splitk_bytes - used;
      }
      if ((rc = tc_gemm(ctx, g, n))) return rc;
    }
  }
  return AG_OK;
}
