// Internal interface between the fused linear+CE driver (ag_flce.cu) and the tcgen05
// tensor-core panels (ag_flce_tc.cu).
#pragma once

#include "ag_common.cuh"

// True when the tensor-core path takes this problem (precision mode, shape, alignment).
bool ag_flce_tc_supported(const ag_flce_desc* d);
// Extra workspace (split / converted operands, dlogits panel, split-K partials) the tensor-core path needs.
size_t ag_flce_tc_scratch_bytes(const ag_flce_desc* d);
// Forward without materialising the logits: they stay in registers, the GEMM epilogue reduces them to per-tile
// (max, sum exp) and picks the target logit; the partials are folded (ag_flce_finish).  Converts X and W
// into operand form inside tc_scratch first.  `logits` (may be null): [N][ag_flce_logits_ld], written beside the statistics.
int64_t ag_flce_logits_ld(const ag_flce_desc* d);
int ag_flce_tc_forward(ag_ctx* ctx, const ag_flce_desc* d, const float* X, const float* W, void* tc_scratch,
                       const int32_t* targets, const float* row_scale, float* run_max, float* run_sum, float* tgt_logit,
                       uint32_t* ticket, float* lse, float* loss, float* logits);
// Folds n_parts partial statistics per row into run_max / run_sum, after the last launch of them into lse and the loss.
// ticket: a word that the launch before has cleared.
int ag_flce_finish(ag_ctx* ctx, const ag_flce_desc* d, const float2* part, int n_parts, const int32_t* targets,
                   const float* row_scale, float* run_max, float* run_sum, const float* tgt_logit, uint32_t* ticket, float* lse,
                   float* loss, bool first, bool last);
// Backward, panel by panel: the logits are recomputed, the GEMM epilogue turns them into dlogits in operand
// form, then dX[r0:r0+rows] += dl . W[v0:v0+vc] and dW[v0:v0+vc] += dl^T . X[r0:r0+rows] (either output may be
// null).  With `logits` of the forward nothing is recomputed: a pass over the panel turns them into dlogits.
int ag_flce_tc_backward(ag_ctx* ctx, const ag_flce_desc* d, const float* X, const float* W, void* tc_scratch,
                        const int32_t* targets, const float* lse, const float* row_scale, const float* dloss,
                        const float* denom, float* dX, float* dW, const float* logits);
// What the backward expects from the kernel before it: 2^-14 * (loss scale of the row) in row_fac for every row,
// `zero_words` words of `zero` cleared, and the largest |elements| of the columns of X in x_max (few rows only, and not
// where the logits are kept).  Null
// pointers when the precision or the shape needs none of it.
struct AgFlceTcInit {
  float* row_fac;
  uint32_t* zero;
  int zero_words;
  uint32_t* x_max;
};
AgFlceTcInit ag_flce_tc_init(const ag_flce_desc* d, void* tc_scratch, bool kept);

// Heads of few multiply-adds take another path (ag_tc_small.cu): operands are split inside the products.
bool ag_flce_small(const ag_flce_desc* d);
// Up to this many rows a CTA of them counts those that take part by itself, beside its products; else denom holds their number.
// Backward, us, counted in a launch of its own / by every CTA: 4096 x 64 x 500 27.9 / 25.3, 16384 x 64 x 300 51.9 / 49.8, 30000 x
// 64 x 300 76.1 / 74.9 (bf16 56.5 / 56.2), 50000 x 64 x 300 114 / 128, 73000 x 32 x 64 88 / 94.
constexpr int64_t AG_FLCE_COUNT_ROWS = 32768;
size_t ag_flce_small_scratch_bytes(const ag_flce_desc* d);
int ag_flce_small_forward(ag_ctx* ctx, const ag_flce_desc* d, const float* X, const float* W, void* scratch,
                          const int32_t* targets, const float* row_scale, float* run_max, float* run_sum, float* tgt_logit,
                          uint32_t* ticket, float* lse, float* loss, float* logits);
int ag_flce_small_backward(ag_ctx* ctx, const ag_flce_desc* d, const float* X, const float* W, void* scratch,
                           const int32_t* targets, const float* lse, const float* row_scale, const float* dloss,
                           const float* denom, float* dX, float* dW, const float* logits);

// Token rows handled per pass over the vocabulary panels (the rows of the logits / dlogits panel held in
// scratch).  148 SMs x 128-row tiles = 74 CTA pairs x 256-row tiles: every GEMM of a full row tile then
// has a whole number of rounds over the SMs in the row direction.
constexpr int64_t AG_FLCE_ROWS_TILE = 148 * 128;

// Operand modes of the tensor-core GEMM (see ag_flce_tc.cu): bf16 values, bf16 (hi, lo) pairs,
// fp16 (hi, lo) pairs with a power-of-two scale per row or column (fp32-grade at the 16-bit MMA rate).
enum AgTcMode { AG_TC_BF16, AG_TC_BF16X3, AG_TC_F16X3 };

// ---- the tensor-core GEMM as a building block (used by the linear + bias + residual op) --------
struct AgTcOperand {
  const void* hi;
  const void* lo;   // null / unused in bf16 mode
  int64_t ld;       // elements between consecutive rows of the array as stored
  int mn_major;     // 0: stored [MN][K] (K contiguous); 1: stored [K][MN] (MN contiguous)
};
// D[M,N] (+)= (A . B^T) * row_mul[m] * col_mul[n] + bias[n] + resid[m,n] with A logically [M][K] and B logically
// [N][K], each stored K-major or MN-major; split-K with an ordered reduction where a workspace is given and the
// problem has few tiles.
struct AgTcGemm {
  int mode = AG_TC_F16X3;
  AgTcOperand A = {}, B = {};
  int M = 0, N = 0, K = 0;
  float* D = nullptr;
  int64_t ldd = 0;
  bool accumulate = false;
  const float *row_mul = nullptr, *col_mul = nullptr, *bias = nullptr, *resid = nullptr;
  int64_t ld_resid = 0;
  float* ws = nullptr;
  size_t ws_bytes = 0;
  int chain_elems = 0;  // longest tensor-core accumulation chain (0: the default of the mode)
};
// One or two independent products in one launch.
int ag_tc_gemm(ag_ctx* ctx, const AgTcGemm* g, int n);
// Operand conversions, src[R][Cc] (row stride lds) -> rows of ldo elements: bf16 values, or fp16 pairs scaled per row
// (inv[R] takes the scale out of the product) or per column (inv[Cc]).
int ag_tc_split_bf16(ag_ctx* ctx, const float* src, int64_t lds, void* dst, int64_t ldo, int64_t R, int Cc);
// The contraction index of a product may be balanced (see TcBalance in ag_flce_tc.cu): bal_max are the maxima of one operand
// at every index (see AgTcMaxima); that operand is converted with bal_up, the other without.
struct AgTcConvert {
  const float* src;
  int64_t lds;
  int64_t R;
  int Cc;
  bool by_column;
  void *hi, *lo;
  int64_t ldo;
  float* inv;
  const uint32_t *bal_max, *bal_bounds;
  bool bal_up;
};
// Bits of the largest |element| of every column or row, and (rows only, may be null) the bounds of them.  `bounds`, and
// `max` by column from more than TC_FEW_ROWS rows on, start at zero.
struct AgTcMaxima {
  const float* src;
  int64_t lds;
  int64_t R;
  int Cc;
  bool by_column;
  uint32_t *max, *bounds;
};
// Column sums of g[R][Cc] in `parts` partial rows (see ag_colsum_partial)
struct AgTcColsum {
  const float* g;
  int64_t R;
  int Cc, parts;
  float* partial;
};
// Up to four conversions, after up to two searches of maxima that they are balanced by, in as few launches as they allow;
// colmax: cleared workspace of a word per column of those scaled by column, needed from more than TC_COLS1_ROWS rows on.
// sums (may be null) share the launch of the maxima.
int ag_tc_convert(ag_ctx* ctx, const AgTcConvert* c, int n, const AgTcMaxima* m, int n_maxima, uint32_t* colmax,
                  size_t colmax_words, const AgTcColsum* sums);

// ---- products of a few tiles straight from fp32 operands (ag_tc_small.cu) -------------------------
struct AgTcsOperand {
  const float* p;
  int64_t ld;
  int mn_major;
};
// D[M,N] (+)= A . B^T + bias[n], or = A . B^T + bias[n] + resid[m,n].  Pointers and row lengths of the operands are whole 16-byte packets; where the
// contiguous extent is not a multiple of 4, the rest of its last packet is zero.  ws: partial outputs of a split contraction.
struct AgTcsGemm {
  AgTcsOperand A = {}, B = {};
  int M = 0, N = 0, K = 0;
  float* D = nullptr;
  int64_t ldd = 0;
  bool accumulate = false;
  const float *bias = nullptr, *resid = nullptr;
  int64_t ld_resid = 0;
  float* ws = nullptr;
  size_t ws_bytes = 0;
};
// The head's fields; dloss, where it is set, also scales the products of dl back (see tcs_dl_shift).
struct AgTcsHead {
  const int32_t* targets;
  int V, rows;
  const float *lse, *row_scale, *dloss, *denom;
  int reduction, ignore_mode;
  float2* part;        // STATS: (max, sum exp) per half column tile and row
  int64_t part_ld;
  float* tgt_logit;    // STATS: logit of the target column
  uint32_t* ticket;    // STATS: cleared for the kernel that follows
  float* logits;       // STATS: written too, where not null; [rows][ld_logits], a multiple of 32
  int64_t ld_logits;
};
// STORE: one or two products, split where that helps.  STATS: logits reduced to partial statistics.  DLOGITS: logits turned
// into dl = 2^shift * scale * (p - onehot), whose row length ldd is padded with zeros.
enum { AG_TCS_STORE, AG_TCS_STATS, AG_TCS_DLOGITS };
// parts: bf16 parts per operand (3 fp32-grade, 2, 1); max_k: longest contraction of a CTA, a multiple of 64.
constexpr int AG_TCS_MAX_K = 2304;    // a a' of a chain is 144 additions then, as many as 768 elements of operand pairs make
constexpr int AG_TCS_MAX_SPLITS = 32;
size_t ag_tcs_split_bytes(int64_t M, int64_t N, int64_t K, int max_k);  // workspace of the splits that a product may take
int ag_tcs_gemm(ag_ctx* ctx, int epi, int parts, const AgTcsGemm* g, int n, int max_k, const AgTcsHead* head, int* tiles_n_out);

// Up to this many rows, one block finds the maxima of 32 columns by itself: saves clearing words for atomics, and a launch
// of the head's backward (forward of a head 333 x 392 x 5000 27.3 against 31.2 us, backward 64.4 against 67.4; 512 x 768 x
// 32768 122.6 / 122.5 and 380 / 372: even there, and 1024 rows cost 4 % more).
constexpr int TC_FEW_ROWS = 512;
// Up to this many rows, one block finds the maxima of 128 columns and converts them too (dW of a projection 768 x 768: 64
// rows 14.6 us against 17.7 with maxima and conversion in launches of their own, 128 rows 17.7 / 18.5, 256 rows 26.4 /
// 20.0, 512 rows 45 / 23; 392 x 5000 and 1536 x 1536 cross at 128 rows too).
constexpr int TC_COLS1_ROWS = 128;

#ifdef __CUDACC__
// partial[part][c] = sum of g over the rows of chunk `part` of `parts` (rows in ascending order), by one thread
__device__ __forceinline__ void ag_colsum_partial(const float* __restrict__ g, int64_t N, int C, int c, int part, int parts,
                                                  float* __restrict__ partial) {
  if (c >= C) return;
  const int64_t per = (N + parts - 1) / parts;
  const int64_t r0 = (int64_t)part * per;
  const int64_t r1 = r0 + per < N ? r0 + per : N;
  float acc = 0.0f;
  int64_t r = r0;
  for (; r + 8 <= r1; r += 8) {  // eight rows in flight, added in row order
    float a[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) a[u] = __ldcs(g + (r + u) * C + c);
#pragma unroll
    for (int u = 0; u < 8; ++u) acc += a[u];
  }
  for (; r < r1; ++r) acc += g[r * C + c];
  partial[(int64_t)part * C + c] = acc;
}

// |x| as ordered bits; Inf and NaN count as zero (they stay Inf and NaN in the pair whatever the scale)
__device__ __forceinline__ uint32_t tc_absbits(float x) {
  const uint32_t b = __float_as_uint(x) & 0x7fffffffu;
  return b < 0x7f800000u ? b : 0u;
}
__device__ __forceinline__ uint4 tc_absbits4(const float4& v) {
  return make_uint4(tc_absbits(v.x), tc_absbits(v.y), tc_absbits(v.z), tc_absbits(v.w));
}
__device__ __forceinline__ uint4 tc_max4(const uint4& a, const uint4& b) {
  return make_uint4(max(a.x, b.x), max(a.y, b.y), max(a.z, b.z), max(a.w, b.w));
}

// Largest |elements| of columns [32 block, 32 block + 32) over all rows, by one block of THREADS = 8 packets x THREADS / 8
// rows: no atomics, nothing to clear.  Row lengths are multiples of 4; s_max: 8 packets per warp.
template <int THREADS>
__device__ __forceinline__ void ag_colmax_few(const float* src, int64_t lds, int R, int Cc, int block, uint32_t* max,
                                              uint4* s_max) {
  const int tx = threadIdx.x & 7, c = (block * 8 + tx) * 4;
  uint4 m = make_uint4(0, 0, 0, 0);
  if (c < Cc) {
#pragma unroll 8
    for (int r = threadIdx.x >> 3; r < R; r += THREADS / 8)
      m = tc_max4(m, tc_absbits4(*reinterpret_cast<const float4*>(src + (int64_t)r * lds + c)));
  }
#pragma unroll
  for (int o = 8; o < 32; o *= 2)
    m = tc_max4(m, make_uint4(__shfl_xor_sync(0xffffffffu, m.x, o), __shfl_xor_sync(0xffffffffu, m.y, o),
                              __shfl_xor_sync(0xffffffffu, m.z, o), __shfl_xor_sync(0xffffffffu, m.w, o)));
  if ((threadIdx.x & 31) < 8) s_max[(threadIdx.x >> 5) * 8 + tx] = m;
  __syncthreads();
  if (threadIdx.x >= 8 || c >= Cc) return;
#pragma unroll
  for (int w = 1; w < THREADS / 32; ++w) m = tc_max4(m, s_max[w * 8 + tx]);
  *reinterpret_cast<uint4*>(max + c) = m;
}
#endif
