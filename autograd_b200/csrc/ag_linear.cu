// Linear projection with fused bias + residual epilogue: out = act . W + b + x.
//
// This is the node that closes every attention / MLP branch of the reference models and feeds the
// next norm (backend.py:2040-2058 forward, :2249-2259 backward).  The GEMMs run on the tcgen05
// kernel of ag_flce_tc.cu with scaled fp16 pairs (fp32-grade; the mode that callers select as AG_CE_3XTF32) or
// bf16; bias and residual are added in its epilogue while the accumulator is in registers, so the projection
// output is written once and `out` may alias `x` (the reference aliases them when x dies here, runtime.py:397-417).
//   forward : out[N,C]  = act[N,K] . W[K,C] + b[C] + x[N,C]     (W read MN-major)
//   backward: dx   += dout
//             dact += dout . W^T                                 (both K-major as stored)
//             dW   += act^T . dout          (both MN-major; split-K with ordered reduction)
//             db   += column sums of dout   (two passes, fixed order, no atomics)
// act, W and dout are only converted to the operand format; the GEMM reads them in whichever orientation each
// product needs, so no transposed copy is made.  An fp16 pair is scaled along the index that is not contracted:
// by row where the operand is read K-major, by column where it is read MN-major; along the contracted index the pair of
// operands is balanced by the maxima of the smaller one (W by row forward and by column for dact, dout by row for dW).  The
// search costs a launch forward, none backward (the bias gradient's partial sums share it), and its reads: 35 of 2160 us
// at 16384 x 5120 -> 1280.
#include "ag_flce.cuh"

namespace {

inline size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

struct LinPlan {
  bool bf16;
  int64_t ldk, ldc;                                         // row lengths of the operands with K / C columns
  size_t act, act_lo, w, w_lo;                              // operands of forward and backward
  size_t row_inv, col_inv, col_inv2;                        // scales of fp16 pairs
  size_t max, max_words, row_max;                           // maxima they are made from (see LinMaxima)
  size_t dout, dout_lo, dout2, dout2_lo, splitk, splitk_bytes, colsum;  // backward only
  size_t total_fwd, total_bwd;
};

// Words of maxima: bounds of the row maxima; maxima of the columns that a contraction is balanced by; of the columns that
// the conversions scale; of rows.  What is found by atomics is cleared before: all but the last, if `atomics` (with few
// rows a block finds each on its own).
struct LinMaxima {
  uint32_t *bounds, *cols, *scaled, *rows;
  size_t scaled_words;
};
int lin_maxima(ag_ctx* ctx, const LinPlan& p, unsigned char* s, int C, bool atomics, LinMaxima* m) {
  uint32_t* w = reinterpret_cast<uint32_t*>(s + p.max);
  const size_t at = 4 + ((size_t)C + 3) / 4 * 4;
  *m = {atomics ? w : nullptr, w + 4, w + at, reinterpret_cast<uint32_t*>(s + p.row_max), p.max_words - at};
  if (atomics) {
    AG_CUDA(ctx, cudaMemsetAsync(w, 0, p.max_words * 4, ctx->stream));
    ag_enqueued(ctx);
  }
  return AG_OK;
}

constexpr int COLSUM_ROWS = 256;  // partial rows of the bias-gradient reduction

LinPlan lin_plan(int64_t N, int K, int C, int precision) {
  LinPlan p = {};
  p.bf16 = precision == AG_CE_BF16;
  auto up8 = [](int x) { return ((int64_t)x + 7) & ~(int64_t)7; };
  p.ldk = up8(K);
  p.ldc = up8(C);
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t o = off; off += up256(bytes); return o; };
  auto pair = [&](size_t elems, size_t& hi, size_t& lo) {
    hi = take(elems * 2);
    lo = p.bf16 ? hi : take(elems * 2);
  };
  pair((size_t)N * p.ldk, p.act, p.act_lo);
  pair((size_t)K * p.ldc, p.w, p.w_lo);
  p.row_inv = take((size_t)(N > K ? N : K) * 4 * 2);  // [act or dout | w]
  p.col_inv = take((size_t)(K > C ? K : C) * 4);
  p.col_inv2 = take((size_t)C * 4);
  p.max_words = 4 + 2 * (size_t)C + K + 8;
  p.max = take(p.max_words * 4);
  p.row_max = take((size_t)(N > K ? N : K) * 4);
  p.total_fwd = off;
  pair((size_t)N * p.ldc, p.dout, p.dout_lo);
  p.dout2 = p.dout;
  p.dout2_lo = p.dout_lo;
  if (!p.bf16) pair((size_t)N * p.ldc, p.dout2, p.dout2_lo);  // scaled by column, for dW
  p.splitk_bytes = up256((size_t)16 * K * C * sizeof(float));
  p.splitk = take(p.splitk_bytes);
  p.colsum = take((size_t)COLSUM_ROWS * C * sizeof(float));
  p.total_bwd = off;
  return p;
}

__global__ void __launch_bounds__(256)
colsum_partial_kernel(const float* __restrict__ g, int64_t N, int C, float* __restrict__ partial) {
  ag_pdl_wait();
  ag_colsum_partial(g, N, C, blockIdx.x * 256 + threadIdx.x, blockIdx.y, gridDim.y, partial);
}

// The partial sums of 32 columns by eight warps, one class of partial rows each, added in order.  One thread per column waited
// for P / 8 loads one after the other in five blocks: 256 x 1280 22 us.
__global__ void __launch_bounds__(256)
colsum_final_kernel(const float* __restrict__ partial, int P, int C, float* __restrict__ out) {
  ag_pdl_wait();
  __shared__ float s_sum[8][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, c = blockIdx.x * 32 + x;
  float acc = 0.0f;
  if (c < C) {
#pragma unroll 8
    for (int p = y; p < P; p += 8) acc += partial[(int64_t)p * C + c];
  }
  s_sum[y][x] = acc;
  __syncthreads();
  if (y || c >= C) return;
  acc = out[c];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc += s_sum[i][x];
  out[c] = acc;
}

int colsum_final(ag_ctx* ctx, const AgTcColsum& q, float* out) {
  AG_LAUNCH_PDL(ctx, "colsum_final_kernel", colsum_final_kernel, (q.Cc + 31) / 32, 256, 0, (const float*)q.partial, q.parts,
                q.Cc, out);
  return AG_OK;
}

// dx += dout and db += column sums of dout in one pass: 32 columns per block, 32 rows at a time, the sums of the 32 row
// classes added in order.  For short batches, which three launches for the two would keep waiting: a block walks all rows, so
// that from 1024 rows on the launches win, later where there are columns for many blocks.  Backward, us, one pass / apart, of
// K 64 to C 64, 256 to 256, 64 to 640, 64 to 2048: 256 rows 11.9 / 14.2, 13.5 / 15.8, 13.2 / 15.9, 15.8 / 18.8; 768 rows 16.6 / 16.4,
// 17.0 / 17.2, 16.6 / 17.3, 21.1 / 22.9; 896 rows 16.6 / 16.3, 18.7 / 18.7, 17.7 / 18.7, 22.9 / 25.7; 1024 rows 17.3 / 15.7, 19.3 /
// 18.2, 18.8 / 18.1, 23.5 / 25.8; 1536 rows 20.8 / 16.9, 23.6 / 20.0, 23.4 / 20.7, 29.6 / 29.2; bf16 the same.
// A last, incomplete batch of partial sums costs the launches up to 3 us: 897 rows, 64 to 64, 16.9 / 19.7.
inline bool lin_one_pass(int64_t N, int C) { return N < (C >= 1536 ? 1536 : 1024); }
__global__ void __launch_bounds__(1024)
residual_bias_kernel(const float* __restrict__ g, int N, int C, float* __restrict__ dx, float* __restrict__ db) {
  ag_pdl_wait();
  __shared__ float s_sum[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, c = blockIdx.x * 32 + x;
  float acc = 0.0f;
  if (c < C) {
#pragma unroll 4
    for (int r = y; r < N; r += 32) {
      const int64_t at = (int64_t)r * C + c;
      const float v = g[at];
      if (dx) dx[at] += v;
      acc += v;
    }
  }
  s_sum[y][x] = acc;
  __syncthreads();
  if (y == 0 && c < C) {
    float t = db[c];
#pragma unroll
    for (int i = 0; i < 32; ++i) t += s_sum[i][x];
    db[c] = t;
  }
}

// Short products go straight from fp32 memory (ag_tc_small.cu).  As with the heads the rows beyond 128 count; what the other
// path converts, N (K + C) elements, moves the line a little.  Forward + backward, us, operand pairs / this path: 16 x 64 x 64
// 28 / 12, 64 x 768 x 768 66 / 24, 128 x 5120 x 2048 197 / 102, 512 x 1536 x 1536 95 / 70, 3000 x 512 x 1024 103 / 98 (1.5e9),
// 400 x 5120 x 1280 183 / 154 (1.8e9), 1500 x 5120 x 256 179 / 127 (1.8e9), 2000 x 512 x 2048 118 / 111 (2.0e9), 16384 x 400 x 320
// 214 / 153 (2.1e9); 2048 x 1024 x 1024 100 / 111 (2.0e9), 1024 x 1536 x 1536 108 / 120 (2.1e9), 700 x 2048 x 2000 135 / 149.  bf16:
// 3000 x 512 x 1024 70 / 62, 400 x 5120 x 1280 101 / 98, 16384 x 400 x 320 128 / 104, 1024 x 1536 x 1536 70 / 78.
// Few columns: what the other path converts, reads and writes again is the activations, N K elements however few columns they meet,
// while a multiply-add here costs what it costs.  So up to 128 columns this path is ahead at any size, and beyond them by how much
// they are more.  Backward has more to convert, the forward no split of the contraction to lose.  Operand pairs / this path, us:
//   16384 x 5120 x 128 forward 194 / 160, backward 572 / 428; 16384 x 3312 x 88 142 / 112 and 408 / 287; 16384 x 3312 x 192 159 / 186 and
//   431 / 386; 8000 x 3312 x 256 104 / 114 and 250 / 216; 8000 x 1024 x 384 55 / 63 and 129 / 106; 16384 x 1024 x 256 68 / 64 and 185 /
//   143; 16384 x 256 x 640 70 / 58 and 152 / 113; 8000 x 3312 x 384 120 / 143 and 274 / 298; 8000 x 1024 x 640 79 / 87 and 160 / 164;
//   bf16 16384 x 5120 x 128 129 / 109 and 369 / 311; 8000 x 3312 x 256 65 / 69 and 155 / 145; 8000 x 5120 x 256 90 / 99 and 204 / 212.
bool lin_fits(int64_t N, int K, int C) {
  constexpr int64_t most = (int64_t)AG_TCS_MAX_SPLITS * AG_TCS_MAX_K;
  return N <= most && C <= most && K <= most / 2 && (double)K * C < (1 << 30) && (double)N * (K > C ? K : C) < (1 << 30);
}
bool lin_short(int64_t N, int K, int C) {
  return lin_fits(N, K, C) && ((double)N - 128.0) * K * C <= 1.8e9 + 40.0 * ((double)N * K + (double)N * C);
}
bool lin_narrow(int64_t N, int K, int C, bool backward, bool bf16) {
  const double nk = (double)N * K, nc = (double)N * C, free = !backward ? 140.0 : bf16 ? 200.0 : 240.0;
  return lin_fits(N, K, C) && nk * (C - free) <= (backward ? 1.8e9 : 1.5e9) + free * nc;
}
// Longest contraction of a CTA in the forward: three times the elements of a chain of operand pairs make as many additions
int lin_small_max_k(int chunk, int K) {
  const int least = ((K + 63) / 64 + AG_TCS_MAX_SPLITS - 1) / AG_TCS_MAX_SPLITS * 64, most = 3 * chunk / 64 * 64;
  return most > least ? most : least;
}
struct LinSmallPlan {
  size_t dact, dact_bytes, dw, dw_bytes, fwd_bytes, total_bwd, total;
};
LinSmallPlan lin_small_plan(int64_t N, int K, int C) {
  LinSmallPlan p = {};
  // for the shortest chains that a context may ask for: the plan is made without one
  p.fwd_bytes = ag_tcs_split_bytes(N, C, K, lin_small_max_k(64, K));
  p.dact_bytes = ag_tcs_split_bytes(N, K, C, AG_TCS_MAX_K);
  p.dw = up256(p.dact_bytes);
  p.dw_bytes = ag_tcs_split_bytes(K, C, N, AG_TCS_MAX_K);
  p.total_bwd = p.dw + up256(p.dw_bytes);
  const size_t colsum = up256((size_t)COLSUM_ROWS * C * sizeof(float));  // of long batches, before the products
  if (p.total_bwd < colsum) p.total_bwd = colsum;
  p.total = p.total_bwd < up256(p.fwd_bytes) ? up256(p.fwd_bytes) : p.total_bwd;
  return p;
}

size_t lin_narrow_room(int64_t N, int K, int C, bool backward, int chunk) {
  return backward ? lin_small_plan(N, K, C).total_bwd : ag_tcs_split_bytes(N, C, K, lin_small_max_k(chunk, K));
}

// The route of a call, and the bytes that it has to bring.  Few columns bring those of the operand pairs and are taken this way where
// they suffice: long outputs of a context with short chains may need more (14359 x 200 x 2180 forward, chains of 64: 250 MB, pairs 13).
bool lin_route(const LinPlan& pairs, int64_t N, int K, int C, bool backward, int chunk, size_t scratch_bytes, size_t* need) {
  if (lin_short(N, K, C)) {
    *need = lin_small_plan(N, K, C).total;
    return true;
  }
  *need = backward ? pairs.total_bwd : pairs.total_fwd;
  return lin_narrow(N, K, C, backward, pairs.bf16) && scratch_bytes >= lin_narrow_room(N, K, C, backward, chunk);
}

int lin_small_forward(ag_ctx* ctx, const float* x, const float* act, const float* w, const float* b, float* out, int64_t N,
                      int K, int C, int parts, unsigned char* s) {
  const int max_k = lin_small_max_k(ctx->linear_k_chunk, K);
  AgTcsGemm g;
  g.A = AgTcsOperand{act, K, 0};
  g.B = AgTcsOperand{w, C, 1};
  g.M = (int)N; g.N = C; g.K = K;
  g.D = out; g.ldd = C;
  g.bias = b; g.resid = x; g.ld_resid = C;
  g.ws = reinterpret_cast<float*>(s);
  g.ws_bytes = lin_short(N, K, C) ? lin_small_plan(N, K, C).fwd_bytes : ag_tcs_split_bytes(N, C, K, max_k);
  return ag_tcs_gemm(ctx, AG_TCS_STORE, parts, &g, 1, max_k, nullptr, nullptr);
}

int lin_small_backward(ag_ctx* ctx, const float* dout, const float* act, const float* w, float* dact, float* dw, int64_t N,
                       int K, int C, int parts, unsigned char* s) {
  const LinSmallPlan p = lin_small_plan(N, K, C);
  AgTcsGemm g[2];
  int n = 0;
  if (dact) {
    AgTcsGemm& q = g[n++];
    q.A = AgTcsOperand{dout, C, 0};
    q.B = AgTcsOperand{w, C, 0};
    q.M = (int)N; q.N = K; q.K = C;
    q.D = dact; q.ldd = K; q.accumulate = true;
    q.ws = reinterpret_cast<float*>(s);
    q.ws_bytes = p.dact_bytes;
  }
  if (dw) {
    AgTcsGemm& q = g[n++];
    q.A = AgTcsOperand{act, K, 1};
    q.B = AgTcsOperand{dout, C, 1};
    q.M = K; q.N = C; q.K = (int)N;
    q.D = dw; q.ldd = C; q.accumulate = true;
    q.ws = reinterpret_cast<float*>(s + p.dw);
    q.ws_bytes = p.dw_bytes;
  }
  return n ? ag_tcs_gemm(ctx, AG_TCS_STORE, parts, g, n, AG_TCS_MAX_K, nullptr, nullptr) : AG_OK;
}

int check_shape(ag_ctx* ctx, int64_t N, int K, int C, int precision) {
  AG_REQUIRE(ctx, N > 0 && K > 0 && C > 0 && N < (1ll << 31), "linear_add: bad shape N=%lld K=%d C=%d", (long long)N, K, C);
  AG_REQUIRE(ctx, precision == AG_CE_3XTF32 || precision == AG_CE_BF16,
             "linear_add: precision must be AG_CE_3XTF32 or AG_CE_BF16 (tensor-core op)");
  const int q = precision == AG_CE_BF16 ? 8 : 4;
  AG_REQUIRE(ctx, K % q == 0 && C % q == 0, "linear_add: K and C must be multiples of %d for the TMA operand rows", q);
  return AG_OK;
}

}  // namespace

extern "C" size_t ag_linear_add_scratch_bytes(int64_t N, int K, int C, int precision) {
  if (N <= 0 || K <= 0 || C <= 0) return 0;
  const LinPlan p = lin_plan(N, K, C, precision);
  if (lin_short(N, K, C)) return lin_small_plan(N, K, C).total;
  size_t most = p.total_fwd > p.total_bwd ? p.total_fwd : p.total_bwd;
  for (int backward = 0; backward < 2; ++backward) {
    const size_t room = lin_narrow(N, K, C, backward, p.bf16) ? lin_narrow_room(N, K, C, backward, AG_LINEAR_K_CHUNK) : 0;
    if (room > most) most = room;
  }
  return most;
}

extern "C" int ag_linear_add_forward(ag_ctx* ctx, const float* x, const float* act, const float* w, const float* b,
                                     float* out, int64_t N, int K, int C, int precision, void* scratch,
                                     size_t scratch_bytes) {
  if (!ctx) return AG_ERR_INVALID;
  int rc = check_shape(ctx, N, K, C, precision);
  if (rc) return rc;
  AG_REQUIRE(ctx, act && w && out, "ag_linear_add_forward: null pointer");
  const LinPlan p = lin_plan(N, K, C, precision);
  size_t need = 0;
  const bool small = lin_route(p, N, K, C, false, ctx->linear_k_chunk, scratch_bytes, &need);
  if (!scratch || scratch_bytes < need)
    AG_FAIL(ctx, AG_ERR_SCRATCH, "ag_linear_add_forward: scratch has %zu bytes, needs %zu", scratch_bytes, need);
  AG_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "ag_linear_add_forward: scratch not 256-byte aligned");
  unsigned char* s = static_cast<unsigned char*>(scratch);
  if (small) return lin_small_forward(ctx, x, act, w, b, out, N, K, C, p.bf16 ? 1 : 3, s);
  // B[n = C][k = K] is W[K][C] as stored with the contraction index as row index: MN-major.
  AgTcGemm g;
  g.A = AgTcOperand{s + p.act, s + p.act_lo, p.ldk, 0};
  g.B = AgTcOperand{s + p.w, s + p.w_lo, p.ldc, 1};
  g.M = (int)N; g.N = C; g.K = K;
  g.D = out; g.ldd = C;
  g.bias = b; g.resid = x; g.ld_resid = C;
  if (p.bf16) {
    g.mode = AG_TC_BF16;
    if ((rc = ag_tc_split_bf16(ctx, act, K, s + p.act, p.ldk, N, K)) || (rc = ag_tc_split_bf16(ctx, w, C, s + p.w, p.ldc, K, C)))
      return rc;
  } else {
    float* row_inv = reinterpret_cast<float*>(s + p.row_inv);
    float* col_inv = reinterpret_cast<float*>(s + p.col_inv);
    LinMaxima m;
    if ((rc = lin_maxima(ctx, p, s, C, K > TC_COLS1_ROWS, &m))) return rc;
    const AgTcMaxima mx = {w, C, K, C, false, m.rows, m.bounds};
    const AgTcConvert cv[2] = {{act, K, N, K, false, s + p.act, s + p.act_lo, p.ldk, row_inv, m.rows, m.bounds, false},
                               {w, C, K, C, true, s + p.w, s + p.w_lo, p.ldc, col_inv, m.rows, m.bounds, true}};
    if ((rc = ag_tc_convert(ctx, cv, 2, &mx, 1, m.scaled, m.scaled_words, nullptr))) return rc;
    g.mode = AG_TC_F16X3;
    g.row_mul = row_inv;
    g.col_mul = col_inv;
    g.chain_elems = ctx->linear_k_chunk;
  }
  return ag_tc_gemm(ctx, &g, 1);
}

extern "C" int ag_linear_add_backward(ag_ctx* ctx, const float* dout, const float* act, const float* w, float* dx,
                                      float* dact, float* dw, float* db, int64_t N, int K, int C, int precision,
                                      void* scratch, size_t scratch_bytes) {
  if (!ctx) return AG_ERR_INVALID;
  int rc = check_shape(ctx, N, K, C, precision);
  if (rc) return rc;
  AG_REQUIRE(ctx, dout, "ag_linear_add_backward: null dout");
  AG_REQUIRE(ctx, (!dact || w) && (!dw || act), "ag_linear_add_backward: dact needs w, dw needs act");
  const LinPlan p = lin_plan(N, K, C, precision);
  size_t need = 0;
  const bool small = lin_route(p, N, K, C, true, ctx->linear_k_chunk, scratch_bytes, &need);
  if (!scratch || scratch_bytes < need)
    AG_FAIL(ctx, AG_ERR_SCRATCH, "ag_linear_add_backward: scratch has %zu bytes, needs %zu", scratch_bytes, need);
  AG_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "ag_linear_add_backward: scratch not 256-byte aligned");
  unsigned char* s = static_cast<unsigned char*>(scratch);
  if (small && db && lin_one_pass(N, C)) {
    AG_REQUIRE(ctx, !dx || (ag_aligned16(dout) && ag_aligned16(dx)), "ag_linear_add_backward: pointers must be 16-byte aligned");
    AG_LAUNCH_PDL(ctx, "residual_bias_kernel", residual_bias_kernel, (C + 31) / 32, 1024, 0, dout, (int)N, C, dx, db);
    return lin_small_backward(ctx, dout, act, w, dact, dw, N, K, C, p.bf16 ? 1 : 3, s);
  }
  if (dx) {
    rc = ag_add_backward(ctx, dout, dx, nullptr, N * (int64_t)C);
    if (rc) return rc;
  }
  // a partial row per 64 rows of dout at least: the final pass adds them up, a class of them per warp
  const int64_t chunks = (N + 63) / 64;
  const AgTcColsum sums = {dout, N, C, (int)(chunks < COLSUM_ROWS ? chunks : COLSUM_ROWS),
                           reinterpret_cast<float*>(s + (small ? 0 : p.colsum))};
  const bool with_maxima = db && !p.bf16 && !small && (dact || dw);  // the partial sums share the launch of the maxima
  if (db && !with_maxima) {
    AG_LAUNCH_PDL(ctx, "colsum_partial_kernel", colsum_partial_kernel, dim3((C + 255) / 256, sums.parts), 256, 0, dout, N, C,
                  sums.partial);
    if ((rc = colsum_final(ctx, sums, db))) return rc;
  }
  if (!dact && !dw) return AG_OK;
  if (small) return lin_small_backward(ctx, dout, act, w, dact, dw, N, K, C, p.bf16 ? 1 : 3, s);
  const int mode = p.bf16 ? AG_TC_BF16 : AG_TC_F16X3;
  if (p.bf16 && (rc = ag_tc_split_bf16(ctx, dout, C, s + p.dout, p.ldc, N, C))) return rc;
  // The two products are independent: one launch deals the tiles of both.
  AgTcGemm g[2];
  AgTcConvert cv[4];
  AgTcMaxima mx[2];
  LinMaxima m = {};
  int n = 0, n_cv = 0, n_mx = 0;
  if (!p.bf16 && (rc = lin_maxima(ctx, p, s, C, N > TC_COLS1_ROWS || K > TC_FEW_ROWS, &m))) return rc;
  if (dact) {
    // dact[N,K] += dout[N,C] . (W[K,C])^T : both K-major as stored
    AgTcGemm& q = g[n++];
    q.mode = mode;
    q.A = AgTcOperand{s + p.dout, s + p.dout_lo, p.ldc, 0};
    q.B = AgTcOperand{s + p.w, s + p.w_lo, p.ldc, 0};
    q.M = (int)N; q.N = K; q.K = C;
    q.D = dact; q.ldd = K; q.accumulate = true;
    if (p.bf16) {
      if ((rc = ag_tc_split_bf16(ctx, w, C, s + p.w, p.ldc, K, C))) return rc;
    } else {
      float* row_inv = reinterpret_cast<float*>(s + p.row_inv);
      float* w_inv = row_inv + (N > K ? N : K);
      mx[n_mx++] = {w, C, K, C, true, m.cols, nullptr};
      cv[n_cv++] = {dout, C, N, C, false, s + p.dout, s + p.dout_lo, p.ldc, row_inv, m.cols, nullptr, false};
      cv[n_cv++] = {w, C, K, C, false, s + p.w, s + p.w_lo, p.ldc, w_inv, m.cols, nullptr, true};
      q.row_mul = row_inv;
      q.col_mul = w_inv;
    }
  }
  if (dw) {
    // dW[K,C] += act^T . dout : the contraction index (token row) is the row index of both as stored
    AgTcGemm& q = g[n++];
    q.mode = mode;
    q.A = AgTcOperand{s + p.act, s + p.act_lo, p.ldk, 1};
    q.B = AgTcOperand{s + p.dout2, s + p.dout2_lo, p.ldc, 1};
    q.M = K; q.N = C; q.K = (int)N;
    q.D = dw; q.ldd = C; q.accumulate = true;
    q.ws = reinterpret_cast<float*>(s + p.splitk);
    q.ws_bytes = p.splitk_bytes;
    if (p.bf16) {
      if ((rc = ag_tc_split_bf16(ctx, act, K, s + p.act, p.ldk, N, K))) return rc;
    } else {
      float* k_inv = reinterpret_cast<float*>(s + p.col_inv);
      float* c_inv = reinterpret_cast<float*>(s + p.col_inv2);
      mx[n_mx++] = {dout, C, N, C, false, m.rows, m.bounds};
      cv[n_cv++] = {act, K, N, K, true, s + p.act, s + p.act_lo, p.ldk, k_inv, m.rows, m.bounds, false};
      cv[n_cv++] = {dout, C, N, C, true, s + p.dout2, s + p.dout2_lo, p.ldc, c_inv, m.rows, m.bounds, true};
      q.row_mul = k_inv;
      q.col_mul = c_inv;
    }
  }
  if (n_cv && (rc = ag_tc_convert(ctx, cv, n_cv, mx, n_mx, m.scaled, m.scaled_words, with_maxima ? &sums : nullptr))) return rc;
  if (with_maxima && (rc = colsum_final(ctx, sums, db))) return rc;
  return ag_tc_gemm(ctx, g, n);
}
