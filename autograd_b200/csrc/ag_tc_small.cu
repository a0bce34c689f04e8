// Products of a few tiles, straight from fp32 memory (interface in ag_flce.cuh).
//
// A head or projection of a few hundred rows is a chain of short launches: with operands converted beforehand, what the
// conversions need (maxima of channels, scales by row and by column, bounds of the columns of dl) made 12 launches of 4 to
// 27 us of which the products themselves were five.  Here sixteen warps of a CTA load fp32 elements,
// split them into bf16 parts in registers and store those as tcgen05 operands in shared memory, one thread issues the
// MMAs, eight more warps are the epilogue, beside the next tile.  No operand is written to memory, and nothing is scaled: three bf16 parts carry
// the 24 bits of an fp32 element at its own exponent, down to 2^-110.  Below that the last part has no bits left (bf16 ends at
// 2^-133) and an element keeps 2^-134 absolute: errors of the terms are 1e-7 to 2^-110, 4e-7 at 2^-114, 2e-5 at 2^-120.  A scale
// would have to be found before the products, in a launch of its own; the gradients of the logits carry one from the start.
//
//   parts = 3 (fp32-grade): x = a + b + c exactly (a: the upper 16 bits; b: the rest, rounded; c: what is left, 8 bits).
//               Six of the nine products; b c', c b' and c c' are about 2^-23 of a product at most.
//   parts = 2 (bf16x3): a = bf16(x), b = bf16(x - a), three products.      parts = 1 (bf16): one product.
// a a' is summed in an accumulator of its own, the smaller products in another one: the accumulator cuts off, 2^-24 or so
// of its value per addition, and this way the large one takes a third of the additions that (hi, lo) pairs make there.
//
// A stage is 64 contraction elements of 128 rows and BN columns.  Bound: a stage takes 2600 clocks, of which the products need
// 1540 and reading and writing shared memory (192 KB and 96 KB) 2300; what is left is the latency of L2, as 64 KB per SM are
// under way at a time, in the registers of the loading warps.  Narrower tiles save little of it.  A first stage takes 1.6 us
// after the wait for the kernel before, an epilogue 1.4-2.5.
// Measured, forward + backward against operand pairs: head 333 x 392 x 5003 97 -> 72 us, 16 x 64 x 256 55 -> 30, 64 x 1024 x
// 20000 303 -> 215; projection 64 x 768 x 768 66 -> 24, 333 x 392 x 2048 80 -> 39.
#include <atomic>

#include "ag_flce.cuh"
#include "ag_tc.cuh"

namespace {

// Warps 0-15 load and split (with eight of them a stage took 4300 clocks: two warps per scheduler do not cover the latency of
// what a packet takes), 16-23 are the epilogue, 24 issues MMAs (registers move between groups of four).  The 72 registers a
// thread that the block starts with are shared out again as 16 x 32 x 72, 8 x 32 x 88 and 4 x 32 x 40 (64512 both ways):
// beside 227 KB of shared memory there is next to no L1, so a register spilled in a loop waits for L2.
constexpr int TCS_LOAD_WARPS = 16, TCS_EPI_WARPS = 8;
constexpr int TCS_MMA_WARP = TCS_LOAD_WARPS + TCS_EPI_WARPS;
constexpr int TCS_THREADS = 32 * (TCS_MMA_WARP + 4);
constexpr int TCS_STAGING = TCS_EPI_WARPS * 2048;  // per epilogue warp: 32 rows of 64 bytes on their way to memory
constexpr uint32_t TCS_ROW = 128;                 // bytes of a row of 64 elements of one part

enum { TCS_STORE, TCS_STATS, TCS_DLOGITS };

struct TcsOperand {
  const float* p;
  int ld;
  int mn_major;  // 0: stored [MN][K]; 1: stored [K][MN]
  int mn, k;     // extents; the contiguous one is rounded up to a packet of 4 (what lies there is zero or not stored)
};

struct TcsProblem {
  TcsOperand A, B;
  int M, N, K, k_stages;
  int tiles_m, tiles_n, splits, k_per;  // k_per: stages per split
  float* D;
  int64_t ldd, split_stride;
  int accumulate;
  const float* bias;
  const float* resid;
  int64_t ld_resid;
};

struct TcsLaunch {
  TcsProblem pr[2];
  int tiles0, tiles;  // of problem 0, of both
  AgTcsHead head;
  int* status;
  int trigger;  // let the next kernel be scheduled early
};

__device__ __forceinline__ uint32_t tcs_pack_bf16(float x, float y) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float tcs_lo16(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float tcs_hi16(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

__device__ __forceinline__ float2 tcs_sub2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tsub.rn.f32x2 r, a, b;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// The parts of a packet of four elements, 8 bytes of each, at s, s + stride, s + 2 stride
template <int PARTS>
__device__ __forceinline__ void tcs_put(unsigned char* s, uint32_t stride, const float4& v) {
  uint2 a;
  float2 a01, a23;
  if (PARTS == 3) {  // the upper halves: never rounded up to Inf
    a.x = __byte_perm(__float_as_uint(v.x), __float_as_uint(v.y), 0x7632);
    a.y = __byte_perm(__float_as_uint(v.z), __float_as_uint(v.w), 0x7632);
    a01 = make_float2(tcs_hi16(__float_as_uint(v.x)), tcs_hi16(__float_as_uint(v.y)));
    a23 = make_float2(tcs_hi16(__float_as_uint(v.z)), tcs_hi16(__float_as_uint(v.w)));
  } else {
    a.x = tcs_pack_bf16(v.x, v.y);
    a.y = tcs_pack_bf16(v.z, v.w);
    a01 = make_float2(tcs_lo16(a.x), tcs_hi16(a.x));
    a23 = make_float2(tcs_lo16(a.y), tcs_hi16(a.y));
  }
  *reinterpret_cast<uint2*>(s) = a;
  if (PARTS == 1) return;
  const float2 r01 = tcs_sub2(make_float2(v.x, v.y), a01), r23 = tcs_sub2(make_float2(v.z, v.w), a23);
  const uint2 b = make_uint2(tcs_pack_bf16(r01.x, r01.y), tcs_pack_bf16(r23.x, r23.y));
  *reinterpret_cast<uint2*>(s + stride) = b;
  if (PARTS == 2) return;
  const float2 c01 = tcs_sub2(r01, make_float2(tcs_lo16(b.x), tcs_hi16(b.x)));
  const float2 c23 = tcs_sub2(r23, make_float2(tcs_lo16(b.y), tcs_hi16(b.y)));
  *reinterpret_cast<uint2*>(s + 2 * stride) = make_uint2(tcs_pack_bf16(c01.x, c01.y), tcs_pack_bf16(c23.x, c23.y));
}

// How far dl is scaled up on its way through the panel, so that every part of it is a normal number wherever the fp32 value
// is (the parts reach 16 bits further down); the exponent of the loss scale, up to 2^60, is taken out.  dX and dW are scaled
// down again.
__device__ __forceinline__ float tcs_dl_shift(float dloss) {
  const int e = (int)((__float_as_uint(dloss) >> 23) & 0xffu) - 127;
  return (float)(16 - min(max(e, -60), 60));
}

// A packet of four, zero where it is outside its operand; no branch, so that several are under way at once.
__device__ __forceinline__ float4 tcs_load4(const float* p, uint32_t inside) {
  float4 v;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
      "@q ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w)
      : "l"(p), "r"(inside));
  return v;
}

// One operand of a tile as one of the 512 threads sees it: packet t & 15 of rows t / 16 + 32 i.  A row is 64 contiguous
// elements: of K, or (MN-major) of a group of 64 columns, rows 0-63 being the first group's k.  Offsets in bytes: operands
// are smaller than 4 GB.
template <int ROWS>
struct TcsLoader {
  uint32_t at;
  int k;          // contraction index of row i: k + 32 (i & 1) where K is the row index, else k
  uint32_t mask;  // rows inside the operand
  uint32_t now;   // those of them whose k is too
  bool whole;     // all of them, in every lane of the warp
  int rows;       // i below this hold anything of the operand: the others are neither loaded nor stored
  __device__ __forceinline__ void here(const TcsOperand& o) {
    now = k < o.k ? mask : 0u;
    if (o.mn_major && k + 32 >= o.k) now &= 0x5u;
    whole = __all_sync(0xffffffffu, now == (1u << (ROWS / 32)) - 1);
  }
  __device__ __forceinline__ void init(const TcsOperand& o, int mn0, int k0) {
    const int p4 = (threadIdx.x & 15) * 4, row = threadIdx.x >> 4, inside = min(o.mn - mn0, ROWS);
    mask = 0;
    rows = o.mn_major ? (inside + 63) / 64 * 2 : (inside + 31) / 32;
    if (o.mn_major) {
      k = k0 + row;
      at = ((uint32_t)k * (uint32_t)o.ld + mn0 + p4) * 4u;
#pragma unroll
      for (int g = 0; g < ROWS / 64; ++g)
        if (mn0 + 64 * g + p4 < o.mn) mask |= 3u << (2 * g);
    } else {
      k = k0 + p4;
      at = ((uint32_t)(mn0 + row) * (uint32_t)o.ld + k) * 4u;
#pragma unroll
      for (int i = 0; i < ROWS / 32; ++i)
        if (mn0 + row + 32 * i < o.mn) mask |= 1u << i;
    }
    here(o);
  }
  __device__ __forceinline__ void load(const TcsOperand& o, float4 (&v)[ROWS / 32]) const {
    const uint32_t s1 = 128u * (uint32_t)o.ld, s2 = o.mn_major ? 256u : 2u * s1;
    const char* base = reinterpret_cast<const char*>(o.p);
    if (whole) {
#pragma unroll
      for (int i = 0; i < ROWS / 32; ++i)
        v[i] = __ldcg(reinterpret_cast<const float4*>(base + (at + (i & 1) * s1 + (i >> 1) * s2)));
    } else {
#pragma unroll
      for (int i = 0; i < ROWS / 32; ++i)
        v[i] = tcs_load4(reinterpret_cast<const float*>(base + (at + (i & 1) * s1 + (i >> 1) * s2)), now & (1u << i));
    }
  }
  __device__ __forceinline__ void next(const TcsOperand& o) {
    at += o.mn_major ? 256u * (uint32_t)o.ld : 256u;
    k += 64;
    here(o);
  }
};

struct TcsTile {
  int which, split, tm, tn, k_first, n_stages;
};
// splits outermost, row tiles innermost (they share the column operand)
__device__ __forceinline__ TcsTile tcs_tile(const TcsLaunch& L, int tile) {
  TcsTile t;
  t.which = tile >= L.tiles0;
  const TcsProblem& p = L.pr[t.which];
  if (t.which) tile -= L.tiles0;
  t.split = tile / (p.tiles_m * p.tiles_n);
  tile -= t.split * p.tiles_m * p.tiles_n;
  t.tn = tile / p.tiles_m;
  t.tm = tile - t.tn * p.tiles_m;
  t.k_first = t.split * p.k_per;
  t.n_stages = min(p.k_per, p.k_stages - t.k_first);
  return t;
}

__device__ __forceinline__ void tcs_tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// 16 columns of 32 rows on their way to D, in the layout of the store: lane l has piece l & 3 of rows l / 4 + 8 i.
struct TcsExtra {
  float4 v[4];
  __device__ __forceinline__ void load(const float* from, int64_t ld, int rows, int cols) {
    const int r4 = threadIdx.x >> 2 & 7, piece = threadIdx.x & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = tcs_load4(from + (int64_t)(r4 + 8 * i) * ld + piece * 4, r4 + 8 * i < rows && cols >= 16 ? 1u : 0u);
  }
};
__device__ __forceinline__ void tcs_store16(unsigned char* s, const float (&v)[16], const TcsExtra& extra, bool with_extra,
                                            const float* bias, float* D, int64_t ldd, int rows) {
  const int lane = threadIdx.x & 31, r4 = lane >> 2, piece = lane & 3;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j) *tc_stage_at(s, lane, j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  __syncwarp();
  float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (bias) b4 = make_float4(bias[piece * 4], bias[piece * 4 + 1], bias[piece * 4 + 2], bias[piece * 4 + 3]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (r4 + 8 * i >= rows) continue;
    float4 t = *tc_stage_at(s, r4 + 8 * i, piece);
    if (with_extra) { t.x += extra.v[i].x; t.y += extra.v[i].y; t.z += extra.v[i].z; t.w += extra.v[i].w; }
    if (bias) { t.x += b4.x; t.y += b4.y; t.z += b4.z; t.w += b4.w; }
    *reinterpret_cast<float4*>(D + (int64_t)(r4 + 8 * i) * ldd + piece * 4) = t;
  }
}

// A persistent CTA per SM; the accumulators of two tiles alternate, so that the next tile is loaded and multiplied beside an
// epilogue.
template <int EPI, int PARTS, int BN>
__global__ void __launch_bounds__(TCS_THREADS, 1) tcs_gemm_kernel(const __grid_constant__ TcsLaunch L) {
  constexpr int NA = 4, NB = BN / 32;  // packets per thread and stage
  constexpr uint32_t A_PART = 128 * TCS_ROW, B_PART = BN * TCS_ROW, STAGE = PARTS * (A_PART + B_PART);
  constexpr uint32_t ACC = PARTS == 1 ? BN : 2 * BN;  // columns of tensor memory: a a', and the smaller products
  constexpr int WIDTH = BN / 2;                       // columns of a warp in the epilogue
  extern __shared__ unsigned char tc_smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[2], empty[2], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort, s_count[TCS_EPI_WARPS];
  volatile int* abort_flag = &s_abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      ag_mbar_init(&full[s], TCS_LOAD_WARPS);
      ag_mbar_init(&empty[s], 1);
      ag_mbar_init(&acc_full[s], 1);
      ag_mbar_init(&acc_empty[s], TCS_EPI_WARPS);
    }
    s_abort = 0;
    ag_fence_mbar_init();
  }
  if (warp == TCS_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ag_smem_u32(&tmem_slot)),
                 "r"(2 * ACC)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (L.trigger) ag_pdl_trigger();  // a single wave
  // every role waits for the kernels before this one right before it touches what they write
  bool expired = false;

  if (warp >= TCS_MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == TCS_MMA_WARP && lane == 0) {
      const uint32_t tiles_u = ag_smem_u32(tiles) >> 4;
      int buf = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 1;
      for (int at = blockIdx.x; !expired && at < L.tiles; at += gridDim.x) {
        const TcsTile t = tcs_tile(L, at);
        const TcsProblem& p = L.pr[t.which];
        TcDesc dA, dB;
        dA.init(p.A.mn_major);
        dB.init(p.B.mn_major);
        // instruction descriptor: D fp32, A and B bf16, operand majors, N >> 3 at bit 17, M >> 4 at bit 24; the last column
        // tile is as wide as it has to be, the last stage as long
        const uint32_t n16 = min(BN, (p.N - t.tn * BN + 15) & ~15);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)p.A.mn_major << 15) |
                               ((uint32_t)p.B.mn_major << 16) | ((n16 >> 3) << 17) | (8u << 24);
        const uint32_t d = tmem + (uint32_t)acc * ACC;
        if (!tc_wait(&acc_empty[acc], acc_phase, abort_flag)) {
          expired = true;
          break;
        }
        for (int s = 0; s < t.n_stages; ++s) {
          if (!tc_wait(&full[buf], phase, abort_flag)) {
            expired = true;
            break;
          }
          tc_fence_after();
          const uint32_t a0 = tiles_u + (uint32_t)buf * (STAGE >> 4) + dA.lo_const;
          const uint32_t b0 = tiles_u + (uint32_t)buf * (STAGE >> 4) + ((PARTS * A_PART) >> 4) + dB.lo_const;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            if ((t.k_first + s) * TC_BK + kk * 16 >= p.K) break;
            const uint32_t a = a0 + (uint32_t)kk * dA.step, b = b0 + (uint32_t)kk * dB.step;
            const uint32_t more = (s | kk) != 0;  // the first product of an accumulator starts it
            auto product = [&](uint32_t to, int i, int j, uint32_t add) {
              tc_mma<2, false>(to, a + (uint32_t)i * (A_PART >> 4), TcDesc::hi, b + (uint32_t)j * (B_PART >> 4), TcDesc::hi,
                               idesc, add);
            };
            if (PARTS == 3) {
              product(d + BN, 0, 2, more);
              product(d + BN, 2, 0, 1u);
              product(d + BN, 1, 1, 1u);
            }
            if (PARTS >= 2) {
              product(d + BN, 0, 1, PARTS == 3 ? 1u : more);
              product(d + BN, 1, 0, 1u);
            }
            product(d, 0, 0, more);
          }
          tc_commit(&empty[buf]);
          buf ^= 1;
          phase ^= buf == 0;
        }
        tc_commit(&acc_full[acc]);
        acc ^= 1;
        acc_phase ^= acc == 0;
      }
    }
  } else if (warp < TCS_LOAD_WARPS) {
    // ------------------------------------------------------------------ loads and splits
    // a 128-byte row is swizzled in 16-byte pieces by its number modulo 8, rows 32 apart alike
    const uint32_t my_row = threadIdx.x >> 4, piece = (threadIdx.x & 15) >> 1;
    unsigned char* mine = tiles + my_row * TCS_ROW + ((piece ^ (my_row & 7u)) << 4) + ((threadIdx.x & 1) << 3);
    int buf = 0, at = blockIdx.x;
    uint32_t phase = 1;  // the first use of a stage waits for nothing
    TcsLoader<128> la;
    TcsLoader<BN> lb;
    TcsTile t = tcs_tile(L, at);
    const TcsProblem* p = &L.pr[t.which];
    la.init(p->A, t.tm * TC_BM, t.k_first * TC_BK);
    lb.init(p->B, t.tn * BN, t.k_first * TC_BK);
    float4 ra[NA], rb[NB];
    ag_pdl_wait();
    la.load(p->A, ra);
    lb.load(p->B, rb);
    int left = t.n_stages;
    while (left) {
      const int a_rows = la.rows, b_rows = lb.rows;  // of the stage that is stored now
      if (--left) {
        la.next(p->A);
        lb.next(p->B);
      } else if ((at += gridDim.x) < L.tiles) {  // the first stage of the next tile
        t = tcs_tile(L, at);
        p = &L.pr[t.which];
        la.init(p->A, t.tm * TC_BM, t.k_first * TC_BK);
        lb.init(p->B, t.tn * BN, t.k_first * TC_BK);
        left = t.n_stages;
      } else {
        la.now = lb.now = 0u;
        la.whole = lb.whole = false;
      }
      if (!tc_wait(&empty[buf], phase, abort_flag)) {
        expired = true;
        break;
      }
      unsigned char *sa = mine + (uint32_t)buf * STAGE, *sb = sa + PARTS * A_PART;
#pragma unroll
      for (int i = 0; i < NA; ++i)
        if (i < a_rows) tcs_put<PARTS>(sa + i * 32 * TCS_ROW, A_PART, ra[i]);
      la.load(p->A, ra);
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (i < b_rows) tcs_put<PARTS>(sb + i * 32 * TCS_ROW, B_PART, rb[i]);
      lb.load(p->B, rb);
      ag_fence_proxy_async();
      __syncwarp();
      if (lane == 0) ag_mbar_arrive(&full[buf]);
      buf ^= 1;
      phase ^= buf == 0;
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
    const int quarter = warp & 3, slice = (warp - TCS_LOAD_WARPS) >> 2;  // its lanes of tensor memory, its half of the columns
    unsigned char* stg = tiles + 2 * STAGE + (warp - TCS_LOAD_WARPS) * 2048;
    const AgTcsHead& h = L.head;
    ag_pdl_wait();
    float dloss = 0.0f, denom = 1.0f, shift = 0.0f;
    if (h.dloss) {
      dloss = h.dloss[0];
      shift = tcs_dl_shift(dloss);
    }
    if (EPI == TCS_DLOGITS && !h.row_scale) {
      denom = h.denom ? h.denom[0] : (float)h.rows;
      if (!h.denom && h.reduction != AG_CE_MEAN_ALL_ROWS) {  // the CTA counts the rows that take part
        int n = 0;
#pragma unroll 4
        for (int i = (warp - TCS_LOAD_WARPS) * 32 + lane; i < h.rows; i += 32 * TCS_EPI_WARPS) {
          const int target = h.targets[i];
          n += target >= 0 && target < h.V ? 1 : 0;
        }
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) s_count[warp - TCS_LOAD_WARPS] = n;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        n = 0;
        for (int w = 0; w < TCS_EPI_WARPS; ++w) n += s_count[w];
        denom = (float)(n > 0 ? n : 1);
      }
    }
    if (EPI == TCS_STATS && blockIdx.x == 0 && warp == TCS_LOAD_WARPS && lane == 0) *h.ticket = 0u;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int at = blockIdx.x; at < L.tiles; at += gridDim.x) {
      const TcsTile t = tcs_tile(L, at);
      const TcsProblem& p = L.pr[t.which];
      const int r0 = t.tm * TC_BM + quarter * 32, r = r0 + lane;
      const int col = t.tn * BN + slice * WIDTH;
      const int rows = p.M - r0 < 32 ? p.M - r0 : 32, n_valid = p.N - col;
      const bool row_in = r < p.M;
      const int target = EPI != TCS_STORE && row_in ? h.targets[r] : -1;
      const bool valid = target >= 0 && target < h.V;
      const int hit = valid ? target - col : -1;
      float e = 0.0f, sc = 0.0f;
      if (EPI == TCS_DLOGITS && row_in) {
        e = h.lse[r];
        sc = h.row_scale ? dloss * h.row_scale[r] : dloss / denom;
        if (!valid && h.ignore_mode == AG_CE_IGNORE_MASKED) sc = 0.0f;
      }
      float* D = p.D + (int64_t)t.split * p.split_stride + (int64_t)r0 * p.ldd + col;
      const float* resid = p.resid ? p.resid + (int64_t)r0 * p.ld_resid + col : nullptr;
      const bool vec = (p.ldd & 3) == 0 && (reinterpret_cast<uintptr_t>(p.D) & 15u) == 0 && (p.split_stride & 3) == 0 &&
                       (!resid || ((p.ld_resid & 3) == 0 && (reinterpret_cast<uintptr_t>(p.resid) & 15u) == 0));
      // the columns of a dl panel are padded with zeros up to its pitch
      const int width = EPI == TCS_DLOGITS ? (int)p.ldd - col : n_valid;
      // what is added to a block is requested a block ahead
      const float* more = p.accumulate ? D : resid;
      const int64_t ld_more = p.accumulate ? p.ldd : p.ld_resid;
      const bool with_extra = EPI == TCS_STORE && vec && more;
      TcsExtra extra;
      if (with_extra) {
        // the rest is asked for at L2 meanwhile: a block ahead in registers is 16 KB per SM, not enough for memory's latency
        // (dW 18000 x 1024 of 64 rows: 7 us per tile of 128 x 128 without)
        if (row_in) {
#pragma unroll
          for (int c = 16; c < WIDTH; c += 32)
            if (c < width) asm volatile("prefetch.global.L2 [%0];" ::"l"(more + (int64_t)lane * ld_more + c));
        }
        extra.load(more, ld_more, rows, width);
      }
      const float one = tc_exp2(EPI == TCS_STORE ? -shift : shift);
      // dl = p * one * sc, the larger factor first.  The shift is no part of the exponent of p: there it would take bits of the
      // argument, an error of 2^-18 of p at a loss gradient of 2^-60 instead of 2^-22.
      const float first = shift < 0.0f ? sc : one, second = shift < 0.0f ? one : sc;
      float mx = -INFINITY, sum = 0.0f;
      if (!tc_wait(&acc_full[acc], acc_phase, abort_flag)) {
        expired = true;
        break;
      }
      tc_fence_after();
      const uint32_t from = tmem + (uint32_t)acc * ACC + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(slice * WIDTH);
#pragma unroll 1
      for (int c = 0; c < WIDTH; c += 16) {
        float v[16], small[16];
        tcs_tmem_ld16(from + c, reinterpret_cast<uint32_t(&)[16]>(v));
        if (PARTS > 1) tcs_tmem_ld16(from + BN + c, reinterpret_cast<uint32_t(&)[16]>(small));
        tc_tmem_ld_wait();
        if (PARTS > 1) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] += small[j];
        }
        if (EPI == TCS_STATS) {
          if (h.logits && row_in && c < n_valid) {  // whole sectors: the pitch is a multiple of 32
            float* dst = h.logits + (int64_t)r * h.ld_logits + col + c;
#pragma unroll
            for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
          }
          float top = mx, tl = 0.0f;
          const int here = hit - c, left = n_valid - c;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (j == here) tl = v[j];
            if (j >= left) v[j] = -INFINITY;
            top = fmaxf(top, v[j]);
          }
          if (here >= 0 && here < 16 && here < left) h.tgt_logit[r] = tl;
          const float ref = top == -INFINITY ? 0.0f : top;
          sum *= tc_exp2((mx - ref) * kLog2e);  // 0 the first time
          mx = top;
#pragma unroll
          for (int j = 0; j < 16; ++j) sum += tc_exp2((v[j] - ref) * kLog2e);
          continue;
        }
        if (EPI == TCS_DLOGITS) {
          const int here = hit - c, live = sc != 0.0f ? n_valid - c : 0;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float q = tc_exp2((v[j] - e) * kLog2e) - (j == here ? 1.0f : 0.0f);
            v[j] = j < live ? q * first * second : 0.0f;
          }
        } else if (h.dloss) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] *= one;
        }
        if (rows <= 0 || c >= width) continue;
        const float* bias = EPI == TCS_STORE && p.bias ? p.bias + col + c : nullptr;
        if (vec && width - c >= 16) {
          TcsExtra next;
          if (with_extra) next.load(more + c + 16, ld_more, rows, c + 16 < WIDTH ? width - c - 16 : 0);
          tcs_store16(stg, v, extra, with_extra, bias, D + c, p.ldd, rows);
          if (with_extra) extra = next;
        } else {  // a row pitch or base that is not 16-byte aligned, or the last columns
          tc_store_cols16(stg, lane, v, D + c, p.ldd, rows, width - c, false, p.accumulate, bias, resid ? resid + c : nullptr,
                          p.ld_resid);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) ag_mbar_arrive(&acc_empty[acc]);
      if (EPI == TCS_STATS && row_in) h.part[(int64_t)(2 * t.tn + slice) * h.part_ld + r] = make_float2(mx, sum);
      acc ^= 1;
      acc_phase ^= acc == 0;
    }
  }
  if (expired && lane == 0) atomicOr(L.status, AG_STATUS_WAIT_EXPIRED);
  tc_fence_before();
  __syncthreads();
  if (warp == TCS_MMA_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * ACC) : "memory");
  }
}

// ---------------------------------------------------------------------------- ordered sums of split contractions
// D (+)= bias + resid + P[0] + P[1] + ..., for the split problems of a launch.  VEC: whole 16-byte packets everywhere.
struct TcsReduce {
  const float* P;
  int splits, M, N;
  float* D;
  int64_t ldd;
  int accumulate;
  const float* bias;
  const float* resid;
  int64_t ld_resid;
  int blocks, share;  // share: threads that add up an element, each a range of consecutive splits
};
struct TcsReduces {
  TcsReduce job[2];
};

// A small result of many splits is a few blocks of threads that each wait for a chain of loads from L2: there eight warps take
// consecutive shares of the splits (dX of 221 x 104 took 20 us with cold caches; that head over 42525 columns, together with the
// threads of ce_finish_kernel, 139.5 -> 125.3 us, 77 x 272 x 41264 171 -> 159, 469 x 72 x 14880 105 -> 96).  Where the blocks of shared sums would exceed four per SM the
// chip is full either way, and a thread adds up all splits of its packet.
constexpr int TCS_SHARE = 8;  // warps of a block

template <bool VEC>
__device__ __forceinline__ void tcs_add(float (&a)[VEC ? 4 : 1], const float* p) {
  if constexpr (VEC) {
    const float4 x = __ldcg(reinterpret_cast<const float4*>(p));
    a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w;
  } else {
    a[0] += __ldcg(p);
  }
}

template <bool VEC>
__device__ __forceinline__ void tcs_put(float* d, const float (&a)[VEC ? 4 : 1]) {
  if constexpr (VEC) *reinterpret_cast<float4*>(d) = make_float4(a[0], a[1], a[2], a[3]);
  else d[0] = a[0];
}

template <bool VEC>
__global__ void __launch_bounds__(256) tcs_reduce_kernel(const __grid_constant__ TcsReduces R) {
  ag_pdl_wait();
  const int which = (int)blockIdx.x >= R.job[0].blocks;
  const TcsReduce& j = R.job[which];
  const int block = (int)blockIdx.x - (which ? R.job[0].blocks : 0);
  const int64_t total = (int64_t)j.M * j.N;
  constexpr int W = VEC ? 4 : 1;
  const int per_row = j.N / W;
  if (j.share > 1) {  // one warp per range, 32 packets a block
    __shared__ float s_part[TCS_SHARE][32 * W];
    const int lane = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int64_t i = (int64_t)block * 32 + lane;
    const bool in = i < total / W;
    const int per = (j.splits + TCS_SHARE - 1) / TCS_SHARE, end = min(j.splits, (y + 1) * per);
    float a[W] = {};
    if (in) {
      const float* src = j.P + i * W;
#pragma unroll 4
      for (int s = y * per; s < end; ++s) tcs_add<VEC>(a, src + (int64_t)s * total);
    }
#pragma unroll
    for (int u = 0; u < W; ++u) s_part[y][lane * W + u] = a[u];
    __syncthreads();
    if (y || !in) return;
    const int m = (int)(i / per_row), n = (int)(i - (int64_t)m * per_row) * W;
    float* d = j.D + (int64_t)m * j.ldd + n;
    float b[W] = {};
    if (j.accumulate) tcs_add<VEC>(b, d);
#pragma unroll
    for (int u = 0; u < W; ++u) {
      for (int q = 0; q < TCS_SHARE; ++q) b[u] += s_part[q][lane * W + u];
      if (j.bias) b[u] += j.bias[n + u];
    }
    if (j.resid) tcs_add<VEC>(b, j.resid + (int64_t)m * j.ld_resid + n);
    tcs_put<VEC>(d, b);
    return;
  }
  for (int64_t i = (int64_t)block * 256 + threadIdx.x; i < total / W; i += (int64_t)j.blocks * 256) {
    const int m = (int)(i / per_row), n = (int)(i - (int64_t)m * per_row) * W;
    const float* src = j.P + (int64_t)m * j.N + n;
    float* d = j.D + (int64_t)m * j.ldd + n;
    float a[W] = {};
    if (j.accumulate) tcs_add<VEC>(a, d);
#pragma unroll 8
    for (int s = 0; s < j.splits; ++s) tcs_add<VEC>(a, src + (int64_t)s * total);
    if (j.bias) {
#pragma unroll
      for (int u = 0; u < W; ++u) a[u] += j.bias[n + u];
    }
    if (j.resid) tcs_add<VEC>(a, j.resid + (int64_t)m * j.ld_resid + n);
    tcs_put<VEC>(d, a);
  }
}

// ---------------------------------------------------------------------------- host side
template <int EPI, int PARTS, int BN>
int tcs_launch(ag_ctx* ctx, int grid, const TcsLaunch& L) {
  static std::atomic<bool> attr_done[AG_MAX_DEVICES];
  constexpr int SMEM = 1024 + 2 * PARTS * (128 + BN) * (int)TCS_ROW + TCS_STAGING;
  auto kern = tcs_gemm_kernel<EPI, PARTS, BN>;
  if (!attr_done[ag_dev_slot(ctx)].load(std::memory_order_relaxed)) {  // the same for every caller: may be done twice
    AG_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    attr_done[ag_dev_slot(ctx)].store(true, std::memory_order_relaxed);
  }
  AG_LAUNCH_PDL(ctx, "tcs_gemm_kernel", kern, grid, TCS_THREADS, (size_t)SMEM, L);
  return AG_OK;
}

template <int EPI>
int tcs_launch_any(ag_ctx* ctx, int parts, int bn, int grid, const TcsLaunch& L) {
  if (parts == 3) return bn == 64 ? tcs_launch<EPI, 3, 64>(ctx, grid, L) : tcs_launch<EPI, 3, 128>(ctx, grid, L);
  if (parts == 2) return bn == 64 ? tcs_launch<EPI, 2, 64>(ctx, grid, L) : tcs_launch<EPI, 2, 128>(ctx, grid, L);
  return bn == 64 ? tcs_launch<EPI, 1, 64>(ctx, grid, L) : tcs_launch<EPI, 1, 128>(ctx, grid, L);
}

// SM clocks of a stage, of what a tile takes besides (its epilogue runs beside the next tile), of the sums that follow split
// contractions and of every split in them.
double tcs_stage_clocks(int parts, int bn) {
  if (parts == 3) return bn == 64 ? 2200.0 : 2600.0;
  if (parts == 2) return bn == 64 ? 1900.0 : 2200.0;
  return bn == 64 ? 1700.0 : 1900.0;
}
// Launches up to this long hide the next one's latency (projection 2123 x 160 x 112, 8.4 us with the next kernel scheduled early, 9.0
// without).  Beside longer ones its CTAs only wait, and they start in an SM whose L1 is what 208 KB of shared memory leave (head
// 333 x 392 x 5003 76.1 / 74.3, 128 x 64 x 65536 127.3 / 120.0).
// A launch on at most half of the SMs leaves room for that, however long it is (bf16 300 x 1128 x 478 48.4 / 49.9, 64 x 1024 x 800
// 65.6 / 66.8); up to all of them it does not (projection 73 x 1840 x 736 11.6 / 11.2, head 440 x 328 x 3212 43.2 / 42.4).
constexpr double TCS_TRIGGER_CLOCKS = 14000.0;
constexpr double TCS_TILE_CLOCKS = 1500.0, TCS_SUM_CLOCKS = 5000.0, TCS_SPLIT_CLOCKS = 350.0;

// The longest path over `units` CTAs to which t0 tiles of cost c0, then t1 of cost c1 are dealt in turn: it is that of the first
// CTA, or of the last one of a round that takes a tile of either kind more.
double tcs_makespan(int t0, double c0, int t1, double c1, int units) {
  const int total = t0 + t1;
  if (total <= units) return t1 && c1 > c0 ? c1 : c0;
  double most = 0.0;
  const int at[] = {0, t0 % units - 1, t0 % units, total % units - 1, total % units, units - 1};
  for (int j : at) {
    if (j < 0 || j >= units) continue;
    const int n0 = j < t0 ? (t0 - j - 1) / units + 1 : 0, n = (total - j - 1) / units + 1;
    const double load = n0 * c0 + (n - n0) * c1;
    if (load > most) most = load;
  }
  return most;
}

constexpr int kTcsSplits[] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, AG_TCS_MAX_SPLITS};

struct TcsChoice {
  int bn, splits[2], k_per[2];
  double clocks;  // of the launch and the sums that follow it, by the model
};

// One way to cut a product of a launch
struct TcsCut {
  int splits, k_per, tiles;
  double tile, sums;
};
// Tile width and splits by the clocks of the launch and of the sums that follow it.  Runs on every call: a few dozen to a few
// hundred combinations, 0.1 to 1.5 us.
TcsChoice tcs_choose(const ag_ctx* ctx, int epi, int parts, const AgTcsGemm* g, int n, int max_stages) {
  TcsChoice best = {};
  double best_cost = 1e300;
  for (int bn : {128, 64}) {
    TcsCut cuts[2][sizeof(kTcsSplits) / sizeof(int)];
    int n_cuts[2] = {0, 0};
    for (int i = 0; i < n; ++i) {
      const int k_stages = (g[i].K + TC_BK - 1) / TC_BK;
      const int64_t tiles = (int64_t)((g[i].M + 127) / 128) * ((g[i].N + bn - 1) / bn);
      for (int want : kTcsSplits) {
        if (want > k_stages || (want > 1 && epi != TCS_STORE)) break;
        TcsCut c;
        c.k_per = (k_stages + want - 1) / want;
        c.splits = (k_stages + c.k_per - 1) / c.k_per;
        const size_t partial = (size_t)c.splits * g[i].M * g[i].N * sizeof(float);
        if ((c.splits > 1 && partial > g[i].ws_bytes) || (epi == TCS_STORE && c.k_per > max_stages)) continue;
        if (tiles * c.splits > (1 << 28)) continue;
        c.tiles = (int)(tiles * c.splits);
        c.tile = c.k_per * tcs_stage_clocks(parts, bn) + TCS_TILE_CLOCKS;
        c.sums = c.splits > 1 ? c.splits * TCS_SPLIT_CLOCKS + (double)partial / 3000.0 : 0.0;
        cuts[i][n_cuts[i]++] = c;
      }
    }
    if (!n_cuts[0] || (n == 2 && !n_cuts[1])) continue;
    const TcsCut none = {1, 1, 0, 0.0, 0.0};
    for (int a = 0; a < n_cuts[0]; ++a) {
      for (int b = 0; b < (n == 2 ? n_cuts[1] : 1); ++b) {
        const TcsCut &c0 = cuts[0][a], &c1 = n == 2 ? cuts[1][b] : none;
        const double cost = tcs_makespan(c0.tiles, c0.tile, c1.tiles, c1.tile, ctx->sm_count) + c0.sums + c1.sums +
                            (c0.splits > 1 || c1.splits > 1 ? TCS_SUM_CLOCKS : 0.0);
        if (cost < best_cost) {
          best_cost = cost;
          best = {bn, {c0.splits, c1.splits}, {c0.k_per, c1.k_per}, cost};
        }
      }
    }
  }
  return best;
}

}  // namespace

size_t ag_tcs_split_bytes(int64_t M, int64_t N, int64_t K, int max_k) {
  const int64_t k_stages = (K + TC_BK - 1) / TC_BK, tiles = ((M + 127) / 128) * ((N + 127) / 128);
  int64_t room = 1;
  for (int s : kTcsSplits)
    if (s <= k_stages && s * tiles <= 512) room = s;  // finer ones only add to the sums that follow
  for (int s : kTcsSplits)
    if ((k_stages + s - 1) / s <= max_k / TC_BK) {
      if (s > room) room = s;
      break;
    }
  return room > 1 ? (size_t)room * M * N * sizeof(float) : 0;
}

int ag_tcs_gemm(ag_ctx* ctx, int epi, int parts, const AgTcsGemm* g, int n, int max_k, const AgTcsHead* head, int* tiles_n_out) {
  static_assert((int)AG_TCS_STORE == TCS_STORE && (int)AG_TCS_STATS == TCS_STATS && (int)AG_TCS_DLOGITS == TCS_DLOGITS, "");
  const TcsChoice c = tcs_choose(ctx, epi, parts, g, n, max_k / TC_BK);
  AG_REQUIRE(ctx, c.bn, "tcs_gemm: no split of the contraction fits its workspace");
  TcsLaunch L = {};
  if (head) L.head = *head;
  L.status = ctx->d_status;
  TcsReduces R = {};
  int64_t ctas = 0, n_red = 0, red_blocks = 0;
  bool vec = true;
  for (int i = 0; i < n; ++i) {
    const AgTcsGemm& q = g[i];
    TcsProblem& p = L.pr[i];
    for (const AgTcsOperand* o : {&q.A, &q.B})
      AG_REQUIRE(ctx, ag_aligned16(o->p) && o->ld % 4 == 0, "tcs_gemm: rows must be whole 16-byte packets");
    AG_REQUIRE(ctx, (q.A.mn_major ? q.K : q.M) * q.A.ld < (1ll << 30) && (q.B.mn_major ? q.K : q.N) * q.B.ld < (1ll << 30),
               "tcs_gemm: operand of 4 GB or more");
    const int k4 = (q.K + 3) & ~3;
    p.A = TcsOperand{q.A.p, (int)q.A.ld, q.A.mn_major, q.M, q.A.mn_major ? q.K : k4};
    p.B = TcsOperand{q.B.p, (int)q.B.ld, q.B.mn_major, q.N, q.B.mn_major ? q.K : k4};
    p.M = q.M; p.N = q.N; p.K = q.K;
    p.k_stages = (q.K + TC_BK - 1) / TC_BK;
    p.tiles_m = (q.M + 127) / 128;
    p.tiles_n = (q.N + c.bn - 1) / c.bn;
    p.splits = c.splits[i];
    p.k_per = c.k_per[i];
    p.D = q.D; p.ldd = q.ldd; p.accumulate = q.accumulate ? 1 : 0;
    p.bias = q.bias; p.resid = q.resid; p.ld_resid = q.ld_resid;
    if (p.splits > 1) {
      TcsReduce& j = R.job[n_red++];
      j = TcsReduce{q.ws, p.splits, q.M, q.N, q.D, q.ldd, p.accumulate, q.bias, q.resid, q.ld_resid, 0, 1};
      vec = vec && q.N % 4 == 0 && q.ldd % 4 == 0 && ag_aligned16(q.D) && ag_aligned16(q.ws) &&
            (!q.resid || (q.ld_resid % 4 == 0 && ag_aligned16(q.resid)));
      p.D = q.ws; p.ldd = q.N; p.accumulate = 0; p.bias = nullptr; p.resid = nullptr;
      p.split_stride = (int64_t)q.M * q.N;
    }
    const int64_t t = (int64_t)p.tiles_m * p.tiles_n * p.splits;
    if (i == 0) L.tiles0 = (int)t;
    ctas += t;
  }
  AG_REQUIRE(ctx, ctas < (1ll << 31), "tcs_gemm: too many tiles");
  L.tiles = (int)ctas;
  L.trigger = c.clocks < TCS_TRIGGER_CLOCKS || ctas <= ctx->sm_count / 2;
  const int grid = (int)(ctas < ctx->sm_count ? ctas : ctx->sm_count);
  if (tiles_n_out) *tiles_n_out = L.pr[0].tiles_n;
  int rc = epi == TCS_STATS     ? tcs_launch_any<TCS_STATS>(ctx, parts, c.bn, grid, L)
           : epi == TCS_DLOGITS ? tcs_launch_any<TCS_DLOGITS>(ctx, parts, c.bn, grid, L)
                                : tcs_launch_any<TCS_STORE>(ctx, parts, c.bn, grid, L);
  if (rc || !n_red) return rc;
  for (int i = 0; i < n_red; ++i) {
    TcsReduce& j = R.job[i];
    const int64_t packets = (int64_t)j.M * j.N / (vec ? 4 : 1), most = (int64_t)ctx->sm_count * 4;
    const int64_t shared = (packets + 31) / 32, want = (packets + 255) / 256;
    if (j.splits >= TCS_SHARE && shared <= most) j.share = TCS_SHARE;
    j.blocks = (int)(j.share > 1 ? shared : want > most ? most : want);
    red_blocks += j.blocks;
  }
  if (vec) AG_LAUNCH_PDL(ctx, "tcs_reduce_kernel", tcs_reduce_kernel<true>, (int)red_blocks, 256, 0, R);
  else AG_LAUNCH_PDL(ctx, "tcs_reduce_kernel", tcs_reduce_kernel<false>, (int)red_blocks, 256, 0, R);
  return AG_OK;
}

// =========================================================================================
// The head
// =========================================================================================
namespace {

// Folds the partial statistics of one launch into those of the rows, after the last launch into the loss.  A block takes 8
// rows, T / 8 threads for each: the maxima first, then the sums scaled to it, in a fixed order.  The block that finishes last adds
// the blocks' sums (run_sum and run_max hold a block's sum and count of rows in its first row), in a fixed order too.
constexpr int CE_ROWS = 8, CE_HELD = 4;  // rows of a block; partials of a thread that stay in registers
template <int T>
__global__ void __launch_bounds__(T)
ce_finish_kernel(const float2* __restrict__ part, int64_t part_ld, int n_parts, int rows, const float* __restrict__ tgt_logit,
                 const int32_t* __restrict__ targets, const float* __restrict__ row_scale, float* __restrict__ lse,
                 float* __restrict__ loss, int V, int reduction, float* run_max, float* run_sum, uint32_t* ticket, int first,
                 int last) {
  constexpr int LANES = T / CE_ROWS, WARPS = T / 32;
  __shared__ float s_max[WARPS][CE_ROWS], s_sum[WARPS][CE_ROWS];
  __shared__ int s_cnt[WARPS];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = threadIdx.x & 7, y = threadIdx.x >> 3;
  const int r = blockIdx.x * CE_ROWS + k;
  const bool in = r < rows;
  ag_pdl_wait();
  const int t = in && y == 0 ? targets[r] : -1;
  const bool take = t >= 0 && t < V;
  const float tl = take && last ? tgt_logit[r] : 0.0f, weight = take && row_scale ? row_scale[r] : 1.0f;
  const float2 before = in && y == 0 && !first ? make_float2(run_max[r], run_sum[r]) : make_float2(-INFINITY, 0.0f);
  float2 held[CE_HELD];
  float m = before.x;
#pragma unroll
  for (int i = 0; i < CE_HELD; ++i) {
    held[i] = in && y + LANES * i < n_parts ? __ldcg(part + (int64_t)(y + LANES * i) * part_ld + r) : make_float2(-INFINITY, 0.0f);
    m = fmaxf(m, held[i].x);
  }
#pragma unroll 4
  for (int i = y + LANES * CE_HELD; i < n_parts; i += LANES)
    if (in) m = fmaxf(m, __ldcg(part + (int64_t)i * part_ld + r).x);
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
  if (lane < 8) s_max[warp][lane] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < WARPS; ++w) m = fmaxf(m, s_max[w][k]);
  // a part without a valid column is (-inf, 0); a NaN among the logits is one in the sums, whatever the maximum is
  float s = 0.0f;
  auto add = [&](const float2& v) { s += v.y == 0.0f ? 0.0f : v.y * expf(v.x - m); };
  add(before);
#pragma unroll
  for (int i = 0; i < CE_HELD; ++i) add(held[i]);
#pragma unroll 4
  for (int i = y + LANES * CE_HELD; i < n_parts; i += LANES)
    if (in) add(__ldcg(part + (int64_t)i * part_ld + r));
  s += __shfl_xor_sync(0xffffffffu, s, 8);
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  if (lane < 8) s_sum[warp][lane] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = 0.0f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) s += s_sum[w][k];
    if (!last) {
      if (y == 0 && in) {
        run_max[r] = m;
        run_sum[r] = s;
      }
      return;
    }
    float acc = 0.0f;
    if (y == 0 && in) {
      const float e = m + logf(s);
      lse[r] = e;
      if (take) acc = (e - tl) * weight;
    }
    acc = ag_warp_sum(acc);
    const int cnt = __popc(__ballot_sync(0xffffffffu, take));
    if (lane == 0) {
      run_sum[blockIdx.x * CE_ROWS] = acc;
      run_max[blockIdx.x * CE_ROWS] = __int_as_float(cnt);
      __threadfence();
      s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
  }
  if (!last) return;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  float acc = 0.0f;
  int cnt = 0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += T) {
    acc += __ldcg(run_sum + b * CE_ROWS);
    cnt += __float_as_int(__ldcg(run_max + b * CE_ROWS));
  }
  acc = ag_warp_sum(acc);
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) {
    s_sum[warp][0] = acc;
    s_cnt[warp] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < WARPS; ++w) {
      acc += s_sum[w][0];
      cnt += s_cnt[w];
    }
    float denom = 1.0f;
    if (!row_scale) denom = reduction == AG_CE_MEAN_ALL_ROWS ? (float)rows : (float)(cnt > 0 ? cnt : 1);
    loss[0] = acc / denom;
  }
}


// dl of kept logits, as the epilogue of TCS_DLOGITS makes it: a thread per packet of four columns, the columns up to the
// panel's pitch zero.
__global__ void __launch_bounds__(256)
tcs_kept_dlogits_kernel(const __grid_constant__ AgTcsHead h, float* __restrict__ dl, int ldc) {
  ag_pdl_wait();
  ag_pdl_trigger();
  const int per_row = ldc >> 2;
  const float dloss = h.dloss[0], shift = tcs_dl_shift(dloss), one = tc_exp2(shift);
  const float mean = h.row_scale ? 0.0f : dloss / (h.denom ? h.denom[0] : (float)h.rows);
  const int64_t total = (int64_t)h.rows * per_row;
#pragma unroll 2
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
    const int r = (int)(i / per_row), c = (int)(i - (int64_t)r * per_row) * 4;
    const float4 l = *reinterpret_cast<const float4*>(h.logits + (int64_t)r * h.ld_logits + c);  // its pitch is no smaller
    const float e = h.lse[r];
    const int target = h.targets[r];
    const bool valid = target >= 0 && target < h.V;
    float sc = h.row_scale ? dloss * h.row_scale[r] : mean;
    if (!valid && h.ignore_mode == AG_CE_IGNORE_MASKED) sc = 0.0f;
    const float first = shift < 0.0f ? sc : one, second = shift < 0.0f ? one : sc;
    const int hit = valid ? target - c : -1, live = sc != 0.0f ? h.V - c : 0;
    float v[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float q = tc_exp2((v[j] - e) * kLog2e) - (j == hit ? 1.0f : 0.0f);
      v[j] = j < live ? q * first * second : 0.0f;
    }
    *reinterpret_cast<float4*>(dl + (int64_t)r * ldc + c) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

int tcs_parts(int precision) { return precision == AG_CE_BF16 ? 1 : precision == AG_CE_BF16X3 ? 2 : 3; }

struct SmallPlan {
  int64_t ldc;
  size_t panel, ws_dx, dx_bytes, ws_dw, dw_bytes, total;
};
SmallPlan small_plan(const ag_flce_desc* d) {
  SmallPlan p = {};
  auto up256 = [](size_t x) { return (x + 255) & ~(size_t)255; };
  p.ldc = (d->V + 15) / 16 * 16;
  // forward: partial statistics, 16 bytes per row and tile of 64 columns at most, where the backward has dl
  p.panel = 0;
  p.ws_dx = up256((size_t)d->N * p.ldc * 4);
  p.dx_bytes = ag_tcs_split_bytes(d->N, d->C, d->V, AG_TCS_MAX_K);
  p.ws_dw = p.ws_dx + up256(p.dx_bytes);
  p.dw_bytes = ag_tcs_split_bytes(d->V, d->C, d->N, AG_TCS_MAX_K);
  p.total = p.ws_dw + up256(p.dw_bytes);
  return p;
}

}  // namespace

// Which heads: a multiply-add costs about twice what it does on converted operands, a converted element of W more than a
// hundred multiply-adds.  So the rows beyond 128 count, times the table.  Forward + backward, us, operand pairs / this path:
//   16 x 64 x 256 55 / 30, 64 x 1024 x 20000 303 / 215, 128 x 1536 x 65536 1194 / 898, 333 x 392 x 5003 98 / 72,
//   512 x 768 x 4096 117 / 104, 1024 x 1024 x 2048 131 / 124 (1.9e9), 256 x 768 x 32768 382 / 399 (3.2e9),
//   1000 x 400 x 8192 189 / 222 (2.9e9), 2048 x 768 x 4096 212 / 333 (6.0e9);
//   bf16: 700 x 200 x 10000 122 / 87 (1.1e9), 1024 x 384 x 4096 88 / 69 (1.4e9), 3000 x 64 x 10000 132 / 157 (1.8e9).
// Up to 128 rows that leaves heads of any size, at which this path is ahead in every mode: bf16x3 16 x 1536 x 65536 823 / 604,
//   64 x 1024 x 20000 217 / 174, 128 x 768 x 32768 271 / 210, 128 x 2304 x 73728 1391 / 1193; bf16 618 / 553, 167 / 155, 198 / 178,
//   1001 / 917; fp32-grade 128 x 2304 x 73728 2023 / 1523.
// Statistics and dl are not split along C, so C ends where their accumulation chain does (2304); nor are dX and dW beyond 32
// chains of that, so V and N end at 73728.  Larger heads take the operand pairs, however few rows they have.
// The panel of dl keeps the size that vocab_chunk allows.
bool ag_flce_small(const ag_flce_desc* d) {
  if (!ag_flce_tc_supported(d)) return false;
  constexpr int64_t most = (int64_t)AG_TCS_MAX_SPLITS * AG_TCS_MAX_K;
  if (d->V > most || d->N > most || d->C > AG_TCS_MAX_K) return false;
  if (d->vocab_chunk < d->V && d->N * d->V > (int64_t)d->vocab_chunk * AG_FLCE_ROWS_TILE) return false;
  return ((double)d->N - 128.0) * d->V * d->C <= (d->precision == AG_CE_3XTF32 ? 2.0e9 : 1.4e9);
}

size_t ag_flce_small_scratch_bytes(const ag_flce_desc* d) { return small_plan(d).total; }

int ag_flce_finish(ag_ctx* ctx, const ag_flce_desc* d, const float2* part, int n_parts, const int32_t* targets,
                   const float* row_scale, float* run_max, float* run_sum, const float* tgt_logit, uint32_t* ticket, float* lse,
                   float* loss, bool first, bool last) {
  const int blocks = (int)((d->N + CE_ROWS - 1) / CE_ROWS);
  auto launch = [&](auto kern, int threads) -> int {
    AG_LAUNCH_PDL(ctx, "ce_finish_kernel", kern, blocks, threads, 0, part, d->N, n_parts, (int)d->N, tgt_logit, targets, row_scale,
                  lse, loss, d->V, d->reduction, run_max, run_sum, ticket, first ? 1 : 0, last ? 1 : 0);
    return AG_OK;
  };
  // Few blocks are bound by latency, each a chain of loads that depend on the maxima of those before: beyond the partials that 32
  // threads hold per row it gets 128, so that one round of loads remains (221 rows x 333 partials took 20 us with cold caches;
  // for the head of that size see TCS_SHARE).  Many blocks hide it, and of 256 threads more of them are on an SM.  So the large
  // blocks are for little more than one wave of two per SM, than two waves where the partials are three rounds of loads.  Forward
  // passes of bf16 heads of 64 columns, us, 128 / 32 threads per row: 17000 tokens, 1500 rows 35.7 / 36.3, 2400 55.0 / 55.8, 3000
  // 57.7 / 56.5, 8192 103 / 93; 50257 tokens, 1500 59.7 / 62.1, 3000 104.1 / 104.6, 4096 135.0 / 134.6, 6000 193 / 190; 151936
  // tokens, 4096 378 / 382, 6000 550 / 547; 32768 tokens, 16384 335 / 320.
  const int quarter_waves = n_parts >= 3 * 1024 / CE_ROWS ? 17 : 9;
  const bool few = 4 * (int64_t)blocks <= (int64_t)quarter_waves * ctx->sm_count;
  return few && n_parts > 256 / CE_ROWS * CE_HELD ? launch(ce_finish_kernel<1024>, 1024) : launch(ce_finish_kernel<256>, 256);
}

int ag_flce_small_forward(ag_ctx* ctx, const ag_flce_desc* d, const float* X, const float* W, void* scratch,
                          const int32_t* targets, const float* row_scale, float* run_max, float* run_sum, float* tgt_logit,
                          uint32_t* ticket, float* lse, float* loss, float* logits) {
  const SmallPlan p = small_plan(d);
  AgTcsHead h = {};
  h.targets = targets;
  h.V = d->V;
  h.rows = (int)d->N;
  h.part = reinterpret_cast<float2*>(static_cast<unsigned char*>(scratch) + p.panel);
  h.part_ld = d->N;
  h.tgt_logit = tgt_logit;
  h.ticket = ticket;
  h.logits = logits;
  h.ld_logits = ag_flce_logits_ld(d);
  AgTcsGemm g;
  g.A = AgTcsOperand{X, d->C, 0};
  g.B = AgTcsOperand{W, d->C, 0};
  g.M = (int)d->N; g.N = d->V; g.K = d->C;
  int tiles_n = 0;
  if (int rc = ag_tcs_gemm(ctx, AG_TCS_STATS, tcs_parts(d->precision), &g, 1, AG_TCS_MAX_K, &h, &tiles_n)) return rc;
  return ag_flce_finish(ctx, d, h.part, 2 * tiles_n, targets, row_scale, run_max, run_sum, tgt_logit, ticket, lse, loss, true, true);
}

int ag_flce_small_backward(ag_ctx* ctx, const ag_flce_desc* d, const float* X, const float* W, void* scratch,
                           const int32_t* targets, const float* lse, const float* row_scale, const float* dloss,
                           const float* denom, float* dX, float* dW, const float* logits) {
  const SmallPlan p = small_plan(d);
  unsigned char* b = static_cast<unsigned char*>(scratch);
  float* dl = reinterpret_cast<float*>(b + p.panel);
  const int parts = tcs_parts(d->precision);
  AgTcsHead h = {};
  h.targets = targets;
  h.V = d->V;
  h.rows = (int)d->N;
  h.lse = lse; h.row_scale = row_scale; h.dloss = dloss; h.denom = denom;
  h.reduction = d->reduction;
  h.ignore_mode = d->ignore_mode;
  AgTcsGemm g[2];
  if (logits) {
    h.logits = const_cast<float*>(logits);
    h.ld_logits = ag_flce_logits_ld(d);
    const int64_t blocks = (d->N * (p.ldc / 4) + 511) / 512, most = (int64_t)ctx->sm_count * 8;
    AG_LAUNCH_PDL(ctx, "tcs_kept_dlogits_kernel", tcs_kept_dlogits_kernel, (int)(blocks < most ? blocks : most), 256, 0, h, dl,
                  (int)p.ldc);
  } else {
    g[0].A = AgTcsOperand{X, d->C, 0};
    g[0].B = AgTcsOperand{W, d->C, 0};
    g[0].M = (int)d->N; g[0].N = d->V; g[0].K = d->C;
    g[0].D = dl;
    g[0].ldd = p.ldc;
    if (int rc = ag_tcs_gemm(ctx, AG_TCS_DLOGITS, parts, g, 1, AG_TCS_MAX_K, &h, nullptr)) return rc;
  }
  int n = 0;
  if (dW) {  // dW += dl^T . X: the contraction index is the row index of both
    AgTcsGemm& q = g[n++];
    q = AgTcsGemm{};
    q.A = AgTcsOperand{dl, p.ldc, 1};
    q.B = AgTcsOperand{X, d->C, 1};
    q.M = d->V; q.N = d->C; q.K = (int)d->N;
    q.D = dW; q.ldd = d->C; q.accumulate = true;
    q.ws = reinterpret_cast<float*>(b + p.ws_dw);
    q.ws_bytes = p.dw_bytes;
  }
  if (dX) {  // dX += dl . W
    AgTcsGemm& q = g[n++];
    q = AgTcsGemm{};
    q.A = AgTcsOperand{dl, p.ldc, 0};
    q.B = AgTcsOperand{W, d->C, 1};
    q.M = (int)d->N; q.N = d->C; q.K = d->V;
    q.D = dX; q.ldd = d->C; q.accumulate = true;
    q.ws = reinterpret_cast<float*>(b + p.ws_dx);
    q.ws_bytes = p.dx_bytes;
  }
  return ag_tcs_gemm(ctx, AG_TCS_STORE, parts, g, n, AG_TCS_MAX_K, &h, nullptr);
}
