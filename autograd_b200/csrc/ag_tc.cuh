// What the tensor-core kernels share (ag_flce_tc.cu, ag_tc_small.cu): tcgen05 instructions, shared-memory matrix
// descriptors, bounded waits, stores of accumulator rows.
#pragma once

#include "ag_common.cuh"

namespace {

constexpr int TC_BM = 128;
constexpr int TC_BK = 64;        // elements of K per stage: 128 bytes
constexpr int TC_MN_GROUP = 64;  // elements of MN per 128-byte row of an MN-major tile
constexpr uint32_t TC_WAIT_LIMIT = 1u << 22;
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ag_smem_u32(bar))
               : "memory");
}

// One MMA from the two halves of each shared-memory descriptor (low word: address and leading byte
// offset, high word: stride byte offset, version, layout).  ACC = 2: accumulate flag from a register
// (the first MMA of a stage), ACC = 1: always accumulate (no predicate set-up instruction).
// PAIR: the instruction spans a pair of CTAs (cta_group::2, M = 256): issued by the leader CTA only,
// it reads A rows and B columns from the shared memory of both CTAs at the same offsets and writes
// 128 accumulator rows into the tensor memory of each.
#define TC_MMA_ASM(GROUP, SETP)                                                              \
  "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t" SETP "\n\t"                                     \
  "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"                                           \
  "tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %5, p;\n\t}"
template <int ACC, bool PAIR>
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                       uint32_t idesc, uint32_t accumulate) {
#define TC_MMA_CASE(GROUP)                                                                                        \
  if (ACC == 2)                                                                                                  \
    asm volatile(TC_MMA_ASM(GROUP, "setp.ne.b32 p, %6, 0;")::"r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo),       \
                 "r"(b_hi), "r"(idesc), "r"(accumulate)                                                          \
                 : "memory");                                                                                    \
  else                                                                                                           \
    asm volatile(TC_MMA_ASM(GROUP, "setp.eq.b32 p, 0, 0;")::"r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo),        \
                 "r"(b_hi), "r"(idesc)                                                                           \
                 : "memory");
  if (PAIR) { TC_MMA_CASE("2") } else { TC_MMA_CASE("1") }
#undef TC_MMA_CASE
}

// Shared-memory matrix descriptors (version 1, Blackwell), as two 32-bit words.
//   low word : bits 0-13 start address >> 4, bits 16-29 leading byte offset >> 4
//   high word: bits 0-13 stride byte offset >> 4, bit 14 version, bits 29-31 layout type
// K-major operand, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart (stride byte
// offset 64), leading byte offset unused (1), layout 2; one MMA consumes 32 bytes of K inside the row,
// so consecutive MMAs advance the start address by 2 units.
// MN-major operand: the tile is stored as [MN group][k row][128 bytes of MN]; consecutive MN groups
// are TC_BK * 128 bytes apart (leading byte offset), the swizzle atom is 8 k rows (stride byte offset 64,
// layout 2).  One MMA consumes 16 k-rows of 128 bytes: 128 address units.
struct TcDesc {
  uint32_t lo_const, step;
  static constexpr uint32_t hi = 64u | (1u << 14) | (2u << 29);
  __device__ __forceinline__ void init(int mn_major) {
    lo_const = (mn_major ? (((uint32_t)TC_BK * 128u) >> 4) & 0x3FFFu : 1u) << 16;
    step = mn_major ? 128u : 2u;
  }
};

__device__ __forceinline__ void tc_tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
      "%23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tc_tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Bounded wait that also gives up when another role of the CTA has already given up.
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t i = 0; i < TC_WAIT_LIMIT; ++i) {
    if (ag_mbar_try_wait(bar, parity)) return true;
    if ((i & 127u) == 127u) {
      if (*abort_flag) return false;
      __nanosleep(20);
    }
  }
  *abort_flag = 1;
  return false;
}

__device__ __forceinline__ float tc_exp2(float x) {  // 2^x by the PTX instruction, ~2 ulp
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// ---------------------------------------------------------------------------- epilogue stores
// An epilogue lane owns one row of the tile, so storing from its registers would touch 32 rows per
// instruction, a sector each.  Every warp passes blocks of 32 rows x 64 bytes through shared memory instead
// (16-byte pieces, swizzled by the row so that neither side has bank conflicts) and accesses memory with
// four lanes per row.
__device__ __forceinline__ float4* tc_stage_at(unsigned char* s, int row, int piece) {
  return reinterpret_cast<float4*>(s + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4));
}

// 16 columns of a 32-row block (rows x cols of it are inside the output): D (+)= v (+ bias) (+ resid), v[] = the lane's row
__device__ __forceinline__ void tc_store_cols16(unsigned char* s, int lane, const float* v, float* D, int64_t ldd, int rows,
                                                int cols, bool vec, int accumulate, const float* bias, const float* resid,
                                                int64_t ld_resid) {
  const int r4 = lane >> 2, piece = lane & 3;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j) *tc_stage_at(s, lane, j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  __syncwarp();
  if (vec && cols >= 16) {
    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bias) b4 = make_float4(bias[piece * 4], bias[piece * 4 + 1], bias[piece * 4 + 2], bias[piece * 4 + 3]);
    float* d = D + (int64_t)r4 * ldd + piece * 4;
    const float* q = resid + (int64_t)r4 * ld_resid + piece * 4;
    // what has to be read of the block is requested before anything waits
    float4 old[4];
    if (accumulate || resid) {
      const float* from = accumulate ? d : q;
      const int64_t ld = 8 * (accumulate ? ldd : ld_resid);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (r4 + 8 * i < rows) old[i] = *reinterpret_cast<const float4*>(from + i * ld);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (r4 + 8 * i >= rows) continue;
      float4 t = *tc_stage_at(s, r4 + 8 * i, piece);
      if (accumulate || resid) { t.x += old[i].x; t.y += old[i].y; t.z += old[i].z; t.w += old[i].w; }
      if (bias) { t.x += b4.x; t.y += b4.y; t.z += b4.z; t.w += b4.w; }
      if (accumulate && resid) {
        const float4 o = *reinterpret_cast<const float4*>(q + i * 8 * ld_resid);
        t.x += o.x; t.y += o.y; t.z += o.z; t.w += o.w;
      }
      *reinterpret_cast<float4*>(d + i * 8 * ldd) = t;
    }
  } else {  // a row pitch or base that is not 16-byte aligned, or the last columns: two rows per instruction
    const int c = lane & 15;
    if (c < cols) {
      for (int r = lane >> 4; r < rows; r += 2) {
        float t = reinterpret_cast<const float*>(tc_stage_at(s, r, c >> 2))[c & 3];
        float* d = D + (int64_t)r * ldd + c;
        if (accumulate) t += *d;
        if (bias) t += bias[c];
        if (resid) t += resid[(int64_t)r * ld_resid + c];
        *d = t;
      }
    }
  }
}

}  // namespace
