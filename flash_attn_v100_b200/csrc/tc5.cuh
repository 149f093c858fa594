// 5th-generation tensor core helpers (tcgen05 + TMEM), sm_100a.
#pragma once
#include "common.cuh"

namespace fa {

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// MMAs are issued with the whole warp converged by one elected lane (elect.sync): the addresses and descriptors are then
// uniform across the warp, which keeps the instruction stream of the issuing warp short.  Commits are issued the same
// way, so that they track the MMAs of the same thread.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
      : "memory");
}

// Runs of four or eight MMAs, D[tmem] (+)= A * B, issued as one sequence: the lane is elected once, and an operand's place in step i is its place in step
// 0 plus a constant, OFF::a(i) and OFF::b(i), in units of the descriptor (16 bytes) or in columns of tensor memory.  `accumulate` is for the first
// step; the others always add.  Alone on an SM such a run takes 64.5 cycles per MMA of 128 x 128 x 16, 128.5 of 128 x 256 x 16, and 44 to 49 of anything
// with up to 64 columns, whatever its rows.  Against one election, two 64-bit sums and a predicate per MMA, which delay the issuing warp beside busy
// ones: packed prompts (16 of 128 to 4096 tokens, 32 heads on 8 of 128) 999 -> 986 us, heads of 256 (2 x 2048 tokens) 137.5 -> 135.7, gated recurrence
// (16 x 1024 tokens, 32 heads of 128) 236.5 -> 235.1.
#define FA_MMA_FIRST(A)                                               \
  "elect.sync _|q, 0xffffffff;\n\t"                                   \
  "setp.ne.b32 p, %4, 0;\n\t"                                         \
  "setp.eq.u32 t, %3, %3;\n\t"                                        \
  "@q tcgen05.mma.cta_group::1.kind::f16 [%0], " A ", %2, %3, p;\n\t"
#define FA_MMA_SS(ia, ib)                                             \
  "add.u32 x, al, %" #ia ";\n\tadd.u32 y, bl, %" #ib ";\n\t"          \
  "mov.b64 a, {x, ah};\n\tmov.b64 b, {y, bh};\n\t"                    \
  "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
#define FA_MMA_TS(ia, ib)                                             \
  "add.u32 x, %1, %" #ia ";\n\tadd.u32 y, bl, %" #ib ";\n\t"          \
  "mov.b64 b, {y, bh};\n\t"                                           \
  "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %3, t;\n\t"
#define FA_MMA_REGS "{\n\t.reg .pred p, q, t;\n\t.reg .b32 x, y, al, ah, bl, bh;\n\t.reg .b64 a, b;\n\t"
#define FA_MMA_OFF3 "n"(OFF::a(1)), "n"(OFF::b(1)), "n"(OFF::a(2)), "n"(OFF::b(2)), "n"(OFF::a(3)), "n"(OFF::b(3))
#define FA_MMA_OFF7 FA_MMA_OFF3, "n"(OFF::a(4)), "n"(OFF::b(4)), "n"(OFF::a(5)), "n"(OFF::b(5)), "n"(OFF::a(6)), "n"(OFF::b(6)), "n"(OFF::a(7)), "n"(OFF::b(7))

// A and B in shared memory.
template <class OFF>
__device__ __forceinline__ void tc_mma_ss4(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(FA_MMA_REGS "mov.b64 {al, ah}, %1;\n\tmov.b64 {bl, bh}, %2;\n\t" FA_MMA_FIRST("%1") FA_MMA_SS(5, 6) FA_MMA_SS(7, 8) FA_MMA_SS(9, 10) "}" ::"r"(d_tmem),
               "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), FA_MMA_OFF3
               : "memory");
}
template <class OFF>
__device__ __forceinline__ void tc_mma_ss8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(FA_MMA_REGS "mov.b64 {al, ah}, %1;\n\tmov.b64 {bl, bh}, %2;\n\t" FA_MMA_FIRST("%1") FA_MMA_SS(5, 6) FA_MMA_SS(7, 8) FA_MMA_SS(9, 10)
                   FA_MMA_SS(11, 12) FA_MMA_SS(13, 14) FA_MMA_SS(15, 16) FA_MMA_SS(17, 18) "}" ::"r"(d_tmem),
               "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), FA_MMA_OFF7
               : "memory");
}
// A in tensor memory, B in shared memory.
template <class OFF>
__device__ __forceinline__ void tc_mma_ts8(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(FA_MMA_REGS "mov.b64 {bl, bh}, %2;\n\t" FA_MMA_FIRST("[%1]") FA_MMA_TS(5, 6) FA_MMA_TS(7, 8) FA_MMA_TS(9, 10) FA_MMA_TS(11, 12) FA_MMA_TS(13, 14)
                   FA_MMA_TS(15, 16) FA_MMA_TS(17, 18) "}" ::"r"(d_tmem),
               "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), FA_MMA_OFF7
               : "memory");
}
#undef FA_MMA_FIRST
#undef FA_MMA_SS
#undef FA_MMA_TS
#undef FA_MMA_REGS
#undef FA_MMA_OFF3
#undef FA_MMA_OFF7

// Steps of 16 along K in 128-byte-swizzled slabs.
// Operands along K: four steps of 32 bytes per slab of 64 columns, slabs ASLAB and BSLAB bytes apart.
template <uint32_t ASLAB, uint32_t BSLAB>
struct StepsAlongK {
  static constexpr uint32_t a(int i) { return (uint32_t)(i >> 2) * (ASLAB >> 4) + (uint32_t)(i & 3) * 2u; }
  static constexpr uint32_t b(int i) { return (uint32_t)(i >> 2) * (BSLAB >> 4) + (uint32_t)(i & 3) * 2u; }
};
// A along K (slabs of ASLAB bytes), B along its columns: 16 rows of 128 bytes.
template <uint32_t ASLAB>
struct StepsByRowsB {
  static constexpr uint32_t a(int i) { return (uint32_t)(i >> 2) * (ASLAB >> 4) + (uint32_t)(i & 3) * 2u; }
  static constexpr uint32_t b(int i) { return (uint32_t)i * 128u; }
};
// Both along their rows and columns.
struct StepsByRows {
  static constexpr uint32_t a(int i) { return (uint32_t)i * 128u; }
  static constexpr uint32_t b(int i) { return (uint32_t)i * 128u; }
};
// A in tensor memory (16 16-bit columns = 8 columns), B along its columns; the rows of B start again after ROWS16 steps.
template <int ROWS16 = 8>
struct StepsTmemA {
  static constexpr uint32_t a(int i) { return (uint32_t)i * 8u; }
  static constexpr uint32_t b(int i) { return (uint32_t)(i % ROWS16) * 128u; }
};
// An operand in two parts, APART (A) or BPART (B) behind one another, by the other: four steps of OFF from step FIRST on, each with both parts, so that the small sums
// of the low part join the large ones step by step.  (All steps of the high part first, then those of the low one: the state of a gated recurrence 0.3 % further from 64 bits.)
template <class OFF, int FIRST, uint32_t APART, uint32_t BPART>
struct InTurn {
  static constexpr uint32_t a(int i) { return OFF::a(FIRST + i / 2) - OFF::a(FIRST) + (uint32_t)(i % 2) * APART; }
  static constexpr uint32_t b(int i) { return OFF::b(FIRST + i / 2) - OFF::b(FIRST) + (uint32_t)(i % 2) * BPART; }
};
// Eight steps with both parts.
template <class OFF, uint32_t APART, uint32_t BPART>
__device__ __forceinline__ void tc_mma_ss8_parts(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  tc_mma_ss8<InTurn<OFF, 0, APART, BPART>>(d_tmem, a_desc, b_desc, idesc, accumulate);
  tc_mma_ss8<InTurn<OFF, 4, APART, BPART>>(d_tmem, a_desc + OFF::a(4), b_desc + OFF::b(4), idesc, 1u);
}
template <class OFF, uint32_t APART>
__device__ __forceinline__ void tc_mma_ts8_parts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  tc_mma_ts8<InTurn<OFF, 0, APART, 0>>(d_tmem, a_tmem, b_desc, idesc, accumulate);
  tc_mma_ts8<InTurn<OFF, 4, APART, 0>>(d_tmem, a_tmem + OFF::a(4), b_desc + OFF::b(4), idesc, 1u);
}

__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// Shared-memory matrix descriptor for 128-byte-swizzled tiles made of 128-byte rows.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)2 << 61;  // 128-byte swizzle
  return d;
}

}  // namespace fa
