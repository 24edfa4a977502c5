// tcgen05 and tiled-TMA wrappers of the prefill kernels.
#pragma once

#include <cuda.h>  // CUtensorMap's type only

#include "common.cuh"

namespace tc {

DRB_DEV void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {  // one full warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
DRB_DEV void tmem_dealloc(uint32_t base, uint32_t cols) {  // one full warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}
DRB_DEV void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
DRB_DEV void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, groups of eight rows group_stride bytes apart.
DRB_DEV uint64_t smem_desc(const void* p, uint32_t group_stride) {
  const uint64_t addr = (uint64_t)(smem_u32(p) >> 4) & 0x3FFFull;
  return addr | (1ull << 16) /* leading offset: unused with swizzle */ | ((uint64_t)(group_stride >> 4) << 32) |
         (1ull << 46) /* descriptor version */ | (2ull << 61) /* SWIZZLE_128B */;
}

// Instruction descriptor for kind::f16: fp16 x fp16 -> fp32, both operands K-major, M = 128, N = n.
DRB_DEV uint32_t instr_desc_f16(int n) {
  return (1u << 4) /* D = f32 */ | (0u << 7) /* A = f16 */ | (0u << 10) /* B = f16 */ | ((uint32_t)(n >> 3) << 17) | (128u >> 4 << 24);
}

// D [128 lanes, n columns] (+)= A . B^T with A in tensor memory: 128 lanes, two halves (k even, k odd) per column, eight
// columns per K = 16. One thread (elect_one).
DRB_DEV void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

// Arrives on `bar` once every MMA issued so far by this thread has completed.
DRB_DEV void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 32 consecutive columns of this warp's 32 lanes; complete after tmem_wait_st.
DRB_DEV void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, "
      "%19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
      "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
      "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
DRB_DEV void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 16 consecutive fp32 columns of this warp's 32 lanes.
DRB_DEV void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Lanes 0..15 (v[0]) and 16..31 (v[1]) of this warp's 32 x 16 columns, either half in the layout of mma.sync accumulators: thread 4 i + c
// gets lane i, columns 2 c and 2 c + 1 in v[.][0], v[.][1], lane i + 8 in v[.][2], v[.][3]; the next eight columns in v[.][4..7].
DRB_DEV void tmem_ld_halves16(uint32_t taddr, uint32_t (&v)[2][8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(v[0][0]), "=&r"(v[0][1]), "=&r"(v[0][2]), "=&r"(v[0][3]), "=&r"(v[0][4]), "=&r"(v[0][5]), "=&r"(v[0][6]), "=&r"(v[0][7]), "=&r"(v[1][0]),
        "=&r"(v[1][1]), "=&r"(v[1][2]), "=&r"(v[1][3]), "=&r"(v[1][4]), "=&r"(v[1][5]), "=&r"(v[1][6]), "=&r"(v[1][7])
      : "r"(taddr), "r"(taddr + (16u << 16))
      : "memory");
}

DRB_DEV void tmem_ld16(uint32_t taddr, uint32_t (&v)[2][8]) { tmem_ld16(taddr, reinterpret_cast<uint32_t(&)[16]>(v)); }

// Byte offset of 16-byte chunk c (0..7) of row r inside a K-major 128-byte-swizzled tile.
DRB_DEV uint32_t swz_off(int r, int c) { return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4)); }

// Two floats -> packed fp16 (lo, hi), round to nearest, clamped to the largest finite fp16: the operands of the
// tensor-core path are fp16, whose range ends at 65504 where bf16 and fp32 carry on. An outlier beyond it then
// degrades (it is clamped) instead of turning a token's whole output row into NaN through an infinity.
DRB_DEV uint32_t f2h2_sat(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
DRB_DEV __half f2h_sat(float v) {
  unsigned short h;
  asm("cvt.rn.satfinite.f16.f32 %0, %1;" : "=h"(h) : "f"(v));
  return __ushort_as_half(h);
}

// ---- tiled TMA loads into shared memory, completing on an mbarrier; the tensor maps live in kernel parameter space --------
DRB_DEV void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                   smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
               : "memory");
}
DRB_DEV void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                   smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
               : "memory");
}
DRB_DEV void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}
// Four rows of a 2-D map whose box is one row, from column c0 on.
DRB_DEV void tma_gather4(void* dst, const CUtensorMap* map, int c0, int r0, int r1, int r2, int r3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(smem_u32(bar))
      : "memory");
}

}  // namespace tc
