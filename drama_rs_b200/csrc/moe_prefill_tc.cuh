// The expert-grouped prefill GEMMs (dr_moe_prefill, dr_moe_prefill_fp8, drb_moe_prefill_block and its peer-store form) on
// the 5th-generation tensor cores, with the dequantised weights handed over in TENSOR memory.
//
//   gate/up:  for expert e with its tokens  D[128, nt] = W_tile[128, 2048] . X_e[nt, 2048]^T
//             (the tile is 64 gate rows and their 64 up rows), epilogue silu(g) * u -> act
//   down:     D[128, nt] = Wd_tile[128, 512] . act_e[nt, 512]^T -> y
//
// The weight rows are the MMA's M = 128 dimension and the tokens its N dimension (16 .. 64): most experts see a handful
// of tokens. Weights are int4 (scale and min per 64 inputs), block-FP8 (one f32 scale per 128 x 128 block) or, for the
// shared expert, int8; every one becomes an fp16 operand with one rounding, accumulated in fp32.
//
// What bounds it. A weight is read once from HBM, so the floor is 1.77 MB (int4) or 3 MB (FP8) per expert hit at the copy
// rate. Between HBM and the tensor core stands the conversion: 1.6 thread-instructions per int4 weight, 40 us for 256
// experts on all issue slots. An A operand in SHARED memory would add its store, its read by the MMA and the raw bytes'
// two passes, 5 bytes per weight through 128 B per cycle = 113 us, more than HBM takes; in tensor memory the same tile
// costs one tcgen05.st (measured 700 B per cycle and multiprocessor), the MMA reads it there (14, 19, 32 cycles for
// N = 16, 32, 64; from shared memory never below 39), and shared memory carries the raw bytes only.
//
// Roles, one block of 24 warps (FP8: 20) per multiprocessor, meeting only on mbarriers, every wait bounded (common.cuh):
//   16 convert warps (FP8: 8)  a step is 256 inputs of 128 rows; groups of eight warps take turns. A thread converts 128 inputs of
//                 one row: four (int4) or eight (8-bit) 16-byte pieces out of the swizzled raw stage, two 32-column
//                 tcgen05.st. Three stages: 128 columns each, with a token tile in shared memory.
//   MMA warp      sixteen K = 16 instructions per step, one commit that frees the stage
//   loader warp   tiled TMA: 128 rows x 128 bytes per request with the 128-byte swizzle; a gate/up tile is 64 gate rows and
//                 their 64 up rows, which a 4-D view of the weight tensor expresses; an int4 item's scales are requested while the item before
//                 still asks for its stages
//   token warp    the tokens' fp16 rows: groups of eight consecutive rows by one TMA request per step (4 KB: eight rows of
//                 four 128-byte swizzled columns), scattered rows by tile::gather4 (512 bytes per request; it costs the copy
//                 engine 19 cycles against 49 for the 4 KB box)
//   table warp    the items' rows, result rows and row factors, ahead of everybody
//   4 epilogue warps (FP8: 8)  drain an item's accumulator while the next item's MMAs fill the other one
//
// Work items: (shared expert or expert, group of up to 64 tokens, 128-row tile), enumerated from the device-side
// counts by a prefix sum each block computes for itself, the shared expert's items first, walked round robin.
// Replaces kernels/drama.cu:799-1109 of the reference (k_moe_pf_gate_up, k_moe_pf_down and their FP8 forms) together with
// the cuBLAS shared expert of src/engine.rs:351-355, 560-562.
#pragma once

#include <cuda.h>  // CUtensorMap and the encode function's type only: the entry point is resolved at run time

#include "common.cuh"
#include "tcgen05.cuh"

namespace pft {

using namespace tc;

constexpr int H = 2048, I = 512;
constexpr int GROUP_WARPS = 8, EPI_WARPS = 4;   // warps of a convert group / of an epilogue set
constexpr int MAX_WARPS = 24;
constexpr int TILE_M = 128;
constexpr int STEP_K = 256;
constexpr int MAX_NT = 64;                      // tokens per work item at most
constexpr int NST = 3;                          // stages: an A tile in tensor memory with its token tile in shared memory
constexpr int A_COLS = STEP_K / 2;              // 32-bit columns of one A tile
constexpr int A_COL0 = 128;                     // ahead of them: the accumulators
constexpr int TMEM_COLS = 512;
static_assert(A_COL0 + NST * A_COLS <= TMEM_COLS, "tensor memory");
constexpr int ROW_BYTES = 128;
constexpr int RAW_BYTES = TILE_M * ROW_BYTES;   // 16 KB: 256 int4 or 128 8-bit inputs of the tile's 128 rows
constexpr int NTAB = 4;
constexpr int MAX_E = 1024;                     // experts per launch; more are taken by further launches
constexpr int CTL_BYTES = 1024;
constexpr int SET_BYTES = (MAX_E + 2) * 4 + 8;
constexpr int TOKEN_STRIDE = 2 * H * 2;         // bytes between prepared token rows (k_prep_rows): fp16 row | factor

struct Tab {  // one work item
  int cols, used, mt, shared;   // accumulator columns (the MMA's N); those in use, in eights
  int full, srow, start;        // contiguous rows: so many boxes of eight from row srow on, and one more from row start (-1: none)
  int quads;                    // rows fetched by number: so many fours of rows[], behind the boxes
  __align__(16) int rows[MAX_NT];
  __align__(16) int dst[MAX_NT];    // result row of each column, -1: none
  __align__(16) float fac[MAX_NT];  // what the column's token row was divided by
};
struct Ctl {
  uint64_t rawfull[10], rawempty[10];      // a raw stage has landed / has been read (one arrival per convert warp of a group)
  uint64_t smfull[4];                      // an int4 item's scales have landed
  uint64_t full[NST];                      // a stage is complete: the A tile (one arrival per convert warp of a group) and the token tile (TMA)
  uint64_t done[NST];                      // the MMAs that read it have completed (tcgen05.commit)
  uint64_t accfull[4], accfree[4];         // an accumulator is complete (tcgen05.commit) / has been drained (one arrival per epilogue warp)
  uint64_t tabfull[NTAB], tabempty[NTAB];  // written / read for the last time (token, MMA and epilogue warps)
  int wtot[MAX_WARPS];                     // the prefix sum's warp totals
  uint32_t tmem_base;
};
static_assert(sizeof(Ctl) <= CTL_BYTES, "control block");

// Sizes of k_grouped<GEMM, FMT, .> and its shared memory: control block | raw stages | token tiles | int4 scales | tables | item prefix.
template <int GEMM, int FMT>
struct Smem {
  static constexpr int NT = FMT == 1 ? 32 : 64;    // tokens per item
  static constexpr int NACC = FMT == 1 ? 4 : 2;    // accumulators: int4: one per item; FP8: one per 128 inputs (see k_grouped)
  static constexpr int B_BYTES = NT * STEP_K * 2;  // one token tile
  static_assert(NT <= MAX_NT && NT * NACC <= A_COL0, "tensor memory");
  // int4: conversion is the work, two groups take turns at the steps and one set of epilogue warps follows. FP8: a weight takes half
  // an instruction to convert, but every 128 inputs have an accumulator to drain: one group, two sets that take
  // turns at the items, each with two accumulators of its own (with one set the MMAs waited for it a third of the time).
  static constexpr int GROUPS = FMT == 1 ? 1 : 2, SETS = FMT == 1 ? 2 : 1;
  static constexpr int CONV_WARPS = GROUPS * GROUP_WARPS;
  static constexpr int MMA_WARP = CONV_WARPS + SETS * EPI_WARPS, LOAD_WARP = MMA_WARP + 1, TOKEN_WARP = MMA_WARP + 2, TABLE_WARP = MMA_WARP + 3;
  static constexpr int THREADS = (TABLE_WARP + 1) * 32;  // 768 / 640
  static_assert(TABLE_WARP < MAX_WARPS, "warps");
  static constexpr int NRAW = FMT == 1 ? 10 : GEMM == 0 ? 5 : 6;           // what fits; four are enough for the copy rate (a stream of such boxes alone: 6.2 TB/s with 4, 6.5 with 6)
  static constexpr int NSM = FMT != 0 ? 0 : GEMM == 0 ? 2 : 4;             // slots for an int4 item's (scale, min) pairs: see the loader
  static constexpr int SMB = TILE_M * ((GEMM == 0 ? H : I) / 64) * 4;      // bytes of one
  static constexpr size_t BYTES = 1024 /* alignment slack */ + CTL_BYTES + NRAW * RAW_BYTES + NST * B_BYTES + NSM * SMB + NTAB * sizeof(Tab) + SET_BYTES;
  static_assert(BYTES <= 232448, "shared memory");
};

// ---- weights -> fp16 ---------------------------------------------------------------------------------------------
// A nibble in bits 0..3 of a 16-bit half, or-ed into 0x6400, is the half 1024 + q; a nibble in bits 4..7, or-ed into
// 0x5400, is the half 64 + q (the unit in the last place of 64 is 1/16). Subtracting the offset is exact, the fused
// multiply-add q*s + m rounds once.
// A nibble in bits 4..7 with nothing above it is the subnormal half q * 2^-20: with the scale times 2^20 (exact, while it stays
// below 2^-4) the fused multiply-add needs no subtraction and rounds the same number.
// The offsets live in registers the compiler cannot rebuild from immediates: it would, once per use.
struct NibbleConst {
  uint32_t k1024, k64, mixed;  // (1024, 1024), (64, 64), (1024, 64)
  DRB_DEV NibbleConst() {
    asm volatile("mov.b32 %0, 0x64006400;" : "=r"(k1024));
    asm volatile("mov.b32 %0, 0x54005400;" : "=r"(k64));
    asm volatile("mov.b32 %0, 0x54006400;" : "=r"(mixed));
  }
};
template <uint32_t MASK>
DRB_DEV uint32_t mask_or(uint32_t w, uint32_t c) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "n"(MASK), "r"(c));
  return r;
}
DRB_DEV uint32_t sub_fma(uint32_t t, uint32_t off, __half2 s2, __half2 m2) {
  const __half2 r = __hfma2(__hsub2(*reinterpret_cast<const __half2*>(&t), *reinterpret_cast<const __half2*>(&off)), s2, m2);
  return *reinterpret_cast<const uint32_t*>(&r);
}
// Eight nibbles of one word in the order (0,4) (1,5) (2,6) (3,7): one shift serves both upper pairs; 13 instructions, SMALL
// (every scale of the warp below 2^-4): 11. The token rows have to come in the same order. Issue slots are what the conversion
// runs out of; the fp16 and the integer pipe take one instruction every other cycle each, and get six and five of the eleven.
template <bool SMALL>
DRB_DEV void dequant8_perm(uint32_t w, __half2 s2, __half2 m2, __half2 big, const NibbleConst& c, uint32_t* o) {
  const uint32_t w8 = w >> 8;
  auto upper = [&](uint32_t v) {
    if (!SMALL) return sub_fma(mask_or<0x00F000F0u>(v, c.k64), c.k64, s2, m2);
    const uint32_t t = v & 0x00F000F0u;
    const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&t), big, m2);
    return *reinterpret_cast<const uint32_t*>(&r);
  };
  o[0] = sub_fma(mask_or<0x000F000Fu>(w, c.k1024), c.k1024, s2, m2);
  o[1] = upper(w);
  o[2] = sub_fma(mask_or<0x000F000Fu>(w8, c.k1024), c.k1024, s2, m2);
  o[3] = upper(w8);
}
// The same in k order: a byte holds a consecutive pair, a permute puts it into both halves. 16 instructions.
DRB_DEV void dequant8_nat(uint32_t w, __half2 s2, __half2 m2, const NibbleConst& c, uint32_t* o) {
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = sub_fma(mask_or<0x00F0000Fu>(prmt(w, 0u, 0x1111u * i), c.mixed), c.mixed, s2, m2);
}
// Eight int8 weights (two words) times one fp16 scale, in k order or in the order of dequant8_perm. 0x6400 | (b ^ 0x80) is
// the half 1024 + 128 + b; subtracting 1152 is exact, the product rounds once.
template <bool PERM>
DRB_DEV void dequant8_i8(uint32_t w0, uint32_t w1, __half2 s2, uint32_t* o) {
  const __half2 k1152 = __half2half2(__ushort_as_half((unsigned short)0x6480));
  const uint32_t u0 = w0 ^ 0x80808080u, u1 = w1 ^ 0x80808080u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t t;
    if (PERM) t = lop3_and_or(prmt(u0, u1, (uint32_t)(i | (i << 4) | ((4 + i) << 8) | ((4 + i) << 12))), 0x00FF00FFu, 0x64006400u);
    else t = prmt(i < 2 ? u0 : u1, 0x64646464u, (i & 1) ? 0x4342u : 0x4140u);
    const __half2 r = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&t), k1152), s2);
    o[i] = *reinterpret_cast<const uint32_t*>(&r);
  }
}
// Four E4M3 weights, in k order: every one is an fp16 number. The block scales stay out of the operands (see k_grouped).
DRB_DEV void dequant4_e4m3(uint32_t w, uint32_t* o) {
  asm("{.reg .b16 lo, hi; mov.b32 {lo, hi}, %2; cvt.rn.f16x2.e4m3x2 %0, lo; cvt.rn.f16x2.e4m3x2 %1, hi;}" : "=r"(o[0]), "=r"(o[1]) : "r"(w));
}
// ---- token rows ----------------------------------------------------------------------------------------------------
// 16-bit rows -> fp16 rows in slot order at a stride of TOKEN_STRIDE bytes: routed slot s from row (row_of ? row_of[s] : s)
// of x into row (dst_row_of ? dst_row_of[s] : s) of dst, shared row r from row r of x into sh_dst; in the order of dequant8_perm
// when PERM. The down kernel's outputs serve as the buffers (they are written after the gate/up kernel has read the rows), each
// slot's row in the place of its result, so that no other row of y is touched; a row's factor sits behind its 4 KB. bf16 rows carry a wider range than fp16: a row whose largest magnitude lies outside [2^-4, 2^15) is divided
// by a power of two (the factor; the gate/up epilogue multiplies it back), every other row keeps its values.
// Only the experts' own slots are read and written: offsets may leave gaps, whose row_of says nothing and whose rows of y are the
// caller's. Every block makes the prefix sum of the counts for itself and looks a row's expert up in it.
// One warp per row; L2 traffic only (8 KB per slot, 20 MB at 300 rows: 4 us).
constexpr int PREP_THREADS = 256;
template <bool BF16, bool PERM>
__global__ void __launch_bounds__(PREP_THREADS)
    k_prep_rows(const uint4* __restrict__ x, const int* __restrict__ row_of, const int* __restrict__ offsets, const int* __restrict__ counts, int E,
                const int* __restrict__ dst_row_of, unsigned char* __restrict__ dst, int rows_sh, unsigned char* __restrict__ sh_dst) {
  __shared__ int first[MAX_E], offs[MAX_E], wtot[PREP_THREADS / 32];  // rows of the experts before e; e's first slot
  pdl_wait();
  pdl_launch_dependents();
  constexpr int PER_T = MAX_E / PREP_THREADS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int c[PER_T], sum = 0;
#pragma unroll
  for (int j = 0; j < PER_T; ++j) {
    const int e = threadIdx.x * PER_T + j;
    c[j] = sum;
    if (e < E) sum += max(__ldcg(counts + e), 0), offs[e] = __ldcg(offsets + e);
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) wtot[warp] = incl;
  __syncthreads();
  int before = incl - sum, total = 0;
#pragma unroll
  for (int w = 0; w < PREP_THREADS / 32; ++w) before += w < warp ? wtot[w] : 0, total += wtot[w];
#pragma unroll
  for (int j = 0; j < PER_T; ++j) first[threadIdx.x * PER_T + j] = before + c[j];
  __syncthreads();
  constexpr int PER = H / 8 / 32;
  for (int i = blockIdx.x * (PREP_THREADS / 32) + warp; i < total + rows_sh; i += gridDim.x * (PREP_THREADS / 32)) {
    const bool sh = i >= total;
    int row = i - total, to = row;  // the shared expert's
    if (!sh) {
      int e = 0;  // the last expert with first[e] <= i, and so the one that owns row i
#pragma unroll
      for (int step = MAX_E / 2; step > 0; step >>= 1)
        if (e + step < E && first[e + step] <= i) e += step;
      const int slot = offs[e] + (i - first[e]);
      row = row_of ? __ldcg(row_of + slot) : slot;
      to = dst_row_of ? __ldcg(dst_row_of + slot) : slot;
    }
    const uint4* p = x + (size_t)row * (H / 8);
    unsigned char* out = (sh ? sh_dst : dst) + (size_t)to * TOKEN_STRIDE;
    uint4 v[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) v[j] = __ldcg(p + j * 32 + lane);
    float inv = 1.f;
    if (BF16) {
      uint32_t m = 0u;  // bf16 with the sign bit cleared orders like an integer
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
        for (int q = 0; q < 4; ++q) m = max(m, max(w[q] & 0x7fffu, (w[q] >> 16) & 0x7fffu));
      }
      m = __reduce_max_sync(0xffffffffu, m);
      const int e = (int)(m >> 7);  // biased exponent of the largest magnitude
      float fac = 1.f;
      if (m != 0u && e < 255 && (e < 127 - 4 || e >= 127 + 15)) {
        const int ec = min(max(e, 2), 252);
        fac = __uint_as_float((uint32_t)ec << 23), inv = __uint_as_float((uint32_t)(254 - ec) << 23);
      }
      if (lane == 0) *reinterpret_cast<float*>(out + H * 2) = fac;
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      uint4 o = v[j];
      if (BF16) {
        const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
        uint32_t* op = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int q = 0; q < 4; ++q) op[q] = f2h2_sat(__uint_as_float(w[q] << 16) * inv, __uint_as_float(w[q] & 0xffff0000u) * inv);
      }
      if (PERM) o = make_uint4(prmt(o.x, o.z, 0x5410u), prmt(o.x, o.z, 0x7632u), prmt(o.y, o.w, 0x5410u), prmt(o.y, o.w, 0x7632u));
      reinterpret_cast<uint4*>(out)[j * 32 + lane] = o;
    }
  }
}

// SiLU for a result that is rounded to fp16: the division within 2 units of the last fp32 place.
DRB_DEV float silu_fast(float x) { return __fdividef(x, 1.f + expf(-x)); }

// *p = v unless at < 0.
DRB_DEV void store_valid(__half* p, uint32_t two, int at) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\t@p st.global.b32 [%0], %1;\n\t}" ::"l"(p), "r"(two), "r"(at) : "memory");
}
DRB_DEV void store_valid(float* p, float v, int at) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v), "r"(at) : "memory");
}

DRB_DEV void lds128(uint32_t addr, uint32_t* v) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}
DRB_DEV void lds64(uint32_t addr, uint32_t& a, uint32_t& b) {
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "r"(addr) : "memory");
}
DRB_DEV __half2 dup_low(uint32_t v) {
  const uint32_t r = prmt(v, 0u, 0x1010u);
  return *reinterpret_cast<const __half2*>(&r);
}
DRB_DEV __half2 dup_high(uint32_t v) {
  const uint32_t r = prmt(v, 0u, 0x3232u);
  return *reinterpret_cast<const __half2*>(&r);
}

// ---- the grouped GEMM ----------------------------------------------------------------------------------------------
// A position in a ring of N mbarriers and the parity its next completion has there, moved without a division: a convert
// warp's step is 104 instructions of conversion, and index arithmetic had grown to 60 more.
template <int N>
struct Ring {
  int i = 0;
  uint32_t par = 0;
  DRB_DEV void next(int k = 1) {  // k < N
    i += k;
    if (i >= N) i -= N, par ^= 1u;
  }
};
// Bounded wait on barrier bars[r.i]; after one that ran out no later wait of the thread spins.
template <unsigned ERR, int N>
DRB_DEV void wait_at(uint64_t* bars, const Ring<N>& r, unsigned& spent) {
  mbar_wait_ring<ERR>(smem_u32(bars) + 8 * r.i, r.par, spent);
}

// gate/up: unit (0..15) of a quadrant that the i-th lane of its half h holds. The epilogue reads sixteen lanes at a time in the layout of an
// mma.sync accumulator: thread (i, .) gets lanes i and i + 8, its unit's gate and up values for two tokens each, from either half.
// The two halves' units lie beside one another in act's order (int4: dequant8_perm's, where unit k + 4 follows unit k; FP8: k, k + 1), so a
// thread's two results for a token go out as one 32-bit store; the higher unit is in half 0 for i >= 4, which gives the eight lanes of a
// half eight different row numbers mod 8, and so their reads of the swizzled weights different banks. With gate and up rows in
// neighbouring lanes every value crossed by a shuffle and two selects, and every result was a store of its own: prefill of 300, 700 and
// 2048 rows 134.9, 180.7, 310.1 -> 134.0, 179.2, 307.4 us; nothing at 64.
template <int FMT>
DRB_DEV int epi_unit(int h, int i) {
  if (FMT == 0) return i + (h == 0 ? (i < 4 ? 0 : 8) : 4);
  return 2 * i + ((h == 1) != (i >= 4) ? 1 : 0);
}

struct Maps {
  CUtensorMap q;             // the routed experts' weights
  CUtensorMap sm;            // int4 gate/up: their (scale, min) pairs, the same view
  CUtensorMap sh;            // the shared expert's int8 weights
  CUtensorMap tok8, tok1;    // routed token rows: boxes of eight rows x four 128-byte columns / single rows for gather4
  CUtensorMap shtok8, shtok1;
};
struct Args {
  const void* scales;        // int4: (scale, min) [E, R, K/64];  FP8: f32 [E, R/128, K/128]
  const __half* shs;         // the shared expert's scales [R, K/128]
  void *dst, *sh_dst;        // gate/up: act fp16 [., I];  down: y f32 [., H]
  const int *offsets, *counts;
  const int* row_of;         // gate/up: slot -> row of the token rows (PREP = false: of x; true: of y, where they are prepared), or NULL
  const int* dst_row_of;     // down: slot -> row of dst, or NULL
  const unsigned char *fac, *sh_fac;  // prepared bf16 rows: where the factors lie (row i at i * TOKEN_STRIDE + 4096), or NULL
  float* const* peer_y;      // down, routed results only: every rank's result buffer, or NULL. dst_row_of[slot] = s * cap + j
  int peer_cap, peer_rank;   //   names the token's source rank s and its slot j there; the row is stored straight into
                             //   rank s's buffer at row rank * cap + j over NVLink
  int E, rows_sh;
};

// GEMM = 0: gate/up + SwiGLU; 1: down. FMT = 0: int4 experts; 1: block-FP8 experts.
// FP8: a tile row's weights share one f32 scale over 128 inputs. Multiplied into the fp16 operand it would cost every weight
// a rounding (measured 4.2e-4 per row against 2.1e-4); here the operands are exact, the MMAs of each 128 inputs have an
// accumulator of their own (a ring of four), and the epilogue warps sum scale * accumulator in fp32 as they complete.
// PREP (gate/up): the token rows are prepared (contiguous in slot order, or through row_of; int4: permuted); otherwise they are
// gathered through row_of in k order. The down kernel's rows are the act array, contiguous, int4: permuted by the gate/up epilogue.
template <int GEMM, int FMT, bool PREP>
__global__ void __launch_bounds__(Smem<GEMM, FMT>::THREADS, 1) k_grouped(const __grid_constant__ Maps maps, const Args a) {
  constexpr int K = GEMM == 0 ? H : I;
  constexpr int R = GEMM == 0 ? 2 * I : H;
  constexpr int MT = R / TILE_M;         // tiles per expert: 8 / 16
  constexpr int NSTEP = K / STEP_K;      // steps per item: 8 / 2
  constexpr bool PERM = FMT == 0 && PREP;
  using S = Smem<GEMM, FMT>;
  constexpr int NRAW = S::NRAW, NSM = S::NSM, SMB = S::SMB, NT = S::NT, NACC = S::NACC, B_BYTES = S::B_BYTES;
  constexpr int GROUPS = S::GROUPS, SETS = S::SETS, CONV_WARPS = S::CONV_WARPS, THREADS = S::THREADS;
  constexpr int MMA_WARP = S::MMA_WARP, LOAD_WARP = S::LOAD_WARP, TOKEN_WARP = S::TOKEN_WARP, TABLE_WARP = S::TABLE_WARP;
  constexpr int SET_ACC = NACC / SETS;  // accumulators of an epilogue set
  extern __shared__ unsigned char dyn_raw[];
  unsigned char* dyn = dyn_raw + (-smem_u32(dyn_raw) & 1023u);  // an offset, not a rounded address: loads stay shared-memory loads
  Ctl& ctl = *reinterpret_cast<Ctl*>(dyn);
  unsigned char* raw = dyn + CTL_BYTES;
  unsigned char* bring = raw + NRAW * RAW_BYTES;
  unsigned char* smbuf = bring + NST * B_BYTES;
  Tab* tabs = reinterpret_cast<Tab*>(smbuf + NSM * SMB);
  int* base = reinterpret_cast<int*>(tabs + NTAB);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NRAW; ++s) mbar_init(&ctl.rawfull[s], 1), mbar_init(&ctl.rawempty[s], GROUP_WARPS);
    for (int s = 0; s < NSM; ++s) mbar_init(&ctl.smfull[s], 1);
    for (int s = 0; s < NST; ++s) mbar_init(&ctl.full[s], GROUP_WARPS + 1), mbar_init(&ctl.done[s], 1);
    for (int s = 0; s < NACC; ++s) mbar_init(&ctl.accfull[s], 1), mbar_init(&ctl.accfree[s], EPI_WARPS);
    for (int s = 0; s < NTAB; ++s) mbar_init(&ctl.tabfull[s], 1), mbar_init(&ctl.tabempty[s], 2 + EPI_WARPS);
    mbar_fence_init();
  }
  if (warp == MMA_WARP) tmem_alloc(&ctl.tmem_base, TMEM_COLS);
  if (GEMM == 0) {
    pdl_wait();  // counts, offsets and the token rows
    pdl_launch_dependents();
  }
  // The down kernel follows the gate/up kernel, which lets its dependents start only after its own wait: counts and
  // offsets are final by now, and so the weights can be requested while the last gate/up items still run.
  // Items per set (set 0: the shared expert, set 1 + e: expert e), exclusive prefix in base[].
  const int n_sets = a.E + 1;
  {
    constexpr int PER = (MAX_E + 1 + THREADS - 1) / THREADS;
    int it[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int s = threadIdx.x * PER + j;
      const int cnt = s >= n_sets ? 0 : s == 0 ? a.rows_sh : __ldcg(a.counts + s - 1);
      it[j] = sum, sum += ((cnt + NT - 1) / NT) * MT;
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) ctl.wtot[warp] = incl;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    int before = incl - sum;
    for (int w = 0; w < warp; ++w) before += ctl.wtot[w];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int s = threadIdx.x * PER + j;
      if (s <= n_sets) base[s] = before + it[j];  // base[n_sets]: the total
    }
    __syncthreads();
  }
  const uint32_t tmem = ctl.tmem_base;
  const int total_items = base[n_sets];

  struct Item {
    bool shared;
    int e, mt, n0;
  };
  int cur = 0;  // the item's set: items come in ascending order, so the search goes on where it stood (whole warps)
  auto decode = [&](int item) {
    for (;;) {
      const int s = cur + 1 + lane;
      const int n = __popc(__ballot_sync(0xffffffffu, s < n_sets && base[s] <= item));
      cur += n;
      if (n < 32) break;
    }
    Item it;
    it.shared = FMT == 0 && cur == 0;
    it.e = cur - 1;
    const int local = item - base[cur];
    it.mt = local % MT;
    it.n0 = (local / MT) * NT;
    return it;
  };
  // weight row of tile row r: a gate/up tile is 64 gate rows and their 64 up rows
  auto weight_row = [&](int mt, int r) { return GEMM == 0 ? (r >> 6) * I + mt * (TILE_M / 2) + (r & 63) : mt * TILE_M + r; };

  unsigned spent = 0;  // see mbar_wait_ring

  if (warp < CONV_WARPS) {
    // ================= convert warps =================
    // The groups of eight take turns at the steps; within a group, warp (half h, lane quarter q4) converts
    // inputs [128 h, +128) of the step's 256 for its 32 rows. The waits and arrivals of a step cost a warp as many instructions as
    // 64 inputs of conversion do, so a thread takes 128 of every other step and not 64 of each (it measured 243 instructions
    // per 64 inputs before, 104 of them conversion).
    const int q4 = warp & 3, half = (warp >> 2) & 1, group = warp >> 3;
    // This thread's tile row; it fills tensor-memory lane 32 q4 + lane. gate/up: lanes 0..7 and 16..23 take gate rows, the eight
    // behind each the same units' up rows: see epi_unit.
    const int r = GEMM == 0 ? ((lane >> 3) & 1) * 64 + q4 * 16 + epi_unit<FMT>(lane >> 4, lane & 7) : q4 * 32 + lane;
    const NibbleConst nc;
    const uint32_t acol = tmem + ((uint32_t)(q4 * 32) << 16) + A_COL0 + half * 64;
    const unsigned char* xrow = raw + swz_off(r, 0);  // piece p of the row stands at xrow + piece(p)
    auto piece = [&](int p) { return (((r & 7) ^ p) - (r & 7)) << 4; };
    const uint32_t x_row = smem_u32(raw) + swz_off(r, 4 * half);  // int4: this thread's first piece
    Ring<NRAW> rr;     // raw stages
    Ring<NST> ra;      // stages; every one starts free
    ra.par = 1;
    ra.next(group);
    auto a_wait = [&]() {  // the MMAs that read this stage's tiles must have completed
      wait_at<DRB_ERR_TMEM>(ctl.done, ra, spent);
      tc_fence_after();
    };
    auto a_done = [&]() {
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.full[ra.i]);
      ra.next(GROUPS);
    };
    Ring<(NSM ? NSM : 1)> rs;  // int4 items' scales
    for (int item = blockIdx.x; item < total_items; item += gridDim.x) {
      const Item it = decode(item);
      if (FMT == 0 && !it.shared) {
        wait_at<DRB_ERR_FULL_WAIT>(ctl.smfull, rs, spent);
        // (scale, min) of this row's groups 4 step + 2 half, + 1: gate/up: piece `step` of a swizzled row; down: 16 bytes a step
        const uint32_t sm_a = smem_u32(smbuf) + rs.i * SMB + (GEMM == 0 ? swz_off(r, 0) : r * 32) + 8 * half;
        rs.next();
        rr.next(group);
#pragma unroll 1
        for (int step = group; step < NSTEP; step += GROUPS) {
          uint32_t sm[2];
          lds64(GEMM == 0 ? sm_a ^ (step << 4) : sm_a + 16 * step, sm[0], sm[1]);
          a_wait();  // ahead of the raw stage: see the loader
          wait_at<DRB_ERR_FULL_WAIT>(ctl.rawfull, rr, spent);
          const bool small = __all_sync(0xffffffffu, max(sm[0] & 0x7fffu, sm[1] & 0x7fffu) < 0x2C00u);  // both scales below 2^-4
          // piece 4 half + j of the row stands at xa ^ 16 j: in the swizzled row the piece's number is xor-ed into the address
          uint32_t xa = x_row + rr.i * RAW_BYTES;
          uint32_t to = acol + ra.i * A_COLS;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint32_t w[8];
            lds128(xa, w), lds128(xa ^ 16u, w + 4);
            xa ^= 32u;
            const __half2 s2 = dup_low(sm[0]), m2 = dup_high(sm[0]);
            sm[0] = sm[1];
            uint32_t o[32];
            if (!PERM && GEMM == 0) {
#pragma unroll
              for (int j = 0; j < 8; ++j) dequant8_nat(w[j], s2, m2, nc, o + 4 * j);
              tmem_st32(to, o);
            } else if (small) {
              const __half2 k1024 = *reinterpret_cast<const __half2*>(&nc.k1024);
              const __half2 big = __hmul2(__hmul2(s2, k1024), k1024);
#pragma unroll
              for (int j = 0; j < 8; ++j) dequant8_perm<true>(w[j], s2, m2, big, nc, o + 4 * j);
              tmem_st32(to, o);
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j) dequant8_perm<false>(w[j], s2, m2, s2, nc, o + 4 * j);
              tmem_st32(to, o);
            }
            to += 32;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl.rawempty[rr.i]);
          rr.next(step + GROUPS < NSTEP ? GROUPS : GROUPS - group);
          a_done();
        }
      } else {  // 8-bit weights: a step is two raw stages, one per half
        const int wrow = weight_row(it.mt, r);
        const __half* ssrow = a.shs + (size_t)wrow * (K / 128) + half;
        __half s_next = __half();  // shared expert: one scale per 128 inputs, fetched a step ahead
        if (FMT == 0) s_next = __ldg(ssrow + 2 * group);
        rr.next(2 * group);
#pragma unroll 1
        for (int step = group; step < NSTEP; step += GROUPS) {
          const __half2 s2 = __half2half2(s_next);
          if (FMT == 0 && step + GROUPS < NSTEP) s_next = __ldg(ssrow + 2 * (step + GROUPS));
          // both stages are waited for although this warp reads one: an arrival must not run a ring's length ahead
          if (GROUPS > 1) a_wait();  // ahead of the raw stages: see the loader
          const int sa = rr.i;
          wait_at<DRB_ERR_FULL_WAIT>(ctl.rawfull, rr, spent);
          rr.next();
          const int sb = rr.i;
          wait_at<DRB_ERR_FULL_WAIT>(ctl.rawfull, rr, spent);
          rr.next(2 * (step + GROUPS < NSTEP ? GROUPS : GROUPS - group) - 1);
          const unsigned char* xp = xrow + (half ? sb : sa) * RAW_BYTES;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint32_t o[32];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 x = *reinterpret_cast<const uint4*>(xp + piece(4 * g + j));
              const uint32_t w[4] = {x.x, x.y, x.z, x.w};
              if (FMT == 1) {
#pragma unroll
                for (int q = 0; q < 4; ++q) dequant4_e4m3(w[q], o + 8 * j + 2 * q);
              } else {
#pragma unroll
                for (int q = 0; q < 2; ++q) dequant8_i8<FMT == 0 && (PREP || GEMM == 1)>(w[2 * q], w[2 * q + 1], s2, o + 8 * j + 4 * q);
              }
            }
            if (GROUPS == 1 && g == 0) a_wait();  // one group: the first conversion needs no tensor memory yet
            tmem_st32(acol + ra.i * A_COLS + g * 32, o);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl.rawempty[sa]), mbar_arrive(&ctl.rawempty[sb]);
          a_done();
        }
      }
    }
  } else if (warp == MMA_WARP) {
    // ================= MMA warp =================
    Ring<NTAB> rt;
    Ring<SET_ACC> rc;  // FP8: an item takes an even number of turns of its set's two accumulators, so the next item finds it as it was
    Ring<NST> ra;
    rc.par = 1;  // the accumulators start free
    unsigned steps = 0;
    int acc0 = 0;  // the item's first accumulator: 0, FP8: of the set whose turn it is
    static_assert(FMT == 0 || (K / 128 / SET_ACC) % 2 == 0, "even turns");
    const uint64_t bdesc0 = smem_desc(bring, 4096);  // eight-row groups lie 4 KB apart: four 1 KB columns each
    for (int item = blockIdx.x; item < total_items; item += gridDim.x) {
      wait_at<DRB_ERR_FULL_WAIT>(ctl.tabfull, rt, spent);
      const uint32_t idesc = instr_desc_f16(tabs[rt.i].cols), d = tmem + (uint32_t)((acc0 + rc.i) * NT);
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.tabempty[rt.i]);
      rt.next();
      if (FMT == 0) wait_at<DRB_ERR_TMEM>(ctl.accfree, rc, spent);
#pragma unroll 1
      for (int step = 0; step < NSTEP; ++step) {
        wait_at<DRB_ERR_TMEM>(ctl.full, ra, spent);
        if (FMT == 0) {
          tc_fence_after();
          if (elect_one()) {
            const uint32_t ac = tmem + A_COL0 + ra.i * A_COLS;
            const uint64_t bd = bdesc0 + (uint32_t)(ra.i * (B_BYTES >> 4));
            mma_f16_ts(d, ac, bd, idesc, step > 0);
#pragma unroll
            for (int k16 = 1; k16 < STEP_K / 16; ++k16) mma_f16_ts(d, ac + 8 * k16, bd + (uint64_t)((k16 >> 2) * 64 + (k16 & 3) * 2), idesc, true);
            mma_commit(&ctl.done[ra.i]);
            if (step == NSTEP - 1) mma_commit(&ctl.accfull[rc.i]);
          }
        } else {
#pragma unroll
          for (int kb = 0; kb < 2; ++kb) {
            wait_at<DRB_ERR_TMEM>(ctl.accfree + acc0, rc, spent);
            tc_fence_after();
            if (elect_one()) {
              const uint32_t ac = tmem + A_COL0 + ra.i * A_COLS, dk = tmem + (uint32_t)((acc0 + rc.i) * NT);
              const uint64_t bd = bdesc0 + (uint32_t)(ra.i * (B_BYTES >> 4));
#pragma unroll
              for (int k16 = 8 * kb; k16 < 8 * kb + 8; ++k16)
                mma_f16_ts(dk, ac + 8 * k16, bd + (uint64_t)((k16 >> 2) * 64 + (k16 & 3) * 2), idesc, k16 > 8 * kb);
              mma_commit(&ctl.accfull[acc0 + rc.i]);
              if (kb == 1) mma_commit(&ctl.done[ra.i]);
            }
            __syncwarp();
            rc.next();
          }
        }
        __syncwarp();
        ra.next();
      }
      if (FMT == 0) rc.next();
      if (SETS > 1) acc0 ^= SET_ACC;
      steps += NSTEP;
    }
    // The block must not end before the completion arrivals it is owed have landed: the last one of every stage.
    for (unsigned k = 0; k < NST && k < steps; ++k) {
      const unsigned n = steps - 1 - k;
      mbar_wait_ring<DRB_ERR_TMEM>(smem_u32(&ctl.done[n % NST]), (n / NST) & 1, spent);
    }
  } else if (warp == LOAD_WARP) {
    // ================= loader =================
    // The (scale, min) pairs of an int4 item go to one of NSM slots. They are requested while the item before still asks for its stages: with
    // the item's own first stage they came half a thousand cycles after the convert warps (300 rows 134.4 -> 132.8 us, 2048 rows 312.2 ->
    // 306.6). Behind request SM_AT of that item the raw stage NRAW requests back has been read, so every item more than NSM - 1
    // items back is finished with its slot.
    constexpr int SM_AT = NSTEP == 8 ? NRAW - 1 : 1;
    static_assert(NSM == 0 || (NSM - 2) * NSTEP + SM_AT + 1 >= NRAW, "scale slots");
    // A wait for a raw stage tests one bit of its phase, so it tells "landed" from "in flight" only once the stage's use before
    // this one is known to have landed; boxes land in any order. A group's own uses it has waited for itself. With two groups a
    // stage also passes from one to the other, and there the stage's MMAs vouch: after a_wait() of step s everything up to step s - NST
    // has been converted. A step takes one raw stage or two, so the use NRAW requests back lies at least NRAW / 2 steps back: NST or more,
    // or two, which is the group's own. Hence NRAW, and a_wait() in front of the raw stages in either branch.
    static_assert(GROUPS == 1 || (GROUPS == 2 && NST == 3 && NRAW >= 5), "raw stages");
    Ring<NRAW> rr;
    Ring<(NSM ? NSM : 1)> rs;
    rr.par = 1;  // every raw stage starts free
    auto scales = [&](const Item& it) {  // one thread
      unsigned char* sp = smbuf + rs.i * SMB;
      mbar_expect_tx(&ctl.smfull[rs.i], SMB);
      if (GEMM == 0) tma_load_4d(sp, &maps.sm, 0, it.mt * (TILE_M / 2), 0, it.e, &ctl.smfull[rs.i]);
      else bulk_g2s(sp, static_cast<const unsigned char*>(a.scales) + (size_t)(it.e * R + it.mt * TILE_M) * (K / 64) * 4, SMB, &ctl.smfull[rs.i]);
    };
    Item next = {};
    if ((int)blockIdx.x < total_items) next = decode(blockIdx.x);
    if (FMT == 0 && (int)blockIdx.x < total_items && !next.shared) {
      if (elect_one()) scales(next);
      __syncwarp();
      rs.next();
    }
    for (int item = blockIdx.x; item < total_items; item += gridDim.x) {
      const Item it = next;
      const bool eight = FMT == 1 || it.shared, more = item + (int)gridDim.x < total_items;
      const int nraw = NSTEP * (eight ? 2 : 1), unit0 = it.mt * (TILE_M / 2), e = it.shared ? 0 : it.e, row0 = e * R + it.mt * TILE_M;
      const CUtensorMap* map = it.shared ? &maps.sh : &maps.q;
#pragma unroll 1
      for (int n = 0; n < nraw; ++n) {
        wait_at<DRB_ERR_EMPTY_WAIT>(ctl.rawempty, rr, spent);
        __syncwarp();
        if (elect_one()) {
          uint64_t* bar = &ctl.rawfull[rr.i];
          mbar_expect_tx(bar, RAW_BYTES);
          if (GEMM == 0) tma_load_4d(raw + (size_t)rr.i * RAW_BYTES, map, n * ROW_BYTES, unit0, 0, e, bar);
          else tma_load_2d(raw + (size_t)rr.i * RAW_BYTES, map, n * ROW_BYTES, row0, bar);
        }
        __syncwarp();
        rr.next();
        if (n == SM_AT) {
          if (more) next = decode(item + gridDim.x);
          if (FMT == 0 && more && !next.shared) {
            if (elect_one()) scales(next);
            __syncwarp();
            rs.next();
          }
        }
      }
    }
  } else if (warp == TOKEN_WARP) {
    // ================= token warp =================
    if (GEMM == 1) pdl_wait();  // the gate/up kernel's activations
    Ring<NTAB> rt;
    Ring<NST> ra;
    ra.par = 1;  // every stage starts free
    for (int item = blockIdx.x; item < total_items; item += gridDim.x) {
      wait_at<DRB_ERR_FULL_WAIT>(ctl.tabfull, rt, spent);
      const Tab& tab = tabs[rt.i];
      const int srow = tab.srow, full = tab.full, start = tab.start, quads = tab.quads;
      const unsigned bytes = (full + (start >= 0)) * 4096 + quads * 2048;
      const CUtensorMap *m8 = tab.shared ? &maps.shtok8 : &maps.tok8, *m1 = tab.shared ? &maps.shtok1 : &maps.tok1;
#pragma unroll 1
      for (int step = 0; step < NSTEP; ++step) {
        wait_at<DRB_ERR_EMPTY_WAIT>(ctl.done, ra, spent);
        __syncwarp();
        if (elect_one()) {
          unsigned char* bp = bring + ra.i * B_BYTES;
          uint64_t* bar = &ctl.full[ra.i];
          mbar_expect_tx(bar, bytes);
          if (start >= 0) tma_load_3d(bp + full * 4096, m8, 0, start, step * 4, bar);
#pragma unroll 1
          for (int g = 0; g < full; ++g) tma_load_3d(bp + g * 4096, m8, 0, srow + 8 * g, step * 4, bar);
#pragma unroll 1
          for (int q = 0; q < quads; ++q) {
            const int4 row = *reinterpret_cast<const int4*>(&tab.rows[4 * q]);
            unsigned char* qp = bp + (full + (q >> 1)) * 4096 + (q & 1) * 512;
#pragma unroll
            for (int c = 0; c < 4; ++c) tma_gather4(qp + c * 1024, m1, step * STEP_K + c * 64, row.x, row.y, row.z, row.w, bar);
          }
        }
        __syncwarp();
        ra.next();
      }
      if (lane == 0) mbar_arrive(&ctl.tabempty[rt.i]);
      rt.next();
    }
  } else if (warp == TABLE_WARP) {
    // ================= table warp =================
    Ring<NTAB> rt;
    rt.par = 1;
    for (int item = blockIdx.x; item < total_items; item += gridDim.x) {
      const Item it = decode(item);
      wait_at<DRB_ERR_EMPTY_WAIT>(ctl.tabempty, rt, spent);
      Tab& tab = tabs[rt.i];
      const int cnt = it.shared ? a.rows_sh : __ldcg(a.counts + it.e);
      const int nt = min(NT, cnt - it.n0);
      const int srow = (it.shared ? 0 : __ldcg(a.offsets + it.e)) + it.n0, end = srow + nt, rest = nt & 7;
      // Contiguous rows go by boxes of eight. What is left over takes one more box, of the last eight rows: no row beyond
      // the item's end is touched, and the columns of rows that it repeats (or that are not the item's) have no result
      // row. Among the array's first eight rows, and for scattered rows, gather4 fetches the rows by number.
      const bool contig = GEMM == 1 || it.shared || (PREP && !a.row_of);
      const int full = contig ? nt >> 3 : 0;
      const int start = contig && rest && end >= 8 ? end - 8 : -1;
      const int quads = start < 0 ? (nt - 8 * full + 3) >> 2 : 0;
      const int cols = ((start >= 0 ? 8 * full + 8 : nt) + 15) & ~15;
      const unsigned char* fac = it.shared ? a.sh_fac : a.fac;
      for (int t = lane; t < cols; t += 32) {
        const int slot = start >= 0 && t >= 8 * full ? start + (t - 8 * full) : srow + t;
        const bool own = slot >= srow + (t >= 8 * full ? 8 * full : 0) && slot < end;
        if (GEMM == 0) {
          float f = 1.f;
          if (own && fac) f = __ldcg(reinterpret_cast<const float*>(fac + (size_t)(a.row_of && !it.shared ? __ldcg(a.row_of + slot) : slot) * TOKEN_STRIDE + H * 2));
          tab.fac[t] = f;
        }
        tab.dst[t] = !own ? -1 : (GEMM == 1 && !it.shared && a.dst_row_of) ? __ldcg(a.dst_row_of + slot) : slot;
      }
      for (int t = lane; t < 4 * quads; t += 32) {
        const int slot = srow + min(8 * full + t, nt - 1);
        tab.rows[t] = (GEMM == 0 && !it.shared && a.row_of) ? __ldcg(a.row_of + slot) : slot;
      }
      if (lane == 0) tab.cols = cols, tab.used = (start >= 0 ? 8 * full + 8 : nt + 7) & ~7, tab.mt = it.mt, tab.shared = it.shared, tab.full = full, tab.srow = srow, tab.start = start, tab.quads = quads;
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.tabfull[rt.i]);
      rt.next();
    }
  } else {
    // ================= epilogue warps =================
    if (GEMM == 1) pdl_wait();  // y may still be read as the gate/up kernel's token rows
    const int q4 = warp & 3, set = SETS > 1 ? (warp - CONV_WARPS) / EPI_WARPS : 0;
    const int acc0 = set * SET_ACC;
    const uint32_t quadrant = tmem + ((uint32_t)(q4 * 32) << 16);
    Ring<NTAB> rt;
    Ring<SET_ACC> rc;
    if (SETS > 1) rt.next(set);  // a table slot serves one set only: NTAB is a multiple of SETS
    for (int item = blockIdx.x + set * gridDim.x; item < total_items; item += SETS * gridDim.x) {
      wait_at<DRB_ERR_FULL_WAIT>(ctl.tabfull, rt, spent);
      const Tab& tab = tabs[rt.i];
      const int cols = FMT == 1 ? tab.cols : tab.used, mt = tab.mt;
      const bool sh = tab.shared != 0, peers = GEMM == 1 && a.peer_y && !sh;
      // gate/up: the place in act of this thread's two units (see epi_unit). down: the column of y of this thread's row.
      const int i8 = lane >> 2;
      __half* const act = static_cast<__half*>(sh ? a.sh_dst : a.dst) + mt * (TILE_M / 2) + q4 * 16 + (FMT == 0 ? 8 * (i8 >> 2) + 2 * (i8 & 3) : 2 * i8);
      float* const y = static_cast<float*>(sh ? a.sh_dst : a.dst) + mt * TILE_M + q4 * 32 + lane;
      const bool swap = lane & 16;  // half 1 holds the lower unit
      // The results of eight columns. The stores carry their own predicate: behind a branch on it the arithmetic of one column
      // waited for the store of the one before (gate/up, 64 columns: 7000 cycles per item).
      auto units = [&](int c0, const uint32_t* h0, const uint32_t* h1) {  // gate/up: tokens 2 (lane % 4) and the next
        const int2 d2 = *reinterpret_cast<const int2*>(&tab.dst[c0 + 2 * (lane & 3)]);
        const float2 f2 = *reinterpret_cast<const float2*>(&tab.fac[c0 + 2 * (lane & 3)]);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const float f = t ? f2.y : f2.x;
          auto unit = [&](const uint32_t* h) { return silu_fast(__uint_as_float(h[t]) * f) * (__uint_as_float(h[2 + t]) * f); };
          const float r0 = unit(h0), r1 = unit(h1);
          const int dt = t ? d2.y : d2.x;
          store_valid(act + (ptrdiff_t)dt * I, f2h2_sat(swap ? r1 : r0, swap ? r0 : r1), dt);
        }
      };
      auto columns = [&](int c0, const uint32_t(&v)[8]) {  // down
#pragma unroll
        for (int i4 = 0; i4 < 8; i4 += 4) {
          const int4 d4 = *reinterpret_cast<const int4*>(&tab.dst[c0 + i4]);
          const int dst[4] = {d4.x, d4.y, d4.z, d4.w};
          if (peers) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (dst[i] < 0) continue;
              const int s = dst[i] / a.peer_cap;
              a.peer_y[s][((size_t)a.peer_rank * a.peer_cap + (dst[i] - s * a.peer_cap)) * H + mt * TILE_M + q4 * 32 + lane] = __uint_as_float(v[i4 + i]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) store_valid(y + (ptrdiff_t)dst[i] * H, __uint_as_float(v[i4 + i]), dst[i]);
          }
        }
      };
      if (FMT == 1) {
        // FP8: the columns' sums over the accumulators; gate/up: [column block of 16][as tmem_ld_halves16]
        float sum[FMT == 1 ? NT : 1];
        // Lane l holds a scale: gate/up: input block l % 16 of the gate rows' (l < 16) or the up rows' block row; down: l % 4.
        const Item it = decode(item);
        const float* se = static_cast<const float*>(a.scales) + (size_t)it.e * (R / 128) * (K / 128);
        const float sv = __ldg(se + (weight_row(mt, GEMM == 0 ? 64 * (lane >> 4) : 0) >> 7) * (K / 128) + lane % (K / 128));
#pragma unroll
        for (int c = 0; c < NT; ++c) sum[c] = 0.f;
#pragma unroll 1
        for (int kb = 0; kb < K / 128; ++kb) {
          const float s = __shfl_sync(0xffffffffu, sv, kb), su = GEMM == 0 ? __shfl_sync(0xffffffffu, sv, kb + 16) : s;
          wait_at<DRB_ERR_TMEM>(ctl.accfull + acc0, rc, spent);
          tc_fence_after();
#pragma unroll
          for (int c0 = 0; c0 < NT; c0 += 16)
            if (c0 < cols) {
              const uint32_t acc = quadrant + (uint32_t)((acc0 + rc.i) * NT + c0);
              uint32_t v[16];
              if (GEMM == 0) tmem_ld_halves16(acc, reinterpret_cast<uint32_t(&)[2][8]>(v));
              else tmem_ld16(acc, v);
#pragma unroll
              for (int i = 0; i < 16; ++i) sum[c0 + i] = fmaf(i & 2 ? su : s, __uint_as_float(v[i]), sum[c0 + i]);
            }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl.accfree[acc0 + rc.i]);
          rc.next();
        }
#pragma unroll
        for (int c0 = 0; c0 < NT; c0 += 8)
          if (c0 < cols) {
            uint32_t v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              // down: columns in order; gate/up: the four of half 0, then the four of half 1
              const int at = GEMM == 1 ? c0 + i : (c0 & ~15) + 8 * (i >> 2) + ((c0 >> 1) & 4) + (i & 3);
              v[i] = __float_as_uint(sum[FMT == 1 ? at : 0]);
            }
            if (GEMM == 0) units(c0, v, v + 4);
            else columns(c0, v);
          }
      } else {
        wait_at<DRB_ERR_TMEM>(ctl.accfull, rc, spent);
        tc_fence_after();
        const uint32_t acc = quadrant + (uint32_t)(rc.i * NT);
#pragma unroll 1
        for (int c0 = 0; c0 < cols; c0 += 16) {
          uint32_t v[2][8];
          if (GEMM == 0) tmem_ld_halves16(acc + (uint32_t)c0, v);
          else tmem_ld16(acc + (uint32_t)c0, v);
          if (c0 + 16 >= cols) {  // everything is in registers: the accumulator is free
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl.accfree[rc.i]);
          }
          if (GEMM == 0) units(c0, v[0], v[1]);
          else columns(c0, v[0]);
          if (c0 + 8 < cols) {
            if (GEMM == 0) units(c0 + 8, v[0] + 4, v[1] + 4);
            else columns(c0 + 8, v[1]);
          }
        }
        rc.next();
      }
      if (peers) __threadfence_system();  // before the flag that a later kernel writes to the peers
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.tabempty[rt.i]);
      rt.next(SETS);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == MMA_WARP) tmem_dealloc(tmem, TMEM_COLS);
}

// ---- host side ---------------------------------------------------------------------------------------------------
// Tensor maps with the 128-byte swizzle. cuTensorMapEncodeTiled is a driver entry point: it is looked up through the
// runtime once, so the library has no link-time dependency on the driver. The map functions return 0 or -3.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn g_encode = nullptr;

static cudaError_t resolve_encode() {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult status;
  cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &status);
  if (e != cudaSuccess) return e;
  if (status != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
  g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  return cudaSuccess;
}

static int encode(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* p, const cuuint64_t* dims, const cuuint64_t* strides,
                  const cuuint32_t* box) {
  if (!g_encode) return -3;
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return g_encode(map, type, rank, const_cast<void*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? 0
             : -3;
}

// Down projection: [rows, row_bytes] row-major, boxes of 128 rows x 128 bytes.
static int map_rows(CUtensorMap* map, const void* p, uint64_t rows, uint64_t row_bytes) {
  const cuuint64_t dims[2] = {row_bytes, rows}, strides[1] = {row_bytes};
  const cuuint32_t box[2] = {ROW_BYTES, TILE_M};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, p, dims, strides, box);
}

// Gate/up: [experts][2 (gate | up)][units][row_bytes] seen as (row byte, unit, gate|up, expert); a box is 128 bytes of
// 64 units' gate rows and then of their up rows.
static int map_gate_up(CUtensorMap* map, const void* p, uint64_t experts, uint64_t units, uint64_t row_bytes) {
  const cuuint64_t dims[4] = {row_bytes, units, 2, experts}, strides[3] = {row_bytes, units * row_bytes, 2 * units * row_bytes};
  const cuuint32_t box[4] = {ROW_BYTES, TILE_M / 2, 2, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, p, dims, strides, box);
}

// fp16 token rows of k inputs at a stride of stride bytes. How many there are is known on the device only; the kernel asks
// for rows that exist, and the maps' row extent is not a limit.
static int map_tokens(CUtensorMap* m8, CUtensorMap* m1, const void* p, uint64_t k, uint64_t stride) {
  const cuuint64_t rows = 1ull << 28;
  const cuuint64_t dims3[3] = {64, rows, k / 64}, strides3[2] = {stride, 128};
  const cuuint32_t box3[3] = {64, 8, STEP_K / 64};
  const cuuint64_t dims2[2] = {k, rows}, strides2[1] = {stride};
  const cuuint32_t box2[2] = {64, 1};
  if (encode(m8, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, p, dims3, strides3, box3)) return -3;
  return encode(m1, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p, dims2, strides2, box2);
}

// One grouped expert block: gate/up, then down.
struct Block {
  int fmt;                                  // 0: int4, 1: block FP8
  const void *gu_w, *gu_s, *d_w, *d_s;      // routed experts
  const void *sgu_q, *sgu_s, *sd_q, *sd_s;  // shared expert (rows_sh > 0)
  const void* x;                            // 16-bit rows [., H]
  bool x_bf16;
  bool prepared;                            // y and sh_out hold the prepared rows already (x is not used)
  const int *row_of, *offsets, *counts, *y_row_of;
  void *act, *y, *sh_act, *sh_out;
  int rows_sh, E;
  float* const* peer_y;
  int peer_cap, peer_rank;
};

template <int FMT>
static int run_block(const Block& b, const DrbDevice& dev, cudaStream_t st) {
  constexpr int WB = FMT == 0 ? 2 : 1;  // weights per byte
  // Rows are prepared wherever there is a buffer for them: y and sh_out, which are written last. With the results going to
  // peers y is not this call's to write: the fp16 rows are gathered as they are.
  const bool prep = b.peer_y == nullptr;
  if (!prep && (b.x_bf16 || FMT != 0)) return -1;
  // Results are stored float by float, so y and sh_out may start at any float. Prepared rows start at the next 16-byte boundary: the
  // 4 KB and the factor fill half of a row's stride, so the last one still ends inside the buffer.
  auto align16 = [](void* p) { return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15); };
  unsigned char* tok = align16(b.y);
  unsigned char* shtok = align16(b.sh_out);
  // What the kernels read in 16-byte pieces, before anything is launched.
  auto odd = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  if ((!b.prepared && odd(b.x)) || (b.E > 0 && (odd(b.gu_w) || odd(b.d_w) || odd(b.act) || (FMT == 0 && (odd(b.gu_s) || odd(b.d_s))))) ||
      (b.rows_sh > 0 && (odd(b.sgu_q) || odd(b.sd_q) || odd(b.sh_act))))
    return -3;
  if (prep && !b.prepared) {
    // Both the preparing launch and the gate/up launch behind it wait for their predecessor themselves, ahead of the first read, and so
    // may start under it: 20 rows over FP8 experts 54.8 -> 50.4 us, 300 rows 137.0 -> 132.7.
    auto kp = b.x_bf16 ? k_prep_rows<true, FMT == 0> : k_prep_rows<false, FMT == 0>;
    for (int e0 = 0; e0 == 0 || e0 < b.E; e0 += MAX_E)  // the shared expert's rows with the first experts
      drb_launch(kp, dim3(2 * dev.sms), dim3(PREP_THREADS), 0, st, dev.pdl, static_cast<const uint4*>(b.x), b.row_of, b.offsets + e0, b.counts + e0,
                 b.E - e0 < MAX_E ? b.E - e0 : MAX_E, b.y_row_of, tok, e0 == 0 ? b.rows_sh : 0, shtok);
  }
  // Every gate/up launch before the first down launch: y holds the token rows until then.
  const bool sh_on = b.rows_sh > 0;
  for (int gemm = 0; gemm < 2; ++gemm) {
    for (int e0 = 0; e0 == 0 || e0 < b.E; e0 += MAX_E) {
      const int ne = b.E - e0 < MAX_E ? b.E - e0 : MAX_E;
      const bool sh = sh_on && e0 == 0;
      const size_t row = (gemm == 0 ? H : I) / WB, rows = gemm == 0 ? 2 * I : H, cols = gemm == 0 ? H : I;
      const size_t s_bytes = FMT == 0 ? rows * (cols / 64) * 4 : (rows / 128) * (cols / 128) * 4;  // scales per expert
      const unsigned char* w = static_cast<const unsigned char*>(gemm == 0 ? b.gu_w : b.d_w) + rows * row * e0;
      const unsigned char* sc = static_cast<const unsigned char*>(gemm == 0 ? b.gu_s : b.d_s) + s_bytes * e0;
      Maps m = {};
      Args a = {};
      if (gemm == 0) {
        if (ne > 0 && (map_gate_up(&m.q, w, ne, I, row) || (FMT == 0 && map_gate_up(&m.sm, sc, ne, I, (H / 64) * 4)))) return -3;
        if (ne > 0 && map_tokens(&m.tok8, &m.tok1, prep ? tok : b.x, H, prep ? TOKEN_STRIDE : H * 2)) return -3;
        if (sh && map_gate_up(&m.sh, b.sgu_q, 1, I, H)) return -3;
        if (sh && map_tokens(&m.shtok8, &m.shtok1, prep ? shtok : b.x, H, prep ? TOKEN_STRIDE : H * 2)) return -3;
        a.dst = b.act, a.sh_dst = b.sh_act, a.row_of = prep ? b.y_row_of : b.row_of;
        if (prep && b.x_bf16) a.fac = tok, a.sh_fac = shtok;
      } else {
        if (ne > 0 && (map_rows(&m.q, w, (uint64_t)ne * H, row) || map_tokens(&m.tok8, &m.tok1, b.act, I, I * 2))) return -3;
        if (sh && (map_rows(&m.sh, b.sd_q, H, I) || map_tokens(&m.shtok8, &m.shtok1, b.sh_act, I, I * 2))) return -3;
        a.dst = b.y, a.sh_dst = b.sh_out, a.dst_row_of = b.y_row_of;
        a.peer_y = b.peer_y, a.peer_cap = b.peer_cap, a.peer_rank = b.peer_rank;
      }
      a.scales = sc, a.shs = static_cast<const __half*>(gemm == 0 ? b.sgu_s : b.sd_s);
      a.offsets = b.offsets + e0, a.counts = b.counts + e0, a.E = ne > 0 ? ne : 0, a.rows_sh = sh ? b.rows_sh : 0;
      if (gemm == 0)
        drb_launch(prep ? k_grouped<0, FMT, true> : k_grouped<0, FMT, FMT != 0>, dim3(dev.sms), dim3(Smem<0, FMT>::THREADS), Smem<0, FMT>::BYTES, st, dev.pdl && prep && b.E <= MAX_E, m, a);
      else  // only the first one follows the gate/up kernel
        drb_launch(k_grouped<1, FMT, true>, dim3(dev.sms), dim3(Smem<1, FMT>::THREADS), Smem<1, FMT>::BYTES, st, dev.pdl && b.E <= MAX_E, m, a);
    }
  }
  return 0;
}

template <typename Kn>
static cudaError_t configure_one(Kn kernel, size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return e != cudaSuccess ? e : drb_carveout(kernel);
}

static cudaError_t configure_all() {
  cudaError_t e;
  if ((e = resolve_encode()) != cudaSuccess) return e;
  if ((e = drb_carveout(k_prep_rows<false, false>)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_prep_rows<false, true>)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_prep_rows<true, false>)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_prep_rows<true, true>)) != cudaSuccess) return e;
  if ((e = configure_one(k_grouped<0, 0, true>, Smem<0, 0>::BYTES)) != cudaSuccess) return e;
  if ((e = configure_one(k_grouped<0, 0, false>, Smem<0, 0>::BYTES)) != cudaSuccess) return e;
  if ((e = configure_one(k_grouped<1, 0, true>, Smem<1, 0>::BYTES)) != cudaSuccess) return e;
  if ((e = configure_one(k_grouped<0, 1, true>, Smem<0, 1>::BYTES)) != cudaSuccess) return e;
  return configure_one(k_grouped<1, 1, true>, Smem<1, 1>::BYTES);
}

}  // namespace pft
