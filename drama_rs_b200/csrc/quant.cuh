// Checkpoint quantisers on the GPU: the reference's converter (tools/convert.py) turns bf16/fp8 expert weights
// into the int4 / int8 layouts the kernels stream. These two kernels restate its per-group procedures operation by
// operation in IEEE fp32 (no fused multiply-add, round-to-nearest division, fp16 rounding of scale and min), so that
// codes and scales come out as the reference writes them. That includes the ORDER of the 64-term sums that decide
// between two clipping candidates: eight running sums over the inputs 8 i + j (i ascending), then
// ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7)): the order of the CPU restatement of the converter, which
// reproduces the converter's own output on the committed fixture bit for bit. (The converter's sums are a library's
// vectorised reduction whose exact order depends on the host's vector width; where two candidates' errors agree to
// the last bit, its pick is not defined by its source.)
//
//   drb_quant_q4: tools/convert.py:44-89 (`quant_q4_groups`: 24-step clipping search, least-squares refit) and
//                 92-101 (`quant_q4`: packing, low nibble = even k). Eight lanes per group of 64 inputs.
//   drb_quant_q8: tools/convert.py:33-41 (`quant_q8`). One warp per group of 128 inputs.
#pragma once

#include "common.cuh"

namespace quant {

constexpr int STEPS = 24;
// float32(1.0 - 0.5 * i / 24), the reference's shrink factors
__constant__ float c_shrink[STEPS] = {1.0f,        0.97916669f, 0.95833331f, 0.9375f,     0.91666669f, 0.89583331f, 0.875f,      0.85416669f,
                                      0.83333331f, 0.8125f,     0.79166669f, 0.77083331f, 0.75f,       0.72916669f, 0.70833331f, 0.6875f,
                                      0.66666669f, 0.64583331f, 0.625f,      0.60416669f, 0.58333331f, 0.5625f,     0.54166669f, 0.52083331f};

DRB_DEV float half_round(float v) { return __half2float(__float2half_rn(v)); }

// A team of eight lanes owns a group: lane j holds inputs j, 8 + j, ..., 56 + j, which are the terms of the converter's
// running sum j in its order, so a 64-term sum is seven additions in the lane and three exchanges. (With two consecutive
// inputs per lane, one warp per group, the same order took sixteen exchanges and fourteen additions for two inputs: 6.3 ms
// for 134 M weights; 1.48 ms so, 0.93 ms with the candidates passed over that cannot win.)
struct Group {
  unsigned long long v2[4];  // inputs 8 i + j as packed pairs (i = 0, 1), (2, 3), (4, 5), (6, 7)
  unsigned long long n2[4];  // the same, negated
};

DRB_DEV unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
DRB_DEV unsigned long long dup2(float v) { return pack2(v, v); }
DRB_DEV float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// The converter's sum of one packed value per input; every lane of the team gets the total.
DRB_DEV float sum64(const unsigned long long (&t)[4]) {
  float a, b, s;
  unpack2(t[0], a, b);
  s = __fadd_rn(a, b);
#pragma unroll
  for (int i = 1; i < 4; ++i) {
    unpack2(t[i], a, b);
    s = __fadd_rn(__fadd_rn(s, a), b);
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));  // r0 + r1, (r0 + r1) + (r2 + r3), ...
  return s;
}

// The eight codes of a lane: rint((v - lo) / scale) clamped to 0..15, as packed floats. The quotient is taken as a product with
// the reciprocal, within 2^-22 of it, clamped before it is rounded. Where it lands within 1e-5 of an inner rounding boundary
// the candidate n is settled exactly: with d = v - lo (a float, at least scale / 2 here) the remainder d - n scale is exact in
// one fused operation, and it is compared with scale / 2; d's spacing is too coarse for the rounded quotient to reach a
// boundary that the exact one misses. Weights on a bf16 grid make such boundaries common (one value in two thousand), nearly
// all of them exact ties, which go to the even code.
DRB_DEV void codes8(const Group& g, float lo, float scale, float rcp, unsigned long long (&q)[4]) {
  const unsigned long long nlo = dup2(-lo), r2 = dup2(rcp), magic = dup2(12582912.f), nmagic = dup2(-12582912.f), neg1 = dup2(-1.f);
  float worst = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float p0, p1, f0, f1;
    unpack2(mul2(add2(g.v2[i], nlo), r2), p0, p1);
    const unsigned long long p = pack2(fminf(fmaxf(p0, 0.f), 15.f), fminf(fmaxf(p1, 0.f), 15.f));
    q[i] = add2(add2(p, magic), nmagic);  // the nearest integer
    unpack2(fma2(q[i], neg1, p), f0, f1);
    worst = max3(worst, fabsf(f0), fabsf(f1));
  }
  if (worst >= 0.49999f) {
    const float half = 0.5f * scale;
    auto settle = [&](float v, float n) {
      const float e = __fmaf_rn(-n, scale, __fadd_rn(v, -lo));
      const bool odd = ((int)n & 1) != 0;
      const bool move = fabsf(e) > half || (fabsf(e) == half && odd);
      return fminf(fmaxf(move ? (e > 0.f ? n + 1.f : n - 1.f) : n, 0.f), 15.f);
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float v0, v1, n0, n1;
      unpack2(g.v2[i], v0, v1);
      unpack2(q[i], n0, n1);
      q[i] = pack2(settle(v0, n0), settle(v1, n1));
    }
  }
}

// sum of (q * scale + min - v)^2, every operation rounded
DRB_DEV float error8(const Group& g, const unsigned long long (&q)[4], float scale, float lo) {
  const unsigned long long s2 = dup2(scale), lo2 = dup2(lo);
  unsigned long long t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const unsigned long long d = add2(add2(mul2(q[i], s2), lo2), g.n2[i]);
    t[i] = mul2(d, d);
  }
  return sum64(t);
}

// One term of it, for the input v and its code, as the converter computes both.
DRB_DEV float term(float v, float scale, float lo) {
  const float n = fminf(fmaxf(rintf(__fdiv_rn(__fsub_rn(v, lo), scale)), 0.f), 15.f);
  const float d = __fsub_rn(__fadd_rn(__fmul_rn(n, scale), lo), v);
  return __fmul_rn(d, d);
}

constexpr int Q4_THREADS = 256, Q4_GROUPS = Q4_THREADS / 8;
// Six blocks per multiprocessor (40 registers) hide the additions' chains a little better than five: 948 -> 934 us.
// What bounds it: fp32 issue (24 candidates x 9 fp32 operations and 3 comparisons per weight; the packed forms halve the issue
// slots), not memory (4.6 bytes per weight). A candidate's scale, min and reciprocal are the same for the whole group:
// each lane of the team prepares three of the 24 and hands them round.
// A rounded sum of terms that are not negative is at least the rounded sum of any two of them (rounding keeps the order), so the
// terms of the group's smallest and largest input, which clipping hits hardest, bound a candidate's error from below. A
// candidate whose bound is not below the best error so far cannot be taken and is passed over, when that holds for all
// four groups of the warp. The ends outweigh the other 62 inputs' rounding from a shrink of about 0.8 on, the eleventh of the 24.
__global__ void __launch_bounds__(Q4_THREADS, 6) k_quant_q4(const float* __restrict__ w, size_t groups, uint8_t* __restrict__ q,
                                                         __half2* __restrict__ sm) {
  const size_t gi = (size_t)blockIdx.x * Q4_GROUPS + (threadIdx.x >> 3);
  const int j = threadIdx.x & 7;
  const size_t gr = gi < groups ? gi : groups - 1;  // teams beyond the end redo the last group and write nothing
  Group g;
  float gmin = INFINITY, gmax = -INFINITY;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = __ldg(w + gr * 64 + 16 * i + j), b = __ldg(w + gr * 64 + 16 * i + 8 + j);
    gmin = fminf(gmin, fminf(a, b)), gmax = fmaxf(gmax, fmaxf(a, b));
    g.v2[i] = pack2(a, b), g.n2[i] = pack2(-a, -b);
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    gmin = fminf(gmin, __shfl_xor_sync(0xffffffffu, gmin, o));
    gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
  }
  const float center = __fmul_rn(__fadd_rn(gmin, gmax), 0.5f);
  float c_scale[STEPS / 8], c_lo[STEPS / 8], c_rcp[STEPS / 8], c_least[STEPS / 8];  // candidates j, 8 + j, 16 + j
#pragma unroll
  for (int t = 0; t < STEPS / 8; ++t) {
    const float shrink = c_shrink[8 * t + j];
    const float lo_c = __fadd_rn(center, __fmul_rn(__fsub_rn(gmin, center), shrink));
    const float hi_c = __fadd_rn(center, __fmul_rn(__fsub_rn(gmax, center), shrink));
    c_scale[t] = fmaxf(half_round(fmaxf(__fdiv_rn(__fsub_rn(hi_c, lo_c), 15.0f), 1e-10f)), 1e-10f);
    c_lo[t] = half_round(lo_c);
    c_rcp[t] = __frcp_rn(c_scale[t]);
    c_least[t] = __fadd_rn(term(gmin, c_scale[t], c_lo[t]), term(gmax, c_scale[t], c_lo[t]));
  }
  float best_err = 0.f, best_scale = 0.f, best_lo = 0.f, best_rcp = 0.f;
  unsigned long long bq[4];
#pragma unroll
  for (int t = 0; t < STEPS / 8; ++t)
#pragma unroll 2
    for (int i = 0; i < 8; ++i) {
      const bool first = t == 0 && i == 0;
      if (!first && __all_sync(0xffffffffu, __shfl_sync(0xffffffffu, c_least[t], i, 8) >= best_err)) continue;
      const float scale = __shfl_sync(0xffffffffu, c_scale[t], i, 8), lo = __shfl_sync(0xffffffffu, c_lo[t], i, 8);
      const float rcp = __shfl_sync(0xffffffffu, c_rcp[t], i, 8);
      codes8(g, lo, scale, rcp, bq);
      const float err = error8(g, bq, scale, lo);
      if (first || err < best_err) best_err = err, best_scale = scale, best_lo = lo, best_rcp = rcp;
    }
  codes8(g, best_lo, best_scale, best_rcp, bq);
  // One least-squares refinement of (scale, min) given the codes.
  const float n = 64.f;
  unsigned long long t[4];
  const float sq = sum64(bq);
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = mul2(bq[i], bq[i]);
  const float sqq = sum64(t);
  const float sw = sum64(g.v2);
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = mul2(bq[i], g.v2[i]);
  const float sqw = sum64(t);
  const float det = __fsub_rn(__fmul_rn(n, sqq), __fmul_rn(sq, sq));
  const bool ok = fabsf(det) > 1e-6f;
  const float ls_scale = ok ? __fdiv_rn(__fsub_rn(__fmul_rn(n, sqw), __fmul_rn(sq, sw)), det) : best_scale;
  const float ls_min = ok ? __fdiv_rn(__fsub_rn(sw, __fmul_rn(ls_scale, sq)), n) : best_lo;
  const float ls_scale_h = half_round(ls_scale), ls_min_h = half_round(ls_min);
  const float ls_err = error8(g, bq, ls_scale_h, ls_min_h);
  if (ls_err < best_err && ok && ls_scale_h > 0.f) best_scale = ls_scale_h, best_lo = ls_min_h;
  // Packing: this lane's codes are nibble j of words 0..7; three exchanges transpose that to all nibbles of word j.
  uint32_t m = 0u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a, b;
    unpack2(bq[i], a, b);
    m |= ((uint32_t)a << (8 * i)) | ((uint32_t)b << (8 * i + 4));
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    const uint32_t keep = o == 4 ? 0x0000FFFFu : o == 2 ? 0x00FF00FFu : 0x0F0F0F0Fu;  // nibbles whose index lacks bit o
    const uint32_t got = __shfl_xor_sync(0xffffffffu, m, o);
    m = (j & o) ? ((m & ~keep) | ((got & ~keep) >> (4 * o))) : ((m & keep) | ((got & keep) << (4 * o)));
  }
  if (gi < groups) {
    uint8_t* out = q + gi * 32 + 4 * j;
    if ((reinterpret_cast<uintptr_t>(q) & 3) == 0) {
      *reinterpret_cast<uint32_t*>(out) = m;
    } else {
#pragma unroll
      for (int b = 0; b < 4; ++b) out[b] = (uint8_t)(m >> (8 * b));
    }
    if (j == 0) sm[gi] = __halves2half2(__float2half_rn(best_scale), __float2half_rn(best_lo));
  }
}

// Lane l holds inputs 4l .. 4l + 3 of the group of 128.
__global__ void __launch_bounds__(256) k_quant_q8(const float* __restrict__ w, size_t groups, int8_t* __restrict__ q,
                                                  __half* __restrict__ s) {
  const size_t g = (size_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (g >= groups) return;
  const float4 v = reinterpret_cast<const float4*>(w + g * 128)[lane];
  float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  amax = fmaxf(amax, 1e-12f);
  const float scale = fmaxf(half_round(__fdiv_rn(amax, 127.0f)), 1e-12f);
  auto code = [&](float x) { return (int)fminf(fmaxf(rintf(__fdiv_rn(x, scale)), -127.f), 127.f); };
  const char4 o = make_char4((signed char)code(v.x), (signed char)code(v.y), (signed char)code(v.z), (signed char)code(v.w));
  reinterpret_cast<char4*>(q + g * 128)[lane] = o;
  if (lane == 0) s[g] = __float2half_rn(scale);
}

}  // namespace quant

// w: groups x 64 consecutive floats (a [E, N, K] tensor with K a multiple of 64, row-major). q: groups x 32 bytes,
// sm: groups x (scale, min) f16: the layouts of `moe.*.q4` / `moe.*.sm`. No counterpart in the reference's C ABI
// (its quantiser is the Python converter).
extern "C" int drb_quant_q4(const float* w, size_t groups, uint8_t* q, __half2* sm, cudaStream_t st) {
  if (groups == 0) return 0;
  quant::k_quant_q4<<<(unsigned)((groups + quant::Q4_GROUPS - 1) / quant::Q4_GROUPS), quant::Q4_THREADS, 0, st>>>(w, groups, q, sm);
  return 0;
}

// w: groups x 128 consecutive floats; q: the int8 codes; s: one f16 scale per group (`*.q8` / `*.s`).
extern "C" int drb_quant_q8(const float* w, size_t groups, int8_t* q, __half* s, cudaStream_t st) {
  if (groups == 0) return 0;
  quant::k_quant_q8<<<(unsigned)((groups + 7) / 8), 256, 0, st>>>(w, groups, q, s);
  return 0;
}
