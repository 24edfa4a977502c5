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
//   drb_quant_q8: tools/convert.py:33-41 (`quant_q8`). A warp takes four groups of 128 inputs.
#pragma once

#include "common.cuh"

namespace quant {

constexpr int STEPS = 24;
// float32(1.0 - 0.5 * i / 24), the reference's shrink factors
__constant__ float c_shrink[STEPS] = {1.0f,        0.97916669f, 0.95833331f, 0.9375f,     0.91666669f, 0.89583331f, 0.875f,      0.85416669f,
                                      0.83333331f, 0.8125f,     0.79166669f, 0.77083331f, 0.75f,       0.72916669f, 0.70833331f, 0.6875f,
                                      0.66666669f, 0.64583331f, 0.625f,      0.60416669f, 0.58333331f, 0.5625f,     0.54166669f, 0.52083331f};

constexpr float FP16_LEAST = 5.9e-8f;  // just below 2^-24: a scale under it sits at the converter's floor

DRB_DEV float half_round(float v) { return __half2float(__float2half_rn(v)); }

// A team of eight lanes owns a group: lane j holds inputs j, 8 + j, ..., 56 + j, which are the terms of the converter's
// running sum j in its order, so a 64-term sum is seven additions in the lane and three exchanges. (With two consecutive
// inputs per lane, one warp per group, the same order took sixteen exchanges and fourteen additions for two inputs: 6.3 ms
// for 134 M weights, 1.48 ms so.)
struct Group {
  unsigned long long v2[4];  // inputs 8 i + j as packed pairs (i = 0, 1), (2, 3), (4, 5), (6, 7)
};

DRB_DEV float reciprocal(float v) {  // within one unit in the last place
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
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
// boundary that the exact one misses, at a scale that fp16 holds (eleven bits). At the floor of 1e-10, which has 24, it is not, and
// the division itself decides. Weights on a bf16 grid make such boundaries common (one value in two thousand), nearly all of them
// exact ties, which go to the even code.
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
    auto divide = [&](float v) { return fminf(fmaxf(rintf(__fdiv_rn(__fadd_rn(v, -lo), scale)), 0.f), 15.f); };
    const bool floor = scale < FP16_LEAST;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float v0, v1, n0, n1;
      unpack2(g.v2[i], v0, v1);
      unpack2(q[i], n0, n1);
      q[i] = floor ? pack2(divide(v0), divide(v1)) : pack2(settle(v0, n0), settle(v1, n1));
    }
  }
}

// sum of (q * scale + min - v)^2, every operation rounded
DRB_DEV float error8(const Group& g, const unsigned long long (&q)[4], float scale, float lo) {
  const unsigned long long s2 = dup2(scale), lo2 = dup2(lo), neg1 = dup2(-1.f);
  unsigned long long t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const unsigned long long d = fma2(g.v2[i], neg1, add2(mul2(q[i], s2), lo2));
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

// A candidate's error, estimated: in units of its scale and measured from the middle of its range an input is a = |v - min| / scale - 7.5|,
// its code the nearest of 0.5, 1.5, ..., 7.5. With 32 added a float's last place is 2^-18: cutting off the fraction's 18 bits and
// setting the highest of them is the rounding. One packed fused operation, two additions, two logic operations, two minima and two more
// packed operations per two inputs, where the converter's own operations take 22 and a sum across lanes.
constexpr float EST_BASE = 32.f;
constexpr uint32_t EST_MASK = 0xFFFC0000u, EST_HALF = 0x00020000u;
DRB_DEV void estimate2(unsigned long long v2, unsigned long long rcp2, unsigned long long c2, unsigned long long neg1, unsigned long long& sum) {
  float u0, u1;
  unpack2(fma2(v2, rcp2, c2), u0, u1);
  const float r0 = __fadd_rn(fabsf(u0), EST_BASE), r1 = __fadd_rn(fabsf(u1), EST_BASE);
  const float q0 = fminf(__uint_as_float(lop3_and_or(__float_as_uint(r0), EST_MASK, EST_HALF)), EST_BASE + 7.5f);
  const float q1 = fminf(__uint_as_float(lop3_and_or(__float_as_uint(r1), EST_MASK, EST_HALF)), EST_BASE + 7.5f);
  const unsigned long long e = fma2(pack2(q0, q1), neg1, pack2(r0, r1));
  sum = fma2(e, e, sum);
}

constexpr int Q4_THREADS = 256, Q4_WARPS = Q4_THREADS / 32, Q4_GROUPS = Q4_THREADS / 8;
constexpr int Q4_STRIDE = 72;   // floats between a warp's four groups in shared memory: their 16-byte reads share no bank
constexpr float Q4_FLAT = 2e-6f;  // a range below it can bring scales to the converter's floor
constexpr int Q4_LIGHT = 12;    // candidates that are estimated; the others clip a quarter of the range or more
// What bounds it: fp32 and integer issue (an instruction in 0.83 of the cycles, 1030 per warp), not memory (4.6 bytes per weight). Half of
// the time are the estimates, half what a group costs without them: loads, two candidates a lane, one evaluation, refinement, packing
// (134 M bf16 weights: 276 us of 560 with the estimates left out). Of the 24 candidates the first twelve are told apart by
// the estimate, lane j taking candidate j over the group's 64 inputs and candidate 8 + j % 4 over half of them (shared memory, broadcast
// reads), and only those that the estimate's error leaves in the running are evaluated in the converter's operations and order: 1.02
// on average on normal weights: 0.56 ms for 134 M weights. Every candidate evaluated that way took 1.48 ms, the half that a bound by the ends
// leaves 0.93 ms; the estimate for sixteen of them instead of twelve, and with correctly rounded reciprocals and roots, 0.69 ms.
// How far the estimate is off. In units of the scale, with a below 31 (beyond, and wherever something is not a number, the candidate
// is evaluated): the estimate's a by 2^-19 for the sum with 32, 39 * 2^-23 for the reciprocal and 39 * 2^-24 for offset and product, the
// converter's difference by 61 * 2^-24, its choice of code by 2 * 39 * 2^-23 at a boundary; each with 2^-23 |min| / scale for groups far
// from zero. Together less than eta = 2^-15 + 2^-21 |min| / scale per input, so the sums S of 64 squares differ by less than
// 16 eta sqrt(S) + 64 eta^2 (Cauchy), and by 2^-16 S for the additions. Two candidates whose estimates differ by more than both bounds are in
// the right order.
// The last twelve candidates leave the group's smallest and largest input at least a quarter of half the range outside, less what
// rounding scale and min to fp16 moves the ends. On most weights those two inputs alone exceed the best error of the others; where
// they do not, for one of the warp's four groups, a candidate's own terms of the two inputs are looked at. (A rounded sum of terms that are not
// negative is at least the rounded sum of any two of them: rounding keeps the order.) Without that second look groups far from
// zero, or with scales among fp16's last numbers, evaluated all twelve: 67 M weights around 1, or with a range of 5e-5, 319 and 619 us instead of
// 302 and 471. Nearly constant groups, whose estimates could not tell candidates apart, do without them: zeros 285 -> 152 us.
template <bool VEC>
__global__ void __launch_bounds__(Q4_THREADS, 5) k_quant_q4(const float* __restrict__ w, size_t groups, uint8_t* __restrict__ q,
                                                         __half2* __restrict__ sm) {
  __shared__ __align__(16) float stage[Q4_WARPS][4 * Q4_STRIDE];
  const size_t gi = (size_t)blockIdx.x * Q4_GROUPS + (threadIdx.x >> 3);
  const int j = threadIdx.x & 7, lane = threadIdx.x & 31, team = lane >> 3;
  float* const mine = stage[threadIdx.x >> 5] + team * Q4_STRIDE;
  // teams beyond the end redo the last group and write nothing
  if (VEC) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const size_t gr = min(gi - team + 2 * h + (lane >> 4), groups - 1);
      *reinterpret_cast<float4*>(stage[threadIdx.x >> 5] + (2 * h + (lane >> 4)) * Q4_STRIDE + 4 * (lane & 15)) =
          __ldg(reinterpret_cast<const float4*>(w + gr * 64) + (lane & 15));
    }
  } else {
    const size_t gr = min(gi, groups - 1);
#pragma unroll
    for (int i = 0; i < 8; ++i) mine[8 * i + j] = __ldg(w + gr * 64 + 8 * i + j);
  }
  __syncwarp();
  Group g;
  float gmin = INFINITY, gmax = -INFINITY;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = mine[16 * i + j], b = mine[16 * i + 8 + j];
    gmin = fminf(gmin, fminf(a, b)), gmax = fmaxf(gmax, fmaxf(a, b));
    g.v2[i] = pack2(a, b);
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    gmin = fminf(gmin, __shfl_xor_sync(0xffffffffu, gmin, o));
    gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
  }
  const float center = __fmul_rn(__fadd_rn(gmin, gmax), 0.5f);
  const unsigned long long neg1 = dup2(-1.f);
  struct Candidate {
    float scale, lo, rcp;
  };
  auto candidate = [&](float shrink) {
    Candidate c;
    const float lo_c = __fadd_rn(center, __fmul_rn(__fsub_rn(gmin, center), shrink));
    const float hi_c = __fadd_rn(center, __fmul_rn(__fsub_rn(gmax, center), shrink));
    c.scale = fmaxf(half_round(fmaxf(__fdiv_rn(__fsub_rn(hi_c, lo_c), 15.0f), 1e-10f)), 1e-10f);
    c.lo = half_round(lo_c);
    c.rcp = reciprocal(c.scale);
    return c;
  };
  const Candidate ca = candidate(c_shrink[j]), cb = candidate(c_shrink[8 + (j & 3)]);
  const float mid_a = __fmaf_rn(-ca.lo, ca.rcp, -7.5f), mid_b = __fmaf_rn(-cb.lo, cb.rcp, -7.5f);
  unsigned long long sum_a = 0ull, sum_b = 0ull;
  if (__any_sync(0xffffffffu, gmax - gmin < Q4_FLAT)) {
    sum_a = sum_b = dup2(NAN);
  } else {
    const unsigned long long ra = dup2(ca.rcp), ma = dup2(mid_a), rb = dup2(cb.rcp), mb = dup2(mid_b);
    const ulonglong2* chunk = reinterpret_cast<const ulonglong2*>(mine);
#pragma unroll 2
    for (int k = 0; k < 8; ++k) {
      const ulonglong2 v0 = chunk[2 * k], v1 = chunk[2 * k + 1], u = chunk[2 * k + (j >> 2)];
      estimate2(v0.x, ra, ma, neg1, sum_a);
      estimate2(u.x, rb, mb, neg1, sum_b);
      estimate2(v0.y, ra, ma, neg1, sum_a);
      estimate2(v1.x, ra, ma, neg1, sum_a);
      estimate2(u.y, rb, mb, neg1, sum_b);
      estimate2(v1.y, ra, ma, neg1, sum_a);
    }
  }
  // an estimate's two sides; NaN where the candidate has to be evaluated whatever the others are
  auto sides = [&](const Candidate& c, float mid, float s, float& least, float& most) {
    const float eta = 0x1p-15f + 0x1p-21f * fabsf(c.lo) * c.rcp, s2 = c.scale * c.scale;
    const float a0 = fabsf(__fmaf_rn(gmin, c.rcp, mid)), a1 = fabsf(__fmaf_rn(gmax, c.rcp, mid));
    float root;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(root) : "f"(s));
    const float est = a0 < 31.f && a1 < 31.f ? s2 * s : NAN, off = s2 * (17.f * eta * root + 70.f * eta * eta + 0x1p-16f * s) + 1e-42f;
    least = est - off, most = est + off;
  };
  float lo_s, hi_s, least_a, least_b, most_a, most_b;
  unpack2(sum_a, lo_s, hi_s);
  sides(ca, mid_a, lo_s + hi_s, least_a, most_a);
  unpack2(sum_b, lo_s, hi_s);
  float s_b = lo_s + hi_s;
  s_b += __shfl_xor_sync(0xffffffffu, s_b, 4);
  sides(cb, mid_b, s_b, least_b, most_b);
  float bound = fminf(most_a, most_b);  // no candidate whose error exceeds it can be the best: fminf passes NaN over
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) bound = fminf(bound, __shfl_xor_sync(0xffffffffu, bound, o));
  uint32_t open = (__ballot_sync(0xffffffffu, !(least_a > bound)) >> (8 * team)) & 0xffu;  // candidates of this team's group that may be the best
  open |= ((__ballot_sync(0xffffffffu, !(least_b > bound)) >> (8 * team)) & 0xfu) << 8;
  const float far = fmaxf(fabsf(gmin), fabsf(gmax)), half = 0.5f * (gmax - gmin);
  const float clip = 0.2499f * half - 0x1p-10f * (far + half) - 1e-6f;
  const bool heavy = __any_sync(0xffffffffu, !(clip > 0.f && 1.99f * clip * clip >= bound));
  float best_err = 0.f, best_scale = 0.f, best_lo = 0.f;
  unsigned long long bq[4];
  auto evaluate = [&](const Candidate& c, bool first, bool counts) {
    unsigned long long cq[4];
    codes8(g, c.lo, c.scale, c.rcp, cq);
    const float err = error8(g, cq, c.scale, c.lo);
    if (first || (counts && err < best_err)) {
      best_err = err, best_scale = c.scale, best_lo = c.lo;
#pragma unroll
      for (int i = 0; i < 4; ++i) bq[i] = cq[i];
    }
  };
  for (bool first = true; __any_sync(0xffffffffu, open != 0u); first = false) {  // the estimate's own least is always open: every team has one
    const int i = open ? __ffs(open) - 1 : 0;
    auto of = [&](float a, float b) { return __shfl_sync(0xffffffffu, i < 8 ? a : b, i & 7, 8); };
    Candidate c;
    c.scale = of(ca.scale, cb.scale), c.lo = of(ca.lo, cb.lo);
    c.rcp = reciprocal(c.scale);  // handed round as well, it cost a spilled register and 2 %
    evaluate(c, first, open != 0u);
    open &= open - 1u;
    if (best_err == 0.f) open = 0u;  // nothing is less
  }
  if (heavy)
#pragma unroll 1
    for (int i = Q4_LIGHT; i < STEPS && __any_sync(0xffffffffu, best_err != 0.f); ++i) {
      const Candidate c = candidate(c_shrink[i]);
      if (!__all_sync(0xffffffffu, __fadd_rn(term(gmin, c.scale, c.lo), term(gmax, c.scale, c.lo)) >= best_err)) evaluate(c, false, true);
    }
  // This lane's codes as bytes: inputs 8 i + j in byte i of c0 (i < 4) or c1. With 1.5 * 2^23 added a code is the float's lowest byte.
  uint32_t c0, c1;
  {
    uint32_t n[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float a, b;
      unpack2(add2(bq[i], dup2(12582912.f)), a, b);
      n[2 * i] = __float_as_uint(a), n[2 * i + 1] = __float_as_uint(b);
    }
    c0 = prmt(prmt(n[0], n[1], 0x0040u), prmt(n[2], n[3], 0x0040u), 0x5410u);
    c1 = prmt(prmt(n[4], n[5], 0x0040u), prmt(n[6], n[7], 0x0040u), 0x5410u);
  }
  // One least-squares refinement of (scale, min) given the codes. Their sums are whole numbers below 2^24, the same in any order.
  const float n = 64.f;
  uint32_t isum = __dp4a(c0, 0x01010101u, __dp4a(c1, 0x01010101u, 0u)) | (__dp4a(c0, c0, __dp4a(c1, c1, 0u)) << 12);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) isum += __shfl_xor_sync(0xffffffffu, isum, o);
  const float sq = (float)(isum & 0xfffu), sqq = (float)(isum >> 12);
  unsigned long long t[4];
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
  uint32_t m = prmt(c0 | (c0 >> 4), c1 | (c1 >> 4), 0x6420u);
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

// Lane l holds inputs 4l .. 4l + 3 of a group of 128; a warp takes four groups, all of them requested before the first is used.
// Bound by the bytes (5 per weight): 134 M weights take 105 us, 6.4 TB/s; the issue slots stand at 0.74 beside it. (A group per warp, with four
// divisions per lane, took 162.) A quotient is taken as a product with the reciprocal, within 2^-22 of it; where that lands within 1e-4
// of a rounding boundary it is settled by the exact remainder, as in codes8 (a code has seven bits and the scale eleven, so their
// product is exact).
constexpr int Q8_PER = 4, Q8_WARPS = 8;
__global__ void __launch_bounds__(Q8_WARPS * 32) k_quant_q8(const float* __restrict__ w, size_t groups, int8_t* __restrict__ q,
                                                  __half* __restrict__ s) {
  const size_t g0 = ((size_t)blockIdx.x * Q8_WARPS + (threadIdx.x >> 5)) * Q8_PER;
  const int lane = threadIdx.x & 31;
  float4 all[Q8_PER];
#pragma unroll
  for (int i = 0; i < Q8_PER; ++i)
    if (g0 + i < groups) all[i] = __ldg(reinterpret_cast<const float4*>(w + (g0 + i) * 128) + lane);
#pragma unroll
  for (int i = 0; i < Q8_PER; ++i) {
    if (g0 + i >= groups) return;
    const float v[4] = {all[i].x, all[i].y, all[i].z, all[i].w};
    // magnitudes order like their bits; a NaN is passed over
    float amax = fmaxf(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))), 0.f);
    amax = fmaxf(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax))), 1e-12f);
    const float scale = fmaxf(half_round(__fdiv_rn(amax, 127.0f)), 1e-12f);
    const float rcp = reciprocal(scale);
    float n[4], worst = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float p = fminf(fmaxf(v[j] * rcp, -127.f), 127.f);
      n[j] = __fadd_rn(__fadd_rn(p, 12582912.f), -12582912.f);  // the nearest integer
      worst = fmaxf(worst, fabsf(p - n[j]));
    }
    if (scale < FP16_LEAST) {  // at the floor: a scale of 24 bits, whose products are not exact
#pragma unroll
      for (int j = 0; j < 4; ++j) n[j] = fminf(fmaxf(rintf(__fdiv_rn(v[j], scale)), -127.f), 127.f);
    } else if (worst >= 0.4999f) {
      const float half = 0.5f * scale;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = __fmaf_rn(-n[j], scale, v[j]);
        const bool move = fabsf(e) > half || (fabsf(e) == half && ((int)n[j] & 1) != 0);
        if (move) n[j] = fminf(fmaxf(e > 0.f ? n[j] + 1.f : n[j] - 1.f, -127.f), 127.f);
      }
    }
    uint32_t b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = __float_as_uint(__fadd_rn(n[j], 12582912.f));  // the code is the lowest byte
    reinterpret_cast<uint32_t*>(q + (g0 + i) * 128)[lane] = prmt(prmt(b[0], b[1], 0x0040u), prmt(b[2], b[3], 0x0040u), 0x5410u);
    if (lane == 0) s[g0 + i] = __float2half_rn(scale);
  }
}

}  // namespace quant

// w: groups x 64 consecutive floats (a [E, N, K] tensor with K a multiple of 64, row-major). q: groups x 32 bytes,
// sm: groups x (scale, min) f16: the layouts of `moe.*.q4` / `moe.*.sm`. No counterpart in the reference's C ABI
// (its quantiser is the Python converter).
extern "C" int drb_quant_q4(const float* w, size_t groups, uint8_t* q, __half2* sm, cudaStream_t st) {
  if (groups == 0) return 0;
  const auto kernel = (reinterpret_cast<uintptr_t>(w) & 15) == 0 ? quant::k_quant_q4<true> : quant::k_quant_q4<false>;  // w starts at any float
  kernel<<<(unsigned)((groups + quant::Q4_GROUPS - 1) / quant::Q4_GROUPS), quant::Q4_THREADS, 0, st>>>(w, groups, q, sm);
  return 0;
}

// w: groups x 128 consecutive floats; q: the int8 codes; s: one f16 scale per group (`*.q8` / `*.s`).
extern "C" int drb_quant_q8(const float* w, size_t groups, int8_t* q, __half* s, cudaStream_t st) {
  if (groups == 0) return 0;
  constexpr int per_block = quant::Q8_PER * quant::Q8_WARPS;
  quant::k_quant_q8<<<(unsigned)((groups + per_block - 1) / per_block), quant::Q8_WARPS * 32, 0, st>>>(w, groups, q, s);
  return 0;
}
