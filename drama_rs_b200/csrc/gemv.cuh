// Batch-1 weight-streaming GEMVs: dr_gemv_q8, dr_gemv_q8_swiglu, dr_gemv_bf16.
//
// One block per multiprocessor owns a contiguous range of output rows. A producer thread streams that range through a ring
// of shared-memory stages with bulk asynchronous copies; the consumer warps multiply and add up. RMSNorm of the input, the
// residual add, SwiGLU and the L2 prefetch of the next kernel's weights are fused in.
//
// Two blocks fit a multiprocessor: a kernel launched behind another (programmatic dependent launch) becomes resident while
// its predecessor still runs and fills its ring, up to 15 MB chip-wide, before its input exists. What is left on the path
// from one launch to the next, and bounds a chain of them, is the time from the input to the output of a block whose weights
// lie in shared memory.
//
// int8 weights: that time was 4.7 us of a 5.9 us launch (8192 x 2048), 2.7 of it dp4a sums of two warps per scheduler and 1.0
// the conversion of the input by the whole block. The sums now run on the tensor cores (mma.sync m16n8k32 s8: batch 1 has
// too few columns for tcgen05, and the operands need no tensor memory): sixteen weight rows are the M dimension, and the
// N dimension holds the limbs of the input. Over the 128 inputs of a weight scale, x_k = delta * n_k with |n_k| <= 2^27, n split
// into four signed 7-bit limbs: four columns of the eight. The int32 sums are exact, a limb more than the dp4a form had
// and finer than fp32's own rounding of x; scale and delta are applied in fp32. Every warp owns 128 inputs of each 2048 and
// converts only those, for itself.
//
// Replaces kernels/drama.cu:219-315 of the reference (k_gemv_q8, k_gemv_q8_swiglu, k_gemv_bf16
// and their launchers), behind the same C signatures (src/ffi.rs:33-40).
#pragma once

#include "common.cuh"

namespace gemv {

constexpr int BLOCK_BYTES = 112 * 1024;  // two blocks per multiprocessor

// The caller's prefetch hint. A following GEMV of this library fills its rings itself as soon as its blocks are resident, about `skip`
// bytes per multiprocessor from the start of each block's share of the rows; asked for here as well, the same lines twice, it
// slowed both (a chain of 33 projections 135 us instead of 129). So of a region that size what lies behind them is prefetched, and no more
// than 128 KB per multiprocessor: a vocabulary-sized region would only push out what the running kernels still read. This launch's
// blocks, when they are fewer, go over all of the successor's shares. A region of at most 2 MB (a router's, a short projection's) is
// prefetched whole, whoever reads it: chains of GEMVs of 0.5, 1 and 2 MB take the same with the hint as without (1.785, 1.815,
// 1.87 us a launch); at 4 MB the lines asked for twice begin to show (1.90 -> 1.97).
constexpr size_t HINT_WHOLE = 2 << 20;
DRB_DEV void prefetch_hint(const char* pf, size_t pf_bytes, unsigned skip, unsigned sms, unsigned block, unsigned blocks) {
  if (skip == 0 || pf_bytes <= HINT_WHOLE) return prefetch_share(pf, pf_bytes, block, blocks);
  const size_t per = pf_bytes / sms;
  if (!pf || per <= skip) return;
  for (unsigned i = block; i < sms; i += blocks) prefetch_share(pf + i * per + skip, per - skip < 131072 ? per - skip : 131072, 0, 1);
}
constexpr unsigned HINT_SKIP = 96 * 1024;

// ---- int8 weights -----------------------------------------------------------------------------------------------------
namespace q8 {

constexpr int CW = 16, NT = CW * 32, THREADS = NT + 32;  // consumer warps + the producer warp
constexpr int GROUP = 128;                               // inputs per weight scale = per warp and segment
constexpr int BATCH = 64;                                // rows whose partial sums are added up at a time

// K inputs, U = 2: SwiGLU (a tile is eight gate rows and their eight up rows), else 1.
template <int K, int U>
struct Shape {
  static constexpr int STAGES = K < 2048 ? 2 : 3;
  static constexpr int SEG = K < 2048 ? K : 2048;       // inputs of a stage
  static constexpr int NSEG = K / SEG;
  static constexpr int KW = SEG / GROUP;                // warps along K
  static constexpr int RS = CW / KW;                    // 16-row tiles per stage
  static constexpr int ROWS = 16 * RS;                  // weight rows per stage
  static constexpr int PITCH = SEG + 64;                // bytes between rows in a stage: rows r and r + 1 on different banks
  static constexpr int SROW = K / GROUP * 2;            // bytes of scales per row
  static constexpr bool S_COPY = SROW >= 16;            // bulk copies need 16-byte granules
  static constexpr int S_SLOTS = S_COPY ? (NSEG > 1 ? 2 : 3) : 0;  // see the producer
  static constexpr int STAGE_BYTES = ROWS * PITCH;
  static constexpr int WARP_BYTES = 2 * BATCH * 4;      // per warp: limbs on their way to the operand layout, then two batches of partial sums
  static constexpr size_t BYTES = 512 + (size_t)STAGES * STAGE_BYTES + S_SLOTS * ROWS * SROW + CW * WARP_BYTES;
  static_assert(K % SEG == 0 && CW % KW == 0 && BATCH % ROWS == 0 && BYTES <= BLOCK_BYTES, "shape");
  static_assert(U == 1 || RS == 1, "SwiGLU: one tile per stage");
};

struct Ctl {
  uint64_t full[3], empty[3];
  __align__(16) float red[CW];
};
static_assert(sizeof(Ctl) <= 512, "control block");

DRB_DEV void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); }

DRB_DEV void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int K, int U>
__global__ void __launch_bounds__(THREADS, 2)
    k_gemv(const int8_t* __restrict__ W, const __half* __restrict__ S, const float* __restrict__ x, const float* res, float* y, int N,
           const float* __restrict__ nw, float eps, const char* pf, size_t pf_bytes, unsigned pf_skip, unsigned sms) {
  using P = Shape<K, U>;
  constexpr int STAGES = P::STAGES, NSEG = P::NSEG, KW = P::KW, RS = P::RS, ROWS = P::ROWS, SEG = P::SEG, PITCH = P::PITCH, SROW = P::SROW;
  constexpr int SLOTS = P::S_SLOTS ? P::S_SLOTS : 1;
  extern __shared__ __align__(128) unsigned char dyn[];
  Ctl& ctl = *reinterpret_cast<Ctl*>(dyn);
  unsigned char* ring = dyn + 512;
  unsigned char* scales = ring + STAGES * P::STAGE_BYTES;
  unsigned char* own = scales + P::S_SLOTS * ROWS * SROW;  // [warp][WARP_BYTES]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned G = gridDim.x, b = blockIdx.x;
  const int u0 = (int)((long long)N * b / G), u1 = (int)((long long)N * (b + 1) / G);  // this block's outputs
  constexpr int OUT = ROWS / U;                                                          // outputs per stage
  const int ntiles = (u1 - u0 + OUT - 1) / OUT;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(&ctl.full[s], 1), mbar_init(&ctl.empty[s], CW);
    mbar_fence_init();
  }
  __syncthreads();
  pdl_launch_dependents();

  if (warp == CW) {
    // ---------------- producer: weights are constants, so copies start before the dependency wait. A tile's scales come with its
    // first stage into one of S_SLOTS slots; the stage STAGES requests back has been read by then, so the slot's last tile is done.
    static_assert(P::S_SLOTS == 0 || P::S_SLOTS * NSEG >= STAGES + NSEG - 1, "scale slots");
    if (elect_one()) {
      int s = 0;
      uint32_t par = 1;  // every stage starts free
      for (int t = 0; t < ntiles; ++t) {
        const int r0 = u0 + t * OUT, nr = min(OUT, u1 - r0);
        for (int seg = 0; seg < NSEG; ++seg) {
          if (!mbar_wait_hot(&ctl.empty[s], par, DRB_ERR_EMPTY_WAIT)) return;
          unsigned char* dst = ring + s * P::STAGE_BYTES;
          const bool sc = P::S_COPY && seg == 0;
          mbar_expect_tx(&ctl.full[s], (unsigned)(nr * U * (SEG + (sc ? SROW : 0))));
#pragma unroll 1
          for (int u = 0; u < U; ++u) {
            const int8_t* src = W + ((size_t)u * N + r0) * K + seg * SEG;
#pragma unroll 1
            for (int r = 0; r < nr; ++r) bulk_g2s(dst + (u * 8 + r) * PITCH, src + (size_t)r * K, SEG, &ctl.full[s]);
            if (sc)
              bulk_g2s(scales + (t % SLOTS * ROWS + u * 8) * SROW, reinterpret_cast<const unsigned char*>(S) + ((size_t)u * N + r0) * SROW,
                       (unsigned)(nr * SROW), &ctl.full[s]);
          }
          if (++s == STAGES) s = 0, par ^= 1u;
        }
      }
      prefetch_hint(pf, pf_bytes, pf_skip, sms, b, G);
    }
    return;
  }

  // ---------------- consumers: warp (sub, kw) multiplies tile `sub` of a stage with inputs [128 kw, +128) of its segment
  const int kw = warp % KW, sub = warp / KW, g = lane >> 2, t4 = lane & 3;
  float* mine = reinterpret_cast<float*>(own + warp * P::WARP_BYTES);
  // The operand of a stage goes to registers and the stage back to the producer before the tensor cores have used it; the first
  // one even before the input exists, so that a block has one stage more than its ring holds on the way (8192 x 2048 needs
  // four stages of three: the fourth came only after the input, a microsecond of each launch).
  constexpr bool EARLY = NSEG <= 2;  // longer rows have no registers to spare while the input is converted
  bool dead = false;                 // a wait ran out once: no later wait spins (the error word is set, the results are void)
  int s = 0;
  uint32_t par = 0;
  uint4 v0, v1, w0, w1;  // rows g and g + 8 of the tile, two pieces each
  __half sc0 = __half(), sc1 = __half();
  auto release = [&]() {
    __syncwarp();
    if (lane == 0) mbar_arrive(&ctl.empty[s]);
    if (++s == STAGES) s = 0, par ^= 1u;
  };
  auto operand = [&]() { return ring + s * P::STAGE_BYTES + (sub * 16 + g) * PITCH + kw * GROUP + 16 * t4; };
  auto load = [&](int t, int q) {
    if (!P::S_COPY) {
      const int row = u0 + t * OUT + sub * 16 + g;
      sc0 = row < u1 ? __ldg(S + (size_t)row * (K / GROUP) + kw) : __half();
      sc1 = row + 8 < u1 ? __ldg(S + (size_t)(row + 8) * (K / GROUP) + kw) : __half();
    }
    if (!dead) dead = !mbar_wait_hot(&ctl.full[s], par, DRB_ERR_FULL_WAIT);
    const unsigned char* rp = operand();
    v0 = *reinterpret_cast<const uint4*>(rp), w0 = *reinterpret_cast<const uint4*>(rp + 8 * PITCH);
    if (EARLY) v1 = *reinterpret_cast<const uint4*>(rp + 64), w1 = *reinterpret_cast<const uint4*>(rp + 8 * PITCH + 64);
    if (P::S_COPY) {
      const unsigned char* sp = scales + (t % SLOTS * ROWS + sub * 16 + g) * SROW + 2 * (q * KW + kw);
      sc0 = *reinterpret_cast<const __half*>(sp), sc1 = *reinterpret_cast<const __half*>(sp + 8 * SROW);
    }
    if (EARLY) release();
  };
  // The norm weights are brought as far as L2 before the input may be read (they may be the work of the launch before).
  float4 wv[NSEG], xv[NSEG];
  if (nw && sub == 0 && (lane & 7) == 0)
#pragma unroll
    for (int q = 0; q < NSEG; ++q) prefetch_line_l2(nw + q * SEG + kw * GROUP + 4 * lane);
  if (EARLY) load(0, 0);
  pdl_wait();  // x and res come from the previous kernel
#pragma unroll
  for (int q = 0; q < NSEG; ++q) {
    xv[q] = __ldcg(reinterpret_cast<const float4*>(x + q * SEG + kw * GROUP) + lane);
    if (EARLY && nw) wv[q] = __ldcg(reinterpret_cast<const float4*>(nw + q * SEG + kw * GROUP) + lane);
  }
  // Thread o < bo writes output o of every batch; the first batch's residual is requested now.
  constexpr int bo = BATCH / U;
  const bool writer = (int)threadIdx.x < bo;
  float add = 0.f;
  if (res && writer && u0 + (int)threadIdx.x < u1) add = __ldcg(res + u0 + threadIdx.x);
  // RMSNorm: the sum is linear in the input, so the rows meet x * nw and the outputs get 1 / rms at the end, where the warps meet
  // anyway: nothing waits for the sum of squares in front of the conversion (a chain of 33 projections, half of them normed, 129.6 ->
  // 125.5 us).
  float ss = 0.f;
  if (nw) {
#pragma unroll
    for (int q = 0; q < NSEG; ++q) {
      ss += (xv[q].x * xv[q].x + xv[q].y * xv[q].y) + (xv[q].z * xv[q].z + xv[q].w * xv[q].w);
      if (!EARLY) wv[q] = __ldcg(reinterpret_cast<const float4*>(nw + q * SEG + kw * GROUP) + lane);
      xv[q] = make_float4(xv[q].x * wv[q].x, xv[q].y * wv[q].y, xv[q].z * wv[q].z, xv[q].w * wv[q].w);
    }
  }
  // Limbs. Lane l holds inputs 4 l .. 4 l + 3 of the 128; the operand wants, in lane (g, t4), limb g of inputs 16 t4 + 4 i and
  // 64 + 16 t4 + 4 i: the order in which a lane's two 16-byte pieces of a weight row come (any order serves a sum).
  uint32_t bf[NSEG][8];
  float delta[NSEG];
  uint32_t* sw = reinterpret_cast<uint32_t*>(mine);
#pragma unroll
  for (int q = 0; q < NSEG; ++q) {
    const float v[4] = {xv[q].x, xv[q].y, xv[q].z, xv[q].w};
    const float m = __uint_as_float(__reduce_max_sync(
        0xffffffffu, __float_as_uint(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))))));
    // m / 2^27, kept away from the subnormals, whose reciprocal is infinite
    const float d = fmaxf(m * (1.f / 134217728.f), 1.1754944e-38f);
    const float inv = 1.f / d;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int n = __float2int_rn(v[i] * inv);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const int lo = l < 3 ? ((n + 64) & 127) - 64 : n;
        n = (n - lo) >> 7;
        w[l] |= (uint32_t)(lo & 0xff) << (8 * i);
      }
    }
    __syncwarp();
#pragma unroll
    for (int l = 0; l < 4; ++l) sw[32 * l + lane] = w[l];
    __syncwarp();
    uint4 p = make_uint4(0u, 0u, 0u, 0u), r = p;
    if (g < 4) p = *reinterpret_cast<const uint4*>(sw + 32 * g + 4 * t4), r = *reinterpret_cast<const uint4*>(sw + 32 * g + 16 + 4 * t4);
    bf[q][0] = p.x, bf[q][1] = p.y, bf[q][2] = p.z, bf[q][3] = p.w, bf[q][4] = r.x, bf[q][5] = r.y, bf[q][6] = r.z, bf[q][7] = r.w;
    // lanes t4 = 0 hold the sums of limbs 0 and 1, lanes t4 = 1 those of limbs 2 and 3; the rest have none
    delta[q] = t4 == 0 ? d : t4 == 1 ? d * 16384.f : 0.f;
  }
  __syncwarp();  // before partial sums overwrite the limbs
  if (nw) {
    ss = warp_sum(ss);
    if (lane == 0) ctl.red[warp] = ss;  // read behind the first batch's barrier
  }
  float inv_rms = 1.f;

  for (int t = 0; t < ntiles; ++t) {
    float a0 = 0.f, a1 = 0.f;  // rows g and g + 8 of the tile
#pragma unroll
    for (int q = 0; q < NSEG; ++q) {
      if (!EARLY) load(t, q);
      int c[4] = {0, 0, 0, 0}, e[4] = {0, 0, 0, 0};
      mma_s8(c, v0.x, w0.x, v0.y, w0.y, bf[q][0], bf[q][1]);
      if (EARLY) {
        mma_s8(e, v1.x, w1.x, v1.y, w1.y, bf[q][4], bf[q][5]);
        mma_s8(c, v0.z, w0.z, v0.w, w0.w, bf[q][2], bf[q][3]);
        mma_s8(e, v1.z, w1.z, v1.w, w1.w, bf[q][6], bf[q][7]);
      } else {  // the second pieces in the registers of the first
        mma_s8(c, v0.z, w0.z, v0.w, w0.w, bf[q][2], bf[q][3]);
        const unsigned char* rp = operand() + 64;
        v0 = *reinterpret_cast<const uint4*>(rp), w0 = *reinterpret_cast<const uint4*>(rp + 8 * PITCH);
        release();
        mma_s8(c, v0.x, w0.x, v0.y, w0.y, bf[q][4], bf[q][5]);
        mma_s8(c, v0.z, w0.z, v0.w, w0.w, bf[q][6], bf[q][7]);
      }
      // |a limb's sum| <= 128 * 128 * 64 = 2^20: limb + 128 * next limb stays an exact integer
      a0 = fmaf(__half2float(sc0) * delta[q], (float)((c[0] + e[0]) + ((c[1] + e[1]) << 7)), a0);
      a1 = fmaf(__half2float(sc1) * delta[q], (float)((c[2] + e[2]) + ((c[3] + e[3]) << 7)), a1);
      if (EARLY) {
        if (q + 1 < NSEG) load(t, q + 1);
        else if (t + 1 < ntiles) load(t + 1, 0);
      }
    }
    a0 += __shfl_xor_sync(0xffffffffu, a0, 1);
    a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
    constexpr int TB = BATCH / ROWS;  // tiles per batch
    float* buf = mine + (t / TB & 1) * BATCH;
    if (t4 == 0) buf[t % TB * 16 + g] = a0, buf[t % TB * 16 + 8 + g] = a1;
    if (t % TB == TB - 1 || t == ntiles - 1) {
      // The batch's outputs: one thread each adds the warps' parts in order. The other buffer takes the next batch, which ends in
      // this barrier again before anyone comes back to this buffer.
      consumer_sync();
      const int o = (int)threadIdx.x, first = u0 + t / TB * bo;
      if (writer) {
        if (nw && t < TB) {
          float tot = 0.f;
#pragma unroll
          for (int w = 0; w < KW; w += 4) {  // the warps of tile 0: each input once
            const float4 v = *reinterpret_cast<const float4*>(&ctl.red[w]);
            tot += (v.x + v.y) + (v.z + v.w);
          }
          inv_rms = rsqrtf(tot / K + eps);
        }
        const int tile = o / (16 / U), row = o % (16 / U);  // within the batch
        const float* pp = reinterpret_cast<const float*>(own + (RS > 1 ? tile * KW : 0) * P::WARP_BYTES) + (t / TB & 1) * BATCH + (RS > 1 ? 0 : tile * 16) + row;
        float r0 = 0.f, r1 = 0.f;
#pragma unroll
        for (int w = 0; w < KW; ++w) {
          r0 += pp[w * (P::WARP_BYTES / 4)];
          if (U == 2) r1 += pp[w * (P::WARP_BYTES / 4) + 8];
        }
        r0 *= inv_rms;
        if (first + o < u1) y[first + o] = U == 2 ? silu_f(r0) * (r1 * inv_rms) : r0 + add;
        add = res && first + bo + o < u1 ? __ldcg(res + first + bo + o) : 0.f;  // the next batch's
      }
    }
  }
}

template <int K, int U>
int launch(const int8_t* W, const __half* S, const float* x, const float* res, float* y, int N, const float* nw, float eps, const char* pf,
           size_t pf_bytes, cudaStream_t st) {
  const DrbDevice& dev = drb_device(st);
  if (!dev.ready) return -2;
  if (N <= 0) return 0;
  drb_launch(k_gemv<K, U>, dim3(N < dev.sms ? N : dev.sms), dim3(THREADS), Shape<K, U>::BYTES, st, dev.pdl, W, S, x, res, y, N, nw, eps, pf, pf_bytes,
             dev.pdl ? HINT_SKIP : 0u, (unsigned)dev.sms);
  return 0;
}

template <int K, int U>
cudaError_t configure() {
  const cudaError_t e = cudaFuncSetAttribute(k_gemv<K, U>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<K, U>::BYTES);
  return e != cudaSuccess ? e : drb_carveout(k_gemv<K, U>);
}

}  // namespace q8

// ---- bf16 weights, K = 2048 ---------------------------------------------------------------------------------------------
// Consumer warps keep the fp32 activations in registers and take a row of the stage each: packed fp32 FMAs, one reduction.
namespace bf16 {

constexpr int K = 2048, CW = 8, NT = CW * 32, THREADS = NT + 32;
constexpr int ROW_BYTES = K * 2, STAGE_BYTES = CW * ROW_BYTES, STAGES = 3, NCH = K / 8 / 32;
constexpr size_t BYTES = 512 + K * 4 + (size_t)STAGES * STAGE_BYTES;
static_assert(BYTES <= BLOCK_BYTES, "two blocks per multiprocessor");

struct Ctl {
  uint64_t full[STAGES], empty[STAGES];
  float red[CW];
};
static_assert(sizeof(Ctl) <= 512, "control block");

DRB_DEV void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); }

__global__ void __launch_bounds__(THREADS, 2)
    k_gemv(const __nv_bfloat16* __restrict__ W, const float* __restrict__ x, float* __restrict__ y, int N, const float* __restrict__ nw, float eps,
           const char* pf, size_t pf_bytes, unsigned pf_skip, unsigned sms) {
  extern __shared__ __align__(128) unsigned char dyn[];
  Ctl& ctl = *reinterpret_cast<Ctl*>(dyn);
  float4* xs4 = reinterpret_cast<float4*>(dyn + 512);
  unsigned char* ring = dyn + 512 + K * 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned G = gridDim.x, b = blockIdx.x;
  const int u0 = (int)((long long)N * b / G), u1 = (int)((long long)N * (b + 1) / G);
  const int nchunks = (u1 - u0 + CW - 1) / CW;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(&ctl.full[s], 1), mbar_init(&ctl.empty[s], CW);
    mbar_fence_init();
  }
  __syncthreads();
  pdl_launch_dependents();

  if (warp == CW) {
    // ---------------- producer: weights are constants, so copies start before the dependency wait
    if (elect_one()) {
      for (int c = 0; c < nchunks; ++c) {
        const int s = c % STAGES, r0 = u0 + c * CW;
        if (c >= STAGES && !mbar_wait_hot(&ctl.empty[s], ((c / STAGES) - 1) & 1, DRB_ERR_EMPTY_WAIT)) return;
        const unsigned bytes = (unsigned)(min(CW, u1 - r0) * ROW_BYTES);
        mbar_expect_tx(&ctl.full[s], bytes);
        bulk_g2s(ring + s * STAGE_BYTES, W + (size_t)r0 * K, bytes, &ctl.full[s]);
      }
      prefetch_hint(pf, pf_bytes, pf_skip, sms, b, G);
    }
    return;
  }

  // ---------------- consumers
  float4 wv[2], xv[2];
  if (nw && (lane & 7) == 0)
#pragma unroll
    for (int j = 0; j < 2; ++j) prefetch_line_l2(nw + 4 * (threadIdx.x + j * NT));
  pdl_wait();  // x comes from the previous kernel
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    xv[j] = __ldcg(reinterpret_cast<const float4*>(x) + threadIdx.x + j * NT);
    wv[j] = nw ? __ldcg(reinterpret_cast<const float4*>(nw) + threadIdx.x + j * NT) : make_float4(1.f, 1.f, 1.f, 1.f);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    xs4[swz4(threadIdx.x + j * NT)] = nw ? make_float4(xv[j].x * wv[j].x, xv[j].y * wv[j].y, xv[j].z * wv[j].z, xv[j].w * wv[j].w) : xv[j];
  if (nw) {  // 1 / rms joins at the end, as in the int8 form
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j) ss += xv[j].x * xv[j].x + xv[j].y * xv[j].y + xv[j].z * xv[j].z + xv[j].w * xv[j].w;
    ss = warp_sum(ss);
    if (lane == 0) ctl.red[warp] = ss;
  }
  consumer_sync();
  float inv = 1.f;
  if (nw) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < CW; ++w) t += ctl.red[w];
    inv = rsqrtf(t / K + eps);
  }
  unsigned long long xp[NCH * 4];
#pragma unroll
  for (int i = 0; i < NCH; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float4 v = xs4[swz4(2 * (lane + 32 * i) + e)];
      xp[i * 4 + 2 * e] = pack2(v.x, v.y), xp[i * 4 + 2 * e + 1] = pack2(v.z, v.w);
    }
  // after the first wait of this thread that ran out no later wait spins again: the error word is set, the results are void
  bool dead = false;
  for (int c = 0; c < nchunks; ++c) {
    const int s = c % STAGES, row = u0 + c * CW + warp;
    if (!dead) dead = !mbar_wait_hot(&ctl.full[s], (c / STAGES) & 1, DRB_ERR_FULL_WAIT);
    const unsigned char* rowp = ring + s * STAGE_BYTES + warp * ROW_BYTES;
    unsigned long long a0 = 0ull, a1 = 0ull;
    if (row < u1) {
#pragma unroll
      for (int i = 0; i < NCH; i += 2) {
        a0 = dot8_bf16(*reinterpret_cast<const uint4*>(rowp + 16 * (lane + 32 * i)), xp + i * 4, a0);
        a1 = dot8_bf16(*reinterpret_cast<const uint4*>(rowp + 16 * (lane + 32 * (i + 1))), xp + (i + 1) * 4, a1);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&ctl.empty[s]);
    float p0, p1, p2, p3;
    unpack2(a0, p0, p1);
    unpack2(a1, p2, p3);
    const float d = warp_sum((p0 + p1) + (p2 + p3));
    if (lane == 0 && row < u1) y[row] = d * inv;
  }
}

}  // namespace bf16

static cudaError_t configure_all() {
  cudaError_t e;
  if ((e = q8::configure<512, 1>()) != cudaSuccess) return e;
  if ((e = q8::configure<2048, 1>()) != cudaSuccess) return e;
  if ((e = q8::configure<4096, 1>()) != cudaSuccess) return e;
  if ((e = q8::configure<6144, 1>()) != cudaSuccess) return e;
  if ((e = q8::configure<8192, 1>()) != cudaSuccess) return e;
  if ((e = q8::configure<2048, 2>()) != cudaSuccess) return e;
  if ((e = q8::configure<4096, 2>()) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(bf16::k_gemv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bf16::BYTES)) != cudaSuccess) return e;
  return drb_carveout(bf16::k_gemv);
}

}  // namespace gemv

// y[n] = W[n] . rmsnorm?(x) (+ res[n]); y may alias res. K in {512, 2048, 4096, 6144, 8192}, else -1.
// Reference: kernels/drama.cu:283-294; src/ffi.rs:33-36.
extern "C" int dr_gemv_q8(const int8_t* W, const __half* S, const float* x, const float* res, float* y, int N, int K,
                          const float* nw, float eps, const char* pf, size_t pf_bytes, cudaStream_t st) {
  using namespace gemv::q8;
  switch (K) {
    case 512: return launch<512, 1>(W, S, x, res, y, N, nw, eps, pf, pf_bytes, st);
    case 2048: return launch<2048, 1>(W, S, x, res, y, N, nw, eps, pf, pf_bytes, st);
    case 4096: return launch<4096, 1>(W, S, x, res, y, N, nw, eps, pf, pf_bytes, st);
    case 6144: return launch<6144, 1>(W, S, x, res, y, N, nw, eps, pf, pf_bytes, st);
    case 8192: return launch<8192, 1>(W, S, x, res, y, N, nw, eps, pf, pf_bytes, st);
    default: return -1;
  }
}

// y[j] = silu(W[j] . x) * (W[I + j] . x), W is [2I, K]. K in {2048, 4096}, else -1.
// Reference: kernels/drama.cu:296-305; src/ffi.rs:37-39.
extern "C" int dr_gemv_q8_swiglu(const int8_t* W, const __half* S, const float* x, float* y, int I, int K, const float* nw,
                                 float eps, const char* pf, size_t pf_bytes, cudaStream_t st) {
  using namespace gemv::q8;
  switch (K) {
    case 2048: return launch<2048, 2>(W, S, x, nullptr, y, I, nw, eps, pf, pf_bytes, st);
    case 4096: return launch<4096, 2>(W, S, x, nullptr, y, I, nw, eps, pf, pf_bytes, st);
    default: return -1;
  }
}

// y[n] = W[n] . rmsnorm?(x) for bf16 weights. K == 2048, else -1.
// Reference: kernels/drama.cu:307-315; src/ffi.rs:40.
extern "C" int dr_gemv_bf16(const __nv_bfloat16* W, const float* x, float* y, int N, int K, const float* nw, float eps,
                            const char* pf, size_t pf_bytes, cudaStream_t st) {
  using namespace gemv::bf16;
  if (K != gemv::bf16::K) return -1;
  const DrbDevice& dev = drb_device(st);
  if (!dev.ready) return -2;
  if (N <= 0) return 0;
  drb_launch(k_gemv, dim3(N < dev.sms ? N : dev.sms), dim3(THREADS), BYTES, st, dev.pdl, W, x, y, N, nw, eps, pf, pf_bytes,
             dev.pdl ? gemv::HINT_SKIP : 0u, (unsigned)dev.sms);
  return 0;
}
