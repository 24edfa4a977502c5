// Prefill-side kernels of the MoE path: per-row routing bookkeeping (count / permute / combine and the fused
// grouping step), the launchers of the expert-grouped GEMMs (moe_prefill_tc.cuh), and the elementwise helpers the
// reference's prefill calls around cuBLAS (dequant_q8, f32_to_bf16, swiglu_rows, rmsnorm).
//
// Replaces kernels/drama.cu:744-968 and 1114-1202 of the reference, same C signatures
// (src/ffi.rs:61-77).
#pragma once

#include "common.cuh"
#include "moe_prefill_tc.cuh"
#include "router.cuh"

namespace pf {

constexpr int H = 2048, I = 512;

// ------------------------------------------------------------------------------------------
// bookkeeping

// Histogram of the chosen experts. Each block counts its 1024 pairs in shared memory and adds only its non-empty
// bins to the global counts: a few hundred global atomics per block instead of one per pair on a handful of hot
// addresses (with Zipf routing a fifth of all pairs name the same expert).
constexpr int CNT_BINS = 1024;
__global__ void __launch_bounds__(256) k_count(const int* __restrict__ idx, int n, int* __restrict__ counts) {
  pdl_wait();
  __shared__ int bins[CNT_BINS];
  for (int i = threadIdx.x; i < CNT_BINS; i += blockDim.x) bins[i] = 0;
  __syncthreads();
  const int base = blockIdx.x * 1024;
  int big[4], nbig = 0;  // experts beyond the shared bins go straight to global memory
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = base + j * 256 + threadIdx.x;
    if (i < n) {
      const int e = __ldg(idx + i);
      if (e < CNT_BINS) atomicAdd(&bins[e], 1);
      else big[nbig++] = e;
    }
  }
  for (int j = 0; j < nbig; ++j) atomicAdd(counts + big[j], 1);
  __syncthreads();
  for (int i = threadIdx.x; i < CNT_BINS; i += blockDim.x)
    if (bins[i]) atomicAdd(counts + i, bins[i]);
}

// One warp per (row, k) pair: lane 0 claims the next slot of the pair's expert, the warp copies the row with
// 16-byte accesses. Eight pairs per block.
__global__ void __launch_bounds__(256)
    k_permute(const int* __restrict__ idx, int pairs, int topk, const int* __restrict__ offsets, int* __restrict__ fill,
              int* __restrict__ slot_of, const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ xp, int Hd) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= pairs) return;
  int slot = 0;
  if (lane == 0) {
    const int e = __ldg(idx + i);
    slot = __ldg(offsets + e) + atomicAdd(fill + e, 1);
    slot_of[i] = slot;
  }
  slot = __shfl_sync(0xffffffffu, slot, 0);
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(i / topk) * Hd);
  uint4* dst = reinterpret_cast<uint4*>(xp + (size_t)slot * Hd);
  for (int c = lane; c < Hd / 8; c += 32) dst[c] = __ldg(src + c);
}

// Count, scan and slot assignment in ONE launch of one block (drb_moe_group): what the reference does with a count
// kernel, a download, a host scan, an upload, a memset and the permute kernel's atomics (src/engine.rs:565-580).
// counts[e], offsets[e] (exclusive scan), slot_of[pair] = offsets[e] + rank of the pair among its expert's pairs,
// row_of[slot] = pair / topk. The grouped GEMM reads its operand rows through row_of, so no permuted copy of the
// rows is ever written. e_lo / e_n restrict the grouping to experts [e_lo, e_lo + e_n) (an expert-parallel rank's
// slice; pairs of other experts get slot -1); local expert ids are e - e_lo.
constexpr int GRP_THREADS = 1024, GRP_MAX_E = 1024;
// With cap > 0 the pairs are what an expert-parallel rank received: `world` blocks of blk_rows rows of row_ints
// 32-bit words each; block b holds cap row slots followed by the cap expert ids of those rows (one int each, the
// region padded to whole rows). Pair j = (block j / cap, slot j % cap); its id is read from the block's id region,
// row_of[slot] is the row's index in the buffer (in rows), pair_of[slot] = j. cap = 0: idx is a plain array,
// row_of[slot] = pair / topk, pair_of is not written.
__global__ void __launch_bounds__(GRP_THREADS)
    k_group(const int* __restrict__ idx, int pairs, int topk, int e_lo, int e_n, int* __restrict__ counts,
            int* __restrict__ offsets, int* __restrict__ slot_of, int* __restrict__ row_of, int* __restrict__ pair_of,
            int cap, int blk_rows, int row_ints) {
  pdl_wait();
  __shared__ int cnt[GRP_MAX_E];
  __shared__ int offs[GRP_MAX_E];
  __shared__ int warp_tot[GRP_THREADS / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  auto expert_of = [&](int p) {
    if (cap <= 0) return __ldg(idx + p);
    const int b = p / cap, i = p - b * cap;
    return __ldcg(idx + ((size_t)b * blk_rows + cap) * row_ints + i);
  };
  for (int i = t; i < e_n; i += GRP_THREADS) cnt[i] = 0;
  __syncthreads();
  // rank of every pair among its expert's pairs (the order inside an expert is arbitrary: every slot is computed
  // independently and the combine step sums in a fixed order)
  for (int p = t; p < pairs; p += GRP_THREADS) {
    const int e = expert_of(p) - e_lo;
    slot_of[p] = (e >= 0 && e < e_n) ? atomicAdd(&cnt[e], 1) : -1;
  }
  __syncthreads();
  // exclusive scan of the counts: one value per thread (e_n <= 1024)
  const int c = t < e_n ? cnt[t] : 0;
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int v = warp_tot[lane], in2 = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, in2, o);
      if (lane >= o) in2 += u;
    }
    warp_tot[lane] = in2 - v;  // exclusive over the warps
  }
  __syncthreads();
  if (t < e_n) {
    const int o = warp_tot[warp] + incl - c;
    offs[t] = o;
    counts[t] = c;
    offsets[t] = o;
  }
  __syncthreads();
  for (int p = t; p < pairs; p += GRP_THREADS) {
    const int e = expert_of(p) - e_lo;
    if (e >= 0 && e < e_n) {
      const int slot = offs[e] + slot_of[p];
      slot_of[p] = slot;
      if (cap <= 0) {
        row_of[slot] = p / topk;
      } else {
        const int b = p / cap;
        row_of[slot] = b * blk_rows + (p - b * cap);
        pair_of[slot] = p;
      }
    }
  }
}

// Expert-parallel dispatch, sender side, step 1 (one block): every (row, k) pair gets a slot in the block of the rank
// that owns its expert. send is `world` blocks of blk_rows rows of row_ints words (layout as in k_group); the pair's
// local expert id goes to the block's id region, unused slots get the id `per` (one past the owner's last expert:
// the owner's grouping skips them). slot_of[pair] = owner * cap + slot (what the combine step indexes the returned
// results with), dst_row[pair] = the row of `send` that the pair's row must be copied to (-1: dropped).
// A pair that finds its block full is dropped, its slot_of points at a valid slot of the block, and *overflow is set:
// the step's result is then void and the caller must repeat it with a larger capacity. Nothing waits or faults.
// With `peers` (device array of every rank's receive buffer) block o is not a part of `send` but this rank's slot in
// peer o's receive buffer: the ids and rows are stored straight into the owner's memory over NVLink, and every
// thread fences at system scope after its stores (the flag that announces them is written by a later kernel).
__global__ void __launch_bounds__(GRP_THREADS)
    k_ep_plan(const int* __restrict__ idx, int pairs, int per, int world, int cap, int blk_rows, int row_ints,
              int* __restrict__ send_local, int* __restrict__ slot_of, int* __restrict__ dst_row, unsigned* __restrict__ overflow,
              int* const* __restrict__ peers, int rank) {
  pdl_wait();
  __shared__ int cnt[64];
  __shared__ int* blk[64];
  const int t = threadIdx.x;
  if (t < 64) cnt[t] = 0;
  if (t < world) blk[t] = peers ? peers[t] + (size_t)rank * blk_rows * row_ints : send_local + (size_t)t * blk_rows * row_ints;
  __syncthreads();
  for (int p = t; p < pairs; p += GRP_THREADS) {
    const int e = __ldg(idx + p);
    const int o = e / per;
    const int r = atomicAdd(&cnt[o], 1);
    if (r < cap) {
      blk[o][(size_t)cap * row_ints + r] = e - o * per;
      slot_of[p] = o * cap + r;
      dst_row[p] = o * blk_rows + r;
    } else {
      atomicExch(overflow, 1u);
      slot_of[p] = o * cap;
      dst_row[p] = -1;
    }
  }
  __syncthreads();
  for (int j = t; j < world * cap; j += GRP_THREADS) {
    const int o = j / cap, r = j - o * cap;
    if (r >= cnt[o]) blk[o][(size_t)cap * row_ints + r] = per;
  }
  if (peers) __threadfence_system();
}

// Step 2: one warp per pair copies its row (row_bytes each, 16-byte accesses) to its place in the send buffer.
__global__ void __launch_bounds__(256)
    k_ep_scatter(const unsigned char* __restrict__ rows, int pairs, int topk, const int* __restrict__ dst_row,
                 unsigned char* __restrict__ send, int row_bytes, unsigned char* const* __restrict__ peers, int rank, int blk_rows) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int p = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (p >= pairs) return;
  const int d = __ldg(dst_row + p);
  if (d < 0) return;
  const uint4* src = reinterpret_cast<const uint4*>(rows + (size_t)(p / topk) * row_bytes);
  uint4* dst;
  if (peers) {
    const int o = d / blk_rows;
    dst = reinterpret_cast<uint4*>(peers[o] + ((size_t)rank * blk_rows + (d - o * blk_rows)) * row_bytes);
  } else {
    dst = reinterpret_cast<uint4*>(send + (size_t)d * row_bytes);
  }
  for (int c = lane; c < row_bytes / 16; c += 32) dst[c] = __ldg(src + c);
  if (peers) __threadfence_system();
}

// The exchange of an expert-parallel step over NVLink peer stores (drb_ep_put / drb_ep_signal / drb_ep_wait): block p of
// this rank's send buffer goes straight into peer p's receive buffer, slot `rank`, with 16-byte stores; every
// writing thread fences at system scope after its stores, so that the flag the next kernel writes to the peer
// can only be seen after the data.
__global__ void __launch_bounds__(256)
    k_ep_put(const uint4* __restrict__ send, uint4* const* __restrict__ peer_recv, int rank, size_t block_vecs) {
  pdl_wait();
  const int p = blockIdx.y;
  const uint4* src = send + (size_t)p * block_vecs;
  uint4* dst = peer_recv[p] + (size_t)rank * block_vecs;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < block_vecs; i += (size_t)gridDim.x * blockDim.x) dst[i] = __ldg(src + i);
  __threadfence_system();
}

// ++*step; then peer p's flag word `rank` takes the new step number (one thread per peer).
__global__ void __launch_bounds__(64) k_ep_signal(unsigned* const* __restrict__ peer_flags, int world, int rank, unsigned* __restrict__ step) {
  pdl_wait();
  __shared__ unsigned now;
  if (threadIdx.x == 0) now = ++*step;
  __syncthreads();
  __threadfence_system();
  if ((int)threadIdx.x < world) {
    volatile unsigned* f = peer_flags[threadIdx.x] + rank;
    *f = now;
  }
}

// ++*step; then waits until every peer's flag has reached the new step number. Bounded: a peer that never signals
// costs `limit` polls, sets the error word and lets the step run on (its result is void).
__global__ void __launch_bounds__(64) k_ep_wait(const unsigned* __restrict__ flags, int world, unsigned* __restrict__ step, unsigned limit) {
  pdl_wait();
  __shared__ unsigned now;
  if (threadIdx.x == 0) now = ++*step;
  __syncthreads();
  if ((int)threadIdx.x < world) {
    const volatile unsigned* f = flags + threadIdx.x;
    unsigned it = 0;
    // signed distance: the counters wrap together
    while ((int)(*f - now) < 0) {
      if (++it >= limit) {
        atomicMax(&g_drb_error, (unsigned)DRB_ERR_GRID_WAIT);
        break;
      }
      if (it > 64) __nanosleep(it > 4096 ? 256 : 32);
    }
  }
  __threadfence_system();
}

// k_ep_signal and k_ep_wait in one launch: announce this rank's stores to every peer, then wait for every peer's.
__global__ void __launch_bounds__(64)
    k_ep_sync(unsigned* const* __restrict__ peer_flags, const unsigned* __restrict__ flags, int world, int rank, unsigned* __restrict__ steps,
              unsigned limit) {
  pdl_wait();
  __shared__ unsigned now_s, now_w;
  if (threadIdx.x == 0) now_s = ++steps[0], now_w = ++steps[1];
  __syncthreads();
  __threadfence_system();
  if ((int)threadIdx.x < world) {
    volatile unsigned* out = peer_flags[threadIdx.x] + rank;
    *out = now_s;
    const volatile unsigned* f = flags + threadIdx.x;
    unsigned it = 0;
    while ((int)(*f - now_w) < 0) {
      if (++it >= limit) {
        atomicMax(&g_drb_error, (unsigned)DRB_ERR_GRID_WAIT);
        break;
      }
      if (it > 64) __nanosleep(it > 4096 ? 256 : 32);
    }
  }
  __threadfence_system();
}

// x[r] += sigmoid(sgate[r]) * shared[r] + sum_k w[r,k] * Y[slot_of[r,k]], k ascending (fixed order, so
// the result does not depend on how slots were handed out). Two forms, one float4 of 1024 columns per thread.
//
// Top-8: block (r, c) takes rows r, r + gridDim.x, ... Bound by Y's bytes from L2 or HBM; all of a thread's rows are requested before the
// first is used (in a loop over a runtime topk every row waited for the one before, 13 us at 300 rows instead of 5). A row's
// slots, weights and gate lie spread over the lanes of each warp and are fetched a row ahead: behind them its data would wait for two
// trips instead of one. 2048 rows 44.5 -> 35.8 us, 300 rows 4.3 -> 3.5, against a block per row.
constexpr int CMB_TOPK = 8, CMB_BLOCKS = 4;  // resident blocks per multiprocessor
__global__ void __launch_bounds__(256, CMB_BLOCKS)
    k_combine8(float* __restrict__ x, const float* __restrict__ Y, const int* __restrict__ slot_of,
               const float* __restrict__ wts, const float* __restrict__ sgate, const float* __restrict__ shared, int rows, int Hd) {
  constexpr int TK = CMB_TOPK;
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, first = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (first - 4 * lane >= Hd) return;
  const bool in = first < Hd;
  const int c = in ? first : Hd - 4;  // whole warps stay for the shuffles
  auto head = [&](unsigned r) -> int {  // lane k < TK the slot of pair k, TK + k its weight, 2 TK the gate
    if (lane < TK) return __ldcg(slot_of + (size_t)r * TK + lane);
    if (lane < 2 * TK) return __float_as_int(__ldcg(wts + (size_t)r * TK + lane - TK));
    return __float_as_int(__ldcg(sgate + r));
  };
  const unsigned n = rows;  // unsigned: a stride past the last row may leave int's range
  int next = head(blockIdx.x);
  for (unsigned r = blockIdx.x; r < n; r += gridDim.x) {
    const int now = next;
    if (r + gridDim.x < n) next = head(r + gridDim.x);
    float4* xo = reinterpret_cast<float4*>(x + (size_t)r * Hd + c);
    const float4 sh = __ldcg(reinterpret_cast<const float4*>(shared + (size_t)r * Hd + c));
    float4 o = __ldcg(xo), v[TK];
#pragma unroll
    for (int k = 0; k < TK; ++k) v[k] = __ldcg(reinterpret_cast<const float4*>(Y + (size_t)__shfl_sync(0xffffffffu, now, k) * Hd + c));
    const float sg = sigmoid_f(__int_as_float(__shfl_sync(0xffffffffu, now, 2 * TK)));
    float4 acc = make_float4(sg * sh.x, sg * sh.y, sg * sh.z, sg * sh.w);
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      const float w = __int_as_float(__shfl_sync(0xffffffffu, now, TK + k));
      acc.x += w * v[k].x, acc.y += w * v[k].y, acc.z += w * v[k].z, acc.w += w * v[k].w;
    }
    o.x += acc.x, o.y += acc.y, o.z += acc.z, o.w += acc.w;
    if (in) *xo = o;
  }
}

// Any topk: block (r, c) takes row r. With many rows eight resident blocks per multiprocessor cover one another's trips; walking over rows in
// four of them, as above, lost (H = 2048, 2048 rows of 2, 16, 32 pairs: 8.3, 61, 110 us, and 12.0, 83, 153). FEW: at most three blocks per
// multiprocessor, where the chain of trips is what there is: four pairs' slots, then four rows (one row of 16, 32 pairs 4.1, 6.6 -> 2.9, 4.2 us;
// 64 rows of 16 4.3 -> 3.1). With four, 290 rows of 4 to 16
// took 20 to 30 % longer so.
template <bool FEW>
__global__ void __launch_bounds__(256, FEW ? 6 : 8)
    k_combine(float* __restrict__ x, const float* __restrict__ Y, const int* __restrict__ slot_of, const float* __restrict__ wts,
              const float* __restrict__ sgate, const float* __restrict__ shared, int topk, int Hd) {
  pdl_wait();
  pdl_launch_dependents();
  const int r = blockIdx.x, c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (c >= Hd) return;
  float4* xo = reinterpret_cast<float4*>(x + (size_t)r * Hd + c);
  const float gate = __ldcg(sgate + r);
  const float4 sh = __ldcg(reinterpret_cast<const float4*>(shared + (size_t)r * Hd + c));
  float4 o = __ldcg(xo);
  const float sg = sigmoid_f(gate);
  float4 acc = make_float4(sg * sh.x, sg * sh.y, sg * sh.z, sg * sh.w);
  const int* slots = slot_of + (size_t)r * topk;
  const float* weights = wts + (size_t)r * topk;
  auto row = [&](int slot) { return __ldcg(reinterpret_cast<const float4*>(Y + (size_t)slot * Hd + c)); };
  auto add = [&](float w, const float4& v) { acc.x += w * v.x, acc.y += w * v.y, acc.z += w * v.z, acc.w += w * v.w; };
  if (FEW) {
    int k = 0;
    for (; k + 4 <= topk; k += 4) {
      int s[4];
      float w[4];
      float4 v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = __ldcg(slots + k + i), w[i] = __ldcg(weights + k + i);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = row(s[i]);
#pragma unroll
      for (int i = 0; i < 4; ++i) add(w[i], v[i]);
    }
#pragma unroll 1
    for (; k < topk; ++k) add(__ldcg(weights + k), row(__ldcg(slots + k)));
  } else {
    for (int k = 0; k < topk; ++k) add(__ldcg(wts + (size_t)r * topk + k), row(__ldcg(slot_of + (size_t)r * topk + k)));
  }
  o.x += acc.x, o.y += acc.y, o.z += acc.z, o.w += acc.w;
  *xo = o;
}

// ------------------------------------------------------------------------------------------
// elementwise

__global__ void k_dequant_q8(const int8_t* __restrict__ W, const __half* __restrict__ S, __nv_bfloat16* __restrict__ out,
                             size_t n_elems, int K) {
  pdl_wait();
  const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 16;
  if (i >= n_elems) return;
  const size_t row = i / K, col = i % K;
  const float s = __half2float(S[row * (K / 128) + col / 128]);
  const uint4 v = *reinterpret_cast<const uint4*>(W + i);
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
  __align__(16) __nv_bfloat16 o[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) o[j] = __float2bfloat16((float)(int8_t)(u[j >> 2] >> (8 * (j & 3))) * s);
  reinterpret_cast<uint4*>(out + i)[0] = reinterpret_cast<uint4*>(o)[0];
  reinterpret_cast<uint4*>(out + i)[1] = reinterpret_cast<uint4*>(o)[1];
}

__global__ void k_f32_to_bf16(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, size_t n) {
  pdl_wait();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16(x[i]);
}

// y[r, j] = silu(h[r, j]) * h[r, I + j] in bf16; h has row stride 2I.
__global__ void k_swiglu_rows(const float* __restrict__ h, __nv_bfloat16* __restrict__ y, int rows, int Id) {
  pdl_wait();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)rows * Id) return;
  const size_t r = i / Id, j = i % Id;
  y[i] = __float2bfloat16(silu_f(h[r * 2 * Id + j]) * h[r * 2 * Id + Id + j]);
}

// Row-wise RMSNorm ("+1" already folded into w). Writes f32 and/or a 16-bit copy: bf16, or (F16) fp16 clamped to its range.
template <bool F16>
__global__ void __launch_bounds__(256)
    k_rmsnorm(const float* __restrict__ x, const float* __restrict__ w, float* y, __nv_bfloat16* yb, int D, float eps) {
  pdl_wait();
  __shared__ float red[9];
  const float* xr = x + (size_t)blockIdx.x * D;
  float ss = 0.f;
  for (int i = threadIdx.x; i < D; i += blockDim.x) ss += xr[i] * xr[i];
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < 8; ++i) t += red[i];
    red[8] = rsqrtf(t / D + eps);
  }
  __syncthreads();
  const float inv = red[8];
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    const float v = xr[i] * inv * w[i];
    if (y) y[(size_t)blockIdx.x * D + i] = v;
    if (yb) {
      if (F16) reinterpret_cast<__half*>(yb)[(size_t)blockIdx.x * D + i] = tc::f2h_sat(v);
      else yb[(size_t)blockIdx.x * D + i] = __float2bfloat16(v);
    }
  }
}

// Router logits whose value for a row does not depend on how many rows are computed together: every (row, output) sum is
// formed in one fixed order whatever the launch's shape. A library GEMM picks its kernel by the batch size (measured:
// logits of the same row differ by 1.2e-6 between a batch of 300 and a batch of 38), which would let the routing of
// a row depend on how the rows are spread over the GPUs.
//
// A block takes 16 rows and the 8-output tiles blockIdx.y, blockIdx.y + gridDim.y, ...; warp w takes inputs [256 w, +256) of
// all of them on mma.sync m16n8k16 bf16, with the rows as the A operand in its registers for the whole launch. The weights are
// bf16 already; an fp16 row value (eleven bits) is the exact sum of two bf16 values, and the low part's products are the
// addend of the high part's. Every instruction starts from zero and its sixteen products join one of a warp's four running sums by
// an fp32 addition, so nothing is lost to the tensor core's own accumulation over long sums; the running sums and then the eight
// warps' sums are added as a tree. Relative error against fp64 (2-norm, 300 x 257 logits): fp16 rows 8.4e-8, bf16 rows 7.5e-8 (with
// one running sum and the warps one behind the other 1.04e-7 and 9.4e-8; as a chain of fp32 FMAs 1.08e-7 and 8.0e-8).
// Which input a lane takes as which of an instruction's sixteen is the same permutation on both sides, chosen so that a lane's
// share of two instructions is one 16-byte load.
// Bound by the weights' way from L2 (1 MB per 16 rows, 64 bytes per clock at the instruction rate); at few rows by latency.
// SRC: what the rows come from. LOGITS_NORM: fp32 rows, RMS-normalised here (sums in k_rmsnorm's order) and rounded to fp16;
// blocks with y = 0 also store them. LOGITS_F16 / LOGITS_BF16: 16-bit rows as they are.
constexpr int RL_K = 2048, RL_WARPS = 8, RL_ROWS = 16, RL_TILE = 8;
constexpr int RL_SEG = RL_K / RL_WARPS;                 // inputs per warp
constexpr int RL_STRIDE = RL_K * 2 + 64;                // bytes per staged row: the fragments' loads meet no bank twice
constexpr int RL_STAGE = RL_ROWS * RL_STRIDE;
constexpr int RL_PART = RL_ROWS * RL_TILE;              // floats per warp and tile
enum LogitsSrc { LOGITS_NORM, LOGITS_F16, LOGITS_BF16 };
constexpr size_t logits_smem(int tiles) { return RL_STAGE + (size_t)tiles * RL_WARPS * RL_PART * 4; }
constexpr int RL_MAX_TILES = (232448 - RL_STAGE) / (RL_WARPS * RL_PART * 4);  // tiles of one block

DRB_DEV void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

// Two fp16 values as the sum of two pairs of bf16 values; exact.
DRB_DEV void split_f16x2(uint32_t v, uint32_t& hi, uint32_t& lo) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
  const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(f.x - __uint_as_float(hi << 16), f.y - __uint_as_float(hi & 0xffff0000u));
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

template <int SRC>
__global__ void __launch_bounds__(RL_WARPS * 32, 1)
    k_router_logits(const void* __restrict__ src, const float* __restrict__ nw, float eps, __half* __restrict__ rows16,
                    const __nv_bfloat16* __restrict__ w, const float* bias, float* logits, int rows, int e1, float beta, int* __restrict__ zero, int n_zero) {
  extern __shared__ __align__(16) unsigned char dyn[];
  float* part = reinterpret_cast<float*>(dyn + RL_STAGE);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int r0 = blockIdx.x * RL_ROWS, nr = min(RL_ROWS, rows - r0);
  const int tiles = (e1 + RL_TILE - 1) / RL_TILE;
  constexpr int LOADS = RL_SEG / 32;  // 16-byte loads of a lane per row and segment
  const int k0 = warp * RL_SEG + 8 * q;
  uint4 b[LOADS];
  auto fetch = [&](int tile) {
    const uint4* p = reinterpret_cast<const uint4*>(w + (size_t)min(tile * RL_TILE + g, e1 - 1) * RL_K + k0);
#pragma unroll
    for (int j = 0; j < LOADS; ++j) b[j] = __ldg(p + 4 * j);
  };
  // the row groups start at different tiles: in step, all of them would ask L2 for the same lines at once
  const int mine = (tiles - (int)blockIdx.y + (int)gridDim.y - 1) / (int)gridDim.y;  // tiles of this block, at least one
  int t = (int)(blockIdx.x % (unsigned)mine);
  // the first tile's weights as far as L2: they too may be the work of the launch before
  prefetch_line_l2(w + (size_t)min((int)(blockIdx.y + t * gridDim.y) * RL_TILE + g, e1 - 1) * RL_K + warp * RL_SEG + 64 * q);
  pdl_launch_dependents();
  pdl_wait();
  fetch(blockIdx.y + t * gridDim.y);
  if (zero && blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = threadIdx.x; i < n_zero; i += blockDim.x) zero[i] = 0;
  constexpr int RPW = RL_ROWS / RL_WARPS;  // rows warp + RL_WARPS p; all requested before the first is used
  if (SRC == LOGITS_NORM) {
    // k_rmsnorm's sums: its thread t adds the squares of inputs t + 256 i in turn; each warp's 32 threads by butterfly, the
    // eight warps in order
    float v[RPW][RL_K / 32];
#pragma unroll
    for (int p = 0; p < RPW; ++p) {
      const float* xr = static_cast<const float*>(src) + (size_t)(r0 + warp + RL_WARPS * p) * RL_K;
      const bool in = warp + RL_WARPS * p < nr;
#pragma unroll
      for (int i = 0; i < RL_K / 32; ++i) v[p][i] = in ? __ldcg(xr + 32 * i + lane) : 0.f;
    }
    float inv[RPW];
#pragma unroll
    for (int p = 0; p < RPW; ++p) {
      float t = 0.f;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < RL_K / 256; ++i) ss += v[p][8 * i + s] * v[p][8 * i + s];
        t += warp_sum(ss);
      }
      inv[p] = rsqrtf(t / RL_K + eps);
    }
#pragma unroll
    for (int i = 0; i < RL_K / 32; ++i) {
      const int k = 32 * i + lane;
      const float f = __ldg(nw + k);
#pragma unroll
      for (int p = 0; p < RPW; ++p)
        reinterpret_cast<__half*>(dyn + (warp + RL_WARPS * p) * RL_STRIDE)[k] =
            warp + RL_WARPS * p < nr ? tc::f2h_sat(v[p][i] * inv[p] * f) : __half(0.f);
    }
  } else {
#pragma unroll
    for (int p = 0; p < RPW; ++p) {
      const int r = warp + RL_WARPS * p;
      const uint4* xr = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(src) + (size_t)(r0 + r) * RL_K);
#pragma unroll
      for (int i = 0; i < RL_K / 256; ++i)
        reinterpret_cast<uint4*>(dyn + r * RL_STRIDE)[32 * i + lane] = r < nr ? __ldcg(xr + 32 * i + lane) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if (SRC == LOGITS_NORM && blockIdx.y == 0) {
    __syncwarp();
#pragma unroll
    for (int p = 0; p < RPW; ++p) {
      const int r = warp + RL_WARPS * p;
      uint4* out = reinterpret_cast<uint4*>(rows16 + (size_t)(r0 + r) * RL_K);
      if (r < nr)
#pragma unroll
        for (int i = 0; i < RL_K / 256; ++i) out[32 * i + lane] = reinterpret_cast<const uint4*>(dyn + r * RL_STRIDE)[32 * i + lane];
    }
  }
  __syncthreads();
  // this warp's A fragments, two instructions per 16-byte piece: rows g and g + 8
  uint32_t ah[2 * LOADS][4], al[2 * LOADS][4];
#pragma unroll
  for (int j = 0; j < LOADS; ++j) {
    const uint4 u = *reinterpret_cast<const uint4*>(dyn + g * RL_STRIDE + 2 * (k0 + 32 * j));
    const uint4 v = *reinterpret_cast<const uint4*>(dyn + (g + 8) * RL_STRIDE + 2 * (k0 + 32 * j));
    const uint32_t f[2][4] = {{u.x, v.x, u.y, v.y}, {u.z, v.z, u.w, v.w}};
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (SRC == LOGITS_BF16) ah[2 * j + s][i] = f[s][i];
        else split_f16x2(f[s][i], ah[2 * j + s][i], al[2 * j + s][i]);
      }
  }
  for (int n = 0; n < mine; ++n) {
    uint4 c[LOADS];
#pragma unroll
    for (int j = 0; j < LOADS; ++j) c[j] = b[j];
    const int now = t;
    if (++t == mine) t = 0;
    if (n + 1 < mine) fetch(blockIdx.y + t * gridDim.y);
    float acc[4][4] = {};
#pragma unroll
    for (int j = 0; j < LOADS; ++j) {
      const uint32_t f[4] = {c[j].x, c[j].y, c[j].z, c[j].w};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const float z[4] = {0.f, 0.f, 0.f, 0.f};
        float d[4];
        if (SRC == LOGITS_BF16) {
          mma_bf16(d, ah[2 * j + s], f[2 * s], f[2 * s + 1], z);
        } else {
          float l[4];
          mma_bf16(l, al[2 * j + s], f[2 * s], f[2 * s + 1], z);
          mma_bf16(d, ah[2 * j + s], f[2 * s], f[2 * s + 1], l);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[(2 * j + s) & 3][i] += d[i];
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[0][i] = (acc[0][i] + acc[2][i]) + (acc[1][i] + acc[3][i]);
    float* p = part + (now * RL_WARPS + warp) * RL_PART + g * RL_TILE + 2 * q;
    *reinterpret_cast<float2*>(p) = make_float2(acc[0][0], acc[0][1]);
    *reinterpret_cast<float2*>(p + 8 * RL_TILE) = make_float2(acc[0][2], acc[0][3]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < mine * RL_PART; i += RL_WARPS * 32) {
    const int m = i / RL_PART, at = i % RL_PART, r = at / RL_TILE, o = (blockIdx.y + m * gridDim.y) * RL_TILE + at % RL_TILE;
    if (o >= e1 || r >= nr) continue;
    float u[RL_WARPS];
#pragma unroll
    for (int s = 0; s < RL_WARPS; ++s) u[s] = part[(m * RL_WARPS + s) * RL_PART + at];
    const float v = ((u[0] + u[1]) + (u[2] + u[3])) + ((u[4] + u[5]) + (u[6] + u[7]));
    const size_t at_out = (size_t)(r0 + r) * e1 + o;
    logits[at_out] = beta != 0.f ? fmaf(beta, bias[at_out], v) : v;
  }
}

// As many blocks side by side as share out the tiles of all the row groups over the multiprocessors, at least as many as the
// partial sums of a block's tiles need to fit into its shared memory.
template <int SRC>
static int launch_logits(const void* src, const float* nw, float eps, __half* rows16, const __nv_bfloat16* w, const float* bias, float* logits,
                         int rows, int e1, float beta, int* zero, int n_zero, cudaStream_t st) {
  const DrbDevice& dev = drb_device(st);
  if (!dev.ready) return -2;
  const int gx = (rows + RL_ROWS - 1) / RL_ROWS, tiles = (e1 + RL_TILE - 1) / RL_TILE;
  const int gy = min(tiles, max((tiles + RL_MAX_TILES - 1) / RL_MAX_TILES, dev.sms / gx));
  drb_launch(k_router_logits<SRC>, dim3(gx, gy), dim3(RL_WARPS * 32), logits_smem((tiles + gy - 1) / gy), st, dev.pdl, src, nw, eps, rows16, w, bias,
             logits, rows, e1, beta, zero, n_zero);
  return 0;
}

template <int SRC>
static cudaError_t configure_logits() {
  const cudaError_t e = cudaFuncSetAttribute(k_router_logits<SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)logits_smem(RL_MAX_TILES));
  return e != cudaSuccess ? e : drb_carveout(k_router_logits<SRC>);
}

// Two warps per row, behind the routing: the row's slots (the exclusive scan of the expert counts, which every block makes for
// itself, plus the rank that router::k_moe_topk took with its count) and its copies for the grouped GEMMs: one per chosen
// expert in slot order, one for the shared expert. Grouping and copying in one launch over the whole chip: as a launch
// of one block and one of its own they took 7 + 6 us at 300 rows, 25 + 18 us at 2048.
constexpr int SC_ROWS = 2, SC_THREADS = SC_ROWS * 64;  // two warps per row, each half of it
__global__ void __launch_bounds__(SC_THREADS)
    k_scatter_rows(const __half* __restrict__ rows16, const int* __restrict__ idx, int rows, int topk, const int* __restrict__ counts, int E,
                   int* __restrict__ offsets, int* __restrict__ slot_of, const int* __restrict__ rank, int* __restrict__ row_of,
                   unsigned char* __restrict__ dst, unsigned char* __restrict__ sh_dst) {
  __shared__ int offs[256], tot[SC_THREADS / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  constexpr int CPT = 256 / SC_THREADS, PER = H / 8 / 64;
  int r = blockIdx.x * SC_ROWS + (warp >> 1);
  auto load = [&](int row, uint4(&v)[PER]) {
    const uint4* src = reinterpret_cast<const uint4*>(rows16 + (size_t)row * H) + (warp & 1) * 32 * PER;
#pragma unroll
    for (int j = 0; j < PER; ++j) v[j] = row < rows ? __ldcg(src + 32 * j + lane) : make_uint4(0u, 0u, 0u, 0u);
  };
  uint4 v[PER];
  load(r, v);
  int c[CPT], sum = 0;
#pragma unroll
  for (int j = 0; j < CPT; ++j) c[j] = sum, sum += CPT * t + j < E ? __ldcg(counts + CPT * t + j) : 0;
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) tot[warp] = incl;
  __syncthreads();
  int before = incl - sum;
  for (int q = 0; q < warp; ++q) before += tot[q];
#pragma unroll
  for (int j = 0; j < CPT; ++j) {
    offs[CPT * t + j] = before + c[j];
    if (blockIdx.x == 0 && CPT * t + j < E) offsets[CPT * t + j] = before + c[j];
  }
  __syncthreads();
  for (; r < rows; r += gridDim.x * SC_ROWS) {
    int slot = 0;
    if (lane < topk) {
      const int p = r * topk + lane;
      slot = offs[__ldcg(idx + p)] + __ldcg(rank + p);
      if ((warp & 1) == 0) {
        slot_of[p] = slot;
        row_of[slot] = r;
      }
    }
#pragma unroll
    for (int j = 0; j < PER; ++j)
      v[j] = make_uint4(prmt(v[j].x, v[j].z, 0x5410u), prmt(v[j].x, v[j].z, 0x7632u), prmt(v[j].y, v[j].w, 0x5410u), prmt(v[j].y, v[j].w, 0x7632u));
    for (int k = 0; k <= topk; ++k) {
      const int to = __shfl_sync(0xffffffffu, slot, k & 31);
      uint4* out = reinterpret_cast<uint4*>(k < topk ? dst + (size_t)to * pft::TOKEN_STRIDE : sh_dst + (size_t)r * pft::TOKEN_STRIDE) + (warp & 1) * 32 * PER;
#pragma unroll
      for (int j = 0; j < PER; ++j) out[32 * j + lane] = v[j];
    }
    load(r + gridDim.x * SC_ROWS, v);
  }
}

// router::k_moe_topk and k_scatter_rows in one launch for up to 32 rows, where a launch's way costs more than its work. Block r
// copies row r; every block forms the routing of all the rows for itself, a warp per row, so nothing crosses blocks: the experts'
// rows are bit masks, a pair's rank is the number of rows before it in its expert's mask.
// A whole call: 49.3 -> 46.5 us at 5 rows, 73.6 -> 68.8 at 16, 77.8 -> 75.7 at 20, 91.8 -> 90.6 at 32; the redundant part grows with the
// rows, and beyond 32 a block has no warp per row.
constexpr int FEW_ROWS = 32, FEW_MIN_THREADS = 512;  // blocks of 32 threads per row, but at least so many for the copies
__global__ void __launch_bounds__(FEW_ROWS * 32)
    k_route_few(const float* __restrict__ logits, const __half* __restrict__ rows16, int rows, int E, int topk, int* __restrict__ idx,
                float* __restrict__ wts, float* __restrict__ sgate, int* __restrict__ counts, int* __restrict__ offsets, int* __restrict__ slot_of,
                int* __restrict__ row_of, unsigned char* __restrict__ dst, unsigned char* __restrict__ sh_dst) {
  __shared__ unsigned mask[256];
  __shared__ int offs[256], tot[8], to[32];
  pdl_launch_dependents();
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, row = blockIdx.x;
  if (t < 256) mask[t] = 0u;
  __syncthreads();
  pdl_wait();
  constexpr int PIECES = H / 8;  // 16-byte pieces of a row; threads t, t + 256, ... hold piece t and share out the copies
  uint4 v = __ldcg(reinterpret_cast<const uint4*>(rows16 + (size_t)row * H) + (t & (PIECES - 1)));
  int mine = 0;  // lane k < topk of warp r: the k-th expert of row r
  if (warp < rows) {
    const float* l = logits + (size_t)warp * (E + 1);
    float w;
    mine = router::route_row([&](int e) { return __ldcg(l + e); }, E, topk, lane, w);
    if (lane < topk) {
      atomicOr(&mask[mine], 1u << warp);
      if (warp == row) idx[row * topk + lane] = mine, wts[row * topk + lane] = w;
    }
    if (warp == row && lane == 0) sgate[row] = __ldcg(l + E);
  }
  __syncthreads();
  const int c = t < 256 ? __popc(mask[t]) : 0;
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31 && warp < 8) tot[warp] = incl;
  __syncthreads();
  if (t < 256) {
    int before = incl - c;
    for (int q = 0; q < warp; ++q) before += tot[q];
    offs[t] = before;
    if (row == 0 && t < E) offsets[t] = before, counts[t] = c;
  }
  __syncthreads();
  if (warp == row && lane < topk) {
    const int slot = offs[mine] + __popc(mask[mine] & ((1u << row) - 1u));
    to[lane] = slot, slot_of[row * topk + lane] = slot, row_of[slot] = row;
  }
  __syncthreads();
  v = make_uint4(prmt(v.x, v.z, 0x5410u), prmt(v.x, v.z, 0x7632u), prmt(v.y, v.w, 0x5410u), prmt(v.y, v.w, 0x7632u));
  for (int k = t / PIECES; k <= topk; k += blockDim.x / PIECES)
    reinterpret_cast<uint4*>(k < topk ? dst + (size_t)to[k] * pft::TOKEN_STRIDE : sh_dst + (size_t)row * pft::TOKEN_STRIDE)[t & (PIECES - 1)] = v;
}

// offsets[e] = sum of counts[0..e): the exclusive scan the reference does on the host between two launches
// (src/engine.rs:567-574). One block, any number of experts.
__global__ void __launch_bounds__(256) k_offsets(const int* __restrict__ counts, int E, int* __restrict__ offsets) {
  pdl_wait();
  __shared__ int warp_tot[8];
  __shared__ int carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < E; base += 256) {
    const int i = base + threadIdx.x;
    const int c = i < E ? counts[i] : 0;
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int before = carry;
    for (int w = 0; w < warp; ++w) before += warp_tot[w];
    if (i < E) offsets[i] = before + incl - c;
    __syncthreads();
    if (threadIdx.x == 255) carry = before + incl;
    __syncthreads();
  }
}

static cudaError_t configure_all() {
  cudaError_t e;
  if ((e = drb_carveout(k_offsets)) != cudaSuccess) return e;
  if ((e = configure_logits<LOGITS_NORM>()) != cudaSuccess) return e;
  if ((e = configure_logits<LOGITS_F16>()) != cudaSuccess) return e;
  if ((e = configure_logits<LOGITS_BF16>()) != cudaSuccess) return e;
  if ((e = drb_carveout(k_scatter_rows)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_route_few)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_count)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_permute)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_combine8)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_combine<true>)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_combine<false>)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_group)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_ep_plan)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_ep_scatter)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_ep_put)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_dequant_q8)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_f32_to_bf16)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_swiglu_rows)) != cudaSuccess) return e;
  if ((e = drb_carveout(k_rmsnorm<true>)) != cudaSuccess) return e;
  return drb_carveout(k_rmsnorm<false>);
}

}  // namespace pf

// Reference: kernels/drama.cu:750-753; src/ffi.rs:65. counts must be zeroed by the caller.
extern "C" int dr_moe_count(const int* idx, int n, int* counts, cudaStream_t st) {
  if (n <= 0) return 0;
  pf::k_count<<<(n + 1023) / 1024, 256, 0, st>>>(idx, n, counts);
  return 0;
}

// No counterpart in the reference, which downloads the counts and scans them on the host (src/engine.rs:567-574):
// with this call the prefill sequence needs no host round trip and can be captured in a graph.
extern "C" int drb_moe_offsets(const int* counts, int e, int* offsets, cudaStream_t st) {
  if (e <= 0) return 0;
  pf::k_offsets<<<1, 256, 0, st>>>(counts, e, offsets);
  return 0;
}

// logits [rows, e1] = xb [rows, h] . w [e1, h]^T + beta * logits, with per-row results that do not depend on `rows`
// (see k_router_logits). The reference computes these logits with cublasGemmEx (src/engine.rs:554); this call is for
// hosts that spread rows over several GPUs and need the same routing at every split. h == 2048, else -1.
extern "C" int drb_router_logits(const __nv_bfloat16* xb, const __nv_bfloat16* w, float* logits, int rows, int e1, int h,
                                 float beta, cudaStream_t st) {
  if (h != pf::RL_K) return -1;
  if (rows <= 0 || e1 <= 0) return 0;
  return pf::launch_logits<pf::LOGITS_BF16>(xb, nullptr, 0.f, nullptr, w, logits, logits, rows, e1, beta, nullptr, 0, st);
}

// The two calls above for rows kept in fp16 (no counterpart in the reference, whose prefill rounds the normalised rows
// to bf16: src/engine.rs:499): drb_rmsnorm_f16 writes the normalised rows as fp16 (clamped to +-65504),
// drb_router_logits_f16 reads them. With drb_moe_prefill_block(x_f16 = 1) the whole block then works on rows with
// eleven significant bits instead of eight.
extern "C" int drb_rmsnorm_f16(const float* x, const float* w, __half* yh, int rows, int D, float eps, cudaStream_t st) {
  if (rows <= 0) return 0;
  pf::k_rmsnorm<true><<<rows, 256, 0, st>>>(x, w, nullptr, reinterpret_cast<__nv_bfloat16*>(yh), D, eps);
  return 0;
}
extern "C" int drb_router_logits_f16(const __half* xh, const __nv_bfloat16* w, float* logits, int rows, int e1, int h, float beta,
                                     cudaStream_t st) {
  if (h != pf::RL_K) return -1;
  if (rows <= 0 || e1 <= 0) return 0;
  return pf::launch_logits<pf::LOGITS_F16>(xh, nullptr, 0.f, nullptr, w, logits, logits, rows, e1, beta, nullptr, 0, st);
}

// Reference: kernels/drama.cu:774-778; src/ffi.rs:66-69. fill must be zeroed by the caller.
extern "C" int dr_moe_permute(const int* idx, int rows, int topk, const int* offsets, int* fill, int* slot_of,
                              const __nv_bfloat16* x, __nv_bfloat16* xp, int H, cudaStream_t st) {
  if (H % 8 != 0) return -1;
  if (rows * topk <= 0) return 0;
  pf::k_permute<<<(rows * topk + 7) / 8, 256, 0, st>>>(idx, rows * topk, topk, offsets, fill, slot_of, x, xp, H);
  return 0;
}

// Reference: kernels/drama.cu:793-797; src/ffi.rs:70-73.
extern "C" int dr_moe_combine(float* x, const float* Y, const int* slot_of, const float* wts, const float* sgate,
                              const float* shared, int rows, int topk, int H, cudaStream_t st) {
  if (H % 4 != 0) return -1;
  if (rows <= 0 || H <= 0) return 0;
  const DrbDevice& dev = drb_device(st);
  const int gy = (H + 1023) / 1024;
  if (topk == pf::CMB_TOPK) {
    const int gx = max(1, pf::CMB_BLOCKS * (dev.ready ? dev.sms : 1) / gy);  // what is resident at once
    drb_launch(pf::k_combine8, dim3(rows < gx ? rows : gx, gy), dim3(256), 0, st, dev.ready && dev.pdl, x, Y, slot_of, wts, sgate, shared, rows, H);
  } else {
    const bool few = topk >= 4 && (long long)rows * gy <= 3 * dev.sms;
    drb_launch(few ? pf::k_combine<true> : pf::k_combine<false>, dim3(rows, gy), dim3(256), 0, st, dev.ready && dev.pdl, x, Y, slot_of, wts, sgate,
               shared, topk, H);
  }
  return 0;
}

// act: scratch of 16 bits per (slot, j); this implementation keeps the SwiGLU intermediate there as fp16
// (values beyond +-65504 are clamped to that range).
// Reference: kernels/drama.cu:961-968; src/ffi.rs:61-64. H = 2048 and I = 512 only, else -1.
extern "C" int dr_moe_prefill(const uint8_t* gu_q, const __half2* gu_sm, const uint8_t* d_q, const __half2* d_sm,
                              const __nv_bfloat16* xp, const int* offsets, const int* counts, __nv_bfloat16* act, float* y,
                              int E, int H, int I, cudaStream_t st) {
  if (H != pf::H || I != pf::I) return -1;
  if (E <= 0) return 0;
  const DrbDevice& dev = drb_device(st);
  if (!dev.ready) return -2;
  pft::Block b = {};
  b.gu_w = gu_q, b.gu_s = gu_sm, b.d_w = d_q, b.d_s = d_sm, b.sgu_s = gu_sm, b.sd_s = d_sm, b.x = xp, b.x_bf16 = true;
  b.offsets = offsets, b.counts = counts, b.act = act, b.y = y, b.E = E;
  return pft::run_block<0>(b, dev, st);
}

// No counterpart in the reference. Count, exclusive scan and slot assignment of the (row, k) pairs in one launch:
// counts[e_n], offsets[e_n], slot_of[rows * topk] (-1 for pairs whose expert lies outside [e_lo, e_lo + e_n)),
// row_of[slot] = row. Replaces dr_moe_count + the host scan + dr_moe_permute of src/engine.rs:565-580 when the
// grouped GEMM is drb_moe_prefill_block, which reads its rows through row_of. e_n <= 1024, else -1.
extern "C" int drb_moe_group(const int* idx, int rows, int topk, int e_lo, int e_n, int* counts, int* offsets, int* slot_of,
                             int* row_of, cudaStream_t st) {
  if (e_n <= 0 || e_n > pf::GRP_MAX_E || topk <= 0) return -1;
  drb_launch(pf::k_group, dim3(1), dim3(pf::GRP_THREADS), 0, st, false, idx, rows * topk, topk, e_lo, e_n, counts, offsets,
             slot_of, row_of, (int*)nullptr, 0, 0, 0);
  return 0;
}

// Expert parallelism (no counterpart in the reference, which is single-GPU). Rows travel between ranks in a buffer of
// `world` blocks; a block is blk_rows = cap + ceil(4 cap / row_bytes) rows of row_bytes bytes: cap row slots, then the
// cap local expert ids of those rows (int32), padded to whole rows. One collective moves rows and ids together.
//   drb_ep_pack    sender: places this rank's (row, k) pairs (idx [rows, topk], experts per rank `per`) into `send`,
//                  slot_of [rows * topk] = owner * cap + slot for the combine step, dst_row [rows * topk] scratch.
//                  *overflow (device word, zeroed by the caller) is set when a block was full: the result is void then.
//   drb_ep_group   owner: groups the received world * cap pairs by local expert: counts / offsets [per],
//                  slot_of [world * cap] scratch, row_of [slot] = row of `recv` (operand gather of the grouped GEMM),
//                  pair_of [slot] = position of the pair in receive order (where the result row goes).
// row_bytes % 16 == 0, world <= 64, per <= 1024; -1 otherwise.
extern "C" int drb_ep_block_rows(int cap, int row_bytes) { return cap + (4 * cap + row_bytes - 1) / row_bytes; }
extern "C" int drb_ep_pack(const void* rows, const int* idx, int n_rows, int topk, int per, int world, int cap, int row_bytes,
                           void* send, int* slot_of, int* dst_row, unsigned* overflow, cudaStream_t st) {
  if (row_bytes % 16 != 0 || world <= 0 || world > 64 || per <= 0 || cap <= 0 || topk <= 0) return -1;
  const int pairs = n_rows * topk;
  const int blk_rows = drb_ep_block_rows(cap, row_bytes);
  drb_launch(pf::k_ep_plan, dim3(1), dim3(pf::GRP_THREADS), 0, st, false, idx, pairs, per, world, cap, blk_rows, row_bytes / 4,
             (int*)send, slot_of, dst_row, overflow, (int* const*)nullptr, 0);
  if (pairs > 0)
    drb_launch(pf::k_ep_scatter, dim3((pairs + 7) / 8), dim3(256), 0, st, false, (const unsigned char*)rows, pairs, topk,
               (const int*)dst_row, (unsigned char*)send, row_bytes, (unsigned char* const*)nullptr, 0, blk_rows);
  return 0;
}
// drb_ep_pack with the blocks stored straight into the owners' receive buffers (peer_recv: device array of `world`
// pointers as for drb_ep_put; this rank's block in peer o's buffer is block `rank`). Follow with drb_ep_signal.
extern "C" int drb_ep_pack_peers(const void* rows, const int* idx, int n_rows, int topk, int per, int world, int cap, int row_bytes,
                                 void* const* peer_recv, int rank, int* slot_of, int* dst_row, unsigned* overflow, cudaStream_t st) {
  if (row_bytes % 16 != 0 || world <= 0 || world > 64 || per <= 0 || cap <= 0 || topk <= 0 || !peer_recv || rank < 0 || rank >= world)
    return -1;
  const int pairs = n_rows * topk;
  const int blk_rows = drb_ep_block_rows(cap, row_bytes);
  drb_launch(pf::k_ep_plan, dim3(1), dim3(pf::GRP_THREADS), 0, st, false, idx, pairs, per, world, cap, blk_rows, row_bytes / 4,
             (int*)nullptr, slot_of, dst_row, overflow, reinterpret_cast<int* const*>(peer_recv), rank);
  if (pairs > 0)
    drb_launch(pf::k_ep_scatter, dim3((pairs + 7) / 8), dim3(256), 0, st, false, (const unsigned char*)rows, pairs, topk,
               (const int*)dst_row, (unsigned char*)nullptr, row_bytes, reinterpret_cast<unsigned char* const*>(peer_recv), rank, blk_rows);
  return 0;
}
extern "C" int drb_ep_group(const void* recv, int world, int cap, int row_bytes, int per, int* counts, int* offsets, int* slot_of,
                            int* row_of, int* pair_of, cudaStream_t st) {
  if (row_bytes % 16 != 0 || world <= 0 || per <= 0 || per > pf::GRP_MAX_E || cap <= 0) return -1;
  drb_launch(pf::k_group, dim3(1), dim3(pf::GRP_THREADS), 0, st, false, (const int*)recv, world * cap, 1, 0, per, counts, offsets,
             slot_of, row_of, pair_of, cap, drb_ep_block_rows(cap, row_bytes), row_bytes / 4);
  return 0;
}

// The expert-parallel exchange over NVLink peer stores instead of a library collective (no counterpart in the
// reference). peer_recv / peer_flags: device arrays of `world` pointers, entry p = rank p's receive buffer / flag
// array (memory every rank can store to: symmetric memory), this rank's own included.
//   drb_ep_put     block p (block_bytes each) of `send` -> peer p's receive buffer at slot `rank`
//   drb_ep_signal  ++*step (device word, zero at start on every rank); peer p's flag [rank] = *step
//   drb_ep_wait    ++*step (another device word, zero at start); returns once flags [0, world) have all reached it, or
//                  after poll_limit polls (error word set, the step's result is void)
// One exchange = put, signal on the sender; wait on the receiver before it reads. A rank starts the next exchange
// into a peer's buffer only after that peer's reply to the current one, so a buffer is never overwritten while it
// is read. block_bytes % 16 == 0, world <= 64, else -1.
extern "C" int drb_ep_put(const void* send, void* const* peer_recv, int world, int rank, size_t block_bytes, cudaStream_t st) {
  if (!send || !peer_recv || world <= 0 || world > 64 || rank < 0 || rank >= world || block_bytes % 16 != 0) return -1;
  if (block_bytes == 0) return 0;
  const size_t vecs = block_bytes / 16;
  const unsigned per = (unsigned)((vecs + 4095) / 4096);  // about sixteen 16-byte stores per thread
  drb_launch(pf::k_ep_put, dim3(per < 1 ? 1 : (per > 64 ? 64 : per), (unsigned)world), dim3(256), 0, st, false,
             static_cast<const uint4*>(send), reinterpret_cast<uint4* const*>(peer_recv), rank, vecs);
  return 0;
}
extern "C" int drb_ep_signal(unsigned* const* peer_flags, int world, int rank, unsigned* step, cudaStream_t st) {
  if (!peer_flags || !step || world <= 0 || world > 64 || rank < 0 || rank >= world) return -1;
  drb_launch(pf::k_ep_signal, dim3(1), dim3(64), 0, st, false, peer_flags, world, rank, step);
  return 0;
}
// drb_ep_signal followed by drb_ep_wait in one launch; steps: two device words (signalled, awaited), zero at start.
extern "C" int drb_ep_sync(unsigned* const* peer_flags, const unsigned* flags, int world, int rank, unsigned* steps, unsigned poll_limit,
                           cudaStream_t st) {
  if (!peer_flags || !flags || !steps || world <= 0 || world > 64 || rank < 0 || rank >= world || poll_limit == 0) return -1;
  drb_launch(pf::k_ep_sync, dim3(1), dim3(64), 0, st, false, peer_flags, flags, world, rank, steps, poll_limit);
  return 0;
}
extern "C" int drb_ep_wait(const unsigned* flags, int world, unsigned* step, unsigned poll_limit, cudaStream_t st) {
  if (!flags || !step || world <= 0 || world > 64 || poll_limit == 0) return -1;
  drb_launch(pf::k_ep_wait, dim3(1), dim3(64), 0, st, false, flags, world, step, poll_limit);
  return 0;
}

// drb_moe_prefill_block and drb_moe_prefill_block_peers (no counterpart in the reference). The routed experts AND the
// int8 shared expert of one prefill block in two launches: dr_moe_prefill with (a) the operand rows read in place through row_of (xb holds the normalised rows in row
// order, [rows, H], bf16 or with x_f16 != 0 fp16; nothing is permuted) and (b) the shared expert as one more expert that owns every row, its
// int8 weights dequantised into the same tensor-core tiles (sh_act: fp16 scratch [rows, I]; sh_out: f32 [rows, H]).
// The reference runs the shared expert through cuBLAS on weights dequantised to bf16 (src/engine.rs:351-355, 560-562);
// here no library GEMM and no bf16 copy of the weights is involved. rows_sh = 0 skips the shared expert, E = 0 the
// routed ones. y_row_of (or NULL): slot -> row of y for the routed results. Limits as dr_moe_prefill.
// Every pointer of a part that runs must be a valid device address; with E = 0 or rows_sh = 0 the arrays of the part
// that does not run are not used, but must still be valid addresses (any buffer will do, NULL will not): the compiler
// may issue a load ahead of the branch that decides whether its value is needed. row_of and y_row_of may be NULL.
static int prefill_block_impl(const uint8_t* gu_q, const __half2* gu_sm, const uint8_t* d_q, const __half2* d_sm,
                                     const int8_t* sgu_q, const __half* sgu_s, const int8_t* sd_q, const __half* sd_s,
                                     const __nv_bfloat16* xb, const int* row_of, const int* offsets, const int* counts,
                                     __nv_bfloat16* act, float* y, __nv_bfloat16* sh_act, float* sh_out, int rows_sh, int E,
                                     int H, int I, int x_f16, const int* y_row_of, float* const* peer_y, int peer_cap, int peer_rank, cudaStream_t st) {
  if (H != pf::H || I != pf::I) return -1;
  if (E <= 0 && rows_sh <= 0) return 0;
  if (!gu_q || !gu_sm || !d_q || !d_sm || !sgu_q || !sgu_s || !sd_q || !sd_s || !xb || !offsets || !counts || !act || !y || !sh_act || !sh_out)
    return -1;
  const DrbDevice& dev = drb_device(st);
  if (!dev.ready) return -2;
  pft::Block b = {};
  b.gu_w = gu_q, b.gu_s = gu_sm, b.d_w = d_q, b.d_s = d_sm, b.sgu_q = sgu_q, b.sgu_s = sgu_s, b.sd_q = sd_q, b.sd_s = sd_s;
  b.x = xb, b.x_bf16 = !x_f16, b.row_of = row_of, b.offsets = offsets, b.counts = counts, b.y_row_of = y_row_of;
  b.act = act, b.y = y, b.sh_act = sh_act, b.sh_out = sh_out, b.rows_sh = rows_sh > 0 ? rows_sh : 0, b.E = E > 0 ? E : 0;
  b.peer_y = peer_y, b.peer_cap = peer_cap, b.peer_rank = peer_rank;
  return pft::run_block<0>(b, dev, st);
}

extern "C" int drb_moe_prefill_block(const uint8_t* gu_q, const __half2* gu_sm, const uint8_t* d_q, const __half2* d_sm,
                                     const int8_t* sgu_q, const __half* sgu_s, const int8_t* sd_q, const __half* sd_s,
                                     const __nv_bfloat16* xb, const int* row_of, const int* offsets, const int* counts,
                                     __nv_bfloat16* act, float* y, __nv_bfloat16* sh_act, float* sh_out, int rows_sh, int E,
                                     int H, int I, int x_f16, const int* y_row_of, cudaStream_t st) {
  return prefill_block_impl(gu_q, gu_sm, d_q, d_sm, sgu_q, sgu_s, sd_q, sd_s, xb, row_of, offsets, counts, act, y, sh_act, sh_out, rows_sh, E,
                            H, I, x_f16, y_row_of, nullptr, 0, 0, st);
}
// drb_moe_prefill_block on an expert-parallel rank, with the routed results stored straight into the home ranks'
// buffers: y_row_of[slot] = s * cap + j names the token's source rank s and its slot j in this rank's receive
// order; its result row goes to peer_y[s] (device array of every rank's result buffer [world * cap, h] f32) at row
// rank * cap + j, over NVLink, from the down GEMM's epilogue. Follow with drb_ep_signal; the home rank's
// drb_ep_wait then covers the results. fp16 rows only. y is not written.
extern "C" int drb_moe_prefill_block_peers(const uint8_t* gu_q, const __half2* gu_sm, const uint8_t* d_q, const __half2* d_sm,
                                           const int8_t* sgu_q, const __half* sgu_s, const int8_t* sd_q, const __half* sd_s,
                                           const __nv_bfloat16* xb, const int* row_of, const int* offsets, const int* counts,
                                           __nv_bfloat16* act, float* y, __nv_bfloat16* sh_act, float* sh_out, int rows_sh, int E,
                                           int H, int I, const int* y_row_of, float* const* peer_y, int cap, int rank,
                                           cudaStream_t st) {
  if (!peer_y || !y_row_of || cap <= 0 || rank < 0) return -1;
  return prefill_block_impl(gu_q, gu_sm, d_q, d_sm, sgu_q, sgu_s, sd_q, sd_s, xb, row_of, offsets, counts, act, y, sh_act, sh_out, rows_sh, E,
                            H, I, 1, y_row_of, peer_y, cap, rank, st);
}

// One MoE block over `rows` rows in one call (include/dramakernels.h): what MoePrefill's own sequence of calls does, in six
// launches (five up to 32 rows), each started while the one before drains.
struct drb_prefill_buffers {
  float* x;
  __half* rows16;
  float* logits;
  const float* logit_bias;
  int* idx;
  float *wts, *sgate;
  int *counts, *offsets, *slot_of, *row_of;
  __nv_bfloat16* act;
  float* y;
  __nv_bfloat16* sh_act;
  float* sh_out;
};
extern "C" int drb_moe_prefill_layer(const drb_moe_layer* w, const drb_prefill_buffers* b, int rows, int e, int topk, int h, int i, float eps,
                                     cudaStream_t st) {
  if (!w || !b || h != pf::H || i != pf::I || e < 1 || e > 256 || topk < 1 || topk > e || topk > 32) return -1;
  if (rows <= 0) return 0;
  // every pointer but logit_bias, before anything is launched; those that are read or written in 16-byte pieces on 16 bytes
  const void* vec[] = {b->x, b->rows16, b->y, b->sh_out, b->act, b->sh_act, w->router, w->gu_q, w->gu_sm, w->d_q, w->d_sm, w->sgu_q, w->sd_q};
  const void* word[] = {b->logits, b->idx, b->wts, b->sgate, b->counts, b->offsets, b->slot_of, b->row_of, w->post_norm, w->sgu_s, w->sd_s};
  for (const void* p : vec)
    if (!p) return -1;
  for (const void* p : word)
    if (!p) return -1;
  for (const void* p : vec)
    if (reinterpret_cast<uintptr_t>(p) & 15) return -3;
  const DrbDevice& dev = drb_device(st);
  if (!dev.ready) return -2;
  const int r = pf::launch_logits<pf::LOGITS_NORM>(b->x, static_cast<const float*>(w->post_norm), eps, b->rows16,
                                                   static_cast<const __nv_bfloat16*>(w->router), b->logit_bias, b->logits, rows, e + 1,
                                                   b->logit_bias ? 1.f : 0.f, b->counts, e, st);
  if (r != 0) return r;
  if (rows <= pf::FEW_ROWS) {
    drb_launch(pf::k_route_few, dim3(rows), dim3(rows * 32 <= pf::FEW_MIN_THREADS ? pf::FEW_MIN_THREADS : pf::FEW_ROWS * 32), 0, st, dev.pdl, (const float*)b->logits, (const __half*)b->rows16, rows, e, topk, b->idx,
               b->wts, b->sgate, b->counts, b->offsets, b->slot_of, b->row_of, reinterpret_cast<unsigned char*>(b->y), reinterpret_cast<unsigned char*>(b->sh_out));
  } else {
    // The pairs' ranks: two warps read each, so they do not share slot_of's place; act is free until the gate/up kernel writes it.
    int* rank = reinterpret_cast<int*>(b->act);
    drb_launch(router::k_moe_topk<true>, dim3((rows + router::TOPK_ROWS - 1) / router::TOPK_ROWS), dim3(router::TOPK_ROWS * 32), 0, st, dev.pdl,
               (const float*)b->logits, rows, e, topk, e + 1, b->idx, b->wts,
               b->sgate, b->counts, rank);
    const int blocks = (rows + pf::SC_ROWS - 1) / pf::SC_ROWS;
    drb_launch(pf::k_scatter_rows, dim3(blocks < 8 * dev.sms ? blocks : 8 * dev.sms), dim3(pf::SC_THREADS), 0, st, dev.pdl, (const __half*)b->rows16,
               (const int*)b->idx, rows, topk, (const int*)b->counts, e, b->offsets, b->slot_of, (const int*)rank, b->row_of,
               reinterpret_cast<unsigned char*>(b->y), reinterpret_cast<unsigned char*>(b->sh_out));
  }
  pft::Block k = {};
  k.gu_w = w->gu_q, k.gu_s = w->gu_sm, k.d_w = w->d_q, k.d_s = w->d_sm;
  k.sgu_q = w->sgu_q, k.sgu_s = w->sgu_s, k.sd_q = w->sd_q, k.sd_s = w->sd_s;
  k.prepared = true, k.row_of = b->row_of, k.offsets = b->offsets, k.counts = b->counts;
  k.act = b->act, k.y = b->y, k.sh_act = b->sh_act, k.sh_out = b->sh_out, k.rows_sh = rows, k.E = e;
  const int g = pft::run_block<0>(k, dev, st);
  if (g != 0) return g;
  return dr_moe_combine(b->x, b->y, b->slot_of, b->wts, b->sgate, b->sh_out, rows, topk, h, st);
}

// dr_moe_prefill over block-FP8 experts (include/dramakernels.h). Reference: kernels/drama.cu:971-1109; src/ffi.rs:52-55.
extern "C" int dr_moe_prefill_fp8(const uint8_t* gu_w, const float* gu_s, const uint8_t* d_w, const float* d_s,
                                  const __nv_bfloat16* xp, const int* offsets, const int* counts, __nv_bfloat16* act, float* y,
                                  int E, int H, int I, cudaStream_t st) {
  if (H != pf::H || I != pf::I) return -1;
  if (E <= 0) return 0;
  const DrbDevice& dev = drb_device(st);
  if (!dev.ready) return -2;
  pft::Block b = {};
  b.gu_w = gu_w, b.gu_s = gu_s, b.d_w = d_w, b.d_s = d_s, b.x = xp, b.x_bf16 = true;
  b.offsets = offsets, b.counts = counts, b.act = act, b.y = y, b.E = E;
  return pft::run_block<1>(b, dev, st);
}

// Reference: kernels/drama.cu:1130-1134; src/ffi.rs:74. K a multiple of 128.
extern "C" int dr_dequant_q8(const int8_t* W, const __half* S, __nv_bfloat16* out, int N, int K, cudaStream_t st) {
  if (K % 128 != 0) return -1;
  const size_t n = (size_t)N * K;
  if (n == 0) return 0;
  pf::k_dequant_q8<<<(unsigned)((n / 16 + 255) / 256), 256, 0, st>>>(W, S, out, n, K);
  return 0;
}

// Reference: kernels/drama.cu:1163-1166; src/ffi.rs:75.
extern "C" int dr_f32_to_bf16(const float* x, __nv_bfloat16* y, size_t n, cudaStream_t st) {
  if (n == 0) return 0;
  pf::k_f32_to_bf16<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, y, n);
  return 0;
}

// Reference: kernels/drama.cu:1176-1180; src/ffi.rs:76.
extern "C" int dr_swiglu_rows(const float* h, __nv_bfloat16* y, int rows, int I, cudaStream_t st) {
  const size_t n = (size_t)rows * I;
  if (n == 0) return 0;
  pf::k_swiglu_rows<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(h, y, rows, I);
  return 0;
}

// Reference: kernels/drama.cu:1198-1202; src/ffi.rs:77.
extern "C" int dr_rmsnorm(const float* x, const float* w, float* y, __nv_bfloat16* yb, int rows, int D, float eps,
                          cudaStream_t st) {
  if (rows <= 0) return 0;
  pf::k_rmsnorm<false><<<rows, 256, 0, st>>>(x, w, y, yb, D, eps);
  return 0;
}
