// Mixture-of-experts routing on the device, in three kernels that replace ~15 eager tensor ops per
// layer and direction (softmax, bias add, top-k, gather, renormalise, counts; stable sort, cumsum
// and scatter for the slot assignment; gather * weight + sum over k for the combine):
//
//   pico_moe_route       one warp per token: fp32 softmax over the E router logits, selection of
//                        the top-k experts on probs (+ bias when loss-free balancing is on), weights
//                        = the un-biased probabilities, renormalised over the k selected; also the
//                        per-expert row counts. Backward: pico_moe_route_bwd (weights -> logits,
//                        plus an optional dense gradient w.r.t. the probabilities, which is how the
//                        auxiliary balancing loss enters).
//   pico_moe_slots       one CTA per expert: position of every routed row inside its expert's queue
//                        in row order (deterministic), and the table row_of_slot[e * C + pos] = row
//                        for the rows that fit the capacity C (-1 elsewhere).
//   pico_moe_combine     y[t] = sum_k w[t,k] * expert_out[e(t,k) * C + pos(t,k)] over the rows that
//                        fit the capacity, k in fixed order; backward: pico_moe_combine_bwd gives the
//                        gradient of expert_out (each slot has exactly one reader, so no atomics)
//                        and of the weights (one dot product per routed row).
//
//   pico_moe_layout      the dropless layout of all experts on one GPU: every expert's rows in row order,
//                        its segment padded to whole 128-row GEMM tiles; row <-> slot tables, segment
//                        starts and tile owners, without a host read.
//   pico_moe_gather      x_slots[s] = x[row_of_slot[s] / k], zeros in padding slots.
//   pico_moe_scatter_sum y[t] = sum_k w[t,k] * x_slots[slot_of_row[t,k]] (w == NULL: weights of one): the
//                        weighted combine, and the backward pass of the gather.
//
// Reference: picotron/expert_parallel/expert_parallel.py:168-224 (router, balancing, weighting),
// :271-341 (dropless execution), capacity_moe.py:44-57 (slot assignment).
#include <cuda_bf16.h>
#include <math_constants.h>

#include "../common/host.h"
#include "../common/ptx.cuh"
#include "elementwise.h"

namespace pico {

constexpr int kMaxExpertsPerLane = 8;   // E <= 256
constexpr int kMaxTopK = 8;

__device__ __forceinline__ float route_warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float route_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// logits: bf16 [T, E] (row stride ldl). probs: fp32 [T, E]. idx: int32 [T, k]. w: fp32 [T, k].
// counts: int32 [E], must be zero on entry. A warp takes a token, kPerLane experts a lane (8 for up to 256 experts did
// four times the work at 64); lane j keeps the j-th choice, so nothing is indexed at run time, and the rows per expert
// are counted in the block first. Bound by the chain of k arg-max rounds of a token; 8192 tokens, 64 experts, top-6:
// 35.0 -> 9.5 us; 2048 tokens 11.7 -> 4.5; 8192 tokens, 256 experts, top-8 28.9 -> 22.8.
template <int kPerLane>
__global__ void __launch_bounds__(256)
moe_route_kernel(const __nv_bfloat16* __restrict__ logits, int64_t ldl, const float* __restrict__ bias,
                 float* __restrict__ probs, int32_t* __restrict__ idx, float* __restrict__ w,
                 int32_t* __restrict__ counts, int T, int E, int k, int renorm) {
  __shared__ int32_t hits[32 * kPerLane];
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int e = threadIdx.x; e < 32 * kPerLane; e += blockDim.x) hits[e] = 0;
  __syncthreads();
  for (int t = warp; t < T; t += nwarps) {
    float p[kPerLane], s[kPerLane];
    float mx = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
      const int e = lane + 32 * i;
      p[i] = e < E ? __bfloat162float(logits[(int64_t)t * ldl + e]) : -CUDART_INF_F;
      mx = fmaxf(mx, p[i]);
    }
    mx = route_warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
      p[i] = (lane + 32 * i) < E ? __expf(p[i] - mx) : 0.f;
      sum += p[i];
    }
    sum = route_warp_sum(sum);
    const float inv = 1.f / sum;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
      const int e = lane + 32 * i;
      p[i] *= inv;
      if (e < E) {
        probs[(int64_t)t * E + e] = p[i];
        s[i] = p[i] + (bias ? bias[e] : 0.f);
      } else {
        s[i] = 0.f;                        // no expert: never chosen
      }
    }
    // k rounds of arg-max over the warp; ties go to the lower expert index. `open` holds the entries of this lane
    // that may still be chosen: k <= E, so some lane always has one, and the choice stays inside [0, E) whatever the
    // scores are. A score that is not a number counts as the lowest one (a row whose softmax is not finite takes its
    // first k experts); its weight carries the NaN into the output.
    unsigned open = 0;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) open |= (unsigned)(lane + 32 * i < E) << i;
    float mine_w = 0.f, wsum = 0.f;
    int mine_e = 0;
    for (int j = 0; j < k; ++j) {
      float best = -CUDART_INF_F;
      int best_e = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < kPerLane; ++i) {
        const int e = lane + 32 * i;
        const float key = isnan(s[i]) ? -CUDART_INF_F : s[i];
        if ((open >> i & 1) != 0 && (key > best || (key == best && e < best_e))) {
          best = key;
          best_e = e;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
        if (ob > best || (ob == best && oe < best_e)) {
          best = ob;
          best_e = oe;
        }
      }
      // the lane that owns the winner hands out its un-biased probability and retires the entry
      float pw = 0.f;
#pragma unroll
      for (int i = 0; i < kPerLane; ++i)
        if (lane + 32 * i == best_e) {
          pw = p[i];
          open &= ~(1u << i);
        }
      pw = __shfl_sync(0xffffffffu, pw, best_e & 31);
      if (lane == j) {
        mine_w = pw;
        mine_e = best_e;
      }
      wsum += pw;
    }
    if (lane < k) {
      const float scale = (renorm && k > 1) ? 1.f / wsum : 1.f;
      idx[(int64_t)t * k + lane] = mine_e;
      w[(int64_t)t * k + lane] = mine_w * scale;
      atomicAdd(hits + mine_e, 1);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x)
    if (hits[e] != 0) atomicAdd(counts + e, hits[e]);
}

// dlogits[t, :] (fp32) from dw[t, :k] and (optional) dprobs[t, :E].
__global__ void __launch_bounds__(256)
moe_route_bwd_kernel(const float* __restrict__ probs, const int32_t* __restrict__ idx, const float* __restrict__ w,
                     const float* __restrict__ dw, const float* __restrict__ dprobs, float* __restrict__ dlogits,
                     int T, int E, int k, int renorm) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int t = warp; t < T; t += nwarps) {
    float p[kMaxExpertsPerLane], g[kMaxExpertsPerLane];
#pragma unroll
    for (int i = 0; i < kMaxExpertsPerLane; ++i) {
      const int e = lane + 32 * i;
      p[i] = e < E ? probs[(int64_t)t * E + e] : 0.f;
      g[i] = (e < E && dprobs) ? dprobs[(int64_t)t * E + e] : 0.f;
    }
    // w_j = p_j / S over the selected set (S = 1 without renormalisation):
    // dL/dp_j = (dw_j - sum_i dw_i w_i) / S, with S = p_j / w_j for any selected j
    float dot = 0.f, S = 1.f;
    if (renorm && k > 1) {
      float psel = 0.f;
      for (int j = 0; j < k; ++j) {
        dot += dw[(int64_t)t * k + j] * w[(int64_t)t * k + j];
        const int e = idx[(int64_t)t * k + j];
        float pj = 0.f;
#pragma unroll
        for (int i = 0; i < kMaxExpertsPerLane; ++i)
          if (lane + 32 * i == e) pj = p[i];
        psel += __shfl_sync(0xffffffffu, pj, e & 31);
      }
      S = psel;
    }
    for (int j = 0; j < k; ++j) {
      const int e = idx[(int64_t)t * k + j];
      const float gj = (renorm && k > 1) ? (dw[(int64_t)t * k + j] - dot) / S : dw[(int64_t)t * k + j];
#pragma unroll
      for (int i = 0; i < kMaxExpertsPerLane; ++i)
        if (lane + 32 * i == e) g[i] += gj;
    }
    // softmax backward: dlogit_e = p_e (g_e - sum_e' g_e' p_e')
    float gp = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxExpertsPerLane; ++i) gp += g[i] * p[i];
    gp = route_warp_sum(gp);
#pragma unroll
    for (int i = 0; i < kMaxExpertsPerLane; ++i) {
      const int e = lane + 32 * i;
      if (e < E) dlogits[(int64_t)t * E + e] = p[i] * (g[i] - gp);
    }
  }
}

// One CTA per expert e: pos[r] = number of rows r' < r with idx[r'] == e, for the rows of expert e;
// row_of_slot[e * C + pos] = r when pos < C (the table must hold -1 on entry).
__global__ void __launch_bounds__(1024)
moe_slots_kernel(const int32_t* __restrict__ idx, int R, int C, int32_t* __restrict__ pos,
                 int32_t* __restrict__ row_of_slot) {
  const int e = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ int warp_tot[32];
  __shared__ int running;
  if (threadIdx.x == 0) running = 0;
  __syncthreads();
  for (int base = 0; base < R; base += blockDim.x) {
    const int r = base + threadIdx.x;
    const bool mine = r < R && idx[r] == e;
    const unsigned ballot = __ballot_sync(0xffffffffu, mine);
    const int before = __popc(ballot & ((1u << lane) - 1u));
    if (lane == 0) warp_tot[warp] = __popc(ballot);
    __syncthreads();
    int off = running;
    for (int wi = 0; wi < warp; ++wi) off += warp_tot[wi];
    if (mine) {
      const int ps = off + before;
      pos[r] = ps;
      if (row_of_slot != nullptr && ps < C) row_of_slot[(int64_t)e * C + ps] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int tot = 0;
      for (int wi = 0; wi < (int)(blockDim.x >> 5); ++wi) tot += warp_tot[wi];
      running += tot;
    }
    __syncthreads();
  }
}

// y[t, :] = sum_j [pos < C] w[t,j] * out[(idx[t,j] * C + pos[t,j]), :]; one warp per token, d % 8 == 0.
__global__ void __launch_bounds__(256)
moe_combine_kernel(const __nv_bfloat16* __restrict__ out, const int32_t* __restrict__ idx,
                   const int32_t* __restrict__ pos, const float* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   int T, int k, int C, int d) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nvec = d / 8;
  for (int t = warp; t < T; t += nwarps) {
    for (int v = lane; v < nvec; v += 32) {
      float acc[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = 0.f;
      for (int j = 0; j < k; ++j) {
        const int ps = pos[(int64_t)t * k + j];
        if (ps >= C) continue;
        const float wj = w[(int64_t)t * k + j];
        const uint4 raw = reinterpret_cast<const uint4*>(out + ((int64_t)idx[(int64_t)t * k + j] * C + ps) * d)[v];
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = __bfloat1622float2(h[i]);
          acc[2 * i] += wj * f.x;
          acc[2 * i + 1] += wj * f.y;
        }
      }
      uint4 o;
      __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      reinterpret_cast<uint4*>(y + (int64_t)t * d)[v] = o;
    }
  }
}

// One CTA per expert. Expert e's segment starts at the sum of the padded counts before it; its rows keep row
// order. Every thread takes kLayoutRows consecutive rows of a pass (one 16-byte load per four), so a
// pass costs one block scan for 16384 rows; a scan per 1024 rows (moe_slots_kernel) took 70 us for 49152
// rows, most of it barriers.
// Nothing is written or named outside the tables, whatever idx and counts hold: a row of no expert, or one that its
// expert's count leaves no slot, gets slot -1 and a slot of no row holds -1, and the status words report it.
constexpr int kLayoutThreads = 1024;
constexpr int kLayoutRows = 16;
constexpr int kLayoutBadRow = 3200, kLayoutBadCount = 3201;   // sites in the status words
__global__ void __launch_bounds__(kLayoutThreads)
moe_layout_kernel(const int32_t* __restrict__ idx, const int32_t* __restrict__ counts, int R, int E, int max_tiles,
                  int32_t* __restrict__ slot_of_row, int32_t* __restrict__ row_of_slot,
                  int32_t* __restrict__ seg_start, int32_t* __restrict__ tile_group, int* status) {
  const int e = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ int warp_tot[kLayoutThreads / 32];
  __shared__ unsigned s_before[kLayoutThreads / 32];
  // padded rows of the experts before this one (E <= 256 < blockDim.x), no more than the tables hold
  const unsigned room = 128u * max_tiles;
  auto padded_rows = [&](int i) { return ((unsigned)min(max(counts[i], 0), R) + 127u) & ~127u; };
  unsigned before = (int)threadIdx.x < e ? min(padded_rows(threadIdx.x), room) : 0u;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before = min(before + __shfl_xor_sync(0xffffffffu, before, o), room);
  if (lane == 0) s_before[warp] = before;
  __syncthreads();
  before = 0;
#pragma unroll
  for (int i = 0; i < 256 / 32; ++i) before = min(before + s_before[i], room);
  const int seg = (int)before;
  const int padded = (int)min(padded_rows(e), room - before);
  const int n = min(max(counts[e], 0), padded);
  if (threadIdx.x == 0) {
    seg_start[e] = seg;
    if (e == E - 1) seg_start[E] = seg + padded;
  }
  for (int i = threadIdx.x; i < padded / 128; i += blockDim.x) tile_group[seg / 128 + i] = e;
  if (e == E - 1)
    for (int i = (seg + padded) / 128 + threadIdx.x; i < max_tiles; i += blockDim.x) tile_group[i] = -1;
  int running = 0;                       // rows of this expert before the current pass
  for (int base = 0; base < R; base += kLayoutThreads * kLayoutRows) {
    const int r0 = base + threadIdx.x * kLayoutRows;
    uint32_t hit = 0, none = 0;          // which of this thread's rows belong to the expert, and which to none
    auto look = [&](int q, int v) {
      hit |= (uint32_t)(v == e) << q;
      none |= (uint32_t)((unsigned)v >= (unsigned)E) << q;
    };
    if (r0 + kLayoutRows <= R) {
#pragma unroll
      for (int q = 0; q < kLayoutRows; q += 4) {
        const int4 v = *reinterpret_cast<const int4*>(idx + r0 + q);   // idx is 16-byte aligned, r0 a multiple of 16
        look(q, v.x);
        look(q + 1, v.y);
        look(q + 2, v.z);
        look(q + 3, v.w);
      }
    } else {
      for (int q = 0; q < kLayoutRows && r0 + q < R; ++q) look(q, idx[r0 + q]);
    }
    for (; e == 0 && none != 0; none &= none - 1) {    // one CTA answers for the rows of no expert
      const int r = r0 + __ffs(none) - 1;
      slot_of_row[r] = -1;
      report_error(status, PICO_ERR_BOUNDS, kLayoutBadRow, r);
    }
    const int c = __popc(hit);
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    __syncthreads();                     // the previous pass's readers are done with warp_tot
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int w = warp_tot[lane];              // 32 warps: one total per lane
    int wincl = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, wincl, o);
      if (lane >= o) wincl += v;
    }
    const int warps_before = __shfl_sync(0xffffffffu, wincl - w, warp);
    const int total = __shfl_sync(0xffffffffu, wincl, 31);
    int pos = running + warps_before + incl - c;
    while (hit != 0) {
      const int q = __ffs(hit) - 1;
      hit &= hit - 1;
      slot_of_row[r0 + q] = pos < n ? seg + pos : -1;
      if (pos < n) row_of_slot[seg + pos] = r0 + q;
      ++pos;
    }
    running += total;
  }
  for (int i = min(running, n) + threadIdx.x; i < padded; i += blockDim.x) row_of_slot[seg + i] = -1;
  if (threadIdx.x == 0 && running != counts[e]) report_error(status, PICO_ERR_BOUNDS, kLayoutBadCount, e);
}

// One warp per slot; slots at or past *used are left alone.
__global__ void __launch_bounds__(256)
moe_gather_kernel(const __nv_bfloat16* __restrict__ x, const int32_t* __restrict__ row_of_slot,
                  const int32_t* __restrict__ used, __nv_bfloat16* __restrict__ out, int slots, int k, int d) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;   // row_grid: up to 2^28 blocks
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int nvec = d / 8;
  const int n = min(slots, *used);
  for (int64_t s = warp; s < n; s += nwarps) {
    const int row = row_of_slot[s];
    uint4* dst = reinterpret_cast<uint4*>(out + s * d);
    if (row < 0) {
      for (int v = lane; v < nvec; v += 32) dst[v] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const uint4* src = reinterpret_cast<const uint4*>(x + (int64_t)(row / k) * d);
    int v = lane;
    for (; v + 96 < nvec; v += 128) {    // four loads in flight
      const uint4 a = src[v], b = src[v + 32], c = src[v + 64], e = src[v + 96];
      dst[v] = a;
      dst[v + 32] = b;
      dst[v + 64] = c;
      dst[v + 96] = e;
    }
    for (; v < nvec; v += 32) dst[v] = src[v];
  }
}

// One warp per token, fp32 sums in the order of k. kHasW: weighted by w[t, j]. A row without a slot (-1, which the
// layout reports) makes its token's sum NaN.
template <bool kHasW>
__global__ void __launch_bounds__(256)
moe_scatter_sum_kernel(const __nv_bfloat16* __restrict__ x, const int32_t* __restrict__ slot_of_row,
                       const float* __restrict__ w, __nv_bfloat16* __restrict__ y, int T, int k, int d) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nvec = d / 8;
  for (int t = warp; t < T; t += nwarps) {
    int slot[kMaxTopK];
    float wt[kMaxTopK];
    bool lost = false;
#pragma unroll
    for (int j = 0; j < kMaxTopK; ++j) {
      slot[j] = j < k ? slot_of_row[(int64_t)t * k + j] : 0;
      wt[j] = kHasW && j < k ? w[(int64_t)t * k + j] : 1.f;
      lost |= slot[j] < 0;
    }
    for (int v = lane; v < nvec; v += 32) {
      uint4 raw[kMaxTopK];               // all k rows' loads in flight
#pragma unroll
      for (int j = 0; j < kMaxTopK; ++j)
        if (j < k) raw[j] = reinterpret_cast<const uint4*>(x + (int64_t)max(slot[j], 0) * d)[v];
      float acc[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll
      for (int j = 0; j < kMaxTopK; ++j) {
        if (j < k) {
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(h[i]);
            acc[2 * i] += kHasW ? wt[j] * f.x : f.x;
            acc[2 * i + 1] += kHasW ? wt[j] * f.y : f.y;
          }
        }
      }
      uint4 o;
      __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      if (lost) o = make_uint4(~0u, ~0u, ~0u, ~0u);       // bf16 NaNs
      reinterpret_cast<uint4*>(y + (int64_t)t * d)[v] = o;
    }
  }
}

// One warp per slot s of the [E*C, d] expert-output table: row = row_of_slot[s];
// dout[s, :] = w[row] * dy[row / k, :] (zeros for an empty slot) and dw[row] = <dy[row / k], out[s]>.
// dw must be zero on entry for the rows that did not fit the capacity (they get no slot).
__global__ void __launch_bounds__(256)
moe_combine_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ out,
                       const int32_t* __restrict__ row_of_slot, const float* __restrict__ w,
                       const int32_t* __restrict__ used, __nv_bfloat16* __restrict__ dout, float* __restrict__ dw,
                       int64_t slots, int k, int d) {
  if (used != nullptr) slots = min(slots, (int64_t)*used);   // fill level known only on the device
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int nvec = d / 8;
  for (int64_t s = warp; s < slots; s += nwarps) {
    const int row = row_of_slot[s];
    if (row < 0) {
      for (int v = lane; v < nvec; v += 32) reinterpret_cast<uint4*>(dout + s * d)[v] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const float wr = w[row];
    const int t = row / k;
    float dot = 0.f;
    for (int v = lane; v < nvec; v += 32) {
      const uint4 g = reinterpret_cast<const uint4*>(dy + (int64_t)t * d)[v];
      const uint4 o = reinterpret_cast<const uint4*>(out + s * d)[v];
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g);
      const __nv_bfloat162* oh = reinterpret_cast<const __nv_bfloat162*>(&o);
      uint4 r;
      __nv_bfloat162* rh = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 gf = __bfloat1622float2(gh[i]);
        const float2 of = __bfloat1622float2(oh[i]);
        dot += gf.x * of.x + gf.y * of.y;
        rh[i] = __floats2bfloat162_rn(wr * gf.x, wr * gf.y);
      }
      reinterpret_cast<uint4*>(dout + s * d)[v] = r;
    }
    dot = route_warp_sum(dot);
    if (lane == 0) dw[row] = dot;
  }
}

static int route_check(const char* what, int T, int E, int k) {
  if (T < 0 || E < 1 || E > 32 * kMaxExpertsPerLane || k < 1 || k > kMaxTopK || k > E) {
    pico_host::set_error("%s: %d tokens, %d experts (max %d), top-%d (max %d)", what, T, E, 32 * kMaxExpertsPerLane, k,
                         kMaxTopK);
    return -2;
  }
  return 0;
}

// A warp per row, the rows in order of memory (8192 tokens x 6, width 2048: gather 57.3 -> 54.4 us, gradient of the
// weighted sum 106 -> 98; the sums, which jump about, gained nothing).
static int row_grid(int64_t rows) {
  const int64_t blocks = (rows + 7) / 8;
  return (int)(blocks < 1 ? 1 : blocks < INT32_MAX ? blocks : INT32_MAX);
}

static int warp_grid(int64_t items) {
  int64_t blocks = (items + 7) / 8;       // 8 warps per CTA
  const int cap = pico_host::num_sms() * 8;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : (int)blocks;
}

}  // namespace pico

using namespace pico;

extern "C" int pico_moe_route(const void* logits, int64_t ldl, const float* bias, float* probs, int32_t* idx,
                              float* w, int32_t* counts, int T, int E, int k, int renorm, cudaStream_t stream) {
  if (int rc = route_check("moe_route", T, E, k)) return rc;
  if (T == 0) return 0;
  auto kern = E <= 32 ? moe_route_kernel<1> : E <= 64 ? moe_route_kernel<2> : E <= 128 ? moe_route_kernel<4>
                                                                                     : moe_route_kernel<8>;
  const int cap = pico_host::num_sms() * 4, grid = warp_grid(T);
  kern<<<grid < cap ? grid : cap, 256, 0, stream>>>((const __nv_bfloat16*)logits, ldl, bias, probs, idx, w, counts, T, E,
                                                    k, renorm);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) pico_host::set_error("moe_route: %s", cudaGetErrorString(e));
  return (int)e;
}

extern "C" int pico_moe_route_bwd(const float* probs, const int32_t* idx, const float* w, const float* dw,
                                  const float* dprobs, float* dlogits, int T, int E, int k, int renorm,
                                  cudaStream_t stream) {
  if (int rc = route_check("moe_route_bwd", T, E, k)) return rc;
  if (T == 0) return 0;
  moe_route_bwd_kernel<<<warp_grid(T), 256, 0, stream>>>(probs, idx, w, dw, dprobs, dlogits, T, E, k, renorm);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) pico_host::set_error("moe_route_bwd: %s", cudaGetErrorString(e));
  return (int)e;
}

extern "C" int pico_moe_slots(const int32_t* idx, int R, int E, int C, int32_t* pos, int32_t* row_of_slot,
                              cudaStream_t stream) {
  if (R < 0 || E < 1 || C < 0) {
    pico_host::set_error("moe_slots: %d rows, %d experts, capacity %d", R, E, C);
    return -2;
  }
  if (R == 0) return 0;
  moe_slots_kernel<<<E, 1024, 0, stream>>>(idx, R, C, pos, row_of_slot);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) pico_host::set_error("moe_slots: %s", cudaGetErrorString(e));
  return (int)e;
}

extern "C" int pico_moe_combine(const void* out, const int32_t* idx, const int32_t* pos, const float* w, void* y,
                                int T, int k, int C, int d, cudaStream_t stream) {
  if (d % 8 != 0 || k < 1 || k > kMaxTopK) {
    pico_host::set_error("moe_combine: row width %d must be a multiple of 8, top-%d at most %d", d, k, kMaxTopK);
    return -2;
  }
  if (T <= 0) return 0;
  moe_combine_kernel<<<warp_grid(T), 256, 0, stream>>>((const __nv_bfloat16*)out, idx, pos, w, (__nv_bfloat16*)y, T,
                                                      k, C, d);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) pico_host::set_error("moe_combine: %s", cudaGetErrorString(e));
  return (int)e;
}

extern "C" int pico_moe_layout(const int32_t* idx, const int32_t* counts, int R, int E, int max_tiles,
                               int32_t* slot_of_row, int32_t* row_of_slot, int32_t* seg_start, int32_t* tile_group,
                               cudaStream_t stream) {
  if (R < 0 || E < 1 || E > 32 * kMaxExpertsPerLane || max_tiles < (R + 127) / 128 + (E < R ? E : R) ||
      (reinterpret_cast<uintptr_t>(idx) & 15) != 0) {
    pico_host::set_error("moe_layout: %d rows, %d experts (max %d), %d tiles (at least rows / 128 + experts that can "
                         "have rows), 16-byte aligned indices", R, E, 32 * kMaxExpertsPerLane, max_tiles);
    return -2;
  }
  moe_layout_kernel<<<E, kLayoutThreads, 0, stream>>>(idx, counts, R, E, max_tiles, slot_of_row, row_of_slot, seg_start,
                                                     tile_group, pico_status_buffer());
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) pico_host::set_error("moe_layout: %s", cudaGetErrorString(e));
  return (int)e;
}

extern "C" int pico_moe_gather(const void* x, const int32_t* row_of_slot, const int32_t* used, void* out, int slots,
                               int k, int d, cudaStream_t stream) {
  if (d % 8 != 0 || k < 1) {
    pico_host::set_error("moe_gather: row width %d must be a multiple of 8", d);
    return -2;
  }
  if (slots <= 0) return 0;
  moe_gather_kernel<<<row_grid(slots), 256, 0, stream>>>((const __nv_bfloat16*)x, row_of_slot, used,
                                                         (__nv_bfloat16*)out, slots, k, d);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) pico_host::set_error("moe_gather: %s", cudaGetErrorString(e));
  return (int)e;
}

extern "C" int pico_moe_scatter_sum(const void* x, const int32_t* slot_of_row, const float* w, void* y, int T, int k,
                                    int d, cudaStream_t stream) {
  if (d % 8 != 0 || k < 1 || k > kMaxTopK) {
    pico_host::set_error("moe_scatter_sum: row width %d must be a multiple of 8, top-%d at most %d", d, k, kMaxTopK);
    return -2;
  }
  if (T <= 0) return 0;
  if (w != nullptr)
    moe_scatter_sum_kernel<true><<<warp_grid(T), 256, 0, stream>>>((const __nv_bfloat16*)x, slot_of_row, w,
                                                                  (__nv_bfloat16*)y, T, k, d);
  else
    moe_scatter_sum_kernel<false><<<warp_grid(T), 256, 0, stream>>>((const __nv_bfloat16*)x, slot_of_row, nullptr,
                                                                   (__nv_bfloat16*)y, T, k, d);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) pico_host::set_error("moe_scatter_sum: %s", cudaGetErrorString(e));
  return (int)e;
}

extern "C" int pico_moe_combine_bwd(const void* dy, const void* out, const int32_t* row_of_slot, const float* w,
                                    const int32_t* used, void* dout, float* dw, int64_t slots, int k, int d,
                                    cudaStream_t stream) {
  if (d % 8 != 0 || k < 1) {
    pico_host::set_error("moe_combine_bwd: row width %d must be a multiple of 8", d);
    return -2;
  }
  if (slots <= 0) return 0;
  moe_combine_bwd_kernel<<<row_grid(slots), 256, 0, stream>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)out,
                                                              row_of_slot, w, used, (__nv_bfloat16*)dout, dw, slots,
                                                              k, d);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) pico_host::set_error("moe_combine_bwd: %s", cudaGetErrorString(e));
  return (int)e;
}
