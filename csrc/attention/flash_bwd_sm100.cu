// Flash attention backward for sm_100a on tcgen05 tensor cores.
//
// One CTA owns a block of 128 keys of one (batch, kv head), or where there are too few of those for the chip a share of
// its steps (pico_attention_bwd_splits); K_j and V_j stay resident in shared
// memory and the dK_j / dV_j accumulators stay in tensor memory while the CTA walks every query
// block (and every query head of the group, for grouped-query attention) that can see those keys.
// All score tiles are computed transposed (keys = tensor-memory lanes, queries = columns):
//
//   S^T  = K_j Q_i^T             dP^T = V_j dO_i^T                 (tensor cores -> TMEM)
//   P^T  = exp(S^T*scale - lse)  dS^T = P^T * (dP^T - delta)       (two or four threads per key row)
//   dV_j += P^T dO_i             dK_j += dS^T Q_i                  (A operand from TMEM)
//   dQ_i  = dS K_j               -> fp32 tile, TMA reduce-add into the global dQ accumulator
//
// With the keys on the lanes P^T and dS^T are, as packed bf16 in tensor memory, the A operands of
// the dV and dK products; only dS goes through shared memory (read transposed through an MN-major
// descriptor by the dQ product). Shared-memory traffic is what binds first here: with P and dS both
// read from shared memory the tile needed ~370 KB (2900 cycles at 128 B/clk) against ~2000 tensor
// cycles for head_dim 64; now it is ~270 KB.
//
// Roles: W softmax warps (arithmetic and the dK / dV epilogue), then four warps that drain dQ and stage lse /
// delta, one that issues every tcgen05.mma and one (one thread) every TMA load. W = 16 at head_dim 64 (four
// threads per key row, 32 queries each, 704 threads of 80 registers): with 8 the exponentials of a tile took
// 1800 cycles against 1024 for the special-function unit (a warp's dependent instructions issue every 3
// cycles; 16384 tokens: 3510 and 3284 us). W = 8 at head_dim 128, where the tensor cores have more to do and the
// drain, which dP of the next step waits for, holds two chunks in registers (437 us; with 16 warps 499).
// The MMA warp issues
//   dV(i) S(i+1) | dK(i) dQ(i) dP(i+1)
// so that the exponentials of step i+1 run under dK(i) / dQ(i) / dP(i+1) and the dS arithmetic under
// dV(i+1) / S(i+2); the two score tiles need no second buffer:
//   S   is overwritten by S(i+1) after P(i) was published (all of S(i) is in registers then)
//   P   is overwritten once S(i+1) has landed (the in-order pipe ran dV(i) before it)
//   dP  is overwritten by dP(i+1) behind dK(i) / dQ(i); dS lies over the dP columns of its own thread
// Measured (causal, B200, one call with its pre- and post-pass after an L2 flush; 546, 5740 and 701 us with P and dS
// through shared memory and one serial chain per tile): 4 x 2048 x 32 heads x 64: 347 us; 1 x 16384 x 32/8 heads x
// 64: 3131 us; 1 x 4096 x 32 x 128: 441 us.
// What binds it now is the chain of a tile through the softmax warps (exponentials, dS, their barriers).
//
// delta = rowsum(dO * O) comes from a small pre-pass; the dQ accumulator is scaled and converted to
// bf16 by a post-pass. Where q and k carry a rotary embedding, the post-pass also rotates dQ and dK back (dK in the
// main kernel's epilogue measured 8 us more per call: 32 rows of the tables per load). Every wait is bounded.
#include <cuda_bf16.h>
#include <math_constants.h>

#include <cstring>

#include "../common/host.h"
#include "../common/ptx.cuh"
#include "attention.h"

namespace pico {

constexpr int kBM = 128;   // query rows per step
constexpr int kBN = 128;   // keys per CTA
constexpr int kBwdDrainThreads = 128;
constexpr float kBwdLog2e = 1.4426950408889634f;

template <int D>
struct BwdCfg {
  static constexpr int kWarps = (D == 64) ? 16 : 8;         // softmax warps
  static constexpr int kParts = kWarps / 4;                 // threads of a key row
  static constexpr int kCols = 128 / kParts;                // queries of a thread
  static constexpr int kThreads = kWarps * 32 + kBwdDrainThreads + 64;
  static constexpr int kTile = 128 * D * 2;                 // one bf16 [128, D] tile
  static constexpr int kQStages = 2;                        // Q_i is read by S(i) and, a step later, by dK(i)
  static constexpr int kDoStages = (D == 64) ? 2 : 1;       // dO_i: dP(i) and dV(i)
  static constexpr int kDs = 2 * 128 * 128;                 // bf16 dS, two panels of 64 queries
  static constexpr int kStaging = 2 * 128 * 128;            // two fp32 dQ chunks of 32 columns
  static constexpr int kTiles = (2 + kQStages + kDoStages) * kTile + kDs + kStaging;
  static constexpr int kStats = 2 * 2 * 128 * 4;            // lse and delta of the queries, two stages
  // kv_full, q_full/q_empty, do_full/do_empty, stat_full[2], s_full, p_ready, dp_full, ds_ready, dq_full, dq_free,
  // all_done
  static constexpr int kNumBars = 1 + 2 * kQStages + 2 * kDoStages + 2 + 7;
  static constexpr int kSmemBytes = kTiles + kStats + kNumBars * 8 + 16;
  static constexpr int kPanels = D / 64;
  // TMEM columns. head_dim 64 has room for P and dQ; at head_dim 128 P lies over S (each part of
  // the queries over its own columns) and dQ over dP
  static constexpr int kTmS = 0, kTmDp = 128, kTmDv = 256, kTmDk = 256 + D;
  static constexpr int kTmDq = (D == 64) ? 384 : kTmDp;
  static constexpr int kTmP = (D == 64) ? 448 : kTmS;
  static constexpr int kTmPPart = (D == 64) ? kCols / 2 : kCols;   // column distance of the parts of P
  static constexpr int kSteps = kCols / 16;                 // 16-query MMA steps of a part
  static constexpr int kTmemCols = 512;
};

struct BwdMaps {
  CUtensorMap q, k, v, dout, dq_accum;
};

__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ dout,
                                  float* __restrict__ delta, float* __restrict__ dq_accum, PicoAttnParams p,
                                  int64_t do_batch_stride, int64_t do_row_stride) {
  ahead_wait();
  ahead_next();
  // also clears the dQ accumulator, 32 bytes per lane: a launch less than a memset of its own
  // head_dim / 8 adjacent lanes per (batch, row, head), 16 bytes of each operand per lane; the
  // heads of a row are contiguous, so a warp reads one 512-byte run of each tensor
  const int gsz = p.head_dim >> 3;            // 8 or 16 lanes per item
  const int per_warp = 32 / gsz;
  const int64_t total = (int64_t)p.batch * p.seq_q * p.heads;
  const int lane = threadIdx.x & 31;
  const int sub = lane / gsz, li = lane % gsz;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w * per_warp < total; w += warps) {
    const int64_t item = w * per_warp + sub;
    float acc = 0.f;
    int h = 0, row = 0, b = 0;
    if (item < total) {
      h = (int)(item % p.heads);
      const int64_t t = item / p.heads;
      row = (int)(t % p.seq_q);
      b = (int)(t / p.seq_q);
      const uint4 ov = *reinterpret_cast<const uint4*>(out + b * p.o_batch_stride + row * p.o_row_stride +
                                                      h * p.head_dim + li * 8);
      const uint4 dv = *reinterpret_cast<const uint4*>(dout + b * do_batch_stride + row * do_row_stride +
                                                      h * p.head_dim + li * 8);
      float4* acc_row = reinterpret_cast<float4*>(dq_accum + item * p.head_dim + li * 8);   // [b, seq, heads, d]
      acc_row[0] = make_float4(0.f, 0.f, 0.f, 0.f);
      acc_row[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&ov);
      const __nv_bfloat162* d2 = reinterpret_cast<const __nv_bfloat162*>(&dv);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = __bfloat1622float2(o2[i]);
        const float2 g = __bfloat1622float2(d2[i]);
        acc += a.x * g.x + a.y * g.y;
      }
    }
    for (int off = gsz >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (item < total && li == 0) delta[((int64_t)b * p.heads + h) * p.seq_q + row] = acc;
  }
}

// The post-pass where there is more to do than attn_dq_convert_kernel does: dq from its accumulator, rotated back
// before the rounding (kRope), dk rotated back in place (kRope) or, where the steps of a key block were split, dk and
// dv as the sums of their splits' slabs, in order. An item is 8 columns of the first half of a head and the 8 of the
// second half that they were rotated with. Bytes bind it; a rotation of its own read and wrote dq once more. Whole
// backward, post-pass and rotation / this, us: 4 x 2048 x 32 x 64: 350 / 340; 8 x 1024 x 15/5 x 64: 92 / 86; 1 x 128 x
// 9/3 x 64: 15.2 / 13.9.
template <bool kRope>
__global__ void attn_finish_kernel(const float* __restrict__ acc, const float* __restrict__ slabs, int splits,
                                   __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk,
                                   __nv_bfloat16* __restrict__ dv, PicoAttnParams p, int64_t dq_batch_stride,
                                   int64_t dq_row_stride, int64_t dk_batch_stride, int64_t dk_row_stride,
                                   int64_t dv_batch_stride, int64_t dv_row_stride) {
  ahead_wait();
  ahead_next();
  const int half = p.head_dim / 2, per_head = half / 8;
  const int64_t q_items = (int64_t)p.batch * p.seq_q * p.heads * per_head;
  const int64_t kv_items = (int64_t)p.batch * p.seq_k * p.kv_heads * per_head;
  const int64_t items = q_items + (splits > 1 ? 2 : kRope ? 1 : 0) * kv_items;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < items;
       i += (int64_t)gridDim.x * blockDim.x) {
    const bool is_q = i < q_items, is_v = i >= q_items + kv_items;
    const int64_t n = is_q ? i : is_v ? i - q_items - kv_items : i - q_items;
    const int heads = is_q ? p.heads : p.kv_heads, seq = is_q ? p.seq_q : p.seq_k;
    const int v = (int)(n % per_head) * 8;
    const int64_t u = n / per_head;
    const int head = (int)(u % heads);
    const int64_t t = u / heads;
    const int row = (int)(t % seq);
    const int64_t b = t / seq;
    __nv_bfloat16* dst = (is_q ? dq + b * dq_batch_stride + row * dq_row_stride
                          : is_v ? dv + b * dv_batch_stride + row * dv_row_stride
                                 : dk + b * dk_batch_stride + row * dk_row_stride) + head * p.head_dim + v;
    float lo[8], hi[8];
    if (is_q || splits > 1) {
      const int64_t slab = (int64_t)p.batch * p.seq_k * p.kv_heads * p.head_dim;
      const float* src = (is_q ? acc : slabs + (is_v ? slab : 0)) + u * p.head_dim + v;
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        *reinterpret_cast<float4*>(lo + j) = *reinterpret_cast<const float4*>(src + j);
        *reinterpret_cast<float4*>(hi + j) = *reinterpret_cast<const float4*>(src + half + j);
      }
      if (!is_q) {
#pragma unroll 2
        for (int sp = 1; sp < splits; ++sp) {
          src += 2 * slab;
#pragma unroll
          for (int j = 0; j < 8; j += 4) {
            const float4 l = *reinterpret_cast<const float4*>(src + j);
            const float4 h = *reinterpret_cast<const float4*>(src + half + j);
            lo[j] += l.x; lo[j + 1] += l.y; lo[j + 2] += l.z; lo[j + 3] += l.w;
            hi[j] += h.x; hi[j + 1] += h.y; hi[j + 2] += h.z; hi[j + 3] += h.w;
          }
        }
      }
    } else {
      const uint4 l = *reinterpret_cast<const uint4*>(dst), h = *reinterpret_cast<const uint4*>(dst + half);
      const uint32_t lw[4] = {l.x, l.y, l.z, l.w}, hw[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        lo[2 * j] = __uint_as_float(lw[j] << 16);
        lo[2 * j + 1] = __uint_as_float(lw[j] & 0xffff0000u);
        hi[2 * j] = __uint_as_float(hw[j] << 16);
        hi[2 * j + 1] = __uint_as_float(hw[j] & 0xffff0000u);
      }
    }
    // dS is kept unscaled by the main kernel, and so are the slabs; a dk that is read back has its scale
    const float sc = is_v || (!is_q && splits == 1) ? 1.f : p.sm_scale;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      lo[j] *= sc;
      hi[j] *= sc;
    }
    if (kRope && !is_v) {
      const int64_t at = (int64_t)(p.rope_pos0 + row) * half + v;
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        float c[4], s[4];
        *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(p.rope_cos + at + j);
        *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(p.rope_sin + at + j);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float a = lo[j + k], g = hi[j + k];
          lo[j + k] = a * c[k] + g * s[k];
          hi[j + k] = g * c[k] - a * s[k];
        }
      }
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(lo[0], lo[1]), pack_bf16x2(lo[2], lo[3]),
                                                pack_bf16x2(lo[4], lo[5]), pack_bf16x2(lo[6], lo[7]));
    *reinterpret_cast<uint4*>(dst + half) = make_uint4(pack_bf16x2(hi[0], hi[1]), pack_bf16x2(hi[2], hi[3]),
                                                       pack_bf16x2(hi[4], hi[5]), pack_bf16x2(hi[6], hi[7]));
  }
}

__global__ void attn_dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq,
                                       PicoAttnParams p, int64_t dq_batch_stride, int64_t dq_row_stride) {
  ahead_wait();
  ahead_next();
  const float sc = p.sm_scale;   // dS is kept unscaled by the main kernel
  const int hd = p.heads * p.head_dim;
  const int64_t nvec = (int64_t)p.batch * p.seq_q * hd / 8;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nvec;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = i * 8;
    const int col = (int)(e % hd);
    const int64_t t = e / hd;
    const int row = (int)(t % p.seq_q);
    const int b = (int)(t / p.seq_q);
    const float4 a = reinterpret_cast<const float4*>(acc + e)[0];
    const float4 c = reinterpret_cast<const float4*>(acc + e)[1];
    uint4 o;
    o.x = pack_bf16x2(a.x * sc, a.y * sc);
    o.y = pack_bf16x2(a.z * sc, a.w * sc);
    o.z = pack_bf16x2(c.x * sc, c.y * sc);
    o.w = pack_bf16x2(c.z * sc, c.w * sc);
    *reinterpret_cast<uint4*>(dq + b * dq_batch_stride + row * dq_row_stride + col) = o;
  }
}

// uniform yes/no across `kThreads` threads of named barrier `kId` (they share barriers afterwards)
template <int kId, int kThreads>
__device__ __forceinline__ int all_agree(bool ok) {
  int all_ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t"
      "}\n"
      : "=r"(all_ok)
      : "r"((int)ok), "n"(kId), "n"(kThreads)
      : "memory");
  return all_ok;
}

template <int D, bool kSplit>
__global__ void __launch_bounds__(BwdCfg<D>::kThreads, 1)
flash_bwd_kernel(const __grid_constant__ BwdMaps maps, const float* __restrict__ lse,
                 const float* __restrict__ delta, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv,
                 const PicoAttnParams p, int64_t dk_batch_stride, int64_t dk_row_stride,
                 int64_t dv_batch_stride, int64_t dv_row_stride, float* __restrict__ slabs, int splits,
                 int* status) {
  using Cfg = BwdCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0) {   // swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) report_error(status, PICO_ERR_BOUNDS, 2998, (int)(smem_u32(smem) & 1023u));
    return;
  }
  uint8_t* sK = smem;
  uint8_t* sV = sK + Cfg::kTile;
  uint8_t* sQ = sV + Cfg::kTile;                          // [kQStages]
  uint8_t* sdO = sQ + Cfg::kQStages * Cfg::kTile;         // [kDoStages]
  uint8_t* sdS = sdO + Cfg::kDoStages * Cfg::kTile;       // rows = keys, 64 queries of 128 bytes per panel
  uint8_t* staging = sdS + Cfg::kDs;                      // [2] fp32 dQ chunks
  float* stats = reinterpret_cast<float*>(smem + Cfg::kTiles);   // [2][lse 128 | delta 128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kTiles + Cfg::kStats);
  uint64_t* kv_full = bars;
  uint64_t* q_full = kv_full + 1;
  uint64_t* q_empty = q_full + Cfg::kQStages;
  uint64_t* do_full = q_empty + Cfg::kQStages;
  uint64_t* do_empty = do_full + Cfg::kDoStages;
  uint64_t* stat_full = do_empty + Cfg::kDoStages;
  uint64_t* s_full = stat_full + 2;
  uint64_t* p_ready = s_full + 1;
  uint64_t* dp_full = p_ready + 1;
  uint64_t* ds_ready = dp_full + 1;
  uint64_t* dq_full = ds_ready + 1;
  uint64_t* dq_free = dq_full + 1;
  uint64_t* all_done = dq_free + 1;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(all_done + 1);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // warp-uniform
  const int lane = threadIdx.x & 31;
  // blocks are dispatched x-fastest: under a causal mask key block 0 has the most query blocks to
  // walk, so every (head, batch) of the heavy key blocks starts before any light one
  const int kv_block = kSplit ? blockIdx.z / splits : blockIdx.z, split = kSplit ? blockIdx.z % splits : 0;
  const int kv_head = blockIdx.x;
  const int batch = blockIdx.y;
  const int group = p.heads / p.kv_heads;
  const int k0 = kv_block * kBN;
  const int num_q_blocks = (p.seq_q + kBM - 1) / kBM;
  // first query block that can see any key of this block
  int i_min = 0;
  if (p.causal) {
    const int first_key_pos = p.k_pos0 + k0;
    const int need = first_key_pos - p.q_pos0 - (kBM - 1);   // q0 >= need
    i_min = need <= 0 ? 0 : (need + kBM - 1) / kBM;
  }
  const int nqb = max(0, num_q_blocks - i_min);
  // this split's stretch of the steps (query blocks of the first head of the group, then of the next, ...)
  const int first = kSplit ? (int)((int64_t)nqb * group * split / splits) : 0;
  const int total = kSplit ? (int)((int64_t)nqb * group * (split + 1) / splits) - first : nqb * group;
  const int g0 = kSplit && nqb > 0 ? first / nqb : 0, i0 = i_min + (kSplit && nqb > 0 ? first % nqb : 0);

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < Cfg::kQStages; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
    }
    for (int s = 0; s < Cfg::kDoStages; ++s) {
      mbar_init(&do_full[s], 1);
      mbar_init(&do_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) mbar_init(&stat_full[s], kBwdDrainThreads);
    mbar_init(s_full, 1);
    mbar_init(p_ready, Cfg::kWarps);
    mbar_init(dp_full, 1);
    mbar_init(ds_ready, Cfg::kWarps);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, kBwdDrainThreads);
    mbar_init(all_done, 1);
    *abort_word = 0;
    mbar_fence_init();
    tma_prefetch_desc(&maps.q);
    tma_prefetch_desc(&maps.k);
    tma_prefetch_desc(&maps.v);
    tma_prefetch_desc(&maps.dout);
    tma_prefetch_desc(&maps.dq_accum);
  }
  if (warp == Cfg::kWarps + 4) {
    tmem_alloc(tmem_ptr_smem, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);
  ahead_wait();
  ahead_next();

  if (warp == Cfg::kWarps + 5) {
    // ---------------------------------------------------------------------------- TMA loads
    if (lane == 0 && total > 0) {
      mbar_arrive_expect_tx(kv_full, 2 * Cfg::kTile);
#pragma unroll
      for (int pn = 0; pn < Cfg::kPanels; ++pn)
        tma_load_4d(sK + pn * 16384, &maps.k, kv_full, pn * 64, kv_head, k0, batch);
      int g = g0, i = i0;
      for (int it = 0; it < total; ++it) {
        const int head = kv_head * group + g;
        const int qs = it % Cfg::kQStages, ds = it % Cfg::kDoStages;
        if (it >= Cfg::kQStages &&
            !mbar_wait(&q_empty[qs], (it / Cfg::kQStages - 1) & 1, abort_word, status, 2010))
          break;
        mbar_arrive_expect_tx(&q_full[qs], Cfg::kTile);
#pragma unroll
        for (int pn = 0; pn < Cfg::kPanels; ++pn)
          tma_load_4d(sQ + qs * Cfg::kTile + pn * 16384, &maps.q, &q_full[qs], pn * 64, head, i * kBM, batch);
        if (it == 0) {
#pragma unroll
          for (int pn = 0; pn < Cfg::kPanels; ++pn)
            tma_load_4d(sV + pn * 16384, &maps.v, kv_full, pn * 64, kv_head, k0, batch);
        }
        if (it >= Cfg::kDoStages &&
            !mbar_wait(&do_empty[ds], (it / Cfg::kDoStages - 1) & 1, abort_word, status, 2011))
          break;
        mbar_arrive_expect_tx(&do_full[ds], Cfg::kTile);
#pragma unroll
        for (int pn = 0; pn < Cfg::kPanels; ++pn)
          tma_load_4d(sdO + ds * Cfg::kTile + pn * 16384, &maps.dout, &do_full[ds], pn * 64, head, i * kBM, batch);
        if (++i == num_q_blocks) {
          i = i_min;
          ++g;
        }
      }
    }
  } else if (warp == Cfg::kWarps + 4) {
    // ---------------------------------------------------------------------------- MMA issue (converged warp)
    if (total > 0) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);   // S^T, dP^T: both operands K-major
      constexpr uint32_t idesc_v = umma_idesc_bf16(128, D, 0, 1);     // dV, dK: A from TMEM, B MN-major
      constexpr uint32_t idesc_q = umma_idesc_bf16(128, D, 1, 1);     // dQ: both operands MN-major
      // descriptors of the first stage of each tile, K-major (scores) and MN-major (gradients)
      constexpr uint32_t kStep = Cfg::kTile >> 4;
      const uint64_t k_d = umma_smem_desc(smem_u32(sK), 16, 1024), v_d = umma_smem_desc(smem_u32(sV), 16, 1024);
      const uint64_t q_d = umma_smem_desc(smem_u32(sQ), 16, 1024), do_d = umma_smem_desc(smem_u32(sdO), 16, 1024);
      const uint64_t k_mn = umma_smem_desc(smem_u32(sK), 16384, 1024), q_mn = umma_smem_desc(smem_u32(sQ), 16384, 1024);
      const uint64_t do_mn = umma_smem_desc(smem_u32(sdO), 16384, 1024);
      const uint64_t ds_mn = umma_smem_desc(smem_u32(sdS), 16384, 1024);
      auto issue_scores = [&](uint32_t d_tmem, uint64_t a_d, uint64_t b_d) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          tc_mma_f16_ss_warp(d_tmem, a_d + off, b_d + off, idesc_s, kk != 0 ? 1u : 0u);
        }
      };
      bool ok = mbar_wait_warp(kv_full, 0, abort_word, status, 2000) &&
                mbar_wait_warp(&q_full[0], 0, abort_word, status, 2020);
      if (ok) {
        tc_fence_after();
        issue_scores(tmem_base + Cfg::kTmS, k_d, q_d);
        tc_commit_warp(s_full);
        ok = mbar_wait_warp(&do_full[0], 0, abort_word, status, 2021);
      }
      if (ok) {
        tc_fence_after();
        issue_scores(tmem_base + Cfg::kTmDp, v_d, do_d);
        tc_commit_warp(dp_full);
      }
      for (int it = 0; it < total && ok; ++it) {
        const int qs = it % Cfg::kQStages, ds = it % Cfg::kDoStages;
        if (!mbar_wait_warp(p_ready, it & 1, abort_word, status, 2040)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)   // contraction over the 128 queries, 16 (8 packed columns) per step
          tc_mma_f16_ts_warp(tmem_base + Cfg::kTmDv,
                             tmem_base + Cfg::kTmP + kk / Cfg::kSteps * Cfg::kTmPPart + kk % Cfg::kSteps * 8,
                             do_mn + ds * kStep + (kk * 2048 >> 4), idesc_v, (it | kk) != 0 ? 1u : 0u);
        tc_commit_warp(&do_empty[ds]);
        if (it + 1 < total) {
          const int nq = (it + 1) % Cfg::kQStages;
          if (!mbar_wait_warp(&q_full[nq], ((it + 1) / Cfg::kQStages) & 1, abort_word, status, 2022)) break;
          tc_fence_after();
          issue_scores(tmem_base + Cfg::kTmS, k_d, q_d + nq * kStep);
          tc_commit_warp(s_full);
        }
        if (!mbar_wait_warp(ds_ready, it & 1, abort_word, status, 2041)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          tc_mma_f16_ts_warp(tmem_base + Cfg::kTmDk,
                             tmem_base + Cfg::kTmDp + kk / Cfg::kSteps * Cfg::kCols + kk % Cfg::kSteps * 8,
                             q_mn + qs * kStep + (kk * 2048 >> 4), idesc_v, (it | kk) != 0 ? 1u : 0u);
        tc_commit_warp(&q_empty[qs]);
        // dQ has its own columns at head_dim 64: the previous tile must have been drained; at head_dim 128
        // that wait came before dP(it), whose columns it shares
        if (D == 64 && it >= 1 && !mbar_wait_warp(dq_free, (it - 1) & 1, abort_word, status, 2042)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)   // contraction over the 128 keys
          tc_mma_f16_ss_warp(tmem_base + Cfg::kTmDq, ds_mn + (kk * 2048 >> 4), k_mn + (kk * 2048 >> 4),
                             idesc_q, kk != 0 ? 1u : 0u);
        tc_commit_warp(dq_full);
        if (it + 1 == total) tc_commit_warp(all_done);
        if (it + 1 < total) {
          const int nd = (it + 1) % Cfg::kDoStages;
          if (!mbar_wait_warp(&do_full[nd], ((it + 1) / Cfg::kDoStages) & 1, abort_word, status, 2023)) break;
          if (D != 64 && !mbar_wait_warp(dq_free, it & 1, abort_word, status, 2043)) break;
          tc_fence_after();
          issue_scores(tmem_base + Cfg::kTmDp, v_d, do_d + nd * kStep);
          tc_commit_warp(dp_full);
        }
      }
    }
  } else if (warp >= Cfg::kWarps) {
    // ---------------------------------------------------------------------------- dQ drain, lse / delta
    const int dt = threadIdx.x - Cfg::kWarps * 32;      // 0..127: query of the tile = TMEM lane
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    // statistics of the queries of step `it`: rows past the end and rows without keys get lse = +inf
    // (probability 0)
    auto load_stat = [&](int g, int i, float& l, float& dl) {
      const int q_idx = i * kBM + dt;
      l = CUDART_INF_F;
      dl = 0.f;
      if (q_idx < p.seq_q) {
        const int64_t off = ((int64_t)batch * p.heads + kv_head * group + g) * p.seq_q + q_idx;
        l = lse[off];
        dl = delta[off];
      }
    };
    auto put_stat = [&](int slot, float l, float dl) {
      stats[slot * 256 + dt] = (l == -CUDART_INF_F || l == CUDART_INF_F) ? -CUDART_INF_F : -l * kBwdLog2e;
      stats[slot * 256 + 128 + dt] = -dl;
      mbar_arrive(&stat_full[slot]);
    };
    int sg = g0, si = i0;                                // step whose statistics are loaded next
    auto stat_next = [&]() {
      if (++si == num_q_blocks) {
        si = i_min;
        ++sg;
      }
    };
    for (int it = 0; it < 2 && it < total; ++it) {
      float l, dl;
      load_stat(sg, si, l, dl);
      put_stat(it, l, dl);
      stat_next();
    }
    int g = g0, i = i0;
    for (int it = 0; it < total; ++it) {
      float l = 0.f, dl = 0.f;
      if (it + 2 < total) {
        load_stat(sg, si, l, dl);
        stat_next();
      }
      if (!all_agree<2, kBwdDrainThreads>(mbar_wait(dq_full, it & 1, abort_word, status, 2200))) break;
      tc_fence_after();
      // dQ(it) is complete, so every reader of this step's statistics is done
      if (it + 2 < total) put_stat(it & 1, l, dl);
      const int head = kv_head * group + g;
      // chunks of 32 columns through two staging tiles, kHeld of them in registers at a time
      constexpr int kHeld = (D == 64) ? 1 : 2;
#pragma unroll
      for (int c0 = 0; c0 < D / 32; c0 += kHeld) {
        uint32_t v[kHeld][32];
#pragma unroll
        for (int c = 0; c < kHeld; ++c) tmem_ld_32x32b_x32(tmem_base + Cfg::kTmDq + lane_base + (c0 + c) * 32, v[c]);
        tmem_ld_wait();
        if (c0 + kHeld == D / 32) {
          tc_fence_before();
          mbar_arrive(dq_free);
        }
        // the last read-out of these staging tiles must be over
        if (dt == 0) tma_store_wait_read<2 - kHeld>();
        named_barrier_sync(3, kBwdDrainThreads);
#pragma unroll
        for (int c = 0; c < kHeld; ++c) {
          uint8_t* srow = staging + ((c0 + c) & 1) * 16384 + dt * 128;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(srow + ((j ^ (dt & 7)) << 4)) =
                make_uint4(v[c][4 * j], v[c][4 * j + 1], v[c][4 * j + 2], v[c][4 * j + 3]);
        }
        fence_proxy_async_smem();
        named_barrier_sync(3, kBwdDrainThreads);
        if (dt == 0) {
#pragma unroll
          for (int c = 0; c < kHeld; ++c)
            tma_reduce_add_4d(&maps.dq_accum, staging + ((c0 + c) & 1) * 16384, (c0 + c) * 32, head, i * kBM, batch);
          tma_store_commit();
        }
      }
      if (++i == num_q_blocks) {
        i = i_min;
        ++g;
      }
    }
    if (dt == 0) tma_store_wait<0>();
  } else {
    // ---------------------------------------------------------------------------- softmax arithmetic
    // kParts warps share a TMEM lane quarter (key rows) and split the queries
    constexpr int kCols = Cfg::kCols;
    const int part = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tm_s = tmem_base + Cfg::kTmS + lane_base + part * kCols;
    const uint32_t tm_dp = tmem_base + Cfg::kTmDp + lane_base + part * kCols;   // dS lies over its first half
    const uint32_t tm_p = tmem_base + Cfg::kTmP + lane_base + part * Cfg::kTmPPart;
    const uint64_t scale2 = f2_pack(p.sm_scale * kBwdLog2e, p.sm_scale * kBwdLog2e);
    uint8_t* ds_row = sdS + (part * kCols >> 6) * 16384 + row * 128;
    const int ds_chunk = (part * kCols & 63) >> 3;          // first 16-byte chunk of this thread in its row
    // keys past the end see no query
    const bool key_valid = k0 + row < p.seq_k;
    const int key_pos = p.k_pos0 + k0 + row - p.q_pos0;     // in query indices
    bool alive = true;
    int i = i0;
    for (int it = 0; it < total; ++it) {
      const int q0 = i * kBM;
      const float* st = stats + (it & 1) * 256 + part * kCols;
      const bool need_mask = (p.causal && p.k_pos0 + k0 + kBN - 1 > p.q_pos0 + q0) || k0 + kBN > p.seq_k;
      // queries with column < q_lo are invisible to this key
      int q_lo = p.causal ? key_pos - q0 - part * kCols : 0;
      if (!key_valid) q_lo = kCols;
      alive = mbar_wait_warp(&stat_full[it & 1], (it >> 1) & 1, abort_word, status, 2099) &&
              mbar_wait_warp(s_full, it & 1, abort_word, status, 2100);
      if (!alive) break;
      tc_fence_after();
      uint32_t pr[kCols];
#pragma unroll
      for (int h = 0; h < kCols; h += 32) tmem_ld_32x32b_x32(tm_s + h, *reinterpret_cast<uint32_t (*)[32]>(&pr[h]));
      tmem_ld_wait();
      uint32_t pk[kCols / 2];
#pragma unroll
      for (int c = 0; c < kCols; c += 4) {
        const float4 nl = *reinterpret_cast<const float4*>(st + c);     // -lse * log2(e), the same for all lanes
        float e0, e1, e2, e3;
        const uint64_t s01 = f2_pack(__uint_as_float(pr[c]), __uint_as_float(pr[c + 1]));
        const uint64_t s23 = f2_pack(__uint_as_float(pr[c + 2]), __uint_as_float(pr[c + 3]));
        f2_unpack(f2_fma(s01, scale2, f2_pack(nl.x, nl.y)), e0, e1);
        f2_unpack(f2_fma(s23, scale2, f2_pack(nl.z, nl.w)), e2, e3);
        e0 = exp2f(e0);
        e1 = exp2f(e1);
        e2 = exp2f(e2);
        e3 = exp2f(e3);
        if (need_mask) {
          e0 = c >= q_lo ? e0 : 0.f;
          e1 = c + 1 >= q_lo ? e1 : 0.f;
          e2 = c + 2 >= q_lo ? e2 : 0.f;
          e3 = c + 3 >= q_lo ? e3 : 0.f;
        }
        pr[c] = __float_as_uint(e0);
        pr[c + 1] = __float_as_uint(e1);
        pr[c + 2] = __float_as_uint(e2);
        pr[c + 3] = __float_as_uint(e3);
        pk[c / 2] = pack_bf16x2(e0, e1);
        pk[c / 2 + 1] = pack_bf16x2(e2, e3);
      }
#pragma unroll
      for (int h = 0; h < kCols; h += 32)
        tmem_st_32x32b_x16(tm_p + h / 2, *reinterpret_cast<uint32_t (*)[16]>(&pk[h / 2]));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);      // one arrival per warp
      alive = mbar_wait_warp(dp_full, it & 1, abort_word, status, 2101);
      if (!alive) break;
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < kCols; h += 32) {
        uint32_t dpv[32], dsp[16];
        tmem_ld_32x32b_x32(tm_dp + h, dpv);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          const float4 nd = *reinterpret_cast<const float4*>(st + 128 + h + c);   // -delta
          float s0, s1, s2, s3;
          const uint64_t p01 = f2_pack(__uint_as_float(pr[h + c]), __uint_as_float(pr[h + c + 1]));
          const uint64_t p23 = f2_pack(__uint_as_float(pr[h + c + 2]), __uint_as_float(pr[h + c + 3]));
          const uint64_t d01 = f2_pack(__uint_as_float(dpv[c]), __uint_as_float(dpv[c + 1]));
          const uint64_t d23 = f2_pack(__uint_as_float(dpv[c + 2]), __uint_as_float(dpv[c + 3]));
          f2_unpack(f2_mul(p01, f2_add(d01, f2_pack(nd.x, nd.y))), s0, s1);
          f2_unpack(f2_mul(p23, f2_add(d23, f2_pack(nd.z, nd.w))), s2, s3);
          dsp[c / 2] = pack_bf16x2(s0, s1);
          dsp[c / 2 + 1] = pack_bf16x2(s2, s3);
        }
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4)
          *reinterpret_cast<uint4*>(ds_row + (((ds_chunk + h / 8 + q4) ^ (row & 7)) << 4)) =
              make_uint4(dsp[4 * q4], dsp[4 * q4 + 1], dsp[4 * q4 + 2], dsp[4 * q4 + 3]);
        tmem_st_32x32b_x16(tm_dp + h / 2, dsp);   // over columns that are in registers already
      }
      fence_proxy_async_smem();
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready);
      if (++i == num_q_blocks) i = i_min;
    }
    // ---- dK / dV of this key block: 32-column chunks of dV, then of dK, dealt to the parts
    if (alive && total > 0) alive = mbar_wait_warp(all_done, 0, abort_word, status, 2102);
    if (alive) {
      tc_fence_after();
      const int kidx = k0 + row;
      __nv_bfloat16* dk_row = dk + (int64_t)batch * dk_batch_stride + (int64_t)kidx * dk_row_stride + kv_head * D;
      __nv_bfloat16* dv_row = dv + (int64_t)batch * dv_batch_stride + (int64_t)kidx * dv_row_stride + kv_head * D;
#pragma unroll 1
      for (int n = part; n < 2 * (D / 32); n += Cfg::kParts) {
        const bool is_dk = n >= D / 32;
        const int c = is_dk ? n - D / 32 : n;
        __nv_bfloat16* dst = (is_dk ? dk_row : dv_row) + c * 32;
        const float sc = is_dk ? p.sm_scale : 1.f;
        uint32_t v[32];
        if (total > 0) {
          tmem_ld_32x32b_x32(tmem_base + (is_dk ? Cfg::kTmDk : Cfg::kTmDv) + lane_base + c * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;
        }
        if (kSplit && key_valid) {
          float* part = slabs + ((((int64_t)(2 * split + (is_dk ? 0 : 1)) * p.batch + batch) * p.seq_k + kidx) *
                                     p.kv_heads + kv_head) * D + c * 32;
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            *reinterpret_cast<uint4*>(part + 4 * q4) =
                make_uint4(v[4 * q4], v[4 * q4 + 1], v[4 * q4 + 2], v[4 * q4 + 3]);
        } else if (key_valid) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(v[8 * q4 + 0]) * sc, __uint_as_float(v[8 * q4 + 1]) * sc);
            o.y = pack_bf16x2(__uint_as_float(v[8 * q4 + 2]) * sc, __uint_as_float(v[8 * q4 + 3]) * sc);
            o.z = pack_bf16x2(__uint_as_float(v[8 * q4 + 4]) * sc, __uint_as_float(v[8 * q4 + 5]) * sc);
            o.w = pack_bf16x2(__uint_as_float(v[8 * q4 + 6]) * sc, __uint_as_float(v[8 * q4 + 7]) * sc);
            *reinterpret_cast<uint4*>(dst + q4 * 8) = o;
          }
        }
      }
    }
  }

  if (*abort_word) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == Cfg::kWarps + 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

template <int D, bool kSplit>
static int launch_bwd(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                      void* dk, void* dv, const float* delta, float* dq_accum, const PicoAttnParams* p,
                      int64_t do_batch_stride, int64_t do_row_stride, int64_t dk_batch_stride,
                      int64_t dk_row_stride, int64_t dv_batch_stride, int64_t dv_row_stride, float* slabs,
                      int splits, cudaStream_t stream) {
  using Cfg = BwdCfg<D>;
  BwdMaps maps;
  const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  int rc = pico_host::make_tmap_bshd(&maps.q, q, bf, 2, D, p->heads, p->seq_q, p->batch, p->q_row_stride * 2,
                                     p->q_batch_stride * 2, 64, kBM);
  if (rc) return rc;
  rc = pico_host::make_tmap_bshd(&maps.k, k, bf, 2, D, p->kv_heads, p->seq_k, p->batch, p->k_row_stride * 2,
                                 p->k_batch_stride * 2, 64, kBN);
  if (rc) return rc;
  rc = pico_host::make_tmap_bshd(&maps.v, v, bf, 2, D, p->kv_heads, p->seq_k, p->batch, p->v_row_stride * 2,
                                 p->v_batch_stride * 2, 64, kBN);
  if (rc) return rc;
  rc = pico_host::make_tmap_bshd(&maps.dout, dout, bf, 2, D, p->heads, p->seq_q, p->batch, do_row_stride * 2,
                                 do_batch_stride * 2, 64, kBM);
  if (rc) return rc;
  const uint64_t acc_row = (uint64_t)p->heads * D * 4;
  rc = pico_host::make_tmap_bshd(&maps.dq_accum, dq_accum, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, D, p->heads,
                                 p->seq_q, p->batch, acc_row, acc_row * p->seq_q, 32, kBM);
  if (rc) return rc;
  auto kern = flash_bwd_kernel<D, kSplit>;
  static int attr_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) {
      pico_host::set_error("attention bwd: cudaFuncSetAttribute(%d): %s", Cfg::kSmemBytes, cudaGetErrorString(e));
      return (int)e;
    }
    attr_dev = dev;
  }
  dim3 grid(p->kv_heads, p->batch, (p->seq_k + kBN - 1) / kBN * splits);
  pico_host::launch_ahead(kern, grid, Cfg::kThreads, Cfg::kSmemBytes, stream, maps, lse, delta, (__nv_bfloat16*)dk,
                          (__nv_bfloat16*)dv, *p, dk_batch_stride, dk_row_stride, dv_batch_stride, dv_row_stride,
                          slabs, splits, pico_status_buffer());
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    pico_host::set_error("attention bwd launch: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

}  // namespace pico

// How many CTAs share the steps of a key block: the smallest modelled time, in steps (1.7 us at head_dim 64, 2.9 at
// 128). CTAs are dealt heavy ones first, so the longest (under a causal mask that of the first keys, all query blocks
// of all heads of the group) or the mean sets the time, each with ~3 steps around its own; a split costs its slabs,
// written and read once, and ~2 steps for the longer post-pass. Measured, whole backward, us, unsplit / split: 1 x 8192
// x 4/1 heads x 128 (64 CTAs) 691 / 206; 4 x 2048 x 4/1 x 64 (64) 110 / 49; 1 x 4096 x 1 x 64 (32) 54 / 28; 1 x 256 x
// 9/3 x 64 (6) 17.9 / 15.8; where the model says no, 2 x 2048 x 8 x 128 (256): 70 / 111 in two.
extern "C" int pico_attention_bwd_splits(const PicoAttnParams* p) {
  const int64_t key_blocks = (p->seq_k + pico::kBN - 1) / pico::kBN, q_blocks = (p->seq_q + pico::kBM - 1) / pico::kBM;
  if (p->kv_heads <= 0 || p->batch <= 0 || key_blocks <= 0 || p->heads < p->kv_heads) return 1;
  const double sms = pico_host::num_sms(), ctas = (double)key_blocks * p->kv_heads * p->batch;
  if (ctas >= 4 * sms) return 1;
  const int64_t group = p->heads / p->kv_heads;
  int64_t longest = 0, sum = 0;
  for (int64_t j = 0; j < key_blocks; ++j) {
    int64_t seen = q_blocks;                           // query blocks that see a key of block j
    if (p->causal) {
      const int64_t need = (int64_t)p->k_pos0 + j * pico::kBN - p->q_pos0 - (pico::kBM - 1);
      seen -= need <= 0 ? 0 : (need + pico::kBM - 1) / pico::kBM;
    }
    if (seen <= 0) continue;
    longest = seen * group > longest ? seen * group : longest;
    sum += seen * group;
  }
  const double work = (double)sum * p->kv_heads * p->batch;
  // slab bytes per split at 5 TB/s, in steps
  const double slab = 16.0 * p->batch * p->seq_k * p->kv_heads * p->head_dim / 5e6 / (p->head_dim == 64 ? 1.7 : 2.9);
  int best = 1;
  // a split that is modelled to gain less than 15 % (as 3 x 1333 x 15/5 x 64, 69.0 / 69.9 in two) is left
  double best_time = 0;
  for (int n = 1; n <= 16 && n <= longest && key_blocks * n <= 65535; ++n) {
    const double own = (double)((longest + n - 1) / n) + 3, mean = (work + 3 * ctas * n) / sms;
    const double time = (own > mean ? own : mean) + (n > 1 ? 2 + n * slab : 0);
    if (n == 1) {
      best_time = time * 0.85;
    } else if (time < best_time) {
      best = n;
      best_time = time;
    }
  }
  return best;
}

extern "C" int pico_attention_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout,
                                  const float* lse, void* dq, void* dk, void* dv, float* delta, float* dq_accum,
                                  const PicoAttnParams* p, int64_t do_batch_stride, int64_t do_row_stride,
                                  int64_t dq_batch_stride, int64_t dq_row_stride, int64_t dk_batch_stride,
                                  int64_t dk_row_stride, int64_t dv_batch_stride, int64_t dv_row_stride,
                                  float* slabs, int splits, cudaStream_t stream) {
  using namespace pico;
  if (splits < 1 || (splits > 1 && slabs == nullptr)) {
    pico_host::set_error("attention bwd: %d splits need slabs", splits);
    return -2;
  }
  if (p->batch <= 0 || p->seq_q <= 0 || p->seq_k <= 0 || p->heads <= 0) return 0;
  if (p->head_dim != 64 && p->head_dim != 128) {
    pico_host::set_error("attention: head_dim %d not supported (64 or 128)", p->head_dim);
    return -2;
  }
  if (p->heads % p->kv_heads != 0) {
    pico_host::set_error("attention: heads (%d) must be a multiple of kv_heads (%d)", p->heads, p->kv_heads);
    return -2;
  }
  const int64_t rows = (int64_t)p->batch * p->seq_q * p->heads;
  const int sms = pico_host::num_sms();
  {
    int64_t blocks = (rows * (p->head_dim / 8) + 255) / 256;
    if (blocks > sms * 16) blocks = sms * 16;
    pico_host::launch_ahead(attn_delta_kernel, (int)blocks, 256, 0, stream, (const __nv_bfloat16*)out,
                            (const __nv_bfloat16*)dout, delta, dq_accum, *p, do_batch_stride, do_row_stride);
  }
  auto launch = p->head_dim == 64 ? (splits > 1 ? launch_bwd<64, true> : launch_bwd<64, false>)
                                  : (splits > 1 ? launch_bwd<128, true> : launch_bwd<128, false>);
  const int rc = launch(q, k, v, dout, lse, dk, dv, delta, dq_accum, p, do_batch_stride, do_row_stride, dk_batch_stride,
                        dk_row_stride, dv_batch_stride, dv_row_stride, slabs, splits, stream);
  if (rc) return rc;
  if (p->rope_cos != nullptr || splits > 1) {
    const int64_t items = (rows + (splits > 1 ? 2 : 1) * (int64_t)p->batch * p->seq_k * p->kv_heads) *
                          (p->head_dim / 16);
    int64_t blocks = (items + 255) / 256;
    if (blocks > sms * 16) blocks = sms * 16;
    pico_host::launch_ahead(p->rope_cos != nullptr ? attn_finish_kernel<true> : attn_finish_kernel<false>, (int)blocks,
                            256, 0, stream, dq_accum, slabs, splits, (__nv_bfloat16*)dq, (__nv_bfloat16*)dk,
                            (__nv_bfloat16*)dv, *p, dq_batch_stride, dq_row_stride, dk_batch_stride, dk_row_stride,
                            dv_batch_stride, dv_row_stride);
  } else {
    int64_t nvec = rows * p->head_dim / 8;
    int64_t blocks = (nvec + 255) / 256;
    if (blocks > sms * 16) blocks = sms * 16;
    pico_host::launch_ahead(attn_dq_convert_kernel, (int)blocks, 256, 0, stream, dq_accum, (__nv_bfloat16*)dq, *p,
                            dq_batch_stride, dq_row_stride);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    pico_host::set_error("attention bwd: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}
