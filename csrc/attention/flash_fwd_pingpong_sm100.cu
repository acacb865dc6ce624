// Flash attention forward for sm_100a, two query tiles per CTA.
//
// One CTA owns 256 query rows of one (batch, head) as two 128-row tiles A and B and walks the
// key/value sequence in blocks of 128. The score tiles are visited in the order
//   A(0) B(0) A(1) B(1) ...
// and score tile u lives in tensor-memory buffer u % kSBufs:
//
//   warps 0-3  : softmax of tile A  (one thread per query row, all 128 key columns of the block)
//   warps 4-7  : softmax of tile B
//   warp  8    : tcgen05.mma issue: S(u) = Q_t K_j^T and O_t += P(u) V_j
//   warp  9    : TMA loads (one thread): Q tiles once, K and V blocks into rings
//
// Tensor memory: kSBufs score buffers of 128 fp32 columns | O_A | O_B (head_dim columns each). At
// head_dim 64 there is room for three score buffers: S(u+3) is issued right behind the product
// that consumed P(u), so when a softmax group has published P(u) its next tile S(u+2) has been in
// tensor memory for half a period and the group never waits for the tensor cores. (Two buffers and
// the query tiles in tensor memory instead, the earlier form, needed 2250 cycles per 128x128 tile:
// each group waited for its own P V and Q K^T products every step, and the groups drifted into
// lock-step, competing for the exponential unit and then both waiting.) At head_dim 128 two
// buffers fill the 512 columns; there P is published in two halves so that P V of the first 64 keys
// runs under the exponentials of the rest.
//
// A softmax thread owns a whole row, so the row maximum and sum need no exchange between threads; the
// row stays in registers (the softmax warpgroups take the registers of the issue warps with
// setmaxnreg: 2 x 128 x 208 + 128 x 88 = 64512 = 384 x 168, what the block is launched with). P is
// written as packed bf16 pairs over the first 64 columns of its own score buffer and is the TMEM A
// operand of O_t += P V_j. The accumulator is rescaled lazily: only when the running maximum grew by
// more than 2^8, which the fp32 range of the un-normalised probabilities absorbs.
//
// Measured (causal, B200, one call after an L2 flush; before this form 218, 2111 and 206 us): 4 x 2048 x 32 heads x
// 64: 146 us; 1 x 16384 x 32/8 heads x 64: 1459 us; 1 x 4096 x 32 x 128: 154 us. At head_dim 64 the softmax warps never wait now
// (165 of 2700 cycles per pair of tiles); two threads per row, three-input maxima or a share of the
// exponentials on the FMA pipe changed that by less than 3 % or made it slower.
//
// Every wait is bounded (common/ptx.cuh); a CTA that gives up frees its TMEM and returns.
#include <cuda_bf16.h>
#include <math_constants.h>

#include <cstring>

#include "../common/host.h"
#include "../common/ptx.cuh"
#include "attention.h"

namespace pico {
namespace pp {

constexpr int kTileM = 128;            // rows of one query tile
constexpr int kCtaM = 2 * kTileM;      // rows per CTA
constexpr int kBlockN = 128;
constexpr int kGroupThreads = 128;
constexpr int kThreads = 3 * kGroupThreads;   // two softmax warpgroups, one with the issue warps
constexpr int kSoftmaxRegs = 208, kIssueRegs = 88;
static_assert(2 * kGroupThreads * kSoftmaxRegs + kGroupThreads * kIssueRegs <= kThreads * 168, "register split");
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescaleThreshold = 8.0f;

template <int D>
struct Cfg {
  static constexpr int kQBytes = kTileM * D * 2;          // one query tile
  static constexpr int kKVBytes = kBlockN * D * 2;        // one K or V block
  static constexpr int kKStages = (D == 64) ? 4 : 2;
  static constexpr int kVStages = (D == 64) ? 4 : 2;
  static constexpr int kSBufs = (D == 64) ? 3 : 2;        // score buffers in tensor memory
  static constexpr int kPParts = (D == 64) ? 1 : 2;       // pieces in which P is published
  static constexpr int kTiles = 2 * kQBytes + (kKStages + kVStages) * kKVBytes;
  // q_full[2], k_full/k_empty[kKStages], v_full/v_empty[kVStages], s_full[kSBufs],
  // p_ready[kSBufs][kPParts], pv_done[2]
  static constexpr int kNumBars = 2 + 2 * kKStages + 2 * kVStages + kSBufs + kSBufs * kPParts + 2;
  static constexpr int kSmemBytes = kTiles + kNumBars * 8 + 16;
  static constexpr int kTmemCols = 512;
  static constexpr int kTmO = kSBufs * kBlockN;
  static constexpr int kPanels = D / 64;
  static_assert(kTmO + 2 * D <= kTmemCols, "tensor memory");
};

struct Maps {
  CUtensorMap q, k, v;
};

// number of key blocks a tile whose last valid row is `last_row` (index in the local sequence) needs
__device__ __forceinline__ int blocks_needed(const PicoAttnParams& p, int first_row, int last_row) {
  if (last_row < first_row) return 0;
  int n = (p.seq_k + kBlockN - 1) / kBlockN;
  if (p.causal) {
    const int visible = p.q_pos0 + last_row - p.k_pos0 + 1;
    n = visible <= 0 ? 0 : min(n, (visible + kBlockN - 1) / kBlockN);
  }
  return n;
}

// Walks the score tiles of a CTA in issue order: A(0) B(0) A(1) ...; a tile that has no block j is left out.
// Carries the K or V ring position of its block j along (the issue warp has no cycles for divisions).
struct TileSeq {
  int t, j, stage;
  uint32_t parity;
  __device__ __forceinline__ TileSeq(int n0) : t(n0 > 0 ? 0 : 1), j(0), stage(0), parity(0) {}
  template <int kStages>
  __device__ __forceinline__ void next(int n0, int n1) {
    if (t == 0 && j < n1) {
      t = 1;
      return;
    }
    ++j;
    t = j < n0 ? 0 : 1;
    if (++stage == kStages) {
      stage = 0;
      parity ^= 1;
    }
  }
};

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
flash_fwd_pingpong_kernel(const __grid_constant__ Maps maps, __nv_bfloat16* __restrict__ out,
                          float* __restrict__ lse, const PicoAttnParams p, int* status) {
  using C = Cfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0) {   // swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) report_error(status, PICO_ERR_BOUNDS, 2999, (int)(smem_u32(smem) & 1023u));
    return;
  }
  uint8_t* sQ = smem;                                   // [2]
  uint8_t* sK = sQ + 2 * C::kQBytes;                    // [kKStages]
  uint8_t* sV = sK + C::kKStages * C::kKVBytes;         // [kVStages]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kTiles);
  uint64_t* q_full = bars;
  uint64_t* k_full = q_full + 2;
  uint64_t* k_empty = k_full + C::kKStages;
  uint64_t* v_full = k_empty + C::kKStages;
  uint64_t* v_empty = v_full + C::kVStages;
  uint64_t* s_full = v_empty + C::kVStages;
  uint64_t* p_ready = s_full + C::kSBufs;               // [buffer][part]
  uint64_t* pv_done = p_ready + C::kSBufs * C::kPParts; // one phase per P V product of the tile
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(pv_done + 2);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // warp-uniform
  const int lane = threadIdx.x & 31;
  // heavy (late) query tiles first so the causal triangle balances across the grid
  const int num_q = (p.seq_q + kCtaM - 1) / kCtaM;
  // blocks are dispatched x-fastest: every (head, batch) of the heaviest query block starts before
  // any lighter block, so the tail of the grid consists of the shortest CTAs
  const int q_blk = num_q - 1 - (int)blockIdx.z;
  const int head = blockIdx.x;
  const int batch = blockIdx.y;
  const int kv_head = head / (p.heads / p.kv_heads);
  const int q0 = q_blk * kCtaM;

  const int n0 = blocks_needed(p, q0, min(q0 + kTileM, p.seq_q) - 1);              // key blocks of tile A
  const int n1 = blocks_needed(p, q0 + kTileM, min(q0 + kCtaM, p.seq_q) - 1);      // ... of tile B
  const int n_max = max(n0, n1);

  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1);
      mbar_init(&pv_done[t], 1);
    }
    for (int s = 0; s < C::kKStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < C::kVStages; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int s = 0; s < C::kSBufs; ++s) mbar_init(&s_full[s], 1);
    for (int s = 0; s < C::kSBufs * C::kPParts; ++s) mbar_init(&p_ready[s], kGroupThreads);
    *abort_word = 0;
    mbar_fence_init();
    tma_prefetch_desc(&maps.q);
    tma_prefetch_desc(&maps.k);
    tma_prefetch_desc(&maps.v);
  }
  if (warp == 8) {
    tmem_alloc(tmem_ptr_smem, C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);
  ahead_wait();
  ahead_next();
  // optional timeline of the first CTA (performance debugging): SM clock stamps, 256 per role;
  // roles: 0 = softmax A (thread 0), 1 = softmax B (thread 128)
  const bool tracing = p.trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 &&
                       (threadIdx.x & 127) == 0;
  int trace_n = 0;
#define PP_STAMP(role)                                                                          \
  do {                                                                                          \
    if (tracing && trace_n < 256) p.trace[(role) * 256 + trace_n++] = (unsigned long long)clock64(); \
  } while (0)

  if (warp >= 8) {
    setmaxnreg_dec<kIssueRegs>();
    if (warp == 9 && lane == 0 && n_max > 0) {
      // -------------------------------------------------------------------------- TMA loads
      auto load_q = [&](int t) {
        mbar_arrive_expect_tx(&q_full[t], C::kQBytes);
#pragma unroll
        for (int pn = 0; pn < C::kPanels; ++pn)
          tma_load_4d(sQ + t * C::kQBytes + pn * 16384, &maps.q, &q_full[t], pn * 64, head, q0 + t * kTileM, batch);
      };
      if (n0 > 0) load_q(0);
      for (int j = 0; j < n_max; ++j) {
        const int ks = j % C::kKStages, vs = j % C::kVStages;
        if (j >= C::kKStages &&
            !mbar_wait(&k_empty[ks], ((j / C::kKStages) - 1) & 1, abort_word, status, 2010))
          break;
        mbar_arrive_expect_tx(&k_full[ks], C::kKVBytes);
#pragma unroll
        for (int pn = 0; pn < C::kPanels; ++pn)
          tma_load_4d(sK + ks * C::kKVBytes + pn * 16384, &maps.k, &k_full[ks], pn * 64, kv_head, j * kBlockN, batch);
        if (j == 0 && n1 > 0) load_q(1);
        if (j >= C::kVStages &&
            !mbar_wait(&v_empty[vs], ((j / C::kVStages) - 1) & 1, abort_word, status, 2011))
          break;
        mbar_arrive_expect_tx(&v_full[vs], C::kKVBytes);
#pragma unroll
        for (int pn = 0; pn < C::kPanels; ++pn)
          tma_load_4d(sV + vs * C::kKVBytes + pn * 16384, &maps.v, &v_full[vs], pn * 64, kv_head, j * kBlockN, batch);
      }
    } else if (warp == 8 && n_max > 0) {
      // -------------------------------------------------------------------------- MMA issue (converged warp)
      constexpr uint32_t idesc_s = umma_idesc_bf16(kTileM, kBlockN, 0, 0);
      constexpr uint32_t idesc_o = umma_idesc_bf16(kTileM, D, 0, 1);
      const int total = n0 + n1;
      const uint64_t q_desc = umma_smem_desc(smem_u32(sQ), 16, 1024), k_desc = umma_smem_desc(smem_u32(sK), 16, 1024);
      const uint64_t v_desc = umma_smem_desc(smem_u32(sV), 16384, 1024);
      // Each wait for operands comes before the wait for P, so that P V and the next Q K^T go out back to
      // back once P is there.
      auto wait_k = [&](const TileSeq& w) -> bool {
        if (w.j == 0 && !mbar_wait_warp(&q_full[w.t], 0, abort_word, status, 2000 + w.t)) return false;
        // the first tile that reads K_j waits for it to land
        return !(w.t == 0 || w.j >= n0) || mbar_wait_warp(&k_full[w.stage], w.parity, abort_word, status, 2020);
      };
      // S(u) = Q_t K_j^T into score buffer `buf`; releases K_j after its last reader
      auto issue_s = [&](const TileSeq& w, int buf) {
        const uint64_t q_d = q_desc + (uint32_t)(w.t * (C::kQBytes >> 4));
        const uint64_t k_d = k_desc + (uint32_t)(w.stage * (C::kKVBytes >> 4));
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          tc_mma_f16_ss_warp(tmem_base + buf * kBlockN, q_d + off, k_d + off, idesc_s, kk != 0 ? 1u : 0u);
        }
        tc_commit_warp(&s_full[buf]);
        if (w.t == 1 || w.j >= n1) tc_commit_warp(&k_empty[w.stage]);   // last reader of K_j
      };
      TileSeq ahead(n0), now(n0);
      int left = total;                 // score tiles not issued yet
      bool ok = true;
      for (int i = 0; i < C::kSBufs && left > 0 && ok; ++i, --left) {
        ok = wait_k(ahead);
        tc_fence_after();
        if (ok) issue_s(ahead, i);
        ahead.next<C::kKStages>(n0, n1);
      }
      int buf = 0;
      uint32_t parity = 0;
      for (int u = 0; u < total && ok; ++u) {
        // O_t += P(u) V_j, then S(u + kSBufs) over the buffer whose P that product reads
        if ((now.t == 0 || now.j >= n0) &&
            !mbar_wait_warp(&v_full[now.stage], now.parity, abort_word, status, 2040))
          break;
        if (left > 0 && !wait_k(ahead)) break;
        const uint64_t v_d = v_desc + (uint32_t)(now.stage * (C::kKVBytes >> 4));
        const uint32_t o_tmem = tmem_base + C::kTmO + now.t * D;
        const uint32_t p_tmem = tmem_base + buf * kBlockN;   // packed bf16 pairs over the first 64 columns
        constexpr int kSteps = kBlockN / 16 / C::kPParts;
#pragma unroll
        for (int part = 0; part < C::kPParts; ++part) {
          ok = ok && mbar_wait_warp(&p_ready[buf * C::kPParts + part], parity, abort_word, status, 2030 + part);
          tc_fence_after();
          if (ok) {
#pragma unroll
            for (int kk = part * kSteps; kk < (part + 1) * kSteps; ++kk)
              tc_mma_f16_ts_warp(o_tmem, p_tmem + kk * 8, v_d + (kk * 2048 >> 4), idesc_o,
                                 (now.j | kk) != 0 ? 1u : 0u);
          }
        }
        if (!ok) break;
        tc_commit_warp(&pv_done[now.t]);
        if (now.t == 1 || now.j >= n1) tc_commit_warp(&v_empty[now.stage]);  // last reader of V_j
        if (left > 0) {
          issue_s(ahead, buf);
          --left;
          ahead.next<C::kKStages>(n0, n1);
        }
        now.next<C::kVStages>(n0, n1);
        if (++buf == C::kSBufs) {
          buf = 0;
          parity ^= 1;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------------------- softmax + epilogue
    setmaxnreg_inc<kSoftmaxRegs>();
    const int t = warp >> 2;                        // tile of this group
    const int row = (warp & 3) * 32 + lane;         // row inside the tile = TMEM lane
    const int q_row = q0 + t * kTileM + row;        // row in the local query sequence
    const bool valid_row = q_row < p.seq_q;
    const int q_pos = p.q_pos0 + q_row;
    const float scale_log2 = p.sm_scale * kLog2e;
    const uint64_t scale2 = f2_pack(scale_log2, scale_log2);
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tmem_o = tmem_base + C::kTmO + t * D + lane_base;
    const int n_mine = t == 0 ? n0 : n1;
    float m_run = -CUDART_INF_F;   // running max of the scaled scores (log2 units)
    float l_run = 0.f;
    bool alive = true;
    // keys with index >= k_limit are invisible to this row
    int k_limit = p.seq_k;
    if (p.causal) k_limit = min(k_limit, q_pos - p.k_pos0 + 1);
    for (int j = 0; j < n_mine; ++j) {
      const int u = t == 0 ? j + min(j, n1) : j + min(j + 1, n0);    // place in the issue order
      const int buf = u % C::kSBufs;
      const uint32_t tmem_s = tmem_base + buf * kBlockN + lane_base;
      PP_STAMP(t);
      // warp-uniform outcome: the lanes of a warp stay together through the votes below
      if (!__all_sync(0xffffffffu, mbar_wait(&s_full[buf], (u / C::kSBufs) & 1, abort_word, status, 2100 + t))) {
        alive = false;
        break;
      }
      tc_fence_after();
      PP_STAMP(t);
      const int k_base = j * kBlockN;
      const bool need_mask =
          (p.causal && (p.k_pos0 + k_base + kBlockN - 1 > p.q_pos0 + q0 + t * kTileM)) || (k_base + kBlockN > p.seq_k);
      // the whole S row (128 fp32) comes into registers with four loads in flight and one wait
      uint32_t sv[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(tmem_s + c * 32, sv[c]);
      tmem_ld_wait();
      // ---- masking: on the few blocks that need it (diagonal, ragged end) invisible scores become
      // -inf in place, so the arithmetic below exists only once in the instruction stream
      // (exp2(-inf) = 0; the kernel is large enough for instruction fetch to matter)
      if (need_mask) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int lim = k_limit - (k_base + c * 32);   // columns [0, lim) of the chunk are visible
#pragma unroll
          for (int i = 0; i < 32; ++i)
            sv[c][i] = i < lim ? sv[c][i] : __float_as_uint(-CUDART_INF_F);
        }
      }
      // ---- row maximum: four chains of three-input maxima
      float mx;
      {
        float m[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          m[c] = fmaxf(__uint_as_float(sv[c][0]), __uint_as_float(sv[c][1]));
#pragma unroll
          for (int i = 2; i < 32; i += 2)
            m[c] = fmaxf(fmaxf(m[c], __uint_as_float(sv[c][i])), __uint_as_float(sv[c][i + 1]));
        }
        mx = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
      }
      mx *= scale_log2;   // scale > 0, so the maximum commutes with the scaling (-inf stays -inf)
      const float m_new = fmaxf(m_run, mx);
      const bool grow = (m_new - m_run > kRescaleThreshold) || (m_run == -CUDART_INF_F);
      const float m_use = grow ? m_new : m_run;
      const float alpha = (m_run == -CUDART_INF_F) ? 0.f : exp2f(m_run - m_use);
      // Each phase of pv_done is waited for once, before this group publishes the P of the next product
      // (a parity wait must be less than two phases behind): here if the accumulator has to be
      // rescaled, else below, where the product has long been done.
      bool pv_seen = j == 0;
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        pv_seen = true;
        if (!__all_sync(0xffffffffu, mbar_wait(&pv_done[t], (j - 1) & 1, abort_word, status, 2110 + t))) {
          alive = false;
          break;
        }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tmem_o + c * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
          tmem_st_32x32b_x32(tmem_o + c * 32, v);
        }
        tmem_st_wait();
      }
      l_run *= alpha;
      m_run = m_use;
      // ---- probabilities -> packed bf16 P over the first 64 columns of the buffer, row sum
      // exp2(s*scale - m) is one fused multiply-add per element; a row that has seen no key yet
      // (m = -inf) uses offset 0: all its scores are -inf and give 0
      const float neg_m = (m_run == -CUDART_INF_F) ? 0.f : -m_run;
      const uint64_t neg_m2 = f2_pack(neg_m, neg_m);
      uint64_t sum[4] = {0, 0, 0, 0};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float e0, e1;
          f2_unpack(f2_fma(f2_pack(__uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1])), scale2, neg_m2), e0, e1);
          e0 = exp2f(e0);
          e1 = exp2f(e1);
          sum[(i >> 1) & 3] = f2_add(sum[(i >> 1) & 3], f2_pack(e0, e1));
          pk[i / 2] = pack_bf16x2(e0, e1);
        }
        tmem_st_32x32b_x16(tmem_s + c * 16, pk);
        if (((c + 1) * C::kPParts) % 4 == 0) {     // this part of P is complete
          tmem_st_wait();
          if (!pv_seen) {
            pv_seen = true;
            alive = __all_sync(0xffffffffu, mbar_wait(&pv_done[t], (j - 1) & 1, abort_word, status, 2105 + t));
          }
          tc_fence_before();
          mbar_arrive(&p_ready[buf * C::kPParts + ((c + 1) * C::kPParts) / 4 - 1]);
        }
      }
      {
        float a, b;
        f2_unpack(f2_add(f2_add(sum[0], sum[1]), f2_add(sum[2], sum[3])), a, b);
        l_run += a + b;
      }
      PP_STAMP(t);
      if (!alive) break;
    }
    // ---- epilogue: normalise and store this thread's output row
    if (alive) {
      bool ok = true;
      if (n_mine > 0)
        ok = __all_sync(0xffffffffu, mbar_wait(&pv_done[t], (n_mine - 1) & 1, abort_word, status, 2200 + t));
      if (ok) {
        tc_fence_after();
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        __nv_bfloat16* orow =
            out + (int64_t)batch * p.o_batch_stride + (int64_t)q_row * p.o_row_stride + head * D;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t v[32];
          if (n_mine > 0) {
            tmem_ld_32x32b_x32(tmem_o + c * 32, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          if (valid_row) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(v[8 * q4 + 0]) * inv, __uint_as_float(v[8 * q4 + 1]) * inv);
              o.y = pack_bf16x2(__uint_as_float(v[8 * q4 + 2]) * inv, __uint_as_float(v[8 * q4 + 3]) * inv);
              o.z = pack_bf16x2(__uint_as_float(v[8 * q4 + 4]) * inv, __uint_as_float(v[8 * q4 + 5]) * inv);
              o.w = pack_bf16x2(__uint_as_float(v[8 * q4 + 6]) * inv, __uint_as_float(v[8 * q4 + 7]) * inv);
              *reinterpret_cast<uint4*>(orow + c * 32 + q4 * 8) = o;
            }
          }
        }
        if (valid_row && lse != nullptr) {
          const float val = l_run > 0.f ? (m_run + log2f(l_run)) / kLog2e : -CUDART_INF_F;
          lse[((int64_t)batch * p.heads + head) * p.seq_q + q_row] = val;
        }
      }
    }
  }

  // ---------------------------------------------------------------------- teardown
  if (*abort_word) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <int D>
static int launch(const void* q, const void* k, const void* v, void* out, float* lse, const PicoAttnParams* p,
                  cudaStream_t stream) {
  using C = Cfg<D>;
  Maps maps;
  int rc = pico_host::make_tmap_bshd(&maps.q, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, D, p->heads, p->seq_q,
                                     p->batch, p->q_row_stride * 2, p->q_batch_stride * 2, 64, kTileM);
  if (rc) return rc;
  rc = pico_host::make_tmap_bshd(&maps.k, k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, D, p->kv_heads, p->seq_k,
                                 p->batch, p->k_row_stride * 2, p->k_batch_stride * 2, 64, kBlockN);
  if (rc) return rc;
  rc = pico_host::make_tmap_bshd(&maps.v, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, D, p->kv_heads, p->seq_k,
                                 p->batch, p->v_row_stride * 2, p->v_batch_stride * 2, 64, kBlockN);
  if (rc) return rc;
  auto kern = flash_fwd_pingpong_kernel<D>;
  static int attr_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) {
      pico_host::set_error("attention fwd: cudaFuncSetAttribute(%d): %s", C::kSmemBytes, cudaGetErrorString(e));
      return (int)e;
    }
    attr_dev = dev;
  }
  dim3 grid(p->heads, p->batch, (p->seq_q + kCtaM - 1) / kCtaM);
  pico_host::launch_ahead(kern, grid, kThreads, C::kSmemBytes, stream, maps, (__nv_bfloat16*)out, lse, *p,
                          pico_status_buffer());
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    pico_host::set_error("attention fwd launch: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

}  // namespace pp
}  // namespace pico

extern "C" int pico_attention_fwd(const void* q, const void* k, const void* v, void* out, float* lse,
                                  const PicoAttnParams* p, cudaStream_t stream) {
  if (p->batch <= 0 || p->seq_q <= 0 || p->heads <= 0) return 0;
  if (p->heads % p->kv_heads != 0) {
    pico_host::set_error("attention: heads (%d) must be a multiple of kv_heads (%d)", p->heads, p->kv_heads);
    return -2;
  }
  if ((p->o_row_stride % 8) != 0 || (p->o_batch_stride % 8) != 0 || (reinterpret_cast<uintptr_t>(out) & 15)) {
    pico_host::set_error("attention: output must be 16-byte aligned with strides that are multiples of 8");
    return -2;
  }
  if (p->head_dim == 64) return pico::pp::launch<64>(q, k, v, out, lse, p, stream);
  if (p->head_dim == 128) return pico::pp::launch<128>(q, k, v, out, lse, p, stream);
  pico_host::set_error("attention: head_dim %d not supported (64 or 128)", p->head_dim);
  return -2;
}
