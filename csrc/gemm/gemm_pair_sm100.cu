// Persistent bf16 GEMM for sm_100a on CTA pairs (tcgen05 cta_group::2).
//
//   D[M,N] (=|+=) op(A)[M,K] * op(B)[K,N]        fp32 accumulation in tensor memory
//
// Two CTAs on neighbouring SMs form a cluster and work on one 256 x BN tile: each holds 128 rows of A
// and BN/2 columns of B in its shared memory and 128 rows of the accumulator in its tensor memory.
// What binds the one-CTA kernel (gemm_bf16_sm100.cu) at large sizes is operand traffic: a 128 x 256
// tile brings 48 KB from L2 for each 64-deep K slice and reads all of it from shared memory again. A
// pair brings 32 KB per SM for the same work, so the ring is 6 stages deep instead of 4, and
// draws less power, which is what sets the clock in a long step. A 256 x 128 tile measured two thirds of
// the rate of 256 x 256 (1019 against 1540 TFLOP/s at 8192 x 2048 x 2048 in whole rounds), so BN is 256.
//
// Roles in each CTA:
//   warp 0    : TMA producer  - this CTA's halves of A and B; both CTAs' copies complete on the
//                               first CTA's barrier
//   warp 1    : MMA issuer    - first CTA only; its commits release the stage in both CTAs
//   warps 2-5 : epilogue      - this CTA's 128 rows: tcgen05.ld, convert, swizzled staging, TMA store
//                               (or TMA reduce-add for D +=); accumulators are double buffered
// SwiGLU tiles have eight epilogue warps, 2-9, two for each quarter of the accumulator's lanes, and
//   warps 10, 11: movers      - bring what the epilogue reads into the staging buffers ahead of it (it works in place)
//                               and send its results away
//
// SwiGLU epilogues, for the gated MLP y = (silu(x Wg^T) * (x Wu^T)) Wd^T:
//   forward : a tile has 128 gate columns and the same 128 up columns (the first CTA loads the rows of Wg, the second
//             those of Wu); gate | up and the activation leave from the same registers
//   backward: the gradient of the activation, dy Wd, meets gate and up in the epilogue and leaves as their gradients;
//             it is never stored
// What a pass of its own over gate | up took (402 MB forward, 671 MB backward for 8192 rows of 2 x 8192) then runs
// under the main loop, 16 thousand cycles per tile at K = 2048. Values are rounded to bf16 before the activation, as
// that pass reads them. Product and pass / fused, us: 8192 rows, 2048 -> 8192: forward 420 / 363, backward 306 / 226;
// 16384, 2048 -> 5632: 566 / 496, 414 / 338; 8192, 960 -> 2560: 77 / 65, 71 / 55 (eight in a row on another machine:
// 412 / 356, 326 / 246; 573 / 503, 440 / 321; 98 / 77, 80 / 61). The movers' four buffers cost a stage of operands; six
// buffers and four stages measured 393 and 284 us in the first line, and with four epilogue warps the short ones 1 us
// more.
//
// Work split: output tiles are dealt to the pairs in whole rounds; where D is accumulated (weight
// gradients) the tiles of the last, partial round are cut along K into equal shares for all pairs, so that
// round costs its share and not a whole one (256 tiles on 74 pairs: 3.46 rounds instead of 4). A share is
// shorter than a tile, so a pair has at most one piece that does not begin its tile. That one goes to the pair's own
// fp32 slab; the first piece of a tile is added to D like a whole tile, and add_pieces_kernel then adds the slabs to D
// in the order of K: the same bits on each run. (Reduce-adding every piece to D needs no second kernel, but then the
// sums depend on which pair is done first.) Measured, dW += dY^T X of 8192 tokens, uncut, cut, cut without an order:
// 6144 x 2048 165, 158, 149 us; 960 x 960 (16 tiles) 52, 29, 24 us; 2048 x 2048 (64 tiles) 67, 77, 66 us.
//
// Row groups (the experts' products: rows of A and D in segments of whole 128-row tiles, one matrix B each): a pair
// takes two neighbouring row tiles of one group, so each CTA's half of B serves both. The last tile of an odd segment
// goes alone, its second CTA's rows are computed and dropped. Which tiles lead a pair is found at the start of the
// kernel from the group of every row tile: no host read, no layout beside the one-CTA kernel's. One CTA / pairs, us:
// 49152 rows of 64 experts, 2048 -> 2 x 1024 with the activation 427 / 373, its backward 286 / 231, 2048 x 1024 200 /
// 189; 8192 rows of 8 experts 70 / 60, 48 / 39, 34 / 31.
//
// Reduction groups (the experts' weight gradients: D a stack of [M, N] blocks, each summed over its own stretch of K):
// the tiles of all groups in turn, none cut. With K short the fp32 reductions bind them more than the tensor cores (4.1
// TB/s read and written). One CTA / pairs, us: 64 experts, 53248 rows, 2048 x 2048 539 / 515, 2048 x 1024 308 / 259.
//
// Operand layouts and raggedness as in gemm_bf16_sm100.cu.
#include <cuda_bf16.h>

#include <cstring>

#include "../common/host.h"
#include "../common/ptx.cuh"
#include "gemm_kernels.h"

namespace pico {
namespace pair {

constexpr int BM = 128;                   // rows of one CTA; a pair works on 2 * BM
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int kStagingBytes = 128 * 128;

constexpr int kMaxRowTiles = 640;         // of a product with row groups; their list takes the rest of shared memory

enum Groups : int { kNoGroups, kRowGroups, kSumGroups };

template <int BN, int OUT, int kGroups = kNoGroups>
struct Cfg {
  static constexpr bool kGate = OUT == GEMM_OUT_SWIGLU, kGateBwd = OUT == GEMM_OUT_SWIGLU_BWD;
  static constexpr bool kMovers = kGate || kGateBwd;
  static constexpr int kEpilogueThreads = kMovers ? 256 : 128;
  static constexpr int kFirstMover = 2 + kEpilogueThreads / 32;
  static constexpr int kThreads = 64 + kEpilogueThreads + (kMovers ? 64 : 0);
  static constexpr int kABytes = BM * BK * 2;
  static constexpr int kBBytes = (BN / 2) * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = kMovers ? 5 : 6;
  static constexpr int kNumStaging = kMovers ? 4 : 2;
  static constexpr int kTiles = kStages * kStageBytes + kNumStaging * kStagingBytes;
  static constexpr int kSmemBytes = kTiles + (2 * kStages + 4 + 3 * kNumStaging) * 8 + 16 +
                                    (kGroups == kRowGroups ? kMaxRowTiles * 4 : 0);
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");
  static constexpr int kTmemCols = 2 * BN;
};

// One stretch of work of a pair: K blocks [kb0, kb1) of output tile (m, n), in units of pair tiles.
// With row groups: the rows begin at `row`, the second CTA has none where the tile is alone, B is that of group grp.
struct Work {
  int m, n, kb0, kb1;
  int row, grp;                             // reduction groups: D's block is `grp`
  bool alone;
};

// The output tiles and the order in which they are worked on.
struct Tiles {
  int num_m, num_n, num_kb;

  __device__ __forceinline__ Tiles(int M, int N, int K, int BN)
      : num_m((M + 2 * BM - 1) / (2 * BM)), num_n((N + BN - 1) / BN), num_kb((K + BK - 1) / BK) {}
  // consecutive tiles (= pairs running at the same time) cover a compact block of the output so
  // that slices of A and B are shared through L2
  __device__ __forceinline__ void place(int tile, Work& w) const {
    constexpr int kGroup = 8;
    const int per_group = kGroup * num_n;
    const int g = tile / per_group;
    const int first_m = g * kGroup;
    const int gsize = min(kGroup, num_m - first_m);
    const int r = tile - g * per_group;
    w.m = first_m + r % gsize;
    w.n = r / gsize;
  }
};

// Walks a pair's work: whole tiles first, then its share of the tiles that are cut along K.
template <int kGroups>
struct Schedule : Tiles {
  const int* seg_start;                     // reduction groups: where each begins in K
  const uint32_t* lead;                     // row groups: the row tiles that lead a pair, see list_pairs
  int whole, pairs;                         // `whole` tiles are not cut
  int next;                                 // next whole tile of this pair
  int64_t unit, unit_end;                   // this pair's K blocks of the cut tiles

  __device__ __forceinline__ Schedule(int M, int N, int K, int BN, int whole_, int pair_id, int pairs_,
                                      const uint32_t* lead_, int num_lead, const int* seg_start_)
      : Tiles(M, N, K, BN), seg_start(seg_start_), lead(lead_), whole(whole_), pairs(pairs_), next(pair_id) {
    if (kGroups == kRowGroups) {
      num_m = num_lead;
      whole = num_m * num_n;
    }
    const int64_t units = kGroups == kSumGroups ? 0 : (int64_t)(num_m * num_n - whole) * num_kb;
    unit = units * pair_id / pairs;
    unit_end = units * (pair_id + 1) / pairs;
  }
  __device__ __forceinline__ bool get(Work& w) {
    int tile;
    if (kGroups == kSumGroups) {
      const int per_group = num_m * num_n;
      do {
        if (next >= whole) return false;
        tile = next;
        next += pairs;
        w.grp = tile / per_group;
        tile -= w.grp * per_group;
        w.kb0 = __ldg(seg_start + w.grp) / BK;
        w.kb1 = __ldg(seg_start + w.grp + 1) / BK;
      } while (w.kb1 <= w.kb0);
    } else if (next < whole) {
      tile = next;
      next += pairs;
      w.kb0 = 0;
      w.kb1 = num_kb;
    } else if (unit < unit_end) {
      const int64_t t = unit / num_kb;
      tile = whole + (int)t;
      w.kb0 = (int)(unit - t * num_kb);
      const int64_t left = unit_end - unit;
      w.kb1 = (int)min((int64_t)num_kb, w.kb0 + left);
      unit += w.kb1 - w.kb0;
    } else {
      return false;
    }
    place(tile, w);
    w.row = w.m * 2 * BM;
    w.alone = false;
    if (kGroups == kRowGroups) {
      const uint32_t e = lead[w.m];
      w.row = (int)(e & 0x7fffu) * BM;
      w.alone = (e & 0x8000u) == 0;
      w.grp = (int)(e >> 16);
    }
    return true;
  }
};

// The row tiles that lead a pair: those at an even place in their segment. Entry: the tile | 0x8000 where the next tile
// is of the same group | group << 16. Called by one warp; returns their number.
__device__ __forceinline__ int list_pairs(const int* __restrict__ tile_group, int num_tiles, uint32_t* list, int lane) {
  int count = 0, begin = 0, prev = -2;               // begin: of the segment that the tiles before this stretch end in
  for (int base = 0; base < num_tiles; base += 32) {
    const int t = base + lane;
    const int g = t < num_tiles ? __ldg(tile_group + t) : -1;
    const int after = t + 1 < num_tiles ? __ldg(tile_group + t + 1) : -1;
    int before = __shfl_up_sync(0xffffffffu, g, 1);
    if (lane == 0) before = prev;
    const uint32_t begins = __ballot_sync(0xffffffffu, g != before);
    const uint32_t upto = begins & (0xffffffffu >> (31 - lane));
    const int seg = upto != 0 ? base + 31 - __clz(upto) : begin;
    const bool leads = g >= 0 && ((t - seg) & 1) == 0;
    const uint32_t all = __ballot_sync(0xffffffffu, leads);
    if (leads) list[count + __popc(all & ((1u << lane) - 1u))] =
        (uint32_t)t | (after == g ? 0x8000u : 0u) | ((uint32_t)g << 16);
    count += __popc(all);
    if (begins != 0) begin = base + 31 - __clz(begins);
    prev = __shfl_sync(0xffffffffu, g, 31);
  }
  return count;
}

// What an epilogue reads and writes.
struct OutMaps {
  CUtensorMap d;                // D; SwiGLU forward: the activation
  CUtensorMap slabs;            // of the cut tiles
  CUtensorMap gate, up;         // SwiGLU: written forward, read backward
  CUtensorMap d_gate, d_up;     // their gradients
};

// The buffers of the staging ring in their order of use, and the parity of the rounds it has made.
template <int kCount>
struct Ring {
  int b = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++b == kCount) {
      b = 0;
      phase ^= 1;
    }
  }
};

__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ float swiglu(float g, float u) { return g / (1.f + __expf(-g)) * u; }
// gradients of gate (returned) and up
__device__ __forceinline__ float swiglu_grad(float g, float u, float d, float& du) {
  const float sg = 1.f / (1.f + __expf(-g));
  du = d * (g * sg);
  return d * u * sg * (1.f + g * (1.f - sg));
}

template <int BN, int A_MN, int B_MN, int OUT, int kGroups>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Cfg<BN, OUT, kGroups>::kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const __grid_constant__ OutMaps out, int M, int N, int K, int whole, int keep_gate,
                 const int* group_array, int* status) {
  using C = Cfg<BN, OUT, kGroups>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* staging = smem + C::kStages * C::kStageBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + C::kTiles);
  uint64_t* empty_bar = full_bar + C::kStages;
  uint64_t* tmem_full = empty_bar + C::kStages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* in_full = tmem_empty + 2;             // movers only, per staging buffer: the epilogue may work on it,
  uint64_t* out_full = in_full + C::kNumStaging;  // is done,
  uint64_t* out_sent = out_full + C::kNumStaging; // and the result has been read from it
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(out_sent + C::kNumStaging);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  if ((smem_u32(smem) & 1023u) != 0) {   // swizzled tiles need 1024-byte alignment; the same in both CTAs
    if (threadIdx.x == 0) report_error(status, PICO_ERR_BOUNDS, 998, (int)(smem_u32(smem) & 1023u));
    return;
  }

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // warp-uniform
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();        // 0 issues the MMAs
  const int pair_id = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], C::kMovers ? 16 : 2);  // from each CTA's epilogue: one arrival, or one of each warp
    }
    for (int b = 0; b < C::kNumStaging; ++b) {
      mbar_init(&in_full[b], 1);
      mbar_init(&out_full[b], C::kEpilogueThreads);
      mbar_init(&out_sent[b], 1);
    }
    *abort_word = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(C::kGateBwd ? &out.gate : &out.d);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_ptr_smem, C::kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                             // the other CTA's barriers exist before anything arrives there
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);
  ahead_wait();
  ahead_next();
  uint32_t* lead = reinterpret_cast<uint32_t*>(const_cast<int*>(abort_word) + 2);
  int num_lead = 0;
  if (kGroups == kRowGroups) {
    if (warp == 0) {
      const int n = list_pairs(group_array, (M + BM - 1) / BM, lead, lane);
      if (lane == 0) abort_word[1] = n;
    }
    __syncthreads();
    num_lead = abort_word[1];
  }
  Schedule<kGroups> sched(M, N, K, BN, whole, pair_id, pairs, lead, num_lead, group_array);
  Work w;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      while (ok && sched.get(w)) {
        const int m0 = w.row + (int)rank * BM;
        const int b0 = kGroups != kRowGroups ? 0 : w.grp * (B_MN == 0 ? N : K);   // this group's B in the stack
        // SwiGLU forward: gate columns in the first CTA, the up columns of the same numbers in the second
        const int n0 = C::kGate ? w.n * (BN / 2) + (int)rank * (N / 2) : w.n * BN + (int)rank * (BN / 2);
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_wait(&empty_bar[s], phase ^ 1, abort_word, status, 100 + s)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + s * C::kStageBytes;
          uint8_t* sb = sa + C::kABytes;
          // both CTAs' bytes are counted on the first CTA's barrier
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * C::kStageBytes);
          const uint32_t bar = cluster_map(&full_bar[s], 0);
          const int k0 = kb * BK;
          if (A_MN == 0) {
            tma_load_2d_pair(sa, &tmap_a, bar, k0, m0);  // box 64(K) x 128(M)
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)            // boxes 64(M) x 64(K)
              tma_load_2d_pair(sa + j * (64 * BK * 2), &tmap_a, bar, m0 + j * 64, k0);
          }
          if (B_MN == 0) {
            tma_load_2d_pair(sb, &tmap_b, bar, k0, b0 + n0);  // box 64(K) x BN/2
          } else {
#pragma unroll
            for (int j = 0; j < BN / 128; ++j)           // boxes 64(N) x 64(K)
              tma_load_2d_pair(sb + j * (64 * BK * 2), &tmap_b, bar, n0 + j * 64, b0 + k0);
          }
          if (++s == C::kStages) {
            s = 0;
            phase ^= 1;
          }
        }
      }
      // The commits that release the last stages arrive here from the first CTA's tensor core, which no barrier of its
      // threads orders: neither CTA may go away before they have (a stage that was never filled counts as released).
      for (int i = 0; ok && i < C::kStages; ++i) {
        ok = mbar_wait(&empty_bar[s], phase ^ 1, abort_word, status, 150 + s);
        if (++s == C::kStages) {
          s = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (converged warp)
    if (rank == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      // descriptors of the first stage; a stage further is kStageStep further
      constexpr uint32_t kStageStep = C::kStageBytes >> 4;
      const uint64_t a_desc = umma_smem_desc(smem_u32(smem), A_MN == 0 ? 16 : 64 * BK * 2, 1024);
      const uint64_t b_desc = umma_smem_desc(smem_u32(smem) + C::kABytes, B_MN == 0 ? 16 : 64 * BK * 2, 1024);
      int s = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      while (ok && sched.get(w)) {
        if (!mbar_wait_warp(&tmem_empty[acc], acc_phase ^ 1, abort_word, status, 200 + acc)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_wait_warp(&full_bar[s], phase, abort_word, status, 300 + s)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t a_d = a_desc + (uint32_t)s * kStageStep, b_d = b_desc + (uint32_t)s * kStageStep;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            // K-major: step 32 bytes inside the swizzle row; MN-major: step 16 k-rows.
            constexpr uint32_t kStepA = (A_MN == 0 ? UMMA_K * 2 : UMMA_K * 128) >> 4;
            constexpr uint32_t kStepB = (B_MN == 0 ? UMMA_K * 2 : UMMA_K * 128) >> 4;
            tc_mma_f16_ss_pair(d_tmem, a_d + k * kStepA, b_d + k * kStepB, idesc, ((kb - w.kb0) | k) != 0 ? 1u : 0u);
          }
          tc_commit_pair(&empty_bar[s]);  // stage reusable in both CTAs once these MMAs have read it
          if (++s == C::kStages) {
            s = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        tc_commit_pair(&tmem_full[acc]);  // accumulator complete
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else if (warp >= C::kFirstMover) {
    // ------------------------------------------------------------------ loads (first) and stores (second) of staging
    if (lane == 0) {
      Ring<C::kNumStaging> r;
      bool ok = true;
      // one buffer: fetched from `src` (NULL: nothing to fetch), sent to the same place of `dst`
      auto move = [&](const CUtensorMap* src, const CUtensorMap* dst, int x, int y) {
        uint8_t* sbuf = staging + r.b * kStagingBytes;
        if (warp == C::kFirstMover) {
          ok = ok && mbar_wait(&out_sent[r.b], r.phase ^ 1, abort_word, status, 500 + r.b);
          if (!ok) return;
          if (src == nullptr) {
            mbar_arrive(&in_full[r.b]);
          } else {
            mbar_arrive_expect_tx(&in_full[r.b], kStagingBytes);
            tma_load_2d(sbuf, src, &in_full[r.b], x, y);
          }
        } else {
          ok = ok && mbar_wait(&out_full[r.b], r.phase, abort_word, status, 550 + r.b);
          if (!ok) return;
          tma_store_2d(dst, sbuf, x, y);
          tma_store_commit();
          tma_store_wait_read<0>();
          mbar_arrive(&out_sent[r.b]);
        }
        r.next();
      };
      while (ok && sched.get(w)) {
        const int m0 = w.row + (int)rank * BM;
        if (m0 >= M || (kGroups == kRowGroups && rank != 0 && w.alone)) continue;
        if (C::kGate) {
          const int n0 = w.n * (BN / 2);
          for (int c = 0; ok && c < BN / 128 && n0 + c * 64 < N / 2; ++c) {
            if (keep_gate) {
              move(nullptr, &out.gate, n0 + c * 64, m0);
              move(nullptr, &out.up, n0 + c * 64, m0);
            }
            move(nullptr, &out.d, n0 + c * 64, m0);
          }
        } else {
          const int n0 = w.n * BN;
          for (int c = 0; ok && c < BN / 64 && n0 + c * 64 < N; ++c) {
            move(&out.gate, &out.d_gate, n0 + c * 64, m0);
            move(&out.up, &out.d_up, n0 + c * 64, m0);
          }
        }
      }
      if (warp != C::kFirstMover) tma_store_wait<0>();
    }
  } else if (C::kMovers) {
    // ------------------------------------------------------------------ epilogue in the movers' buffers
    const int quarter = warp & 3;                 // TMEM lane quarter this warp may access
    const int h = (warp - 2) >> 2;                // and the 32 of a chunk's 64 columns it works on
    const int row = quarter * 32 + lane;          // row of this CTA's half tile owned by this thread
    Ring<C::kNumStaging> r;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    // this thread's row of the buffer whose turn it is, once it may be worked on
    auto take = [&]() {
      ok = ok && mbar_wait_warp(&in_full[r.b], r.phase, abort_word, status, 600 + r.b);
      return staging + r.b * kStagingBytes + row * 128;
    };
    while (ok && sched.get(w)) {
      const int m0 = w.row + (int)rank * BM;
      if (!mbar_wait_warp(&tmem_full[acc], acc_phase, abort_word, status, 400 + acc)) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + acc * BN + ((uint32_t)(quarter * 32) << 16);
      if (m0 >= M || (kGroups == kRowGroups && rank != 0 && w.alone)) {
        // nothing of this CTA's half lies in D
      } else if (C::kGate) {
        const int n0 = w.n * (BN / 2);
#pragma unroll 1
        for (int c = 0; c < BN / 128 && n0 + c * 64 < N / 2; ++c) {
          int bufs[3] = {0, 0, 0};
          uint8_t* rows[3] = {staging, staging, staging};
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            if (i < 2 && !keep_gate) continue;
            rows[i] = take();
            bufs[i] = r.b;
            r.next();
          }
          if (!ok) break;
          uint32_t g[32], u[32];
          tmem_ld_32x32b_x32(t_row + c * 64 + h * 32, g);
          tmem_ld_32x32b_x32(t_row + BN / 2 + c * 64 + h * 32, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t gw[4], uw[4], aw[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int e = 8 * j + 2 * i;
              gw[i] = pack_bf16x2(__uint_as_float(g[e]), __uint_as_float(g[e + 1]));
              uw[i] = pack_bf16x2(__uint_as_float(u[e]), __uint_as_float(u[e + 1]));
              aw[i] = pack_bf16x2(swiglu(bf16_lo(gw[i]), bf16_lo(uw[i])), swiglu(bf16_hi(gw[i]), bf16_hi(uw[i])));
            }
            const int at = ((h * 4 + j) ^ (row & 7)) << 4;
            if (keep_gate) {
              *reinterpret_cast<uint4*>(rows[0] + at) = make_uint4(gw[0], gw[1], gw[2], gw[3]);
              *reinterpret_cast<uint4*>(rows[1] + at) = make_uint4(uw[0], uw[1], uw[2], uw[3]);
            }
            *reinterpret_cast<uint4*>(rows[2] + at) = make_uint4(aw[0], aw[1], aw[2], aw[3]);
          }
          fence_proxy_async_smem();
          if (keep_gate) {
            mbar_arrive(&out_full[bufs[0]]);
            mbar_arrive(&out_full[bufs[1]]);
          }
          mbar_arrive(&out_full[bufs[2]]);
        }
      } else {
        const int n0 = w.n * BN;
#pragma unroll 1
        for (int c = 0; c < BN / 64 && n0 + c * 64 < N; ++c) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(t_row + c * 64 + h * 32, v);
          uint8_t* grow = take();
          const int gb = r.b;
          r.next();
          uint8_t* urow = take();
          const int ub = r.b;
          r.next();
          tmem_ld_wait();
          if (!ok) break;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int at = ((h * 4 + j) ^ (row & 7)) << 4;
            uint4* gp = reinterpret_cast<uint4*>(grow + at);
            uint4* up = reinterpret_cast<uint4*>(urow + at);
            const uint4 gq = *gp, uq = *up;
            const uint32_t gw[4] = {gq.x, gq.y, gq.z, gq.w}, uw[4] = {uq.x, uq.y, uq.z, uq.w};
            uint32_t dg[4], du[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t* d = &v[8 * j + 2 * i];
              float u0, u1;
              const float g0 = swiglu_grad(bf16_lo(gw[i]), bf16_lo(uw[i]), __uint_as_float(d[0]), u0);
              const float g1 = swiglu_grad(bf16_hi(gw[i]), bf16_hi(uw[i]), __uint_as_float(d[1]), u1);
              dg[i] = pack_bf16x2(g0, g1);
              du[i] = pack_bf16x2(u0, u1);
            }
            *gp = make_uint4(dg[0], dg[1], dg[2], dg[3]);
            *up = make_uint4(du[0], du[1], du[2], du[3]);
          }
          fence_proxy_async_smem();
          mbar_arrive(&out_full[gb]);
          mbar_arrive(&out_full[ub]);
        }
      }
      // accumulator drained by this warp: hand it back to the issuing CTA's MMA warp
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_map(&tmem_empty[acc], 0));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    constexpr int kNumStaging = C::kNumStaging, kEpilogueThreads = C::kEpilogueThreads;
    const int et = threadIdx.x - 64;             // 0..127
    const int quarter = warp & 3;                 // TMEM lane quarter this warp may access
    const int row = quarter * 32 + lane;          // row of this CTA's half tile owned by this thread
    constexpr int kColsPerChunk = (OUT == GEMM_OUT_BF16) ? 64 : 32;  // 128 bytes of output per row
    constexpr int kChunks = BN / kColsPerChunk;
    int acc = 0;
    uint32_t acc_phase = 0;
    int buf = 0;
    while (sched.get(w)) {
      const int m0 = w.row + (int)rank * BM;
      const int n0 = w.n * BN;
      const bool ok = mbar_wait(&tmem_full[acc], acc_phase, abort_word, status, 400 + acc);
      // uniform decision for the four epilogue warps (they share named barriers below)
      int all_ok;
      asm volatile(
          "{\n\t"
          ".reg .pred p, q;\n\t"
          "setp.ne.b32 p, %1, 0;\n\t"
          "barrier.cta.red.and.pred q, 2, 128, p;\n\t"
          "selp.u32 %0, 1, 0, q;\n\t"
          "}\n"
          : "=r"(all_ok)
          : "r"((int)ok)
          : "memory");
      if (!all_ok) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + acc * BN + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < kChunks; ++c) {
        // skip what lies entirely outside D (uniform across threads)
        if (n0 + c * kColsPerChunk >= N || m0 >= M || (kGroups == kRowGroups && rank != 0 && w.alone)) break;
        uint8_t* sbuf = staging + buf * kStagingBytes;
        if (et == 0) tma_store_wait_read<kNumStaging - 1>();
        named_barrier_sync(1, kEpilogueThreads);
        uint8_t* srow = sbuf + row * 128;
        if (OUT == GEMM_OUT_BF16) {
          uint32_t v[2][32];
          tmem_ld_32x32b_x32(t_row + c * 64, v[0]);
          tmem_ld_32x32b_x32(t_row + c * 64 + 32, v[1]);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t* x = &v[j >> 2][8 * (j & 3)];
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(x[0]), __uint_as_float(x[1]));
            o.y = pack_bf16x2(__uint_as_float(x[2]), __uint_as_float(x[3]));
            o.z = pack_bf16x2(__uint_as_float(x[4]), __uint_as_float(x[5]));
            o.w = pack_bf16x2(__uint_as_float(x[6]), __uint_as_float(x[7]));
            *reinterpret_cast<uint4*>(srow + ((j ^ (row & 7)) << 4)) = o;
          }
        } else {
          uint32_t v[32];
          tmem_ld_32x32b_x32(t_row + c * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(srow + ((j ^ (row & 7)) << 4)) =
                make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        fence_proxy_async_smem();
        named_barrier_sync(1, kEpilogueThreads);
        if (et == 0) {
          const int y = m0 + (kGroups == kSumGroups ? w.grp * M : 0);
          if (OUT == GEMM_OUT_F32_ACC && kGroups == kNoGroups && w.kb0 != 0)   // not the first piece: this pair's slab
            tma_store_2d(&out.slabs, sbuf, c * kColsPerChunk, (2 * pair_id + (int)rank) * BM);
          else if (OUT == GEMM_OUT_F32_ACC)
            tma_reduce_add_2d(&out.d, sbuf, n0 + c * kColsPerChunk, y);
          else
            tma_store_2d(&out.d, sbuf, n0 + c * kColsPerChunk, y);
          tma_store_commit();
        }
        buf ^= 1;
      }
      // accumulator drained: hand it back to the issuing CTA's MMA warp
      tc_fence_before();
      named_barrier_sync(1, kEpilogueThreads);
      if (et == 0) mbar_arrive_cluster(cluster_map(&tmem_empty[acc], 0));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (et == 0) tma_store_wait<0>();
  }

  // ---------------------------------------------------------------------- teardown
  if (*abort_word) {
    // give copies that were already issued time to land before shared memory goes away
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();     // the other CTA's MMAs read this one's shared memory, its arrivals land here
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem_base, C::kTmemCols);
}

// Pieces of the cut tiles that do not begin their tile, added to D in the order of K. blockIdx.y is the cut tile, a
// block takes 4 * kRows rows of it, a thread four columns of kRows rows; the loads of kBatch pieces are in flight at a
// time.
template <int kRows, int kBatch>
__global__ void __launch_bounds__(256)
add_pieces_kernel(const float* __restrict__ slabs, float* __restrict__ D, int64_t ldd, int M, int N, int K, int whole,
                  int pairs) {
  const int cut = blockIdx.y, rest = gridDim.y;
  const Tiles tiles(M, N, K, 256);
  Work w;
  tiles.place(whole + cut, w);
  // the pairs whose share begins inside this tile, floor(rest * num_kb * p / pairs) in (cut * num_kb,
  // (cut + 1) * num_kb): num_kb * (rest * p - cut * pairs) >= pairs, and rest * p < (cut + 1) * pairs
  const int first = (cut * pairs + (pairs + tiles.num_kb - 1) / tiles.num_kb + rest - 1) / rest;
  const int last = ((cut + 1) * pairs + rest - 1) / rest;      // exclusive
  const int row = blockIdx.x * 4 * kRows + (threadIdx.x >> 6), col = (threadIdx.x & 63) * 4;
  const int m = w.m * 256 + row, n = w.n * 256 + col;
  float* dst = D + m * ldd + n;
  const float* src = slabs + (int64_t)first * kGemmSlab + row * 256 + col;
  ahead_wait();
  ahead_next();
  if (n >= N) return;
  if (n + 4 <= N) {
    float4 acc[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
      if (m + 4 * r < M) acc[r] = *reinterpret_cast<const float4*>(dst + 4 * r * ldd);
    for (int p = first; p < last; p += kBatch, src += (int64_t)kBatch * kGemmSlab) {
      float4 v[kBatch][kRows];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
#pragma unroll
        for (int r = 0; r < kRows; ++r)
          if (p + b < last && m + 4 * r < M)
            v[b][r] = *reinterpret_cast<const float4*>(src + (int64_t)b * kGemmSlab + 4 * r * 256);
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        if (p + b < last) {
#pragma unroll
          for (int r = 0; r < kRows; ++r) {
            acc[r].x += v[b][r].x;
            acc[r].y += v[b][r].y;
            acc[r].z += v[b][r].z;
            acc[r].w += v[b][r].w;
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r)
      if (m + 4 * r < M) *reinterpret_cast<float4*>(dst + 4 * r * ldd) = acc[r];
  } else {
    for (int r = 0; r < kRows && m + 4 * r < M; ++r) {
      for (int i = 0; n + i < N; ++i) {
        float acc = dst[4 * r * ldd + i];
        for (int p = 0; p < last - first; ++p) acc += src[(int64_t)p * kGemmSlab + 4 * r * 256 + i];
        dst[4 * r * ldd + i] = acc;
      }
    }
  }
}

static int pairs_launched(const GemmPlan& plan) {
  return plan.whole == plan.tiles && plan.tiles < plan.pairs ? plan.tiles : plan.pairs;
}

// Maps of the operands, the kernel's attributes and its launch.
// groups, group_array: row groups and the group of every row tile (B has a matrix for each), or the beginnings of
// reduction groups.
template <int BN, int A_MN, int B_MN, int OUT, int kGroups = kNoGroups>
static int start(const GemmPlan& plan, const void* A, const void* B, const OutMaps& out, int M, int N, int K, int lda,
                 int ldb, int keep_gate, cudaStream_t stream, int groups = 1, const int* group_array = nullptr) {
  using C = Cfg<BN, OUT, kGroups>;
  using pico_host::Swizzle;
  const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap ta, tb;
  if (kGroups != kRowGroups) groups = 1;           // in the maps of the operands
  int rc = A_MN == 0 ? pico_host::make_tmap_2d(&ta, A, bf, 2, K, M, (uint64_t)lda * 2, 64, BM, Swizzle::B128)
                     : pico_host::make_tmap_2d(&ta, A, bf, 2, M, K, (uint64_t)lda * 2, 64, 64, Swizzle::B128);
  if (rc) return rc;
  rc = B_MN == 0 ? pico_host::make_tmap_2d(&tb, B, bf, 2, K, (uint64_t)N * groups, (uint64_t)ldb * 2, 64, BN / 2,
                                           Swizzle::B128)
                 : pico_host::make_tmap_2d(&tb, B, bf, 2, N, (uint64_t)K * groups, (uint64_t)ldb * 2, 64, 64,
                                           Swizzle::B128);
  if (rc) return rc;
  auto kern = gemm_pair_kernel<BN, A_MN, B_MN, OUT, kGroups>;
  static int attr_dev = -1;  // per template instantiation
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) {
      pico_host::set_error("cudaFuncSetAttribute(smem=%d): %s", C::kSmemBytes, cudaGetErrorString(e));
      return (int)e;
    }
    attr_dev = dev;
  }
  pico_host::launch_ahead(kern, 2 * pairs_launched(plan), C::kThreads, C::kSmemBytes, stream, ta, tb, out, M, N, K,
                          plan.whole, keep_gate, group_array, pico_status_buffer());
  return 0;
}

static int launched() {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    pico_host::set_error("gemm launch: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

template <int BN, int A_MN, int B_MN, int OUT>
static int launch(const GemmPlan& plan, const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb,
                  int ldd, float* slabs, cudaStream_t stream) {
  using pico_host::Swizzle;
  OutMaps out = {};
  int rc = OUT == GEMM_OUT_BF16
               ? pico_host::make_tmap_2d(&out.d, D, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, N, M, (uint64_t)ldd * 2, 64,
                                         BM, Swizzle::B128)
               : pico_host::make_tmap_2d(&out.d, D, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, N, M, (uint64_t)ldd * 4, 32,
                                         BM, Swizzle::B128);
  if (rc) return rc;
  const bool cut = plan.whole < plan.tiles;
  if (cut) {
    if (OUT != GEMM_OUT_F32_ACC || slabs == nullptr) {
      pico_host::set_error("pair gemm: tiles cut along K need an accumulated result and scratch");
      return -2;
    }
    rc = pico_host::make_tmap_2d(&out.slabs, slabs, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, 256,
                                 (uint64_t)plan.pairs * 256, 256 * 4, 32, BM, Swizzle::B128);
    if (rc) return rc;
  }
  rc = start<BN, A_MN, B_MN, OUT>(plan, A, B, out, M, N, K, lda, ldb, 0, stream);
  if (rc) return rc;
  if (cut) {
    // few tiles have many pieces each (up to 18): short threads with many loads in flight, latency binds; else two or
    // three, and fewer and longer threads
    const int rest = plan.tiles - plan.whole;
    const bool few = rest < 16;
    pico_host::launch_ahead(few ? add_pieces_kernel<1, 8> : add_pieces_kernel<4, 1>, dim3(few ? 64 : 16, rest), 256, 0,
                            stream, slabs, (float*)D, (int64_t)ldd, M, N, K, plan.whole, plan.pairs);
  }
  return launched();
}

template <int BN>
static int dispatch(const GemmPlan& plan, const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb,
                    int ldd, int a_mn, int b_mn, int out_mode, float* slabs, cudaStream_t st) {
#define PICO_CASE(AM, BMJ, OM)                                 \
  if (a_mn == AM && b_mn == BMJ && out_mode == OM)             \
    return launch<BN, AM, BMJ, OM>(plan, A, B, D, M, N, K, lda, ldb, ldd, slabs, st);
  PICO_CASE(0, 0, GEMM_OUT_BF16)
  PICO_CASE(0, 1, GEMM_OUT_BF16)
  PICO_CASE(1, 1, GEMM_OUT_BF16)
  PICO_CASE(1, 1, GEMM_OUT_F32_ACC)
#undef PICO_CASE
  return kGemmPairUnsupported;
}

}  // namespace pair

bool gemm_pair_has(int a_mn, int b_mn, int out_mode) {
  return (out_mode == GEMM_OUT_BF16 && !(a_mn == 1 && b_mn == 0)) ||
         (out_mode == GEMM_OUT_F32_ACC && a_mn == 1 && b_mn == 1);
}

int gemm_pair(const GemmPlan& plan, const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb,
              int ldd, int a_mn, int b_mn, int out_mode, float* slabs, cudaStream_t stream) {
  return pair::dispatch<256>(plan, A, B, D, M, N, K, lda, ldb, ldd, a_mn, b_mn, out_mode, slabs, stream);
}

// `tiles` has room for one short tile per group, so from twice the groups on a group has about two. One CTA / pairs,
// us, up, activation, down and their input gradients in all, width 2048 and 1024: 64 groups, 128 tiles (8192 rows) 389 /
// 391 to 160 tiles 478 / 423, 208 tiles 668 / 672, 256 tiles 690 / 660 (rounds of whole tiles differ); 8 groups, 24 tiles
// 103 / 95. Below that there are fewer pair tiles than pairs and their epilogues show: 8 groups, 16 tiles 64 / 68, 20
// tiles 52 / 55. Plain products are held against the one-CTA kernel by gemm_pair_rows_pay too. With the activation
// inside, the narrow ones lose on the GPU as well (8 groups, 24 tiles, 256 x 256: forward 8.1 / 9.8, backward 7.8 / 10.6;
// 128 tiles 13.7 / 14.7, 13.1 / 11.7), but there the host sets the time, and one operator takes it less than three: forward
// and backward of an expert layer of width 256 to 1024, 24 to 272 tiles, 700 / 630 with 8 experts, 830 / 755 with 16.
bool gemm_pair_takes_rows(int M, int groups) {
  const int tiles = (M + pair::BM - 1) / pair::BM;
  return tiles <= pair::kMaxRowTiles && tiles >= 2 * (int64_t)groups && tiles >= 24 &&
         groups < 32768 && pico_host::num_sms() >= 2;
}

// Cycles of both kernels, as in plan_gemm: 512 for a K block of a round of pairs, though a round takes no less than its
// epilogue's ~5000, and ~1000 to list the pairs; on the one-CTA kernel 333 for a K block of 128-wide tiles in one wave,
// 573 for one of a round of 256-wide tiles. So narrow products with few row tiles, and short ones, stay there. One CTA /
// pairs, us, 8 groups: 24 row tiles, N = K = 256 4.9 / 6.8, 512 5.9 / 8.2, 1024 10.4 / 11.1; 64, N = K = 512 7.8 / 8.8;
// 128, N = 2048, K = 1024 56 / 49; 384, N = 1024, K = 256 32.9 / 41.1, K = 1024 84 / 74. Over 1100 products (N 256 ..
// 4096, K 128 .. 4096, 24 .. 384 row tiles, 8 .. 64 groups) the choice is 0.3 % slower than the better one on average;
// pairs for all of them 7.4 %, for none 4.0 %.
bool gemm_pair_rows_pay(int sms, int M, int N, int K, int bn) {
  const auto parts = [](int64_t n, int64_t of) { return (n + of - 1) / of; };
  if (sms < 2) return false;
  const int64_t kb = parts(K, pair::BK), rows = parts(M, pair::BM), round = kb * 512 > 5000 ? kb * 512 : 5000;
  const int64_t one = parts(rows * parts(N, bn), sms) * kb * (bn < 256 ? 333 : 573);
  return parts(parts(rows, 2) * parts(N, 256), sms / 2) * round + 1000 < one;
}

int gemm_pair_rows(const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb, int ldd, int b_mn,
                   const int* tile_group, int groups, cudaStream_t stream) {
  const GemmPlan plan{true, 256, pico_host::num_sms() / 2, INT32_MAX, INT32_MAX};     // counted in the kernel
  pair::OutMaps out = {};
  int rc = pico_host::make_tmap_2d(&out.d, D, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, N, M, (uint64_t)ldd * 2, 64,
                                   pair::BM, pico_host::Swizzle::B128);
  if (rc) return rc;
  auto start = b_mn ? pair::start<256, 0, 1, GEMM_OUT_BF16, pair::kRowGroups>
                    : pair::start<256, 0, 0, GEMM_OUT_BF16, pair::kRowGroups>;
  rc = start(plan, A, B, out, M, N, K, lda, ldb, 0, stream, groups, tile_group);
  return rc ? rc : pair::launched();
}

// Four rounds and more; with fewer the last one costs more than wider tiles save (8 groups of 320 rows, 2048 x 1024,
// 256 tiles: 21.8 us on one CTA, 23.6 on pairs; 16 groups of 584, 512 tiles: 63.9, 63.2).
bool gemm_pair_takes_sums(int M, int N, int groups) {
  return (int64_t)((M + 255) / 256) * ((N + 255) / 256) * groups >= 4 * (pico_host::num_sms() / 2) &&
         pico_host::num_sms() >= 2;
}

int gemm_pair_sums(const void* A, const void* B, float* D, int M, int N, int K, int lda, int ldb, int ldd,
                   const int* seg_start, int groups, cudaStream_t stream) {
  const int64_t tiles = (int64_t)((M + 255) / 256) * ((N + 255) / 256) * groups;
  if (tiles > INT32_MAX) {
    pico_host::set_error("grouped gemm: too many tiles");
    return -2;
  }
  const GemmPlan plan{true, 256, pico_host::num_sms() / 2, (int)tiles, (int)tiles};
  pair::OutMaps out = {};
  const int rc = pico_host::make_tmap_2d(&out.d, D, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, N, (uint64_t)M * groups,
                                         (uint64_t)ldd * 4, 32, pair::BM, pico_host::Swizzle::B128);
  if (rc) return rc;
  const int rc2 = pair::start<256, 1, 1, GEMM_OUT_F32_ACC, pair::kSumGroups>(plan, A, B, out, M, N, K, lda, ldb, 0,
                                                                             stream, groups, seg_start);
  return rc2 ? rc2 : pair::launched();
}

// All tiles of an [M, N] product whole. With row groups odd segments take a pair tile more each, so their number is found
// in the kernel and the grid has all pairs (32 row tiles in 8 odd segments on a grid for 16 pair tiles of each column:
// two rounds, 13.9 us instead of 9.8 forward, 15.8 instead of 10.6 backward, 256 x 256).
static int whole_plan(int M, int N, bool row_groups, GemmPlan& plan) {
  const int64_t tiles = (int64_t)((M + 255) / 256) * ((N + 255) / 256);
  const int sms = pico_host::num_sms();
  if (tiles > INT32_MAX || sms < 2) {
    pico_host::set_error("swiglu gemm: too many tiles, or fewer than two SMs");
    return -2;
  }
  const int count = row_groups ? INT32_MAX : (int)tiles;
  plan = GemmPlan{true, 256, sms / 2, count, count};
  return 0;
}

// The two halves of a [rows, 2 * I] buffer as matrices of their own, so that a tile past I is clipped in each.
static int half_maps(CUtensorMap* gate, CUtensorMap* up, const void* gu, int rows, int I) {
  const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const uint64_t pitch = (uint64_t)I * 4;
  const int rc = pico_host::make_tmap_2d(gate, gu, bf, 2, I, rows, pitch, 64, pair::BM, pico_host::Swizzle::B128);
  return rc ? rc : pico_host::make_tmap_2d(up, (const char*)gu + (int64_t)I * 2, bf, 2, I, rows, pitch, 64, pair::BM,
                                           pico_host::Swizzle::B128);
}

}  // namespace pico

// The fused form ends on an epilogue that nothing overlaps, 3 to 5 us longer than that of the plain product; the pass
// it saves takes its launch and its bytes. So it pays from some number of activations on, where the plain product runs
// on pairs too (elsewhere its narrower tiles waste less). Measured, product and pass / fused, us:
//   forward           512 x 960 x 2560 12.3 / 13.1, 256 x 2048 x 8192 18.9 / 19.2, 4096 x 576 x 1536 21.4 / 21.1
//   .. without gate|up 512 x 576 x 1536 8.3 / 8.6, 512 x 960 x 2560 12.3 / 10.9, 256 x 2048 x 8192 18.9 / 16.9
//   backward          1024 x 960 x 2560 13.8 / 14.3, 4096 x 576 x 1536 20.0 / 18.7
// and off pairs, 300 x 4096 x 11008: 77 / 89 forward, 47 / 58 backward.
extern "C" int pico_gemm_swiglu_pays(int M, int I, int K, int keep_gate, int backward) {
  if (M <= 0 || I <= 0 || K <= 0 || I > INT32_MAX / 2) return 0;
  const pico::GemmPlan plan = pico::plan_gemm(pico_host::num_sms(), M, backward ? I : 2 * I, K, 0, backward,
                                              pico::GEMM_OUT_BF16, 0, false);
  return plan.pair && (int64_t)M * I >= (backward ? 4000000 : keep_gate ? 2500000 : 1250000);
}

extern "C" int pico_gemm_swiglu_pairs(int M, int I, int row_groups, int backward) {
  pico::GemmPlan plan;
  return M <= 0 || I <= 0 || pico::whole_plan(M, backward ? I : 2 * I, row_groups != 0, plan)
             ? 0 : pico::pair::pairs_launched(plan);
}

static bool row_groups_ok(int M, int K, int groups, bool whole_k) {
  if (pico::gemm_pair_takes_rows(M, groups) && (!whole_k || K % pico::pair::BK == 0)) return true;
  pico_host::set_error("swiglu gemm: row groups of two tiles and more on average, 24 to %d tiles, K (%d) a multiple of "
                       "%d backward", pico::pair::kMaxRowTiles, K, pico::pair::BK);
  return false;
}

extern "C" int pico_gemm_rows_on_pairs(int M, int groups) { return pico::gemm_pair_takes_rows(M, groups); }

extern "C" int pico_gemm_swiglu(const void* x, const void* w, void* gate_up, void* act, int M, int I, int K, int ldx,
                                int ldw, const int* tile_group, int groups, cudaStream_t stream) {
  if (M <= 0 || I <= 0 || K <= 0) return 0;
  if (tile_group != nullptr && !row_groups_ok(M, K, groups, false)) return -2;
  if (I > INT32_MAX / 2) {
    pico_host::set_error("swiglu gemm: width %d", I);
    return -2;
  }
  pico::GemmPlan plan;
  int rc = pico::whole_plan(M, 2 * I, tile_group != nullptr, plan);
  if (rc) return rc;
  pico::pair::OutMaps out = {};
  rc = pico_host::make_tmap_2d(&out.d, act, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, I, M, (uint64_t)I * 2, 64,
                               pico::pair::BM, pico_host::Swizzle::B128);
  if (!rc && gate_up != nullptr) rc = pico::half_maps(&out.gate, &out.up, gate_up, M, I);
  auto start = tile_group != nullptr ? pico::pair::start<256, 0, 0, pico::GEMM_OUT_SWIGLU, pico::pair::kRowGroups>
                                     : pico::pair::start<256, 0, 0, pico::GEMM_OUT_SWIGLU>;
  if (!rc) rc = start(plan, x, w, out, M, 2 * I, K, ldx, ldw, gate_up != nullptr, stream, groups, tile_group);
  return rc ? rc : pico::pair::launched();
}

extern "C" int pico_gemm_swiglu_bwd(const void* dy, const void* w, const void* gate_up, void* d_gate_up, int M, int I,
                                    int K, int lddy, int ldw, const int* tile_group, int groups,
                                    cudaStream_t stream) {
  if (M <= 0 || I <= 0 || K <= 0) return 0;
  if (tile_group != nullptr && !row_groups_ok(M, K, groups, true)) return -2;
  pico::GemmPlan plan;
  int rc = pico::whole_plan(M, I, tile_group != nullptr, plan);
  if (rc) return rc;
  pico::pair::OutMaps out = {};
  rc = pico::half_maps(&out.gate, &out.up, gate_up, M, I);
  if (!rc) rc = pico::half_maps(&out.d_gate, &out.d_up, d_gate_up, M, I);
  auto start = tile_group != nullptr ? pico::pair::start<256, 0, 1, pico::GEMM_OUT_SWIGLU_BWD, pico::pair::kRowGroups>
                                     : pico::pair::start<256, 0, 1, pico::GEMM_OUT_SWIGLU_BWD>;
  if (!rc) rc = start(plan, dy, w, out, M, I, K, lddy, ldw, 1, stream, groups, tile_group);
  return rc ? rc : pico::pair::launched();
}
