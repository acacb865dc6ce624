// What the translation units of the GEMM family share.
#pragma once
#include <cuda_runtime.h>

namespace pico {

enum GemmOutMode : int {
  GEMM_OUT_BF16 = 0,
  GEMM_OUT_F32 = 1,
  GEMM_OUT_F32_ACC = 2,
  GEMM_OUT_SWIGLU = 3,        // pico_gemm_swiglu and its backward, pair kernel only
  GEMM_OUT_SWIGLU_BWD = 4,
};

constexpr int kGemmPairUnsupported = -10;

// What a plain product runs on: the CTA-pair kernel (256 x 256 tiles) or the one-CTA kernel with 128 x bn tiles.
// Pair kernel: `whole` of the `tiles` output tiles are dealt to the pairs as they are, the others (the last, partial
// round of an accumulating product) are cut along K into equal shares for all pairs, which takes scratch of
// kGemmSlab floats per pair (has_scratch).
struct GemmPlan {
  bool pair;
  int bn;
  int pairs, tiles, whole;
};
constexpr int kGemmSlab = 256 * 256;
GemmPlan plan_gemm(int sms, int M, int N, int K, int a_mn_major, int b_mn_major, int out_mode, int max_ctas,
                   bool has_scratch);

// CTA-pair kernel; operands as pico_gemm_bf16, `plan` as plan_gemm gives it for them, slabs: its scratch, 16-byte
// aligned (not read where nothing is cut).
bool gemm_pair_has(int a_mn_major, int b_mn_major, int out_mode);
int gemm_pair(const GemmPlan& plan, const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb,
              int ldd, int a_mn_major, int b_mn_major, int out_mode, float* slabs, cudaStream_t stream);

// bf16 D with row groups (PicoGemmComm::tile_group, K-major A, B stacked) on the same kernel, whether their number and
// size suit it, and whether the plain product is then faster than on the one-CTA kernel's tiles of width bn.
bool gemm_pair_takes_rows(int M, int groups);
bool gemm_pair_rows_pay(int sms, int M, int N, int K, int bn);
int gemm_pair_rows(const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb, int ldd,
                   int b_mn_major, const int* tile_group, int groups, cudaStream_t stream);

// D += with reduction groups (PicoGemmComm::seg_start; MN-major operands, M a multiple of 128) on the same kernel.
bool gemm_pair_takes_sums(int M, int N, int groups);
int gemm_pair_sums(const void* A, const void* B, float* D, int M, int N, int K, int lda, int ldb, int ldd,
                   const int* seg_start, int groups, cudaStream_t stream);

}  // namespace pico
