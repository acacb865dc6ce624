// Device code of the RMSNorm kernels, shared by the launchers in norm.cu and by the
// allocation-free entry point in norm_noalloc.cu.
#pragma once
#include <cuda_bf16.h>

#include "../common/ptx.cuh"

namespace pico {

constexpr int kNormThreads = 256;
constexpr int kMaxVec = 8;  // vectors of 8 bf16 per thread kept in registers: H <= 16384

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < kNormThreads / 32) ? red[lane] : 0.f;
  return warp_sum(t);
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return v;
}

template <int NV>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ h_out, float* __restrict__ rstd_out, int rows, int H,
                   float eps) {
  ahead_wait();
  ahead_next();
  __shared__ float red[kNormThreads / 32];
  const int nvec = H / 8;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * H);
    const uint4* rr = residual ? reinterpret_cast<const uint4*>(residual + (size_t)row * H) : nullptr;
    float vals[NV][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * kNormThreads;
      if (v < nvec) {
        unpack8(xr[v], vals[i]);
        if (rr) {
          float r[8];
          unpack8(rr[v], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) vals[i][j] += r[j];
          // the summed stream is rounded to bf16 before it is normalised, as an unfused
          // add followed by a norm would do
          uint4 hv = pack8(vals[i]);
          unpack8(hv, vals[i]);
          if (h_out) reinterpret_cast<uint4*>(h_out + (size_t)row * H)[v] = hv;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += vals[i][j] * vals[i][j];
      }
    }
    ss = block_sum(ss, red);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * kNormThreads;
      if (v < nvec) {
        float wv[8], o[8];
        unpack8(reinterpret_cast<const uint4*>(w)[v], wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = vals[i][j] * rstd * wv[j];
        reinterpret_cast<uint4*>(y + (size_t)row * H)[v] = pack8(o);
      }
    }
  }
}

// Warp-per-row forward for H <= 1024: lane l owns vectors l, l + 32, ...; no block barrier, all loads of a row in
// flight at once. The block-per-row kernel above leaves half of its threads idle at H = 960 and waits for
// two barriers per row (8192 rows: 12.7 us there, 8.7 here).
template <int NVW>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                        const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                        __nv_bfloat16* __restrict__ h_out, float* __restrict__ rstd_out, int rows, int H,
                        float eps) {
  ahead_wait();
  ahead_next();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = H / 8;
  for (int row = blockIdx.x * (kNormThreads / 32) + warp; row < rows; row += gridDim.x * (kNormThreads / 32)) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * H);
    uint4 hv[NVW], rv[NVW];
#pragma unroll
    for (int i = 0; i < NVW; ++i) {
      const int v = lane + i * 32;
      hv[i] = v < nvec ? xr[v] : make_uint4(0, 0, 0, 0);
    }
    if (residual) {
      const uint4* rr = reinterpret_cast<const uint4*>(residual + (size_t)row * H);
#pragma unroll
      for (int i = 0; i < NVW; ++i) {
        const int v = lane + i * 32;
        rv[i] = v < nvec ? rr[v] : make_uint4(0, 0, 0, 0);
      }
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NVW; ++i) {
      float f[8];
      unpack8(hv[i], f);
      if (residual) {
        float r[8];
        unpack8(rv[i], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += r[j];
        // the summed stream is rounded to bf16 before it is normalised, as an unfused add followed by a
        // norm would do
        hv[i] = pack8(f);
        unpack8(hv[i], f);
        const int v = lane + i * 32;
        if (h_out && v < nvec) reinterpret_cast<uint4*>(h_out + (size_t)row * H)[v] = hv[i];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (lane == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int i = 0; i < NVW; ++i) {
      const int v = lane + i * 32;
      if (v < nvec) {
        float f[8], wv[8], o[8];
        unpack8(hv[i], f);
        unpack8(reinterpret_cast<const uint4*>(w)[v], wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = f[j] * rstd * wv[j];
        reinterpret_cast<uint4*>(y + (size_t)row * H)[v] = pack8(o);
      }
    }
  }
}

// dw partials: dw_partial[blockIdx.x][H] fp32
template <int NV>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dh,
                   float* __restrict__ dw_partial, int rows, int H) {
  ahead_wait();
  ahead_next();
  __shared__ float red[kNormThreads / 32];
  const int nvec = H / 8;
  float dw_acc[NV][8];
  float wv[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * kNormThreads;
#pragma unroll
    for (int j = 0; j < 8; ++j) dw_acc[i][j] = 0.f;
    if (v < nvec) unpack8(reinterpret_cast<const uint4*>(w)[v], wv[i]);
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float rstd = rstd_in[row];
    float g[NV][8], hv[NV][8];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * kNormThreads;
      if (v < nvec) {
        float d[8];
        unpack8(reinterpret_cast<const uint4*>(dy + (size_t)row * H)[v], d);
        unpack8(reinterpret_cast<const uint4*>(h + (size_t)row * H)[v], hv[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          g[i][j] = d[j] * wv[i][j];
          dot += g[i][j] * hv[i][j];
          dw_acc[i][j] += d[j] * hv[i][j] * rstd;
        }
      }
    }
    dot = block_sum(dot, red);
    const float c = dot / (float)H * rstd * rstd * rstd;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * kNormThreads;
      if (v < nvec) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rstd * g[i][j] - hv[i][j] * c;
        if (dres) {
          float r[8];
          unpack8(reinterpret_cast<const uint4*>(dres + (size_t)row * H)[v], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        reinterpret_cast<uint4*>(dh + (size_t)row * H)[v] = pack8(o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * kNormThreads;
    if (v < nvec) {
      float4* out = reinterpret_cast<float4*>(dw_partial + (size_t)blockIdx.x * H + (size_t)v * 8);
      out[0] = make_float4(dw_acc[i][0], dw_acc[i][1], dw_acc[i][2], dw_acc[i][3]);
      out[1] = make_float4(dw_acc[i][4], dw_acc[i][5], dw_acc[i][6], dw_acc[i][7]);
    }
  }
}

// Row-group variant for H = 2048 * NV: one CTA works on R rows at a time, every thread owning NV
// vectors of 8 columns of each row. The R row dot products share one pair of barriers, the
// weight-gradient partials are 8 * NV registers per thread, so many CTAs fit an SM and enough
// loads are in flight to keep the memory system busy (a warp per row would hold 8 * H / 256 partials per
// lane: 64 at H = 2048, which measured a quarter of the copy bandwidth).
template <int NV, int R>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_bwd_rows_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h,
                        const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                        const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dh,
                        float* __restrict__ dw_partial, int rows, int H) {
  ahead_wait();
  ahead_next();
  constexpr int kWarps = kNormThreads / 32;
  __shared__ float red[R][kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = H / 8;                       // == NV * kNormThreads
  float dw_acc[NV][8];
  float wv[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) dw_acc[i][j] = 0.f;
    unpack8(reinterpret_cast<const uint4*>(w)[threadIdx.x + i * kNormThreads], wv[i]);
  }
  const float inv_h = 1.f / (float)H;
  for (int row0 = blockIdx.x * R; row0 < rows; row0 += gridDim.x * R) {
    uint4 draw[R][NV], hraw[R][NV];
    float rstd[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = row0 + r;
      rstd[r] = row < rows ? rstd_in[row] : 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        // zeros past the end: a copy of the last row times rstd = 0 would be NaN where that row has an infinity
        const size_t off = (size_t)row * nvec + threadIdx.x + i * kNormThreads;
        draw[r][i] = row < rows ? reinterpret_cast<const uint4*>(dy)[off] : make_uint4(0, 0, 0, 0);
        hraw[r][i] = row < rows ? reinterpret_cast<const uint4*>(h)[off] : make_uint4(0, 0, 0, 0);
      }
    }
    float dot[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      dot[r] = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        float d[8], hv[8];
        unpack8(draw[r][i], d);
        unpack8(hraw[r][i], hv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dot[r] += d[j] * wv[i][j] * hv[j];
          dw_acc[i][j] += d[j] * hv[j] * rstd[r];
        }
      }
      dot[r] = warp_sum(dot[r]);
    }
    __syncthreads();                            // the previous iteration's readers are done with red
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) red[r][warp] = dot[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = row0 + r;
      if (row >= rows) break;
      float tot = 0.f;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) tot += red[r][k];
      const float c = tot * inv_h * rstd[r] * rstd[r] * rstd[r];
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        float d[8], hv[8], o[8];
        unpack8(draw[r][i], d);
        unpack8(hraw[r][i], hv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rstd[r] * d[j] * wv[i][j] - hv[j] * c;
        const size_t off = (size_t)row * nvec + threadIdx.x + i * kNormThreads;
        if (dres) {
          float rr[8];
          unpack8(reinterpret_cast<const uint4*>(dres)[off], rr);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += rr[j];
        }
        reinterpret_cast<uint4*>(dh)[off] = pack8(o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float4* out = reinterpret_cast<float4*>(dw_partial + (size_t)blockIdx.x * H +
                                            (size_t)(threadIdx.x + i * kNormThreads) * 8);
    out[0] = make_float4(dw_acc[i][0], dw_acc[i][1], dw_acc[i][2], dw_acc[i][3]);
    out[1] = make_float4(dw_acc[i][4], dw_acc[i][5], dw_acc[i][6], dw_acc[i][7]);
  }
}

// The same row-group scheme with the next group's rows already in flight while the current group
// is reduced and written: the loads of group g+1 are issued before the barriers of group g, so the
// memory system never idles between the load and the store phase of a CTA. kThreads = 256 holds H = 2048
// exactly; narrower rows take the next multiple of a warp above H / 8 threads, so that the last few idle and
// not half of 256.
template <int kThreads, int R>
__global__ void __launch_bounds__(kThreads)
rmsnorm_bwd_rows_pf_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h,
                           const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                           const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dh,
                           float* __restrict__ dw_partial, int rows, int H) {
  ahead_wait();
  ahead_next();
  constexpr int kWarps = kThreads / 32;
  __shared__ float red[R][kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = H / 8;                       // <= kThreads
  const bool act = (int)threadIdx.x < nvec;
  const int col = act ? (int)threadIdx.x : 0;     // idle threads read column 0 and add nothing
  float dw_acc[8], wv[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) dw_acc[j] = 0.f;
  unpack8(reinterpret_cast<const uint4*>(w)[col], wv);
  const float inv_h = 1.f / (float)H;
  uint4 dnext[R], hnext[R];
  float rnext[R];
  auto load = [&](int row0) {                   // zeros past the end, as above
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = row0 + r;
      const size_t off = (size_t)row * nvec + col;
      rnext[r] = row < rows ? rstd_in[row] : 0.f;
      dnext[r] = row < rows ? reinterpret_cast<const uint4*>(dy)[off] : make_uint4(0, 0, 0, 0);
      hnext[r] = row < rows ? reinterpret_cast<const uint4*>(h)[off] : make_uint4(0, 0, 0, 0);
    }
  };
  const int stride = gridDim.x * R;
  int row0 = blockIdx.x * R;
  if (row0 < rows) load(row0);
  for (; row0 < rows; row0 += stride) {
    uint4 draw[R], hraw[R];
    float rstd[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      rstd[r] = rnext[r];
      draw[r] = dnext[r];
      hraw[r] = hnext[r];
    }
    if (row0 + stride < rows) load(row0 + stride);
    float dot[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      dot[r] = 0.f;
      float d[8], hv[8];
      unpack8(draw[r], d);
      unpack8(hraw[r], hv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (act) dot[r] += d[j] * wv[j] * hv[j];
        dw_acc[j] += d[j] * hv[j] * rstd[r];
      }
      dot[r] = warp_sum(dot[r]);
    }
    __syncthreads();                            // the previous iteration's readers are done with red
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) red[r][warp] = dot[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = row0 + r;
      if (row >= rows) break;
      float tot = 0.f;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) tot += red[r][k];
      const float c = tot * inv_h * rstd[r] * rstd[r] * rstd[r];
      float d[8], hv[8], o[8];
      unpack8(draw[r], d);
      unpack8(hraw[r], hv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rstd[r] * d[j] * wv[j] - hv[j] * c;
      const size_t off = (size_t)row * nvec + col;
      if (dres) {
        float rr[8];
        unpack8(reinterpret_cast<const uint4*>(dres)[off], rr);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += rr[j];
      }
      if (act) reinterpret_cast<uint4*>(dh)[off] = pack8(o);
    }
  }
  if (!act) return;
  float4* out = reinterpret_cast<float4*>(dw_partial + (size_t)blockIdx.x * H + (size_t)col * 8);
  out[0] = make_float4(dw_acc[0], dw_acc[1], dw_acc[2], dw_acc[3]);
  out[1] = make_float4(dw_acc[4], dw_acc[5], dw_acc[6], dw_acc[7]);
}

// dw[H] (=|+=) sum_p partial[p][H]; fixed summation order (deterministic)
static __global__ void colsum_kernel(const float* __restrict__ partial, int nparts, int H,
                                     float* __restrict__ out_f32, __nv_bfloat16* __restrict__ out_bf16,
                                     int accumulate) {
  ahead_wait();
  ahead_next();
  // block = 32 columns x (blockDim.x / 32) row groups; each thread sums every groups-th partial row of its column,
  // the sub-sums are then added in a fixed order. What binds it is the latency of the strided loads, so they
  // are spread over 1024 threads and unrolled (592 x 960 partials: 6.6 us with 256 threads)
  __shared__ float red[32][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5, groups = blockDim.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (c < H) {
#pragma unroll 8
    for (int p = ry; p < nparts; p += groups) s += partial[(size_t)p * H + c];
  }
  red[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && c < H) {
    float t = 0.f;
    for (int k = 0; k < groups; ++k) t += red[k][cx];
    if (out_f32) out_f32[c] = accumulate ? out_f32[c] + t : t;
    if (out_bf16) out_bf16[c] = __float2bfloat16(accumulate ? __bfloat162float(out_bf16[c]) + t : t);
  }
}

}  // namespace pico
