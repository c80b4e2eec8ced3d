// gemv_row.cu — the products of a decode step of one sequence (one bf16 row), with what stands between them folded in.
//
// One token of a small model is a chain of dependent launches of a few microseconds each, most of it the way from one
// launch to the next.  Here a product takes its input's norm along (every CTA norms the row itself: one read of x, two block
// sums) and finishes its result itself (activation, or the residual update of x in place), so a layer is five launches
// instead of seven.  A warp group (WPR warps) owns the whole sum of R output rows; its lanes take 16 bytes of a
// weight row at a time, all of a row's loads in flight, the first tile's before the wait for the kernel in front
// (weights don't change).  Sums: 8 NL FMAs a lane, then the lanes and warps in pairs.
// Bound by the chain: release of the launch, one L2 round trip for the row, the sums.
//
// Which layers take it (forward.cu), us a token, with their norms and products as launches of their own / here (vocabulary of
// 4096; width, feed-forward, layers):
//   768, 3072, 12 (GPT-2 small)  289 / 213     2048, 8192, 4   201 / 187     4096, 8192, 2    189 / 179 (all heads with keys of
//   1600, 6400, 8                341 / 287     3072, 8192, 4   286 / 264                       their own: 205 / 194)
// Rows wider than 4096 are better off without the norm in front, which every CTA repeats: 5120, 6144, 2 199 / 217; 8192,
// 4096, 2 269 / 277; 8192, 8192, 2 344 / 352; 5120, 384, 4 with 8 heads 122 / 144.  And the attention's output product pays only
// where the feed-forward follows here too: behind it alone a norm is launched all the same, and the residual update that this
// norm would have done costs the product its split sums (2048, 8192, 4: 201 / 209; 4096, 14336, 2: 251 / 253).  What is left
// then, the first layer's projections, is worth it in narrow models (routed experts, 1024, 3 layers 158 / 156; 4096, 14336, 1
// layer 138 / 140).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace nvllm {

constexpr int GR_THREADS = 256, GR_WARPS = GR_THREADS / 32;

__device__ __forceinline__ void widen8(const uint4& v, float (&o)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 f = __bfloat1622float2(h[i]);
    o[2 * i] = f.x;
    o[2 * i + 1] = f.y;
  }
}

// R: output rows of a warp group (2: a gate / up pair); WPR: its warps; NL: 16-byte pieces of a row per lane; NORM: the row is
// x, normed here
template <int R, int WPR, int NL, bool NORM>
__global__ void __launch_bounds__(GR_THREADS) gemv_row_kernel(GemvRowArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  extern __shared__ __align__(16) bf16 xn[];  // NORM: the normed row
  __shared__ float red[32];
  __shared__ float part[2][GR_WARPS][R];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int per = GR_WARPS / WPR * R;  // output rows of a tile
  const int wr = warp / WPR, wk = warp % WPR;
  const int tiles = (a.N + per - 1) / per;
  constexpr int kstep = WPR * 256;
  const int k0 = wk * 256 + lane * 8;
  uint4 w[R][NL];
  auto fetch = [&](int tile) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int n = tile * per + wr * R + r;
#pragma unroll
      for (int i = 0; i < NL; i++) {
        const int k = k0 + i * kstep;
        w[r][i] = k < a.K && n < a.N ? ld_once16(a.W + (size_t)n * a.K + k) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };
  int tile = blockIdx.x;
  fetch(tile);
  uint4 act[NL];
  float x_old = 0.f;
  const bool resid = a.epi == TC5_EPI_RESID;
  const bool writer = wk == 0 && lane == 0;
  if (NORM) {
    float4 v[WPR], g[WPR];  // K <= 1024 WPR
    const int pieces = a.K / 4;
#pragma unroll
    for (int j = 0; j < WPR; j++) {
      const int i = threadIdx.x + j * GR_THREADS;
      if (i < pieces) g[j] = __ldg(reinterpret_cast<const float4*>(a.norm_w) + i);
    }
    pdl_wait();
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < WPR; j++) {
      const int i = threadIdx.x + j * GR_THREADS;
      v[j] = i < pieces ? __ldcg(reinterpret_cast<const float4*>(a.x) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const bool ln = a.norm_b != nullptr;
#pragma unroll
    for (int j = 0; j < WPR; j++)
      sum += ln ? (v[j].x + v[j].y) + (v[j].z + v[j].w) : (v[j].x * v[j].x + v[j].y * v[j].y) + (v[j].z * v[j].z + v[j].w * v[j].w);
    float tot = block_sum(sum, red), mean = 0.f;
    if (ln) {
      mean = tot / (float)a.K;
      sum = 0.f;
#pragma unroll
      for (int j = 0; j < WPR; j++) {
        if (threadIdx.x + j * GR_THREADS >= pieces) continue;
        const float d0 = v[j].x - mean, d1 = v[j].y - mean, d2 = v[j].z - mean, d3 = v[j].w - mean;
        sum += (d0 * d0 + d1 * d1) + (d2 * d2 + d3 * d3);
      }
      tot = block_sum(sum, red);
    }
    const float inv = 1.0f / sqrtf(tot / (float)a.K + a.eps);
#pragma unroll
    for (int j = 0; j < WPR; j++) {
      const int i = threadIdx.x + j * GR_THREADS;
      if (i >= pieces) continue;
      float4 o = make_float4((v[j].x - mean) * inv * g[j].x, (v[j].y - mean) * inv * g[j].y, (v[j].z - mean) * inv * g[j].z,
                             (v[j].w - mean) * inv * g[j].w);
      if (ln) {
        const float4 b = __ldg(reinterpret_cast<const float4*>(a.norm_b) + i);
        o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w;
      }
      __nv_bfloat162 p[2] = {__floats2bfloat162_rn(o.x, o.y), __floats2bfloat162_rn(o.z, o.w)};
      *reinterpret_cast<uint2*>(xn + 4 * i) = *reinterpret_cast<const uint2*>(p);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NL; i++) {
      const int k = k0 + i * kstep;
      act[i] = k < a.K ? *reinterpret_cast<const uint4*>(xn + k) : make_uint4(0u, 0u, 0u, 0u);
    }
  } else {
    pdl_wait();
#pragma unroll
    for (int i = 0; i < NL; i++) {
      const int k = k0 + i * kstep;
      act[i] = k < a.K ? __ldcg(reinterpret_cast<const uint4*>(a.A + k)) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  for (int it = 0; tile < tiles; tile += gridDim.x, it++) {
    const int n = tile * per + wr * R;
    if (resid && writer && n < a.N) x_old = __ldcg(a.x + n);
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      acc[r] = 0.f;
#pragma unroll
      for (int i = 0; i < NL; i++) {
        float wf[8], af[8];
        widen8(w[r][i], wf);
        widen8(act[i], af);
#pragma unroll
        for (int e = 0; e < 8; e++) acc[r] = fmaf(wf[e], af[e], acc[r]);
      }
    }
    if (tile + (int)gridDim.x < tiles) fetch(tile + gridDim.x);
#pragma unroll
    for (int r = 0; r < R; r++) acc[r] = warp_sum(acc[r]);
    if (WPR > 1) {
      if (lane == 0)
#pragma unroll
        for (int r = 0; r < R; r++) part[it & 1][warp][r] = acc[r];
      __syncthreads();
      if (writer)
#pragma unroll
        for (int r = 0; r < R; r++) {
          float s = part[it & 1][warp][r];
#pragma unroll
          for (int j = 1; j < WPR; j++) s += part[it & 1][warp + j][r];
          acc[r] = s;
        }
    }
    if (writer && n < a.N) {
      if (resid) {
        a.x[n] = x_old + a.m * (acc[0] + (a.bias ? a.bias[n] : 0.f));
      } else if (a.epi == TC5_EPI_SWIGLU) {
        a.act[n >> 1] = __float2bfloat16_rn(glu_unit(acc[0], acc[R - 1], 0.f));
      } else if (a.epi == TC5_EPI_GELU) {
        a.act[n] = __float2bfloat16_rn(gelu_tanh(acc[0] + (a.bias ? a.bias[n] : 0.f)));
      } else {
        a.out[n] = acc[0];
      }
    }
  }
  TRACE_EXIT(tr);
}

bool gemv_row_fits(int K, bool norm) { return K >= 8 && K <= (norm ? 4096 : 8192) && (K % 8) == 0; }

template <int R, int WPR, int NL, bool NORM>
static cudaError_t gemv_row_launch(cudaStream_t st, const GemvRowArgs& a) {
  const int ctas = std::min(ceil_div(a.N, GR_WARPS / WPR * R), 4 * std::max(1, a.sm_count));
  return launch_k(gemv_row_kernel<R, WPR, NL, NORM>, dim3(ctas), dim3(GR_THREADS), NORM ? (size_t)a.K * 2 : 0, st, a, next_trace(50));
}
// as few warps to a row as take it in four pieces a lane
template <int R, bool NORM>
static cudaError_t gemv_row_pick(cudaStream_t st, const GemvRowArgs& a) {
  if constexpr (!NORM)
    if (a.K > 4096) return gemv_row_launch<R, 8, 4, NORM>(st, a);
  if (a.K > 2048) return gemv_row_launch<R, 4, 4, NORM>(st, a);
  if (a.K > 1024) return gemv_row_launch<R, 2, 4, NORM>(st, a);
  if (a.K > 768) return gemv_row_launch<R, 1, 4, NORM>(st, a);
  if (a.K > 256) return gemv_row_launch<R, 1, 3, NORM>(st, a);
  return gemv_row_launch<R, 1, 1, NORM>(st, a);
}

cudaError_t launch_gemv_row(cudaStream_t st, const GemvRowArgs& a) {
  if (!gemv_row_fits(a.K, a.norm_w != nullptr) || (a.epi == TC5_EPI_SWIGLU && (a.N & 1)) || a.N < 1) return cudaErrorInvalidValue;
  if (a.epi == TC5_EPI_SWIGLU) return a.norm_w ? gemv_row_pick<2, true>(st, a) : gemv_row_pick<2, false>(st, a);
  return a.norm_w ? gemv_row_pick<1, true>(st, a) : gemv_row_pick<1, false>(st, a);
}

}  // namespace nvllm
