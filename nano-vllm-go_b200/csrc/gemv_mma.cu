// gemv_mma.cu — skinny bf16 GEMM (2 <= M <= 8 rows of activations) that streams the weights once.
//
//   C[m, n] = alpha * sum_k A[m, k] W[n, k], A [M, lda] and W [N, K] bf16, fp32 accumulation.
//
// Bound by the HBM stream of W (N K 2 bytes); at eight rows the arithmetic on the CUDA cores took four times as long
// as that stream (a conversion per weight and 8 FMAs), so the products run on mma.sync m16n8k16: 16 weight rows are
// the M side, the <= 8 activation rows the N side.  Each mma starts from zero, and the four of a chunk are added to four
// fp32 sums that meet in pairs at the end, as the warps' do: 16 products are added inside the tensor core, which drops
// bits, all else is short chains of ordinary fp32 addition.  Against float64, relative to chains of FMAs on the CUDA
// cores: 0.93 to 1.06 times their error from 768 of k on (1.11 to 1.29 times with two mma's in a row and one sum).
// The order of k inside a product is free as long as both operands agree: a lane reads 16 contiguous bytes of a weight
// row and the same 16 of its activation row and feeds their four 2-element pieces to two mma's.
//
// The warps of a CTA share its k range in chunks of 64 and work alone: each has a ring of chunks (its 16 MT weight
// rows and the activation rows) in shared memory that it fills by cp.async, 128 contiguous bytes of a row to eight
// lanes, so a warp keeps several chunks in flight without a register or a barrier; 100 KB in flight per SM cover
// the latency.  (Weights straight to registers, 64 bytes of a row at a time, held 2.6 TB/s: every wait for one
// step waited for the step requested last.)  The warps' sums meet in shared memory: most shapes need no split-K
// slices in global memory at all, and a CTA that holds whole sums can apply the feed-forward's activation itself.
// Alone with a cold L2 (a launch and its two events are 8 us of it): 18176 x 4544 at 8 rows 90.5 -> 42.5 us, at 2 rows
// 45.8 -> 42.4; 2048 x 8192 at 8 rows 27.0 -> 15.6; 768 x 768 10.3 -> 8.0.  Inside a step of two Falcon layers 5.6 TB/s.
// At one row the CUDA-core kernel is as fast alone and faster in a chain of small products (GPT-2 small: 344 against
// 363 us per token), so it keeps that row count.
#include "common.cuh"
#include "kernels.h"
#include "mma.cuh"

namespace nvllm {

__device__ __forceinline__ uint4 ld_shared16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

constexpr int GM_CK = 64;  // k of a chunk: 128 bytes of a row

// byte offset of 16-byte piece c of row r: odd rows swap their halves, so the two rows that eight lanes read at once
// lie in different banks
__device__ __forceinline__ uint32_t gm_at(int r, int c) { return (uint32_t)(r * 128 + ((c ^ ((r & 1) << 2)) << 4)); }

// MT: 16-row weight tiles per warp; NW warps; NS chunks in a warp's ring
template <int MT, int NW, int NS>
__global__ void __launch_bounds__(NW * 32)
gemv_mma_kernel(GemvMmaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  constexpr uint32_t W_BYTES = 16 * MT * 128, STAGE = W_BYTES + 8 * 128;
  extern __shared__ __align__(128) uint8_t ring[];  // [warp][stage][weights | activations]
  __shared__ float fin[8][16 * MT];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int n0 = blockIdx.x * 16 * MT;
  const int ks = blockIdx.y * a.KC, ke = min(a.K, ks + a.KC);
  const int chunks = (ke - ks + GM_CK - 1) / GM_CK;  // of this CTA; warp w takes chunks w, w + NW, ...
  const int mine = (chunks - warp + NW - 1) / NW;
  const uint32_t base = smem_addr(ring) + (uint32_t)warp * NS * STAGE;
  // loader: lane covers 16 bytes (piece lc) of rows lr, lr + 4, ...
  const int lr = lane >> 3, lc = lane & 7;
  auto fetch_w = [&](int i) {  // K is a multiple of 8: a piece is all inside or all outside (zeros)
    const uint32_t st = base + (uint32_t)(i % NS) * STAGE;
    const int k = ks + (warp + i * NW) * GM_CK + lc * 8;
    const bool in = k < ke;
#pragma unroll
    for (int r = lr; r < 16 * MT; r += 4)
      cp_async16_once(st + gm_at(r, lc), a.W + (size_t)min(n0 + r, a.N - 1) * a.K + (in ? k : 0), in);
  };
  auto fetch_a = [&](int i) {
    const uint32_t st = base + (uint32_t)(i % NS) * STAGE + W_BYTES;
    const int k = ks + (warp + i * NW) * GM_CK + lc * 8;
    const bool in = k < ke;
#pragma unroll
    for (int r = lr; r < 8; r += 4)
      cp_async16(st + gm_at(r, lc), a.A + (size_t)min(r, a.M - 1) * a.lda + (in ? k : 0), in && r < a.M);
  };
  // the weights are immutable: the ring's first chunks are requested before the dependency resolves
#pragma unroll
  for (int i = 0; i < NS - 1; i++)
    if (i < mine) fetch_w(i);
  pdl_wait();
#pragma unroll
  for (int i = 0; i < NS - 1; i++) {
    if (i < mine) fetch_a(i);
    cp_async_commit();
  }
  float acc[4][MT][4] = {};  // [mma of a chunk]
  for (int i = 0; i < mine; i++) {
    cp_async_wait<NS - 2>();
    __syncwarp();  // chunk i has arrived for every lane, and every lane is done with the stage that is filled next
    if (i + NS - 1 < mine) {
      fetch_w(i + NS - 1);
      fetch_a(i + NS - 1);
    }
    cp_async_commit();
    const uint32_t st = base + (uint32_t)(i % NS) * STAGE;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const uint4 x = ld_shared16(st + W_BYTES + gm_at(g, 4 * j + q));
#pragma unroll
      for (int t = 0; t < MT; t++) {
        const uint4 lo = ld_shared16(st + gm_at(16 * t + g, 4 * j + q)), hi = ld_shared16(st + gm_at(16 * t + g + 8, 4 * j + q));
        float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
        mma16816(d0, lo.x, hi.x, lo.y, hi.y, x.x, x.y);
        mma16816(d1, lo.z, hi.z, lo.w, hi.w, x.z, x.w);
#pragma unroll
        for (int e = 0; e < 4; e++) {
          acc[2 * j][t][e] += d0[e];
          acc[2 * j + 1][t][e] += d1[e];
        }
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();  // the rings are done with: the warps' sums take their place
  float (*red)[8][16 * MT] = reinterpret_cast<float (*)[8][16 * MT]>(ring);
#pragma unroll
  for (int i = 0; i < MT; i++) {  // fragment: weight rows g and g + 8, activation rows 2 q and 2 q + 1
    float s[4];
#pragma unroll
    for (int e = 0; e < 4; e++) s[e] = (acc[0][i][e] + acc[1][i][e]) + (acc[2][i][e] + acc[3][i][e]);
    red[warp][2 * q][16 * i + g] = s[0];
    red[warp][2 * q + 1][16 * i + g] = s[1];
    red[warp][2 * q][16 * i + g + 8] = s[2];
    red[warp][2 * q + 1][16 * i + g + 8] = s[3];
  }
  __syncthreads();
  for (int e = tid; e < a.M * 16 * MT; e += NW * 32) {
    const int m = e / (16 * MT), r = e % (16 * MT), n = n0 + r;
    float p[NW];
#pragma unroll
    for (int w = 0; w < NW; w++) p[w] = red[w][m][r];
#pragma unroll
    for (int o = 1; o < NW; o <<= 1)
#pragma unroll
      for (int w = 0; w < NW; w += 2 * o) p[w] += p[w + o];
    float v = a.alpha * p[0];
    if (a.epi == TC5_EPI_PARTIAL) {
      if (n < a.N) a.out[(size_t)blockIdx.y * a.split_stride + (size_t)m * a.ldo + n] = v;
    } else if (a.epi == TC5_EPI_SWIGLU) {
      fin[m][r] = v;
    } else if (n < a.N) {
      if (a.epi_bias) v += a.epi_bias[n];
      a.epi_out[(size_t)m * a.epi_ld + n] = from_f32<bf16>(a.epi == TC5_EPI_RELU2 ? relu2(v) : gelu_tanh(v));
    }
  }
  if (a.epi == TC5_EPI_SWIGLU) {  // rows 2 j and 2 j + 1 of the weights are gate and up of column j
    __syncthreads();
    for (int e = tid; e < a.M * 8 * MT; e += NW * 32) {
      const int m = e / (8 * MT), j = e % (8 * MT);
      if (n0 + 2 * j + 1 < a.N)
        a.epi_out[(size_t)m * a.epi_ld + n0 / 2 + j] = from_f32<bf16>(glu_unit(fin[m][2 * j], fin[m][2 * j + 1], a.glu_limit));
    }
  }
  TRACE_EXIT(tr);
}

// 32 weight rows per CTA where that still gives two CTAs per SM, else 16; then k is split over CTAs until there
// are two per SM, each keeping at least 256 of k.  `most` bounds the slices.
GemvMmaPlan gemv_mma_plan(int N, int K, int most) {
  GemvMmaPlan p;
  p.mt = ceil_div(N, 32) >= 296 ? 2 : 1;
  const int tiles = ceil_div(N, 16 * p.mt);
  int S = 1;
  while (S < most && tiles * S < 296 && K / (S + 1) >= 256) S++;
  p.KC = ceil_div(ceil_div(K, GM_CK), S) * GM_CK;
  p.S = ceil_div(K, p.KC);
  return p;
}

template <int MT, int NW, int NS>
static cudaError_t gemv_mma_launch(cudaStream_t st, const GemvMmaArgs& a, const GemvMmaPlan& p) {
  constexpr int smem = NW * NS * (16 * MT + 8) * 128;
  const cudaError_t e = cudaFuncSetAttribute(gemv_mma_kernel<MT, NW, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  return launch_k(gemv_mma_kernel<MT, NW, NS>, dim3(ceil_div(a.N, 16 * MT), p.S), dim3(NW * 32), smem, st, a, next_trace(11));
}
cudaError_t launch_gemv_mma(cudaStream_t st, const GemvMmaArgs& a, const GemvMmaPlan& p) {
  return p.mt == 2 ? gemv_mma_launch<2, 4, 5>(st, a, p) : gemv_mma_launch<1, 8, 4>(st, a, p);
}

}  // namespace nvllm
