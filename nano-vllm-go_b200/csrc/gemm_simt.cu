// gemm_simt.cu — CUDA-core matrix kernels.
//
//  * gemv_kernel: skinny weight-streaming split-K GEMV: M <= 8 in fp32 mode, one row in bf16 mode (more: gemv_mma.cu).
//    Weights [N,K] are read exactly once with 16-byte streaming loads (L1 no-allocate), one
//    warp per R output rows, activations staged in shared memory as fp32, fp32 accumulate.
//    HBM-bound: algorithmic bytes = N*K*sizeof(W).
//  * gemm_f32_kernel: register-tiled packed-FMA GEMM of the fp32 PARITY mode for few rows and small weights (the others:
//    gemm_f32_tc5.cu), and its grouped (MoE expert) GEMM with row gather.
//  * gemm_simt_kernel: 64x64x16 fp32-FMA tiles on bf16 operands that the tcgen05 path cannot address.
//
// All compute C[m,n] = alpha * sum_k A[m,k] * W[n,k]  (reference tensor.go:62-88 MatMul with
// the weight held [out,in]) and write fp32 split-K partials.
#include "common.cuh"
#include "kernels.h"
#include "mma.cuh"

namespace nvllm {

// ------------------------------------------------------------------ GEMV
struct GemvPlan {
  int warps, R, KC, S;
};
static GemvPlan gemv_plan(int M, int N, int K) {
  GemvPlan p;
  p.warps = 8;
  p.R = (M > 2) ? 4 : 2;
  int kc_max = (M > 4) ? 1024 : 2048;  // fp32 activations in smem: M*KC*4 <= 32 KB
  p.KC = kc_max;
  auto ctas = [&](int R, int KC) { return ceil_div(N, p.warps * R) * ceil_div(K, KC); };
  // fill 148 SMs x 2 CTAs when the matrix is small: first shrink the K chunk, then R
  while (ctas(p.R, p.KC) < 296 && p.KC > 512) p.KC /= 2;
  while (ctas(p.R, p.KC) < 296 && p.R > 1) p.R /= 2;
  if (p.KC > K) p.KC = ceil_div(K, 256) * 256;
  p.S = ceil_div(K, p.KC);
  return p;
}
int gemv_splits(int M, int N, int K) { return gemv_plan(M, N, K).S; }

// 8 weight elements as loaded (the conversion to fp32 is deferred to the use)
template <typename WT> struct Raw8;
template <> struct Raw8<bf16> {
  uint4 v;
  __device__ __forceinline__ void ld(const bf16* p) { v = ld_once16(p); }
  __device__ __forceinline__ void cvt(float (&o)[8]) const {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      float2 f = __bfloat1622float2(h[i]);
      o[2 * i] = f.x;
      o[2 * i + 1] = f.y;
    }
  }
};
template <> struct Raw8<float> {
  uint4 a, b;
  __device__ __forceinline__ void ld(const float* p) {
    a = ld_stream16(p);
    b = ld_stream16(p + 4);
  }
  __device__ __forceinline__ void cvt(float (&o)[8]) const {
    o[0] = __uint_as_float(a.x); o[1] = __uint_as_float(a.y); o[2] = __uint_as_float(a.z); o[3] = __uint_as_float(a.w);
    o[4] = __uint_as_float(b.x); o[5] = __uint_as_float(b.y); o[6] = __uint_as_float(b.z); o[7] = __uint_as_float(b.w);
  }
};

// The weights are immutable: every warp issues the loads of its first GEMV_PF k-iterations
// BEFORE griddepcontrol.wait, so the HBM stream of this GEMV runs under the tail of the kernel
// in front of it (a single-sequence decode step is a chain of ~100 such dependent launches).
constexpr int GEMV_PF = 2;
template <typename T, int M, int R>
__global__ void __launch_bounds__(256)
gemv_kernel(const T* __restrict__ A, int lda, const T* __restrict__ W, int N, int K, int KC,
            float* __restrict__ out, int ldo, size_t split_stride, float alpha, GemvPre pre, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  extern __shared__ float a_s[];  // [M][KC]
  const int ks = blockIdx.y * KC;
  const int ke = min(K, ks + KC);
  const int klen = ke - ks;
  Raw8<T> wpre[GEMV_PF][R];
  {
    const int lane_ = threadIdx.x & 31, warp_ = threadIdx.x >> 5, nw_ = blockDim.x >> 5;
    const int n0_ = (blockIdx.x * nw_ + warp_) * R;
    if (n0_ < N) {
#pragma unroll
      for (int it = 0; it < GEMV_PF; it++) {
        const int k = lane_ * 8 + it * 256;
        if (k < klen) {
#pragma unroll
          for (int r = 0; r < R; r++) wpre[it][r].ld(W + (size_t)min(n0_ + r, N - 1) * K + ks + k);
        }
      }
    }
  }
  pdl_wait();
  if (pre.mode == 0) {
    for (int i = threadIdx.x * 8; i < M * KC; i += blockDim.x * 8) {
      const int m = i / KC, k = i % KC;
      float v[8];
      if (k < klen) {
        load8(A + (size_t)m * lda + ks + k, v);
      } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = 0.f;
      }
      store8(a_s + i, v);
    }
  } else {
    // the activation kernel's work (act_kernel): SwiGLU over interleaved gate / up columns or
    // tanh-GELU of the FFN up projection's split-K slices (transformer.go:50-78)
    for (int i = threadIdx.x; i < M * KC; i += blockDim.x) {
      const int m = i / KC, k = i % KC;
      float y = 0.f;
      if (k < klen) {
        const int col = ks + k;
        if (pre.swiglu == 1) {
          float g = 0.f, u = 0.f;
          for (int sl = 0; sl < pre.Sh; sl++) {
            const float* hrow = pre.hp + (size_t)sl * pre.hstride + (size_t)m * pre.hld + 2 * col;
            g += hrow[0];
            u += hrow[1];
          }
          y = glu_unit(g, u, pre.glu_limit);
        } else {
          float hsum = 0.f;
          for (int sl = 0; sl < pre.Sh; sl++) hsum += pre.hp[(size_t)sl * pre.hstride + (size_t)m * pre.hld + col];
          if (pre.hbias) hsum += pre.hbias[col];
          y = pre.swiglu == 2 ? relu2(hsum) : gelu_tanh(hsum);
        }
        y = to_f32(from_f32<T>(y));
      }
      a_s[i] = y;
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int n0 = (blockIdx.x * nwarps + warp) * R;
  if (n0 >= N) return;
  float acc[R][M];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int m = 0; m < M; m++) acc[r][m] = 0.f;
  const T* wrow[R];
#pragma unroll
  for (int r = 0; r < R; r++) wrow[r] = W + (size_t)min(n0 + r, N - 1) * K + ks;

  auto fma_block = [&](const float (&w)[R][8], int k) {
#pragma unroll
    for (int m = 0; m < M; m++) {
      float a[8];
      load8(a_s + m * KC + k, a);
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[r][m] = fmaf(w[r][j], a[j], acc[r][m]);
    }
  };
#pragma unroll
  for (int it = 0; it < GEMV_PF; it++) {
    const int k = lane * 8 + it * 256;
    if (k < klen) {
      float w[R][8];
#pragma unroll
      for (int r = 0; r < R; r++) wpre[it][r].cvt(w[r]);
      fma_block(w, k);
    }
  }
#pragma unroll 2
  for (int k = lane * 8 + GEMV_PF * 256; k < klen; k += 256) {
    float w[R][8];
#pragma unroll
    for (int r = 0; r < R; r++) load8_stream(wrow[r] + k, w[r]);
#pragma unroll
    for (int m = 0; m < M; m++) {
      float a[8];
      load8(a_s + m * KC + k, a);
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[r][m] = fmaf(w[r][j], a[j], acc[r][m]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int m = 0; m < M; m++) {
      float v = warp_sum(acc[r][m]);
      if (lane == 0 && n0 + r < N)
        out[(size_t)blockIdx.y * split_stride + (size_t)m * ldo + n0 + r] = alpha * v;
    }
  TRACE_EXIT(tr);
}

template <typename T, int M>
static cudaError_t gemv_dispatch_r(cudaStream_t st, const GemmArgs& g, const GemvPlan& p, const GemvPre& pre) {
  dim3 grid(ceil_div(g.N, p.warps * p.R), p.S);
  size_t smem = (size_t)M * p.KC * sizeof(float);
#define GV(RR)                                                                                     \
  (void)launch_k(gemv_kernel<T, M, RR>, dim3(grid), dim3(p.warps * 32), smem, st,                                     \
      (const T*)g.A, g.lda, (const T*)g.W, g.N, g.K, p.KC, g.out, g.ldo, g.split_stride, g.alpha, \
      pre, next_trace(11))
  if (p.R == 4) GV(4);
  else if (p.R == 2) GV(2);
  else GV(1);
#undef GV
  return cudaGetLastError();
}
template <typename T>
static cudaError_t gemv_dispatch_m(cudaStream_t st, const GemmArgs& g, const GemvPlan& p, const GemvPre& pre) {
  switch (g.M) {
    case 1: return gemv_dispatch_r<T, 1>(st, g, p, pre);
    case 2: return gemv_dispatch_r<T, 2>(st, g, p, pre);
    case 3: return gemv_dispatch_r<T, 3>(st, g, p, pre);
    case 4: return gemv_dispatch_r<T, 4>(st, g, p, pre);
    case 5: return gemv_dispatch_r<T, 5>(st, g, p, pre);
    case 6: return gemv_dispatch_r<T, 6>(st, g, p, pre);
    case 7: return gemv_dispatch_r<T, 7>(st, g, p, pre);
    case 8: return gemv_dispatch_r<T, 8>(st, g, p, pre);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_gemv(cudaStream_t st, GemmArgs& g, const GemvPre* pre_in) {
  GemvPre pre{};
  if (pre_in) pre = *pre_in;
  if (g.M < 1 || g.M > 8 || (g.K % 8) != 0) return cudaErrorInvalidValue;
  if (pre.mode != 0 && pre.mode != 2) return cudaErrorInvalidValue;
  GemvPlan p = gemv_plan(g.M, g.N, g.K);
  g.S = p.S;
  if (g.out_capacity && (size_t)p.S * g.split_stride > g.out_capacity) return cudaErrorInvalidValue;
  if (g.adt == DT_F32 && g.wdt == DT_F32) return gemv_dispatch_m<float>(st, g, p, pre);
  if (g.adt == DT_BF16 && g.wdt == DT_BF16) {
    if (g.M < GEMV_MMA_ROWS) return gemv_dispatch_r<bf16, 1>(st, g, p, pre);
    if (pre.mode != 0) return cudaErrorInvalidValue;
    // gemv_mma_plan stays within the slices that the callers have room for
    const GemvMmaPlan mp = gemv_mma_plan(g.N, g.K, p.S);
    g.S = mp.S;
    GemvMmaArgs a{};
    a.A = (const bf16*)g.A; a.W = (const bf16*)g.W; a.lda = g.lda; a.M = g.M; a.N = g.N; a.K = g.K; a.KC = mp.KC;
    a.out = g.out; a.ldo = g.ldo; a.split_stride = g.split_stride; a.alpha = g.alpha;
    return launch_gemv_mma(st, a, mp);
  }
  return cudaErrorInvalidValue;
}

// ------------------------------------------------------------------ tiled SIMT GEMM
constexpr int SBM = 64, SBN = 64, SBK = 16;

__device__ __forceinline__ void load4(const bf16* p, float (&v)[4]) {
  uint2 r = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
  float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

__global__ void __launch_bounds__(256)
gemm_simt_kernel(GemmArgs g, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float As[2][SBK][SBM + 4];
  __shared__ float Ws[2][SBK][SBN + 4];
  int row0, rows_valid;
  const bf16* W = (const bf16*)g.W;
  if (g.tile_expert) {
    if ((int)blockIdx.x >= *g.n_tiles) return;
    row0 = g.tile_row0[blockIdx.x];
    rows_valid = g.tile_rows[blockIdx.x];
    W += (size_t)g.tile_expert[blockIdx.x] * g.expert_stride;
  } else {
    row0 = blockIdx.x * SBM;
    rows_valid = min(SBM, g.M - row0);
  }
  const int col0 = blockIdx.y * SBN;
  const bf16* A = (const bf16*)g.A;
  const int tid = threadIdx.x;
  // loader mapping: 64 rows x 16 k = 256 threads x 4 consecutive k
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  int arow = -1;
  if (lr < rows_valid) arow = g.a_rows ? g.a_rows[row0 + lr] : row0 + lr;
  const int wrow = (col0 + lr < g.N) ? col0 + lr : -1;
  const bf16* ap = (arow >= 0) ? A + (size_t)arow * g.lda : nullptr;
  const bf16* wp = (wrow >= 0) ? W + (size_t)wrow * g.K : nullptr;
  const int ty = tid >> 4, tx = tid & 15;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;

  float ra[4], rw[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int j = 0; j < 4; j++) ra[j] = rw[j] = 0.f;
    if (k0 + lk < g.K) {  // K % 4 == 0 is guaranteed (K % 8 == 0)
      if (ap) load4(ap + k0 + lk, ra);
      if (wp) load4(wp + k0 + lk, rw);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      As[buf][lk + j][lr] = ra[j];
      Ws[buf][lk + j][lr] = rw[j];
    }
  };
  const int nk = ceil_div(g.K, SBK);
  fetch(0);
  stash(0);
  __syncthreads();
  for (int kb = 0; kb < nk; kb++) {
    const int buf = kb & 1;
    if (kb + 1 < nk) fetch((kb + 1) * SBK);
#pragma unroll
    for (int k = 0; k < SBK; k++) {
      float4 a4 = *reinterpret_cast<const float4*>(&As[buf][k][ty * 4]);
      float4 b4 = *reinterpret_cast<const float4*>(&Ws[buf][k][tx * 4]);
      const float a[4] = {a4.x, a4.y, a4.z, a4.w};
      const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (kb + 1 < nk) {
      stash(buf ^ 1);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r = ty * 4 + i;
    if (r >= rows_valid) continue;
    float* orow = g.out + (size_t)(row0 + r) * g.ldo;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int c = col0 + tx * 4 + j;
      if (c < g.N) orow[c] = g.alpha * acc[i][j];
    }
  }
  TRACE_EXIT(tr);
}

// ------------------------------------------------------------------ tiled fp32 GEMM
// C tile of 8 MI x 64 by four warps, a lane holds MI x 4 sums, each as a packed pair: the even and the odd k of every
// step of two, added at the end, so that the 16-byte pieces of A and W feed the packed FMA (f32x2, two IEEE
// fp32 operations) as they lie in memory.  A and W go to shared memory in steps of 32 k by 16-byte cp.async, three
// stages deep; rows are 36 floats apart, which puts the 8 (4) rows that a warp reads at once on different
// banks.  k is split over CTAs (fp32 slices, summed by the consumer) so that the SMs get equal shares.
// Bound by latency and, next to it, by shared memory: per 4 k a lane reads 4 + MI pieces, four passes of the SM's shared
// memory each, for 8 MI packed FMAs, at MI = 8 48 passes beside 32 cycles of the FMA lanes; with 138 registers three
// CTAs (nine warps) fit an SM, and both are little more than half busy (57 % and 55 % in a product of 300 x 2304 x 768).
// MI = 2 / 4 keep tiles of 16 / 32 rows for small steps, which are bound by the weights.
// GPT-2 small, four prompts of 50 to 100 tokens (now on gemm_f32_tc5.cu): the step's 48 matrix products 7.24 -> 2.04 ms
// against tiles of 64 x 64 x 16 with scalar FMAs, operands transposed through registers and one k range (60 to 240 CTAs of
// the chip's 296); 32 TFLOP/s in the widest, three CTAs per SM (four at 128 registers each: 2.50 ms).
constexpr int FG_BN = 64, FG_BK = 32, FG_PITCH = 36, FG_STAGES = 3, FG_THREADS = 128;

template <int MI>
__global__ void __launch_bounds__(FG_THREADS)
gemm_f32_kernel(GemmArgs g, int kc, Trace tr) {
  TRACE_ENTRY(tr);
  constexpr int BM = 8 * MI;
  extern __shared__ __align__(16) float fsm[];  // [stage][BM + 64][pitch]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  int row0, rows_valid;
  const float* W = (const float*)g.W;
  if (g.tile_expert) {
    if ((int)blockIdx.x >= *g.n_tiles) return;
    row0 = g.tile_row0[blockIdx.x];
    rows_valid = g.tile_rows[blockIdx.x];
    W += (size_t)g.tile_expert[blockIdx.x] * g.expert_stride;
  } else {
    row0 = blockIdx.x * BM;
    rows_valid = min(BM, g.M - row0);
  }
  const int col0 = blockIdx.y * FG_BN;
  const int ks = blockIdx.z * kc, ke = min(g.K, ks + kc);
  const int nk = (ke - ks + FG_BK - 1) / FG_BK;
  // loader: 8 pieces of 16 bytes per row and step, 16 rows at a time
  const int lr = tid >> 3, lp = (tid & 7) * 4;
  constexpr int LA = (BM + 15) / 16;
  const float* ap[LA];
#pragma unroll
  for (int i = 0; i < LA; i++) {
    const int r = lr + 16 * i;
    ap[i] = r < rows_valid ? (const float*)g.A + (size_t)(g.a_rows ? g.a_rows[row0 + r] : row0 + r) * g.lda + ks + lp : nullptr;
  }
  const float* wp[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int n = col0 + lr + 16 * i;
    wp[i] = n < g.N ? W + (size_t)n * g.K + ks + lp : nullptr;
  }
  const float* any = (const float*)g.A;  // a valid address for pieces that are filled with zeros
  auto fetch = [&](int kb) {
    if (kb < nk) {
      float* dst = fsm + (kb % FG_STAGES) * (BM + FG_BN) * FG_PITCH + lr * FG_PITCH + lp;
      const int k = kb * FG_BK;
      const bool in = ks + k + lp < ke;  // K and the k ranges are multiples of 4
#pragma unroll
      for (int i = 0; i < LA; i++)
        if (lr + 16 * i < BM) cp_async16(smem_addr(dst + 16 * i * FG_PITCH), ap[i] && in ? ap[i] + k : any, ap[i] && in);
#pragma unroll
      for (int i = 0; i < 4; i++) cp_async16(smem_addr(dst + (BM + 16 * i) * FG_PITCH), wp[i] && in ? wp[i] + k : any, wp[i] && in);
    }
    cp_async_commit();
  };
  const int am = (warp >> 1) * 4 + (lane >> 3), wn = (warp & 1) * 8 + (lane & 7);
  unsigned long long acc[MI][4];
#pragma unroll
  for (int i = 0; i < MI; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
#pragma unroll
  for (int i = 0; i + 1 < FG_STAGES; i++) fetch(i);
  for (int kb = 0; kb < nk; kb++) {
    cp_async_wait<FG_STAGES - 2>();
    __syncthreads();  // step kb has arrived, and step kb - 1's buffer is free
    fetch(kb + FG_STAGES - 1);
    const float* a_s = fsm + (kb % FG_STAGES) * (BM + FG_BN) * FG_PITCH + am * FG_PITCH;
    const float* w_s = fsm + (kb % FG_STAGES) * (BM + FG_BN) * FG_PITCH + (BM + wn) * FG_PITCH;
#pragma unroll
    for (int k = 0; k < FG_BK; k += 4) {
      ulonglong2 w[4];
#pragma unroll
      for (int j = 0; j < 4; j++) w[j] = *reinterpret_cast<const ulonglong2*>(w_s + 16 * j * FG_PITCH + k);
#pragma unroll
      for (int i = 0; i < MI; i++) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(a_s + 8 * i * FG_PITCH + k);
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fma2(a.x, w[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fma2(a.y, w[j].y, acc[i][j]);
      }
    }
  }
  // The kernels behind this one are let in here and not at its start.  They release each other at once, so that the next
  // product's CTAs used to come in while these still filled the SMs unevenly, and stayed where they came in: six on one SM,
  // two on most.  (Between them a norm of a step takes most of an SM's registers, which made it worse.)  Decode steps of
  // 9, 12, 16 sequences in fp32, us released at the start / here: GPT-2 787 / 576, 785 / 580, 879 / 586; four Llama-1B layers
  // 581 / 516, 582 / 520, 579 / 527; a delta-rule and a window layer 373 / 294, 424 / 314, 481 / 313.  (Eight blocks of k
  // earlier 629, 537 and 326 in those of 9.)
  pdl_launch_dependents();
  float* out = g.out + (size_t)blockIdx.z * g.split_stride;
#pragma unroll
  for (int i = 0; i < MI; i++) {
    const int r = 8 * i + am;
    if (r >= rows_valid) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int n = col0 + 16 * j + wn;
      float lo, hi;
      unpack2(acc[i][j], lo, hi);
      if (n < g.N) out[(size_t)(row0 + r) * g.ldo + n] = g.alpha * (lo + hi);
    }
  }
  TRACE_EXIT(tr);
}

template <int MI>
static cudaError_t gemm_f32_launch(cudaStream_t st, const GemmArgs& g, dim3 grid, int kc) {
  constexpr size_t smem = (size_t)FG_STAGES * (8 * MI + FG_BN) * FG_PITCH * sizeof(float);
  if (smem > 48 * 1024) {  // (an attribute of the device's kernel: set on whichever device is current)
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<MI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  return launch_k(gemm_f32_kernel<MI>, grid, dim3(FG_THREADS), smem, st, g, kc, next_trace(12));
}

static cudaError_t launch_gemm_f32(cudaStream_t st, GemmArgs& g) {
  const int mi = g.tile_expert || g.M > 32 ? 8 : g.M > 16 ? 4 : 2;
  const int mt = g.tile_expert ? g.max_tiles : ceil_div(g.M, 8 * mi), nt = ceil_div(g.N, FG_BN);
  g.S = 1;
  if (mt == 0 || nt == 0) return cudaSuccess;
  // slices: up to the eight that a consumer sums with one batch of loads, each at least 128 of k, as many as the buffer
  // has room for (grouped tiles write one slice): the count with the least work on the fullest SM, in steps of 32 k
  // plus two for a CTA's fill and its results; an SM with fewer than three CTAs runs them at a lower rate (two cost 2.4,
  // one 1.8 where three cost 3), and a consumer reads every slice (0.3).  Against the best of all eight counts, each
  // timed alone with a cold L2, 9 to 800 rows, 768 to 8192 columns and 768 to 8192 of k: the count chosen is within
  // 10 % in 57 of 63 shapes, 17 % behind at worst (9 rows of 768 x 768, 10.0 us against 8.6)
  int S = 1;
  if (!g.tile_expert && g.out_capacity) {
    double best = 1e30;
    for (int s = 1; s <= 8 && (s == 1 || g.K / s >= 128) && (s == 1 || (size_t)s * g.split_stride <= g.out_capacity); s++) {
      const int per_sm = ceil_div(mt * nt * s, 148), steps = ceil_div(ceil_div(g.K, FG_BK), s);
      const double cost = (per_sm >= 3 ? per_sm : per_sm == 2 ? 2.4 : 1.8) * (steps + 2.0) + 0.3 * s;
      if (cost < best) {
        best = cost;
        S = s;
      }
    }
  }
  const int kc = ceil_div(ceil_div(g.K, FG_BK), S) * FG_BK;
  g.S = ceil_div(g.K, kc);
  const dim3 grid(mt, nt, g.S);
  if (mi == 8) return gemm_f32_launch<8>(st, g, grid, kc);
  if (mi == 4) return gemm_f32_launch<4>(st, g, grid, kc);
  return gemm_f32_launch<2>(st, g, grid, kc);
}

cudaError_t launch_gemm_simt(cudaStream_t st, GemmArgs& g) {
  if ((g.K % 8) != 0) return cudaErrorInvalidValue;
  if (gemm_f32_tc5_fits(g)) return launch_gemm_f32_tc5(st, g);
  if (g.adt == DT_F32 && g.wdt == DT_F32) return launch_gemm_f32(st, g);
  g.S = 1;
  dim3 grid(g.tile_expert ? g.max_tiles : ceil_div(g.M, SBM), ceil_div(g.N, SBN));
  if (grid.x == 0 || grid.y == 0) return cudaSuccess;
  if (g.adt != DT_BF16 || g.wdt != DT_BF16) return cudaErrorInvalidValue;
  (void)launch_k(gemm_simt_kernel, dim3(grid), dim3(256), 0, st, g, next_trace(12));
  return cudaGetLastError();
}

}  // namespace nvllm
