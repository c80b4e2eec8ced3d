// gemm_f32_tc5.cu — fp32 GEMM on the tensor cores: every fp32 operand as the exact sum of three bf16 parts.
//
// x = hi + mid + lo with hi = bf16(x), mid = bf16(x - hi), lo = x - hi - mid (24 bits = 3 x 8, each part rounded to
// nearest, so mid <= 2^-9 |x| and lo <= 2^-18 |x|).  Exact down to some 2^-110: below, lo falls under bf16's smallest
// subnormal, and an operand is off by up to 2^-134.  Of the nine products of parts the six above 2^-27 of the whole are
// summed; what is left out is below the rounding of one fp32 product.  The tensor core's fp32 sums drop bits where an
// FMA rounds, so no sum stays in it for long: each stage of 64 k starts from zero in tensor memory, in two
// accumulators by size (hi hi; the other five), and is added to fp32 registers, which round to nearest.
//
// Weights are the UMMA M side (128 rows), tokens the N side (BT rows).  (MMAs are only ordered among those of one shape
// on one accumulator, so the parts of the token tile are not joined to wider MMAs.)  Sixteen warps fetch fp32 pieces from
// global memory one stage ahead, split them and store the parts in the 128-byte swizzle; one warp issues the MMAs; eight
// warps sum the stages (tensor memory, double-buffered) and write the tile.  Persistent: units (weight tile, token tile,
// k slice) go round the CTAs.
//
// An operand with a part that is not finite (infinity, NaN, or a value that bf16 rounds to infinity) turns into NaN in the
// split, and products out of range into infinities of both signs, where fp32 arithmetic may have an infinity: results that
// are not finite are computed again with FMAs, by a warp each, until the sum is NaN.
//
// Bound by the MMAs' reads of shared memory (24 MMAs a stage, 60 cycles each at BT = 64, 79 at 128) with the splitters
// close behind: with eight of their warps instead of sixteen a stage took 1.57 / 1.85 us instead of 1.19 / 1.55.
// GPT-2 small, four prompts of 50 to 100 tokens: the whole step 2.69 -> 1.70 ms against the SIMT tiles; 2048 x 8192 x
// 2048 44 -> 188 TFLOP/s.  Relative error (2-norm) against float64, SIMT / this kernel: 300 x 2304 x 768 3.5e-7 / 9.7e-8,
// 300 x 768 x 3072 7.0e-7 / 1.5e-7, 9 to 300 rows and 64 to 8192 of k 1.1e-7..1.1e-6 / 7e-8..2.2e-7.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "gemm_tc5.cuh"
#include "kernels.h"

namespace nvllm {

constexpr int FT_SUM = 8, FT_SPLIT = 16;  // warps that sum the stages, warps that split; a warpgroup for the MMAs between them
constexpr int FT_THREADS = 32 * (FT_SUM + 4 + FT_SPLIT);
// registers per thread after the roles part: 2 x 104 + 40 + 4 x 64 for the seven warpgroups that start with 72 each
constexpr int FT_REGS = 72, FT_REGS_SUM = 104, FT_REGS_MMA = 40, FT_REGS_SPLIT = 64;
static_assert(2 * FT_REGS_SUM + FT_REGS_MMA + 4 * FT_REGS_SPLIT <= 7 * FT_REGS, "no more than the launch brought");

template <int BT> struct FtSizes {
  static constexpr int STAGES = BT > 32 ? 2 : 3;
  static constexpr uint32_t W_PART = TC_BN * TC_BK * 2, A_PART = BT * TC_BK * 2;
  static constexpr uint32_t STAGE = 3 * (W_PART + A_PART);
  static constexpr uint32_t ACC = 2 * BT;  // accumulator columns of a stage
  static constexpr int NC = BT / 2, CHUNK = NC < 32 ? NC : 32;  // tokens of a summing warp; of them staged at a time
  static constexpr uint32_t OUT = 2 * CHUNK * TC_BN * 4;        // results on their way out, of both halves of the tokens
  static constexpr size_t SMEM = (size_t)STAGES * STAGE + OUT + 1024;
};

struct F32Tc5Args {
  const float *A, *W;
  int lda, M, N, K;
  int n_tiles, m_tiles, S, kc;  // kc: k of a slice, a multiple of TC_BK
  float* out;
  int ldo;
  size_t split_stride;
  float alpha;
  int* flag;
  int wide;  // rows of `out` start on 16-byte boundaries
  int late;  // W comes from the kernel in front
};

struct F8 {  // eight consecutive values, as the packed operations take them
  unsigned long long v[4];
};
// 32 bytes on their own boundary, no line kept in L1
// (volatile: not before the wait for the kernel that wrote them)
__device__ __forceinline__ F8 ld_piece(const float* p) {
  F8 r;
  asm volatile("ld.global.L1::no_allocate.v4.b64 {%0, %1, %2, %3}, [%4];"
               : "=l"(r.v[0]), "=l"(r.v[1]), "=l"(r.v[2]), "=l"(r.v[3]) : "l"(p));
  return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint32_t round_bf16x2(unsigned long long v) {
  float a, b;
  unpack2(v, a, b);
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ unsigned long long widen_bf16x2(uint32_t h) {
  return pack2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u));
}
__device__ __forceinline__ void split2(unsigned long long x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = round_bf16x2(x);
  const unsigned long long r = sub2(x, widen_bf16x2(hi));
  mid = round_bf16x2(r);
  lo = round_bf16x2(sub2(r, widen_bf16x2(mid)));
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint32_t (&v)[4]) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void tmem_ld_32x8_nowait(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// the whole warp: sum of a[k] w[k], k0 <= k < k1 (multiples of 8), in fp32; ends early once it is NaN.  Rare: kept out of the
// kernel's registers.
__device__ __noinline__ float warp_dot(const float* a, const float* w, int k0, int k1, int lane) {
  float v = 0.f;
  for (int k = k0 + 4 * lane; __any_sync(0xffffffffu, k < k1) && !__any_sync(0xffffffffu, v != v);) {
#pragma unroll
    for (int i = 0; i < 4; i++, k += 128) {
      if (k >= k1) continue;
      const float4 x = __ldcg(reinterpret_cast<const float4*>(a + k)), y = __ldcg(reinterpret_cast<const float4*>(w + k));
      v = fmaf(x.x, y.x, v);
      v = fmaf(x.y, y.y, v);
      v = fmaf(x.z, y.z, v);
      v = fmaf(x.w, y.w, v);
    }
  }
  return warp_sum(v);
}

template <int BT>
__global__ void __launch_bounds__(FT_THREADS, 1) gemm_f32_tc5_kernel(F32Tc5Args g, Trace tr) {
  using Z = FtSizes<BT>;
  TRACE_ENTRY(tr);
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long bar_s[2 * Z::STAGES + 4];
  __shared__ uint32_t tmem_s, dead_s;
  const uint32_t tiles = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_full = smem_u32(bar_s), bar_empty = bar_full + 8 * Z::STAGES;
  const uint32_t bar_dfull = bar_empty + 8 * Z::STAGES, bar_dempty = bar_dfull + 16;
  volatile uint32_t* dead = &dead_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();
  if (warp == FT_SUM) {
    if (lane == 0) {
      dead_s = 0;
      for (int s = 0; s < Z::STAGES; s++) {
        mbar_init(bar_full + 8 * s, FT_SPLIT);
        mbar_init(bar_empty + 8 * s, 1);
      }
      for (int b = 0; b < 2; b++) {
        mbar_init(bar_dfull + 8 * b, 1);
        mbar_init(bar_dempty + 8 * b, FT_SUM);
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"((uint32_t)(2 * Z::ACC))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_s;
  const int units = g.n_tiles * g.m_tiles * g.S;
  // unit u: the k slices of a tile and the token tiles of a weight tile run next to each other
  auto unit = [&](int u, int& n0, int& m0, int& split, int& k0, int& k1) {
    split = u % g.S;
    const int r = u / g.S;
    m0 = (r % g.m_tiles) * BT;
    n0 = (r / g.m_tiles) * TC_BN;
    k0 = split * g.kc;
    k1 = min(g.K, k0 + g.kc);
  };

  if (warp >= FT_SUM + 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FT_REGS_SPLIT));
    // ---- splitters: thread (rows r0 + 64 i, piece q of 8 k) of the weight tile, then of the token tile; the pieces of
    // the next stage are fetched as soon as this stage's are split
    const int ct = threadIdx.x - 32 * (FT_SUM + 4);
    const int q = ct & 7, r0 = ct >> 3;
    constexpr int NW = TC_BN / 64, NA = (BT + 63) / 64;
    F8 w[NW], a[NA];
    auto fetch_w = [&](int n0, int k, int k1) {
      const int n = n0 + r0;
      const float* p = g.W + (size_t)n * g.K + k + 8 * q;
      const bool in = k + 8 * q < k1;
#pragma unroll
      for (int i = 0; i < NW; i++) w[i] = in && n + 64 * i < g.N ? ld_piece(p + (size_t)(64 * i) * g.K) : F8{};
    };
    auto fetch_a = [&](int m0, int k, int k1) {
      const int m = m0 + r0;
      const float* p = g.A + (size_t)m * g.lda + k + 8 * q;
      const bool in = k + 8 * q < k1 && (BT >= 64 || r0 < BT);
#pragma unroll
      for (int i = 0; i < NA; i++) a[i] = in && m + 64 * i < g.M ? ld_piece(p + (size_t)(64 * i) * g.lda) : F8{};
    };
    const uint32_t at0 = (uint32_t)(r0 * 128) + (((q ^ r0) & 7) << 4);  // 64 rows on: 8192 bytes on, the same swizzle
    auto put = [&](const F8& v, uint32_t at, uint32_t part) {
      uint32_t h[4], m[4], l[4];
#pragma unroll
      for (int e = 0; e < 4; e++) split2(v.v[e], h[e], m[e], l[e]);
      st_shared_v4(at, h);
      st_shared_v4(at + part, m);
      st_shared_v4(at + 2 * part, l);
    };
    int u = blockIdx.x, n0, m0, split, k, k1, i = 0;
    unit(u, n0, m0, split, k, k1);
    if (!g.late) fetch_w(n0, k, k1);  // weights don't change: before the kernel in front is done
    pdl_wait();
    if (g.late) fetch_w(n0, k, k1);
    fetch_a(m0, k, k1);
    for (;; i++) {
      k += TC_BK;  // the next stage
      if (k >= k1) {
        u += gridDim.x;
        if (u < units) unit(u, n0, m0, split, k, k1);
      }
      const int s = i % Z::STAGES;
      if (!wait_limited(bar_empty + 8 * s, ((i / Z::STAGES) & 1) ^ 1, dead, g.flag)) break;
      const uint32_t base = tiles + s * Z::STAGE + at0;
#pragma unroll
      for (int j = 0; j < NW; j++) put(w[j], base + 8192 * j, Z::W_PART);
      if (u < units) fetch_w(n0, k, k1);
#pragma unroll
      for (int j = 0; j < NA; j++)
        if (BT >= 64 || r0 < BT) put(a[j], base + 3 * Z::W_PART + 8192 * j, Z::A_PART);
      if (u < units) fetch_a(m0, k, k1);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_full + 8 * s);
      if (u >= units) break;
    }
  } else if (warp >= FT_SUM) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FT_REGS_MMA));
    // ---- MMAs: fp32 accumulate, bf16 x bf16, both K-major, M = 128, N = BT
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BT >> 3) << 17) | ((uint32_t)(TC_BN >> 4) << 24);
    pdl_wait();  // (the limit of the waits counts from the dependency, not from this CTA's start)
    int i = 0;
    bool ok = true;
    for (int u = blockIdx.x; warp == FT_SUM && ok && u < units; u += gridDim.x) {
      int n0, m0, split, k0, k1;
      unit(u, n0, m0, split, k0, k1);
      for (int k = k0; k < k1; k += TC_BK, i++) {
        const int s = i % Z::STAGES, b = i & 1;
        if (!(ok = wait_limited(bar_dempty + 8 * b, ((i >> 1) & 1) ^ 1, dead, g.flag))) break;
        if (!(ok = wait_limited(bar_full + 8 * s, (i / Z::STAGES) & 1, dead, g.flag))) break;
        tc_fence_after();
        const uint32_t wt = tiles + s * Z::STAGE, acc = tmem + b * Z::ACC;
        const uint64_t wh = make_smem_desc(wt), wm = make_smem_desc(wt + Z::W_PART), wl = make_smem_desc(wt + 2 * Z::W_PART);
        const uint32_t at = wt + 3 * Z::W_PART;
        const uint64_t ah = make_smem_desc(at), am = make_smem_desc(at + Z::A_PART), al = make_smem_desc(at + 2 * Z::A_PART);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < TC_BK / 16; kk++) {
            tc_mma_bf16(acc, wh + 2 * kk, ah + 2 * kk, IDESC, kk != 0);
            tc_mma_bf16(acc + BT, wh + 2 * kk, am + 2 * kk, IDESC, kk != 0);
            tc_mma_bf16(acc + BT, wm + 2 * kk, ah + 2 * kk, IDESC, 1);
            tc_mma_bf16(acc + BT, wh + 2 * kk, al + 2 * kk, IDESC, 1);
            tc_mma_bf16(acc + BT, wm + 2 * kk, am + 2 * kk, IDESC, 1);
            tc_mma_bf16(acc + BT, wl + 2 * kk, ah + 2 * kk, IDESC, 1);
          }
          tc_commit(bar_empty + 8 * s);
          tc_commit(bar_dfull + 8 * b);
        }
        __syncwarp();
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FT_REGS_SUM));
    // ---- sums of the stages: thread = weight row n, half of the tokens
    constexpr int NC = Z::NC;
    const int qr = warp & 3, c0 = (warp >> 2) * NC;
    pdl_wait();
    int i = 0;
    bool ok = true;
    for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
      int n0, m0, split, k0, k1;
      unit(u, n0, m0, split, k0, k1);
      float sum[NC];
#pragma unroll
      for (int c = 0; c < NC; c++) sum[c] = 0.f;
      for (int k = k0; k < k1; k += TC_BK, i++) {
        const int b = i & 1;
        if (!(ok = wait_limited(bar_dfull + 8 * b, (i >> 1) & 1, dead, g.flag))) break;
        tc_fence_after();
        const uint32_t acc = tmem + ((uint32_t)(qr * 32) << 16) + b * Z::ACC + c0;
#pragma unroll
        for (int c = 0; c < NC; c += 8) {
          uint32_t x[8], y[8];
          tmem_ld_32x8_nowait(acc + c, x);
          tmem_ld_32x8_nowait(acc + BT + c, y);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 8; e++)
            sum[c + e] += __uint_as_float(x[e]) + __uint_as_float(y[e]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_dempty + 8 * b);
      }
      if (!warps_agree<32 * FT_SUM>(ok)) break;
      const int n = n0 + qr * 32 + lane;
      float* out = g.out + (size_t)split * g.split_stride + (size_t)(m0 + c0) * g.ldo;
      // through shared memory, a row of 128 columns per store: short code (what a launch runs once, it also fetches once)
      float* stage = reinterpret_cast<float*>(smem_raw + (tiles - smem_u32(smem_raw)) + Z::STAGES * Z::STAGE) + (warp >> 2) * (Z::CHUNK * TC_BN);
#pragma unroll
      for (int cc = 0; cc < NC; cc += Z::CHUNK) {
        named_bar(2 + (warp >> 2), 128);  // the chunk before is out
#pragma unroll
        for (int c = 0; c < Z::CHUNK; c++) stage[c * TC_BN + qr * 32 + lane] = g.alpha * sum[cc + c];
        uint32_t odd = 0;  // of the chunk's tokens, those whose result is not finite
#pragma unroll
        for (int c = 0; c < Z::CHUNK; c++) odd |= (uint32_t)(fabsf(sum[cc + c]) < INFINITY ? 0 : 1) << c;
        // (rows past M or N count for nothing: their zeros turn into NaN where the other operand has one)
        const int valid = n < g.N ? min(Z::CHUNK, g.M - m0 - c0 - cc) : 0;
        if (valid < Z::CHUNK) odd &= valid > 0 ? (1u << valid) - 1 : 0u;
        for (unsigned lanes; (lanes = __ballot_sync(0xffffffffu, odd != 0)) != 0;) {
          const int who = __ffs(lanes) - 1, c = __ffs(__shfl_sync(0xffffffffu, odd, who)) - 1;
          const float v = g.alpha * warp_dot(g.A + (size_t)(m0 + c0 + cc + c) * g.lda, g.W + (size_t)__shfl_sync(0xffffffffu, n, who) * g.K, k0, k1, lane);
          if (lane == who) {
            stage[c * TC_BN + qr * 32 + lane] = v;
            odd &= odd - 1;
          }
        }
        named_bar(2 + (warp >> 2), 128);
        const int nn = n0 + 4 * lane, rows = min(Z::CHUNK, g.M - m0 - c0 - cc);
#pragma unroll 2
        for (int c = qr; c < rows; c += 4) {
          const float4 v = *reinterpret_cast<const float4*>(stage + c * TC_BN + 4 * lane);
          float* o = out + (size_t)(cc + c) * g.ldo + nn;
          if (g.wide && nn + 3 < g.N) {
            *reinterpret_cast<float4*>(o) = v;
          } else {
            if (nn < g.N) o[0] = v.x;
            if (nn + 1 < g.N) o[1] = v.y;
            if (nn + 2 < g.N) o[2] = v.z;
            if (nn + 3 < g.N) o[3] = v.w;
          }
        }
      }
    }
  }
  __syncwarp();
  if (*dead) {  // a wait ran out: the MMAs in flight retire before the shared memory is given up
    const unsigned long long t0 = gtime();
    while (gtime() - t0 < TC_DRAIN_NS) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  TRACE_EXIT(tr);
  if (warp == FT_SUM)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(2 * Z::ACC)) : "memory");
}

template <int BT>
static cudaError_t launch_f32_tc5(cudaStream_t st, const F32Tc5Args& a, int ctas) {
  using Z = FtSizes<BT>;
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc5_kernel<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Z::SMEM);
  if (e != cudaSuccess) return e;
  return launch_k(gemm_f32_tc5_kernel<BT>, dim3(ctas), dim3(FT_THREADS), Z::SMEM, st, a, next_trace(49));
}

// From 17 rows on, and from 33 where the weights are small: below, the SIMT tiles are the faster ones (a stage costs the
// same with any number of rows).  Alone with a cold L2, us, SIMT / this kernel, N x K:
//   rows   768 x 768    2304 x 768   768 x 3072   8192 x 2048     rows   768 x 768    2304 x 768   768 x 3072   8192 x 2048
//     16    9.8 / 12.1   12.0 / 12.5  14.5 / 16.7  33.7 / 32.1     100   13.4 / 14.2  20.5 / 14.4  31.1 / 22.4   108 / 39
//     32   11.2 / 12.2   14.0 / 12.6  19.1 / 16.7  40.4 / 32.7     300   35.7 / 23.7  54.7 / 24.7   120 / 63     294 / 109
//     64   13.2 / 12.4   15.9 / 13.3  22.0 / 18.5  60.9 / 35.5    2048   75.4 / 30.0   179 / 52     275 / 83    1548 / 366
// K below 256 leaves nothing to split: 300 x 64 x 64 9.4 / 10.3.
bool gemm_f32_tc5_takes(const GemmArgs& g) {
  return g.adt == DT_F32 && g.wdt == DT_F32 && g.wait_flag && !g.tile_expert && !g.a_rows && (g.K % 8) == 0 && (g.lda % 8) == 0 &&
         (((uintptr_t)g.A | (uintptr_t)g.W) & 31) == 0;  // 32-byte loads
}
bool gemm_f32_tc5_fits(const GemmArgs& g) {
  return gemm_f32_tc5_takes(g) && g.K >= 256 && (g.M > 32 || (g.M > 16 && (size_t)g.N * g.K >= (size_t)1 << 20));
}

// Token tile and slices (up to the eight that a consumer sums with one batch of loads, as many as the buffer has room
// for) by what the fullest CTA takes, in us: a stage costs 1.0 / 1.2 / 1.55 with 32 / 64 / 128 rows, the first pieces and
// the last results of a launch 4 / 4 / 6, and a consumer reads every slice (0.3).
cudaError_t launch_gemm_f32_tc5(cudaStream_t st, GemmArgs& g) {
  F32Tc5Args a{};
  a.A = (const float*)g.A; a.W = (const float*)g.W; a.lda = g.lda; a.M = g.M; a.N = g.N; a.K = g.K;
  a.out = g.out; a.ldo = g.ldo; a.split_stride = g.split_stride; a.alpha = g.alpha; a.flag = g.wait_flag; a.late = g.w_late;
  a.wide = (((uintptr_t)g.out | (uintptr_t)(g.ldo * 4) | (uintptr_t)(g.split_stride * 4)) & 15) == 0;
  a.n_tiles = ceil_div(g.N, TC_BN);
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int steps = ceil_div(g.K, TC_BK);
  int bt = 0, S = 1;
  double best = 1e30;
  for (int b = g.M > 32 ? 64 : 32; b <= 128 && (b < 64 || b / 2 < g.M); b *= 2)
    for (int s = 1; s <= 8 && s <= steps && (s == 1 || (size_t)s * g.split_stride <= g.out_capacity); s++) {
      const int per = ceil_div(steps, s), rounds = ceil_div(a.n_tiles * ceil_div(g.M, b) * ceil_div(steps, per), sms);
      const double cost = rounds * per * (b == 128 ? 1.55 : b == 64 ? 1.2 : 1.0) + (b == 128 ? 6 : 4) + 0.3 * (rounds + s);
      if (cost < best) {
        best = cost;
        bt = b;
        S = s;
      }
    }
  a.m_tiles = ceil_div(g.M, bt);
  a.kc = ceil_div(steps, S) * TC_BK;
  g.S = a.S = ceil_div(g.K, a.kc);
  const int ctas = std::min(a.n_tiles * a.m_tiles * a.S, sms);
  return bt == 128 ? launch_f32_tc5<128>(st, a, ctas) : bt == 64 ? launch_f32_tc5<64>(st, a, ctas) : launch_f32_tc5<32>(st, a, ctas);
}

}  // namespace nvllm
