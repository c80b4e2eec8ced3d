// gemm_tc5.cuh — what the tcgen05 GEMM kernels share: the one-CTA kernel of gemm_tcgen05.cu, the CTA-pair
// kernel of gemm_tc5_pair.cu and the fp32 kernel of gemm_f32_tc5.cu.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"
#include "tc5.cuh"
#include "tma.cuh"

namespace nvllm {

constexpr int TC_BN = 128;  // weight rows per CTA (UMMA M)
constexpr int TC_BK = 64;   // k elements per stage = one 128-byte swizzle row of bf16
constexpr int TC_THREADS = 192;
// k-blocks that a stage of the one-CTA kernel's ring holds (one wait each for producer and MMAs)
__host__ __device__ constexpr int tc5_stage_blocks(int BT) { return BT <= 128 ? 2 : 1; }

// The work of a launch: units (token tile, weight tile, k split) dealt out round-robin.
struct Tc5Sched {
  int units, n_tiles, S, kbps, nkb_total;
  // grouped (mixture-of-experts) mode, g_expert != nullptr: token tile t covers rows
  // [g_row0[t], g_row0[t] + g_rows[t]) of the expert-sorted activations and multiplies expert
  // g_expert[t]'s [g_N, K] weight matrix (experts stacked row-wise in W); the tile list lives
  // on the device (moe_sort_kernel), so units = *g_ntiles * n_tiles is read after the wait
  const int* g_expert;
  const int* g_row0;
  const int* g_rows;
  const int* g_ntiles;
  int g_N;
  // decode-sized grouped GEMMs: raw weight base / bytes per weight row / expert count for the
  // speculative L2 prefetch before the dependency resolves (null = off)
  const uint8_t* g_wbase;
  int g_row_bytes, g_E;
};
// the RMSNorm-fold arguments of Tc5Args (kernels.h), as the kernel takes them
struct Tc5Fuse {
  const float* rs_ssq;
  int rs_parts, rs_ld;
  float rs_inv_h, rs_eps;
  float* x;
  bf16* xb;
  float* ssq;
  int ssq_ld;
  const float* bias;
  float m;
  const float* g;  // weight of the norm that reads x next: xb = bf16(x * g); null = ones
  int cl;          // > 1: the S k-splits of an output tile are one thread-block cluster of `cl` CTAs
  float glu_limit; // != 0: the gated epilogue computes another unit than silu(g) u (common.cuh glu_unit)
};
__device__ __forceinline__ void named_bar(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
// thread-block cluster primitives (the fused-residual split-K epilogue)
__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_release() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait_acquire() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// v[c] of every lane -> lane l gets sum over lanes of v[l]  (31 shuffles instead of 32 x 5)
__device__ __forceinline__ float warp_transpose_sum(float (&v)[32], int lane) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < off; i++) {
      const float send = up ? v[i] : v[i + off];
      const float keep = up ? v[i + off] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  return v[0];
}
// ---- bounded waits: a kernel whose wait ran out raises its caller's flag, lets its copies land and returns
constexpr unsigned long long TC_WAIT_NS = 2000000000ull, TC_DRAIN_NS = 20000000ull;
// whole warp; false when the wait ran out (here or anywhere in the CTA)
__device__ __forceinline__ bool wait_limited(uint32_t bar, uint32_t parity, volatile uint32_t* dead, int* flag) {
#pragma unroll 1
  for (int i = 0; i < 64; i++)
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const unsigned long long t0 = gtime();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; i++)
      if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    const bool over = *dead != 0 || gtime() - t0 > TC_WAIT_NS;
    if (__any_sync(0xffffffffu, over)) {
      *dead = 1;
      if (flag) *reinterpret_cast<volatile int*>(flag) = 1;
      return false;
    }
  }
}
// the same for short paths: a wait that need not wait costs little more than the test
__device__ __forceinline__ bool wait_short(uint32_t bar, uint32_t parity, volatile uint32_t* dead, int* flag) {
  return __all_sync(0xffffffffu, mbar_try_wait(bar, parity)) || wait_limited(bar, parity, dead, flag);
}
// the N threads of the epilogue warps go on together or not at all (they share barriers further on)
template <int N>
__device__ __forceinline__ bool warps_agree(bool ok) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, 4, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all)
      : "r"((uint32_t)ok), "n"(N)
      : "memory");
  return all != 0;
}
// rot: CTAs working on the same k range start at different k-blocks (and wrap), so that at any
// instant they pull DIFFERENT activation tiles out of L2 — otherwise every CTA of a skinny
// GEMM requests the same 8 KB A tile at the same time and the few L2 slices holding it pace
// the whole kernel (measured: ~390 ns per k-block with W already in shared memory).
struct Tc5Unit {
  int n0;     // first output column (weight row inside the expert)
  int wrow;   // first weight row in the stacked weight tensor (TMA coordinate)
  int m0;     // first token row
  int m_end;  // one past the last valid token row of this tile
  int kb0, nkb, split, rot;
};
__device__ __forceinline__ Tc5Unit tc5_unit(const Tc5Sched& sc, int u, int BT, int M) {
  Tc5Unit t;
  t.split = u % sc.S;
  const int r = u / sc.S;
  const int nt = r % sc.n_tiles, mt = r / sc.n_tiles;
  t.n0 = nt * TC_BN;
  if (sc.g_expert) {
    t.m0 = sc.g_row0[mt];
    t.m_end = t.m0 + sc.g_rows[mt];
    t.wrow = sc.g_expert[mt] * sc.g_N + t.n0;
  } else {
    t.m0 = mt * BT;
    t.m_end = M;
    t.wrow = t.n0;
  }
  t.kb0 = t.split * sc.kbps;
  t.nkb = min(sc.kbps, sc.nkb_total - t.kb0);
  t.rot = (nt + 5 * mt) % t.nkb;
  return t;
}
__device__ __forceinline__ int tc5_kb(int kb0, int kb, int rot, int nkb) {
  const int k = kb + rot;
  return kb0 + (k >= nkb ? k - nkb : k);
}

}  // namespace nvllm
