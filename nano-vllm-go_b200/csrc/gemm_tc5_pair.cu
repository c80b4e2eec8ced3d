// gemm_tc5_pair.cu — the tcgen05 GEMM for many token rows: two CTAs of a cluster work on one output tile
// (cta_group::2) of 256 weight rows x 256 token rows.
//
// The one-CTA kernel (gemm_tcgen05.cu) loads 128 weight rows and 256 token rows for every 128 x 256 product; at full
// tensor rate its 148 CTAs would draw 96 bytes per clock and SM out of L2, more than L2 delivers, and that is
// what bounds it once a step has more than a few hundred rows.  Here each CTA of a pair loads its own 128 weight rows
// and 128 of the 256 token rows, the tensor cores of both read both halves of the token tile, and the draw
// is 64 bytes per clock and SM.  The stage shrinks from 48 to 32 KB, so six fit where four did.
//
// Roles per CTA: warp 0 loads (TMA; both CTAs' loads report to the leader's barrier), warp 1 of the leader issues
// the MMAs for both, warps 2-9 read their own CTA's accumulator (128 weight rows x 256 tokens in TMEM,
// double-buffered; two warps take the 32-token chunks of a quarter of the rows in turn) and apply the epilogue under
// the next tile's MMAs.  The residual epilogue fetches the rows of x that
// a chunk updates one chunk ahead.
//
// Measured inside whole steps, TFLOP/s of all products against the one-CTA kernel: Llama-3.2-1B layers, 64 prompts of 256
// to 512 tokens 1078 -> 1383; Llama-3.2-3B layers, 7936 rows 1207 -> 1352; Falcon-7B layers, 2048 rows 1278 -> 1386;
// squared-ReLU layers of 2048 x 12288, 18 k rows 1345 -> 1518; routed experts of 1024 x 512, 150 k rows 783 -> 953, and
// 975 with their second product (512 of k) on the one-CTA kernel, where it is now.  With
// four epilogue warps instead of eight the first five were 1200, 1292, 1331, 1280 and 781: at 1024 to 2048 of k a tile's
// epilogue took longer than its products.  What bounds it now is the clock under the power limit (tensor pipe 92 %
// busy at 1.3 GHz in the widest product) and, below 2048 of k, the epilogue.
//
// The waits of the loading, MMA and epilogue loops have a limit: past it the kernel sets its launch's flag in host memory
// (WaitFlag), leaves its loops, gives the copies in flight time to land, frees its tensor memory and returns; the host
// reports the step as failed.
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "gemm_tc5.cuh"
#include "kernels.h"

namespace nvllm {

constexpr int PR_BT = 256;                               // token rows of a pair's tile
constexpr int PR_STAGES = 6;
constexpr uint32_t PR_W_BYTES = TC_BN * TC_BK * 2;       // of one CTA: its 128 weight rows
constexpr uint32_t PR_A_BYTES = (PR_BT / 2) * TC_BK * 2; // and its half of the token rows
constexpr uint32_t PR_STAGE_BYTES = PR_W_BYTES + PR_A_BYTES;
constexpr int PR_EPI = 8, PR_THREADS = 64 + 32 * PR_EPI; // epilogue warps: two for each 32 lanes of tensor memory
constexpr int HEADS_TOKENS = 16, HEADS_PITCH = TC_BN + 4;
constexpr size_t PR_SMEM = (size_t)PR_STAGES * PR_STAGE_BYTES + 1024 + 16 * PR_STAGES + 64;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// a load of this CTA's tile that reports to the barrier of the pair's leader (peer bit of the address cleared)
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const void* map, uint32_t bar, int c0, int c1, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(dst), "l"(map), "r"(bar & 0xFEFFFFFFu), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the MMAs issued so far arrive on this barrier of both CTAs when they have retired
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void arrive_at(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// unit u of the pair: tc5_unit with weight tiles of 256 rows, this CTA's half of them
__device__ __forceinline__ Tc5Unit pair_unit(const Tc5Sched& sc, int u, int M, int rank) {
  Tc5Unit t;
  const int nt = u % sc.n_tiles, mt = u / sc.n_tiles;
  t.split = 0;
  t.n0 = nt * 2 * TC_BN + rank * TC_BN;
  if (sc.g_expert) {
    t.m0 = sc.g_row0[mt];
    t.m_end = t.m0 + sc.g_rows[mt];
    t.wrow = sc.g_expert[mt] * sc.g_N + t.n0;
  } else {
    t.m0 = mt * PR_BT;
    t.m_end = M;
    t.wrow = t.n0;
  }
  t.kb0 = 0;
  t.nkb = sc.nkb_total;
  t.rot = (nt + 5 * mt) % t.nkb;
  return t;
}

__global__ void __launch_bounds__(PR_THREADS, 1)
gemm_tc5_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA, int M, int N, Tc5Sched sc,
                     float* __restrict__ out, int ldo, float alpha, int w_reused, int epi, bf16* __restrict__ epi_out,
                     int epi_ld, const float* __restrict__ epi_bias, Tc5Fuse fz, Tc5Heads hs, int* flag, Trace tr) {
  const unsigned long long t_entry = trace_on(tr) ? gtime() : 0ull;
  unsigned long long t_wait = 0;
  __shared__ __align__(16) union {
    uint8_t act[PR_EPI][32 * 48];
    float heads[2][HEADS_TOKENS][HEADS_PITCH];
  } epi_stage;
  __shared__ int pos_s[2][PR_BT], slot_s[2][PR_BT];
  __shared__ float rstd_s[2][PR_BT];
  __shared__ float ssq_s[2][2][4][32];  // [half][chunk parity]
  __shared__ uint32_t dead_s;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t tiles = (smem_u32(smem_raw) + 1023u) & ~1023u;  // SWIZZLE_128B needs 1024 B
  const uint32_t bars = tiles + PR_STAGES * PR_STAGE_BYTES;
  // full[s] at bars + 8 s (the leader's counts both CTAs' bytes), empty[s] behind them, tmem_full[2], tmem_empty[2]
  const uint32_t bar_tfull = bars + 16 * PR_STAGES;
  const uint32_t bar_tempty = bar_tfull + 16;
  const uint32_t tmem_slot = bar_tempty + 16;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  volatile uint32_t* dead = &dead_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const bool grouped = sc.g_expert != nullptr;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  pdl_launch_dependents();

  if (warp == 0 && lane == 0) {
    dead_s = 0;
    for (int s = 0; s < PR_STAGES; s++) {
      mbar_init(bars + 8 * s, 1);
      mbar_init(bars + 8 * (PR_STAGES + s), 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(bar_tfull + 8 * b, 1);
      mbar_init(bar_tempty + 8 * b, 2 * PR_EPI);  // one arrival per epilogue warp of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmW) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"((uint32_t)(2 * PR_BT))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive_release();  // the peer's barriers are initialised and its tensor memory is allocated
  cluster_wait_acquire();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;

  if (warp == 0) {
    uint64_t pol_w, pol_a;
    if (w_reused) asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_w));
    else asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_w));
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_a));
    // weight tiles of the first stages before the dependency resolves (a grouped GEMM learns its
    // experts from the previous kernel)
    int pre = 0;
    if (!grouped) {
      int u = pair, kb = 0;
      while (pre < PR_STAGES && u < sc.units) {
        const Tc5Unit t = pair_unit(sc, u, M, rank);
        const uint32_t full = bars + 8 * pre;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(full, 2 * PR_STAGE_BYTES);
          tma_load_pair(tiles + pre * PR_STAGE_BYTES, &tmW, full, tc5_kb(t.kb0, kb, t.rot, t.nkb) * TC_BK, t.wrow, pol_w);
        }
        __syncwarp();
        pre++;
        if (++kb == t.nkb) {
          kb = 0;
          u += pairs;
        }
      }
    }
    pdl_wait();
    if (trace_on(tr)) t_wait = gtime();
    const int units = grouped ? *sc.g_ntiles * sc.n_tiles : sc.units;
    int i = 0;
    bool ok = true;
    for (int u = pair; ok && u < units; u += pairs) {
      const Tc5Unit t = pair_unit(sc, u, M, rank);
      for (int kb = 0; kb < t.nkb; kb++, i++) {
        const int s = i % PR_STAGES;
        const uint32_t full = bars + 8 * s, dst = tiles + s * PR_STAGE_BYTES;
        const int k = tc5_kb(t.kb0, kb, t.rot, t.nkb) * TC_BK;
        const bool ahead = i < pre;
        if (!ahead && !(ok = wait_limited(bars + 8 * (PR_STAGES + s), ((i / PR_STAGES) & 1) ^ 1, dead, flag))) break;
        if (elect_one()) {
          if (!ahead) {
            if (rank == 0) mbar_expect_tx(full, 2 * PR_STAGE_BYTES);
            tma_load_pair(dst, &tmW, full, k, t.wrow, pol_w);
          }
          tma_load_pair(dst + PR_W_BYTES, &tmA, full, k, t.m0 + rank * (PR_BT / 2), pol_a);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // fp32 accumulate, bf16 x bf16, both K-major, N = 256, M = 256 over the two CTAs
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(PR_BT >> 3) << 17) |
                                 ((uint32_t)((2 * TC_BN) >> 4) << 24);
      // the tile list is the previous kernel's output; and the limit of the waits below counts from here, not from
      // this CTA's start: the kernels in front may take longer than it (an all-reduce waits up to 5 s for a late peer)
      pdl_wait();
      const int units = grouped ? *sc.g_ntiles * sc.n_tiles : sc.units;
      int i = 0, lu = 0;
      bool ok = true;
      for (int u = pair; ok && u < units; u += pairs, lu++) {
        const int buf = lu & 1;
        if (!(ok = wait_limited(bar_tempty + 8 * buf, ((lu >> 1) & 1) ^ 1, dead, flag))) break;  // both epilogues drained it
        tc_fence_after();
        const uint32_t tacc = tmem_base + (uint32_t)(buf * PR_BT);
        for (int kb = 0; kb < sc.nkb_total; kb++, i++) {
          const int s = i % PR_STAGES;
          if (!(ok = wait_limited(bars + 8 * s, (i / PR_STAGES) & 1, dead, flag))) break;
          tc_fence_after();
          const uint32_t wt = tiles + s * PR_STAGE_BYTES;
          const uint64_t wdesc = make_smem_desc(wt), adesc = make_smem_desc(wt + PR_W_BYTES);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < TC_BK / 16; kk++) mma_pair(tacc, wdesc + 2 * kk, adesc + 2 * kk, idesc, (kb | kk) != 0);
            commit_pair(bars + 8 * (PR_STAGES + s));
            if (kb == sc.nkb_total - 1) commit_pair(bar_tfull + 8 * buf);
          }
          __syncwarp();
        }
      }
    }
  } else {
    // epilogue: warp w may touch TMEM lanes [32 (w % 4), +32)
    const int q = warp & 3, half = (warp - 2) >> 2, et = threadIdx.x - 64;
    pdl_wait();
    const int units = grouped ? *sc.g_ntiles * sc.n_tiles : sc.units;
    int lu = 0;
    for (int u = pair; u < units; u += pairs, lu++) {
      const Tc5Unit t = pair_unit(sc, u, M, rank);
      const int n0 = t.n0, m0 = t.m0, Me = t.m_end, buf = lu & 1;
      const float* rs = nullptr;
      if (fz.rs_ssq) {
        // folded RMSNorm: 1 / sqrt(mean(x^2) + eps) per token row (tensor.go:211-224)
        float* w = rstd_s[buf];
        for (int c = et; c < PR_BT; c += 32 * PR_EPI) {
          const int mm = m0 + c;
          float ssum = 0.f;
          if (mm < Me) {
#pragma unroll 8
            for (int p = 0; p < fz.rs_parts; p++) ssum += __ldcg(fz.rs_ssq + (size_t)p * fz.rs_ld + mm);
          }
          w[c] = 1.0f / sqrtf(ssum * fz.rs_inv_h + fz.rs_eps);
        }
        if (!hs.hd) named_bar(1, 32 * PR_EPI);
        rs = w;
      }
      if (hs.hd) {
        for (int c = et; c < PR_BT && m0 + c < Me; c += 32 * PR_EPI) {
          pos_s[buf][c] = __ldcg(hs.positions + m0 + c);
          slot_s[buf][c] = __ldcg(hs.slots + m0 + c);
        }
        named_bar(1, 32 * PR_EPI);
      }
      const int n = n0 + q * 32 + lane;
      const bool n_ok = n < N;
      const uint32_t lanes = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * PR_BT);
      const bool resid = epi == TC5_EPI_RESID;
      float xv[32];  // RESID: the rows of x of the coming chunk
      auto fetch_x = [&](int c0) {
        const float* x = fz.x + (size_t)(m0 + c0) * N + n;
#pragma unroll
        for (int c = 0; c < 32; c++) xv[c] = n_ok && m0 + c0 + c < Me ? x[(size_t)c * N] : 0.f;
      };
      if (resid) fetch_x(32 * half);
      if (!warps_agree<256>(wait_limited(bar_tfull + 8 * buf, (lu >> 1) & 1, dead, flag))) break;
      tc_fence_after();
      auto load_acc = [&](int c0, uint32_t (&r)[32]) {
        __syncwarp();  // the load is the whole warp's: lanes past the last column have skipped the previous chunk's stores
        tmem_ld_32x32(lanes + (uint32_t)c0, r);
        if (rs) {
#pragma unroll
          for (int c = 0; c < 32; c++) r[c] = __float_as_uint(__uint_as_float(r[c]) * rs[c0 + c]);
        }
      };
      if (hs.hd) {
        // Query, key and value heads, instead of fp32 sums that a kernel of their own reads back: bias, rotation of the
        // halves of a head (rope.go), bf16; queries to epi_out, keys and values to their pages.  A head's halves are in the
        // accumulators of different warps, so 16 tokens at a time go through shared memory; there a thread takes eight
        // entries of either half of one token's head.  24.4 k rows of 32 + 16 heads of 64, K = 2048: 229 us and 151-169 for
        // the other kernel -> one product of 206; whole steps: Llama-3.2-1B layers, 64 prompts 11.58 -> 11.14 ms; 3B layers,
        // 4 k rows 3.93 -> 3.73; 18.7 k rows of 16 + 16 heads 5.17 -> 4.97.
        float (*stg)[HEADS_PITCH] = epi_stage.heads[half];
        const int tid = et & 127, tt = tid >> 3, g = tid & 7, hd = hs.hd, hh = hd == 64 ? g >> 2 : 0;
        const int j = hd == 64 ? (g & 3) * 8 : g * 8;      // entry of the half
        const int col = hh * 64 + j, swap = hh;            // (odd heads read their second 16 bytes first: other banks)
        const int head = (n0 + hh * 64) / hd;
        const bool is_v = head >= hs.nh + hs.nkv, live = head < hs.nh + 2 * hs.nkv;
        const bool rot = hs.cosT && !is_v && live;
        float ba[8], bb[8];
#pragma unroll
        for (int i = 0; i < 8; i++) ba[i] = bb[i] = 0.f;
        if (epi_bias && live) {
          load8(epi_bias + n0 + col, ba);
          load8(epi_bias + n0 + col + hd / 2, bb);
        }
        float cs[8], sn[8];
        auto fetch_rotation = [&](int c) {  // of the coming token
          if (rot && m0 + c < Me) {
            const size_t at = (size_t)pos_s[buf][c] * (hd / 2) + j;
            load8(hs.cosT + at, cs);
            load8(hs.sinT + at, sn);
          }
        };
        fetch_rotation(32 * half + tt);
#pragma unroll 1
        for (int c0 = 32 * half; c0 < PR_BT && m0 + c0 < Me; c0 += 64) {
          uint32_t r[32];
          load_acc(c0, r);
#pragma unroll
          for (int s = 0; s < 32; s += HEADS_TOKENS) {
#pragma unroll
            for (int c = 0; c < HEADS_TOKENS; c++) stg[c][q * 32 + lane] = alpha * __uint_as_float(r[s + c]);
            named_bar(2 + half, 128);
            const int c = c0 + s + tt, m = m0 + c;
            if (live && m < Me) {
              float a[8], b[8];
#pragma unroll
              for (int i = 0; i < 2; i++) {
                const int o = 4 * (i ^ swap);
                const float4 va = *reinterpret_cast<const float4*>(&stg[tt][col + o]);
                const float4 vb = *reinterpret_cast<const float4*>(&stg[tt][col + hd / 2 + o]);
                const int e = 4 * i;
                a[e] = va.x; a[e + 1] = va.y; a[e + 2] = va.z; a[e + 3] = va.w;
                b[e] = vb.x; b[e + 1] = vb.y; b[e + 2] = vb.z; b[e + 3] = vb.w;
              }
              if (swap) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                  const float ta = a[i], tb = b[i];
                  a[i] = a[i + 4]; a[i + 4] = ta;
                  b[i] = b[i + 4]; b[i + 4] = tb;
                }
              }
#pragma unroll
              for (int i = 0; i < 8; i++) {
                a[i] += ba[i];
                b[i] += bb[i];
              }
              if (rot) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                  const float ra = a[i] * cs[i] - b[i] * sn[i], rb = b[i] * cs[i] + a[i] * sn[i];
                  a[i] = ra;
                  b[i] = rb;
                }
              }
              bf16* dst;
              if (head < hs.nh) {
                dst = epi_out + (size_t)m * epi_ld + head * hd + j;
              } else {
                const int slot = slot_s[buf][c], kvh = head - hs.nh - (is_v ? hs.nkv : 0);
                dst = (is_v ? hs.vpool : hs.kpool) + (((size_t)(slot / KV_BLOCK) * hs.nkv + kvh) * KV_BLOCK + slot % KV_BLOCK) * hd + j;
              }
              store8(dst, a);
              store8(dst + hd / 2, b);
            }
            const int cn = s == 0 ? c + HEADS_TOKENS : c + 64 - HEADS_TOKENS;
            if (cn < PR_BT) fetch_rotation(cn);
            named_bar(2 + half, 128);
          }
        }
      } else if (epi == TC5_EPI_PARTIAL) {
#pragma unroll 1
        for (int c0 = 32 * half; c0 < PR_BT && m0 + c0 < Me; c0 += 64) {
          uint32_t r[32];
          load_acc(c0, r);
          if (!n_ok) continue;
          float* op = out + (size_t)(m0 + c0) * ldo + n;
          if (m0 + c0 + 32 <= Me) {
#pragma unroll
            for (int c = 0; c < 32; c++) op[(size_t)c * ldo] = alpha * __uint_as_float(r[c]);
          } else {
#pragma unroll
            for (int c = 0; c < 32; c++)
              if (m0 + c0 + c < Me) op[(size_t)c * ldo] = alpha * __uint_as_float(r[c]);
          }
        }
      } else if (epi == TC5_EPI_SWIGLU) {
        // interleaved gate / up rows (weights.cu): even lane = gate j, odd lane = up j; the pair splits the 32 tokens.
        // Staged per warp in shared memory ([32 tokens][16 columns], rows 48 B apart) for 16-byte stores.
        const int odd = lane & 1, pr = lane >> 1;
        uint8_t* stg = epi_stage.act[warp - 2];
        const int j0 = (n0 + q * 32) >> 1;
        // (a choice of the unit per token keeps a lane's sixteen from overlapping: 64 prompts of 384 through four layers of
        // routed experts 4.34 ms so, 4.23 with the choice outside; 64 of 512 through four Llama-1B layers 10.4 and 10.1, where
        // the runs of one side differ by as much)
        auto glu_rows = [&](auto unit) {
#pragma unroll 1
          for (int c0 = 32 * half; c0 < PR_BT && m0 + c0 < Me; c0 += 64) {
            uint32_t r[32];
            load_acc(c0, r);
#pragma unroll
            for (int c = 0; c < 16; c++) {
              const float mine = __uint_as_float(odd ? r[c + 16] : r[c]);
              const float send = __uint_as_float(odd ? r[c] : r[c + 16]);
              const float got = __shfl_xor_sync(0xffffffffu, send, 1);
              const float g = alpha * (odd ? got : mine), up = alpha * (odd ? mine : got);
              *reinterpret_cast<bf16*>(stg + (c + (odd ? 16 : 0)) * 48 + pr * 2) = __float2bfloat16_rn(unit(g, up));
            }
            __syncwarp();
            const int m = m0 + c0 + lane;
            if (m < Me) {
              bf16* orow = epi_out + (size_t)m * epi_ld + j0;
#pragma unroll
              for (int hh = 0; hh < 2; hh++)
                if (2 * (j0 + hh * 8) < N)
                  *reinterpret_cast<uint4*>(orow + hh * 8) = *reinterpret_cast<const uint4*>(stg + lane * 48 + hh * 16);
            }
            __syncwarp();
          }
        };
        if (fz.glu_limit == 0.f) glu_rows([](float g, float up) { return __fdividef(g, 1.0f + __expf(-g)) * up; });
        else glu_rows([&](float g, float up) { return glu_unit(g, up, fz.glu_limit); });
      } else if (resid) {
        // x = x + m * (proj + bias) (generic_model.go:359-365, 383-389), the row rounded to bf16 for the next folded
        // norm and its sum of squares over this CTA's columns
        const float b = (fz.bias && n_ok) ? fz.bias[n] : 0.f;
        const float gn = (fz.g && n_ok) ? fz.g[n] : 1.f;
        const int nt = n0 / TC_BN;
        int chunk = 0;
#pragma unroll 1
        for (int c0 = 32 * half; c0 < PR_BT && m0 + c0 < Me; c0 += 64, chunk++) {
          uint32_t r[32];
          load_acc(c0, r);
          float v[32];
#pragma unroll
          for (int c = 0; c < 32; c++) v[c] = xv[c] + fz.m * (alpha * __uint_as_float(r[c]) + b);
          if (c0 + 64 < PR_BT && m0 + c0 + 64 < Me) fetch_x(c0 + 64);
          const size_t base = (size_t)(m0 + c0) * N + n;
          if (n_ok && m0 + c0 + 32 <= Me) {
#pragma unroll
            for (int c = 0; c < 32; c++) {
              fz.x[base + (size_t)c * N] = v[c];
              fz.xb[base + (size_t)c * N] = __float2bfloat16_rn(v[c] * gn);
              v[c] *= v[c];
            }
          } else {
#pragma unroll
            for (int c = 0; c < 32; c++) {
              const bool in = n_ok && m0 + c0 + c < Me;
              if (in) {
                fz.x[base + (size_t)c * N] = v[c];
                fz.xb[base + (size_t)c * N] = __float2bfloat16_rn(v[c] * gn);
              }
              v[c] = in ? v[c] * v[c] : 0.f;
            }
          }
          const float tot = warp_transpose_sum(v, lane);  // token c0 + lane over this warp's 32 columns
          float (*sq)[32] = ssq_s[half][chunk & 1];
          sq[q][lane] = tot;
          named_bar(2 + half, 128);  // the four warps of this chunk
          if (q == 0 && n0 < N && m0 + c0 + lane < Me)
            fz.ssq[(size_t)nt * fz.ssq_ld + m0 + c0 + lane] =
                ((sq[0][lane] + sq[1][lane]) + sq[2][lane]) + sq[3][lane];
        }
      } else {
        // gelu_tanh(h + b1) (transformer.go:67-78), or relu(h)^2 for TC5_EPI_RELU2
        const float b = (epi_bias && n_ok) ? epi_bias[n] : 0.f;
#pragma unroll 1
        for (int c0 = 32 * half; c0 < PR_BT && m0 + c0 < Me; c0 += 64) {
          uint32_t r[32];
          load_acc(c0, r);
          bf16* op = epi_out + (size_t)(m0 + c0) * epi_ld + n;
          if (!n_ok) continue;
          if (epi == TC5_EPI_RELU2) {
#pragma unroll
            for (int c = 0; c < 32; c++) r[c] = __float_as_uint(relu2(alpha * __uint_as_float(r[c]) + b));
          } else {
#pragma unroll
            for (int c = 0; c < 32; c++) r[c] = __float_as_uint(gelu_tanh(alpha * __uint_as_float(r[c]) + b));
          }
          if (m0 + c0 + 32 <= Me) {
#pragma unroll
            for (int c = 0; c < 32; c++) op[(size_t)c * epi_ld] = __float2bfloat16_rn(__uint_as_float(r[c]));
          } else {
#pragma unroll
            for (int c = 0; c < 32; c++)
              if (m0 + c0 + c < Me) op[(size_t)c * epi_ld] = __float2bfloat16_rn(__uint_as_float(r[c]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_at(cluster_map(bar_tempty + 8 * buf, 0));
    }
  }
  __syncwarp();
  if (*dead) {  // a wait ran out: the copies in flight land before the shared memory is given up
    const unsigned long long t0 = gtime();
    while (gtime() - t0 < TC_DRAIN_NS) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive_release();  // the leader's MMAs read the peer's shared memory, the peer's warps arrive on the leader's barriers
  cluster_wait_acquire();
  if (threadIdx.x == 0 && trace_on(tr)) trace_rec(tr, t_entry, t_wait, (unsigned long long)epi);
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * PR_BT)) : "memory");
}

// ------------------------------------------------------------------ host side
namespace {
struct PairDevice {
  bool known = false;
  int pairs = 0;  // CTA pairs that are resident at once; 0: the kernel is not used on this device
  int sms = 0;
};
std::mutex g_pair_mu;
PairDevice g_pair_dev[64];
}  // namespace

cudaError_t WaitFlag::create() {
  cudaError_t e = cudaHostAlloc((void**)&host, sizeof(int), cudaHostAllocMapped);
  if (e != cudaSuccess) {
    host = nullptr;
    return e;
  }
  *host = 0;
  e = cudaHostGetDevicePointer((void**)&dev, host, 0);
  if (e != cudaSuccess) destroy();
  return e;
}
void WaitFlag::destroy() {
  if (host) cudaFreeHost(host);
  host = dev = nullptr;
}
void WaitFlag::raise() {
  if (host) __atomic_store_n(host, 1, __ATOMIC_RELEASE);
}
bool WaitFlag::take() { return host && __atomic_exchange_n(host, 0, __ATOMIC_ACQ_REL) != 0; }

// Once per device, outside any stream capture (handle creation): kernel attributes, resident pairs
int tc5_pair_init(int dev) {
  std::lock_guard<std::mutex> g(g_pair_mu);
  if (dev < 0 || dev >= 64) return 0;
  PairDevice& d = g_pair_dev[dev];
  if (d.known) return d.pairs;
  int n = 0;
  if (cudaFuncSetAttribute(gemm_tc5_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PR_SMEM) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(PR_THREADS);
    cfg.dynamicSmemBytes = PR_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_tc5_pair_kernel, &cfg) != cudaSuccess) n = 0;
  }
  if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 0;
  (void)cudaGetLastError();
  d.pairs = n;
  d.known = true;
  return n;
}
// Products of 256-row token tiles with one k range are taken over, where rounding the weight tiles up to 256 rows does not
// cost more rounds of the persistent schedule than the pair gains:
//  * epilogues that work on the accumulator (activation, residual, the row scales of a folded norm), for which the pair has
//    twice the warps, and attention projections, which save the launch that would rotate and place them: up to 1.15 times
//    the rounds.  All products of a step's layers with these on pairs against
//    not, 384 to 4544 wide, 520 to 20000 rows: activations 1.06 to 1.6 times as fast, residuals 1.0 to 1.08.  (With more
//    rounds they lose: Falcon-7B layers, 780 rows 627 us against 590, 2040 rows 1252 against 1220.)
//  * plain fp32 results: up to 1.1 times the rounds; from 768 of k on, a single round from 3072 of k on.  Time of the
//    one-CTA kernel over that of pairs, alone with a cold L2, 156 shapes:
//      k                        512        640        768        1024       2048       4096       8192
//      one round             .89- .93   .90- .94   .97-1.04   .92-1.00   .97-1.04     1.07
//      two                   .98-1.02   .99-1.00  1.01-1.03  1.00-1.07  1.02-1.09  1.09-1.10     1.15
//      three to seven        .92- .99   .93-1.05  1.00-1.06  1.01-1.08  1.05-1.09  1.06-1.09  1.10-1.15
//      13 rounds for 12      .96- .97                        1.06-1.09  1.04-1.05  1.04-1.06
//      8 for 7, 9 for 8      .94- .96                        1.03-1.06  1.00-1.04   .98-1.00     1.02
bool tc5_pair_fits(const Tc5Args& a, int bt, int S) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  const int pairs = g_pair_dev[dev].pairs, sms = g_pair_dev[dev].sms;
  if (pairs <= 0 || !a.wait_flag || bt != PR_BT || S != 1 || a.N <= TC_BN) return false;
  const long mt = a.g_experts > 0 ? a.M / PR_BT + a.g_experts : ceil_div(a.M, PR_BT);
  const long one = (mt * ceil_div(a.N, TC_BN) + sms - 1) / sms;
  const long two = (mt * ceil_div(a.N, 2 * TC_BN) + pairs - 1) / pairs;
  const bool plain = a.epi == TC5_EPI_PARTIAL && !a.rs_ssq && !a.heads;
  if (plain) return two * 10 <= one * 11 && a.K >= (one > 1 ? 768 : 3072);
  return two * 20 <= one * 23;
}

cudaError_t launch_gemm_tc5_pair(cudaStream_t st, const Tc5Args& a, const TmaDesc* tw, const TmaDesc* ta) {
  int dev = 0;
  cudaGetDevice(&dev);
  const int pairs = g_pair_dev[dev].pairs;
  if (pairs <= 0 || !a.wait_flag) return cudaErrorInvalidValue;
  if (a.heads && (a.epi != TC5_EPI_PARTIAL || !a.epi_out || a.g_experts > 0 || (a.heads->hd != 64 && a.heads->hd != 128))) return cudaErrorInvalidValue;
  if (a.epi == TC5_EPI_RESID && (!a.res_x || !a.res_xb || !a.res_ssq || a.g_experts > 0)) return cudaErrorInvalidValue;
  Tc5Sched sc{};
  sc.nkb_total = sc.kbps = ceil_div(a.K, TC_BK);
  sc.S = 1;
  sc.n_tiles = ceil_div(a.N, 2 * TC_BN);
  int m_tiles = ceil_div(a.M, PR_BT);
  if (a.g_experts > 0) {
    sc.g_expert = a.g_tile_expert;
    sc.g_row0 = a.g_tile_row0;
    sc.g_rows = a.g_tile_rows;
    sc.g_ntiles = a.g_n_tiles;
    sc.g_N = a.N;
    m_tiles = min(a.g_max_tiles, a.M / PR_BT + a.g_experts);  // upper bound; the kernel reads the count
  }
  sc.units = sc.n_tiles * m_tiles;
  int n = min(sc.units, pairs);
  if (a.max_ctas > 0 && a.epi != TC5_EPI_RESID) n = max(1, min(n, a.max_ctas / 2));
  const bool w_reused = a.g_experts > 0 ? a.M > 2 * PR_BT * a.g_experts : m_tiles > 1;
  const Tc5Fuse fz{a.rs_ssq, a.rs_parts, a.rs_ld, a.rs_inv_h, a.rs_eps, a.res_x, (bf16*)a.res_xb, a.res_ssq,
                   a.res_ssq_ld, a.res_bias, a.res_m, a.res_g, 0, a.glu_limit};
  return launch_k_cluster(gemm_tc5_pair_kernel, dim3(2 * n), dim3(PR_THREADS), PR_SMEM, st, 2,
                          *reinterpret_cast<const CUtensorMap*>(tw), *reinterpret_cast<const CUtensorMap*>(ta), a.M, a.N, sc,
                          a.out, a.ldo, a.alpha, w_reused ? 1 : 0, a.epi, (bf16*)a.epi_out, a.epi_ld, a.epi_bias, fz,
                          a.heads ? *a.heads : Tc5Heads{}, a.wait_flag,
                          next_trace(46));
}

}  // namespace nvllm
