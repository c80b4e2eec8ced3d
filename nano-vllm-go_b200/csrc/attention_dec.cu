// attention_dec.cu — bf16 paged decode attention for small query-head groups
// (G = n_heads / n_kv_heads <= 8: GPT-2 MHA, Llama / Granite GQA), sm_100a.
//
// Same semantics as attention_mma.cu's decode kernel (reference attention.go:354-421: scores =
// (q.k)*scale, keys after the query masked, softmax, P.V; q head h uses kv head h / G) and the
// same fused prologue (split-K sum of the QKV GEMM partials + bias, rotate_half RoPE
// rope.go:153-205, K/V append through the block table).  What differs is how the stream is fed
// and which way round the MMAs sit — the decode step's attention is a pure HBM stream and the
// older kernel was issue-bound at ~900 instructions per warp per 128-key tile:
//
//  * K/V tiles arrive by TMA (one elected lane of a dedicated producer warp issues 2*HD/64
//    bulk tensor copies per tile, SWIZZLE_128B, completion on an mbarrier) — no per-thread
//    cp.async address arithmetic; the consumer warps never issue a load.  full/empty mbarrier
//    ring, no __syncthreads per tile, so the four consumer warps drift freely.
//  * "keys are the M rows": S^T[key][head] = K[key][d] . Q^T[d][head] with the K tile as the
//    ldmatrix-fed A operand and the (<= 8, zero-padded) query heads as the 8 columns of the
//    m16n8k16 B operand held in registers; O^T[d][head] = V^T[d][key] . P^T[key][head] with V
//    through ldmatrix.trans and P^T turned from accumulator layout into a B fragment by
//    movmatrix.  Per 16 keys x 64 dims: 4 + 4 ldmatrix.x4, 4 + 4 mma, 2 movmatrix — a 16-row
//    query tile with 4 real rows would need twice the MMAs and 4x the accumulator registers.
//  * the row maximum is a 3-shuffle reduction over the 8 key lanes; row sums stay per-thread
//    partials until the head is finished.
#include <stdlib.h>

#include "common.cuh"
#include "kernels.h"
#include "mma.cuh"
#include "tma.cuh"

namespace nvllm {

constexpr int DT_CONSUMERS = 4;                       // consumer warps
constexpr int DT_THREADS = (DT_CONSUMERS + 1) * 32;   // + the TMA producer warp

__device__ __forceinline__ void consumer_bar() {
  asm volatile("bar.sync 1, %0;" ::"n"(DT_CONSUMERS * 32) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
// 16-byte chunk c of key row r in a TMA-written tile: HD/64 panels of [BN][128 B], SWIZZLE_128B
template <int BN>
__device__ __forceinline__ uint32_t tile_off_t(int r, int c) {
  return (uint32_t)((c >> 3) * (BN * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}

template <int HD>
struct DecSmem {
  static constexpr int QROW = HD * 2 + 16;  // padded query row: conflict-free 32-bit reads
  static constexpr int Q_BYTES = 8 * QROW;  // per packed kv head
  static constexpr int RS = HD + 2;
  static constexpr int RED_BYTES = DT_CONSUMERS * 8 * RS * 4;
};

// KPC = kv heads per CTA (1, 2, 4).  The four consumer warps split into KPC groups of
// WPH = 4 / KPC warps; group i owns head i of the CTA for the whole kernel, its warps split each
// 64-key tile of that head between them.  The tiles of the KPC heads are interleaved in the
// ring, so the groups stream concurrently and never wait for each other: no CTA-wide barrier
// after the prologue, a WPH-warp merge per head (none at all for KPC = 4).
template <int HD, int BN, int STAGES, int KPC>
__global__ void __launch_bounds__(DT_THREADS, (HD == 64 && BN == 64 && STAGES <= 4) ? 3 : 2)
attn_decode_t_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     AttnArgs a, int G, Trace tr) {
  constexpr int kpc = KPC;
  constexpr int WPH = DT_CONSUMERS / KPC;  // warps per head
  const unsigned long long t_entry = trace_on(tr) ? gtime() : 0ull;
  pdl_launch_dependents();
  using SM = DecSmem<HD>;
  constexpr int PANELS = HD / 64;
  constexpr uint32_t TILE_BYTES = BN * HD * 2;
  constexpr int WK = BN / WPH;  // keys per consumer warp per tile
  constexpr int MT = WK / 16;
  constexpr int RS = SM::RS;
  static_assert(WK % 16 == 0, "tile too small for the consumer warps");
  // tile f = j * KPC + head sits in stage f % STAGES: with STAGES a multiple of KPC a stage only
  // ever holds tiles of ONE head, so exactly one warp group waits on / releases its barriers
  // (a group that skipped a phase of a barrier would see a stale parity as "complete")
  static_assert(STAGES % KPC == 0, "each ring stage must belong to one head group");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sK = (raw + 1023u) & ~1023u;  // SWIZZLE_128B panels need 1024 B alignment
  uint8_t* smem = smem_raw + (sK - raw);
  const uint32_t sV = sK + STAGES * TILE_BYTES;
  uint8_t* p_after = smem + 2 * STAGES * TILE_BYTES;
  float* red = reinterpret_cast<float*>(p_after);                       // [4][8][HD + 2]
  uint8_t* q_gen = p_after + SM::RED_BYTES;                             // [kpc][8][QROW]
  const uint32_t sQ = sK + 2 * STAGES * TILE_BYTES + SM::RED_BYTES;
  bf16* s_newkv = reinterpret_cast<bf16*>(q_gen + kpc * SM::Q_BYTES);   // [kpc][2][HD]
  const uint32_t bars = sQ + kpc * SM::Q_BYTES + kpc * 2 * HD * 2;      // full[STAGES], empty[STAGES]

  const int seq = blockIdx.x;
  const int kvh0 = blockIdx.y * kpc;
  const int split = blockIdx.z;
  const int len = a.seq_len[seq];  // step state: stable before the wait
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int* bt = a.block_tables + (size_t)seq * a.max_blocks;
  // this split's key range, in whole tiles
  const int tiles_total = (len + BN - 1) / BN;
  const int tps = (tiles_total + a.n_splits - 1) / a.n_splits;
  const int tile_begin = split * tps;
  const int n_tiles = max(0, min(tps, tiles_total - tile_begin));
  const int F = n_tiles * kpc;  // flat (head, tile) work list
  const bool fused = a.qkv_p != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(bars + 8 * s, 1);
      mbar_init(bars + 8 * (STAGES + s), WPH);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == DT_CONSUMERS) {
    // ------------------------------------------------------------ producer warp
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmK) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmV) : "memory");
    }
    // Rows past the sequence end hold whatever the pool block holds (zeros or finite stale
    // values): their scores are masked to -inf, so they contribute exactly 0.  The only row
    // the previous kernel (rope_kv, unfused mode) writes is position len - 1: tiles that end
    // before it were written by earlier steps and are requested BEFORE the dependency
    // resolves.  Fused mode patches that row in shared memory, so nothing here depends on the
    // previous kernel at all.
    bool waited = fused;
    const uint64_t once = l2_once();
    for (int f = 0; f < F; f++) {
      const int stage = f % STAGES;
      const int hh = f % KPC, j = f / KPC;  // heads interleaved tile by tile
      const int k0 = (tile_begin + j) * BN;
      if (!waited && k0 + BN > len - 1) {
        pdl_wait();
        waited = true;
      }
      if (f >= STAGES) mbar_wait(bars + 8 * (STAGES + stage), ((f / STAGES) - 1) & 1);
      const int blk = bt[k0 / KV_BLOCK];
      const int row = (blk * a.nkv + kvh0 + hh) * KV_BLOCK + (k0 % KV_BLOCK);
      const uint32_t full = bars + 8 * stage;
      if (elect_one()) {
        mbar_expect_tx(full, 2 * TILE_BYTES);
#pragma unroll
        for (int p = 0; p < PANELS; p++) {
          tma_load_2d_hint(sK + stage * TILE_BYTES + p * (BN * 128), &tmK, full, p * 64, row, once);
          tma_load_2d_hint(sV + stage * TILE_BYTES + p * (BN * 128), &tmV, full, p * 64, row, once);
        }
      }
      __syncwarp();
    }
    if (!waited) pdl_wait();
    return;
  }

  // -------------------------------------------------------------- consumer warps
  const int g = lane >> 2, t = lane & 3;
  const int mi = lane >> 3, lr = lane & 7;
  const bool has_new = fused && n_tiles > 0 && tile_begin + n_tiles == tiles_total;
  // Fused prologue = split-K sum + bias, rotate_half RoPE at position len - 1, bf16: what
  // rope_kv_kernel does for a decode token, for this CTA's query heads and its kv heads.  One
  // item = 4 + 4 floats (x at column j, its rotation partner at j + HD/2) of one real query
  // head row or of the new K / V row.  Everything that does not depend on the QKV GEMM — item
  // geometry, cos / sin, bias, the pool slot, the zero padding rows — is done BEFORE the
  // dependency resolves; after it there is one round trip for the partial slices.
  constexpr int HALF = HD / 2, VPH = HALF / 4;
  constexpr int NT = DT_CONSUMERS * 32;
  const int pos = len - 1;
  const int q_items = G * VPH, kv_items = has_new ? 2 * VPH : 0;
  const int per_head = q_items + kv_items;
  const int n_items = fused ? per_head * kpc : 0;
  struct Item {
    int hh, r, which, j, col;
    bool is_q, rot;
    float4 c, sn, bx, by;
  };
  auto prep = [&](int it0) {
    Item I;
    I.hh = it0 / per_head;
    const int it = it0 - I.hh * per_head;
    I.is_q = it < q_items;
    I.r = I.is_q ? it / VPH : 0;
    I.which = I.is_q ? 0 : (it - q_items) / VPH;  // 0 = K, 1 = V
    I.j = (I.is_q ? it % VPH : (it - q_items) % VPH) * 4;
    const int kvh = kvh0 + I.hh;
    I.col = (I.is_q ? kvh * G + I.r : a.nh + I.which * a.nkv + kvh) * HD + I.j;
    I.rot = a.cosT != nullptr && (I.is_q || I.which == 0);
    I.c = I.sn = I.bx = I.by = make_float4(0.f, 0.f, 0.f, 0.f);
    if (I.rot) {
      I.c = __ldg(reinterpret_cast<const float4*>(a.cosT + (size_t)pos * HALF + I.j));
      I.sn = __ldg(reinterpret_cast<const float4*>(a.sinT + (size_t)pos * HALF + I.j));
    }
    if (a.qkv_bias) {
      I.bx = __ldg(reinterpret_cast<const float4*>(a.qkv_bias + I.col));
      I.by = __ldg(reinterpret_cast<const float4*>(a.qkv_bias + I.col + HALF));
    }
    return I;
  };
  Item first;
  if ((int)threadIdx.x < n_items) first = prep(threadIdx.x);
  const int new_blk = has_new ? bt[pos / KV_BLOCK] : 0;
  // query rows >= G are MMA padding: zero
  for (int i = threadIdx.x; i < kpc * (8 - G) * (HD / 8); i += NT) {
    const int hh = i / ((8 - G) * (HD / 8)), rem = i % ((8 - G) * (HD / 8));
    const int r = G + rem / (HD / 8), c = rem % (HD / 8);
    *reinterpret_cast<uint4*>(q_gen + hh * SM::Q_BYTES + r * SM::QROW + c * 16) = make_uint4(0, 0, 0, 0);
  }
  pdl_wait();
  const unsigned long long t_wait = trace_on(tr) ? gtime() : 0ull;
  if (!fused) {
    // Q rows (bf16, written by rope_kv) -> padded shared rows
    constexpr int CPR = HD / 8;
    for (int i = threadIdx.x; i < kpc * G * CPR; i += NT) {
      const int hh = i / (G * CPR), r = (i / CPR) % G, c = i % CPR;
      *reinterpret_cast<uint4*>(q_gen + hh * SM::Q_BYTES + r * SM::QROW + c * 16) =
          *reinterpret_cast<const uint4*>((const bf16*)a.q + (size_t)seq * a.nh * HD +
                                          (size_t)((kvh0 + hh) * G + r) * HD + c * 8);
    }
  } else {
    const float* rowp = a.qkv_p + (size_t)seq * a.qkv_ld;
    for (int it0 = threadIdx.x; it0 < n_items; it0 += NT) {
      const Item I = it0 == (int)threadIdx.x ? first : prep(it0);
      float4 x = I.bx, y = I.by;
      for (int q0 = 0; q0 < a.qkv_S; q0 += 8) {
        // up to 8 slices of both halves in flight at once: one L2 round trip
        float4 px[8], py[8];
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (q0 + q < a.qkv_S) {
            const float* pp = rowp + (size_t)(q0 + q) * a.qkv_stride + I.col;
            px[q] = *reinterpret_cast<const float4*>(pp);
            py[q] = *reinterpret_cast<const float4*>(pp + HALF);
          }
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (q0 + q < a.qkv_S) {
            x.x += px[q].x; x.y += px[q].y; x.z += px[q].z; x.w += px[q].w;
            y.x += py[q].x; y.y += py[q].y; y.z += py[q].z; y.w += py[q].w;
          }
      }
      if (I.rot) {
        const float4 x0 = x, y0 = y, c = I.c, sn = I.sn;
        x.x = x0.x * c.x - y0.x * sn.x; y.x = y0.x * c.x + x0.x * sn.x;
        x.y = x0.y * c.y - y0.y * sn.y; y.y = y0.y * c.y + x0.y * sn.y;
        x.z = x0.z * c.z - y0.z * sn.z; y.z = y0.z * c.z + x0.z * sn.z;
        x.w = x0.w * c.w - y0.w * sn.w; y.w = y0.w * c.w + x0.w * sn.w;
      }
      const uint2 lo = make_uint2(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w));
      const uint2 hi = make_uint2(pack_bf16(y.x, y.y), pack_bf16(y.z, y.w));
      if (I.is_q) {
        uint8_t* qr = q_gen + I.hh * SM::Q_BYTES + I.r * SM::QROW;
        *reinterpret_cast<uint2*>(qr + I.j * 2) = lo;
        *reinterpret_cast<uint2*>(qr + (I.j + HALF) * 2) = hi;
      } else {
        bf16* nk = s_newkv + ((size_t)I.hh * 2 + I.which) * HD;
        *reinterpret_cast<uint2*>(nk + I.j) = lo;
        *reinterpret_cast<uint2*>(nk + I.j + HALF) = hi;
        // this CTA covers the end of the sequence: it appends the row to the paged pool
        bf16* pool = I.which ? (bf16*)a.vpool : (bf16*)a.kpool;
        bf16* dst = pool + (((size_t)new_blk * a.nkv + kvh0 + I.hh) * KV_BLOCK + (pos % KV_BLOCK)) * HD + I.j;
        *reinterpret_cast<uint2*>(dst) = lo;
        *reinterpret_cast<uint2*>(dst + HALF) = hi;
      }
    }
  }
  consumer_bar();  // Q and the new K / V rows are visible to the four warps
  const unsigned long long t_prol = tr.buf ? gtime() : 0ull;
  unsigned long long t_first = 0, t_fin0 = 0;

  uint32_t qb[HD / 16][2];
  float o[HD / 16][4];
  float m[2], l[2];
  const float scale_log2 = a.scale * 1.4426950408889634f;
  const int limit = len - 1;

  const int hh = warp / WPH, wi = warp % WPH;  // this warp's head and its slot in the group
  {
    const uint32_t q = sQ + hh * SM::Q_BYTES + g * SM::QROW + t * 4;
#pragma unroll
    for (int ks = 0; ks < HD / 16; ks++) {
      qb[ks][0] = lds32(q + ks * 32);
      qb[ks][1] = lds32(q + ks * 32 + 16);
    }
#pragma unroll
    for (int dt = 0; dt < HD / 16; dt++)
#pragma unroll
      for (int i = 0; i < 4; i++) o[dt][i] = 0.f;
    m[0] = m[1] = -INFINITY;
    l[0] = l[1] = 0.f;
  }
  for (int j = 0; j < n_tiles; j++) {
    const int f = j * KPC + hh;
    const int stage = f % STAGES;
    mbar_wait(bars + 8 * stage, (f / STAGES) & 1);
    if (tr.buf && j == 0) t_first = gtime();
    const uint32_t tK = sK + stage * TILE_BYTES, tV = sV + stage * TILE_BYTES;
    const int k0 = (tile_begin + j) * BN;
    const int key0 = wi * WK;
    bool patched = false;
    if (has_new && j == n_tiles - 1) {
      // the tile landed with whatever the pool held at position len - 1: the warp that owns
      // that key row overwrites it with the K / V built in the prologue
      const int row = len - 1 - k0;
      if (row >= key0 && row < key0 + WK) {
        for (int i = lane; i < 2 * (HD / 8); i += 32) {
          const int which = i / (HD / 8), c = i % (HD / 8);
          st_shared16((which ? tV : tK) + tile_off_t<BN>(row, c),
                      *reinterpret_cast<const uint4*>(s_newkv + ((size_t)hh * 2 + which) * HD + c * 8));
        }
        __syncwarp();
        patched = true;
      }
    }
    // ---- S^T = K . Q^T for this warp's WK keys
    float s[MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
#pragma unroll
      for (int i = 0; i < 4; i++) s[mt][i] = 0.f;
#pragma unroll
      for (int ks = 0; ks < HD / 16; ks++) {
        uint32_t a0, a1, a2, a3;
        ldsm_x4(tK + tile_off_t<BN>(key0 + mt * 16 + lr + (mi & 1) * 8, ks * 2 + (mi >> 1)), a0, a1,
                a2, a3);
        mma16816(s[mt], a0, a1, a2, a3, qb[ks][0], qb[ks][1]);
      }
    }
    if (k0 + BN > len) {
#pragma unroll
      for (int mt = 0; mt < MT; mt++) {
        const int kp = k0 + key0 + mt * 16 + g;
        if (kp > limit) s[mt][0] = s[mt][1] = -INFINITY;
        if (kp + 8 > limit) s[mt][2] = s[mt][3] = -INFINITY;
      }
    }
    // ---- online softmax: this thread holds heads 2t (e = 0) and 2t + 1 (e = 1)
    float corr[2], mu[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      float mx = -INFINITY;
#pragma unroll
      for (int mt = 0; mt < MT; mt++) mx = fmaxf(mx, fmaxf(s[mt][e], s[mt][2 + e]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
      const float m_new = fmaxf(m[e], mx);
      const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
      corr[e] = exp2f((m[e] - m_use) * scale_log2);  // m = -inf => 0
      m[e] = m_new;
      mu[e] = m_use * scale_log2;
      float rs = 0.f;
#pragma unroll
      for (int mt = 0; mt < MT; mt++) {
        const float p0 = exp2f(fmaf(s[mt][e], scale_log2, -mu[e]));
        const float p1 = exp2f(fmaf(s[mt][2 + e], scale_log2, -mu[e]));
        s[mt][e] = p0;
        s[mt][2 + e] = p1;
        rs += p0 + p1;
      }
      l[e] = l[e] * corr[e] + rs;  // per-thread partial; the key lanes are reduced at the end
    }
#pragma unroll
    for (int dt = 0; dt < HD / 16; dt++) {
      o[dt][0] *= corr[0];
      o[dt][1] *= corr[1];
      o[dt][2] *= corr[0];
      o[dt][3] *= corr[1];
    }
    // ---- O^T += V^T . P^T
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
      const uint32_t b0 = movmatrix_t(pack_bf16(s[mt][0], s[mt][1]));
      const uint32_t b1 = movmatrix_t(pack_bf16(s[mt][2], s[mt][3]));
#pragma unroll
      for (int dt = 0; dt < HD / 16; dt++) {
        uint32_t a0, a1, a2, a3;
        ldsm_x4_t(tV + tile_off_t<BN>(key0 + mt * 16 + lr + (mi >> 1) * 8, dt * 2 + (mi & 1)), a0, a1,
                  a2, a3);
        mma16816(o[dt], a0, a1, a2, a3, b0, b1);
      }
    }
    // ---- release the stage
    if (patched) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bars + 8 * (STAGES + stage));

  }
  if (n_tiles > 0) {
    if (tr.buf && hh == 0) t_fin0 = gtime();
    // ---- finish this group's head: row sums over the 8 key lanes, then either write straight
    // from the registers (one warp per head) or merge the group's WPH warps through `red`
#pragma unroll
    for (int e = 0; e < 2; e++) {
      l[e] += __shfl_xor_sync(0xffffffffu, l[e], 4);
      l[e] += __shfl_xor_sync(0xffffffffu, l[e], 8);
      l[e] += __shfl_xor_sync(0xffffffffu, l[e], 16);
    }
    const int h0 = (kvh0 + hh) * G;
    if constexpr (WPH == 1) {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int r = 2 * t + e;
        if (r >= G) continue;
        const float inv = 1.f / l[e];
        bf16* op = (bf16*)a.out + (size_t)seq * a.nh * HD + (size_t)(h0 + r) * HD;
#pragma unroll
        for (int dt = 0; dt < HD / 16; dt++) {
          op[dt * 16 + g] = __float2bfloat16_rn(o[dt][e] * inv);
          op[dt * 16 + 8 + g] = __float2bfloat16_rn(o[dt][2 + e] * inv);
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int r = 2 * t + e;
        if (r >= G) continue;
        float* rr = red + ((size_t)warp * 8 + r) * RS;
#pragma unroll
        for (int dt = 0; dt < HD / 16; dt++) {
          rr[dt * 16 + g] = o[dt][e];
          rr[dt * 16 + 8 + g] = o[dt][2 + e];
        }
        if (g == 0) {
          rr[HD] = m[e];
          rr[HD + 1] = l[e];
        }
      }
      // immediate barrier ids: a register id would make ptxas reserve all 16 named barriers
      if constexpr (WPH == DT_CONSUMERS) {
        consumer_bar();
      } else {
        if (hh == 0) asm volatile("bar.sync 2, 64;" ::: "memory");
        else asm volatile("bar.sync 3, 64;" ::: "memory");
      }
      const int w0 = hh * WPH;
      for (int idx = threadIdx.x - w0 * 32; idx < G * HD; idx += WPH * 32) {
        const int r = idx / HD, d = idx % HD;
        float mn = -INFINITY;
#pragma unroll
        for (int w = 0; w < WPH; w++) mn = fmaxf(mn, red[((size_t)(w0 + w) * 8 + r) * RS + HD]);
        float lt = 0.f, at = 0.f;
#pragma unroll
        for (int w = 0; w < WPH; w++) {
          const float* rr = red + ((size_t)(w0 + w) * 8 + r) * RS;
          const float c = (rr[HD] == -INFINITY) ? 0.f : exp2f((rr[HD] - mn) * scale_log2);
          lt += rr[HD + 1] * c;
          at += rr[d] * c;
        }
        const int h = h0 + r;
        if (a.n_splits == 1) {
          ((bf16*)a.out)[(size_t)seq * a.nh * HD + (size_t)h * HD + d] = __float2bfloat16_rn(at / lt);
        } else {
          float* rec = a.ws + (((size_t)seq * a.nh + h) * a.n_splits + split) * (HD + 2);
          rec[d] = at;
          if (d == 0) {
            rec[HD] = (mn == -INFINITY) ? -INFINITY : mn * a.scale;  // combine kernel works in exp()
            rec[HD + 1] = lt;
          }
        }
      }
    }
  }
  if (n_tiles == 0) {  // empty split: (0, -inf, 0) records
    for (int idx = threadIdx.x; idx < kpc * G * HD; idx += DT_CONSUMERS * 32) {
      const int h = kvh0 * G + idx / HD, d = idx % HD;
      float* rec = a.ws + (((size_t)seq * a.nh + h) * a.n_splits + split) * (HD + 2);
      rec[d] = 0.f;
      if (d == 0) {
        rec[HD] = -INFINITY;
        rec[HD + 1] = 0.f;
      }
    }
  }
  if (threadIdx.x == 0 && trace_on(tr))
    trace_rec(tr, t_entry, t_wait,
              (((t_prol - t_wait) & 0x1fffff) << 42) | (((t_first - t_wait) & 0x1fffff) << 21) |
                  ((t_fin0 - t_wait) & 0x1fffff));
}

// ------------------------------------------------------------------ launcher
bool attn_decode_t_supported(const AttnArgs& a) {
  static const int off = getenv("NVLLM_ATTN_T") ? atoi(getenv("NVLLM_ATTN_T")) == 0 : 0;
  if (off) return false;
  return attn_mma_supported(a.qdt, a.kvdt, a.hd) && a.nkv > 0 && a.nh % a.nkv == 0 &&
         a.nh / a.nkv <= 8 && a.pool_blocks > 0;
}

template <int HD, int BN, int STAGES, int KPC>
static cudaError_t decode_t_launch(cudaStream_t st, const AttnArgs& a, int G) {
  using SM = DecSmem<HD>;
  constexpr int kpc = KPC;
  const size_t smem = 1024 + (size_t)2 * STAGES * BN * HD * 2 + SM::RED_BYTES +
                      (size_t)kpc * SM::Q_BYTES + (size_t)kpc * 2 * HD * 2 + 16 * STAGES;
  const int pool_rows = a.pool_blocks * a.nkv * KV_BLOCK;
  const TmaDesc* tk = tma_map_cached(a.kpool, pool_rows, HD, BN);
  const TmaDesc* tv = tma_map_cached(a.vpool, pool_rows, HD, BN);
  if (!tk || !tv) return cudaErrorInvalidValue;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(attn_decode_t_kernel<HD, BN, STAGES, KPC>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  (void)launch_k(attn_decode_t_kernel<HD, BN, STAGES, KPC>, dim3(a.n_seqs, a.nkv / kpc, a.n_splits),
                 dim3(DT_THREADS), smem, st, *reinterpret_cast<const CUtensorMap*>(tk),
                 *reinterpret_cast<const CUtensorMap*>(tv), a, G, next_trace(4));
  return cudaGetLastError();
}

// kv heads per CTA can be forced with NVLLM_ATTN_T_KPC (1, 2, 4) for experiments.
// The order of a row's sums follows it: a replayed graph is kept for one choice only (run.cu), so that a step's results
// do not depend on the lengths that the handle saw before.
int attn_decode_heads(int n_seqs, int nh, int nkv, int max_len, int n_splits, int sm_count) {
  if (nkv <= 0 || nh % nkv) return 1;
  const int G = nh / nkv;
  // read per launch (not cached): the parity tests switch it between runners
  const char* kpc_s = getenv("NVLLM_ATTN_T_KPC");
  const int kpc_env = kpc_s ? atoi(kpc_s) : 0;
  // The fixed cost of a CTA (launch, prologue, first-tile latency) is ~4 us against ~0.6 us
  // per 64-key tile: when the step has more (sequence, kv head) pairs than resident CTA slots,
  // pack 2 heads per CTA while the grid still covers ~1.6 CTAs per SM.  (4 heads per CTA with
  // one stage per head measured slower — cfg3 1810 vs 1775 us/step, cfg2 1231 vs 1088 — and is
  // only reachable through the knob.)
  int kpc = 1;
  if (n_splits == 1) {
    const int sm = sm_count > 0 ? sm_count : 148;
    while (kpc < 2 && nkv % (kpc * 2) == 0 &&
           (long)n_seqs * (nkv / (kpc * 2)) * 10 >= (long)sm * 16)
      kpc *= 2;
    // heads by themselves (G = 1) and short contexts: two of them to a CTA merge over two warps each instead of four
    // (GPT-2 alone, us a step: 30 tokens 220 -> 210, 150 209 -> 201, 300 216 -> 213; eight sequences of 450 268 -> 271)
    if (kpc == 1 && G == 1 && nkv % 2 == 0 && max_len <= 256) kpc = 2;
    if ((kpc_env == 1 || kpc_env == 2 || kpc_env == 4) && nkv % kpc_env == 0) kpc = kpc_env;
  }
  return kpc;
}

cudaError_t launch_attn_decode_t(cudaStream_t st, const AttnArgs& a) {
  if (a.n_seqs <= 0) return cudaSuccess;
  const int G = a.nh / a.nkv, kpc = attn_decode_heads(a.n_seqs, a.nh, a.nkv, a.max_len, a.n_splits, a.sm_count);
  if (a.hd == 64) {
    // 4 heads: one 16 KB stage per head (3 CTAs / SM, 12 head streams per SM in flight)
    if (kpc == 4) return decode_t_launch<64, 64, 4, 4>(st, a, G);
    if (kpc == 2) return decode_t_launch<64, 64, 6, 2>(st, a, G);
    if (a.n_splits > 1) return decode_t_launch<64, 64, 6, 1>(st, a, G);
    return decode_t_launch<64, 64, 4, 1>(st, a, G);
  }
  // head dim 128: 32 KB stages; at most 2 heads per CTA
  if (kpc >= 2) return decode_t_launch<128, 64, 2, 2>(st, a, G);
  return decode_t_launch<128, 64, 3, 1>(st, a, G);
}

}  // namespace nvllm
