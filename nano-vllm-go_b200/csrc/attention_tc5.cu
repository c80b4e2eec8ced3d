// attention_tc5.cu — paged causal prefill attention on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory, operands by TMA), bf16, head dim 64 / 128.
//
// Reference math: scores = Q K^T * scale, causal mask, row softmax, P V
// (purego/tensor/attention.go:354-421 GQA, :127-191 MHA, mqa.go:184-243 MQA), K / V read through
// the scheduler's block tables, the cached prefix of a sequence (NumCachedTokens) attended but
// not recomputed.
//
// Options (AttnArgs, compiled in by OPT): a sink in the softmax's denominator (score 0 or
// learned per head) and the output of a head times a gate per (token, head), both outside the per-score
// loop (OPT 1); besides, a window of keys (OPT 2), whose key tiles start at the first query's first key.  Capped scores and distance penalties stay with the mma.sync kernels of attention_window.cu: a
// transform of every score in the softmax warps (tried: 3.5 to 5.7 ms against 0.97 ms plain, 16 x 4096 tokens,
// 16 heads of 64) made this kernel slower than those.
//
// Persistent, two CTAs per SM: an item is 128 queries of one sequence x one query head, dealt out by a counter, heaviest
// first.  Per key tile (BN keys):
//   scheduler     the next items' rows, positions and key tiles, up to four ahead (every warp finds the CTA's first item
//                 itself, before the wait for the kernel in front)
//   TMA warp      Q of the item, K / V tiles of the paged pool (one (block, kv head) slab is contiguous;
//                 2-D tensor map over the layer's pool, SWIZZLE_128B) -> shared memory, two stages each
//   MMA warp      S = Q K^T   (128 x BN, K-major x K-major, accumulator in TMEM), issued as soon as the softmax warps
//                 have the tile before in registers
//                 O += P V    (128 x hd; P from tensor memory, V as the MN-major operand —
//                 the pool keeps V [key][hd], so no transpose anywhere)
//   softmax warps thread r owns query row r (TMEM lane r): the S row is read into registers
//                 once (all tcgen05.ld issued, one wait), row max, exp2 / row sum, bf16 P
//                 back to tensor memory.  O stays in TMEM across the
//                 tiles (accumulating MMAs); it is rescaled there only when the running
//                 maximum has grown by more than a factor 2^8 ("lazy" flash rescaling), and
//                 read once, under the next item's first tile — nothing but the final output leaves the SM
// Bound by the softmax warps of the SM's two CTAs: row maximum and 128 exp2 a row take 2400 cycles a tile of 128 keys where
// the special-function units alone would take 1024 of each, and 2600 an item go to its hand-over (prompts of 256 to 512
// tokens, 2.1 tiles an item).  With one CTA per item, S only after the P V before it and P through shared memory (which
// costs a proxy fence): 4150 a tile and 4000 an item.  Per launch, 64 such prompts, 32 heads of 64: 255 -> 195 us; 16 heads
// 73 -> 58; 16 x 256 queries on 3840 cached keys, 24 heads of 128: 409 -> 348 (711 -> 834 TFLOP/s); one prompt of 2048, 71
// heads of 64: 97 -> 86.
// Windows, per launch against the mma.sync kernel of attention_window.cu, 32 heads of 64 / 128, us: 8 x 2000 tokens, window 32
// 170 -> 76 / 307 -> 102, 128 232 -> 76 / 413 -> 112, 1024 618 -> 219 / 1051 -> 257; 16 x 600, window 512 229 -> 85 / 375 -> 99;
// one prompt of 40 tokens 10.4 -> 7.8 / 12.7 -> 7.6; faster at every size tried, so every layer that fits takes this kernel.
#include <cuda.h>
#include <stdlib.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "gemm_tc5.cuh"
#include "tc5.cuh"
#include "tma.cuh"

namespace nvllm {

namespace {

constexpr int PT_BM = 128;       // queries per CTA (UMMA M)
constexpr int PT_THREADS = 256;  // warps 0-3 softmax (warpgroup 0), warp 4 TMA, warp 5 MMA, warp 6 scheduler, 7 idle
constexpr int PT_ITEMS = 4;      // items known ahead

// a query tile of one head: its first row and query position, rows in use, key tiles (0: no more items)
struct PtItem {
  int seq, head, row, pos, rows, n_tiles, first;  // first: key tile
};

template <int HD>
struct PtCfg {
  static constexpr int BN = HD == 64 ? 128 : 64;  // keys per tile
  static constexpr int ST = 2;                     // stages of K and of V
  static constexpr int SUB = HD / 64;              // 64-column (128-byte) sub-tiles of a head row
  static constexpr uint32_t Q_BYTES = PT_BM * HD * 2;
  static constexpr uint32_t KV_BYTES = BN * HD * 2;
  static constexpr uint32_t TILES = Q_BYTES + 2 * ST * KV_BYTES;
  static constexpr uint32_t SMEM = TILES + 512;    // barriers, items, tensor-memory address
  static constexpr uint32_t TMEM_COLS = 256;       // S: BN columns at 0, O: HD columns at BN, P: BN / 2 columns behind
  static_assert(BN + HD + BN / 2 <= 256, "two CTAs share the tensor memory");
  static_assert(2 * (SMEM + 1024) <= 233472, "and the shared memory");
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

}  // namespace

// OPT: which options of AttnArgs are compiled in (1: sink, gate per head; 2: the window too)
template <int HD, int OPT>
__global__ void __launch_bounds__(PT_THREADS, 2)
attn_prefill_tc5_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV, AttnArgs a, Trace tr) {
  using Cf = PtCfg<HD>;
  constexpr int BN = Cf::BN, SUB = Cf::SUB, ST = Cf::ST;
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  extern __shared__ __align__(1024) uint8_t smem_raw[];  // (no static shared memory in front of it)
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t sQ = base;
  const uint32_t sK = sQ + Cf::Q_BYTES;
  const uint32_t sV = sK + ST * Cf::KV_BYTES;
  const uint32_t bars = sV + ST * Cf::KV_BYTES;
  const uint32_t b_qfull = bars, b_qempty = bars + 8, b_kfull = bars + 16, b_kempty = bars + 32, b_vfull = bars + 48,
                 b_vempty = bars + 64, b_sfull = bars + 80, b_sread = bars + 88, b_pready = bars + 96, b_ofull = bars + 104,
                 b_ifull = bars + 112, b_iempty = bars + 112 + 8 * PT_ITEMS;
  uint8_t* tail = smem_raw + Cf::TILES + 112 + 16 * PT_ITEMS;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(tail);
  volatile uint32_t* dead = reinterpret_cast<uint32_t*>(tail + 4);
  PtItem* items = reinterpret_cast<PtItem*>(tail + 16);
  static_assert(112 + 16 * PT_ITEMS + 16 + PT_ITEMS * sizeof(PtItem) <= 512, "the tail of the shared memory");
  if (base & 1023) {  // (the swizzle's atoms would not line up; the host's layout rules this out)
    if (threadIdx.x == 0 && a.wait_flag) *reinterpret_cast<volatile int*>(a.wait_flag) = 1;
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_items = a.n_qtiles * a.nh, grid = (int)gridDim.x;
  auto item_at = [&](int t) {
    // heaviest tiles (latest queries of a sequence see the most keys) first, the heads of a tile next to each other
    PtItem w;
    const int tile = a.n_qtiles - 1 - t / a.nh;
    w.head = t % a.nh;
    w.seq = a.tile_seq[tile];
    const int q0 = a.tile_q0[tile], first = a.cu_q[w.seq];
    w.row = first + q0;
    w.rows = min(PT_BM, a.cu_q[w.seq + 1] - first - q0);
    w.pos = a.seq_start[w.seq] + q0;
    w.first = OPT > 1 ? max(0, w.pos - a.window + 1) / BN : 0;
    w.n_tiles = (w.pos + w.rows + BN - 1) / BN - w.first;  // keys up to pos + rows are visible to this tile
    return w;
  };

  if (warp == 4 && lane == 0) {
    mbar_init(b_qfull, 1);
    mbar_init(b_qempty, 1);
    for (int s = 0; s < ST; s++) {
      mbar_init(b_kfull + 8 * s, 1);
      mbar_init(b_kempty + 8 * s, 1);
      mbar_init(b_vfull + 8 * s, 1);
      mbar_init(b_vempty + 8 * s, 1);
    }
    mbar_init(b_sfull, 1);
    mbar_init(b_sread, 4);   // one arrival per softmax warp
    mbar_init(b_pready, 4);
    mbar_init(b_ofull, 1);
    for (int s = 0; s < PT_ITEMS; s++) {
      mbar_init(b_ifull + 8 * s, 1);
      mbar_init(b_iempty + 8 * s, 6);  // TMA, MMA and softmax warps
    }
    *dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmQ) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmK) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmV) : "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot_ptr)),
                 "r"(Cf::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  const uint32_t tS = tmem_base, tO = tmem_base + BN, tP = tO + HD;
  auto wait = [&](uint32_t bar, int parity) { return wait_short(bar, (uint32_t)parity & 1, dead, a.wait_flag); };
  // the CTA's item `it` > 0 once it is known (n_tiles == 0: there are no more); false when the wait ran out
  auto next_item = [&](int it, PtItem& w) {
    if (n_items <= grid) {
      w.n_tiles = 0;
      return true;
    }
    const int s = (it - 1) % PT_ITEMS;
    if (!wait(b_ifull + 8 * s, (it - 1) / PT_ITEMS)) return false;
    w = items[s];
    __syncwarp();
    if (lane == 0) mbar_arrive(b_iempty + 8 * s);
    return true;
  };

  if (warp >= 4) {
    // warpgroup 1 (TMA warp 4, MMA warp 5, scheduler warp 6, an idle warp) hands its registers to the softmax
    // warpgroup, whose threads carry a whole fp32 output row
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    PtItem w = item_at(blockIdx.x);  // (what it reads came with the step: no kernel writes it)
    // Q and this step's K / V rows are the previous kernels' output (and the limit of the waits counts from the wait for them)
    if (warp == 6) {
      // ---------------------------------------------------------------- scheduler
      pdl_wait();
      if (n_items > grid) {
        auto draw = [&](int t) { return lane != 0 ? 0 : a.tickets ? grid + atomicAdd(a.tickets, 1) : t + grid; };
        auto drawn = [&](int d) {
          d = __shfl_sync(0xffffffffu, d, 0);
          // the counter is zero again for the next launch: n_items draws in all, of each CTA one past the end
          if (a.tickets && d - grid == n_items - 1 && lane == 0) *a.tickets = 0;
          return d;
        };
        int t = drawn(draw(blockIdx.x));
        for (int it = 0;; it++) {
          const bool more = t < n_items;
          const int d = more ? draw(t) : 0;  // the item after this one
          w.n_tiles = 0;
          if (more) w = item_at(t);
          const int s = it % PT_ITEMS;
          if (!wait(b_iempty + 8 * s, it / PT_ITEMS + 1)) break;
          if (elect_one()) {
            items[s] = w;
            mbar_arrive(b_ifull + 8 * s);
          }
          __syncwarp();
          if (!more) break;
          t = drawn(d);
        }
      }
    } else if (warp == 4) {
      // ---------------------------------------------------------------- TMA producer
      int g = 1;  // key tiles so far
      bool ok = true;
      {  // the first item's queries and first key tile: short code behind the wait, which a launch fetches while it counts
        const int k0 = w.first * BN;
        const int prow = (a.block_tables[(size_t)w.seq * a.max_blocks + k0 / KV_BLOCK] * a.nkv + w.head / (a.nh / a.nkv)) * KV_BLOCK + k0 % KV_BLOCK;
        const bool one = elect_one();
        if (one) {
          mbar_expect_tx(b_qfull, Cf::Q_BYTES);
          mbar_expect_tx(b_kfull, Cf::KV_BYTES);
          mbar_expect_tx(b_vfull, Cf::KV_BYTES);
        }
        pdl_wait();
        if (one) {
          for (int s = 0; s < SUB; s++) tma_load_2d(sQ + s * (PT_BM * 128), &tmQ, b_qfull, w.head * HD + 64 * s, w.row);
          for (int s = 0; s < SUB; s++) tma_load_2d(sK + s * (BN * 128), &tmK, b_kfull, 64 * s, prow);
          for (int s = 0; s < SUB; s++) tma_load_2d(sV + s * (BN * 128), &tmV, b_vfull, 64 * s, prow);
        }
        __syncwarp();
      }
      for (int it = 0; ok && w.n_tiles > 0; it++) {
        const int* bt = a.block_tables + (size_t)w.seq * a.max_blocks;
        const int kvh = w.head / (a.nh / a.nkv);
        if (it > 0) {
          if (!wait(b_qempty, it - 1)) break;
          if (elect_one()) {
            mbar_expect_tx(b_qfull, Cf::Q_BYTES);
            for (int s = 0; s < SUB; s++) tma_load_2d(sQ + s * (PT_BM * 128), &tmQ, b_qfull, w.head * HD + 64 * s, w.row);
          }
          __syncwarp();
        }
        for (int j = it == 0 ? 1 : 0; j < w.n_tiles; j++, g++) {
          const int k0 = (w.first + j) * BN, st = g % ST;
          const int prow = (bt[k0 / KV_BLOCK] * a.nkv + kvh) * KV_BLOCK + (k0 % KV_BLOCK);
          if (!(ok = wait(b_kempty + 8 * st, g / ST + 1))) break;
          if (elect_one()) {
            mbar_expect_tx(b_kfull + 8 * st, Cf::KV_BYTES);
            for (int s = 0; s < SUB; s++)
              tma_load_2d(sK + st * Cf::KV_BYTES + s * (BN * 128), &tmK, b_kfull + 8 * st, 64 * s, prow);
          }
          __syncwarp();
          if (!(ok = wait(b_vempty + 8 * st, g / ST + 1))) break;
          if (elect_one()) {
            mbar_expect_tx(b_vfull + 8 * st, Cf::KV_BYTES);
            for (int s = 0; s < SUB; s++)
              tma_load_2d(sV + st * Cf::KV_BYTES + s * (BN * 128), &tmV, b_vfull + 8 * st, 64 * s, prow);
          }
          __syncwarp();
        }
        ok = ok && next_item(it + 1, w);
      }
    } else if (warp == 5) {
      // ---------------------------------------------------------------- MMA issuer
      // instruction descriptors (cute/arch/mma_sm100_desc.hpp): fp32 accumulate, bf16 x bf16,
      // M = 128; S: N = BN, both operands K-major; O: N = hd, B (= V) MN-major (bit 16)
      constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                                   ((uint32_t)(PT_BM >> 4) << 24);
      constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) |
                                   ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(PT_BM >> 4) << 24);
      auto scores = [&](int g, bool last) {
        const int st = g % ST;
        if (!wait(b_kfull + 8 * st, g / ST)) return false;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int s = 0; s < SUB; s++) {
            const uint64_t qd = make_smem_desc(sQ + s * (PT_BM * 128));
            const uint64_t kd = make_smem_desc(sK + st * Cf::KV_BYTES + s * (BN * 128));
#pragma unroll
            for (int kk = 0; kk < 4; kk++) tc_mma_bf16(tS, qd + 2 * kk, kd + 2 * kk, idesc_s, (s | kk) != 0);
          }
          tc_commit(b_kempty + 8 * st);
          tc_commit(b_sfull);
          if (last) tc_commit(b_qempty);  // the next item's queries may come
        }
        __syncwarp();
        return true;
      };
      int g = 0;
      bool ok = true;
      PtItem wn;
      pdl_wait();
      for (int it = 0; ok && w.n_tiles > 0; it++, w = wn) {
        const int n_tiles = w.n_tiles;
        // (the previous item's last S has been read: its P V came after)
        if (!wait(b_qfull, it) || !scores(g, n_tiles == 1)) break;
        for (int j = 0; j < n_tiles; j++, g++) {
          // under the softmax of this tile: S of the next one, or what the next item is (with its S ahead of this item's
          // last P V the 64 prompts above took 216 us, and 198 in this order)
          if (j + 1 < n_tiles) ok = wait(b_sread, g) && scores(g + 1, j + 2 == n_tiles);
          else ok = next_item(it + 1, wn);
          const int st = g % ST;
          // P_j is in tensor memory, its O there may be written
          if (!(ok = ok && wait(b_vfull + 8 * st, g / ST) && wait(b_pready, g))) break;
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < BN / 16; kk++) {
              const uint64_t vd = make_smem_desc_mn(sV + st * Cf::KV_BYTES + kk * 2048, BN * 128);
              tc_mma_bf16_ta(tO, tP + 8 * kk, vd, idesc_o, (j | kk) != 0);
            }
            tc_commit(b_vempty + 8 * st);
            tc_commit(b_ofull);
          }
          __syncwarp();
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + output
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    PtItem w = item_at(blockIdx.x);
    pdl_wait();
    const int q = warp;  // TMEM lane quadrant of this warp
    const int r = q * 32 + lane;
    constexpr float LOG2E = 1.4426950408889634f;
    const float sl2 = a.scale * LOG2E;
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    // O accumulates in TMEM across the key tiles (the P V MMAs run with accumulate = 1).  The
    // exponent reference m_used only follows the running maximum when it has grown by more than
    // 2^RESCALE_LOG2 in probability — then, and only then, O (TMEM) and l are rescaled; in
    // between, p = exp2(s - m_used) may exceed 1 by at most that factor, harmless in fp32 / bf16.
    constexpr float RESCALE_LOG2 = 8.f;
    int g = 0;
    bool ok = true;
    // the finished item whose O waits in tensor memory
    bf16* o_row = nullptr;
    float o_inv = 0.f;
    bool o_pending = false;
    auto output = [&] {
#pragma unroll 1
      for (int c0 = 0; c0 < HD; c0 += 32) {
        uint32_t rr[32];
        tmem_ld_32x32(tO + lane_off + (uint32_t)c0, rr);
        if (o_row) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = __uint_as_float(rr[c + i]) * o_inv;
            store8(o_row + c0 + c, v);
          }
        }
      }
      __syncwarp();
      o_pending = false;
    };
    for (int it = 0; ok && w.n_tiles > 0; it++) {
      const int n_tiles = w.n_tiles;
      float m_used = -INFINITY, l_run = 0.f;
      for (int j = 0; j < n_tiles; j++, g++) {
        // columns of this tile up to which the warp's first row sees keys (its last row: 31 more)
        const int lim = w.pos + q * 32 - (w.first + j) * BN;
        const int low = lim - a.window + 1;  // and from which on (OPT 2)
        if (!(ok = wait(b_sfull, g))) break;
        tc_fence_after();
        // the whole S row of this tile in registers: all loads issued, one wait
        uint32_t sr[BN];
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) tmem_ld_32x32_nowait(tS + lane_off + (uint32_t)c0, &sr[c0]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(b_sread);
        float mx = -INFINITY;
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) {
          if (c0 > lim + 31 || (OPT > 1 && c0 + 31 < low)) continue;  // no row of the warp sees these keys: p = 0 below
          if (OPT > 1 && c0 < low + 31) {
#pragma unroll
            for (int c = 0; c < 32; c++)
              if (c0 + c < low + lane) sr[c0 + c] = 0xff800000u;
          }
          if (c0 + 31 > lim) {
#pragma unroll
            for (int c = 0; c < 32; c++)
              if (c0 + c > lim + lane) sr[c0 + c] = 0xff800000u;  // -inf: p = 0
          }
          float m[4];
#pragma unroll
          for (int c = 0; c < 4; c++) m[c] = __uint_as_float(sr[c0 + c]);
#pragma unroll
          for (int c = 4; c < 32; c++) m[c & 3] = fmaxf(m[c & 3], __uint_as_float(sr[c0 + c]));
          mx = fmaxf(mx, fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])));
        }
        // rows of the tile that see no key yet (mx = -inf) keep their reference
        const bool grow = (mx - m_used) * sl2 > RESCALE_LOG2 || (m_used == -INFINITY && mx > -INFINITY);
        const float m_new = grow ? mx : m_used;
        const float corr = (m_used == -INFINITY) ? 0.f : ex2((m_used - m_new) * sl2);
        const bool rescale = __any_sync(0xffffffffu, grow);
        if (rescale) l_run *= corr;
        m_used = m_new;
        const float mb = (m_used == -INFINITY) ? 0.f : m_used * sl2;
        const unsigned long long sl2_2 = pack2(sl2, sl2), mb_2 = pack2(-mb, -mb);
        float sum = 0.f;
        uint32_t pk[BN / 2];
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) {
          if (c0 > lim + 31 || (OPT > 1 && c0 + 31 < low)) {
#pragma unroll
            for (int c = 0; c < 32; c += 2) pk[(c0 + c) / 2] = 0;
            continue;
          }
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float p0, p1;
            unpack2(fma2(pack2(__uint_as_float(sr[c0 + c]), __uint_as_float(sr[c0 + c + 1])), sl2_2, mb_2), p0, p1);
            p0 = ex2(p0);
            p1 = ex2(p1);
            sum += p0 + p1;
            __nv_bfloat162 b2 = __floats2bfloat162_rn(p0, p1);
            pk[(c0 + c) / 2] = *reinterpret_cast<uint32_t*>(&b2);
          }
        }
        l_run += sum;
        // the P V before has retired: P may be overwritten, and O rescaled or read
        if (g > 0 && !(ok = wait(b_ofull, g - 1))) break;
        tc_fence_after();
        if (rescale && j > 0) {  // tile 0's P V overwrites O: nothing to rescale yet
#pragma unroll 1
          for (int c0 = 0; c0 < HD; c0 += 32) {
            uint32_t rr[32];
            tmem_ld_32x32(tO + lane_off + (uint32_t)c0, rr);
#pragma unroll
            for (int c = 0; c < 32; c++) rr[c] = __float_as_uint(__uint_as_float(rr[c]) * corr);
            tmem_st_32x32(tO + lane_off + (uint32_t)c0, rr);
          }
          tmem_st_wait();
        }
        if (o_pending) output();
#pragma unroll
        for (int c = 0; c < BN / 2; c += 32)
          tmem_st_32x32(tP + lane_off + (uint32_t)c, reinterpret_cast<const uint32_t(&)[32]>(pk[c]));
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(b_pready);
      }
      if (!ok) break;
      if (OPT && a.sink && m_used > -INFINITY)  // the sink: a term of the denominator without key or value
        l_run += ex2((a.sink_w ? a.sink_w[w.head] : 0.f) * LOG2E - m_used * sl2);
      o_inv = 1.0f / l_run;
      if (OPT && a.head_gate && r < w.rows) o_inv *= a.head_gate[(size_t)(w.row + r) * a.gate_ld + w.head];
      o_row = r < w.rows ? (bf16*)a.out + (size_t)(w.row + r) * a.nh * HD + (size_t)w.head * HD : nullptr;
      o_pending = true;
      ok = next_item(it + 1, w);
    }
    if (ok && o_pending && wait(b_ofull, g - 1)) {
      tc_fence_after();
      output();
    }
  }
  __syncwarp();
  if (*dead) {  // a wait ran out: the copies in flight land before the shared memory is given up
    const unsigned long long t0 = gtime();
    while (gtime() - t0 < TC_DRAIN_NS) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(Cf::TMEM_COLS)
                 : "memory");
  }
  TRACE_EXIT(tr);
}

// ------------------------------------------------------------------ launcher
bool attn_prefill_tc5_enabled() {
  static const bool on = !(getenv("NVLLM_ATTN_PREFILL_TC5") && atoi(getenv("NVLLM_ATTN_PREFILL_TC5")) == 0);
  return on;
}

template <int HD, int OPT>
static cudaError_t prefill_tc5_launch(cudaStream_t st, const AttnArgs& a) {
  using Cf = PtCfg<HD>;
  const int pool_rows = a.pool_blocks * a.nkv * KV_BLOCK;
  const TmaDesc* tq = tma_map_cached(a.q, a.total_rows, a.nh * HD, PT_BM);
  const TmaDesc* tk = tma_map_cached(a.kpool, pool_rows, HD, Cf::BN);
  const TmaDesc* tv = tma_map_cached(a.vpool, pool_rows, HD, Cf::BN);
  if (!tq || !tk || !tv) return cudaErrorInvalidValue;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc5_kernel<HD, OPT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cf::SMEM);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  const int ctas = std::min(a.n_qtiles * a.nh, 2 * std::max(1, a.sm_count));
  (void)launch_k(attn_prefill_tc5_kernel<HD, OPT>, dim3(ctas), dim3(PT_THREADS), Cf::SMEM, st,
                 *reinterpret_cast<const CUtensorMap*>(tq), *reinterpret_cast<const CUtensorMap*>(tk),
                 *reinterpret_cast<const CUtensorMap*>(tv), a, next_trace(13));
  return cudaGetLastError();
}

// needs AttnArgs::pool_blocks / total_rows and a tile list built with 128-query tiles
cudaError_t launch_attn_prefill_tc5(cudaStream_t st, const AttnArgs& a) {
  if (a.n_qtiles <= 0) return cudaSuccess;
  if (a.pool_blocks <= 0 || a.total_rows <= 0) return cudaErrorInvalidValue;
  if (a.window > 0) {
    AttnArgs b = a;
    // (a window past the longest sequence limits nothing, and the masks' differences of positions stay within 32 bits)
    b.window = (int)std::min((long long)a.window, (long long)a.max_blocks * KV_BLOCK);
    return a.hd == 64 ? prefill_tc5_launch<64, 2>(st, b) : prefill_tc5_launch<128, 2>(st, b);
  }
  if (a.sink || a.head_gate) return a.hd == 64 ? prefill_tc5_launch<64, 1>(st, a) : prefill_tc5_launch<128, 1>(st, a);
  return a.hd == 64 ? prefill_tc5_launch<64, 0>(st, a) : prefill_tc5_launch<128, 0>(st, a);
}

}  // namespace nvllm
