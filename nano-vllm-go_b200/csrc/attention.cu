// attention.cu — paged attention (MHA / GQA / MQA) reading K/V straight through
// the scheduler's block tables (block = 256 positions, nanovllm/sequence.go:52).
//
// Semantics follow the reference: scores = (q.k) * scale, causal mask
// j > kv_len - q_len + i (attention.go:164-169,374-380, mqa.go:216-222), row
// softmax, P.V.  The reference writes -1e10 into masked scores; exp(-1e10 - max)
// is exactly 0 in fp32, so skipping those keys is identical.  q head h uses kv
// head h / (n_heads / n_kv_heads) (attention.go:337-339).
//
//  * attn_prefill_kernel: flash-style (online softmax, no S x S score tensor).
//    CTA = 32 queries of one sequence x one head; 4 threads per query each own
//    hd/4 dims; K/V tiles of 64 keys staged in shared memory as fp32.  Bound by the latency of its
//    shared-memory reads and sums.  In small steps, with one or two CTAs per SM, a scheduler has one warp to
//    issue from: there four groups of 128 threads share the keys of a tile (16 each) and merge at the end
//    (prefill_groups has the rule and both sides' times).
//  * attn_decode_kernel: one new token per sequence.  CTA = (sequence, group of
//    GC query heads sharing a kv head, KV split).  HBM-bound: each K/V row is
//    read once with 16-byte loads by hd/8 lanes; online softmax in registers;
//    split partials merged by attn_combine_kernel.
#include <stdlib.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace nvllm {

constexpr int PF_KT = 64;  // keys per shared-memory tile (divides KV_BLOCK)
constexpr size_t pf_smem(int hd, int groups) {  // K and V tiles; then the groups' results: m, l and a row each
  return sizeof(float) * std::max((size_t)2 * PF_KT * hd, (size_t)(groups - 1) * ATTN_PREFILL_QTILE * (hd + 4));
}

// the groups' results of a query (maximum, sum, row; 4 threads each) meet in the first one
template <int HD, int GROUPS>
__device__ __forceinline__ void merge_groups(float* smem, int grp, int qi, int sub, float m, float& l, float (&acc)[HD / 4]) {
  constexpr int NV = HD / 16;
  __syncthreads();
  if (grp > 0) {
    float* mine = smem + ((size_t)(grp - 1) * ATTN_PREFILL_QTILE + qi) * (HD + 4);
    if (sub == 0) {
      mine[HD] = m;
      mine[HD + 1] = l;
    }
#pragma unroll
    for (int v = 0; v < NV; v++)
      *reinterpret_cast<float4*>(mine + v * 16 + sub * 4) = make_float4(acc[v * 4], acc[v * 4 + 1], acc[v * 4 + 2], acc[v * 4 + 3]);
  }
  __syncthreads();
  if (grp > 0) return;
  // (key 0 is the first group's: a valid query's m is finite)
  const float* other[GROUPS - 1];
  float top = m;
#pragma unroll
  for (int g = 0; g < GROUPS - 1; g++) {
    other[g] = smem + ((size_t)g * ATTN_PREFILL_QTILE + qi) * (HD + 4);
    top = fmaxf(top, other[g][HD]);
  }
  const float c0 = expf(m - top);
  l *= c0;
#pragma unroll
  for (int i = 0; i < HD / 4; i++) acc[i] *= c0;
#pragma unroll
  for (int g = 0; g < GROUPS - 1; g++) {
    const float c = expf(other[g][HD] - top);  // a group that saw no key: exp(-inf) = 0
    l = fmaf(other[g][HD + 1], c, l);
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const float4 o = *reinterpret_cast<const float4*>(other[g] + v * 16 + sub * 4);
      acc[v * 4] = fmaf(o.x, c, acc[v * 4]);
      acc[v * 4 + 1] = fmaf(o.y, c, acc[v * 4 + 1]);
      acc[v * 4 + 2] = fmaf(o.z, c, acc[v * 4 + 2]);
      acc[v * 4 + 3] = fmaf(o.w, c, acc[v * 4 + 3]);
    }
  }
}

template <typename QT, typename KT, int HD, int GROUPS>
__global__ void __launch_bounds__(128 * GROUPS)
attn_prefill_kernel(AttnArgs a) {
  pdl_launch_dependents();
  extern __shared__ float smem[];
  float* Ks = smem;               // [PF_KT][HD]
  float* Vs = smem + PF_KT * HD;  // [PF_KT][HD]
  constexpr int DPT = HD / 4;     // dims per thread
  constexpr int NV = DPT / 4;     // float4 per thread
  const int tile = blockIdx.x;
  const int head = blockIdx.y;
  const int seq = a.tile_seq[tile];
  const int q0 = a.tile_q0[tile];
  const int n_new = a.cu_q[seq + 1] - a.cu_q[seq];
  const int start = a.seq_start[seq];
  const int kvh = head / (a.nh / a.nkv);
  const int grp = threadIdx.x >> 7, qi = (threadIdx.x & 127) >> 2, sub = threadIdx.x & 3;
  const int qidx = q0 + qi;  // index among the new tokens of this sequence
  const bool qvalid = qidx < n_new;
  const int qpos = start + qidx;
  const int row = a.cu_q[seq] + qidx;
  const int* bt = a.block_tables + (size_t)seq * a.max_blocks;

  const int blk0 = bt[0];
  float q[DPT], acc[DPT];
#pragma unroll
  for (int i = 0; i < DPT; i++) acc[i] = 0.f;
  pdl_wait();  // (what is read above came with the step)
  if (qvalid) {
    const QT* qp = (const QT*)a.q + (size_t)row * a.nh * HD + head * HD;
#pragma unroll
    for (int v = 0; v < NV; v++)
#pragma unroll
      for (int j = 0; j < 4; j++) q[v * 4 + j] = to_f32(qp[v * 16 + sub * 4 + j]) * a.scale;
  } else {
#pragma unroll
    for (int i = 0; i < DPT; i++) q[i] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  const int kv_end = min(start + q0 + ATTN_PREFILL_QTILE, start + n_new);  // keys [0, kv_end)
  const KT* kpool = (const KT*)a.kpool;
  const KT* vpool = (const KT*)a.vpool;

  for (int k0 = 0; k0 < kv_end; k0 += PF_KT) {
    const int nk = min(PF_KT, kv_end - k0);
    const int blk = k0 == 0 ? blk0 : bt[k0 / KV_BLOCK];
    const size_t base = (((size_t)blk * a.nkv + kvh) * KV_BLOCK + (k0 % KV_BLOCK)) * HD;
    __syncthreads();
    for (int i = threadIdx.x * 8; i < nk * HD; i += blockDim.x * 8) {
      float v[8];
      load8(kpool + base + i, v);
      store8(Ks + i, v);
      load8(vpool + base + i, v);
      store8(Vs + i, v);
    }
    __syncthreads();
    // causal: key position <= query position.  The trip count must be warp-uniform (the
    // shuffles below name all 32 lanes), so every lane runs to the warp's largest jmax and
    // masks its own tail.
    const int jmax = qvalid ? max(0, min(nk, qpos - k0 + 1)) : 0;
    const int jlim = min(__reduce_max_sync(0xffffffffu, jmax), (grp + 1) * (PF_KT / GROUPS));
    for (int j0 = grp * (PF_KT / GROUPS); j0 < jlim; j0 += 8) {
      float s[8];
      float cmax = -INFINITY;
#pragma unroll
      for (int jj = 0; jj < 8; jj++) {
        const int j = j0 + jj;
        float d = 0.f;
        if (j < jmax) {
          const float* kr = Ks + j * HD + sub * 4;
#pragma unroll
          for (int v = 0; v < NV; v++) {
            float4 k4 = *reinterpret_cast<const float4*>(kr + v * 16);
            d = fmaf(q[v * 4 + 0], k4.x, d);
            d = fmaf(q[v * 4 + 1], k4.y, d);
            d = fmaf(q[v * 4 + 2], k4.z, d);
            d = fmaf(q[v * 4 + 3], k4.w, d);
          }
        }
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        s[jj] = (j < jmax) ? d : -INFINITY;
        cmax = fmaxf(cmax, s[jj]);
      }
      if (cmax == -INFINITY) continue;  // nothing visible to this query in the chunk (no shuffles below)
      const float m_new = fmaxf(m, cmax);
      const float corr = __expf(m - m_new);  // m = -inf on the first chunk -> 0
      l *= corr;
#pragma unroll
      for (int i = 0; i < DPT; i++) acc[i] *= corr;
#pragma unroll
      for (int jj = 0; jj < 8; jj++) {
        const int j = j0 + jj;
        if (j < jmax) {
          const float p = expf(s[jj] - m_new);
          l += p;
          const float* vr = Vs + j * HD + sub * 4;
#pragma unroll
          for (int v = 0; v < NV; v++) {
            float4 v4 = *reinterpret_cast<const float4*>(vr + v * 16);
            acc[v * 4 + 0] = fmaf(p, v4.x, acc[v * 4 + 0]);
            acc[v * 4 + 1] = fmaf(p, v4.y, acc[v * 4 + 1]);
            acc[v * 4 + 2] = fmaf(p, v4.z, acc[v * 4 + 2]);
            acc[v * 4 + 3] = fmaf(p, v4.w, acc[v * 4 + 3]);
          }
        }
      }
      m = m_new;
    }
  }
  if constexpr (GROUPS > 1) merge_groups<HD, GROUPS>(smem, grp, qi, sub, m, l, acc);
  if (grp == 0 && qvalid) {
    const float inv = 1.0f / l;
    QT* op = (QT*)a.out + (size_t)row * a.nh * HD + head * HD;
#pragma unroll
    for (int v = 0; v < NV; v++)
#pragma unroll
      for (int j = 0; j < 4; j++) op[v * 16 + sub * 4 + j] = from_f32<QT>(acc[v * 4 + j] * inv);
  }
}

// How many groups share a tile's keys.  With four, an SM holds one CTA (two of heads up to 32) and a CTA is through a tile in
// 0.6 of the time; with one it holds six, and a full chip gets through more tiles.  So four while the time is that of the
// longest CTA: x = all CTAs' tiles over SMs x the longest one's up to 1.0 where that is one tile, and to 2.8 (4 for heads up
// to 32) from six on; and one up to 32 keys, of which two groups would have none.  Time with four over time with one, whole
// fp32 steps of four layers of 768, x in front; heads: 12 of 64, 32 of 64, 12 of 32, 16 of 128:
//    9 tokens         0.06 1.10   0.17 1.14   0.06 1.07   0.08 1.01      2 x 300    0.96 0.91   2.56 0.97   0.96 0.81   1.28 0.89
//   48                0.17 0.95   0.45 0.99   0.17 0.94   0.22 0.92      6 x 300    2.87 1.01   7.67 1.16   2.87 0.97   3.83 1.03
//    4 x 40           0.62 0.90   1.64 1.05   0.62 0.97   0.82 0.96      1000       1.36 0.70   3.63 1.04   1.36 0.61   1.81 0.95
//   16 x 40           2.47 1.10   6.57 1.22   2.47 1.02   3.29 1.09      3 x 1000   4.08 1.04   10.9 1.17   4.08 0.90   5.44 1.02
//    8 x 80           1.24 1.03   3.31 1.18   1.24 0.94   1.66 1.07      2000       2.60 0.85   6.92 1.08   2.60 0.81   3.46 0.94
//    2 x 130          0.43 0.83   1.14 0.91   0.43 0.88   0.57 0.89      2 x 2000   5.19 1.04   13.8 1.16   5.19 0.95   6.92 1.02
static int prefill_groups(const AttnArgs& a) {
  if (a.max_len <= PF_KT / 2) return 1;
  const double longest = ceil_div(a.max_len, PF_KT);
  const double tiles = a.nh * (a.pairs / (ATTN_PREFILL_QTILE * PF_KT) + 0.75 * a.n_qtiles);  // (a CTA's last tile is half full)
  const double most = std::min(0.6 + 0.4 * longest, a.hd <= 32 ? 4.0 : 2.8);
  return tiles <= most * longest * std::max(1, a.sm_count) ? 4 : 1;
}

template <typename QT, typename KT, int HD, int GROUPS>
static cudaError_t prefill_launch(cudaStream_t st, const AttnArgs& a) {
  constexpr size_t smem = pf_smem(HD, GROUPS);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(attn_prefill_kernel<QT, KT, HD, GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  (void)launch_k(attn_prefill_kernel<QT, KT, HD, GROUPS>, dim3(a.n_qtiles, a.nh), dim3(128 * GROUPS), smem, st, a);
  return cudaGetLastError();
}
template <typename QT, typename KT, int HD>
static cudaError_t prefill_hd(cudaStream_t st, const AttnArgs& a) {
  return prefill_groups(a) == 4 ? prefill_launch<QT, KT, HD, 4>(st, a) : prefill_launch<QT, KT, HD, 1>(st, a);
}
template <typename QT, typename KT>
static cudaError_t prefill_dispatch(cudaStream_t st, const AttnArgs& a) {
  switch (a.hd) {
    case 16: return prefill_hd<QT, KT, 16>(st, a);
    case 32: return prefill_hd<QT, KT, 32>(st, a);
    case 64: return prefill_hd<QT, KT, 64>(st, a);
    case 128: return prefill_hd<QT, KT, 128>(st, a);
    default: return cudaErrorInvalidValue;
  }
}

int attn_prefill_qtile(int qdt, int kvdt, int hd) {
  if (attn_mma_supported(qdt, kvdt, hd)) return attn_prefill_tc5_enabled() ? 128 : 64;
  return ATTN_PREFILL_QTILE;
}

int attn_decode_splits(int qdt, int kvdt, int n_seqs, int nh, int nkv, int hd, int max_len,
                       long long sum_len, int sm_count) {
  int ctas, max_splits;
  if (attn_mma_supported(qdt, kvdt, hd)) {
    const int G = nh / nkv;
    ctas = n_seqs * nkv * ((G + 15) / 16);
    max_splits = (max_len + attn_decode_mma_tile(hd) - 1) / attn_decode_mma_tile(hd);
    // Where a context is left whole: its second half would cost less than the launch that joins the parts.  The more CTAs
    // there are, the more of their memory time one hides under another's, and the longer that holds.  Resident steps, us
    // split / whole (12 GPT-2 layers, heads by themselves; four Llama-1B layers, groups of four; two of Falcon, one group):
    //   GPT-2    1 x 250 226 / 213, 350 230 / 220, 500 225 / 228    4 x 250 256 / 242, 420 251 / 258    8 x 450 302 / 270, 900 319 / 306
    //   Llama    1 x 250 196 / 190, 500 190 / 192    8 x 500 189 / 182, 1500 206 / 202, 2500 219 / 226    16 x 700 221 / 205, 2500 256 / 254
    //            24 x 1500 250 / 228    32 x 1000 240 / 219
    //   Falcon   8 x 250 197 / 195, 700 200 / 202    16 x 700 210 / 217
    // The others' work has to be there for that: the longest context may exceed what they keep the chip busy with (mean * ctas
    // / 300 tokens of one CTA's time; twice that at head size 128, with twice the bytes) by the cost of the launch and of the
    // parts' own starts (800 tokens, and 6 per CTA).  One context of the first length, the others as long / half / a quarter /
    // a twentieth, us split / whole:
    //   Llama-1B  16 x 2000  245 / 242  233 / 233  225 / 229  220 / 226     32 x 4000  348 / 330  293 / 294  268 / 279  248 / 266
    //             36 x 4000  384 / 366  318 / 320  289 / 299  265 / 285
    //   head size 128 (two Llama-3B layers)
    //              7 x 500   149 / 138  148 / 136  147 / 137  145 / 136     14 x 1500  175 / 159  164 / 156  161 / 155  158 / 154
    //             16 x 2000  186 / 171  172 / 165  166 / 163  162 / 162     28 x 4000  298 / 281  226 / 236  201 / 215  184 / 198
    // (Not met by it: 160 to 230 CTAs of head size 128, some SMs with twice the CTAs of the others: 20 x 3000 229 / 239 stays
    // whole, and so does 28 x 4000 with halves.)
    const int whole = G > 8 ? 256 : 352;
    const double rest = (double)sum_len / n_seqs * ctas * hd / (300 * 64);
    if (max_len <= whole || (G <= 8 && ctas >= 56 && max_len <= min(20.0 * ctas, 800 + 6.0 * ctas + rest))) return 1;
  } else {
    const int G = nh / nkv;
    int gc = 1;
    for (int c = 4; c >= 1; c--)
      if (G % c == 0) {
        gc = c;
        break;
      }
    ctas = n_seqs * (nh / gc);
    max_splits = (max_len + 255) / 256;
  }
  int ns = (2 * sm_count + ctas - 1) / ctas;
  ns = min(ns, max_splits);
  return max(1, min(ns, 32));
}

cudaError_t launch_attn_prefill(cudaStream_t st, const AttnArgs& a) {
  if (a.n_qtiles <= 0) return cudaSuccess;
  if (attn_mma_supported(a.qdt, a.kvdt, a.hd)) {
    if (attn_prefill_tc5_enabled() && a.pool_blocks > 0 && a.total_rows > 0)
      return launch_attn_prefill_tc5(st, a);
    return launch_attn_prefill_mma(st, a);
  }
  if (a.qdt == DT_F32 && a.kvdt == DT_F32) return prefill_dispatch<float, float>(st, a);
  if (a.qdt == DT_F32 && a.kvdt == DT_BF16) return prefill_dispatch<float, bf16>(st, a);
  if (a.qdt == DT_BF16 && a.kvdt == DT_BF16) return prefill_dispatch<bf16, bf16>(st, a);
  return cudaErrorInvalidValue;
}

// ------------------------------------------------------------------- decode
// split partial record: [hd] unnormalised accumulator, then m, l
template <typename QT, typename KT, int HD, int GC>
__global__ void __launch_bounds__(128)
attn_decode_kernel(AttnArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int LPT = HD / 8;    // lanes per token row
  constexpr int TPI = 32 / LPT;  // token rows per warp iteration
  constexpr int NW = 4;
  __shared__ float sm_acc[NW][GC][HD];
  __shared__ float sm_ml[NW][GC][2];
  const int seq = blockIdx.x;
  const int hg = blockIdx.y;  // group of GC consecutive q heads
  const int split = blockIdx.z;
  const int h0 = hg * GC;
  const int kvh = h0 / (a.nh / a.nkv);
  const int len = a.seq_len[seq];
  int chunk = (len + a.n_splits - 1) / a.n_splits;
  chunk = ((chunk + 63) / 64) * 64;
  const int t0 = split * chunk;
  const int t1 = min(len, t0 + chunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = lane / LPT, sub = lane % LPT;
  const int* bt = a.block_tables + (size_t)seq * a.max_blocks;
  const KT* kpool = (const KT*)a.kpool;
  const KT* vpool = (const KT*)a.vpool;

  float q[GC][8], acc[GC][8], m[GC], l[GC];
  const QT* qp = (const QT*)a.q + (size_t)seq * a.nh * HD + h0 * HD + sub * 8;
#pragma unroll
  for (int g = 0; g < GC; g++) {
    load8(qp + g * HD, q[g]);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      q[g][i] *= a.scale;
      acc[g][i] = 0.f;
    }
    m[g] = -INFINITY;
    l[g] = 0.f;
  }
  // warp-uniform trip count (the shuffles name all 32 lanes); lanes past t1 are masked
  for (int tb = t0 + warp * TPI; tb < t1; tb += NW * TPI) {
    const int t = tb + slot;
    const bool valid = t < t1;
    const int tc = valid ? t : t1 - 1;
    const int blk = bt[tc / KV_BLOCK];
    const size_t off = (((size_t)blk * a.nkv + kvh) * KV_BLOCK + (tc % KV_BLOCK)) * HD + sub * 8;
    float k[8], v[8];
    load8(kpool + off, k);
    load8(vpool + off, v);
#pragma unroll
    for (int g = 0; g < GC; g++) {
      float d = 0.f;
#pragma unroll
      for (int i = 0; i < 8; i++) d = fmaf(q[g][i], k[i], d);
#pragma unroll
      for (int o = 1; o < LPT; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if (!valid) continue;
      if (d > m[g]) {  // rescale only when the running max moves
        const float corr = __expf(m[g] - d);
        l[g] *= corr;
#pragma unroll
        for (int i = 0; i < 8; i++) acc[g][i] *= corr;
        m[g] = d;
      }
      const float p = expf(d - m[g]);
      l[g] += p;
#pragma unroll
      for (int i = 0; i < 8; i++) acc[g][i] = fmaf(p, v[i], acc[g][i]);
    }
  }
  // merge the TPI token slots of the warp (lanes with equal `sub`)
#pragma unroll
  for (int g = 0; g < GC; g++) {
#pragma unroll
    for (int o = LPT; o < 32; o <<= 1) {
      const float mo = __shfl_xor_sync(0xffffffffu, m[g], o);
      const float lo = __shfl_xor_sync(0xffffffffu, l[g], o);
      const float mn = fmaxf(m[g], mo);
      const float c0 = (m[g] == -INFINITY) ? 0.f : __expf(m[g] - mn);
      const float c1 = (mo == -INFINITY) ? 0.f : __expf(mo - mn);
      l[g] = l[g] * c0 + lo * c1;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float ao = __shfl_xor_sync(0xffffffffu, acc[g][i], o);
        acc[g][i] = acc[g][i] * c0 + ao * c1;
      }
      m[g] = mn;
    }
    if (slot == 0) {
#pragma unroll
      for (int i = 0; i < 8; i++) sm_acc[warp][g][sub * 8 + i] = acc[g][i];
      if (sub == 0) {
        sm_ml[warp][g][0] = m[g];
        sm_ml[warp][g][1] = l[g];
      }
    }
  }
  __syncthreads();
  // merge the 4 warps; thread d handles dim d of every head of the group
  for (int idx = threadIdx.x; idx < GC * HD; idx += blockDim.x) {
    const int g = idx / HD, d = idx % HD;
    float mn = -INFINITY;
#pragma unroll
    for (int w = 0; w < NW; w++) mn = fmaxf(mn, sm_ml[w][g][0]);
    float lt = 0.f, at = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) {
      const float mw = sm_ml[w][g][0];
      const float c = (mw == -INFINITY) ? 0.f : __expf(mw - mn);
      lt += sm_ml[w][g][1] * c;
      at += sm_acc[w][g][d] * c;
    }
    const int h = h0 + g;
    if (a.n_splits == 1) {
      ((QT*)a.out)[(size_t)seq * a.nh * HD + h * HD + d] = from_f32<QT>(at / lt);
    } else {
      float* rec = a.ws + (((size_t)seq * a.nh + h) * a.n_splits + split) * (HD + 2);
      rec[d] = at;
      if (d == 0) {
        rec[HD] = mn;
        rec[HD + 1] = lt;
      }
    }
  }
}

template <typename QT>
__global__ void attn_combine_kernel(AttnArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.x, h = blockIdx.y, HD = a.hd;
  const float* rec0 = a.ws + (((size_t)seq * a.nh + h) * a.n_splits) * (HD + 2);
  float mn = -INFINITY;
  for (int s = 0; s < a.n_splits; s++) mn = fmaxf(mn, rec0[(size_t)s * (HD + 2) + HD]);
  for (int d = threadIdx.x; d < HD; d += blockDim.x) {
    float lt = 0.f, at = 0.f;
    for (int s = 0; s < a.n_splits; s++) {
      const float* rec = rec0 + (size_t)s * (HD + 2);
      const float ms = rec[HD];
      const float c = (ms == -INFINITY) ? 0.f : __expf(ms - mn);
      lt += rec[HD + 1] * c;
      at += rec[d] * c;
    }
    ((QT*)a.out)[(size_t)seq * a.nh * HD + h * HD + d] = from_f32<QT>(at / lt);
  }
  TRACE_EXIT(tr);
}

template <typename QT, typename KT, int HD>
static cudaError_t decode_dispatch_gc(cudaStream_t st, const AttnArgs& a) {
  const int G = a.nh / a.nkv;
  int gc = 1;
  for (int c = 4; c >= 1; c--)
    if (G % c == 0) {
      gc = c;
      break;
    }
  dim3 grid(a.n_seqs, a.nh / gc, a.n_splits);
  switch (gc) {
    case 4: (void)launch_k(attn_decode_kernel<QT, KT, HD, 4>, dim3(grid), dim3(128), 0, st, a); break;
    case 3: (void)launch_k(attn_decode_kernel<QT, KT, HD, 3>, dim3(grid), dim3(128), 0, st, a); break;
    case 2: (void)launch_k(attn_decode_kernel<QT, KT, HD, 2>, dim3(grid), dim3(128), 0, st, a); break;
    default: (void)launch_k(attn_decode_kernel<QT, KT, HD, 1>, dim3(grid), dim3(128), 0, st, a); break;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (a.n_splits > 1) {
    (void)launch_k(attn_combine_kernel<QT>, dim3(dim3(a.n_seqs, a.nh)), dim3(min(128, a.hd)), 0, st, a, next_trace(14));
    e = cudaGetLastError();
  }
  return e;
}
template <typename QT, typename KT>
static cudaError_t decode_dispatch(cudaStream_t st, const AttnArgs& a) {
  switch (a.hd) {
    case 16: return decode_dispatch_gc<QT, KT, 16>(st, a);
    case 32: return decode_dispatch_gc<QT, KT, 32>(st, a);
    case 64: return decode_dispatch_gc<QT, KT, 64>(st, a);
    case 128: return decode_dispatch_gc<QT, KT, 128>(st, a);
  }
  return cudaErrorInvalidValue;
}

// true: launch_attn_decode takes the QKV GEMM partials (AttnArgs::qkv_p) and does the RoPE +
// KV append of the decoded token itself; the caller then skips launch_rope_kv
bool attn_decode_fuses_rope(int qdt, int kvdt, int hd) {
  static const bool on = [] {
    const char* e = getenv("NVLLM_FUSE_ROPE");
    return e ? atoi(e) != 0 : true;
  }();
  return on && attn_mma_supported(qdt, kvdt, hd);
}

cudaError_t launch_attn_decode(cudaStream_t st, const AttnArgs& a) {
  if (a.n_seqs <= 0) return cudaSuccess;
  if (a.qkv_p && !attn_decode_fuses_rope(a.qdt, a.kvdt, a.hd)) return cudaErrorInvalidValue;
  if (attn_mma_supported(a.qdt, a.kvdt, a.hd)) {
    // small head groups: TMA-fed, keys-as-M-rows kernel (attention_dec.cu); Falcon's 71-head
    // MQA group keeps the 16-query-row kernel
    cudaError_t e = attn_decode_t_supported(a) ? launch_attn_decode_t(st, a)
                                               : launch_attn_decode_mma(st, a);
    if (e != cudaSuccess || a.n_splits == 1) return e;
    (void)launch_k(attn_combine_kernel<bf16>, dim3(dim3(a.n_seqs, a.nh)), dim3(min(128, a.hd)), 0, st, a, next_trace(14));
    return cudaGetLastError();
  }
  if (a.qdt == DT_F32 && a.kvdt == DT_F32) return decode_dispatch<float, float>(st, a);
  if (a.qdt == DT_F32 && a.kvdt == DT_BF16) return decode_dispatch<float, bf16>(st, a);
  if (a.qdt == DT_BF16 && a.kvdt == DT_BF16) return decode_dispatch<bf16, bf16>(st, a);
  return cudaErrorInvalidValue;
}

}  // namespace nvllm
