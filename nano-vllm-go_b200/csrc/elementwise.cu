// elementwise.cu — HBM-bound kernels of the forward pass: embedding gather,
// fused residual-add + LayerNorm/RMSNorm, SwiGLU/GELU, RoPE + paged KV append,
// on-device sampling, weight repack.  All accesses are 16-byte vectors over the
// contiguous (hidden) dimension; one CTA per token row.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "moe_route.cuh"
#include "kernels.h"

namespace nvllm {

// ------------------------------------------------------------------ embedding
// generic_model.go:567-592 embedWithOffset + :298-302 EmbeddingMultiplier
template <typename WT>
__global__ void embed_kernel(const int* __restrict__ tokens, const int* __restrict__ positions,
                             const WT* __restrict__ wte, const WT* __restrict__ wpe, int max_pos,
                             float mult, float* __restrict__ x, int H, bf16* __restrict__ xb,
                             float* __restrict__ ssq, const float* __restrict__ g,
                             const double* __restrict__ pos_freq, WT* __restrict__ y, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_wait();  // step prologue: later kernels may read the step state before their own wait
  pdl_launch_dependents();
  __shared__ float red[32];
  float lsq = 0.f;
  const int t = blockIdx.x;
  const int tok = tokens[t];
  const int pos = positions[t];
  const WT* er = wte + (size_t)tok * H;
  const bool add_pos = (wpe != nullptr) && (pos < max_pos);
  const WT* pr = add_pos ? wpe + (size_t)pos * H : nullptr;
  for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
    float v[8];
    load8(er + i, v);
    if (add_pos) {
      float p[8];
      load8(pr + i, p);
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] += p[j];
    }
    if (mult != 0.f) {
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] *= mult;
    }
    if (pos_freq) {
      // sinusoidal positions: entries (2k, 2k + 1) get sin / cos of pos * pos_freq[k]
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        double sn, cs;
        sincos((double)pos * pos_freq[(i + j) >> 1], &sn, &cs);
        v[j] += (float)sn;
        v[j + 1] += (float)cs;
      }
    }
    store8(x + (size_t)t * H + i, v);
    if (y) store8(y + (size_t)t * H + i, v);
    if (xb) {
      float gv[8], o[8];
      load8(g + i, gv);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        lsq += v[j] * v[j];
        o[j] = v[j] * gv[j];
      }
      store8(xb + (size_t)t * H + i, o);
    }
  }
  if (xb) {
    const float tot = block_sum(lsq, red);
    if (threadIdx.x == 0) ssq[t] = tot;
  }
  TRACE_EXIT(tr);
}

// The same for prompts: a warp per row, four neighbouring entries per lane (whole sectors in every access), eight pieces of the
// row in flight, no block barriers.  Bound by memory.  24 k rows of 2048, bf16 copy and sums of squares: 174 -> 95 us; 18.7 k of
// 1024 50 -> 23.  A row's chain is eight times as long as in a block of its own, so there have to be enough of them: twelve to
// an SM, and with sines (fp64, which a warp computes one piece after another) sixty-four.  A block / a warp per row, us:
//   rows                1024         1536         1792         2048         4096         8192        16000        24000
//   width  768       2.0 / 4.6    2.5 / 4.5    4.9 / 4.5    6.6 / 4.7   10.7 / 8.5   19.9 / 12.9
//         2048       5.9 / 9.3    8.9 / 9.7   10.3 / 9.2   11.9 / 9.3   22.9 / 19.8  45.7 / 29.2
//         4544       7.6 / 8.9   10.8 / 9.1   11.7 / 9.2   14.5 / 10.1  27.5 / 22.6  54.0 / 36.4
//         2048, sines 6.4 / 14.7  8.9 / 14.9               11.9 / 14.8  22.4 / 31.1  45.5 / 45.0  85.4 / 75.2  130 / 112
constexpr int EMBED_WARPS = 8, EMBED_MIN_ROWS = 12 * 148, EMBED_MIN_ROWS_SINES = 64 * 148;
template <typename WT>
__global__ void __launch_bounds__(32 * EMBED_WARPS) embed_rows_kernel(const int* __restrict__ tokens, const int* __restrict__ positions, int T,
                                                                      const WT* __restrict__ wte, const WT* __restrict__ wpe, int max_pos,
                                                                      float mult, float* __restrict__ x, int H, bf16* __restrict__ xb,
                                                                      float* __restrict__ ssq, const float* __restrict__ g,
                                                                      const double* __restrict__ pos_freq, WT* __restrict__ y, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_wait();  // step prologue, as above
  pdl_launch_dependents();
  constexpr int U = 8;
  const int lane = threadIdx.x & 31, t = blockIdx.x * EMBED_WARPS + (threadIdx.x >> 5);
  if (t < T) {
    const int tok = tokens[t], pos = positions[t];
    const WT* er = wte + (size_t)tok * H;
    const WT* pr = wpe != nullptr && pos < max_pos ? wpe + (size_t)pos * H : nullptr;
    auto get = [](const WT* p, float (&o)[4]) {
      if constexpr (sizeof(WT) == 4) {
        const float4 f = *reinterpret_cast<const float4*>(p);
        o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
      } else {
        const uint2 u = *reinterpret_cast<const uint2*>(p);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
      }
    };
    float lsq = 0.f;
    for (int i0 = 4 * lane; i0 < H; i0 += 128 * U) {
      float v[U][4];
#pragma unroll
      for (int u = 0; u < U; u++)
        if (i0 + 128 * u < H) get(er + i0 + 128 * u, v[u]);
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + 128 * u;
        if (i >= H) break;
        if (pr) {
          float p[4];
          get(pr + i, p);
#pragma unroll
          for (int j = 0; j < 4; j++) v[u][j] += p[j];
        }
        if (mult != 0.f) {
#pragma unroll
          for (int j = 0; j < 4; j++) v[u][j] *= mult;
        }
        if (pos_freq) {
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            double sn, cs;
            sincos((double)pos * pos_freq[(i + j) >> 1], &sn, &cs);
            v[u][j] += (float)sn;
            v[u][j + 1] += (float)cs;
          }
        }
        store4(x + (size_t)t * H + i, v[u]);
        if (y) store4(y + (size_t)t * H + i, v[u]);
        if (xb) {
          const float4 gv = *reinterpret_cast<const float4*>(g + i);
          const float o[4] = {v[u][0] * gv.x, v[u][1] * gv.y, v[u][2] * gv.z, v[u][3] * gv.w};
#pragma unroll
          for (int j = 0; j < 4; j++) lsq += v[u][j] * v[u][j];
          store4(xb + (size_t)t * H + i, o);
        }
      }
    }
    if (xb) {
      lsq = warp_sum(lsq);
      if (lane == 0) ssq[t] = lsq;
    }
  }
  TRACE_EXIT(tr);
}

cudaError_t launch_embed(cudaStream_t st, int wdt, const int* tokens, const int* positions,
                         const void* wte, const void* wpe, int max_pos, float mult, float* x, int T,
                         int H, void* xb, float* ssq, const float* g, const double* pos_freq, void* y) {
  if (T <= 0) return cudaSuccess;
  if ((xb == nullptr) != (ssq == nullptr) || (xb && !g)) return cudaErrorInvalidValue;
  if (T >= (pos_freq ? EMBED_MIN_ROWS_SINES : EMBED_MIN_ROWS) && H % 8 == 0) {
    const dim3 grid(ceil_div(T, EMBED_WARPS)), block(32 * EMBED_WARPS);
    return wdt == DT_F32 ? launch_k(embed_rows_kernel<float>, grid, block, 0, st, tokens, positions, T, (const float*)wte, (const float*)wpe,
                                    max_pos, mult, x, H, (bf16*)xb, ssq, g, pos_freq, (float*)y, next_trace(5))
                         : launch_k(embed_rows_kernel<bf16>, grid, block, 0, st, tokens, positions, T, (const bf16*)wte, (const bf16*)wpe,
                                    max_pos, mult, x, H, (bf16*)xb, ssq, g, pos_freq, (bf16*)y, next_trace(5));
  }
  int threads = min(256, max(32, ((H / 8 + 31) / 32) * 32));
  if (wdt == DT_F32)
    (void)launch_k(embed_kernel<float>, dim3(T), dim3(threads), 0, st, tokens, positions, (const float*)wte,
                                               (const float*)wpe, max_pos, mult, x, H, (bf16*)xb, ssq, g, pos_freq, (float*)y, next_trace(5));
  else
    (void)launch_k(embed_kernel<bf16>, dim3(T), dim3(threads), 0, st, tokens, positions, (const bf16*)wte,
                                              (const bf16*)wpe, max_pos, mult, x, H, (bf16*)xb, ssq, g, pos_freq, (bf16*)y, next_trace(5));
  return cudaGetLastError();
}

// ------------------------------------------------- fused residual add + norm
// tensor.go:193-250 LayerNorm (RMSNorm when bias == nil), fused with the
// residual combine of generic_model.go:320-326 / :359-365 / :405-416:
//   x <- x + m1 * (sum_s p1[s] + bias1) + m2 * (sum_s p2[s] + bias2);  y = norm(x)
// The updated row is staged in shared memory so x is read once and written once.
// TAPS != 0 (NormArgs::conv_taps; > 0 at compile time, -1 read from the arguments): the normed row passes the
// causal convolution of a step with one row per sequence before it goes out.  Its tail in the state slot was
// last written in an earlier step, which the step's first kernel has waited for: it is fetched, like
// the weights, before this kernel's own dependency resolves.
template <typename YT, int TAPS>
__global__ void __launch_bounds__(512) norm_kernel(NormArgs a, Trace tr) {
  const unsigned long long t_entry = trace_on(tr) ? gtime() : 0ull;
  pdl_launch_dependents();
  extern __shared__ float row[];
  __shared__ float red[32];
  const int H = a.H;
  // norm weights / biases are immutable: fetch the first vector's worth before the
  // dependency resolves (they come from HBM on first touch)
  const int i0 = threadIdx.x * 8;
  float w0[8], b0[8], bias1_0[8], bias2_0[8];
#pragma unroll
  for (int j = 0; j < 8; j++) w0[j] = b0[j] = bias1_0[j] = bias2_0[j] = 0.f;
  if (i0 < H) {
    if (a.y || a.y_f32 || a.post) {
      if (a.w) load8(a.w + i0, w0);
      else
#pragma unroll
        for (int j = 0; j < 8; j++) w0[j] = 1.f;
      if (a.b) load8(a.b + i0, b0);
    }
    if (a.p1 && a.bias1) load8(a.bias1 + i0, bias1_0);
    if (a.p2 && a.bias2) load8(a.bias2 + i0, bias2_0);
  }
  constexpr int KEEP0 = TAPS > 1 ? TAPS - 1 : 1;  // earlier rows fetched ahead
  float tail0[KEEP0][8], cw0[TAPS > 0 ? TAPS : 1][8];
  float* tail = nullptr;
  int cpos = 0;
  if constexpr (TAPS != 0) {
    if (TAPS > 1 || a.conv_taps > 1) {  // (one tap: no earlier rows, a model without state slots)
      tail = a.conv_pool + (size_t)a.conv_slots[blockIdx.x] * a.conv_slot_floats + a.conv_tail_off;
      cpos = a.conv_pos[blockIdx.x];
    }
    if constexpr (TAPS > 0) {
      if (i0 < H) {
#pragma unroll
        for (int j = 0; j < TAPS; j++) load8(a.conv_w + (size_t)j * H + i0, cw0[j]);
#pragma unroll
        for (int j = 0; j + 1 < TAPS; j++) load8(tail + (size_t)j * H + i0, tail0[j]);
      }
    }
  }
  pdl_wait();
  const unsigned long long t_wait = trace_on(tr) ? gtime() : 0ull;
  const int orow = blockIdx.x;
  const int r = a.row_idx ? a.row_idx[orow] - a.row_bias : orow;
  float* xr = a.x + (size_t)r * H;
  if (a.post) {
    // the norm sits on the addend: x <- x + rmsnorm(sum_s p1[s]) * w; y = x in the act dtype
    float lsq = 0.f;
    for (int i = i0; i < H; i += blockDim.x * 8) {
      float acc[8];
      sum_partials8(a.p1 + (size_t)r * H + i, a.S1, a.stride1, acc);
      store8(row + i, acc);
#pragma unroll
      for (int j = 0; j < 8; j++) lsq += acc[j] * acc[j];
    }
    const float inv = 1.0f / sqrtf(block_sum(lsq, red) / (float)H + a.eps);
    YT* yr = a.y ? (YT*)a.y + (size_t)orow * H : nullptr;
    for (int i = i0; i < H; i += blockDim.x * 8) {
      float v[8], w[8];
      load8(xr + i, v);
      if (i == i0) {
#pragma unroll
        for (int j = 0; j < 8; j++) w[j] = w0[j];
      } else {
        load8(a.w + i, w);
      }
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = fmaf(row[i + j] * inv, w[j], v[j]);
      store8(xr + i, v);
      if (yr) store8(yr + i, v);
    }
    if (threadIdx.x == 0 && trace_on(tr)) trace_rec(tr, t_entry, t_wait, 0ull);
    return;
  }
  const bool upd = (a.p1 != nullptr) || (a.p2 != nullptr) || (a.xadd != nullptr) || (a.xadd_table != nullptr);
  const YT* xtab = a.xadd_table ? (const YT*)a.xadd_table + (size_t)a.xadd_tokens[r] * H : nullptr;
  const bool ln = a.b != nullptr || a.centered != 0;  // LayerNorm (with or without the additive term)
  float lsum = 0.f;
  for (int i = i0; i < H; i += blockDim.x * 8) {
    float v[8];
    load8(xr + i, v);
    if (a.p1) {
      float acc[8];
      if (a.comb_rows) {
#pragma unroll
        for (int j = 0; j < 8; j++) acc[j] = 0.f;
        // slot order (moe.go:116-118), four slots at a time: the index / weight loads of all
        // four first, then all four row loads, then the ordered accumulation — two L2 round
        // trips per four slots instead of two per slot
        for (int s0 = 0; s0 < a.comb_k; s0 += 4) {
          int prow[4];
          float cw[4], pv[4][8];
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (s0 + q < a.comb_k) {
              prow[q] = a.comb_rows[(size_t)r * a.comb_k + s0 + q];
              cw[q] = a.comb_w[(size_t)r * a.comb_k + s0 + q];
            }
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (s0 + q < a.comb_k && prow[q] >= 0) load8(a.p1 + (size_t)prow[q] * H + i, pv[q]);
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (s0 + q < a.comb_k && prow[q] >= 0) {
#pragma unroll
              for (int j = 0; j < 8; j++) acc[j] += cw[q] * pv[q][j];
            }
        }
      } else if (a.p1_bf16) {
        load8(reinterpret_cast<const bf16*>(a.p1) + (size_t)r * H + i, acc);
      } else {
        sum_partials8(a.p1 + (size_t)r * H + i, a.S1, a.stride1, acc);
      }
      if (a.bias1) {
        float p[8];
        if (i == i0) {
#pragma unroll
          for (int j = 0; j < 8; j++) p[j] = bias1_0[j];
        } else {
          load8(a.bias1 + i, p);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) acc[j] += p[j];
      }
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = v[j] + a.m1 * acc[j];
    }
    if (a.p2) {
      float acc[8];
      sum_partials8(a.p2 + (size_t)r * H + i, a.S2, a.stride2, acc);
      if (a.bias2) {
        float p[8];
        if (i == i0) {
#pragma unroll
          for (int j = 0; j < 8; j++) p[j] = bias2_0[j];
        } else {
          load8(a.bias2 + i, p);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) acc[j] += p[j];
      }
      const float m2 = a.row_m2 ? a.m2 * a.row_m2[r] : a.m2;
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = v[j] + m2 * acc[j];
    }
    if (a.xadd) {
      float p[8];
      load8(a.xadd + i, p);
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] += p[j];
    }
    if (xtab) {
      float p[8];
      load8(xtab + i, p);
      const float m = a.xadd_mult != 0.f ? a.xadd_mult : 1.f;
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = fmaf(p[j], m, v[j]);
    }
    if (upd && !a.row_idx) store8(xr + i, v);  // (gathered rows may repeat: the last norm, whose input nothing reads again)
    store8(row + i, v);
    if (ln) {
#pragma unroll
      for (int j = 0; j < 8; j++) lsum += v[j];
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) lsum += v[j] * v[j];
    }
  }
  if (a.y == nullptr && a.y_f32 == nullptr) return;
  if (a.plain) {  // no norm: the updated row itself goes out (each thread reads back what it staged)
    YT* yp = (YT*)a.y + (size_t)orow * H;
    for (int i = i0; i < H; i += blockDim.x * 8) {
      float o[8];
      load8(row + i, o);
      store8(yp + i, o);
    }
    if (threadIdx.x == 0 && trace_on(tr)) trace_rec(tr, t_entry, t_wait, 0ull);
    return;
  }
  unsigned long long t_loads = 0ull, t_red = 0ull;
  // eight entries of the normed row -> convolution -> outputs
  auto emit = [&](int i, float (&o)[8]) {
    if constexpr (TAPS != 0) {
      const int taps = TAPS > 0 ? TAPS : a.conv_taps, keep = taps - 1;
      float y[8], prev[8];
#pragma unroll
      for (int e = 0; e < 8; e++) y[e] = o[e];
      auto tap = [&](int j, const float (&u)[8], const float (&cw)[8]) {
#pragma unroll
        for (int e = 0; e < 8; e++) y[e] = fmaf(cw[e], u[e], y[e]);
        if (j > 0) store8(tail + (size_t)(j - 1) * H + i, u);  // this row is one position further back next time
      };
      if constexpr (TAPS > 0) {
        if (i != i0) {
#pragma unroll
          for (int j = 0; j < TAPS; j++) load8(a.conv_w + (size_t)j * H + i, cw0[j]);
#pragma unroll
          for (int j = 0; j + 1 < TAPS; j++) load8(tail + (size_t)j * H + i, tail0[j]);
        }
#pragma unroll
        for (int j = 0; j + 1 < TAPS; j++) {
          if (TAPS - 1 - j > cpos) {  // before the sequence's start: whatever the slot held counts as zero
#pragma unroll
            for (int e = 0; e < 8; e++) tail0[j][e] = 0.f;
          }
          tap(j, tail0[j], cw0[j]);
        }
        tap(TAPS - 1, o, cw0[TAPS - 1]);
      } else {
        float cw[8];
        for (int j = 0; j < keep; j++) {
          load8(a.conv_w + (size_t)j * H + i, cw);
          load8(tail + (size_t)j * H + i, prev);
          if (keep - j > cpos) {
#pragma unroll
            for (int e = 0; e < 8; e++) prev[e] = 0.f;
          }
          tap(j, prev, cw);
        }
        load8(a.conv_w + (size_t)keep * H + i, cw);
        tap(keep, o, cw);
      }
#pragma unroll
      for (int e = 0; e < 8; e++) o[e] = y[e];
    }
    if (a.y) store8((YT*)a.y + (size_t)orow * H + i, o);
    if (a.y_f32) store8(a.y_f32 + (size_t)orow * H + i, o);
    if (a.router || a.gate_w) store8(row + i, o);  // each thread overwrites only what it alone reads
  };
  if (a.groups > 1 && !ln) {
    // RMS norm in equal parts: a warp sums the squares of one part at a time
    __shared__ float ginv[64];
    __syncthreads();
    const int part = H / a.groups;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int g = warp; g < a.groups; g += nw) {
      float sq = 0.f;
      for (int i = lane; i < part; i += 32) {
        const float v = row[g * part + i];
        sq = fmaf(v, v, sq);
      }
      sq = warp_sum(sq);
      if (lane == 0) ginv[g] = 1.0f / sqrtf(sq / (float)part + a.eps);
    }
    __syncthreads();
    for (int i = i0; i < H; i += blockDim.x * 8) {
      float w[8], o[8];
      if (i == i0) {
#pragma unroll
        for (int j = 0; j < 8; j++) w[j] = w0[j];
      } else if (a.w) load8(a.w + i, w);
      else
#pragma unroll
        for (int j = 0; j < 8; j++) w[j] = 1.f;
#pragma unroll
      for (int j = 0; j < 8; j++) o[j] = row[i + j] * ginv[(i + j) / part] * w[j];
      emit(i, o);
    }
  } else {
  t_loads = tr.buf ? gtime() : 0ull;
  float tot = block_sum(lsum, red);
  t_red = tr.buf ? gtime() : 0ull;
  float mean = 0.f, inv;
  if (ln) {
    mean = tot / (float)H;
    float lv = 0.f;
    for (int i = i0; i < H; i += blockDim.x * 8) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        float d = row[i + j] - mean;
        lv += d * d;
      }
    }
    float var = block_sum(lv, red) / (float)H;
    inv = 1.0f / sqrtf(var + a.eps);
  } else {
    inv = 1.0f / sqrtf(tot / (float)H + a.eps);
  }
  for (int i = i0; i < H; i += blockDim.x * 8) {
    float w[8], bb[8], o[8];
    if (i == i0) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        w[j] = w0[j];
        bb[j] = b0[j];
      }
    } else {
      if (a.w) load8(a.w + i, w);
      else
#pragma unroll
        for (int j = 0; j < 8; j++) w[j] = 1.f;
      if (a.b) load8(a.b + i, bb);
      else
#pragma unroll
        for (int j = 0; j < 8; j++) bb[j] = 0.f;
    }
    if (ln) {
#pragma unroll
      for (int j = 0; j < 8; j++) o[j] = (row[i + j] - mean) * inv * w[j] + bb[j];
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) o[j] = row[i + j] * inv * w[j];
    }
    emit(i, o);
  }
  }
  if (a.gate_w) {  // one number per token: sigmoid(normed row . gate_w), fp32
    float d = 0.f;
    for (int i = i0; i < H; i += blockDim.x * 8) {
      float g[8];
      load8(a.gate_w + i, g);
#pragma unroll
      for (int j = 0; j < 8; j++) d = fmaf(row[i + j], g[j], d);
    }
    d = block_sum(d, red);
    if (threadIdx.x == 0) a.gate_out[orow] = 1.0f / (1.0f + expf(-d));
  }
  if (a.router) {
    __shared__ float probs[MOE_MAX_E];
    __syncthreads();
    if (a.route.identity > 0) {
      // the chosen identity experts return the row itself: their weight times it joins x here, where both are at hand
      __shared__ float id_w;
      moe_route_row(row, a.router, H, a.E, a.topk, probs, (size_t)orow, a.topk_idx, a.topk_w, a.route, &id_w);
      __syncthreads();
      const float wi = id_w;
      if (wi != 0.f)
        for (int i = i0; i < H; i += blockDim.x * 8) {
          float v[8];
          load8(xr + i, v);  // (this thread's own store above)
#pragma unroll
          for (int j = 0; j < 8; j++) v[j] = fmaf(wi, row[i + j], v[j]);
          store8(xr + i, v);
        }
    } else {
      moe_route_row(row, a.router, H, a.E, a.topk, probs, (size_t)orow, a.topk_idx, a.topk_w, a.route);
    }
  }
  if (threadIdx.x == 0 && trace_on(tr))
    trace_rec(tr, t_entry, t_wait, ((t_loads - t_wait) << 32) | (t_red - t_wait));
}

// The same with a row in registers, four entries per thread and vector, V vectors, and all loads of a row in flight at once,
// the expert rows of a combine (COMB) and up to SL slices of an addend included.  norm_kernel keeps eight entries per
// thread (a warp's 16-byte loads then touch every sector twice), stages the row in shared memory and needs 128 registers
// for all its options.
// Prompts (SL = 1; their addends need no summing over slices): bound by memory.  Per launch inside whole steps: 6446 rows of
// 2048 with one addend 55 -> 31 us (5.9 TB/s); 18 k rows of 2048, norm on the addend 148 -> 86 us; 2048 rows of 4544,
// LayerNorm and two addends 54 -> 24 us; 18.7 k rows of 1024 through combines of eight expert rows and routing 161 -> 140
// us.  From 512 rows on (every SM has more than three).
// Steps of fewer rows (SL = 8): bound by one L2 round trip, two block sums at most and the way in and out of the launch;
// weights and biases are loaded before the dependency resolves.  64 rows of 2048 with eight slices, from the release to the last
// exit: 4.9 -> 2.7 us; 16 decode steps of 64 sequences through four Llama-1B layers 4668 -> 4330 us, of 128 through routed
// experts (every second norm) 5694 -> 5505.  Threads and vectors are such that no form spills (two vectors with the weights
// ahead did; a step of 64 sequences through two Llama-3B layers 147.8 us so, 144.5 without).
constexpr int NR_MAX_V = 4, NR_THREADS = 512, NR_STEP_MAX_V = 5;
constexpr int nr_step_threads(int V, bool comb) { return V <= (comb ? 1 : 2) ? 640 : 512; }
template <typename YT, int V, int COMB, int SL>
__global__ void __launch_bounds__(SL > 1 ? nr_step_threads(V, COMB > 0) : NR_THREADS, SL > 1 ? 1 : 2) norm_rows_kernel(NormArgs a, Trace tr) {
  const unsigned long long t_entry = trace_on(tr) ? gtime() : 0ull;
  pdl_launch_dependents();
  __shared__ float red[32];
  const int H = a.H;
  constexpr bool STEP = SL > 1, AHEAD = STEP && V == 1;  // (two vectors leave no registers for the weights)
  auto get = [](const float* p, float (&o)[4]) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
  };
  float wa[AHEAD ? V : 1][4], ba[AHEAD ? V : 1][4], b1a[AHEAD ? V : 1][4], b2a[AHEAD ? V : 1][4];
  if constexpr (AHEAD) {
#pragma unroll
    for (int k = 0; k < V; k++) {
      const int i = ((int)threadIdx.x + k * (int)blockDim.x) * 4;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        wa[k][j] = 1.f;
        ba[k][j] = b1a[k][j] = b2a[k][j] = 0.f;
      }
      if (i >= H) continue;
      if (a.w) get(a.w + i, wa[k]);
      if (a.b) get(a.b + i, ba[k]);
      if (a.p1 && a.bias1) get(a.bias1 + i, b1a[k]);
      if (a.p2 && a.bias2) get(a.bias2 + i, b2a[k]);
    }
  }
  pdl_wait();
  const unsigned long long t_wait = trace_on(tr) ? gtime() : 0ull;
  const int orow = blockIdx.x;
  const int r = STEP && a.row_idx ? a.row_idx[orow] - a.row_bias : orow;
  float* xr = a.x + (size_t)r * H;
  float v[V][4], acc[V][4];
  int prow[COMB ? COMB : 1];
  float cw[COMB ? COMB : 1];
  if constexpr (COMB > 0) {
#pragma unroll
    for (int q = 0; q < COMB; q++) {
      prow[q] = q < a.comb_k ? a.comb_rows[(size_t)r * a.comb_k + q] : -1;
      cw[q] = q < a.comb_k ? a.comb_w[(size_t)r * a.comb_k + q] : 0.f;
    }
  }
#pragma unroll
  for (int k = 0; k < V; k++) {
    const int i = ((int)threadIdx.x + k * (int)blockDim.x) * 4;
#pragma unroll
    for (int j = 0; j < 4; j++) v[k][j] = acc[k][j] = 0.f;
    if (i >= H) continue;
    get(xr + i, v[k]);
    float p2[4] = {0.f, 0.f, 0.f, 0.f}, b[4];
    float s2[SL][4];
    if (STEP && a.p2 && !a.post) {  // (ahead of the first addend, a load behind a branch costs prompts 0.4 us of 8 a launch)
#pragma unroll
      for (int q = 0; q < SL; q++)
        if (q == 0 || q < a.S2) get(a.p2 + (size_t)q * a.stride2 + (size_t)r * H + i, s2[q]);
    }
    if constexpr (COMB > 0) {
      float pv[COMB][4];
#pragma unroll
      for (int q = 0; q < COMB; q++)
        if (prow[q] >= 0) get(a.p1 + (size_t)prow[q] * H + i, pv[q]);
#pragma unroll
      for (int q = 0; q < COMB; q++)  // slot order (moe.go:116-118)
        if (prow[q] >= 0) {
#pragma unroll
          for (int j = 0; j < 4; j++) acc[k][j] += cw[q] * pv[q][j];
        }
    } else if constexpr (!STEP) {
      if (a.p1) get(a.p1 + (size_t)r * H + i, acc[k]);
    } else if (a.p1) {
      float s1[SL][4];
#pragma unroll
      for (int q = 0; q < SL; q++)
        if (q == 0 || q < a.S1) get(a.p1 + (size_t)q * a.stride1 + (size_t)r * H + i, s1[q]);
#pragma unroll
      for (int q = 0; q < SL; q++)
        if (q == 0 || q < a.S1) {
#pragma unroll
          for (int j = 0; j < 4; j++) acc[k][j] += s1[q][j];
        }
    }
    if (a.post) continue;
    if constexpr (!STEP) {
      if (a.p2) get(a.p2 + (size_t)r * H + i, p2);
    } else if (a.p2) {
#pragma unroll
      for (int q = 0; q < SL; q++)
        if (q == 0 || q < a.S2) {
#pragma unroll
          for (int j = 0; j < 4; j++) p2[j] += s2[q][j];
        }
    }
    if (a.p1 && a.bias1) {
      if constexpr (!AHEAD) get(a.bias1 + i, b);
#pragma unroll
      for (int j = 0; j < 4; j++) acc[k][j] += AHEAD ? b1a[AHEAD ? k : 0][j] : b[j];
    }
    if (a.p2 && a.bias2) {
      if constexpr (!AHEAD) get(a.bias2 + i, b);
#pragma unroll
      for (int j = 0; j < 4; j++) p2[j] += AHEAD ? b2a[AHEAD ? k : 0][j] : b[j];
    }
    if (a.p1)
#pragma unroll
      for (int j = 0; j < 4; j++) v[k][j] = v[k][j] + a.m1 * acc[k][j];
    if (a.p2)
#pragma unroll
      for (int j = 0; j < 4; j++) v[k][j] = v[k][j] + a.m2 * p2[j];
    if ((a.p1 || a.p2) && !(STEP && a.row_idx)) store4(xr + i, v[k]);  // (gathered rows may repeat, see norm_kernel)
  }
  if (a.y || a.y_f32 || a.post) {
    const bool ln = a.b != nullptr || a.centered != 0;
    float part = 0.f;
#pragma unroll
    for (int k = 0; k < V; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) part += a.post ? acc[k][j] * acc[k][j] : ln ? v[k][j] : v[k][j] * v[k][j];  // (zeros past the row)
    const float tot = block_sum(part, red);
    float mean = 0.f, inv;
    if (ln && !a.post) {
      mean = tot / (float)H;
      float lv = 0.f;
#pragma unroll
      for (int k = 0; k < V; k++)
        if (((int)threadIdx.x + k * (int)blockDim.x) * 4 < H) {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const float d = v[k][j] - mean;
            lv += d * d;
          }
        }
      inv = 1.0f / sqrtf(block_sum(lv, red) / (float)H + a.eps);
    } else {
      inv = 1.0f / sqrtf(tot / (float)H + a.eps);
    }
#pragma unroll
    for (int k = 0; k < V; k++) {
      const int i = ((int)threadIdx.x + k * (int)blockDim.x) * 4;
      if (i >= H) continue;
      float w[4] = {1.f, 1.f, 1.f, 1.f}, b[4] = {0.f, 0.f, 0.f, 0.f}, o[4];
      if constexpr (AHEAD) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          w[j] = wa[k][j];
          b[j] = ba[k][j];
        }
      } else {
        if (a.w) get(a.w + i, w);
        if (a.b) get(a.b + i, b);
      }
      if (a.post) {
#pragma unroll
        for (int j = 0; j < 4; j++) o[j] = fmaf(acc[k][j] * inv, w[j], v[k][j]);
        store4(xr + i, o);
      } else if (ln) {
#pragma unroll
        for (int j = 0; j < 4; j++) o[j] = (v[k][j] - mean) * inv * w[j] + b[j];
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) o[j] = v[k][j] * inv * w[j];
      }
      if (a.y) store4((YT*)a.y + (size_t)orow * H + i, o);
      if (a.y_f32 && !a.post) store4(a.y_f32 + (size_t)orow * H + i, o);
    }
  }
  if (threadIdx.x == 0 && trace_on(tr))  // what the row took in: 1 an addend (2: expert rows), 4 a second one, 8 normed on it
    trace_rec(tr, t_entry, t_wait, (a.p1 ? 1ull : 0ull) | (COMB ? 2ull : 0ull) | (a.p2 ? 4ull : 0ull) | (a.post ? 8ull : 0ull));
}
// no option of norm_kernel that these kernels lack; at most eight expert rows
static bool norm_rows_plain(const NormArgs& a) {
  return a.H % 8 == 0 && !a.router && !a.gate_w && !a.plain && a.groups <= 1 && !a.xadd && !a.xadd_table && !a.row_m2 &&
         !a.conv_taps && !a.p1_bf16 && (!a.p1 || !a.comb_rows || a.comb_k <= 8) &&
         (!a.post || (a.p1 && a.w && !a.comb_rows && !a.p2 && !a.row_idx));
}
// many rows, at most one slice per addend
static bool norm_rows_fit(const NormArgs& a) {
  return norm_rows_plain(a) && a.n_rows >= 512 && a.H <= NR_MAX_V * NR_THREADS * 4 && !a.row_idx &&
         (!a.p1 || a.comb_rows || a.S1 == 1) && (!a.p2 || a.S2 == 1);
}
struct NrShape {
  int V, threads;
};
static NrShape nr_shape(int H, bool step, bool comb) {
  NrShape s{1, 0};
  while (H > s.V * 4 * (step ? nr_step_threads(s.V, comb) : NR_THREADS)) s.V++;
  s.threads = ceil_div(ceil_div(H, 4 * s.V), 32) * 32;
  return s;
}
// Few rows, at most eight slices (what the products of a step are split into).  Up to which row: norm_kernel has two CTAs of
// up to 2048 entries on an SM where these take all of its registers, and is ahead from the fourth wave of them on, with
// expert rows from the second; rows of four vectors and more are too long a chain for a second wave.  Whole steps of few
// layers, norm_kernel / these:
//   rows            1            16           64           128          192          256          384          448          511
//   width  768  199 / 198    437 / 363    490 / 425    613 / 548    789 / 734    891 / 828   1143 / 1107  1219 / 1200  1311 / 1298
//         2048  188 / 187    200 / 188    218 / 195    261 / 250    376 / 367    404 / 397    563 / 560    585 / 591    612 / 622
//         3072  144 / 144    134 / 132    150 / 145    179 / 176    247 / 244    268 / 265    389 / 391    414 / 416    432 / 434
//         4544  259 / 259    208 / 202    234 / 228    277 / 272    377 / 367    410 / 403    574 / 565    605 / 591    628 / 615
//         5120  278 / 270    274 / 255    292 / 270    335 / 317    432 / 411    468 / 449    612 / 590    658 / 634    706 / 678
//         6144  332 / 330    295 / 286    313 / 302    360 / 352    458 / 452    497 / 493    655 / 650    707 / 704    747 / 750
//         8192  373 / 378    346 / 343    363 / 360    419 / 418    521 / 527    566 / 575    668 / 663    689 / 687    749 / 748
//        10240  327 / 329    326 / 319    354 / 344    427 / 420    611 / 612    684 / 689    929 / 950    988 /1012   1020 / 1043
//   experts 1024  182 / 172  197 / 189    222 / 213    250 / 244    314 / 309    342 / 337    430 / 429    454 / 455    485 / 485
//           2048  171 / 162  190 / 181    204 / 195    240 / 233    308 / 308    350 / 351    439 / 444    478 / 486    512 / 520
static bool norm_step_fit(const NormArgs& a) {
  if (!norm_rows_plain(a) || a.n_rows >= 512 || a.H > NR_STEP_MAX_V * nr_step_threads(NR_STEP_MAX_V, false) * 4 ||
      (a.p1 && !a.comb_rows && a.S1 > 8) || (a.p2 && a.S2 > 8))
    return false;
  const bool comb = a.p1 && a.comb_rows;
  const NrShape s = nr_shape(a.H, true, comb);
  if (s.V >= 4) return a.n_rows <= 148;
  const bool alone = s.threads * (comb ? 80 : 96) > 32768;  // on its SM, by its registers
  return !alone || a.H > 2048 || a.n_rows <= (comb ? 148 : 3 * 148);
}
template <typename YT, int SL>
static cudaError_t launch_norm_rows(cudaStream_t st, const NormArgs& a) {
  const bool comb = a.p1 && a.comb_rows;
  const auto [V, threads] = nr_shape(a.H, SL > 1, comb);
#define NR(V_)                                                                                                           \
  (comb ? launch_k(norm_rows_kernel<YT, V_, 8, SL>, dim3(a.n_rows), dim3(threads), 0, st, a, next_trace(SL > 1 ? 53 : 47)) \
        : launch_k(norm_rows_kernel<YT, V_, 0, SL>, dim3(a.n_rows), dim3(threads), 0, st, a, next_trace(SL > 1 ? 53 : 47)))
  if constexpr (SL > 1)
    if (V == 5) return NR(5);
  return V == 1 ? NR(1) : V == 2 ? NR(2) : V == 3 ? NR(3) : NR(4);
#undef NR
}

// The step form with the row's routing behind it (mixture-of-experts layers, up to 1024 rows): 16 warps, each the logits of
// experts w, w + 16, ... from the normed row in shared memory.  The first RT_AHEAD 16-byte pieces of a lane's router rows
// are loaded before the dependency resolves (32 experts of 1024: all of them), neighbouring lanes neighbouring pieces, and up to
// 32 experts are chosen with a lane each.  128 rows of 1024 with eight slices and 32 experts, from the release to the last exit:
// 10 -> 5.9 us; with the sort of moe.cu, 16 decode steps of 128 sequences through four layers of 32 experts 5410 -> 5100 us.
// One step of 64 / 192 / 384 / 512 sequences, norm_kernel / this: 222 / 209, 336 / 308, 464 / 420, 524 / 477; prompts of 1008
// rows in all 703 / 638.
constexpr int RT_THREADS = 512, RT_AHEAD = 16, RT_MAX_V = 4;
template <typename YT, int V, int COMB>
__global__ void __launch_bounds__(RT_THREADS, 1) norm_route_kernel(NormArgs a, Trace tr) {
  const unsigned long long t_entry = trace_on(tr) ? gtime() : 0ull;
  pdl_launch_dependents();
  extern __shared__ __align__(16) float row[];
  __shared__ float red[32], probs[MOE_MAX_E], chs[MOE_MAX_E], gsc[MOE_MAX_E];
  const int H = a.H, r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = RT_THREADS / 32;
  auto get = [](const float* p, float (&o)[4]) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
  };
  // piece m of this warp's router rows: expert warp + NW (m / nch), entries 128 (m % nch) + 4 lane
  const int nch = (H + 127) / 128, pieces = (a.E > warp ? (a.E - warp + NW - 1) / NW : 0) * nch;
  auto piece = [&](int j, int c, float (&o)[4]) {
    const int i = 128 * c + 4 * lane;
    o[0] = o[1] = o[2] = o[3] = 0.f;
    if (i < H) get(a.router + (size_t)(warp + NW * j) * H + i, o);
  };
  float ahead[RT_AHEAD][4];
  {
    int j = 0, c = 0;
#pragma unroll
    for (int m = 0; m < RT_AHEAD; m++) {
      if (m < pieces) piece(j, c, ahead[m]);
      if (++c == nch) c = 0, j++;
    }
  }
  pdl_wait();
  const unsigned long long t_wait = trace_on(tr) ? gtime() : 0ull;
  float* xr = a.x + (size_t)r * H;
  int prow[COMB ? COMB : 1];
  float cw[COMB ? COMB : 1];
  if constexpr (COMB > 0) {
#pragma unroll
    for (int q = 0; q < COMB; q++) {
      prow[q] = q < a.comb_k ? a.comb_rows[(size_t)r * a.comb_k + q] : -1;
      cw[q] = q < a.comb_k ? a.comb_w[(size_t)r * a.comb_k + q] : 0.f;
    }
  }
  const bool ln = a.b != nullptr || a.centered != 0;
  float v[V][4], part = 0.f;
#pragma unroll
  for (int k = 0; k < V; k++) {
    const int i = ((int)threadIdx.x + k * RT_THREADS) * 4;
#pragma unroll
    for (int j = 0; j < 4; j++) v[k][j] = 0.f;
    if (i >= H) continue;
    get(xr + i, v[k]);
    if (a.p1) {
      float s1[8][4], acc[4] = {0.f, 0.f, 0.f, 0.f}, b[4];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        if (COMB ? prow[COMB ? q : 0] >= 0 : q < a.S1)
          get(a.p1 + (COMB ? (size_t)prow[COMB ? q : 0] * H : (size_t)q * a.stride1 + (size_t)r * H) + i, s1[q]);
      }
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (COMB ? prow[COMB ? q : 0] >= 0 : q < a.S1) {
#pragma unroll
          for (int j = 0; j < 4; j++) acc[j] += COMB ? cw[COMB ? q : 0] * s1[q][j] : s1[q][j];
        }
      if (a.bias1) {
        get(a.bias1 + i, b);
#pragma unroll
        for (int j = 0; j < 4; j++) acc[j] += b[j];
      }
#pragma unroll
      for (int j = 0; j < 4; j++) v[k][j] = v[k][j] + a.m1 * acc[j];
      store4(xr + i, v[k]);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) part += ln ? v[k][j] : v[k][j] * v[k][j];
  }
  const float tot = block_sum(part, red);
  float mean = 0.f, inv;
  if (ln) {
    mean = tot / (float)H;
    float lv = 0.f;
#pragma unroll
    for (int k = 0; k < V; k++)
      if (((int)threadIdx.x + k * RT_THREADS) * 4 < H) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float d = v[k][j] - mean;
          lv += d * d;
        }
      }
    inv = 1.0f / sqrtf(block_sum(lv, red) / (float)H + a.eps);
  } else {
    inv = 1.0f / sqrtf(tot / (float)H + a.eps);
  }
#pragma unroll
  for (int k = 0; k < V; k++) {
    const int i = ((int)threadIdx.x + k * RT_THREADS) * 4;
    if (i >= H) continue;
    float w[4] = {1.f, 1.f, 1.f, 1.f}, b[4] = {0.f, 0.f, 0.f, 0.f}, o[4];
    if (a.w) get(a.w + i, w);
    if (a.b) get(a.b + i, b);
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = ln ? (v[k][j] - mean) * inv * w[j] + b[j] : v[k][j] * inv * w[j];
    if (a.y) store4((YT*)a.y + (size_t)r * H + i, o);
    if (a.y_f32) store4(a.y_f32 + (size_t)r * H + i, o);
    store4(row + i, o);
  }
  __syncthreads();
  {
    int j = 0, c = 0;
    float acc = 0.f;
    auto take = [&](const float (&p)[4]) {
      const int i = 128 * c + 4 * lane;
      if (i < H) {
        float y[4];
        get(row + i, y);
#pragma unroll
        for (int e = 0; e < 4; e++) acc = fmaf(y[e], p[e], acc);
      }
      if (++c == nch) {
        acc = warp_sum(acc);
        const int e = warp + NW * j;
        if (lane == 0) probs[e] = a.route.bias ? acc + a.route.bias[e] : acc;
        acc = 0.f;
        c = 0;
        j++;
      }
    };
#pragma unroll
    for (int m = 0; m < RT_AHEAD; m++)
      if (m < pieces) take(ahead[m]);
    for (int m = RT_AHEAD; m < pieces; m += 8) {
      float p[8][4];
      int jj = j, cc = c;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        if (m + q < pieces) piece(jj, cc, p[q]);
        if (++cc == nch) cc = 0, jj++;
      }
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (m + q < pieces) take(p[q]);
    }
  }
  __syncthreads();
  if (warp == 0) {
    if (a.E <= 32 && !a.route.correction && !(a.route.groups > 1 && a.route.keep < a.route.groups))
      moe_select_lanes(lane < a.E ? probs[lane] : 0.f, a.E, a.topk, (size_t)r, a.topk_idx, a.topk_w, a.route);
    else
      moe_select_row(probs, chs, gsc, a.E, a.topk, (size_t)r, a.topk_idx, a.topk_w, a.route);
  }
  if (threadIdx.x == 0 && trace_on(tr)) trace_rec(tr, t_entry, t_wait, 0ull);
}
// (identity experts need the row itself again; more rows fill the SMs without 16 warps to a row)
static bool norm_route_fit(const NormArgs& a) {
  return a.router && a.route.identity == 0 && a.n_rows <= 1024 && a.E <= MOE_MAX_E && a.topk <= 32 && a.H % 8 == 0 &&
         a.H <= RT_MAX_V * RT_THREADS * 4 && !a.p2 && !a.row_idx && !a.gate_w && !a.plain && !a.post && a.groups <= 1 && !a.xadd &&
         !a.xadd_table && !a.row_m2 && !a.conv_taps && !a.p1_bf16 && (!a.p1 || (a.comb_rows ? a.comb_k <= 8 : a.S1 <= 8));
}
template <typename YT>
static cudaError_t launch_norm_route(cudaStream_t st, const NormArgs& a) {
  const int V = ceil_div(a.H, RT_THREADS * 4);
  const size_t smem = (size_t)a.H * sizeof(float);
  const bool comb = a.p1 && a.comb_rows;
#define NR(V_)                                                                                                        \
  (comb ? launch_k(norm_route_kernel<YT, V_, 8>, dim3(a.n_rows), dim3(RT_THREADS), smem, st, a, next_trace(54))       \
        : launch_k(norm_route_kernel<YT, V_, 0>, dim3(a.n_rows), dim3(RT_THREADS), smem, st, a, next_trace(54)))
  return V == 1 ? NR(1) : V == 2 ? NR(2) : V == 3 ? NR(3) : NR(4);
#undef NR
}

cudaError_t launch_norm(cudaStream_t st, const NormArgs& a) {
  if (a.n_rows <= 0) return cudaSuccess;
  if (a.groups > 64 || (a.groups > 1 && a.H % a.groups) || (a.plain && !a.y)) return cudaErrorInvalidValue;
  if (norm_rows_fit(a)) return a.ydt == DT_F32 ? launch_norm_rows<float, 1>(st, a) : launch_norm_rows<bf16, 1>(st, a);
  if (norm_step_fit(a)) return a.ydt == DT_F32 ? launch_norm_rows<float, 8>(st, a) : launch_norm_rows<bf16, 8>(st, a);
  if (norm_route_fit(a)) return a.ydt == DT_F32 ? launch_norm_route<float>(st, a) : launch_norm_route<bf16>(st, a);
  int threads = min(512, max(64, ((a.H / 8 + 31) / 32) * 32));
  // fused router, decode-sized batches (latency-bound: fewer row CTAs than two waves): 16 warps
  // so that each takes two experts of a 32-expert layer in one pass; prefill keeps the
  // occupancy of the narrow CTA (measured: 512 threads cost cfg3 prefill 35 -> 44 ms)
  if (a.router && a.n_rows <= 1024) threads = 512;
  size_t smem = (size_t)a.H * sizeof(float);
  if (a.conv_taps < 0 || a.conv_taps > INPUT_CONV_MAX_TAPS || (a.conv_taps > 0 && (a.post || a.plain || a.row_idx)))
    return cudaErrorInvalidValue;
#define NK(TP_)                                                                                                        \
  do {                                                                                                                 \
    if (a.ydt == DT_F32) (void)launch_k(norm_kernel<float, TP_>, dim3(a.n_rows), dim3(threads), smem, st, a, next_trace(2)); \
    else (void)launch_k(norm_kernel<bf16, TP_>, dim3(a.n_rows), dim3(threads), smem, st, a, next_trace(2));             \
  } while (0)
  if (a.conv_taps == 0) NK(0);
  else if (a.conv_taps == 2) NK(2);
  else if (a.conv_taps == 3) NK(3);
  else if (a.conv_taps == 4) NK(4);
  else NK(-1);
#undef NK
  return cudaGetLastError();
}

// ---------------------------------------------------------------- activations
template <typename OT>
__global__ void act_kernel(int T, int F, const float* __restrict__ h, int S, size_t stride,
                           const float* __restrict__ bias, int swiglu, OT* __restrict__ out, float glu_limit,
                           Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  const int act2 = swiglu == 2;  // squared ReLU: a plain (ungated) activation
  if (act2) swiglu = 0;
  const int ld = swiglu ? 2 * F : F;
  const size_t nvec = (size_t)T * (F / 8);
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec;
       v += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(v / (F / 8));
    const int j = (int)(v % (F / 8)) * 8;
    float g[8], o[8];
#pragma unroll
    for (int i = 0; i < 8; i++) g[i] = 0.f;
    if (!swiglu) sum_partials8(h + (size_t)t * ld + j, S, stride, g);
    if (swiglu) {
      // W1 rows are stored interleaved (weights.cu): column 2j = gate j, 2j + 1 = up j
      float a[8], b[8];
      sum_partials8(h + (size_t)t * ld + 2 * j, S, stride, a);
      sum_partials8(h + (size_t)t * ld + 2 * j + 8, S, stride, b);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        o[i] = glu_unit(a[2 * i], a[2 * i + 1], glu_limit);
        o[4 + i] = glu_unit(b[2 * i], b[2 * i + 1], glu_limit);
      }
    } else {
      if (bias) {
        float p[8];
        load8(bias + j, p);
#pragma unroll
        for (int i = 0; i < 8; i++) g[i] += p[i];
      }
#pragma unroll
      for (int i = 0; i < 8; i++) o[i] = act2 ? relu2(g[i]) : gelu_tanh(g[i]);
    }
    store8(out + (size_t)t * F + j, o);
  }
  TRACE_EXIT(tr);
}

cudaError_t launch_act(cudaStream_t st, int odt, int T, int F, const float* h, int S, size_t stride,
                       const float* bias, int swiglu, void* out, float glu_limit) {
  if (T <= 0) return cudaSuccess;
  size_t nvec = (size_t)T * (F / 8);
  // few rows: small CTAs, so that the slices come in through many SMs
  int threads = nvec < (size_t)148 * 512 ? 64 : 256;
  int blocks = (int)min((size_t)148 * 16, (nvec + threads - 1) / threads);
  if (odt == DT_F32)
    (void)launch_k(act_kernel<float>, dim3(blocks), dim3(threads), 0, st, T, F, h, S, stride, bias, swiglu, (float*)out, glu_limit, next_trace(6));
  else
    (void)launch_k(act_kernel<bf16>, dim3(blocks), dim3(threads), 0, st, T, F, h, S, stride, bias, swiglu, (bf16*)out, glu_limit, next_trace(6));
  return cudaGetLastError();
}

// ------------------------------------------------------------------ PolyNorm
// CTA per token: the row's split-K slices summed into shared memory while its sums of z^2, z^4 and z^6 are taken,
// then one pass that applies the cubic with its three normalisers.
template <typename OT>
__global__ void __launch_bounds__(256) poly_norm_kernel(int n, int ld, const float* __restrict__ h, int S, size_t stride,
                                                        const float* __restrict__ coef, float eps, OT* __restrict__ out,
                                                        Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  extern __shared__ float row[];  // [ld]
  __shared__ float red[32];
  const float ca = coef[0], cb = coef[1], cc = coef[2], ce = coef[3];
  pdl_wait();
  const size_t t = blockIdx.x;
  float s1 = 0.f, s2 = 0.f, s3 = 0.f;
  for (int i = threadIdx.x * 8; i < ld; i += blockDim.x * 8) {
    float z[8];
    sum_partials8(h + t * ld + i, S, stride, z);
    store8(row + i, z);
#pragma unroll
    for (int e = 0; e < 8; e++)
      if (i + e < n) {
        const float q = z[e] * z[e], c = q * z[e];
        s1 += q;
        s2 = fmaf(q, q, s2);
        s3 = fmaf(c, c, s3);
      }
  }
  s1 = block_sum(s1, red);
  s2 = block_sum(s2, red);
  s3 = block_sum(s3, red);
  const float inv_n = 1.0f / (float)n;
  const float n1 = ca / sqrtf(s1 * inv_n + eps), n2 = cb / sqrtf(s2 * inv_n + eps), n3 = cc / sqrtf(s3 * inv_n + eps);
  for (int i = threadIdx.x * 8; i < ld; i += blockDim.x * 8) {
    float z[8], o[8];
    load8(row + i, z);
#pragma unroll
    for (int e = 0; e < 8; e++) o[e] = i + e < n ? fmaf(fmaf(fmaf(n3, z[e], n2), z[e], n1), z[e], ce) : 0.f;
    store8(out + t * ld + i, o);
  }
  TRACE_EXIT(tr);
}

cudaError_t launch_poly_norm(cudaStream_t st, int odt, int T, int n, int ld, const float* h, int S, size_t stride,
                             const float* coef, float eps, void* out) {
  if (T <= 0) return cudaSuccess;
  if (n <= 0 || n > ld || (ld & 7) || S < 1) return cudaErrorInvalidValue;
  const size_t smem = (size_t)ld * sizeof(float);
  const int threads = min(256, max(64, ((ld / 8 + 31) / 32) * 32));
  if (odt == DT_F32) {
    if (smem > 48 * 1024) cudaFuncSetAttribute(poly_norm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    (void)launch_k(poly_norm_kernel<float>, dim3(T), dim3(threads), smem, st, n, ld, h, S, stride, coef, eps, (float*)out, next_trace(6));
  } else {
    if (smem > 48 * 1024) cudaFuncSetAttribute(poly_norm_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    (void)launch_k(poly_norm_kernel<bf16>, dim3(T), dim3(threads), smem, st, n, ld, h, S, stride, coef, eps, (bf16*)out, next_trace(6));
  }
  return cudaGetLastError();
}

// ------------------------------------------------------- per-layer token input
// g[t, j] = gelu_tanh(W_gate x)[t, j] * table[token[t]][col0 + j]: the split-K slices of the gate
// projection summed, the activation in fp32, the token's entries of the layer's part of the table
template <typename OT, typename WT>
__global__ void token_gate_kernel(int T, int n, const float* __restrict__ h, int S, size_t stride, int ld_h,
                                  const int* __restrict__ tokens, const WT* __restrict__ table, int ld_table, int col0,
                                  OT* __restrict__ out, int ld_out, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  const size_t total = (size_t)T * ld_out;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / ld_out), j = (int)(i % ld_out);
    float o = 0.f;
    if (j < n) {
      float z = 0.f;
      for (int s = 0; s < S; s++) z += h[(size_t)s * stride + (size_t)t * ld_h + j];
      o = gelu_tanh(z) * to_f32(table[(size_t)tokens[t] * ld_table + col0 + j]);
    }
    out[i] = from_f32<OT>(o);
  }
  TRACE_EXIT(tr);
}

cudaError_t launch_token_gate(cudaStream_t st, int odt, int wdt, int T, int n, const float* h, int S, size_t stride, int ld_h,
                              const int* tokens, const void* table, int ld_table, int col0, void* out, int ld_out) {
  if (T <= 0) return cudaSuccess;
  const size_t total = (size_t)T * ld_out;
  const int blocks = (int)min((size_t)148 * 16, (total + 255) / 256);
  if (odt == DT_F32 && wdt == DT_F32)
    (void)launch_k(token_gate_kernel<float, float>, dim3(blocks), dim3(256), 0, st, T, n, h, S, stride, ld_h, tokens,
                   (const float*)table, ld_table, col0, (float*)out, ld_out, next_trace(6));
  else if (odt == DT_BF16 && wdt == DT_BF16)
    (void)launch_k(token_gate_kernel<bf16, bf16>, dim3(blocks), dim3(256), 0, st, T, n, h, S, stride, ld_h, tokens,
                   (const bf16*)table, ld_table, col0, (bf16*)out, ld_out, next_trace(6));
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

// ------------------------------------------------------- RoPE + paged KV append
// One CTA per token.  Work items are (head, 8-wide vector of the first half):
// rotate_half pairs element i with i + hd/2 (rope.go:187-201).
template <typename QT, typename KT>
__global__ void rope_kv_kernel(int nh, int nkv, int hd, const float* __restrict__ qkv, int S,
                               size_t stride, const float* __restrict__ bias,
                               const int* __restrict__ positions, const int* __restrict__ slots,
                               const float* __restrict__ cosT, const float* __restrict__ sinT,
                               QT* __restrict__ q_out, KT* __restrict__ kpool,
                               KT* __restrict__ vpool, Trace tr) {
  const unsigned long long t_entry = trace_on(tr) ? gtime() : 0ull;
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const int half = hd / 2;
  const int vph = half / 8;  // vectors per half head
  const int ncols = (nh + 2 * nkv) * hd;
  // positions / slots were written by the step's first kernel (which triggers its dependents
  // only after its own wait) or by the host copy: stable here.  Fetch them and the first
  // item's RoPE factors before the dependency on the QKV GEMM resolves.
  const int pos = positions[t];
  const int slot = slots[t];
  const int blk = slot / KV_BLOCK, off = slot % KV_BLOCK;
  const int items = (nh + 2 * nkv) * vph;
  float c0v[8], s0v[8];
#pragma unroll
  for (int i = 0; i < 8; i++) c0v[i] = s0v[i] = 0.f;
  const int it_first = blockIdx.y * blockDim.x + threadIdx.x;
  if (cosT != nullptr && it_first < items) {
    const int j = (it_first % vph) * 8;
    load8(cosT + (size_t)pos * half + j, c0v);
    load8(sinT + (size_t)pos * half + j, s0v);
  }
  pdl_wait();
  const unsigned long long t_wait = trace_on(tr) ? gtime() : 0ull;
  for (int it = blockIdx.y * blockDim.x + threadIdx.x; it < items; it += gridDim.y * blockDim.x) {
    const int head = it / vph;
    const int j = (it % vph) * 8;
    const int c0 = head * hd + j;
    float a[8], b[8];
    const float* base = qkv + (size_t)t * ncols + c0;
    sum_partials8(base, S, stride, a);
    sum_partials8(base + half, S, stride, b);
    if (bias) {
      float p[8];
      load8(bias + c0, p);
#pragma unroll
      for (int i = 0; i < 8; i++) a[i] += p[i];
      load8(bias + c0 + half, p);
#pragma unroll
      for (int i = 0; i < 8; i++) b[i] += p[i];
    }
    const bool is_v = head >= nh + nkv;
    if (cosT != nullptr && !is_v) {
      float c[8], sn[8];
      if (it == it_first) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          c[i] = c0v[i];
          sn[i] = s0v[i];
        }
      } else {
        load8(cosT + (size_t)pos * half + j, c);
        load8(sinT + (size_t)pos * half + j, sn);
      }
#pragma unroll
      for (int i = 0; i < 8; i++) {
        float ra = a[i] * c[i] - b[i] * sn[i];
        float rb = b[i] * c[i] + a[i] * sn[i];
        a[i] = ra;
        b[i] = rb;
      }
    }
    if (head < nh) {
      QT* dst = q_out + (size_t)t * nh * hd + head * hd + j;
      store8(dst, a);
      store8(dst + half, b);
    } else {
      const int kvh = is_v ? head - nh - nkv : head - nh;
      KT* pool = is_v ? vpool : kpool;
      KT* dst = pool + (((size_t)blk * nkv + kvh) * KV_BLOCK + off) * hd + j;
      store8(dst, a);
      store8(dst + half, b);
    }
  }
  if (threadIdx.x == 0) trace_rec(tr, t_entry, t_wait, 0);
}

cudaError_t launch_rope_kv(cudaStream_t st, int qdt, int kvdt, int T, int nh, int nkv, int hd,
                           const float* qkv, int S, size_t stride, const float* bias,
                           const int* positions, const int* slots, const float* cosT,
                           const float* sinT, void* q_out, void* kpool, void* vpool) {
  if (T <= 0) return cudaSuccess;
  int items = (nh + 2 * nkv) * (hd / 16);
  // few tokens (decode): split each token's heads over several CTAs — a CTA pulls S partial
  // slices of its columns out of L2 and one SM's intake would pace the kernel
  int groups = 1;
  while (T * groups < 256 && items / (groups * 2) >= 32) groups *= 2;
  int per = (items + groups - 1) / groups;
  int threads = min(256, max(32, ((per + 31) / 32) * 32));
#define RK(QT, KT)                                                                              \
  (void)launch_k(rope_kv_kernel<QT, KT>, dim3(T, groups), dim3(threads), 0, st, nh, nkv, hd, qkv, S, stride, bias, positions,   \
                                                slots, cosT, sinT, (QT*)q_out, (KT*)kpool,      \
                                                (KT*)vpool, next_trace(3))
  if (qdt == DT_F32 && kvdt == DT_F32) RK(float, float);
  else if (qdt == DT_F32 && kvdt == DT_BF16) RK(float, bf16);
  else if (qdt == DT_BF16 && kvdt == DT_BF16) RK(bf16, bf16);
  else return cudaErrorInvalidValue;
#undef RK
  return cudaGetLastError();
}

// ------------------------------------------------------------------- sampling
struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax argmax_merge(ArgMax a, ArgMax b) {
  // larger value wins; equal values keep the lower index (first-max rule)
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

// order-preserving float -> uint32 key; the low word ~index makes atomicMax keep the LOWEST
// index among equal values (first-max rule of cmd/ask/main.go:389-402)
__device__ __forceinline__ unsigned long long argmax_key(float v, int i) {
  uint32_t b = __float_as_uint(v);
  b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  return ((unsigned long long)b << 32) | (uint32_t)(~(uint32_t)i);
}

// Tensor-parallel LM head: the row's logits are V / vsplit slices gathered rank-major.  One
// CTA (blockIdx.y == 0) per row; same arithmetic and scan order as the plain path below.
__device__ __noinline__ void sample_split_rows(const float* __restrict__ logits, int V, int n,
                                               int vsplit, const float* __restrict__ temperature,
                                               const float* __restrict__ uniforms,
                                               int* __restrict__ out_tokens, float* red,
                                               ArgMax* amred, float* scan, int* winner) {
  if (blockIdx.y != 0) return;
  const int s = blockIdx.x;
  auto at = [&](int v) -> float {
    const int r = v / vsplit;
    return logits[(size_t)r * n * vsplit + (size_t)s * vsplit + (v - r * vsplit)];
  };
  const float temp = temperature ? temperature[s] : 0.f;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (!(temp > 0.f)) {
    ArgMax am = {-INFINITY, 0x7fffffff};
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
      const float v = at(i);
      if (v > am.v) { am.v = v; am.i = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax ot = {__shfl_xor_sync(0xffffffffu, am.v, o), __shfl_xor_sync(0xffffffffu, am.i, o)};
      am = argmax_merge(am, ot);
    }
    if (lane == 0) amred[w] = am;
    __syncthreads();
    if (w == 0) {
      ArgMax r = (lane < nw) ? amred[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ArgMax ot = {__shfl_xor_sync(0xffffffffu, r.v, o), __shfl_xor_sync(0xffffffffu, r.i, o)};
        r = argmax_merge(r, ot);
      }
      if (lane == 0) out_tokens[s] = (r.i == 0x7fffffff) ? 0 : r.i;
    }
    return;
  }
  const int chunk = (V + blockDim.x - 1) / blockDim.x;
  const int lo = min(V, (int)threadIdx.x * chunk), hi = min(V, lo + chunk);
  float mx = -INFINITY;
  for (int i = lo; i < hi; i++) mx = fmaxf(mx, at(i) / temp);
  mx = block_max(mx, red);
  float csum = 0.f;
  for (int i = lo; i < hi; i++) csum += expf(at(i) / temp - mx);
  scan[threadIdx.x] = csum;
  __syncthreads();
  for (int o = 1; o < (int)blockDim.x; o <<= 1) {
    float add = (threadIdx.x >= (unsigned)o) ? scan[threadIdx.x - o] : 0.f;
    __syncthreads();
    scan[threadIdx.x] += add;
    __syncthreads();
  }
  const float total = scan[blockDim.x - 1];
  const float r = uniforms[s] * total;
  if (threadIdx.x == 0) *winner = V - 1;
  __syncthreads();
  const float incl = scan[threadIdx.x];
  const float excl = incl - csum;
  const bool mine = (incl >= r) && (threadIdx.x == 0 || scan[threadIdx.x - 1] < r) && (hi > lo);
  if (mine) {
    float run = excl;
    int pick = hi - 1;
    for (int i = lo; i < hi; i++) {
      run += expf(at(i) / temp - mx);
      if (run >= r) {
        pick = i;
        break;
      }
    }
    atomicMin(winner, pick);
  }
  __syncthreads();
  if (threadIdx.x == 0) out_tokens[s] = *winner;
}

// grid (n_seqs, chunks).  Greedy rows: every CTA reduces its slice of the vocabulary and
// merges with one 64-bit atomicMax; the last CTA of the row (atomic ticket) publishes the
// token and re-arms the scratch, so the kernel needs no separate init.  Temperature rows: CTA
// chunk 0 runs the whole softmax / inverse-CDF draw.
__global__ void sample_kernel(const float* __restrict__ logits, int ldl, int V,
                              const float* __restrict__ temperature,
                              const float* __restrict__ uniforms, int* __restrict__ out_tokens,
                              unsigned long long* __restrict__ amax, int* __restrict__ ticket,
                              int vsplit, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  const float temp = temperature ? temperature[blockIdx.x] : 0.f;  // step state: stable before the wait
  pdl_wait();
  __shared__ float red[32];
  __shared__ ArgMax amred[32];
  __shared__ float scan[1024];
  __shared__ int winner;
  const int s = blockIdx.x;
  if (vsplit > 0) {
    sample_split_rows(logits, V, gridDim.x, vsplit, temperature, uniforms, out_tokens, red, amred,
                      scan, &winner);
    TRACE_EXIT(tr);
    return;
  }
  const float* l = logits + (size_t)s * ldl;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (!(temp > 0.f)) {
    const int chunks = gridDim.y;
    const int per = ((V + chunks - 1) / chunks + 3) & ~3;
    const int lo = blockIdx.y * per, hi = min(V, lo + per);
    ArgMax am = {-INFINITY, 0x7fffffff};
    // the forward pass has ldl % 8 == 0 and `per` % 4 == 0 (16-byte aligned slices); the
    // single-operator entry point may pass any row stride
    const bool vec = ((reinterpret_cast<uintptr_t>(l + lo)) & 15) == 0;
    constexpr int U = 4;  // pieces of a thread in flight
    const int step = (int)blockDim.x * 4;
    for (int i0 = lo + (int)threadIdx.x * 4; i0 < hi; i0 += U * step) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; u++)
        if (vec && i0 + u * step + 3 < hi) v[u] = *reinterpret_cast<const float4*>(l + i0 + u * step);
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + u * step;
        if (vec && i + 3 < hi) {
          if (v[u].x > am.v) { am.v = v[u].x; am.i = i; }
          if (v[u].y > am.v) { am.v = v[u].y; am.i = i + 1; }
          if (v[u].z > am.v) { am.v = v[u].z; am.i = i + 2; }
          if (v[u].w > am.v) { am.v = v[u].w; am.i = i + 3; }
        } else {
          for (int j = i; j < min(hi, i + 4); j++) {
            const float w_ = l[j];
            if (w_ > am.v) { am.v = w_; am.i = j; }
          }
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax ot = {__shfl_xor_sync(0xffffffffu, am.v, o), __shfl_xor_sync(0xffffffffu, am.i, o)};
      am = argmax_merge(am, ot);
    }
    if (lane == 0) amred[w] = am;
    __syncthreads();
    if (w == 0) {
      ArgMax r = (lane < nw) ? amred[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ArgMax ot = {__shfl_xor_sync(0xffffffffu, r.v, o), __shfl_xor_sync(0xffffffffu, r.i, o)};
        r = argmax_merge(r, ot);
      }
      if (lane == 0) {
        if (chunks == 1) {
          out_tokens[s] = (r.i == 0x7fffffff) ? 0 : r.i;
        } else {
          if (r.i != 0x7fffffff) atomicMax(amax + s, argmax_key(r.v, r.i));
          __threadfence();
          if (atomicAdd(ticket + s, 1) == chunks - 1) {
            __threadfence();
            const unsigned long long k = atomicExch(amax + s, 0ull);
            out_tokens[s] = k ? (int)(~(uint32_t)(k & 0xffffffffu)) : 0;
            ticket[s] = 0;
          }
        }
      }
    }
    TRACE_EXIT(tr);
    return;
  }
  if (blockIdx.y != 0) return;
  // temperature sampling: sampling.go:70-74 (divide), :105-128 (softmax), :196-217 (inverse CDF).
  // Each thread owns a contiguous chunk so that prefix sums follow index order.
  const int chunk = (V + blockDim.x - 1) / blockDim.x;
  const int lo = min(V, (int)threadIdx.x * chunk), hi = min(V, lo + chunk);
  float mx = -INFINITY;
  for (int i = lo; i < hi; i++) mx = fmaxf(mx, l[i] / temp);
  mx = block_max(mx, red);
  float csum = 0.f;
  for (int i = lo; i < hi; i++) csum += expf(l[i] / temp - mx);
  scan[threadIdx.x] = csum;
  __syncthreads();
  // inclusive scan over <= 1024 chunk sums (Hillis-Steele)
  for (int o = 1; o < (int)blockDim.x; o <<= 1) {
    float add = (threadIdx.x >= (unsigned)o) ? scan[threadIdx.x - o] : 0.f;
    __syncthreads();
    scan[threadIdx.x] += add;
    __syncthreads();
  }
  const float total = scan[blockDim.x - 1];
  const float r = uniforms[s] * total;
  if (threadIdx.x == 0) winner = V - 1;  // sampling.go:212-214 clamp
  __syncthreads();
  const float incl = scan[threadIdx.x];
  const float excl = incl - csum;
  // first chunk whose inclusive prefix reaches r
  const bool mine = (incl >= r) && (threadIdx.x == 0 || scan[threadIdx.x - 1] < r) && (hi > lo);
  if (mine) {
    float run = excl;
    int pick = hi - 1;
    for (int i = lo; i < hi; i++) {
      run += expf(l[i] / temp - mx);
      if (run >= r) {
        pick = i;
        break;
      }
    }
    atomicMin(&winner, pick);
  }
  __syncthreads();
  if (threadIdx.x == 0) out_tokens[s] = winner;
  TRACE_EXIT(tr);
}

cudaError_t launch_sample(cudaStream_t st, const float* logits, int ldl, int V, int n,
                          const float* temperature, const float* uniforms, int* out_tokens,
                          unsigned long long* amax, int* ticket, int vsplit) {
  if (n <= 0) return cudaSuccess;
  // A CTA of a large vocabulary: at most 4096 logits up to 262144 of them, all its loads in flight (8192 one after another: 16
  // steps of GPT-2 alone 3800 us, 3763 so; a few more than 4096, by rounding the CTAs down, cost a step of one to 128 rows of
  // 32000 / 50257 / 128256 another 0.3 to 1.8 us).
  const int chunks = (amax && ticket && vsplit == 0 && V >= 16384) ? min(64, ceil_div(V, 4096)) : 1;
  (void)launch_k(sample_kernel, dim3(n, chunks), dim3(chunks > 1 ? 256 : 1024), 0, st, logits, ldl,
                 V, temperature, uniforms, out_tokens, amax, ticket, vsplit, next_trace(7));
  return cudaGetLastError();
}

__global__ void advance_kernel(int n, const int* __restrict__ sampled, int* tokens, int* positions,
                               int* slots, int* seq_len, const int* __restrict__ block_tables,
                               int max_blocks, int max_pos, Trace tr) {
  TRACE_ENTRY(tr);
  // Step prologue: later kernels read the step state BEFORE their own griddepcontrol.wait, so
  // the dependents are released only after this kernel's writes (the embedding kernel that
  // follows additionally waits for this grid's completion before it releases its own).
  pdl_wait();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    tokens[i] = sampled[i];
    int pos = positions[i] + 1;
    if (pos >= max_pos) pos = max_pos - 1;  // the host bounds every sequence; never index past the table
    int bi = pos / KV_BLOCK;
    if (bi >= max_blocks) bi = max_blocks - 1;
    positions[i] = pos;
    seq_len[i] = pos + 1;
    slots[i] = block_tables[(size_t)i * max_blocks + bi] * KV_BLOCK + pos % KV_BLOCK;
  }
  __threadfence();
  pdl_launch_dependents();
  TRACE_EXIT(tr);
}

cudaError_t launch_advance(cudaStream_t st, int n, const int* sampled, int* tokens, int* positions,
                           int* slots, int* seq_len, const int* block_tables, int max_blocks,
                           int max_pos) {
  if (n <= 0) return cudaSuccess;
  (void)launch_k(advance_kernel, dim3((n + 127) / 128), dim3(128), 0, st, n, sampled, tokens, positions, slots, seq_len,
                                                 block_tables, max_blocks, max_pos, next_trace(8));
  return cudaGetLastError();
}

// ------------------------------------------------------------- recurrent state
// The state of a step's sequences aside (restore = 0) and back: copy [n][slot_floats], behind it the n slots.  Bound by
// memory, once in and once out; the copy leaves L2 first.  32 slots of 1.1 MB: 16 us.
__global__ void __launch_bounds__(256) state_copy_kernel(int n, const int* __restrict__ slots, float* __restrict__ pool, size_t slot_floats,
                                                         float* __restrict__ copy, int* __restrict__ copy_slots, int restore, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_wait();
  const int r = blockIdx.y, slot = restore ? copy_slots[r] : slots[r];
  if (!restore && blockIdx.x == 0 && threadIdx.x == 0) copy_slots[r] = slot;
  float *live = pool + (size_t)slot * slot_floats, *aside = copy + (size_t)r * slot_floats;
  const size_t step = (size_t)gridDim.x * 256, first = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (slot_floats % 4 == 0) {
    const float4* src = reinterpret_cast<const float4*>(restore ? aside : live);
    float4* dst = reinterpret_cast<float4*>(restore ? live : aside);
    const size_t m = slot_floats / 4;
    for (size_t i = first; i < m; i += 4 * step) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (i + u * step < m) v[u] = restore ? __ldcs(src + i + u * step) : __ldcg(src + i + u * step);
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (i + u * step < m) {
          if (restore) dst[i + u * step] = v[u];
          else __stcs(dst + i + u * step, v[u]);
        }
    }
  } else {
    for (size_t i = first; i < slot_floats; i += step) {
      if (restore) live[i] = __ldcs(aside + i);
      else __stcs(aside + i, __ldcg(live + i));
    }
  }
  // a step's kernels read the state ahead of their own waits: they are released after the writes (see advance_kernel)
  __threadfence();
  pdl_launch_dependents();
  TRACE_EXIT(tr);
}
cudaError_t launch_state_copy(cudaStream_t st, int n, const int* slots, float* pool, size_t slot_floats, float* copy, int* copy_slots,
                              bool restore) {
  const unsigned per = (unsigned)std::max<size_t>(1, std::min<size_t>((slot_floats + 4095) / 4096, (size_t)ceil_div(148 * 8, n)));
  return launch_k(state_copy_kernel, dim3(per, (unsigned)n), dim3(256), 0, st, n, slots, pool, slot_floats, copy, copy_slots, restore ? 1 : 0,
                  next_trace(55));
}

// ------------------------------------------------------------- results
// To pinned host memory by a kernel: a few KB are over in one trip across the bus, where the copy engine holds the stream for
// some 10 us.  16 decode steps, copies / kernel: 64 sequences of four Llama-1B layers 4140 / 4022 us (the same steps without
// any copy 3760), GPT-2 alone 3565 / 3490, one sampled step of Falcon layers with its logits 335 / 323.  (The way in stays
// with the copy engine, which starts while the host prepares the launch: requests through delta-rule layers 3860 with a
// kernel, 3780 so.)
// tokens [n], and rows [n][V] of logits that are ldl apart, to pinned memory; CTA 0 has the tokens
__global__ void __launch_bounds__(256) copy_out_kernel(int n, const int* __restrict__ tokens, int* __restrict__ out_tokens,
                                                       const float* __restrict__ logits, int ldl, int V, float* __restrict__ out_logits,
                                                       Trace tr) {
  TRACE_ENTRY(tr);
  pdl_wait();
  pdl_launch_dependents();
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < n; i += 256) out_tokens[i] = __ldcg(tokens + i);
  } else {
    const size_t step = (size_t)(gridDim.x - 1) * 256;
    const bool vec = V % 4 == 0 && ldl % 4 == 0;
    const int per = vec ? V / 4 : V;
    for (size_t i = (size_t)(blockIdx.x - 1) * 256 + threadIdx.x; i < (size_t)n * per; i += step) {
      const size_t r = i / per, c = i % per;
      if (vec) reinterpret_cast<float4*>(out_logits)[i] = __ldcg(reinterpret_cast<const float4*>(logits + r * ldl) + c);
      else out_logits[i] = __ldcg(logits + r * ldl + c);
    }
  }
  TRACE_EXIT(tr);
}
cudaError_t launch_copy_out(cudaStream_t st, int n, const int* tokens, int* out_tokens, const float* logits, int ldl, int V, float* out_logits) {
  const size_t vecs = out_logits ? ((size_t)n * V + 1023) / 1024 : 0;
  return launch_k(copy_out_kernel, dim3(1 + (unsigned)std::min<size_t>(vecs, 64)), dim3(256), 0, st, n, tokens, out_tokens, logits, ldl, V,
                  out_logits, next_trace(56));
}

// ------------------------------------------------------------- weight repack
template <typename ST> __device__ __forceinline__ float src_to_f32(ST v);
template <> __device__ __forceinline__ float src_to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float src_to_f32<bf16>(bf16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float src_to_f32<__half>(__half v) { return __half2float(v); }

// dst[n * row_mul + row_add, k] = src[k, n] for k < K, n < N; src rows are ld_src apart (a
// column slice of a wider matrix: tensor-parallel shards).  32x32 tiles through shared memory
// so both sides are coalesced.  row_mul = 2: [gate | up] halves become interleaved rows (gate j
// -> 2j, up j -> 2j + 1) so that a GEMM tile holds matching gate / up rows for the fused
// SwiGLU epilogue.
template <typename ST, typename DT>
__global__ void transpose_convert_kernel(const ST* __restrict__ src, size_t ld_src, int K, int N,
                                         DT* __restrict__ dst, int ld_dst, int row_mul,
                                         int row_add) {
  __shared__ float tile[32][33];
  const int n0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    int k = k0 + r, n = n0 + threadIdx.x;
    tile[r][threadIdx.x] = (k < K && n < N) ? src_to_f32<ST>(src[(size_t)k * ld_src + n]) : 0.f;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    int n = n0 + r, k = k0 + threadIdx.x;
    if (n < N && k < K)
      dst[((size_t)n * row_mul + row_add) * ld_dst + k] = from_f32<DT>(tile[threadIdx.x][r]);
  }
}

cudaError_t launch_transpose_convert(cudaStream_t st, int sdt_api, const void* src, size_t ld_src,
                                     int K, int N, int ddt, void* dst, int ld_dst, int row_mul,
                                     int row_add) {
  if (K <= 0 || N <= 0) return cudaSuccess;
  dim3 grid((N + 31) / 32, (K + 31) / 32), block(32, 8);
#define TC(ST, DT)                                                                            \
  transpose_convert_kernel<ST, DT><<<grid, block, 0, st>>>((const ST*)src, ld_src, K, N, (DT*)dst, \
                                                           ld_dst, row_mul, row_add)
  if (ddt == DT_F32) {
    if (sdt_api == 0) TC(float, float);
    else if (sdt_api == 1) TC(bf16, float);
    else TC(__half, float);
  } else {
    if (sdt_api == 0) TC(float, bf16);
    else if (sdt_api == 1) TC(bf16, bf16);
    else TC(__half, bf16);
  }
#undef TC
  return cudaGetLastError();
}

// glu_I > 0: src is a stack of [2 glu_I, cols] matrices whose first glu_I rows are GLU gates and
// last glu_I rows the matching ups (HF MoE input_linear, generic_loader.go:578-586); dst
// interleaves them (gate j -> row 2j, up j -> row 2j + 1) so that a 128-row weight tile holds
// complete gate / up pairs for the fused SwiGLU epilogue.
template <typename ST, typename DT>
__global__ void convert_kernel(const ST* __restrict__ src, size_t n, DT* __restrict__ dst, int glu_I,
                               int cols) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    size_t o = i;
    if (glu_I > 0) {
      const size_t row = i / cols, c = i - row * cols;
      const size_t e = row / (2 * (size_t)glu_I), q = row - e * 2 * glu_I;
      const size_t g = q / glu_I, j = q - g * glu_I;
      o = (e * 2 * glu_I + 2 * j + g) * cols + c;
    }
    dst[o] = from_f32<DT>(src_to_f32<ST>(src[i]));
  }
}

cudaError_t launch_convert(cudaStream_t st, int sdt_api, const void* src, size_t n, int ddt,
                           void* dst, int glu_I, int cols) {
  if (n == 0) return cudaSuccess;
  int blocks = (int)min((size_t)148 * 8, (n + 255) / 256);
#define CV(ST, DT) \
  convert_kernel<ST, DT><<<blocks, 256, 0, st>>>((const ST*)src, n, (DT*)dst, glu_I, cols)
  if (ddt == DT_F32) {
    if (sdt_api == 0) CV(float, float);
    else if (sdt_api == 1) CV(bf16, float);
    else CV(__half, float);
  } else {
    if (sdt_api == 0) CV(float, bf16);
    else if (sdt_api == 1) CV(bf16, bf16);
    else CV(__half, bf16);
  }
#undef CV
  return cudaGetLastError();
}

// dst[(n * row_mul + row_add) * ld_dst + k] = src[n * ld_src + k] for n < N rows, k < K: a row
// range of a [out, in] (PyTorch / safetensors) linear taken as it lies — the device layout has
// the same orientation, so loading is a strided copy + dtype conversion, no transpose
template <typename ST, typename DT>
__global__ void copy_rows_kernel(const ST* __restrict__ src, size_t ld_src, int N, int K,
                                 DT* __restrict__ dst, int ld_dst, int row_mul, int row_add) {
  const size_t total = (size_t)N * K;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t n = i / K;
    const int k = (int)(i - n * K);
    dst[(n * row_mul + row_add) * ld_dst + k] = from_f32<DT>(src_to_f32<ST>(src[n * ld_src + k]));
  }
}
cudaError_t launch_copy_rows(cudaStream_t st, int sdt_api, const void* src, size_t ld_src, int N,
                             int K, int ddt, void* dst, int ld_dst, int row_mul, int row_add) {
  if (N <= 0 || K <= 0) return cudaSuccess;
  const size_t total = (size_t)N * K;
  int blocks = (int)min((size_t)148 * 8, (total + 255) / 256);
#define CR(ST, DT) \
  copy_rows_kernel<ST, DT><<<blocks, 256, 0, st>>>((const ST*)src, ld_src, N, K, (DT*)dst, ld_dst, row_mul, row_add)
  if (ddt == DT_F32) {
    if (sdt_api == 0) CR(float, float);
    else if (sdt_api == 1) CR(bf16, float);
    else CR(__half, float);
  } else {
    if (sdt_api == 0) CR(float, bf16);
    else if (sdt_api == 1) CR(bf16, bf16);
    else CR(__half, bf16);
  }
#undef CR
  return cudaGetLastError();
}

__global__ void fill_kernel(float* p, size_t n, float v) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    p[i] = v;
}
cudaError_t launch_fill(cudaStream_t st, float* p, size_t n, float v) {
  fill_kernel<<<148 * 8, 256, 0, st>>>(p, n, v);
  return cudaGetLastError();
}

// out[i] = sum_s p[s*stride + i]   (split-K partials of the LM head -> logits)
__global__ void reduce_partials_kernel(const float* __restrict__ p, int S, size_t stride, size_t n,
                                       float* __restrict__ out, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    float acc = 0.f;
    for (int s = 0; s < S; s++) acc += p[(size_t)s * stride + i];
    out[i] = acc;
  }
  TRACE_EXIT(tr);
}
cudaError_t launch_reduce_partials(cudaStream_t st, const float* p, int S, size_t stride, size_t n,
                                   float* out) {
  if (n == 0) return cudaSuccess;
  int blocks = (int)min((size_t)148 * 8, (n + 255) / 256);
  (void)launch_k(reduce_partials_kernel, dim3(blocks), dim3(256), 0, st, p, S, stride, n, out, next_trace(10));
  return cudaGetLastError();
}

// Build the decode-step state of n sequences from the state of the prefill step that just
// sampled `sampled`: next position = seq_len, KV slot through the block table.
__global__ void make_decode_state_kernel(int n, int mb, const int* __restrict__ sampled,
                                         const int* __restrict__ src_seq_len,
                                         const int* __restrict__ src_bt,
                                         const int* __restrict__ src_temp,
                                         const int* __restrict__ src_uni, int* tokens,
                                         int* positions, int* slots, int* cu_q, int* seq_start,
                                         int* seq_len, int* last_row, int* bt, int* temp, int* uni,
                                         Trace tr) {
  TRACE_ENTRY(tr);
  // step prologue: dependents are released after the writes below (see advance_kernel)
  pdl_wait();
  const int i = blockIdx.x;
  for (int b = threadIdx.x; b < mb; b += blockDim.x) bt[(size_t)i * mb + b] = src_bt[(size_t)i * mb + b];
  if (threadIdx.x == 0) {
    const int pos = src_seq_len[i];
    int bi = pos / KV_BLOCK;
    if (bi >= mb) bi = mb - 1;  // the host checks the range before launching
    tokens[i] = sampled[i];
    positions[i] = pos;
    slots[i] = src_bt[(size_t)i * mb + bi] * KV_BLOCK + pos % KV_BLOCK;
    cu_q[i] = i;
    if (i == n - 1) cu_q[n] = n;
    seq_start[i] = pos;
    seq_len[i] = pos + 1;
    last_row[i] = i;
    temp[i] = src_temp[i];
    uni[i] = src_uni[i];
  }
  __threadfence();
  __syncthreads();
  pdl_launch_dependents();
  TRACE_EXIT(tr);
}
cudaError_t launch_make_decode_state(cudaStream_t st, int n, int mb, const int* sampled,
                                     const int* src_seq_len, const int* src_bt, const int* src_temp,
                                     const int* src_uni, int* tokens, int* positions, int* slots,
                                     int* cu_q, int* seq_start, int* seq_len, int* last_row, int* bt,
                                     int* temp, int* uni) {
  if (n <= 0) return cudaSuccess;
  (void)launch_k(make_decode_state_kernel, dim3(n), dim3(64), 0, st, n, mb, sampled, src_seq_len, src_bt, src_temp, src_uni,
                                             tokens, positions, slots, cu_q, seq_start, seq_len,
                                             last_row, bt, temp, uni, next_trace(8));
  return cudaGetLastError();
}

}  // namespace nvllm
