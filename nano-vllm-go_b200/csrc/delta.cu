// delta.cu — the gated delta rule mixer of a model given as a list of layers
// (nvllm_mixer_kind NVLLM_MIXER_DELTA), for a ragged batch of sequences, between its two
// projections (ordinary GEMMs, forward_layered.cu).
//
// Per head, with a dim x vdim state S kept in fp32 per state slot, for every token in order:
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// q, k (kv_heads x dim, shared by heads / kv_heads heads each) and v (heads x vdim) come from
// the fused input projection through a causal convolution over time per channel (taps from the
// layer, zeros before the sequence start, the last column is the current token's), SiLU, and for
// q / k a division by the head's Euclidean length (eps 1e-6 under the root; q also by sqrt(dim)).
// beta = sigmoid(W_b x), g = exp(-exp(A_log) softplus(W_a x + dt_bias)) per head.  The read-out
// of a head is divided by its root mean square over vdim, multiplied by a weight shared by the
// heads and by silu(W_g x), and goes to the output projection.
//
//   delta_prep_kernel  per token: split-K sum of the projection, convolution (the taps - 1
//                      inputs before the step's first token come from the slot's tail), SiLU,
//                      unit lengths; beta and g.  All fp32.
//   delta_scan_kernel  one CTA per (sequence, head, block of value columns).  A value column of
//                      the state is independent of the others: it lives in the registers of LPC
//                      lanes (dim / LPC entries each), the inner products of a token are
//                      reduced with shuffles inside that lane group.  Token inputs arrive in
//                      double-buffered shared-memory tiles of 16 tokens (cp.async), so the loop
//                      over tokens never waits for memory.  The state is read from the slot when
//                      the sequence has earlier tokens (zero otherwise) and written back at the
//                      end; the sequence's CTAs also roll the convolution tail forward.  Compile-time sizes:
//                      delta_scan_columns_kernel, and delta_scan_packed_kernel for many columns.
//   delta_out_kernel   one CTA per token, a warp per head: RMS over vdim, weight, gate -> act dtype.
#include <stdlib.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "mma.cuh"

namespace nvllm {

namespace {
__device__ __forceinline__ int seq_of_row(const int* __restrict__ cu_q, int n_seqs, int row) {
  int lo = 0, hi = n_seqs - 1;  // last s with cu_q[s] <= row
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_q[mid] <= row) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
__device__ __forceinline__ float sum_slices(const float* __restrict__ p, int S, size_t stride) {
  float acc = 0.f;
  for (int s = 0; s < S; s++) acc += p[(size_t)s * stride];
  return acc;
}
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }
// SiLU of the convolution outputs and of the output gate: exact in the fp32 mode, fast
// intrinsics (relative error about 1e-6, far below the bf16 rounding that follows) otherwise
template <bool FAST>
__device__ __forceinline__ float silu_t(float x) {
  return FAST ? __fdividef(x, 1.0f + __expf(-x)) : silu(x);
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
}  // namespace

constexpr int DELTA_MAX_TAPS = 8;

// grid (T, Y), 256 threads.  The channels of a row are cut into units that a WARP finishes on
// its own: the G query heads, the G key heads (a unit = one head, whose length the warp needs)
// and the value channels in pieces of 32 * MAXV; the warps of the row's CTAs take the units in
// turn.  A lane holds up to MAXV channels of its unit; all their taps' loads are in flight at once.
template <int MAXV, bool FAST>
__global__ void __launch_bounds__(256) delta_prep_kernel(DeltaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  // one row per sequence (a decode step): row t is sequence t, no search through the offsets
  const int s = a.T == a.n_seqs ? t : seq_of_row(a.cu_q, a.n_seqs, t);
  const int r0 = a.cu_q[s];
  const int li = t - r0;                 // index among the step's rows of the sequence
  const int pos = a.positions[r0] + li;  // position in the sequence
  const float* tail = a.state_pool + (size_t)a.state_slots[s] * a.slot_floats + a.tail_off;  // [taps - 1][conv_ch]
  constexpr int PIECE = 32 * MAXV;
  const int v_units = ceil_div(a.n_v, PIECE);
  const int n_units = 2 * a.G + v_units;
  const float qmul = 1.0f / sqrtf((float)a.dim);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int u = blockIdx.y * nw + warp; u < n_units; u += gridDim.y * nw) {
    const bool head = u < 2 * a.G;
    const int c0 = head ? u * a.dim : a.n_q + a.n_k + (u - 2 * a.G) * PIECE;
    const int cn = head ? a.dim : min(PIECE, a.conv_ch - c0);
    float val[MAXV];
#pragma unroll
    for (int i = 0; i < MAXV; i++) val[i] = 0.f;
    for (int k = 0; k < a.taps; k++) {  // tap k reads the token taps - 1 - k positions earlier
      const int back = a.taps - 1 - k;
      const float* src = nullptr;
      int S = 1;
      size_t stride = 0;
      if (li - back >= 0) { src = a.in_p + (size_t)(t - back) * a.in_ld; S = a.in_S; stride = a.in_stride; }
      else if (pos - back >= 0) src = tail + (size_t)(a.taps - 1 + li - back) * a.conv_ch;
      if (!src) continue;  // before the start of the sequence: zeros
#pragma unroll
      for (int i = 0; i < MAXV; i++) {
        const int c = c0 + lane + 32 * i;
        if (lane + 32 * i < cn) val[i] = fmaf(sum_slices(src + c, S, stride), a.conv_w[c * a.taps + k], val[i]);
      }
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < MAXV; i++) {
      val[i] = (lane + 32 * i < cn) ? silu_t<FAST>(val[i]) : 0.f;
      ss += val[i] * val[i];
    }
    float mul = 1.f;
    if (head) {  // unit length; the queries also carry 1 / sqrt(dim)
      mul = 1.0f / sqrtf(warp_sum(ss) + 1e-6f);
      if (u < a.G) mul *= qmul;
    }
#pragma unroll
    for (int i = 0; i < MAXV; i++)
      if (lane + 32 * i < cn) a.qkv[(size_t)t * a.conv_ch + c0 + lane + 32 * i] = val[i] * mul;
  }
  if (blockIdx.y == 0 && threadIdx.x < a.H) {
    const int h = threadIdx.x;
    const float* p = a.in_p + (size_t)t * a.in_ld + a.conv_ch;
    const float b = sum_slices(p + h, a.in_S, a.in_stride);
    const float d = sum_slices(p + a.H + h, a.in_S, a.in_stride);
    a.bg[(size_t)t * 2 * a.H + h] = 1.0f / (1.0f + expf(-b));
    a.bg[(size_t)t * 2 * a.H + a.H + h] = expf(-expf(a.a_log[h]) * softplus(d + a.dt_bias[h]));
  }
  TRACE_EXIT(tr);
}

// The same for steps of many rows, DP_ROWS neighbouring rows per CTA: a warp keeps the taps of its unit (a head of up to
// 128 channels, or 128 value channels; four per lane) and slides a window of rows over them, so a row of the projection
// is read once, 16 bytes at a time, instead of once per tap with a search for its sequence in front.  Bound by
// memory (the projection's columns once, the results once): 18 k rows of 4096 channels 195 us, 950 us with a row per
// CTA.  Fewer rows than 1024 keep that kernel, which spreads a row over several CTAs.
constexpr int DP_ROWS = 8;
__device__ __forceinline__ float4 sum_slices4(const float* __restrict__ p, int S, size_t stride) {
  float4 acc = *reinterpret_cast<const float4*>(p);
  for (int s = 1; s < S; s++) {
    const float4 v = *reinterpret_cast<const float4*>(p + (size_t)s * stride);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  return acc;
}
template <int TAPS, bool FAST>
__global__ void __launch_bounds__(256) delta_prep_rows_kernel(DeltaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  const int t0 = blockIdx.x * DP_ROWS, t1 = min(a.T, t0 + DP_ROWS);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int u = blockIdx.y * 8 + warp;  // this warp's unit
  const bool head = u < 2 * a.G;
  const int c0 = head ? u * a.dim : a.n_q + a.n_k + (u - 2 * a.G) * 128;
  const int cn = head ? a.dim : min(128, a.conv_ch - c0);
  const bool on = 4 * lane < cn;  // heads and pieces are multiples of 4 channels; a unit past the last has none
  const int c = c0 + 4 * lane;
  float wv[4][TAPS];  // immutable: fetched before the dependency resolves
#pragma unroll
  for (int e = 0; e < 4; e++)
#pragma unroll
    for (int k = 0; k < TAPS; k++) wv[e][k] = on ? a.conv_w[(size_t)(c + e) * TAPS + k] : 0.f;
  pdl_wait();
  const float qmul = 1.0f / sqrtf((float)a.dim);
  int s = seq_of_row(a.cu_q, a.n_seqs, t0);
  int first = a.cu_q[s], last = a.cu_q[s + 1], pos0 = a.positions[first];
  float4 win[TAPS];  // the last TAPS rows, the current one last
  // the rows in front of row t: of the step, of the slot's tail, or zeros before the sequence's start
  auto refill = [&](int t) {
    const float* tail = a.state_pool + (size_t)a.state_slots[s] * a.slot_floats + a.tail_off;
    const int li = t - first, pos = pos0 + li;
#pragma unroll
    for (int k = 0; k + 1 < TAPS; k++) {
      const int back = TAPS - 1 - k;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (on) {
        if (li - back >= 0) v = sum_slices4(a.in_p + (size_t)(t - back) * a.in_ld + c, a.in_S, a.in_stride);
        else if (pos - back >= 0) v = *reinterpret_cast<const float4*>(tail + (size_t)(TAPS - 1 + li - back) * a.conv_ch + c);
      }
      win[k + 1] = v;  // moves to k when row t enters
    }
  };
  refill(t0);
  for (int t = t0; t < t1; t++) {
    if (t >= last) {  // the next sequence (every sequence of a step has rows)
      s++;
      first = last;
      last = a.cu_q[s + 1];
      pos0 = a.positions[first];
      refill(t);
    }
#pragma unroll
    for (int k = 0; k + 1 < TAPS; k++) win[k] = win[k + 1];
    win[TAPS - 1] = on ? sum_slices4(a.in_p + (size_t)t * a.in_ld + c, a.in_S, a.in_stride) : make_float4(0.f, 0.f, 0.f, 0.f);
    float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < TAPS; k++) {
      y[0] = fmaf(win[k].x, wv[0][k], y[0]);
      y[1] = fmaf(win[k].y, wv[1][k], y[1]);
      y[2] = fmaf(win[k].z, wv[2][k], y[2]);
      y[3] = fmaf(win[k].w, wv[3][k], y[3]);
    }
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      y[e] = silu_t<FAST>(y[e]);
      ss += y[e] * y[e];
    }
    float mul = 1.f;
    if (head) {  // unit length; the queries also carry 1 / sqrt(dim)
      mul = 1.0f / sqrtf(warp_sum(on ? ss : 0.f) + 1e-6f);
      if (u < a.G) mul *= qmul;
    }
    if (on)
      *reinterpret_cast<float4*>(a.qkv + (size_t)t * a.conv_ch + c) = make_float4(y[0] * mul, y[1] * mul, y[2] * mul, y[3] * mul);
  }
  if (blockIdx.y == 0)
    for (int i = threadIdx.x; i < (t1 - t0) * a.H; i += blockDim.x) {
      const int t = t0 + i / a.H, h = i % a.H;
      const float* q = a.in_p + (size_t)t * a.in_ld + a.conv_ch;
      const float b = sum_slices(q + h, a.in_S, a.in_stride);
      const float d = sum_slices(q + a.H + h, a.in_S, a.in_stride);
      a.bg[(size_t)t * 2 * a.H + h] = 1.0f / (1.0f + expf(-b));
      a.bg[(size_t)t * 2 * a.H + a.H + h] = expf(-expf(a.a_log[h]) * softplus(d + a.dt_bias[h]));
    }
  TRACE_EXIT(tr);
}
// rows, units and tails that start on 16-byte boundaries, heads of one warp, enough rows to fill the chip eight at a time
static bool delta_prep_rows_fit(const DeltaArgs& a) {
  return a.T >= 1024 && a.taps >= 2 && a.taps <= 4 && a.dim <= 128 && a.dim % 4 == 0 && a.n_v % 4 == 0 && a.in_ld % 4 == 0 &&
         a.in_stride % 4 == 0 && a.tail_off % 4 == 0 && a.slot_floats % 4 == 0;
}
template <int TAPS>
static cudaError_t delta_prep_rows(cudaStream_t st, const DeltaArgs& a) {
  const dim3 grid(ceil_div(a.T, DP_ROWS), ceil_div(2 * a.G + ceil_div(a.n_v, 128), 8));
  return a.fast_act ? launch_k(delta_prep_rows_kernel<TAPS, true>, grid, dim3(256), 0, st, a, next_trace(34))
                    : launch_k(delta_prep_rows_kernel<TAPS, false>, grid, dim3(256), 0, st, a, next_trace(34));
}

cudaError_t launch_delta_prep(cudaStream_t st, const DeltaArgs& a) {
  if (a.T <= 0) return cudaSuccess;
  if (a.taps < 1 || a.taps > DELTA_MAX_TAPS || a.H > 256 || a.dim > 1024) return cudaErrorInvalidValue;
  if (delta_prep_rows_fit(a)) {
    if (a.taps == 4) return delta_prep_rows<4>(st, a);
    return a.taps == 3 ? delta_prep_rows<3>(st, a) : delta_prep_rows<2>(st, a);
  }
  const int maxv = a.dim <= 128 ? 4 : a.dim <= 256 ? 8 : 32;
  const int n_units = 2 * a.G + ceil_div(a.n_v, 32 * maxv);
  // few rows (decode): a row's units spread over several CTAs
  const int ny = a.T >= 2048 ? 1 : std::min(ceil_div(n_units, 8), std::max(1, 2048 / a.T));
  const dim3 grid(a.T, ny);
  if (a.fast_act) {
    if (maxv == 4) (void)launch_k(delta_prep_kernel<4, true>, grid, dim3(256), 0, st, a, next_trace(34));
    else if (maxv == 8) (void)launch_k(delta_prep_kernel<8, true>, grid, dim3(256), 0, st, a, next_trace(34));
    else (void)launch_k(delta_prep_kernel<32, true>, grid, dim3(256), 0, st, a, next_trace(34));
  } else {
    if (maxv == 4) (void)launch_k(delta_prep_kernel<4, false>, grid, dim3(256), 0, st, a, next_trace(34));
    else if (maxv == 8) (void)launch_k(delta_prep_kernel<8, false>, grid, dim3(256), 0, st, a, next_trace(34));
    else (void)launch_k(delta_prep_kernel<32, false>, grid, dim3(256), 0, st, a, next_trace(34));
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------------ scan
constexpr int DELTA_TT = 16;  // tokens per shared-memory tile

// block = VC * LPC threads: thread (jl = tid / LPC, p = tid % LPC) holds rows d = r * LPC + p,
// r < R, of value column vbase + jl
template <int R>
__global__ void __launch_bounds__(256) delta_scan_kernel(DeltaArgs a, int LPC, int VC, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float sm[];
  const int dim = a.dim, vdim = a.vdim;
  const int s = blockIdx.x, h = blockIdx.y, vbase = blockIdx.z * VC;
  const int r0 = a.cu_q[s], r1 = a.cu_q[s + 1];
  const int n_new = r1 - r0;
  const int start = a.positions[r0];
  float* slot = a.state_pool + (size_t)a.state_slots[s] * a.slot_floats;
  const int tid = threadIdx.x;
  const int p = tid % LPC, jl = tid / LPC;
  const int col = vbase + jl;
  const bool col_ok = jl < VC && col < vdim;
  const int kvh = h / (a.H / a.G);

  // convolution tail of the slot: after this step it holds the inputs of the last taps - 1
  // positions.  The sequence's CTAs share the channels, a thread per channel, old values read
  // before any write (the prep kernel, which also reads the tail, finished before this kernel's wait).
  if (a.taps > 1) {
    float* tail = slot + a.tail_off;
    const int part = h * gridDim.z + blockIdx.z, parts = a.H * gridDim.z;  // the sequence's CTAs share the channels
    for (int c = part * blockDim.x + tid; c < a.conv_ch; c += parts * blockDim.x) {
      float nv[DELTA_MAX_TAPS];
#pragma unroll
      for (int j = 0; j < DELTA_MAX_TAPS - 1; j++) {
        if (j >= a.taps - 1) break;
        const int q = n_new - (a.taps - 1) + j;  // row of the step that lands in tail[j]; < 0: an older input
        if (q >= 0) nv[j] = sum_slices(a.in_p + (size_t)(r0 + q) * a.in_ld + c, a.in_S, a.in_stride);
        else nv[j] = (start + q >= 0) ? tail[(size_t)(j + n_new) * a.conv_ch + c] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < DELTA_MAX_TAPS - 1; j++) {
        if (j >= a.taps - 1) break;
        tail[(size_t)j * a.conv_ch + c] = nv[j];
      }
    }
  }

  float* S_g = slot + a.state_off + (size_t)h * dim * vdim;
  float S[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int d = r * LPC + p;
    S[r] = (start > 0 && col_ok && d < dim) ? S_g[(size_t)d * vdim + col] : 0.f;
  }
  // tile of DELTA_TT tokens: q [TT][dim], k [TT][dim], v [TT][VC], beta [TT], g [TT]
  const int tile_floats = DELTA_TT * (2 * dim + VC + 2);
  const float* qg = a.qkv + (size_t)kvh * dim;
  const float* kg = a.qkv + a.n_q + (size_t)kvh * dim;
  const float* vg = a.qkv + a.n_q + a.n_k + (size_t)h * vdim + vbase;
  const int vcn = min(VC, vdim - vbase);
  auto issue = [&](int t0, int buf) {
    float* b = sm + buf * tile_floats;
    const int nt = min(DELTA_TT, n_new - t0);
    const uint32_t qb = smem_addr(b), kb = smem_addr(b + DELTA_TT * dim), vb = smem_addr(b + 2 * DELTA_TT * dim),
                   bb = smem_addr(b + DELTA_TT * (2 * dim + VC));
    for (int i = tid; i < nt * dim; i += blockDim.x) {
      const int tt = i / dim, d = i % dim;
      const size_t rowo = (size_t)(r0 + t0 + tt) * a.conv_ch;
      cp_async4(qb + 4 * i, qg + rowo + d);
      cp_async4(kb + 4 * i, kg + rowo + d);
    }
    for (int i = tid; i < nt * vcn; i += blockDim.x) {
      const int tt = i / vcn, j = i % vcn;
      cp_async4(vb + 4 * (tt * VC + j), vg + (size_t)(r0 + t0 + tt) * a.conv_ch + j);
    }
    for (int i = tid; i < nt * 2; i += blockDim.x) {
      const int tt = i >> 1, w = i & 1;
      cp_async4(bb + 4 * (w * DELTA_TT + tt), a.bg + (size_t)(r0 + t0 + tt) * 2 * a.H + w * a.H + h);
    }
  };
  issue(0, 0);
  cp_async_commit();
  float* og = a.o + (size_t)h * vdim + col;
  const int HV = a.H * vdim;
  for (int t0 = 0, it = 0; t0 < n_new; t0 += DELTA_TT, it++) {
    const int buf = it & 1;
    if (t0 + DELTA_TT < n_new) issue(t0 + DELTA_TT, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const float* b = sm + buf * tile_floats;
    const float* qs = b;
    const float* ks = b + DELTA_TT * dim;
    const float* vs = b + 2 * DELTA_TT * dim;
    const float* bs = b + DELTA_TT * (2 * dim + VC);
    const int nt = min(DELTA_TT, n_new - t0);
    for (int tt = 0; tt < nt; tt++) {
      const float beta = bs[tt], g = bs[DELTA_TT + tt];
      const float v = col_ok ? vs[tt * VC + jl] : 0.f;
      float kr[R];
      float dot = 0.f;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int d = r * LPC + p;
        kr[r] = d < dim ? ks[tt * dim + d] : 0.f;
        S[r] *= g;
        dot = fmaf(S[r], kr[r], dot);
      }
      for (int o = 1; o < LPC; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      const float u = beta * (v - dot);
      float out = 0.f;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int d = r * LPC + p;
        S[r] = fmaf(kr[r], u, S[r]);
        const float qv = d < dim ? qs[tt * dim + d] : 0.f;
        out = fmaf(S[r], qv, out);
      }
      for (int o = 1; o < LPC; o <<= 1) out += __shfl_xor_sync(0xffffffffu, out, o);
      if (p == 0 && col_ok) og[(size_t)(r0 + t0 + tt) * HV] = out;
    }
    __syncthreads();  // the buffer may be refilled
  }
  cp_async_wait<0>();
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int d = r * LPC + p;
    if (col_ok && d < dim) S_g[(size_t)d * vdim + col] = S[r];
  }
  TRACE_EXIT(tr);
}


// The same scan with compile-time sizes, dim = R * LPC: lane p of a column holds the R
// neighbouring rows p R .. p R + R - 1, the keys and queries of a token sit in shared memory as
// LPC segments of R + 4 floats (the padding puts the lanes' 16-byte reads in different banks),
// no bounds checks in the token loop, four partial sums per inner product; one column per
// thread and two CTAs per SM, or two columns per thread (CC = 2) and one.
template <int R, int LPC, int CC>
__global__ void __launch_bounds__(256, CC == 1 ? 2 : 1) delta_scan_columns_kernel(DeltaArgs a, int VC, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  constexpr int DIM = R * LPC, RP = R + 4, KL = LPC * RP;
  const int vdim = a.vdim;
  const int s = blockIdx.x, h = blockIdx.y, vbase = blockIdx.z * VC;
  const int r0 = a.cu_q[s], r1 = a.cu_q[s + 1];
  const int n_new = r1 - r0;
  const int start = a.positions[r0];
  float* slot = a.state_pool + (size_t)a.state_slots[s] * a.slot_floats;
  const int tid = threadIdx.x;
  const int p = tid % LPC, jl = tid / LPC;  // the thread's CC columns: vbase + jl + cc * (VC / CC)
  const int VH = VC / CC;
  bool col_ok[CC];
  int col[CC];
#pragma unroll
  for (int cc = 0; cc < CC; cc++) {
    col[cc] = vbase + jl + cc * VH;
    col_ok[cc] = jl < VH && col[cc] < vdim;
  }
  const int kvh = h / (a.H / a.G);

  if (a.taps > 1) {  // roll the convolution tail forward (see the generic kernel)
    float* tail = slot + a.tail_off;
    const int part = h * gridDim.z + blockIdx.z, parts = a.H * gridDim.z;
    for (int c = part * blockDim.x + tid; c < a.conv_ch; c += parts * blockDim.x) {
      float nv[DELTA_MAX_TAPS];
#pragma unroll
      for (int j = 0; j < DELTA_MAX_TAPS - 1; j++) {
        if (j >= a.taps - 1) break;
        const int q = n_new - (a.taps - 1) + j;
        if (q >= 0) nv[j] = sum_slices(a.in_p + (size_t)(r0 + q) * a.in_ld + c, a.in_S, a.in_stride);
        else nv[j] = (start + q >= 0) ? tail[(size_t)(j + n_new) * a.conv_ch + c] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < DELTA_MAX_TAPS - 1; j++) {
        if (j >= a.taps - 1) break;
        tail[(size_t)j * a.conv_ch + c] = nv[j];
      }
    }
  }

  float* S_g = slot + a.state_off + (size_t)h * DIM * vdim;
  float S[CC][R];
#pragma unroll
  for (int cc = 0; cc < CC; cc++)
#pragma unroll
    for (int r = 0; r < R; r++) S[cc][r] = (start > 0 && col_ok[cc]) ? S_g[(size_t)(p * R + r) * vdim + col[cc]] : 0.f;
  // tile of DELTA_TT tokens: q [TT][KL], k [TT][KL], v [TT][VC], beta [TT], g [TT]
  const int tile_floats = DELTA_TT * (2 * KL + VC + 2);
  const float* qg = a.qkv + (size_t)kvh * DIM;
  const float* kg = a.qkv + a.n_q + (size_t)kvh * DIM;
  const float* vg = a.qkv + a.n_q + a.n_k + (size_t)h * vdim + vbase;
  const int vcn = min(VC, vdim - vbase);
  auto issue = [&](int t0, int buf) {
    float* b = sm + buf * tile_floats;
    const int nt = min(DELTA_TT, n_new - t0);
    const uint32_t qb = smem_addr(b), kb = smem_addr(b + DELTA_TT * KL), vb = smem_addr(b + 2 * DELTA_TT * KL),
                   bb = smem_addr(b + DELTA_TT * (2 * KL + VC));
    for (int i = tid; i < nt * (DIM / 4); i += blockDim.x) {  // 16 bytes at a time: rows and segments are 16-byte aligned
      const int tt = i / (DIM / 4), d = (i % (DIM / 4)) * 4;
      const size_t rowo = (size_t)(r0 + t0 + tt) * a.conv_ch;
      const int so = tt * KL + (d / R) * RP + d % R;
      cp_async16(qb + 4 * so, qg + rowo + d, true);
      cp_async16(kb + 4 * so, kg + rowo + d, true);
    }
    for (int i = tid; i < nt * vcn; i += blockDim.x) {
      const int tt = i / vcn, j = i % vcn;
      cp_async4(vb + 4 * (tt * VC + j), vg + (size_t)(r0 + t0 + tt) * a.conv_ch + j);
    }
    for (int i = tid; i < nt * 2; i += blockDim.x) {
      const int tt = i >> 1, w = i & 1;
      cp_async4(bb + 4 * (w * DELTA_TT + tt), a.bg + (size_t)(r0 + t0 + tt) * 2 * a.H + w * a.H + h);
    }
  };
  issue(0, 0);
  cp_async_commit();
  const int HV = a.H * vdim;
  float* og = a.o + (size_t)h * vdim;
  for (int t0 = 0, it = 0; t0 < n_new; t0 += DELTA_TT, it++) {
    const int buf = it & 1;
    if (t0 + DELTA_TT < n_new) issue(t0 + DELTA_TT, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const float* b = sm + buf * tile_floats;
    const float* qs = b + p * RP;
    const float* ks = b + DELTA_TT * KL + p * RP;
    const float* vs = b + 2 * DELTA_TT * KL;
    const float* bs = b + DELTA_TT * (2 * KL + VC);
    const int nt = min(DELTA_TT, n_new - t0);
    for (int tt = 0; tt < nt; tt++) {
      const float beta = bs[tt], g = bs[DELTA_TT + tt];
      float v[CC], dot[CC], out[CC];
#pragma unroll
      for (int cc = 0; cc < CC; cc++) v[cc] = col_ok[cc] ? vs[tt * VC + jl + cc * VH] : 0.f;
      float kr[R];
      float d4[CC][4];
#pragma unroll
      for (int cc = 0; cc < CC; cc++) d4[cc][0] = d4[cc][1] = d4[cc][2] = d4[cc][3] = 0.f;
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(ks + tt * KL + r);
        kr[r] = k4.x; kr[r + 1] = k4.y; kr[r + 2] = k4.z; kr[r + 3] = k4.w;
#pragma unroll
        for (int cc = 0; cc < CC; cc++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            S[cc][r + e] *= g;
            d4[cc][e] = fmaf(S[cc][r + e], kr[r + e], d4[cc][e]);
          }
      }
#pragma unroll
      for (int cc = 0; cc < CC; cc++) {
        dot[cc] = (d4[cc][0] + d4[cc][1]) + (d4[cc][2] + d4[cc][3]);
#pragma unroll
        for (int o = 1; o < LPC; o <<= 1) dot[cc] += __shfl_xor_sync(0xffffffffu, dot[cc], o);
        dot[cc] = beta * (v[cc] - dot[cc]);  // u: what the token writes into the column
        d4[cc][0] = d4[cc][1] = d4[cc][2] = d4[cc][3] = 0.f;
      }
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 q4 = *reinterpret_cast<const float4*>(qs + tt * KL + r);
        const float qv[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int cc = 0; cc < CC; cc++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            S[cc][r + e] = fmaf(kr[r + e], dot[cc], S[cc][r + e]);
            d4[cc][e] = fmaf(S[cc][r + e], qv[e], d4[cc][e]);
          }
      }
#pragma unroll
      for (int cc = 0; cc < CC; cc++) {
        out[cc] = (d4[cc][0] + d4[cc][1]) + (d4[cc][2] + d4[cc][3]);
#pragma unroll
        for (int o = 1; o < LPC; o <<= 1) out[cc] += __shfl_xor_sync(0xffffffffu, out[cc], o);
        if (p == 0 && col_ok[cc]) og[(size_t)(r0 + t0 + tt) * HV + col[cc]] = out[cc];
      }
    }
    __syncthreads();  // the buffer may be refilled
  }
  cp_async_wait<0>();
#pragma unroll
  for (int cc = 0; cc < CC; cc++)
    if (col_ok[cc]) {
#pragma unroll
      for (int r = 0; r < R; r++) S_g[(size_t)(p * R + r) * vdim + col[cc]] = S[cc][r];
    }
  TRACE_EXIT(tr);
}

// The same for many columns (delta_packed_fits) with packed operations, dim = R * LPC.  Lane p of a column holds the R
// neighbouring rows p R .. p R + R - 1 of CC neighbouring columns as packed pairs of rows; the keys and queries of a
// token sit in shared memory as LPC segments of R + 4 floats (the padding puts the lanes' 16-byte reads in different
// banks).  The inner products of the CC columns are summed by shuffles that scatter them over the lanes.  Three fp32 operations per state entry and token instead of four:
//   * the state is kept as S / c with c the product of the decays since the last rescaling, so a token multiplies one
//     number by g; S k and S q are taken in one pass over the old state, the update adds k (u / c)^T, and
//     o = c (S / c) q + (k . q) u.  c starts at one in every tile of tokens (the state is multiplied by the previous
//     tile's c), and whenever it falls below 1e-18 inside one, so u / c stays far from overflow.
//   * k . q, c, 1 / c and the multipliers are made once per token and CTA when a tile has arrived.
// Bound by fp32 issue and, about equally, by shared-memory reads: a 16-byte read costs its four quarter-warps a pass
// each even where they read the same bytes, so eight lanes with four columns (28 reads and 12 shuffles for 96
// packed operations) replace four lanes with two columns.  Four CTAs of 128 threads per SM.  16 sequences of 750 to
// 1500 tokens, 16 heads of 128 x 128: 1502 us; delta_scan_columns_kernel 1905 us.
constexpr float DELTA_RESCALE = 1e-18f;
template <int R, int LPC, int CC>
__global__ void __launch_bounds__(128, 4) delta_scan_packed_kernel(DeltaArgs a, int VC, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  __shared__ float4 tok_s[DELTA_TT];  // of a token: c, 1 / c, k . q, beta
  __shared__ float mul_s[DELTA_TT];   // what multiplies the state before it
  constexpr int DIM = R * LPC, RP = R + 4, KL = LPC * RP;
  const int vdim = a.vdim;
  const int s = blockIdx.x, h = blockIdx.y, vbase = blockIdx.z * VC;
  const int r0 = a.cu_q[s], r1 = a.cu_q[s + 1];
  const int n_new = r1 - r0;
  const int start = a.positions[r0];
  float* slot = a.state_pool + (size_t)a.state_slots[s] * a.slot_floats;
  const int tid = threadIdx.x;
  const int p = tid % LPC, jl = tid / LPC;  // the thread's columns: vbase + CC jl + cc
  // after the shuffles a lane holds one inner product: of column mc, with k (typ 0) or q (typ 1)
  static_assert((CC == 2 || CC == 4) && 2 * CC <= LPC, "a lane for every inner product");
  const int mc = p & (CC - 1), typ = (p / CC) & 1, lane0 = (tid & 31) - p;
  const int vcn = min(VC, vdim - vbase);
  const int kvh = h / (a.H / a.G);

  if (a.taps > 1) {  // roll the convolution tail forward (see the generic kernel)
    float* tail = slot + a.tail_off;
    const int part = h * gridDim.z + blockIdx.z, parts = a.H * gridDim.z;
    for (int c = part * blockDim.x + tid; c < a.conv_ch; c += parts * blockDim.x) {
      float nv[DELTA_MAX_TAPS];
#pragma unroll
      for (int j = 0; j < DELTA_MAX_TAPS - 1; j++) {
        if (j >= a.taps - 1) break;
        const int q = n_new - (a.taps - 1) + j;
        if (q >= 0) nv[j] = sum_slices(a.in_p + (size_t)(r0 + q) * a.in_ld + c, a.in_S, a.in_stride);
        else nv[j] = (start + q >= 0) ? tail[(size_t)(j + n_new) * a.conv_ch + c] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < DELTA_MAX_TAPS - 1; j++) {
        if (j >= a.taps - 1) break;
        tail[(size_t)j * a.conv_ch + c] = nv[j];
      }
    }
  }

  float* S_g = slot + a.state_off + (size_t)h * DIM * vdim + vbase;
  unsigned long long S[CC][R / 2];
#pragma unroll
  for (int cc = 0; cc < CC; cc++)
#pragma unroll
    for (int r = 0; r < R; r += 2) {
      const bool ok = start > 0 && CC * jl + cc < vcn;
      const float* src = S_g + (size_t)(p * R + r) * vdim + CC * jl + cc;
      S[cc][r / 2] = ok ? pack2(src[0], src[vdim]) : 0ull;
    }
  // tile of DELTA_TT tokens: q [TT][KL], k [TT][KL], v [TT][VC], beta [TT], g [TT]
  const int tile_floats = DELTA_TT * (2 * KL + VC + 2);
  const float* qg = a.qkv + (size_t)kvh * DIM;
  const float* kg = a.qkv + a.n_q + (size_t)kvh * DIM;
  const float* vg = a.qkv + a.n_q + a.n_k + (size_t)h * vdim + vbase;
  auto issue = [&](int t0, int buf) {
    float* b = sm + buf * tile_floats;
    const int nt = min(DELTA_TT, n_new - t0);
    const uint32_t qb = smem_addr(b), kb = smem_addr(b + DELTA_TT * KL), vb = smem_addr(b + 2 * DELTA_TT * KL),
                   bb = smem_addr(b + DELTA_TT * (2 * KL + VC));
    for (int i = tid; i < nt * (DIM / 4); i += blockDim.x) {  // 16 bytes at a time: rows and segments are 16-byte aligned
      const int tt = i / (DIM / 4), d = (i % (DIM / 4)) * 4;
      const size_t rowo = (size_t)(r0 + t0 + tt) * a.conv_ch;
      const int so = tt * KL + (d / R) * RP + d % R;
      cp_async16(qb + 4 * so, qg + rowo + d, true);
      cp_async16(kb + 4 * so, kg + rowo + d, true);
    }
    for (int i = tid; i < nt * vcn; i += blockDim.x) {
      const int tt = i / vcn, j = i % vcn;
      cp_async4(vb + 4 * (tt * VC + j), vg + (size_t)(r0 + t0 + tt) * a.conv_ch + j);
    }
    for (int i = tid; i < nt * 2; i += blockDim.x) {
      const int tt = i >> 1, w = i & 1;
      cp_async4(bb + 4 * (w * DELTA_TT + tt), a.bg + (size_t)(r0 + t0 + tt) * 2 * a.H + w * a.H + h);
    }
  };
  issue(0, 0);
  cp_async_commit();
  const int HV = a.H * vdim;
  float* og = a.o + (size_t)h * vdim + vbase;
  float c_end = 1.f;  // (last warp) c after the previous tile
  for (int t0 = 0, it = 0; t0 < n_new; t0 += DELTA_TT, it++) {
    const int buf = it & 1;
    if (t0 + DELTA_TT < n_new) issue(t0 + DELTA_TT, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const float* b = sm + buf * tile_floats;
    const float* qs = b + p * RP;
    const float* ks = b + DELTA_TT * KL + p * RP;
    const float* vs = b + 2 * DELTA_TT * KL;
    const float* bs = b + DELTA_TT * (2 * KL + VC);
    const int nt = min(DELTA_TT, n_new - t0);
    for (int i0 = 0; i0 < DELTA_TT * LPC; i0 += blockDim.x) {  // k . q: LPC neighbouring lanes share a token
      const int i = i0 + tid, tt = i / LPC;
      float dot = 0.f;
      if (tt < nt) {
        const float* kk = b + DELTA_TT * KL + tt * KL + (i % LPC) * RP;
        const float* qq = b + tt * KL + (i % LPC) * RP;
        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < R; r += 4) {
          const float4 k4 = *reinterpret_cast<const float4*>(kk + r), q4 = *reinterpret_cast<const float4*>(qq + r);
          d.x = fmaf(k4.x, q4.x, d.x); d.y = fmaf(k4.y, q4.y, d.y);
          d.z = fmaf(k4.z, q4.z, d.z); d.w = fmaf(k4.w, q4.w, d.w);
        }
        dot = (d.x + d.y) + (d.z + d.w);
      }
#pragma unroll
      for (int o = 1; o < LPC; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (i % LPC == 0 && tt < nt) tok_s[tt].z = dot;
    }
    if (tid >= (int)blockDim.x - 32) {  // the last warp: lane tt makes c of token tt, the product of the decays up to it
      const int tt = tid & 31;
      float c = tt < nt ? bs[DELTA_TT + tt] : 1.f;
#pragma unroll
      for (int o = 1; o < DELTA_TT; o <<= 1) {
        const float before = __shfl_up_sync(0xffffffffu, c, o);
        if (tt >= o) c *= before;
      }
      const float last = __shfl_sync(0xffffffffu, c, nt - 1);
      if (last >= DELTA_RESCALE) {
        if (tt < nt) {
          tok_s[tt].x = c;
          tok_s[tt].y = 1.0f / c;
          tok_s[tt].w = bs[tt];
          mul_s[tt] = tt == 0 ? c_end : 1.f;
        }
        c_end = last;
      } else {  // strong decays: one lane goes through the tokens and rescales where it has to
        float cc = 1.f;
        for (int j = 0; j < nt; j++) {
          cc *= bs[DELTA_TT + j];
          float m = j == 0 ? c_end : 1.f;
          if (cc < DELTA_RESCALE) {
            m *= cc;
            cc = 1.f;
          }
          if (tt == 0) {
            mul_s[j] = m;
            tok_s[j].x = cc;
            tok_s[j].y = 1.0f / cc;
            tok_s[j].w = bs[j];
          }
        }
        c_end = cc;
      }
    }
    __syncthreads();
    for (int tt = 0; tt < nt; tt++) {
      const float4 tk = tok_s[tt];
      const float m = mul_s[tt];
      if (m != 1.f) {
        const unsigned long long mm = pack2(m, m);
#pragma unroll
        for (int cc = 0; cc < CC; cc++)
#pragma unroll
          for (int r = 0; r < R / 2; r++) S[cc][r] = mul2(S[cc][r], mm);
      }
      const float v = CC * jl + mc < vcn ? vs[tt * VC + CC * jl + mc] : 0.f;
      unsigned long long kr[R / 2], dk[CC], dq[CC];
#pragma unroll
      for (int cc = 0; cc < CC; cc++) dk[cc] = dq[cc] = 0ull;
#pragma unroll
      for (int r = 0; r < R / 2; r += 2) {
        const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(ks + tt * KL + 2 * r);
        const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(qs + tt * KL + 2 * r);
        kr[r] = k2.x;
        kr[r + 1] = k2.y;
#pragma unroll
        for (int cc = 0; cc < CC; cc++) {
          dk[cc] = fma2(S[cc][r], k2.x, dk[cc]);
          dq[cc] = fma2(S[cc][r], q2.x, dq[cc]);
        }
#pragma unroll
        for (int cc = 0; cc < CC; cc++) {
          dk[cc] = fma2(S[cc][r + 1], k2.y, dk[cc]);
          dq[cc] = fma2(S[cc][r + 1], q2.y, dq[cc]);
        }
      }
      float w[2][CC];  // [k / q][column]
#pragma unroll
      for (int cc = 0; cc < CC; cc++) {
        float x0, x1;
        unpack2(dk[cc], x0, x1);
        w[0][cc] = x0 + x1;
        unpack2(dq[cc], x0, x1);
        w[1][cc] = x0 + x1;
      }
      // halve the columns, then the two kinds, over the lanes; lanes beyond those bits add up
#pragma unroll
      for (int o = 1; o < CC; o <<= 1) {
        const bool up = (p & o) != 0;
#pragma unroll
        for (int t = 0; t < 2; t++)
#pragma unroll
          for (int cc = 0; cc < CC / 2 / o; cc++) {
            const float give = up ? w[t][2 * cc] : w[t][2 * cc + 1], keep = up ? w[t][2 * cc + 1] : w[t][2 * cc];
            w[t][cc] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
      }
      float e = (typ ? w[1][0] : w[0][0]) + __shfl_xor_sync(0xffffffffu, typ ? w[0][0] : w[1][0], CC);
#pragma unroll
      for (int o = 2 * CC; o < LPC; o <<= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
      e *= tk.x;
      const float mine = tk.w * (v - e);  // u on the lanes of typ 0
      const float u = __shfl_sync(0xffffffffu, mine, lane0 + mc);
      if (p >= CC && p < 2 * CC && CC * jl + mc < vcn) og[(size_t)(r0 + t0 + tt) * HV + CC * jl + mc] = fmaf(tk.z, u, e);
      unsigned long long wu[CC];
#pragma unroll
      for (int cc = 0; cc < CC; cc++) {
        const float x = __shfl_sync(0xffffffffu, mine, lane0 + cc) * tk.y;
        wu[cc] = pack2(x, x);
      }
#pragma unroll
      for (int r = 0; r < R / 2; r += 2)
#pragma unroll
        for (int cc = 0; cc < CC; cc++) {
          S[cc][r] = fma2(kr[r], wu[cc], S[cc][r]);
          S[cc][r + 1] = fma2(kr[r + 1], wu[cc], S[cc][r + 1]);
        }
    }
    __syncthreads();  // the buffer and the token values may be refilled
  }
  cp_async_wait<0>();
  if (tid == (int)blockDim.x - 1) mul_s[0] = c_end;
  __syncthreads();
  const float c = mul_s[0];
#pragma unroll
  for (int cc = 0; cc < CC; cc++)
    if (CC * jl + cc < vcn) {
#pragma unroll
      for (int r = 0; r < R; r += 2) {
        float lo, hi;
        unpack2(S[cc][r / 2], lo, hi);
        float* dst = S_g + (size_t)(p * R + r) * vdim + CC * jl + cc;
        dst[0] = c * lo;
        dst[vdim] = c * hi;
      }
    }
  TRACE_EXIT(tr);
}

template <int R, int LPC, int CC>
static cudaError_t delta_scan_packed_launch(cudaStream_t st, const DeltaArgs& a) {
  constexpr int MOST = CC * 128 / LPC;  // columns of 128 threads
  const int VC = std::min(MOST, (a.vdim + CC - 1) / CC * CC);
  const int threads = (VC / CC * LPC + 31) / 32 * 32;
  const dim3 grid(a.n_seqs, a.H, ceil_div(a.vdim, VC));
  const size_t smem = (size_t)2 * DELTA_TT * (2 * LPC * (R + 4) + VC + 2) * sizeof(float);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(delta_scan_packed_kernel<R, LPC, CC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  return launch_k(delta_scan_packed_kernel<R, LPC, CC>, grid, dim3(threads), smem, st, a, VC, next_trace(48));
}

template <int R, int LPC>
static cudaError_t delta_scan_columns_launch(cudaStream_t st, const DeltaArgs& a) {
  // two columns per thread (the key / query reads from shared memory, which bound the one-column
  // form, serve both) when the head has the columns for it
  const bool cc2 = a.vdim >= 2 * (256 / LPC);
  const int VC = std::min((cc2 ? 2 : 1) * (256 / LPC), a.vdim);
  const int threads = cc2 ? 256 : (VC * LPC + 31) / 32 * 32;
  const dim3 grid(a.n_seqs, a.H, ceil_div(a.vdim, VC));
  const size_t smem = (size_t)2 * DELTA_TT * (2 * LPC * (R + 4) + VC + 2) * sizeof(float);
  auto run = [&](auto kernel) -> cudaError_t {
    if (smem > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    return launch_k(kernel, grid, dim3(threads), smem, st, a, VC, next_trace(35));
  };
  return cc2 ? run(delta_scan_columns_kernel<R, LPC, 2>) : run(delta_scan_columns_kernel<R, LPC, 1>);
}

// The packed kernel does less work per token, but its chain from one token to the next is longer (two exchanges between
// lanes more, the multipliers' reads) and several of its small CTAs share an SM even where others are empty: it pays where
// the columns kernel needs a second wave (one CTA of two columns a thread per SM, two of one column) and the sequences
// have some tokens.  16 heads, convolution + scan + norm of a layer, us, columns against packed: 128 x 128, 16 sequences
// of 16 / 64 / 300 tokens 65 / 116 / 504 against 62 / 101 / 427, 32 of 300 994 against 748, but 8 of 300 256 against 321, one
// of 1100 788 against 1190 (the scan alone), decode of 32 48 against 55; 64 x 64, 32 of 64 / 300 85 / 370 against 79 / 331,
// 24 of 300 295 against 300, 16 of 300 187 against 232; 48 x 48, 32 of 300 352 against 330.  Heads of 16, 32, 96 and
// 256 are slower in it at every size (one sequence of 300: 56 against 95, 72 against 134, 133 against 210, 297 against
// 352; 32 of 300: 138 against 181, 181 against 242, 728 against 842, 4700 against 5550).
static bool delta_packed_fits(const DeltaArgs& a) {
  if (a.dim != 48 && a.dim != 64 && a.dim != 128) return false;
  const bool cc2 = a.vdim >= 128;  // two columns per thread in delta_scan_columns_kernel
  const long ctas = (long)a.n_seqs * a.H * ceil_div(a.vdim, cc2 ? 128 : 64);
  return ctas > (cc2 ? 148 : 440) && a.T >= 16 * a.n_seqs;
}
cudaError_t launch_delta_scan(cudaStream_t st, const DeltaArgs& a) {
  if (a.n_seqs <= 0) return cudaSuccess;
  if (a.dim > 1024 || a.H % a.G) return cudaErrorInvalidValue;
  // compile-time sizes for the usual head widths (rows of the step's inputs must be 16-byte aligned)
  static const bool fixed_on = !(getenv("NVLLM_DELTA_FIXED") && atoi(getenv("NVLLM_DELTA_FIXED")) == 0);
  if (fixed_on && a.conv_ch % 4 == 0 && a.n_q % 4 == 0 && a.n_k % 4 == 0) {
    const bool packed = delta_packed_fits(a);
    switch (a.dim) {
      case 16: return delta_scan_columns_launch<4, 4>(st, a);
      case 32: return delta_scan_columns_launch<8, 4>(st, a);
      case 48: return packed ? delta_scan_packed_launch<12, 4, 2>(st, a) : delta_scan_columns_launch<12, 4>(st, a);
      case 64: return packed ? delta_scan_packed_launch<8, 8, 4>(st, a) : delta_scan_columns_launch<16, 4>(st, a);
      case 96: return delta_scan_columns_launch<24, 4>(st, a);
      case 128: return packed ? delta_scan_packed_launch<16, 8, 4>(st, a) : delta_scan_columns_launch<32, 4>(st, a);
      case 256: return delta_scan_columns_launch<32, 8>(st, a);
    }
  }
  // registers per thread R and lanes per column LPC (a power of two): R * LPC >= dim
  int R = 4;
  while (R < 32 && R * 4 < a.dim) R *= 2;
  int LPC = 1;
  while (R * LPC < a.dim) LPC *= 2;
  int VC = 256 / LPC;
  if (VC > a.vdim) VC = a.vdim;
  int threads = VC * LPC;
  threads = (threads + 31) / 32 * 32;  // whole warps: every lane takes part in the shuffles
  const dim3 grid(a.n_seqs, a.H, ceil_div(a.vdim, VC));
  const size_t smem = (size_t)2 * DELTA_TT * (2 * a.dim + VC + 2) * sizeof(float);
#define DS(RR)                                                                                        \
  {                                                                                                   \
    if (smem > 48 * 1024)                                                                             \
      cudaFuncSetAttribute(delta_scan_kernel<RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    (void)launch_k(delta_scan_kernel<RR>, grid, dim3(threads), smem, st, a, LPC, VC, next_trace(35));   \
  }
  if (R == 4) DS(4)
  else if (R == 8) DS(8)
  else if (R == 16) DS(16)
  else DS(32)
#undef DS
  return cudaGetLastError();
}

// ------------------------------------------------------------------ gated norm of the read-out
// heads of up to 128 columns that start on 16-byte boundaries: four columns per lane (bound by memory; 18 k rows of 16
// heads of 128: 83 us, 215 us with 4-byte accesses)
template <typename OT>
__global__ void __launch_bounds__(256) delta_out_vec_kernel(DeltaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  constexpr bool FAST = sizeof(OT) == 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int t = blockIdx.x, vdim = a.vdim;
  const bool on = 4 * lane < vdim;
  const float4 w = on ? *reinterpret_cast<const float4*>(a.onorm_w + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
  pdl_wait();
  if (a.roll) {  // behind delta_step_kernel: the tail of the q and k channels moves on by the row that it left in qkv
    float* tail = a.state_pool + (size_t)a.state_slots[t] * a.slot_floats + a.tail_off;
    for (int c = 4 * (blockIdx.y * blockDim.x + threadIdx.x); c < a.n_q + a.n_k; c += 4 * gridDim.y * blockDim.x) {
      float4 nv[3];
#pragma unroll
      for (int k = 0; k < 3; k++)
        if (k + 2 < a.taps) nv[k] = __ldcg(reinterpret_cast<const float4*>(tail + (size_t)(k + 1) * a.conv_ch + c));
      const float4 last = __ldcg(reinterpret_cast<const float4*>(a.qkv + (size_t)t * a.conv_ch + c));
#pragma unroll
      for (int k = 0; k < 3; k++)
        if (k + 2 < a.taps) *reinterpret_cast<float4*>(tail + (size_t)k * a.conv_ch + c) = nv[k];
      *reinterpret_cast<float4*>(tail + (size_t)(a.taps - 2) * a.conv_ch + c) = last;
    }
  }
  OT* out = (OT*)a.out + (size_t)t * a.o_ld;
  const float* gate = a.in_p + (size_t)t * a.in_ld + a.conv_ch + 2 * a.H + 4 * lane;
  const float* o = a.o + (size_t)t * a.H * vdim + 4 * lane;
  for (int h = blockIdx.y * nw + warp; h < a.H; h += gridDim.y * nw) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 v = on ? *reinterpret_cast<const float4*>(o + (size_t)h * vdim) : zero;
    const float4 g = on ? sum_slices4(gate + (size_t)h * vdim, a.in_S, a.in_stride) : zero;
    const float inv = 1.0f / sqrtf(warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w) / (float)vdim + a.eps);
    const float r[4] = {v.x * inv * w.x * silu_t<FAST>(g.x), v.y * inv * w.y * silu_t<FAST>(g.y),
                        v.z * inv * w.z * silu_t<FAST>(g.z), v.w * inv * w.w * silu_t<FAST>(g.w)};
    if (on) store4(out + h * vdim + 4 * lane, r);
  }
  if (blockIdx.y == 0)
    for (int c = a.H * vdim + threadIdx.x; c < a.o_ld; c += blockDim.x) out[c] = from_f32<OT>(0.f);
  TRACE_EXIT(tr);
}

template <typename OT, int MV>
__global__ void __launch_bounds__(256) delta_out_kernel(DeltaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int vdim = a.vdim;
  OT* out = (OT*)a.out + (size_t)t * a.o_ld;
  const float* gate = a.in_p + (size_t)t * a.in_ld + a.conv_ch + 2 * a.H;
  // heads of up to 32 * MV columns stay in registers: read-outs and gates are loaded together
  constexpr bool FAST = sizeof(OT) == 2;
  for (int h = blockIdx.y * nw + warp; h < a.H; h += gridDim.y * nw) {
    const float* o = a.o + (size_t)t * a.H * vdim + (size_t)h * vdim;
    if (vdim <= 32 * MV) {
      float ov[MV], gv[MV];
#pragma unroll
      for (int c = 0; c < MV; c++) {
        const int i = lane + 32 * c;
        ov[c] = i < vdim ? o[i] : 0.f;
        gv[c] = i < vdim ? sum_slices(gate + h * vdim + i, a.in_S, a.in_stride) : 0.f;
      }
      float ss = 0.f;
#pragma unroll
      for (int c = 0; c < MV; c++) ss += ov[c] * ov[c];
      const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)vdim + a.eps);
#pragma unroll
      for (int c = 0; c < MV; c++) {
        const int i = lane + 32 * c;
        if (i < vdim) out[h * vdim + i] = from_f32<OT>(ov[c] * inv * a.onorm_w[i] * silu_t<FAST>(gv[c]));
      }
      continue;
    }
    float ss = 0.f;
    for (int i = lane; i < vdim; i += 32) ss += o[i] * o[i];
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)vdim + a.eps);
    for (int i = lane; i < vdim; i += 32) {
      const float gt = sum_slices(gate + h * vdim + i, a.in_S, a.in_stride);
      out[h * vdim + i] = from_f32<OT>(o[i] * inv * a.onorm_w[i] * silu(gt));
    }
  }
  if (blockIdx.y == 0)
    for (int c = a.H * vdim + threadIdx.x; c < a.o_ld; c += blockDim.x) out[c] = from_f32<OT>(0.f);
  TRACE_EXIT(tr);
}

static bool delta_out_vec_fits(const DeltaArgs& a) {  // (the gates' columns start behind 2 H entries of the projection)
  return a.vdim <= 128 && a.vdim % 4 == 0 && (a.conv_ch + 2 * a.H) % 4 == 0 && a.in_ld % 4 == 0 && a.in_stride % 4 == 0 && a.o_ld % 4 == 0;
}

// ------------------------------------------------------------------ one token per sequence
// Decode steps, preparation and scan as one launch: a CTA per (sequence, head, 64 value columns) makes its head's q and k
// and its own v itself and holds its DIM x 64 entries of the state, two columns per lane and DIM / 8 rows per warp, in
// registers.  State, tail and filter are loaded before the wait for the projection (the kernels that wrote them belong to
// the step before), so the state streams in under the projection's end; then one round of loads (the projection's
// slices), two block sums.  Bound by the state's stream, once in and once out.  The tail of the v channels moves on here;
// that of q and k, which other CTAs still read, in the kernel behind (roll).  32 sequences, 16 heads of 128 x 128, us a layer
// with the gated norm: 48 -> 20.
constexpr int DS_VC = 64;
__device__ __forceinline__ float sum_slices8(const float* __restrict__ p, int S, size_t stride) {
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = i < S ? p[(size_t)i * stride] : 0.f;  // all in flight
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++)
    if (i < S) acc += v[i];
  return acc;
}
template <int DIM, int TAPS, bool FAST>
__global__ void __launch_bounds__(256, 3) delta_step_kernel(DeltaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  constexpr int RW = DIM / 8, NCH = 2 * DIM + DS_VC, NI = (NCH + 255) / 256;
  __shared__ float qkv[NCH];  // q | k | v
  __shared__ float part[8][DS_VC];
  __shared__ float bg[2];
  const int t = blockIdx.x, h = blockIdx.y, vbase = blockIdx.z * DS_VC;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hpg = a.H / a.G, kvh = h / hpg;
  const int pos = a.positions[t];  // (one row per sequence)
  float* slot = a.state_pool + (size_t)a.state_slots[t] * a.slot_floats;
  float* tail = slot + a.tail_off;
  float2* S_g = reinterpret_cast<float2*>(slot + a.state_off + ((size_t)h * DIM + warp * RW) * a.vdim + vbase) + lane;
  const int ld2 = a.vdim / 2;
  float2 st[RW];
#pragma unroll
  for (int r = 0; r < RW; r++) st[r] = pos > 0 ? __ldcg(S_g + (size_t)r * ld2) : make_float2(0.f, 0.f);
  int ch[NI];
  float old[NI][TAPS - 1], cw[NI][TAPS];
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int j = tid + 256 * i;
    ch[i] = j < DIM ? kvh * DIM + j : j < 2 * DIM ? a.n_q + kvh * DIM + (j - DIM) : a.n_q + a.n_k + h * a.vdim + vbase + (j - 2 * DIM);
    if (j >= NCH) continue;
#pragma unroll
    for (int k = 0; k < TAPS; k++) cw[i][k] = a.conv_w[(size_t)ch[i] * TAPS + k];
#pragma unroll
    for (int k = 0; k + 1 < TAPS; k++) old[i][k] = pos - (TAPS - 1 - k) >= 0 ? __ldcg(tail + (size_t)k * a.conv_ch + ch[i]) : 0.f;
  }
  pdl_wait();
  const float* in = a.in_p + (size_t)t * a.in_ld;
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int j = tid + 256 * i;
    if (j >= NCH) continue;
    const float x = sum_slices8(in + ch[i], a.in_S, a.in_stride);
    float v = 0.f;
#pragma unroll
    for (int k = 0; k + 1 < TAPS; k++) v = fmaf(old[i][k], cw[i][k], v);
    v = fmaf(x, cw[i][TAPS - 1], v);
    qkv[j] = silu_t<FAST>(v);
    if (j >= 2 * DIM) {
#pragma unroll
      for (int k = 0; k + 2 < TAPS; k++) tail[(size_t)k * a.conv_ch + ch[i]] = old[i][k + 1];
      tail[(size_t)(TAPS - 2) * a.conv_ch + ch[i]] = x;
    } else if (blockIdx.z == 0 && h % hpg == 0) {
      a.qkv[(size_t)t * a.conv_ch + ch[i]] = x;  // for the roll
    }
  }
  if (tid >= 254) {
    const float* p = in + a.conv_ch;
    if (tid == 254) bg[0] = 1.0f / (1.0f + expf(-sum_slices8(p + h, a.in_S, a.in_stride)));
    else bg[1] = expf(-expf(a.a_log[h]) * softplus(sum_slices8(p + a.H + h, a.in_S, a.in_stride) + a.dt_bias[h]));
  }
  __syncthreads();
  if (warp < 2) {  // unit lengths of q and k; the query also carries 1 / sqrt(dim)
    float* v = qkv + warp * DIM;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < DIM / 32; i++) ss += v[lane + 32 * i] * v[lane + 32 * i];
    float mul = 1.0f / sqrtf(warp_sum(ss) + 1e-6f);
    if (warp == 0) mul *= 1.0f / sqrtf((float)DIM);
#pragma unroll
    for (int i = 0; i < DIM / 32; i++) v[lane + 32 * i] *= mul;
  }
  __syncthreads();
  const float beta = bg[0], g = bg[1];
  const float *q = qkv + warp * RW, *k = qkv + DIM + warp * RW;
  auto column_sum = [&](float2 mine) {  // over the warps, every thread its two columns
    *reinterpret_cast<float2*>(&part[warp][2 * lane]) = mine;
    __syncthreads();
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int w = 0; w < 8; w++) {
      const float2 o = *reinterpret_cast<const float2*>(&part[w][2 * lane]);
      s.x += o.x;
      s.y += o.y;
    }
    return s;
  };
  float2 acc = make_float2(0.f, 0.f);
#pragma unroll
  for (int r = 0; r < RW; r++) {
    st[r].x *= g;
    st[r].y *= g;
    acc.x = fmaf(st[r].x, k[r], acc.x);
    acc.y = fmaf(st[r].y, k[r], acc.y);
  }
  const float2 sk = column_sum(acc);
  const float2 v = *reinterpret_cast<const float2*>(&qkv[2 * DIM + 2 * lane]);
  const float2 u = make_float2(beta * (v.x - sk.x), beta * (v.y - sk.y));
  acc = make_float2(0.f, 0.f);
#pragma unroll
  for (int r = 0; r < RW; r++) {
    st[r].x = fmaf(k[r], u.x, st[r].x);
    st[r].y = fmaf(k[r], u.y, st[r].y);
    S_g[(size_t)r * ld2] = st[r];
    acc.x = fmaf(st[r].x, q[r], acc.x);
    acc.y = fmaf(st[r].y, q[r], acc.y);
  }
  __syncthreads();  // `part` has been read
  const float2 o = column_sum(acc);
  if (warp == 0) *reinterpret_cast<float2*>(a.o + (size_t)t * a.H * a.vdim + (size_t)h * a.vdim + vbase + 2 * lane) = o;
  TRACE_EXIT(tr);
}
// sizes that divide into the kernel's tiles, a read-out that the vector form of the gated norm takes (it rolls the tail)
bool delta_step_fits(const DeltaArgs& a) {
  return a.T == a.n_seqs && (a.dim == 64 || a.dim == 128) && a.vdim % DS_VC == 0 && a.taps >= 2 && a.taps <= 4 && a.in_S <= 8 &&
         a.H % a.G == 0 && delta_out_vec_fits(a) && a.n_q % 4 == 0 && a.n_k % 4 == 0 && a.conv_ch % 4 == 0 && a.tail_off % 4 == 0 &&
         a.state_off % 2 == 0 && a.slot_floats % 4 == 0;
}
template <int DIM, int TAPS>
static cudaError_t delta_step_launch(cudaStream_t st, const DeltaArgs& a) {
  const dim3 grid(a.T, a.H, a.vdim / DS_VC);
  return a.fast_act ? launch_k(delta_step_kernel<DIM, TAPS, true>, grid, dim3(256), 0, st, a, next_trace(51))
                    : launch_k(delta_step_kernel<DIM, TAPS, false>, grid, dim3(256), 0, st, a, next_trace(51));
}
cudaError_t launch_delta_step(cudaStream_t st, const DeltaArgs& a) {
  if (a.T <= 0) return cudaSuccess;
  if (!delta_step_fits(a)) return cudaErrorInvalidValue;
  if (a.dim == 64) return a.taps == 4 ? delta_step_launch<64, 4>(st, a) : a.taps == 3 ? delta_step_launch<64, 3>(st, a) : delta_step_launch<64, 2>(st, a);
  return a.taps == 4 ? delta_step_launch<128, 4>(st, a) : a.taps == 3 ? delta_step_launch<128, 3>(st, a) : delta_step_launch<128, 2>(st, a);
}

cudaError_t launch_delta_out(cudaStream_t st, int odt, const DeltaArgs& a) {
  if (a.T <= 0) return cudaSuccess;
  const dim3 grid(a.T, a.T >= 1024 ? 1 : ceil_div(a.H, 8));  // few rows (decode): a row's heads spread over several CTAs
  if (a.roll && !delta_out_vec_fits(a)) return cudaErrorInvalidValue;
  if (delta_out_vec_fits(a))
    return odt == DT_F32 ? launch_k(delta_out_vec_kernel<float>, grid, dim3(256), 0, st, a, next_trace(36))
                         : launch_k(delta_out_vec_kernel<bf16>, grid, dim3(256), 0, st, a, next_trace(36));
  if (odt == DT_F32) (void)launch_k(delta_out_kernel<float, 8>, grid, dim3(256), 0, st, a, next_trace(36));
  else if (a.vdim <= 128) (void)launch_k(delta_out_kernel<bf16, 4>, grid, dim3(256), 0, st, a, next_trace(36));
  else (void)launch_k(delta_out_kernel<bf16, 8>, grid, dim3(256), 0, st, a, next_trace(36));
  return cudaGetLastError();
}

}  // namespace nvllm
