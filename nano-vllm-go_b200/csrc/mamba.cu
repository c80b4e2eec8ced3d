// mamba.cu — Mamba2 block of the Granite-4 hybrid (purego/tensor/mamba2.go:72-351), for a ragged batch of sequences.  The two projections are
// ordinary GEMMs (forward.cu); this file holds what sits between them:
//   mamba_conv_rows_kernel  sum of the in_proj split-K slices, causal conv1d over the xBC columns
//                       (zero-padded at the start of every CALL, like causalConv1d :209-270 — the
//                       reference never reads its ConvCache), SiLU; dt = softplus(dt + bias) and the
//                       head's decay exp(-exp(A_log) dt)
//   mamba_scan_tile_kernel  the selective scan (:273-351), sequential over a sequence's new tokens;
//                       the SSM state lives per KV BLOCK (handle.h) and is read / written through
//                       the block table
//   mamba_gate_norm_kernel  y * silu(gate), RMS norm over E with eps 1e-5, * Norm (:139-173)
// mamba_conv_kernel and mamba_scan_kernel take what the first two do not: decode and other short steps (the
// convolution), taps other than 4, rows or heads that are no multiples of 16 bytes, states other than 16 / 32 / 64 / 128.
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

// 16-byte accesses of the row kernels: four neighbouring channels per thread
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 sum_slices4(const float* __restrict__ p, int S, size_t stride) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s = 0; s < S; s++) {
    const float4 v = ld4(p + (size_t)s * stride);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  return acc;
}
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void st4(bf16* p, float a, float b, float c, float d) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&lo);
  u.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = u;
}

// step size softplus(z) (mamba2.go:369-376) and decay exp(-exp(A_log) dt) of a (token, head), through double
__device__ __forceinline__ void store_step(const MambaArgs& a, int t, int h, float z) {
  const float dt = (float)log(1.0 + exp((double)z));
  const float A = a.a_log ? -(float)exp((double)a.a_log[h]) : 0.f;
  a.dt[(size_t)t * a.nh + h] = make_float2(dt, a.a_log ? (float)exp((double)(A * dt)) : 1.0f);
}

}  // namespace

// grid (T, ceil(conv / 256)); proj: [S][T][P] split-K slices of x @ in_proj^T, columns
// [gate (E) | xBC (conv) | dt (heads)]
__global__ void __launch_bounds__(256)
mamba_conv_kernel(MambaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int s = seq_of_row(a.cu_q, a.n_seqs, t);
  const int li = t - a.cu_q[s];  // index of the token inside this call's rows of its sequence
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c < a.conv) {
    float sum = 0.f;
    for (int k = 0; k < a.K; k++) {
      const int back = a.K - 1 - k;  // tap k reads the token `back` rows earlier
      if (li - back >= 0)
        sum += sum_slices(a.proj + (size_t)(t - back) * a.P + a.E + c, a.S, a.stride) * a.conv_w[c * a.K + k];
    }
    if (a.conv_b) sum += a.conv_b[c];
    a.xbc[(size_t)t * a.conv + c] = silu(sum);
  }
  if (blockIdx.y == 0 && threadIdx.x < a.nh) {
    const int h = threadIdx.x;
    float dt = sum_slices(a.proj + (size_t)t * a.P + a.E + a.conv + h, a.S, a.stride);
    if (a.dt_bias) dt += a.dt_bias[h];
    store_step(a, t, h, dt);
  }
  TRACE_EXIT(tr);
}

// grid (n_seqs, heads), block = head_dim threads (thread d owns state[d][0..N))
template <int NMAX>
__global__ void __launch_bounds__(128)
mamba_scan_kernel(MambaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float sB[NMAX], sC[NMAX];
  const int s = blockIdx.x, h = blockIdx.y, d = threadIdx.x;
  const int r0 = a.cu_q[s], r1 = a.cu_q[s + 1];
  const int start = a.positions[r0];  // position of the first new token
  const int* bt = a.block_tables + (size_t)s * a.max_blocks;
  const size_t per_layer = (size_t)a.nh * a.hd * a.N;
  const size_t per_block = (size_t)a.n_mamba * per_layer;
  float st[NMAX];
#pragma unroll
  for (int i = 0; i < NMAX; i++) st[i] = 0.f;
  if (start > 0 && d < a.hd) {
    // the state after position start - 1 sits in that position's block
    const float* src = a.ssm_pool + (size_t)bt[(start - 1) / KV_BLOCK] * per_block + (size_t)a.layer * per_layer +
                       ((size_t)h * a.hd + d) * a.N;
#pragma unroll
    for (int i = 0; i < NMAX; i++)
      if (i < a.N) st[i] = src[i];
  }
  int grp = h * a.G / a.nh;
  if (grp >= a.G) grp = a.G - 1;
  const float Dh = a.d_skip ? a.d_skip[h] : 0.f;
  for (int t = r0; t < r1; t++) {
    __syncthreads();  // the previous token's sB / sC have been consumed
    for (int i = threadIdx.x; i < a.N; i += blockDim.x) {
      sB[i] = a.xbc[(size_t)t * a.conv + a.E + (size_t)grp * a.N + i];
      sC[i] = a.xbc[(size_t)t * a.conv + a.E + (size_t)a.G * a.N + (size_t)grp * a.N + i];
    }
    __syncthreads();
    if (d < a.hd) {
      const float2 step = a.dt[(size_t)t * a.nh + h];
      const float dt = step.x, abar = step.y;
      const float u = a.xbc[(size_t)t * a.conv + (size_t)h * a.hd + d];
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < NMAX; i++)
        if (i < a.N) {
          st[i] = abar * st[i] + dt * sB[i] * u;  // mamba2.go:325-331
          sum += sC[i] * st[i];                   // :335-340, s ascending
        }
      a.y[(size_t)t * a.E + (size_t)h * a.hd + d] = sum + Dh * u;
      const int pos = start + (t - r0);
      if ((pos + 1) % KV_BLOCK == 0 || t == r1 - 1) {
        // snapshot: the state after the last token written into this block
        float* dst = a.ssm_pool + (size_t)bt[pos / KV_BLOCK] * per_block + (size_t)a.layer * per_layer +
                     ((size_t)h * a.hd + d) * a.N;
#pragma unroll
        for (int i = 0; i < NMAX; i++)
          if (i < a.N) dst[i] = st[i];
      }
    }
  }
  TRACE_EXIT(tr);
}

// ------------------------------------------------------------------ block-pooled path, 16-byte rows
// Rows, segments and split-K slices of the projection start on 16-byte boundaries (E is a multiple of 8).
static bool mamba_rows_aligned(const MambaArgs& a) { return a.P % 4 == 0 && a.conv % 4 == 0 && a.stride % 4 == 0; }

// Convolution of MC_ROWS neighbouring rows, four channels per thread: the K taps of a channel quad stay in
// registers and every row of the projection is read once per window instead of once per tap (bound by memory:
// one read of the xBC columns and one write).  blockIdx.y == 0 also makes the steps and decays of its rows.
// 16 sequences of 256 to 512 tokens (6446 rows), 6144 channels: 131 us (2.4 TB/s), 465 us with one channel and token
// per thread and K strided loads each.
constexpr int MC_ROWS = 8;
template <int K>
__global__ void __launch_bounds__(256) mamba_conv_rows_kernel(MambaArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  const int t0 = blockIdx.x * MC_ROWS, t1 = min(a.T, t0 + MC_ROWS);
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  float wv[4][K], bias[4] = {0.f, 0.f, 0.f, 0.f};  // immutable: fetched before the dependency resolves
  if (c < a.conv) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
      for (int k = 0; k < K; k++) wv[q][k] = a.conv_w[(size_t)(c + q) * K + k];
      if (a.conv_b) bias[q] = a.conv_b[c + q];
    }
  }
  pdl_wait();
  int s = seq_of_row(a.cu_q, a.n_seqs, t0);
  int first = a.cu_q[s], last = a.cu_q[s + 1];  // rows of the sequence that the current row belongs to
  if (c < a.conv) {
    float4 u[K];  // the window: u[K - 1] is the current row's input
#pragma unroll
    for (int k = 0; k + 1 < K; k++) {
      const int t = t0 - (K - 1) + k;
      u[k + 1] = t >= first ? sum_slices4(a.proj + (size_t)t * a.P + a.E + c, a.S, a.stride) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int t = t0; t < t1; t++) {
      while (t >= last) {
        s++;
        first = last;
        last = a.cu_q[s + 1];
      }
#pragma unroll
      for (int k = 0; k + 1 < K; k++) {
        u[k] = u[k + 1];
        if (t - (K - 1 - k) < first) u[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      u[K - 1] = sum_slices4(a.proj + (size_t)t * a.P + a.E + c, a.S, a.stride);
      float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < K; k++) {
        y[0] += u[k].x * wv[0][k]; y[1] += u[k].y * wv[1][k];
        y[2] += u[k].z * wv[2][k]; y[3] += u[k].w * wv[3][k];
      }
      st4(a.xbc + (size_t)t * a.conv + c, silu(y[0] + bias[0]), silu(y[1] + bias[1]), silu(y[2] + bias[2]), silu(y[3] + bias[3]));
    }
  }
  if (blockIdx.y == 0)
    for (int i = threadIdx.x; i < (t1 - t0) * a.nh; i += blockDim.x) {
      const int t = t0 + i / a.nh, h = i % a.nh;
      const float z = sum_slices(a.proj + (size_t)t * a.P + a.E + a.conv + h, a.S, a.stride);
      store_step(a, t, h, a.dt_bias ? z + a.dt_bias[h] : z);
    }
  TRACE_EXIT(tr);
}

// Selective scan.  L lanes share R rows of a head's state (lane q holds entries 4 L j + 4 q .. + 3 of each, as packed
// pairs in registers), L hd / R threads make a head and HPC heads of one group a CTA.  Per token a lane reads N / L
// entries of B and of C for R N / L state entries and spends three packed instructions per entry pair; the L partial
// read-outs of a row meet by shuffles that scatter the rows over the lanes.  B, C, u and the (step, decay) pairs of the
// next MS_TC tokens arrive by cp.async under the current ones.
// Two fp32 operations per state entry and token: the state is kept as S / c, c the product of the decays since the chunk
// of tokens began, so a token adds (dt u / c) B and reads c (S / c) C; the state is multiplied by the last chunk's c when
// the next one begins, and by c inside one whenever that falls below 1e-18 (nothing leaves fp32's range).  c and
// dt / c are made once per token and head.
// Bound by instruction issue, half of it those operations; a 16-byte read of shared memory brings eight different pieces
// to eight lanes (four lanes per row where the state has only 16 entries).  6446 rows in 16 sequences, 64 heads of
// 64 x 128: 582 us (659 with the CTAs in the order of the sequences: 1024 of them in 592 places); before that, 730 us with
// four lanes and three operations per entry, 7405 us with a thread per row, scalar
// operations and the decay computed in every thread.  The order comes from the host, which knows the lengths, and only where
// they differ: counted in every CTA it made a decode step of 128 / 256 / 512 sequences (one such layer and one of attention)
// 305 / 746 / 3120 us long, 280 / 483 / 816 so.  Half the rows per lane doubles the threads of a head when few
// (sequence, head) pairs are to be shared out.
constexpr int MS_TC = 16;
constexpr float MS_RESCALE = 1e-18f;
constexpr int MS_MAX_HPC = 16;  // heads of a CTA
template <int R, int L, int NJ>
__global__ void __launch_bounds__(512) mamba_scan_tile_kernel(MambaArgs a, int hpc, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  constexpr int N = 4 * L * NJ;
  extern __shared__ __align__(16) float sm[];
  __shared__ float4 tok_s[2 * MS_TC * MS_MAX_HPC];  // [half][token][head]: c, dt / c, what multiplies the state before it
  const int tid = threadIdx.x, nt = blockDim.x, tph = L * a.hd / R;
  const int hl = tid / tph, ht = tid % tph, q = ht % L, d0 = ht / L * R;
  const int uw = hpc * a.hd, row = 2 * N + uw + 2 * hpc;  // floats of a staged token: B | C | u | (step, decay)
  const int rowp = (row + 3) & ~3;
  pdl_wait();
  // the CTAs of the longest sequence first, then the next one's: what starts last, in SMs that others have left, is short
  int s = blockIdx.x, part = blockIdx.y;
  if (a.order) {
    const int at = blockIdx.x + gridDim.x * blockIdx.y;
    part = at % gridDim.y;
    s = a.order[at / gridDim.y];
  }
  const int h0 = part * hpc, h = h0 + hl;
  const int r0 = a.cu_q[s], r1 = a.cu_q[s + 1];
  if (r0 >= r1) return;
  const int start = a.positions[r0];  // position of the first new token
  const int* bt = a.block_tables + (size_t)s * a.max_blocks;
  const size_t per_layer = (size_t)a.nh * a.hd * N;
  const size_t per_block = (size_t)a.n_mamba * per_layer;
  const size_t mine = (size_t)a.layer * per_layer + ((size_t)h * a.hd + d0) * N + 4 * q;
  const int grp = h0 / (a.nh / a.G);
  const float* base = a.xbc + a.E + (size_t)grp * N;
  auto fetch = [&](int t0, int buf) {
    const int n = min(MS_TC, r1 - t0);
    float* dst = sm + buf * MS_TC * rowp;
    for (int i = tid; i < n * (N / 2 + uw / 4); i += nt) {
      const int t = i / (N / 2 + uw / 4), p = i % (N / 2 + uw / 4);
      const float* x = a.xbc + (size_t)(t0 + t) * a.conv;
      const float* src = p < N / 4 ? base + (size_t)(t0 + t) * a.conv + 4 * p
                         : p < N / 2 ? base + (size_t)(t0 + t) * a.conv + (size_t)a.G * N + 4 * (p - N / 4)
                                     : x + (size_t)h0 * a.hd + 4 * (p - N / 2);
      cp_async16(smem_addr(dst + t * rowp + 4 * p), src, true);
    }
    for (int i = tid; i < n * hpc; i += nt) {
      const int t = i / hpc, k = i % hpc;
      *reinterpret_cast<float2*>(dst + t * rowp + 2 * N + uw + 2 * k) = a.dt[(size_t)(t0 + t) * a.nh + h0 + k];
    }
    cp_async_commit();
  };
  fetch(r0, 0);
  unsigned long long st[R][2 * NJ];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int j = 0; j < 2 * NJ; j++) st[r][j] = 0ull;
  if (start > 0) {
    // the state after position start - 1 sits in that position's block
    const float* src = a.ssm_pool + (size_t)bt[(start - 1) / KV_BLOCK] * per_block + mine;
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src + (size_t)r * N + 4 * L * j);
        st[r][2 * j] = v.x;
        st[r][2 * j + 1] = v.y;
      }
  }
  const float Dh = a.d_skip ? a.d_skip[h] : 0.f;
  auto scale = [&](float m) {
    const unsigned long long mm = pack2(m, m);
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int j = 0; j < 2 * NJ; j++) st[r][j] = mul2(st[r][j], mm);
  };
  float c_end = 1.f;  // c after the last token
  for (int t0 = r0, buf = 0; t0 < r1; t0 += MS_TC, buf ^= 1) {
    cp_async_wait<0>();
    __syncthreads();  // this chunk has arrived, and everybody is done with the other buffer
    const int n = min(MS_TC, r1 - t0);
    for (int i = tid; i < n * hpc; i += nt) {  // token t of head k: the decays up to it
      const int t = i / hpc, k = i % hpc;
      const float* w = sm + buf * MS_TC * rowp + 2 * N + uw + 2 * k;
      float c = 1.f, m = 1.f;
      for (int j = 0; j <= t; j++) {
        c *= w[j * rowp + 1];
        m = 1.f;
        if (c < MS_RESCALE) {
          m = c;
          c = 1.f;
        }
      }
      tok_s[(buf * MS_TC + t) * MS_MAX_HPC + k] = make_float4(c, w[t * rowp] / c, m, 0.f);
    }
    if (t0 + MS_TC < r1) fetch(t0 + MS_TC, buf ^ 1);
    __syncthreads();
    if (c_end != 1.f) scale(c_end);
    float* yp = a.y + (size_t)t0 * a.E + (size_t)h * a.hd + d0 + q;
    // snapshots: the state after the last token written into a block
    const int pos0 = start + (t0 - r0);
    int snap = min(KV_BLOCK - 1 - pos0 % KV_BLOCK, r1 - 1 - t0);
    for (int t = 0; t < n; t++, yp += a.E) {
      const float* x = sm + (buf * MS_TC + t) * rowp;
      const float4 tk = tok_s[(buf * MS_TC + t) * MS_MAX_HPC + hl];
      const float* u = x + 2 * N + hl * a.hd + d0;
      if (tk.z != 1.f) scale(tk.z);
      c_end = tk.x;
      unsigned long long du[R], acc[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        const float v = tk.y * u[r];
        du[r] = pack2(v, v);
      }
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        const ulonglong2 B = *reinterpret_cast<const ulonglong2*>(x + 4 * L * j + 4 * q);
        const ulonglong2 Cc = *reinterpret_cast<const ulonglong2*>(x + N + 4 * L * j + 4 * q);
#pragma unroll
        for (int r = 0; r < R; r++) {
          st[r][2 * j] = fma2(du[r], B.x, st[r][2 * j]);  // mamba2.go:325-331
          st[r][2 * j + 1] = fma2(du[r], B.y, st[r][2 * j + 1]);
          acc[r] = j == 0 ? mul2(Cc.x, st[r][0]) : fma2(Cc.x, st[r][2 * j], acc[r]);  // :335-340
          acc[r] = fma2(Cc.y, st[r][2 * j + 1], acc[r]);
        }
      }
      float y[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        float lo, hi;
        unpack2(acc[r], lo, hi);
        y[r] = lo + hi;
      }
      // lanes q < R end up with row d0 + q
#pragma unroll
      for (int o = 1; o < R; o <<= 1) {
        const bool up = (q & o) != 0;
#pragma unroll
        for (int r = 0; r < R / 2 / o; r++) {
          const float give = up ? y[2 * r] : y[2 * r + 1], keep = up ? y[2 * r + 1] : y[2 * r];
          y[r] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
      float out = y[0];
#pragma unroll
      for (int o = R; o < L; o <<= 1) out += __shfl_xor_sync(0xffffffffu, out, o);
      if (q < R) *yp = tk.x * out + Dh * u[q];
      if (t == snap) {
        snap = min(snap + KV_BLOCK, r1 - 1 - t0);
        float* dst = a.ssm_pool + (size_t)bt[(pos0 + t) / KV_BLOCK] * per_block + mine;
        const unsigned long long cc = pack2(tk.x, tk.x);
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
          for (int j = 0; j < NJ; j++)
            *reinterpret_cast<ulonglong2*>(dst + (size_t)r * N + 4 * L * j) =
                make_ulonglong2(mul2(st[r][2 * j], cc), mul2(st[r][2 * j + 1], cc));
      }
    }
  }
  TRACE_EXIT(tr);
}

// one CTA per token row: y[t, :] * silu(gate[t, :]) -> RMS norm (eps 1e-5, mamba2.go:150-166)
// -> * Norm -> act dtype (the out_proj GEMM's input).  V = 4: 16-byte accesses (aligned rows): 68 us for 6446 rows
// of 4096 (bound by memory: gates, scan outputs and results once), 129 us with 4-byte ones.
template <typename OT, int V>
__global__ void __launch_bounds__(256)
mamba_gate_norm_kernel(MambaArgs a, OT* __restrict__ out, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float row[];
  __shared__ float red[32];
  const int t = blockIdx.x;
  float lsq = 0.f;
  for (int i = threadIdx.x * V; i < a.E; i += blockDim.x * V) {
    const float* g = a.proj + (size_t)t * a.P + i;
    const float* y = a.y + (size_t)t * a.E + i;
    if constexpr (V == 4) {
      const float4 g4 = sum_slices4(g, a.S, a.stride), y4 = ld4(y);
      const float4 v = make_float4(y4.x * silu(g4.x), y4.y * silu(g4.y), y4.z * silu(g4.z), y4.w * silu(g4.w));
      st4(row + i, v.x, v.y, v.z, v.w);
      lsq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    } else {
      const float v = *y * silu(sum_slices(g, a.S, a.stride));
      row[i] = v;
      lsq += v * v;
    }
  }
  const float tot = block_sum(lsq, red);
  const float rms = 1.0f / sqrtf(tot / (float)a.E + 1e-5f);
  OT* o = out + (size_t)t * a.E;
  for (int i = threadIdx.x * V; i < a.E; i += blockDim.x * V) {
    if constexpr (V == 4) {
      const float4 v = ld4(row + i), w = a.norm_w ? ld4(a.norm_w + i) : make_float4(1.f, 1.f, 1.f, 1.f);
      st4(o + i, v.x * rms * w.x, v.y * rms * w.y, v.z * rms * w.z, v.w * rms * w.w);
    } else {
      o[i] = from_f32<OT>(row[i] * rms * (a.norm_w ? a.norm_w[i] : 1.f));
    }
  }
  TRACE_EXIT(tr);
}

// ------------------------------------------------------------------ Mamba-2 with state slots
// The Mamba-2 mixer of a model given as a list of layers (forward_layered.cu).  Its state
// S (N x vdim per head, fp32) and the last taps - 1 inputs of its convolution live in the
// sequence's state slot; the recurrence itself runs in the linear-recurrence scan of linrec.cu.
//   mamba2_slot_prep_kernel  one CTA per token: split-K sum of the input projection, causal convolution
//                            over x | B | C (inputs before the step's first row from the slot's tail, zeros
//                            before the sequence's start), + bias, SiLU; dt = softplus(dt + bias) (fp32, no
//                            clamp), the head's decay exp(-exp(A_log) dt), and dt x (the scan's values)
//   mamba2_slot_out_kernel   one CTA per token: y = read-out + D x, times silu(z), RMS norm in norm_groups
//                            equal parts (eps of the model), times the weight -> act dtype
// every row, segment and tail of the two kernels starts on a 16-byte boundary
__device__ __forceinline__ bool m2_rows_aligned(const Mamba2SlotArgs& a) {
  const int inner = a.heads * a.vdim, gn = a.G * a.N;
  return (a.vdim % 4 == 0) && (gn % 4 == 0) && (a.in_ld % 4 == 0) && (a.in_stride % 4 == 0) && (inner % 4 == 0);
}

template <int TAPS>
__global__ void __launch_bounds__(256) mamba2_slot_prep_kernel(Mamba2SlotArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  constexpr int MT = TAPS > 0 ? TAPS : 8;
  const int taps = TAPS > 0 ? TAPS : a.taps;
  const int t = blockIdx.x;
  const int inner = a.heads * a.vdim, ch = inner + 2 * a.G * a.N;
  __shared__ int s_seq;
  __shared__ float s_dt[256];
  if (a.T == a.n_seqs) {
    if (threadIdx.x == 0) s_seq = t;
  } else {
    for (int i = threadIdx.x; i < a.n_seqs; i += blockDim.x)
      if (a.cu_q[i] <= t && t < a.cu_q[i + 1]) s_seq = i;
  }
  // step sizes and decays of the heads (at most 256 heads)
  for (int hh = threadIdx.x; hh < a.heads; hh += blockDim.x) {
    const float z = sum_slices(a.in_p + (size_t)t * a.in_ld + inner + ch + hh, a.in_S, a.in_stride) + a.dt_bias[hh];
    const float dt = z > 20.f ? z : log1pf(expf(z));  // softplus; above 20 the two agree to fp32 rounding
    s_dt[hh] = dt;
    a.decay[(size_t)t * a.heads + hh] = expf(-expf(a.a_log[hh]) * dt);
  }
  __syncthreads();
  const int s = s_seq;
  const int li = t - a.cu_q[s], pos = a.positions[t], keep = taps - 1;
  const float* tail = a.state_pool + (size_t)a.state_slots[s] * a.slot_floats + a.tail_off;
  const float* src[MT];
  bool part[MT];  // the row is one of this step's partials (slices to sum)
#pragma unroll
  for (int j = 0; j < MT; j++) {
    src[j] = nullptr;
    part[j] = false;
    if (j < taps) {
      const int back = keep - j;
      if (back <= li) { src[j] = a.in_p + (size_t)(t - back) * a.in_ld + inner; part[j] = true; }
      else if (back <= pos) src[j] = tail + (size_t)(keep - (back - li)) * ch;
    }
  }
  const bool one = a.in_S == 1;
  if (TAPS == 4 && m2_rows_aligned(a)) {
    // four channels per thread: their 16 taps are 64 contiguous bytes, every tap's inputs one 16-byte load
    for (int c = threadIdx.x * 4; c < ch; c += blockDim.x * 4) {
      float y[4], wv[4][4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float4 w4 = ld4(a.conv_w + (size_t)(c + k) * 4);
        wv[k][0] = w4.x; wv[k][1] = w4.y; wv[k][2] = w4.z; wv[k][3] = w4.w;
        y[k] = a.conv_b ? a.conv_b[c + k] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (!src[j]) continue;  // before the sequence's start: zeros
        const float4 u = (one || !part[j]) ? ld4(src[j] + c) : sum_slices4(src[j] + c, a.in_S, a.in_stride);
        y[0] = fmaf(wv[0][j], u.x, y[0]); y[1] = fmaf(wv[1][j], u.y, y[1]);
        y[2] = fmaf(wv[2][j], u.z, y[2]); y[3] = fmaf(wv[3][j], u.w, y[3]);
      }
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; k++) v[k] = a.fast_act ? __fdividef(y[k], 1.0f + __expf(-y[k])) : silu(y[k]);
      st4(a.xbc + (size_t)t * ch + c, v[0], v[1], v[2], v[3]);
      if (c < inner) {
        const float dt = s_dt[c / a.vdim];
        st4(a.dtx + (size_t)t * inner + c, v[0] * dt, v[1] * dt, v[2] * dt, v[3] * dt);
      }
    }
    TRACE_EXIT(tr);
    return;
  }
  for (int c = threadIdx.x; c < ch; c += blockDim.x) {
    float u[MT], wv[MT];
#pragma unroll
    for (int j = 0; j < MT; j++) {
      u[j] = 0.f;
      wv[j] = j < taps ? a.conv_w[(size_t)c * taps + j] : 0.f;
      if (j < taps && src[j]) u[j] = (one || !part[j]) ? src[j][c] : sum_slices(src[j] + c, a.in_S, a.in_stride);
    }
    float y = a.conv_b ? a.conv_b[c] : 0.f;
#pragma unroll
    for (int j = 0; j < MT; j++) y = fmaf(wv[j], u[j], y);
    const float v = a.fast_act ? __fdividef(y, 1.0f + __expf(-y)) : silu(y);
    a.xbc[(size_t)t * ch + c] = v;
    if (c < inner) a.dtx[(size_t)t * inner + c] = v * s_dt[c / a.vdim];
  }
  TRACE_EXIT(tr);
}

template <typename OT>
__global__ void __launch_bounds__(256) mamba2_slot_out_kernel(Mamba2SlotArgs a, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float row[];
  __shared__ float ginv[64];
  const int t = blockIdx.x;
  const int inner = a.heads * a.vdim, ch = inner + 2 * a.G * a.N;
  const int part = inner / a.norm_groups;
  const bool vec = m2_rows_aligned(a);
  if (vec) {
    for (int i = threadIdx.x * 4; i < inner; i += blockDim.x * 4) {
      const float4 z = sum_slices4(a.in_p + (size_t)t * a.in_ld + i, a.in_S, a.in_stride);
      const float4 x = ld4(a.xbc + (size_t)t * ch + i);
      const float4 o = ld4(a.o + (size_t)t * inner + i);
      const float d = a.d_skip[i / a.vdim];
      const float zz[4] = {z.x, z.y, z.z, z.w};
      const float yy[4] = {o.x + d * x.x, o.y + d * x.y, o.z + d * x.z, o.w + d * x.w};
#pragma unroll
      for (int k = 0; k < 4; k++) row[i + k] = yy[k] * (a.fast_act ? __fdividef(zz[k], 1.0f + __expf(-zz[k])) : silu(zz[k]));
    }
  } else {
    for (int i = threadIdx.x; i < inner; i += blockDim.x) {
      const float z = sum_slices(a.in_p + (size_t)t * a.in_ld + i, a.in_S, a.in_stride);
      const float x = a.xbc[(size_t)t * ch + i];
      const float y = a.o[(size_t)t * inner + i] + a.d_skip[i / a.vdim] * x;
      row[i] = y * (a.fast_act ? __fdividef(z, 1.0f + __expf(-z)) : silu(z));
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int g = warp; g < a.norm_groups; g += nw) {
    float sq = 0.f;
    for (int i = lane; i < part; i += 32) {
      const float v = row[g * part + i];
      sq = fmaf(v, v, sq);
    }
    sq = warp_sum(sq);
    if (lane == 0) ginv[g] = 1.0f / sqrtf(sq / (float)part + a.eps);
  }
  __syncthreads();
  OT* op = (OT*)a.out + (size_t)t * a.o_ld;
  if (vec && part % 4 == 0 && a.o_ld % 4 == 0) {
    for (int i = threadIdx.x * 4; i < a.o_ld; i += blockDim.x * 4) {
      if (i < inner) {  // inner and o_ld are multiples of 4: a quad is all inside or all padding
        const float4 r4 = ld4(row + i), w4 = ld4(a.norm_w + i);
        const float gi = ginv[i / part];
        st4(op + i, r4.x * gi * w4.x, r4.y * gi * w4.y, r4.z * gi * w4.z, r4.w * gi * w4.w);
      } else {
        st4(op + i, 0.f, 0.f, 0.f, 0.f);
      }
    }
  } else {
    for (int i = threadIdx.x; i < a.o_ld; i += blockDim.x)
      op[i] = from_f32<OT>(i < inner ? row[i] * ginv[i / part] * a.norm_w[i] : 0.f);
  }
  TRACE_EXIT(tr);
}

// Steps with one row per sequence: convolution, step size, decay and the recurrence of a (sequence, head)
// pair as ONE launch (mamba2_slot_prep_kernel and the scan of linrec.cu in one).  CTA = (sequence, head), 256
// threads.  Phase 1: the head's step size and decay; the convolution (+ bias, SiLU) of the head's vdim
// channels of x and of its group's N channels of B and of C into shared memory (the x channels also to xbc,
// where mamba2_slot_out_kernel reads them for the D skip).  Phase 2: the head's state [N][vdim] goes once
// through the registers, VW columns per thread and 256 / (vdim / VW) rows in flight:
// S <- decay S + B_n (dt x_p), y_p += S C_n, written back in place; the rows' partial read-outs meet in shared
// memory.  A sequence at position 0 starts from zeros whatever the slot holds.
// VW = 4: 16-byte loads and stores (vdim a multiple of 4); VW = 1 otherwise.
constexpr int M2D_THREADS = 256;
template <int TAPS, int VW>
__global__ void __launch_bounds__(M2D_THREADS) mamba2_slot_decode_kernel(Mamba2SlotArgs a, float* __restrict__ o, Trace tr) {
  TRACE_ENTRY(tr);
  pdl_launch_dependents();
  pdl_wait();
  constexpr int MT = TAPS > 0 ? TAPS : 8;
  const int taps = TAPS > 0 ? TAPS : a.taps;
  const int t = blockIdx.x, hh = blockIdx.y;
  const int P = a.vdim, N = a.N;
  const int inner = a.heads * P, gn = a.G * N, ch = inner + 2 * gn;
  const int g = hh / (a.heads / a.G);
  extern __shared__ __align__(16) float m2d_smem[];
  float* xs = m2d_smem;       // [P]  dt * silu(conv x)
  float* Bs = xs + ((P + 3) & ~3);  // [N]
  float* Cs = Bs + N;         // [N]
  float* red = Cs + N;        // [rows in flight][P]
  __shared__ float s_dt, s_decay;
  if (threadIdx.x == 0) {
    const float z = sum_slices(a.in_p + (size_t)t * a.in_ld + inner + ch + hh, a.in_S, a.in_stride) + a.dt_bias[hh];
    const float dt = z > 20.f ? z : log1pf(expf(z));
    s_dt = dt;
    s_decay = expf(-expf(a.a_log[hh]) * dt);
  }
  const int pos = a.positions[t], keep = taps - 1;
  const float* tail = a.state_pool + (size_t)a.state_slots[t] * a.slot_floats + a.tail_off;
  const float* cur = a.in_p + (size_t)t * a.in_ld + inner;
  __syncthreads();
  const float dt = s_dt, decay = s_decay;
  // the head's P + 2 N convolution channels
  for (int i = threadIdx.x; i < P + 2 * N; i += blockDim.x) {
    const int c = i < P ? hh * P + i : (i < P + N ? inner + g * N + (i - P) : inner + gn + g * N + (i - P - N));
    float y = a.conv_b ? a.conv_b[c] : 0.f;
#pragma unroll
    for (int j = 0; j < MT; j++) {
      if (j >= taps) continue;
      const int back = keep - j;  // the input `back` positions before this token
      float u = 0.f;
      if (back == 0) u = a.in_S == 1 ? cur[c] : sum_slices(cur + c, a.in_S, a.in_stride);
      else if (back <= pos) u = tail[(size_t)(keep - back) * ch + c];
      y = fmaf(a.conv_w[(size_t)c * taps + j], u, y);
    }
    const float v = a.fast_act ? __fdividef(y, 1.0f + __expf(-y)) : silu(y);
    if (i < P) {
      xs[i] = v * dt;
      a.xbc[(size_t)t * ch + c] = v;
    } else if (i < P + N) {
      Bs[i - P] = v;
    } else {
      Cs[i - P - N] = v;
    }
  }
  __syncthreads();
  // the recurrence
  const int cols = P / VW;                       // column units of VW
  const int rows_par = M2D_THREADS / cols;       // rows in flight (the launcher keeps cols <= 256)
  const int u = threadIdx.x % cols, rg = threadIdx.x / cols;
  float* state = const_cast<float*>(a.state_pool) + (size_t)a.state_slots[t] * a.slot_floats + a.state_off + (size_t)hh * N * P;
  const bool has_prev = pos > 0;
  float acc[VW], xv[VW];
#pragma unroll
  for (int e = 0; e < VW; e++) { acc[e] = 0.f; xv[e] = xs[u * VW + e]; }
  if (rg < rows_par) {
#pragma unroll 4
    for (int n = rg; n < N; n += rows_par) {
      float* sp = state + (size_t)n * P + u * VW;
      float sv[VW];
      if (VW == 4) {
        const float4 q4 = has_prev ? *reinterpret_cast<const float4*>(sp) : make_float4(0.f, 0.f, 0.f, 0.f);
        sv[0] = q4.x; sv[1 % VW] = q4.y; sv[2 % VW] = q4.z; sv[3 % VW] = q4.w;
      } else {
        sv[0] = has_prev ? sp[0] : 0.f;
      }
      const float bn = Bs[n], cn = Cs[n];
#pragma unroll
      for (int e = 0; e < VW; e++) {
        sv[e] = fmaf(decay, sv[e], bn * xv[e]);
        acc[e] = fmaf(sv[e], cn, acc[e]);
      }
      if (VW == 4) *reinterpret_cast<float4*>(sp) = make_float4(sv[0], sv[1 % VW], sv[2 % VW], sv[3 % VW]);
      else sp[0] = sv[0];
    }
#pragma unroll
    for (int e = 0; e < VW; e++) red[(size_t)rg * P + u * VW + e] = acc[e];
  }
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    float y = 0.f;
    for (int r = 0; r < rows_par; r++) y += red[(size_t)r * P + p];
    o[(size_t)t * inner + hh * P + p] = y;
  }
  TRACE_EXIT(tr);
}

bool mamba2_slot_decode_ok(const Mamba2SlotArgs& a) {
  static const bool on = !(getenv("NVLLM_MAMBA2_DECODE_FUSED") && atoi(getenv("NVLLM_MAMBA2_DECODE_FUSED")) == 0);
  const int cols = a.vdim % 4 == 0 ? a.vdim / 4 : a.vdim;
  return on && a.T == a.n_seqs && cols <= M2D_THREADS && a.taps >= 1 && a.taps <= 8 && a.heads % a.G == 0;
}

// o: [T, inner] read-outs (what the scan would have written); a.state_off: the layer's state inside a slot
cudaError_t launch_mamba2_slot_decode(cudaStream_t st, const Mamba2SlotArgs& a, float* o) {
  if (a.T <= 0) return cudaSuccess;
  if (!mamba2_slot_decode_ok(a)) return cudaErrorInvalidValue;
  const bool v4 = a.vdim % 4 == 0;
  const int cols = v4 ? a.vdim / 4 : a.vdim;
  const size_t smem = ((size_t)((a.vdim + 3) & ~3) + 2 * a.N + (size_t)(M2D_THREADS / cols) * a.vdim) * sizeof(float);
  const dim3 grid(a.T, a.heads);
#define M2D(TP_, VW_)                                                                                               \
  {                                                                                                                  \
    if (smem > 48 * 1024)                                                                                            \
      cudaFuncSetAttribute(mamba2_slot_decode_kernel<TP_, VW_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    (void)launch_k(mamba2_slot_decode_kernel<TP_, VW_>, grid, dim3(M2D_THREADS), smem, st, a, o, next_trace(21));     \
  }
  if (v4) {
    if (a.taps == 4) M2D(4, 4) else if (a.taps == 3) M2D(3, 4) else if (a.taps == 2) M2D(2, 4) else M2D(0, 4)
  } else {
    M2D(0, 1)
  }
#undef M2D
  return cudaGetLastError();
}

cudaError_t launch_mamba2_slot_prep(cudaStream_t st, const Mamba2SlotArgs& a) {
  if (a.T <= 0) return cudaSuccess;
  if (a.taps < 1 || a.taps > 8 || a.heads > 256) return cudaErrorInvalidValue;
  if (a.taps == 2) (void)launch_k(mamba2_slot_prep_kernel<2>, dim3(a.T), dim3(256), 0, st, a, next_trace(20));
  else if (a.taps == 3) (void)launch_k(mamba2_slot_prep_kernel<3>, dim3(a.T), dim3(256), 0, st, a, next_trace(20));
  else if (a.taps == 4) (void)launch_k(mamba2_slot_prep_kernel<4>, dim3(a.T), dim3(256), 0, st, a, next_trace(20));
  else (void)launch_k(mamba2_slot_prep_kernel<0>, dim3(a.T), dim3(256), 0, st, a, next_trace(20));
  return cudaGetLastError();
}

cudaError_t launch_mamba2_slot_out(cudaStream_t st, int odt, const Mamba2SlotArgs& a) {
  if (a.T <= 0) return cudaSuccess;
  const int inner = a.heads * a.vdim;
  if (a.norm_groups < 1 || a.norm_groups > 64 || inner % a.norm_groups) return cudaErrorInvalidValue;
  const size_t smem = (size_t)inner * sizeof(float);
  if (odt == DT_F32) {
    if (smem > 48 * 1024) cudaFuncSetAttribute(mamba2_slot_out_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    (void)launch_k(mamba2_slot_out_kernel<float>, dim3(a.T), dim3(256), smem, st, a, next_trace(22));
  } else {
    if (smem > 48 * 1024) cudaFuncSetAttribute(mamba2_slot_out_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    (void)launch_k(mamba2_slot_out_kernel<bf16>, dim3(a.T), dim3(256), smem, st, a, next_trace(22));
  }
  return cudaGetLastError();
}

// Windows of rows pay where sequences have several rows and there are some 100 CTAs of them.  Convolution, scan and norm
// of a step, with a row per CTA against windows, us: decode of 16 / 64 / 128 sequences, 6144 channels, 14.6 / 79 / 137.7
// against 18.6 / 86 / 139.9, 2304 channels and 64 / 256 sequences 18.6 / 41.8 against 26.9 / 47.5; one prompt of 16 / 64
// tokens 13.1 / 31.0 against 17.5 / 32.8; from there on windows are ahead (96 CTAs: 128 tokens 53.3 against 52.2, 2304
// channels and 256 tokens 62.6 against 57; 2048 tokens 709 against 508).
static bool mamba_conv_rows_fit(const MambaArgs& a) {
  return a.K == 4 && mamba_rows_aligned(a) && a.T >= 2 * a.n_seqs && ceil_div(a.T, MC_ROWS) * ceil_div(a.conv, 1024) >= 96;
}
cudaError_t launch_mamba_conv(cudaStream_t st, const MambaArgs& a) {
  if (a.T <= 0) return cudaSuccess;
  if (mamba_conv_rows_fit(a)) {
    const dim3 grid(ceil_div(a.T, MC_ROWS), ceil_div(a.conv, 1024));
    (void)launch_k(mamba_conv_rows_kernel<4>, grid, dim3(256), 0, st, a, next_trace(20));
  } else {
    (void)launch_k(mamba_conv_kernel, dim3(a.T, ceil_div(a.conv, 256)), dim3(256), 0, st, a, next_trace(20));
  }
  return cudaGetLastError();
}

// heads of a CTA of the tiled scan, 0 where it does not fit: whole warps, the heads of a CTA from one group
static int mamba_scan_hpc(const MambaArgs& a, int R, int L) {
  if (!mamba_rows_aligned(a) || a.hd % 4 != 0) return 0;
  if (a.N != 16 && a.N != 32 && a.N != 64 && a.N != 128) return 0;
  const int tph = L * a.hd / R, per_group = a.nh / a.G;
  int hpc = 1;
  while (hpc * 2 * tph <= 128 && per_group % (hpc * 2) == 0) hpc *= 2;
  return hpc * tph % 32 == 0 && hpc * tph <= 512 && hpc <= MS_MAX_HPC ? hpc : 0;
}
template <int R, int L, int NJ>
static cudaError_t mamba_scan_tiles(cudaStream_t st, const MambaArgs& a, int hpc) {
  const dim3 grid(a.n_seqs, a.nh / hpc), block(hpc * L * a.hd / R);
  const size_t smem = (size_t)2 * MS_TC * ((2 * a.N + hpc * a.hd + 2 * hpc + 3) & ~3) * sizeof(float);
  if (smem > 32 * 1024) {  // (beside the kernel's own 8 KB the default limit is 40 KB)
    const cudaError_t e = cudaFuncSetAttribute(mamba_scan_tile_kernel<R, L, NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  return launch_k(mamba_scan_tile_kernel<R, L, NJ>, grid, block, smem, st, a, hpc, next_trace(21));
}
// R rows per lane, or half as many: twice the warps per head and half the state per lane, the shorter chain per token
// while the grid leaves schedulers idle (148 SMs x 4, two warps each)
template <int R, int L, int NJ>
static bool mamba_scan_try(cudaStream_t st, const MambaArgs& a, cudaError_t* e) {
  const int half = mamba_scan_hpc(a, R / 2, L), whole = mamba_scan_hpc(a, R, L);
  if (whole && (!half || (long)a.n_seqs * a.nh * (L * a.hd / R) / 32 > 148 * 8)) *e = mamba_scan_tiles<R, L, NJ>(st, a, whole);
  else if (half) *e = mamba_scan_tiles<R / 2, L, NJ>(st, a, half);
  else return false;
  return true;
}
cudaError_t launch_mamba_scan(cudaStream_t st, const MambaArgs& a) {
  if (a.n_seqs <= 0) return cudaSuccess;
  const int threads = max(32, ((a.hd + 31) / 32) * 32);
  if (threads > 128 || a.N > 128) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  if (a.N == 16 ? mamba_scan_try<2, 4, 1>(st, a, &e) : a.N == 32 ? mamba_scan_try<4, 8, 1>(st, a, &e)
      : a.N == 64 ? mamba_scan_try<4, 8, 2>(st, a, &e) : a.N == 128 && mamba_scan_try<4, 8, 4>(st, a, &e))
    return e;
  const dim3 grid(a.n_seqs, a.nh);
  if (a.N <= 16) (void)launch_k(mamba_scan_kernel<16>, grid, dim3(threads), 0, st, a, next_trace(21));
  else if (a.N <= 32) (void)launch_k(mamba_scan_kernel<32>, grid, dim3(threads), 0, st, a, next_trace(21));
  else if (a.N <= 64) (void)launch_k(mamba_scan_kernel<64>, grid, dim3(threads), 0, st, a, next_trace(21));
  else (void)launch_k(mamba_scan_kernel<128>, grid, dim3(threads), 0, st, a, next_trace(21));
  return cudaGetLastError();
}

template <typename OT>
static cudaError_t mamba_gate_norm(cudaStream_t st, const MambaArgs& a, OT* out) {
  const size_t smem = (size_t)a.E * sizeof(float);
  if (mamba_rows_aligned(a))
    (void)launch_k(mamba_gate_norm_kernel<OT, 4>, dim3(a.T), dim3(256), smem, st, a, out, next_trace(22));
  else
    (void)launch_k(mamba_gate_norm_kernel<OT, 1>, dim3(a.T), dim3(256), smem, st, a, out, next_trace(22));
  return cudaGetLastError();
}
cudaError_t launch_mamba_gate_norm(cudaStream_t st, const MambaArgs& a, int odt, void* out) {
  if (a.T <= 0) return cudaSuccess;
  return odt == DT_F32 ? mamba_gate_norm(st, a, (float*)out) : mamba_gate_norm(st, a, (bf16*)out);
}

}  // namespace nvllm
