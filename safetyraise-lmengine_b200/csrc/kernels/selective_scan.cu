// The selective scan: a recurrent mixer with a state S [channels, N] per request, written and read token by token.
//
//   x <- silu(conv(x) + conv_bias)         a short causal convolution per channel over time (zeros before the start)
//   dt = softplus(dt_raw + dt_bias)        per channel; dt_raw is a projection of the token
//   S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c x_c B_n
//   y_c = sum_n S[c, n] C_n + D_c x_c;     out_c = y_c * silu(z_c)
//
// A (negative), D per channel and the biases are float32; B and C [N] come per token from a projection of x.  What a
// request carries from step to step lies in its slot, float32: S of every channel, then the last taps - 1 inputs of
// every channel's convolution.  Everything here is float32 arithmetic; only `out` (the input of the output product)
// and the optional second copy of x (the input of the B / C / dt product) are written in the activation dtype.
//
//   conv   one thread per (token, four neighbouring channels; one where rows do not allow 16-byte accesses): reads
//          the step's inputs, and the slot's carried inputs for the first taps - 1 tokens of an entry
//   scan   one block per (entry, 16 channels): two or four warps walk the entry's tokens in order, 4 lanes (8 from 17
//          states on) sharing a channel's N states, through chunks of 16 tokens in shared memory; the lanes' partial sums
//          of 8 tokens are added in one exchange of 6 shuffles (7).  Four more warps fetch the chunks several ahead
//          (cp.async), form the step sizes, and gate and write a finished chunk's y as a block; at the end the walkers
//          renew the slot's S and carried inputs.
//          A channel's sums do not depend on what else is in the step or on how the tokens were cut into steps.
#include <math_constants.h>

#include "common.cuh"

namespace srlm {

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// state of a slot: [channels * N] S, then [channels * (taps - 1)] carried inputs, oldest first
template <typename TL, int V>
__global__ void scan_conv_kernel(const float* __restrict__ xz, long long ld, const float* __restrict__ conv_w,
                                 const float* __restrict__ conv_b, const float* __restrict__ state, long long state_stride,
                                 const int* __restrict__ entry_of_token, const int* __restrict__ cu_q,
                                 const int* __restrict__ slots, float* __restrict__ x_out, TL* __restrict__ x_low,
                                 int T, int channels, int N, int taps) {
  pdl_wait();
  pdl_trigger();
  const int per_token = channels / V;                      // V neighbouring channels a thread (V divides channels)
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)T * per_token) return;
  const int t = (int)(idx / per_token), c = (int)(idx - (long long)t * per_token) * V;
  const int e = entry_of_token[t];
  const int i = t - cu_q[e];                               // the token's place in its entry
  const float* carry = state + (size_t)slots[e] * state_stride + (size_t)channels * N + (size_t)c * (taps - 1);
  float acc[V], v[V];
#pragma unroll
  for (int u = 0; u < V; ++u) acc[u] = conv_b ? conv_b[c + u] : 0.f;
  for (int j = 0; j < taps; ++j) {
    const int back = taps - 1 - j;                         // tap j weighs the input `back` tokens ago
    if (back <= i) {
      const float* src = xz + (size_t)(t - back) * ld + c;
      if constexpr (V == 4) {
        const float4 f = *reinterpret_cast<const float4*>(src);
        v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
      } else {
#pragma unroll
        for (int u = 0; u < V; ++u) v[u] = src[u];
      }
    } else {
#pragma unroll
      for (int u = 0; u < V; ++u) v[u] = carry[(size_t)u * (taps - 1) + taps - 1 + i - back];
    }
#pragma unroll
    for (int u = 0; u < V; ++u) acc[u] = fmaf(conv_w[(size_t)(c + u) * taps + j], v[u], acc[u]);
  }
#pragma unroll
  for (int u = 0; u < V; ++u) acc[u] = silu_f(acc[u]);
  const size_t at = (size_t)t * channels + c;
  if constexpr (V == 4) {
    *reinterpret_cast<float4*>(x_out + at) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  } else {
#pragma unroll
    for (int u = 0; u < V; ++u) x_out[at + u] = acc[u];
  }
  if (x_low) {
    if constexpr (V == 4 && sizeof(TL) == 2) {               // four 16-bit values in one 8-byte store
      TL low[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) low[u] = from_float<TL>(acc[u]);
      *reinterpret_cast<uint2*>(x_low + at) = *reinterpret_cast<const uint2*>(low);
    } else {
#pragma unroll
      for (int u = 0; u < V; ++u) x_low[at + u] = from_float<TL>(acc[u]);
    }
  }
}

// The same convolution for rows that allow 16-byte accesses and 2 to 4 taps: a thread owns four neighbouring channels
// over a run of tokens, holds their weights and the rows of the last TAPS - 1 tokens in registers, and reads every
// row once.  The sums are formed in the order of the kernel above (bias, then the taps from the oldest on).
template <typename TL, int TAPS>
__global__ void scan_conv_rows_kernel(const float* __restrict__ xz, long long ld, const float* __restrict__ conv_w,
                                      const float* __restrict__ conv_b, const float* __restrict__ state,
                                      long long state_stride, const int* __restrict__ entry_of_token,
                                      const int* __restrict__ cu_q, const int* __restrict__ slots,
                                      float* __restrict__ x_out, TL* __restrict__ x_low, int T, int channels, int N,
                                      int run) {
  pdl_wait();
  pdl_trigger();
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (c >= channels) return;
  const int t_begin = blockIdx.y * run, t_end = min(T, t_begin + run);
  float w[4][TAPS], bias[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    bias[u] = conv_b ? conv_b[c + u] : 0.f;
#pragma unroll
    for (int j = 0; j < TAPS; ++j) w[u][j] = conv_w[(size_t)(c + u) * TAPS + j];
  }
  float4 prev[TAPS - 1];                                   // prev[k]: the row of token t - (TAPS - 1) + k
#pragma unroll
  for (int k = 0; k < TAPS - 1; ++k) {
    const int row = t_begin - (TAPS - 1) + k;
    prev[k] = row >= 0 ? *reinterpret_cast<const float4*>(xz + (size_t)row * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll 4
  for (int t = t_begin; t < t_end; ++t) {
    const int e = entry_of_token[t];
    const int i = t - cu_q[e];                             // the token's place in its entry
    const float4 cur = *reinterpret_cast<const float4*>(xz + (size_t)t * ld + c);
    float acc[4] = {bias[0], bias[1], bias[2], bias[3]};
#pragma unroll
    for (int j = 0; j < TAPS; ++j) {
      const int back = TAPS - 1 - j;                       // tap j weighs the input `back` tokens ago
      float v[4];
      if (back <= i) {                                     // a row of this step (and of this entry)
        const float4 f = back == 0 ? cur : prev[j];
        v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
      } else {                                             // ahead of the portion: the slot's carried inputs
        const float* carry = state + (size_t)slots[e] * state_stride + (size_t)channels * N + (size_t)c * (TAPS - 1);
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = carry[(size_t)u * (TAPS - 1) + TAPS - 1 + i - back];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = fmaf(w[u][j], v[u], acc[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = silu_f(acc[u]);
    const size_t at = (size_t)t * channels + c;
    *reinterpret_cast<float4*>(x_out + at) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    if (x_low) {
      if constexpr (sizeof(TL) == 2) {
        TL low[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) low[u] = from_float<TL>(acc[u]);
        *reinterpret_cast<uint2*>(x_low + at) = *reinterpret_cast<const uint2*>(low);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) x_low[at + u] = from_float<TL>(acc[u]);
      }
    }
#pragma unroll
    for (int k = 0; k + 1 < TAPS - 1; ++k) prev[k] = prev[k + 1];
    prev[TAPS - 2] = cur;
  }
}

constexpr int kScanChannels = 16, kScanChunk = 16;
constexpr int scan_helpers(bool lengthy) { return lengthy ? 256 : 128; }

__device__ __forceinline__ void scan_cp_async_4(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void scan_cp_async_16(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void scan_cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void scan_cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kScanStates = 128;                           // most states of a channel

// 2^x for x <= 0 (a decay): the hardware's approximation, 2 ulp, zero below 2^-126
__device__ __forceinline__ float scan_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two neighbouring floats as one operand: an instruction of the FMA pipe for both, each rounded as alone.
typedef unsigned long long Pair;
__device__ __forceinline__ Pair pair_of(float lo, float hi) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
  return p;
}
__device__ __forceinline__ float2 halves_of(Pair p) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p));
  return f;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
  Pair p;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
  return p;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair p;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(a), "l"(b), "l"(c));
  return p;
}
__device__ __forceinline__ Pair scan_exp2(Pair p) {
  const float2 f = halves_of(p);
  return pair_of(scan_exp2(f.x), scan_exp2(f.y));
}

// n neighbouring pairs of shared memory (n a power of two; the address a multiple of min(n, 2) pairs)
template <int PAIRS>
__device__ __forceinline__ void scan_load_row(const float* src, Pair (&dst)[PAIRS]) {
  if constexpr (PAIRS == 1) {
    dst[0] = *reinterpret_cast<const Pair*>(src);
  } else {
#pragma unroll
    for (int k = 0; k < PAIRS; k += 2) {
      const ulonglong2 f = *reinterpret_cast<const ulonglong2*>(src + 2 * k);
      dst[k] = f.x, dst[k + 1] = f.y;
    }
  }
}

// A chunk of 16 tokens lies in shared memory while the block walks it: B and C of every token, zero behind N up to
// the lanes' reach; per (token, channel) the raw dt, x and z, each a plane of its own; per (token, channel) the pair of
// the step size and its product with x; and the block's y ahead of the gate.  Places behind an entry's last token hold
// dt = 0, dt x = 0, B = 0: S <- fma(1, S, 0) leaves every state as it is, so the walk has no branch.
//
// The block's last four warps fetch, prepare and finish; the others walk.  While the walkers are on chunk j the
// helpers turn the raw step sizes of chunk j + 1 into softplus(dt + bias) and its product with x, gate and write the y
// of chunk j - 1, issue the fetch of chunk j + K - 2 into the buffer chunk j - 2 has left, and wait until their own
// copies of chunk j + 2 have landed: K buffers of operands (a fetch has K - 4 walks of a chunk to arrive: a chunk's walk
// is about as long as a trip to DRAM), two of the pairs and of y, one barrier a chunk.  Every round commits one group of
// copies, an empty one behind the entry's end, so that "all but the last K - 4 groups" always names chunk j + 2.  A
// helper reads what other helpers fetched, and overwrites what other helpers read, only with a barrier in between.
//
// Bound by a chunk's dependent instructions, of the walkers (75 cycles a token in the form for two blocks an SM) and of the
// helpers alike, and with several blocks an SM by their number: 2,048 tokens, 4,096 channels of 16 states 107 us (2,048
// channels 88).  With 8 lanes a channel and a state an instruction 132 (105); pairs of states in 4 lanes 133, with both groups
// of a chunk and 96 registers in flight 111, with a copy a helper 107.  8 lanes of a pair each: 74 us at 2,048 channels, where
// an SM has one block, and 119 at 4,096.
constexpr int scan_buffers(int np) { return np <= 16 ? 8 : np <= 32 ? 7 : np <= 64 ? 6 : 5; }
constexpr int kScanPlane = kScanChunk * kScanChannels;
constexpr int kScanYRow = kScanChannels + 4;               // floats from a token's y to the next: a channel's lanes share no bank
// floats of shared memory: two of steps, two of y, `held` buffers (B | C up to the lanes' reach, three planes)
constexpr int scan_floats(int np, int held) {
  return 2 * 2 * kScanPlane + 2 * kScanChunk * kScanYRow + held * (kScanChunk * 2 * np + 3 * kScanPlane);
}
template <int HELPERS>
__device__ __forceinline__ void scan_helpers_meet() { asm volatile("bar.sync 1, %0;" ::"n"(HELPERS) : "memory"); }

// WIDE: channels, N, the rows and the pointers allow copies of 16 bytes.  LENGTHY (with WIDE): a long walk of few blocks
// LANES of a channel hold NPL states each, neighbours
template <typename TO, int LANES, int NPL, bool WIDE, bool LENGTHY>
__global__ void __launch_bounds__(LANES * kScanChannels + scan_helpers(LENGTHY), LENGTHY ? 2 : NPL <= 4 ? 5 : NPL <= 8 ? 4 : 3)
selective_scan_kernel(const float* __restrict__ x, const float* __restrict__ xz, long long ld_xz,
                      const float* __restrict__ dbc, long long ld_dbc, int b_off, const float* __restrict__ dt_raw,
                      const float* __restrict__ dt_bias, const float* __restrict__ A, const float* __restrict__ D,
                      float* __restrict__ state, long long state_stride, const int* __restrict__ cu_q,
                      const int* __restrict__ slots, TO* __restrict__ out, int channels, int N, int taps) {
  constexpr int NP = NPL * LANES;                           // states a channel's lanes reach, >= N
  constexpr int GROUP = LANES == 4 ? 8 : NPL <= 4 ? 4 : 2;  // tokens whose independent work the compiler interleaves
  constexpr int BC = kScanChunk * 2 * NP, YS = kScanPlane, WALKERS = LANES * kScanChannels, PAIRS = NPL / 2;
  constexpr int HELPERS = scan_helpers(LENGTHY), UNROLL = LENGTHY && NPL <= 4 ? kScanChunk / GROUP : 1;
  constexpr int K = scan_buffers(NP);
  pdl_wait();
  extern __shared__ __align__(16) float scan_smem[];
  float2* step_s = reinterpret_cast<float2*>(scan_smem);    // [2][chunk][channels of the block]: dt, dt x
  float* y_s = scan_smem + 2 * 2 * YS;                      // [2][chunk][kScanYRow]
  // K buffers, of which a launch has those that its longest entry fills (chunk j lies in buffer j % K): [3][chunk][channels of the
  // block], raw dt, x, z, then [chunk][2 NP], B and C
  constexpr int BUF = 3 * YS + BC;
  float* raw_s = y_s + 2 * kScanChunk * kScanYRow;
  float* bc_s = raw_s + 3 * YS;
  const int e = blockIdx.y, c0 = blockIdx.x * kScanChannels;
  const bool walker = threadIdx.x < WALKERS;
  const int tid = walker ? threadIdx.x : threadIdx.x - WALKERS;           // place among the walkers, or among the helpers
  const int lane = tid % LANES, ch = tid / LANES;
  const int c = c0 + ch;
  const bool live = c < channels;
  const int t0 = cu_q[e], q_len = cu_q[e + 1] - t0;
  float* slot = state + (size_t)slots[e] * state_stride;
  const int n_chunks = (q_len + kScanChunk - 1) / kScanChunk;

  // what a helper copies of every chunk where there are more helpers than copies of either kind: a piece of B or C, a piece of a
  // plane (raw dt, x, z: 64 pieces each)
  const int bc_i = tid / 8, raw_p = (tid - 64) / 64, raw_i = (tid - 64) % 64 / 4, raw_c = c0 + (tid - 64) % 4 * 4;
  const int bc_n = tid % 4 * 4;
  const float* bc_from = dbc + (size_t)(t0 + bc_i) * ld_dbc + b_off + (tid % 8 / 4) * N + bc_n;
  const bool raw_on = raw_c < channels;
  const long long raw_ld = raw_p == 2 ? ld_xz : channels;
  const float* raw_from = (raw_p == 0 ? dt_raw : raw_p == 1 ? x : xz + channels) + (size_t)(t0 + raw_i) * raw_ld + raw_c;
  // helpers: the fetch of chunk j, one group of copies (an empty one behind the last chunk)
  auto stage = [&](int j) {
    if (j >= n_chunks) {
      scan_cp_async_commit();
      return;
    }
    const int base = j * kScanChunk, n_here = min(kScanChunk, q_len - base);
    float* bc = bc_s + (j % K) * BUF;
    float* raw = raw_s + (j % K) * BUF;
    if constexpr (LENGTHY && NP == 16) {                    // 128 pieces of B and C, 192 of the planes
      if (tid < 128 && bc_i < n_here && bc_n < N) scan_cp_async_16(bc + 4 * tid, bc_from + (size_t)j * kScanChunk * ld_dbc);
      if (tid < 128 && (bc_i >= n_here || bc_n >= N)) *reinterpret_cast<float4*>(bc + 4 * tid) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (tid >= 64 && raw_on && raw_i < n_here) scan_cp_async_16(raw + 4 * (tid - 64), raw_from + (size_t)j * kScanChunk * raw_ld);
      scan_cp_async_commit();
      return;
    }
    constexpr int V = WIDE ? 4 : 1;                         // floats a copy
    for (int idx = tid; idx < BC / V; idx += HELPERS) {
      const int i = idx / (2 * NP / V), r = idx % (2 * NP / V) * V, half = r / NP, n = r % NP;
      float* dst = bc + idx * V;
      if (i < n_here && n < N) {
        const float* src = dbc + (size_t)(t0 + base + i) * ld_dbc + b_off + half * N + n;
        if constexpr (WIDE) scan_cp_async_16(dst, src);
        else scan_cp_async_4(dst, src);
      } else {
#pragma unroll
        for (int u = 0; u < V; ++u) dst[u] = 0.f;
      }
    }
    for (int idx = tid; idx < YS / V; idx += HELPERS) {
      const int i = idx / (kScanChannels / V), cc = idx % (kScanChannels / V) * V;
      if (i >= n_here || c0 + cc >= channels) continue;
      const size_t t = (size_t)(t0 + base + i);
      const float* from[3] = {dt_raw + t * channels + c0 + cc, x + t * channels + c0 + cc, xz + t * ld_xz + channels + c0 + cc};
#pragma unroll
      for (int p = 0; p < 3; ++p)
        if constexpr (WIDE) scan_cp_async_16(raw + p * YS + idx * V, from[p]);
        else scan_cp_async_4(raw + p * YS + idx * V, from[p]);
    }
    scan_cp_async_commit();
  };
  // a helper's channel is the same at all its (token, channel) places
  const int hc = c0 + tid % kScanChannels;
  const float bias = !walker && dt_bias && hc < channels ? dt_bias[hc] : 0.f, skip = !walker && hc < channels ? D[hc] : 0.f;
  // helpers: the step sizes of chunk j, all of whose copies have landed and were waited for ahead of a barrier
  auto prepare = [&](int j) {
    const int n_here = min(kScanChunk, q_len - j * kScanChunk);
    const float* raw = raw_s + (j % K) * BUF;
    float2* step = step_s + (j & 1) * YS;
#pragma unroll
    for (int u = 0; u < YS / HELPERS; ++u) {
      const int idx = tid + u * HELPERS;
      const bool on = idx / kScanChannels < n_here && hc < channels;
      const float dt = on ? softplus_f(raw[idx] + bias) : 0.f;
      step[idx] = make_float2(dt, on ? dt * raw[YS + idx] : 0.f);
    }
  };
  // helpers: y of chunk j, gated and written: out = (y + D x) * silu(z)
  auto finish = [&](int j) {
    const int base = j * kScanChunk, n_here = min(kScanChunk, q_len - base);
    const float* raw = raw_s + (j % K) * BUF;
    const float* ys = y_s + (j & 1) * kScanChunk * kScanYRow;
    if (hc >= channels) return;
#pragma unroll
    for (int u = 0; u < YS / HELPERS; ++u) {
      const int idx = tid + u * HELPERS;
      const int i = idx / kScanChannels;
      if (i < n_here)
        out[(size_t)(t0 + base + i) * channels + hc] = from_float<TO>((ys[i * kScanYRow + idx % kScanChannels] + skip * raw[YS + idx]) * silu_f(raw[2 * YS + idx]));
    }
  };

  Pair S[PAIRS], a[PAIRS];                                  // a lane's states are neighbours: n = lane * NPL + k
  // Many states of short walks: pairs of S and A by one access each, N being even with WIDE (a step of 64 requests of one token, by
  // single numbers | by pairs: 4,096 channels of 64 states 112 | 91 us, 1,024 of 128 84 | 58; with fewer states a lane, or a
  // walk that hides its ends, the registers of both forms cost up to 8 % more than this gives).
  const bool whole = WIDE && !LENGTHY && NPL >= 8 && (((uintptr_t)slot | (uintptr_t)A) & 7) == 0;
  if (walker && whole) {
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
      const int n = lane * NPL + 2 * k;
      const size_t at = (size_t)c * N + n;
      float2 s = make_float2(0.f, 0.f), f = s;
      if (live && n < N) s = *reinterpret_cast<const float2*>(slot + at), f = *reinterpret_cast<const float2*>(A + at);
      S[k] = pair_of(s.x, s.y);
      a[k] = pair_of(f.x * kLog2e, f.y * kLog2e);           // exp(dt A) = 2^(dt A log2 e)
    }
  } else if (walker) {
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
      const int n = lane * NPL + 2 * k;
      const bool on = live && n < N, two = live && n + 1 < N;
      const float *s_at = slot + (size_t)c * N + n, *a_at = A + (size_t)c * N + n;
      S[k] = pair_of(on ? s_at[0] : 0.f, two ? s_at[1] : 0.f);
      a[k] = pair_of(on ? a_at[0] * kLog2e : 0.f, two ? a_at[1] * kLog2e : 0.f);
    }
  } else if (n_chunks > 0) {
    for (int j = 0; j < K - 2; ++j) stage(j);
    scan_cp_async_wait<K - 4>();                            // the helper's own copies of chunks 0 and 1
    scan_helpers_meet<HELPERS>();
    prepare(0);
  }
  for (int j = 0; j < n_chunks; ++j) {
    __syncthreads();       // chunk j lies prepared, chunk j + 1 has landed; the y of chunk j - 1 lies in its buffer
    if (!walker) {
      stage(j + K - 2);                                     // into the buffer of chunk j - 2, which was finished in round j - 1
      if (j + 1 < n_chunks) prepare(j + 1);
      if (j > 0) finish(j - 1);
      scan_cp_async_wait<K - 4>();
      continue;
    }
    const int n_here = min(kScanChunk, q_len - j * kScanChunk);
    const float* bc = bc_s + (j % K) * BUF;
    const float2* step = step_s + (j & 1) * YS;
    float* ys = y_s + (j & 1) * kScanChunk * kScanYRow;
#pragma unroll UNROLL
    for (int i0 = 0; i0 < (UNROLL > 1 ? kScanChunk : n_here); i0 += GROUP) {
      float y[GROUP];
#pragma unroll
      for (int u = 0; u < GROUP; ++u) {
        const int i = i0 + u;
        const float2 v = step[i * kScanChannels + ch];
        const Pair dt = pair_of(v.x, v.x), dtx = pair_of(v.y, v.y);
        Pair Bv[PAIRS], Cv[PAIRS], sum;
        scan_load_row<PAIRS>(bc + i * 2 * NP + lane * NPL, Bv);
        scan_load_row<PAIRS>(bc + i * 2 * NP + NP + lane * NPL, Cv);
#pragma unroll
        for (int k = 0; k < PAIRS; ++k) {
          S[k] = fma2(scan_exp2(mul2(dt, a[k])), S[k], mul2(dtx, Bv[k]));
          sum = k ? fma2(S[k], Cv[k], sum) : mul2(S[k], Cv[k]);
        }
        const float2 f = halves_of(sum);
        y[u] = f.x + f.y;
      }
      // the lanes' partial sums of GROUP tokens, added across the lanes: each round a lane hands half of what it
      // holds to its partner and keeps the other half, so 8 tokens cost 4 + 2 exchanges among 4 lanes, and lane l ends with
      // two tokens' sums; a group of fewer tokens than lanes ends with plain rounds (both partners then hold the sum)
      int held = GROUP, tok = 0;
#pragma unroll
      for (int o = LANES / 2; o > 0; o >>= 1) {
        if (held > 1) {
          const int h = held / 2;
          const bool upper = (lane & o) != 0;
#pragma unroll
          for (int u = 0; u < GROUP / 2; ++u)
            if (u < h) {
              const float send = upper ? y[u] : y[u + h], keep = upper ? y[u + h] : y[u];
              y[u] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
          tok += upper ? h : 0;
          held = h;
        } else {
          y[0] += __shfl_xor_sync(0xffffffffu, y[0], o);
        }
      }
      if (GROUP >= LANES || (lane & (LANES / GROUP - 1)) == 0) {
#pragma unroll
        for (int u = 0; u < (GROUP > LANES ? GROUP / LANES : 1); ++u) ys[(i0 + tok + u) * kScanYRow + ch] = y[u];
      }
    }
  }
  pdl_trigger();             // a long walk: the kernel behind would only sit on the SMs meanwhile
  __syncthreads();
  if (!walker) {
    if (n_chunks > 0) finish(n_chunks - 1);
    return;
  }
#pragma unroll
  for (int k = 0; k < PAIRS; ++k) {
    const int n = lane * NPL + 2 * k;
    const float2 f = halves_of(S[k]);
    if (whole) {
      if (live && n < N) *reinterpret_cast<float2*>(slot + (size_t)c * N + n) = f;
      continue;
    }
    if (live && n < N) slot[(size_t)c * N + n] = f.x;
    if (live && n + 1 < N) slot[(size_t)c * N + n + 1] = f.y;
  }
  // the carried inputs: the last taps - 1 inputs of the channel, of this step or, for a short one, shifted up
  if (live && lane == 0 && taps > 1) {
    float* carry = slot + (size_t)channels * N + (size_t)c * (taps - 1);
    for (int j = 0; j < taps - 1; ++j) {
      const int i = q_len - (taps - 1) + j;                 // place in the entry of the input that lands in carry[j]
      carry[j] = i >= 0 ? xz[(size_t)(t0 + i) * ld_xz + c] : carry[j + q_len];     // reads ahead of what it has written
    }
  }
}

// out = (wa * a / sqrt(mean(a^2) + eps) + wb * b / sqrt(mean(b^2) + eps)) / 2: two sublayers that read the same input,
// each result normed with its own weight, averaged.  One block per token; sums in float32 in an order fixed by the width
// and the block's size.  V elements a thread and access (V = 4 where rows and pointers allow 16 bytes of float32); a
// thread keeps its first PER accesses of a and b in registers for the second pass and reads the rest again.
template <typename TI, typename TO, int V, int PER>
__global__ void paired_rmsnorm_mean_kernel(const TI* __restrict__ a, const float* __restrict__ wa, const TI* __restrict__ b,
                                           const float* __restrict__ wb, float eps, TO* __restrict__ out, int H) {
  pdl_wait();
  pdl_trigger();
  __shared__ float scratch[32];
  const size_t base = (size_t)blockIdx.x * H;
  const int step = blockDim.x * V;
  float ua[PER][V], ub[PER][V];
  float sa = 0.f, sb = 0.f;
  auto fetch = [&](int i, float (&u)[V], float (&v)[V]) {
    if constexpr (V == 4 && sizeof(TI) == 4) {
      const float4 f = *reinterpret_cast<const float4*>(a + base + i), g = *reinterpret_cast<const float4*>(b + base + i);
      u[0] = f.x, u[1] = f.y, u[2] = f.z, u[3] = f.w;
      v[0] = g.x, v[1] = g.y, v[2] = g.z, v[3] = g.w;
    } else {
#pragma unroll
      for (int k = 0; k < V; ++k) u[k] = to_float(a[base + i + k]), v[k] = to_float(b[base + i + k]);
    }
  };
  int r = 0;
  for (int i = threadIdx.x * V; i < H; i += step, ++r) {
    float u[V], v[V];
    fetch(i, u, v);
#pragma unroll
    for (int k = 0; k < V; ++k) sa = fmaf(u[k], u[k], sa), sb = fmaf(v[k], v[k], sb);
#pragma unroll
    for (int p = 0; p < PER; ++p)
      if (p == r) {
#pragma unroll
        for (int k = 0; k < V; ++k) ua[p][k] = u[k], ub[p][k] = v[k];
      }
  }
  const float ia = 1.0f / sqrtf(block_sum(sa, scratch) / (float)H + eps);
  const float ib = 1.0f / sqrtf(block_sum(sb, scratch) / (float)H + eps);
  r = 0;
  for (int i = threadIdx.x * V; i < H; i += step, ++r) {
    float u[V], v[V];
    bool kept = false;
#pragma unroll
    for (int p = 0; p < PER; ++p)
      if (p == r) {
        kept = true;
#pragma unroll
        for (int k = 0; k < V; ++k) u[k] = ua[p][k], v[k] = ub[p][k];
      }
    if (!kept) fetch(i, u, v);
#pragma unroll
    for (int k = 0; k < V; ++k)
      out[base + i + k] = from_float<TO>(0.5f * (u[k] * ia * wa[i + k] + v[k] * ib * wb[i + k]));
  }
}

}  // namespace srlm

using namespace srlm;

// xz float32 [T, ld >= channels]: the inputs of the convolution in its first `channels` columns.  conv_w float32
// [channels, taps] (last column: the current token's), conv_b float32 [channels] or null.  state float32
// [slots, state_stride]: per slot channels * N of S, then channels * (taps - 1) carried inputs (read here, renewed by
// srlm_selective_scan).  x_out float32 [T, channels]; x_low [T, channels] in low_dtype, or null.
extern "C" int srlm_scan_conv(const float* xz, long long ld, const float* conv_w, const float* conv_b, const float* state,
                              long long state_stride, const int* entry_of_token, const int* cu_q, const int* slots,
                              float* x_out, void* x_low, int low_dtype, int T, int channels, int N, int taps,
                              cudaStream_t stream) {
  if (T <= 0) return ST_OK;
  if (channels <= 0 || N <= 0 || taps <= 0 || ld < channels || state_stride < (long long)channels * (N + taps - 1))
    return refuse(ST_BAD_SIZE, "scan_conv: channels=%d N=%d taps=%d ld=%lld state_stride=%lld", channels, N, taps, ld,
                  state_stride);
  // four neighbouring channels a thread where rows and pointers allow 16-byte accesses (the sums are the same)
  const bool wide = channels % 4 == 0 && ld % 4 == 0 && ((uintptr_t)xz | (uintptr_t)x_out | (uintptr_t)x_low) % 16 == 0;
  const long long total = (long long)T * (wide ? channels / 4 : channels);
  const dim3 grid((unsigned)((total + 255) / 256));
  if (wide && taps >= 2 && taps <= 4) {                      // rows read once, weights in registers
    const int run = T >= 512 ? 16 : 4;
    const dim3 rows_grid((channels / 4 + 127) / 128, (T + run - 1) / run);
#define SRLM_CONV_ROWS(TL, TAPS, LOW)                                                                                   \
  launch_pdl(scan_conv_rows_kernel<TL, TAPS>, rows_grid, dim3(128), 0, stream, xz, ld, conv_w, conv_b, state,          \
             state_stride, entry_of_token, cu_q, slots, x_out, LOW, T, channels, N, run)
#define SRLM_CONV_TAPS(TL, LOW)                                  \
  switch (taps) {                                                \
    case 2: SRLM_CONV_ROWS(TL, 2, LOW); break;                   \
    case 3: SRLM_CONV_ROWS(TL, 3, LOW); break;                   \
    default: SRLM_CONV_ROWS(TL, 4, LOW); break;                  \
  }
    if (!x_low) { SRLM_CONV_TAPS(float, (float*)nullptr) }
    else if (low_dtype == DT_BF16) { SRLM_CONV_TAPS(bf16, (bf16*)x_low) }
    else return refuse(ST_BAD_DTYPE, "scan_conv: the second copy of x is bfloat16 (dtype %d)", low_dtype);
#undef SRLM_CONV_TAPS
#undef SRLM_CONV_ROWS
    return launched();
  }
#define SRLM_CONV(TL, V, LOW)                                                                                          \
  launch_pdl(scan_conv_kernel<TL, V>, grid, dim3(256), 0, stream, xz, ld, conv_w, conv_b, state, state_stride,        \
             entry_of_token, cu_q, slots, x_out, LOW, T, channels, N, taps)
  if (!x_low) {
    if (wide) SRLM_CONV(float, 4, (float*)nullptr);
    else SRLM_CONV(float, 1, (float*)nullptr);
  } else if (low_dtype == DT_BF16) {
    if (wide) SRLM_CONV(bf16, 4, (bf16*)x_low);
    else SRLM_CONV(bf16, 1, (bf16*)x_low);
  } else {
    return refuse(ST_BAD_DTYPE, "scan_conv: the second copy of x is bfloat16 (dtype %d)", low_dtype);
  }
#undef SRLM_CONV
  return launched();
}

// x float32 [T, channels] (behind the convolution); xz float32 [T, ld_xz >= 2 channels]: the convolution's inputs, then z;
// dbc float32 [T, ld_dbc]: B in columns [b_off, b_off + N), C in the N columns behind them; dt_raw float32
// [T, channels]; dt_bias, D float32 [channels]; A float32 [channels, N]; out [T, channels] in out_dtype.  max_q_len: the
// most tokens an entry brings (an upper bound will do).
extern "C" int srlm_selective_scan(const float* x, const float* xz, long long ld_xz, const float* dbc, long long ld_dbc,
                                   int b_off, const float* dt_raw, const float* dt_bias, const float* A, const float* D,
                                   float* state, long long state_stride, const int* cu_q, const int* slots, void* out,
                                   int out_dtype, int n_entries, int max_q_len, int channels, int N, int taps,
                                   cudaStream_t stream) {
  if (n_entries <= 0) return ST_OK;
  if (channels <= 0 || N <= 0 || N > kScanStates || taps <= 0 || ld_xz < 2ll * channels || b_off < 0 ||
      ld_dbc < b_off + 2ll * N || state_stride < (long long)channels * (N + taps - 1) || n_entries > 65535)
    return refuse(ST_BAD_SIZE, "selective_scan: channels=%d N=%d (at most %d) taps=%d ld_xz=%lld ld_dbc=%lld b_off=%d "
                  "state_stride=%lld", channels, N, kScanStates, taps, ld_xz, ld_dbc, b_off, state_stride);
  const dim3 grid((channels + kScanChannels - 1) / kScanChannels, n_entries);
  // four lanes a channel up to 16 states, eight beyond (64 states: 8 a lane, half the registers)
  const int lanes = N <= 16 ? 4 : 8;
  int npl = 2;
  while (npl * lanes < N) npl <<= 1;
  const bool early = max_q_len <= 4 * kScanChunk;      // a long walk starts on an empty GPU, its blocks spread evenly
  // at most two blocks an SM: more registers and helpers for each (2,048 tokens, 4,096 channels 107 us, 133 without;
  // 8,192 channels 218, 204 without)
  const bool roomy = !early && (long long)grid.x * grid.y <= 2 * 148;
  // copies of 16 bytes: neither four channels nor four states straddle an edge
  const bool wide = channels % 4 == 0 && N % 4 == 0 && b_off % 4 == 0 && ld_dbc % 4 == 0 && ld_xz % 4 == 0 &&
                    ((uintptr_t)x | (uintptr_t)xz | (uintptr_t)dbc | (uintptr_t)dt_raw) % 16 == 0;
  // a step of short portions (decode) needs no ring: with one, fewer of its many blocks share an SM (64 requests of
  // one token, 8,192 channels of 16 states: the layer 237 us, without it and with the registers
  // of five blocks an SM 206)
  const int chunks = (max_q_len + kScanChunk - 1) / kScanChunk;
  const int held = chunks < 1 ? 1 : chunks < scan_buffers(npl * lanes) ? chunks : scan_buffers(npl * lanes);
  const size_t smem = (size_t)scan_floats(npl * lanes, held) * sizeof(float);
#define SRLM_SCAN_AS(TO, LANES, NPL, W, LONG)                                                                           \
  do {                                                                                                                  \
    auto kern = selective_scan_kernel<TO, LANES, NPL, W, LONG>;                                                         \
    const cudaError_t got =                                                                                             \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                             \
    if (got != cudaSuccess) return refuse((int)got, "selective_scan: cannot get %zu bytes of shared memory", smem);     \
    launch_pdl_if(early, kern, grid, dim3(LANES * kScanChannels + scan_helpers(LONG)), smem, stream, x, xz, ld_xz, dbc, \
                  ld_dbc, b_off, dt_raw, dt_bias, A, D, state, state_stride, cu_q, slots, (TO*)out, channels, N, taps); \
  } while (0)
#define SRLM_SCAN(TO, LANES, NPL)                                   \
  do {                                                              \
    if (wide && roomy) SRLM_SCAN_AS(TO, LANES, NPL, true, true);   \
    else if (wide) SRLM_SCAN_AS(TO, LANES, NPL, true, false);       \
    else SRLM_SCAN_AS(TO, LANES, NPL, false, false);                \
  } while (0)
#define SRLM_SCAN_N(TO)                                   \
  switch (lanes * 100 + npl) {                            \
    case 402: SRLM_SCAN(TO, 4, 2); break;                 \
    case 404: SRLM_SCAN(TO, 4, 4); break;                 \
    case 804: SRLM_SCAN(TO, 8, 4); break;                 \
    case 808: SRLM_SCAN(TO, 8, 8); break;                 \
    default: SRLM_SCAN(TO, 8, 16);                        \
  }
  if (out_dtype == DT_F32) { SRLM_SCAN_N(float) }
  else if (out_dtype == DT_BF16) { SRLM_SCAN_N(bf16) }
  else return refuse(ST_BAD_DTYPE, "selective_scan: output dtype %d", out_dtype);
#undef SRLM_SCAN_N
#undef SRLM_SCAN
#undef SRLM_SCAN_AS
  return launched();
}

// a, b [T, H] in in_dtype; wa, wb float32 [H]; out [T, H] in out_dtype
extern "C" int srlm_paired_rmsnorm_mean(const void* a, const float* wa, const void* b, const float* wb, float eps, void* out,
                                        int in_dtype, int out_dtype, int T, int H, cudaStream_t stream) {
  if (T <= 0) return ST_OK;
  if (H <= 0 || !(eps > 0.f) || !wa || !wb) return refuse(ST_BAD_SIZE, "paired_rmsnorm_mean: H=%d eps=%g", H, (double)eps);
  const bool wide = H % 4 == 0 && ((uintptr_t)a | (uintptr_t)b) % 16 == 0;
  const int v = wide ? 4 : 1;
  int block = 64;
  while (block < 1024 && block * 2 * v < H) block <<= 1;      // two accesses a thread, kept in registers between the passes
#define SRLM_PAIRED(TI, TO)                                                                                              \
  do {                                                                                                                   \
    if (wide) launch_pdl(paired_rmsnorm_mean_kernel<TI, TO, 4, 2>, dim3(T), dim3(block), 0, stream, (const TI*)a, wa,    \
                         (const TI*)b, wb, eps, (TO*)out, H);                                                            \
    else launch_pdl(paired_rmsnorm_mean_kernel<TI, TO, 1, 2>, dim3(T), dim3(block), 0, stream, (const TI*)a, wa,         \
                    (const TI*)b, wb, eps, (TO*)out, H);                                                                 \
  } while (0)
  if (in_dtype == DT_F32 && out_dtype == DT_F32) SRLM_PAIRED(float, float);
  else if (in_dtype == DT_F32 && out_dtype == DT_BF16) SRLM_PAIRED(float, bf16);
  else if (in_dtype == DT_BF16 && out_dtype == DT_BF16) SRLM_PAIRED(bf16, bf16);
  else return refuse(ST_BAD_DTYPE, "paired_rmsnorm_mean: input dtype %d with output dtype %d", in_dtype, out_dtype);
#undef SRLM_PAIRED
  return launched();
}
