// The gated delta rule (delta_rule.cu) for long portions: chunks of 16 tokens.
//
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q            (in this order, per token)
//
// What 16 tokens do to S and v, all columns of S share.  With P_i = g_1 .. g_i, D_ij = g_(j+1) .. g_i and R_j = D_16,j (products
// within the chunk, so nothing grows), N_ij = (k_i . k_j) D_ij (j < i), M_ij = (q_i . k_j) D_ij (j <= i):
//   X = (I + diag(beta) N)^-1 diag(beta):   u = X (v - [P_i k_i . S]),   o_i = P_i q_i . S + (M u)_i
// and, with the products by X and M taken ahead of S,
//   kx = X [P_i k_i],  qm = [P_i q_i] - M kx,  ke_j = R_j k_j,  u0 = X v,  o0 = M u0,  whole = P_16:
//   u = u0 - kx . S,   o = o0 + qm . S,   S <- whole S + sum_j ke_j u_j
//
//   delta_chunks       a block per (chunk, head): convolution, silu, unit vectors, beta, decays, and the record of the chunk;
//                      bound by instructions (silu, the products by X and M) at 20 warps an SM.
//   delta_chunk_walk   a block per (entry, head, 16 columns of S) walks the records: three products a chunk on tensor cores,
//                      S in the accumulators; bound by the latency of a chunk (two exchanges between the eight warps).  Blocks
//                      start in the order of their entries' lengths, the longest first: entries of 486, 458 and 1,056 tokens
//                      163 us in the step's order, where the longest waited for places, 126 so.
// 2,000 tokens, 16 heads of 128 x 128, one entry: 77 + 153 us; the kernels that go token by token: 98 + 610 us.
//
// The products of the walk are mma.sync m16n8k8 on tf32 operands, each operand split into two tf32 numbers (high, and the rest)
// and each product formed as high high + high low + low high.  Relative error against float64 (2-norm; 16 to 2,000 tokens, decays
// from fast to nearly one), outputs and state: 1.3e-7 to 2.1e-7 and 5e-8 to 2.1e-7; the kernels that go token by token in float32
// FMAs: 1.3e-7 to 3.7e-6 and 1.4e-7 to 5.2e-6, never below.  It takes the sums of their own in mma_split (one running sum in the
// tensor core: up to 2.9 times the token walk's error) and the scalars of a token in 64 bits (up to 1.7 times without).
#include "state_walk.cuh"

namespace srlm {
namespace chunks {

constexpr int TOK = 16, DK = 128, TAPS = 4;
constexpr int LD = DK + 8;                     // floats from a staged token to the next: 8 modulo 32 banks

__host__ __device__ inline int record_floats(int dv) { return 3 * TOK * DK + 2 * TOK * dv + 4; }

struct Home {
  int entry, t0, n, first;                     // first: the entry's first token in the step
};
// Chunks of an entry of `len` tokens: none where it goes token by token (fewer than `least` tokens).
__device__ __forceinline__ int chunks_of(int len, int least) { return len < least ? 0 : (len + TOK - 1) / TOK; }
__device__ __forceinline__ Home home_of(const int* __restrict__ cu_q, int n_entries, int least, int index) {
  int base = 0;
  for (int e = 0; e < n_entries; ++e) {
    const int a = cu_q[e], len = cu_q[e + 1] - a, mine = chunks_of(len, least);
    if (index < base + mine) {
      const int at = (index - base) * TOK;
      return Home{e, a + at, min(TOK, len - at), a};
    }
    base += mine;
  }
  return Home{-1, 0, 0, 0};
}

struct Sizes {
  int H, G, dv, C;                             // value heads, q / k heads, value size, convolved channels
};

__global__ void __launch_bounds__(128, 5)
delta_chunks_kernel(const float* __restrict__ proj, long long ldp, const float* __restrict__ conv_w, int taps,
                    const float* __restrict__ a_log, const float* __restrict__ dt_bias, const float* __restrict__ state,
                    long long state_stride, const int* __restrict__ cu_q, int n_entries, const int* __restrict__ slots,
                    float* __restrict__ records, int least, int first_chunk, Sizes z, float unit_eps) {
  pdl_wait();
  pdl_trigger();
  __shared__ __align__(16) float k_s[TOK][DK + 4], q_s[TOK][DK + 4];
  __shared__ __align__(16) float x_s[TOK][TOK], m_s[TOK][TOK], n_s[TOK][TOK];
  // what multiplies a whole token or a pair of tokens is formed in 64 bits and rounded once
  __shared__ double d_s[TOK][TOK], unit_k[TOK], unit_q[TOK], g_s[TOK], pre_s[TOK];
  __shared__ float beta_s[TOK], fade_k[TOK], fade_q[TOK], last_k[TOK];   // P_i / |k_i|, P_i / (|q_i| sqrt(DK)), R_i / |k_i|
  const Home home = home_of(cu_q, n_entries, least, first_chunk + blockIdx.x);
  if (home.entry < 0) return;
  const int h = blockIdx.y, kh = h / (z.H / z.G), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* carry = state + (size_t)slots[home.entry] * state_stride + (size_t)z.H * DK * z.dv;   // [C][taps - 1]
  const bool inner = home.n == TOK && home.t0 - home.first >= TAPS - 1;
  // the convolved and activated channel c of the chunk's tokens (0 where there is none)
  auto convolve = [&](int c, float (&y)[TOK]) {
    float in[TOK + TAPS - 1], w[TAPS];
    if (inner) {                               // a whole chunk, its past among the step's tokens
      const float* at = proj + (size_t)(home.t0 - (TAPS - 1)) * ldp + c;
#pragma unroll
      for (int i = 0; i < TOK + TAPS - 1; ++i, at += ldp) in[i] = *at;
    } else {
#pragma unroll
    for (int i = 0; i < TOK + TAPS - 1; ++i) {
      const int t = home.t0 + i - (TAPS - 1), local = t - home.first;
      in[i] = 0.f;
      if (i - (TAPS - 1) < home.n) {
        if (local >= 0) in[i] = proj[(size_t)t * ldp + c];
        else if (local + taps - 1 >= 0) in[i] = carry[(size_t)c * (taps - 1) + taps - 1 + local];
      }
    }
    }
#pragma unroll
    for (int j = 0; j < TAPS; ++j) w[j] = j >= TAPS - taps ? conv_w[(size_t)c * taps + j - (TAPS - taps)] : 0.f;
#pragma unroll
    for (int i = 0; i < TOK; ++i) {
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < TAPS; ++j) s = fmaf(w[j], j >= TAPS - taps ? in[i + j] : 0.f, s);
      y[i] = i < home.n ? s / (1.f + expf(-s)) : 0.f;
    }
  };
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {
    float y[TOK];
    convolve((part * z.G + kh) * DK + tid, y);
#pragma unroll
    for (int i = 0; i < TOK; ++i) (part ? k_s : q_s)[i][tid] = y[i];
  }
  // The scalars in 64 bits take long chains of instructions: side by side, in lanes and warps of their own.
  if (warp == 1 && lane < TOK) {
    float b = 0.f;
    if (lane < home.n) b = (float)(1. / (1. + exp(-(double)proj[(size_t)(home.t0 + lane) * ldp + z.C + h])));
    beta_s[lane] = b;
  }
  if (warp == 0) {                             // lane i: g_i; then column i of D, and P
    const bool on = lane < min(home.n, TOK);
    const double a = on ? (double)proj[(size_t)(home.t0 + lane) * ldp + z.C + z.H + h] + dt_bias[h] : 0.;
    const bool far = a > 20.;
    const double e = exp(lane < TOK ? (far ? -a : a) : (double)a_log[h]);        // the upper lanes: exp(a_log)
    const double rate = __shfl_sync(0xffffffffu, e, TOK), l = log1p(e);
    const double g = on ? exp(-rate * (far ? a + l : l)) : 1.;
    if (lane < TOK) g_s[lane] = g;
    __syncwarp();
    if (lane < TOK) {
      double p = 1., d = 1.;
      for (int i = 0; i <= lane; ++i) p *= g_s[i];
      pre_s[lane] = p;
      for (int i = 0; i < TOK; ++i) {
        if (i > lane) d *= g_s[i];
        d_s[i][lane] = i >= lane ? d : 0.;
      }
    }
  }
  __syncthreads();
  {
    float mine = 0.f;                          // lane j: of the warp's j-th token of k, then of q
#pragma unroll
    for (int j = 0; j < 2 * TOK / 4; ++j) {
      const int v = warp + 4 * j, i = v % TOK;
      const float4 x = *reinterpret_cast<const float4*>((v < TOK ? k_s[i] : q_s[i]) + 4 * lane);
      const float ss = warp_sum((x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w));
      if (lane == j) mine = ss;
    }
    if (lane < 2 * TOK / 4) {
      const int v = warp + 4 * lane, i = v % TOK;
      const double one = v < TOK ? 1. : 1. / sqrt((double)DK);
      (v < TOK ? unit_k : unit_q)[i] = i < home.n ? one / sqrt((double)mine + unit_eps) : 0.;      // a place without a token
    }
  }
  // k_i . k_j (threads 0 .. 63) and q_i . k_j (64 .. 127): rows i, i + 8, columns j, j + 8
  {
    const int i = (tid & 63) >> 3, j = tid & 7;
    const float* a0 = tid < 64 ? k_s[i] : q_s[i];
    const float* a1 = tid < 64 ? k_s[i + 8] : q_s[i + 8];
    float part[2][2][4] = {};
#pragma unroll 4
    for (int c = 0; c < DK; c += 4) {
      const float4 a[2] = {*reinterpret_cast<const float4*>(a0 + c), *reinterpret_cast<const float4*>(a1 + c)};
      const float4 b[2] = {*reinterpret_cast<const float4*>(k_s[j] + c), *reinterpret_cast<const float4*>(k_s[j + 8] + c)};
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          part[x][y][0] = fmaf(a[x].x, b[y].x, part[x][y][0]);
          part[x][y][1] = fmaf(a[x].y, b[y].y, part[x][y][1]);
          part[x][y][2] = fmaf(a[x].z, b[y].z, part[x][y][2]);
          part[x][y][3] = fmaf(a[x].w, b[y].w, part[x][y][3]);
        }
    }
    __syncthreads();                           // the unit factors and D are here
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int r = i + 8 * x, c = j + 8 * y;
        const float sum = (part[x][y][0] + part[x][y][1]) + (part[x][y][2] + part[x][y][3]);
        const double s = sum * unit_k[c] * d_s[r][c];            // D is 0 above the diagonal
        if (tid < 64) n_s[r][c] = r > c ? (float)(s * unit_k[r]) : 0.f;
        else m_s[r][c] = (float)(s * unit_q[r]);
      }
  }
  if (tid < TOK) {
    fade_k[tid] = (float)(pre_s[tid] * unit_k[tid]);
    fade_q[tid] = (float)(pre_s[tid] * unit_q[tid]);
    last_k[tid] = (float)(d_s[TOK - 1][tid] * unit_k[tid]);
  }
  __syncthreads();
  if (tid < TOK) {                             // column tid of X, forward along the rows
    float x[TOK];
#pragma unroll
    for (int i = 0; i < TOK; ++i) {
      float s = i == tid ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) s = fmaf(-n_s[i][j], x[j], s);
      x[i] = beta_s[i] * s;
      x_s[i][tid] = x[i];
    }
  }
  __syncthreads();
  float* rec = records + ((size_t)blockIdx.x * z.H + h) * record_floats(z.dv);
  // x_i <- sum_(j <= i) A_ij x_j, from the last row up
  auto lower = [&](const float (*A)[TOK], float (&x)[TOK]) {
#pragma unroll
    for (int i = TOK - 1; i >= 0; --i) {
      float s = 0.f;
#pragma unroll
      for (int j = 0; j <= i; j += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&A[i][j]);
        s = fmaf(a.x, x[j], s);
        if (j + 1 <= i) s = fmaf(a.y, x[j + 1], s);
        if (j + 2 <= i) s = fmaf(a.z, x[j + 2], s);
        if (j + 3 <= i) s = fmaf(a.w, x[j + 3], s);
      }
      x[i] = s;
    }
  };
  // the key channel tid first, then the value columns tid, tid + 128, ..
#pragma unroll 1
  for (int c = tid - DK; c < z.dv; c += DK) {
    float x[TOK];
    if (c < 0) {
#pragma unroll
      for (int i = 0; i < TOK; ++i) {
        rec[(2 * TOK + i) * DK + tid] = last_k[i] * k_s[i][tid];
        x[i] = fade_k[i] * k_s[i][tid];
      }
    } else {
      convolve(2 * z.G * DK + h * z.dv + c, x);
    }
    float* out = rec + (c < 0 ? tid : 3 * TOK * DK + c);
    const int ld = c < 0 ? DK : z.dv;
    lower(x_s, x);
#pragma unroll
    for (int i = 0; i < TOK; ++i) out[i * ld] = x[i];
    lower(m_s, x);
#pragma unroll
    for (int i = 0; i < TOK; ++i) out[(TOK + i) * ld] = c < 0 ? fmaf(fade_q[i], q_s[i][tid], -x[i]) : x[i];
  }
  if (tid == 0) rec[3 * TOK * DK + 2 * TOK * z.dv] = (float)pre_s[TOK - 1];
}

// ---- the walk -----------------------------------------------------------------------------------------------------------
constexpr int COLS = 16, WARPS = 8, ROWS = DK / WARPS, STAGES = 3, THREADS = 32 * WARPS;
constexpr int STAGE = 3 * TOK * LD + 2 * TOK * COLS + 4;       // kx | qm | ke | u0, o0 of the block's columns | whole
constexpr int U_LD = 24;                                       // floats from a token of u to the next: 24 modulo 32 banks
constexpr int SUM_LD = 20, SUMS = TOK * SUM_LD;                // a warp's sums [token][column]: lanes two tokens apart share no bank
constexpr int WALK_SMEM = (STAGES * STAGE + 2 * WARPS * SUMS + TOK * U_LD) * (int)sizeof(float);

struct Split {                                 // x = hi + lo up to 2^-23 of x
  uint32_t hi, lo;
};
// hi: x rounded to the 11 bits of a tf32 number (integer arithmetic: the conversion instruction runs at a quarter of its
// rate); the rest fits 12 bits, of which the product reads 11.  A NaN stays one in lo.
__device__ __forceinline__ Split split(float x) {
  Split s;
  s.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  s.lo = __float_as_uint(x - __uint_as_float(s.hi));
  return s;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// A sum of a tensor-core product is cut off, not rounded, behind its 24th bit, each time that it is written.  So the products
// of the high parts (`large`, one product a sum) and those with a rest (`small`, 2^-11 of it) have sums of their own, which
// float32 additions join.
__device__ __forceinline__ void mma_split(float (&small)[4], float (&large)[4], const Split (&a)[4], const Split (&b)[2]) {
  mma_tf32(small, a[0].lo, a[1].lo, a[2].lo, a[3].lo, b[0].hi, b[1].hi);
  mma_tf32(small, a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[0].lo, b[1].lo);
  mma_tf32(large, a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[0].hi, b[1].hi);
}

// A warp holds 16 columns x 16 rows of S as two accumulator tiles [column][8 rows]: lane (g, t) = (lane / 4, lane % 4) has
// columns g, g + 8 and rows 2 t, 2 t + 1 of each.  As the left operand of the next product the same registers serve, with
// the product's k-th place t standing for row 2 t and t + 4 for row 2 t + 1 (on both sides).
__global__ void __launch_bounds__(THREADS, 2)
delta_chunk_walk_kernel(const float* __restrict__ records, float* __restrict__ state, long long state_stride,
                        const int* __restrict__ cu_q, int n_entries, const int* __restrict__ slots,
                        float* __restrict__ o_out, int least, int first_chunk, int n_chunks, Sizes z) {
  pdl_wait();
  pdl_trigger();
  // the records are those of the step's chunks first_chunk .. first_chunk + n_chunks - 1, of the entry's those from..to - 1
  extern __shared__ __align__(16) float chunk_smem[];
  float* p_sums = chunk_smem + STAGES * STAGE;           // [warp][SUMS]: kx . S
  float* q_sums = p_sums + WARPS * SUMS;                 // qm . S
  float* u_s = q_sums + WARPS * SUMS;                    // [token][U_LD]
  // the blockIdx.z-th longest of the entries, and the place of its first record: the blocks of the longest entry start first
  int e = n_entries, base = 0;
  if (n_entries == 1) {
    e = 0;
    base = -first_chunk;
  } else if (n_entries <= THREADS) {
    __shared__ int found[2];
    const int t = threadIdx.x;
    if (t < n_entries) {
      const int len = cu_q[t + 1] - cu_q[t];
      int longer = 0, before = -first_chunk;
#pragma unroll 4
      for (int x = 0; x < n_entries; ++x) {
        const int other = cu_q[x + 1] - cu_q[x];
        longer += other > len || (other == len && x < t);
        before += x < t ? chunks_of(other, least) : 0;
      }
      if (longer == (int)blockIdx.z) found[0] = t, found[1] = before;
    }
    __syncthreads();
    e = __reduce_max_sync(0xffffffffu, found[0]);        // (the same in every lane, which the compiler can see)
    base = __reduce_max_sync(0xffffffffu, found[1]);
  } else {                                               // more than one a thread: in the step's order
#pragma unroll 8
    for (int x = 0, seen = 0, before = -first_chunk; x < n_entries; ++x) {       // no way out: the loads do not wait for each other
      const int mine = chunks_of(cu_q[x + 1] - cu_q[x], least);
      const bool it = mine > 0 && seen == (int)blockIdx.z;
      e = it ? x : e;
      base = it ? before : base;
      seen += mine > 0;
      before += mine;
    }
  }
  if (e == n_entries) return;
  const int h = blockIdx.y, c0 = blockIdx.x * COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int first = cu_q[e], n = cu_q[e + 1] - first;
  const int from = max(0, -base), to = min(chunks_of(n, least), n_chunks - base);
  if (from >= to) return;
  const int rec_floats = record_floats(z.dv);
  auto fetch = [&](int s) {
    if (s < to) {
      const float* src = records + ((size_t)(base + s) * z.H + h) * rec_floats;
      float* dst = chunk_smem + (s % STAGES) * STAGE;
#pragma unroll
      for (int i = 0; i < 3 * TOK * DK / 4 / THREADS; ++i) {
        const int idx = tid + i * THREADS, row = idx / (DK / 4), c = (idx % (DK / 4)) * 4;
        state_copy_16(dst + row * LD + c, src + row * DK + c);
      }
      if (tid < 2 * TOK * COLS / 4) {
        const int row = tid / (COLS / 4), c = (tid % (COLS / 4)) * 4;
        state_copy_16(dst + 3 * TOK * LD + row * COLS + c, src + 3 * TOK * DK + row * z.dv + c0 + c);
      }
      if (tid == THREADS - 1) state_copy_4(dst + 3 * TOK * LD + 2 * TOK * COLS, src + 3 * TOK * DK + 2 * TOK * z.dv);
    }
    state_copy_commit();
  };
#pragma unroll
  for (int s = from; s < from + STAGES - 1; ++s) fetch(s);
  float* S_head = state + (size_t)slots[e] * state_stride + (size_t)h * z.dv * DK;
  float S[2][4];
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const float2 v = *reinterpret_cast<const float2*>(S_head + (size_t)(c0 + g + 8 * half) * DK + warp * ROWS + 8 * x + 2 * t);
      S[x][2 * half] = v.x;
      S[x][2 * half + 1] = v.y;
    }
  const int tok = tid / COLS, col = tid % COLS;          // what the thread finishes of a chunk: one u and one o
  // the warp's sums [token][column] of a product, left for the others
  auto leave = [&](float* to, const float (&c)[2][4]) {
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int v = 0; v < 4; ++v) to[warp * SUMS + (8 * y + 2 * t + (v & 1)) * SUM_LD + g + (v >> 1) * 8] = c[y][v];
  };
  auto gather = [&](const float* from) {
    float sum = 0.f;
#pragma unroll
    for (int x = 0; x < WARPS; ++x) sum += from[x * SUMS + tok * SUM_LD + col];
    return sum;
  };
  // kx . S or qm . S over the warp's rows, 16 tokens
  auto product = [&](const float* rows, const Split (&a)[2][4], float (&c)[2][4]) {
    float large[2][2][4] = {};
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const float2 r = *reinterpret_cast<const float2*>(rows + (8 * y + g) * LD + warp * ROWS + 8 * x + 2 * t);
        const Split b[2] = {split(r.x), split(r.y)};
        mma_split(c[y], large[x][y], a[x], b);
      }
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int v = 0; v < 4; ++v) c[y][v] += large[0][y][v] + large[1][y][v];
  };
  float o0 = 0.f;
  auto finish = [&](int s) {                             // the thread's o of chunk s
    if (s * TOK + tok < n) o_out[((size_t)(first + s * TOK + tok) * z.H + h) * z.dv + c0 + col] = o0 + gather(q_sums);
  };
  for (int s = from; s < to; ++s) {
    state_copy_wait<STAGES - 2>();
    __syncthreads();                                     // chunk s is here for all; chunk s - 1 is read by all
    if (s > from) finish(s - 1);
    fetch(s + STAGES - 1);
    const float* st = chunk_smem + (s % STAGES) * STAGE;
    Split a[2][4];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      a[x][0] = split(S[x][0]);
      a[x][1] = split(S[x][2]);
      a[x][2] = split(S[x][1]);
      a[x][3] = split(S[x][3]);
    }
    float p[2][4] = {}, w[2][4] = {};
    product(st, a, p);
    leave(p_sums, p);
    __syncthreads();
    u_s[tok * U_LD + col] = st[3 * TOK * LD + tid] - gather(p_sums);
    product(st + TOK * LD, a, w);                        // does not wait for u: its sums are gathered a chunk later
    o0 = st[3 * TOK * LD + TOK * COLS + tid];
    const float whole = st[3 * TOK * LD + 2 * TOK * COLS];
    __syncthreads();
    float small[2][4] = {}, large[2][2][4] = {};
#pragma unroll
    for (int y = 0; y < 2; ++y) {                        // eight tokens
      const float* at = u_s + (8 * y + t) * U_LD + g;
      const Split ua[4] = {split(at[0]), split(at[8]), split(at[4 * U_LD]), split(at[4 * U_LD + 8])};
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float* ke = st + (2 * TOK + 8 * y + t) * LD + warp * ROWS + 8 * x + g;
        const Split b[2] = {split(ke[0]), split(ke[4 * LD])};
        mma_split(small[x], large[x][y], ua, b);
      }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int v = 0; v < 4; ++v) S[x][v] = fmaf(whole, S[x][v], (large[x][0][v] + large[x][1][v]) + small[x][v]);
    leave(q_sums, w);
  }
  __syncthreads();
  finish(to - 1);
  state_copy_wait<0>();
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int half = 0; half < 2; ++half)
      *reinterpret_cast<float2*>(S_head + (size_t)(c0 + g + 8 * half) * DK + warp * ROWS + 8 * x + 2 * t) =
          make_float2(S[x][2 * half], S[x][2 * half + 1]);
}

}  // namespace chunks
}  // namespace srlm

using namespace srlm;

// Floats of a chunk's record for one head, 0 where these sizes go token by token.
extern "C" int srlm_delta_chunk_record(int dk, int dv, int taps) {
  return dk == chunks::DK && dv > 0 && dv % chunks::COLS == 0 && dv <= 1024 && taps >= 1 && taps <= chunks::TAPS
             ? chunks::record_floats(dv) : 0;
}

// proj float32 [T, ldp] and state as in delta_rule.cu, whose limits hold for an entry of any length.  Serves the entries of
// `least` tokens and more: the chunks first_chunk .. first_chunk + n_chunks - 1 of those that they have together, entry by entry;
// a step whose chunks do not all fit `records` (float32 [n_chunks, H, record]) is several calls, in order.  n_long:
// how many entries they are.  o_out float32 [T, H dv].  Renews S; the carried inputs of the convolution are read and stay.
extern "C" int srlm_delta_chunks(const float* proj, long long ldp, const float* conv_w, const float* a_log, const float* dt_bias,
                                 float* state, long long state_stride, const int* cu_q, const int* slots, int n_entries,
                                 float* records, int least, int n_long, int first_chunk, int n_chunks, float* o_out, int H,
                                 int G, int dk, int dv, int taps, float unit_eps, cudaStream_t stream) {
  if (n_entries <= 0 || n_long <= 0 || n_chunks <= 0) return ST_OK;
  const long long C = 2LL * G * dk + (long long)H * dv;
  if (!srlm_delta_chunk_record(dk, dv, taps) || first_chunk < 0 || H <= 0 || G <= 0 || H % G || H > 65535 || n_entries > 65535 ||
      n_long > n_entries || ldp < C + 2LL * H || C * 4 > 200 * 1024 || state_stride < (long long)H * dk * dv + C * (taps - 1))
    return refuse(ST_BAD_SIZE, "delta_chunks: H=%d G=%d dk=%d dv=%d taps=%d ldp=%lld state=%lld entries=%d", H, G, dk, dv, taps,
                  ldp, state_stride, n_entries);
  if ((uintptr_t)state % 8 || state_stride % 2 || (uintptr_t)records % 16)
    return refuse(ST_BAD_ALIGN, "delta_chunks: states start on 8 bytes, records on 16");
  const chunks::Sizes z{H, G, dv, (int)C};
  launch_pdl(chunks::delta_chunks_kernel, dim3(n_chunks, H), dim3(128), 0, stream, proj, ldp, conv_w, taps, a_log, dt_bias,
             (const float*)state, state_stride, cu_q, n_entries, slots, records, least, first_chunk, z, unit_eps);
  const cudaError_t e = cudaFuncSetAttribute(chunks::delta_chunk_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             chunks::WALK_SMEM);
  if (e != cudaSuccess) return refuse((int)e, "delta_chunks: cannot get %d bytes of shared memory", chunks::WALK_SMEM);
  // (not ahead of time: blocks that start while the chunks' kernel drains would share the SMs that happen to be free)
  launch_pdl_if(false, chunks::delta_chunk_walk_kernel, dim3(dv / chunks::COLS, H, n_long), dim3(chunks::THREADS),
                chunks::WALK_SMEM, stream, (const float*)records, state, state_stride, cu_q, n_entries, slots, o_out,
                least, first_chunk, n_chunks, z);
  return launched();
}
