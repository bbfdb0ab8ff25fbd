// Paged causal attention for a ragged batch, plain FMA arithmetic in float32.
//
// A row (token, query head) walks its request's keys in blocks of 32 aligned to
// multiples of 32 from the start of the sequence, one running softmax, a score one
// chain of FMAs over the head, an output one chain over the keys: the order of
// every sum depends only on the token's position, so the result is the same however
// the tokens were cut into steps or batched.  This is the attention of the float32
// path, and the reference the tensor-core kernels are tested against.  Formula:
// src/model/math.rs:102-155 (scale 1/sqrt(hd) or the given one, query head h reads
// KV head h / (nq/nkv), online softmax).
//
// A block serves up to 32 rows that read the same KV head: the query heads of a run of tokens of one request.  Keys and
// values of a span of keys are copied to shared memory once for all rows, the next span in flight under the current one.  Eight
// warps form the scores, a lane a key; then each warp owns up to four rows, a lane the dimensions lane + 32 i.  Bound by the
// warps' waits for one another and for shared memory between two barriers, which a second block on the SM fills.  Three shapes with
// the same sums (pick_shape):
//  * paired: spans of 64 keys (32 for heads above 64), two blocks an SM.  Prompts: 2,048 tokens, 32 heads of 128 in 2.05 ms, of 64
//    in 16 heads 0.69 (2.79 and 1.06 with one block an SM and spans twice as long, 34.2 with a warp a row that read its keys
//    from global memory).
//  * long: spans of 128 / 64 / 32 keys (heads up to 64 / 128 / 256), one block an SM, where the blocks are fewer than the SMs and
//    the chain of spans of the longest request is the time (8 requests of 2,048, 32 heads of 128: 0.14 ms; paired, 0.31
//    where it was 0.19).
//  * small: 8 rows and spans of 32 keys without a second buffer, several blocks an SM, for many requests of few rows, or few keys:
//    they hide the trips to memory that a short request consists of (64 requests of 16 keys, 32 heads of 64: 118 us in the long
//    shape, which leaves such a request an SM, 15 in the small one, 19 with the warp a row).
#include <math_constants.h>

#include "common.cuh"

namespace srlm {

enum SimtShape { SMALL, PAIRED, LONG };      // (see pick_shape)

template <int DIMS, SimtShape SHAPE>          // DIMS: dimensions a lane owns, heads up to 32 * DIMS
struct SimtForm {
  static constexpr int KEYS = SHAPE == SMALL ? 32 : SHAPE == PAIRED ? (DIMS <= 2 ? 64 : 32) : DIMS <= 2 ? 128 : DIMS <= 4 ? 64 : 32;
  static constexpr int THREADS = SHAPE == SMALL ? 128 : 256, WARPS = THREADS / 32;
  static constexpr int STAGES = SHAPE == SMALL ? 1 : 2, ROWS = SHAPE == SMALL ? 8 : 32, OWN = ROWS / WARPS;
  static constexpr int BLOCKS = SHAPE == SMALL ? (DIMS <= 2 ? 8 : DIMS <= 4 ? 5 : 3) : SHAPE == PAIRED ? 2 : 1;      // an SM
};

// Floats from a staged key to the next: an odd number of 16-byte pieces, so that lanes on neighbouring keys share no bank.
__host__ __device__ __forceinline__ int simt_key_ld(int hd) { return 4 * (((hd + 3) / 4) | 1); }
__host__ __device__ __forceinline__ int simt_row_ld(int hd) { return (hd + 3) / 4 * 4; }

template <typename F>
static size_t simt_smem(int hd) {
  return sizeof(float) * ((size_t)F::STAGES * F::KEYS * (simt_key_ld(hd) + simt_row_ld(hd)) + (size_t)F::ROWS * simt_row_ld(hd) +
                          (size_t)F::ROWS * F::KEYS) + sizeof(long long) * 2 * F::KEYS;
}

// Scores of `NR` neighbouring rows against a lane's key.
template <int NR>
__device__ __forceinline__ void simt_scores(const float* __restrict__ kp, const float* __restrict__ qs, int ldq, int pieces,
                                            float (&dot)[NR]) {
#pragma unroll
  for (int r = 0; r < NR; ++r) dot[r] = 0.f;
#pragma unroll 4
  for (int c = 0; c < pieces; ++c) {
    const float4 k = *reinterpret_cast<const float4*>(kp + 4 * c);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const float4 x = *reinterpret_cast<const float4*>(qs + r * ldq + 4 * c);
      dot[r] = fmaf(x.x, k.x, dot[r]);
      dot[r] = fmaf(x.y, k.y, dot[r]);
      dot[r] = fmaf(x.z, k.z, dot[r]);
      dot[r] = fmaf(x.w, k.w, dot[r]);
    }
  }
}

struct SimtYes { static constexpr bool value = true; };
struct SimtNo { static constexpr bool value = false; };
template <int N> struct SimtOwn { static constexpr int value = N; };

// The rows of tokens t0 .. t0 + tokens - 1 (one request) and heads h_lo .. h_lo + heads - 1 of KV head kvh.
template <typename TA, int DIMS, bool COPY, SimtShape SHAPE>       // COPY: float32 rows of whole 16-byte pieces, fetched asynchronously
__device__ void simt_rows(const TA* __restrict__ q, const TA* __restrict__ k_cache, const TA* __restrict__ v_cache,
                          TA* __restrict__ out, const int* __restrict__ table, const int* __restrict__ positions, int t0,
                          int tokens, int nq, int nkv, int kvh, int h_lo, int heads, int hd, int page_size, float scale,
                          int window) {
  typedef SimtForm<DIMS, SHAPE> Form;
  constexpr int KEYS = Form::KEYS, STAGES = Form::STAGES, SA_ROWS = Form::ROWS, SA_OWN = Form::OWN,
                SA_THREADS = Form::THREADS, SA_WARPS = Form::WARPS;
  extern __shared__ __align__(16) float simt_sh[];
  const int g = nq / nkv;
  const int rows = tokens * heads;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ldk = simt_key_ld(hd), ldv = simt_row_ld(hd), pieces = ldv / 4;
  float* k_sh = simt_sh;                                     // [STAGES][KEYS][ldk]
  float* v_sh = k_sh + STAGES * KEYS * ldk;                  // [STAGES][KEYS][ldv]
  float* q_sh = v_sh + STAGES * KEYS * ldv;                  // [SA_ROWS][ldv]
  float* s_sh = q_sh + SA_ROWS * ldv;                        // [SA_ROWS][KEYS]: scores, then weights
  long long* at_sh = reinterpret_cast<long long*>(s_sh + SA_ROWS * KEYS);      // [2][KEYS]: cache row of a key, or -1

  for (int i = tid; i < SA_ROWS * ldv; i += SA_THREADS) {
    const int r = i / ldv, d = i % ldv;
    const bool there = r < rows && d < hd;
    q_sh[i] = there ? to_float(q[((size_t)(t0 + r / heads) * nq + kvh * g + h_lo + r % heads) * hd + d]) : 0.f;
  }
  int first = 0x7fffffff, last = -1;                         // keys that some row of the block sees
  for (int i = 0; i < tokens; ++i) {
    const int p = positions[t0 + i];
    first = min(first, window > 0 ? max(0, p - window + 1) : 0);
    last = max(last, p);
  }
  first = first / KEYS * KEYS;
  const int spans = last / KEYS - first / KEYS + 1;
  auto locate = [&](int span) {
    if (tid < KEYS) {
      const int j = first + span * KEYS + tid;
      at_sh[(span & 1) * KEYS + tid] =
          j <= last ? (((long long)table[j / page_size] * nkv + kvh) * page_size + j % page_size) * hd : -1;
    }
  };
  auto fetch = [&](int span) {
    if (span < spans) {
      float* kd = k_sh + span % STAGES * KEYS * ldk;
      float* vd = v_sh + span % STAGES * KEYS * ldv;
      const long long* at = at_sh + (span & 1) * KEYS;
      for (int i = tid; i < KEYS * pieces; i += SA_THREADS) {
        const int key = i / pieces, c = (i % pieces) * 4;
        const long long row = at[key];
        if (row < 0) continue;                               // nobody uses what this place holds
        if constexpr (COPY) {
          const unsigned int ka = (unsigned int)__cvta_generic_to_shared(kd + key * ldk + c);
          const unsigned int va = (unsigned int)__cvta_generic_to_shared(vd + key * ldv + c);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ka), "l"(k_cache + row + c) : "memory");
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(va), "l"(v_cache + row + c) : "memory");
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            kd[key * ldk + c + e] = c + e < hd ? to_float(k_cache[row + c + e]) : 0.f;
            vd[key * ldv + c + e] = c + e < hd ? to_float(v_cache[row + c + e]) : 0.f;
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // the rows that this warp owns behind the scores: warp, warp + 8, ...
  float acc[SA_OWN][DIMS], m[SA_OWN], z[SA_OWN];
  int low[SA_OWN], high[SA_OWN];
#pragma unroll
  for (int o = 0; o < SA_OWN; ++o) {
    const int r = warp + o * SA_WARPS;
    const int p = r < rows ? positions[t0 + r / heads] : -1;
    low[o] = r < rows ? (window > 0 ? max(0, p - window + 1) : 0) : 0x7fffffff;
    high[o] = p;
    m[o] = -CUDART_INF_F;
    z[o] = 0.f;
#pragma unroll
    for (int i = 0; i < DIMS; ++i) acc[o][i] = 0.f;
  }

  locate(0);
  __syncthreads();
  if constexpr (STAGES == 2) {
    fetch(0);
    locate(1);
    __syncthreads();
  }
  for (int span = 0; span < spans; ++span) {
    fetch(span + STAGES - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
    __syncthreads();                                         // the span has arrived, the places of the next are read
    const int j0 = first + span * KEYS;
    const int here = min(KEYS / 32, (last - j0) / 32 + 1);   // blocks of 32 keys that somebody may see
    {
      const float* ks = k_sh + span % STAGES * KEYS * ldk;
      constexpr int EACH = SHAPE == SMALL ? 2 : 8;           // rows a task: two where a span is one block of keys for four warps
      const bool few = rows <= 2;
      const int groups = few ? 1 : (rows + EACH - 1) / EACH;
      for (int task = warp; task < groups * here; task += SA_WARPS) {
        const int kb = task % here * 32, r0 = task / here * EACH;
        const float* kp = ks + (kb + lane) * ldk;
        if (SHAPE == SMALL || few) {
          float dot[2];
          simt_scores<2>(kp, q_sh + r0 * ldv, ldv, pieces, dot);
#pragma unroll
          for (int r = 0; r < 2; ++r) s_sh[(r0 + r) * KEYS + kb + lane] = dot[r] * scale;
        } else {
          float dot[8];
          simt_scores<8>(kp, q_sh + r0 * ldv, ldv, pieces, dot);
#pragma unroll
          for (int r = 0; r < 8; ++r) s_sh[(r0 + r) * KEYS + kb + lane] = dot[r] * scale;
        }
      }
    }
    locate(span + STAGES);
    __syncthreads();
    const float* vs = v_sh + span % STAGES * KEYS * ldv;
    auto values = [&](auto own) {                            // own: rows a warp owns, at most; with one nothing branches by row
                                                             // (a request of 700 keys, 16 heads over 8 of 64: 42 -> 27 us)
#pragma unroll 1
      for (int kb = 0; kb < 32 * here; kb += 32) {
        const int jb = j0 + kb, j = jb + lane;
        bool any = false, all = true;                        // (uniform over the warp)
#pragma unroll
        for (int o = 0; o < decltype(own)::value; ++o) {
          if (decltype(own)::value > 1 && warp + o * SA_WARPS >= rows) continue;
          float* sp = s_sh + (warp + o * SA_WARPS) * KEYS + kb + lane;
          const bool valid = j >= low[o] && j <= high[o];
          float p = 0.f;
          if (__any_sync(0xffffffffu, valid)) {              // else the row does not see this block: nothing changes
            const float s = valid ? *sp : -CUDART_INF_F;
            const float m_new = fmaxf(m[o], warp_max(s));
            const float alpha = expf(m[o] - m_new);          // m = -inf at first: exp(-inf) = 0
            p = valid ? expf(s - m_new) : 0.f;
            z[o] = z[o] * alpha + warp_sum(p);
            m[o] = m_new;
#pragma unroll
            for (int i = 0; i < DIMS; ++i) acc[o][i] *= alpha;
            any = true;
          }
          all &= __all_sync(0xffffffffu, p != 0.f);
          *sp = p;
        }
        if (!any) continue;
        __syncwarp();
        const float* vp = vs + (size_t)kb * ldv + lane;
        // a weight of zero (a key out of the row's sight, or one far below the maximum) leaves its value unread
        auto add = [&](auto tested) {
#pragma unroll 2
          for (int jj = 0; jj < 32; jj += 4) {
            float v[4][DIMS];
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
              for (int i = 0; i < DIMS; ++i) v[e][i] = lane + 32 * i < ldv ? vp[(jj + e) * ldv + 32 * i] : 0.f;
#pragma unroll
            for (int o = 0; o < decltype(own)::value; ++o) {
              if (decltype(own)::value > 1 && warp + o * SA_WARPS >= rows) continue;
              const float4 w = *reinterpret_cast<const float4*>(s_sh + (warp + o * SA_WARPS) * KEYS + kb + jj);
              const float ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (!decltype(tested)::value || ws[e] != 0.f)
#pragma unroll
                  for (int i = 0; i < DIMS; ++i) acc[o][i] = fmaf(ws[e], v[e][i], acc[o][i]);
            }
          }
        };
        if (all) add(SimtNo{}); else add(SimtYes{});
      }
    };
    if (rows > SA_WARPS) values(SimtOwn<SA_OWN>{});
    else if (warp < rows) values(SimtOwn<1>{});
    __syncthreads();                                         // the span's buffers and scores are free
  }
#pragma unroll
  for (int o = 0; o < SA_OWN; ++o) {
    const int r = warp + o * SA_WARPS;
    if (r >= rows) continue;
    TA* dst = out + ((size_t)(t0 + r / heads) * nq + kvh * g + h_lo + r % heads) * hd;
    const float inv = 1.f / z[o];
#pragma unroll
    for (int i = 0; i < DIMS; ++i) {
      const int d = lane + 32 * i;
      if (d < hd) dst[d] = from_float<TA>(acc[o][i] * inv);
    }
  }
}

// A block is (tile of tokens, KV head, lane of runs): of the runs of tokens of one request within the tile, it serves the
// of_lane-th and every lanes-th behind it.  Where an SM holds one block or two, those with most keys should not come last: the
// tiles are taken from both ends, the requests of a step's front (its decoding ones) and the end of its prompts first (300 tokens
// beside 5 requests of up to 700 keys, 16 heads of 64: 68 us where the runs behind a tile's first came last, 56 now).
template <typename TA, int DIMS, bool COPY, SimtShape SHAPE>
__global__ void __launch_bounds__((SimtForm<DIMS, SHAPE>::THREADS), (SimtForm<DIMS, SHAPE>::BLOCKS))
paged_attention_simt_kernel(const TA* __restrict__ q, const TA* __restrict__ k_cache, const TA* __restrict__ v_cache,
                            TA* __restrict__ out, const int* __restrict__ block_table, int table_stride,
                            const int* __restrict__ entry_of_token, const int* __restrict__ positions, int T, int nq,
                            int nkv, int hd, int page_size, float scale, int window, int tile_tokens, int head_groups) {
  constexpr int ROWS = SimtForm<DIMS, SHAPE>::ROWS;
  const int g = nq / nkv, tiles = (T + tile_tokens - 1) / tile_tokens;
  int tile, place, of_lane, lanes;
  if constexpr (SHAPE == SMALL) {
    tile = blockIdx.x, place = blockIdx.y, of_lane = blockIdx.z, lanes = gridDim.z;
  } else {
    const int turn = blockIdx.z * gridDim.y + blockIdx.y;
    if (turn >= tiles) return;
    tile = turn & 1 ? tiles - 1 - turn / 2 : turn / 2;
    lanes = gridDim.x / (nkv * head_groups), place = blockIdx.x / lanes, of_lane = blockIdx.x % lanes;
  }
  const int kvh = place / head_groups, h_lo = place % head_groups * ROWS;
  const int heads = min(g - h_lo, ROWS);                  // (tile_tokens is 1 where a group has more heads than rows)
  const int t_end = min((tile + 1) * tile_tokens, T);
  int run = 0;
  for (int t = tile * tile_tokens; t < t_end; ++run) {
    const int entry = entry_of_token[t];
    int tokens = 1;
    while (t + tokens < t_end && entry_of_token[t + tokens] == entry) ++tokens;
    if (run % lanes == of_lane)
      simt_rows<TA, DIMS, COPY, SHAPE>(q, k_cache, v_cache, out, block_table + (size_t)entry * table_stride, positions, t, tokens, nq,
                                nkv, kvh, h_lo, heads, hd, page_size, scale, window);
    t += tokens;
  }
}

// Which shape.  Requests of up to 8 rows (decode): the small one once there are more of them than SMs (us, long | small: 16 heads
// over 8 of 64, 64 requests of 700 keys 174 | 79, of 16 27 | 7; below that the long spans win, 4 requests of 700 43 | 76; with
// a warp's one row unrolled by itself the small one takes 69 for the 64 requests of 700, the long one 27 for the 4).
// Prompts: the small one where they see few keys (16 over 8 heads of 64, 20 tokens 12.4 | 7.5), or where the heads are wide,
// whose spans are short in all, and its finer blocks fill the GPU better (us, paired | small, 16 over 8 of 128: 300 tokens
// 69 | 63, 500 tokens 133 | 125; 32 over 4 of 128, 40 tokens behind 500 keys 103 long | 74).  Else two blocks an SM once there are
// more blocks than SMs (16 over 8 of 64, us, long | paired: 1,000 tokens 280 | 206; 256 tokens behind 1,500 keys, 128 blocks,
// 222 | 233).
static SimtShape pick_shape(int T, int nq, int nkv, int hd, int runs, int most_keys) {
  const int g = nq / nkv, rows = 32, tile_tokens = g >= rows ? 1 : rows / g;
  if (runs > T) runs = T;
  const long long tiles = (T + tile_tokens - 1) / tile_tokens;
  const long long blocks = (tiles > runs ? tiles : runs) * nkv * ((g + rows - 1) / rows);      // of the large form
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 148;
  if ((long long)T * g <= 8ll * runs) return blocks > sms ? SMALL : LONG;
  if ((most_keys > 0 && most_keys <= 128) || (hd > 64 && blocks <= 2 * sms)) return SMALL;
  return blocks > sms && hd <= 128 ? PAIRED : LONG;
}

template <typename TA, int DIMS, bool COPY, SimtShape SHAPE>
static int run_simt_form(const void* q, const void* k_cache, const void* v_cache, void* out, const int* block_table,
                         int table_stride, const int* entry_of_token, const int* positions, int T, int nq, int nkv, int hd,
                         int page_size, float scale, int window, int runs, cudaStream_t stream) {
  typedef SimtForm<DIMS, SHAPE> Form;
  const size_t smem = simt_smem<Form>(hd);
  const auto kernel = paged_attention_simt_kernel<TA, DIMS, COPY, SHAPE>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int g = nq / nkv, head_groups = (g + Form::ROWS - 1) / Form::ROWS;
  const int tile_tokens = g >= Form::ROWS ? 1 : Form::ROWS / g;
  const int z = runs < 1 ? 1 : runs < tile_tokens ? runs : tile_tokens;
  const int tiles = (T + tile_tokens - 1) / tile_tokens, most = 65535, places = nkv * head_groups;
  const dim3 grid = SHAPE == SMALL ? dim3(tiles, places, z) : dim3(places * z, tiles < most ? tiles : most, (tiles + most - 1) / most);
  kernel<<<grid, Form::THREADS, smem, stream>>>(
      (const TA*)q, (const TA*)k_cache, (const TA*)v_cache, (TA*)out, block_table, table_stride, entry_of_token, positions, T,
      nq, nkv, hd, page_size, scale, window, tile_tokens, head_groups);
  return launched();
}

template <typename TA, int DIMS, bool COPY>
static int run_simt(const void* q, const void* k_cache, const void* v_cache, void* out, const int* block_table,
                    int table_stride, const int* entry_of_token, const int* positions, int T, int nq, int nkv, int hd,
                    int page_size, float scale, int window, int runs, int most_keys, cudaStream_t stream) {
  const auto go = [&](auto run_form) {
    return run_form(q, k_cache, v_cache, out, block_table, table_stride, entry_of_token, positions, T, nq, nkv, hd, page_size, scale,
                    window, runs, stream);
  };
  const SimtShape shape = pick_shape(T, nq, nkv, hd, runs, most_keys);
  if (shape == SMALL) return go(run_simt_form<TA, DIMS, COPY, SMALL>);
  if constexpr (DIMS <= 4) {
    if (shape == PAIRED) return go(run_simt_form<TA, DIMS, COPY, PAIRED>);
  }
  return go(run_simt_form<TA, DIMS, COPY, LONG>);
}

template <typename TA, bool COPY, typename... Args>
static int run_simt_dims(int hd, Args... args) {
  if (hd <= 64) return run_simt<TA, 2, COPY>(args...);
  if (hd <= 128) return run_simt<TA, 4, COPY>(args...);
  return run_simt<TA, 8, COPY>(args...);
}

}  // namespace srlm

using namespace srlm;

// runs: how many requests' tokens may stand beside each other in a tile of tokens (a hint: it spreads them over blocks);
// most_keys: no request of the step has more keys (a hint too; 0: not known).
extern "C" int srlm_paged_attention_simt(const void* q, const void* k_cache, const void* v_cache,
                                         void* out, int act_dtype, int cache_dtype,
                                         const int* block_table, int table_stride,
                                         const int* entry_of_token, const int* positions, int T, int nq,
                                         int nkv, int hd, int page_size, float scale, int window, int runs,
                                         int most_keys, cudaStream_t stream) {
  if (T <= 0) return ST_OK;
  if (nq <= 0 || nkv <= 0 || nq % nkv || hd <= 0 || hd > 256 || page_size <= 0 ||
      nkv * ((nq / nkv + 7) / 8) > 65535)
    return refuse(ST_BAD_SIZE,
                  "paged_attention_simt: nq=%d nkv=%d hd=%d page_size=%d (needs nq %% nkv == 0, hd <= %d)",
                  nq, nkv, hd, page_size, 256);
  if (act_dtype != cache_dtype)
    return refuse(ST_BAD_DTYPE, "paged_attention_simt: cache dtype %d differs from activations %d",
                  cache_dtype, act_dtype);
  if (act_dtype == DT_F32) {
    if (hd % 4 == 0 && ((uintptr_t)k_cache | (uintptr_t)v_cache) % 16 == 0)
      return run_simt_dims<float, true>(hd, q, k_cache, v_cache, out, block_table, table_stride, entry_of_token, positions, T,
                                        nq, nkv, hd, page_size, scale, window, runs, most_keys, stream);
    return run_simt_dims<float, false>(hd, q, k_cache, v_cache, out, block_table, table_stride, entry_of_token, positions, T,
                                       nq, nkv, hd, page_size, scale, window, runs, most_keys, stream);
  }
  if (act_dtype != DT_BF16) return refuse(ST_BAD_DTYPE, "dtype code %d is not known", act_dtype);
  return run_simt_dims<bf16, false>(hd, q, k_cache, v_cache, out, block_table, table_stride, entry_of_token, positions, T, nq,
                                    nkv, hd, page_size, scale, window, runs, most_keys, stream);
}
