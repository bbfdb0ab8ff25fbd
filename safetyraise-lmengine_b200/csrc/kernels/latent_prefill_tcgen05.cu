// Prompts of an attention over a cached latent, in the heads' own space, on the 5th-generation tensor cores: keys of
// 128 + 64 elements (a head's unrotated key, formed for the step from the latent; the rotated part, which the heads share,
// from the pages) and values of 128.
//
// The plan is attention_prefill_tcgen05.cu's, with a KV head per query head: a block takes up to 256 tokens of one entry and
// one head as two tiles of 128 rows and walks the keys in tiles of 128; S = Q K^T and O += P V are tcgen05.mma with
// accumulators in tensor memory, P is bfloat16 over the columns of S, one thread owns a row's softmax.  What differs: O is
// rescaled whenever a row's maximum has grown, and a row's sum is that of the rounded weights (with sums of the unrounded
// ones and a maximum that may lag by 2^8, so that the largest weight is rounded too, the layer's error against float64 was
// 0.5 % above that of the kernel on mma.sync, 1.3 % at 300 tokens behind 1,000; so it is 0.1 % below; it costs 9 us of 166
// in a layer of 1,800 tokens); an operand row is three panels of 64 elements, two fetched from the step's matrix of keys and
// values (one box of 128 rows) and one from the pages (a box a page); the queries arrive in float32 as projected and are
// rotated and rounded on their way into shared memory; a head's output gate is applied to the float32 sums as they leave.
//
// Shared memory holds 96 KB of queries, two K tiles (96 KB) and one V tile (32 KB): a V tile is fetched under the S product
// and the softmax that follow the product that freed it.  Bound by the softmax (one exponential and about nine other
// instructions a score), the rescaling and the MMA issue of the longest block.  1,800 tokens behind 200, 16 heads: 62 us (485 on
// mma.sync, plus 30 for the rotation and the gate by themselves).
#include "attention_tcgen05.cuh"

namespace srlm {
namespace lfmha {

using namespace fmha;

constexpr int BR = 128, KT = 128, DIM = 128, ROT = 64, DV = 128;
constexpr int PANEL = 128 * 128;                         // bytes: 128 rows of 64 elements
constexpr int QK_BYTES = 3 * PANEL, V_BYTES = 2 * PANEL;
constexpr int K_STAGES = 2;
constexpr int THREADS = 320;                             // warp 0: TMA, warp 1: MMA, warps 2-5 and 6-9: softmax
constexpr int SMEM = 2 * QK_BYTES + K_STAGES * QK_BYTES + V_BYTES + 24 * 8 + 1024;
static_assert(SMEM <= 227 * 1024, "");

struct Args {
  const float* q;            // heads x (128 | 64) lead a token's row of ldq floats
  long long ldq;
  bool q_vec;                // see load_queries
  const float* cos_t;        // [T, pairs]
  const float* sin_t;
  int pairs;
  bool halves;               // partners (i, i + pairs), else (2i, 2i + 1)
  const float* gate;         // logit of head h of token t: gate[t * ld_gate + h], or null
  long long ld_gate;
  bf16* out;                 // [T, heads, 128]
  const int* block_table;
  int table_stride;
  const int* cu_q;
  const int* kv_lens;
  const int* cu_kv;          // row of key 0 of an entry in the matrix of keys and values (may be negative: see the caller)
  const int* work;           // (entry, block of tiles_per_block x 128 tokens)
  int heads, page_size, rank, v_off, tiles_per_block, window;
  float scale_log2;
  int* err_flag;
};

__device__ __forceinline__ void load8(const float* src, float (&x)[8]) {
  const float4 lo = __ldg(reinterpret_cast<const float4*>(src)), hi = __ldg(reinterpret_cast<const float4*>(src + 4));
  x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w;
  x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
}
// Element r of a query's rotated part: x, partner, cosine and sine -> the turned element.
__device__ __forceinline__ float turned(float x, float partner, float c, float s, bool second) {
  return second ? x * c + partner * s : x * c - partner * s;
}
__device__ __forceinline__ void put8(uint32_t at, const float (&x)[8]) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(pack2(x[0], x[1])), "r"(pack2(x[2], x[3])),
               "r"(pack2(x[4], x[5])), "r"(pack2(x[6], x[7])) : "memory");
}

// `rows` query rows of a head -> shared memory, turned and rounded, in the swizzled K-major layout (zeros beyond the entry's
// rows).  A thread has four pieces (of eight elements) in flight, two of the rotated part, whose cosines and sines come
// with them (with scalar reads of the tables a tile of 128 rows took 12 us instead of 4); more pieces unrolled make code that
// every block fetches cold: with eight and four, a block of 5 rows took 12.3 us instead of 10.3.
template <bool VEC>              // whole 16-byte pieces everywhere: rows, tables, and pairs that do not straddle a piece
__device__ __forceinline__ void load_queries(const Args& a, uint32_t q_tiles, int rows, bool two, int first_token, int left,
                                             int head, int tid, int threads) {
  auto place = [&](int row, int c) {       // a block of one row tile keeps it in slot 1
    return tile_addr(q_tiles + (two ? row >> 7 : 1) * QK_BYTES, row & 127, c);
  };
  auto source = [&](int row) { return a.q + (size_t)(first_token + row) * a.ldq + (size_t)head * (DIM + ROT); };
  constexpr int PLAIN = DIM / 8, TURNED = ROT / 8, QB = 4, RB = 2;
#pragma unroll 1
  for (int base = tid; base < rows * PLAIN; base += threads * QB) {
    float x[QB][8];
#pragma unroll
    for (int j = 0; j < QB; ++j) {
      const int idx = base + j * threads, row = idx / PLAIN, d = (idx % PLAIN) * 8;
      const bool there = idx < rows * PLAIN && row < left;
#pragma unroll
      for (int i = 0; i < 8; ++i) x[j][i] = 0.f;
      if (there) {
        if constexpr (VEC) {
          load8(source(row) + d, x[j]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) x[j][i] = __ldg(source(row) + d + i);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < QB; ++j) {
      const int idx = base + j * threads;
      if (idx < rows * PLAIN) put8(place(idx / PLAIN, idx % PLAIN), x[j]);
    }
  }
#pragma unroll 1
  for (int base = tid; base < rows * TURNED; base += threads * RB) {
    float x[RB][8], y[RB][8], c[RB][8], s[RB][8];
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int idx = base + j * threads, row = idx / TURNED, r0 = (idx % TURNED) * 8;
      const bool there = idx < rows * TURNED && row < left;
#pragma unroll
      for (int i = 0; i < 8; ++i) x[j][i] = y[j][i] = s[j][i] = 0.f, c[j][i] = 1.f;
      if (!there) continue;
      const float* src = source(row) + DIM;
      const float* ct = a.cos_t + (size_t)(first_token + row) * a.pairs;
      const float* st = a.sin_t + (size_t)(first_token + row) * a.pairs;
      if constexpr (VEC) {
        load8(src + r0, x[j]);
        if (r0 < 2 * a.pairs) {
          if (a.halves) {
            const bool second = r0 >= a.pairs;
            load8(src + (second ? r0 - a.pairs : r0 + a.pairs), y[j]);
            load8(ct + (second ? r0 - a.pairs : r0), c[j]);
            load8(st + (second ? r0 - a.pairs : r0), s[j]);
          } else {
            const float4 c4 = __ldg(reinterpret_cast<const float4*>(ct + r0 / 2)), s4 = __ldg(reinterpret_cast<const float4*>(st + r0 / 2));
            c[j][0] = c[j][1] = c4.x; c[j][2] = c[j][3] = c4.y; c[j][4] = c[j][5] = c4.z; c[j][6] = c[j][7] = c4.w;
            s[j][0] = s[j][1] = s4.x; s[j][2] = s[j][3] = s4.y; s[j][4] = s[j][5] = s4.z; s[j][6] = s[j][7] = s4.w;
#pragma unroll
            for (int i = 0; i < 8; ++i) y[j][i] = x[j][i ^ 1];
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = r0 + i;
          x[j][i] = __ldg(src + r);
          if (r < 2 * a.pairs) {
            const bool second = a.halves ? r >= a.pairs : r & 1;
            const int pair = a.halves ? (second ? r - a.pairs : r) : r >> 1;
            y[j][i] = __ldg(src + (a.halves ? (second ? r - a.pairs : r + a.pairs) : r ^ 1));
            c[j][i] = __ldg(ct + pair);
            s[j][i] = __ldg(st + pair);
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int idx = base + j * threads, r0 = (idx % TURNED) * 8;
      if (idx < rows * TURNED) {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[j][i] = turned(x[j][i], y[j][i], c[j][i], s[j][i], a.halves ? r0 + i >= a.pairs : i & 1);
        put8(place(idx / TURNED, PLAIN + idx % TURNED), x[j]);
      }
    }
  }
}

__global__ void __launch_bounds__(THREADS, 1)
latent_prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap map_rows, const __grid_constant__ CUtensorMap map_pages,
                              const Args a) {
  extern __shared__ uint8_t lfmha_smem_raw[];
  uint8_t* smem = lfmha_smem_raw + ((1024u - (s32(lfmha_smem_raw) & 1023u)) & 1023u);
  uint8_t* q_t = smem;                                   // [2] Q tiles
  uint8_t* k_t = q_t + 2 * QK_BYTES;                     // [K_STAGES] K tiles
  uint8_t* v_t = k_t + K_STAGES * QK_BYTES;              // the V tile
  uint64_t* k_full = reinterpret_cast<uint64_t*>(v_t + V_BYTES);
  uint64_t* k_empty = k_full + K_STAGES;
  uint64_t* v_full = k_empty + K_STAGES;
  uint64_t* v_empty = v_full + 1;
  uint64_t* s_full = v_empty + 1;                        // [2]: per row tile
  uint64_t* p_ready = s_full + 2;                        // [2]
  uint64_t* o_done = p_ready + 2;                        // [2]
  uint64_t* v_clean = o_done + 2;                        // [2]: V rows without a key of the request are zeroed
  uint64_t* q_full = v_clean + 2;                        // the Q tiles are written (every warp but the producer)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_full + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < K_STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    mbar_init(v_full, 1);
    mbar_init(v_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 4);
      mbar_init(&o_done[i], 1);
      mbar_init(&v_clean[i], 1);
    }
    mbar_init(q_full, THREADS / 32 - 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_rows) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_pages) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  // heads fastest: the work list is sorted by length, and blocks start in the order of their index
  const int item = blockIdx.x / a.heads, head = blockIdx.x % a.heads;
  const int e = a.work[2 * item], bt = a.work[2 * item + 1];
  const int q0 = a.cu_q[e], q_len = a.cu_q[e + 1] - q0, kv_len = a.kv_lens[e], start = kv_len - q_len;
  const int* table = a.block_table + (size_t)e * a.table_stride;
  // Row tile 1 is always there and holds the block's last rows; row tile 0, when the block has two, the 128 before them
  const int r_block = bt * a.tiles_per_block * BR;
  const bool two = a.tiles_per_block == 2 && r_block + BR < q_len;
  const int r_first[2] = {r_block, two ? r_block + BR : r_block};
  const int r_last1 = min(q_len, r_first[1] + BR) - 1;
  const int first_key = a.window > 0 ? max(0, start + r_block - a.window + 1) : 0;
  const int jb0 = first_key / KT * KT;
  const int end1 = start + r_last1 + 1, end0 = two ? start + r_first[1] : 0;
  const int n_tiles1 = (end1 - jb0 + KT - 1) / KT;
  const int n_tiles0 = end0 > jb0 ? (end0 - jb0 + KT - 1) / KT : 0;
  // V tiles with rows that hold no key of this request (beyond its length, before the window)
  const bool dirty_first = jb0 < first_key;
  const bool dirty_last = jb0 + n_tiles1 * KT > kv_len;

  if (warp != 0) {
    // while warp 0 already fetches the first keys
    const int rows = (two ? 2 : 1) * BR, threads = THREADS - 32;
    if (a.q_vec) load_queries<true>(a, s32(q_t), rows, two, q0 + r_block, q_len - r_block, head, threadIdx.x - 32, threads);
    else load_queries<false>(a, s32(q_t), rows, two, q0 + r_block, q_len - r_block, head, threadIdx.x - 32, threads);
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(q_full);
  }

  if (warp == 0) {
    // ---------------- TMA producer (lane 0 and a lane a page box; the warp zeroes dirty V rows) ----------------
    const int ps = a.page_size, box_rows = ps < KT ? ps : KT, boxes = KT / box_rows;
    const int row0 = a.cu_kv[e];
    bool ok = true;
    auto load_k = [&](int t) {
      uint8_t* tile = k_t + (t % K_STAGES) * QK_BYTES;
      uint64_t* full = &k_full[t % K_STAGES];
      const int jb = jb0 + t * KT;
      if (lane == 0) {
        mbar_expect_tx(full, QK_BYTES);
        tma_load_2d(tile, &map_rows, full, head * DIM, row0 + jb);
        tma_load_2d(tile + PANEL, &map_rows, full, head * DIM + 64, row0 + jb);
      }
      __syncwarp();
      if (lane < boxes) {
        const int key = jb + lane * box_rows, pg = key / ps;
        const int page = (pg < a.table_stride && key < kv_len) ? max(table[pg], 0) : 0;
        tma_load_2d(tile + 2 * PANEL + lane * box_rows * 128, &map_pages, full, a.rank, page * ps + key % ps);
      }
    };
    auto load_v = [&](int t) {
      ok = mbar_wait(v_empty, (t & 1) ^ 1, a.err_flag, 67);
      if (!ok) return;
      const int jb = jb0 + t * KT;
      if (lane == 0) {
        mbar_expect_tx(v_full, V_BYTES);
        tma_load_2d(v_t, &map_rows, v_full, a.v_off + head * DV, row0 + jb);
        tma_load_2d(v_t + PANEL, &map_rows, v_full, a.v_off + head * DV + 64, row0 + jb);
      }
      __syncwarp();
      const bool df = dirty_first && t == 0, dl = dirty_last && t == n_tiles1 - 1;
      if (df || dl) {
        ok = mbar_wait(v_full, t & 1, a.err_flag, 69);
        if (!ok) return;
        const int bad_to = df ? first_key - jb : 0;            // rows [0, bad_to) and [bad_from, KT)
        const int bad_from = dl ? max(kv_len - jb, 0) : KT;
        const uint32_t vt = s32(v_t);
        for (int idx = lane; idx < KT * 16; idx += 32) {
          const int row = idx >> 4, c = idx & 15;
          if (row < bad_to || row >= bad_from)
            asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(tile_addr(vt, row, c)), "r"(0) : "memory");
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&v_clean[df ? 0 : 1]);      // each is used once
      }
    };
    for (int t = 0; t < n_tiles1 && ok; ++t) {
      ok = mbar_wait(&k_empty[t % K_STAGES], ((t / K_STAGES) & 1) ^ 1, a.err_flag, 61);
      if (!ok) break;
      load_k(t);
      if (t >= 1) load_v(t - 1);
    }
    if (ok) load_v(n_tiles1 - 1);
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const uint32_t idesc_s = umma_idesc(KT, false), idesc_o = umma_idesc(DV, true);
      bool ok = true;
      auto wait_k = [&](int t) {
        ok = ok && mbar_wait(&k_full[t % K_STAGES], (t / K_STAGES) & 1, a.err_flag, 62);
        fence_after();
      };
      const uint64_t q_desc = umma_desc(s32(q_t), 0, 1024), k_desc = umma_desc(s32(k_t), 0, 1024);
      const uint64_t v_desc = umma_desc(s32(v_t), PANEL, 1024);
      auto issue_s = [&](int i, int t) {            // S_i = Q_i . K_t^T
        if (!ok) return;
        const uint64_t qd = q_desc + (uint64_t)(i * (QK_BYTES >> 4));
        const uint64_t kd = k_desc + (uint64_t)((t % K_STAGES) * (QK_BYTES >> 4));
#pragma unroll
        for (int ks = 0; ks < (DIM + ROT) / 16; ++ks) {
          const uint32_t off = ((ks >> 2) * PANEL + (ks & 3) * 32) >> 4;         // panel, then 32 bytes per k-step
          umma_bf16(tmem + i * 128, qd + off, kd + off, idesc_s, ks != 0);
        }
        umma_commit(&s_full[i]);
      };
      auto issue_pv = [&](int i, int t) {           // O_i += P_i . V_t
        ok = ok && mbar_wait(&p_ready[i], t & 1, a.err_flag, 63);
        if (!ok) return;
        fence_after();
        const uint32_t d = tmem + 256 + i * 128, p = tmem + i * 128;
#pragma unroll
        for (int kk = 0; kk < KT / 16; ++kk)        // 16 keys: 8 columns of P, 2048 bytes of V
          umma_bf16_ts(d, p + kk * 8, v_desc + kk * (2048 >> 4), idesc_o, t != 0 || kk != 0);
        umma_commit(&o_done[i]);
      };
      ok = mbar_wait(q_full, 0, a.err_flag, 71);
      wait_k(0);
      if (n_tiles0 > 0) issue_s(0, 0);
      issue_s(1, 0);
      if (ok) umma_commit(&k_empty[0]);
      for (int t = 0; t < n_tiles1 && ok; ++t) {
        ok = mbar_wait(v_full, t & 1, a.err_flag, 68);
        if (ok && dirty_first && t == 0) ok = mbar_wait(&v_clean[0], 0, a.err_flag, 70);
        else if (ok && dirty_last && t == n_tiles1 - 1) ok = mbar_wait(&v_clean[1], 0, a.err_flag, 70);
        if (!ok) break;
        const bool more = t + 1 < n_tiles1;
        if (t < n_tiles0) issue_pv(0, t);
        if (more) wait_k(t + 1);
        if (t + 1 < n_tiles0) issue_s(0, t + 1);
        issue_pv(1, t);
        if (ok) umma_commit(v_empty);
        if (more) {
          issue_s(1, t + 1);
          if (ok) umma_commit(&k_empty[(t + 1) % K_STAGES]);
        }
      }
    }
    __syncwarp();
  } else {
    // ---------------- softmax: one row per thread, warps 2-5 row tile 0, warps 6-9 row tile 1 ----------------
    const int i = (warp - 2) >> 2;
    const int n_tiles = i ? n_tiles1 : n_tiles0;
    const int ew = warp & 3;
    const int row = ew * 32 + lane;                        // TMEM lane = row of the tile
    const uint32_t lane_addr = (uint32_t)(ew * 32) << 16;
    const uint32_t s_addr = tmem + i * 128 + lane_addr, o_addr = tmem + 256 + i * 128 + lane_addr;
    const int r = r_first[i] + row;
    const int r_end = i ? q_len : r_first[1];              // rows of this tile: [r_first, min(r_first + 128, r_end))
    const int rr = min(r, r_end - 1);
    const int pos = start + rr;
    const int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    // every row of the tile sees all keys of tiles within [lo_max, pos_min]
    const int pos_min = start + r_first[i], pos_max = start + min(r_first[i] + BR, r_end) - 1;
    const int lo_max = a.window > 0 ? max(0, pos_max - a.window + 1) : 0;
    float m_run = -CUDART_INF_F, l_run = 0.f;
    bool ok = true;
    for (int t = 0; t < n_tiles && ok; ++t) {
      const int jb = jb0 + t * KT;
      ok = mbar_wait(&s_full[i], t & 1, a.err_flag, 64);
      if (!ok) break;
      fence_after();
      const bool full = jb >= lo_max && jb + KT - 1 <= pos_min;
      const int k_lo = max(0, lo - jb), k_hi = min(KT, pos - jb + 1);
      Row srow;
      load_row(s_addr, srow);
      const float mx = (full ? row_max<false>(srow, 0, KT) : row_max<true>(srow, k_lo, k_hi)) * a.scale_log2;
      const float m_new = fmaxf(mx, m_run);
      if (t > 0 && __any_sync(0xffffffffu, m_new != m_run)) {
        const float alpha = m_new == m_run ? 1.f : ex2(m_run - m_new);     // m_run = -inf gives 0
        ok = mbar_wait(&o_done[i], (t - 1) & 1, a.err_flag, 65);          // P.V of the tile before is in O
        fence_after();
#pragma unroll 1
        for (int c = 0; c < DV; c += 16) {
          uint32_t v[16];
          tmem_ld16(o_addr + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
          tmem_st16(o_addr + c, v);
        }
      }
      if (m_new != m_run) l_run *= ex2(m_run - m_new);
      m_run = m_new;
      const float base = m_run == -CUDART_INF_F ? 0.f : m_run;
      l_run += full ? row_exp<false, true>(s_addr, srow, a.scale_log2, base, 0, KT)
                    : row_exp<true, true>(s_addr, srow, a.scale_log2, base, k_lo, k_hi);
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[i]);
    }
    if (ok && n_tiles > 0) ok = mbar_wait(&o_done[i], (n_tiles - 1) & 1, a.err_flag, 66);
    fence_after();
    if (n_tiles > 0 && __all_sync(0xffffffffu, ok)) {      // the loads are warp-wide: rows beyond the tile run them too
      const bool mine = r < min(r_first[i] + BR, r_end);
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const float open = a.gate ? 1.f / (1.f + expf(-a.gate[(size_t)(q0 + rr) * a.ld_gate + head])) : 1.f;
      bf16* dst = a.out + ((size_t)(q0 + rr) * a.heads + head) * DV;
      auto done = [&](uint32_t x) { return __uint_as_float(x) * inv * open; };
#pragma unroll 1
      for (int c = 0; c < DV; c += 32) {
        uint32_t v[32];
        tmem_ld32(o_addr + c, v);
        tmem_wait_ld();
        if (mine) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            *reinterpret_cast<uint4*>(dst + c + 8 * q) =
                make_uint4(pack2(done(v[8 * q]), done(v[8 * q + 1])), pack2(done(v[8 * q + 2]), done(v[8 * q + 3])),
                           pack2(done(v[8 * q + 4]), done(v[8 * q + 5])), pack2(done(v[8 * q + 6]), done(v[8 * q + 7])));
        }
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

static bool make_map(CUtensorMap* m, const void* ptr, long long cols, long long rows, long long ld, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace lfmha
}  // namespace srlm

using namespace srlm;

// 1 if srlm_latent_prefill_tcgen05 takes these sizes (a rank whose rotated part starts on 16 bytes; pages that a tile of
// 128 keys holds a whole number of, or that hold a whole number of tiles).
extern "C" int srlm_latent_prefill_tcgen05_takes(int dim, int rot, int dv, int rank, int page_size) {
  return dim == lfmha::DIM && rot == lfmha::ROT && dv == lfmha::DV && rank > 0 && rank % 8 == 0 &&
         (page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64 || (page_size > 0 && page_size % 128 == 0));
}

// q float32, heads x (128 | 64) leading rows of ldq elements, unrotated; cos, sin float32 [tokens, pairs]; pages bfloat16,
// one KV head, rows [latent (rank) | rotated key part (64)]; kv_rows bfloat16 [kv_count, ld_rows]: per row the heads'
// unrotated keys (heads x 128) and, from column v_off, their values (heads x 128); row cu_kv[e] + j holds key j of entry e
// (rows of keys that nobody sees need not exist).  gate: float32 logits, head h of token t at gate[t * ld_gate + h], or null.
extern "C" int srlm_latent_prefill_tcgen05(const float* q, long long ldq, const float* cos_t, const float* sin_t, int pairs,
                                           int halves, const void* pages, long long num_pages, const void* kv_rows,
                                           long long kv_count, long long ld_rows, const int* cu_kv, const float* gate,
                                           long long ld_gate, void* out, const int* block_table, int table_stride,
                                           const int* cu_q, const int* kv_lens, const int* work, int n_work,
                                           int tiles_per_block, int heads, int dim, int rot, int dv, int rank, int v_off,
                                           int page_size, float scale, int window, int* err_flag, cudaStream_t stream) {
  if (n_work <= 0) return ST_OK;
  if (!srlm_latent_prefill_tcgen05_takes(dim, rot, dv, rank, page_size) || heads <= 0 || pairs < 0 || 2 * pairs > rot ||
      (pairs && (!cos_t || !sin_t)) || ldq < (long long)heads * (dim + rot) || tiles_per_block < 1 || tiles_per_block > 2 ||
      kv_count <= 0 || ld_rows % 8 || v_off % 8 || v_off < 0 || ld_rows < v_off + (long long)heads * dv ||
      num_pages * (long long)page_size > 0x7fffffffll || kv_count > 0x7fffffffll)
    return refuse(ST_BAD_SIZE, "latent_prefill_tcgen05: heads=%d dim=%d rot=%d dv=%d rank=%d ld=%lld v_off=%d page_size=%d", heads,
                  dim, rot, dv, rank, ld_rows, v_off, page_size);
  if ((((uintptr_t)pages | (uintptr_t)kv_rows | (uintptr_t)out) & 15) != 0)
    return refuse(ST_BAD_ALIGN, "latent_prefill_tcgen05: pages, rows and output must be 16-byte aligned");
  CUtensorMap rows_map, pages_map;
  if (!lfmha::make_map(&rows_map, kv_rows, ld_rows, kv_count, ld_rows, lfmha::KT) ||
      !lfmha::make_map(&pages_map, pages, rank + rot, num_pages * page_size, rank + rot, page_size < lfmha::KT ? page_size : lfmha::KT))
    return refuse(ST_BAD_SIZE, "latent_prefill_tcgen05: cuTensorMapEncodeTiled refused the operands");
  const cudaError_t e = cudaFuncSetAttribute(lfmha::latent_prefill_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             lfmha::SMEM);
  if (e != cudaSuccess) return refuse((int)e, "latent_prefill_tcgen05: cannot get %d bytes of shared memory", lfmha::SMEM);
  const bool q_vec = ldq % 4 == 0 && pairs % (halves ? 8 : 4) == 0 && (((uintptr_t)q | (uintptr_t)cos_t | (uintptr_t)sin_t) & 15) == 0;
  lfmha::Args a{q, ldq, q_vec, cos_t, sin_t, pairs, halves != 0, gate, ld_gate, (bf16*)out,
                block_table, table_stride, cu_q, kv_lens, cu_kv, work, heads, page_size, rank, v_off, tiles_per_block, window,
                scale * 1.4426950408889634f, err_flag};
  launch_pdl(lfmha::latent_prefill_tcgen05_kernel, dim3(n_work * heads), dim3(lfmha::THREADS), lfmha::SMEM, stream, rows_map,
             pages_map, a);
  return launched();
}
