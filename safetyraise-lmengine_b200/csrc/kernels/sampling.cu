// Sampling over float32 logits [n, V]: greedy argmax (ties go to the lowest id,
// src/frontend/sampling.rs:181-189) and a non-finite check (sampling.rs:97-99).
#include <math_constants.h>

#include "common.cuh"

namespace srlm {

constexpr uint32_t kMaxCluster = 8;

// A row may be shared by the blocks of a thread-block cluster: block `rank` of `nranks` takes the
// elements [lo, hi) of the row, lo a multiple of 4.
struct Slice {
  int lo, hi;
};
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {       // every thread of every block of the cluster
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the 64-bit word at `mine` (an address in this block's shared memory) in block `rank` of the cluster
__device__ __forceinline__ unsigned long long peer_u64(const void* mine, uint32_t rank) {
  uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(mine)), remote;
  unsigned long long v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ Slice slice_of(int V) {
  const int n = (int)cluster_size(), r = (int)cluster_rank();
  const int chunk = ((V + n - 1) / n + 3) & ~3;
  Slice s;
  s.lo = min(V, r * chunk);
  s.hi = min(V, s.lo + chunk);
  return s;
}

// Calls f(i, row[i]) for this thread's share of the elements [sl.lo, sl.hi) of a row, every index once,
// in ascending order per thread.  Rows of a multiple of 4 floats on a 16-byte boundary are read as
// float4, four loads in flight.
template <typename F>
__device__ __forceinline__ void for_each_of_row(const float* __restrict__ row, int V, Slice sl, F f) {
  if ((V & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
    const float4* row4 = reinterpret_cast<const float4*>(row);
    const int n4 = sl.hi >> 2, step = blockDim.x;          // sl.lo and V are multiples of 4, so sl.hi is
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = (sl.lo >> 2) + threadIdx.x; j < n4; j += 4 * step) {
      const bool has1 = j + step < n4, has2 = j + 2 * step < n4, has3 = j + 3 * step < n4;
      const float4 a = row4[j];
      const float4 b = has1 ? row4[j + step] : zero;
      const float4 c = has2 ? row4[j + 2 * step] : zero;
      const float4 d = has3 ? row4[j + 3 * step] : zero;
      f(4 * j, a.x); f(4 * j + 1, a.y); f(4 * j + 2, a.z); f(4 * j + 3, a.w);
      if (has1) { const int i = 4 * (j + step); f(i, b.x); f(i + 1, b.y); f(i + 2, b.z); f(i + 3, b.w); }
      if (has2) { const int i = 4 * (j + 2 * step); f(i, c.x); f(i + 1, c.y); f(i + 2, c.z); f(i + 3, c.w); }
      if (has3) { const int i = 4 * (j + 3 * step); f(i, d.x); f(i + 1, d.y); f(i + 2, d.z); f(i + 3, d.w); }
    }
  } else {
    for (int i = sl.lo + threadIdx.x; i < sl.hi; i += blockDim.x) f(i, row[i]);
  }
}

// larger value first, then the lower id: one 64-bit word whose maximum is the argmax with ties to the
// lowest id
__device__ __forceinline__ uint32_t order_key(float v) {   // larger value -> larger key; -0 counts as +0
  uint32_t b = __float_as_uint(v);
  if (b == 0x80000000u) b = 0u;
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ unsigned long long best_word(float v, int i) {
  return ((unsigned long long)order_key(v) << 32) | (uint32_t)(0x7fffffff - i);
}

// The best (value, id) of the elements [sl.lo, sl.hi) over the block, then over the cluster; the same
// word in every thread of every block.  `slot`: one 64-bit word of shared memory, `warp_best`: 32.
// FLAG: `flag`, which `adjust` may set, becomes whether any thread of the cluster has set it.  It travels as the one bit that
// a word leaves free.
template <bool FLAG, typename F>
__device__ unsigned long long cluster_best(const float* row, int V, Slice sl, unsigned long long* warp_best,
                                           unsigned long long* slot, bool& flag, F adjust) {
  constexpr unsigned long long kFlag = 0x80000000ull;
  auto join = [](unsigned long long a, unsigned long long b) {
    if (!FLAG) return b > a ? b : a;
    const unsigned long long x = a & ~kFlag, y = b & ~kFlag;
    return (y > x ? y : x) | ((a | b) & kFlag);
  };
  unsigned long long best = 0;
  for_each_of_row(row, V, sl, [&](int i, float x) {
    const unsigned long long w = best_word(adjust(i, x), i);
    best = w > best ? w : best;
  });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other > best ? other : best;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (FLAG && __any_sync(0xffffffffu, flag)) best |= kFlag;
  if (lane == 0) warp_best[warp] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long b = 0;
    for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) b = join(b, warp_best[w]);
    *slot = b;
  }
  cluster_sync();
  best = 0;
  for (uint32_t r = 0; r < cluster_size(); ++r) best = join(best, peer_u64(slot, r));
  cluster_sync();                       // nobody rewrites its slot while another block still reads it
  if (FLAG) {
    flag = (best & kFlag) != 0;
    best &= ~kFlag;
  }
  return best;
}

// One cluster of blocks per row.  out_token[row] = argmax; bad[0] set if a logit is not finite.
__global__ void argmax_kernel(const float* __restrict__ logits, long long row_stride, int V,
                              int* __restrict__ out_token, int* __restrict__ bad) {
  __shared__ unsigned long long warp_best[32];
  __shared__ unsigned long long slot;
  const int r = blockIdx.x / cluster_size();
  const float* row = logits + (size_t)r * row_stride;
  bool nonfinite = false;
  const unsigned long long best = cluster_best<false>(row, V, slice_of(V), warp_best, &slot, nonfinite, [&](int, float x) {
    if (!isfinite(x)) nonfinite = true;
    return x;
  });
  if (nonfinite) atomicExch(bad, 1);
  if (cluster_rank() == 0 && threadIdx.x == 0) out_token[r] = best ? 0x7fffffff - (int)(uint32_t)best : 0;
}

}  // namespace srlm

using namespace srlm;

// One cluster of `cluster` blocks per row (1: plain blocks).
template <typename... KArgs, typename... Args>
static void launch_rows(void (*kernel)(KArgs...), int rows, int cluster, int block, size_t smem, cudaStream_t stream,
                        Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows * cluster);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
// Blocks per row: a long row is shared by a cluster of up to 8 (the portable size), each block a slice,
// as long as the clusters of all rows find room on the GPU at once.
// whole_sms: a block fills an SM, and the GPU's clusters of SMs hold 15 clusters of 8 such blocks or 36 of 4 at a time
// (16 rows: 128 us in clusters of 8, which take two rounds, 85 us in clusters of 4, although a quarter of 151,936 values no
// longer fits a block's shared memory beside the bins).  The counts are those of the 148 SMs of a B200.
static int blocks_per_row(int V, int rows, bool whole_sms = false) {
  int c = V >= 32768 ? 8 : V >= 8192 ? 2 : 1;
  while (c > 1 && (rows * c > 148 || (whole_sms && rows > (c == 8 ? 15 : c == 4 ? 36 : 74)))) c >>= 1;
  return c;
}

extern "C" int srlm_argmax(const float* logits, long long row_stride, int n, int V, int* out_token,
                           int* bad_flag, cudaStream_t stream) {
  if (n <= 0) return ST_OK;
  if (V <= 0 || row_stride < V) return refuse(ST_BAD_SIZE, "argmax: V=%d stride=%lld", V, row_stride);
  const int block = V >= 4096 ? 1024 : 256;
  launch_rows(argmax_kernel, n, blocks_per_row(V, n), block, 0, stream, logits, row_stride, V, out_token, bad_flag);
  return launched();
}

// ---------------------------------------------------------------------------
// Temperature / top-k / top-p sampling with a repetition penalty, one block (for a
// long row a cluster of 8 blocks, each with a slice of the row, their sums combined
// through distributed shared memory) per row, in the reference's order of operations (src/frontend/sampling.rs:92-158):
//   penalty -> (temperature == 0: argmax) -> value / temperature -> order by
//   value descending and id ascending -> keep top_k -> softmax over the kept ->
//   keep the shortest prefix whose mass >= top_p -> draw = u * kept mass ->
//   first element whose running mass reaches the draw.
// Nothing is sorted.  The adjusted values are written once to a scratch row; "the
// element at which a running total in sorted order reaches a target" is then found
// by a radix search over the 32 bits of the order key, 8 bits a pass: a pass adds
// the elements that match the prefix found so far into 256 bins, and a scan of the
// bins from the top (by one warp) gives the next 8 bits.  Counts (top-k) and masses are integers
// (a mass is exp(v - max) in units of 2^-31), so the sums do not depend on the
// order of the additions: the same token on every run.  Elements with equal keys
// are ordered by id; a tie on a boundary is resolved by a search over the ids.
// About a dozen passes over the row instead of a hundred; a block's slice of the row lies in shared memory where it fits.
// A top-k of a few hundred ends its search for the boundary at the first digit down to which a list takes all elements: these
// are collected and ordered.  Its first pass counts while the values are adjusted.
// Bound by what a pass costs beside its elements: the bins' copies, their sums, the exchange in the cluster (3 to 4 us).
// 8 rows of 151,936, top-k 50, top-p 0.9, penalty: 154 us with 64-bit additions and the bins scanned by one thread, 85 us
// without either, 40 us with the collected list behind all four digits, 27 us with the list behind the digit (two here) that
// bounds it; without a top-k 114 -> 63 us.
// ---------------------------------------------------------------------------
namespace srlm {

typedef unsigned long long u64;

__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}
// exp(v - vmax) in units of 2^-31: 2^31 for the maximum, 0 below about 2^-31 of it
__device__ __forceinline__ uint32_t mass_of(float v, float vmax) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"((v - vmax) * 1.4426950408889634f));
  return (uint32_t)(e * 2147483648.0f);
}

__device__ __forceinline__ int block_sum_i(int v, int* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  int t = lane < nw ? scratch[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// The kept set: key > kth, or key == kth and id <= id_cut.
struct Kept {
  uint32_t kth;
  int id_cut;
  __device__ __forceinline__ bool has(uint32_t key, int i) const {
    return key > kth || (key == kth && i <= id_cut);
  }
};

constexpr int REPLICAS = 32;          // one copy of the bins per lane: the lanes of a warp never meet
constexpr int REPLICA_STRIDE = 257;   // in bins: the copies of a bin fall on different banks
// A bin's copy is two 32-bit sums, of the masses' lower 16 bits and of the rest (a 64-bit addition in shared memory is a loop
// of compare-and-swap).  A lane adds at most 2^16 elements of a part of a slice, so the lower sums stay below 2^32.
constexpr int COPY_WORDS = REPLICAS * REPLICA_STRIDE;
constexpr int MAX_PART = 32 << 15;

struct Shared {
  u64 bins[256];          // the pass in progress: the sums over the whole row
  u64 mine[2][256];       // ... and over this block's slice (read by the other blocks of the cluster), by turns: a pass
                          // writes one while slower blocks may still read the other
  u64 first[256];         // masses of the kept set by the top 8 bits of the key (reused by both searches)
  u64 found[3];           // digit, sum above it, its own bin
  u64 low_id[256];        // smallest id of this block's slice that fell into each bin (kept for shift == 0)
  u64 low_all[256];       // ... and of the whole row
  u64 word;               // one word for the other blocks to read
  u64 total;
  unsigned long long warp_best[32];
  int is[32];
};

// The sum over the cluster of one integer per block (the same in every thread of every block).
__device__ u64 cluster_sum(u64 mine, Shared& sh) {
  __syncthreads();
  if (threadIdx.x == 0) sh.word = mine;
  cluster_sync();
  u64 sum = 0;
  const uint32_t n = cluster_size();
#pragma unroll
  for (uint32_t r = 0; r < kMaxCluster; ++r) sum += r < n ? peer_u64(&sh.word, r) : 0;
  cluster_sync();
  return sum;
}

// By one warp: the digit, from the top, at which `above + bins` first reaches `target` (0 if none does), the sum above that
// digit, and the digit's own bin.
__device__ __forceinline__ void scan_bins(const u64* bins, u64 above, u64 target, u64* found) {
  const int lane = threadIdx.x;
  u64 b[8], own = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    b[j] = bins[255 - 8 * lane - j];
    own += b[j];
  }
  u64 through = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u64 up = __shfl_up_sync(0xffffffffu, through, o);
    if (lane >= o) through += up;
  }
  const unsigned hits = __ballot_sync(0xffffffffu, above + through >= target);
  if (lane == (hits ? __ffs(hits) - 1 : 31)) {
    u64 acc = above + through - own, bin = b[7];
    int at = 7;
    bool hit = false;
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      if (hit) continue;
      if (acc + b[j] >= target) hit = true, at = j, bin = b[j];
      else acc += b[j];
    }
    found[0] = (u64)(255 - 8 * lane - at);
    found[1] = acc;
    found[2] = bin;
  }
}

// One radix pass: adds `weight(v)` of every element for which `match(key, i)` holds into the bin of its
// digit at `shift`, then scans the bins from the top: the digit at which `above + bins` first reaches
// `target`, the sum above that digit, and the digit's own bin go to sh.found.  The keys of a row share
// few leading digits, so every lane adds into a copy of the bins of its own (`copies`, in dynamic shared
// memory); the copies are summed before the scan.  Integer additions: any order gives the same sums.
// COUNT: every weight is 1.  turn: passes that fill alternate between 0 and 1.  counted: the copies hold the slice's counts.
template <bool COUNT, typename Match, typename Weight>
__device__ __forceinline__ void radix_pass(const float* v, int V, Slice sl, int shift, u64 above, u64 target, int& turn,
                                           Shared& sh, uint32_t* copies, Match match, Weight weight, bool fill, bool counted = false) {
  if (fill) {
    u64* mine = sh.mine[turn];
    turn ^= 1;
    if (shift == 0)
      for (int i = threadIdx.x; i < 256; i += blockDim.x) sh.low_id[i] = 0x7fffffffull;
    uint32_t* lane_copy = copies + (threadIdx.x & (REPLICAS - 1)) * REPLICA_STRIDE;
    for (int lo = sl.lo; lo == sl.lo || lo < sl.hi; lo += MAX_PART) {      // one part, for every vocabulary that there is
      const Slice part{counted ? sl.hi : lo, counted ? sl.hi : min(sl.hi, lo + MAX_PART)};
      if (!counted) {
        for (int i = threadIdx.x; i < (COUNT ? 1 : 2) * COPY_WORDS; i += blockDim.x) copies[i] = 0;
        __syncthreads();
      }
      for_each_of_row(v, V, part, [&](int i, float x) {
        const uint32_t key = order_key(x);
        if (match(key, i)) {
          const uint32_t d = (key >> shift) & 255u;
          if (COUNT) {
            atomicAdd(&lane_copy[d], 1u);
          } else {
            const uint32_t w = weight(x);
            if (w) {
              atomicAdd(&lane_copy[d], w & 0xffffu);
              atomicAdd(&lane_copy[COPY_WORDS + d], w >> 16);
            }
          }
          if (shift == 0) atomicMin(&sh.low_id[d], (u64)i);
        }
      });
      __syncthreads();
      const int d = threadIdx.x >> 2, quarter = threadIdx.x & 3;          // 1024 threads: four a bin, eight copies each
      u64 sum = 0;
#pragma unroll
      for (int c = 0; c < REPLICAS / 4; ++c) {
        const int at = (4 * c + quarter) * REPLICA_STRIDE + d;
        sum += copies[at];
        if (!COUNT) sum += (u64)copies[COPY_WORDS + at] << 16;
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      if (quarter == 0) mine[d] = lo == sl.lo ? sum : mine[d] + sum;
      __syncthreads();
      if (counted) break;
    }
    cluster_sync();                       // every block's slice is in its `mine`
    const uint32_t n = cluster_size();
    for (int d = threadIdx.x; d < 256; d += blockDim.x) {
      u64 sum = 0, low = 0x7fffffffull;
#pragma unroll
      for (uint32_t r = 0; r < kMaxCluster; ++r) {
        if (r >= n) break;
        sum += peer_u64(&mine[d], r);
        if (shift == 0) { const u64 other = peer_u64(&sh.low_id[d], r); low = other < low ? other : low; }
      }
      sh.bins[d] = sum;
      if (shift == 0) sh.low_all[d] = low;
    }
    __syncthreads();
  }
  if (threadIdx.x < 32) scan_bins(sh.bins, above, target, sh.found);
  __syncthreads();
}

// The n-th (1-based) smallest id among the elements of the kept set whose key is `key`.
// `first_id`: the smallest such id if the caller knows it (the last radix pass records it), else -1.
__device__ int nth_holder(const float* v, int V, Slice sl, uint32_t key, const Kept& kept, u64 n, u64 holders,
                          int first_id, Shared& sh) {
  if (n <= 1 && first_id >= 0) return first_id;
  // the smallest and the largest holder: one word per block, (0x7fffffff - smallest) above largest + 1
  unsigned long long best = 0;
  {
    int lo = 0x7fffffff, hi = -1;
    for_each_of_row(v, V, sl, [&](int i, float x) {
      if (order_key(x) == key && kept.has(key, i)) { lo = min(lo, i); hi = max(hi, i); }
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh.warp_best[warp] = ((unsigned long long)(uint32_t)(0x7fffffff - lo) << 32) | (uint32_t)(hi + 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t a = 0, b = 0;
      for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) {
        a = max(a, (uint32_t)(sh.warp_best[w] >> 32));
        b = max(b, (uint32_t)sh.warp_best[w]);
      }
      sh.word = ((unsigned long long)a << 32) | b;
    }
    cluster_sync();
    uint32_t a = 0, b = 0;
    for (uint32_t r = 0; r < cluster_size(); ++r) {
      const unsigned long long w = peer_u64(&sh.word, r);
      a = max(a, (uint32_t)(w >> 32));
      b = max(b, (uint32_t)w);
    }
    cluster_sync();
    best = ((unsigned long long)a << 32) | b;
  }
  int a = 0x7fffffff - (int)(uint32_t)(best >> 32), b = (int)(uint32_t)best - 1;
  if (n <= 1) return a;
  if (n >= holders) return b;
  while (a < b) {                         // smallest id c with #{holders with id <= c} >= n
    const int mid = a + (b - a) / 2;
    int part = 0;
    for_each_of_row(v, V, sl, [&](int i, float x) { part += (i <= mid && order_key(x) == key && kept.has(key, i)); });
    const u64 count = cluster_sum((u64)block_sum_i(part, sh.is), sh);
    if (count >= n) b = mid; else a = mid + 1;
  }
  return a;
}

// The element of the kept set at which the running mass, in the order of key descending and id
// ascending, first reaches `target` (1 <= target <= total mass).  sh.first must hold the kept set's
// masses by the top 8 bits of the key.
__device__ void select_by_mass(const float* v, int V, Slice sl, const Kept& kept, float vmax, u64 target, Shared& sh,
                               uint32_t* copies, int& turn, uint32_t* key_sel, int* id_sel, u64* mass_through) {
  uint32_t prefix = 0;
  u64 above = 0;
  for (int level = 0; level < 4; ++level) {
    const int shift = 24 - 8 * level;
    if (level == 0) {
      for (int i = threadIdx.x; i < 256; i += blockDim.x) sh.bins[i] = sh.first[i];
      __syncthreads();
    }
    const uint32_t pre = prefix;
    radix_pass<false>(v, V, sl, shift, above, target, turn, sh, copies,
                      [&](uint32_t key, int i) { return kept.has(key, i) && (key >> (shift + 8)) == pre; },
                      [&](float x) { return mass_of(x, vmax); }, level != 0);
    prefix = (prefix << 8) | (uint32_t)sh.found[0];
    above = sh.found[1];
  }
  const u64 own = sh.found[2];                         // mass of the elements with this very key
  const int first_id = (int)sh.low_all[prefix & 255u];
  __syncthreads();
  const u64 w = (u64)mass_of(key_value(prefix), vmax);
  const u64 holders = w ? own / w : 1;
  u64 need = w ? (target > above ? (target - above + w - 1) / w : 1) : 1;
  if (need < 1) need = 1;
  if (need > holders) need = holders;
  *key_sel = prefix;
  *id_sel = nth_holder(v, V, sl, prefix, kept, need, holders, first_id == 0x7fffffff ? -1 : first_id, sh);
  *mass_through = above + need * w;
}

// The choice among few elements (top-k of at most kList; `kept`: those k, or at most kList with them among these): block 0 of the
// cluster collects them, orders them by key descending and id ascending, and reads the cutoff and the draw off the running
// masses of the first k: the element that the searches above would find.  -> its id in block 0's thread 0, -1 where no kept element has a mass (the adjusted maximum is not a finite
// number); the other blocks return at once.  lists: 3 * kList words of shared memory, at the same place in every block.
constexpr int kList = 512;
__device__ int select_from_list(const float* v, int V, Slice sl, const Kept& kept, int k, float vmax, float tp, float uniform,
                                Shared& sh, u64* lists) {
  u64 *own = lists, *all = lists + kList, *sorted = lists + 2 * kList;
  __syncthreads();
  if (threadIdx.x == 0) sh.is[0] = 0;
  __syncthreads();
  for_each_of_row(v, V, sl, [&](int i, float x) {
    const uint32_t key = order_key(x);
    if (kept.has(key, i)) {
      const int at = atomicAdd(&sh.is[0], 1);
      if (at < kList) own[at] = ((u64)key << 32) | (uint32_t)(0x7fffffff - i);
    }
  });
  __syncthreads();
  if (threadIdx.x == 0) sh.word = (u64)min(sh.is[0], kList);
  cluster_sync();
  int n = 0;
  if (cluster_rank() == 0) {
    for (uint32_t r = 0; r < cluster_size(); ++r) {
      const int count = min((int)peer_u64(&sh.word, r), kList - n);
      for (int j = threadIdx.x; j < count; j += blockDim.x) all[n + j] = peer_u64(&own[j], r);
      n += count;
    }
  }
  cluster_sync();
  if (cluster_rank() != 0) return 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const u64 mine = all[i];
    int before = 0;
    for (int j = 0; j < n; ++j) before += all[j] > mine;
    sorted[before] = mine;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return 0;
  n = min(n, k);
  const int lane = threadIdx.x, per = (n + 31) / 32, lo = min(n, lane * per), hi = min(n, lo + per);
  auto mass = [&](int i) { return (u64)mass_of(key_value((uint32_t)(sorted[i] >> 32)), vmax); };
  u64 own_mass = 0;
  for (int i = lo; i < hi; ++i) own_mass += mass(i);
  u64 through = own_mass;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u64 up = __shfl_up_sync(0xffffffffu, through, o);
    if (lane >= o) through += up;
  }
  const u64 total = __shfl_sync(0xffffffffu, through, 31);
  if (total == 0) return -1;
  // the first element whose running mass reaches `target` (1 .. total), and that mass
  auto reach = [&](u64 target, u64* mass_through) {
    const int lane_of = __ffs(__ballot_sync(0xffffffffu, through >= target)) - 1;
    u64 acc = through - own_mass;
    int at = lo;
    if (lane == lane_of)
      for (; at < hi; ++at) {
        acc += mass(at);
        if (acc >= target) break;
      }
    *mass_through = __shfl_sync(0xffffffffu, acc, lane_of);
    return __shfl_sync(0xffffffffu, at, lane_of);
  };
  u64 kept_mass = total, unused;
  int cut = n - 1;
  if (tp < 1.f) {
    u64 target = (u64)ceil((double)tp * (double)total);
    target = target < 1 ? 1 : (target > total ? total : target);
    cut = reach(target, &kept_mass);
  }
  u64 draw = (u64)ceil((double)uniform * (double)kept_mass);
  draw = draw < 1 ? 1 : (draw > kept_mass ? kept_mass : draw);
  return 0x7fffffff - (int)(uint32_t)sorted[min(reach(draw, &unused), cut)];
}

// One block per row.  hist_offsets[row]..hist_offsets[row+1] index `history` (ids for the penalty).
// scratch: one row of V floats per row of logits.
__global__ void __launch_bounds__(1024)
sample_kernel(const float* __restrict__ logits, long long row_stride, int V,
              const float* __restrict__ temperature, const int* __restrict__ top_k,
              const float* __restrict__ top_p, const float* __restrict__ penalty,
              const float* __restrict__ uniform, const int* __restrict__ history,
              const int* __restrict__ hist_offsets, float* __restrict__ scratch, int slice_room,
              int* __restrict__ out_token, int* __restrict__ bad) {
  extern __shared__ __align__(16) float dyn_smem[];  // [the slice's adjusted values], the copies of the bins, the penalty's bitmap
  __shared__ Shared sh;
  const int r = blockIdx.x / cluster_size();
  const Slice sl = slice_of(V);
  const float* row = logits + (size_t)r * row_stride;
  // the adjusted values: in shared memory where the slice fits, else in the scratch row.  (Indexed like the row; slices
  // begin on a multiple of 4, so a slice in shared memory keeps the row's alignment of 16 bytes.)
  float* v = slice_room ? dyn_smem - sl.lo : scratch + (size_t)r * V;
  uint32_t* copies = reinterpret_cast<uint32_t*>(dyn_smem + slice_room);
  uint32_t* seen_bits = copies + 2 * COPY_WORDS;                                   // ceil(V / 32) words
  int turn = 0;
  const float temp = temperature[r];
  const float pen = penalty ? penalty[r] : 1.f;
  const bool use_pen = pen != 1.f && history;
  if (use_pen) {
    const int words = (V + 31) >> 5;
    for (int i = threadIdx.x; i < words; i += blockDim.x) seen_bits[i] = 0u;
    __syncthreads();
    for (int i = hist_offsets[r] + threadIdx.x; i < hist_offsets[r + 1]; i += blockDim.x) {
      const int tok = history[i];
      if (tok >= 0 && tok < V) atomicOr(&seen_bits[tok >> 5], 1u << (tok & 31));
    }
    __syncthreads();
  }
  // the adjusted values, once (each block its slice); their argmax (ties to the lowest id) and the
  // non-finite check, over the whole row
  // and, for a top-k, the counts of the first pass of its search
  const int k = top_k ? top_k[r] : 0;
  const bool cuts = k > 0 && k < V && temp > 0.f;
  uint32_t* lane_copy = copies + (threadIdx.x & (REPLICAS - 1)) * REPLICA_STRIDE;
  if (cuts) {
    for (int i = threadIdx.x; i < COPY_WORDS; i += blockDim.x) copies[i] = 0;
    __syncthreads();
  }
  bool nonfinite = false;
  const unsigned long long best = cluster_best<true>(row, V, sl, sh.warp_best, &sh.word, nonfinite, [&](int i, float x) {
    if (!isfinite(x)) nonfinite = true;
    if (use_pen && (seen_bits[i >> 5] >> (i & 31) & 1u)) x = x < 0.f ? x * pen : x / pen;
    if (temp > 0.f) x = x / temp;
    v[i] = x;
    if (cuts) atomicAdd(&lane_copy[order_key(x) >> 24], 1u);
    return x;
  });
  const float bv = key_value((uint32_t)(best >> 32));
  const int bi = best ? 0x7fffffff - (int)(uint32_t)best : 0;
  const bool writer = cluster_rank() == 0 && threadIdx.x == 0;
  // the decision is the same in every block of the cluster: they meet again at every pass
  if (nonfinite || !(temp > 0.f)) {
    if (writer) {
      if (nonfinite) atomicExch(bad, 1);
      out_token[r] = bi;
    }
    return;
  }
  // top-k: the k-th largest key, and the id cut among the elements equal to it
  Kept kept{0u, 0x7fffffff};
  if (cuts) {
    uint32_t prefix = 0;
    u64 above = 0;
    bool few = false;                   // no more elements down to the boundary's digit than a list takes: it is ordered whole
    for (int level = 0; level < 4 && !few; ++level) {
      const int shift = 24 - 8 * level;
      const uint32_t pre = prefix;
      radix_pass<true>(v, V, sl, shift, above, (u64)k, turn, sh, copies,
                       [&](uint32_t key, int) { return (key >> (shift + 8)) == pre; },
                       [](float) { return 1u; }, true, level == 0);
      prefix = (prefix << 8) | (uint32_t)sh.found[0];
      above = sh.found[1];
      few = k <= kList && above + sh.found[2] <= (u64)kList;
      kept.kth = prefix << shift;
    }
    const u64 ties = sh.found[2];
    const int first_id = (int)sh.low_all[prefix & 255u];
    __syncthreads();
    if (!few && above + ties > (u64)k)     // a tie on the boundary: keep the lowest ids among the equal
      kept.id_cut = nth_holder(v, V, sl, prefix, Kept{0u, 0x7fffffff}, (u64)k - above, ties,
                               first_id == 0x7fffffff ? -1 : first_id, sh);
  }
  if (cuts && k <= kList) {
    const int id = select_from_list(v, V, sl, kept, k, bv, top_p[r], uniform[r], sh, reinterpret_cast<u64*>(copies));
    if (writer) {
      if (id < 0) atomicExch(bad, 1);
      out_token[r] = id < 0 ? bi : id;
    }
    return;
  }
  // the kept set's masses by the top 8 bits of the key; their sum is the softmax denominator
  radix_pass<false>(v, V, sl, 24, 0, ~(u64)0, turn, sh, copies, [&](uint32_t key, int i) { return kept.has(key, i); },
                    [&](float x) { return mass_of(x, bv); }, true);
  for (int i = threadIdx.x; i < 256; i += blockDim.x) sh.first[i] = sh.bins[i];
  if (threadIdx.x == 0) sh.total = sh.found[1] + sh.found[2];      // no bin reaches the target: all above bin 0, and bin 0
  __syncthreads();
  const u64 total = sh.total;
  if (total == 0) {                       // the same in every block: the bins hold the whole row
    if (writer) { atomicExch(bad, 1); out_token[r] = bi; }
    cluster_sync();                     // no block leaves while another reads its shared memory
    return;
  }
  // top-p cutoff: the shortest prefix whose mass >= top_p
  const float tp = top_p[r];
  uint32_t key_cut = 0;
  int id_cut = 0x7fffffff;
  u64 kept_mass = total;
  if (tp < 1.f) {
    u64 target = (u64)ceil((double)tp * (double)total);
    target = target < 1 ? 1 : (target > total ? total : target);
    select_by_mass(v, V, sl, kept, bv, target, sh, copies, turn, &key_cut, &id_cut, &kept_mass);
  }
  // the draw
  u64 draw = (u64)ceil((double)uniform[r] * (double)kept_mass);
  draw = draw < 1 ? 1 : (draw > kept_mass ? kept_mass : draw);
  uint32_t key_sel;
  int id_sel;
  u64 through;
  select_by_mass(v, V, sl, kept, bv, draw, sh, copies, turn, &key_sel, &id_sel, &through);
  // never beyond the cutoff element (the reference falls back to the last kept element)
  if (key_sel < key_cut || (key_sel == key_cut && id_sel > id_cut)) id_sel = id_cut;
  if (writer) out_token[r] = id_sel;
  cluster_sync();                       // no block leaves while another reads its shared memory
}

}  // namespace srlm

// scratch: n rows of V floats that the kernel may overwrite.
extern "C" int srlm_sample(const float* logits, long long row_stride, int n, int V, const float* temperature,
                           const int* top_k, const float* top_p, const float* penalty, const float* uniform,
                           const int* history, const int* hist_offsets, float* scratch, int* out_token,
                           int* bad_flag, cudaStream_t stream) {
  if (n <= 0) return ST_OK;
  if (V <= 0 || row_stride < V) return refuse(ST_BAD_SIZE, "sample: V=%d stride=%lld", V, row_stride);
  if (!scratch) return refuse(ST_BAD_SIZE, "sample: a scratch row of V floats per row of logits is needed");
  const int cluster = blocks_per_row(V, n, true);
  const int slice = ((V + cluster - 1) / cluster + 3) & ~3;
  const size_t fixed = (size_t)2 * COPY_WORDS * 4 + (history ? (size_t)((V + 31) / 32) * 4 : 0);
  if (fixed > 190 * 1024) return refuse(ST_BAD_SIZE, "sample: vocabulary %d is too large for the penalty bitmap", V);
  const int room = fixed + (size_t)slice * 4 <= 190 * 1024 ? slice : 0;
  const size_t smem = fixed + (size_t)room * 4;
  const cudaError_t e = cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 190 * 1024);
  if (e != cudaSuccess) return refuse((int)e, "sample: cannot get 190 KB of shared memory");
  launch_rows(sample_kernel, n, cluster, 1024, smem, stream, logits, row_stride, V, temperature, top_k, top_p,
              penalty, uniform, history, hist_offsets, scratch, room, out_token, bad_flag);
  return launched();
}
