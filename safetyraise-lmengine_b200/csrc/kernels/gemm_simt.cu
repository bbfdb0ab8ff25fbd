// C[M,N] = A[M,K] . W[N,K]^T with float32 FMA accumulation (no tensor cores,
// no reduced-precision mode).  Every output element is one chain of FMAs over k
// in the order 0..K-1 whatever M, N and the tile are, so a row's result does not
// depend on the batch, bit for bit.  This is the matrix product of the float32
// path and the reference twin of the tensor-core GEMM.  Formula:
// src/artifact/mod.rs:377-405.
//
// Two forms, with the same sums:
//  * tiles: a block forms BM x BN outputs from slabs of 32 k's, small tiles and large ones each in a form of their own.
//    Bound by the FMA pipes; the tile is chosen by size (see `pick_tile`).
//  * few rows (M <= 16, see `few_rows`): a warp streams 8 weight rows through a ring of its own, a lane owns up to four outputs.  Bound by
//    the chain of K dependent FMAs (4 cycles each) for small weights (8 x 4,096 x 4,096: 33 us, 195 in tiles), by memory for
//    large ones (1 x 24,576 x 4,096: 85 us, 484 in tiles).
#include <algorithm>

#include "common.cuh"

namespace srlm {

constexpr int BK = 32, KLD = BK + 4;      // rows of a slab lie an odd number of 16-byte pieces apart: neighbouring rows'
constexpr int STAGES = 3;                 // 16-byte reads share no bank

__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {     // not valid: zeros, nothing is read
  const unsigned int at = (unsigned int)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_committed() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copies_waited() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// ROWS x BK elements of a matrix, rows of a slab KLD apart; what lies outside the matrix is zero.
template <typename T, int ROWS, int THREADS>
struct Slab {
  static constexpr int PIECES = ROWS * (BK / 4) / THREADS;
  static_assert(ROWS * (BK / 4) % THREADS == 0, "");
  float4 v[PIECES];
  static __device__ __forceinline__ void copy(float* dst, const T* src, long long ld, int row0, int rows, int k0, int K, int tid) {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int idx = tid + p * THREADS, r = idx / (BK / 4), c = (idx % (BK / 4)) * 4;
      const bool valid = row0 + r < rows && k0 + c < K;
      copy16(dst + r * KLD + c, reinterpret_cast<const float*>(valid ? src + (size_t)(row0 + r) * ld + k0 + c : src), valid);
    }
  }
  __device__ __forceinline__ void load(const T* __restrict__ src, long long ld, int row0, int rows, int k0, int K, int tid) {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int idx = tid + p * THREADS, r = row0 + idx / (BK / 4), k = k0 + (idx % (BK / 4)) * 4;
      v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && k < K) {
        const T* at = src + (size_t)r * ld + k;
        v[p].x = to_float(at[0]);
        if (k + 1 < K) v[p].y = to_float(at[1]);
        if (k + 2 < K) v[p].z = to_float(at[2]);
        if (k + 3 < K) v[p].w = to_float(at[3]);
      }
    }
  }
  __device__ __forceinline__ void store(float* dst, int tid) const {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int idx = tid + p * THREADS;
      *reinterpret_cast<float4*>(dst + idx / (BK / 4) * KLD + (idx % (BK / 4)) * 4) = v[p];
    }
  }
};

// A lane's place in a warp's 4 x 8 threads: lanes i and i ^ 1 read the same row of W, i and i ^ 2 the same row of A.
__device__ __forceinline__ int lane_row(int lane) { return (lane & 1) | (lane >> 2 & 2); }
__device__ __forceinline__ int lane_col(int lane) { return (lane >> 1 & 3) | (lane >> 2 & 4); }

// Small tiles, for sizes whose large tiles leave SMs idle: slabs lie row by row, as asynchronous copies bring them, and four to eight
// warps an SM quarter hide the reads.  (32 x 32 outputs in the layout above: 305 x 1,024 x 3,072 in 124 us, 83 here.)
// A thread forms TM x TN outputs, rows BM / TM and columns BN / TN apart.  VEC: float32 rows of whole 16-byte pieces.
template <typename TA, typename TW, typename TO, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_tn_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TO* __restrict__ C, int M, int N,
                    int K, long long lda, long long ldw, long long ldc) {
  constexpr int THREADS = (BM / TM) * (BN / TN), DM = BM / TM, DN = BN / TN, RING = VEC ? STAGES : 2;
  // the body of the loop over k stays below 256 FMAs: unrolled over the whole slab (2,048 FMAs, 34 KB of code) a warp waited
  // for instructions 0.7 cycles an instruction
  constexpr int WHOLE = 256 / (4 * TM * TN), PIECES_A_TURN = WHOLE < 1 ? 1 : WHOLE > BK / 4 ? BK / 4 : WHOLE;
  extern __shared__ __align__(16) float slabs[];             // RING x (BM rows of A, BN rows of W) x KLD
  static_assert(DM % 4 == 0 && DN % 8 == 0, "");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = warp / (DN / 8) * 4 + lane_row(lane), tn = warp % (DN / 8) * 8 + lane_col(lane);
  float acc[TM][TN] = {};
  Slab<TA, BM, THREADS> a_slab;
  Slab<TW, BN, THREADS> w_slab;
  const int steps = (K + BK - 1) / BK;
  auto place = [&](int s) { return slabs + (s % RING) * (BM + BN) * KLD; };
  auto fetch = [&](int s) {
    if (s < steps) {
      Slab<TA, BM, THREADS>::copy(place(s), A, lda, m0, M, s * BK, K, tid);
      Slab<TW, BN, THREADS>::copy(place(s) + BM * KLD, W, ldw, n0, N, s * BK, K, tid);
    }
    copies_committed();
  };
  if constexpr (VEC) {
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
  } else {
    a_slab.load(A, lda, m0, M, 0, K, tid);
    w_slab.load(W, ldw, n0, N, 0, K, tid);
  }
  for (int s = 0; s < steps; ++s) {
    if constexpr (VEC) {
      copies_waited<STAGES - 2>();
      __syncthreads();                                       // slab s is here; everyone has left slab s - 1
      fetch(s + STAGES - 1);
    } else {
      a_slab.store(place(s), tid);                           // (two slabs back, which everyone has left)
      w_slab.store(place(s) + BM * KLD, tid);
      __syncthreads();
      if (s + 1 < steps) {
        a_slab.load(A, lda, m0, M, (s + 1) * BK, K, tid);
        w_slab.load(W, ldw, n0, N, (s + 1) * BK, K, tid);
      }
    }
    const float* as = place(s) + tm * KLD;
    const float* ws = place(s) + (BM + tn) * KLD;
#pragma unroll PIECES_A_TURN
    for (int k = 0; k < BK; k += 4) {
      float4 a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * DM * KLD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + j * DN * KLD + k);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j)
            acc[i][j] = fmaf(e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w,
                             e == 0 ? w[j].x : e == 1 ? w[j].y : e == 2 ? w[j].z : w[j].w, acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + tm + i * DM;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tn + j * DN;
      if (n < N) C[(size_t)m * ldc + n] = from_float<TO>(acc[i][j]);
    }
  }
}

// ROWS x BK elements of a matrix on their way to shared memory, where they lie k by k: four rows a 16-byte piece, four floats of
// padding behind four k's, so that a warp's stores (4 rows by 32 k's) and reads (neighbouring fours of one k) share no bank.
// What lies outside the matrix is zero.
template <typename T, int ROWS, int THREADS, bool VEC>
struct KSlab {
  static constexpr int PIECES = ROWS * (BK / 4) / THREADS, GROUP = 4 * ROWS + 4, FLOATS = BK / 4 * GROUP;
  static_assert(ROWS * (BK / 4) % THREADS == 0, "");
  float4 v[PIECES];
  __device__ __forceinline__ void load(const T* __restrict__ src, long long ld, int row0, int rows, int k0, int K, int tid) {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int idx = tid + p * THREADS, r = row0 + idx / (BK / 4), k = k0 + (idx % (BK / 4)) * 4;
      v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && k < K) {
        const T* at = src + (size_t)r * ld + k;
        if constexpr (VEC) {
          v[p] = *reinterpret_cast<const float4*>(at);
        } else {
          v[p].x = to_float(at[0]);
          if (k + 1 < K) v[p].y = to_float(at[1]);
          if (k + 2 < K) v[p].z = to_float(at[2]);
          if (k + 3 < K) v[p].w = to_float(at[3]);
        }
      }
    }
  }
  __device__ __forceinline__ void store(float* dst, int tid) const {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int idx = tid + p * THREADS, r = idx / (BK / 4), c = idx % (BK / 4);
      float* at = dst + c * GROUP + r;
      at[0] = v[p].x;
      at[ROWS] = v[p].y;
      at[2 * ROWS] = v[p].z;
      at[3 * ROWS] = v[p].w;
    }
  }
};

// Large tiles.  Slabs lie k by k, so that a read brings four rows of one k and two columns are one packed FMA (the same two sums,
// half the instructions: a warp an SM quarter then issues its reads between the FMAs instead of before them).  Bound by
// the FMA pipes, 70 % busy for 2,048 x 6,144 x 4,096: 1.99 ms where a tile of the form below took 2.26; with single FMAs 2.32.
// A thread forms TM x TN outputs: rows in fours BM / TM fours apart, columns in fours BN / TN fours apart.  VEC: float32 rows of
// whole 16-byte pieces.
template <typename TA, typename TW, typename TO, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_tn_pairs_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TO* __restrict__ C, int M, int N,
                    int K, long long lda, long long ldw, long long ldc) {
  constexpr int THREADS = (BM / TM) * (BN / TN), DM = BM / TM, DN = BN / TN, PIECES = BK / 4;
  extern __shared__ __align__(16) float slabs[];             // 2 x (a slab of A, one of W)
  static_assert(DM % 4 == 0 && DN % 8 == 0 && TM % 4 == 0 && TN % 4 == 0, "");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = warp / (DN / 8) * 4 + lane_row(lane), tn = warp % (DN / 8) * 8 + lane_col(lane);
  float2 acc[TM][TN / 2] = {};
  typedef KSlab<TA, BM, THREADS, VEC> SlabA;
  typedef KSlab<TW, BN, THREADS, VEC> SlabW;
  SlabA a_slab;
  SlabW w_slab;
  const int steps = (K + BK - 1) / BK;
  auto place = [&](int s) { return slabs + (s & 1) * (SlabA::FLOATS + SlabW::FLOATS); };
  auto load = [&](int s) {
    a_slab.load(A, lda, m0, M, s * BK, K, tid);
    w_slab.load(W, ldw, n0, N, s * BK, K, tid);
  };
  auto store = [&](int s) {
    a_slab.store(place(s), tid);
    w_slab.store(place(s) + SlabA::FLOATS, tid);
  };
  float4 a[2][TM / 4], w[2][TN / 4];
  auto read = [&](int set, const float* ap, const float* wp, int k) {
#pragma unroll
    for (int i = 0; i < TM / 4; ++i) a[set][i] = *reinterpret_cast<const float4*>(ap + k * BM + 4 * i * DM);
#pragma unroll
    for (int j = 0; j < TN / 4; ++j) w[set][j] = *reinterpret_cast<const float4*>(wp + k * BN + 4 * j * DN);
  };
  auto multiply = [&](int set) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const float4 x = a[set][i / 4];
      const float xi = i % 4 == 0 ? x.x : i % 4 == 1 ? x.y : i % 4 == 2 ? x.z : x.w;
      const float2 xx = make_float2(xi, xi);
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        const float4 y = w[set][j / 2];
        acc[i][j] = fma2(xx, j % 2 ? make_float2(y.z, y.w) : make_float2(y.x, y.y), acc[i][j]);
      }
    }
  };
  load(0);
  store(0);
  if (steps > 1) load(1);
  __syncthreads();
  auto a_at = [&](int s) { return place(s) + 4 * tm; };
  auto w_at = [&](int s) { return place(s) + SlabA::FLOATS + 4 * tn; };
  const float *ap = a_at(0), *wp = w_at(0);
  read(0, ap, wp, 0);
  for (int s = 0; s < steps; ++s) {
#pragma unroll 1
    for (int c = 0; c < PIECES; ++c) {
      read(1, ap, wp, 1);
      multiply(0);
      read(0, ap, wp, 2);
      multiply(1);
      read(1, ap, wp, 3);
      multiply(0);
      ap += SlabA::GROUP;
      wp += SlabW::GROUP;
      if (c == PIECES / 2 && s + 1 < steps) {                // (everyone has left slab s - 1, which lay there)
        store(s + 1);
        if (s + 2 < steps) load(s + 2);
      }
      if (c == PIECES - 1) {
        __syncthreads();                                     // slab s + 1 is here; everyone has read slab s
        ap = a_at(s + 1);
        wp = w_at(s + 1);
      }
      read(0, ap, wp, 0);                                    // (behind the last slab: numbers that nobody uses)
      multiply(1);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + 4 * (tm + i / 4 * DM) + i % 4;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + 4 * (tn + j / 4 * DN) + j % 4;
      if (n < N) C[(size_t)m * ldc + n] = from_float<TO>(j % 2 ? acc[i][j / 2].y : acc[i][j / 2].x);
    }
  }
}

// ---- few rows -----------------------------------------------------------------------------------------------------
constexpr int FEW_M = 16, FEW_N = 8, FEW_K = 128, FEW_STAGES = 4;
constexpr int FEW_LD = FEW_K + 4;

template <int MINE>                       // rows of A a lane multiplies with its weight row: M <= 4 * MINE
__global__ void __launch_bounds__(32)
gemm_tn_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                   long long lda, long long ldw, long long ldc) {
  extern __shared__ __align__(16) float few_sh[];          // FEW_STAGES x (FEW_N weight rows, then 4 * MINE rows of A) x FEW_LD
  constexpr int STAGE = (FEW_N + 4 * MINE) * FEW_LD;
  const int lane = threadIdx.x, n0 = blockIdx.x * FEW_N;
  const int slabs = (K + FEW_K - 1) / FEW_K;
  auto fetch = [&](int s) {
    if (s < slabs) {
      float* dst = few_sh + (s % FEW_STAGES) * STAGE + 4 * lane;
      const int k = s * FEW_K + 4 * lane;                  // a row of a slab is one piece a lane
#pragma unroll
      for (int r = 0; r < FEW_N; ++r) {
        const bool valid = k < K && n0 + r < N;
        copy16(dst + r * FEW_LD, valid ? W + (size_t)(n0 + r) * ldw + k : W, valid);
      }
#pragma unroll
      for (int r = 0; r < 4 * MINE; ++r) {
        const bool valid = k < K && r < M;
        copy16(dst + (FEW_N + r) * FEW_LD, valid ? A + (size_t)r * lda + k : A, valid);
      }
    }
    copies_committed();
  };
#pragma unroll
  for (int s = 0; s < FEW_STAGES - 1; ++s) fetch(s);
  const int n = lane_col(lane), m = lane_row(lane);
  float acc[MINE] = {};
  for (int s = 0; s < slabs; ++s) {
    copies_waited<FEW_STAGES - 2>();
    __syncwarp();                                          // slab s has arrived; every lane has left slab s - 1
    fetch(s + FEW_STAGES - 1);
    const float* w = few_sh + (s % FEW_STAGES) * STAGE + n * FEW_LD;
    const float* a = few_sh + (s % FEW_STAGES) * STAGE + (FEW_N + m) * FEW_LD;
    constexpr int AHEAD = 4;                               // 16-byte pieces read ahead of the chains of FMAs
    float4 y[2][AHEAD], x[2][AHEAD][MINE];
    auto read = [&](int g) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        y[g & 1][i] = *reinterpret_cast<const float4*>(w + 4 * (g * AHEAD + i));
#pragma unroll
        for (int j = 0; j < MINE; ++j)
          x[g & 1][i][j] = *reinterpret_cast<const float4*>(a + 4 * j * FEW_LD + 4 * (g * AHEAD + i));
      }
    };
    read(0);
#pragma unroll 2
    for (int g = 0; g < FEW_K / 4 / AHEAD; ++g) {
      if (g + 1 < FEW_K / 4 / AHEAD) read(g + 1);
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
#pragma unroll
        for (int j = 0; j < MINE; ++j) acc[j] = fmaf(x[g & 1][i][j].x, y[g & 1][i].x, acc[j]);
#pragma unroll
        for (int j = 0; j < MINE; ++j) acc[j] = fmaf(x[g & 1][i][j].y, y[g & 1][i].y, acc[j]);
#pragma unroll
        for (int j = 0; j < MINE; ++j) acc[j] = fmaf(x[g & 1][i][j].z, y[g & 1][i].z, acc[j]);
#pragma unroll
        for (int j = 0; j < MINE; ++j) acc[j] = fmaf(x[g & 1][i][j].w, y[g & 1][i].w, acc[j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < MINE; ++j)
    if (m + 4 * j < M && n0 + n < N) C[(size_t)(m + 4 * j) * ldc + n0 + n] = acc[j];
}

template <int MINE>
static int run_few(const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldw, long long ldc,
                   cudaStream_t stream) {
  constexpr int smem = (int)sizeof(float) * FEW_STAGES * (FEW_N + 4 * MINE) * FEW_LD;
  if constexpr (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_tn_few_kernel<MINE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
  }
  gemm_tn_few_kernel<MINE><<<(N + FEW_N - 1) / FEW_N, 32, smem, stream>>>((const float*)A, (const float*)W, (float*)C, M, N, K,
                                                                        lda, ldw, ldc);
  return launched();
}

// ---- dispatch -----------------------------------------------------------------------------------------------------
template <typename TA, typename TW, typename TO, int BM, int BN, int TM, int TN>
static int run_tile(const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldw,
                    long long ldc, bool vec, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  constexpr int threads = (BM / TM) * (BN / TN);
  auto go = [&](auto kernel, int floats) {
    const int smem = (int)sizeof(float) * floats;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    kernel<<<grid, threads, smem, stream>>>((const TA*)A, (const TW*)W, (TO*)C, M, N, K, lda, ldw, ldc);
    return launched();
  };
  constexpr bool f32 = sizeof(TA) == 4 && sizeof(TW) == 4;
  if constexpr (BM >= 64) {
    constexpr int floats = 2 * (KSlab<TA, BM, threads, false>::FLOATS + KSlab<TW, BN, threads, false>::FLOATS);
    if constexpr (f32) {
      if (vec) return go(gemm_tn_pairs_kernel<TA, TW, TO, BM, BN, TM, TN, true>, floats);
    }
    if constexpr (BN > 64) return refuse(ST_BAD_SIZE, "gemm_tn_simt: a tile of %d columns takes whole pieces", BN);
    else return go(gemm_tn_pairs_kernel<TA, TW, TO, BM, BN, TM, TN, false>, floats);
  } else {
    if constexpr (f32) {
      if (vec) return go(gemm_tn_simt_kernel<TA, TW, TO, BM, BN, TM, TN, true>, STAGES * (BM + BN) * KLD);
    }
    return go(gemm_tn_simt_kernel<TA, TW, TO, BM, BN, TM, TN, false>, 2 * (BM + BN) * KLD);
  }
}

static int device_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return n > 0 ? n : 148;
}

// The tile whose blocks cost least.  `cycles`: what an SM spends on a k of one block where few blocks share it, measured; large
// tiles reuse what they read, small ones leave no SM idle (a block of 64 x 128 alone on its SM takes 112).  us in tiles of
// 64 x 128, 64 x 64, 32 x 64, 32 x 32: 2,048 x 6,144 x 4,096 1,984, 2,101, 2,537, 2,710; 305 x 6,144 x 1,024 98.7, 110, 114,
// 111; 500 x 1,024 x 2,048 108, 73.8, 78.9, 71.0; 305 x 1,024 x 3,072 160, 109, 116, 82.  Rows that are no whole 16-byte pieces
// (not `vec`) are fetched number by number, which blocks beside each other hide: `first` is the time of blocks that have an SM
// each, `each` what one more costs (us at 1,001 k; 300 x 8,192 in the last three tiles: 149, 173, 204; 24 x 8,192: 47, 34, 31;
// in 64 x 128, which is then not taken, 160 and 65).
static int pick_tile(int M, int N, bool vec) {
  struct Tile { int bm, bn, cycles, first, each; };
  static const Tile tiles[] = {{64, 128, 100, 0, 0}, {64, 64, 62, 46, 34}, {32, 64, 37, 31, 21}, {32, 32, 18, 21, 12}};
  const int sms = device_sms();
  int best = -1;
  long long least = 0;
  for (int i = vec ? 0 : 1; i < 4; ++i) {
    if ((M + tiles[i].bm - 1) / tiles[i].bm > 65535) continue;          // more tiles than a grid has rows
    const long long blocks = (long long)((M + tiles[i].bm - 1) / tiles[i].bm) * ((N + tiles[i].bn - 1) / tiles[i].bn);
    const long long cost = vec ? (blocks + sms - 1) / sms * tiles[i].cycles + (i == 0 ? 12 : 0)
                               : std::max((long long)tiles[i].first * sms, blocks * tiles[i].each);
    if (best < 0 || cost < least) best = i, least = cost;
  }
  return best;
}

// Whether few rows are streamed or taken in tiles.  A block of the streaming form is one warp with up to four outputs a lane: the
// more rows and the more of them an SM holds, the more the tiles' reuse wins; with few k's the streaming form is all ramp.  us,
// streamed | tiles: 4 x 8,192 x 128 6.5 | 4.8, x 512 10.6 | 12.2; 8 x 32,000 x 512 35 | 33, x 1,024 48 | 63; 16 x 2,048 x 1,024
// 10.9 | 16.3; 16 x 4,096 x 1,024 17.1 | 16.3, x 2,048 27.6 | 30.4; 16 x 8,192 x 4,096 92 | 80.
static bool few_rows(int M, int N, int K) {
  if (M <= 2 || M > FEW_M) return M <= 2;
  if (N >= 2048 && K < FEW_K) return false;
  if (M <= 8) return K >= 512 ? M <= 4 || N < 16384 || K >= 1024 : N < 4096;
  return N <= 2048 || (N <= 4096 && K >= 2048);
}

template <typename TA, typename TW, typename TO>
static int run(const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldw,
               long long ldc, cudaStream_t stream) {
  const bool vec = sizeof(TA) == 4 && sizeof(TW) == 4 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
                   ((uintptr_t)A | (uintptr_t)W) % 16 == 0;
  if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4 && sizeof(TO) == 4) {
    if (vec && few_rows(M, N, K)) {
      if (M <= 4) return run_few<1>(A, W, C, M, N, K, lda, ldw, ldc, stream);
      if (M <= 8) return run_few<2>(A, W, C, M, N, K, lda, ldw, ldc, stream);
      return run_few<4>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    }
  }
  switch (pick_tile(M, N, vec)) {
    case 0: return run_tile<TA, TW, TO, 64, 128, 8, 8>(A, W, C, M, N, K, lda, ldw, ldc, vec, stream);
    case 1: return run_tile<TA, TW, TO, 64, 64, 8, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, stream);
    case 2: return run_tile<TA, TW, TO, 32, 64, 4, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, stream);
    default: return run_tile<TA, TW, TO, 32, 32, 4, 2>(A, W, C, M, N, K, lda, ldw, ldc, vec, stream);
  }
}

}  // namespace srlm

using namespace srlm;

extern "C" int srlm_gemm_tn_simt(const void* A, int a_dtype, const void* W, int w_dtype, void* C,
                                 int c_dtype, int M, int N, int K, long long lda, long long ldw,
                                 long long ldc, cudaStream_t stream) {
  if (M <= 0) return ST_OK;
  if (N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N)
    return refuse(ST_BAD_SIZE, "gemm_tn_simt: M=%d N=%d K=%d lda=%lld ldw=%lld ldc=%lld", M, N, K, lda,
                  ldw, ldc);
  if ((M + 63) / 64 > 65535)
    return refuse(ST_BAD_SIZE, "gemm_tn_simt: M=%d exceeds %d rows", M, 65535 * 64);
  if (a_dtype == DT_F32 && w_dtype == DT_F32 && c_dtype == DT_F32)
    return run<float, float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (a_dtype == DT_BF16 && w_dtype == DT_BF16 && c_dtype == DT_BF16)
    return run<bf16, bf16, bf16>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (a_dtype == DT_BF16 && w_dtype == DT_BF16 && c_dtype == DT_F32)
    return run<bf16, bf16, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  return refuse(ST_BAD_DTYPE, "gemm_tn_simt: dtypes (%d, %d) -> %d are not offered", a_dtype, w_dtype,
                c_dtype);
}
