// What the attention kernels on tcgen05 tensor cores share: mbarriers with bounded waits, TMA loads, MMA issue and
// descriptors, tensor-memory loads and stores, and the softmax of a row of 128 scores held by one thread.
#pragma once

#include <cuda.h>
#include <math_constants.h>

#include <mutex>

#include "common.cuh"

namespace srlm {
namespace fmha {

constexpr long long WAIT_CYCLES = 4000000000ll;

__device__ __forceinline__ uint32_t s32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(s32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err_flag, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (clock64() - t0 > WAIT_CYCLES) {
      atomicExch(err_flag, code);
      return false;
    }
  }
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(s32(dst)), "l"(map), "r"(s32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar)) : "memory");
}
// D[tmem] (+)= A[tmem, bfloat16 pairs per column] . B[smem]
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 128-byte swizzled operand tile.  K-major: rows of 128 bytes along K, 8-row groups 1024 bytes apart
// (the leading offset is unused).  MN-major: rows of 128 bytes along MN (64 elements), 8 k-rows per
// 1024-byte group (stride offset), the next 64 elements of MN `lead` bytes further (leading offset).
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lead_bytes, uint32_t stride_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lead_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((stride_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ uint32_t umma_idesc(int n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn_major ? (1u << 16) : 0u) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// 16-byte chunk `c16` (of 16) of row `row` in a tile of two 64-element panels [128 rows][128 bytes].
__device__ __forceinline__ uint32_t tile_addr(uint32_t tile, int row, int c16) {
  return tile + (uint32_t)(c16 >> 3) * (128 * 128) + (uint32_t)row * 128 + (uint32_t)(((c16 & 7) ^ (row & 7)) << 4);
}


// One row of S (128 keys) in registers: the four loads are in flight together.
struct Row {
  uint32_t a[32], b[32], c[32], d[32];
};
__device__ __forceinline__ void load_row(uint32_t s_addr, Row& r) {
  tmem_ld32(s_addr, r.a);
  tmem_ld32(s_addr + 32, r.b);
  tmem_ld32(s_addr + 64, r.c);
  tmem_ld32(s_addr + 96, r.d);
  tmem_wait_ld();
}
// The maximum of the keys [k_lo, k_hi) of the row (all 128 keys when not MASKED).
template <bool MASKED>
__device__ __forceinline__ float row_max(const Row& r, int k_lo, int k_hi) {
  float m0 = -CUDART_INF_F, m1 = -CUDART_INF_F, m2 = -CUDART_INF_F, m3 = -CUDART_INF_F;
  auto part = [&](const uint32_t (&v)[32], int c) {
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const int k = c + j;
      if (!MASKED || (k >= k_lo && k < k_hi)) m0 = fmaxf(m0, __uint_as_float(v[j]));
      if (!MASKED || (k + 1 >= k_lo && k + 1 < k_hi)) m1 = fmaxf(m1, __uint_as_float(v[j + 1]));
      if (!MASKED || (k + 2 >= k_lo && k + 2 < k_hi)) m2 = fmaxf(m2, __uint_as_float(v[j + 2]));
      if (!MASKED || (k + 3 >= k_lo && k + 3 < k_hi)) m3 = fmaxf(m3, __uint_as_float(v[j + 3]));
    }
  };
  part(r.a, 0);
  part(r.b, 32);
  part(r.c, 64);
  part(r.d, 96);
  return fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
}
// P = exp2(S * scale - base) as bfloat16 pairs over the first 64 columns of S; returns the row sum, of the weights as they are
// or (ROUNDED) as the product with V reads them: a row's weights then add up to one exactly, and the rounding of one that
// outweighs the others cancels.
template <bool MASKED, bool ROUNDED = false>
__device__ __forceinline__ float row_exp(uint32_t s_addr, const Row& r, float scale, float base, int k_lo, int k_hi) {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  const float nb = -base;
  auto part = [&](const uint32_t (&v)[32], int c) {
    uint32_t pk[16];
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      float p0 = ex2(fmaf(__uint_as_float(v[j]), scale, nb));
      float p1 = ex2(fmaf(__uint_as_float(v[j + 1]), scale, nb));
      float p2 = ex2(fmaf(__uint_as_float(v[j + 2]), scale, nb));
      float p3 = ex2(fmaf(__uint_as_float(v[j + 3]), scale, nb));
      if (MASKED) {
        const int k = c + j;
        p0 = (k >= k_lo && k < k_hi) ? p0 : 0.f;
        p1 = (k + 1 >= k_lo && k + 1 < k_hi) ? p1 : 0.f;
        p2 = (k + 2 >= k_lo && k + 2 < k_hi) ? p2 : 0.f;
        p3 = (k + 3 >= k_lo && k + 3 < k_hi) ? p3 : 0.f;
      }
      const uint32_t lo = pk[j >> 1] = pack2(p0, p1), hi = pk[(j >> 1) + 1] = pack2(p2, p3);
      if (ROUNDED) {
        p0 = __uint_as_float(lo << 16), p1 = __uint_as_float(lo & 0xffff0000u);
        p2 = __uint_as_float(hi << 16), p3 = __uint_as_float(hi & 0xffff0000u);
      }
      s0 += p0; s1 += p1; s2 += p2; s3 += p3;
    }
    tmem_st16(s_addr + (c >> 1), pk);
  };
  part(r.a, 0);
  part(r.b, 32);
  part(r.c, 64);
  part(r.d, 96);
  return (s0 + s1) + (s2 + s3);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
        qr == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

}  // namespace fmha
}  // namespace srlm
