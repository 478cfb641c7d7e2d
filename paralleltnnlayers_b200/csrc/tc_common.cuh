// sm_100a building blocks used by the tensor-core kernels: mbarrier, TMA (cp.async.bulk.tensor),
// tcgen05 (TMEM allocation, MMA, commit, load), descriptors.  Inline PTX only.
//
// Every wait is bounded: a wait that runs out returns false, the kernel records the failure in a
// status word and leaves through its normal exit (TMEM released), so a lost signal can never hang the GPU.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace b200cp {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier -----------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait on a phase parity.  Returns false when the limit is reached.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit_cycles = 1500000000ll) {
  const uint32_t a = smem_u32(bar);
  const long long t0 = clock64();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > limit_cycles) return false;  // about a second: record and leave, never hang
  }
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// generic-proxy writes to shared memory -> visible to the async proxy (TMA, tcgen05.mma)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- TMA --------------------------------------------------------------------------
// 3-D tiled load (no multicast): coordinates (x = innermost, y, z).  x * 4 bytes must be a multiple of 16.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// 4-D tiled load (no multicast): coordinates (x = innermost, y, z, w); x * 4 bytes must be a multiple of 16, the other
// coordinates may start outside the tensor (out-of-range elements arrive as the map's fill value: zero).
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z,
                                            int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// One lane of a converged warp.  The compiler keeps the descriptors of tcgen05 instructions that follow in uniform registers, which
// it cannot after a comparison of the thread index: 24 products of 128 x 32 x 16 are issued in 770 cycles instead of 1210.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
  return one != 0;
}

// ---- TMEM -------------------------------------------------------------------------
// One full warp allocates `ncols` (power of two, >= 32) columns; the base address lands in *slot (shared).
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- descriptors -------------------------------------------------------------------
// Shared-memory matrix descriptor (sm_100 format): start address, leading / stride byte offsets
// (all in units of 16 bytes), descriptor version 1, swizzle mode in bits 61..63
// (0 none, 1 = 128 B span with 32-byte atoms, 2 = 128 B span with 16-byte atoms).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t swizzle) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)(swizzle & 7) << 61;
  return d;
}
constexpr uint32_t kSwizzleNone = 0, kSwizzle128B_32B = 1, kSwizzle128B = 2;

// Instruction descriptor for kind::tf32 with fp32 accumulation, M = 128.
// a_mn / b_mn: 1 when the operand is MN-major (contiguous along M / N), 0 when K-major.
__host__ __device__ constexpr uint32_t make_idesc_tf32(uint32_t n, uint32_t a_mn, uint32_t b_mn) {
  return (1u << 4)      // D format: F32
         | (2u << 7)    // A format: TF32
         | (2u << 10)   // B format: TF32
         | (a_mn << 15) | (b_mn << 16) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.
__device__ __forceinline__ void mma_tf32_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}
// The mbarrier receives one arrival when every previously issued MMA of this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// TMEM -> registers: the warp reads its own 32-lane quarter, `N` consecutive 32-bit columns per thread.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ---- tf32 split --------------------------------------------------------------------
// hi = x rounded to tf32 (10-bit mantissa), lo = x - hi (exact in fp32).  hi*b + lo*b recovers x*b
// to about 2^-21 relative once lo is itself cut to tf32 by the tensor core.
// Round to nearest, ties away from zero, as cvt.rna.tf32.f32 does for finite x below the overflow threshold:
// half an ulp added to the magnitude bits, low 13 bits cut (two integer instructions).
__device__ __forceinline__ float tf32_hi(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}

// ---- scaled fp16 split: x = (hi + lo) * 2^e with one exponent per row (gemm_tc.cu) ---------------------------------
// 2^e for e in [-126, 127]
__device__ __forceinline__ float exp2_int(int e) { return __int_as_float((e + 127) << 23); }
// v * 2^e for e in [-252, 254], in two steps of the same sign
__device__ __forceinline__ float scale_by(float v, int e) {
  const int h = e >> 1;
  return v * exp2_int(h) * exp2_int(e - h);
}

// Exponent e of a row whose largest magnitude has these bits: x * 2^-e is below 2^15.  (Infinities and NaN leave the
// finite values of their row in range and themselves non-finite.)
__device__ __forceinline__ int row_exponent(unsigned bits, int least) {
  return bits == 0 ? 0 : max((int)(bits >> 23) - 141, least);
}
constexpr int kLeast = -126, kLeastConv = -100;   // 2^-e and (convolutions) 2^(e - 24) stay normal numbers

// the largest and the least of three magnitudes, one instruction; a NaN is neither, but the largest with most_nan
#define B200CP_MAGNITUDES(name, op)                                                                                            \
  __device__ __forceinline__ float name(float a, float b, float c) {                                                           \
    float d;                                                                                                                   \
    asm("{\n.reg .f32 x, y;\nabs.f32 x, %2;\nabs.f32 y, %3;\n" op ".f32 %0, %1, x, y;\n}" : "=f"(d) : "f"(a), "f"(b), "f"(c)); \
    return d;                                                                                                                  \
  }
B200CP_MAGNITUDES(most_of, "max")
B200CP_MAGNITUDES(most_nan, "max.NaN")
B200CP_MAGNITUDES(least_of, "min")
#undef B200CP_MAGNITUDES
__device__ __forceinline__ unsigned abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
constexpr int kRowShift = 24;   // of totals that take a power of two per step: see SplitGemm::ea
// ---- three bf16 parts -------------------------------------------------------------------------------------------------
// Two values as three bf16 parts each, x = p[0] + p[1] + p[2] exactly (each part with its own exponent; the last may fall below the
// smallest float).  The first is cut off, so that no finite value becomes infinite; the other two are rounded, so that what a
// product leaves out (p[1] p[2], 2^-24 of it) has no preferred sign.
struct Bf3 {
  uint32_t p[3];
};
constexpr float kLift = 131072.f;   // 2^17: values times it have normal parts wherever they are normal themselves
__device__ __forceinline__ Bf3 split3(float a, float b) {
  Bf3 out;
  const uint32_t x = __float_as_uint(a), y = __float_as_uint(b);
  out.p[0] = __byte_perm(x, y, 0x7632);
  a -= __uint_as_float(x & 0xffff0000u);
  b -= __uint_as_float(y & 0xffff0000u);
  const __nv_bfloat162 m = __floats2bfloat162_rn(a, b);
  const float2 f = __bfloat1622float2(m);
  const __nv_bfloat162 l = __floats2bfloat162_rn(a - f.x, b - f.y);
  out.p[1] = *reinterpret_cast<const uint32_t*>(&m);
  out.p[2] = *reinterpret_cast<const uint32_t*>(&l);
  return out;
}
// The same with a first part of six bits, rounded: the products of two of them have twelve, so that an instruction adds sixteen without
// cutting any off unless one is 2^-12 of another (with eight bits 2^-8, and the sums of an instruction are 2e-8 too small in the mean).
// The three parts still hold all 24 bits; the second is up to 2^-6 of the value, so that its products with the third count too.  (A value
// that would round to infinity, within 1 % of the largest, is cut off instead and may lose its last bit; without FINITE it becomes one.)
template <bool FINITE>
__device__ __forceinline__ Bf3 split3_short(float a, float b) {
  Bf3 out;
  const auto first = [](float v) {
    const uint32_t u = __float_as_uint(v), up = u + 0x20000u;
    return (FINITE && (up & 0x7f800000u) == 0x7f800000u ? u : up) & 0xfffc0000u;
  };
  const uint32_t x = first(a), y = first(b);
  out.p[0] = __byte_perm(x, y, 0x7632);
  a -= __uint_as_float(x);
  b -= __uint_as_float(y);
  const __nv_bfloat162 m = __floats2bfloat162_rn(a, b);
  const float2 f = __bfloat1622float2(m);
  const __nv_bfloat162 l = __floats2bfloat162_rn(a - f.x, b - f.y);
  out.p[1] = *reinterpret_cast<const uint32_t*>(&m);
  out.p[2] = *reinterpret_cast<const uint32_t*>(&l);
  return out;
}
// Instruction descriptor for kind::f16 with K-major operands and fp32 accumulation, M = 128 (one CTA): fp16, or bf16.
__host__ __device__ constexpr uint32_t make_idesc_f16(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }
__host__ __device__ constexpr uint32_t make_idesc_bf16(uint32_t n) { return make_idesc_f16(n) | (1u << 7) | (1u << 10); }
__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

}  // namespace tc

// host: cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda)
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
PFN_encodeTiled get_encode_tiled();

}  // namespace b200cp
