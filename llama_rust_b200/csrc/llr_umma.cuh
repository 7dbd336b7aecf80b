// What the kernels on tcgen05.mma share: mbarrier wrappers with bounded waits and shared-memory descriptors; for those that feed it
// dequantized tiles (llr_gemm_tc.cu, llr_gemm_i8.cu) the packed-byte ring's geometry and the Q6_K code unpacking.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "llr_formats.cuh"
#include "llr_kernels.cuh"

namespace llr {
namespace umma {

constexpr int BM = 128;     // weight rows per CTA = UMMA M
constexpr int MACRO = 256;  // columns per packed-byte ring stage
constexpr int TC_SPIN = 1 << 24;
constexpr int SMEM_LIMIT = 232448;  // 227 KB opt-in maximum per CTA

// packed bytes per row per macro-step, and the ring's row pitch (odd multiple of 16 bytes)
template <int DT> struct Pk;
template <> struct Pk<DT_Q4_K> { static constexpr int RB = 144, PITCH = 144; };
template <> struct Pk<DT_Q8_0> { static constexpr int RB = 272, PITCH = 272; };
template <> struct Pk<DT_Q5_0> { static constexpr int RB = 176, PITCH = 176; };
template <> struct Pk<DT_Q4_0> { static constexpr int RB = 144, PITCH = 144; };
template <> struct Pk<DT_Q5_1> { static constexpr int RB = 192, PITCH = 208; };
template <> struct Pk<DT_Q4_1> { static constexpr int RB = 160, PITCH = 176; };
template <> struct Pk<DT_Q5_K> { static constexpr int RB = 176, PITCH = 176; };
// Q6_K blocks are 210 bytes: the block of macro-step ms starts at 210*ms, which is a multiple of 16 bytes only
// for every eighth step.  The copy starts at the 16-byte boundary below (TMA needs that) and is 240 bytes wide
// (14 bytes of lead at most + 210, rounded up to an odd number of 16-byte chunks); the decoder adds the lead back.
template <> struct Pk<DT_Q6_K> { static constexpr int RB = 210, PITCH = 240; };

__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* b, int n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity) {
  for (int spins = 0; spins < TC_SPIN; ++spins) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(s32(b)), "r"(parity) : "memory");
    if (ok) return true;
  }
  return false;
}

// both barriers tested in one go, so that the two round trips to the barrier unit overlap
__device__ __forceinline__ bool bar_wait2(uint64_t* a, uint32_t pa, uint64_t* b, uint32_t pb) {
  for (int spins = 0; spins < TC_SPIN; ++spins) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p, q; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4; "
        "and.pred p, p, q; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok) : "r"(s32(a)), "r"(pa), "r"(s32(b)), "r"(pb) : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(pred));
  return pred != 0;
}

// K-major, 128-byte swizzle shared-memory matrix descriptor: rows of 128 bytes, eight-row
// groups 1024 bytes apart, descriptor version 1 (sm_100), layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t smem_desc_u(uint32_t saddr) {
  const uint64_t addr = (uint64_t)(saddr >> 4) & 0x3fffu;
  return addr | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

constexpr uint32_t DESC_HI = 64u | (1u << 14) | (2u << 29);  // its high word; the low word of addresses below 2^18 without leading offset: address / 16

__device__ __forceinline__ float h2f(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }
// Shared memory is addressed through 32-bit shared-window addresses and explicit ld/st.shared:
// the tile base is aligned by integer arithmetic, which would otherwise turn every access
// into a generic-address load or store.
template <int NCH> __device__ __forceinline__ void lds_chunks(uint32_t p, uint32_t (&w)[4 * NCH]) {
#pragma unroll
  for (int i = 0; i < NCH; ++i)
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(w[4 * i]), "=r"(w[4 * i + 1]), "=r"(w[4 * i + 2]), "=r"(w[4 * i + 3]) : "r"(p + 16 * i));
}

// 32 bytes at byte offset off (even, the same for all threads of the CTA) of a row in the packed ring, as eight
// words: three aligned 16-byte loads, then a shift by whole words (four cases, uniform branch) and by a half word.
__device__ __forceinline__ void lds_32_at(uint32_t prow, int off, uint32_t (&q)[8]) {
  uint32_t w[12];
  lds_chunks<3>(prow + (uint32_t)(off & ~15), w);
  const uint32_t hs = (uint32_t)(off & 2) * 8u;
  switch ((off & 15) >> 2) {
    case 0:
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = __funnelshift_r(w[i], w[i + 1], hs);
      break;
    case 1:
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = __funnelshift_r(w[i + 1], w[i + 2], hs);
      break;
    case 2:
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = __funnelshift_r(w[i + 2], w[i + 3], hs);
      break;
    default:
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = __funnelshift_r(w[i + 3], w[i + 4], hs);
      break;
  }
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t p) {
  uint32_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(p));
  return v;
}
// Q6_K sub-block sb (32 columns) of the block that starts `lead` bytes into the ring row: the six-bit codes
// c = ql nibble | two qh bits << 4 of columns 4i..4i+3 in the bytes of c[i], the two signed scales (columns 0..15,
// 16..31) and d.  Layout of dequant_q6_k_row (langtax/src/quant.rs): per 128 columns, ql bytes 64n + 32(j & 1) + l
// give nibble j >> 1, qh bytes 32n + l give bits 2j.., scales 8n + 2j + l / 16.
__device__ __forceinline__ void q6k_codes(uint32_t prow, int lead, int sb, uint32_t (&c)[8], float& d, int& s0, int& s1) {
  const int n = sb >> 2, j = sb & 3;
  uint32_t ql[8], qh[8];
  lds_32_at(prow, lead + 64 * n + 32 * (j & 1), ql);
  lds_32_at(prow, lead + 128 + 32 * n, qh);
  const uint32_t sc = lds_u16(prow + (uint32_t)(lead + 192 + 8 * n + 2 * j));
  d = h2f(lds_u16(prow + (uint32_t)(lead + 208)));
  s0 = (int)(int8_t)(sc & 255u);
  s1 = (int)(int8_t)(sc >> 8);
  const int nsh = 4 * (j >> 1), hsh = 2 * j;
#pragma unroll
  for (int i = 0; i < 8; ++i) c[i] = ((ql[i] >> nsh) & 0x0f0f0f0fu) | (((qh[i] >> hsh) & 0x03030303u) << 4);
}

}  // namespace umma
}  // namespace llr
