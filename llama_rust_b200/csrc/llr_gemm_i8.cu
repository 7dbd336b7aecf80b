// Products of more activation rows than the decode kernel takes at once, with 32-bit results, for the K-quants (Q4_K, Q5_K,
// Q6_K) on the integer tensor cores of the 5th generation: what llr_gemv_stream.cu does for 1..8 rows, with the same sums in the
// same order, so that a row's result keeps its bits whatever batch it is in.
//
// The arithmetic is llr_mma_common.cuh's: activations as four signed base-256 digits of a per-block integer, exact integer dot
// products, one int -> float conversion and one multiply-add per (row, 256-column block, digit).  The integers are formed
// another way: sub-block scale times code is a 16-bit integer, written as an unsigned low byte and a signed high byte, and the
// sums over a block's 256 columns are two chains of tcgen05.mma.kind::i8 (M = 128 weight rows, N = 4 digits of TB activation
// rows, K = 32).  Low and high sums are joined as lo + 256 hi: the same integer that the decode kernel adds up sub-block by
// sub-block with its scales.
//
// What bounds it: the decode kernel spends an integer multiply-add per (row, 32 columns, activation row, digit) on the scales
// and reads the weights again for every eight rows (14336 x 4096 Q4_K: 20 us a pass).  Here the weights are decoded once for
// up to 24 rows (1.6 instructions per weight) and the scales cost nothing per activation row; what is left is the drain, about
// 20 instructions per (row, block, activation row).
//
// A CTA owns 128 weight rows, TB activation rows and a range of units.  A unit is what one warp of the decode kernel owns of
// 4096 columns: blocks w and w + 8.  Its result is one float per (row, activation row); the floats of the eight units of a
// part are added in order, then the parts.  28 warps:
//   * sixteen dequantize: packed bytes (TMA ring) -> low | high bytes in tensor memory (A operand, stages of 128 columns); each
//     decodes 64 columns of 32 weight rows of every block before it waits for a free stage, since the ring holds one to three
//     blocks and its round trip is what the MMAs would otherwise wait for;
//   * eight drain: accumulators of a finished unit -> floats, the mins, the sums over units, and the stores; two warps share
//     the 32 tensor-memory lanes (weight rows) of a quarter, half of the activation rows each, and fetch the next activation row's
//     accumulators while they work on one;
//   * one copies packed weights, one digit tiles and the blocks' sums and scales, two issue the MMAs.
// (Eight dequantizing warps, one issuing warp that waited for every 64 columns: 44 us instead of 34 for 24 rows of Q4_K
// 14336 x 4096, 37 instead of 30 for 16 rows.)
// Both blocks of a unit have accumulators of their own (2 x 2 x 4 TB columns of tensor memory), the rest holds the A ring.
// Few row tiles: the units are spread over several CTAs (grid z), each unit's floats go to memory and a second kernel adds
// them in the same order.
// Measured, passes of the decode kernel -> this: 24 rows Q4_K 14336 x 4096 62 -> 34 us, 4096 x 4096 34 -> 15, 1024 x 4096
// 28 -> 10; Q6_K 4096 x 14336 124 -> 47, 32000 x 4096 138 -> 71; 48 rows Q4_K 4096 x 4096 68 -> 23.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "llr_formats.cuh"
#include "llr_kernels.cuh"
#include "llr_mma_common.cuh"
#include "llr_tmap.cuh"
#include "llr_umma.cuh"

namespace llr {
namespace {
using namespace umma;

constexpr int DQ = 16, DR = 8;  // dequantizing and draining warps
// Registers per thread: the drain keeps two activation rows' accumulators in flight, the others need few.  All warpgroups give or
// take at their start; the sum is what the block was launched with (28 warps x 72).
constexpr int REG_DQ = 64, REG_DR = 104, REG_REST = 40;
static_assert(4 * REG_DQ + 2 * REG_DR + REG_REST <= 7 * 72, "register split");
constexpr int W_PACKED = DQ + DR, W_DIG = W_PACKED + 1, W_MMA = W_DIG + 1, THREADS = 32 * (W_MMA + 2);  // two MMA warps
constexpr int PART_BLOCKS = 16, PART_UNITS = 8;  // of 4096 columns
constexpr int AUX = 48;  // bytes per (block, activation row): eight sums of 32 columns, 2^-e, padding

template <int DT, int TB> struct ILay {
  static constexpr int N = 4 * TB;             // digit planes of TB activation rows
  static constexpr int ACC = 2 * 2 * N;        // accumulator columns: (low, high) of a unit's two blocks
  static constexpr int A_COLS = 64;            // 128 weight columns: 4 sub-blocks x (low, high) x 8 words
  static constexpr int NA = (512 - ACC) / A_COLS;
  static constexpr int IMG = N * 256;          // digits of one block, as the MMA reads them
  static constexpr int REC = IMG + TB * AUX;   // a block's record in memory
  static constexpr int NB = 4, NX = 4;
  static constexpr int P_STAGE = BM * Pk<DT>::PITCH;
  static constexpr int B = 0, X = NB * IMG, P = X + NX * TB * AUX;
  static constexpr int FIXED = 1024 /*alignment*/ + 64 /*chunk reads may pass a row's end*/ + 16 + 512 /*barriers*/;
  static constexpr int FIT = (SMEM_LIMIT - FIXED - P) / P_STAGE, NPK = FIT > 6 ? 6 : FIT;
  static constexpr int BAR = (P + NPK * P_STAGE + 64 + 15) / 16 * 16;
  static constexpr int TOTAL = BAR + 512 + 1024;
  static_assert(NA >= 2 && NA % 2 == 0 && NPK >= 2 && P % 128 == 0 && IMG % 1024 == 0 && REC % 16 == 0, "rings");
  static_assert((2 * NA + 2 * NB + 2 * NX + 2 * NPK + 2) * 8 + 8 <= 512 && TOTAL <= SMEM_LIMIT, "shared memory");
};

// How the columns of a row fall into units: `blocks` 256-column blocks.
__host__ __device__ __forceinline__ int units_of(int blocks) {
  const int rest = blocks % PART_BLOCKS;
  return blocks / PART_BLOCKS * PART_UNITS + (rest < PART_UNITS ? rest : PART_UNITS);
}
__device__ __forceinline__ int unit_blocks(int u, int blocks, int& first) {
  const int part = u / PART_UNITS, w = u % PART_UNITS;
  first = part * PART_BLOCKS + w;
  return first + PART_UNITS < blocks ? 2 : 1;
}

// kind::i8: D s32, A u8 or s8 (tensor memory), B s8 (shared memory, K-major), M = 128
template <int N, bool SIGNED_A> __host__ __device__ constexpr uint32_t desc_i8() {
  return (2u << 4) | ((SIGNED_A ? 1u : 0u) << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

typedef unsigned long long pair;
__device__ __forceinline__ pair fma2(pair a, pair b, pair c) {
  pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ pair mul2(pair a, pair b) {
  pair d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ pair pack2(float lo, float hi) { return (pair)__float_as_uint(hi) << 32 | __float_as_uint(lo); }
__device__ __forceinline__ float low2(pair p) { return __uint_as_float((uint32_t)p); }
__device__ __forceinline__ float high2(pair p) { return __uint_as_float((uint32_t)(p >> 32)); }

// 16-bit products of four columns, (c0, c2) and (c1, c3) -> their low and high bytes in column order
__device__ __forceinline__ void split_bytes(uint32_t p02, uint32_t p13, uint32_t& lo, uint32_t& hi) {
  lo = __byte_perm(p02, p13, 0x6240);
  hi = __byte_perm(p02, p13, 0x7351);
}

// Sub-block 2 G + S (32 columns) of the row at prow: o[0..7] low bytes, o[8..15] high bytes.
// Q4_K: 16 scale code, Q5_K: scale code, Q6_K: 4 scale (code - 32), the multiples that the decode kernel sums too.
template <int DT, int S>
__device__ __forceinline__ void decode32(uint32_t prow, int lead, int G, uint32_t (&o)[16]) {
  if constexpr (DT == DT_Q6_K) {
    uint32_t c[8];
    float d;
    int sc[2];
    q6k_codes(prow, lead, 2 * G + S, c, d, sc[0], sc[1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      // both halves of 4 scale (code - 32) + 32768 lie in [16384, 49152]; flipping the top bit takes the 32768 off again
      const uint32_t k = 4u * (uint32_t)sc[i >> 2], bias = 0x80008000u - 32u * k * 0x10001u;
      split_bytes((c[i] & 0x00ff00ffu) * k + bias, ((c[i] >> 8) & 0x00ff00ffu) * k + bias, o[i], o[8 + i]);
      o[8 + i] ^= 0x80808080u;
    }
  } else {
    constexpr bool K5 = DT == DT_Q5_K;
    uint32_t h[4], q[8];
    lds_chunks<1>(prow, h);
    lds_chunks<2>(prow + (K5 ? 48 : 16) + 32 * G, q);
    const uint32_t sc = G < 2 ? h[1] & 0x3f3f3f3fu : (h[3] & 0x0f0f0f0fu) | ((h[1] >> 2) & 0x30303030u);
    const uint32_t s = (sc >> (16 * (G & 1) + 8 * S)) & 255u;
    if constexpr (K5) {
      uint32_t f[8];
      lds_chunks<2>(prow + 16, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t a = ((q[i] >> (4 * S)) & 0x0f0f0f0fu) | (((f[i] >> (2 * G + S)) & 0x01010101u) << 4);
        split_bytes((a & 0x00ff00ffu) * s, ((a >> 8) & 0x00ff00ffu) * s, o[i], o[8 + i]);
      }
    } else {
      constexpr uint32_t M = S ? 0x00f000f0u : 0x000f000fu;
      const uint32_t k = S ? s : 16u * s;
#pragma unroll
      for (int i = 0; i < 8; ++i) split_bytes((q[i] & M) * k, ((q[i] >> 8) & M) * k, o[i], o[8 + i]);
    }
  }
}

// What the drain needs of a block's header: d, and dmin times the eight mins in pairs ((0, 1), (2, 3), ...)
template <int DT> struct Head { float d; pair m[4]; };
template <int DT>
__device__ __forceinline__ void read_head(uint32_t prow, int lead, Head<DT>& H) {
  if constexpr (DT == DT_Q6_K) {
    H.d = h2f(lds_u16(prow + (uint32_t)(lead + 208)));
  } else {
    uint32_t h[4];
    lds_chunks<1>(prow, h);
    H.d = h2f(h[0] & 0xffffu);
    const float dmin = h2f(h[0] >> 16);
    const uint32_t lo = h[2] & 0x3f3f3f3fu, hi = ((h[3] >> 4) & 0x0f0f0f0fu) | ((h[2] >> 2) & 0x30303030u);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      H.m[i] = pack2(dmin * (float)((lo >> (16 * i)) & 255u), dmin * (float)((lo >> (16 * i + 8)) & 255u));
      H.m[2 + i] = pack2(dmin * (float)((hi >> (16 * i)) & 255u), dmin * (float)((hi >> (16 * i + 8)) & 255u));
    }
  }
}

// four digit sums of one activation row
__device__ __forceinline__ void tmem_ld4(uint32_t addr, int (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&o)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]),
                 "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(o[15]) : "memory");
}

// One activation row of a finished unit of NBK blocks; its sums and scale lie at xa[k] + off
template <int DT, int NBK>
__device__ __forceinline__ float join(const int (&v)[NBK][2][4], const Head<DT> (&H)[2], const uint32_t (&xa)[2], uint32_t off) {
  constexpr float W0 = DT == DT_Q4_K ? 0.0625f : DT == DT_Q6_K ? 0.25f : 1.f;  // weights of the digits: 256^p, and 1/16 or 1/4 for the codes' multiples
  const pair w01 = pack2(W0, W0 * 256.f), w23 = pack2(W0 * 65536.f, W0 * 16777216.f);
  pair s01 = 0, s23 = 0, m01 = 0, m23 = 0;
#pragma unroll
  for (int k = 0; k < NBK; ++k) {
    float xs;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(xs) : "r"(xa[k] + off + 32));
    const float m = __fmul_rn(H[k].d, xs);
    const pair mm = pack2(m, m);  // times the weight as the decode kernel does it: the scales of tiny activations round there
    const int* l = v[k][0];
    const int* h = v[k][1];
    s01 = fma2(pack2((float)(l[0] + 256 * h[0]), (float)(l[1] + 256 * h[1])), mul2(mm, w01), s01);
    s23 = fma2(pack2((float)(l[2] + 256 * h[2]), (float)(l[3] + 256 * h[3])), mul2(mm, w23), s23);
    if constexpr (DT != DT_Q6_K) {
      pair c[4];
      asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];" : "=l"(c[0]), "=l"(c[1]) : "r"(xa[k] + off));
      asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];" : "=l"(c[2]), "=l"(c[3]) : "r"(xa[k] + off + 16));
      m01 = fma2(H[k].m[0], c[0], fma2(H[k].m[2], c[2], m01));
      m23 = fma2(H[k].m[1], c[1], fma2(H[k].m[3], c[3], m23));
    }
  }
  float r = __fadd_rn(__fadd_rn(low2(s01), high2(s01)), __fadd_rn(low2(s23), high2(s23)));
  if constexpr (DT != DT_Q6_K) r = __fsub_rn(r, __fadd_rn(__fadd_rn(low2(m01), high2(m01)), __fadd_rn(low2(m23), high2(m23))));
  return r;
}

struct Args {
  const uint8_t* rec;  // digit records [token tile][block]
  float* y;            // the result, or (several CTAs along z) the units' floats [unit][activation row][weight row]
  int rows, blocks, tokens;
};

template <int DT, int TB>
__global__ void __launch_bounds__(THREADS, 1)
gemm_i8_kernel(const __grid_constant__ CUtensorMap wmap, const Args P, int* __restrict__ err) {
  using L = ILay<DT, TB>;
  constexpr int NA = L::NA, NB = L::NB, NX = L::NX, NPK = L::NPK, N = L::N, PITCH = Pk<DT>::PITCH, RB = Pk<DT>::RB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_a = (uint64_t*)(smem + L::BAR);
  uint64_t* empty_a = full_a + NA;
  uint64_t* full_b = empty_a + NA;
  uint64_t* empty_b = full_b + NB;
  uint64_t* full_x = empty_b + NB;
  uint64_t* empty_x = full_x + NX;
  uint64_t* pk_full = empty_x + NX;
  uint64_t* pk_empty = pk_full + NPK;
  uint64_t* acc_full = pk_empty + NPK;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = (int)blockIdx.x * BM, tok0 = (int)blockIdx.y * TB;
  const int units = units_of(P.blocks), u_begin = (int)((int64_t)units * blockIdx.z / gridDim.z), u_end = (int)((int64_t)units * (blockIdx.z + 1) / gridDim.z);

  if (tid == 0) {
    for (int s = 0; s < NA; ++s) { bar_init(&full_a[s], 8); bar_init(&empty_a[s], 2); }
    for (int s = 0; s < NB; ++s) { bar_init(&full_b[s], 1); bar_init(&empty_b[s], 2); }
    for (int s = 0; s < NX; ++s) { bar_init(&full_x[s], 1); bar_init(&empty_x[s], DR); }
    for (int s = 0; s < NPK; ++s) { bar_init(&pk_full[s], 1); bar_init(&pk_empty[s], DQ + DR); }
    bar_init(acc_full, 2);
    bar_init(acc_empty, DR);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // only now: a dependent that is placed here finds its tensor memory after this block has its own, and does not wait with it for this grid
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  bool ok = true;
  auto wait = [&](uint64_t* bar, int n, int ring) {  // n-th use of a ring: its stage n % ring
    if (ok && !bar_wait(bar + n % ring, (uint32_t)((n / ring) & 1))) { ok = false; report_error(err, 3); }
  };
  auto wait_free = [&](uint64_t* bar, int n, int ring) {
    if (ok && !bar_wait(bar + n % ring, (uint32_t)(((n / ring) & 1) ^ 1))) { ok = false; report_error(err, 3); }
  };

  if (warp < DQ) {
    // ------------------------------------------------------------ dequantization: columns 64 G .. 64 G + 63 of every block
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_DQ));
    const int q = warp & 3, G = warp >> 2;
    const uint32_t a_dst = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)L::ACC;
    int n = 0;
    for (int u = u_begin; u < u_end; ++u) {
      int first;
      const int nb = unit_blocks(u, P.blocks, first);
      for (int k = 0; k < nb; ++k, ++n) {
        const int b = first + PART_UNITS * k, lead = DT == DT_Q6_K ? (b * RB) & 15 : 0, st = 2 * n + (G >> 1);
        wait(pk_full, n, NPK);
        const uint32_t prow = s32(smem + L::P) + (uint32_t)((n % NPK) * L::P_STAGE + (32 * q + lane) * PITCH), dst = a_dst + (uint32_t)(st % NA * L::A_COLS + 32 * (G & 1));
        uint32_t o[2][16];  // decoded before a stage is free: what follows, up to the MMA, is the latency that the short ring has to cover
        decode32<DT, 0>(prow, lead, G, o[0]);
        decode32<DT, 1>(prow, lead, G, o[1]);
        __syncwarp();
        if (lane == 0) bar_arrive(&pk_empty[n % NPK]);
        wait_free(empty_a, st, NA);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_st16(dst, o[0]);
        tmem_st16(dst + 16, o[1]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(&full_a[st % NA]);
      }
    }
  } else if (warp < DQ + DR) {
    // -------------------------------------------------------------------------------------------------------- drain
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REG_DR));
    constexpr int TW = TB / 2;  // activation rows of this warp
    const int q = warp & 3, half = (warp - DQ) >> 2, row = row0 + 32 * q + lane;
    const uint32_t acc = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(4 * TW * half);
    const bool split = gridDim.z > 1;
    float sum[TW], carry[TW];
#pragma unroll
    for (int t = 0; t < TW; ++t) sum[t] = carry[t] = 0.f;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // y may still be read by an earlier kernel
    int n = 0;
    for (int u = u_begin; u < u_end; ++u) {
      int first;
      const int nb = unit_blocks(u, P.blocks, first);
      Head<DT> H[2];
      uint32_t xa[2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (k < nb) {
          const int b = first + PART_UNITS * k;
          wait(pk_full, n + k, NPK);
          read_head<DT>(s32(smem + L::P) + (uint32_t)((n + k) % NPK * L::P_STAGE + (32 * q + lane) * PITCH), DT == DT_Q6_K ? (b * RB) & 15 : 0, H[k]);
          __syncwarp();
          if (lane == 0) bar_arrive(&pk_empty[(n + k) % NPK]);
          wait(full_x, n + k, NX);
          xa[k] = s32(smem + L::X) + (uint32_t)(((n + k) % NX * TB + half * TW) * AUX);
        }
      wait(acc_full, u - u_begin, 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      auto unit = [&](auto NBK_) {
        constexpr int NBK = decltype(NBK_)::value;
        int v[2][NBK][2][4];
        auto fetch = [&](int t, int (&d)[NBK][2][4]) {
#pragma unroll
          for (int k = 0; k < NBK; ++k) {
            tmem_ld4(acc + (uint32_t)(2 * N * k + 4 * t), d[k][0]);
            tmem_ld4(acc + (uint32_t)(2 * N * k + N + 4 * t), d[k][1]);
          }
        };
        fetch(0, v[0]);
#pragma unroll
        for (int t = 0; t < TW; ++t) {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (t + 1 < TW) fetch(t + 1, v[(t + 1) & 1]);
          const float r = join<DT, NBK>(v[t & 1], H, xa, (uint32_t)(t * AUX));
          if (split) {
            const int tok = tok0 + TW * half + t;
            if (row < P.rows && tok < P.tokens) P.y[((int64_t)u * P.tokens + tok) * P.rows + row] = r;
          } else {
            sum[t] = __fadd_rn(sum[t], r);
          }
        }
      };
      if (nb == 2) unit(std::integral_constant<int, 2>{});
      else unit(std::integral_constant<int, 1>{});
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        bar_arrive(acc_empty);
        bar_arrive(&empty_x[n % NX]);
        if (nb == 2) bar_arrive(&empty_x[(n + 1) % NX]);
      }
      n += nb;
      if (!split && (u % PART_UNITS == PART_UNITS - 1 || u == units - 1)) {  // a part is complete
#pragma unroll
        for (int t = 0; t < TW; ++t) {
          carry[t] = u < PART_UNITS ? sum[t] : __fadd_rn(sum[t], carry[t]);
          sum[t] = 0.f;
        }
      }
    }
    if (!split && row < P.rows) {
#pragma unroll
      for (int t = 0; t < TW; ++t) {
        const int tok = tok0 + TW * half + t;
        if (tok < P.tokens) P.y[(int64_t)tok * P.rows + row] = carry[t];
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  } else {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_REST));
   if (warp == W_PACKED) {
    if (lane == 0) {
      int n = 0;
      for (int u = u_begin; u < u_end; ++u) {
        int first;
        const int nb = unit_blocks(u, P.blocks, first);
        for (int k = 0; k < nb; ++k, ++n) {
          const int b = first + PART_UNITS * k, ps = n % NPK;
          wait_free(pk_empty, n, NPK);
          bar_expect(&pk_full[ps], BM * PITCH);
          // x in 32-bit words, rounded down to 16 bytes (Q6_K only); rows and words past the matrix read as zero
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
              ::"r"(s32(smem + L::P + ps * L::P_STAGE)), "l"(&wmap), "r"(((b * RB) & ~15) / 4), "r"(row0), "r"(s32(&pk_full[ps])) : "memory");
        }
      }
    }
   } else if (warp == W_DIG) {
    if (lane == 0) {
      asm volatile("griddepcontrol.wait;" ::: "memory");  // the records are the kernel before's output
      int n = 0;
      auto copy = [&](uint8_t* dst, const uint8_t* src, uint32_t bytes, uint64_t* bar) {
        bar_expect(bar, bytes);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(s32(dst)), "l"(src), "r"(bytes), "r"(s32(bar)) : "memory");
      };
      for (int u = u_begin; u < u_end; ++u) {
        int first;
        const int nb = unit_blocks(u, P.blocks, first);
        for (int k = 0; k < nb; ++k, ++n) {
          const uint8_t* src = P.rec + ((int64_t)blockIdx.y * P.blocks + first + PART_UNITS * k) * L::REC;
          wait_free(empty_b, n, NB);
          copy(smem + L::B + n % NB * L::IMG, src, L::IMG, &full_b[n % NB]);
          wait_free(empty_x, n, NX);
          copy(smem + L::X + n % NX * TB * AUX, src + L::IMG, TB * AUX, &full_x[n % NX]);
        }
      }
    }
   } else {
    // Two warps issue, one the low bytes' MMAs and one the high bytes' (accumulators of their own): a stage's wait, its MMAs and its
    // commit take one warp longer than the tensor pipe needs for them.  Converged loops, one elected lane issues: addresses and
    // descriptors stay in uniform registers.
    const int high = warp - W_MMA;
    const uint32_t td = __shfl_sync(0xffffffffu, tmem, 0), sb = __shfl_sync(0xffffffffu, s32(smem + L::B), 0);
    const uint32_t idesc = high ? desc_i8<N, true>() : desc_i8<N, false>();
    int n = 0;
    for (int u = u_begin; u < u_end; ++u) {
      int first;
      const int nb = unit_blocks(u, P.blocks, first);
      wait_free(acc_empty, u - u_begin, 1);
      for (int k = 0; k < nb; ++k, ++n) {
        wait(full_b, n, NB);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int st = 2 * n + h;
          wait(full_a, st, NA);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (elect_one()) {
            const uint32_t ta = td + (uint32_t)(L::ACC + st % NA * L::A_COLS + 8 * high), acc = td + (uint32_t)(2 * N * k + N * high);
            const uint64_t db = smem_desc_u(sb + (uint32_t)(n % NB * L::IMG + h * (N * 128)));
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              const uint32_t more = h + s ? 1u : 0u;
              asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p; }"
                           ::"r"(acc), "r"(ta + 16 * s), "l"(db + 2 * s), "r"(idesc), "r"(more) : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(&empty_a[st % NA])) : "memory");
            if (h == 1) {
              asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(&empty_b[n % NB])) : "memory");
              if (k == nb - 1) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(acc_full)) : "memory");
            }
          }
          __syncwarp();
        }
      }
    }
   }
  }
  __syncthreads();
  if (warp == W_MMA) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// Activations -> records: a warp per (block, place in a token tile).  Places without an activation row are zero.
// A record's digits lie as the MMA reads them: two panels of 128 columns, a row of 128 bytes per plane (4 t + p), 16-byte chunks
// swizzled with the row number's low three bits.
__global__ void __launch_bounds__(256)
digit_records_kernel(const float* x, uint8_t* __restrict__ rec, int cols, int tokens, int tile, int places) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, place = (int)blockIdx.y * 8 + (threadIdx.x >> 5), b = blockIdx.x, blocks = gridDim.x;
  if (place >= places) return;
  const int tt = place / tile, t = place % tile, n = 4 * tile;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (place < tokens) {
    const float4* xp = (const float4*)(x + (int64_t)place * cols + b * 256 + 8 * lane);
    const float4 a = xp[0], c = xp[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
  }
  uint32_t pk[4][2];
  float sum, scale;
  mma::split_block(v, pk, sum, scale);
  uint8_t* r = rec + ((int64_t)tt * blocks + b) * (n * 256 + tile * AUX);
  const int panel = lane >> 4, chunk = (lane & 15) >> 1;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int row = 4 * t + p;
    *(uint2*)(r + panel * n * 128 + row * 128 + ((chunk ^ (row & 7)) << 4) + 8 * (lane & 1)) = make_uint2(pk[p][0], pk[p][1]);
  }
  float* aux = (float*)(r + n * 256 + t * AUX);
  if ((lane & 3) == 0) aux[lane >> 2] = sum;
  if (lane == 0) *(float4*)(aux + 8) = make_float4(scale, 0.f, 0.f, 0.f);
}

// The units' floats -> y: eight units of a part in order from zero, then the parts, as the reducer of the decode kernel adds them
__global__ void __launch_bounds__(256)
add_units_kernel(const float* part, float* __restrict__ y, int64_t n, int units) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float carry = 0.f;
    for (int u0 = 0; u0 < units; u0 += PART_UNITS) {
      float v[PART_UNITS];
#pragma unroll
      for (int w = 0; w < PART_UNITS; ++w) v[w] = u0 + w < units ? part[(int64_t)(u0 + w) * n + i] : 0.f;
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < PART_UNITS; ++w) s = __fadd_rn(s, v[w]);
      carry = u0 == 0 ? s : __fadd_rn(s, carry);
    }
    y[i] = carry;
  }
}

// Activation rows per tile: as few tiles as 24 rows each allow, the rows spread evenly over them (13 at least: I8_MIN_TOKENS)
int tile_rows(int64_t tokens) {
  const int64_t tiles = (tokens + 23) / 24, per = (tokens + tiles - 1) / tiles;
  return per > 16 ? 24 : 16;
}
// CTAs that share a tile's units.  More than one only where the row tiles leave most SMs idle: the units' floats then go through
// memory and a second kernel.
int unit_slices(const MatView& m, int64_t tokens) {
  const int tb = tile_rows(tokens), units = units_of((int)(m.cols / MACRO));
  const int64_t tiles = (m.rows + BM - 1) / BM * ((tokens + tb - 1) / tb);
  int s = 1;
  while (2 * s <= units && tiles * 2 * s <= 148) s *= 2;
  return s;
}
size_t record_bytes(const MatView& m, int64_t tokens) {
  const int tb = tile_rows(tokens);
  return (size_t)((tokens + tb - 1) / tb) * (size_t)(m.cols / MACRO) * (size_t)(4 * tb * 256 + tb * AUX);
}

template <int DT, int TB>
cudaError_t launch_tb(const MatView& m, const CUtensorMap& wmap, const Args& a, int slices, cudaStream_t stream, int* err) {
  auto kern = gemm_i8_kernel<DT, TB>;
  constexpr int smem = ILay<DT, TB>::TOTAL;
  static PerDevice ready;  // per instantiation
  std::atomic<int>& slot = ready.here();
  if (slot.load(std::memory_order_relaxed) == 0) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    slot.store(1, std::memory_order_relaxed);
  }
  const dim3 grid((unsigned)((m.rows + BM - 1) / BM), (unsigned)((a.tokens + TB - 1) / TB), (unsigned)slices);
  return launch_overlapped(kern, grid, THREADS, smem, stream, wmap, a, err);
}
template <int DT>
cudaError_t launch_dt(const MatView& m, const Args& a, int tb, int slices, cudaStream_t stream, int* err) {
  EncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return cudaErrorNotSupported;
  CUtensorMap wmap;  // packed weights as rows of 32-bit words; one box = 128 rows x the ring pitch
  const cuuint64_t dims[2] = {(cuuint64_t)(m.row_bytes / 4), (cuuint64_t)m.rows}, strides[1] = {(cuuint64_t)m.row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)(Pk<DT>::PITCH / 4), (cuuint32_t)BM}, estr[2] = {1, 1};
  if (enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, (void*)m.w, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  return tb == 24 ? launch_tb<DT, 24>(m, wmap, a, slices, stream, err) : launch_tb<DT, 16>(m, wmap, a, slices, stream, err);
}

}  // namespace

bool gemm_i8_supported(const MatView& m, int64_t tokens) {
  return (m.dtype == DT_Q4_K || m.dtype == DT_Q5_K || m.dtype == DT_Q6_K) && tokens >= I8_MIN_TOKENS && tokens <= I8_MAX_TOKENS && gemv_mma_supported(m);
}

size_t gemm_i8_scratch_bytes(const MatView& m, int64_t tokens) {
  const int s = unit_slices(m, tokens);
  return (record_bytes(m, tokens) + 255) / 256 * 256 + (s > 1 ? (size_t)units_of((int)(m.cols / MACRO)) * (size_t)tokens * (size_t)m.rows * 4 : 0);
}

cudaError_t launch_gemm_i8(const MatView& m, const float* x, float* y, int64_t tokens, void* scratch, cudaStream_t stream, int* err, uint64_t* launches, bool x_staged) {
  const int tb = tile_rows(tokens), tiles = (int)((tokens + tb - 1) / tb), blocks = (int)(m.cols / MACRO), slices = unit_slices(m, tokens);
  uint8_t* rec = (uint8_t*)scratch;
  float* part = (float*)(rec + (record_bytes(m, tokens) + 255) / 256 * 256);
  cudaError_t e = cudaSuccess;
  if (!x_staged) {
    e = launch_overlapped(digit_records_kernel, dim3((unsigned)blocks, (unsigned)((tiles * tb + 7) / 8)), 256, 0, stream, x, rec, (int)m.cols, (int)tokens, tb,
                          tiles * tb);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  const Args a{rec, slices > 1 ? part : y, (int)m.rows, blocks, (int)tokens};
  e = m.dtype == DT_Q4_K ? launch_dt<DT_Q4_K>(m, a, tb, slices, stream, err) : m.dtype == DT_Q5_K ? launch_dt<DT_Q5_K>(m, a, tb, slices, stream, err)
                                                                             : launch_dt<DT_Q6_K>(m, a, tb, slices, stream, err);
  if (e != cudaSuccess) return e;
  if (launches) ++*launches;
  if (slices > 1) {
    const int64_t n = tokens * m.rows;
    const int64_t grid = std::min<int64_t>((n + 255) / 256, 148 * 8);
    e = launch_overlapped(add_units_kernel, dim3((unsigned)grid), 256, 0, stream, (const float*)part, y, n, units_of(blocks));
    if (e == cudaSuccess && launches) ++*launches;
  }
  return e;
}

}  // namespace llr
