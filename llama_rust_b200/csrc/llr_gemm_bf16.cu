// Matrix products with bfloat16 weights for many activation rows on the 5th-generation tensor cores: both operands come
// through TMA into 128-byte swizzled shared memory, tcgen05.mma accumulates in tensor memory (f32), the epilogue reads the
// accumulators with tcgen05.ld.
//
//   y[t][z * rows + r] = sum_c W[z * rows + r][c] * x[t][z * xk + c]        z < batch
//
// With batch 1 this is the chunk form of gemm_f32_x for BF16 weights (langtax/src/quant.rs:6144, :6760); with more it is
// a product per head (a head's rows of W against that head's slice of the activation row).  Activations are bfloat16
// rows (x16); results are f32, or bfloat16 for the product that follows, optionally multiplied by the sigmoid of a
// per-head gate.
//
// With `glu` W stacks gate | up (2 rows rows) and the results are gated units: a tile then holds as many gate rows
// as up rows, so that a thread of the epilogue has both factors of each result.
//
// One CTA computes a tile of 128 or 256 activation rows x bn <= BN weight rows: the activation rows are the MMA's M dimension (one
// tensor-memory lane each), so that a thread of the epilogue holds consecutive results of one activation row and stores
// them as vectors.  One warp issues the TMA loads and one the MMAs; four read the accumulators, eight in wide tiles.  Tiles of 256 activation
// rows have a ring per operand, a warp of MMAs for each half and sixteen for the results.
// Two CTAs fit an SM at BN <= 128 (96 KB of stages, 128 columns of tensor memory each), so one tile's epilogue overlaps another's
// loads.  Wide tiles are bound by what the SMs draw from L2, so 256 activation rows share a stage's weights where that saves waves
// (tile_shape).  Up to 64 activation rows the product is a stream of weights: a stage then holds 32 or 64 activation rows (the MMA
// reads on into the weights behind them: rows of its result that nobody looks at), tiles of 32 .. 128 weight rows spread it over the SMs
// (stream_width) and up to sixteen stages of it are under way; plain results of 33 rows and more against very many weight rows go by whole
// tiles again (launch_gemm_bf16).  16384 x 2048 gated, 32 rows: 25 -> 18 us.  A K range may be cut into
// slices (gridDim.z): slice s leaves its partial sums at y + s * slice_stride and the reader adds them in slice order.  Every wait is
// bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "llr_formats.cuh"
#include "llr_kernels.cuh"
#include "llr_tmap.cuh"
#include "llr_umma.cuh"

namespace llr {
namespace {

using umma::bar_expect;
using umma::bar_init;
using umma::bar_wait;
using umma::bar_wait2;
using umma::elect_one;
using umma::DESC_HI;  // operand tiles are K-major 128-byte swizzled rows, eight-row groups 1024 bytes apart
using umma::s32;

constexpr int BM = 128;  // activation rows per MMA = UMMA M
constexpr int BK = 64;   // columns per stage: one 128-byte swizzle row

// RT: tiles of BM activation rows per CTA; 0: at most 64 activation rows, stages and their number by the launch
template <int BN, int RT> struct Lay {
  static constexpr int A_STAGE = RT * BM * 128, B_STAGE = BN * 128, STAGE = A_STAGE + B_STAGE;
  static constexpr int NS = RT == 0 ? 16 : RT == 2 ? 8 : BN == 256 ? 4 : BN == 128 ? 3 : 4;  // 192, 96, 96 KB
  static constexpr int NB = 4;  // two tiles of activation rows: stages of weights, beside a ring of at most NS single tiles
  static constexpr int EPI = BN < 256 ? 4 : RT == 2 ? 16 : 8, W_TMA = EPI, W_MMA = EPI + 1, THREADS = (EPI + 2 + (RT == 2)) * 32;  // epilogue warps first
  static constexpr int TOTAL = RT == 2 ? umma::SMEM_LIMIT : 1024 /*alignment*/ + NS * STAGE + 512;
  static constexpr int TMEM_COLS = RT == 0 ? BN : RT * BN;
};

// kind::f16: f32 accumulator, both operands bfloat16, M = 128, N = bn
__device__ __forceinline__ uint32_t mma_desc(int bn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

struct Args {
  float* y;
  __nv_bfloat16* y16;
  const float* gate;   // gate[t * gate_ld + z]: results times its sigmoid
  int64_t y_ld, gate_ld, slice_stride;
  int tokens, rows, nk, xk;  // nk: 64-column steps of the whole K range
  int batch, slices, bn;
  int a_rows, stages;  // activation rows of a stage, stages (RT 0)
  GluShape glu;
};

// 32 accumulator columns of this warp's 32 lanes
__device__ __forceinline__ void load32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr) : "memory");
}

__device__ __forceinline__ void load8(uint32_t taddr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr) : "memory");
}

// operands by the low words of their descriptors
__device__ __forceinline__ void mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t add) {
  asm volatile("{ .reg .pred p; .reg .b64 a, b; setp.ne.b32 p, %5, 0; mov.b64 a, {%1, %3}; mov.b64 b, {%2, %3}; "
               "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p; }"
               ::"r"(d), "r"(a), "r"(b), "r"(DESC_HI), "r"(idesc), "r"(add) : "memory");
}

template <int BN, int RT, bool GLU>
__global__ void __launch_bounds__(Lay<BN, RT>::THREADS)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const Args a, int* __restrict__ err) {
  using L = Lay<BN, RT>;
  constexpr int W_TMA = L::W_TMA, W_MMA = L::W_MMA;
  constexpr bool STREAM = RT == 0, PAIR = RT == 2;
  const int NS = STREAM || PAIR ? a.stages : L::NS, A_STAGE = STREAM ? a.a_rows * 128 : L::A_STAGE, STAGE = STREAM ? A_STAGE + a.bn * 128 : L::STAGE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // behind the stages, and behind what the last one's MMA reads past its activation rows
  uint64_t* full = (uint64_t*)(smem + (PAIR ? NS * BM * 128 + L::NB * a.bn * 128 : NS * STAGE + (STREAM ? BM * 128 : 0)));
  uint64_t* empty = full + L::NS;
  uint64_t* full_b = empty + L::NS;  // PAIR: of the weights' ring
  uint64_t* empty_b = full_b + L::NB;
  uint64_t* done = empty_b + L::NB;
  uint32_t* tmem_slot = (uint32_t*)(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bn = a.bn, width = GLU ? bn / 2 : bn;  // results per activation row of the tile
  // token tiles run fastest: the CTAs that share weight rows run at the same time, and the weights are read from HBM once
  const int row0 = blockIdx.y * width, tok0 = blockIdx.x * ((STREAM ? 1 : RT) * BM);
  const int z = (int)blockIdx.z / a.slices, slice = (int)blockIdx.z % a.slices;
  const int per = (a.nk + a.slices - 1) / a.slices, k0 = slice * per, k1 = min(a.nk, k0 + per);  // never empty: the launcher sees to it

  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; ++s) { bar_init(&full[s], 1); bar_init(&empty[s], 1); }
    if (PAIR)
      for (int s = 0; s < L::NB; ++s) { bar_init(&full_b[s], 1); bar_init(&empty_b[s], 2); }
    bar_init(done, PAIR ? 2 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(L::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // only now: a dependent that is placed here finds its tensor memory after this block has its own, and does not wait with it for this grid
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  bool ok = true;

  if (PAIR && warp == W_TMA) {
    // Two rings: weights four steps deep, tiles of 128 activation rows three or four for each half.  Stages of both tiles and the weights together were three
    // (64 KB each), and a place that is free only once all eight MMAs of a step are done came back late: steps of 0.62 us instead of 0.47.
    const uint32_t base = __shfl_sync(0xffffffffu, s32(smem), 0), base_b = base + (uint32_t)(NS * BM * 128);
    auto load_w = [&](int k, int s) {
      bar_expect(&full_b[s], (uint32_t)(bn * 128));  // boxes are always complete: what lies outside the matrices is filled with zeros
      asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                   ::"r"(base_b + (uint32_t)(s * bn * 128)), "l"(&wmap), "r"(k * BK), "r"(z * a.rows + row0), "r"(s32(&full_b[s])) : "memory");
      if constexpr (GLU)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(base_b + (uint32_t)(s * bn * 128 + width * 128)), "l"(&wmap), "r"(k * BK), "r"(a.rows + row0), "r"(s32(&full_b[s])) : "memory");
    };
    const bool leader = elect_one();
    const int ahead = min(L::NB, k1 - k0);
    if (leader)
      for (int s = 0; s < ahead; ++s) load_w(k0 + s, s);
    __syncwarp();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint32_t s = 0, lap = 0, sb = 0, lb = 0;
    for (int k = k0; k < k1; ++k) {
      if (k - k0 >= ahead) {
        if (ok && !bar_wait(&empty_b[sb], lb ^ 1)) { ok = false; report_error(err, 5); }
        if (ok && leader) load_w(k, (int)sb);
      }
      if (++sb == (uint32_t)L::NB) { sb = 0; lb ^= 1; }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (ok && !bar_wait(&empty[s], lap ^ 1)) { ok = false; report_error(err, 5); }
        if (ok && leader) {
          bar_expect(&full[s], BM * 128);
          asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                       ::"r"(base + s * (uint32_t)(BM * 128)), "l"(&xmap), "r"(z * a.xk + k * BK), "r"(tok0 + BM * r), "r"(s32(&full[s])) : "memory");
        }
        if (++s == (uint32_t)NS) { s = 0; lap ^= 1; }
      }
    }
    __syncwarp();
  } else if (PAIR && (warp == W_MMA || warp == W_MMA + 1)) {
    // A warp per tile of activation rows: asking a barrier takes 100 ns, and the tensor pipe holds no more than a few MMAs ready, so that one
    // thread that asks for weights and two tiles in turn leaves it idle in between (steps of 0.65 us instead of 0.47).
    const int r = warp - W_MMA;
    const uint32_t idesc = mma_desc(bn), td = __shfl_sync(0xffffffffu, tmem, 0) + (uint32_t)(r * BN), base = __shfl_sync(0xffffffffu, s32(smem), 0) >> 4;
    const uint32_t base_b = base + (uint32_t)(NS * BM * 128 / 16);
    const bool leader = elect_one();
    int s = r, sb = 0;
    uint32_t lap = 0, lb = 0;
    for (int k = k0; k < k1; ++k) {
      if (ok && !bar_wait2(&full_b[sb], lb, &full[s], lap)) { ok = false; report_error(err, 5); }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (leader) {
        const uint32_t la = base + (uint32_t)(s * (BM * 128 / 16)), lw = base_b + (uint32_t)(sb * (bn * 128 / 16)), first = k > k0 ? 1u : 0u;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) mma(td, la + (uint32_t)(2 * kk), lw + (uint32_t)(2 * kk), idesc, kk > 0 ? 1u : first);
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(&empty[s])) : "memory");
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(&empty_b[sb])) : "memory");
      }
      if ((s += 2) >= NS) { s -= NS; lap ^= 1; }
      if (++sb == L::NB) { sb = 0; lb ^= 1; }
    }
    if (leader)
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(done)) : "memory");
    __syncwarp();
  } else if (warp == W_TMA) {
    const uint32_t base = __shfl_sync(0xffffffffu, s32(smem), 0);
    auto load_w = [&](int k, int s) {
      bar_expect(&full[s], (uint32_t)(A_STAGE + bn * 128));  // boxes are always complete: what lies outside the matrices is filled with zeros
      asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                   ::"r"(base + (uint32_t)(s * STAGE + A_STAGE)), "l"(&wmap), "r"(k * BK), "r"(z * a.rows + row0), "r"(s32(&full[s])) : "memory");
      if constexpr (GLU)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(base + (uint32_t)(s * STAGE + A_STAGE + width * 128)), "l"(&wmap), "r"(k * BK), "r"(a.rows + row0), "r"(s32(&full[s])) : "memory");
    };
    // the first stages' weights are on their way while the kernel before this one still runs; its results are waited for
    const int ahead = min(NS, k1 - k0);
    for (int s = 0; s < ahead; ++s) {
      if (elect_one()) load_w(k0 + s, s);
      __syncwarp();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool leader = elect_one();
    uint32_t s = 0, lap = 0;
    for (int k = k0; k < k1; ++k) {
      if (ok && !bar_wait(&empty[s], lap ^ 1)) { ok = false; report_error(err, 5); }
      if (ok && leader) {
        if (k - k0 >= ahead) load_w(k, (int)s);
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(base + s * (uint32_t)STAGE), "l"(&xmap), "r"(z * a.xk + k * BK), "r"(tok0), "r"(s32(&full[s])) : "memory");
      }
      if (++s == (uint32_t)NS) { s = 0; lap ^= 1; }
    }
    __syncwarp();
  } else if (warp == W_MMA) {
    // One thread issues, and what it needs per step is kept ready: a step of four MMAs of N = 128 takes 256 cycles, and with a division
    // for its stage, an election and 64-bit descriptors the step took 600.
    const uint32_t idesc = mma_desc(bn), td = __shfl_sync(0xffffffffu, tmem, 0), base = __shfl_sync(0xffffffffu, s32(smem), 0) >> 4;
    const bool leader = elect_one();
    uint32_t s = 0, lap = 0, lo = base;  // low words of the operands' descriptors: addresses below 2^18, in units of 16 bytes
    for (int k = k0; k < k1; ++k) {
      if (ok && !bar_wait(&full[s], lap)) { ok = false; report_error(err, 5); }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (leader) {
        const uint32_t lb = lo + (uint32_t)(A_STAGE / 16), first = k > k0 ? 1u : 0u;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) mma(td, lo + (uint32_t)(2 * kk), lb + (uint32_t)(2 * kk), idesc, kk > 0 ? 1u : first);
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(&empty[s])) : "memory");
      }
      lo += (uint32_t)(STAGE / 16);
      if (++s == (uint32_t)NS) { s = 0; lap ^= 1; lo = base; }
    }
    if (leader)
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(done)) : "memory");
    __syncwarp();
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");  // gates; results may still be read by an earlier kernel
    if (!bar_wait(done, 0)) { ok = false; report_error(err, 5); }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int n_live = min(width, a.rows - row0);
    // The code of an epilogue runs once per block, cold: straight-line gated units for 32 columns took 8 us to fetch (28672 x 4096
    // gated, 512 rows: 118 -> 107 us with eight).  Few columns per
    // round, and a stream of weights, whose results lie in one or two warps' lanes, spreads them over all four through shared memory.
    if constexpr (STREAM) {
      float* turn = (float*)smem;  // every stage has been read
      const int pitch = bn + 1;
      float g[2] = {1.f, 1.f};  // gates of tokens lane, 32 + lane
      if (a.gate) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
          if (32 * k + lane < a.tokens) g[k] = 1.0f / (1.0f + expf(-a.gate[(int64_t)(32 * k + lane) * a.gate_ld + z]));
      }
      if (32 * warp < a.a_rows) {
#pragma unroll 1
        for (int c0 = 0; c0 < bn; c0 += 32) {
          uint32_t v[32];
          load32(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c0, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c0 + j < bn) turn[(32 * warp + lane) * pitch + c0 + j] = __uint_as_float(v[j]);
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * L::EPI) : "memory");
#pragma unroll 1
      for (int t = warp; t < a.tokens; t += L::EPI) {
        const float gate = __shfl_sync(~0u, t < 32 ? g[0] : g[1], t & 31);
        const int64_t off = (int64_t)t * a.y_ld + (int64_t)z * a.rows + row0;
#pragma unroll 1
        for (int c = lane; c < n_live; c += 32) {
          float f = turn[t * pitch + c];
          if constexpr (GLU) f = gated_unit(f, turn[t * pitch + width + c], a.glu);
          else f = a.gate ? f * gate : f;
          if (a.y) a.y[slice * a.slice_stride + off + c] = f;
          if (a.y16) a.y16[off + c] = __float2bfloat16_rn(f);
        }
        __syncwarp();
      }
    } else {
      // warps 4.. read the second tile of activation rows, the next four or eight every other run of columns
      constexpr int W = GLU ? 8 : 16;  // columns of a round: plain results are short code, and eight cost 65 rows 3 % (2048 columns, 2048 weight rows 23.1 -> 22.0 us)
      const int r = PAIR ? (warp >> 2) & 1 : 0, t = tok0 + BM * r + 32 * (warp & 3) + lane;
      constexpr int C_STEP = W * L::EPI / (4 * RT);
      const int64_t off = (int64_t)t * a.y_ld + (int64_t)z * a.rows + row0;
      float* y = a.y ? a.y + slice * a.slice_stride + off : nullptr;
      __nv_bfloat16* y16 = a.y16 ? a.y16 + off : nullptr;
      float gate = 1.f;
      if (a.gate && t < a.tokens) gate = 1.0f / (1.0f + expf(-a.gate[(int64_t)t * a.gate_ld + z]));
      const bool vec = ((a.y_ld | a.rows) & 7) == 0;  // every run of eight results starts on a 16-byte boundary in either format
      const uint32_t taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(r * BN);
      const int c_first = W * (warp / (4 * RT));
      uint32_t v[2][W], u[2][W];  // the next round's are on their way while one is worked on
      auto fetch = [&](int c0, int k) {
#pragma unroll
        for (int j = 0; j < W; j += 8) {
          load8(taddr + (uint32_t)(c0 + j), v[k] + j);
          if constexpr (GLU) load8(taddr + (uint32_t)(width + c0 + j), u[k] + j);
        }
      };
      auto finish = [&](int c0, int k) {
        if (t >= a.tokens) return;
        float f[W];
#pragma unroll
        for (int j = 0; j < W; ++j) {
          if constexpr (GLU) f[j] = gated_unit(__uint_as_float(v[k][j]), __uint_as_float(u[k][j]), a.glu);
          else f[j] = a.gate ? __uint_as_float(v[k][j]) * gate : __uint_as_float(v[k][j]);
        }
        if (vec) {  // rows is a multiple of eight here
#pragma unroll
          for (int j = 0; j < W; j += 8)
            if (c0 + j < n_live) {
              if (y) {
                *(float4*)(y + c0 + j) = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
                *(float4*)(y + c0 + j + 4) = make_float4(f[j + 4], f[j + 5], f[j + 6], f[j + 7]);
              }
              if (y16) {
                __nv_bfloat162 h[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[j + 2 * i], f[j + 2 * i + 1]);
                *(uint4*)(y16 + c0 + j) = *(const uint4*)h;
              }
            }
        } else {
#pragma unroll
          for (int j = 0; j < W; ++j)
            if (c0 + j < n_live) {
              if (y) y[c0 + j] = f[j];
              if (y16) y16[c0 + j] = __float2bfloat16_rn(f[j]);
            }
        }
      };
      if (c_first < n_live) fetch(c_first, 0);
#pragma unroll 1
      for (int c0 = c_first; c0 < n_live; c0 += 2 * C_STEP) {
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + C_STEP < n_live) fetch(c0 + C_STEP, 1);
        finish(c0, 0);
        __syncwarp();
        if (c0 + C_STEP < n_live) {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (c0 + 2 * C_STEP < n_live) fetch(c0 + 2 * C_STEP, 0);
          finish(c0 + C_STEP, 1);
          __syncwarp();
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == W_MMA) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS) : "memory");
  }
}

bool encode_rows(CUtensorMap* map, const void* base, int64_t cols, int64_t rows, int64_t ld, int box_rows) {
  EncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  const cuuint32_t one[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A stream's shared memory: alignment, stages, what the last stage's MMA reads past its activation rows, barriers.  Two blocks share an SM's
// 228 KB, of which each takes a kilobyte unasked: 95 KB of stages, three at the widest (four there left one block per SM, 18432 x 4096
// gated, 64 rows: 86 -> 74 us; one block with the full ring 82).
constexpr int STREAM_REST = 1024 + BM * 128 + 512, STREAM_STAGES = 200 * 1024, STREAM_STAGES_OF_TWO = 228 * 1024 / 2 - 1024 - STREAM_REST;
constexpr int STREAM_SMEM = STREAM_STAGES + STREAM_REST;
static_assert(STREAM_STAGES_OF_TWO / ((64 + 128) * 128) >= 3, "a ring");

template <int BN, int RT, bool GLU>
cudaError_t launch_tiles(const Bf16Product& p, const Args& a, cudaStream_t stream, int* err) {
  CUtensorMap xmap, wmap;
  const int width = GLU ? a.bn / 2 : a.bn;  // rows of one box of W
  if (!encode_rows(&xmap, p.x16, p.x_cols, p.tokens, p.x_ld, RT == 0 ? a.a_rows : BM) || !encode_rows(&wmap, p.w, p.cols, (int64_t)p.rows * (GLU ? 2 : p.batch), p.cols, width))
    return cudaErrorInvalidValue;
  const int smem = RT == 0 ? a.stages * (a.a_rows + a.bn) * 128 + STREAM_REST : RT == 2 ? 1024 + (a.stages * BM + Lay<BN, RT>::NB * a.bn) * 128 + 512 : Lay<BN, RT>::TOTAL;
  static PerDevice ready;
  std::atomic<int>& slot = ready.here();
  if (slot.load(std::memory_order_relaxed) == 0) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_bf16_kernel<BN, RT, GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, RT == 0 ? STREAM_SMEM : Lay<BN, RT>::TOTAL);
    if (e != cudaSuccess) return e;
    slot.store(1, std::memory_order_relaxed);
  }
  constexpr int TOK = RT == 0 ? BM : RT * BM;
  const dim3 grid((unsigned)((p.tokens + TOK - 1) / TOK), (unsigned)((p.rows + width - 1) / width), (unsigned)(p.batch * a.slices));
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidValue;
  return launch_overlapped(gemm_bf16_kernel<BN, RT, GLU>, grid, Lay<BN, RT>::THREADS, smem, stream, xmap, wmap, a, err);
}

// Two tiles of activation rows: single tiles in their ring, as many as fit beside the weights, an EVEN number.  The halves take the places in
// turn, and a barrier says no more than the parity of its phase: a half that shared a place with the other and got ahead of it by a lap --
// copies need not arrive in order -- would take the phase of two laps ago for its own, multiply a tile that is not there and free it twice.
constexpr int pair_stages(int bn) { return std::min(8, (Lay<256, 2>::TOTAL - 1024 - 512 - Lay<256, 2>::NB * bn * 128) / (BM * 128)) & ~1; }
constexpr bool even_rings() {
  for (int bn = 160; bn <= 256; bn += 16)
    if (pair_stages(bn) % 2 != 0 || pair_stages(bn) < 4) return false;
  return true;
}
static_assert(even_rings(), "a place of the ring belongs to one half");

constexpr int SMS = 148;
int tiles_of(int tokens, int rows, int batch, int bn, int rt = 1) { return ((tokens + rt * BM - 1) / (rt * BM)) * ((rows + bn - 1) / bn) * batch; }
// Shape of a tile.  Few tiles: 128 or 64 weight rows.  Many: 160 .. 256 weight rows (a multiple of `step`, so that both halves of a
// gated tile are whole eight-row groups) and one or two tiles of 128 activation rows, for which the waves over the SMs cost least.
// What a wave costs was measured at 4096 columns, 512 activation rows: 27 / 31 / 33 us with 160 / 224 / 256 weight rows, 43 / 54 /
// 58 us with two tiles of activation rows (50 at 224 since those have two rings, an issuing thread each and sixteen warps for
// results).  The stages come from L2 at about 50 bytes a cycle and SM, which is what bounds a wave; the second tile of activation rows
// uses a stage's weights again.  28672 x 4096: 126 -> 111 us (107 with the short epilogue, 101 with two rings), 16384 x 2048: 54 -> 44,
// 10240 x 4096: 64 -> 54, and with the wide tile from 120 tiles on (132 before) 8192 x 4096: 43 -> 39.
struct Tile { int bn, rt; };
Tile tile_shape(int tokens, int rows, int batch, int step = 16) {
  if (tiles_of(tokens, rows, batch, 256) < 120) return {rows > 64 ? 128 : 64, 1};
  Tile best{256, 1};
  int cost = 1 << 30;
  for (int rt = 1; rt <= 2; ++rt)
    for (int bn = 256; bn >= 160; bn -= step) {
      const int c = (tiles_of(tokens, rows, batch, bn, rt) + SMS - 1) / SMS * (rt == 1 ? 5 * bn + 1410 : 12 * bn + 1640);
      if (c < cost) { cost = c; best = {bn, rt}; }
    }
  return best;
}

// At most 64 activation rows: the width of a tile, for which the weights an SM draws (in waves of a tile per SM, the activations of a
// tile at half their bytes: they come from L2) are fewest.  The stages then fill an SM's shared memory, or half of it where blocks share one.
constexpr int STREAM_TOKENS = 64;
int stream_width(int tokens, int rows, int batch, int slices) {
  int best = 128;
  int64_t cost = INT64_MAX;
  for (int bn = 128; bn >= 32; bn -= 16) {
    const int64_t waves = ((int64_t)tiles_of(tokens, rows, batch, bn) * slices + SMS - 1) / SMS, c = waves * (bn + (tokens > 32 ? 32 : 16));
    if (c < cost) { cost = c; best = bn; }
  }
  return best;
}

}  // namespace

bool gemm_bf16_supported(const void* w, int64_t rows, int64_t cols) {
  return rows > 0 && rows < (1 << 28) && cols > 0 && cols < (1 << 28) && cols % 8 == 0 && ((uintptr_t)w & 15) == 0;
}

// K slices of a product without heads: as many as keep the grid within one wave of two CTAs per SM, every slice at
// least 512 columns long
int gemm_bf16_slices(int tokens, int rows, int cols) {
  const int bn = tile_shape(tokens, rows, 1).bn;
  if (bn > 128) return 1;
  const int tiles = tiles_of(tokens, rows, 1, bn), nk = (cols + BK - 1) / BK;
  int s = 1;
  while (s < 8 && tiles * s * 2 <= 296 && nk / (s * 2) >= 8) s *= 2;
  while (s > 1 && (s - 1) * ((nk + s - 1) / s) >= nk) s /= 2;  // no empty slice
  return s;
}

cudaError_t launch_gemm_bf16(const Bf16Product& p, cudaStream_t stream, int* err, uint64_t* launches) {
  if (p.tokens <= 0) return cudaSuccess;
  if (!gemm_bf16_supported(p.w, p.rows, p.cols) || p.batch < 1 || p.x_ld % 8 != 0 || (p.batch > 1 && p.xk % 8 != 0) || ((uintptr_t)p.x16 & 15) != 0 ||
      (((uintptr_t)p.y | (uintptr_t)p.y16) & 15) != 0 || p.slices < 1 || (p.slices > 1 && (p.batch != 1 || p.y16 || p.gate || p.glu)) ||
      (p.glu && (p.batch != 1 || p.gate)))
    return cudaErrorInvalidValue;
  Args a{};
  a.y = p.y; a.y16 = (__nv_bfloat16*)p.y16; a.gate = p.gate;
  a.y_ld = p.y_ld; a.gate_ld = p.gate_ld; a.slice_stride = p.slice_stride;
  a.tokens = p.tokens; a.rows = p.rows; a.nk = (p.cols + BK - 1) / BK; a.xk = p.xk;
  a.batch = p.batch; a.slices = p.slices;
  if ((a.slices - 1) * ((a.nk + a.slices - 1) / a.slices) >= a.nk) return cudaErrorInvalidValue;
  if (launches) ++*launches;
  if (p.glu) a.glu = *p.glu;
  // Plain results of 33 to 64 rows leave the stream at one and a half tiles of 128 weight rows per SM: what the tiles then write is no longer
  // hidden behind weights (4096 columns, 64 rows, streamed and not: 24576 weight rows 56.1 / 56.5 us, 28672 62.9 / 61.7, 128256 205.6 / 196.7).
  // Gated units, half as many, stay (128256: 206 / 203, and 1 to 8 % faster streamed everywhere below).
  if (p.tokens <= 32 || (p.tokens <= STREAM_TOKENS && (p.glu || 2 * tiles_of(p.tokens, p.rows, p.batch, 128) <= 3 * SMS))) {
    a.bn = stream_width(p.tokens, p.rows * (p.glu ? 2 : 1), p.batch, p.slices);
    a.a_rows = p.tokens > 32 ? 64 : 32;
    const bool alone = (int64_t)tiles_of(p.tokens, p.rows * (p.glu ? 2 : 1), p.batch, a.bn) * p.slices <= SMS;
    a.stages = std::min(16, (alone ? STREAM_STAGES : STREAM_STAGES_OF_TWO) / ((a.a_rows + a.bn) * 128));
    return p.glu ? launch_tiles<128, 0, true>(p, a, stream, err) : launch_tiles<128, 0, false>(p, a, stream, err);
  }
  if (p.glu) {
    const Tile tile = tile_shape(p.tokens, 2 * p.rows, 1, 32);
    a.bn = std::max(tile.bn, 128);
    a.stages = pair_stages(a.bn);
    return tile.rt == 2 ? launch_tiles<256, 2, true>(p, a, stream, err) : a.bn > 128 ? launch_tiles<256, 1, true>(p, a, stream, err)
                                                                                     : launch_tiles<128, 1, true>(p, a, stream, err);
  }
  const Tile tile = tile_shape(p.tokens, p.rows, p.batch);
  a.bn = tile.bn;
  a.stages = pair_stages(a.bn);
  if (tile.rt == 2) return launch_tiles<256, 2, false>(p, a, stream, err);
  if (a.bn > 128) return launch_tiles<256, 1, false>(p, a, stream, err);
  return a.bn == 128 ? launch_tiles<128, 1, false>(p, a, stream, err) : launch_tiles<64, 1, false>(p, a, stream, err);
}

}  // namespace llr
