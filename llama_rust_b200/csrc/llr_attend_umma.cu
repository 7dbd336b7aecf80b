// Prompt attention on the 5th-generation tensor cores: rows of ONE sequence at consecutive positions against the keys and values
// they see, grouped-query heads or one latent for every head.
//
// The keys and values that any row of a group sees are first gathered from their pages into contiguous binary16 rows
// (span_gather_kernel), which TMA then copies as 128-byte swizzled tiles.  A block takes one kv head and 128 (row, query head) pairs in
// row-major order -- all query heads of a kv head share its keys, so any ratio of heads fills the tile -- and walks the keys
// that any of its rows sees, NK at a time:
//   scores   S = Q K^T      tcgen05.mma, Q and K from shared memory (K-major), f32 accumulators in tensor memory, two buffers
//   weights  P = 2^(S - m)  one pair per lane of tensor memory; binary16 back into tensor memory (SPLIT: and the rest)
//   sums     O += P V       tcgen05.mma, P from tensor memory, V from shared memory as it lies (dimensions run fastest: MN-major)
// Queries (rescaled per pair by a power of two), keys, values and the exponentials are binary16 operands; scores and sums are f32;
// scale, distance bias, mask, maxima, exponentials and their sums are f32.
//
// The weights lie where the scores lay.  The reference m of a row moves only when the row's maximum has grown by more than 8 (a factor
// of 256: exponentials stay far inside binary16's range), so O is rarely read back and rescaled.  (That, and two sets of warps that take
// turns, are published for attention on this chip and the one before: FlashAttention-4 and -3.)  Two schedules:
//   values of at most 128 dimensions, NK = 128: four warps take the even steps, four the odd ones, either four with sums and references
//     of their own that meet at the end; while one set waits for the tensor cores the other has the exponentials (eight warps a step, half
//     of its keys each, took 2.0 us a step instead of 1.2: the registers then hold too little)
//   more, NK = 64: eight warps a step, half of its keys each.  A block has 256 value dimensions and blocks of the other parts form the
//     scores again: 1.5 times the operations of one pass with a latent of 512, whose sums would leave no column for scores.  The first
//     256 columns of the queries are operands in tensor memory, which leaves a ring of two and a half steps (with all of them in shared
//     memory the ring held a step and a half, and a step took 2.9 us, most of it waiting for copies).
// Keys and values come through a ring of chunk pairs, 2 x [NK keys][64 dimensions], one pair of barriers each (a chunk alone is four
// MMAs of 45 to 64 cycles: waiting for its barrier and freeing it took 460); where values are the keys, a block reads the pairs of its own
// dimensions last and keeps them until the sums have used them.
//
// Bound: the exponentials (16 a cycle and SM) and the MMAs, 1024 cycles each per 128 keys of 128 dimensions; for a latent of 512 the
// scores' operand traffic in shared memory.  The code is kept short (scores are masked and biased by rolled loops over 32 of them, in
// place): a launch finds the instruction caches cold, and straight-line code then runs at eight instructions in 50 ns.  Unrolled,
// steps with masks or biases took 5 to 9 us instead of one, and a pass over the results 12.
// Weights rounded to binary16 are a third of the error where scores are spread by a nat.  A reference per slice (four runs of 32 keys on
// mma.sync) rounded more of the large ones to 1; with two references for all keys the Llama walk was further from 64 bits (512 rows, 4 heads of 128
// over one, scores spread by 1 / 2 / 3 nats: 3.39 / 4.90 / 5.72e-4 -> 3.43 / 4.94 / 5.75e-4).  So there (SPLIT) a weight is two binary16 numbers, it
// and what rounding has left of it, in the 32 columns of the scores of its 32 keys, and the second product has two MMAs for one: 3.15 / 4.83 /
// 5.69e-4, which is what rounding queries, keys and values costs; a launch of the walk, 512 rows, 32 heads of 128 over 8, 20.9 -> 21.0 us.  Layered decoders, whose
// products are bfloat16, are as far from 64 bits either way (1.573e-3, 1.574e-3).
// Measured, one launch: 2048 pairs x 8 kv heads of 128 dimensions, 1500 keys, window 1024, biases and gates 100 -> 35 us (mma.sync, 64
// pairs a block, before); 512 rows x 32 heads, latent of 512, window 1024 169 -> 75 us.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cfloat>

#include "llr_attend.cuh"
#include "llr_kernels.cuh"
#include "llr_tmap.cuh"
#include "llr_umma.cuh"

namespace llr {
namespace {

using umma::bar_arrive;
using umma::bar_expect;
using umma::bar_init;
using umma::bar_wait;
using umma::elect_one;
using umma::DESC_HI;
using umma::s32;

__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *(const uint32_t*)&h;
}
__device__ __forceinline__ float exp2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The list of keys a group of rows sees: kept tokens before the first row's window, then every position from there to the
// last row.
struct GroupKeys {
  int lo, nk, n;
  __device__ __forceinline__ int at(int m) const { return m < nk ? m : lo + m - nk; }
  __device__ __forceinline__ int index(int j) const { return j < nk ? j : j - lo + nk; }  // of a position in the list
};
__device__ __forceinline__ GroupKeys group_keys(int first, int rows, int window, int keep_first) {
  const int lo = window > 0 ? max(0, first - window + 1) : 0, nk = min(keep_first, lo);
  return GroupKeys{lo, nk, nk + first + rows - lo};
}

// The groups of one launch: group i has the rows [t0, t0 + rows), blocks [keys_at[i], keys_at[i + 1]) of the gather and
// [tiles_at[i], tiles_at[i + 1]) of the attention.  Row m of the gathered keys of kv head h is row row0 + h * keys + m of the
// matrix of all keys (of all values): the groups follow each other in it.  A group alone fills a few SMs (a prompt of 24 rows:
// eight blocks), and a ragged batch has dozens: with a launch each, 24 groups of 30 rows took 16 x (5 + 30) us per layer one
// after the other.
constexpr int SPAN_GROUPS = 64;
struct SpanBatch {
  int n;
  int t0[SPAN_GROUPS], rows[SPAN_GROUPS], keys[SPAN_GROUPS], row0[SPAN_GROUPS], keys_at[SPAN_GROUPS + 1], tiles_at[SPAN_GROUPS + 1];
};
__device__ __forceinline__ int span_group(const int* at, int n, int block) {
  int i = 0;
  while (i + 1 < n && block >= at[i + 1]) ++i;
  return i;
}

// One warp per key row: grid (keys / 8 of all groups, kv head).  What is not a number must reach the rows that see it and no others, but a
// masked weight of zero times an infinity is not zero.  So where a value is not finite as binary16 the row's KEY says so: scores that do
// not see it are masked by selection, those that do make their whole row not a number.  A latent is both operands at once and is bounded
// instead, NaN included.  With that, every value that a tile reads behind its last key -- another head's, another group's, zeros
// behind the last -- is finite and meets a weight of zero.
__global__ void __launch_bounds__(256)
span_gather_kernel(SpanShape sh, LayerKv kv, RowMap rows, const __grid_constant__ SpanBatch b, __half* __restrict__ k16, __half* __restrict__ v16) {
  pdl_enter();
  const int gi = span_group(b.keys_at, b.n, blockIdx.x), t0 = b.t0[gi];
  const GroupKeys gk = group_keys(row_position(rows, t0), b.rows[gi], sh.window, sh.keep_first);
  const int m = (blockIdx.x - b.keys_at[gi]) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, head = blockIdx.y, seq = row_sequence(rows, t0);
  if (m >= b.keys[gi]) return;
  const int64_t row = (int64_t)b.row0[gi] + (int64_t)head * b.keys[gi] + m;
  const bool latent = v16 == nullptr;
  const int j = gk.at(m);
  const int64_t page = kv.table[(int64_t)seq * kv.max_blocks + j / kv.block_tokens], in_page = (int64_t)head * kv.block_tokens + j % kv.block_tokens;
  const float* ks = kv.k + page * kv.k_block + in_page * sh.dk;
  auto operand = [&](float x) { return latent || (sh.saturate && fabsf(x) <= FLT_MAX) ? fminf(fmaxf(x, -65504.f), 65504.f) : x; };
  auto words = [&](const float* src) {  // dk and dv are multiples of eight
    const float4 x = *(const float4*)src;
    return make_uint2(pack_h2(operand(x.x), operand(x.y)), pack_h2(operand(x.z), operand(x.w)));
  };
  for (int i = 4 * lane; i < sh.dk; i += 128) *(uint2*)(k16 + row * sh.dk + i) = words(ks + i);
  if (latent) return;
  bool special = false;
  auto finite = [&](uint32_t w) {
    const bool not_finite = (w & 0x7c00u) == 0x7c00u || (w & 0x7c000000u) == 0x7c000000u;
    special |= not_finite;
    return not_finite ? 0u : w;
  };
  const float* vs = kv.v + page * kv.v_block + in_page * sh.dv;
  for (int i = 4 * lane; i < sh.dv; i += 128) {
    const uint2 w = words(vs + i);
    *(uint2*)(v16 + row * sh.dv + i) = make_uint2(finite(w.x), finite(w.y));
  }
  if (__any_sync(~0u, special))  // the same lanes wrote the key
    for (int i = 4 * lane; i < sh.dk; i += 128) *(uint2*)(k16 + row * sh.dk + i) = make_uint2(0x7fff7fffu, 0x7fff7fffu);
}

constexpr int PAIRS = 128;
constexpr int PART = 256;       // value dimensions of a block
constexpr int OUT_PITCH = 144;  // bytes of a row of 32 results on their way out
// KC: chunks of 64 columns of a query; NK: keys of a step (128 where one part of 128 dimensions holds all values)
template <int KC, int NK> struct Lay {
  static constexpr bool ALT = NK == 128;           // two sets of four warps take the steps in turn
  static constexpr int SOFT = 8, W_TMA = SOFT, W_MMA = SOFT + 1, THREADS = (SOFT + 2) * 32;
  static constexpr int QT = KC >= 8 ? 4 : 0;       // query chunks in tensor memory
  static constexpr int Q = (KC - QT) * PAIRS * 128, CHUNK = NK * 128, SLOT = 2 * CHUNK;
  static constexpr int RED = 2 * 2 * PAIRS * 4;    // what warps tell each other: [parity of the step][half][pair]
  static constexpr int BIAS = KC <= 4 ? 16384 : 0; // distance biases of the block's heads, where they fit
  static constexpr int SPACE = (umma::SMEM_LIMIT - Q - RED - BIAS - 512) / SLOT;
  static constexpr int NS = SPACE > 10 ? 10 : SPACE;  // two steps of 4 pairs + 2 kept of the step before where values are keys
  static constexpr int AT_BIAS = Q + NS * SLOT, AT_RED = AT_BIAS + BIAS, AT_BAR = AT_RED + RED, NEED = AT_BAR + 512;
  static constexpr int TOTAL = NEED + 1024 > umma::SMEM_LIMIT ? umma::SMEM_LIMIT : NEED + 1024;
  static constexpr int S_COL = PART, Q_COL = S_COL + 2 * NK;  // tensor memory columns; sums start at 0 (and at 128 those of the odd steps)
  // last slots of the ring, through which the queries pass: as binary16 on their way to tensor memory, or (short ones) as f32
  static constexpr bool RAW = KC <= 2;
  static constexpr int TMP = RAW ? KC * PAIRS * 256 / SLOT : QT * PAIRS * 128 / SLOT, AT_TMP = Q + (NS - TMP) * SLOT;
  static_assert(Q_COL + 32 * QT <= 512 && (2 * NS + 7) * 8 + 8 <= 512 && Q + NS * SLOT >= 2 * SOFT * 32 * OUT_PITCH + 2048 && TMP <= NS, "");
};

struct Shape {
  int parts;   // of the values
  bool shared; // values are the keys
};

__device__ __forceinline__ void tld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tst32(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]),
        "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "f"(v[16]), "f"(v[17]), "f"(v[18]), "f"(v[19]), "f"(v[20]), "f"(v[21]),
        "f"(v[22]), "f"(v[23]), "f"(v[24]), "f"(v[25]), "f"(v[26]), "f"(v[27]), "f"(v[28]), "f"(v[29]), "f"(v[30]), "f"(v[31])
      : "memory");
}
__device__ __forceinline__ void tst16(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
                 "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
               : "memory");
}
__device__ __forceinline__ void tld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tst_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void t_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void t_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar)) : "memory");
}
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, int col, int row, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(col), "r"(row), "r"(s32(bar)) : "memory");
}
// kind::f16 with binary16 operands and f32 accumulators, M = 128
__host__ __device__ constexpr uint32_t mma_desc(int n, bool mn_major_b) {
  return (1u << 4) | ((mn_major_b ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(PAIRS >> 4) << 24);
}

__device__ __forceinline__ void mma_ss(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t add) {
  asm volatile("{ .reg .pred p; .reg .b64 a, b; setp.ne.b32 p, %5, 0; mov.b64 a, {%1, %3}; mov.b64 b, {%2, %3}; "
               "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p; }"
               ::"r"(d), "r"(a), "r"(b), "r"(DESC_HI), "r"(idesc), "r"(add) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t add) {  // the first operand in tensor memory
  asm volatile("{ .reg .pred p; .reg .b64 b; setp.ne.b32 p, %5, 0; mov.b64 b, {%2, %3}; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p; }"
               ::"r"(d), "r"(a), "r"(b), "r"(DESC_HI), "r"(idesc), "r"(add) : "memory");
}

// grid (tiles of all groups x parts, kv head)
template <int KC, int NK, bool SPLIT>
__global__ void __launch_bounds__(Lay<KC, NK>::THREADS, 1)
span_umma_kernel(const float* q, int64_t q_ld, SpanShape sh, Shape ms, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                 RowMap rows, const __grid_constant__ SpanBatch b, SpanOut so, int* __restrict__ err) {
  using L = Lay<KC, NK>;
  constexpr int NS = L::NS, NC = L::ALT ? NK : NK / 2, CB = L::ALT ? 64 : NC, W_TMA = L::W_TMA, W_MMA = L::W_MMA;  // NC: keys of a step that one thread turns into weights, CB at a time
  constexpr bool ALT = L::ALT;
  extern __shared__ __align__(1024) uint8_t raw[];
  const uint32_t base = (s32(raw) + 1023u) & ~1023u;
  uint8_t* smem = raw + (base - s32(raw));
  float* red = (float*)(smem + L::AT_RED);
  uint64_t* full = (uint64_t*)(smem + L::AT_BAR);
  uint64_t *empty = full + NS, *s_full = empty + NS, *p_full = s_full + 2, *sums = p_full + 2, *q_full = sums + 2;  // sums, like the others, by step parity
  uint32_t* tmem_slot = (uint32_t*)(q_full + 1);
  const int warp = __shfl_sync(~0u, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (base - s32(raw) + L::NEED > L::TOTAL) {  // shared memory not where its alignment says: the same for every thread of the grid
    if (threadIdx.x == 0) report_error(err, 5);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; ++s) { bar_init(&full[s], 1); bar_init(&empty[s], 1); }
    for (int i = 0; i < 2; ++i) { bar_init(&s_full[i], 1); bar_init(&p_full[i], ALT ? 4 : 8); bar_init(&sums[i], 1); }
    bar_init(q_full, L::SOFT);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  t_before();
  __syncthreads();
  t_after();
  const uint32_t tmem = __shfl_sync(~0u, *tmem_slot, 0);
  const int head = blockIdx.y, gq = sh.n_head / sh.n_kv;
  // biases of the block's heads, in units of ln 2; heads start eight banks apart
  constexpr float LOG2E = 1.4426950408889634f;
  const int bias_pitch = (sh.bias_len + 31) / 32 * 32 + 8;
  const bool staged = sh.bias && (int64_t)gq * bias_pitch * 4 <= L::BIAS;
  if (staged && warp < L::SOFT)
    for (int i = threadIdx.x; i < gq * sh.bias_len; i += L::SOFT * 32) {
      const int g = i / sh.bias_len;
      ((float*)(smem + L::AT_BIAS))[g * bias_pitch + i - g * sh.bias_len] = sh.bias[(int64_t)head * gq * sh.bias_len + i] * LOG2E;
    }
  // dependents may be placed from here on: they find their tensor memory only after this block has its own
  pdl_enter();

  const int part = ms.parts > 1 ? (int)blockIdx.x % ms.parts : 0, tile = (int)blockIdx.x / ms.parts;
  const int gi = span_group(b.tiles_at, b.n, tile), t0 = b.t0[gi], tokens = b.rows[gi];
  // the last rows first: in a window that is still filling they see the most keys
  const int pairs = tokens * gq, pair0 = (b.tiles_at[gi + 1] - 1 - tile) * PAIRS;
  const int p_first = row_position(rows, t0);
  const GroupKeys gk = group_keys(p_first, tokens, sh.window, sh.keep_first);
  const int pa = p_first + pair0 / gq, pb = p_first + min(pairs - 1, pair0 + PAIRS - 1) / gq;  // positions of the tile's rows
  // The steps: NK rows of the group's list each.  Those that hold kept tokens before the tile's window start at its head, the others
  // at the window's first key or behind those.
  const int lo = sh.window > 0 ? max(0, pa - sh.window + 1) : 0, kept = min(sh.keep_first, lo), kept_steps = (kept + NK - 1) / NK;
  const int w0 = max(kept_steps * NK, gk.index(lo)), steps = kept_steps + max(0, (gk.index(pb) - w0 + NK) / NK);
  auto step_row = [&](int j) { return j < kept_steps ? j * NK : w0 + (j - kept_steps) * NK; };
  // pairs of chunks: a step's keys, the block's own values; the first own pair
  const int own_dims = min(sh.dv - part * PART, PART), kc = (sh.dk + 127) / 128, vc = (own_dims + 127) / 128, own0 = part * (PART / 128);
  // the order in which a step's key chunks are read: where they are values too, the block's own come last
  auto pair = [&](int i) { return !ms.shared ? i : i < kc - vc ? (i < own0 ? i : i + vc) : own0 + i - (kc - vc); };
  bool ok = true;

  if (warp == W_TMA) {
    if (elect_one()) {
      const int row0 = b.row0[gi] + head * b.keys[gi];
      int s = 0, lap = 0;
      bool first = true;
      auto load = [&](const CUtensorMap* map, int cols, int col, int row) {
        if (L::TMP > 0 && first && s == NS - L::TMP) {  // the queries have left these slots
          first = false;
          if (ok && !bar_wait(q_full, 0)) { ok = false; report_error(err, 5); }
        }
        if (ok && !bar_wait(&empty[s], (uint32_t)((lap & 1) ^ 1))) { ok = false; report_error(err, 5); }
        if (ok) {
          const bool two = col + 64 < cols;
          const uint32_t dst = base + (uint32_t)(L::Q + s * L::SLOT);
          bar_expect(&full[s], two ? L::SLOT : L::CHUNK);  // boxes are always complete: what lies outside the matrix is filled with zeros
          load_box(dst, map, col, row, &full[s]);
          if (two) load_box(dst + L::CHUNK, map, col + 64, row, &full[s]);
        }
        if (++s == NS) { s = 0; ++lap; }
      };
      auto keys = [&](int j) { for (int i = 0; i < kc; ++i) load(&kmap, sh.dk, 128 * pair(i), row0 + step_row(j)); };
      keys(0);
      for (int j = 0; j < steps; ++j) {
        if (j + 1 < steps) keys(j + 1);
        if (!ms.shared) for (int i = 0; i < vc; ++i) load(&vmap, sh.dv, 128 * (own0 + i), row0 + step_row(j));
      }
    }
    __syncwarp();
  } else if (warp == W_MMA) {
    const bool leader = elect_one();
    int s = 0, lap = 0;  // the ring's next slot
    const uint32_t q_lo = base >> 4, r_lo = (base + (uint32_t)L::Q) >> 4;  // low words of descriptors: addresses below 2^18
    auto arrived = [&] {
      if (ok && !bar_wait(&full[s], (uint32_t)(lap & 1))) { ok = false; report_error(err, 5); }
    };
    auto next = [&] { if (++s == NS) { s = 0; ++lap; } };
    auto scores = [&](int j) {
      const uint32_t d = tmem + (uint32_t)(L::S_COL + (j & 1) * NK);
      for (int i = 0; i < kc; ++i) {
        const int c = pair(i), k16 = (sh.dk - 128 * c + 15) / 16;
        const uint32_t lb = r_lo + (uint32_t)(s * (L::SLOT / 16));
        arrived();
        t_after();
        if (leader) {
          if (2 * c < L::QT) {
            const uint32_t ta = tmem + (uint32_t)(L::Q_COL + 64 * c);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              if (kk < k16) mma_ts(d, ta + (uint32_t)(8 * kk), lb + (uint32_t)((kk >> 2) * (L::CHUNK / 16) + 2 * (kk & 3)), mma_desc(NK, false), (uint32_t)(i | kk));
          } else {
            const uint32_t la = q_lo + (uint32_t)((2 * c - L::QT) * (PAIRS * 128 / 16));
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              if (kk < k16)
                mma_ss(d, la + (uint32_t)((kk >> 2) * (PAIRS * 128 / 16) + 2 * (kk & 3)), lb + (uint32_t)((kk >> 2) * (L::CHUNK / 16) + 2 * (kk & 3)),
                       mma_desc(NK, false), (uint32_t)(i | kk));
          }
          if (!(ms.shared && i >= kc - vc)) commit(&empty[s]);
        }
        next();
      }
      if (leader) commit(&s_full[j & 1]);
    };
    int own = kc - vc;  // where values are keys: the slot of the step's first own pair
    auto weighted = [&](int j) {
      if (ok && !bar_wait(&p_full[j & 1], (uint32_t)((j >> 1) & 1))) { ok = false; report_error(err, 5); }
      const uint32_t p = tmem + (uint32_t)(L::S_COL + (j & 1) * NK), acc = (uint32_t)(ALT ? j >> 1 : j);
      for (int i = 0; i < vc;) {
        // pairs that follow each other in the ring are one operand: 64 columns apart in the descriptor's leading offset
        const int at = ms.shared ? own : s;
        int run = 0;
        for (; i + run < vc && at + run < NS; ++run)
          if (!ms.shared) { arrived(); next(); }
        t_after();
        const uint32_t lb = r_lo + (uint32_t)(at * (L::SLOT / 16)) + ((uint32_t)(L::CHUNK / 16) << 16);
        const uint32_t idesc = mma_desc(min(128 * run, (own_dims - 128 * i + 15) & ~15), true), o = tmem + (uint32_t)((ALT ? 128 * (j & 1) : 0) + 128 * i);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < NK / 16; ++kk) {  // sixteen keys: two groups of eight 128-byte rows
            const uint32_t pk = p + (uint32_t)(SPLIT ? 32 * (kk >> 1) + 8 * (kk & 1) : 8 * kk);
            mma_ts(o, pk, lb + (uint32_t)(128 * kk), idesc, acc | (uint32_t)kk);
            if constexpr (SPLIT) mma_ts(o, pk + 16, lb + (uint32_t)(128 * kk), idesc, 1u);
          }
          for (int k = 0; k < run; ++k) commit(&empty[at + k]);
        }
        i += run;
        if (ms.shared && (own += run) == NS) own = 0;
      }
      if (ms.shared && (own += kc - vc) >= NS) own -= NS;
      if (leader) commit(&sums[j & 1]);
    };
    if (ok && !bar_wait(q_full, 0)) { ok = false; report_error(err, 5); }
    t_after();
    scores(0);
    if (ALT && steps > 1) scores(1);
    for (int j = 0; j < steps; ++j) {
      if (!ALT && j + 1 < steps) scores(j + 1);
      weighted(j);
      if (ALT && j + 2 < steps) scores(j + 2);  // over the weights of step j, behind the sums that read them
    }
    __syncwarp();
  } else {  // scores are kept in units of ln 2: exp(x) = exp2(x log2 e)
    const int wg = warp >> 2, set = ALT ? wg : 0, half = ALT ? 0 : wg, row = 32 * (warp & 3) + lane, p = pair0 + row, pc = min(p, pairs - 1);
    const uint32_t t_lane = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    auto all_warps = [] { asm volatile("bar.sync 1, %0;" ::"n"(L::SOFT * 32) : "memory"); };
    // ---- queries: eight lanes per pair; the power of two that brings the largest magnitude into [2^9, 2^10).  One that is not finite stays so:
    // it meets its own row only
    {
      constexpr int OWN = PAIRS / L::SOFT;  // pairs of a warp
      const bool quads = ((uintptr_t)q & 15) == 0 && (q_ld & 3) == 0;
      auto source = [&](int r) {
        const int rc = min(pair0 + r, pairs - 1);
        return q + (int64_t)(t0 + rc / gq) * q_ld + (int64_t)(head * gq + rc % gq) * sh.dk;
      };
      auto fetch = [&](const float* src, int i) {
        return quads ? *(const float4*)(src + i) : make_float4(src[i], src[i + 1], src[i + 2], src[i + 3]);  // dk is a multiple of eight
      };
      const uint32_t own_raw = base + (uint32_t)(L::AT_TMP + warp * OWN * KC * 256);
      if (L::RAW && quads) {  // all of a warp's pairs are on their way at once
#pragma unroll 1
        for (int r = lane >> 3; r < OWN; r += 4) {
          const float* src = source(warp * OWN + r);
#pragma unroll
          for (int c = 0; c < 2 * KC; ++c) {
            const int i = 32 * c + 4 * (lane & 7);
            if (i < sh.dk) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(own_raw + (uint32_t)(r * KC * 256 + 4 * i)), "l"(src + i) : "memory");
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
      }
      auto tile_of = [&](int c) { return c < L::QT ? L::AT_TMP + c * PAIRS * 128 : (c - L::QT) * PAIRS * 128; };
#pragma unroll 1
      for (int r0 = lane >> 3; r0 < OWN; r0 += 4) {
        const int r = warp * OWN + r0;
        const float* src = source(r);
        float4 v[2 * KC];
        float most = 0.f;
#pragma unroll
        for (int c = 0; c < 2 * KC; ++c) {
          const int i = 32 * c + 4 * (lane & 7);
          v[c] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (pair0 + r < pairs && i < sh.dk) v[c] = L::RAW && quads ? *(const float4*)(smem + L::AT_TMP + (r * KC * 256 + 4 * i)) : fetch(src, i);
        }
#pragma unroll
        for (int c = 0; c < 2 * KC; ++c) most = fmaxf(fmaxf(most, fmaxf(fabsf(v[c].x), fabsf(v[c].y))), fmaxf(fabsf(v[c].z), fabsf(v[c].w)));
#pragma unroll
        for (int k = 4; k > 0; k >>= 1) most = fmaxf(most, __shfl_xor_sync(~0u, most, k));
        const int be = (int)((__float_as_uint(most) >> 23) & 0xff);
        const int e = (be == 0 || be == 255) ? 0 : min(126, max(-126, 136 - be));
        const float up = __uint_as_float((uint32_t)(127 + e) << 23), down = __uint_as_float((uint32_t)(127 - e) << 23);
#pragma unroll
        for (int c = 0; c < 2 * KC; ++c)  // 16-byte pieces of a 128-byte row lie where their number XOR the row says
          *(uint2*)(smem + tile_of(c >> 1) + r * 128 + (((4 * (c & 1) + ((lane & 7) >> 1)) ^ (r & 7)) << 4) + 8 * (lane & 1)) =
              make_uint2(pack_h2(v[c].x * up, v[c].y * up), pack_h2(v[c].z * up, v[c].w * up));
        if ((lane & 7) == 0) red[r] = down * sh.scale;
      }
    }
    all_warps();
    if constexpr (L::QT > 0) {
#pragma unroll 1
      for (int c = wg; c < L::QT; c += 2) {
        float w[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) *(float4*)(w + 4 * i) = *(const float4*)(smem + L::AT_TMP + c * PAIRS * 128 + row * 128 + ((i ^ (row & 7)) << 4));
        tst32(t_lane + (uint32_t)(L::Q_COL + 32 * c), w);
      }
      tst_wait();
      t_before();
    }
    const float f = red[row] * LOG2E;  // every thread has its own before the first scores exist, and with them the first exchange
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) bar_arrive(q_full);
    const int g = pc % gq, h = head * gq + g, pos = p_first + pc / gq;  // this thread's pair
    const int i_lo = p_first + min(pair0 + 32 * (warp & 3), pairs - 1) / gq, i_hi = p_first + min(pair0 + 32 * (warp & 3) + 31, pairs - 1) / gq;  // positions of this warp's
    const float* bias = staged ? (const float*)(smem + L::AT_BIAS) + g * bias_pitch : sh.bias ? sh.bias + (int64_t)h * sh.bias_len : nullptr;
    const float unit = staged ? 1.f : LOG2E, far = bias ? bias[sh.bias_len - 1] * unit : 0.f;
    // rows of the list that this pair sees: its window, and the kept tokens (whose rows are their positions)
    const int see_lo = sh.window > 0 ? gk.index(max(0, pos - sh.window + 1)) : 0, see_hi = gk.index(pos), see_kept = min(sh.keep_first - 1, see_hi);
    auto bits = [](int a, int b) {  // bits a .. b of a word, as far as they are in it
      a = max(a, 0);
      b = min(b, 31);
      return a > b ? 0u : (~0u << a) & (~0u >> (31 - b));
    };
    float m = -CUDART_INF_F, l = 0.f;  // the row's reference, and the sum of this thread's exponentials
    if (sh.sink && set == 0) {  // the sink is the first score: the reference starts there, and one thread of a row's counts it
      m = sh.sink[h] * LOG2E;
      l = half == 0 ? 1.f : 0.f;
    }
    auto sums_done = [&](int j) {  // of step j
      if (ok && !bar_wait(&sums[j & 1], (uint32_t)((j >> 1) & 1))) { ok = false; report_error(err, 5); }
    };
    const int o_blocks = (own_dims + 31) / 32;
    float s[CB];
#pragma unroll 1
    for (int j = set; j < steps; j += ALT ? 2 : 1) {
      const uint32_t t_s = t_lane + (uint32_t)(L::S_COL + (j & 1) * NK), t_mine = t_s + (uint32_t)(half * NC);
      const int k_lo = step_row(j) + half * NC, j_lo = gk.at(k_lo), j_hi = gk.at(k_lo + NC - 1);
      const bool all_seen = j_hi <= i_lo && (sh.window <= 0 || i_hi - j_lo < sh.window || j_hi < sh.keep_first);  // warp-uniform
      const bool all_far = !bias || i_lo - j_hi >= sh.bias_len - 1, plain = all_seen && all_far && sh.scale >= 0.f;
      if (ok && !bar_wait(&s_full[j & 1], (uint32_t)((j >> 1) & 1))) { ok = false; report_error(err, 5); }
      t_after();
      if (!plain) {
#pragma unroll 1
        for (int c = 0; c < NC; c += 32) {
          float u[32];
          tld32(t_mine + (uint32_t)c, u);
          tld_wait();
          if (all_far) {
#pragma unroll
            for (int i = 0; i < 32; ++i) u[i] = fmaf(u[i], f, far);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) u[i] = fmaf(u[i], f, bias[min(max(pos - gk.at(k_lo + c + i), 0), sh.bias_len - 1)] * unit);
          }
          const uint32_t seen = bits(see_lo - k_lo - c, see_hi - k_lo - c) | bits(0, see_kept - k_lo - c);
#pragma unroll
          for (int i = 0; i < 32; ++i) u[i] = (seen >> i) & 1u ? u[i] : -CUDART_INF_F;
          tst32(t_mine + (uint32_t)c, u);
        }
        tst_wait();
      }
      float x = -CUDART_INF_F;
#pragma unroll 1
      for (int c = 0; c < NC; c += CB) {
#pragma unroll
        for (int i = 0; i < CB; i += 32) tld32(t_mine + (uint32_t)(c + i), s + i);
        tld_wait();
#pragma unroll
        for (int i = 0; i < CB; ++i) x = fmaxf(x, s[i]);
      }
      if (plain) x = fmaf(x, f, far);
      if (!ALT) {
        float* both = red + (j & 1) * 2 * PAIRS;
        both[half * PAIRS + row] = x;
        all_warps();  // every warp has its scores: weights may take their place
        x = fmaxf(x, both[(half ^ 1) * PAIRS + row]);
      }
      const bool grown = x > m + 8.f;  // the same in both threads of a row
      if (__any_sync(~0u, grown)) {
        const float w = grown ? (m == -CUDART_INF_F ? 0.f : exp2_ftz(m - x)) : 1.f;
        if (grown) m = x;
        l *= w;
        const int before = j - (ALT ? 2 : 1);
        if (before >= 0) {
          sums_done(before);
          t_after();
#pragma unroll 1
          for (int c = half; c < o_blocks; c += ALT ? 1 : 2) {
            float o[32];
            const uint32_t t_o = t_lane + (uint32_t)(128 * set + 32 * c);
            tld32(t_o, o);
            tld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= w;
            tst32(t_o, o);
          }
        }
      }
      // a row that has seen nothing yet: every score is -inf and so is the reference; its exponentials are zero
      const float ref = m == -CUDART_INF_F ? 0.f : m, mul = plain ? f : 1.f, add = plain ? far - ref : -ref;
#pragma unroll 1
      for (int c = 0; c < NC; c += CB) {
        if (ALT) {
#pragma unroll
          for (int i = 0; i < CB; i += 32) tld32(t_mine + (uint32_t)(c + i), s + i);
          tld_wait();
        }
#pragma unroll
        for (int k = 0; k < CB; k += 32) {
          uint32_t e[SPLIT ? 32 : 16];
          float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float e0 = exp2_ftz(fmaf(s[k + 2 * i], mul, add)), e1 = exp2_ftz(fmaf(s[k + 2 * i + 1], mul, add));
            e[i] = pack_h2(e0, e1);
            const float2 r = __half22float2(*(const __half2*)&e[i]);
            if constexpr (SPLIT) e[16 + i] = pack_h2(e0 - r.x, e1 - r.y);
            sum0 += SPLIT ? e0 : r.x;  // the sum of what the weighted sum uses
            sum1 += SPLIT ? e1 : r.y;
          }
          l += sum0 + sum1;
          if constexpr (SPLIT) tst32(t_mine + (uint32_t)(c + k), (const float*)e);
          else tst16(t_s + (uint32_t)((half * NC + c + k) / 2), e);
        }
      }
      tst_wait();
      t_before();
      __syncwarp();
      if (lane == 0) bar_arrive(&p_full[j & 1]);
    }
    // ---- results: the sets' sums meet, a warp turns 32 rows x 32 dimensions at a time over shared memory and stores whole rows
    const bool gated = so.gate && !so.head_gate, vec = ((so.ld & 7) | (gated ? so.gate_ld & 3 : 0)) == 0 &&
                       (((uintptr_t)so.out | (uintptr_t)so.out16 | (gated ? (uintptr_t)so.gate : 0)) & 15) == 0;
    if (steps > 1) sums_done(steps - 2);
    sums_done(steps - 1);  // queries, keys and values have been read: their place is free
    t_after();
    uint8_t *turn = smem + warp * 64 * OUT_PITCH, *gates = turn + 32 * OUT_PITCH;
    int64_t *start = (int64_t*)(smem + L::SOFT * 64 * OUT_PITCH), *gate_start = start + PAIRS;  // of a row's results, of its gates
    all_warps();  // the last exchange has been read
    red[wg * PAIRS + row] = l;
    red[(2 + wg) * PAIRS + row] = m;
    if (wg == 0) {
      start[row] = (int64_t)(t0 + pc / gq) * so.ld + (int64_t)h * sh.dv + part * PART;
      gate_start[row] = (int64_t)(t0 + pc / gq) * so.gate_ld + (int64_t)h * sh.dv + part * PART;
    }
    all_warps();
    const float l0 = red[row], l1 = red[PAIRS + row], m0 = red[2 * PAIRS + row], m1 = red[3 * PAIRS + row];
    float w0 = 1.f, w1 = 1.f;
    if (ALT) {
      const float top = fmaxf(m0, m1);
      w0 = m0 == -CUDART_INF_F ? 0.f : exp2_ftz(m0 - top);
      w1 = m1 == -CUDART_INF_F ? 0.f : exp2_ftz(m1 - top);
    }
    float inv = __fdiv_rn(1.0f, l0 * w0 + l1 * w1) * so.scale;
    if (so.gate && so.head_gate) inv *= __fdiv_rn(1.0f, 1.0f + expf(-so.gate[(int64_t)(t0 + pc / gq) * so.gate_ld + h]));
    w0 *= inv;
    w1 *= inv;
#pragma unroll 1
    for (int c = wg; c < o_blocks; c += L::SOFT / 4) {
      const int d = 32 * c + 4 * (lane & 7);
      const int last = d < own_dims ? min(32, pairs - pair0 - 32 * (warp & 3)) : 0;  // dv is a multiple of eight
      float o[32], o2[32];
      tld32(t_lane + (uint32_t)(32 * c), o);
      if (ALT && steps > 1) tld32(t_lane + (uint32_t)(128 + 32 * c), o2);
      tld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        o[i] *= w0;
        if (ALT && steps > 1) o[i] = fmaf(o2[i], w1, o[i]);
      }
#pragma unroll
      for (int i = 0; i < 32; i += 4) *(float4*)(turn + lane * OUT_PITCH + 4 * i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
      if (gated) {  // gates of rows lane / 8 + 4 k, all on their way at once
        float4 gate[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = (lane >> 3) + 4 * k;
          const float* gp = so.gate + gate_start[32 * (warp & 3) + r] + d;
          gate[k] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r < last) gate[k] = vec ? *(const float4*)gp : make_float4(gp[0], gp[1], gp[2], gp[3]);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) *(float4*)(gates + ((lane >> 3) + 4 * k) * OUT_PITCH + 16 * (lane & 7)) = gate[k];
      }
      __syncwarp();
#pragma unroll 2
      for (int r = lane >> 3; r < last; r += 4) {
        float4 v = *(const float4*)(turn + r * OUT_PITCH + 16 * (lane & 7));
        const int64_t at = start[32 * (warp & 3) + r] + d;
        if (gated) {
          const float4 gv = *(const float4*)(gates + r * OUT_PITCH + 16 * (lane & 7));
          v.x *= __frcp_rn(1.0f + expf(-gv.x));
          v.y *= __frcp_rn(1.0f + expf(-gv.y));
          v.z *= __frcp_rn(1.0f + expf(-gv.z));
          v.w *= __frcp_rn(1.0f + expf(-gv.w));
        }
        if (so.out) {
          if (vec) {
            *(float4*)(so.out + at) = v;
          } else {
            *(float2*)(so.out + at) = make_float2(v.x, v.y);
            *(float2*)(so.out + at + 2) = make_float2(v.z, v.w);
          }
        }
        if (so.out16) {
          __nv_bfloat162 w[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
          __nv_bfloat16* dst = (__nv_bfloat16*)so.out16 + at;
          if (vec) {
            *(uint2*)dst = *(const uint2*)w;
          } else {
            *(__nv_bfloat162*)dst = w[0];
            *(__nv_bfloat162*)(dst + 2) = w[1];
          }
        }
      }
      __syncwarp();
    }
    t_before();
  }
  __syncthreads();
  if (warp == W_MMA) {
    t_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

typedef void (*UmmaKernel)(const float*, int64_t, SpanShape, Shape, const CUtensorMap, const CUtensorMap, RowMap, const SpanBatch, SpanOut, int*);
struct Variant {
  UmmaKernel kernel;
  int nk, smem, threads;
  PerDevice* ready;
};
// Steps of 128 keys where the values fit 128 columns of tensor memory, of 64 otherwise; the queries' chunks are rounded up to an
// instance's.  The longest keys that have 16-bit operands leave a ring of four pairs, which the queries pass through before it starts.
Variant variant(int dk, int dv, bool split) {
  const int kc = (dk + 63) / 64;
#define LLR_V(K, N, S) { static PerDevice ready; return Variant{span_umma_kernel<K, N, S>, N, Lay<K, N>::TOTAL, Lay<K, N>::THREADS, &ready}; }
  if (split) {
    if (dv <= 128 && kc <= 1) LLR_V(1, 128, true)
    if (dv <= 128 && kc <= 2) LLR_V(2, 128, true)
    return Variant{nullptr, 0, 0, 0, nullptr};
  }
  if (dv <= 128) {
    if (kc <= 1) LLR_V(1, 128, false)
    if (kc <= 2) LLR_V(2, 128, false)
    if (kc <= 4) LLR_V(4, 128, false)
  }
  if (kc <= 4) LLR_V(4, 64, false)
  if (kc <= 8) LLR_V(8, 64, false)
  if (kc <= 12) LLR_V(12, 64, false)
  if (kc <= 14) LLR_V(14, 64, false)
#undef LLR_V
  return Variant{nullptr, 0, 0, 0, nullptr};
}

bool encode_rows(CUtensorMap* map, const void* base, int64_t cols, int64_t rows, int box_rows) {
  EncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t one[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)base, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int visible_keys(const SpanShape& sh, const SpanGroup& g) {
  const int lo = sh.window > 0 ? std::max(0, g.first - sh.window + 1) : 0;  // as group_keys
  return std::min(sh.keep_first, lo) + g.first + g.rows - lo;
}

// most keys a group of consecutive rows sees
int span_group_keys(const SpanShape& sh, int rows) {
  return sh.window > 0 ? (int)std::min<int64_t>(sh.n_ctx, (int64_t)sh.window + sh.keep_first + rows) : sh.n_ctx;
}

}  // namespace

size_t span_umma_scratch_floats(const SpanShape& sh, int max_rows) {
  return (size_t)sh.n_kv * span_group_keys(sh, max_rows) * (sh.dk + sh.dv) / 2 + 64;
}

// Heads that have 16-bit operands: those of which 64 queries, 64 keys and 64 values fit 222 KB as binary16, keys padded to 16 columns and values
// to the widths below (beside up to 128 of them; more leave room for a tile of exponentials), and latents up to 512.  Wider heads have f32
// operands whatever the number of rows, although the kernel here could hold some of them: nobody who uses them asked for fewer bits.
static bool sixteen_bit_heads(int dk, int dv, bool shared) {
  if (dv > 512) return false;
  const int kw = (dk + 15) / 16 * 16, vw = dv <= 128 ? (dv + 31) / 32 * 32 : dv <= 192 ? 192 : dv <= 256 ? 256 : dv <= 384 ? 384 : 512;
  return shared ? dk == dv : 2 * kw + vw <= (dv <= 128 ? 1752 : 1680);
}

bool span_umma_supported(const SpanShape& sh, bool shared, const SpanOut& out) {
  return sh.n_kv > 0 && sh.n_head % sh.n_kv == 0 && sh.dk % 8 == 0 && sh.dv % 8 == 0 && sixteen_bit_heads(sh.dk, sh.dv, shared) && variant(sh.dk, sh.dv, sh.split_weights).kernel &&
         (int64_t)sh.n_kv * sh.n_ctx < (1 << 30) && out.ld % 2 == 0 && ((uintptr_t)out.out & 7) == 0 && ((uintptr_t)out.out16 & 3) == 0 &&
         (!out.gate || out.head_gate || (out.gate_ld % 2 == 0 && ((uintptr_t)out.gate & 7) == 0));
}

cudaError_t launch_span_umma(const float* q, int64_t q_ld, const SpanShape& sh, const LayerKv& kv, const RowMap& rows, const SpanGroup* groups, int n_groups,
                             int min_rows, const SpanOut& out, float* scratch, size_t scratch_floats, cudaStream_t s, int* err, uint64_t* launches) {
  const Variant v = variant(sh.dk, sh.dv, sh.split_weights);
  const bool shared = kv.k == kv.v;
  const int gq = sh.n_head / sh.n_kv, width = sh.dk + (shared ? 0 : sh.dv);
  const Shape ms{(sh.dv + PART - 1) / PART, shared};
  cudaError_t e = cudaSuccess;
  std::atomic<int>& slot = v.ready->here();
  if (slot.load(std::memory_order_relaxed) == 0) {
    if ((e = cudaFuncSetAttribute((const void*)v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem)) != cudaSuccess) return e;
    slot.store(1, std::memory_order_relaxed);
  }
  SpanBatch b{};
  int64_t keys = 0;  // rows of the matrices of keys and of values
  auto run_batch = [&] {
    if (b.n == 0) return cudaSuccess;
    __half *k16 = (__half*)scratch, *v16 = shared ? nullptr : k16 + keys * sh.dk;
    CUtensorMap kmap, vmap;
    if (!encode_rows(&kmap, k16, sh.dk, keys, v.nk) || !encode_rows(&vmap, shared ? k16 : v16, sh.dv, keys, v.nk)) return cudaErrorInvalidValue;
    if (launches) *launches += 2;
    cudaError_t ce = launch_walk(span_gather_kernel, dim3(b.keys_at[b.n], sh.n_kv), dim3(256), 0, s, sh, kv, rows, b, k16, v16);
    if (ce == cudaSuccess)
      ce = launch_walk(v.kernel, dim3(b.tiles_at[b.n] * ms.parts, sh.n_kv), dim3(v.threads), v.smem, s, q, q_ld, sh, ms, kmap, vmap, rows, b, out, err);
    b.n = 0;
    keys = 0;
    return ce;
  };
  for (int g = 0; g < n_groups && e == cudaSuccess; ++g) {
    if (groups[g].rows < min_rows) continue;
    if (groups[g].first < 0) return cudaErrorInvalidValue;
    const int mine = visible_keys(sh, groups[g]);
    if ((size_t)((int64_t)sh.n_kv * mine) * width > 2 * scratch_floats) return cudaErrorInvalidValue;
    if (b.n == SPAN_GROUPS || (b.n > 0 && (size_t)(keys + (int64_t)sh.n_kv * mine) * width > 2 * scratch_floats)) e = run_batch();
    const int i = b.n++;
    b.t0[i] = groups[g].t0;
    b.rows[i] = groups[g].rows;
    b.keys[i] = mine;
    b.row0[i] = (int)keys;
    b.keys_at[i + 1] = b.keys_at[i] + (mine + 7) / 8;
    b.tiles_at[i + 1] = b.tiles_at[i] + (int)(((int64_t)groups[g].rows * gq + PAIRS - 1) / PAIRS);
    keys += (int64_t)sh.n_kv * mine;
  }
  return e == cudaSuccess ? run_batch() : e;
}

}  // namespace llr
