// Element-wise and attention kernels of the device-resident Llama walk: what stands between the matrix
// products of Llama::forward_layers (langtax/src/decode.rs:2737-3097) -- rmsnorm_inplace :11498, rope :11578
// (adjacent-pair rotation), store_kv :12059, attend_query :11126 with grouped-query heads, silu :11826,
// the residual adds -- and the greedy argmax of sample.rs:293.  The host walk of the reference runs these on
// the CPU between two executor calls; here a decode step never leaves the device.
//
// Arithmetic follows the reference's formulas; sums that the reference adds sequentially (sum of squares,
// attention scores, softmax denominator, weighted values) are added in a fixed tree / block order here, so
// results are reproducible from run to run and differ from the CPU walk in the last bits only.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <math_constants.h>

#include "llr_attend.cuh"
#include "llr_kernels.cuh"

namespace llr {
namespace {

// first float of the head vector of (sequence, layer, kv head, position) in a paged cache
// A row of the cache is the slot'th of hd floats.  Decode attention looks the slots of a slice up once; they fit 32 bits where
// hd >= 16 (2^32 rows of 64 bytes are more than the device holds), and shared memory in slices of up to SLOT_CHUNK positions.
constexpr int SLOT_CHUNK = 2048;
__host__ __device__ inline int slot_words(int chunk, int hd) { return chunk <= SLOT_CHUNK && hd >= 16 ? chunk : 0; }
__device__ __forceinline__ int64_t kv_slot(const KvView& kv, int seq, int layer, int head, int pos, int n_head_kv) {
  const int b = kv.table[(int64_t)seq * kv.max_blocks + pos / kv.block_tokens];
  return (((int64_t)b * kv.n_layer + layer) * n_head_kv + head) * kv.block_tokens + pos % kv.block_tokens;
}
__device__ __forceinline__ int64_t kv_offset(const KvView& kv, int seq, int layer, int head, int pos, int n_head_kv, int hd) {
  return kv_slot(kv, seq, layer, head, pos, n_head_kv) * hd;
}

// one block per activation row; a row of up to 4096 values stays in registers between the two passes
constexpr int NORM_THREADS = 1024;
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_kernel(float* x, const float* add, const float* __restrict__ w, float* __restrict__ y,
               int n, float eps) {
  pdl_enter();
  __shared__ float sh[32];
  float* xr = x + (int64_t)blockIdx.x * n;
  const float* ar = add ? add + (int64_t)blockIdx.x * n : nullptr;
  float* yr = y + (int64_t)blockIdx.x * n;
  const bool in_regs = n <= 4 * NORM_THREADS && n % 4 == 0;
  float4 keep = make_float4(0.f, 0.f, 0.f, 0.f);
  float ss = 0.f;
  if (in_regs) {
    const int i = 4 * threadIdx.x;
    if (i < n) {
      keep = *(const float4*)(xr + i);
      if (ar) {  // proj + residual (decode.rs:2938, :3050), written back: the new residual stream
        const float4 a = *(const float4*)(ar + i);
        keep.x = __fadd_rn(a.x, keep.x); keep.y = __fadd_rn(a.y, keep.y); keep.z = __fadd_rn(a.z, keep.z); keep.w = __fadd_rn(a.w, keep.w);
        *(float4*)(xr + i) = keep;
      }
      ss = fmaf(keep.x, keep.x, fmaf(keep.y, keep.y, fmaf(keep.z, keep.z, keep.w * keep.w)));
    }
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      float v = xr[i];
      if (ar) { v = __fadd_rn(ar[i], v); xr[i] = v; }
      ss = fmaf(v, v, ss);
    }
  }
  ss = block_sum(ss, sh);
  const float rms = sqrtf(__fadd_rn(__fdiv_rn(ss, (float)(n <= 65535 ? n : 1)), eps));
  const float inv = rms > 0.f ? __fdiv_rn(1.0f, rms) : 0.f;
  if (in_regs) {
    const int i = 4 * threadIdx.x;
    if (i < n) {
      float4 o = make_float4(__fmul_rn(keep.x, inv), __fmul_rn(keep.y, inv), __fmul_rn(keep.z, inv), __fmul_rn(keep.w, inv));
      if (w) {
        const float4 ww = *(const float4*)(w + i);
        o.x = __fmul_rn(o.x, ww.x); o.y = __fmul_rn(o.y, ww.y); o.z = __fmul_rn(o.z, ww.z); o.w = __fmul_rn(o.w, ww.w);
      }
      *(float4*)(yr + i) = o;
    }
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const float t = __fmul_rn(xr[i], inv);
      yr[i] = w ? __fmul_rn(t, w[i]) : t;
    }
  }
}

// One block per token: the cosine and sine of every pair's angle once (all heads of a token turn by the same
// angles), then the rotation of every q and k head, q in place, k and v into the cache (store_kv, decode.rs:12059: the row's sequence, paged).
// Bound: memory latency.  The page is looked up once, values are on their way while the angles are worked out, and four pairs are fetched
// before the first is stored (a pair at a time, and the cache filled from the rotated rows: 512 rows of 32 + 8 heads 15 us).
__global__ void __launch_bounds__(256)
rope_store_kernel(float* q, const float* k, const float* v, KvView kv, RowMap rows, int layer,
                  WalkShape w) {
  pdl_enter();
  __shared__ float s_cos[128], s_sin[128];  // head_dim <= 256
  constexpr int U = 4;
  const int t = blockIdx.x;
  const int pos = row_position(rows, t);
  const int hd = w.head_dim, half = hd / 2, n_kv = w.n_head_kv * half, n = w.n_head * half + n_kv;  // pairs
  const int64_t slot = kv_slot(kv, row_sequence(rows, t), layer, 0, pos, w.n_head_kv);  // heads lie block_tokens slots apart
  auto cached = [&](float* pool, int h, int p) { return (float2*)(pool + (slot + (int64_t)h * kv.block_tokens) * hd + 2 * p); };
  const float2 *qrow = (const float2*)(q + (int64_t)t * w.n_head * hd), *krow = (const float2*)(k + (int64_t)t * w.n_head_kv * hd),
               *vrow = (const float2*)(v + (int64_t)t * w.n_head_kv * hd);
  float2 vv[U];
#pragma unroll
  for (int j = 0; j < U; ++j)
    if ((int)threadIdx.x + 256 * j < n_kv) vv[j] = vrow[threadIdx.x + 256 * j];
  const float theta_scale = w.theta_scale;  // base^(-2/n_rot), computed once on the host in f32 as the reference does
  for (int p = threadIdx.x; p < half; p += blockDim.x) {
    float theta = (float)(pos <= 65535 ? pos : 65535);
    for (int i = 0; i < p; ++i) theta *= theta_scale;  // the reference advances theta multiplicatively in f32
    s_cos[p] = cosf(theta);
    s_sin[p] = sinf(theta);
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < U; ++j) {
    const int i = threadIdx.x + 256 * j;
    if (i < n_kv) *cached(kv.v, i / half, i % half) = vv[j];
  }
  for (int i = threadIdx.x + 256 * U; i < n_kv; i += 256) *cached(kv.v, i / half, i % half) = vrow[i];
  const int nq = n - n_kv;
  for (int i0 = threadIdx.x; i0 < n; i0 += 256 * U) {
    float2 ab[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int i = i0 + 256 * j;
      if (i < n) ab[j] = i < nq ? qrow[i] : krow[i - nq];
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int i = i0 + 256 * j;
      if (i >= n) continue;
      const int h = i / half, p = i % half;
      const float c = s_cos[p], s = s_sin[p];
      const float2 r = make_float2(__fsub_rn(__fmul_rn(ab[j].x, c), __fmul_rn(ab[j].y, s)), __fadd_rn(__fmul_rn(ab[j].x, s), __fmul_rn(ab[j].y, c)));
      if (i < nq) ((float2*)(q + (int64_t)t * w.n_head * hd))[i] = r;
      else *cached(kv.k, h - w.n_head, p) = r;
    }
  }
}

// Attention of one row over one slice of positions.  A block handles the query heads that share a kv head and
// writes, per query head, the slice's maximum score, the sum of exp(score - max) and the exp-weighted sum of value
// rows; attention_combine_kernel merges the slices (the usual two-pass softmax, rearranged so that K and V are read
// once per kv head and by many SMs).  Slices have a fixed length in positions (attention_chunk), whatever the batch: a
// row's result depends on its own sequence only, never on what shares its batch.
// `KV` says where the key and value rows of a position lie: in the paged cache (one row per block: decode steps) or
// in a shared-memory tile that a block fills once for many rows of a prompt chunk.  The arithmetic is this one
// function either way, so both kernels give the same bits.
constexpr int ATT_ROWS = 16;       // rows per block of the tiled kernel
constexpr int ATT_TILE_CHUNK = 128; // longest slice the tiled kernel stages (2 x 128 x head_dim floats: contexts up to 4096 positions)

struct KvGlobal {
  const KvView& kv;
  int sid, layer, hkv, n_head_kv, hd;
  float scale;
  const uint32_t* slots;  // of positions s0, s0 + 1, ... (shared memory), or null
  int s0;
  __device__ __forceinline__ int64_t at(int s) const { return (slots ? (int64_t)slots[s - s0] : kv_slot(kv, sid, layer, hkv, s, n_head_kv)) * hd; }
  __device__ __forceinline__ const float* k(int s) const { return kv.k + at(s); }
  __device__ __forceinline__ const float* v(int s) const { return kv.v + at(s); }
  __device__ __forceinline__ float score(int, int, float dot) const { return __fmul_rn(dot, scale); }
};
struct KvTile {
  const float* kt;
  const float* vt;
  int s0, hd;
  __device__ __forceinline__ const float* k(int s) const { return kt + (s - s0) * hd; }
  __device__ __forceinline__ const float* v(int s) const { return vt + (s - s0) * hd; }
};

// The rotation of rope_store_kernel on n_vec vectors of hd floats in shared memory: one thread per pair
__device__ __forceinline__ void rope_in_place(float* vecs, int n_vec, int hd, int pos, float theta_scale) {
  const int half = hd / 2;
  for (int idx = threadIdx.x; idx < n_vec * half; idx += blockDim.x) {
    float* vec = vecs + (idx / half) * hd;
    const int p = idx % half;
    float theta = (float)(pos <= 65535 ? pos : 65535);
    for (int i = 0; i < p; ++i) theta *= theta_scale;
    const float c = cosf(theta), s = sinf(theta);
    const float a = vec[2 * p], b = vec[2 * p + 1];
    vec[2 * p] = __fsub_rn(__fmul_rn(a, c), __fmul_rn(b, s));
    vec[2 * p + 1] = __fadd_rn(__fmul_rn(a, s), __fmul_rn(b, c));
  }
}

// The rows of a batch that a block of an attention kernel works on: runs [first, first + n) of at most 64 rows of ONE sequence at
// consecutive positions, n << 16 | first.
constexpr int MAX_TILES = 512;
struct RowTiles {
  int n;
  uint32_t run[MAX_TILES];
  __device__ __forceinline__ int begin(int z) const { return (int)(run[z] & 0xffff); }
  __device__ __forceinline__ int end(int z) const { return begin(z) + (int)(run[z] >> 16); }
};

// grid (kv head, position slice, token): one row per block, K and V straight from the paged cache (decode steps).
// With k_new / v_new (a single decode token) the kernel also does what rope_store_kernel does for that token: q is
// rotated as it is loaded, and the block whose slice holds the token's position rotates the new key, writes it and
// the new value into the cache and then reads them back like any other position: one launch less per layer.
template <int G>
__device__ __forceinline__ void attention_partial_row(const float* q, const KvView& kv, float* __restrict__ part, const RowMap& rows, int t, int layer,
                                                      int chunk, const WalkShape& w, const float* k_new, const float* v_new) {
  extern __shared__ float sm[];  // slots[slot_words] | q[gqa][hd] | scores[gqa][chunk] or sums[P][gqa][hd]
  const int hkv = blockIdx.x, split = blockIdx.y;
  const int hd = w.head_dim, gqa = w.n_head / w.n_head_kv;
  const int seq = row_position(rows, t) + 1;  // positions this row attends to
  const int sid = row_sequence(rows, t);
  const int n_split = (int)gridDim.y;
  const int s0 = split * chunk, s1 = min(seq, s0 + chunk);
  if (s0 >= seq) return;  // this row's sequence ends before the slice
  uint32_t* slots = slot_words(chunk, hd) ? (uint32_t*)sm : nullptr;
  float* sq = sm + slot_words(chunk, hd);
  float* sc = sq + gqa * hd;
  if (slots)
    for (int i = threadIdx.x; i < s1 - s0; i += ATT_THREADS) slots[i] = (uint32_t)kv_slot(kv, sid, layer, hkv, s0 + i, w.n_head_kv);
  for (int i = threadIdx.x; i < gqa * hd; i += ATT_THREADS)
    sq[i] = q[((int64_t)t * w.n_head + hkv * gqa) * hd + i];
  if (k_new) {
    const bool mine = s1 == seq;  // the slice that holds the token's own position
    if (mine)
      for (int i = threadIdx.x; i < hd; i += ATT_THREADS) sc[i] = k_new[((int64_t)t * w.n_head_kv + hkv) * hd + i];
    __syncthreads();
    rope_in_place(sq, gqa, hd, seq - 1, w.theta_scale);
    if (mine) {
      rope_in_place(sc, 1, hd, seq - 1, w.theta_scale);
      __syncthreads();
      const int64_t off = kv_offset(kv, sid, layer, hkv, seq - 1, w.n_head_kv, hd);
      for (int i = threadIdx.x; i < hd; i += ATT_THREADS) {
        kv.k[off + i] = sc[i];
        kv.v[off + i] = v_new[((int64_t)t * w.n_head_kv + hkv) * hd + i];
      }
    }
  }
  __syncthreads();
  float* out = part + (((int64_t)t * w.n_head_kv + hkv) * n_split + split) * gqa * (hd + 2);
  attend_slice<ATT_THREADS, G>(KvGlobal{kv, sid, layer, hkv, w.n_head_kv, hd, 1.0f / sqrtf((float)hd), slots, s0}, sq, sc, out, s0, s1, chunk, hd, hd, gqa);
}
template <int G>
__global__ void __launch_bounds__(ATT_THREADS)
attention_partial_kernel(const float* q, KvView kv, float* __restrict__ part, RowMap rows, int layer, int chunk,
                         WalkShape w, const float* k_new, const float* v_new) {
  pdl_enter();
  attention_partial_row<G>(q, kv, part, rows, blockIdx.z, layer, chunk, w, k_new, v_new);
}
// the listed rows of a batch, one per blockIdx.z
template <int G>
__global__ void __launch_bounds__(ATT_THREADS)
attention_rows_kernel(const float* q, KvView kv, float* __restrict__ part, RowMap rows, int layer, int chunk, WalkShape w,
                      const __grid_constant__ RowTiles tiles) {
  pdl_enter();
  attention_partial_row<G>(q, kv, part, rows, tiles.begin(blockIdx.z), layer, chunk, w, nullptr, nullptr);
}

// The same slice of one row done by ONE warp, every elementary sum formed in the order attend_slice forms it (a
// position's score: lanes over the columns in ascending order, then the shuffle tree; a head's softmax: lanes over the
// positions; a dimension's weighted sum: per group of runs of eight positions in ascending order, then the groups in
// order), so the bits are the same.  GQA query heads per kv head and P = ATT_THREADS / head_dim groups are template
// parameters: nothing is predicated, and the loop over the value rows goes over the positions once, each position's
// weights and value row loaded once for all the dimensions and heads a lane owns (the loop is bound by shared-memory
// loads).  sq [GQA][hd] and sc [GQA][max_chunk] are this warp's.
template <int GQA, int P, typename KV>
__device__ __forceinline__ void attend_slice_warp(const KV& src, const float* sq, float* sc, float* out, int s0, int s1, int max_chunk) {
  constexpr int HD = ATT_THREADS / P, ND = HD / 32;
  const int lane = threadIdx.x & 31;
  const float scale = 1.0f / sqrtf((float)HD);
  constexpr int SP = 4;
  for (int sbase = s0; sbase < s1; sbase += SP) {
    float acc[SP][GQA];
    float kvv[SP][ND];
#pragma unroll
    for (int j = 0; j < SP; ++j) {
      const bool live = sbase + j < s1;
      const float* krow = src.k(live ? sbase + j : s0);
#pragma unroll
      for (int u = 0; u < ND; ++u) kvv[j][u] = live ? krow[lane + 32 * u] : 0.f;
#pragma unroll
      for (int g = 0; g < GQA; ++g) acc[j][g] = 0.f;
    }
#pragma unroll
    for (int u = 0; u < ND; ++u)
#pragma unroll
      for (int g = 0; g < GQA; ++g) {
        const float qv = sq[g * HD + lane + 32 * u];
#pragma unroll
        for (int j = 0; j < SP; ++j) acc[j][g] = fmaf(qv, kvv[j][u], acc[j][g]);
      }
#pragma unroll
    for (int j = 0; j < SP; ++j)
      if (sbase + j < s1) {
#pragma unroll
        for (int g = 0; g < GQA; ++g) {
          const float d = warp_sum(acc[j][g]);
          if (lane == 0) sc[g * max_chunk + (sbase + j - s0)] = __fmul_rn(d, scale);
        }
      }
  }
  __syncwarp();
#pragma unroll
  for (int g = 0; g < GQA; ++g) {
    float m = -CUDART_INF_F;
    for (int s = lane; s < s1 - s0; s += 32) m = fmaxf(m, sc[g * max_chunk + s]);
    m = warp_max(m);
    float l = 0.f;
    for (int s = lane; s < s1 - s0; s += 32) {
      const float e = expf(sc[g * max_chunk + s] - m);
      sc[g * max_chunk + s] = e;
      l += e;
    }
    l = warp_sum(l);
    if (lane == 0) { out[g * (HD + 2) + HD] = m; out[g * (HD + 2) + HD + 1] = l; }
  }
  __syncwarp();
  float acc[ND][P][GQA];
#pragma unroll
  for (int k = 0; k < ND; ++k)
#pragma unroll
    for (int grp = 0; grp < P; ++grp)
#pragma unroll
      for (int g = 0; g < GQA; ++g) acc[k][grp][g] = 0.f;
  for (int rb = 0; s0 + 8 * rb < s1; rb += P) {
#pragma unroll
    for (int grp = 0; grp < P; ++grp) {
      const int sb = s0 + 8 * (rb + grp);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (sb + j < s1) {
          float e[GQA], v[ND];
          const float* vrow = src.v(sb + j);
#pragma unroll
          for (int g = 0; g < GQA; ++g) e[g] = sc[g * max_chunk + (sb + j - s0)];
#pragma unroll
          for (int k = 0; k < ND; ++k) v[k] = vrow[lane + 32 * k];
#pragma unroll
          for (int k = 0; k < ND; ++k)
#pragma unroll
            for (int g = 0; g < GQA; ++g) acc[k][grp][g] = fmaf(e[g], v[k], acc[k][grp][g]);
        }
    }
  }
#pragma unroll
  for (int k = 0; k < ND; ++k)
#pragma unroll
    for (int g = 0; g < GQA; ++g) {
      float total = 0.f;
#pragma unroll
      for (int grp = 0; grp < P; ++grp) total += acc[k][grp][g];
      out[g * (HD + 2) + lane + 32 * k] = total;
    }
}

// grid (kv head, position slice, run of up to ATT_ROWS rows of one sequence): the rows share the slice's key and value rows,
// which the block stages in shared memory once; each warp then takes rows of its own, with no block-wide barrier between rows.
// (A block that took the next sixteen rows of a ragged batch, whatever their sequences, staged a slice per sequence one after
// the other: 24 rows of 24 sequences 129 us.)
template <int GQA, int P>
__global__ void __launch_bounds__(ATT_THREADS, 3)
attention_tile_kernel(const float* q, KvView kv, float* __restrict__ part, RowMap rows, int layer, int chunk,
                      WalkShape w, const __grid_constant__ RowTiles tiles) {
  pdl_enter();
  extern __shared__ float sm[];  // k tile [chunk][hd] | v tile [chunk][hd] | per warp: q[gqa][hd], scores[gqa][chunk]
  constexpr int hd = ATT_THREADS / P, gqa = GQA;
  const int hkv = blockIdx.x, split = blockIdx.y;
  const int n_split = (int)gridDim.y;
  const int s0 = split * chunk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = ATT_THREADS / 32;
  float* kt = sm;
  float* vt = kt + chunk * hd;
  float* sq = vt + chunk * hd + warp * gqa * hd;
  float* sc = vt + chunk * hd + nw * gqa * hd + warp * gqa * chunk;
  // the last rows first: in a prompt chunk they attend to the most slices, the blocks of the first rows (which leave at once for
  // the slices beyond them) then fill the tail
  const int t_begin = tiles.begin((int)gridDim.z - 1 - (int)blockIdx.z), t_end = tiles.end((int)gridDim.z - 1 - (int)blockIdx.z);
  const int sid = row_sequence(rows, t_begin), p0 = row_position(rows, t_begin);
  // positions [s0, s0 + need) lie in blocks the sequence owns: a row's position is below its reserved length
  const int need = min(p0 + t_end - t_begin, s0 + chunk) - s0;
  if (need <= 0) return;
  constexpr int vec = hd / 4;
  for (int idx = threadIdx.x; idx < need * vec; idx += ATT_THREADS) {
    const int p = idx / vec, c = idx % vec;
    const int64_t off = kv_offset(kv, sid, layer, hkv, s0 + p, w.n_head_kv, hd);
    ((float4*)(kt + p * hd))[c] = ((const float4*)(kv.k + off))[c];
    ((float4*)(vt + p * hd))[c] = ((const float4*)(kv.v + off))[c];
  }
  __syncthreads();
  for (int r = t_begin + warp; r < t_end; r += nw) {
    const int seq = p0 + r - t_begin + 1;
    if (s0 >= seq) continue;
    const int s1 = min(seq, s0 + chunk);
    for (int i = lane; i < gqa * hd; i += 32) sq[i] = q[((int64_t)r * w.n_head + hkv * gqa) * hd + i];
    __syncwarp();
    float* out = part + (((int64_t)r * w.n_head_kv + hkv) * n_split + split) * gqa * (hd + 2);
    attend_slice_warp<GQA, P>(KvTile{kt, vt, s0, hd}, sq, sc, out, s0, s1, chunk);
    __syncwarp();
  }
}

// Rows that the tensor-core kernel has finished: at most eight groups of 64 rows and more in a batch of 512.
struct RowRanges {
  int n, lo[8], hi[8];
  __device__ __forceinline__ bool has(int t) const {
    for (int i = 0; i < n; ++i)
      if (t >= lo[i] && t < hi[i]) return true;
    return false;
  }
};

// grid (query heads / 4, token), one warp per query head: merges the position slices (at most 32).  Lane sp turns
// slice sp's maximum into the weight exp(m_slice - m); the denominator is the shuffle-tree sum of the weighted slice
// sums; then every lane adds its dimensions over the slices in ascending order, the weights coming by shuffle.
__global__ void __launch_bounds__(128)
attention_combine_kernel(const float* part, float* __restrict__ out, RowMap rows, int chunk, WalkShape w, int heads_per_block,
                         const __grid_constant__ RowRanges finished) {
  pdl_enter();
  // heads_per_block 4: one warp per head (many rows: fewer, fuller blocks); 1: the four warps share a head's
  // dimensions (a decode step has few blocks to fill the device with)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int hq = heads_per_block == 4 ? blockIdx.x * 4 + warp : blockIdx.x, t = blockIdx.y;
  if (hq >= w.n_head) return;
  const int d0 = heads_per_block == 4 ? lane : lane + 32 * warp, dstep = heads_per_block == 4 ? 32 : 128;
  const int hd = w.head_dim, gqa = w.n_head / w.n_head_kv;
  const int hkv = hq / gqa, g = hq % gqa;
  const int seq = row_position(rows, t) + 1;
  if (finished.has(t)) return;  // behind the load: the list's first look into the constant bank takes as long
  const int n_split = (w.n_ctx + chunk - 1) / chunk, used = min(n_split, (seq + chunk - 1) / chunk);
  const float* base = part + ((int64_t)t * w.n_head_kv + hkv) * n_split * gqa * (hd + 2) + g * (hd + 2);
  const int64_t stride = (int64_t)gqa * (hd + 2);
  const float ms = lane < used ? base[lane * stride + hd] : -CUDART_INF_F;
  const float m = warp_max(ms);
  const float e = lane < used ? expf(ms - m) : 0.f;
  const float l = warp_sum(lane < used ? base[lane * stride + hd + 1] * e : 0.f);
  float acc[8];  // head_dim <= 256: up to eight dimensions per lane, all in flight at once
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  for (int sp0 = 0; sp0 < used; sp0 += 4) {  // four slices' records are fetched before the first is used
    float v[4][8];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 8; ++k) v[j][k] = (sp0 + j < used && d0 + dstep * k < hd) ? base[(sp0 + j) * stride + d0 + dstep * k] : 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float es = __shfl_sync(0xffffffffu, e, (sp0 + j) & 31);
      if (sp0 + j < used) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (d0 + dstep * k < hd) acc[k] = fmaf(v[j][k], es, acc[k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (d0 + dstep * k < hd) out[((int64_t)t * w.n_head + hq) * hd + d0 + dstep * k] = l > 0.f ? __fdiv_rn(acc[k], l) : 0.f;
}

__device__ __forceinline__ float swiglu_of(float a, float b) { return __fmul_rn(__fdiv_rn(a, 1.0f + expf(-a)), b); }  // silu(gate) * up (decode.rs:11826, :2984)
__global__ void swiglu_kernel(float* g, const float* u, int64_t n) {
  pdl_enter();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) g[i] = swiglu_of(g[i], u[i]);
}
// the same, four elements per thread and step (n4 = n / 4; g and u 16-byte aligned)
__global__ void swiglu4_kernel(float4* g, const float4* u, int64_t n4) {
  pdl_enter();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 a = g[i], b = u[i];
    g[i] = make_float4(swiglu_of(a.x, b.x), swiglu_of(a.y, b.y), swiglu_of(a.z, b.z), swiglu_of(a.w, b.w));
  }
}
__global__ void add_kernel(float* x, const float* y, int64_t n) {
  pdl_enter();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = __fadd_rn(y[i], x[i]);
}

// one block: index of the first strict maximum (sample.rs:293: `v > best` scanning upwards, so ties go to the
// lower index), its margin over the largest other value, and the position counter advanced for the next step
__global__ void __launch_bounds__(1024)
argmax_kernel(const float* logits, int n, int* __restrict__ out_id, float* __restrict__ out_margin,
              int* pos_dev, int advance, int* count_dev) {
  pdl_enter();
  // with count_dev: out_id[0] is the slot the next step reads its token from, and the token and its margin are also
  // appended at out_id[1 + *count_dev] / out_margin[*count_dev]: every step of a generation is then the same launch
  const int slot = count_dev ? *count_dev : 0;
  logits += (int64_t)blockIdx.x * n;  // one block per row of logits (a single row unless launch_argmax_rows)
  out_id += blockIdx.x;
  if (out_margin) out_margin += blockIdx.x;
  __shared__ float sv[32];
  __shared__ int si[32];
  __shared__ int s_best;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (n > 0) {
    float best = -CUDART_INF_F;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const float v = logits[i];
      if (v > best) { best = v; bi = i; }  // ascending i per thread: the first of equal values stays
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(~0u, best, o);
      const int oi = __shfl_xor_sync(~0u, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
      best = lane < nw ? sv[lane] : -CUDART_INF_F;
      bi = lane < nw ? si[lane] : 0x7fffffff;
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(~0u, best, o);
        const int oi = __shfl_xor_sync(~0u, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      if (lane == 0) s_best = bi == 0x7fffffff ? 0 : bi;  // all NaN or -inf: index 0, as the reference's scan leaves it
    }
    __syncthreads();
    const int win = s_best;
    if (out_margin) {
      float second = -CUDART_INF_F;
      for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (i != win) second = fmaxf(second, logits[i]);
      second = warp_max(second);
      __syncthreads();
      if (lane == 0) sv[warp] = second;
      __syncthreads();
      if (threadIdx.x == 0) {
        float m = -CUDART_INF_F;
        for (int w = 0; w < nw; ++w) m = fmaxf(m, sv[w]);
        out_margin[slot] = logits[win] - m;
      }
    }
    if (threadIdx.x == 0) {
      out_id[0] = win;
      if (count_dev) { out_id[1 + slot] = win; *count_dev = slot + 1; }
    }
  }
  if (threadIdx.x == 0 && pos_dev) *pos_dev += advance;
}

// Two-stage argmax of one long row (a vocabulary): ARG_BLOCKS blocks each reduce a contiguous range to (best value, its
// first index, largest other value of the range); one block merges the ranges in ascending order, so the first of equal
// maxima still wins (sample.rs:293), and applies the bookkeeping of argmax_kernel.
constexpr int ARG_BLOCKS = 128;
__global__ void __launch_bounds__(256)
argmax_part_kernel(const float* logits, int n, float* __restrict__ pbest, int* __restrict__ pidx, float* __restrict__ psecond) {
  pdl_enter();
  __shared__ float sv[8], s2[8];
  __shared__ int si[8];
  const int per = (n + gridDim.x - 1) / gridDim.x;
  const int lo = blockIdx.x * per, hi = min(n, lo + per);
  float best = -CUDART_INF_F, second = -CUDART_INF_F;
  int bi = 0x7fffffff;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const float v = logits[i];
    if (v > best) { second = best; best = v; bi = i; }
    else second = fmaxf(second, v);
  }
  // merge (best, index, second) of two disjoint sets: the larger best wins, ties to the lower index; the loser's best
  // and both seconds compete for second place
  auto merge = [](float& b, int& i, float& s, float ob, int oi, float os) {
    const bool other = ob > b || (ob == b && oi < i);
    const float loser = other ? b : ob;
    s = fmaxf(fmaxf(s, os), loser);
    if (other) { b = ob; i = oi; }
  };
  for (int o = 16; o > 0; o >>= 1) {
    const float ob = __shfl_xor_sync(~0u, best, o), os = __shfl_xor_sync(~0u, second, o);
    const int oi = __shfl_xor_sync(~0u, bi, o);
    merge(best, bi, second, ob, oi, os);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { sv[warp] = best; si[warp] = bi; s2[warp] = second; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) merge(best, bi, second, sv[w], si[w], s2[w]);
    pbest[blockIdx.x] = best; pidx[blockIdx.x] = bi; psecond[blockIdx.x] = second;
  }
}
__global__ void __launch_bounds__(ARG_BLOCKS)
argmax_merge_kernel(const float* pbest, const int* pidx, const float* psecond, int parts,
                    int* __restrict__ out_id, float* __restrict__ out_margin, int* pos_dev, int advance,
                    int* count_dev) {
  pdl_enter();
  if (threadIdx.x != 0) return;  // a hundred-odd triples: one thread, ascending order
  float best = -CUDART_INF_F, second = -CUDART_INF_F;
  int bi = 0x7fffffff;
  for (int p = 0; p < parts; ++p) {
    const float ob = pbest[p], os = psecond[p];
    const int oi = pidx[p];
    const bool other = ob > best || (ob == best && oi < bi);
    const float loser = other ? best : ob;
    second = fmaxf(fmaxf(second, os), loser);
    if (other) { best = ob; bi = oi; }
  }
  const int win = bi == 0x7fffffff ? 0 : bi;
  const int slot = count_dev ? *count_dev : 0;
  out_id[0] = win;
  if (out_margin) out_margin[slot] = best - second;
  if (count_dev) { out_id[1 + slot] = win; *count_dev = slot + 1; }
  if (pos_dev) *pos_dev += advance;
}

__global__ void __launch_bounds__(256) table_entries_kernel(int* __restrict__ table, const int* __restrict__ entries, int n) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) table[(uint32_t)entries[2 * i]] = entries[2 * i + 1];
}

// positions per attention slice: 32, or a thirty-second of the context when that is longer
int attention_chunk(const WalkShape& w) {
  const int c = (w.n_ctx + 31) / 32;
  return c > 32 ? c : 32;
}
int attention_splits(const WalkShape& w) {
  const int c = attention_chunk(w);
  return (w.n_ctx + c - 1) / c;
}

}  // namespace

cudaError_t launch_rmsnorm(float* x, const float* add, const float* w, float* y, int tokens, int n, float eps,
                           cudaStream_t s, uint64_t* launches) {
  if (tokens <= 0) return cudaSuccess;
  if (launches) ++*launches;
  return launch_walk(rmsnorm_kernel, dim3(tokens), dim3(NORM_THREADS), 0, s, x, add, w, y, n, eps);
}

cudaError_t launch_rope_store(float* q, float* k, const float* v, const KvView& kv, const RowMap& rows, int tokens, int layer,
                              const WalkShape& w, cudaStream_t s, uint64_t* launches) {
  if (tokens <= 0) return cudaSuccess;
  if (launches) ++*launches;
  return launch_walk(rope_store_kernel, dim3(tokens), dim3(256), 0, s, q, k, v, kv, rows, layer, w);
}

// the walk's attention as the tensor-core kernel knows it: no window, no bias
static SpanShape span_shape(const WalkShape& w) {
  SpanShape sh{};
  sh.n_head = w.n_head; sh.n_kv = w.n_head_kv; sh.dk = sh.dv = w.head_dim; sh.n_ctx = w.n_ctx;
  sh.scale = 1.0f / sqrtf((float)w.head_dim);
  sh.saturate = false;  // a model whose values leave binary16's range shows it in its logits
  sh.split_weights = true;
  return sh;
}

size_t attention_scratch_floats(int tokens, size_t positions, const WalkShape& w) {
  SpanShape sh = span_shape(w);
  sh.n_ctx = (int)std::min<size_t>(w.n_ctx, positions);
  return std::max((size_t)tokens * w.n_head_kv * attention_splits(w) * (w.n_head / w.n_head_kv) * (w.head_dim + 2), span_umma_scratch_floats(sh, tokens));
}

// The per-row kernels for the heads per group of a shape (the smallest of 1, 2, 4, 8 that holds them) and their shared memory,
// checked and allowed
struct RowKernels {
  void (*partial)(const float*, KvView, float*, RowMap, int, int, WalkShape, const float*, const float*);
  void (*rows)(const float*, KvView, float*, RowMap, int, int, WalkShape, const RowTiles);
  size_t smem;
};
template <int G>
static cudaError_t allow_rows(RowKernels* k) {
  k->partial = attention_partial_kernel<G>;
  k->rows = attention_rows_kernel<G>;
  static PerDevice configured;  // per instantiation: the largest size the kernels have been allowed on this device
  std::atomic<int>& allowed = configured.here();
  if (k->smem > 48 * 1024 && (int)k->smem > allowed.load(std::memory_order_relaxed)) {
    cudaError_t e = cudaFuncSetAttribute(k->partial, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k->smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k->rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k->smem);
    if (e != cudaSuccess) return e;
    allowed.store((int)k->smem, std::memory_order_relaxed);
  }
  return cudaSuccess;
}
static cudaError_t attention_row_kernels(const WalkShape& w, RowKernels* k) {
  const int gqa = w.n_head / w.n_head_kv, max_chunk = attention_chunk(w);
  if (gqa < 1 || gqa > ATT_MAX_GQA || w.n_head % w.n_head_kv != 0 || w.head_dim > ATT_THREADS) return cudaErrorInvalidValue;
  const size_t groups = ATT_THREADS / w.head_dim > 0 ? ATT_THREADS / w.head_dim : 1;
  const size_t score_floats = (size_t)gqa * max_chunk > groups * gqa * w.head_dim ? (size_t)gqa * max_chunk : groups * gqa * w.head_dim;
  const size_t floats = (size_t)gqa * w.head_dim + score_floats + 32;
  if (floats * sizeof(float) > 200 * 1024) return cudaErrorInvalidValue;
  k->smem = (floats + (size_t)slot_words(max_chunk, w.head_dim)) * sizeof(float);
  return gqa == 1 ? allow_rows<1>(k) : gqa == 2 ? allow_rows<2>(k) : gqa <= 4 ? allow_rows<4>(k) : allow_rows<8>(k);
}

cudaError_t launch_attention(const float* q, const KvView& kv, float* out, float* scratch, const RowMap& rows, int layer, const WalkShape& w, cudaStream_t s,
                             uint64_t* launches, const float* k_new, const float* v_new) {
  RowKernels row;
  cudaError_t e = attention_row_kernels(w, &row);
  if (e != cudaSuccess) return e;
  const int splits = attention_splits(w), chunk = attention_chunk(w);
  if (launches) *launches += 2;
  e = launch_walk(row.partial, dim3(w.n_head_kv, splits, 1), dim3(ATT_THREADS), row.smem, s, q, kv, scratch, rows, layer, chunk, w, k_new, v_new);
  if (e != cudaSuccess) return e;
  return launch_walk(attention_combine_kernel, dim3(w.n_head, 1), dim3(128), 0, s, (const float*)scratch, out, rows, chunk, w, 1, RowRanges{});
}

cudaError_t launch_attention_groups(const float* q, const KvView& kv, float* out, float* scratch, const RowMap& rows, int tokens, int layer, const WalkShape& w,
                                    const AttentionGroup* groups, int n_groups, bool tensor_cores, size_t scratch_floats, cudaStream_t s, int* err,
                                    uint64_t* launches) {
  if (tokens <= 0) return cudaSuccess;
  if (tokens > MAX_TILES) return cudaErrorInvalidValue;
  const int gqa = w.n_head_kv > 0 ? w.n_head / w.n_head_kv : 0;
  RowKernels row;
  cudaError_t e = attention_row_kernels(w, &row);
  if (e != cudaSuccess) return e;
  const int splits = attention_splits(w);
  const int max_chunk = attention_chunk(w);
  const AttentionGroup all{0, tokens, rows.first};
  if (!groups) { groups = &all; n_groups = 1; }
  // prompt chunks: rows of a group share the slice's keys and values through a shared-memory tile
  const size_t tile_smem = (2 * (size_t)max_chunk * w.head_dim + (ATT_THREADS / 32) * ((size_t)gqa * w.head_dim + (size_t)gqa * max_chunk)) * sizeof(float);
  void (*tile)(const float*, KvView, float*, RowMap, int, int, WalkShape, const RowTiles) = nullptr;
#define LLR_TILE(G, PP) if (gqa == G && w.head_dim == ATT_THREADS / PP) tile = attention_tile_kernel<G, PP>;
  LLR_TILE(1, 1) LLR_TILE(2, 1) LLR_TILE(4, 1) LLR_TILE(1, 2) LLR_TILE(2, 2) LLR_TILE(4, 2) LLR_TILE(8, 2)
  LLR_TILE(1, 4) LLR_TILE(2, 4) LLR_TILE(4, 4) LLR_TILE(8, 4)
#undef LLR_TILE
  if (max_chunk > ATT_TILE_CHUNK || tile_smem > 200 * 1024) tile = nullptr;
  // groups long enough, when the caller allows 16-bit operands: tensor cores
  const SpanShape span = span_shape(w);
  const SpanOut to_out{out, nullptr, (int64_t)w.n_head * w.head_dim, nullptr, 0, false, 1.0f};
  const bool mma = tensor_cores && (w.head_dim == 64 || w.head_dim == 128) && (gqa & (gqa - 1)) == 0 && span_umma_supported(span, false, to_out);
  // Every group goes to one of three kernels, one launch each: binary16 MMAs (64 rows and more), the tiled f32 kernel (four rows
  // and more: below that a block of eight warps would have work for one to three), the f32 kernel of a block per row.
  RowTiles tiled{}, single{};
  RowRanges finished{};
  SpanGroup big[8];
  int left = 0;
  for (int g = 0; g < n_groups; ++g) {
    const int first = groups[g].first, n = groups[g].rows;
    if (mma && n >= 64 && finished.n < 8) {
      big[finished.n] = SpanGroup{first, n, groups[g].position};
      finished.lo[finished.n] = first;
      finished.hi[finished.n++] = first + n;
      continue;
    }
    RowTiles& to = tile && n >= 4 ? tiled : single;
    const int per = tile && n >= 4 ? ATT_ROWS : 1;
    for (int r = 0; r < n; r += per) to.run[to.n++] = (uint32_t)std::min(per, n - r) << 16 | (uint32_t)(first + r);
    left += n;
  }
  if (finished.n) {
    const int64_t page = (int64_t)kv.n_layer * w.n_head_kv * kv.block_tokens * w.head_dim, at = (int64_t)layer * w.n_head_kv * kv.block_tokens * w.head_dim;
    const LayerKv pages{kv.k + at, kv.v + at, kv.table, kv.block_tokens, kv.max_blocks, page, page};
    e = launch_span_umma(q, (int64_t)w.n_head * w.head_dim, span, pages, rows, big, finished.n, 1, to_out, scratch, scratch_floats, s, err, launches);
    if (e != cudaSuccess || left == 0) return e;
  }
  if (tiled.n) {
    if (launches) ++*launches;
    if (tile_smem > 48 * 1024 && (e = cudaFuncSetAttribute((const void*)tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_smem)) != cudaSuccess) return e;
    e = launch_walk(tile, dim3(w.n_head_kv, splits, tiled.n), dim3(ATT_THREADS), tile_smem, s, q, kv, scratch, rows, layer, max_chunk, w, tiled);
    if (e != cudaSuccess) return e;
  }
  if (single.n) {
    if (launches) ++*launches;
    e = launch_walk(row.rows, dim3(w.n_head_kv, splits, single.n), dim3(ATT_THREADS), row.smem, s, q, kv, scratch, rows, layer, max_chunk, w, single);
    if (e != cudaSuccess) return e;
  }
  if (launches) ++*launches;
  return launch_walk(attention_combine_kernel, dim3(tokens >= 16 ? (w.n_head + 3) / 4 : w.n_head, tokens), dim3(128), 0, s, (const float*)scratch, out, rows,
                     max_chunk, w, tokens >= 16 ? 4 : 1, finished);
}

cudaError_t launch_swiglu(float* g, const float* u, int64_t n, cudaStream_t s, uint64_t* launches) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (launches) ++*launches;
  if (n % 4 == 0 && (((uintptr_t)g | (uintptr_t)u) & 15) == 0) {
    int64_t b4 = (n / 4 + 255) / 256;
    if (b4 > 148 * 8) b4 = 148 * 8;
    return launch_walk(swiglu4_kernel, dim3((unsigned)b4), dim3(256), 0, s, (float4*)g, (const float4*)u, n / 4);
  }
  return launch_walk(swiglu_kernel, dim3((unsigned)blocks), dim3(256), 0, s, g, u, n);
}

cudaError_t launch_table_entries(int* table, const int* entries, int n, cudaStream_t s, uint64_t* launches) {
  if (n <= 0) return cudaSuccess;
  if (launches) ++*launches;
  table_entries_kernel<<<(n + 255) / 256, 256, 0, s>>>(table, entries, n);
  return cudaGetLastError();
}

cudaError_t launch_add(float* x, const float* y, int64_t n, cudaStream_t s, uint64_t* launches) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (launches) ++*launches;
  return launch_walk(add_kernel, dim3((unsigned)blocks), dim3(256), 0, s, x, y, n);
}

cudaError_t launch_argmax_rows(const float* logits, int n_rows, int n, int* out_id, float* out_margin, cudaStream_t s,
                               uint64_t* launches) {
  if (n_rows <= 0) return cudaSuccess;
  if (launches) ++*launches;
  return launch_walk(argmax_kernel, dim3(n_rows), dim3(1024), 0, s, logits, n, out_id, out_margin, (int*)nullptr, 0, (int*)nullptr);
}

cudaError_t launch_argmax_advance(const float* logits, int n, int* out_id, float* out_margin, int* pos_dev, int advance,
                                  int* count_dev, float* part, cudaStream_t s, uint64_t* launches) {
  if (n >= 16384 && part) {  // a vocabulary: spread the scan over the device (part: 3 * ARG_BLOCKS words of scratch)
    if (launches) *launches += 2;
    cudaError_t e = launch_walk(argmax_part_kernel, dim3(ARG_BLOCKS), dim3(256), 0, s, logits, n, part, (int*)(part + ARG_BLOCKS), part + 2 * ARG_BLOCKS);
    if (e != cudaSuccess) return e;
    return launch_walk(argmax_merge_kernel, dim3(1), dim3(ARG_BLOCKS), 0, s, (const float*)part, (const int*)(part + ARG_BLOCKS),
                       (const float*)(part + 2 * ARG_BLOCKS), (int)ARG_BLOCKS, out_id, out_margin, pos_dev, advance, count_dev);
  }
  if (launches) ++*launches;
  return launch_walk(argmax_kernel, dim3(1), dim3(1024), 0, s, logits, n, out_id, out_margin, pos_dev, advance, count_dev);
}

}  // namespace llr
