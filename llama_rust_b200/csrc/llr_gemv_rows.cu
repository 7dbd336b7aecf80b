// Products of the element formats F32, F16 and BF16 in f32 arithmetic, any number of activation rows: gemv_f32 / gemv_f16 of
// langtax/src/quant.rs (:6191, :6144) and their gemm twins.
//
// These formats need no unpacking, so one or two activation rows are a plain stream: one warp per weight row, every lane pulls
// 16-byte pieces of the row straight from HBM with streaming loads (several pieces in flight per lane, no shared
// memory in between), multiplies them into f32 accumulators against activations that stay in L1, and the warp
// finishes with shuffles.  Bound: HBM.  Algorithmic bytes per weight: 4 (F32), 2 (F16, BF16).  More rows share the weights in passes of
// eight or sixteen (gemv_rows_wide_kernel).
// Rows must start 16-byte aligned and hold a multiple of eight columns; other shapes take the shape-agnostic kernel.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "llr_formats.cuh"
#include "llr_kernels.cuh"

namespace llr {
namespace {

constexpr int ROW_WARPS = 8;
// 16-byte pieces in flight per lane: 8 for the 2-byte formats, 4 pairs for F32 (128 bytes per lane either way)
template <int DT> struct Unroll { static constexpr int N = DT == DT_F32 ? 4 : 8; };

__device__ __forceinline__ uint4 ld_stream16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// The raw 16-byte pieces that hold eight consecutive weights starting at element index c of the row: kept as they
// come (32 bytes for F32, 16 for the 2-byte formats) and widened only when they are used, so that the pieces in
// flight cost a quarter of the registers their f32 values would and four CTAs fit an SM.
template <int DT> struct Raw8 { uint4 a, b; };
template <int DT> __device__ __forceinline__ void fetch8(const uint8_t* row, int64_t c, Raw8<DT>& r) {
  if constexpr (DT == DT_F32) {
    r.a = ld_stream16(row + 4 * c);
    r.b = ld_stream16(row + 4 * c + 16);
  } else {
    r.a = ld_stream16(row + 2 * c);
  }
}
template <int DT> __device__ __forceinline__ void widen8(const Raw8<DT>& r, float (&w)[8]) {
  if constexpr (DT == DT_F32) {
    w[0] = __uint_as_float(r.a.x); w[1] = __uint_as_float(r.a.y); w[2] = __uint_as_float(r.a.z); w[3] = __uint_as_float(r.a.w);
    w[4] = __uint_as_float(r.b.x); w[5] = __uint_as_float(r.b.y); w[6] = __uint_as_float(r.b.z); w[7] = __uint_as_float(r.b.w);
  } else {
    const uint32_t u[4] = {r.a.x, r.a.y, r.a.z, r.a.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if constexpr (DT == DT_F16) {
        // exact for every finite value, infinities included; NaN payloads are a matter of the dequantizer, not of a dot product
        const float2 f = __half22float2(*(const __half2*)&u[k]);
        w[2 * k] = f.x; w[2 * k + 1] = f.y;
      } else {
        w[2 * k] = __uint_as_float(u[k] << 16);
        w[2 * k + 1] = __uint_as_float(u[k] & 0xffff0000u);
      }
    }
  }
}

template <int DT, int MT>
__global__ void __launch_bounds__(ROW_WARPS * 32, DT == DT_F32 ? 2 : 4)
gemv_rows_kernel(const uint8_t* __restrict__ W, int64_t row_bytes, int64_t rows, int64_t cols,
                 const float* __restrict__ X, float* __restrict__ Y, int tokens) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
  const int64_t n_warps = (int64_t)gridDim.x * ROW_WARPS;
  for (int64_t row = warp; row < rows; row += n_warps) {
    const uint8_t* wr = W + row * row_bytes;
    float acc[MT];
#pragma unroll
    for (int t = 0; t < MT; ++t) acc[t] = 0.f;
    constexpr int UNROLL = Unroll<DT>::N;
    for (int64_t c0 = 8 * lane; c0 < cols; c0 += 256 * UNROLL) {
      Raw8<DT> raw[UNROLL];
#pragma unroll
      for (int i = 0; i < UNROLL; ++i)
        if (c0 + 256 * i < cols) fetch8<DT>(wr, c0 + 256 * i, raw[i]);
#pragma unroll
      for (int i = 0; i < UNROLL; ++i) {
        const int64_t c = c0 + 256 * i;
        if (c < cols) {
          float w[8];
          widen8<DT>(raw[i], w);
#pragma unroll
          for (int t = 0; t < MT; ++t)
            if (t < tokens) {
              const float4* xp = (const float4*)(X + (int64_t)t * cols + c);
              const float4 a = __ldg(xp), b = __ldg(xp + 1);
              float s = acc[t];
              s = fmaf(w[0], a.x, s); s = fmaf(w[1], a.y, s); s = fmaf(w[2], a.z, s); s = fmaf(w[3], a.w, s);
              s = fmaf(w[4], b.x, s); s = fmaf(w[5], b.y, s); s = fmaf(w[6], b.z, s); s = fmaf(w[7], b.w, s);
              acc[t] = s;
            }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      float v = acc[t];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
      if (lane == 0 && t < tokens) Y[(int64_t)t * rows + row] = v;
    }
  }
}

// Three rows of activations and more.  The kernel above reads every activation from L1 once per weight row: with eight of them a
// warp moves 16 bytes of activations per byte of BF16 weights, and the load path, not HBM, sets the time (32000 x 2048 BF16,
// eight rows: 144 us for 131 MB).  Here a warp works on R weight rows, the CTA's warps share a tile of the activations in shared
// memory, and each value read from it serves R rows.  Activations of two rows lie side by side in the tile, so that one
// fma.rn.f32x2 carries two sums.  A sum is formed as above: per lane in ascending columns, then the shuffles; a row's result
// is the same alone and in a batch of up to 32 rows.  Bound: the FMA pipe and the shared-memory reads, which four weight rows per warp balance.
// Measured, 32000 x 2048 BF16: 3 / 8 / 16 rows 62 / 144 / 287 -> 37 / 49 / 92 us; 4096 x 4104 F32, 7 rows 59 -> 25 us.
// RUNS (batches of more than 32 rows): a lane's sum is closed every 512 columns (256 up to RUN_COLS columns) and added to the row's.  The
// staged kernel, which served such batches at 8 rows per pass (14336 x 4096 F16, 100 rows: 2234 us), rounds as runs of 256 do: relative
// error 1.01e-7 at 2304 columns, 1.12e-7 at 4096, 1.33e-7 at 8192, 2.1e-7 at 28672.  Runs of 512 have 1.05, 1.11, 1.22, 1.7e-7 on
// inputs of one size, and up to a tenth more than runs of 256 on inputs of very different sizes until about 6000 columns.
constexpr int64_t RUN_COLS = 6144;
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ void fma2(unsigned long long& s, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s) : "l"(a), "l"(b));
}
template <int T> struct WideTile { static constexpr int SLOTS = T / 2 * 4 * 32; };  // 16-byte slots: (pair of rows, two columns, lane)
template <int DT, int T, int R, bool RUNS, int S>  // S: 256-column steps that a tile holds
__global__ void __launch_bounds__(ROW_WARPS * 32, S > 1 || R * T * (DT == DT_F32 || RUNS ? 2 : 1) >= 64 ? 1 : 2)
gemv_rows_wide_kernel(const uint8_t* __restrict__ W, int64_t row_bytes, int64_t rows, int64_t cols, const float* __restrict__ X,
                      float* __restrict__ Y, int tokens) {
  constexpr int NP = T / 2, PIECES = S * NP * 64, FILL = (PIECES + ROW_WARPS * 32 - 1) / (ROW_WARPS * 32);  // float4 pairs of a tile, per thread
  constexpr int SLOTS = WideTile<T>::SLOTS;
  __shared__ __align__(16) uint4 tile[2][S * SLOTS];
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t row0 = (int64_t)blockIdx.x * (ROW_WARPS * R) + (tid >> 5) * R;
  const uint8_t* wr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) wr[r] = W + (row0 + r < rows ? row0 + r : rows - 1) * row_bytes;
  unsigned long long acc[R][NP], sum[RUNS ? R : 1][RUNS ? NP : 1];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      acc[r][p] = 0ull;
      if (RUNS) sum[r][p] = 0ull;
    }

  float4 xa[FILL], xb[FILL];
  auto load_x = [&](int64_t c0) {  // four columns of two activation rows per piece; rows and columns beyond the end are zeros
#pragma unroll
    for (int f = 0; f < FILL; ++f) {
      const int piece = f * ROW_WARPS * 32 + tid, p = (piece >> 6) % NP;
      const int64_t c = c0 + 256 * (piece / (NP * 64)) + 4 * (piece & 63);
      xa[f] = xb[f] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (piece < PIECES && c < cols) {
        if (2 * p < tokens) xa[f] = __ldg((const float4*)(X + (int64_t)(2 * p) * cols + c));
        if (2 * p + 1 < tokens) xb[f] = __ldg((const float4*)(X + (int64_t)(2 * p + 1) * cols + c));
      }
    }
  };
  auto store_x = [&](int buf) {
#pragma unroll
    for (int f = 0; f < FILL; ++f) {
      const int piece = f * ROW_WARPS * 32 + tid, p = (piece >> 6) % NP, q = piece & 63;
      if (piece >= PIECES) break;
      float4* at = (float4*)&tile[buf][piece / (NP * 64) * SLOTS + (p * 4 + 2 * (q & 1)) * 32 + (q >> 1)];
      at[0] = make_float4(xa[f].x, xb[f].x, xa[f].y, xb[f].y);
      at[32] = make_float4(xa[f].z, xb[f].z, xa[f].w, xb[f].w);
    }
  };
  Raw8<DT> raw[2][S][R];
  auto load_w = [&](int64_t c0, Raw8<DT> (&to)[S][R]) {
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const int64_t c = c0 + 256 * j + 8 * lane;
      if (c < cols) {
#pragma unroll
        for (int r = 0; r < R; ++r) fetch8<DT>(wr[r], c, to[j][r]);
      }
    }
  };
  load_w(0, raw[0]);
  load_x(0);
  store_x(0);
  __syncthreads();
  auto step = [&](int64_t c0, int buf, Raw8<DT> (&now)[S][R], Raw8<DT> (&next)[S][R]) {
    load_w(c0 + 256 * S, next);
    load_x(c0 + 256 * S);
#pragma unroll
    for (int j = 0; j < S; ++j)
      if (c0 + 256 * j + 8 * lane < cols) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // four columns at a time
          unsigned long long w2[R][4];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            float w[8];
            widen8<DT>(now[j][r], w);
#pragma unroll
            for (int k = 0; k < 4; ++k) w2[r][k] = pack2(w[4 * h + k], w[4 * h + k]);
          }
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const ulonglong2 u = *(const ulonglong2*)&tile[buf][j * SLOTS + (p * 4 + 2 * h) * 32 + lane];
            const ulonglong2 v = *(const ulonglong2*)&tile[buf][j * SLOTS + (p * 4 + 2 * h + 1) * 32 + lane];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              fma2(acc[r][p], w2[r][0], u.x); fma2(acc[r][p], w2[r][1], u.y);
              fma2(acc[r][p], w2[r][2], v.x); fma2(acc[r][p], w2[r][3], v.y);
            }
          }
        }
      }
    store_x(buf ^ 1);
    __syncthreads();
  };
  auto close_run = [&] {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum[RUNS ? r : 0][RUNS ? p : 0]) : "l"(acc[r][p]));
        acc[r][p] = 0ull;
      }
  };
  static_assert(!RUNS || S == 1, "runs are closed between steps");
  for (int64_t c0 = 0; c0 < cols; c0 += 512 * S) {
    step(c0, 0, raw[0], raw[1]);
    if (RUNS && cols <= RUN_COLS) close_run();
    if (c0 + 256 * S < cols) step(c0 + 256 * S, 1, raw[1], raw[0]);
    if (RUNS) close_run();
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const unsigned long long v = RUNS ? sum[RUNS ? r : 0][RUNS ? p : 0] : acc[r][p];
      float a = __uint_as_float((uint32_t)v), b = __uint_as_float((uint32_t)(v >> 32));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) { a += __shfl_xor_sync(~0u, a, o); b += __shfl_xor_sync(~0u, b, o); }
      if (lane == 0 && row0 + r < rows) {
        if (2 * p < tokens) Y[(int64_t)(2 * p) * rows + row0 + r] = a;
        if (2 * p + 1 < tokens) Y[(int64_t)(2 * p + 1) * rows + row0 + r] = b;
      }
    }
}

// Rows i and n + i of a stacked gate | up matrix by one warp, which then has both factors of result i: half the pieces in
// flight per row, two rows at a time.
template <int DT, int MT>
__global__ void __launch_bounds__(ROW_WARPS * 32, (DT == DT_F32 || MT > 2) ? 2 : 4)
gemv_rows_glu_kernel(const uint8_t* __restrict__ W, int64_t row_bytes, int64_t cols, const float* __restrict__ X, float* __restrict__ Y, int tokens,
                     GluShape glu) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5), n_warps = (int64_t)gridDim.x * ROW_WARPS;
  constexpr int UNROLL = Unroll<DT>::N / 2;
  for (int64_t row = warp; row < glu.n; row += n_warps) {
    const uint8_t* wr[2] = {W + row * row_bytes, W + (row + glu.n) * row_bytes};
    float acc[2][MT];
#pragma unroll
    for (int t = 0; t < MT; ++t) acc[0][t] = acc[1][t] = 0.f;
    for (int64_t c0 = 8 * lane; c0 < cols; c0 += 256 * UNROLL) {
      Raw8<DT> raw[2][UNROLL];
#pragma unroll
      for (int i = 0; i < UNROLL; ++i)
        if (c0 + 256 * i < cols) { fetch8<DT>(wr[0], c0 + 256 * i, raw[0][i]); fetch8<DT>(wr[1], c0 + 256 * i, raw[1][i]); }
#pragma unroll
      for (int i = 0; i < UNROLL; ++i) {
        const int64_t c = c0 + 256 * i;
        if (c < cols) {
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            float w[8];
            widen8<DT>(raw[r][i], w);
#pragma unroll
            for (int t = 0; t < MT; ++t)
              if (t < tokens) {
                const float4* xp = (const float4*)(X + (int64_t)t * cols + c);
                const float4 a = __ldg(xp), b = __ldg(xp + 1);
                float s = acc[r][t];
                s = fmaf(w[0], a.x, s); s = fmaf(w[1], a.y, s); s = fmaf(w[2], a.z, s); s = fmaf(w[3], a.w, s);
                s = fmaf(w[4], b.x, s); s = fmaf(w[5], b.y, s); s = fmaf(w[6], b.z, s); s = fmaf(w[7], b.w, s);
                acc[r][t] = s;
              }
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      float a = acc[0][t], b = acc[1][t];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) { a += __shfl_xor_sync(~0u, a, o); b += __shfl_xor_sync(~0u, b, o); }
      if (lane == 0 && t < tokens) {
        Y[(int64_t)t * glu.n + row] = gated_unit(a, b, glu);
      }
    }
  }
}

template <int DT, int MT>
cudaError_t launch_rows_glu(const MatView& m, const float* x, float* y, int tokens, const GluShape& glu, cudaStream_t stream, int sm_count) {
  const int64_t grid = std::min<int64_t>((glu.n + ROW_WARPS - 1) / ROW_WARPS, (int64_t)sm_count * 8);
  gemv_rows_glu_kernel<DT, MT><<<(unsigned)grid, ROW_WARPS * 32, 0, stream>>>(m.w, m.row_bytes, m.cols, x, y, tokens, glu);
  return cudaGetLastError();
}
template <int DT>
cudaError_t launch_rows_glu_mt(const MatView& m, const float* x, float* y, int tokens, const GluShape& glu, cudaStream_t stream, int sm_count) {
  if (tokens == 1) return launch_rows_glu<DT, 1>(m, x, y, tokens, glu, stream, sm_count);
  if (tokens == 2) return launch_rows_glu<DT, 2>(m, x, y, tokens, glu, stream, sm_count);
  if (tokens <= 4) return launch_rows_glu<DT, 4>(m, x, y, tokens, glu, stream, sm_count);
  return launch_rows_glu<DT, 8>(m, x, y, tokens, glu, stream, sm_count);
}

template <int DT, int MT>
cudaError_t launch_rows(const MatView& m, const float* x, float* y, int tokens, cudaStream_t stream, int sm_count) {
  int64_t grid = (m.rows + ROW_WARPS - 1) / ROW_WARPS;
  const int64_t cap = (int64_t)sm_count * 8;  // two waves of the four CTAs of 256 threads an SM holds
  if (grid > cap) grid = cap;
  gemv_rows_kernel<DT, MT><<<(unsigned)grid, ROW_WARPS * 32, 0, stream>>>(m.w, m.row_bytes, m.rows, m.cols, x, y, tokens);
  return cudaGetLastError();
}

template <int DT, int T, int R, bool RUNS = false, int S = 1>
cudaError_t launch_rows_wide(const MatView& m, const float* x, float* y, int tokens, cudaStream_t stream) {
  gemv_rows_wide_kernel<DT, T, R, RUNS, S><<<(unsigned)((m.rows + ROW_WARPS * R - 1) / (ROW_WARPS * R)), ROW_WARPS * 32, 0, stream>>>(
      m.w, m.row_bytes, m.rows, m.cols, x, y, tokens);
  return cudaGetLastError();
}

// four weight rows per warp, two where they would leave SMs without a block
bool few_rows(const MatView& m, int sm_count) { return m.rows < (int64_t)sm_count * 2 * ROW_WARPS * 4; }

template <int DT>
cudaError_t launch_rows_mt(const MatView& m, const float* x, float* y, int tokens, bool runs, cudaStream_t stream, int sm_count) {
  const bool few = few_rows(m, sm_count);
  if (runs) return !few ? launch_rows_wide<DT, 8, 4, true>(m, x, y, tokens, stream)
                   : tokens <= 8 ? launch_rows_wide<DT, 8, 2, true>(m, x, y, tokens, stream) : launch_rows_wide<DT, 16, 2, true>(m, x, y, tokens, stream);
  if (tokens == 1) return launch_rows<DT, 1>(m, x, y, tokens, stream, sm_count);
  if (tokens == 2) return launch_rows<DT, 2>(m, x, y, tokens, stream, sm_count);
  // Up to four activation rows of a matrix that has at most a block per SM: a step of 256 columns is little work, and what a CTA waits
  // for is one trip to memory per tile; tiles of four steps make a quarter of the trips.  From 1024 columns on, where the first
  // tile is full (2048 x 256: 4.2 us with one step, 4.8 with four).  Three rows, weights from HBM, one / four steps a tile, and a
  // warp per weight row (the kernel above): 128 x 28672 F32 88 / 51 / 67 us, BF16 80 / 34 / 71; 1024 x 4096 F32 16.3 / 11.2 / 14.2.
  if (tokens <= 4 && m.cols >= 1024 && m.rows <= (int64_t)sm_count * 2 * ROW_WARPS) return launch_rows_wide<DT, 4, 2, false, 4>(m, x, y, tokens, stream);
  if (tokens <= 4) return few ? launch_rows_wide<DT, 4, 2>(m, x, y, tokens, stream) : launch_rows_wide<DT, 4, 4>(m, x, y, tokens, stream);
  if (tokens <= 8) return few ? launch_rows_wide<DT, 8, 2>(m, x, y, tokens, stream) : launch_rows_wide<DT, 8, 4>(m, x, y, tokens, stream);
  return few ? launch_rows_wide<DT, 16, 2>(m, x, y, tokens, stream) : launch_rows_wide<DT, 16, 4>(m, x, y, tokens, stream);
}

}  // namespace

cudaError_t launch_gemv_rows_glu(const MatView& m, const float* x, float* out, const GluShape& glu, int tokens, cudaStream_t stream, int sm_count,
                                 uint64_t* launches) {
  if (!gemv_rows_supported(m) || m.rows != 2 * (int64_t)glu.n || tokens < 1 || tokens > 8 || ((uintptr_t)x & 15) != 0) return cudaErrorInvalidValue;
  if (launches) ++*launches;
  if (m.dtype == DT_F32) return launch_rows_glu_mt<DT_F32>(m, x, out, tokens, glu, stream, sm_count);
  if (m.dtype == DT_F16) return launch_rows_glu_mt<DT_F16>(m, x, out, tokens, glu, stream, sm_count);
  return launch_rows_glu_mt<DT_BF16>(m, x, out, tokens, glu, stream, sm_count);
}

bool gemv_rows_supported(const MatView& m) {
  if (m.dtype != DT_F32 && m.dtype != DT_F16 && m.dtype != DT_BF16) return false;
  return m.rows > 0 && m.cols > 0 && m.cols % 8 == 0 && m.row_bytes % 16 == 0 && ((uintptr_t)m.w & 15) == 0;
}

cudaError_t launch_gemv_rows(const MatView& m, const float* x, float* y, int64_t tokens, cudaStream_t stream, int sm_count,
                             uint64_t* launches) {
  // A matrix of up to 256 columns is one run: the sums of the kernels without runs are the same.  Runs double the accumulators, so a
  // pass has sixteen rows only where a warp has two weight rows.  33 rows, passes of eight / these / the staged kernel: 2048 x 256
  // 30.9 / 16.5 / 28.8 us, 1024 x 4096 F32 95 / 59 / 150, 32000 x 256 F32 146 / 105 / 124.
  const bool runs = tokens > 32 && m.cols > 256;
  const int64_t pass = runs && !few_rows(m, sm_count) ? 8 : 16;
  for (int64_t t0 = 0; t0 < tokens; t0 += pass) {
    const int nt = (int)(tokens - t0 < pass ? tokens - t0 : pass);
    const float* xp = x + t0 * m.cols;
    float* yp = y + t0 * m.rows;
    cudaError_t e;
    if (m.dtype == DT_F32) e = launch_rows_mt<DT_F32>(m, xp, yp, nt, runs, stream, sm_count);
    else if (m.dtype == DT_F16) e = launch_rows_mt<DT_F16>(m, xp, yp, nt, runs, stream, sm_count);
    else e = launch_rows_mt<DT_BF16>(m, xp, yp, nt, runs, stream, sm_count);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  return cudaSuccess;
}

}  // namespace llr
