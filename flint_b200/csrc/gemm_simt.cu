// General matrix products on the ordinary float32 pipes: y[m,n] = sum_k x[m,k] * W[n,k].
//
// This is the true 32-bit path (plain FFMA, no tensor cores, no reduced-precision mode)
// and the path for shapes that the tensor-core kernel refuses.  Inputs may be float32
// or bfloat16 (widened on load), the accumulator is float32.  It takes any M, N, K.
// One kernel serves four uses:
//   dense            out = x W^T (+ bias) (+ out if accumulate)
//   dense, gated     out = act(x W^T) * (x W_up^T)
//   grouped          rows are sorted by expert; a tile map names each row tile's expert
//   grouped, gated   both
// Reference counterparts: crates/thuban_kernel/wgsl/gemm.wgsl (64x128x32 tiles, ACC=1 for
// the residual add), bias.wgsl, swiglu.wgsl.
#include <stdarg.h>
#include "common.cuh"
#include "scan.cuh"

using namespace flint;

namespace {
constexpr int BM = 64, BN = 64, BK = 16, THREADS = 256;

__device__ __forceinline__ float act_fn(float g, int act) {
  if (act == 0) return g / (1.0f + expf(-g));                       // silu
  return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g)));
}

template <typename TX, typename TW, typename TO, bool GATED>
__global__ void __launch_bounds__(THREADS)
gemm_simt_kernel(const TX* __restrict__ x, int ldx, const TW* __restrict__ w, const float* __restrict__ bias,
                 TO* __restrict__ out, int ldo, int accumulate, int act,
                 const int* __restrict__ tile_expert, const int* __restrict__ tile_row0,
                 const int* __restrict__ n_tiles, const int* __restrict__ offsets, int tile_rows,
                 long long expert_stride, int M, int N, int K, float act_slope, float act_limit) {
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  __shared__ float us[GATED ? BK : 1][BN + 4];

  int expert = 0, row0 = blockIdx.y * BM, row_end = M;
  if (tile_expert) {
    if ((int)blockIdx.y >= *n_tiles) return;
    expert = tile_expert[blockIdx.y];
    row0 = tile_row0[blockIdx.y];
    row_end = min(offsets[expert + 1], row0 + tile_rows);
  }
  const int col0 = blockIdx.x * BN;
  const TW* we = w + (size_t)expert * expert_stride;

  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 16 x 16 threads, 4 x 4 outputs each
  float acc[4][4] = {}, acc_u[GATED ? 4 : 1][4] = {};

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64 rows x 16 k = 1024 elements per operand, 4 per thread; k runs fastest in memory
    for (int i = threadIdx.x; i < BM * BK; i += THREADS) {
      const int r = i / BK, k = i % BK;
      const int gr = row0 + r, gk = k0 + k;
      xs[k][r] = (gr < row_end && gk < K) ? to_f32(x[(size_t)gr * ldx + gk]) : 0.f;
      const int gc = col0 + r;
      const bool ok = gc < N && gk < K;
      const size_t wr = GATED ? paired_gate_row(gc) : gc;      // gated: the up row lies GATE_BLOCK rows further
      ws[k][r] = ok ? to_f32(we[wr * K + gk]) : 0.f;
      if (GATED) us[k][r] = ok ? to_f32(we[(wr + GATE_BLOCK) * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], b[4], u[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[k][tx * 4 + j];
      if (GATED) {
#pragma unroll
        for (int j = 0; j < 4; ++j) u[j] = us[k][tx * 4 + j];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
          if (GATED) acc_u[i][j] = fmaf(a[i], u[j], acc_u[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gr = row0 + ty * 4 + i;
    if (gr >= row_end) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gc = col0 + tx * 4 + j;
      if (gc >= N) continue;
      float v = acc[i][j];
      if (GATED) {          // a gated product's bias is paired like its weight rows and comes before the activation
        float up = acc_u[i][j];
        if (bias) {
          v += bias[paired_gate_row(gc)];
          up += bias[paired_gate_row(gc) + GATE_BLOCK];
        }
        if (act == 2) {     // clamped: gate sigmoid(slope gate) (up + 1)
          v = fminf(v, act_limit);
          up = fminf(fmaxf(up, -act_limit), act_limit);
          v = v / (1.0f + expf(-act_slope * v)) * (up + 1.0f);
        } else {
          v = act_fn(v, act) * up;
        }
      } else if (bias) {
        v += bias[gc];
      }
      const size_t o = (size_t)gr * ldo + gc;
      if (accumulate) v += to_f32(out[o]);
      out[o] = from_f32<TO>(v);
    }
  }
}

// Dense products of many rows and columns in tiles of 128 x 128, 8 x 8 outputs a thread as pairs for the two-wide float32
// instructions, operands read 16 bytes (bfloat16: 8) a load into registers while the tile before is worked on.  What bounds it
// is the float32 pipe: 3,500 rows, N 4,096, K 128 is 3.7 GFLOP, 50 us at its peak; the 64 x 64 tiles above, with scalar
// loads and 16 outputs a thread, took 337 us.  Every output's products are added in the same order (k ascending), so both
// give the same bits.
constexpr int WM = 128, WN = 128, WK = 16;

__device__ __forceinline__ float4 load_four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_four(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                     __uint_as_float(v.y & 0xffff0000u));
}

template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(THREADS, 2)
gemm_simt_wide_kernel(const TX* __restrict__ x, int ldx, const TW* __restrict__ w, const float* __restrict__ bias,
                      TO* __restrict__ out, int ldo, int accumulate, int M, int N, int K) {
  using namespace flint_scan;
  __shared__ __align__(16) float xs[2][WK][WM + 4];
  __shared__ __align__(16) float ws[2][WK][WN + 4];
  const int row0 = blockIdx.y * WM, col0 = blockIdx.x * WN;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;     // rows 4 ty + 0..3 and 64 + 4 ty + 0..3, columns alike
  // loads: 128 rows of four pieces of four; thread i takes pieces i and i + 256
  const int lr = threadIdx.x >> 2, lk = (threadIdx.x & 3) * 4;
  float4 px[2], pw[2];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = row0 + lr + 64 * i, c = col0 + lr + 64 * i, k = k0 + lk;      // K is a multiple of 4
      px[i] = r < M && k < K ? load_four(x + (size_t)r * ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      pw[i] = c < N && k < K ? load_four(w + (size_t)c * K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto stage = [&](int b) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = lr + 64 * i;
      xs[b][lk][r] = px[i].x; xs[b][lk + 1][r] = px[i].y; xs[b][lk + 2][r] = px[i].z; xs[b][lk + 3][r] = px[i].w;
      ws[b][lk][r] = pw[i].x; ws[b][lk + 1][r] = pw[i].y; ws[b][lk + 2][r] = pw[i].z; ws[b][lk + 3][r] = pw[i].w;
    }
  };
  pair_t acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  fetch(0);
  stage(0);
  __syncthreads();
  int b = 0;
  for (int k0 = 0; k0 < K; k0 += WK, b ^= 1) {
    const bool more = k0 + WK < K;
    if (more) fetch(k0 + WK);
#pragma unroll
    for (int k = 0; k < WK; ++k) {
      const float4 a0 = *reinterpret_cast<const float4*>(&xs[b][k][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&xs[b][k][64 + ty * 4]);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&ws[b][k][tx * 4]);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&ws[b][k][64 + tx * 4]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const pair_t aa = pack2(av[i], av[i]);
        acc[i][0] = fma2(aa, b0.x, acc[i][0]);
        acc[i][1] = fma2(aa, b0.y, acc[i][1]);
        acc[i][2] = fma2(aa, b1.x, acc[i][2]);
        acc[i][3] = fma2(aa, b1.y, acc[i][3]);
      }
    }
    if (more) stage(b ^ 1);       // read last before the barrier of the round before
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = row0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 y = unpack2(acc[i][j]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = col0 + (j < 2 ? tx * 4 + 2 * j : 64 + tx * 4 + 2 * (j - 2)) + h;
        if (c >= N) continue;
        float v = h ? y.y : y.x;
        if (bias) v += bias[c];
        const size_t o = (size_t)r * ldo + c;
        if (accumulate) v += to_f32(out[o]);
        out[o] = from_f32<TO>(v);
      }
    }
  }
}
}  // namespace

// x [rows, K] (row stride ldx), w [E, N, K] (gated: [E, paired_rows(N), K], gate and up rows paired in blocks),
// out [rows, N].
// Dense: tile_expert == NULL, rows = M, one "expert".  Grouped: rows of expert e are
// offsets[e] .. offsets[e+1]-1, and tile i covers up to tile_rows (<= 64) rows from tile_row0[i] of
// expert tile_expert[i]; only the first *n_tiles tiles exist (max_tiles bounds the grid).
// A gated product's bias has paired_rows(N) entries and is added before the activation; act 2 is the clamped form with
// act_slope and act_limit.
extern "C" int flint_gemm_simt(const void* x, int x_dtype, int ldx, const void* w, int gated,
                               int w_dtype, const float* bias, void* out, int out_dtype, int ldo,
                               int accumulate, int act, const int* tile_expert,
                               const int* tile_row0, const int* n_tiles, const int* offsets,
                               int max_tiles, int tile_rows, int M, int N, int K, float act_slope, float act_limit,
                               cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return fail("gemm_simt: K=%d", K);
  const long long expert_stride = (long long)(gated ? paired_rows(N) : N) * K;
  if (gated && accumulate) return fail("gemm_simt: a gated product cannot accumulate");
  if (tile_expert && (tile_rows < 1 || tile_rows > BM)) return fail("gemm_simt: row tiles of %d rows (1..%d)", tile_rows, BM);
  const int tiles_m = tile_expert ? max_tiles : (M + BM - 1) / BM;
  if (tiles_m <= 0) return 0;
  if (tiles_m > 65535) return fail("gemm_simt: %d row tiles exceed the grid limit", tiles_m);
  // large tiles where they are at least as many as the multiprocessors (below that the smaller ones spread further), on rows
  // that can be read in whole pieces of four
  const int x_size = x_dtype == FLINT_F32 ? 4 : 2, w_size = w_dtype == FLINT_F32 ? 4 : 2;
  const long long large = (long long)((M + WM - 1) / WM) * ((N + WN - 1) / WN);
  if (!tile_expert && !gated && large >= multiprocessors() && K % 4 == 0 && ldx % 4 == 0 && (uintptr_t)x % (4 * x_size) == 0 &&
      (uintptr_t)w % (4 * w_size) == 0) {
    const dim3 wide((N + WN - 1) / WN, (M + WM - 1) / WM);
    FLINT_DISPATCH_DTYPE(x_dtype, TX, FLINT_DISPATCH_DTYPE(w_dtype, TW, FLINT_DISPATCH_DTYPE(out_dtype, TO,
        (gemm_simt_wide_kernel<TX, TW, TO><<<wide, THREADS, 0, stream>>>((const TX*)x, ldx, (const TW*)w, bias, (TO*)out, ldo,
                                                                         accumulate, M, N, K)))));
    return check_launch("gemm_simt");
  }
  dim3 grid((N + BN - 1) / BN, tiles_m);
#define LAUNCH(TX, TW, TO)                                                                        \
  do {                                                                                            \
    if (gated)                                                                                    \
      gemm_simt_kernel<TX, TW, TO, true><<<grid, THREADS, 0, stream>>>(                           \
          (const TX*)x, ldx, (const TW*)w, bias, (TO*)out, ldo, accumulate, act,                  \
          tile_expert, tile_row0, n_tiles, offsets, tile_rows, expert_stride, M, N, K, act_slope, act_limit);                                     \
    else                                                                                          \
      gemm_simt_kernel<TX, TW, TO, false><<<grid, THREADS, 0, stream>>>(                          \
          (const TX*)x, ldx, (const TW*)w, bias, (TO*)out, ldo, accumulate, act,                  \
          tile_expert, tile_row0, n_tiles, offsets, tile_rows, expert_stride, M, N, K, act_slope, act_limit);                                     \
  } while (0)
  FLINT_DISPATCH_DTYPE(x_dtype, TX, FLINT_DISPATCH_DTYPE(w_dtype, TW,
      FLINT_DISPATCH_DTYPE(out_dtype, TO, LAUNCH(TX, TW, TO))));
#undef LAUNCH
  return check_launch("gemm_simt");
}

extern "C" const char* flint_gemm_simt_last_error() { return g_error; }
