// The walk over the tokens of prompts that the mixers with a matrix state per head share (recurrent.cu, mlstm.cu).
//
// Per request and head a float32 matrix S [D, V] (key dims by value dims) lives in the state slab.
//   gated delta rule:  S <- diag(g_t) S;  u = beta_t (v_t - S^T k_t);  S <- S + k_t u^T;  o_t = S^T q_t
//                      (g_t a decay per key channel, or one number for the head)
//   state space:       S <- a_t S + k_t (w_t v_t)^T;                                      o_t = S^T q_t + skip v_t
// Columns of S are independent.  LANES neighbouring lanes hold CPT columns, lane s of them the rows 4 (s + LANES i) .. + 3
// for i < NR, in registers as pairs for the two-wide float32 instructions.  Tokens are walked one by one in float32 whatever
// the cut of the prompt; their operands are staged through shared memory TB tokens at a time by asynchronous copies in a
// ring of SCAN_STAGES stages, one barrier a stage.  A full stage is laid out flat: the next token's operands are read while
// this one's are worked on, and the outputs' sums over the lanes are made for all its tokens in one exchange.
//
// What bounds it: a prompt has one or two warps of columns a scheduler, so it is the latency of the walk, then the reads of
// the operands from shared memory (16 bytes a lane take four cycles however many lanes read the same) and the float32
// pipes, each about half busy.  3,500 tokens, 128 heads of 128 x 64 (state space): 785 us, before 1,486 with 32 rows a lane,
// four lanes a column, two stages and a sum over the lanes at every token; 32 heads of 128 x 128 (delta rule, a decay per
// channel): 812 us, before 1,568.
#pragma once
#include "common.cuh"

namespace flint_scan {

enum { STATE_SPACE = 0, DELTA_CHANNEL = 1, DELTA_HEAD = 2 };
constexpr int SCAN_STAGES = 4;
constexpr int TB = 8;            // tokens a stage

typedef unsigned long long pair_t;         // two float32 numbers
__device__ __forceinline__ pair_t pack2(float a, float b) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(pair_t p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
  pair_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ pair_t mul2(pair_t a, pair_t b) {
  pair_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t add2(pair_t a, pair_t b) {
  pair_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ void copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// q, k: rows of G key heads of D floats, v rows of H heads of V; every operand has a stride between tokens.  decay: a number
// a head (DELTA_CHANNEL: D numbers a head), w: beta or the write's weight, one a head; head_step: floats between the numbers
// of neighbouring heads of `decay` and `w`.  skip [H] or null.  seq_start [n_seq + 1]: request e brings the rows
// seq_start[e] .. seq_start[e + 1] - 1.  State of (request, head): S row-major [D, V]; or, transposed, [V, D]; then column
// V - 1 takes the value 1 at every token and its output goes to extra[t, head_step h] instead of o, whose rows (and v's) hold
// V - 1 numbers a head.
struct ScanArgs {
  const float* q; long long q_stride;
  const float* k; long long k_stride;
  const float* v; long long v_stride;
  const float* decay; long long decay_stride;
  const float* w; long long w_stride;
  int head_step;
  const float* skip;
  const int* slot;
  const int* seq_start;
  float* state; long long state_stride, head_stride;
  float* o;
  float* extra; long long extra_stride;
  int H, G, D, V;
};

template <int CPT> __device__ __forceinline__ void load_cols(const float* p, float* v) {
  if constexpr (CPT == 2) { const float2 x = *reinterpret_cast<const float2*>(p); v[0] = x.x; v[1] = x.y; }
  else v[0] = *p;
}

// The floats of one token in a stage: q, k (and the decay per channel), padded to the lanes' rows, the block's values, and
// two numbers (a multiple of 4 in all).
template <int LANES, int NR, int CPT, int RULE>
__host__ __device__ constexpr int scan_token_floats(int threads) {
  return (RULE == DELTA_CHANNEL ? 3 : 2) * LANES * 4 * NR + threads / LANES * CPT + 4;
}

// VEC: every operand row starts on a 16-byte boundary and D and the values of a head are multiples of 4, so they are staged
// 16 bytes a copy; else 4 bytes a copy.  Both leave the same numbers in the same places.  Grid: (column blocks, H, n_seq).
template <int LANES, int NR, int CPT, int RULE, bool VEC, bool TRANSPOSED>
__global__ void __launch_bounds__(256, RULE == STATE_SPACE ? 2 : 1)    // two blocks a multiprocessor: 785 us, one 934
token_scan_kernel(const ScanArgs a) {
  extern __shared__ __align__(16) float sm[];
  constexpr int DP = LANES * 4 * NR;
  constexpr bool CHANNEL = RULE == DELTA_CHANNEL;
  constexpr int NV = CHANNEL ? 3 : 2;
  const int threads = blockDim.x, cols = threads / LANES * CPT;
  const int tid = threadIdx.x, sub = tid % LANES, D = a.D, V = a.V;
  const int c0 = blockIdx.x * cols, nc = min(cols, V - c0), col = c0 + tid / LANES * CPT;
  const int h = blockIdx.y, e = blockIdx.z, kh = h / (a.H / a.G);
  const int per_tok = scan_token_floats<LANES, NR, CPT, RULE>(threads), per_stage = TB * per_tok;
  const int ones = TRANSPOSED ? NV * DP + V - 1 - c0 : -1;             // the staged value that is 1 at every token
  for (int i = tid; i < SCAN_STAGES * per_stage; i += threads) {       // dims and columns beyond the last: q = k = v = 0, decay 1
    const int w = i % per_tok;
    sm[i] = (CHANNEL && w >= 2 * DP && w < 3 * DP) || (TRANSPOSED && w == ones && w < NV * DP + cols) ? 1.f : 0.f;
  }
  const int v_live = TRANSPOSED ? min(nc, V - 1 - c0) : nc;            // values staged by copies
  __syncthreads();
  flint::pdl_wait();
  const int r0 = a.seq_start[e], r1 = a.seq_start[e + 1];
  if (r1 <= r0) return;
  float* S_g = a.state + (size_t)a.slot[r0] * a.state_stride + (size_t)h * a.head_stride;
  auto at = [&](int d, int c) -> float* { return TRANSPOSED ? S_g + (size_t)c * D + d : S_g + (size_t)d * V + c; };
  const int o_width = TRANSPOSED ? V - 1 : V;
  const float* q_h = a.q + (size_t)kh * D;
  const float* k_h = a.k + (size_t)kh * D;
  const float* g_h = CHANNEL ? a.decay + (size_t)h * D : a.decay + (size_t)h * a.head_step;
  const float* w_h = a.w + (size_t)h * a.head_step;
  const float* v_h = a.v + (size_t)h * o_width + c0;
  auto fetch = [&](int t0, int st) {
    const int n = min(TB, r1 - t0);
    float* base = sm + st * per_stage;
    if (VEC) {
      // piece j of a token: 16 bytes of q, then of k, then of the decay, then of the values
      const int d4 = D >> 2, pieces = NV * d4 + (v_live >> 2);
      for (int j = tid; j < pieces; j += threads) {
        int part = 0, x = j;                        // which vector, which piece of it
        if (x >= d4) { x -= d4; part = 1; }
        if (part == 1 && x >= d4) { x -= d4; part = 2; }
        if (CHANNEL && part == 2 && x >= d4) { x -= d4; part = 3; }
        const bool val = part == NV;
        const float* src = val ? v_h : part == 0 ? q_h : part == 1 ? k_h : g_h;
        const long long stride = val ? a.v_stride : part == 0 ? a.q_stride : part == 1 ? a.k_stride : a.decay_stride;
        src += (size_t)t0 * stride + 4 * x;
        float* dst = base + part * DP + 4 * x;
        for (int tt = 0; tt < n; ++tt, src += stride, dst += per_tok) copy16(dst, src);
      }
    } else {
      for (int i = tid; i < n * D; i += threads) {
        const int tt = i / D, d = i % D, t = t0 + tt;
        float* dst = base + (size_t)tt * per_tok + d;
        copy4(dst, q_h + (size_t)t * a.q_stride + d);
        copy4(dst + DP, k_h + (size_t)t * a.k_stride + d);
        if (CHANNEL) copy4(dst + 2 * DP, g_h + (size_t)t * a.decay_stride + d);
      }
      for (int i = tid; i < n * v_live; i += threads) {
        const int tt = i / v_live, c = i % v_live;
        copy4(base + (size_t)tt * per_tok + NV * DP + c, v_h + (size_t)(t0 + tt) * a.v_stride + c);
      }
    }
    // the last threads bring the two numbers of a token (the first ones have the most pieces)
    for (int j = threads - 1 - tid; j < 2 * n; j += threads) {
      const int tt = j >> 1;
      float* dst = base + (size_t)tt * per_tok + NV * DP + cols + (j & 1);
      if (!(j & 1)) copy4(dst, w_h + (size_t)(t0 + tt) * a.w_stride);
      else if (!CHANNEL) copy4(dst, g_h + (size_t)(t0 + tt) * a.decay_stride);
    }
  };
#pragma unroll
  for (int s = 0; s < SCAN_STAGES - 1; ++s) {
    if (r0 + s * TB < r1) fetch(r0 + s * TB, s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  pair_t S[CPT][2 * NR];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int d = 4 * (sub + LANES * i);
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      float x[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) x[r] = (col + c < V && d + r < D) ? *at(d + r, col + c) : 0.f;
      S[c][2 * i] = pack2(x[0], x[1]);
      S[c][2 * i + 1] = pack2(x[2], x[3]);
    }
  }
  const float skip_h = a.skip ? a.skip[h] : 0.f;
  struct Token { ulonglong2 k[NR], q[NR], g[CHANNEL ? NR : 1]; float v[CPT], w, decay; };
  auto read = [&](const float* tok, Token& x) {
    const ulonglong2* k2 = reinterpret_cast<const ulonglong2*>(tok + DP) + sub;
    const ulonglong2* g2 = reinterpret_cast<const ulonglong2*>(tok + 2 * DP) + sub;
    const ulonglong2* q2 = reinterpret_cast<const ulonglong2*>(tok) + sub;
#pragma unroll
    for (int i = 0; i < NR; ++i) x.k[i] = k2[LANES * i];
#pragma unroll
    for (int i = 0; i < (CHANNEL ? NR : 0); ++i) x.g[i] = g2[LANES * i];
    load_cols<CPT>(tok + NV * DP + tid / LANES * CPT, x.v);
    x.w = tok[NV * DP + cols];
    x.decay = CHANNEL ? 1.f : tok[NV * DP + cols + 1];
#pragma unroll
    for (int i = 0; i < NR; ++i) x.q[i] = q2[LANES * i];
  };
  // one token through the columns: out[c] is this lane's part of the column's output
  auto walk = [&](const Token& x, float* out) {
    const pair_t dd = pack2(x.decay, x.decay);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const ulonglong2 gg = CHANNEL ? x.g[CHANNEL ? i : 0] : make_ulonglong2(dd, dd);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        S[c][2 * i] = mul2(S[c][2 * i], gg.x);
        S[c][2 * i + 1] = mul2(S[c][2 * i + 1], gg.y);
      }
    }
    float u[CPT];
    if (RULE != STATE_SPACE) {
      float dot[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        pair_t d0 = mul2(S[c][0], x.k[0].x), d1 = mul2(S[c][1], x.k[0].y);
#pragma unroll
        for (int i = 1; i < NR; ++i) {
          d0 = fma2(S[c][2 * i], x.k[i].x, d0);
          d1 = fma2(S[c][2 * i + 1], x.k[i].y, d1);
        }
        const float2 y = unpack2(add2(d0, d1));
        dot[c] = y.x + y.y;
      }
#pragma unroll
      for (int m = LANES / 2; m >= 1; m >>= 1)
#pragma unroll
        for (int c = 0; c < CPT; ++c) dot[c] += __shfl_xor_sync(0xffffffffu, dot[c], m);
#pragma unroll
      for (int c = 0; c < CPT; ++c) u[c] = x.w * (x.v[c] - dot[c]);
    } else {
#pragma unroll
      for (int c = 0; c < CPT; ++c) u[c] = x.w * x.v[c];
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const pair_t uu = pack2(u[c], u[c]);
      pair_t o0, o1;
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        S[c][2 * i] = fma2(x.k[i].x, uu, S[c][2 * i]);
        S[c][2 * i + 1] = fma2(x.k[i].y, uu, S[c][2 * i + 1]);
        o0 = i ? fma2(S[c][2 * i], x.q[i].x, o0) : mul2(S[c][0], x.q[0].x);
        o1 = i ? fma2(S[c][2 * i + 1], x.q[i].y, o1) : mul2(S[c][1], x.q[0].y);
      }
      const float2 y = unpack2(add2(o0, o1));
      out[c] = y.x + y.y;
    }
  };
  auto place = [&](int t, int c) -> float* {           // where the output of token t in column c goes
    return TRANSPOSED && c == V - 1 ? a.extra + (size_t)t * a.extra_stride + (size_t)h * a.head_step
                                    : a.o + ((size_t)t * a.H + h) * o_width + c;
  };
  constexpr int KEEP = TB * CPT / LANES;       // of a full stage's outputs (token-major) a lane ends with these, from sub KEEP
  static_assert(KEEP >= 1, "a full stage has an output for every lane of a column");
  int st = 0;
  for (int t0 = r0; t0 < r1; t0 += TB) {
    asm volatile("cp.async.wait_group %0;" ::"n"(SCAN_STAGES - 2) : "memory");
    __syncthreads();           // this stage has arrived for everyone, and everyone has left the one refilled now
    if (t0 + (SCAN_STAGES - 1) * TB < r1) fetch(t0 + (SCAN_STAGES - 1) * TB, (st + SCAN_STAGES - 1) % SCAN_STAGES);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int n = min(TB, r1 - t0);
    const float* stage = sm + st * per_stage;
    if (n == TB) {
      float out[TB * CPT];
      Token now, next;
      read(stage, now);
#pragma unroll
      for (int tt = 0; tt < TB; ++tt) {
        if (tt + 1 < TB) read(stage + (tt + 1) * per_tok, next);
        walk(now, out + tt * CPT);
        now = next;
      }
      // every lane passes on the half of the outputs that it does not keep
#pragma unroll
      for (int m = LANES / 2, half = TB * CPT / 2; m >= 1; m >>= 1, half >>= 1) {
        const bool hi = sub & m;
#pragma unroll
        for (int i = 0; i < half; ++i)
          out[i] = (hi ? out[half + i] : out[i]) + __shfl_xor_sync(0xffffffffu, hi ? out[i] : out[half + i], m);
      }
#pragma unroll
      for (int r = 0; r < KEEP; ++r) {
        const int tt = (sub * KEEP + r) / CPT, c = (sub * KEEP + r) % CPT;
        const float v_mine = stage[tt * per_tok + NV * DP + tid / LANES * CPT + c];
        if (col + c < V) *place(t0 + tt, col + c) = fmaf(skip_h, v_mine, out[r]);
      }
    } else {
      for (int tt = 0; tt < n; ++tt) {
        float out[CPT];
        Token now;
        read(stage + tt * per_tok, now);
        walk(now, out);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
#pragma unroll
          for (int m = LANES / 2; m >= 1; m >>= 1) out[c] += __shfl_xor_sync(0xffffffffu, out[c], m);
          if (sub == 0 && col + c < V) *place(t0 + tt, col + c) = fmaf(skip_h, now.v[c], out[c]);
        }
      }
    }
    st = (st + 1) % SCAN_STAGES;
  }
  // Only now may the kernel behind this one start: its blocks would wait on the SMs beside the walk's few warps for
  // as long as the walk takes (a prompt of 2,048 tokens ran twice as long with the release at the top).
  flint::pdl_launch();
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int d = 4 * (sub + LANES * i);
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const float2 lo = unpack2(S[c][2 * i]), hi = unpack2(S[c][2 * i + 1]);
      const float x[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (col + c < V && d + r < D) *at(d + r, col + c) = x[r];
    }
  }
}

template <int LANES, int NR, int CPT, int RULE, bool VEC, bool TRANSPOSED>
inline cudaError_t launch_one(const ScanArgs& a, int n_seq, int threads, cudaStream_t stream) {
  auto kernel = token_scan_kernel<LANES, NR, CPT, RULE, VEC, TRANSPOSED>;
  const int cols = threads / LANES * CPT;
  const dim3 grid((unsigned)((a.V + cols - 1) / cols), (unsigned)a.H, (unsigned)n_seq), block((unsigned)threads);
  const size_t smem = (size_t)SCAN_STAGES * TB * scan_token_floats<LANES, NR, CPT, RULE>(threads) * sizeof(float);
  if (smem > 48 * 1024) {        // at every launch, and always the same: the limit is one of the call's device
    const cudaError_t raised = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    SCAN_STAGES * TB * scan_token_floats<LANES, NR, CPT, RULE>(256) * (int)sizeof(float));
    if (raised != cudaSuccess) return raised;
  }
  // An ordinary launch, on an empty chip, where the few blocks get an SM each: started early they land beside the blocks
  // of the kernel before, several to an SM (a prompt of 2,048 tokens then ran half a millisecond longer a layer).
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

// Sixteen lanes a column and two columns a lane for the state-space form, whose walk has no chain between tokens but the
// update: half the operand reads of eight lanes (one request of 957 tokens, 16 heads of 128 x 128: 112 us, eight lanes 164;
// 2,048 tokens of 64 heads of 128 x 64: 280 against 338).  Blocks of 256 threads stage an operand for twice the columns and
// are taken where they still are about as many as there are multiprocessors (280 us against 301).
// Eight lanes for the delta rule, whose dot product waits for the exchange between the lanes at every token, and two columns
// a lane unless that leaves multiprocessors with less than a warp a scheduler (32 heads of 128 columns, 3,500 tokens: 812 us,
// one column 1,130; 16 heads, 1,024 tokens: 277 against 213).
template <int RULE, bool TRANSPOSED>
inline cudaError_t launch_token_scan(const ScanArgs& a, int n_seq, bool vec, cudaStream_t stream) {
  const int sm_count = flint::multiprocessors();
  const long long columns = (long long)n_seq * a.H * a.V;
#define SCAN_ONE(L, NR, C)                                                              \
  return vec ? launch_one<L, NR, C, RULE, true, TRANSPOSED>(a, n_seq, threads, stream) \
             : launch_one<L, NR, C, RULE, false, TRANSPOSED>(a, n_seq, threads, stream)
  if constexpr (RULE == STATE_SPACE) {
    const int threads = columns * 5 >= 32LL * 4 * sm_count ? 256 : 128;
    if (a.D <= 64) SCAN_ONE(16, 1, 2);
    if (a.D <= 128) SCAN_ONE(16, 2, 2);
    SCAN_ONE(16, 4, 2);
  } else {
    const int threads = 128;
    const bool pairs = columns > 4LL * 4 * sm_count;
    if (a.D <= 32) SCAN_ONE(8, 1, 2);
    if (a.D <= 64) SCAN_ONE(8, 2, 2);
    if (a.D <= 128) {
      if (pairs) SCAN_ONE(8, 4, 2);
      SCAN_ONE(8, 4, 1);
    }
    SCAN_ONE(8, 8, 2);
  }
#undef SCAN_ONE
}

}  // namespace flint_scan
