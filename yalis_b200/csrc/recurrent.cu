// Mixers that keep a matrix per head instead of keys and values: linear recurrences
// over a float32 state S [dim, vdim] per (request, head),
//
//   S <- diag(g_t) S                      g_t: a constant per head, a scalar per token, or a vector over dim
//   u  = beta_t (v_t - S^T k_t)           (delta rule)        or   u = v_t   (plain outer-product write)
//   S <- S + k_t u^T
//   o_t = S^T q_t                         (the read-out sees the token's own write)
//
// the selective form, with a step size in front of the write and the token's own value beside the read-out,
//
//   S <- g_t S + k_t (beta_t v_t)^T,   o_t = S^T q_t + D v_t
//
// and the generalized delta rule, whose decay and removal both read the OLD state,
//
//   S <- diag(g_t) S - (a_t * u_t)(u_t^T S) + k_t v_t^T,   o_t = S^T q_t
//
// with a unit key u_t and a removal rate a_t per head and key channel,
//
// with the short causal convolution that feeds some of them and the per-head norm and gate
// that follow them.  Everything here is float32 arithmetic whatever the model's dtype; the
// state and the convolution's tail live in the per-request slot memory of the cache manager.
//
// The columns of S are independent of one another (column j only ever meets v_j), so a thread
// owns 8 or 16 rows of one or two columns in registers, the lanes that share a column sit in one warp, and
// a block walks the tokens of one request in order: a portion of a prompt and a single
// decoded token are the same loop, and the result for a token does not depend on how the
// request was cut into steps or on what else is in the batch.  (Long portions of bfloat16 models may go
// by chunks instead: recurrent_chunks.cu.)
#include "common.cuh"

namespace {

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// ---- what the delta rule reads: convolution, unit length, decay and write strength ------------------
//   y_t[c] = silu(sum_j w[c][K-1-j] x_(t-j)[c]),  x before the request's start = 0
// The last K-1 inputs of every request are kept in its slot: tail[c][0..K-2], oldest first.
// With kv_heads > 0 the first 2 * kv_heads * dim channels are the heads of q and then of k: each head is
// brought to unit length, x / sqrt(sum x^2 + eps), and q multiplied by q_scale.  With a_raw the decay
// g = exp(-exp(a_log[h]) * softplus(a_raw + dt_bias)) (per head, or per head and key channel) and the write
// strength are computed beside it, in float32: beta = sigmoid(b_raw), or without b_raw (one column of a_raw per
// head) the step size itself, beta = softplus(a_raw + dt_bias).  With conv_bias y_t[c] = silu(conv_bias[c] + ...).
// A block takes a tile of consecutive tokens and a piece of the channels; a thread walks the tile with the last K-1
// inputs of its channels in registers.  In steps of single tokens it also writes the new tail (`single`); otherwise
// short_conv_tail_kernel does, once every block has read the old one.
constexpr int kMaxTaps = 16;

struct DeltaPrepareParams {
  const void* x; int x_stride;
  const float* w; const float* conv_bias;
  float* tail; size_t slot_stride;
  const int32_t* req_of_token; const int32_t* q_start; const int32_t* slots;
  float* out; int out_stride;
  int n_tokens, channels, taps, tile, piece, single;
  int kv_heads, dim; float q_scale, unit_eps;
  const void* a_raw; int a_stride, a_cols; const float* a_log; const float* dt_bias;
  const void* b_raw; int b_stride, heads;
  float* g_out; float* beta_out;
};

// V neighbouring inputs as float32 (V = 2: one 4- or 8-byte load).
template <typename T, int V>
__device__ __forceinline__ void load_inputs(const T* p, float (&o)[V]) {
  if constexpr (V == 2) {
    if constexpr (sizeof(T) == 2) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
      o[0] = f.x; o[1] = f.y;
    } else {
      const float2 f = *reinterpret_cast<const float2*>(p);
      o[0] = f.x; o[1] = f.y;
    }
  } else {
    o[0] = to_f32<T>(p[0]);
  }
}

// Decays and write strengths of the tokens n0 .. n1 - 1, shared out among the blocks of a tile.
template <typename T>
__device__ __forceinline__ void rates_and_strengths(const DeltaPrepareParams& p, int n0, int n1) {
  if (p.a_raw != nullptr) {
    const T* a_raw = reinterpret_cast<const T*>(p.a_raw);
    const T* b_raw = reinterpret_cast<const T*>(p.b_raw);
    const int per = p.a_cols / p.heads;           // 1, or dim
    const int first = blockIdx.y * blockDim.x + threadIdx.x, step = gridDim.y * blockDim.x;
    for (int e = first; e < (n1 - n0) * p.a_cols; e += step) {
      const int n = n0 + e / p.a_cols, c = e % p.a_cols;
      if (p.req_of_token[n] < 0) continue;
      const float s = softplus_f(to_f32<T>(a_raw[(size_t)n * p.a_stride + c]) + p.dt_bias[c]);
      p.g_out[(size_t)n * p.a_cols + c] = expf(-expf(p.a_log[c / per]) * s);
      if (b_raw == nullptr) p.beta_out[(size_t)n * p.heads + c] = s;
    }
    for (int e = first; b_raw != nullptr && e < (n1 - n0) * p.heads; e += step) {
      const int n = n0 + e / p.heads, h = e % p.heads;
      if (p.req_of_token[n] >= 0) p.beta_out[(size_t)n * p.heads + h] = sigmoid_f(to_f32<T>(b_raw[(size_t)n * p.b_stride + h]));
    }
  }
}

// KMAX: the most taps (a bound known at compile time keeps the history in registers); V: channels a thread takes.
template <typename T, int KMAX, int V>
__global__ void delta_prepare_kernel(const DeltaPrepareParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int n0 = blockIdx.x * p.tile, n1 = min(n0 + p.tile, p.n_tokens);
  const int c_begin = blockIdx.y * p.piece, c_end = min(c_begin + p.piece, p.channels);
  const int keep = p.taps - 1;
  for (int c = c_begin + (int)threadIdx.x * V; c < c_end; c += (int)blockDim.x * V) {
    float w[KMAX][V], bias[V], hist[KMAX][V];      // place m: the input KMAX - 1 - m tokens back (the last place is unused in hist)
#pragma unroll
    for (int v = 0; v < V; ++v) {
      bias[v] = p.conv_bias ? p.conv_bias[c + v] : 0.f;
#pragma unroll
      for (int m = 0; m < KMAX; ++m) {
        const int lag = KMAX - 1 - m;
        w[m][v] = lag < p.taps ? p.w[(size_t)(c + v) * p.taps + (p.taps - 1 - lag)] : 0.f;
        hist[m][v] = 0.f;
      }
    }
    bool follows = false;                          // hist holds the inputs before token n
    for (int n = n0; n < n1; ++n) {
      const int req = p.req_of_token[n];
      if (req < 0) {
        follows = false;
        continue;
      }
      const int i = n - p.q_start[req];            // index of the token in its request's portion
      const T* xr = reinterpret_cast<const T*>(p.x) + (size_t)n * p.x_stride + c;
      float* tl = p.tail + (size_t)p.slots[req] * p.slot_stride + (size_t)c * keep;
      if (!follows || i == 0) {
#pragma unroll
        for (int m = 0; m < KMAX - 1; ++m) {
          const int lag = KMAX - 1 - m;
          if (lag <= keep) {
            if (i >= lag) {
              load_inputs<T, V>(xr - (size_t)lag * p.x_stride, hist[m]);
            } else {
#pragma unroll
              for (int v = 0; v < V; ++v) hist[m][v] = tl[(size_t)v * keep + (keep + i - lag)];
            }
          }
        }
      }
      load_inputs<T, V>(xr, hist[KMAX - 1]);
      float y[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        float acc = 0.f;
#pragma unroll
        for (int m = 0; m < KMAX; ++m) acc = __fmaf_rn(w[m][v], hist[m][v], acc);     // oldest input first: a fixed order
        y[v] = silu_exact(acc + bias[v]);
      }
      float* o = p.out + (size_t)n * p.out_stride + c;
      if constexpr (V == 2) *reinterpret_cast<float2*>(o) = make_float2(y[0], y[1]);
      else o[0] = y[0];
#pragma unroll
      for (int m = 0; m < KMAX - 1; ++m)
#pragma unroll
        for (int v = 0; v < V; ++v) hist[m][v] = hist[m + 1][v];
      follows = true;
      if (p.single) {
#pragma unroll
        for (int m = 0; m < KMAX - 1; ++m) {
          const int lag = KMAX - 1 - m;            // after the shift: the input lag - 1 tokens back
          if (lag <= keep)
#pragma unroll
            for (int v = 0; v < V; ++v) tl[(size_t)v * keep + (keep - lag)] = hist[m][v];
        }
      }
    }
  }
  rates_and_strengths<T>(p, n0, n1);
  if (p.kv_heads > 0) {
    __syncthreads();                              // the block reads back what it wrote itself
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    // the heads of q, then of k, that lie in this piece (a piece is a multiple of dim channels)
    const int h0 = c_begin / p.dim, h1 = min(c_end, 2 * p.kv_heads * p.dim) / p.dim;
    for (int e = threadIdx.x >> 5; e < (n1 - n0) * max(h1 - h0, 0); e += nw) {
      const int n = n0 + e / (h1 - h0), hh = h0 + e % (h1 - h0);
      if (p.req_of_token[n] < 0) continue;
      float* v = p.out + (size_t)n * p.out_stride + (size_t)hh * p.dim;
      float ss = 0.f;
      for (int d = lane; d < p.dim; d += 32) ss = __fmaf_rn(v[d], v[d], ss);
      ss = warp_sum(ss);
      const float r = (hh < p.kv_heads ? p.q_scale : 1.0f) / sqrtf(ss + p.unit_eps);
      for (int d = lane; d < p.dim; d += 32) v[d] *= r;
    }
  }
}

// The same over portions, for up to four taps and pieces of 128 channels (where heads are brought to unit length, a head each): a warp
// has a piece of two tokens, all of whose inputs it asks for before it needs the first, and holds a head's results until its
// length is known.  Sums in the order of the form above: the same bits.
// What bounds it: expf and the division of silu, some 30 instructions a value, and a block's wait for its rows.  The form above
// waits for a token's index, slot and row before it asks for the next one's, and reads its results back for their length.
// Measured (us with the tails' kernel, L2 flushed, above -> here): 4,096 channels, 16 heads to unit length, a rate per head: 64 tokens
// 13.3 -> 13.3, 256 17.4 -> 15.4, 512 23.6 -> 17.4, 1,024 31.7 -> 23.6, 2,048 46 -> 38; 6,144, 32 heads, a rate per channel: 128 tokens
// 19.5 -> 17.4, 2,048 89 -> 77; 2,304, none: 128 tokens 13.3 -> 15.3, 256 13.3 -> 13.3, 512 17.4 -> 15.4, 3,000 38 -> 36.
// Few values leave it with too few warps in flight, and portions of a few tokens wait for their slots' inputs at every tile (replayed, without a
// flush: 512 channels with two heads, 512 tokens 7.2 -> 7.7, 128 channels 5.0 -> 5.8; 2,304 channels, 256 tokens 6.4 -> 6.8, 512 tokens 9.5 -> 7.6, but of
// 128 requests 11.3 -> 13.0; 4,096 channels, 256 tokens 10.3 -> 8.1): so from 256 tokens and 2^20 values on, eight tokens a request on average.
// Four tokens a warp 38, 83 and 38 for the longest, eight 46, 112 and 46: fewer warps.
constexpr int kConvTile = 2, kConvTileFrom = 256;

template <typename T>
__global__ void __launch_bounds__(256) conv_tile_kernel(const DeltaPrepareParams p) {
  constexpr int LAGS = 3, NJ = 4, TILE = kConvTile;
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, piece = blockIdx.y * 8 + (threadIdx.x >> 5);
  const int n0 = blockIdx.x * TILE, n1 = min(n0 + TILE, p.n_tokens), keep = p.taps - 1;
  if (piece * 128 < p.channels) {
    float x[NJ][TILE + LAGS], w[NJ][LAGS + 1], bias[NJ], y[NJ][TILE];
    const bool quads = p.taps == 4 && ((uintptr_t)p.w & 15) == 0;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = piece * 128 + j * 32 + lane;
      const T* xc = reinterpret_cast<const T*>(p.x) + c;
#pragma unroll
      for (int m = 0; m < TILE + LAGS; ++m) {
        const int n = n0 - LAGS + m;
        x[j][m] = n >= 0 && n < n1 ? to_f32<T>(xc[(size_t)n * p.x_stride]) : 0.f;
      }
      if (quads) {
        const float4 v = load4_f32(p.w + (size_t)c * 4);
        w[j][0] = v.x; w[j][1] = v.y; w[j][2] = v.z; w[j][3] = v.w;
      } else {
#pragma unroll
        for (int lag = 0; lag <= LAGS; ++lag) w[j][LAGS - lag] = lag <= keep ? p.w[(size_t)c * p.taps + keep - lag] : 0.f;
      }
      bias[j] = p.conv_bias ? p.conv_bias[c] : 0.f;
    }
    int index = -1, slot = 0;                       // lane t: of token n0 + t within its request's portion
    if (n0 + lane < n1 && lane < TILE) {
      const int req = p.req_of_token[n0 + lane];
      if (req >= 0) {
        index = n0 + lane - p.q_start[req];
        slot = p.slots[req];
      }
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = piece * 128 + j * 32 + lane;
#pragma unroll
      for (int t = 0; t < TILE; ++t) {
        const int i = __shfl_sync(0xffffffffu, index, t), at = __shfl_sync(0xffffffffu, slot, t);
        float h[LAGS + 1];
#pragma unroll
        for (int m = 0; m <= LAGS; ++m) h[m] = x[j][t + m];
        if (i >= 0 && i < keep) {                   // the portion begins here: what is before it waits in the slot
#pragma unroll
          for (int lag = 1; lag <= LAGS; ++lag)
            if (lag > i && lag <= keep) h[LAGS - lag] = p.tail[(size_t)at * p.slot_stride + (size_t)c * keep + (keep + i - lag)];
        }
        float acc = 0.f;
#pragma unroll
        for (int m = 0; m <= LAGS; ++m)
          if (LAGS - m <= keep) acc = __fmaf_rn(w[j][m], h[m], acc);     // oldest input first
        y[j][t] = silu_exact(acc + bias[j]);
      }
    }
    const bool unit = piece < 2 * p.kv_heads;
#pragma unroll
    for (int t = 0; t < TILE; ++t) {
      if (unit) {
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < NJ; ++j) ss = __fmaf_rn(y[j][t], y[j][t], ss);
        ss = warp_sum(ss);
        const float r = (piece < p.kv_heads ? p.q_scale : 1.0f) / sqrtf(ss + p.unit_eps);
#pragma unroll
        for (int j = 0; j < NJ; ++j) y[j][t] *= r;
      }
      if (__shfl_sync(0xffffffffu, index, t) >= 0) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) p.out[(size_t)(n0 + t) * p.out_stride + piece * 128 + j * 32 + lane] = y[j][t];
      }
    }
  }
  rates_and_strengths<T>(p, n0, n1);
}

// After the step: the tail becomes the last K-1 inputs the request has seen.
template <typename T>
__global__ void short_conv_tail_kernel(const T* x, int x_stride, float* tail,
                                       size_t slot_stride, const int32_t* q_start,
                                       const int32_t* slots, int channels, int taps) {
  // The recurrence that follows holds few blocks that run long: let in while delta_prepare still fills most SMs they
  // would crowd onto the ones that come free first.
  pdl_wait();
  pdl_launch_dependents();
  const int req = blockIdx.x;
  const int a = q_start[req], q_len = q_start[req + 1] - a;
  if (q_len <= 0) return;
  float* tl = tail + (size_t)slots[req] * slot_stride;
  const int keep = taps - 1;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < channels; c += gridDim.y * blockDim.x) {
    float nv[kMaxTaps];
#pragma unroll
    for (int m = 0; m < kMaxTaps; ++m) {
      if (m < keep) {
        const int i = q_len - keep + m;           // index in the portion of the input that lands at place m
        nv[m] = i >= 0 ? to_f32<T>(x[(size_t)(a + i) * x_stride + c]) : tl[(size_t)c * keep + (m + q_len)];
      }
    }
#pragma unroll
    for (int m = 0; m < kMaxTaps; ++m)
      if (m < keep) tl[(size_t)c * keep + m] = nv[m];
  }
}

// ---- the recurrence ------------------------------------------------------------------------------
constexpr int kScanThreads = 128;

struct ScanParams {
  const float* q; int q_stride;      // [N, kv_heads * dim]
  const float* k; int k_stride;
  const float* v; int v_stride;      // [N, heads * vdim]
  const float* decay;                // DECAY 0: [heads]; 1: [N, heads]; 2: [N, heads * dim]
  const float* beta;                 // RULE 1, 3: [N, heads]
  const float* skip;                 // RULE 3: [heads] or null: skip_h v_t is added to the read-out
  const float* unit;                 // RULE 2: unit keys u [N, heads * dim]
  const float* removal;              // RULE 2: a * u [N, heads * dim]
  float* state; size_t slot_stride;  // per slot: [heads][vdim][dim_padded]
  float* out; int out_stride;        // [N, heads * vdim]
  const int32_t* q_start; const int32_t* slots;
  int heads, kv_heads, dim, dim_padded, vdim;
  int wide;                          // 1: rows of q, k and the decay may be copied 16 bytes at a time
  int limit, upto;                   // limit > 0: portions of limit to upto tokens are left to the form by chunks
};

__device__ __forceinline__ void copy_async4(float* smem, const float* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void copy_async16(float* smem, const float* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Two float32 operations in one instruction, each half rounded as the single operation is.
__device__ __forceinline__ uint64_t bits2(float2 v) { return *reinterpret_cast<uint64_t*>(&v); }
__device__ __forceinline__ float2 pair2(uint64_t v) { return *reinterpret_cast<float2*>(&v); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
  return pair2(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)));
  return pair2(d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)));
  return pair2(d);
}
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// Floats of one staging buffer (see the kernel), a multiple of four.
constexpr int scan_buffer_floats(int vec_cols, int tile, int width, int cols) {
  return (vec_cols * tile * width + tile * cols + 2 * tile + 3) & ~3;
}

// What a lane needs of one token, in registers.
template <int ROWS, int COLS, int RULE, int DECAY>
struct ScanToken {
  float4 q[ROWS / 4], k[ROWS / 4];
  float4 g[DECAY == 2 ? ROWS / 4 : 1];                                 // decay vector
  float4 u[RULE == 2 ? ROWS / 4 : 1], a[RULE == 2 ? ROWS / 4 : 1];     // unit key, removal vector
  float v[COLS], beta, decay;
};

// A lane's share of the dot product of a column of the state with a vector: four partial sums, a fixed tree.
template <int Q>
__device__ __forceinline__ float share_dot(const float2 (&S)[2 * Q], const float4 (&x)[Q]) {
  float2 a = mul2(S[0], lo2(x[0])), b = mul2(S[1], hi2(x[0]));
#pragma unroll
  for (int i = 1; i < Q; ++i) {
    a = fma2(S[2 * i], lo2(x[i]), a);
    b = fma2(S[2 * i + 1], hi2(x[i]), b);
  }
  a = add2(a, b);
  return a.x + a.y;
}

// The dot products of a thread's columns: a butterfly over the L lanes (the same order of additions for every token).
template <int Q, int L, int C>
__device__ __forceinline__ void lane_dots(const float2 (&S)[C][2 * Q], const float4 (&x)[Q], float (&dot)[C]) {
#pragma unroll
  for (int cc = 0; cc < C; ++cc) dot[cc] = share_dot<Q>(S[cc], x);
#pragma unroll
  for (int o = 1; o < L; o <<= 1)
#pragma unroll
    for (int cc = 0; cc < C; ++cc) dot[cc] += __shfl_xor_sync(0xffffffffu, dot[cc], o);
}

// Sums over the L lanes of a column of N values a lane holds (one per token and column): halves are exchanged while there
// are several, so N values cost about N shuffles and not N log L.  Afterwards lane l holds the sums of values l N / L ...
// (N >= L), or of value l / (L / N).  Every sum adds the lanes in the same tree, which is also that of one value alone.
template <int N, int L>
__device__ __forceinline__ void lane_sums(float (&r)[N], int l) {
  int n = N;
#pragma unroll
  for (int o = L / 2; o >= 1; o >>= 1) {
    if (n > 1) {
      const bool upper = (l & o) != 0;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        if (i < n / 2) {
          const float send = upper ? r[i] : r[i + n / 2], keep = upper ? r[i + n / 2] : r[i];
          r[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      n >>= 1;
    } else {
      r[0] += __shfl_xor_sync(0xffffffffu, r[0], o);
    }
  }
}

// RULE: 0 plain outer-product write, 1 delta rule, 2 generalized delta rule (needs DECAY 2), 3 plain write of beta v
// with skip_h v beside the read-out.
// DECAY: 0 constant per head, 1 scalar per token and head, 2 vector per token, head and key channel.
// ROWS x COLS: rows and neighbouring columns of the state that a thread keeps.  LANES: lanes that share a column (a power
// of two; ROWS * LANES >= dim).  TILE: tokens staged in shared memory at a time, through two buffers: while one tile is
// walked, the asynchronous copies of the next are in flight.  TILE 1 is the form for single tokens: small blocks, many of
// them per SM.
//
// What bounds a prompt is one warp's stream of instructions (a single request has only heads * vdim * dim / (32 * 16) warps,
// under one per scheduler; a warp issues an instruction every two to three cycles) and, for several requests, the loads from
// shared memory (16 bytes a lane are four passes whatever lanes share).  Hence tokens in groups of four without a run-time
// address or a move between them, a token's vectors loaded while the one before is computed, two float32 operations per
// instruction, and read-outs summed over the lanes four tokens at a time instead of one by one through shared memory.
// Measured for 16 heads of 128 x 128, us for 1 x 2,048 / 4 x 2,048 tokens (8 x 1 rows by columns a thread, a token at a time,
// before): delta rule 473 / 1156 -> 380 / 800, decay per channel 516 -> 430, generalized rule 582 -> 449, plain write
// 300 -> 250, selective 328 / 860 -> 260 / 518; 64 single tokens 37 to 41 -> 29 (134 MB: 4.6 TB/s).
// Why this split: the delta rules' chain (dot product over the lanes, write, next token) is shortest with 16 rows and 8
// lanes (two columns of 8 rows: 488 us); the others read each q and k once for two columns of 8 rows (16 rows: 262 us, and
// 717 for four selective prompts).
template <int ROWS, int LANES, int COLS, int RULE, int DECAY, int TILE>
__global__ void __launch_bounds__(kScanThreads) state_scan_kernel(const ScanParams p) {
  extern __shared__ __align__(16) float sm[];
  constexpr int Q = ROWS / 4;          // 16-byte pieces of a column per thread
  constexpr int L = LANES, C = COLS, cols = kScanThreads / L * C, width = ROWS * L;
  // one buffer: q [TILE][width], k [TILE][width], decay vectors [TILE][width] (DECAY 2), unit keys and removal vectors
  // [TILE][width] each (RULE 2), v [TILE][cols], beta [TILE], decay [TILE]; behind the two buffers the read-outs [TILE][cols]
  constexpr int vec_cols = RULE == 2 ? 5 : (DECAY == 2 ? 3 : 2);
  constexpr int array = TILE * width, buf_floats = scan_buffer_floats(vec_cols, TILE, width, cols);
  pdl_launch_dependents();
  pdl_wait();
  const int req = blockIdx.z, h = blockIdx.y;
  const int t_begin = p.q_start[req], q_len = p.q_start[req + 1] - t_begin;
  if (q_len <= 0 || (p.limit > 0 && q_len >= p.limit && q_len <= p.upto)) return;
  const int tid = threadIdx.x, l = tid % L, c = tid / L;
  const int j = blockIdx.x * cols + c * C;               // the thread's first column
  const int kvh = h / (p.heads / p.kv_heads);
  const int D = p.dim, Dp = p.dim_padded, V = p.vdim;
  float* sp = p.state + (size_t)p.slots[req] * p.slot_stride + ((size_t)h * V + j) * Dp;
  float2 S[C][ROWS / 2];
#pragma unroll
  for (int cc = 0; cc < C; ++cc)
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int d = (i * L + l) * 4;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j + cc < V && d < Dp) x = *reinterpret_cast<const float4*>(sp + (size_t)cc * Dp + d);
      S[cc][2 * i] = lo2(x); S[cc][2 * i + 1] = hi2(x);
    }
  float* outs = sm + 2 * buf_floats;

  // what no copy ever writes: the rows past dim (zeros; ones for the decay)
  const int pad = width - D;
  for (int e = tid; e < 2 * vec_cols * TILE * pad; e += kScanThreads) {
    const int row = e / pad, d = D + (e - row * pad);          // row: (buffer, array, token)
    const int b = row / (vec_cols * TILE), r = row - b * (vec_cols * TILE);
    sm[b * buf_floats + r * width + d] = (r / TILE) == 2 ? 1.f : 0.f;
  }

  auto issue = [&](int t0, int b) {
    float* qs = sm + b * buf_floats;
    float* vs = qs + vec_cols * array;
    float* bs = vs + TILE * cols;
    float* gs = bs + TILE;
    const int tt = min(TILE, q_len - t0);
    auto copy_row = [&](auto copy, int t, int d) {
      const size_t n = (size_t)(t_begin + t0 + t);
      float* to = qs + t * width + d;
      copy(to, p.q + n * p.q_stride + (size_t)kvh * D + d);
      copy(to + array, p.k + n * p.k_stride + (size_t)kvh * D + d);
      if (DECAY == 2) copy(to + 2 * array, p.decay + (n * p.heads + h) * D + d);
      if (RULE == 2) {
        copy(to + 3 * array, p.unit + (n * p.heads + h) * D + d);
        copy(to + 4 * array, p.removal + (n * p.heads + h) * D + d);
      }
    };
    if (p.wide && pad == 0) {                      // a row of a power of two: no division
      for (int e = tid; e < tt * (width / 4); e += kScanThreads) copy_row(copy_async16, e / (width / 4), e % (width / 4) * 4);
    } else if (p.wide) {
      const int quads = D >> 2;
      for (int e = tid; e < tt * quads; e += kScanThreads) copy_row(copy_async16, e / quads, e % quads * 4);
    } else {
      for (int e = tid; e < tt * D; e += kScanThreads) copy_row(copy_async4, e / D, e % D);
    }
    for (int e = tid; e < tt * cols; e += kScanThreads) {
      const int t = e / cols, jj = blockIdx.x * cols + e % cols;
      if (jj < V) copy_async4(vs + e, p.v + (size_t)(t_begin + t0 + t) * p.v_stride + (size_t)h * V + jj);
      else vs[e] = 0.f;
    }
    if (tid < tt) {
      const size_t n = (size_t)(t_begin + t0 + tid);
      if (RULE == 1 || RULE == 3) copy_async4(bs + tid, p.beta + n * p.heads + h);
      if (DECAY == 1) copy_async4(gs + tid, p.decay + n * p.heads + h);
    }
    copy_async_commit();
  };

  const float g_const = DECAY == 0 ? p.decay[h] : 1.f;
  const float skip = (RULE == 3 && p.skip) ? p.skip[h] : 0.f;

  issue(0, 0);
  int b = 0;
  for (int t0 = 0; t0 < q_len; t0 += TILE, b ^= 1) {
    const int tt = min(TILE, q_len - t0);
    if (t0 + TILE < q_len) {
      issue(t0 + TILE, b ^ 1);
      copy_async_wait<1>();
    } else {
      copy_async_wait<0>();
    }
    __syncthreads();
    const float* qp = sm + b * buf_floats + l * 4;         // this lane's first piece of q; the other vectors follow
    const float* vp = sm + b * buf_floats + vec_cols * array + c * C;
    const float* bp = sm + b * buf_floats + vec_cols * array + TILE * cols;
    using Token = ScanToken<ROWS, C, RULE, DECAY>;
    auto load = [&](Token& x, int t) {
      const float* r = qp + t * width;
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        x.q[i] = *reinterpret_cast<const float4*>(r + i * L * 4);
        x.k[i] = *reinterpret_cast<const float4*>(r + array + i * L * 4);
        if constexpr (DECAY == 2) x.g[i] = *reinterpret_cast<const float4*>(r + 2 * array + i * L * 4);
        if constexpr (RULE == 2) {
          x.u[i] = *reinterpret_cast<const float4*>(r + 3 * array + i * L * 4);
          x.a[i] = *reinterpret_cast<const float4*>(r + 4 * array + i * L * 4);
        }
      }
#pragma unroll
      for (int cc = 0; cc < C; ++cc) x.v[cc] = vp[t * cols + cc];
      if constexpr (RULE == 1 || RULE == 3) x.beta = bp[t];
      if constexpr (DECAY == 1) x.decay = bp[TILE + t];
    };
    // one token: the state moves on; this lane's shares of the read-outs
    auto step = [&](const Token& x, float* share) {
      float dot[C];
      if constexpr (RULE == 2) {
        // both the decay and the removal read the old state: the dot products u . S first, then every row in one
        // expression, then the read-out as in the other rules
        lane_dots<Q, L, C>(S, x.u, dot);
#pragma unroll
        for (int cc = 0; cc < C; ++cc) {
          const float2 md = make_float2(-dot[cc], -dot[cc]), vv = make_float2(x.v[cc], x.v[cc]);
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            S[cc][2 * i] = fma2(lo2(x.k[i]), vv, fma2(lo2(x.a[i]), md, mul2(S[cc][2 * i], lo2(x.g[i]))));
            S[cc][2 * i + 1] = fma2(hi2(x.k[i]), vv, fma2(hi2(x.a[i]), md, mul2(S[cc][2 * i + 1], hi2(x.g[i]))));
          }
        }
      } else {
        const float g = DECAY == 1 ? x.decay : g_const;
        const float2 gg = make_float2(g, g);
#pragma unroll
        for (int cc = 0; cc < C; ++cc)
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            S[cc][2 * i] = mul2(S[cc][2 * i], DECAY == 2 ? lo2(x.g[i]) : gg);
            S[cc][2 * i + 1] = mul2(S[cc][2 * i + 1], DECAY == 2 ? hi2(x.g[i]) : gg);
          }
        if constexpr (RULE == 1) lane_dots<Q, L, C>(S, x.k, dot);
#pragma unroll
        for (int cc = 0; cc < C; ++cc) {
          float u = x.v[cc];
          if constexpr (RULE == 1) u = x.beta * (u - dot[cc]);
          if constexpr (RULE == 3) u *= x.beta;
          const float2 uu = make_float2(u, u);
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            S[cc][2 * i] = fma2(lo2(x.k[i]), uu, S[cc][2 * i]);
            S[cc][2 * i + 1] = fma2(hi2(x.k[i]), uu, S[cc][2 * i + 1]);
          }
        }
      }
#pragma unroll
      for (int cc = 0; cc < C; ++cc) {
        share[cc] = share_dot<Q>(S[cc], x.q);
        if (RULE == 3 && l == 0) share[cc] = __fmaf_rn(skip, x.v[cc], share[cc]);   // the token's own value joins the first lane's share
      }
    };
    int t = 0;
    if constexpr (TILE >= 4) {
      if (tt >= 4) {
        Token x[2];
        load(x[0], 0);
#pragma unroll 1
        for (; t + 4 <= tt; t += 4) {
          float r[4 * C];
          load(x[1], t + 1);
          step(x[0], r);
          load(x[0], t + 2);
          step(x[1], r + C);
          load(x[1], t + 3);
          step(x[0], r + 2 * C);
          load(x[0], min(t + 4, TILE - 1));       // (the row past the tile's last token is not used)
          step(x[1], r + 3 * C);
          lane_sums<4 * C, L>(r, l);
          constexpr int per = L >= 4 * C ? 1 : 4 * C / L, share = L >= 4 * C ? L / (4 * C) : 1;
          if (l % share == 0)
#pragma unroll
            for (int i = 0; i < per; ++i) {
              const int at = l / share * per + i;                     // (token, column) of the sum
              outs[(t + at / C) * cols + c * C + at % C] = r[i];
            }
        }
      }
    }
    for (; t < tt; ++t) {
      Token x;
      load(x, t);
      float r[C];
      step(x, r);
      lane_sums<C, L>(r, l);
      constexpr int per = L >= C ? 1 : C / L, share = L >= C ? L / C : 1;
      if (l % share == 0)
#pragma unroll
        for (int i = 0; i < per; ++i) outs[t * cols + c * C + l / share * per + i] = r[i];
    }
    __syncthreads();                // the next round's copies overwrite the other buffer, which the round after reads
    for (int e = tid; e < tt * cols; e += kScanThreads) {
      const int jj = blockIdx.x * cols + e % cols;
      if (jj < V) p.out[(size_t)(t_begin + t0 + e / cols) * p.out_stride + (size_t)h * V + jj] = outs[e];
    }
  }
#pragma unroll
  for (int cc = 0; cc < C; ++cc)
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int d = (i * L + l) * 4;
      if (j + cc < V && d < Dp)
        *reinterpret_cast<float4*>(sp + (size_t)cc * Dp + d) = make_float4(S[cc][2 * i].x, S[cc][2 * i].y, S[cc][2 * i + 1].x, S[cc][2 * i + 1].y);
    }
}

// ---- per-head norm, weight and gate of a mixer's read-out ---------------------------------------------
//   y[n, h, :] = o / sqrt(mean(o^2) + eps) * weight * act(gate[n, h, :]) * out_scale
// GATE: 0 none, 1 silu, 2 sigmoid.
template <typename T>
__global__ void head_norm_gate_kernel(const float* o, int o_stride, const float* __restrict__ weight,
                                      const T* gate, int gate_stride, int gate_kind, T* y,
                                      int y_stride, const int32_t* req_of_token, int heads, int vdim,
                                      float eps, float out_scale, int weight_stride) {
  pdl_launch_dependents();
  pdl_wait();
  // a warp per (token, head): the sum of squares in a fixed order whatever the block holds
  const int n = blockIdx.x, h = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= heads || req_of_token[n] < 0) return;
  const float* op = o + (size_t)n * o_stride + (size_t)h * vdim;
  float ss = 0.f;
  for (int d = lane; d < vdim; d += 32) ss = __fmaf_rn(op[d], op[d], ss);
  ss = warp_sum(ss);
  const float r = 1.0f / sqrtf(ss / (float)vdim + eps);
  for (int d = lane; d < vdim; d += 32) {
    float val = op[d] * r;
    if (weight) val *= weight[(size_t)h * weight_stride + d];
    if (gate_kind) {
      const float z = to_f32<T>(gate[(size_t)n * gate_stride + (size_t)h * vdim + d]);
      val *= gate_kind == 1 ? silu_exact(z) : sigmoid_f(z);
    }
    y[(size_t)n * y_stride + (size_t)h * vdim + d] = from_f32<T>(val * out_scale);
  }
}

// The same for heads of up to 512 values, a multiple of four, on the boundaries of four values: a head stays in registers
// between the sum and the result, everything is read and written once, four values at a time.  2,048 tokens of 16 heads of 128,
// 34 MB: 19 us a value at a time, 15 us this way (ncu, cold), 2.3 TB/s: a warp's chain of load, sum and store leaves little on
// its way.
template <typename T>
__global__ void head_norm_gate_x4_kernel(const float* o, int o_stride, const float* weight, const T* gate, int gate_stride,
                                         int gate_kind, T* y, int y_stride, const int32_t* req_of_token, int heads, int vdim,
                                         float eps, float out_scale, int weight_stride) {
  pdl_launch_dependents();
  pdl_wait();
  const int n = blockIdx.x, h = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= heads || req_of_token[n] < 0) return;
  const float* op = o + (size_t)n * o_stride + (size_t)h * vdim;
  const T* gp = gate_kind ? gate + (size_t)n * gate_stride + (size_t)h * vdim : nullptr;
  float4 v[4], g[4];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int d = i * 128 + lane * 4;
    if (i * 128 >= vdim) break;                    // (uniform)
    v[i] = g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (d < vdim) {
      v[i] = load4_f32(op + d);
      if (gate_kind) g[i] = load4_f32(gp + d);
    }
    ss += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
  }
  ss = warp_sum(ss);
  const float r = 1.0f / sqrtf(ss / (float)vdim + eps);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int d = i * 128 + lane * 4;
    if (d >= vdim) break;
    float4 x = make_float4(v[i].x * r, v[i].y * r, v[i].z * r, v[i].w * r);
    if (weight) {
      const float4 w = load4_f32(weight + (size_t)h * weight_stride + d);
      x.x *= w.x; x.y *= w.y; x.z *= w.z; x.w *= w.w;
    }
    if (gate_kind == 1) {
      x.x *= silu_exact(g[i].x); x.y *= silu_exact(g[i].y); x.z *= silu_exact(g[i].z); x.w *= silu_exact(g[i].w);
    } else if (gate_kind) {
      x.x *= sigmoid_f(g[i].x); x.y *= sigmoid_f(g[i].y); x.z *= sigmoid_f(g[i].z); x.w *= sigmoid_f(g[i].w);
    }
    store4(y + (size_t)n * y_stride + (size_t)h * vdim + d, make_float4(x.x * out_scale, x.y * out_scale, x.z * out_scale, x.w * out_scale));
  }
}

// ---- gate and norm in equal parts -------------------------------------------------------------------------------
//   y = o * act(z);   y[part] <- y / sqrt(mean(y^2 over the part) + eps) * weight * out_scale           (after = 0)
//   y = o / sqrt(mean(o^2 over the part) + eps) * weight * act(z) * out_scale                            (after = 1)
// GATE: 1 silu, 2 sigmoid.  A block per (token, part); a part waits in shared memory between the two passes.  VEC: four
// values at a time (all rows and parts on 16-byte boundaries of float32, 8-byte ones of bfloat16).
__device__ __forceinline__ float gate_value(float z, int kind) { return kind == 1 ? silu_exact(z) : sigmoid_f(z); }

template <typename T, bool VEC>
__global__ void gate_norm_kernel(const float* o, int o_stride, const T* z, int z_stride,
                                 const float* __restrict__ weight, T* y, int y_stride,
                                 const int32_t* req_of_token, int width, float eps, float out_scale, int kind,
                                 int after) {
  extern __shared__ __align__(16) float part_s[];  // [width]
  __shared__ float scratch[32];
  pdl_launch_dependents();
  pdl_wait();
  const int n = blockIdx.x, c0 = blockIdx.y * width;
  if (req_of_token[n] < 0) return;
  const float* op = o + (size_t)n * o_stride + c0;
  const T* zp = z + (size_t)n * z_stride + c0;
  T* yp = y + (size_t)n * y_stride + c0;
  const float* wp = weight + c0;
  float ss = 0.f;
  if constexpr (VEC) {
    for (int c = threadIdx.x * 4; c < width; c += blockDim.x * 4) {
      float4 v = load4_f32(op + c);
      if (!after) {
        const float4 g = load4_f32(zp + c);
        v.x *= gate_value(g.x, kind); v.y *= gate_value(g.y, kind); v.z *= gate_value(g.z, kind); v.w *= gate_value(g.w, kind);
      }
      *reinterpret_cast<float4*>(part_s + c) = v;
      ss = __fmaf_rn(v.x, v.x, ss); ss = __fmaf_rn(v.y, v.y, ss); ss = __fmaf_rn(v.z, v.z, ss); ss = __fmaf_rn(v.w, v.w, ss);
    }
    const float r = out_scale / sqrtf(block_sum(ss, scratch) / (float)width + eps);
    for (int c = threadIdx.x * 4; c < width; c += blockDim.x * 4) {
      float4 v = *reinterpret_cast<const float4*>(part_s + c);
      const float4 w = load4_f32(wp + c);
      v.x *= r * w.x; v.y *= r * w.y; v.z *= r * w.z; v.w *= r * w.w;
      if (after) {
        const float4 g = load4_f32(zp + c);
        v.x *= gate_value(g.x, kind); v.y *= gate_value(g.y, kind); v.z *= gate_value(g.z, kind); v.w *= gate_value(g.w, kind);
      }
      store4(yp + c, v);
    }
  } else {
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
      const float v = after ? op[c] : op[c] * gate_value(to_f32<T>(zp[c]), kind);
      part_s[c] = v;
      ss = __fmaf_rn(v, v, ss);
    }
    const float r = out_scale / sqrtf(block_sum(ss, scratch) / (float)width + eps);
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
      const float v = part_s[c] * r * wp[c];
      yp[c] = from_f32<T>(after ? v * gate_value(to_f32<T>(zp[c]), kind) : v);
    }
  }
}

// ---- what the generalized delta rule reads ------------------------------------------------------------
// From the projections of a token (model dtype): q, k, v as float32; per head and key channel the decay
// g = exp(-rate * sigmoid(w_raw + w_bias)), the unit key u = k / sqrt(sum k^2 + unit_eps) of each head and the
// removal vector sigmoid(a_raw + a_bias) * u.  A block per token, a warp per head in turn; float32 throughout.
// VEC: four neighbouring channels a lane (everything on the boundaries of four values, heads that keep all lanes busy); the sum
// over a head has the same order in both forms.  2,048 tokens of 16 heads of 128: a value a lane 26.8 us, four 22.5; of 24 heads
// of 64, which leave half the lanes idle: 20.3 and 25.5.
template <typename T, bool VEC>
__global__ void general_delta_prepare_kernel(const T* q, const T* k, const T* v,
                                             int in_stride, const T* a_raw, int a_stride,
                                             const float* __restrict__ a_bias, const T* w_raw, int w_stride,
                                             const float* __restrict__ w_bias, float rate, float unit_eps,
                                             const int32_t* req_of_token, int heads, int dim,
                                             float* out, size_t plane) {
  pdl_launch_dependents();
  pdl_wait();
  const int n = blockIdx.x;
  if (req_of_token[n] < 0) return;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, width = heads * dim;
  float* row = out + (size_t)n * width;           // six planes [N, width]: q, k, v, decay, unit, removal
  for (int h = blockIdx.y * nw + (threadIdx.x >> 5); h < heads; h += nw * gridDim.y) {   // a warp per head
    float ss = 0.f;
    for (int d = lane; d < dim; d += 32) {
      const float kv = to_f32<T>(k[(size_t)n * in_stride + h * dim + d]);
      ss = __fmaf_rn(kv, kv, ss);
    }
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss + unit_eps);
    if constexpr (VEC) {
      for (int d = lane * 4; d < dim; d += 128) {
        const int c = h * dim + d;
        const float4 kv = load4_f32(k + (size_t)n * in_stride + c), qv = load4_f32(q + (size_t)n * in_stride + c);
        const float4 vv = load4_f32(v + (size_t)n * in_stride + c), wv = load4_f32(w_raw + (size_t)n * w_stride + c);
        const float4 av = load4_f32(a_raw + (size_t)n * a_stride + c), wb = load4_f32(w_bias + c), ab = load4_f32(a_bias + c);
        const float4 u = make_float4(kv.x * inv, kv.y * inv, kv.z * inv, kv.w * inv);
        auto decay = [&](float z) { return expf(-rate * sigmoid_f(z)); };
        store4(row + c, qv);
        store4(row + 1 * plane + c, kv);
        store4(row + 2 * plane + c, vv);
        store4(row + 3 * plane + c, make_float4(decay(wv.x + wb.x), decay(wv.y + wb.y), decay(wv.z + wb.z), decay(wv.w + wb.w)));
        store4(row + 4 * plane + c, u);
        store4(row + 5 * plane + c, make_float4(sigmoid_f(av.x + ab.x) * u.x, sigmoid_f(av.y + ab.y) * u.y,
                                                sigmoid_f(av.z + ab.z) * u.z, sigmoid_f(av.w + ab.w) * u.w));
      }
    } else {
      for (int d = lane; d < dim; d += 32) {
        const int c = h * dim + d;
        const float kv = to_f32<T>(k[(size_t)n * in_stride + c]);
        const float qv = to_f32<T>(q[(size_t)n * in_stride + c]), vv = to_f32<T>(v[(size_t)n * in_stride + c]);
        const float wv = to_f32<T>(w_raw[(size_t)n * w_stride + c]) + w_bias[c];
        const float av = to_f32<T>(a_raw[(size_t)n * a_stride + c]) + a_bias[c], u = kv * inv;
        row[c] = qv;
        row[1 * plane + c] = kv;
        row[2 * plane + c] = vv;
        row[3 * plane + c] = expf(-rate * sigmoid_f(wv));
        row[4 * plane + c] = u;
        row[5 * plane + c] = sigmoid_f(av) * u;
      }
    }
  }
}

}  // namespace

// out: float32 [6, n_tokens, heads * dim]: q, k, v, decay, unit key, removal vector.
YALIS_API int yalis_general_delta_prepare(const void* q, const void* k, const void* v, int in_stride, const void* a_raw,
                                          int a_stride, const float* a_bias, const void* w_raw, int w_stride,
                                          const float* w_bias, float rate, float unit_eps, const int32_t* req_of_token,
                                          int n_tokens, int heads, int dim, int dtype, float* out,
                                          cudaStream_t stream) {
  if (n_tokens <= 0) return YALIS_OK;
  if (heads <= 0 || dim <= 0) return YALIS_ERR_SHAPE;
  // steps of few tokens: two heads a block, so that a decode step of 8 tokens fills more than 8 SMs
  const int per_block = n_tokens >= 512 ? 8 : 2;
  const int warps = heads < per_block ? heads : per_block;
  const uintptr_t narrow = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)a_raw | (uintptr_t)w_raw;
  const bool vec = dim >= 128 && ((dim | in_stride | a_stride | w_stride) & 3) == 0 && (narrow & (dtype == YALIS_BF16 ? 7 : 15)) == 0 &&
                   (((uintptr_t)a_bias | (uintptr_t)w_bias | (uintptr_t)out) & 15) == 0;
  const dim3 grid(n_tokens, (heads + warps - 1) / warps), block(32 * warps);
  const size_t plane = (size_t)n_tokens * heads * dim;
  YALIS_DISPATCH_DTYPE(dtype, T, {
    auto go = [&](auto kernel) {
      return yalis_launch(kernel, grid, block, 0, stream, (const T*)q, (const T*)k, (const T*)v, in_stride, (const T*)a_raw, a_stride,
                          a_bias, (const T*)w_raw, w_stride, w_bias, rate, unit_eps, req_of_token, heads, dim, out, plane);
    };
    return vec ? go(general_delta_prepare_kernel<T, true>) : go(general_delta_prepare_kernel<T, false>);
  });
  return YALIS_OK;
}

// b_raw null (with a_raw [N, heads]): beta_out receives the step sizes softplus(a_raw + dt_bias).
// single_tokens: no request brings more than one token (the tails are then written by the same kernel).
// a_raw null: no decay and write strength are computed.  kv_heads 0: no head is brought to unit length.
YALIS_API int yalis_delta_prepare(const void* x, int dtype, int x_stride, const float* w, float* tail,
                                  int64_t slot_stride, const int32_t* req_of_token, const int32_t* q_start,
                                  const int32_t* slots, float* out, int out_stride, int n_tokens, int n_requests,
                                  int channels, int taps, int kv_heads, int dim, float q_scale, float unit_eps,
                                  const void* a_raw, int a_stride, int a_cols, const float* a_log, const float* dt_bias,
                                  const void* b_raw, int b_stride, int heads, float* g_out, float* beta_out,
                                  const float* conv_bias, int single_tokens, cudaStream_t stream) {
  if (n_tokens <= 0) return YALIS_OK;
  if (taps < 1 || taps > kMaxTaps || channels <= 0 || kv_heads < 0 || 2 * kv_heads * dim > channels) return YALIS_ERR_SHAPE;
  if (a_raw && (heads <= 0 || a_cols % heads || !a_log || !dt_bias || (!b_raw && a_cols != heads) || !g_out || !beta_out)) return YALIS_ERR_SHAPE;
  DeltaPrepareParams p;
  p.x = x; p.x_stride = x_stride; p.w = w; p.conv_bias = conv_bias; p.tail = tail; p.slot_stride = (size_t)slot_stride;
  p.req_of_token = req_of_token; p.q_start = q_start; p.slots = slots; p.out = out; p.out_stride = out_stride;
  p.n_tokens = n_tokens; p.channels = channels; p.taps = taps; p.single = single_tokens;
  p.kv_heads = kv_heads; p.dim = dim; p.q_scale = q_scale; p.unit_eps = unit_eps;
  p.a_raw = a_raw; p.a_stride = a_stride; p.a_cols = a_cols; p.a_log = a_log; p.dt_bias = dt_bias;
  p.b_raw = b_raw; p.b_stride = b_stride; p.heads = heads; p.g_out = g_out; p.beta_out = beta_out;
  const size_t element = dtype == YALIS_BF16 ? 2 : 4;
  const bool pairs = channels % 2 == 0 && x_stride % 2 == 0 && out_stride % 2 == 0 && ((uintptr_t)x % (2 * element)) == 0 &&
                     ((uintptr_t)out & 7) == 0 && (kv_heads == 0 || dim % 2 == 0);
  const int v = pairs ? 2 : 1, threads = n_tokens >= 512 ? 256 : 128;
  // a piece holds whole heads where heads are brought to unit length
  p.piece = kv_heads > 0 ? (threads * v + dim - 1) / dim * dim : threads * v;
  p.tile = n_tokens >= 1024 ? 8 : (n_tokens >= 256 ? 2 : 1);
  const dim3 grid((n_tokens + p.tile - 1) / p.tile, (channels + p.piece - 1) / p.piece);
  if (grid.y > 65535) return YALIS_ERR_SHAPE;
  const int pieces = (channels / 128 + 7) / 8;
  const bool by_tiles = !single_tokens && n_tokens >= kConvTileFrom && n_tokens >= 8ll * n_requests && (long long)n_tokens * channels >= (1 << 20) &&
                        taps <= 4 && channels % 128 == 0 && (kv_heads == 0 || dim == 128) && pieces <= 65535;
  YALIS_DISPATCH_DTYPE(dtype, T, {
    int st;
    if (by_tiles) st = yalis_launch(conv_tile_kernel<T>, dim3((n_tokens + kConvTile - 1) / kConvTile, pieces), dim3(256), 0, stream, p);
    else if (taps <= 4)
      st = pairs ? yalis_launch(delta_prepare_kernel<T, 4, 2>, grid, dim3(threads), 0, stream, p)
                 : yalis_launch(delta_prepare_kernel<T, 4, 1>, grid, dim3(threads), 0, stream, p);
    else
      st = yalis_launch(delta_prepare_kernel<T, kMaxTaps, 1>, grid, dim3(threads), 0, stream, p);
    if (st != YALIS_OK || taps == 1 || single_tokens) return st;
    return yalis_launch(short_conv_tail_kernel<T>, dim3(n_requests, (channels + 127) / 128), dim3(128), 0, stream, (const T*)x,
                        x_stride, tail, (size_t)slot_stride, q_start, slots, channels, taps);
  });
  return YALIS_OK;
}

template <int ROWS, int LANES, int COLS, int RULE, int DECAY, int TILE>
static int launch_scan_tile(const ScanParams& p, int n_requests, bool early, cudaStream_t stream) {
  constexpr int cols = kScanThreads / LANES * COLS, vec_cols = RULE == 2 ? 5 : (DECAY == 2 ? 3 : 2);
  constexpr size_t smem = (2 * (size_t)scan_buffer_floats(vec_cols, TILE, ROWS * LANES, cols) + TILE * cols) * sizeof(float);
  static_assert(smem <= 200 * 1024, "two buffers and the read-outs fit a block");
  auto kernel = state_scan_kernel<ROWS, LANES, COLS, RULE, DECAY, TILE>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return YALIS_ERR_LAUNCH;
  const dim3 grid((p.vdim + cols - 1) / cols, p.heads, n_requests);
  if (!early) return yalis_launch_after(kernel, grid, dim3(kScanThreads), smem, stream, p);
  return yalis_launch(kernel, grid, dim3(kScanThreads), smem, stream, p);
}

// The staging tile goes by the longest portion: a tile of 16 tokens for portions of two to four holds shared memory that other
// blocks of the SM need (64 requests of two tokens, heads of 256, generalized rule: 225 us, 86 in a tile of two).  Portions up
// to 128 tokens may start before the kernel in front has ended: their blocks do not hold an SM for long.
template <int ROWS, int LANES, int COLS, int RULE, int DECAY>
static int launch_scan(const ScanParams& p, int n_requests, int longest, cudaStream_t stream) {
  if (longest == 1) return launch_scan_tile<ROWS, LANES, COLS, RULE, DECAY, 1>(p, n_requests, true, stream);
  if (longest > 0 && longest <= 4) return launch_scan_tile<ROWS, LANES, COLS, RULE, DECAY, 4>(p, n_requests, true, stream);
  return launch_scan_tile<ROWS, LANES, COLS, RULE, DECAY, (ROWS * LANES > 256 ? 8 : 16)>(p, n_requests, longest > 0 && longest <= 128, stream);
}

// The smallest power of two of lanes that covers dim.  Delta rules: 16 rows of one column a thread; the others 8 rows of two
// neighbouring columns (beyond 256 rows 16 of one).  Sums over a column have one order per rule and dim, whatever the step.
template <int RULE, int DECAY>
static int launch_scan_dim(const ScanParams& p, int n_requests, int longest, cudaStream_t stream) {
  if constexpr (RULE == 1) {
    if (p.dim <= 16) return launch_scan<16, 1, 1, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 32) return launch_scan<16, 2, 1, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 64) return launch_scan<16, 4, 1, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 128) return launch_scan<16, 8, 1, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 256) return launch_scan<16, 16, 1, RULE, DECAY>(p, n_requests, longest, stream);
  } else {
    if (p.dim <= 8) return launch_scan<8, 1, 2, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 16) return launch_scan<8, 2, 2, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 32) return launch_scan<8, 4, 2, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 64) return launch_scan<8, 8, 2, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 128) return launch_scan<8, 16, 2, RULE, DECAY>(p, n_requests, longest, stream);
    if (p.dim <= 256) return launch_scan<8, 32, 2, RULE, DECAY>(p, n_requests, longest, stream);
  }
  return launch_scan<16, 32, 1, RULE, DECAY>(p, n_requests, longest, stream);
}
// decay_kind 0: decay [heads]; 1: decay [N, heads]; 2: decay [N, heads * dim].  delta 1: the delta rule with beta
// [N, heads]; delta 2: the generalized delta rule with unit keys and removal vectors [N, heads * dim] (contiguous,
// kv_heads = heads, decay_kind 2); delta 3: the selective form, beta [N, heads] the step sizes and skip [heads] (or null)
// the token's own value in the read-out (decay_kind 1).
// max_q_len: the longest portion of the step if the caller knows it (0: not known); it only chooses the staging tile.
// limit > 0: portions of limit to upto tokens are left alone.
YALIS_API int yalis_state_scan(const float* q, int q_stride, const float* k, int k_stride, const float* v, int v_stride,
                               const float* decay, int decay_kind, const float* beta, const float* skip, const float* unit,
                               const float* removal, float* state, int64_t slot_stride,
                               float* out, int out_stride, const int32_t* q_start, const int32_t* slots, int n_requests,
                               int heads, int kv_heads, int dim, int vdim, int delta, int max_q_len, int limit, int upto, cudaStream_t stream) {
  if (n_requests <= 0) return YALIS_OK;
  if (dim <= 0 || vdim <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || heads > 65535 || n_requests > 65535)
    return YALIS_ERR_SHAPE;
  if (dim > 512) return YALIS_ERR_SHAPE;
  if (decay_kind < 0 || decay_kind > 2 || !decay || delta < 0 || delta > 3 || (delta == 1 && !beta)) return YALIS_ERR_SHAPE;
  if (delta == 3 && (decay_kind != 1 || !beta)) return YALIS_ERR_SHAPE;
  if (delta == 2 && (decay_kind != 2 || !unit || !removal || kv_heads != heads)) return YALIS_ERR_SHAPE;
  const int dim_padded = (dim + 3) & ~3;
  if ((slot_stride & 3) || ((uintptr_t)state & 15)) return YALIS_ERR_ALIGN;
  ScanParams p;
  p.q = q; p.q_stride = q_stride; p.k = k; p.k_stride = k_stride; p.v = v; p.v_stride = v_stride;
  p.decay = decay; p.beta = beta; p.skip = skip; p.unit = unit; p.removal = removal; p.state = state; p.slot_stride = (size_t)slot_stride; p.out = out;
  p.out_stride = out_stride; p.q_start = q_start; p.slots = slots; p.heads = heads; p.kv_heads = kv_heads;
  p.dim = dim; p.dim_padded = dim_padded; p.vdim = vdim; p.limit = limit; p.upto = upto;
  p.wide = (dim % 4 == 0 && q_stride % 4 == 0 && k_stride % 4 == 0 && !((uintptr_t)q & 15) && !((uintptr_t)k & 15) &&
            (decay_kind != 2 || !((uintptr_t)decay & 15)) &&
            (delta != 2 || (!((uintptr_t)unit & 15) && !((uintptr_t)removal & 15)))) ? 1 : 0;
  const int longest = max_q_len;
  if (delta == 2) return launch_scan_dim<2, 2>(p, n_requests, longest, stream);
  if (delta == 3) return launch_scan_dim<3, 1>(p, n_requests, longest, stream);
  if (delta && decay_kind == 1) return launch_scan_dim<1, 1>(p, n_requests, longest, stream);
  if (delta && decay_kind == 2) return launch_scan_dim<1, 2>(p, n_requests, longest, stream);
  if (delta) return launch_scan_dim<1, 0>(p, n_requests, longest, stream);
  if (decay_kind == 0) return launch_scan_dim<0, 0>(p, n_requests, longest, stream);
  if (decay_kind == 1) return launch_scan_dim<0, 1>(p, n_requests, longest, stream);
  return launch_scan_dim<0, 2>(p, n_requests, longest, stream);
}

YALIS_API int yalis_head_norm_gate(const float* o, int o_stride, const float* weight, const void* gate, int gate_stride,
                                   int gate_kind, void* y, int y_stride, int dtype, const int32_t* req_of_token,
                                   int n_tokens, int heads, int vdim, float eps, float out_scale, int weight_per_head,
                                   cudaStream_t stream) {
  if (n_tokens <= 0) return YALIS_OK;
  if (heads <= 0 || heads > 65535 || vdim <= 0 || gate_kind < 0 || gate_kind > 2 || (gate_kind && !gate)) return YALIS_ERR_SHAPE;
  const int warps = heads < 4 ? heads : 4;
  const uintptr_t narrow = dtype == YALIS_BF16 ? 7 : 15;
  if (vdim <= 512 && ((vdim | o_stride | y_stride | (gate_kind ? gate_stride : 0)) & 3) == 0 &&
      !(((uintptr_t)o | (uintptr_t)weight) & 15) && !(((uintptr_t)y | (uintptr_t)(gate_kind ? gate : nullptr)) & narrow))
    YALIS_DISPATCH_DTYPE(dtype, T,
                         return yalis_launch(head_norm_gate_x4_kernel<T>, dim3(n_tokens, (heads + warps - 1) / warps),
                                             dim3(32 * warps), 0, stream, o, o_stride, weight, (const T*)gate, gate_stride,
                                             gate_kind, (T*)y, y_stride, req_of_token, heads, vdim, eps, out_scale,
                                             weight_per_head ? vdim : 0));
  YALIS_DISPATCH_DTYPE(dtype, T,
                       return yalis_launch(head_norm_gate_kernel<T>, dim3(n_tokens, (heads + warps - 1) / warps),
                                           dim3(32 * warps), 0, stream, o, o_stride, weight, (const T*)gate, gate_stride,
                                           gate_kind, (T*)y, y_stride, req_of_token, heads, vdim, eps, out_scale,
                                           weight_per_head ? vdim : 0));
  return YALIS_OK;
}

// o float32 [N, parts * width]; z (model dtype) the gate's input; weight float32 [parts * width]; y in the model dtype.
// gate_kind 1: silu, 2: sigmoid; after: the gate stands behind the norm.
YALIS_API int yalis_gate_norm(const float* o, int o_stride, const void* z, int z_stride, const float* weight, void* y,
                              int y_stride, int dtype, const int32_t* req_of_token, int n_tokens, int parts, int width,
                              float eps, float out_scale, int gate_kind, int after, cudaStream_t stream) {
  if (n_tokens <= 0) return YALIS_OK;
  if (parts <= 0 || parts > 65535 || width <= 0 || gate_kind < 1 || gate_kind > 2) return YALIS_ERR_SHAPE;
  const int threads = width >= 1024 ? 256 : (width >= 256 ? 128 : 64);
  const size_t smem = (size_t)width * sizeof(float);
  if (smem > 200 * 1024) return YALIS_ERR_SHAPE;
  const uintptr_t narrow = dtype == YALIS_BF16 ? 7 : 15;
  const bool vec = ((width | o_stride | z_stride | y_stride) & 3) == 0 && !(((uintptr_t)o | (uintptr_t)weight) & 15) &&
                   !(((uintptr_t)z | (uintptr_t)y) & narrow);
  YALIS_DISPATCH_DTYPE(dtype, T, {
    auto kernel = vec ? gate_norm_kernel<T, true> : gate_norm_kernel<T, false>;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
      return YALIS_ERR_LAUNCH;
    return yalis_launch(kernel, dim3(n_tokens, parts), dim3(threads), smem, stream, o, o_stride, (const T*)z, z_stride,
                        weight, (T*)y, y_stride, req_of_token, width, eps, out_scale, gate_kind, after);
  });
  return YALIS_OK;
}
