// Paged causal attention, the exact one: any head size up to 256 (even), any
// number of heads and KV groups, any page size, float32 or bfloat16 storage,
// float32 arithmetic throughout.  The general form: one block per (token, head); each warp walks
// every fourth visible key in ascending order with an online softmax and the
// four partial results are merged in warp order.  For a given (position, head)
// the order of every sum is therefore fixed, whatever else is in the batch and
// however the request was cut into steps.  It is the kernel of the float32
// path and the twin against which the faster bfloat16 kernels are tested.
//
//   S = (q . k_j) * scale for keys j with  pos - window < j <= pos   (window 0: all j <= pos)
//   with chunk C > 0 also  j >= floor(pos / C) * C      (position 0 starts the first chunk)
//   S <- S - slope_h * (pos - j)                                        (slopes given only)
//   S <- cap * tanh(S / cap)                                            (cap > 0 only)
//   O = softmax(S) V, or with a sink: exp(S_j) / (exp(z_h) + sum_i exp(S_i)) V  (a key of score z_h and no value;
//   z_h = sink_logits[h], or 0 without that array)
//   O <- O * sigmoid(gate[t, h, :]), or * sigmoid(gate[t, h])           (gate given only)
//   S <- S + rel[h][min(pos - j, rel_len - 1)]                          (a bias per distance, given only)
// Pooled blocks (pool P > 0, with a window): beside the keys of the window a position sees one key and value for every
// block of P positions that lies wholly before it, blocks b < floor((pos - window + 1) / P); they come from pools of
// their own (entry b of the request's block table over entries) and share the softmax with the window's keys.
// Values may have a head size of their own (hsv).
// Two maps (maps = 2): a query head has two queries and a key/value head two keys per position (each of size hs, side by
// side in the query matrix and in a cached row of 2 hs), and one value; each map is a softmax of its own over the visible
// keys.  With O1, O2 the maps' results  O = O1 - lambda * O2,  O <- O / sqrt(mean(O^2) + eps) * out_scale.
// Mask by absolute position: yalis/attention/backend_impl/sdpa_and_flex.py:15-19, 301-307.
// KV head of query head h: h / (nh / g)                                 (:59-67).
#include "common.cuh"

namespace {

constexpr int kWarps = 4;
constexpr int kMaxPerLane = 8;  // head size <= 256

template <typename T>
struct GenericParams {
  const T* q; int q_stride;
  T* out; int out_stride;
  const T* k_pool; const T* v_pool;
  const int32_t* positions; const int32_t* req_of_token; const int32_t* block_table;
  int table_width, page_size, num_pages, nh, g, hs, hsv;
  float scale; int window; float softcap; int sink; float out_scale; int chunk;
  const float* sink_logits; const float* slopes;
  const float* rel; int rel_len;                 // [nh, rel_len] or null
  const T* gate; int gate_stride, gate_per_head; // [N, nh * hsv], or [N, nh] per head
  int pool;                                      // P > 0: pooled blocks before the window
  const T* pk_pool; const T* pv_pool; const int32_t* pool_table;
  int pool_table_width, pool_page_size, pool_num_pages;   // in entries (one per block)
  float lambda, diff_eps;                        // two maps
};

template <typename T, int MAPS>
__global__ void paged_attention_generic_kernel(const GenericParams<T> p) {
  extern __shared__ float smem[];  // per map [kWarps][hsv] accumulators, then m[kWarps], l[kWarps]; two maps: [hsv] besides
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y;
  const int req = p.req_of_token[t];
  if (req < 0) return;
  const int pos = p.positions[t];
  const int kvh = h / (p.nh / p.g);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per_lane = (p.hs + 31) >> 5, per_lane_v = (p.hsv + 31) >> 5;

  float qr[MAPS][kMaxPerLane], acc[MAPS][kMaxPerLane];
  const T* qp = p.q + (size_t)t * p.q_stride + (size_t)h * (MAPS * p.hs);
#pragma unroll
  for (int a = 0; a < MAPS; ++a)
#pragma unroll
    for (int i = 0; i < kMaxPerLane; ++i) {
      const int d = lane + 32 * i;
      qr[a][i] = (i < per_lane && d < p.hs) ? to_f32<T>(qp[a * p.hs + d]) : 0.f;
      acc[a][i] = 0.f;
    }
  float m[MAPS], l[MAPS];
#pragma unroll
  for (int a = 0; a < MAPS; ++a) {
    m[a] = -INFINITY;
    l[a] = 0.f;
  }
  int lo = (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0;
  if (p.chunk > 0) lo = max(lo, (pos / p.chunk) * p.chunk);
  const float slope = p.slopes ? p.slopes[h] : 0.f;
  const int32_t* bt = p.block_table + (size_t)req * p.table_width;
  // the pooled blocks first, then the window's keys: one row of places, of which each warp walks every fourth
  const int blocks = (p.pool > 0 && p.window > 0 && pos - p.window + 1 > 0) ? (pos - p.window + 1) / p.pool : 0;
  for (int at = warp; at < blocks + pos - lo + 1; at += kWarps) {
    const bool pooled = at < blocks;
    const int j = pooled ? at : lo + (at - blocks);
    const int ps = pooled ? p.pool_page_size : p.page_size;
    const int pi = j / ps;
    const int32_t* table = pooled ? p.pool_table + (size_t)req * p.pool_table_width : bt;
    const int page = pi < (pooled ? p.pool_table_width : p.table_width) ? table[pi] : -1;
    if (page < 0 || page >= (pooled ? p.pool_num_pages : p.num_pages)) continue;  // unmapped: treated as masked
    const size_t row = ((size_t)page * p.g + kvh) * ps + (j - pi * ps);
    const T* kp = (pooled ? p.pk_pool : p.k_pool) + row * (MAPS * p.hs);
    const T* vp = (pooled ? p.pv_pool : p.v_pool) + row * p.hsv;
#pragma unroll
    for (int a = 0; a < MAPS; ++a) {
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < kMaxPerLane; ++i) {
        const int d = lane + 32 * i;
        if (i < per_lane && d < p.hs) dot += qr[a][i] * to_f32<T>(kp[a * p.hs + d]);
      }
      float s = warp_sum(dot) * p.scale;
      if (p.slopes && !pooled) s -= slope * (float)(pos - j);
      if (p.rel && !pooled) s += p.rel[(size_t)h * p.rel_len + min(pos - j, p.rel_len - 1)];
      if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
      const float m_new = fmaxf(m[a], s);
      const float corr = expf(m[a] - m_new);
      const float e = expf(s - m_new);
      l[a] = l[a] * corr + e;
#pragma unroll
      for (int i = 0; i < kMaxPerLane; ++i) {
        const int d = lane + 32 * i;
        if (i < per_lane_v && d < p.hsv) acc[a][i] = acc[a][i] * corr + e * to_f32<T>(vp[d]);
      }
      m[a] = m_new;
    }
  }
  const int map_floats = kWarps * p.hsv + 2 * kWarps;
#pragma unroll
  for (int a = 0; a < MAPS; ++a) {
    float* acc_w = smem + a * map_floats + warp * p.hsv;
#pragma unroll
    for (int i = 0; i < kMaxPerLane; ++i) {
      const int d = lane + 32 * i;
      if (i < per_lane_v && d < p.hsv) acc_w[d] = acc[a][i];
    }
    if (lane == 0) {
      smem[a * map_floats + kWarps * p.hsv + warp] = m[a];
      smem[a * map_floats + kWarps * p.hsv + kWarps + warp] = l[a];
    }
  }
  __syncthreads();
  if constexpr (MAPS == 2) {
    __shared__ float scratch[32];
    float* o_s = smem + 2 * map_floats;
    float wgt[2][kWarps];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const float* ms = smem + a * map_floats + kWarps * p.hsv;
      const float* ls = ms + kWarps;
      float mm = -INFINITY, ll = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, ms[w]);
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        wgt[a][w] = ms[w] == -INFINITY ? 0.f : expf(ms[w] - mm);
        ll += ls[w] * wgt[a][w];
      }
#pragma unroll
      for (int w = 0; w < kWarps; ++w) wgt[a][w] = ll > 0.f ? wgt[a][w] / ll : 0.f;
    }
    float ss = 0.f;
    for (int d = threadIdx.x; d < p.hsv; d += blockDim.x) {
      float o[2] = {0.f, 0.f};
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int w = 0; w < kWarps; ++w) o[a] += smem[a * map_floats + w * p.hsv + d] * wgt[a][w];
      const float v = o[0] - p.lambda * o[1];
      o_s[d] = v;
      ss = __fmaf_rn(v, v, ss);
    }
    const float r = p.out_scale / sqrtf(block_sum(ss, scratch) / (float)p.hsv + p.diff_eps);
    T* op = p.out + (size_t)t * p.out_stride + (size_t)h * p.hsv;
    for (int d = threadIdx.x; d < p.hsv; d += blockDim.x) op[d] = from_f32<T>(o_s[d] * r);
    return;
  }
  const float* acc_s = smem;
  const float* m_s = smem + kWarps * p.hsv;
  const float* l_s = m_s + kWarps;
  float mm = -INFINITY;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, m_s[w]);
  const float sink_z = (p.sink && p.sink_logits) ? p.sink_logits[h] : 0.f;
  if (p.sink) mm = fmaxf(mm, sink_z);
  float ll = p.sink ? expf(sink_z - mm) : 0.f;
  float wgt[kWarps];
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    wgt[w] = (m_s[w] == -INFINITY) ? 0.f : expf(m_s[w] - mm);
    ll += l_s[w] * wgt[w];
  }
  T* op = p.out + (size_t)t * p.out_stride + (size_t)h * p.hsv;
  for (int d = threadIdx.x; d < p.hsv; d += blockDim.x) {
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) o += acc_s[w * p.hsv + d] * wgt[w];
    float res = ll > 0.f ? o / ll * p.out_scale : 0.f;
    if (p.gate) {
      const size_t at = (size_t)t * p.gate_stride + (p.gate_per_head ? (size_t)h : (size_t)h * p.hsv + d);
      res *= 1.0f / (1.0f + expf(-to_f32<T>(p.gate[at])));
    }
    op[d] = from_f32<T>(res);
  }
}

// ---- the same for float32 heads of 64 and 128, several queries and heads at a time ------------------------------------------
// The form above spends some sixty instructions a key and head, most of them on the sum over a warp and the two exponentials
// of every key.  Here a warp takes a tile of 32 keys for up to eight (query, head) pairs that share a key/value head: a lane has a
// key's scores for all pairs, so there is one maximum, one sum and one exponential a lane for 32 keys, then the lanes
// share out the head's sizes for the values.  Tiles lie at multiples of 32 positions and warp w walks those whose number is w
// modulo four, in ascending order; what a query does not see counts as nothing.  So here, too, the order of every sum is fixed for a
// given position and head.  The keys of the next tile and the values of this one are on their way while a warp computes.
// A block takes the neighbouring tokens of one request whose positions lie in one aligned group of QT (one, two or four): the first
// of them finds the others, the blocks of the others end at once.
// What bounds it: reads of shared memory (16 bytes of a pair's query are two passes beside four products a lane) and, for few
// blocks, the chain of a tile: copy, scores, maximum, exponential, values (as many as registers leave room for are asked for ahead; behind a
// context's end none is waited for).  Measured (us, general form -> now; with half as many registers and every value of the last tile waited for), 32
// heads on 8 of 64 / 128: one token behind 200 40 -> 5.8 (7.0) / 53 -> 7.1 (7.9), 16 tokens behind 8,000 2,132 -> 262 (259) / 2,400 -> 291 (505), 64
// tokens of their own behind 1,000 679 -> 50 / 1,011 -> 140 (143), a prompt of 250 247 -> 42 (48) / 269 -> 60, of 1,024 3,699 -> 352 (418) / 4,096 -> 552,
// of 16 6.0 -> 4.1 (4.5) / 6.9 -> 5.4 (8.3), of 8 3.8 -> 3.6 (4.2) / 4.4 -> 4.2 (4.9), of 4 3.0 -> 3.5 (4.0) / 3.3 -> 4.1 (4.5): contexts of a few
// keys are the general form's, but which form a token takes must not depend on what runs beside it.
constexpr int kTile = 32;

__device__ __forceinline__ void copy16(float* to, const float* from, bool there) {      // zeros where there is nothing
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from), "r"(there ? 16 : 0));
}
// The largest of a warp's values; NaN counts for nothing.
__device__ __forceinline__ float warp_top(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

template <int D, int PAIRS>
constexpr size_t tiled_smem() {      // queries; per warp: a tile of keys, the weights
  return (PAIRS * D + kWarps * kTile * (D + 4) + kWarps * PAIRS * kTile) * sizeof(float);
}

// D: the head size; HP: heads of a key/value head that a block takes; QT: queries.
// Blocks an SM for a query a block: what shared memory holds (three for a size of 128) or what leaves registers for the values ahead.  Several
// queries: left to the compiler (0; three or two blocks: prompts of 250 to 1,024 3 to 10 % slower).
constexpr int tiled_blocks(int d, int hp, int qt) { return qt > 1 ? 0 : d == 128 ? 3 : hp == 1 ? 6 : hp == 2 ? 5 : 4; }
template <int D, int HP, int QT>
__global__ void __launch_bounds__(kWarps * 32, tiled_blocks(D, HP, QT)) paged_attention_tiled_kernel(const GenericParams<float> p, int n_tokens) {
  constexpr int P = HP * QT, LK = D + 4, V = D / 32;           // rows of keys padded: lanes read 16 bytes of rows of their own
  extern __shared__ __align__(16) float smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int t0 = blockIdx.x, per = p.nh / p.g, parts = per / HP, kvh = blockIdx.y / parts, h0 = kvh * per + (blockIdx.y % parts) * HP;
  const int req = p.req_of_token[t0], pos0 = p.positions[t0];
  if (req < 0) return;
  if (pos0 % QT != 0 && t0 > 0 && p.req_of_token[t0 - 1] == req && p.positions[t0 - 1] == pos0 - 1) return;
  int nq = 1;
  while (nq < QT && (pos0 + nq) % QT != 0 && t0 + nq < n_tokens && p.req_of_token[t0 + nq] == req && p.positions[t0 + nq] == pos0 + nq) ++nq;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* qs = smem;                                            // [pair][D], a missing query is zeros
  float* ks = smem + P * D + warp * kTile * LK;
  float* ws = smem + P * D + kWarps * kTile * LK + warp * P * kTile;
  for (int e = threadIdx.x; e < P * D; e += kWarps * 32) {
    const int pair = e / D, i = pair / HP;
    qs[e] = i < nq ? p.q[(size_t)(t0 + i) * p.q_stride + (size_t)(h0 + pair % HP) * D + e % D] : 0.f;
  }
  __syncthreads();

  auto first = [&](int pos) {                                  // the first key that a position sees
    const int lo = (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0;
    return p.chunk > 0 ? max(lo, (pos / p.chunk) * p.chunk) : lo;
  };
  const int lo = first(pos0), hi = pos0 + nq - 1;              // (a later position's first key is no earlier)
  const int32_t* bt = p.block_table + (size_t)req * p.table_width;
  // the row in the pools of a lane's key, or -1
  auto find = [&](int tile) {
    const int j = tile * kTile + lane, pi = j / p.page_size;
    if (j < lo || j > hi || pi >= p.table_width) return -1;
    const int page = bt[pi];
    return page < 0 || page >= p.num_pages ? -1 : (page * p.g + kvh) * p.page_size + (j - pi * p.page_size);
  };
  auto fetch_keys = [&](int row) {
#pragma unroll
    for (int e = 0; e < kTile * D / 4; e += 32) {
      const int r = (e + lane) / (D / 4), d = (e + lane) % (D / 4) * 4, at = __shfl_sync(0xffffffffu, row, r);
      copy16(ks + r * LK + d, p.k_pool + (at < 0 ? 0 : (size_t)at * D + d), at >= 0);
    }
    asm volatile("cp.async.commit_group;" ::);
  };
  // a lane's sizes (V neighbouring ones) of the values of rows r .. r + 3 of the tile
  auto fetch_values = [&](int row, int r, float (&v)[4][V]) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int at = __shfl_sync(0xffffffffu, row, r + u);
      const float* from = p.v_pool + (size_t)max(at, 0) * D + lane * V;
      if constexpr (V == 4) {
        const float4 x = at >= 0 ? *reinterpret_cast<const float4*>(from) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[u][0] = x.x; v[u][1] = x.y; v[u][2] = x.z; v[u][3] = x.w;
      } else {
        const float2 x = at >= 0 ? *reinterpret_cast<const float2*>(from) : make_float2(0.f, 0.f);
        v[u][0] = x.x; v[u][1] = x.y;
      }
    }
  };

  float acc[P][V], m[P], l[P];
#pragma unroll
  for (int a = 0; a < P; ++a) {
    m[a] = -INFINITY;
    l[a] = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) acc[a][i] = 0.f;
  }
  const int last = hi / kTile;
  int tile = lo / kTile + ((warp - lo / kTile) & (kWarps - 1));
  int row = tile <= last ? find(tile) : -1;
  if (tile <= last) fetch_keys(row);
  for (; tile <= last; tile += kWarps) {
    const int j = tile * kTile + lane, here = row, next = tile + kWarps;
    float v[2][4][V];
    fetch_values(here, 0, v[0]);
    row = next <= last ? find(next) : -1;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    float s[P][4];
#pragma unroll
    for (int a = 0; a < P; ++a) s[a][0] = s[a][1] = s[a][2] = s[a][3] = 0.f;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      const float4 k = *reinterpret_cast<const float4*>(ks + lane * LK + d);
#pragma unroll
      for (int a = 0; a < P; ++a) {
        const float4 q = *reinterpret_cast<const float4*>(qs + a * D + d);
        s[a][0] = __fmaf_rn(q.x, k.x, s[a][0]); s[a][1] = __fmaf_rn(q.y, k.y, s[a][1]);
        s[a][2] = __fmaf_rn(q.z, k.z, s[a][2]); s[a][3] = __fmaf_rn(q.w, k.w, s[a][3]);
      }
    }
    __syncwarp();
    if (next <= last) fetch_keys(row);
    uint32_t seen[QT], any = 0;
    bool whole = true;
#pragma unroll
    for (int i = 0; i < QT; ++i) {
      seen[i] = __ballot_sync(0xffffffffu, i < nq && here >= 0 && j <= pos0 + i && j >= first(pos0 + i));
      whole = whole && seen[i] == 0xffffffffu;
      any |= seen[i];
    }
#pragma unroll
    for (int a = 0; a < P; ++a) {
      const int i = a / HP, h = h0 + a % HP;
      float x = ((s[a][0] + s[a][1]) + (s[a][2] + s[a][3])) * p.scale;
      if (p.slopes) x -= p.slopes[h] * (float)(pos0 + i - j);
      if (p.rel) x += p.rel[(size_t)h * p.rel_len + max(0, min(pos0 + i - j, p.rel_len - 1))];
      if (p.softcap > 0.f) x = p.softcap * tanhf(x / p.softcap);
      const bool see = (seen[i] >> lane) & 1;
      const float top = fmaxf(m[a], warp_top(see ? x : -INFINITY));
      const float e = see ? expf(x - top) : 0.f, corr = seen[i] != 0 ? expf(m[a] - top) : 1.f;
      l[a] = l[a] * corr + e;                                  // this lane's keys; the lanes meet at the end
      m[a] = top;
      ws[a * kTile + lane] = e;
#pragma unroll
      for (int u = 0; u < V; ++u) acc[a][u] *= corr;
    }
    __syncwarp();
    auto add_values = [&](int r, float (&now)[4][V], float (&next)[4][V]) {
      if (r + 4 < kTile) fetch_values(here, r + 4, next);
#pragma unroll
      for (int i = 0; i < QT; ++i) {
        float mine[4][V];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int e = 0; e < V; ++e) mine[u][e] = now[u][e];
        if (!whole) {                                          // what a query does not see must not reach it, be it infinite
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int e = 0; e < V; ++e) mine[u][e] = (seen[i] >> (r + u) & 1) ? mine[u][e] : 0.f;
        }
#pragma unroll
        for (int a = i * HP; a < (i + 1) * HP; ++a) {
          const float4 w = *reinterpret_cast<const float4*>(ws + a * kTile + r);
#pragma unroll
          for (int e = 0; e < V; ++e)
            acc[a][e] = __fmaf_rn(w.w, mine[3][e], __fmaf_rn(w.z, mine[2][e], __fmaf_rn(w.y, mine[1][e], __fmaf_rn(w.x, mine[0][e], acc[a][e]))));
        }
      }
    };
    if (QT > 1 || HP == 4 || any >> (kTile - 4) != 0) {
#pragma unroll
      for (int r = 0; r < kTile; r += 4) add_values(r, v[(r / 4) & 1], v[(r / 4 + 1) & 1]);
    } else {                                                   // a context's end: the values behind it are not waited for
#pragma unroll 1
      for (int r = 0; r < kTile && any >> r != 0; r += 8) {
        add_values(r, v[0], v[1]);
        add_values(r + 4, v[1], v[0]);
      }
    }
    __syncwarp();
  }
  // the warps' shares, added in warp order
  __syncthreads();
  float* share = smem + P * D;                                 // [warp][pair][D], then maxima and sums [warp][pair]
  float* ms = share + kWarps * P * D;
  float* ls = ms + kWarps * P;
#pragma unroll
  for (int a = 0; a < P; ++a) {
    const float sum = warp_sum(l[a]);
#pragma unroll
    for (int e = 0; e < V; ++e) share[(warp * P + a) * D + lane * V + e] = acc[a][e];
    if (lane == 0) {
      ms[warp * P + a] = m[a];
      ls[warp * P + a] = sum;
    }
  }
  __syncthreads();
  for (int a = warp; a < nq * HP; a += kWarps) {
    const int t = t0 + a / HP, h = h0 + a % HP;
    const float z = (p.sink && p.sink_logits) ? p.sink_logits[h] : 0.f;
    float top = p.sink ? z : -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) top = fmaxf(top, ms[w * P + a]);
    float sum = p.sink ? expf(z - top) : 0.f, wgt[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      wgt[w] = ms[w * P + a] == -INFINITY ? 0.f : expf(ms[w * P + a] - top);
      sum += ls[w * P + a] * wgt[w];
    }
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const int d = lane + 32 * e;
      float o = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) o += share[(w * P + a) * D + d] * wgt[w];
      float res = sum > 0.f ? o / sum * p.out_scale : 0.f;
      if (p.gate) res *= 1.0f / (1.0f + expf(-p.gate[(size_t)t * p.gate_stride + (p.gate_per_head ? (size_t)h : (size_t)h * D + d)]));
      p.out[(size_t)t * p.out_stride + (size_t)h * D + d] = res;
    }
  }
}

template <int D, int HP, int QT>
int launch_tiled(const GenericParams<float>& p, int n_tokens, cudaStream_t stream) {
  constexpr int P = HP * QT;
  constexpr size_t smem = tiled_smem<D, P>();
  static_assert(kWarps * P * D + 2 * kWarps * P <= kWarps * kTile * (D + 4) + kWarps * P * kTile, "the shares fit where the tiles were");
  if (cudaFuncSetAttribute(paged_attention_tiled_kernel<D, HP, QT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return YALIS_ERR_LAUNCH;
  return yalis_launch(paged_attention_tiled_kernel<D, HP, QT>, dim3(n_tokens, p.nh / HP), dim3(kWarps * 32), smem, stream, p, n_tokens);
}
// Which form (the bits are the same): as many heads a block, up to four, as leave two blocks an SM (for a size of 128, of whose blocks an SM has three
// places, one and a half: 16 tokens of 32 heads are then one round of blocks, 8.3 -> 5.4 us), since a block's walk over
// the keys is what a step of few tokens waits for (a token behind 8,000, 32 heads of 128 on 8: 180 us with one head a block, 282 with
// four); several queries a block where one makes more than eight blocks an SM (64 tokens behind 1,000 with 16 heads of 64 on
// 16, all of requests of their own: 346 us with eight queries a block).
template <int D>
int launch_tiled_heads(const GenericParams<float>& p, int n_tokens, cudaStream_t stream) {
  const int per = p.nh / p.g;
  const long long pairs = (long long)n_tokens * p.nh, sms = yalis_sm_count();
  const long long many = D == 128 ? 3 * sms / 2 : 2 * sms;
  const int hp = per % 4 == 0 && pairs / 4 > many ? 4 : per % 2 == 0 && pairs / 2 > many ? 2 : 1;
  const bool single = pairs / hp <= 8 * sms;
  if (hp == 4) return single ? launch_tiled<D, 4, 1>(p, n_tokens, stream) : launch_tiled<D, 4, 2>(p, n_tokens, stream);
  if (hp == 2) return single ? launch_tiled<D, 2, 1>(p, n_tokens, stream) : launch_tiled<D, 2, 4>(p, n_tokens, stream);
  return single ? launch_tiled<D, 1, 1>(p, n_tokens, stream) : launch_tiled<D, 1, 4>(p, n_tokens, stream);
}

// Rows of the pools in 16-byte pieces whose numbers fit 32 bits, one map, no pooled blocks.
template <typename T>
bool takes_tiles(const GenericParams<T>& p, int maps) {
  return sizeof(T) == 4 && maps == 1 && p.pool == 0 && p.hs == p.hsv && (p.hs == 64 || p.hs == 128) &&
         ((uintptr_t)p.k_pool | (uintptr_t)p.v_pool) % 16 == 0 && (long long)p.num_pages * p.g * p.page_size < (1ll << 31);
}
int launch_tiles(const GenericParams<float>& p, int n_tokens, cudaStream_t stream) {
  return p.hs == 64 ? launch_tiled_heads<64>(p, n_tokens, stream) : launch_tiled_heads<128>(p, n_tokens, stream);
}
int launch_tiles(const GenericParams<__nv_bfloat16>&, int, cudaStream_t) { return YALIS_ERR_DTYPE; }

}  // namespace

// maps 2: two maps, hs the size of one map's queries and keys; no sink, gate or pooled blocks.
// rel null: no bias per distance.  pool 0: no pooled blocks (the pool_* arguments are not read).
YALIS_API int yalis_paged_attention_generic(const void* q, int q_stride, void* out, int out_stride,
                                            const void* k_pool, const void* v_pool, int dtype,
                                            const int32_t* positions, const int32_t* req_of_token,
                                            const int32_t* block_table, int table_width, int page_size,
                                            int num_pages, int n_tokens, int nh, int g, int hs, int hsv,
                                            float scale, int window, float softcap, int sink, float out_scale,
                                            int chunk, const float* sink_logits, const float* slopes, const void* gate,
                                            int gate_stride, int gate_per_head, const float* rel, int rel_len, int pool,
                                            const void* pk_pool, const void* pv_pool, const int32_t* pool_table,
                                            int pool_table_width, int pool_page_size, int pool_num_pages, int maps,
                                            float lambda, float diff_eps, cudaStream_t stream) {
  if (n_tokens <= 0) return YALIS_OK;
  if (maps != 1 && (maps != 2 || sink || gate || pool > 0)) return YALIS_ERR_SHAPE;
  if (hs <= 0 || hs > 32 * kMaxPerLane || hsv <= 0 || hsv > 32 * kMaxPerLane || g <= 0 || nh % g != 0 || nh > 65535)
    return YALIS_ERR_SHAPE;
  if ((rel && rel_len < 1) || pool < 0 || (pool > 0 && (window <= 0 || chunk > 0 || !pk_pool || !pv_pool || !pool_table || pool_page_size < 1)))
    return YALIS_ERR_SHAPE;
  const size_t smem = (maps * ((size_t)kWarps * hsv + 2 * kWarps) + (maps == 2 ? hsv : 0)) * sizeof(float);
  dim3 grid(n_tokens, nh);
  YALIS_DISPATCH_DTYPE(dtype, T, {
    GenericParams<T> p;
    p.q = (const T*)q; p.q_stride = q_stride; p.out = (T*)out; p.out_stride = out_stride;
    p.k_pool = (const T*)k_pool; p.v_pool = (const T*)v_pool;
    p.positions = positions; p.req_of_token = req_of_token; p.block_table = block_table;
    p.table_width = table_width; p.page_size = page_size; p.num_pages = num_pages;
    p.nh = nh; p.g = g; p.hs = hs; p.hsv = hsv;
    p.scale = scale; p.window = window; p.softcap = softcap; p.sink = sink; p.out_scale = out_scale; p.chunk = chunk;
    p.sink_logits = sink_logits; p.slopes = slopes; p.rel = rel; p.rel_len = rel_len;
    p.gate = (const T*)gate; p.gate_stride = gate_stride; p.gate_per_head = gate_per_head;
    p.pool = pool; p.pk_pool = (const T*)pk_pool; p.pv_pool = (const T*)pv_pool; p.pool_table = pool_table;
    p.pool_table_width = pool_table_width; p.pool_page_size = pool_page_size; p.pool_num_pages = pool_num_pages;
    p.lambda = lambda; p.diff_eps = diff_eps;
    if (takes_tiles(p, maps)) return launch_tiles(p, n_tokens, stream);
    return maps == 2 ? yalis_launch(paged_attention_generic_kernel<T, 2>, grid, dim3(kWarps * 32), smem, stream, p)
                     : yalis_launch(paged_attention_generic_kernel<T, 1>, grid, dim3(kWarps * 32), smem, stream, p);
  });
  return YALIS_OK;
}
