// The recurrences with one decay per head (recurrent.cu has the rules and the form that walks token by token) over long
// portions, sixteen tokens at a time.
//
// Within a chunk, with G_t the product of the decays up to token t, P_ts that of the decays after s up to t and S the state
// before the chunk, the delta rule's writes u solve a triangular system and all else is sums of products:
//
//   u_t + beta_t sum_(s<t) P_ts (k_t . k_s) u_s = beta_t (v_t - G_t S^T k_t),     u = T (v - G S^T k)
//   o_t = G_t S^T q_t + sum_(s<=t) P_ts (q_t . k_s) u_s,     S <- G_16 S + sum_s P_16,s k_s u_s^T
//
// (the plain rule: u = v; the selective form: u = beta v, and skip v beside o).  What does not depend on the state is computed
// for all chunks side by side by the first kernel: k and q in three bfloat16 parts each (as in gemm_f32_mma.cu, but unscaled:
// see below), T, P (q . k) and the decays, whose products are taken in 64 bits.  The second walks the chunks: a block has 16
// columns of a head's state, a warp 32 of its rows, as accumulators of the tensor cores in float32 (transposed, so that
// they are also the operand of the products with k and q).  All sums are float32: products of parts are summed on the tensor cores
// over 16 values at most, small ones first, and added in registers; dot products of a chunk's tokens are added in 64 bits; the state is
// scaled in registers, by a decay of two floats (one rounded factor per chunk would add up over a prompt).
// Parts do not hold everything: an infinity has no difference to its rounded self, the largest values round to one, and of values below 2^-110
// the last parts fall below bfloat16's range.  So the tokens of a block are walked again, one by one, where a read-out or a value of the new
// state is not finite or a read-out lies below 2^-80, and such values are taken from there.  (A portion whose read-outs all lie above that or are zero
// has errors of up to 2^-134 times the other operand besides: nothing beside a read-out for q and k up to 2^20.)
// A chunk starts where its request's portion starts: a long portion's results depend on how the request was cut, by rounding.
// Errors against float64 beside the walk's, read-outs / state in 1e-8 (256 tokens of 16 heads, decays drawn from the named value up to 1,
// twelve seeds): delta rule from 0: 6.4 / 4.6 (8.9 / 5.1), 0.5: 7.3 / 5.1 (9.5 / 6.1), 0.995: 12 / 10 (28 / 32); selective from 0: 2.6 / 4.3
// (5.7 / 4.4), 0.5: 2.6 / 4.5 (5.7 / 5.6); a decay a token from 0: 5.4 / 3.4 (8.2 / 3.6); constant decays from 0.5: 8.0 / 5.2 (13.8 / 13).  With
// single sums on the tensor cores and the chunk's own products first: delta rule from 0: 9.8 / 6.9, from 0.5 10.2 / 7.3.
// What bounds it: for one request the instructions of a chunk's chain, some 2,100 cycles by the delta rule: a warp alone on its
// scheduler issues one in about four cycles (clock counts between the chain's stages), so sums start from no cleared
// registers, the six products of parts are one chain, pairs of float32 operations go in one instruction, and what the chain does not
// need is left to other warps: waiting for copies, by the delta rule the products with q.  For several requests the copies of k and q,
// which the blocks of a head's columns all ask for.
// Measured (us, walk token by token -> both kernels; before copies ran up to four chunks ahead and the chain was shortened), 16
// heads of 128 x 128 (delta rule: 8 key heads; selective: 32 of 128 x 64, one), L2 flushed: delta rule 1 x 2,048 387 -> 169 (196),
// 1 x 128 30.7 -> 29.7 (28), 4 x 901 363 -> 253 (259), 32 x 128 351 -> 275 (282); plain 1 x 2,048 256 -> 116 (155), 4 x 901 223 -> 185 (208),
// 8 x 512 219 -> 192 (237); selective 1 x 2,048 260 -> 110 (144), 4 x 901 236 -> 163 (187), 16 x 256 219 -> 169.  What keeps the errors where
// the walk has them (the last products of a chunk twice, the own token last, 64-bit sums) is 6 to 12 us of 1 x 2,048.
// Not taken: eight row warps and 32 columns a block (for several requests no gain: 282 and 218 for 4 x 901), two chunks in
// shared memory, k and q copied in pieces whose order differs from block to block, the products with q by the reading warps in the
// other rules too (1 x 2,048 plain 175, 4 x 901 214: those warps become the chain).
#include "common.cuh"

namespace {

constexpr int kC = 16;              // tokens of a chunk
constexpr int kD = 128;             // rows of the state
constexpr int kWarps = 4;           // of a block that prepares
constexpr int kPart = kC * kD;      // values of one part of a chunk
// per (chunk, head): T [t][s], P (q . k) [t][s], G [t], P_16,s [s], beta [s], G_16 in two floats
constexpr int kCoefT = 0, kCoefM = 256, kCoefG = 512, kCoefW = 528, kCoefB = 544, kCoefL = 560, kCoef = 564;

struct ChunkParams {
  const float* q; int q_stride;
  const float* k; int k_stride;
  const float* v; int v_stride;
  const float* decay; int decay_kind;           // 0: [heads], 1: [N, heads]
  const float* beta;                            // RULE 1, 3: [N, heads]
  const float* skip;                            // RULE 3: [heads] or null
  float* state; size_t slot_stride;
  float* out; int out_stride;
  const int32_t* q_start; const int32_t* slots;
  int heads, kv_heads, vdim, shortest, longest; // portions of other lengths are left out
  int from, room;                               // the places of chunks that this launch takes: from ... from + room - 1
  __nv_bfloat16* parts;                         // [chunk][kv_head][k, q][3][16][128], 16-byte pieces swapped within rows
  float* coef;                                  // [chunk][head][kCoef]
  int32_t* error;
};

// The tokens of request r that this launch takes, and where its chunks lie: no two requests' chunks share a place.
struct Portion {
  int start, len;                               // len 0: none
  int first;
};
__device__ __forceinline__ Portion portion_of(const ChunkParams& p, int r) {
  const int start = p.q_start[r], len = p.q_start[r + 1] - start, place = start / kC + r - p.from;      // of its first chunk
  const int skip = max(0, -place) * kC;                                                                // taken before
  Portion o = {start + skip, min(len - skip, (p.room - max(0, place)) * kC), max(0, place)};
  if (len < p.shortest || len > p.longest || o.len < 0) o.len = 0;
  return o;
}

__device__ __forceinline__ uint32_t two_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same from zero: no registers are cleared first.
__device__ __forceinline__ void mma0(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// Eight tokens' products: from zero, and on top of another sum, which stays.
__device__ __forceinline__ void half0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(b), "f"(0.f));
}
__device__ __forceinline__ void half_on(float (&d)[4], const float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(b), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// The parts of a product's operands, small products first: (2, 0), (0, 2), (1, 1), (1, 0), (0, 1), (0, 0).
__device__ __forceinline__ constexpr int first_part(int o) { return o == 0 ? 2 : o == 2 || o == 3 ? 1 : 0; }
__device__ __forceinline__ constexpr int second_part(int o) { return o == 1 ? 2 : o == 2 || o == 4 ? 1 : 0; }
// Two float32 operations in one instruction, each rounded as the single one is.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
  return *reinterpret_cast<float2*>(&d);
}
// Two values as three pairs of bfloat16 values whose sums they are.
__device__ __forceinline__ void part2(float a, float b, uint32_t (&o)[3]) {
  float2 x = make_float2(a, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[i] = two_bf16(x.x, x.y);
    if (i < 2) x = fma2(make_float2(__uint_as_float(o[i] << 16), __uint_as_float(o[i] & 0xffff0000u)), make_float2(-1.f, -1.f), x);
  }
}
constexpr uint32_t kSpinLimit = 1u << 22;      // polls of a wait before the block gives up
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy_bulk(void* to, const void* from, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(to)), "l"(from), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool copies_there(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void copy16(void* to, const void* from, bool there) {      // zeros where there is nothing
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(to)), "l"(from), "r"(there ? 16 : 0) : "memory");
}

// A block per chunk, key head and request: parts of k and q, the dot products, then a warp per head of the group.
template <int RULE>
__global__ void __launch_bounds__(kWarps * 32) chunk_prepare_kernel(const ChunkParams p) {
  __shared__ __align__(128) __nv_bfloat16 ps_s[6 * kPart];                     // parts of k, then of q, as they go to memory
  __shared__ float kk[kC * kC], qk[kC * kC], ratio[kWarps][kC * kC];
  pdl_launch_dependents();
  pdl_wait();
  const int req = blockIdx.z, kvh = blockIdx.y;
  const Portion portion = portion_of(p, req);
  const int t0 = portion.start + blockIdx.x * kC, valid = min(kC, portion.len - (int)blockIdx.x * kC);
  if (valid <= 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t chunk = portion.first + (int)blockIdx.x;
  __nv_bfloat16* parts = p.parts + (chunk * p.kv_heads + kvh) * (6 * kPart);
  for (int e = tid; e < 2 * kC * (kD / 8); e += kWarps * 32) {
    const int which = e / (kC * (kD / 8)), t = e / (kD / 8) % kC, c = e % (kD / 8);       // k, then q; a piece of eight values
    float4 x[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    if (t < valid) {
      const float* from = (which ? p.q + (size_t)(t0 + t) * p.q_stride : p.k + (size_t)(t0 + t) * p.k_stride) + kvh * kD + c * 8;
      x[0] = load4_f32(from);
      x[1] = load4_f32(from + 4);
    }
    uint32_t o[4][3];
    part2(x[0].x, x[0].y, o[0]); part2(x[0].z, x[0].w, o[1]); part2(x[1].x, x[1].y, o[2]); part2(x[1].z, x[1].w, o[3]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int at = (which * 3 + i) * kPart + t * kD + ((c ^ (t & 7)) * 8);
      const uint4 piece = make_uint4(o[0][i], o[1][i], o[2][i], o[3][i]);
      *reinterpret_cast<uint4*>(parts + at) = piece;
      *reinterpret_cast<uint4*>(ps_s + at) = piece;
    }
  }
  __syncthreads();
  if (RULE == 1 || warp < 2) {
    // q k by two warps, k k by two, eight of the second operand's tokens each: the products of the first parts, 16 values at a time, are added in
    // 64 bits (a decay of a half leaves of a read-out little but these products), the five small ones in one chain on the tensor cores
    const bool qk_here = warp < 2;
    const int s0 = (warp & 1) * 8;
    const uint32_t as = smem_u32(ps_s) + (qk_here ? 3 * kPart * 2 : 0) + (lane & 15) * (kD * 2);
    const uint32_t bs = smem_u32(ps_s) + (s0 + (lane & 7)) * (kD * 2);
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    float small[2][4];
#pragma unroll
    for (int j = 0; j < kD / 32; ++j) {                            // 32 values
      uint32_t fa[3][2][4], fb[3][4];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        ldmatrix4(fb[i], bs + i * kPart * 2 + (((4 * j + (lane >> 3)) ^ (lane & 7)) << 4));
#pragma unroll
        for (int n = 0; n < 2; ++n) ldmatrix4(fa[i][n], as + i * kPart * 2 + (((4 * j + 2 * n + (lane >> 4)) ^ (lane & 7)) << 4));
      }
      float large[2][4];
#pragma unroll
      for (int o = 0; o < 6; ++o)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const uint32_t(&b)[4] = fb[second_part(o)];
          if (o == 0 && j == 0) mma0(small[n], fa[first_part(o)][n], b[2 * n], b[2 * n + 1]);
          else if (o < 5) mma(small[n], fa[first_part(o)][n], b[2 * n], b[2 * n + 1]);
          else mma0(large[n], fa[first_part(o)][n], b[2 * n], b[2 * n + 1]);
        }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] += (double)large[n][e];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int t = (lane >> 2) + 8 * (e >> 1), s = s0 + 2 * (lane & 3) + (e & 1);
      (qk_here ? qk : kk)[t * kC + s] = (float)(sum[e] + (double)(small[0][e] + small[1][e]));
    }
  }
  __syncthreads();
  const int per = p.heads / p.kv_heads, s = lane & 15;
  float* ps = ratio[warp];
  for (int j = warp; j < per; j += kWarps) {
    const int h = kvh * per + j;
    float* coef = p.coef + (chunk * p.heads + h) * kCoef;
    const float g = s >= valid ? 1.f : p.decay_kind == 0 ? p.decay[h] : p.decay[(size_t)(t0 + s) * p.heads + h];
    const float beta = s >= valid ? 0.f : RULE == 0 ? 1.f : p.beta[(size_t)(t0 + s) * p.heads + h];
    // lane s (and its double s + 16): the products of the decays after s, and of all up to s
    double after = 1.0, upto = 1.0;
#pragma unroll
    for (int t = 0; t < kC; ++t) {
      const double gt = (double)__shfl_sync(0xffffffffu, g, t);
      if (t <= s) upto *= gt;
      else after *= gt;
      if (lane < kC) ps[t * kC + s] = t < s ? 0.f : (float)after;
    }
    __syncwarp();
    const double total = __shfl_sync(0xffffffffu, upto, kC - 1);
    if (lane < kC) {
      coef[kCoefG + s] = (float)upto;
      coef[kCoefW + s] = (float)after;
      coef[kCoefB + s] = beta;
      if (s == 0) {
        coef[kCoefL] = (float)total;
        coef[kCoefL + 1] = (float)(total - (double)(float)total);
      }
    }
    float T[kC];                                // column s of T
#pragma unroll
    for (int t = 0; t < kC; ++t) {
      const float bt = __shfl_sync(0xffffffffu, beta, t);
      if constexpr (RULE == 1) {
        float x = t == s ? 1.f : 0.f;
#pragma unroll
        for (int r = 0; r < t; ++r) {
          const float l = bt * (ps[t * kC + r] * kk[t * kC + r]);
          if (r >= s) x = __fmaf_rn(-l, T[r], x);
        }
        T[t] = t < s ? 0.f : x;
      }
      if (lane < kC) {
        if constexpr (RULE == 1) coef[kCoefT + t * kC + s] = T[t] * beta;
        coef[kCoefM + t * kC + s] = t < s ? 0.f : ps[t * kC + s] * qk[t * kC + s];
      }
    }
    __syncwarp();
  }
}

// A block per 16 columns of a head and request.  Four warps walk: each has 32 rows of the state.  Four
// more form the read-outs of a chunk while those are at the next, from the state's parts that the walking warps leave
// them, one fetches.  All meet once per chunk, when its u are there.  Shared memory: stages of (k and q in parts, coefficients, v
// [t][column]), the state in parts as operands [row warp][part][tile][lane], the row warps' shares of S^T q [row warp][t][column] and of S^T k,
// u [buffer][column][t], v - G S^T k [column][t], u P_16 in parts [buffer][part][t][column].
constexpr int kV = 16, kRowWarps = 4;                                   // columns of a block, row warps
constexpr int kWalk = kRowWarps * 32, kAll = 2 * kWalk + 32;            // threads that walk (as many form read-outs), of the block
constexpr int kRowTiles = kD / (16 * kRowWarps), kStateParts = kRowWarps * 3 * kRowTiles * 32;      // a warp's rows, sixteen at a time; 16-byte pieces
constexpr int kLdT = kC + 4, kShares = kV * kLdT;                       // floats between a column's tokens and the next one's
constexpr int kStage = (6 * kPart * 2 + kCoef * 4 + kC * kV * 4 + 127) / 128 * 128;
template <int RULE, int STAGES>
constexpr size_t walk_smem() {
  return STAGES * kStage + (RULE == 1 ? kStateParts * 16 : 0) + (2 * kRowWarps * kShares + (RULE == 1 ? 3 : 2) * kV * kLdT) * sizeof(float) + 2 * 3 * kC * kV * 2 + STAGES * 8 + 16;
}
template <int ID, int N>
__device__ __forceinline__ void meet() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory"); }
constexpr int kMeetAll = 0, kMeetWalk = 1, kMeetRead = 2, kMeetTaken = 3, kMeetEnd = 4;
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }
__device__ __forceinline__ bool sure(float x) { return finite(x) && fabsf(x) >= 8.3e-25f; }

// A row of a chunk's coefficients.
__device__ __forceinline__ void load_row(const float* m, float (&c)[kC]) {
#pragma unroll
  for (int s = 0; s < kC; s += 4) {
    const float4 x = load4_f32(m + s);
    c[s] = x.x; c[s + 1] = x.y; c[s + 2] = x.z; c[s + 3] = x.w;
  }
}
// Sum over the tokens before t of a coefficient times a column's value: later ones take no part, be they infinite.  (The token's own
// product, the largest where decays are fast, is added last.)
__device__ __forceinline__ float before(const float (&c)[kC], const float (&y)[kC], int t) {
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int s = 0; s < kC; s += 2) {
    if (s < t) a = __fmaf_rn(c[s], y[s], a);
    if (s + 1 < t) b = __fmaf_rn(c[s + 1], y[s + 1], b);
  }
  return a + b;
}

// A warp's rows of the state, transposed and in parts, times 16 tokens' vectors in parts at `from`: its share of S^T k or S^T q.
__device__ __forceinline__ void read_state(const uint32_t (&fs)[3][kRowTiles][4], uint32_t from, float* to, int warp, int lane) {
  constexpr int NJ = kRowTiles;
  const int lt = (lane & 7) + (lane >> 4) * 8;                 // ldmatrix: tokens 0-7 by two pieces, tokens 8-15 by two
  uint32_t f[3][NJ][4];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
      ldmatrix4(f[i][j], from + i * kPart * 2 + lt * (kD * 2) + (((2 * NJ * warp + 2 * j + ((lane >> 3) & 1)) ^ (lt & 7)) << 4));
  float sum[NJ][2][4];
#pragma unroll
  for (int o = 0; o < 6; ++o)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const uint32_t(&b)[4] = f[second_part(o)][j];
        if (o == 0) mma0(sum[j][n], fs[first_part(o)][j], b[2 * n], b[2 * n + 1]);
        else mma(sum[j][n], fs[first_part(o)][j], b[2 * n], b[2 * n + 1]);
      }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {                              // columns lane / 4 and 8 further; two tokens
      float2 y = make_float2(sum[0][n][2 * e], sum[0][n][2 * e + 1]);
#pragma unroll
      for (int j = 1; j < NJ; ++j) {
        y.x += sum[j][n][2 * e];
        y.y += sum[j][n][2 * e + 1];
      }
      *reinterpret_cast<float2*>(to + ((lane >> 2) + 8 * e) * kLdT + 8 * n + 2 * (lane & 3)) = y;
    }
}

// The tokens of a portion one by one, for a column c whose state before it is W, eight lanes a column and sixteen rows a lane: takes the place of
// what the chunks' form did not hold.
template <int RULE>
__device__ __noinline__ void walk_again(const ChunkParams& p, float (&W)[kD / 8], float* column, int start, int len, int h, int kvh, int c) {
  const int lane = threadIdx.x % 8;
  const bool mine = c < p.vdim;
  const float skip = (RULE == 3 && p.skip) ? p.skip[h] : 0.f;
#pragma unroll 1
  for (int n = start; n < start + len; ++n) {
    const float* k = p.k + (size_t)n * p.k_stride + kvh * kD + lane * 4;
    const float* q = p.q + (size_t)n * p.q_stride + kvh * kD + lane * 4;
    const float g = p.decay_kind == 0 ? p.decay[h] : p.decay[(size_t)n * p.heads + h];
    const float v = mine ? p.v[(size_t)n * p.v_stride + (size_t)h * p.vdim + c] : 0.f;
    float u = v, dot = 0.f, read = 0.f;
#pragma unroll
    for (int i = 0; i < kD / 8; ++i) {
      W[i] *= g;
      dot = __fmaf_rn(k[i / 4 * 32 + i % 4], W[i], dot);
    }
    if constexpr (RULE == 1) {
      for (int o = 1; o < 8; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      u = v - dot;
    }
    if constexpr (RULE != 0) u *= p.beta[(size_t)n * p.heads + h];
#pragma unroll
    for (int i = 0; i < kD / 8; ++i) {
      W[i] = __fmaf_rn(k[i / 4 * 32 + i % 4], u, W[i]);
      read = __fmaf_rn(q[i / 4 * 32 + i % 4], W[i], read);
    }
    for (int o = 1; o < 8; o <<= 1) read += __shfl_xor_sync(0xffffffffu, read, o);
    if constexpr (RULE == 3) read = __fmaf_rn(skip, v, read);
    if (mine && lane == 0) {
      float* to = p.out + (size_t)n * p.out_stride + (size_t)h * p.vdim + c;
      if (!sure(*to)) *to = read;
    }
  }
#pragma unroll
  for (int i = 0; i < kD / 8; ++i)
    if (mine && !sure(column[i / 4 * 32 + i % 4])) column[i / 4 * 32 + i % 4] = W[i];
}

template <int RULE, int STAGES>
__global__ void __launch_bounds__(kAll, STAGES == 3 ? 2 : 1) chunk_walk_kernel(const __grid_constant__ ChunkParams p) {
  constexpr int NJ = kRowTiles;
  constexpr bool EARLY = STAGES > 3;                                  // who waits for a chunk's copies: the warp that fetches, or the walking ones
  extern __shared__ __align__(128) unsigned char smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int req = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * kV;
  Portion portion = portion_of(p, req);
  if (portion.len <= 0) return;
  // (that there is a first chunk is kept from the compiler: without the check in front of its loops it orders a chunk's instructions
  // otherwise, 179 us in place of 165 for the delta rule's 1 x 2,048)
  asm volatile("" : "+r"(portion.start), "+r"(portion.len), "+r"(portion.first));
  const int start = portion.start, len = portion.len;
  const int role = threadIdx.x / kWalk, tid = threadIdx.x % kWalk;      // role 0 walks, 1 reads, 2 fetches
  const int lane = tid & 31, kvh = h / (p.heads / p.kv_heads);
  const int chunks = (len + kC - 1) / kC;
  const size_t first = portion.first;
  uint4* state_parts = reinterpret_cast<uint4*>(smem + STAGES * kStage);
  float* shares_q = reinterpret_cast<float*>(state_parts + (RULE == 1 ? kStateParts : 0));      // RULE 1: one buffer
  float* shares_k = shares_q + kRowWarps * kShares;                                             // RULE 1
  float* us = shares_q + 2 * kRowWarps * kShares;
  float* rest = us + 2 * kV * kLdT;
  __nv_bfloat16* ups = reinterpret_cast<__nv_bfloat16*>(rest + (RULE == 1 ? kV * kLdT : 0));
  uint64_t* there = reinterpret_cast<uint64_t*>(ups + 2 * 3 * kC * kV);
  volatile int* lost = reinterpret_cast<volatile int*>(there + STAGES);      // a wait ran out
  volatile int* again = lost + 1;                                            // something was not held
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 33;" ::"r"(smem_u32(&there[s])));      // lane 0 and every lane's copies
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *lost = 0;
    *again = 0;
  }
  __syncthreads();
  auto coef_of = [&](int c) { return reinterpret_cast<const float*>(smem + c % STAGES * kStage + 6 * kPart * 2); };
  // A wait that runs out ends neither the copies nor the meetings; what is formed then is dropped at the end.
  auto await = [&](int c) {
    if (c < chunks && !copies_there(&there[c % STAGES], (c / STAGES) & 1)) *lost = 1;
    __syncwarp();
  };

  if (role == 2) {
    // One copy each for the parts and the coefficients; the values 16 bytes at a time, zeros behind the portion's end and the last
    // column (a bulk copy for every row of 64 bytes took longer than all else).
    auto fetch = [&](int c) {
      if (c >= chunks) return;
      unsigned char* to = smem + c % STAGES * kStage;
      uint64_t* bar = &there[c % STAGES];
      if (lane == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(6 * kPart * 2 + kCoef * 4) : "memory");
        copy_bulk(to, p.parts + ((first + c) * p.kv_heads + kvh) * (6 * kPart), 6 * kPart * 2, bar);
        copy_bulk(to + 6 * kPart * 2, p.coef + ((first + c) * p.heads + h) * kCoef, kCoef * 4, bar);
      }
      __syncwarp();
#pragma unroll
      for (int e = lane; e < kC * kV / 4; e += 32) {
        const int t = e / (kV / 4), d = e % (kV / 4) * 4;
        const bool is = c * kC + t < len && j0 + d < p.vdim;
        copy16(to + 6 * kPart * 2 + kCoef * 4 + e * 16, is ? p.v + (size_t)(start + c * kC + t) * p.v_stride + (size_t)h * p.vdim + j0 + d : p.v, is);
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
    };
    for (int c = 0; c < STAGES - 1; ++c) fetch(c);
    // EARLY: it waits for a chunk's copies before it joins the meeting of the chunk before: past that they are there for all.
    if constexpr (EARLY) await(0);
    meet<kMeetAll, kAll>();
    for (int c = 0; c < chunks; ++c) {
      if constexpr (EARLY) await(c + 1);
      meet<kMeetAll, kAll>();                                   // everyone is done with the chunk before
      fetch(c + STAGES - 1);
    }
    // (all copies end before the block does, also those that a wait gave up on)
    for (int c = max(0, chunks - STAGES); c < chunks; ++c) copies_there(&there[c % STAGES], (c / STAGES) & 1);
    __syncwarp();
    if (lane == 0 && *lost) atomicOr(p.error, YALIS_FLAG_WAIT_RECURRENCE);
    return;
  }

  if (role == 1) {
    // read-outs: a thread has CPT columns of a token
    constexpr int CPT = kC * kV / kWalk;
    const int rt = tid, t = rt / (kV / CPT), v0 = rt % (kV / CPT) * CPT;
    const float skip = (RULE == 3 && p.skip) ? p.skip[h] : 0.f;
    bool all = true;                                          // held by the parts
    meet<kMeetAll, kAll>();
    for (int c = 0; c < chunks; ++c) {
      meet<kMeetAll, kAll>();
      const float* shares = shares_q + (RULE == 1 ? 0 : (c & 1) * kRowWarps * kShares);
      if constexpr (RULE == 1) {
        const int rw = rt / 32;
        uint32_t fs[3][kRowTiles][4];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < kRowTiles; ++j) {
            const uint4 x = state_parts[((rw * 3 + i) * kRowTiles + j) * 32 + lane];
            fs[i][j][0] = x.x; fs[i][j][1] = x.y; fs[i][j][2] = x.z; fs[i][j][3] = x.w;
          }
        if (c + 1 < chunks) asm volatile("bar.arrive %0, %1;" ::"n"(kMeetTaken), "n"(2 * kWalk) : "memory");
        read_state(fs, smem_u32(smem + c % STAGES * kStage) + 3 * kPart * 2, shares_q + rw * kShares, rw, lane);
        meet<kMeetRead, kWalk>();
      }
      const float* coef = coef_of(c);
      const float g = coef[kCoefG + t], own = coef[kCoefM + t * kC + t];
      float o[CPT], row_t[kC];
      load_row(coef + kCoefM + t * kC, row_t);
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        float read = 0.f;
#pragma unroll
        for (int w = 0; w < kRowWarps; ++w) read += shares[w * kShares + (v0 + i) * kLdT + t];
        float y[kC];
        load_row(us + ((c & 1) * kV + v0 + i) * kLdT, y);
        o[i] = __fmaf_rn(own, us[((c & 1) * kV + v0 + i) * kLdT + t], __fmaf_rn(g, read, before(row_t, y, t)));
        if constexpr (RULE == 3) o[i] = __fmaf_rn(skip, coef[kCoef + t * kV + v0 + i], o[i]);
      }
      if (c * kC + t < len && j0 + v0 < p.vdim) {
        float* to = p.out + (size_t)(start + c * kC + t) * p.out_stride + (size_t)h * p.vdim + j0 + v0;
#pragma unroll
        for (int i = 0; i < CPT; i += 2) {
          *reinterpret_cast<float2*>(to + i) = make_float2(o[i], o[i + 1]);
          all = all && (sure(o[i]) || o[i] == 0.f) && (sure(o[i + 1]) || o[i + 1] == 0.f);
        }
      }
    }
    if (!all) *again = 1;
    meet<kMeetEnd, 2 * kWalk>();
    return;
  }

  const int warp = tid / 32;
  // the state, transposed: a lane's columns are col and col + 8, its rows row + 8 n and the one after
  const int col = lane >> 2, row = 16 * NJ * warp + 2 * (lane & 3);
  float* sp = p.state + (size_t)p.slots[req] * p.slot_stride + ((size_t)h * p.vdim + j0 + col) * kD + row;
  float2 S[2 * NJ][2];
#pragma unroll
  for (int n = 0; n < 2 * NJ; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      S[n][e] = j0 + col + 8 * e < p.vdim ? *reinterpret_cast<const float2*>(sp + (size_t)e * 8 * kD + 8 * n) : make_float2(0.f, 0.f);
    }
  static_assert(kC * kV == 2 * kWalk, "two tokens of a column a thread");
  const int v = tid % kV, t = tid / kV * 2;                     // a thread's column, and its first token, in the small sums
  const int tt = (lane & 7) + ((lane >> 3) & 1) * 8;           // ldmatrix: two halves of the tokens by a piece, then by the next

  meet<kMeetAll, kAll>();                                             // the first chunk is there
  for (int c = 0; c < chunks; ++c) {
    // the state in parts: for S^T k here and S^T q by the reading warps, or for S^T q
    uint32_t fs[3][NJ][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t o[3];
        part2(S[2 * j + (i >> 1)][i & 1].x, S[2 * j + (i >> 1)][i & 1].y, o);
        fs[0][j][i] = o[0]; fs[1][j][i] = o[1]; fs[2][j][i] = o[2];
      }
    const uint32_t ks = smem_u32(smem + c % STAGES * kStage), qs = ks + 3 * kPart * 2;
    const float* coef = coef_of(c);
    const float* vs = coef + kCoef;
    if constexpr (RULE == 1) {
      if (c > 0) meet<kMeetTaken, 2 * kWalk>();                 // the reading warps have the last chunk's
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          state_parts[((warp * 3 + i) * NJ + j) * 32 + lane] = make_uint4(fs[i][j][0], fs[i][j][1], fs[i][j][2], fs[i][j][3]);
      if constexpr (!EARLY) await(c);
      read_state(fs, ks, shares_k + warp * kShares, warp, lane);
    } else {
      if constexpr (!EARLY) await(c);
      read_state(fs, qs, shares_q + ((c & 1) * kRowWarps + warp) * kShares, warp, lane);
    }
    // the state's products' operands that do not wait for the others
    uint32_t fk[3][NJ][4];
    auto load_k = [&]() {
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          ldmatrix4_trans(fk[i][j], ks + i * kPart * 2 + tt * (kD * 2) + (((2 * NJ * warp + 2 * j + (lane >> 4)) ^ (tt & 7)) << 4));
    };
    const float2 w = *reinterpret_cast<const float2*>(coef + kCoefW + t), x = make_float2(vs[t * kV + v], vs[(t + 1) * kV + v]);
    float2 u;
    if constexpr (RULE == 1) {
      const float2 g = *reinterpret_cast<const float2*>(coef + kCoefG + t);
      float row[2][kC];
      load_row(coef + kCoefT + t * kC, row[0]);
      load_row(coef + kCoefT + (t + 1) * kC, row[1]);
      meet<kMeetWalk, kWalk>();
      float2 a = make_float2(0.f, 0.f);
#pragma unroll
      for (int r = 0; r < kRowWarps; ++r) {
        const float2 y = *reinterpret_cast<const float2*>(shares_k + r * kShares + v * kLdT + t);
        a.x += y.x;
        a.y += y.y;
      }
      const float2 own = make_float2(coef[kCoefT + t * kC + t], coef[kCoefT + (t + 1) * kC + t + 1]);
      const float2 left = make_float2(__fmaf_rn(-g.x, a.x, x.x), __fmaf_rn(-g.y, a.y, x.y));
      *reinterpret_cast<float2*>(rest + v * kLdT + t) = left;
      meet<kMeetWalk, kWalk>();
      load_k();
      float y[kC];
      load_row(rest + v * kLdT, y);
      u = make_float2(__fmaf_rn(own.x, left.x, before(row[0], y, t)), __fmaf_rn(own.y, left.y, before(row[1], y, t + 1)));
    } else {                                                   // u is known at once
      load_k();
      const float2 b = *reinterpret_cast<const float2*>(coef + kCoefB + t);
      u = make_float2(b.x * x.x, b.y * x.y);
    }
    {                                                          // u, and u times the decays after it in parts
      uint32_t o[3];
      part2(w.x * u.x, w.y * u.y, o);
      *reinterpret_cast<float2*>(us + ((c & 1) * kV + v) * kLdT + t) = u;
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(ups + (((c & 1) * 3 + i) * kV + v) * kC + t) = o[i];
    }
    const float hi = coef[kCoefL], lo = coef[kCoefL + 1];
    meet<kMeetAll, kAll>();
    // the state: u times the decays after its token, times k
    uint32_t fu[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)                                // ldmatrix: two halves of the columns by eight tokens, then by the next
      ldmatrix4(fu[i], smem_u32(ups + (((c & 1) * 3 + i) * kV + tt) * kC + (lane >> 4) * 8));
    // The tensor cores cut off the last bits of a sum and of every small term beside a large one.  The first parts' products of the later
    // eight tokens, the largest where decays are fast, are formed twice: negative, and positive on top of that, which leaves what was
    // cut off.  The small products join that, then the earlier tokens' first parts; all this joins the old state before the negative sum is
    // taken off it.
    float less[NJ][2][4], more[NJ][2][4];
#pragma unroll
    for (int o = -2; o < 6; ++o)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const uint32_t(&b)[4] = fk[o < 0 ? 0 : second_part(o)][j];
          if (o == -2) half0(less[j][n], fu[0][2] ^ 0x80008000u, fu[0][3] ^ 0x80008000u, b[2 * n + 1]);
          else if (o == -1) half_on(more[j][n], less[j][n], fu[0][2], fu[0][3], b[2 * n + 1]);
          else if (o < 5) mma(more[j][n], fu[first_part(o)], b[2 * n], b[2 * n + 1]);
          else half_on(more[j][n], more[j][n], fu[0][0], fu[0][1], b[2 * n]);
        }
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float2& x = S[2 * j + n][e];
          const float2 y = fma2(make_float2(hi, hi), x, fma2(make_float2(lo, lo), x, make_float2(more[j][n][2 * e], more[j][n][2 * e + 1])));
          x = fma2(make_float2(less[j][n][2 * e], less[j][n][2 * e + 1]), make_float2(-1.f, -1.f), y);
        }
  }
  bool whole = true;
#pragma unroll
  for (int n = 0; n < 2 * NJ; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) whole = whole && finite(S[n][e].x) && finite(S[n][e].y);
  if (!whole) *again = 1;
  meet<kMeetEnd, 2 * kWalk>();
  if (*lost) return;
  auto store = [&]() {
#pragma unroll
    for (int n = 0; n < 2 * NJ; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (j0 + col + 8 * e < p.vdim) *reinterpret_cast<float2*>(sp + (size_t)e * 8 * kD + 8 * n) = S[n][e];
  };
  if (!*again) {
    store();
    return;
  }
  float W[kD / 8];                                             // the state before the portion, eight lanes a column
  const int c = j0 + tid / 8;
  float* column = p.state + (size_t)p.slots[req] * p.slot_stride + ((size_t)h * p.vdim + c) * kD + tid % 8 * 4;
#pragma unroll
  for (int i = 0; i < kD / 8; ++i) W[i] = c < p.vdim ? column[i / 4 * 32 + i % 4] : 0.f;
  meet<kMeetWalk, kWalk>();
  store();
  meet<kMeetWalk, kWalk>();
  walk_again<RULE>(p, W, column, start, len, h, kvh, c);
}

template <int RULE, int STAGES>
int launch_walk(const ChunkParams& p, int n_requests, cudaStream_t stream) {
  constexpr size_t smem = walk_smem<RULE, STAGES>();
  if (cudaFuncSetAttribute(chunk_walk_kernel<RULE, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return YALIS_ERR_LAUNCH;
  return yalis_launch_after(chunk_walk_kernel<RULE, STAGES>, dim3((p.vdim + kV - 1) / kV, p.heads, n_requests), dim3(kAll), smem, stream, p);
}

// Chunks in shared memory: three leave room for two blocks on an SM, which cover each other's copies; where there is a block an SM at
// most, five.
template <int RULE>
int launch_chunks(ChunkParams p, int n_requests, int places, cudaStream_t stream) {
  const long long blocks = (long long)((p.vdim + kV - 1) / kV) * p.heads * n_requests;
  const dim3 grid(min((p.longest + kC - 1) / kC, p.room), p.kv_heads, n_requests);
  for (p.from = 0; p.from < places; p.from += p.room) {
    int st = yalis_launch(chunk_prepare_kernel<RULE>, grid, dim3(kWarps * 32), 0, stream, p);
    if (st == YALIS_OK) st = blocks <= yalis_sm_count() ? launch_walk<RULE, 5>(p, n_requests, stream) : launch_walk<RULE, 3>(p, n_requests, stream);
    if (st != YALIS_OK) return st;
  }
  return YALIS_OK;
}

}  // namespace

// float32 values per (chunk, head) of `coef`; a chunk has 6 x 16 x 128 bfloat16 values per key head in `parts`.  places: of chunks in the
// step, n_tokens / 16 + n_requests + 1; room: chunks that parts and coef hold.  Where there are more places the step is taken in
// several launches, to the same bits: between two of them the state is the slots'.
YALIS_API int yalis_state_chunks_coefficients() { return kCoef; }

// The portions of `shortest` to `longest` tokens of a step, the others are left alone.  dim 128, vdim a multiple of four, rows on
// 16-byte boundaries; rule 0: plain, 1: delta, 3: selective; decay_kind 0 or 1 as in yalis_state_scan.
YALIS_API int yalis_state_chunks(const float* q, int q_stride, const float* k, int k_stride, const float* v, int v_stride,
                                 const float* decay, int decay_kind, const float* beta, const float* skip, float* state,
                                 int64_t slot_stride, float* out, int out_stride, const int32_t* q_start, const int32_t* slots,
                                 int n_requests, int heads, int kv_heads, int dim, int vdim, int rule, int longest, int shortest,
                                 int places, int room, void* parts, void* coef, int32_t* error, cudaStream_t stream) {
  if (n_requests <= 0 || longest <= 0) return YALIS_OK;
  if (places <= 0 || places > (1 << 30) || room <= 0) return YALIS_ERR_SHAPE;
  if (dim != kD || vdim <= 0 || vdim % 4 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || heads > 65535 || n_requests > 65535)
    return YALIS_ERR_SHAPE;
  if (decay_kind < 0 || decay_kind > 1 || !decay || (rule != 0 && rule != 1 && rule != 3) || (rule && !beta)) return YALIS_ERR_SHAPE;
  if (((q_stride | k_stride | v_stride | out_stride) & 3) || (slot_stride & 3) ||
      (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state | (uintptr_t)out | (uintptr_t)parts | (uintptr_t)coef) & 15))
    return YALIS_ERR_ALIGN;
  const ChunkParams p = {q, q_stride, k, k_stride, v, v_stride, decay, decay_kind, beta, skip, state, (size_t)slot_stride, out, out_stride,
                         q_start, slots, heads, kv_heads, vdim, shortest, longest, 0, room < places ? room : places, (__nv_bfloat16*)parts, (float*)coef, error};
  if (rule == 0) return launch_chunks<0>(p, n_requests, places, stream);
  if (rule == 1) return launch_chunks<1>(p, n_requests, places, stream);
  return launch_chunks<3>(p, n_requests, places, stream);
}
