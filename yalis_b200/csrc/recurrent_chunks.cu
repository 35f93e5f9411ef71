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
// for all chunks side by side by the first kernel: k and q in three bfloat16 parts each (nothing of a float32 value is lost; see
// gemm_f32_mma.cu), T, P (q . k) and the decays, whose products are taken in 64 bits.  The second walks the chunks: a block has 16
// columns of a head's state, a warp 32 of its rows, as accumulators of the tensor cores in float32 (transposed, so that
// they are also the operand of the products with k and q).  All sums are float32: products of parts are summed on the tensor cores
// over 16 values at most, small ones first, and added in registers; the state is scaled in registers, by a decay of two floats (one
// rounded factor per chunk would add up over a prompt).
// A chunk starts where its request's portion starts: a long portion's results depend on how the request was cut, by rounding.
// Errors against float64 beside the walk's (2,048 tokens, slow decays, read-outs / state): constant decay 1.9e-7 / 7.7e-7 (2.0e-7 /
// 9.4e-7), delta rule 1.4e-7 / 3.6e-7 (1.1e-7 / 3.6e-7), selective 0.7e-7 / 2.2e-7 (1.1e-7 / 5.0e-7).
// What bounds it: for one request the chain of a chunk, some 2,000 cycles: parts of the state, two products, two small sums, the
// state's products; for several the copies of k and q, which the blocks of a head's columns all ask for (3 TB/s).
// Measured (us, walk token by token -> both kernels), 16 heads of 128 x 128 (selective: 32 of 128 x 64): delta rule 1 x 2,048
// 382 -> 186, 1 x 128 26 -> 24, 4 x 901 357 -> 246, 32 x 128 346 -> 270; plain 1 x 2,048 251 -> 145, 4 x 901 217 -> 194,
// 8 x 512 214 -> 225, 32 x 128 195 -> 224; selective 1 x 2,048 256 -> 135, 32 x 128 211 -> 207.
// Not taken: eight row warps (1 x 2,048: 179, 4 x 901: 321), 32 columns a block (304 and 294), two chunks in shared memory (253 and 304),
// four (no gain), k and q copied in pieces whose order differs from block to block (236).
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
  int heads, kv_heads, vdim, shortest;          // portions below `shortest` tokens are left out
  __nv_bfloat16* parts;                         // [chunk][kv_head][k, q][3][16][128], 16-byte pieces swapped within rows
  float* coef;                                  // [chunk][head][kCoef]
  int32_t* error;
};

// The chunks of request r begin here: no two requests' chunks share a place.
__device__ __forceinline__ int first_chunk(int start, int r) { return start / kC + r; }

__device__ __forceinline__ uint32_t two_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// Two values as three pairs of bfloat16 values whose sums they are.
__device__ __forceinline__ void part2(float a, float b, uint32_t (&o)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[i] = two_bf16(a, b);
    if (i < 2) {
      a -= __uint_as_float(o[i] << 16);
      b -= __uint_as_float(o[i] & 0xffff0000u);
    }
  }
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
  constexpr int LD = kD + 4;
  __shared__ __align__(16) float ks[kC * LD];
  __shared__ __align__(16) float qs[kC * LD];
  __shared__ float kk[kC * kC], qk[kC * kC], ratio[kWarps][kC * kC];
  pdl_launch_dependents();
  pdl_wait();
  const int req = blockIdx.z, kvh = blockIdx.y, start = p.q_start[req], len = p.q_start[req + 1] - start;
  const int t0 = start + blockIdx.x * kC, valid = min(kC, start + len - t0);
  if (len < p.shortest || valid <= 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t chunk = first_chunk(start, req) + blockIdx.x;
  __nv_bfloat16* parts = p.parts + (chunk * p.kv_heads + kvh) * (6 * kPart);
  for (int e = tid; e < 2 * kC * (kD / 8); e += kWarps * 32) {
    const int which = e / (kC * (kD / 8)), t = e / (kD / 8) % kC, c = e % (kD / 8);       // k, then q; a piece of eight values
    float4 x[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    if (t < valid) {
      const float* from = (which ? p.q + (size_t)(t0 + t) * p.q_stride : p.k + (size_t)(t0 + t) * p.k_stride) + kvh * kD + c * 8;
      x[0] = load4_f32(from);
      x[1] = load4_f32(from + 4);
    }
    float* to = (which ? qs : ks) + t * LD + c * 8;
    store4(to, x[0]);
    store4(to + 4, x[1]);
    uint32_t o[4][3];
    part2(x[0].x, x[0].y, o[0]); part2(x[0].z, x[0].w, o[1]); part2(x[1].x, x[1].y, o[2]); part2(x[1].z, x[1].w, o[3]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint4*>(parts + (which * 3 + i) * kPart + t * kD + ((c ^ (t & 7)) * 8)) = make_uint4(o[0][i], o[1][i], o[2][i], o[3][i]);
  }
  __syncthreads();
  {
    // two tokens by two, four sums of 32 products each: half of the threads for q k, the others for k k
    const int t = tid % 64 / 8 * 2, s = tid % 8 * 2;
    const float* xs = tid < 64 ? qs : ks;
    if (s <= t + 1 && (RULE == 1 || tid < 64)) {
      float4 a[4] = {};
      auto add = [](float4& c, const float4& x, const float4& y) {
        c.x = __fmaf_rn(x.x, y.x, c.x); c.y = __fmaf_rn(x.y, y.y, c.y); c.z = __fmaf_rn(x.z, y.z, c.z); c.w = __fmaf_rn(x.w, y.w, c.w);
      };
#pragma unroll 4
      for (int d = 0; d < kD; d += 4) {
        const float4 x0 = load4_f32(xs + t * LD + d), x1 = load4_f32(xs + (t + 1) * LD + d);
        const float4 y0 = load4_f32(ks + s * LD + d), y1 = load4_f32(ks + (s + 1) * LD + d);
        add(a[0], x0, y0); add(a[1], x0, y1); add(a[2], x1, y0); add(a[3], x1, y1);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) (tid < 64 ? qk : kk)[(t + i / 2) * kC + s + i % 2] = (a[i].x + a[i].y) + (a[i].z + a[i].w);
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
// more form the read-outs of a chunk while those are at the next, one fetches.  All meet once per chunk, when its u are there;
// everything that the read-outs need lies in two buffers.  Shared memory: stages of (k and q in parts, coefficients, v
// [t][column]), the row warps' shares of S^T q [buffer][row warp][t][column] and of S^T k, u [buffer][column][t], v - G S^T k
// [column][t], u P_16 in parts [buffer][part][t][column].
constexpr int kV = 16, kRowWarps = 4, kStages = 3;                      // columns of a block, row warps, chunks in shared memory
constexpr int kReaders = 4, kWalk = kRowWarps * 32, kAll = kWalk + (kReaders + 1) * 32;
constexpr int kLdV = kV + 4, kLdT = kC + 4, kShares = kC * kLdV;
constexpr int kStage = (6 * kPart * 2 + kCoef * 4 + kC * kV * 4 + 127) / 128 * 128;
template <int RULE>
constexpr size_t walk_smem() {
  return kStages * kStage + (kRowWarps * (RULE == 1 ? 3 : 2) * kShares + (RULE == 1 ? 3 : 2) * kV * kLdT) * sizeof(float) + 2 * 3 * kC * kV * 2 + kStages * 8 + 16;
}
template <int ID, int N>
__device__ __forceinline__ void meet() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory"); }

// Sums over the tokens up to t of a coefficient times a column's value: later ones take no part, be they infinite.
__device__ __forceinline__ float upto(const float* m, const float* y, int t) {
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int s = 0; s < kC; s += 4) {
    const float4 c = load4_f32(m + s), x = load4_f32(y + s);
    a = __fmaf_rn(c.x, s > t ? 0.f : x.x, a); b = __fmaf_rn(c.y, s + 1 > t ? 0.f : x.y, b);
    a = __fmaf_rn(c.z, s + 2 > t ? 0.f : x.z, a); b = __fmaf_rn(c.w, s + 3 > t ? 0.f : x.w, b);
  }
  return a + b;
}

template <int RULE>
__global__ void __launch_bounds__(kAll) chunk_walk_kernel(const ChunkParams p) {
  constexpr int NJ = kD / (16 * kRowWarps);                           // a warp's rows, sixteen at a time
  extern __shared__ __align__(128) unsigned char smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int req = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * kV, start = p.q_start[req], len = p.q_start[req + 1] - start;
  if (len < p.shortest) return;
  const int tid = threadIdx.x, lane = tid & 31, kvh = h / (p.heads / p.kv_heads);
  const int chunks = (len + kC - 1) / kC;
  const size_t first = first_chunk(start, req);
  float* shares_q = reinterpret_cast<float*>(smem + kStages * kStage);
  float* shares_k = shares_q + 2 * kRowWarps * kShares;
  float* us = shares_k + (RULE == 1 ? kRowWarps * kShares : 0);
  float* rest = us + 2 * kV * kLdT;
  __nv_bfloat16* ups = reinterpret_cast<__nv_bfloat16*>(rest + (RULE == 1 ? kV * kLdT : 0));
  uint64_t* there = reinterpret_cast<uint64_t*>(ups + 2 * 3 * kC * kV);
  volatile int* lost = reinterpret_cast<volatile int*>(there + kStages);      // a wait for chunk c ran out: [c & 1]
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 33;" ::"r"(smem_u32(&there[s])));      // lane 0 and every lane's copies
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    lost[0] = lost[1] = 0;
  }
  __syncthreads();
  auto coef_of = [&](int c) { return reinterpret_cast<const float*>(smem + c % kStages * kStage + 6 * kPart * 2); };
  auto await = [&](int c) {                                    // a whole warp
    if (lane == 0 && !copies_there(&there[c % kStages], (c / kStages) & 1)) lost[c & 1] = 1;
    __syncwarp();
  };

  if (tid >= kWalk + kReaders * 32) {
    // One copy each for the parts and the coefficients; the values 16 bytes at a time, zeros behind the portion's end and the last
    // column (a bulk copy for every row of 64 bytes took longer than all else).
    auto fetch = [&](int c) {
      if (c >= chunks) return;
      unsigned char* to = smem + c % kStages * kStage;
      uint64_t* bar = &there[c % kStages];
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
    for (int c = 0; c < kStages - 1; ++c) fetch(c);
    for (int c = 0; c < chunks; ++c) {
      meet<0, kAll>();                                          // everyone is done with the chunk before
      if (lost[c & 1]) {
        // (what was asked for and not waited for ends before the block does)
        for (int n = c; n < min(c + kStages - 1, chunks); ++n) copies_there(&there[n % kStages], (n / kStages) & 1);
        if (lane == 0) atomicOr(p.error, YALIS_FLAG_WAIT_PRODUCT);
        break;
      }
      fetch(c + kStages - 1);
    }
    return;
  }

  if (tid >= kWalk) {
    // read-outs: a thread has CPT columns of a token
    constexpr int CPT = kC * kV / (kReaders * 32);
    const int rt = tid - kWalk, t = rt / (kV / CPT), v0 = rt % (kV / CPT) * CPT;
    const float skip = (RULE == 3 && p.skip) ? p.skip[h] : 0.f;
    for (int c = 0; c < chunks; ++c) {
      await(c);
      meet<0, kAll>();
      if (lost[c & 1]) break;
      const float* coef = coef_of(c);
      const float g = coef[kCoefG + t];
      float o[CPT];
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        float read = 0.f;
#pragma unroll
        for (int w = 0; w < kRowWarps; ++w) read += shares_q[((c & 1) * kRowWarps + w) * kShares + t * kLdV + v0 + i];
        o[i] = __fmaf_rn(g, read, upto(coef + kCoefM + t * kC, us + ((c & 1) * kV + v0 + i) * kLdT, t));
        if constexpr (RULE == 3) o[i] = __fmaf_rn(skip, coef[kCoef + t * kV + v0 + i], o[i]);
      }
      if (c * kC + t < len && j0 + v0 < p.vdim) {
        float* to = p.out + (size_t)(start + c * kC + t) * p.out_stride + (size_t)h * p.vdim + j0 + v0;
#pragma unroll
        for (int i = 0; i < CPT; i += 2) *reinterpret_cast<float2*>(to + i) = make_float2(o[i], o[i + 1]);
      }
    }
    return;
  }

  const int warp = tid / 32;
  // the state, transposed: a lane's columns are col and col + 8, its rows row + 8 n and the one after
  const int col = lane >> 2, row = 16 * NJ * warp + 2 * (lane & 3);
  float* sp = p.state + (size_t)p.slots[req] * p.slot_stride + ((size_t)h * p.vdim + j0 + col) * kD + row;
  float S[2 * NJ][4];
#pragma unroll
  for (int n = 0; n < 2 * NJ; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 x = j0 + col + 8 * e < p.vdim ? *reinterpret_cast<const float2*>(sp + (size_t)e * 8 * kD + 8 * n) : make_float2(0.f, 0.f);
      S[n][2 * e] = x.x; S[n][2 * e + 1] = x.y;
    }
  // parts (of the first operand, of the second), small products first, in two chains that are added: (2, 0), (1, 1), (1, 0) and
  // (0, 2), (0, 1), (0, 0)
  constexpr int order[2][3][2] = {{{2, 0}, {1, 1}, {1, 0}}, {{0, 2}, {0, 1}, {0, 0}}};
  constexpr int CPT = kC * kV / kWalk;                           // a thread's columns of a token in the small sums
  const int t = tid / (kV / CPT), v0 = tid % (kV / CPT) * CPT;
  const int lt = (lane & 7) + (lane >> 4) * 8;                 // ldmatrix: tokens 0-7 by two pieces, tokens 8-15 by two
  const int tt = (lane & 7) + ((lane >> 3) & 1) * 8;           // ldmatrix: two halves of the tokens by a piece, then by the next

  bool whole = true;
  for (int c = 0; c < chunks; ++c) {
    // S^T k and S^T q over this warp's rows
    uint32_t fs[3][NJ][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t o[3];
        part2(S[2 * j + (i >> 1)][2 * (i & 1)], S[2 * j + (i >> 1)][2 * (i & 1) + 1], o);
        fs[0][j][i] = o[0]; fs[1][j][i] = o[1]; fs[2][j][i] = o[2];
      }
    await(c);
    const uint32_t ks = smem_u32(smem + c % kStages * kStage), qs = ks + 3 * kPart * 2;
    const float* coef = coef_of(c);
    const float* vs = coef + kCoef;
    auto read = [&](uint32_t from, float* to) {
      uint32_t f[3][NJ][4];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          ldmatrix4(f[i][j], from + i * kPart * 2 + lt * (kD * 2) + (((2 * NJ * warp + 2 * j + ((lane >> 3) & 1)) ^ (lt & 7)) << 4));
      float sum[NJ][2][2][4] = {};
#pragma unroll
      for (int o = 0; o < 3; ++o)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int n = 0; n < 2; ++n) mma(sum[j][a][n], fs[order[a][o][0]][j], f[order[a][o][1]][j][2 * n], f[order[a][o][1]][j][2 * n + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float y = sum[0][0][n][e] + sum[0][1][n][e];
#pragma unroll
          for (int j = 1; j < NJ; ++j) y += sum[j][0][n][e] + sum[j][1][n][e];
          to[(8 * n + 2 * (lane & 3) + (e & 1)) * kLdV + col + 8 * (e >> 1)] = y;
        }
    };
    if constexpr (RULE == 1) read(ks, shares_k + warp * kShares);
    read(qs, shares_q + ((c & 1) * kRowWarps + warp) * kShares);
    const float w = coef[kCoefW + t];
    float u[CPT];
    if constexpr (RULE == 1) {
      meet<1, kWalk>();
      const float g = coef[kCoefG + t];
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        float a = 0.f;
#pragma unroll
        for (int r = 0; r < kRowWarps; ++r) a += shares_k[r * kShares + t * kLdV + v0 + i];
        rest[(v0 + i) * kLdT + t] = __fmaf_rn(-g, a, vs[t * kV + v0 + i]);
      }
      meet<1, kWalk>();
#pragma unroll
      for (int i = 0; i < CPT; ++i) u[i] = upto(coef + kCoefT + t * kC, rest + (v0 + i) * kLdT, t);
    } else {                                                   // u is known at once
      const float b = coef[kCoefB + t];
#pragma unroll
      for (int i = 0; i < CPT; ++i) u[i] = b * vs[t * kV + v0 + i];
    }
    {                                                          // u, and u times the decays after it in parts
      uint32_t o[3];
      part2(w * u[0], w * u[CPT - 1], o);
#pragma unroll
      for (int i = 0; i < CPT; ++i) us[((c & 1) * kV + v0 + i) * kLdT + t] = u[i];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        __nv_bfloat16* to = ups + (((c & 1) * 3 + i) * kC + t) * kV + v0;
        if constexpr (CPT == 2) *reinterpret_cast<uint32_t*>(to) = o[i];
        else *reinterpret_cast<uint16_t*>(to) = (uint16_t)o[i];
      }
    }
    meet<0, kAll>();
    if (lost[c & 1]) {
      whole = false;
      break;
    }
    // the state: u times the decays after its token, times k
    uint32_t fu[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)                                // ldmatrix: tokens 0-7 by two pieces of columns, tokens 8-15 by two
      ldmatrix4_trans(fu[i], smem_u32(ups + (((c & 1) * 3 + i) * kC + lt) * kV + ((lane >> 3) & 1) * 8));
    const float hi = coef[kCoefL], lo = coef[kCoefL + 1];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      uint32_t f[3][4];
#pragma unroll
      for (int i = 0; i < 3; ++i)
        ldmatrix4_trans(f[i], ks + i * kPart * 2 + tt * (kD * 2) + (((2 * NJ * warp + 2 * j + (lane >> 4)) ^ (tt & 7)) << 4));
      float more[2][2][4] = {};
#pragma unroll
      for (int o = 0; o < 3; ++o)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int n = 0; n < 2; ++n) mma(more[a][n], fu[order[a][o][0]], f[order[a][o][1]][2 * n], f[order[a][o][1]][2 * n + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          S[2 * j + n][e] = __fmaf_rn(hi, S[2 * j + n][e], __fmaf_rn(lo, S[2 * j + n][e], more[0][n][e] + more[1][n][e]));
    }
  }
  if (!whole) return;
#pragma unroll
  for (int n = 0; n < 2 * NJ; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (j0 + col + 8 * e < p.vdim) *reinterpret_cast<float2*>(sp + (size_t)e * 8 * kD + 8 * n) = make_float2(S[n][2 * e], S[n][2 * e + 1]);
}

template <int RULE>
int launch_chunks(const ChunkParams& p, int n_requests, int longest, cudaStream_t stream) {
  constexpr size_t smem = walk_smem<RULE>();
  if (cudaFuncSetAttribute(chunk_walk_kernel<RULE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return YALIS_ERR_LAUNCH;
  const int st = yalis_launch(chunk_prepare_kernel<RULE>, dim3((longest + kC - 1) / kC, p.kv_heads, n_requests), dim3(kWarps * 32), 0, stream, p);
  if (st != YALIS_OK) return st;
  return yalis_launch_after(chunk_walk_kernel<RULE>, dim3((p.vdim + kV - 1) / kV, p.heads, n_requests), dim3(kAll), smem, stream, p);
}

}  // namespace

// float32 values per (chunk, head) of `coef`; a step has n_tokens / 16 + n_requests + 1 chunks at most, each with 6 x 16 x 128
// bfloat16 values per key head in `parts`.
YALIS_API int yalis_state_chunks_coefficients() { return kCoef; }

// The portions of `shortest` tokens and more of a step, the others are left alone.  dim 128, vdim a multiple of four, rows on
// 16-byte boundaries; rule 0: plain, 1: delta, 3: selective; decay_kind 0 or 1 as in yalis_state_scan.  longest: the longest portion.
YALIS_API int yalis_state_chunks(const float* q, int q_stride, const float* k, int k_stride, const float* v, int v_stride,
                                 const float* decay, int decay_kind, const float* beta, const float* skip, float* state,
                                 int64_t slot_stride, float* out, int out_stride, const int32_t* q_start, const int32_t* slots,
                                 int n_requests, int heads, int kv_heads, int dim, int vdim, int rule, int longest, int shortest,
                                 void* parts, void* coef, int32_t* error, cudaStream_t stream) {
  if (n_requests <= 0 || longest <= 0) return YALIS_OK;
  if (dim != kD || vdim <= 0 || vdim % 4 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || heads > 65535 || n_requests > 65535)
    return YALIS_ERR_SHAPE;
  if (decay_kind < 0 || decay_kind > 1 || !decay || (rule != 0 && rule != 1 && rule != 3) || (rule && !beta)) return YALIS_ERR_SHAPE;
  if (((q_stride | k_stride | v_stride | out_stride) & 3) || (slot_stride & 3) ||
      (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state | (uintptr_t)out | (uintptr_t)parts | (uintptr_t)coef) & 15))
    return YALIS_ERR_ALIGN;
  const ChunkParams p = {q, q_stride, k, k_stride, v, v_stride, decay, decay_kind, beta, skip, state, (size_t)slot_stride, out, out_stride,
                         q_start, slots, heads, kv_heads, vdim, shortest, (__nv_bfloat16*)parts, (float*)coef, error};
  if (rule == 0) return launch_chunks<0>(p, n_requests, longest, stream);
  if (rule == 1) return launch_chunks<1>(p, n_requests, longest, stream);
  return launch_chunks<3>(p, n_requests, longest, stream);
}
