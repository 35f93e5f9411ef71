// y = x W^T with float32 operands on the tensor cores.
//
// A float32 value is the sum of three bfloat16 values, the value rounded, what is left rounded, and what is left then
// (8 + 8 + 8 bits of mantissa): nothing is lost.  A product of two such sums is nine products of bfloat16 values, which the
// tensor cores form without rounding; the three smallest (below 2^-26 of the product) are left out.  The six others of 16
// values of k are summed on the tensor cores, the small ones first, and every such sum is added to a float32 sum in registers:
// the tensor cores' additions cut off instead of rounding, so chains of them are kept this short.  An output is one chain over
// ascending k whatever the tile: a row's bits depend on neither the number of rows nor the tile that it falls into.
//
// W is the m side of the products (16 rows) and the tokens are the n side (8).  A block's threads fetch 32 values of k of
// its rows as float32, some steps ahead by asynchronous copies that each reads back itself, part them and lay the parts out in
// shared memory (two stages, pieces of 16 bytes swapped within rows of 64: neither the stores nor ldmatrix meet in a bank).
//
// The parts are those of the values times 2^16: so even the last bit of the smallest float32 value lies in bfloat16's range.  An output is computed again
// in float32 FMAs where its sum is not finite (an infinity has no difference to its rounded self, and values from 2^112 and
// outputs from 2^96 on leave the range at its other end) or below 2^-80 (an output below 2^-112: the small parts' products leave it).
//
// What bounds it: mma.sync, which gives 2,048 products a two cycles and SM (973 a cycle measured alone; 0.64 of that here: the
// warps load and multiply in step with one another), and in small steps the chain of a step: copy, part, barrier, load, twelve
// products.  (tcgen05 would give four times that; a form on it faulted and is not used.)
// Error against float64, 2-norm: 2.1e-7 for K = 2,048, 4.1e-7 for 8,192; of FMAs in four chains 4.1e-7 and 8.1e-7.
#include "common.cuh"

namespace {

constexpr int kStep = 32;                     // values of k per stage
constexpr int kQuads = kStep / 4;             // groups of four of them

struct F32Params {
  const void* x; long long ldx;
  const float* w; long long ldw;
  void* out; long long ldo; int out_dtype;
  int M, N, K;
};

__device__ __forceinline__ uint32_t two_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
constexpr float kScale = 65536.f;
// Two float32 operations in one instruction, each rounded as the single one is.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
  return *reinterpret_cast<float2*>(&d);
}
// Four values times kScale as three groups of four bfloat16 values whose sums they are.
__device__ __forceinline__ void part(const float4 v, uint2 (&o)[3]) {
  const float2 scale = make_float2(kScale, kScale), minus = make_float2(-1.f, -1.f);
  float2 a = mul2(make_float2(v.x, v.y), scale), b = mul2(make_float2(v.z, v.w), scale);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[i] = make_uint2(two_bf16(a.x, a.y), two_bf16(b.x, b.y));
    if (i < 2) {
      a = fma2(make_float2(__uint_as_float(o[i].x << 16), __uint_as_float(o[i].x & 0xffff0000u)), minus, a);
      b = fma2(make_float2(__uint_as_float(o[i].y << 16), __uint_as_float(o[i].y & 0xffff0000u)), minus, b);
    }
  }
}
// Copies to shared memory; zeros where there is nothing to read.
template <int BYTES>
__device__ __forceinline__ void copy_async(void* to, const void* from, bool there) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(to);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(from), "r"(there ? 16 : 0) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(at), "l"(from), "n"(BYTES), "r"(there ? BYTES : 0) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// All warps of the block, from wherever each of them is.
__device__ __forceinline__ void meet() { asm volatile("bar.sync 0;" ::: "memory"); }

// WR x WT warps form the products, MT x NT of 16 rows of W by 8 tokens each; FW warps fetch, AHEAD steps before, and part.
// VECX: rows of x on boundaries of four values.
template <typename TX, int WR, int WT, int MT, int NT, int FW, int AHEAD, bool VECX>
__global__ void __launch_bounds__((WR * WT + FW) * 32) gemm_f32_parts_kernel(const F32Params p) {
  constexpr int ROWS = WR * MT * 16, TOKENS = WT * NT * 8, THREADS = FW * 32;
  constexpr int PART_W = ROWS * kStep * 2, PART_X = TOKENS * kStep * 2, STAGE = 3 * (PART_W + PART_X), FETCH = (ROWS + TOKENS) * kStep * 4;
  constexpr int GW = ROWS * kQuads / THREADS, GX = TOKENS * kQuads / THREADS;       // groups of four that a thread fetches
  static_assert(GW >= 1 && GX >= 1 && NT % 2 == 0 && 2 * STAGE >= ROWS * TOKENS * 4, "whole groups; the sums fit the stages");
  extern __shared__ __align__(128) unsigned char smem[];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x - WR * WT * 32;     // tid: of a thread that fetches
  const int n0 = blockIdx.x * ROWS, m0 = (blockIdx.z * gridDim.y + blockIdx.y) * TOKENS;
  const int steps = (p.K + kStep - 1) / kStep;
  const TX* xs = reinterpret_cast<const TX*>(p.x);

  // group u of step i lies in its own 16 bytes of slot i mod AHEAD, behind the stages
  auto slot = [&](int i, int u) { return smem + 2 * STAGE + (i % AHEAD) * FETCH + (u * THREADS + tid) * 16; };
  auto fetch_w = [&](int i) {
#pragma unroll
    for (int u = 0; u < GW; ++u) {
      const int e = tid + u * THREADS, n = n0 + e / kQuads, k = i * kStep + e % kQuads * 4;
      const bool there = n < p.N && k < p.K;
      copy_async<16>(slot(i, u), there ? p.w + (size_t)n * p.ldw + k : p.w, there);
    }
  };
  auto fetch_x = [&](int i) {
#pragma unroll
    for (int u = 0; u < GX; ++u) {
      const int e = tid + u * THREADS, m = m0 + e / kQuads, k = i * kStep + e % kQuads * 4;
      const bool there = m < p.M && k < p.K;
      const TX* from = there ? xs + (size_t)m * p.ldx + k : xs;
      TX* to = reinterpret_cast<TX*>(slot(i, GW + u));
      if constexpr (VECX) {
        copy_async<4 * sizeof(TX)>(to, from, there);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if constexpr (sizeof(TX) == 4) copy_async<4>(to + j, there ? from + j : xs, there);
          else to[j] = there ? from[j] : from_f32<TX>(0.f);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto put = [&](unsigned char* to, int part_bytes, int e, const float4 v) {
    uint2 o[3];
    part(v, o);
    const int r = e / kQuads, h = e % kQuads;                  // 8 bytes of a row of 64, half a 16-byte piece
    unsigned char* at = to + r * (kStep * 2) + (((h >> 1) ^ ((r >> 1) & 3)) << 4) + (h & 1) * 8;
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(at + i * part_bytes) = o[i];
  };
  auto fill = [&](int i) {
    unsigned char* to = smem + (i & 1) * STAGE;
#pragma unroll
    for (int u = 0; u < GW; ++u) put(to, PART_W, tid + u * THREADS, *reinterpret_cast<const float4*>(slot(i, u)));
#pragma unroll
    for (int u = 0; u < GX; ++u) put(to + 3 * PART_W, PART_X, tid + u * THREADS, load4_f32(reinterpret_cast<const TX*>(slot(i, GW + u))));
  };

  if (warp >= WR * WT) {
    for (int i = 0; i < AHEAD; ++i) fetch_w(i);                // weights do not depend on the kernel in front
    pdl_wait();
    for (int i = 0; i < AHEAD; ++i) fetch_x(i);                // (a group of copies per step, all weights with the first)
    for (int i = 0; i < steps; ++i) {
      asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory");
      fill(i);                                                 // the stage whose products were formed before the last barrier
      fetch_w(i + AHEAD);
      fetch_x(i + AHEAD);
      meet();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else {
    pdl_wait();
    meet();
  }

  float acc[MT][NT][4];
#pragma unroll
  for (int a = 0; a < MT; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;
  // addresses of a lane's rows for ldmatrix: 16 rows of W by 16 k; 16 tokens by 16 k
  const int wr = (warp % WR) * MT * 16 + (lane & 15), wt = (warp / WR) * NT * 8 + (lane & 7) + (lane >> 4) * 8;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t aw = base + wr * (kStep * 2), ax = base + 3 * PART_W + wt * (kStep * 2);
  for (int i = 0; i < steps && warp < WR * WT; ++i) {
    const uint32_t stage = (i & 1) * STAGE;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t cw = ((k * 2 + (lane >> 4)) ^ ((wr >> 1) & 3)) << 4, cx = ((k * 2 + ((lane >> 3) & 1)) ^ ((wt >> 1) & 3)) << 4;
      uint32_t fw[3][MT][4], fx[3][NT / 2][4];
#pragma unroll
      for (int s = 0; s < 3; ++s) {
#pragma unroll
        for (int a = 0; a < MT; ++a) ldmatrix4(fw[s][a], aw + stage + s * PART_W + a * 16 * (kStep * 2) + cw);
#pragma unroll
        for (int b = 0; b < NT / 2; ++b) ldmatrix4(fx[s][b], ax + stage + s * PART_X + b * 16 * (kStep * 2) + cx);
      }
      // parts (of w, of x): the products in ascending order of size, so that few additions meet the whole sum
      constexpr int order[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};
      float sum[MT][NT][4];
#pragma unroll
      for (int a = 0; a < MT; ++a)
#pragma unroll
        for (int b = 0; b < NT; ++b)
#pragma unroll
          for (int c = 0; c < 4; ++c) sum[a][b][c] = 0.f;
#pragma unroll
      for (int j = 0; j < 6; ++j)
#pragma unroll
        for (int a = 0; a < MT; ++a)
#pragma unroll
          for (int b = 0; b < NT; ++b)
            mma(sum[a][b], fw[order[j][0]][a], fx[order[j][1]][b / 2][b % 2 * 2], fx[order[j][1]][b / 2][b % 2 * 2 + 1]);
#pragma unroll
      for (int a = 0; a < MT; ++a)
#pragma unroll
        for (int b = 0; b < NT; ++b)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[a][b][c] += sum[a][b][c];
    }
    if (i + 1 < steps) meet();
  }
  meet();                                             // the last products have read their stage
  // through shared memory to rows of outputs: [token][row of W]
  float* sums = reinterpret_cast<float*>(smem);
  if (warp < WR * WT) {
#pragma unroll
    for (int a = 0; a < MT; ++a)
#pragma unroll
      for (int b = 0; b < NT; ++b)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int r = (warp % WR) * MT * 16 + a * 16 + (lane >> 2) + (c >> 1) * 8, t = (warp / WR) * NT * 8 + b * 8 + (lane & 3) * 2 + (c & 1);
          sums[t * ROWS + r] = acc[a][b][c];
        }
  }
  meet();
  for (int e = threadIdx.x; e < ROWS * TOKENS; e += (WR * WT + FW) * 32) {         // (whole warps: ROWS is a multiple of 32)
    const int t = e / ROWS, r = e % ROWS, m = m0 + t, n = n0 + r;
    float y = sums[e];
    const float size = fabsf(y);
    y *= 1.f / kScale / kScale;
    const bool mine = m < p.M && n < p.N, again = mine && !(size <= 3.402823466e38f && (size >= 8.3e-25f || size == 0.f));
    for (uint32_t todo = __ballot_sync(0xffffffffu, again); todo != 0; todo &= todo - 1) {
      const int who = __ffs(todo) - 1;
      const float* wr = p.w + (size_t)(n - lane + who) * p.ldw;
      const TX* xr = xs + (size_t)m * p.ldx;
      float sum = 0.f;
      for (int k = lane; k < p.K; k += 32) sum = __fmaf_rn(to_f32(xr[k]), wr[k], sum);
      sum = warp_sum(sum);
      if (lane == who) y = sum;
    }
    if (mine) {
      const size_t o = (size_t)m * p.ldo + n;
      if (p.out_dtype == YALIS_F32) reinterpret_cast<float*>(p.out)[o] = y;
      else reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(y);
    }
  }
}

template <typename TX, int WR, int WT, int MT, int NT, int FW, int AHEAD, bool VECX>
int launch_parts(const F32Params& p, cudaStream_t stream) {
  constexpr int ROWS = WR * MT * 16, TOKENS = WT * NT * 8, smem = (ROWS + TOKENS) * kStep * (2 * 3 * 2 + AHEAD * 4);
  if (cudaFuncSetAttribute(gemm_f32_parts_kernel<TX, WR, WT, MT, NT, FW, AHEAD, VECX>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return YALIS_ERR_LAUNCH;
  const int tiles = (p.M + TOKENS - 1) / TOKENS, layers = (tiles + 65534) / 65535;      // more than one dimension of a grid holds
  const dim3 grid((p.N + ROWS - 1) / ROWS, (tiles + layers - 1) / layers, layers);
  return yalis_launch(gemm_f32_parts_kernel<TX, WR, WT, MT, NT, FW, AHEAD, VECX>, grid, dim3((WR * WT + FW) * 32), smem, stream, p);
}

// Which tile (the bits are the same).  Tiles of 32 rows of W by 16 tokens up to four blocks an SM: a step waits for weights and
// for its own chain.  64 x 64 with eight warps of 32 x 16 where that makes a block an SM at most (one block has to fill the SM), with
// four of 32 x 32, which load less from shared memory a product and leave room for a second block, where there are more.
// Measured (us, FMAs on the CUDA cores as it was -> now), columns x K:
//   1 token     3,072 x 2,048  39 -> 26    16,384 x 2,048  116 -> 49    2,048 x 8,192  171 -> 105
//   64 tokens   3,072 x 2,048  62 -> 47    16,384 x 2,048  141 -> 91    2,048 x 8,192  238 -> 172
//   250 tokens  3,072 x 2,048  142 -> 91   16,384 x 2,048  486 -> 315   2,048 x 8,192  461 -> 198    2,048 x 2,048  119 -> 52
//   1,024       3,072 x 2,048  416 -> 269  16,384 x 2,048  1,893 -> 1,238
// (1,024 tokens in tiles of 128 x 128: 1,166 for 16,384 columns, 333 for 3,072: not taken.)
template <typename TX, bool VECX>
int launch_sizes(const F32Params& p, cudaStream_t stream) {
  const long long sms = yalis_sm_count();
  auto blocks = [&](int rows, int tokens) { return (long long)((p.N + rows - 1) / rows) * ((p.M + tokens - 1) / tokens); };
  if (p.M <= 16 || blocks(32, 16) <= 4 * sms) return launch_parts<TX, 2, 1, 1, 2, 2, 6, VECX>(p, stream);
  if (blocks(64, 64) <= sms) return launch_parts<TX, 2, 4, 2, 2, 8, 3, VECX>(p, stream);
  return launch_parts<TX, 2, 2, 2, 4, 4, 3, VECX>(p, stream);
}

}  // namespace

// O[M, N] = X[M, K] . W[N, K]^T, float32 W on 16-byte boundaries, K a multiple of four, X float32 or bfloat16.
YALIS_API int yalis_gemm_f32_parts(const void* X, int x_dtype, long long ldx, const float* W, long long ldw, void* O, int o_dtype,
                                   long long ldo, int M, int N, int K, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return YALIS_OK;
  if (K <= 0 || M > 65535 * 64) return YALIS_ERR_SHAPE;
  if (K % 4 || ldw % 4 || (uintptr_t)W % 16) return YALIS_ERR_ALIGN;
  if ((x_dtype != YALIS_F32 && x_dtype != YALIS_BF16) || (o_dtype != YALIS_F32 && o_dtype != YALIS_BF16)) return YALIS_ERR_DTYPE;
  const F32Params p = {X, ldx, W, ldw, O, ldo, o_dtype, M, N, K};
  const bool vec = ldx % 4 == 0 && (uintptr_t)X % (x_dtype == YALIS_F32 ? 16 : 8) == 0;
  if (x_dtype == YALIS_F32) return vec ? launch_sizes<float, true>(p, stream) : launch_sizes<float, false>(p, stream);
  return vec ? launch_sizes<__nv_bfloat16, true>(p, stream) : launch_sizes<__nv_bfloat16, false>(p, stream);
}
