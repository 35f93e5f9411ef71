// y = x W^T on the CUDA cores: the float32 path's product with small and unaligned weights
// (the others: gemm_f32_mma.cu), and the twin of the tensor-core products in tests.
//
// x [M, K] and W [N, K] are both K-contiguous (a Linear layer's weight as it
// is stored).  Products and sums are float32 FMAs; there is no tensor-core
// instruction and no reduced-precision mode anywhere in this file, so with
// float32 operands the result is a true 32-bit product.  Each output element
// is accumulated in chains over fixed values of k that are added in a fixed
// order, so it does not depend on M, N or the tile a row falls into: a token's
// result is the same bits whatever batch it is computed in.
//
// Operand and output types are independent (float or bfloat16), which lets the
// same kernel serve as the twin of the tensor-core kernels in tests.
#include "common.cuh"

namespace {

// A tile of BM x BN outputs per block, BK values of k at a time through two buffers in shared memory.  The block's threads
// are kGroups groups that each take every output of the tile over their own quarter of every BK values, TM x TN outputs a
// thread; at the end the groups' sums are added in order.  An output is therefore four chains of FMAs over fixed values of
// k, added in a fixed order: the same bits whatever M, N and the tile.  Values of the next tile are loaded to registers while
// the current one is multiplied, 16 bytes at a time where rows are aligned.
//
// What bounds it: the FMAs (128 a cycle and SM) and the loads from shared memory beside them, 16 values for the 64 FMAs of
// 8 x 8 outputs a thread: together 0.43 of the FMA rate for the products of 250 rows.  A step of a few hundred rows has about as
// many tiles as there are SMs: hence four groups, two warps per scheduler from one block, whose waits cover one another.
constexpr int kGroups = 4;

template <typename TA, typename TW, typename TO, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(kGroups * (BM / TM) * (BN / TN), 2)
gemm_tn_simt_kernel(const TA* A, long long lda, const TW* W, long long ldw, TO* O, long long ldo, int M, int N, int K) {
  constexpr int BK = 32, KG = BK / kGroups, PER = (BM / TM) * (BN / TN), THREADS = kGroups * PER, TX = BN / TN;
  constexpr int LA = BM + 4, LW = BN + 4;                  // padded rows: the transposed stores spread over the banks
  constexpr int NA = BM * BK / 4 / THREADS, NW = BN * BK / 4 / THREADS;      // groups of four k values a thread loads
  static_assert(NA >= 1 && NW >= 1 && TM % 4 == 0 && TN % 4 == 0, "whole groups");
  static_assert(BM * BN <= 2 * BK * (LA + LW), "a group's sums fit the buffers");
  __shared__ __align__(16) float buffers[2 * BK * (LA + LW)];
  auto As = [&](int b, int k) { return buffers + (size_t)(b * BK + k) * LA; };
  auto Ws = [&](int b, int k) { return buffers + 2 * BK * LA + (size_t)(b * BK + k) * LW; };
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, group = tid / PER, tx = tid % PER % TX, ty = tid % PER / TX;
  const int m0 = (blockIdx.z * gridDim.y + blockIdx.y) * BM, n0 = blockIdx.x * BN;
  if (m0 >= M) return;                                     // (the last of several layers of blocks)
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  float4 ra[NA], rw[NW];
  // four values of row `row` from k on; zeros outside the matrix
  auto fetch4 = [&](const auto* p, long long ld, int row, int rows, int k) -> float4 {
    if (row >= rows || k >= K) return make_float4(0.f, 0.f, 0.f, 0.f);
    const auto* q = p + (size_t)row * ld + k;
    if constexpr (VEC) return load4_f32(q);                // K is a multiple of four
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = k + u < K ? to_f32(q[u]) : 0.f;
    return make_float4(v[0], v[1], v[2], v[3]);
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int e = tid + i * THREADS;
      ra[i] = fetch4(A, lda, m0 + e / (BK / 4), M, k0 + (e % (BK / 4)) * 4);
    }
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      const int e = tid + i * THREADS;
      rw[i] = fetch4(W, ldw, n0 + e / (BK / 4), N, k0 + (e % (BK / 4)) * 4);
    }
  };
  auto put = [&](int b) {
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int e = tid + i * THREADS, r = e / (BK / 4), k = (e % (BK / 4)) * 4;
      float* to = As(b, k) + r;
      to[0] = ra[i].x; to[LA] = ra[i].y; to[2 * LA] = ra[i].z; to[3 * LA] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      const int e = tid + i * THREADS, r = e / (BK / 4), k = (e % (BK / 4)) * 4;
      float* to = Ws(b, k) + r;
      to[0] = rw[i].x; to[LW] = rw[i].y; to[2 * LW] = rw[i].z; to[3 * LW] = rw[i].w;
    }
  };

  fetch(0);
  put(0);
  __syncthreads();
  int b = 0;
  for (int k0 = 0; k0 < K; k0 += BK, b ^= 1) {
    const bool more = k0 + BK < K;
    if (more) fetch(k0 + BK);
    const float* ap = As(b, group * KG) + ty * 4;
    const float* wp = Ws(b, group * KG) + tx * 4;
#pragma unroll
    for (int kk = 0; kk < KG; ++kk) {
      float a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(ap + kk * LA + (i / 4) * (BM * 4 / TM));
        a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const float4 v = *reinterpret_cast<const float4*>(wp + kk * LW + (j / 4) * (BN * 4 / TN));
        w[j] = v.x; w[j + 1] = v.y; w[j + 2] = v.z; w[j + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    if (more) put(b ^ 1);             // the buffer that the round before read: everyone passed the barrier behind it
    __syncthreads();
  }
  // the groups' sums, in order, through the buffers
  for (int g = 1; g < kGroups; ++g) {
    if (group == g) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) buffers[(i * TN + j) * PER + tid % PER] = acc[i][j];
    }
    __syncthreads();
    if (group == 0) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] += buffers[(i * TN + j) * PER + tid % PER];
    }
    __syncthreads();
  }
  if (group != 0) return;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + (i / 4) * (BM * 4 / TM) + ty * 4 + i % 4;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + (j / 4) * (BN * 4 / TN) + tx * 4 + j % 4;
      if (n < N) O[(size_t)m * ldo + n] = from_f32<TO>(acc[i][j]);
    }
  }
}

template <typename TA, typename TW, typename TO, int BM, int BN, int TM, int TN>
int launch_tile(const void* A, long long lda, const void* W, long long ldw, void* O, long long ldo, int M, int N, int K,
                cudaStream_t stream) {
  // more row tiles than one dimension of a grid holds go on in the next
  const int row_tiles = (M + BM - 1) / BM, layers = (row_tiles + 65534) / 65535;
  const dim3 grid((N + BN - 1) / BN, (row_tiles + layers - 1) / layers, layers), block(kGroups * (BM / TM) * (BN / TN));
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % (4 * sizeof(TA)) == 0 &&
                   (uintptr_t)W % (4 * sizeof(TW)) == 0;
  if (vec)
    return yalis_launch(gemm_tn_simt_kernel<TA, TW, TO, BM, BN, TM, TN, true>, grid, block, 0, stream, (const TA*)A, lda,
                        (const TW*)W, ldw, (TO*)O, ldo, M, N, K);
  return yalis_launch(gemm_tn_simt_kernel<TA, TW, TO, BM, BN, TM, TN, false>, grid, block, 0, stream, (const TA*)A, lda,
                      (const TW*)W, ldw, (TO*)O, ldo, M, N, K);
}

// Which tile: 32 x 128 with 8 x 8 outputs a thread where that makes a block for every other SM at least and the columns fill it,
// else 32 x 32 with 4 x 4: more blocks.
// Measured (us, float32; 64 x 64 tiles with 4 x 4 outputs a thread, as it was -> now), columns x K:
//   250 rows   3,072 x 2,048  227 -> 147    2,048 x 2,048  158 -> 90     16,384 x 2,048  699 -> 494    2,048 x 8,192  610 -> 331
//   1,024 rows 3,072 x 2,048  602 -> 424    2,048 x 2,048  411 -> 287    16,384 x 2,048  2,704 -> 1,907  2,048 x 8,192  1,614 -> 1,104
//   8 rows     3,072 x 2,048  159 -> 71     16,384 x 2,048  221 -> 90    2,048 x 8,192  633 -> 262
// 1,024 rows were faster still in tiles of 128 x 128 with one chain an output (359, 248 and, for K = 8,192, 956), which 250 rows
// do not fill the SMs with; an output's bits must not depend on the tile, so one number of chains serves all sizes.
template <typename TA, typename TW, typename TO>
int launch(const void* A, long long lda, const void* W, long long ldw, void* O, long long ldo, int M, int N, int K,
           cudaStream_t stream) {
  if (((long long)M + 63) / 64 > 65535) return YALIS_ERR_SHAPE;      // (4,194,240 rows)
  const long long sms = yalis_sm_count();
  const long long blocks = (long long)((N + 127) / 128) * ((M + 31) / 32);
  if (blocks >= sms / 2 && N > 64) return launch_tile<TA, TW, TO, 32, 128, 8, 8>(A, lda, W, ldw, O, ldo, M, N, K, stream);
  return launch_tile<TA, TW, TO, 32, 32, 4, 4>(A, lda, W, ldw, O, ldo, M, N, K, stream);
}

}  // namespace

// O[M, N] = A[M, K] . W[N, K]^T with float32 accumulation.
YALIS_API int yalis_gemm_tn_simt(const void* A, int a_dtype, long long lda, const void* W, int w_dtype, long long ldw,
                                 void* O, int o_dtype, long long ldo, int M, int N, int K, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return YALIS_OK;
  if (K <= 0) return YALIS_ERR_SHAPE;
  using bf16 = __nv_bfloat16;
  const int code = a_dtype * 4 + w_dtype * 2 + o_dtype;
  switch (code) {
    case 0: return launch<float, float, float>(A, lda, W, ldw, O, ldo, M, N, K, stream);
    case 1: return launch<float, float, bf16>(A, lda, W, ldw, O, ldo, M, N, K, stream);
    case 2: return launch<float, bf16, float>(A, lda, W, ldw, O, ldo, M, N, K, stream);
    case 3: return launch<float, bf16, bf16>(A, lda, W, ldw, O, ldo, M, N, K, stream);
    case 4: return launch<bf16, float, float>(A, lda, W, ldw, O, ldo, M, N, K, stream);
    case 5: return launch<bf16, float, bf16>(A, lda, W, ldw, O, ldo, M, N, K, stream);
    case 6: return launch<bf16, bf16, float>(A, lda, W, ldw, O, ldo, M, N, K, stream);
    case 7: return launch<bf16, bf16, bf16>(A, lda, W, ldw, O, ldo, M, N, K, stream);
    default: return YALIS_ERR_DTYPE;
  }
}
