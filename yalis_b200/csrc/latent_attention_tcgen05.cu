// Latent attention for prompt portions on the 5th-generation tensor cores, bfloat16 rows.
//
//   out[n, h] = sum_j softmax_j((q_lat[n, h] . c_j + q_rot[n, h] . k_j) scale) c_j,    row j of the cache = [c_j: R | k_j: p]
//
// A block owns 128 rows (token, head) of one request, in token order, and walks the rows of the cache that its tokens see
// 64 at a time.  A tile of the cache is fetched once (TMA, a box per page or part of one and 64 columns) and read twice, as
// the K operand of the scores and, its first R columns, as the V operand:
//
//   S = Q K^T       tcgen05.mma, Q [128][R + p] and the tile K-major in 128B-swizzled shared memory, S in tensor memory, two
//                   buffers of 64 columns;
//   softmax         four warps, a thread per row: mask by position and window, running maximum and sum in float32; the
//                   weights go back to tensor memory over the scores they came from, as two bfloat16 halves (rounding and
//                   rounding of the rest: 16 bits of mantissa, as in the mma.sync form);
//   O += (P_hi + P_lo) V    tcgen05.mma with A from tensor memory and the tile's rows as an MN-major operand; O [128][R]
//                   stays in tensor memory and is rescaled only when a row's maximum has grown by more than 2^8.
//
// One warp looks up pages and issues the copies (a ring of two or three tiles), one issues the products, whichever are ready:
// the scores of tile j + 1 run while the softmax of tile j is computed.  Blocks are numbered so that the heaviest tiles of queries start first.
//
// What bounds it: the latency of a tile's copies.  At R = 256, p = 64 a tile takes about 3,400 cycles (clock stamps in the
// kernel): its copies arrive 2,300 to 4,000 cycles after they are asked for, one tile being on its way at a time beside the two
// in use.  The tensor pipe has work for 1,664 of them (20 products of 128 x 64 x 16, 8 of 128 x 256 x 16), the softmax warps for
// about 1,100.  The tile is 64 rows wide because O (R columns) and two S fill the tensor memory at R = 384, and because three
// tiles of 320 columns beside Q are what shared memory holds.
// Measured: a layer with r = 256, p = 64, 16 heads and 2,048 tokens (products, preparation and gate included) 582 -> 194 us,
// 523 -> 93 us for this kernel (140 with Q loaded piece by piece and products in a fixed order);
// 8 single tokens of 16 heads behind 1,024 rows in 16 shares: 37 -> 17 us for this kernel, 22 -> 8 us for the merge.
//
// With n_splits > 1 the tiles of a request are dealt to that many blocks in contiguous shares, which leave unnormalised sums
// with their maxima (natural logarithm) and sums of weights for latent_merge_kernel.
//
// Limits (else the caller takes the mma.sync form): R 64, 128, 256 or 384, R + p a multiple of 64 that leaves room for two
// tiles beside Q, pages of 8, 16, 32, 64 or 128 rows, operands on 16-byte boundaries.  All waits are bounded (error word,
// copies drained, tensor memory freed).
#include "tcgen05.cuh"

namespace {

constexpr int LM = 128;            // rows of a block
constexpr int LN = 64;             // rows of the cache per tile
constexpr int kLatentThreads = 192;   // warps 0-3 queries, softmax and output; warp 4 copies; warp 5 products
constexpr int kMaxStages = 3;

struct LatentTc {
  const __nv_bfloat16* q_lat; long ql_n, ql_h;
  const float* q_rot; long qr_n, qr_h;
  void* out; int out_bf16; long o_n, o_h;
  const int32_t* positions; const int32_t* q_start;
  const int32_t* block_table; int table_width, page_size, num_pages;
  int heads, p; float scale_log2; int window;
  const float* sink;
  int n_splits; float* part_o; float* part_ml;
  int n_tokens, stages;
  int32_t* error;
};

template <int R>
__global__ void __launch_bounds__(kLatentThreads, 1)
latent_attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map, const LatentTc a) {
  constexpr int COLS = R + 2 * LN <= 256 ? 256 : 512;      // tensor memory: S0, S1, O
  constexpr int COL_S = 0, COL_O = 2 * LN;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int W = R + a.p, subs = W / 64;
  const int q_bytes = LM * W * 2, tile_bytes = LN * W * 2;
  unsigned char* q_s = base;                               // [subs][128 rows][128 B]
  unsigned char* k_s = q_s + q_bytes;                      // [stages][subs][64 rows][128 B]
  uint64_t* bars = reinterpret_cast<uint64_t*>(k_s + a.stages * tile_bytes);
  uint64_t* full = bars;                                   // [kMaxStages]
  uint64_t* empty = bars + kMaxStages;                     // [kMaxStages]
  uint64_t* s_full = bars + 2 * kMaxStages;                // 2
  uint64_t* p_full = s_full + 2;                           // 2
  uint64_t* o_full = p_full + 2;                           // 1: P V of a tile is done
  uint64_t* o_done = o_full + 1;                           // 1: of the last one (o_full may be two phases behind by then)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map)) : "memory");
    for (int i = 0; i < kMaxStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); }
    mbar_init(o_full, 1);
    mbar_init(o_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  // Tensor memory is taken before the next kernel's blocks are let in: one of theirs that held it while it waits for this
  // kernel would never give it up.
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();                                         // the barriers are initialised, the allocation is written
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t tmem = *tmem_slot;
  auto give_back = [&]() {
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
  };
  const int req = blockIdx.y, split = blockIdx.z;
  const int q0 = a.q_start[req], q_len = a.q_start[req + 1] - q0;
  // the last tiles of a portion see the most rows: they go first
  const int n_rows = q_len * a.heads, row0 = (int)(gridDim.x - 1 - blockIdx.x) * LM;
  if (row0 >= n_rows) {                                    // (uniform)
    give_back();
    return;
  }
  const int rows_here = min(LM, n_rows - row0);
  const int pos_first = a.positions[q0 + row0 / a.heads];
  const int pos_last = a.positions[q0 + (row0 + rows_here - 1) / a.heads];
  const int lo = (a.window > 0 && pos_first - a.window + 1 > 0) ? pos_first - a.window + 1 : 0;
  const int tile_lo = lo / LN, all_tiles = pos_last / LN - tile_lo + 1;
  const int per_split = (all_tiles + a.n_splits - 1) / a.n_splits;
  const int tile_base = tile_lo + split * per_split;
  const int n_tiles = min(per_split, all_tiles - split * per_split);
  if (n_tiles <= 0) {                                      // a share without tiles (uniform)
    for (int r = tid; r < rows_here; r += kLatentThreads) {
      const size_t at = ((size_t)split * a.n_tokens + q0 + (row0 + r) / a.heads) * a.heads + (row0 + r) % a.heads;
      *reinterpret_cast<float2*>(a.part_ml + at * 2) = make_float2(-INFINITY, 0.f);
    }
    give_back();
    return;
  }
  // The queries, as bfloat16, into the swizzled K-major layout: 16-byte piece c of row r lies at piece c ^ (r & 7) of its
  // 128 bytes.  Rows past the last one hold anything: nothing of theirs is stored.  (The copy warp leaves this to the others and starts on the tiles.)
  if (warp != 4) {
    // Loads in batches before their stores: the compiler cannot tell that a store to shared memory leaves the next load
    // alone, and a trip to memory per 16 bytes made this a third of a block's time.
    const int first = warp == 5 ? 128 + lane : tid;        // 160 threads
    constexpr int RP = R / 8, BATCH = 8;                   // 16-byte pieces of a row's first part
    auto place = [&](int r, int piece) -> uint4* {
      return reinterpret_cast<uint4*>(q_s + (piece >> 3) * (LM * 128) + r * 128 + (((piece & 7) ^ (r & 7)) << 4));
    };
    const int lat_end = rows_here * RP;
    for (int e0 = first; e0 < lat_end; e0 += 160 * BATCH) {
      uint4 v[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH; ++i) {
        const int e = e0 + i * 160, r = e / RP;
        if (e < lat_end) {
          const int t = (row0 + r) / a.heads, h = row0 + r - t * a.heads;
          v[i] = *reinterpret_cast<const uint4*>(a.q_lat + (size_t)(q0 + t) * a.ql_n + (size_t)h * a.ql_h + (e - r * RP) * 8);
        }
      }
#pragma unroll
      for (int i = 0; i < BATCH; ++i) {
        const int e = e0 + i * 160, r = e / RP;
        if (e < lat_end) *place(r, e - r * RP) = v[i];
      }
    }
    const int pp = a.p / 8, rot_end = rows_here * pp;
    for (int e0 = first; e0 < rot_end; e0 += 160 * (BATCH / 2)) {
      float4 x[BATCH / 2], y[BATCH / 2];
#pragma unroll
      for (int i = 0; i < BATCH / 2; ++i) {
        const int e = e0 + i * 160, r = e / pp;
        if (e < rot_end) {
          const int t = (row0 + r) / a.heads, h = row0 + r - t * a.heads;
          const float* src = a.q_rot + (size_t)(q0 + t) * a.qr_n + (size_t)h * a.qr_h + (e - r * pp) * 8;
          x[i] = load4_f32(src);
          y[i] = load4_f32(src + 4);
        }
      }
#pragma unroll
      for (int i = 0; i < BATCH / 2; ++i) {
        const int e = e0 + i * 160, r = e / pp;
        if (e < rot_end)
          *place(r, RP + e - r * pp) = make_uint4(pack_bf16(x[i].x, x[i].y), pack_bf16(x[i].z, x[i].w), pack_bf16(y[i].x, y[i].y),
                                                  pack_bf16(y[i].z, y[i].w));
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  int armed = 0;                                           // tiles the copy warp has asked for
  const int page_shift = 31 - __clz(a.page_size), box_shift = min(page_shift, 6);
  const int boxes = LN >> box_shift, box_rows = 1 << box_shift;
  const int32_t* bt = a.block_table + (size_t)req * a.table_width;
  auto box_row = [&](int j) -> int {
    // row of the pool at which this lane's box of tile j starts; past the pool (a box of zeros) where the block's queries
    // see none of its rows, and, with the error word raised, where a visible row has no page
    const int key = ((tile_base + j) << 6) + (lane << box_shift);
    const int none = a.num_pages << page_shift;
    if (lane >= boxes || j >= n_tiles || key > pos_last || key + box_rows <= lo) return none;
    const int pi = key >> page_shift, page = pi < a.table_width ? bt[pi] : -1;
    if (page >= 0 && page < a.num_pages) return (page << page_shift) + (key & (a.page_size - 1));
    if (a.error) atomicOr(a.error, YALIS_FLAG_BAD_PAGE);
    return none;
  };
  auto copy_tile = [&](int j, int y) {                     // the warp: tile j into its buffer, box i from row y of lane i
    const int b = j % a.stages;
    if (lane == 0) mbar_expect_tx(&full[b], (uint32_t)tile_bytes);
    armed = j + 1;
    __syncwarp();
    for (int i0 = 0; i0 < boxes * subs; i0 += 32) {
      const int i = i0 + lane, box = min(i / subs, boxes - 1), sub = i - (i / subs) * subs;
      const int row = __shfl_sync(0xffffffffu, y, box);
      if (i < boxes * subs)
        tma_load_2d(k_s + b * tile_bytes + sub * (LN * 128) + (box << box_shift) * 128, &map, sub * 64, row, &full[b]);
    }
    __syncwarp();
  };
  if (warp == 4) {                                         // the first tiles need no buffer to come free
    for (int j = 0; j < min(n_tiles, a.stages); ++j) copy_tile(j, box_row(j));
  }
  __syncthreads();

  if (warp == 4) {
    // ---------------------------------- copies -------------------------------------------------
    int y = box_row(a.stages);
    for (int j = a.stages; j < n_tiles; ++j) {
      const int b = j % a.stages;
      if (!warp_wait(&empty[b], ((j / a.stages) & 1) ^ 1, abort_flag, lane)) break;
      copy_tile(j, y);
      y = box_row(j + 1);                                  // looked up while the tile is on its way
    }
  } else if (warp == 5) {
    // ---------------------------------- products -----------------------------------------------
    const uint32_t elected = elect_one();
    const uint32_t idesc_qk = idesc_f16(LM, LN, false);
    const uint64_t q_desc = desc_kmajor(smem_u32(q_s)), k_desc0 = desc_kmajor(smem_u32(k_s));
    const uint64_t v_desc0 = desc_mnmajor(smem_u32(k_s), LN * 128);
    auto issue_qk = [&](int j) {
      const int b = j % a.stages;
      // the S buffer is free: P(j - 2), which lay in it, was read by a product issued before this one
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t k_desc = k_desc0 + (uint64_t)((b * tile_bytes) >> 4);
      for (int ks = 0; ks < W / 16; ++ks) {
        const uint32_t q_off = (ks >> 2) * (LM * 128) + (ks & 3) * 32, k_off = (ks >> 2) * (LN * 128) + (ks & 3) * 32;
        umma_ss(elected, tmem + COL_S + (j & 1) * LN, q_desc + (q_off >> 4), k_desc + (k_off >> 4), idesc_qk, ks > 0);
      }
      umma_commit(elected, &s_full[j & 1]);
    };
    auto issue_pv = [&](int j) {
      const int b = j % a.stages;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t v_desc = v_desc0 + (uint64_t)((b * tile_bytes) >> 4);
      const uint32_t p_at = tmem + COL_S + (j & 1) * LN;
#pragma unroll
      for (int half = 0; half < 2; ++half)                 // the weights' upper and lower halves
#pragma unroll
        for (int ks = 0; ks < LN / 16; ++ks) {
          // 16 rows = two 8-row swizzle groups = 2048 bytes further; P: 16 bfloat16 = 8 columns further
          const uint32_t acc = (j > 0 || half > 0 || ks > 0) ? 1u : 0u;
          constexpr int N0 = R < 256 ? R : 256;
          umma_ts(elected, tmem + COL_O, p_at + half * (LN / 2) + ks * 8, v_desc + ((ks * 2048) >> 4), idesc_f16(LM, N0, true), acc);
          if constexpr (R > 256)
            umma_ts(elected, tmem + COL_O + 256, p_at + half * (LN / 2) + ks * 8, v_desc + ((4 * LN * 128 + ks * 2048) >> 4),
                    idesc_f16(LM, R - 256, true), acc);
        }
      umma_commit(elected, o_full);
      umma_commit(elected, &empty[b]);
      if (j + 1 == n_tiles) umma_commit(elected, o_done);
    };
    // Whatever is ready goes out: P V of a tile whose weights are there before the scores of the tile after the next, whose
    // rows may still be on their way (waiting for those first held P V back, and with it the buffer they wait for).
    int next_s = 0, next_o = 0;
    for (uint32_t idle = 0; next_o < n_tiles;) {
      if (next_o < next_s && __all_sync(0xffffffffu, mbar_test(&p_full[next_o & 1], (next_o >> 1) & 1))) {
        issue_pv(next_o++);
        idle = 0;
      } else if (next_s < n_tiles && next_s < next_o + 2 &&
                 __all_sync(0xffffffffu, mbar_test(&full[next_s % a.stages], (next_s / a.stages) & 1))) {
        issue_qk(next_s++);
        idle = 0;
      } else if (++idle > kSpinLimit * 4 || ((idle & 1023u) == 1023u && __any_sync(0xffffffffu, *abort_flag))) {
        if (lane == 0) *abort_flag = 1;
        break;
      }
    }
    __syncwarp();
  } else {
    // ---------------------------------- softmax, a thread per row ------------------------------
    const int r = tid;
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    const bool valid = r < rows_here;
    const int tok = q0 + (row0 + (valid ? r : 0)) / a.heads, head = (row0 + (valid ? r : 0)) % a.heads;
    const int pos = valid ? a.positions[tok] : -1;
    const int first = a.window > 0 ? pos - a.window + 1 : 0;         // the row's first visible key
    const int first_of_all = pos_last - (a.window > 0 ? a.window : pos_last + 1) + 1;   // every row sees keys from here ...
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int b = j & 1, key0 = (tile_base + j) * LN;
      if (!warp_wait(&s_full[b], (j >> 1) & 1, abort_flag, lane)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float sv[LN];
      const uint32_t s_addr = lane_base + COL_S + b * LN;
#pragma unroll
      for (int c0 = 0; c0 < LN; c0 += 32) tmem_ld32(s_addr + c0, *reinterpret_cast<uint32_t(*)[32]>(&sv[c0]));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (key0 + LN - 1 > pos_first || key0 < first_of_all || !valid) {      // ... and up to here: else some key is hidden
#pragma unroll
        for (int c = 0; c < LN; ++c)
          if (key0 + c > pos || key0 + c < first) sv[c] = -INFINITY;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < LN; c += 8) {
        mx[0] = max3(mx[0], sv[c], sv[c + 1]); mx[1] = max3(mx[1], sv[c + 2], sv[c + 3]);
        mx[2] = max3(mx[2], sv[c + 4], sv[c + 5]); mx[3] = max3(mx[3], sv[c + 6], sv[c + 7]);
      }
      const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.scale_log2);
      // the older maximum stays unless the new one is more than 2^8 larger: the weights are float32 numbers either way
      const bool grow = (m_new - m_run > 8.0f) || (m_run == -INFINITY && m_new != -INFINITY);
      const float m_use = grow ? m_new : m_run;
      const float mb = (m_use == -INFINITY) ? 0.f : m_use;
      const float corr = grow ? ((m_run == -INFINITY) ? 0.f : ex2(m_run - mb)) : 1.f;
      uint64_t ls2[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
      const uint64_t scale2 = pack2(a.scale_log2, a.scale_log2), nmb2 = pack2(-mb, -mb);
#pragma unroll
      for (int c0 = 0; c0 < LN; c0 += 32) {
        uint32_t hi[16], lw[16];
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          float x0, x1;
          unpack2(fma2(pack2(sv[c0 + c], sv[c0 + c + 1]), scale2, nmb2), x0, x1);
          const float p0 = ex2(x0), p1 = ex2(x1);
          ls2[(c >> 1) & 1] = add2(ls2[(c >> 1) & 1], pack2(p0, p1));
          const uint32_t h = pack_bf16(p0, p1);
          hi[c >> 1] = h;
          lw[c >> 1] = pack_bf16(p0 - __uint_as_float(h << 16), p1 - __uint_as_float(h & 0xffff0000u));
        }
        tmem_st16(s_addr + (c0 >> 1), hi);                           // over the scores, which are in registers now
        tmem_st16(s_addr + LN / 2 + (c0 >> 1), lw);
      }
      float ls[4];
      unpack2(ls2[0], ls[0], ls[1]);
      unpack2(ls2[1], ls[2], ls[3]);
      l_run = l_run * corr + ((ls[0] + ls[1]) + (ls[2] + ls[3]));
      m_run = m_use;
      if (j > 0 && __any_sync(0xffffffffu, grow)) {                  // rescale O (never for the first tile)
        // (the scores of tile j are there, and P V of tile j - 2 was issued before them: the phase waited for is the current one)
        if (!warp_wait(o_full, (j - 1) & 1, abort_flag, lane)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int c0 = 0; c0 < R; c0 += 16) {
          uint32_t o[16];
          tmem_ld16(lane_base + COL_O + c0, o);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int c = 0; c < 16; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * corr);
          tmem_st16(lane_base + COL_O + c0, o);
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      if (key0 + LN - 1 > pos_last) {
        // Last tile: rows past the last visible one may hold anything (even NaN); its scores are taken, so the rows are
        // zeroed now, before they are multiplied by weights of zero.
        if (r < LN && key0 + r > pos_last) {
          unsigned char* kt = k_s + (j % a.stages) * tile_bytes;
          for (int sub = 0; sub < R / 64; ++sub)
#pragma unroll
            for (int c = 0; c < 8; ++c)
              *reinterpret_cast<uint4*>(kt + sub * (LN * 128) + r * 128 + c * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[b]);
    }
    // ---- output ---------------------------------------------------------------------------------
    if (ok) ok = warp_wait(o_done, 0, abort_flag, lane);
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
      float* share = nullptr;
      if (a.n_splits > 1) {
        const size_t at = ((size_t)split * a.n_tokens + tok) * a.heads + head;
        share = a.part_o + at * R;
        if (valid) *reinterpret_cast<float2*>(a.part_ml + at * 2) = make_float2(m_run * 0.6931471805599453f, l_run);
        inv = 1.f;
      } else if (a.sink != nullptr) {                                // the sums stand relative to m_run: the sink joins there
        const float sk = a.sink[head] * 1.4426950408889634f, mf = fmaxf(m_run, sk);
        const float c = m_run == -INFINITY ? 0.f : exp2f(m_run - mf);
        inv = c / (l_run * c + exp2f(sk - mf));
      }
      const size_t base_out = (size_t)tok * a.o_n + (size_t)head * a.o_h;
#pragma unroll 1
      for (int c0 = 0; c0 < R; c0 += 32) {
        uint32_t o[32];
        __syncwarp();                                                // rows past the last one and the others part below
        tmem_ld32(lane_base + COL_O + c0, o);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (!valid) continue;
        if (share == nullptr && a.out_bf16) {
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.out) + base_out + c0;
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(o[c]) * inv, __uint_as_float(o[c + 1]) * inv);
            v.y = pack_bf16(__uint_as_float(o[c + 2]) * inv, __uint_as_float(o[c + 3]) * inv);
            v.z = pack_bf16(__uint_as_float(o[c + 4]) * inv, __uint_as_float(o[c + 5]) * inv);
            v.w = pack_bf16(__uint_as_float(o[c + 6]) * inv, __uint_as_float(o[c + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c) = v;
          }
        } else {
          float* dst = share != nullptr ? share + c0 : reinterpret_cast<float*>(a.out) + base_out + c0;
#pragma unroll
          for (int c = 0; c < 32; c += 4)
            *reinterpret_cast<float4*>(dst + c) = make_float4(__uint_as_float(o[c]) * inv, __uint_as_float(o[c + 1]) * inv,
                                                              __uint_as_float(o[c + 2]) * inv, __uint_as_float(o[c + 3]) * inv);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }

  // ---- exit: drain what was asked for, free tensor memory -------------------------------------------------------------
  __syncthreads();
  if (*abort_flag && tid == 4 * 32) {
    if (a.error) atomicOr(a.error, YALIS_FLAG_WAIT_ATTENTION);
    for (int j = max(0, armed - a.stages); j < armed; ++j)
      for (uint32_t i = 0; i < kSpinLimit; ++i)
        if (mbar_try_wait(&full[j % a.stages], (j / a.stages) & 1)) break;
  }
  __syncthreads();
  give_back();
}

// The pool [pages, 1, page_size, W] as a matrix [pages * page_size, W]; boxes of [min(page, 64) rows, 64 columns].
bool make_latent_map(CUtensorMap* map, const void* pool, long long rows, int W, int page_size) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  cuuint64_t dims[2] = {(cuuint64_t)W, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)W * 2};
  cuuint32_t box[2] = {64u, (cuuint32_t)(page_size < LN ? page_size : LN)};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(pool), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int kLatentSmem = 227 * 1024;

size_t latent_tc_smem(int W, int stages) {
  return 1024 + (size_t)(LM + stages * LN) * W * 2 + (2 * kMaxStages + 6) * 8 + 16;
}

template <int R>
int launch_latent_tc(const CUtensorMap& map, const LatentTc& a, dim3 grid, cudaStream_t stream) {
  const size_t smem = latent_tc_smem(R + a.p, a.stages);
  if (cudaFuncSetAttribute(latent_attention_tcgen05_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return YALIS_ERR_LAUNCH;
  return yalis_launch(latent_attention_tcgen05_kernel<R>, grid, dim3(kLatentThreads), smem, stream, map, a);
}

}  // namespace

// Whether this form takes a latent of r and a rotated part of p sizes in pages of page_size rows.
YALIS_API int yalis_latent_attention_tcgen05_supports(int r, int p, int page_size) {
  const bool page_ok = page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64 || page_size == 128;
  return page_ok && (r == 64 || r == 128 || r == 256 || r == 384) && p >= 0 && p % 64 == 0 &&
         latent_tc_smem(r + p, 2) <= (size_t)kLatentSmem ? 1 : 0;
}

// The kernel above; the merge of n_splits > 1 is the caller's.  q_lat bfloat16, q_rot float32, both on 16-byte boundaries in
// every row; out bfloat16 or float32 likewise.
int yalis_latent_tc_launch(const void* q_lat, long ql_n, long ql_h, const float* q_rot, long qr_n, long qr_h, void* out,
                           int out_bf16, long o_n, long o_h, const void* pool, const int32_t* positions,
                           const int32_t* q_start, const int32_t* block_table, int table_width, int page_size, int num_pages,
                           int n_requests, int n_tokens, int max_q_len, int heads, int r, int p, float scale, int window,
                           const float* sink, int n_splits, float* part_o, float* part_ml, int32_t* error, cudaStream_t stream) {
  LatentTc a;
  a.q_lat = (const __nv_bfloat16*)q_lat; a.ql_n = ql_n; a.ql_h = ql_h; a.q_rot = q_rot; a.qr_n = qr_n; a.qr_h = qr_h;
  a.out = out; a.out_bf16 = out_bf16; a.o_n = o_n; a.o_h = o_h; a.positions = positions; a.q_start = q_start;
  a.block_table = block_table; a.table_width = table_width; a.page_size = page_size; a.num_pages = num_pages;
  a.heads = heads; a.p = p; a.scale_log2 = scale * 1.4426950408889634f; a.window = window; a.sink = sink;
  a.n_splits = n_splits; a.part_o = part_o; a.part_ml = part_ml; a.n_tokens = n_tokens; a.error = error;
  a.stages = latent_tc_smem(r + p, 3) <= (size_t)kLatentSmem ? 3 : 2;
  CUtensorMap map;
  if (!make_latent_map(&map, pool, (long long)num_pages * page_size, r + p, page_size)) return YALIS_ERR_LAUNCH;
  const dim3 grid((unsigned)(((long long)max_q_len * heads + LM - 1) / LM), n_requests, n_splits);
  switch (r) {
    case 64: return launch_latent_tc<64>(map, a, grid, stream);
    case 128: return launch_latent_tc<128>(map, a, grid, stream);
    case 256: return launch_latent_tc<256>(map, a, grid, stream);
    case 384: return launch_latent_tc<384>(map, a, grid, stream);
  }
  return YALIS_ERR_SHAPE;
}
