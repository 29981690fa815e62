// bf16 GEMM for sm_100a: D[M,N] = A[M,K] * B[N,K]^T with fp32 accumulation in tensor memory.
//
// A persistent grid walks output tiles.  Two forms of one kernel:
//   CG = 2  a pair of CTAs (one cluster, tcgen05 cta_group::2) shares a 256 x BN tile: each CTA holds its 128 rows of A
//           and half of the BN rows of B per stage and 128 x BN of the accumulator, so an operand byte in shared memory
//           feeds twice the products of a tile of one CTA;
//   CG = 1  one CTA per 128 x BN tile, for outputs with too few tiles for the pairs or with few rows; with SPLIT, a
//           cluster of CTAs divides the reduction of one tile and adds the parts through distributed shared memory.
// Warp 0 streams operand tiles into a shared-memory ring with TMA (128-byte swizzle), warp 1 (of the leader) issues
// tcgen05.mma into one of two TMEM accumulators, warps 2-5 drain the other one with tcgen05.ld, so the epilogue of
// tile i overlaps the main loop of tile i+1.  The epilogue (+ bias, or added onto an existing fp32 D) goes through
// swizzled shared memory and TMA stores: 128-byte rows instead of one 16-byte piece per row and instruction, and
// accumulation as a TMA reduction in L2, which takes the read of D off the SM.
//
// Either operand can be K-major (reduction dimension contiguous in memory) or MN-major (row/column
// dimension contiguous), which covers the three GEMMs of a linear layer without a transpose pass:
//   forward  y  = x  * w^T : A = x  (K-major),  B = w (K-major)
//   dgrad    dx = dy * w   : A = dy (K-major),  B = w (MN-major)
//   wgrad    dw = dy^T * x : A = dy (MN-major), B = x (MN-major)
// Every wait is bounded; on a time-out the kernel records a status, drains its own TMA copies, frees its
// tensor memory and returns.
#include "common.cuh"

#include <atomic>
#include <mutex>
#include <unordered_map>

namespace jpb {

constexpr int BM = 128, BK = 64, UMMA_K = 16;  // rows of A per CTA, reduction elements per stage and per instruction
constexpr int A_BYTES = BM * BK * 2;           // 16 KiB
constexpr int GEMM_THREADS = 192;
constexpr int SMEM_MAX = 227 * 1024;
constexpr int EPI_BUF = 32 * 128;              // one store of an epilogue warp: 32 rows of 128 bytes
constexpr int EPI_BYTES = 4 * 2 * EPI_BUF;     // two buffers for each of four warps
constexpr int BAR_BYTES = 256;

template <int CG, int BN>
struct Cfg {
  static constexpr int TM = BM * CG;           // rows of an output tile
  static constexpr int B_ROWS = BN / CG;       // rows of B per CTA
  static constexpr int B_BYTES = B_ROWS * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (SMEM_MAX - 1024 - BAR_BYTES - EPI_BYTES) / STAGE_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + BAR_BYTES + 1024;
  static constexpr int TMEM_COLS = 2 * BN;
  static_assert(STAGES >= 4 && STAGES <= 12 && TMEM_COLS <= 512, "");
};

struct GemmParams {
  int M, N, K;
  int ldd;             // elements between rows of D
  int out_fp32;        // D is fp32 (else bf16)
  int accumulate;      // D += result (D must be fp32)
  int bias_fp32;
  const void* bias;    // per-column bias or nullptr
  void* D;
  int* status;
  int tiles_m, tiles_n;
  int split;           // CTAs that share the reduction of one tile (SPLIT form: one tile per cluster of `split` CTAs)
  int tma_store;       // D can be written through map_d (16-byte aligned rows)
  int a_blocked, b_blocked;  // MN-major operand addressed through a 3-D map {64, K, MN/64}: one copy per stage
  // Batched (grouped, equal-sized groups): `batch` problems stacked along the rows of each operand's storage --
  // A [batch*M, K] or [batch*K, M], B [batch*N, K] or [batch*K, N], D [batch*M, N].  Tiles that straddle the
  // end of a problem read rows of the next one; the epilogue masks them (and K must be a multiple of 64).
  int batch;
  int a_off, b_off;          // storage rows per problem of A and B
  // Groups of unequal size inside equal-sized storage: the M rows of a problem (count_k == 0) or its K reduction
  // rows (count_k == 1) are `segs` segments of `seg_rows` rows, and only the first counts[prob * segs + s] rows of
  // segment s hold data (the others are zero).  Output tiles, or 64-row reduction blocks, without a live row are
  // not loaded and not multiplied; an output tile without any is written as zeros (left alone when accumulating).
  const int* counts;         // device memory, or nullptr: every row is live
  int seg_rows, segs, count_k;
};

// Does [lo, hi) of problem `prob` contain a live row?  Every role of the CTA asks the same question about the same
// ranges and gets the same answer (the counts do not change while the kernel runs), so they skip in step.
__device__ __forceinline__ bool range_live(const GemmParams& p, int prob, int lo, int hi) {
  const int* c = p.counts + prob * p.segs;
  int q1 = (hi - 1) / p.seg_rows;
  if (q1 >= p.segs) q1 = p.segs - 1;
  for (int q = lo / p.seg_rows; q <= q1; ++q) {
    const int s = q * p.seg_rows;
    const int e = s + min(__ldg(c + q), p.seg_rows);
    if (e > s && lo < e && hi > s) return true;
  }
  return false;
}
// Is output tile [m0, m0 + rows) of problem `prob` worth computing?
__device__ __forceinline__ bool tile_live(const GemmParams& p, int prob, int m0, int rows) {
  if (p.counts == nullptr) return true;
  return p.count_k ? range_live(p, prob, 0, p.K) : range_live(p, prob, m0, m0 + rows);
}
// The 64-row reduction blocks of a problem that hold data, as a sequence of ranges [lo, hi): one range covering all
// k blocks when the counts do not describe K; otherwise one per non-empty segment (a block shared by two segments is
// visited once).  Every role walks the same sequence.  No division: this runs once per k block in the threads that
// issue the copies and the MMAs.
struct KRanges {
  int q = 0, next = 0, seg_lo = 0;
  __device__ __forceinline__ bool get(const GemmParams& p, int prob, int k_blocks, int& lo, int& hi) {
    if (p.counts == nullptr || !p.count_k) {
      if (q++ > 0) return false;
      lo = 0; hi = k_blocks;
      return true;
    }
    const int* c = p.counts + prob * p.segs;
    for (; q < p.segs; ++q, seg_lo += p.seg_rows) {
      const int n = min(__ldg(c + q), p.seg_rows);
      if (n <= 0) continue;
      lo = max(next, seg_lo / BK);
      hi = min(k_blocks, (seg_lo + n + BK - 1) / BK);
      if (lo >= hi) continue;
      next = hi;
      ++q; seg_lo += p.seg_rows;
      return true;
    }
    return false;
  }
};

// Tile rasterisation: groups of `group_m` row blocks (2048 rows) are walked column by column, so that the tiles in
// flight at any time touch a few row panels of A and column panels of B -- a working set that stays in L2 instead of
// re-streaming all of A for every column of tiles.
// With live-row counts the group is an odd number of blocks high: empty tiles sit at fixed row blocks, a CTA visits
// every gridDim-th tile, and a height that shares a factor with that stride would hand some CTAs twice as many empty
// tiles as others.
constexpr int GROUP_ROWS = 2048;
__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int tiles_n, int& m_blk, int& n_blk, int group_m) {
  const int per_group = group_m * tiles_n;
  const int group = tile / per_group;
  const int first_m = group * group_m;
  const int gm = (tiles_m - first_m) < group_m ? (tiles_m - first_m) : group_m;
  const int in = tile - group * per_group;
  m_blk = first_m + in % gm;
  n_blk = in / gm;
}

// v += bias[col0 .. col0 + 32)
__device__ __forceinline__ void add_bias(float (&v)[32], const GemmParams& p, int col0) {
  if (!p.bias) return;
  if (p.bias_fp32) {
    const float* b = static_cast<const float*>(p.bias) + col0;
#pragma unroll
    for (int j = 0; j < 32; ++j) if (col0 + j < p.N) v[j] += __ldg(b + j);
  } else {
    const __nv_bfloat16* b = static_cast<const __nv_bfloat16*>(p.bias) + col0;
#pragma unroll
    for (int j = 0; j < 32; ++j) if (col0 + j < p.N) v[j] += __bfloat162float(b[j]);
  }
}

// One row of 32 columns straight to memory: outputs whose rows are not 16-byte aligned.  (Unrolled with a test per column:
// a loop that ends at N would index `v` at run time and put it, and every step of the epilogue, into local memory: the
// 128 x 256 outputs of a CTA then took 8000 cycles, longer than the products of 16 k blocks.)
__device__ __forceinline__ void store_row(const float (&v)[32], const GemmParams& p, size_t row, int col0) {
  if (p.out_fp32) {
    float* d = static_cast<float*>(p.D) + row * p.ldd + col0;
#pragma unroll
    for (int j = 0; j < 32; ++j) if (col0 + j < p.N) d[j] = p.accumulate ? d[j] + v[j] : v[j];
  } else {
    __nv_bfloat16* d = static_cast<__nv_bfloat16*>(p.D) + row * p.ldd + col0;
#pragma unroll
    for (int j = 0; j < 32; ++j) if (col0 + j < p.N) d[j] = __float2bfloat16_rn(v[j]);
  }
}

// What bounds it: the tensor cores, given operands in shared memory.  A 128x256x16 product of one CTA reads 12 KiB of
// operands while the copies for the next ones write 12 KiB, at 128 bytes a cycle more than the product's 128 cycles;
// the pair reads and writes 8 KiB each per CTA and stays within them.
template <int CG, int BN, bool SPLIT, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_d, const GemmParams p) {
  using C = Cfg<CG, BN>;
  constexpr int STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  // operand stages need 1024-byte alignment for the 128-byte swizzle pattern
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi = smem + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi + EPI_BYTES);
  uint64_t* full = bars;                  // [STAGES] TMA -> MMA (pair: the leader's counts both CTAs' bytes)
  uint64_t* empty = bars + STAGES;        // [STAGES] MMA -> TMA (pair: each CTA has its own, one commit arrives on both)
  uint64_t* acc_full = bars + 2 * STAGES;   // [2] MMA -> epilogue (likewise)
  uint64_t* acc_empty = bars + 2 * STAGES + 2;  // [2] epilogue -> MMA (pair: the leader's, both CTAs' warps arrive)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = (CG == 2 || SPLIT) ? int(cluster_ctarank()) : 0;
  const int cluster_ctas = SPLIT ? p.split : CG;
  const int first_tile = blockIdx.x / cluster_ctas;
  const int tile_step = gridDim.x / cluster_ctas;
  const int pair_row = CG == 2 ? rank * BM : 0;           // this CTA's rows of a tile
  const int pair_col = CG == 2 ? rank * C::B_ROWS : 0;    // and the rows of B that it fetches
  const int tiles_per_problem = p.tiles_m * p.tiles_n;
  const int num_tiles = tiles_per_problem * p.batch;
  const int group_m = GROUP_ROWS / C::TM - ((p.counts != nullptr && !p.count_k) ? 1 : 0);
  const int k_all = (p.K + BK - 1) / BK;
  // SPLIT: this CTA's share of the reduction blocks (never empty: the host keeps split <= k_all)
  const int k_begin = SPLIT ? int((long long)(k_all) * rank / p.split) : 0;
  const int k_blocks = SPLIT ? int((long long)(k_all) * (rank + 1) / p.split) : k_all;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4 * CG);  // one arrival per epilogue warp
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    if (p.tma_store) tma_prefetch_desc(&map_d);
  }
  if (warp == 1) {
    tmem_alloc_cg<CG>(tmem_slot, C::TMEM_COLS);
    tmem_relinquish_cg<CG>();
  }
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync();  // the peer's barriers are ready before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------- TMA producer --------------------------------------------
    // (all lanes walk the loop; one elected lane issues: see elect_one)
    uint32_t it = 0;
    uint32_t armed = 0;       // bit s set <=> a copy into stage s may still be in flight
    uint32_t armed_phase = 0; // bit s = barrier phase of the latest copy issued into stage s
    bool ok = true;
    for (int tile = first_tile; tile < num_tiles && ok; tile += tile_step) {
      int m_blk, n_blk;
      const int prob = tile / tiles_per_problem;
      tile_coords(tile - prob * tiles_per_problem, p.tiles_m, p.tiles_n, m_blk, n_blk, group_m);
      if (!tile_live(p, prob, m_blk * C::TM, C::TM)) continue;
      const int m0 = m_blk * C::TM + pair_row, n0 = n_blk * BN + pair_col;
      const int a_row = prob * p.a_off, b_row = prob * p.b_off;  // storage-row offsets of this problem
      KRanges kr;
      int kb_lo, kb_hi;
      while (ok && kr.get(p, prob, k_blocks, kb_lo, kb_hi)) for (int kb = SPLIT ? k_begin : kb_lo; kb < kb_hi; ++kb) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!mbar_wait_bounded_warp(&empty[s], ph ^ 1, abort_flag, p.status)) { ok = false; break; }
        uint8_t* sa = smem + s * STAGE_BYTES;
        uint8_t* sb = sa + A_BYTES;
        armed |= 1u << s;
        armed_phase = (armed_phase & ~(1u << s)) | (ph << s);
        const int k0 = kb * BK;
        if (elect_one()) {
          // The peer's bytes may land on the leader's barrier before the leader has announced them: the phase cannot end
          // without the leader's own arrival, which announces both CTAs' bytes, and the peer cannot run ahead into the
          // next phase, since its `empty` barrier waits for the products that the leader issues after this one.
          if (CG == 1 || rank == 0) mbar_expect_tx(&full[s], STAGE_BYTES * CG);
          const uint32_t bar = CG == 2 ? mapa_u32(&full[s], 0) : 0;
          auto load2 = [&](uint8_t* dst, const CUtensorMap* map, int x, int y) {
            if constexpr (CG == 2) tma_load_2d_pair(dst, map, bar, x, y);
            else tma_load_2d(dst, map, &full[s], x, y);
          };
          auto load3 = [&](uint8_t* dst, const CUtensorMap* map, int x, int y, int z) {
            if constexpr (CG == 2) tma_load_3d_pair(dst, map, bar, x, y, z);
            else tma_load_3d(dst, map, &full[s], x, y, z);
          };
          if (!A_MN) {
            load2(sa, &map_a, k0, a_row + m0);              // box {64 k, 128 rows}
          } else if (p.a_blocked) {
            load3(sa, &map_a, 0, a_row + k0, m0 >> 6);      // box {64 m, 64 k, 2 blocks}
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) load2(sa + j * 8192, &map_a, m0 + j * 64, a_row + k0);
          }
          if (!B_MN) {
            load2(sb, &map_b, k0, b_row + n0);              // box {64 k, B_ROWS rows}
          } else if (p.b_blocked) {
            load3(sb, &map_b, 0, b_row + k0, n0 >> 6);      // box {64 n, 64 k, B_ROWS / 64 blocks}
          } else {
#pragma unroll
            for (int j = 0; j < C::B_ROWS / 64; ++j) load2(sb + j * 8192, &map_b, n0 + j * 64, b_row + k0);
          }
        }
        __syncwarp();
        ++it;
      }
    }
    if (!ok) {
      // drain: wait (bounded) until every copy this thread issued has landed, so that no TMA write is
      // still in flight when the CTA's shared memory is released
      const uint64_t t0 = globaltimer_ns();
      if (CG == 2 && rank != 0) {
        // this CTA's copies report to the leader's barriers, which cannot be polled from here: wait out many times the
        // time that a copy takes
        while (globaltimer_ns() - t0 < 2000000) {
        }
      } else {
        for (int s = 0; s < STAGES; ++s) {
          if (!(armed & (1u << s))) continue;
          const uint32_t ph = (armed_phase >> s) & 1;
          while (!mbar_try_wait(&full[s], ph) && globaltimer_ns() - t0 < wait_budget_ns()) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer (the leader's, in a pair) ------------------------
    if (CG == 1 || rank == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(C::TM, BN, A_MN, B_MN);
      constexpr uint32_t A_STEP = (A_MN ? 2048 : 32) >> 4, B_STEP = (B_MN ? 2048 : 32) >> 4;
      const SmemDesc a_desc = A_MN ? make_smem_desc2(smem_u32(smem), 8192, 1024) : make_smem_desc2(smem_u32(smem), 16, 1024);
      const SmemDesc b_desc = B_MN ? make_smem_desc2(smem_u32(smem) + A_BYTES, 8192, 1024)
                                   : make_smem_desc2(smem_u32(smem) + A_BYTES, 16, 1024);
      uint32_t it = 0;
      uint32_t tile_i = 0;
      bool ok = true;
      for (int tile = first_tile; tile < num_tiles && ok; tile += tile_step) {
        const int prob = tile / tiles_per_problem;
        if (p.counts != nullptr) {
          int m_blk, n_blk;
          tile_coords(tile - prob * tiles_per_problem, p.tiles_m, p.tiles_n, m_blk, n_blk, group_m);
          if (!tile_live(p, prob, m_blk * C::TM, C::TM)) continue;
        }
        const uint32_t acc = tile_i & 1;
        const uint32_t acc_ph = (tile_i >> 1) & 1;
        if (!mbar_wait_bounded_warp(&acc_empty[acc], acc_ph ^ 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        bool fresh = true;  // the first product of a tile overwrites the accumulator
        KRanges kr;
        int kb_lo, kb_hi;
        while (ok && kr.get(p, prob, k_blocks, kb_lo, kb_hi)) for (int kb = SPLIT ? k_begin : kb_lo; kb < kb_hi; ++kb) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait_bounded_warp(&full[s], ph, abort_flag, p.status)) { ok = false; break; }
          tc_fence_after();
          const uint32_t off = uint32_t(s * STAGE_BYTES) >> 4;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_bf16_ss2_cg<CG>(d_tmem, a_desc.lo + off + k * A_STEP, a_desc.hi, b_desc.lo + off + k * B_STEP, b_desc.hi, idesc,
                                   !(fresh && k == 0));
            umma_commit_cg<CG>(&empty[s], 3);  // frees the stage (of both CTAs) once these MMAs have read it
          }
          __syncwarp();
          fresh = false;
          ++it;
        }
        if (ok && elect_one()) umma_commit_cg<CG>(&acc_full[acc], 3);
        __syncwarp();
        ++tile_i;
      }
    }
  } else {
    // ------------------------------- epilogue (warps 2..5) ------------------------------------------
    const int quarter = warp & 3;  // TMEM lanes [32*quarter, 32*quarter+32) are visible to this warp
    uint8_t* buf = epi + quarter * 2 * EPI_BUF;
    uint32_t tile_i = 0;
    uint32_t stores = 0;           // TMA stores issued by this warp (two buffers in turn)
    bool ok = true;
    for (int tile = first_tile; tile < num_tiles && ok; tile += tile_step) {
      int m_blk, n_blk;
      const int prob = tile / tiles_per_problem;
      tile_coords(tile - prob * tiles_per_problem, p.tiles_m, p.tiles_n, m_blk, n_blk, group_m);
      const int m0 = m_blk * C::TM + pair_row, n0 = n_blk * BN;
      const int row_w = m0 + quarter * 32;                // first row of this warp within the problem
      if (!tile_live(p, prob, m_blk * C::TM, C::TM)) {    // uniform across the tile: nothing was computed, it is all zeros
        if (p.accumulate) continue;                       // nothing to add
        const int n_end = min(n0 + BN, p.N);              // this warp's 32 rows, one row at a time, lanes along the columns
        for (int rr = 0; rr < 32 && row_w + rr < p.M; ++rr) {
          const size_t row = size_t(prob) * p.M + row_w + rr;
          if (p.out_fp32) {
            float* d = static_cast<float*>(p.D) + row * p.ldd;
            for (int c = n0 + lane; c < n_end; c += 32) d[c] = 0.f;
          } else {
            __nv_bfloat16* d = static_cast<__nv_bfloat16*>(p.D) + row * p.ldd;
            for (int c = n0 + lane; c < n_end; c += 32) d[c] = __float2bfloat16_rn(0.f);
          }
        }
        continue;
      }
      const uint32_t acc = tile_i & 1;
      const uint32_t acc_ph = (tile_i >> 1) & 1;
      if (!mbar_wait_bounded_warp(&acc_full[acc], acc_ph, abort_flag, p.status)) { ok = false; break; }
      tc_fence_after();
      const uint32_t t_acc = tmem_base + (uint32_t(quarter * 32) << 16) + acc * BN;
      if constexpr (SPLIT) {
        // this CTA's part of the sum, fp32 [128][BN], into the operand ring (all its products have been read); 16-byte
        // pieces are rotated by the row so that the lanes' stores fall into different banks
        float* part = reinterpret_cast<float*>(smem);
        const int r = quarter * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t w[32];
          tmem_ld_32x32(t_acc + c * 32, w);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(part + r * BN + c * 32 + ((j ^ (r & 7)) << 2)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
        }
      } else {
        // A warp whose rows lie behind the last one stores nothing and must leave its buffers alone: without a store of its
        // own to count, the wait for the store before last would not cover the last one, which may still be reading.
        const int c_end = row_w < p.M ? BN : 0;
        const int cols = (p.out_fp32 || !p.tma_store) ? 32 : 64;      // columns per step: 128 bytes of a row
#pragma unroll 1
        for (int c = 0; c < c_end; c += cols) {
          const int col0 = n0 + c;
          if (col0 >= p.N) break;  // uniform across the warp
          uint32_t r[32];
          float v[32];
          tmem_ld_32x32(t_acc + c, r);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          add_bias(v, p, col0);
          if (!p.tma_store) {
            if (row_w + lane < p.M) store_row(v, p, size_t(prob) * p.M + row_w + lane, col0);
            continue;
          }
          uint8_t* b = buf + (stores & 1) * EPI_BUF;
          if (lane == 0) bulk_wait_read<1>();               // the store before last has read this buffer
          __syncwarp();
          uint8_t* row = b + lane * 128;
          const int sw = lane & 7;                          // 128-byte swizzle: piece i of row r sits at i ^ (r & 7)
          if (p.out_fp32) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(row + ((j ^ sw) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              *reinterpret_cast<uint4*>(row + ((j ^ sw) << 4)) = make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                                                                            pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7]));
            tmem_ld_32x32(t_acc + c + 32, r);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            add_bias(v, p, col0 + 32);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              *reinterpret_cast<uint4*>(row + (((j + 4) ^ sw) << 4)) = make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                                                                                  pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7]));
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            if (p.accumulate) tma_reduce_add_3d(&map_d, b, col0, row_w, prob);
            else tma_store_3d(&map_d, b, col0, row_w, prob);
            bulk_commit();
          }
          ++stores;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2 && rank != 0) mbar_arrive_cluster(mapa_u32(&acc_empty[acc], 0));
        else mbar_arrive(&acc_empty[acc]);
      }
      ++tile_i;
    }
    if (lane == 0) bulk_wait_all();
  }

  if constexpr (SPLIT) {
    // every part is in its CTA's shared memory: CTA `rank` adds columns [rank, rank + 1) * BN / split of all of them, in
    // the order of the parts, and writes the result, consecutive threads along a row
    __syncwarp();
    cluster_sync();
    int m_blk, n_blk;
    const int prob = first_tile / tiles_per_problem;
    tile_coords(first_tile - prob * tiles_per_problem, p.tiles_m, p.tiles_n, m_blk, n_blk, group_m);
    const int width = BN / p.split, vecs = width >> 2;     // columns, and 4-column pieces, of this CTA
    const uint32_t part0 = smem_u32(smem);
    for (int i = threadIdx.x; i < BM * vecs; i += GEMM_THREADS) {
      const int r = i / vecs, cc = rank * width + (i - r * vecs) * 4;
      const int piece = (cc >> 2) & 7;
      const uint32_t off = uint32_t(r * BN + (cc & ~31) + ((piece ^ (r & 7)) << 2)) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int q = 0; q < p.split; ++q) {
        uint32_t addr;
        float4 w;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(part0 + off), "r"(q));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(w.x), "=f"(w.y), "=f"(w.z), "=f"(w.w) : "r"(addr) : "memory");
        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
      }
      const int row_in = m_blk * C::TM + r, col = n_blk * BN + cc;
      if (row_in >= p.M) continue;
      const float o[4] = {v.x, v.y, v.z, v.w};
      const size_t at = (size_t(prob) * p.M + row_in) * p.ldd + col;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (col + j >= p.N) break;
        float x = o[j];
        if (p.bias) x += p.bias_fp32 ? __ldg(static_cast<const float*>(p.bias) + col + j)
                                     : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col + j]);
        if (p.out_fp32) {
          float* d = static_cast<float*>(p.D) + at + j;
          *d = p.accumulate ? *d + x : x;
        } else {
          static_cast<__nv_bfloat16*>(p.D)[at + j] = __float2bfloat16_rn(x);
        }
      }
    }
  }

  // ------------------------------- teardown -------------------------------------------------------------
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (CG == 2 || SPLIT) cluster_sync();  // a CTA leaves only when nothing of the cluster reads or signals its memory any more
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_cg<CG>(tmem_base, C::TMEM_COLS);
  }
}

// -------------------------------------------------------------------------------------------------------------
// host side: tensor-map cache + launcher
// -------------------------------------------------------------------------------------------------------------
struct MapKey {
  const void* base;
  uint64_t d0, d1, stride;
  uint32_t b0, b1;
  uint64_t d2 = 1;
  bool operator==(const MapKey& o) const {
    return base == o.base && d0 == o.d0 && d1 == o.d1 && stride == o.stride && b0 == o.b0 && b1 == o.b1 && d2 == o.d2;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.base);
    h = h * 1000003u ^ k.d0;
    h = h * 1000003u ^ k.d1;
    h = h * 1000003u ^ k.stride;
    h = h * 1000003u ^ (size_t(k.b0) << 16 | k.b1);
    h = h * 1000003u ^ k.d2;
    return h;
  }
};

static std::mutex g_map_mutex;
static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_map_cache;

// 2-D bf16 map over a row-major matrix with `rows` rows of `cols` contiguous elements.
static int get_map_2d(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t ld_elems,
                      uint32_t box_cols, uint32_t box_rows) {
  MapKey key{base, cols, rows, ld_elems, box_cols, box_rows};
  {
    std::lock_guard<std::mutex> lock(g_map_mutex);
    auto it = g_map_cache.find(key);
    if (it != g_map_cache.end()) {
      *out = it->second;
      return 0;
    }
  }
  uint64_t dims[2] = {cols, rows};
  uint64_t strides[1] = {ld_elems * 2};
  uint32_t box[2] = {box_cols, box_rows};
  int rc = jpb_make_tensor_map(out, base, 2, 2, dims, strides, box, 1);
  if (rc != 0) return rc;
  std::lock_guard<std::mutex> lock(g_map_mutex);
  if (g_map_cache.size() > 4096) g_map_cache.clear();
  g_map_cache.emplace(key, *out);
  return 0;
}

// 3-D bf16 map over an MN-major operand stored as [K rows, mn contiguous] (mn a multiple of 64): dimensions
// {64 within a block, K, mn / 64 blocks}; one copy of box {64, 64, blocks} lands as `blocks` consecutive
// 64x64 swizzled blocks, the layout the MN-major shared-memory descriptors expect.
static int get_map_mn_blocked(CUtensorMap* out, const void* base, uint64_t mn, uint64_t k_rows, uint64_t ld_elems,
                              uint32_t blocks) {
  MapKey key{base, mn, k_rows, ld_elems, 0xB10Cu, blocks};
  {
    std::lock_guard<std::mutex> lock(g_map_mutex);
    auto it = g_map_cache.find(key);
    if (it != g_map_cache.end()) {
      *out = it->second;
      return 0;
    }
  }
  uint64_t dims[3] = {64, k_rows, mn / 64};
  uint64_t strides[2] = {ld_elems * 2, 128};
  uint32_t box[3] = {64, 64, blocks};
  int rc = jpb_make_tensor_map(out, base, 2, 3, dims, strides, box, 1);
  if (rc != 0) return rc;
  std::lock_guard<std::mutex> lock(g_map_mutex);
  if (g_map_cache.size() > 4096) g_map_cache.clear();
  g_map_cache.emplace(key, *out);
  return 0;
}

// Output map {N, M, problems}: a store of 32 rows of 128 bytes is clipped at the end of its own problem.
static int get_map_out(CUtensorMap* out, const void* base, int elem_bytes, uint64_t n, uint64_t m, uint64_t batch, uint64_t ldd) {
  MapKey key{base, n, m, ldd, 0x0D70u, uint32_t(elem_bytes), batch};
  {
    std::lock_guard<std::mutex> lock(g_map_mutex);
    auto it = g_map_cache.find(key);
    if (it != g_map_cache.end()) {
      *out = it->second;
      return 0;
    }
  }
  uint64_t dims[3] = {n, m, batch};
  uint64_t strides[2] = {ldd * elem_bytes, m * ldd * elem_bytes};
  uint32_t box[3] = {uint32_t(128 / elem_bytes), 32, 1};
  int rc = jpb_make_tensor_map(out, base, elem_bytes, 3, dims, strides, box, 1);
  if (rc != 0) return rc;
  std::lock_guard<std::mutex> lock(g_map_mutex);
  if (g_map_cache.size() > 4096) g_map_cache.clear();
  g_map_cache.emplace(key, *out);
  return 0;
}

static int num_sms() {
  static std::atomic<int> sms{0};
  int n = sms.load(std::memory_order_relaxed);
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    sms.store(n, std::memory_order_relaxed);
  }
  return n;
}

// Which form a product takes.  A launch takes about
//     start + sum over waves of max(main + k blocks x step, out) + out     microseconds,
// a wave being as many tiles as there are CTAs (pairs, clusters) at a time and `out` the epilogue of a tile, which overlaps
// the next tile's products.  A step is not shorter than its part of B takes from memory (with few rows of output the product
// is a pass over B).  The constants were fitted to every form's time at 1410 products (outputs of 8 to 8192 rows and
// 128 to 50304 columns, reductions of 8 to 28672, all three layouts, bf16 and accumulated fp32 results; A in L2, B and the
// result taking turns through more memory than L2 holds).  The form with the least estimate is 0.4 % slower than the fastest
// one on average, 31 % at worst (8 x 7776 x 432); without the terms for the epilogue and for B and without the third form
// it was 7 to 12 % and up to three times.
//   256 x 256 pairs       large outputs: 4096^3 100 us (128 columns 132, single CTAs of 128 columns 152)
//   256 x 128 pairs       768 x 1024 x 28672: 102 us, single CTAs of 64 columns 116
//   128 x 256, one CTA    one wave where narrower tiles need a second, and few rows of A, which every tile fetches again:
//                         128 x 22016 x 4096 38 us, 128 columns 49; 8 x 32000 x 4096 53 us, 69; 384 x 11008 x 4096 36 us,
//                         pairs 41
//   128 x 128, 128 x 64   few tiles, and short reductions, whose time is the epilogue's: 768 x 256 x 1024 with 64 columns
//                         8.3 us, 256 10.1
//   divided reductions    cost 2 to 4 us of their own: 128 x 2304 x 4096 16.7 us in two parts, whole 23; in four 20.4, since
//                         only 33 clusters of four CTAs are resident at once and its 36 tiles took two rounds
enum Form { PAIR256, PAIR128, ONE256, ONE128, ONE64, FORMS };
struct Choice {
  int form, split;
};
struct Resident {      // how many fit on the device at once: CTAs, clusters of two and of four
  int ctas, pairs, quads;
};
static Choice choose(long long batch, int M, int N, int K, bool out_fp32, bool counted, const Resident& res) {
  constexpr int tm[FORMS] = {256, 256, 128, 128, 128}, tn[FORMS] = {256, 128, 256, 128, 64};
  constexpr double start[FORMS] = {3.0, 2.1, 2.5, 2.7, 2.9}, main[FORMS] = {0.6, 1.5, 1.1, 0.9, 0.9},
                   step[FORMS] = {0.306, 0.253, 0.372, 0.277, 0.268}, out[FORMS] = {2.8, 2.2, 1.7, 1.1, 0.6};
  constexpr double bytes_per_us = 5.4e6;   // B from memory, all CTAs together
  const double out_scale = out_fp32 ? 1.4 : 1.0;
  // few rows: every CTA asks for the same lines of A at the same time, the more often the narrower its tiles are
  const double few_rows = M < 64 ? 0.037 * (64 - M) / 64 : 0.0;
  const int k_blocks = (K + BK - 1) / BK;
  Choice best{PAIR256, 1};
  double best_t = 1e30;
  auto offer = [&](int f, int split, double extra) {
    const long long row_tiles = (M + tm[f] - 1) / tm[f], tiles = batch * row_tiles * ((N + tn[f] - 1) / tn[f]);
    const int slots = split == 4 ? res.quads : split == 2 || f <= PAIR128 ? res.pairs : res.ctas;
    if (split > 1 && (counted || tiles > slots || k_blocks < 8 * split)) return;
    const long long full_waves = (tiles - 1) / slots;
    const double o = out[f] * out_scale;
    auto wave = [&](double tiles_in_flight) {
      const double own = step[f] + few_rows * (256.0 / tn[f] - 1.0) * tiles_in_flight / slots;
      const double fetch = tiles_in_flight * split * tn[f] * BK * 2 / row_tiles / bytes_per_us;
      const double products = main[f] + (k_blocks + split - 1) / split * (own > fetch ? own : fetch);
      return products > o ? products : o;
    };
    const double t = start[f] + extra + full_waves * wave(slots) + wave(double(tiles - full_waves * slots)) + o;
    if (t < best_t) { best_t = t; best = {f, split}; }
  };
  for (int f = 0; f < FORMS; ++f) offer(f, 1, 0.0);
  offer(ONE64, 2, 3.7);
  offer(ONE64, 4, 2.2);
  return best;
}

// Clusters of `size` CTAs of this kernel that are resident at once.  148 SMs hold 74 pairs but only 33 clusters of four.
template <int CG, int BN, bool SPLIT>
static int resident_clusters(int size) {
  auto kernel = gemm_bf16_kernel<CG, BN, SPLIT, false, false>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<CG, BN>::SMEM_BYTES) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(num_sms() / size * size);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = Cfg<CG, BN>::SMEM_BYTES;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();   // not an error of the launch that follows
    n = 0;
  }
  const int whole = num_sms() / size;
  return n > 0 && n < whole ? n : whole;
}
static const Resident& resident() {
  static const Resident r = {num_sms(), resident_clusters<2, 256, false>(2), resident_clusters<1, 64, true>(4)};
  return r;
}

template <int CG, int BN, bool SPLIT, bool A_MN, bool B_MN>
static int launch(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& md, const GemmParams& p, cudaStream_t stream) {
  using C = Cfg<CG, BN>;
  auto kernel = gemm_bf16_kernel<CG, BN, SPLIT, A_MN, B_MN>;
  static const cudaError_t configured =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
  if (configured != cudaSuccess) return int(configured);
  const int ctas = SPLIT ? p.split : CG;
  const int tiles = p.tiles_m * p.tiles_n * p.batch;
  const int slots = CG == 2 ? resident().pairs : num_sms() / ctas;
  const int clusters = SPLIT ? tiles : (tiles < slots ? tiles : slots);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * ctas);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctas > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ma, mb, md, p);
  return e != cudaSuccess ? int(e) : int(cudaGetLastError());
}
template <int CG, int BN, bool SPLIT>
static int launch_layout(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& md, const GemmParams& p, int a_mn, int b_mn,
                         cudaStream_t s) {
  if (!a_mn && !b_mn) return launch<CG, BN, SPLIT, false, false>(ma, mb, md, p, s);
  if (!a_mn && b_mn) return launch<CG, BN, SPLIT, false, true>(ma, mb, md, p, s);
  if (a_mn && b_mn) return launch<CG, BN, SPLIT, true, true>(ma, mb, md, p, s);
  return launch<CG, BN, SPLIT, true, false>(ma, mb, md, p, s);
}

}  // namespace jpb

// Common entry: `batch` equal-sized problems stacked along the storage rows of A, B and D (batch == 1: one GEMM).
static int gemm_entry(const void* A, const void* B, void* D, const void* bias, int batch, int M, int N, int K, int lda, int ldb,
                      int ldd, int a_mn_major, int b_mn_major, int out_fp32, int accumulate, int bias_fp32, void* stream,
                      const int* counts = nullptr, int seg_rows = 0, int segs = 0, int count_k = 0) {
  using namespace jpb;
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return 0;
  if (counts != nullptr) {
    // segments must tile the counted dimension exactly; a bias would make dead tiles non-zero
    if (seg_rows <= 0 || segs <= 0 || (long long)seg_rows * segs != (count_k ? K : M) || bias != nullptr || K % BK != 0)
      return -JPB_ERR_BAD_ARGUMENT;
  }
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda & 7) || (ldb & 7))
    return -JPB_ERR_BAD_ARGUMENT;
  if (accumulate && !out_fp32) return -JPB_ERR_BAD_ARGUMENT;
  if (batch > 1 && (K % BK != 0 || bias != nullptr)) return -JPB_ERR_BAD_ARGUMENT;
  GemmParams p;
  const uint64_t nb = uint64_t(batch);
  const int a_blocked = a_mn_major && M % 64 == 0, b_blocked = b_mn_major && N % 64 == 0;
  p.a_blocked = a_blocked; p.b_blocked = b_blocked;
  p.batch = batch;
  p.a_off = a_mn_major ? K : M;
  p.b_off = b_mn_major ? K : N;
  p.M = M; p.N = N; p.K = K; p.ldd = ldd; p.out_fp32 = out_fp32; p.accumulate = accumulate;
  p.bias = bias; p.bias_fp32 = bias_fp32; p.D = D; p.status = jpb_status_device_ptr();
  p.counts = counts; p.seg_rows = seg_rows; p.segs = segs; p.count_k = count_k;
  const Choice choice = choose(batch, M, N, K, out_fp32 != 0, counts != nullptr, resident());
  const int tm = choice.form <= PAIR128 ? 256 : 128;
  const int tn = choice.form == PAIR256 || choice.form == ONE256 ? 256 : choice.form == ONE64 ? 64 : 128;
  const int b_rows = choice.form <= PAIR128 ? tn / 2 : tn;  // rows of B per CTA
  p.tiles_m = (M + tm - 1) / tm;
  p.tiles_n = (N + tn - 1) / tn;
  p.split = choice.split;
  CUtensorMap ma, mb, md;
  int rc;
  if (!a_mn_major) rc = get_map_2d(&ma, A, K, nb * M, lda, BK, BM);
  else if (a_blocked) rc = get_map_mn_blocked(&ma, A, M, nb * K, lda, BM / 64);
  else rc = get_map_2d(&ma, A, M, nb * K, lda, 64, BK);
  if (rc) return rc;
  if (!b_mn_major) rc = get_map_2d(&mb, B, K, nb * N, ldb, BK, b_rows);
  else if (b_blocked) rc = get_map_mn_blocked(&mb, B, N, nb * K, ldb, b_rows / 64);
  else rc = get_map_2d(&mb, B, N, nb * K, ldb, 64, BK);
  if (rc) return rc;
  // D through TMA where its rows start on 16-byte boundaries (else with plain stores)
  const int es = out_fp32 ? 4 : 2;
  p.tma_store = choice.split == 1 && (reinterpret_cast<uintptr_t>(D) & 15) == 0 && (uint64_t(ldd) * es) % 16 == 0;
  if (p.tma_store) {
    rc = get_map_out(&md, D, es, N, M, nb, ldd);
    if (rc) return rc;
  } else {
    md = ma;  // not used
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (choice.form) {
    case PAIR256: return launch_layout<2, 256, false>(ma, mb, md, p, a_mn_major, b_mn_major, s);
    case PAIR128: return launch_layout<2, 128, false>(ma, mb, md, p, a_mn_major, b_mn_major, s);
    case ONE256: return launch_layout<1, 256, false>(ma, mb, md, p, a_mn_major, b_mn_major, s);
    case ONE128: return launch_layout<1, 128, false>(ma, mb, md, p, a_mn_major, b_mn_major, s);
    default:
      if (choice.split > 1) return launch_layout<1, 64, true>(ma, mb, md, p, a_mn_major, b_mn_major, s);
      return launch_layout<1, 64, false>(ma, mb, md, p, a_mn_major, b_mn_major, s);
  }
}

// The form that `batch` products [M, K] x [K, N] take, and the parts of their reductions (times 16), on a device that holds
// `ctas` CTAs, `pairs` clusters of two and `quads` of four at once (ctas = 0: this device).  Forms: 0 and 1 pairs of CTAs with
// 256 and 128 columns, 2 to 4 single CTAs with 256, 128 and 64.
JPB_API int jpb_gemm_form(int batch, int M, int N, int K, int out_fp32, int counted, int ctas, int pairs, int quads) {
  const jpb::Resident res = ctas > 0 ? jpb::Resident{ctas, pairs, quads} : jpb::resident();
  if (res.ctas <= 0 || res.pairs <= 0 || res.quads <= 0 || batch <= 0 || M <= 0 || N <= 0 || K <= 0) return -JPB_ERR_BAD_ARGUMENT;
  const jpb::Choice c = jpb::choose(batch, M, N, K, out_fp32 != 0, counted != 0, res);
  return c.form + 16 * c.split;
}

// A: [M,K] with lda (K-major) or stored as [K,M] with lda (MN-major); likewise B for [N,K] / [K,N].
// All leading dimensions in elements; bf16 operands must be 16-byte aligned with lda/ldb multiples of 8.
JPB_API int jpb_gemm_bf16(const void* A, const void* B, void* D, const void* bias, int M, int N, int K, int lda, int ldb,
                          int ldd, int a_mn_major, int b_mn_major, int out_fp32, int accumulate, int bias_fp32,
                          void* stream) {
  return gemm_entry(A, B, D, bias, 1, M, N, K, lda, ldb, ldd, a_mn_major, b_mn_major, out_fp32, accumulate, bias_fp32, stream);
}

// Grouped GEMM with equal-sized groups (the local experts of a mixture-of-experts layer): problem b uses rows
// [b*M, (b+1)*M) of a K-major A (or rows [b*K, (b+1)*K) of an MN-major one), likewise B, and writes rows
// [b*M, (b+1)*M) of D.  One launch, one persistent grid over all problems' tiles.  K must be a multiple of 64.
JPB_API int jpb_gemm_bf16_batched(const void* A, const void* B, void* D, int batch, int M, int N, int K, int lda, int ldb,
                                  int ldd, int a_mn_major, int b_mn_major, int out_fp32, int accumulate, void* stream) {
  return gemm_entry(A, B, D, nullptr, batch, M, N, K, lda, ldb, ldd, a_mn_major, b_mn_major, out_fp32, accumulate, 0, stream);
}

// Grouped GEMM whose groups differ in size (a mixture-of-experts layer after capacity routing: every expert has room
// for the same number of slots, but fills only some).  Storage is that of jpb_gemm_bf16_batched; `counts` (device
// memory, [batch, segs] int32) says how many rows at the start of each `seg_rows`-row segment hold data -- segments of
// the M rows of each problem (count_k = 0: forward and input gradient), or of its K reduction rows (count_k = 1:
// weight gradient).  The other rows must be zero.  Output tiles and 64-row reduction blocks without a live row cost no
// memory traffic and no tensor-core time; the result equals that of jpb_gemm_bf16_batched.
JPB_API int jpb_gemm_bf16_grouped(const void* A, const void* B, void* D, int batch, int M, int N, int K, int lda, int ldb,
                                  int ldd, int a_mn_major, int b_mn_major, int out_fp32, int accumulate, const int* counts,
                                  int seg_rows, int segs, int count_k, void* stream) {
  if (counts == nullptr) return -JPB_ERR_BAD_ARGUMENT;
  return gemm_entry(A, B, D, nullptr, batch, M, N, K, lda, ldb, ldd, a_mn_major, b_mn_major, out_fp32, accumulate, 0, stream,
                    counts, seg_rows, segs, count_k);
}
