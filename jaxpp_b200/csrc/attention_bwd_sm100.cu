// Flash attention backward for sm_100a, as two tcgen05 kernels plus a small pre-pass:
//
//   delta[b,h,q]  = sum_d dO * O                                        (attn_delta_kernel)
//   dK, dV        : one 128-row K/V block at a time; loops over 128-row Q blocks (and, for GQA, over the query heads
//                   sharing the K/V head).  Works on transposed tiles so that each thread owns one K/V row:
//                   S^T = K Q^T and dP^T = V dO^T in TMEM, P^T and dS^T written over them as bf16, from where
//                   dV += P^T dO and dK += dS^T Q take their A operand; dV and dK stay in TMEM over the whole loop.
//   dQ            : one 128-row Q block at a time; loops over 128-row K/V blocks: S = Q K^T, dP = dO V^T, dS written over
//                   S as bf16, dQ += dS K accumulated in TMEM.
//
// Recomputing S and dP in the second kernel costs two extra MMAs per tile pair but needs no atomics and no
// fp32 dQ staging buffer, and the result is deterministic.  The same shared-memory tile serves as a K-major
// operand in one MMA and as an MN-major operand in another (only the descriptor differs), so nothing is
// transposed in memory.  All waits are bounded.
//
// What bounds them: the tensor cores (4 and 3 products of 128 x 128 x head_dim per pair of blocks, 512 cycles each at
// head_dim 128) and the operand fetches from shared memory, which a 128 x 128 x 16 product with both operands there
// already saturates; P^T and dS stay in tensor memory for that reason.  The products of one block are issued while the
// warps work on the other operand of the same block or on the next block: see the order in the MMA warps.
// Causal, 32 heads of 128, all three kernels: 4096 rows 573 us, 16384 rows 7.56 ms; with 128 x 64 blocks and P, dS
// handed over through shared memory 843 us and 10.5 ms.
#include "common.cuh"

namespace jpb {

// Threads of both main kernels: a TMA warp, an MMA warp and two groups of four warps.  A thread owns one row of a tile
// and its group's 64 of the 128 columns.
constexpr int BWD_THREADS = 64 + 2 * 128;

struct AttnBwdParams {
  int B, Sq, Sk, H, Hkv;
  int Sp;              // Sq rounded up to whole blocks: row pitch of lse and delta
  int causal;
  int by_length_kv, by_length_q;   // order of the tiles of the dK/dV and of the dQ kernel, see DkvTiles
  float scale;
  const float* lse;    // [B,H,Sp], already multiplied by log2(e); +inf behind row Sq
  const float* delta;  // [B,H,Sp], already multiplied by the softmax scale; 0 behind row Sq
  __nv_bfloat16 *dq, *dk, *dv;
  int* status;
};

// ---------------------------------------------------------------------------------------------------------
// Writes delta * scale and lse * log2(e): the forms the two main kernels consume, so that their inner loops are
// one fma + ex2 for P and one fma + mul for dS per element.  D / 8 threads per row, 16 bytes of dO and O each.  The rows
// behind Sq, which exist only in the padded outputs, get the values for which P and dS are zero.
template <int D>
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O,
                                  const float* __restrict__ lse, float* __restrict__ delta_s, float* __restrict__ lse2,
                                  float scale, int B, int S, int Sp, int H) {
  constexpr int TPR = D / 8;
  const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / TPR;   // (b, s, h) over padded s
  const int part = threadIdx.x % TPR;
  const bool in = row < (long long)B * Sp * H;
  const int h = in ? int(row % H) : 0;
  const long long bs = row / H;
  const int s = in ? int(bs % Sp) : Sp, b = in ? int(bs / Sp) : 0;
  float acc = 0.f;
  if (s < S) {
    const size_t at = ((size_t(b) * S + s) * H + h) * D + part * 8;
    const uint4 x = *reinterpret_cast<const uint4*>(dO + at), y = *reinterpret_cast<const uint4*>(O + at);
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 u = unpack_bf16(xs[i]), v = unpack_bf16(ys[i]);
      acc += u.x * v.x + u.y * v.y;
    }
  }
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (part == 0 && in) {
    const size_t idx = (size_t(b) * H + h) * Sp + s;
    delta_s[idx] = s < S ? acc * scale : 0.f;
    lse2[idx] = s < S ? lse[(size_t(b) * H + h) * S + s] * 1.4426950408889634f : INFINITY;
  }
}

// ---------------------------------------------------------------------------------------------------------
// dK / dV
// ---------------------------------------------------------------------------------------------------------
template <int D>
struct DkvSmem {
  static constexpr int DB = D / 64;
  static constexpr int TILE = 128 * 128;      // [128 rows x 64 elements] bf16
  static constexpr int T_BYTES = DB * TILE;   // a block of K, V, Q or dO
  // Stages: Q of block g+1 is needed soon after dK of block g-1 has released its stage, dO a whole block later.
  static constexpr int NSQ = D == 128 ? 3 : 4, NSD = D == 128 ? 2 : 4;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + T_BYTES;
  static constexpr int OFF_Q = OFF_V + T_BYTES;
  static constexpr int OFF_DO = OFF_Q + NSQ * T_BYTES;
  static constexpr int OFF_ST = OFF_DO + NSD * T_BYTES;   // two buffers: lse [128] and delta [128], fp32
  static constexpr int OFF_BAR = OFF_ST + 2 * 1024;
  static constexpr int TOTAL = OFF_BAR + 256;   // no slack for alignment: the kernel checks its base address
  static_assert(TOTAL <= 227 * 1024, "");
};

enum { K1_KV = 0, K1_KVE = 1, K1_QF = 2, K1_DOF = 6, K1_QE = 10, K1_DOE = 14, K1_SF = 18, K1_DPF = 19, K1_PF = 20, K1_DSF = 21,
       K1_ACC = 22, K1_ST = 23, K1_N = 25 };

// Work distribution of the persistent dK/dV kernel, one of two orders:
//   by length  single kv blocks, the ones that the most queries see first, dealt to the CTAs back and forth: every CTA gets
//              the same number of query blocks to within one short tile (32 heads x 32 blocks on 148 SMs: 7 % of the time
//              idle less than with pairs).  All heads are in flight at once.
//   pairs      a work item is a pair of kv blocks (j, n_kvb-1-j) of one (batch, kv head): under a causal mask the two
//              together see the same number of query blocks whatever j is, so items have equal cost and a round-robin over
//              the CTAs is balanced; consecutive items belong to the same head, whose Q / dO stream they share -- taken
//              where the streams of all heads together do not stay in L2.  Tile k of a CTA is half (k & 1) of its item
//              number (k >> 1).
struct DkvTiles {
  int n_kvb, n_pairs, n_items, nq, causal, Sq, Sk, Hkv, heads, by_length;
  __device__ __forceinline__ bool get(int k, int& jb, int& hk, int& b, int& i_start, int& per_head) const {
    int hb;
    bool none = false;
    if (by_length) {
      const int G = gridDim.x;
      const int tile = k * G + ((k & 1) ? G - 1 - int(blockIdx.x) : int(blockIdx.x));
      if (tile >= n_kvb * heads) return false;
      jb = tile / heads;
      hb = tile - jb * heads;
    } else {
      const int item = blockIdx.x + (k >> 1) * gridDim.x;
      if (item >= n_items) return false;
      hb = item / n_pairs;
      const int pi = item - hb * n_pairs;
      jb = (k & 1) ? n_kvb - 1 - pi : pi;
      none = (k & 1) && n_kvb - 1 - pi == pi;    // odd block count: the middle block is its item's only tile
    }
    hk = hb % Hkv;
    b = hb / Hkv;
    i_start = 0;
    if (causal) {
      const int first_q = jb * 128 - (Sk - Sq);  // first query row that sees this kv block
      i_start = first_q > 0 ? first_q / 128 : 0;
    }
    per_head = nq > i_start ? nq - i_start : 0;
    if (none) per_head = -1;
    return true;
  }
};

// 64 values of this thread's row, packed to bf16 in place: columns [0, 32) of the 64 columns at `taddr`
__device__ __forceinline__ void st_packed(uint32_t taddr, const float (&v)[64]) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = pack_bf16(v[c * 32 + 2 * i], v[c * 32 + 2 * i + 1]);
    tmem_st_32x16(taddr + c * 16, w);
  }
  tc_wait_st();
}

// Stores `C` accumulator columns of this thread's row as bf16.
template <int C>
__device__ __forceinline__ void store_acc(uint32_t taddr, __nv_bfloat16* dst, bool row_ok) {
#pragma unroll
  for (int c = 0; c < C / 16; ++c) {
    uint32_t a[16];
    tmem_ld_32x16(taddr + c * 16, a);
    tc_wait_ld();
    if (row_ok) {
#pragma unroll
      for (int i = 0; i < 16; i += 8) {
        uint4 v;
        v.x = pack_bf16(__uint_as_float(a[i]), __uint_as_float(a[i + 1]));
        v.y = pack_bf16(__uint_as_float(a[i + 2]), __uint_as_float(a[i + 3]));
        v.z = pack_bf16(__uint_as_float(a[i + 4]), __uint_as_float(a[i + 5]));
        v.w = pack_bf16(__uint_as_float(a[i + 6]), __uint_as_float(a[i + 7]));
        *reinterpret_cast<uint4*>(dst + c * 16 + i) = v;
      }
    }
  }
}

template <int D>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                     const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                     const AttnBwdParams p) {
  using L = DkvSmem<D>;
  constexpr int NSQ = L::NSQ, NSD = L::NSD;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {   // the swizzled tiles need it; uniform over the grid
    if (threadIdx.x == 0) report_status(p.status, JPB_ERR_BAD_ARGUMENT);
    return;
  }
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + K1_N);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.H / p.Hkv;
  DkvTiles tiles;
  tiles.n_kvb = (p.Sk + 127) / 128;
  tiles.n_pairs = (tiles.n_kvb + 1) / 2;
  tiles.n_items = tiles.n_pairs * p.Hkv * p.B;
  tiles.nq = (p.Sq + 127) / 128; tiles.causal = p.causal; tiles.Sq = p.Sq; tiles.Sk = p.Sk; tiles.Hkv = p.Hkv;
  tiles.heads = p.Hkv * p.B; tiles.by_length = p.by_length_kv;

  if (threadIdx.x == 0) {
    mbar_init(&bar[K1_KV], 1);
    mbar_init(&bar[K1_KVE], 1);
    for (int s = 0; s < NSQ; ++s) { mbar_init(&bar[K1_QF + s], 1); mbar_init(&bar[K1_QE + s], 1); }
    for (int s = 0; s < NSD; ++s) { mbar_init(&bar[K1_DOF + s], 1); mbar_init(&bar[K1_DOE + s], 1); }
    for (int s = 0; s < 2; ++s) mbar_init(&bar[K1_ST + s], 1);
    mbar_init(&bar[K1_SF], 1); mbar_init(&bar[K1_DPF], 1); mbar_init(&bar[K1_ACC], 1);
    mbar_init(&bar[K1_PF], 8); mbar_init(&bar[K1_DSF], 8);   // one arrival per warp of the two groups
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&map_q); tma_prefetch_desc(&map_do); tma_prefetch_desc(&map_k); tma_prefetch_desc(&map_v);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // columns: S^T 128 (P^T over it), dP^T 128 (dS^T over it), dV (D), dK (D).  Of each 64 columns of S^T or dP^T the first
  // 32 take the packed values: every warp overwrites only columns that it alone reads.
  const uint32_t t_s = tmem_base, t_dp = tmem_base + 128, t_dv = tmem_base + 256, t_dk = tmem_base + 256 + D;

  // Every role walks the same tiles in the same order.  `g` counts the (kv block, q block) iterations of this
  // CTA over all its tiles and `tile_i` its non-empty tiles: the barrier phases follow these two counters, so the
  // operand ring, the S / P hand-offs and the K/V buffer carry over from one tile to the next without a drain.
  if (warp == 0) {
    if (lane == 0) {
      uint32_t armed = 0, armed_phase = 0;
      auto arm = [&](int id, uint32_t ph, uint32_t bytes) {
        mbar_expect_tx(&bar[id], bytes);
        armed |= 1u << id;
        armed_phase = (armed_phase & ~(1u << id)) | (ph << id);
      };
      bool ok = true;
      uint32_t g = 0, tile_i = 0;
      int jb, hk, b, i_start, per_head;
      for (int k = 0; ok && tiles.get(k, jb, hk, b, i_start, per_head); ++k) {
        const int n_iter = per_head * G;
        if (n_iter <= 0) continue;
        // K / V of the previous tile are read by its S and dP MMAs only: free once the last of them is done
        if (tile_i > 0 && !mbar_wait_bounded(&bar[K1_KVE], (tile_i - 1) & 1, abort_flag, p.status)) { ok = false; break; }
        arm(K1_KV, tile_i & 1, 2 * L::T_BYTES);
#pragma unroll
        for (int d = 0; d < L::DB; ++d) {
          tma_load_4d(smem + L::OFF_K + d * L::TILE, &map_k, &bar[K1_KV], d * 64, hk, jb * 128, b);
          tma_load_4d(smem + L::OFF_V + d * L::TILE, &map_v, &bar[K1_KV], d * 64, hk, jb * 128, b);
        }
        for (int t = 0; t < n_iter && ok; ++t, ++g) {
          const int sq = g % NSQ, sd = g % NSD, st = g & 1;
          const int h = hk * G + t / per_head;
          const int q0 = (i_start + t % per_head) * 128;
          const size_t stat = (size_t(b) * p.H + h) * p.Sp + q0;
          if (!mbar_wait_bounded(&bar[K1_QE + sq], ((g / NSQ) & 1) ^ 1, abort_flag, p.status)) { ok = false; break; }
          arm(K1_QF + sq, (g / NSQ) & 1, L::T_BYTES);
#pragma unroll
          for (int d = 0; d < L::DB; ++d)
            tma_load_4d(smem + L::OFF_Q + sq * L::T_BYTES + d * L::TILE, &map_q, &bar[K1_QF + sq], d * 64, h, q0, b);
          if (!mbar_wait_bounded(&bar[K1_DOE + sd], ((g / NSD) & 1) ^ 1, abort_flag, p.status)) { ok = false; break; }
          arm(K1_DOF + sd, (g / NSD) & 1, L::T_BYTES);
#pragma unroll
          for (int d = 0; d < L::DB; ++d)
            tma_load_4d(smem + L::OFF_DO + sd * L::T_BYTES + d * L::TILE, &map_do, &bar[K1_DOF + sd], d * 64, h, q0, b);
          // the warps have read the statistics of iteration g - 2 before its dK product, which releases its Q stage
          if (g > 1 && !mbar_wait_bounded(&bar[K1_QE + (g - 2) % NSQ], ((g - 2) / NSQ) & 1, abort_flag, p.status)) { ok = false; break; }
          arm(K1_ST + st, (g >> 1) & 1, 1024);
          bulk_load(smem + L::OFF_ST + st * 1024, p.lse + stat, 512, &bar[K1_ST + st]);
          bulk_load(smem + L::OFF_ST + st * 1024 + 512, p.delta + stat, 512, &bar[K1_ST + st]);
        }
        ++tile_i;
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        for (int id = 0; id < K1_N; ++id) {   // only the barriers of copies are ever armed
          if (!(armed & (1u << id))) continue;
          while (!mbar_try_wait(&bar[id], (armed_phase >> id) & 1) && globaltimer_ns() - t0 < wait_budget_ns()) {
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);  // [kv x q] = K-major x K-major
      constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, 0, 1);  // [kv x d] = TMEM (P^T) x MN-major (dO / Q)
      // descriptor words that do not change from one MMA to the next are computed here, once (see SmemDesc)
      const SmemDesc dk_ = make_smem_desc2(smem_u32(smem + L::OFF_K), 16, 1024);    // K, V, Q, dO as K-major operands
      const SmemDesc dv_ = make_smem_desc2(smem_u32(smem + L::OFF_V), 16, 1024);
      const SmemDesc dq_ = make_smem_desc2(smem_u32(smem + L::OFF_Q), 16, 1024);
      const SmemDesc do_ = make_smem_desc2(smem_u32(smem + L::OFF_DO), 16, 1024);
      const SmemDesc dqm_ = make_smem_desc2(smem_u32(smem + L::OFF_Q), L::TILE, 1024);   // Q / dO as MN-major operands
      const SmemDesc dom_ = make_smem_desc2(smem_u32(smem + L::OFF_DO), L::TILE, 1024);
      constexpr uint32_t T16 = L::T_BYTES >> 4;
      bool ok = true;
      auto kmajor = [&](uint32_t d, const SmemDesc& a, const SmemDesc& bb, uint32_t stage) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = ((k >> 2) * L::TILE + (k & 3) * 32) >> 4;
          umma_bf16_ss2(d, a.lo + off, a.hi, bb.lo + stage * T16 + off, bb.hi, idesc_s, k != 0);
        }
      };
      auto accumulate = [&](uint32_t d, uint32_t a, const SmemDesc& bb, uint32_t stage, uint32_t acc) {
#pragma unroll
        for (int k = 0; k < 128 / 16; ++k)  // reduction over the 128 query rows, 8 packed columns per step
          umma_bf16_ts2(d, a + (k >> 2) * 64 + (k & 3) * 8, bb.lo + stage * T16 + k * 128, bb.hi, idesc_acc, k ? 1u : acc);
      };
      uint32_t g = 0, tile_i = 0;
      int jb, hk, b, i_start, per_head;
      for (int k = 0; ok && tiles.get(k, jb, hk, b, i_start, per_head); ++k) {
        const int n_iter = per_head * G;
        if (n_iter <= 0) continue;
        if (!mbar_wait_bounded(&bar[K1_KV], tile_i & 1, abort_flag, p.status)) { ok = false; break; }
        // Per iteration: dV, the next S^T, dK, the next dP^T.  S^T of the next block overwrites the P^T that dV has just
        // read and dP^T the dS^T of dK (the tensor core runs products in the order of issue), so while the warps take
        // the exponentials of a block the tensor core runs dK and dP^T, and while they form dS^T it runs dV and S^T.
        auto issue_s = [&](uint32_t gg) -> bool {
          if (!mbar_wait_bounded(&bar[K1_QF + gg % NSQ], (gg / NSQ) & 1, abort_flag, p.status)) return false;
          tc_fence_after();
          kmajor(t_s, dk_, dq_, gg % NSQ);
          umma_commit(&bar[K1_SF]);
          return true;
        };
        auto issue_dp = [&](uint32_t gg) -> bool {
          if (!mbar_wait_bounded(&bar[K1_DOF + gg % NSD], (gg / NSD) & 1, abort_flag, p.status)) return false;
          tc_fence_after();
          kmajor(t_dp, dv_, do_, gg % NSD);
          umma_commit(&bar[K1_DPF]);
          return true;
        };
        if (!issue_s(g) || !issue_dp(g)) { ok = false; break; }
        for (int t = 0; t < n_iter; ++t, ++g) {
          const uint32_t sq = g % NSQ, sd = g % NSD;
          const bool more = t + 1 < n_iter;
          if (!more) umma_commit(&bar[K1_KVE]);  // the last S / dP of this tile are done: K and V may be replaced
          if (!mbar_wait_bounded(&bar[K1_PF], g & 1, abort_flag, p.status)) { ok = false; break; }
          tc_fence_after();
          accumulate(t_dv, t_s, dom_, sd, t != 0);
          umma_commit(&bar[K1_DOE + sd]);
          if (more && !issue_s(g + 1)) { ok = false; break; }
          if (!mbar_wait_bounded(&bar[K1_DSF], g & 1, abort_flag, p.status)) { ok = false; break; }
          tc_fence_after();
          accumulate(t_dk, t_dp, dqm_, sq, t != 0);
          umma_commit(&bar[K1_QE + sq]);
          if (more) { if (!issue_dp(g + 1)) { ok = false; break; } }
          else umma_commit(&bar[K1_ACC]);
        }
        ++tile_i;
      }
    }
  } else {
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;  // kv row within the block == TMEM lane
    const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
    const float sl2 = p.scale * 1.4426950408889634f;
    constexpr int EC = D / 2;         // accumulator columns per warp group in the epilogue
    const int grp = (warp - 2) >> 2;  // which 64 of the 128 query columns this warp group handles
    const int cb = grp * 64;
    const int off = p.Sk - p.Sq;
    bool ok = true;
    uint32_t g = 0, tile_i = 0;
    int jb, hk, b, i_start, per_head;
    for (int k = 0; ok && tiles.get(k, jb, hk, b, i_start, per_head); ++k) {
      if (per_head < 0) continue;  // not a tile (middle block already done)
      const int n_iter = per_head * G;
      const int kv0 = jb * 128;
      const int kv = kv0 + r;
      const bool row_ok = kv < p.Sk;
      __nv_bfloat16* dk_row = p.dk + ((size_t(b) * p.Sk + kv) * p.Hkv + hk) * D;
      __nv_bfloat16* dv_row = p.dv + ((size_t(b) * p.Sk + kv) * p.Hkv + hk) * D;
      if (n_iter == 0) {
        if (row_ok) {
          for (int i = grp * EC; i < (grp + 1) * EC; i += 8) {
            *reinterpret_cast<uint4*>(dk_row + i) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(dv_row + i) = make_uint4(0, 0, 0, 0);
          }
        }
        continue;
      }
      for (int t = 0; t < n_iter && ok; ++t, ++g) {
        const int q0 = (i_start + t % per_head) * 128 + cb;
        // Warp-uniform: must some column of this group's 64 be masked?  Columns behind Sq need nothing (their lse is +inf
        // and their delta 0), rows behind Sk are not stored.
        const bool diag = p.causal && kv0 + 127 > q0 + off;
        const int hidden = kv - off - q0;   // columns i < hidden do not see this kv row
        const float* st = reinterpret_cast<const float*>(smem + L::OFF_ST + (g & 1) * 1024) + cb;
        if (!mbar_wait_bounded_warp(&bar[K1_ST + (g & 1)], (g >> 1) & 1, abort_flag, p.status)) { ok = false; break; }
        if (!mbar_wait_bounded_warp(&bar[K1_SF], g & 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        float pv[64];
        {
          uint32_t a[2][32];
          tmem_ld_32x32(t_s + lane_addr + cb, a[0]);
          tmem_ld_32x32(t_s + lane_addr + cb + 32, a[1]);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            const float4 l = *reinterpret_cast<const float4*>(st + i);   // the same address in every lane
            pv[i] = exp2f(fmaf(__uint_as_float(a[i >> 5][i & 31]), sl2, -l.x));
            pv[i + 1] = exp2f(fmaf(__uint_as_float(a[i >> 5][(i & 31) + 1]), sl2, -l.y));
            pv[i + 2] = exp2f(fmaf(__uint_as_float(a[i >> 5][(i & 31) + 2]), sl2, -l.z));
            pv[i + 3] = exp2f(fmaf(__uint_as_float(a[i >> 5][(i & 31) + 3]), sl2, -l.w));
          }
        }
        if (diag) {
#pragma unroll
          for (int i = 0; i < 64; ++i) if (i < hidden) pv[i] = 0.f;
        }
        st_packed(t_s + lane_addr + cb, pv);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar[K1_PF]);
        if (!mbar_wait_bounded_warp(&bar[K1_DPF], g & 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t a[2][32];
          tmem_ld_32x32(t_dp + lane_addr + cb, a[0]);
          tmem_ld_32x32(t_dp + lane_addr + cb + 32, a[1]);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            const float4 dl = *reinterpret_cast<const float4*>(st + 128 + i);
            pv[i] *= fmaf(__uint_as_float(a[i >> 5][i & 31]), p.scale, -dl.x);
            pv[i + 1] *= fmaf(__uint_as_float(a[i >> 5][(i & 31) + 1]), p.scale, -dl.y);
            pv[i + 2] *= fmaf(__uint_as_float(a[i >> 5][(i & 31) + 2]), p.scale, -dl.z);
            pv[i + 3] *= fmaf(__uint_as_float(a[i >> 5][(i & 31) + 3]), p.scale, -dl.w);
          }
        }
        if (diag) {   // 0 times a non-finite factor is not 0
#pragma unroll
          for (int i = 0; i < 64; ++i) if (i < hidden) pv[i] = 0.f;
        }
        st_packed(t_dp + lane_addr + cb, pv);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar[K1_DSF]);
      }
      if (!ok) break;
      // dK / dV of this tile: the accumulators are complete when the last iteration's MMAs are.  The next tile's
      // first accumulating MMA is issued only after these warps hand over its P^T, i.e. after this read.
      if (!mbar_wait_bounded_warp(&bar[K1_ACC], tile_i & 1, abort_flag, p.status)) { ok = false; break; }
      ++tile_i;
      tc_fence_after();
      store_acc<EC>(t_dv + lane_addr + grp * EC, dv_row + grp * EC, row_ok);
      store_acc<EC>(t_dk + lane_addr + grp * EC, dk_row + grp * EC, row_ok);
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// ---------------------------------------------------------------------------------------------------------
// dQ
// ---------------------------------------------------------------------------------------------------------
template <int D>
struct DqSmem {
  static constexpr int DB = D / 64;
  static constexpr int TILE = 128 * 128;      // [128 rows x 64 elements] bf16
  static constexpr int T_BYTES = DB * TILE;
  // Stages: K of block g+1 is needed right after dQ of block g-1 has released its stage, V a whole block later.
  static constexpr int NSK = D == 128 ? 3 : 4, NSV = D == 128 ? 2 : 4;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_DO = OFF_Q + T_BYTES;
  static constexpr int OFF_K = OFF_DO + T_BYTES;
  static constexpr int OFF_V = OFF_K + NSK * T_BYTES;
  static constexpr int OFF_BAR = OFF_V + NSV * T_BYTES;
  static constexpr int TOTAL = OFF_BAR + 256 + 1024;
  static_assert(TOTAL <= 227 * 1024, "");
};

// K2_SF / K2_DSF come in pairs, indexed by the parity of the iteration (two S buffers)
enum { K2_Q = 0, K2_QFREE = 1, K2_KF = 2, K2_VF = 6, K2_KE = 10, K2_VE = 14, K2_SF = 18, K2_DPF = 20, K2_DPR = 21, K2_DSF = 22,
       K2_ACC = 24, K2_N = 25 };

// Work distribution of the persistent dQ kernel, in the same two orders: single query blocks, the ones that see the most
// kv blocks first, or pairs of query blocks (i, num_m-1-i) of one (batch, head).
struct DqTiles {
  int num_m, n_pairs, n_items, H, causal, Sq, Sk, heads, by_length;
  __device__ __forceinline__ bool get(int k, int& m_blk, int& h, int& b, int& n_iter) const {
    int hb;
    bool none = false;
    if (by_length) {
      const int G = gridDim.x;
      const int tile = k * G + ((k & 1) ? G - 1 - int(blockIdx.x) : int(blockIdx.x));
      if (tile >= num_m * heads) return false;
      m_blk = tile / heads;
      hb = tile - m_blk * heads;
      m_blk = num_m - 1 - m_blk;
    } else {
      const int item = blockIdx.x + (k >> 1) * gridDim.x;
      if (item >= n_items) return false;
      hb = item / n_pairs;
      const int pi = item - hb * n_pairs;
      m_blk = (k & 1) ? pi : num_m - 1 - pi;   // the heavier block of the pair first
      none = (k & 1) && num_m - 1 - pi == pi;  // odd block count: the middle block is its item's only tile
    }
    h = hb % H;
    b = hb / H;
    n_iter = (Sk + 127) / 128;
    if (causal) {
      const int last = (m_blk * 128 + 127 + (Sk - Sq)) / 128 + 1;
      n_iter = last < n_iter ? last : n_iter;
      if (n_iter < 1) n_iter = 1;
    }
    if (none) n_iter = 0;
    return true;
  }
};

template <int D>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                   const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const AttnBwdParams p) {
  using L = DqSmem<D>;
  constexpr int NSK = L::NSK, NSV = L::NSV;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + K2_N);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int Gq = p.H / p.Hkv;
  DqTiles tiles;
  tiles.num_m = (p.Sq + 127) / 128;
  tiles.n_pairs = (tiles.num_m + 1) / 2;
  tiles.n_items = tiles.n_pairs * p.H * p.B;
  tiles.H = p.H; tiles.causal = p.causal; tiles.Sq = p.Sq; tiles.Sk = p.Sk;
  tiles.heads = p.H * p.B; tiles.by_length = p.by_length_q;

  if (threadIdx.x == 0) {
    mbar_init(&bar[K2_Q], 1);
    mbar_init(&bar[K2_QFREE], 1);
    for (int s = 0; s < NSK; ++s) { mbar_init(&bar[K2_KF + s], 1); mbar_init(&bar[K2_KE + s], 1); }
    for (int s = 0; s < NSV; ++s) { mbar_init(&bar[K2_VF + s], 1); mbar_init(&bar[K2_VE + s], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bar[K2_SF + i], 1); mbar_init(&bar[K2_DSF + i], 8); }
    mbar_init(&bar[K2_DPF], 1); mbar_init(&bar[K2_DPR], 8); mbar_init(&bar[K2_ACC], 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&map_q); tma_prefetch_desc(&map_do); tma_prefetch_desc(&map_k); tma_prefetch_desc(&map_v);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // columns: two S buffers of 128 (dS over them, packed into the first 32 of each 64), dP 128, dQ (D)
  const uint32_t t_dp = tmem_base + 256, t_dq = tmem_base + 384;

  // As in the dK/dV kernel: every role walks the same tiles; `g` counts this CTA's (q block, kv block) iterations
  // over all its tiles and `tile_i` its tiles, and the barrier phases follow those two counters.
  if (warp == 0) {
    if (lane == 0) {
      uint32_t armed = 0, armed_phase = 0;
      auto arm = [&](int id, uint32_t ph, uint32_t bytes) {
        mbar_expect_tx(&bar[id], bytes);
        armed |= 1u << id;
        armed_phase = (armed_phase & ~(1u << id)) | (ph << id);
      };
      bool ok = true;
      uint32_t g = 0, tile_i = 0;
      int m_blk, h, b, n_iter;
      for (int k = 0; ok && tiles.get(k, m_blk, h, b, n_iter); ++k) {
        if (n_iter <= 0) continue;
        const int hk = h / Gq;
        // Q / dO of the previous tile are read by its S and dP MMAs only
        if (tile_i > 0 && !mbar_wait_bounded(&bar[K2_QFREE], (tile_i - 1) & 1, abort_flag, p.status)) { ok = false; break; }
        arm(K2_Q, tile_i & 1, 2 * L::T_BYTES);
#pragma unroll
        for (int d = 0; d < L::DB; ++d) {
          tma_load_4d(smem + L::OFF_Q + d * L::TILE, &map_q, &bar[K2_Q], d * 64, h, m_blk * 128, b);
          tma_load_4d(smem + L::OFF_DO + d * L::TILE, &map_do, &bar[K2_Q], d * 64, h, m_blk * 128, b);
        }
        for (int t = 0; t < n_iter && ok; ++t, ++g) {
          const int sk = g % NSK, sv = g % NSV;
          if (!mbar_wait_bounded(&bar[K2_KE + sk], ((g / NSK) & 1) ^ 1, abort_flag, p.status)) { ok = false; break; }
          arm(K2_KF + sk, (g / NSK) & 1, L::T_BYTES);
#pragma unroll
          for (int d = 0; d < L::DB; ++d)
            tma_load_4d(smem + L::OFF_K + sk * L::T_BYTES + d * L::TILE, &map_k, &bar[K2_KF + sk], d * 64, hk, t * 128, b);
          if (!mbar_wait_bounded(&bar[K2_VE + sv], ((g / NSV) & 1) ^ 1, abort_flag, p.status)) { ok = false; break; }
          arm(K2_VF + sv, (g / NSV) & 1, L::T_BYTES);
#pragma unroll
          for (int d = 0; d < L::DB; ++d)
            tma_load_4d(smem + L::OFF_V + sv * L::T_BYTES + d * L::TILE, &map_v, &bar[K2_VF + sv], d * 64, hk, t * 128, b);
        }
        ++tile_i;
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        for (int id = 0; id < K2_KE; ++id) {
          if (id == K2_QFREE || !(armed & (1u << id))) continue;
          while (!mbar_try_wait(&bar[id], (armed_phase >> id) & 1) && globaltimer_ns() - t0 < wait_budget_ns()) {
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);  // [q x kv]
      constexpr uint32_t idesc_dq = make_idesc_bf16(128, D, 0, 1);   // [q x d] = TMEM (dS) x MN-major (K)
      const SmemDesc dq_ = make_smem_desc2(smem_u32(smem + L::OFF_Q), 16, 1024);
      const SmemDesc do_ = make_smem_desc2(smem_u32(smem + L::OFF_DO), 16, 1024);
      const SmemDesc dk_ = make_smem_desc2(smem_u32(smem + L::OFF_K), 16, 1024);
      const SmemDesc dv_ = make_smem_desc2(smem_u32(smem + L::OFF_V), 16, 1024);
      const SmemDesc dkm_ = make_smem_desc2(smem_u32(smem + L::OFF_K), L::TILE, 1024);   // K as MN-major operand
      constexpr uint32_t T16 = L::T_BYTES >> 4;
      bool ok = true;
      auto kmajor = [&](uint32_t d, const SmemDesc& a, const SmemDesc& bb, uint32_t stage) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = ((k >> 2) * L::TILE + (k & 3) * 32) >> 4;
          umma_bf16_ss2(d, a.lo + off, a.hi, bb.lo + stage * T16 + off, bb.hi, idesc_s, k != 0);
        }
      };
      // S of iteration gg, over the dS of iteration gg - 2: its product with K has been issued before
      auto issue_s = [&](uint32_t gg) -> bool {
        if (!mbar_wait_bounded(&bar[K2_KF + gg % NSK], (gg / NSK) & 1, abort_flag, p.status)) return false;
        tc_fence_after();
        kmajor(tmem_base + (gg & 1) * 128, dq_, dk_, gg % NSK);
        umma_commit(&bar[K2_SF + (gg & 1)]);
        return true;
      };
      // dP of iteration gg, once the warps have read that of iteration gg - 1
      auto issue_dp = [&](uint32_t gg) -> bool {
        if (!mbar_wait_bounded(&bar[K2_VF + gg % NSV], (gg / NSV) & 1, abort_flag, p.status)) return false;
        if (gg > 0 && !mbar_wait_bounded(&bar[K2_DPR], (gg - 1) & 1, abort_flag, p.status)) return false;
        tc_fence_after();
        kmajor(t_dp, do_, dv_, gg % NSV);
        umma_commit(&bar[K2_VE + gg % NSV]);
        umma_commit(&bar[K2_DPF]);
        return true;
      };
      uint32_t g = 0, tile_i = 0;
      int m_blk, h, b, n_iter;
      for (int k = 0; ok && tiles.get(k, m_blk, h, b, n_iter); ++k) {
        if (n_iter <= 0) continue;
        if (!mbar_wait_bounded(&bar[K2_Q], tile_i & 1, abort_flag, p.status)) { ok = false; break; }
        if (!issue_s(g) || !issue_dp(g)) { ok = false; break; }
        for (int t = 0; t < n_iter; ++t, ++g) {
          // S of the next block runs while the warps take this one's exponentials; dP of the next block and dQ of this one
          // while they take the next one's
          if (t + 1 < n_iter) {
            if (!issue_s(g + 1) || !issue_dp(g + 1)) { ok = false; break; }
          } else {
            umma_commit(&bar[K2_QFREE]);   // the last S / dP of this tile: Q and dO may be replaced
          }
          const uint32_t s = g % NSK, bf = g & 1;
          if (!mbar_wait_bounded(&bar[K2_DSF + bf], (g >> 1) & 1, abort_flag, p.status)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < 128 / 16; ++kk)  // reduction over the 128 kv rows
            umma_bf16_ts2(t_dq, tmem_base + bf * 128 + (kk >> 2) * 64 + (kk & 3) * 8, dkm_.lo + s * T16 + kk * 128, dkm_.hi, idesc_dq,
                          (t | kk) != 0);
          umma_commit(&bar[K2_KE + s]);
          if (t + 1 == n_iter) umma_commit(&bar[K2_ACC]);
        }
        ++tile_i;
      }
    }
  } else {
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
    const float sl2 = p.scale * 1.4426950408889634f;
    const int off = p.Sk - p.Sq;
    constexpr int EC = D / 2;         // dQ columns per warp group in the epilogue
    const int grp = (warp - 2) >> 2;  // which 64 of the 128 kv columns this warp group handles
    const int cb = grp * 64;
    bool ok = true;
    uint32_t g = 0, tile_i = 0;
    int m_blk, h, b, n_iter;
    for (int k = 0; ok && tiles.get(k, m_blk, h, b, n_iter); ++k) {
      if (n_iter <= 0) continue;
      const int m0 = m_blk * 128;
      const int qi = m0 + r;
      const bool row_ok = qi < p.Sq;
      const size_t stat = (size_t(b) * p.H + h) * p.Sp + qi;   // the padded rows exist up to whole blocks
      const float lse_r = p.lse[stat], dl_r = p.delta[stat];
      for (int t = 0; t < n_iter && ok; ++t, ++g) {
        const uint32_t bf = g & 1;
        const uint32_t t_sb = tmem_base + bf * 128 + lane_addr + cb;
        // warp-uniform: is some (query row, kv column) of this warp group's 128 x 64 block hidden?
        const int kv_first = t * 128 + cb;
        const bool edge = kv_first + 63 >= p.Sk || (p.causal && kv_first + 63 > m0 + off);
        const int limit = (p.causal ? min(qi + off, p.Sk - 1) : p.Sk - 1) - kv_first;   // last visible column
        if (!mbar_wait_bounded_warp(&bar[K2_SF + bf], (g >> 1) & 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        float pv[64];
        {
          uint32_t a[2][32];
          tmem_ld_32x32(t_sb, a[0]);
          tmem_ld_32x32(t_sb + 32, a[1]);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 64; ++i) pv[i] = exp2f(fmaf(__uint_as_float(a[i >> 5][i & 31]), sl2, -lse_r));
        }
        if (!mbar_wait_bounded_warp(&bar[K2_DPF], g & 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t a[2][32];
          tmem_ld_32x32(t_dp + lane_addr + cb, a[0]);
          tmem_ld_32x32(t_dp + lane_addr + cb + 32, a[1]);
          tc_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar[K2_DPR]);
#pragma unroll
          for (int i = 0; i < 64; ++i) pv[i] *= fmaf(__uint_as_float(a[i >> 5][i & 31]), p.scale, -dl_r);
        }
        if (edge) {
#pragma unroll
          for (int i = 0; i < 64; ++i) if (i > limit) pv[i] = 0.f;
        }
        st_packed(t_sb, pv);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar[K2_DSF + bf]);
      }
      if (!ok) break;
      // dQ of this tile; the next tile's first accumulating MMA needs a dS hand-over from these warps, which comes
      // after this read of the accumulator
      if (!mbar_wait_bounded_warp(&bar[K2_ACC], tile_i & 1, abort_flag, p.status)) { ok = false; break; }
      ++tile_i;
      tc_fence_after();
      store_acc<EC>(t_dq + lane_addr + grp * EC, p.dq + ((size_t(b) * p.Sq + qi) * p.H + h) * D + grp * EC, row_ok);
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// 4-D map over [B, S, Hn, D] bf16 with a box of [128 rows of S] x [64 elements of D]
static int make_map_rows(CUtensorMap* out, const void* base, int B, int S, int Hn, int D) {
  uint64_t dims[4] = {uint64_t(D), uint64_t(Hn), uint64_t(S), uint64_t(B)};
  uint64_t strides[3] = {uint64_t(D) * 2, uint64_t(Hn) * D * 2, uint64_t(S) * Hn * D * 2};
  uint32_t box[4] = {64, 1, 128, 1};
  return jpb_make_tensor_map(out, base, 2, 4, dims, strides, box, 1);
}

static int padded_rows(int Sq) { return (Sq + 127) / 128 * 128; }

template <int D>
static int launch_bwd(const void* dO, const void* q, const void* k, const void* v, const void* o, const float* lse, float* delta,
                      float* lse2, const AttnBwdParams& p, cudaStream_t stream) {
  CUtensorMap mq, mdo, mk, mv;
  int rc = 0;
  rc |= make_map_rows(&mq, q, p.B, p.Sq, p.H, D);
  rc |= make_map_rows(&mdo, dO, p.B, p.Sq, p.H, D);
  rc |= make_map_rows(&mk, k, p.B, p.Sk, p.Hkv, D);
  rc |= make_map_rows(&mv, v, p.B, p.Sk, p.Hkv, D);
  if (rc) return rc;
  auto k1 = attn_bwd_dkdv_kernel<D>;
  auto k2 = attn_bwd_dq_kernel<D>;
  static const cudaError_t configured1 = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, DkvSmem<D>::TOTAL);
  static const cudaError_t configured2 = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, DqSmem<D>::TOTAL);
  if (configured1 != cudaSuccess || configured2 != cudaSuccess) return -3;
  const long long rows = (long long)p.B * p.Sp * p.H;
  attn_delta_kernel<D><<<(unsigned)((rows * (D / 8) + 255) / 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(dO), static_cast<const __nv_bfloat16*>(o), lse, delta, lse2, p.scale, p.B, p.Sq, p.Sp, p.H);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int n_kvb = (p.Sk + 127) / 128;
  const int items = (p.by_length_kv ? n_kvb : (n_kvb + 1) / 2) * p.Hkv * p.B;  // see DkvTiles
  const int g1 = items < sms ? items : sms;
  k1<<<g1, BWD_THREADS, DkvSmem<D>::TOTAL, stream>>>(mq, mdo, mk, mv, p);
  const int num_m = (p.Sq + 127) / 128;
  const int items2 = (p.by_length_q ? num_m : (num_m + 1) / 2) * p.H * p.B;  // see DqTiles
  const int g2 = items2 < sms ? items2 : sms;
  k2<<<g2, BWD_THREADS, DqSmem<D>::TOTAL, stream>>>(mq, mdo, mk, mv, p);
  return int(cudaGetLastError());
}

}  // namespace jpb

// Scratch needed by jpb_attention_bwd: two fp32 vectors [B,H,Sq rounded up to 128] (delta * scale, lse * log2 e).
JPB_API long long jpb_attention_bwd_scratch_bytes(int B, int Sq, int Sk, int H, int Hkv, int D) {
  (void)Sk; (void)Hkv; (void)D;
  return (long long)B * H * jpb::padded_rows(Sq) * 4 * 2;
}

// All tensors contiguous bf16: dO/q/o/dq [B,Sq,H,D], k/v/dk/dv [B,Sk,Hkv,D]; lse [B,H,Sq] fp32.
// `scratch` must hold jpb_attention_bwd_scratch_bytes() and start on a 16-byte boundary; `reserved` is unused (pass NULL).
JPB_API int jpb_attention_bwd(const void* dO, const void* q, const void* k, const void* v, const void* o, const float* lse,
                              void* dq, void* dk, void* dv, void* scratch, void* reserved, int B, int Sq, int Sk, int H,
                              int Hkv, int D, int causal, float scale, void* stream) {
  using namespace jpb;
  (void)reserved;
  if (H % Hkv != 0 || (D != 64 && D != 128) || (reinterpret_cast<uintptr_t>(scratch) & 15)) return -JPB_ERR_BAD_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  AttnBwdParams p;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.H = H; p.Hkv = Hkv; p.causal = causal; p.scale = scale;
  p.Sp = padded_rows(Sq);
  // half of the L2 cache: the Q and dO (K and V) of all heads that the tiles in flight stream through
  p.by_length_kv = (long long)B * Sq * H * D * 4 <= 64ll * 1024 * 1024;
  p.by_length_q = (long long)B * Sk * Hkv * D * 4 <= 64ll * 1024 * 1024;
  float* delta = static_cast<float*>(scratch);
  float* lse2 = delta + (size_t)B * H * p.Sp;
  p.lse = lse2; p.delta = delta;
  p.dq = static_cast<__nv_bfloat16*>(dq); p.dk = static_cast<__nv_bfloat16*>(dk); p.dv = static_cast<__nv_bfloat16*>(dv);
  p.status = jpb_status_device_ptr();
  return D == 128 ? launch_bwd<128>(dO, q, k, v, o, lse, delta, lse2, p, s) : launch_bwd<64>(dO, q, k, v, o, lse, delta, lse2, p, s);
}
