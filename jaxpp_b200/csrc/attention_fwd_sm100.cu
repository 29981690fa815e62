// Flash attention forward for sm_100a (causal or full, MHA/GQA, head_dim 64 or 128, bf16 in/out).
//
// One CTA handles two tiles of 128 query rows of one (batch, head) or, with HALVES, one tile whose keys are halved.  Warp 0
// streams the Q tiles once and K/V blocks of 128 rows through a shared-memory ring with TMA; warp 1 issues tcgen05.mma; warps
// 2-5 and 6-9 are the softmax of one tile each: a thread owns one query row, reads its 128 columns of S = Q K^T from TMEM, and
// writes the probabilities back over them as bf16, from where O += P V takes its A operand.  S, P and O never leave tensor
// memory.
//
// What bounds it: a block of 128 x 128 scores costs 16384 exponentials (1024 cycles of the SM's special-function
// units) and two products (1024 cycles of the tensor cores at head_dim 128).  Both would be busy all the time if a
// tile's softmax could overlap its own products, which depend on it; with two tiles in turn the tensor cores work on
// one while the exponentials of the other are taken.  A thread per row needs no exchange of maxima between warps.
// O is rescaled in TMEM only when some row's maximum has moved by enough to matter.
// Causal, 32 heads of 128: 4096 rows 140 us (980 TFLOP/s), 16384 rows 1.88 ms (1170); with one tile per CTA and its
// columns split among four warp groups, all in step with each other, 224 us and 2.63 ms.
//
// HALVES is for grids that leave SMs without a pair of tiles: the two softmax groups take the first and the second 64 keys of
// every block as two independent sums over the same tile, which meet at the end.  Two buffers for the scores of a half let S
// run ahead of P V, so a half waits for neither its own products nor the other half.  4 heads of 128, 4096 causal rows: 47 us,
// with two tiles per CTA on half the SMs 68, and 51 with one tile whose columns were split among four warp groups in step with
// each other.  The MMA warp must issue from uniform code for that (see elect_one): from one lane of a divergent branch every
// product cost about 120 cycles, whatever its size, and the same case took 59 us.
// All waits are bounded and report through the status word.
#include "common.cuh"

namespace jpb {

constexpr int ATT_BM = 128;   // query rows per tile, two tiles per CTA
constexpr int ATT_BN = 128;   // kv rows per block
constexpr int ATT_THREADS = 64 + 2 * 128;

struct AttnParams {
  int B, Sq, Sk, H, Hkv;
  int causal;
  int items;          // CTAs per (batch, head)
  int head_major;     // order of the CTAs: all of a head first, or the longest of every head first
  float scale;
  __nv_bfloat16* o;   // [B, Sq, H, D]
  float* lse;         // [B, H, Sq]
  int* status;
};

template <int D, bool HALVES>
struct AttnSmem {
  static constexpr int TILE = 128 * 64 * 2;           // one [128 rows x 64 elements] swizzled block, 16 KiB
  static constexpr int DB = D / 64;                   // 64-element blocks along head_dim
  static constexpr int NS = D == 128 ? (HALVES ? 3 : 2) : 4;   // K/V stages
  static constexpr int T_BYTES = DB * TILE;           // a tile of Q, K or V
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = OFF_Q + (HALVES ? 1 : 2) * T_BYTES;
  static constexpr int OFF_V = OFF_K + NS * T_BYTES;
  static constexpr int OFF_BAR = OFF_V + NS * T_BYTES;
  static constexpr int OFF_ML = OFF_Q;                // (maximum, sum) of half rows, once nothing reads Q any more
  static constexpr int TOTAL = OFF_BAR + 256 + 1024;
  static_assert(TOTAL <= 227 * 1024, "");
};

// barriers: Q per tile, K/V full and empty per stage, S ready / P ready / O complete per tile; with HALVES, S and P of half t
// have two of each (t + 2 * parity of the block), and BAR_PV counts the products P V of a half
enum { BAR_Q = 0, BAR_KF = 2, BAR_VF = 6, BAR_KE = 10, BAR_VE = 14, BAR_SF = 18, BAR_PF = 22, BAR_O = 26, BAR_PV = 28, BAR_N = 30 };

__host__ __device__ __forceinline__ int att_blocks(const AttnParams& p, int m0) {  // kv blocks that tile m0 sees
  if (m0 >= p.Sq) return 0;
  int n = (p.Sk + ATT_BN - 1) / ATT_BN;
  if (p.causal) {
    const int last = (m0 + ATT_BM - 1 + (p.Sk - p.Sq)) / ATT_BN + 1;
    n = last < n ? last : n;
    if (n < 1) n = 1;
  }
  return n;
}

// The softmax warps' 256 threads meet: named barrier 1.
__device__ __forceinline__ void softmax_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

template <int D, bool HALVES>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attention_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  using L = AttnSmem<D, HALVES>;
  constexpr int NS = L::NS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + BAR_N);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float2* row_ml = reinterpret_cast<float2*>(smem + L::OFF_ML);   // HALVES: [2][128] maximum and sum of each half of a row
  constexpr int BN = HALVES ? ATT_BN / 2 : ATT_BN;                // kv rows of a block that one softmax thread sees

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int heads = p.H * p.B;
  const int bh = p.head_major ? blockIdx.x / p.items : blockIdx.x % heads;
  const int item = p.items - 1 - (p.head_major ? blockIdx.x % p.items : blockIdx.x / heads);  // longest causal tiles first
  const int h = bh % p.H, b = bh / p.H;
  const int hk = h / (p.H / p.Hkv);
  const int m0 = item * (HALVES ? 1 : 2) * ATT_BM;
  const int n0 = att_blocks(p, m0), n1 = HALVES ? n0 : att_blocks(p, m0 + ATT_BM);  // n1 is 0 or at least n0
  const int n_blocks = n0 > n1 ? n0 : n1;

  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&bar[BAR_Q + t], 1);
      for (int b = 0; b < 4; b += 2) {
        mbar_init(&bar[BAR_SF + t + b], 1);
        mbar_init(&bar[BAR_PF + t + b], 4);   // one arrival per softmax warp of the tile
      }
      mbar_init(&bar[BAR_O + t], 1);
      mbar_init(&bar[BAR_PV + t], 1);
    }
    for (int s = 0; s < NS; ++s) {
      mbar_init(&bar[BAR_KF + s], 1);
      mbar_init(&bar[BAR_VF + s], 1);
      mbar_init(&bar[BAR_KE + s], 1);
      mbar_init(&bar[BAR_VE + s], 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // columns: S of tile 0 and 1 (P, packed bf16, over the first 64 of each), O of tile 0 and 1; with HALVES, the 128 columns of
  // a half are two buffers of 64 for S (P over the first 32 of each)
  const uint32_t tmem_o = tmem_base + 256;

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------- TMA producer -------------------------------------------
      uint32_t armed = 0, armed_phase = 0;  // indexed by barrier id, for draining after an abort
      auto arm = [&](int id, uint32_t ph, uint32_t bytes) {
        mbar_expect_tx(&bar[id], bytes);
        armed |= 1u << id;
        armed_phase = (armed_phase & ~(1u << id)) | (ph << id);
      };
      auto load_q = [&](int t) {
        arm(BAR_Q + t, 0, L::T_BYTES);
#pragma unroll
        for (int d = 0; d < L::DB; ++d)
          tma_load_4d(smem + L::OFF_Q + t * L::T_BYTES + d * L::TILE, &map_q, &bar[BAR_Q + t], d * 64, h, m0 + t * ATT_BM, b);
      };
      auto load_kv = [&](const CUtensorMap* map, int full, int empty, int off, int j) -> bool {
        const int s = j % NS;
        const uint32_t ph = (j / NS) & 1;
        if (!mbar_wait_bounded(&bar[empty + s], ph ^ 1, abort_flag, p.status)) return false;
        arm(full + s, ph, L::T_BYTES);
#pragma unroll
        for (int d = 0; d < L::DB; ++d)
          tma_load_4d(smem + off + s * L::T_BYTES + d * L::TILE, map, &bar[full + s], d * 64, hk, j * ATT_BN, b);
        return true;
      };
      load_q(0);
      bool ok = load_kv(&map_k, BAR_KF, BAR_KE, L::OFF_K, 0);
      if (!HALVES && n1 > 0) load_q(1);
      // K runs one block ahead of V: a K stage is free as soon as S of its block has been computed (early), a V
      // stage only after P V of its block (late)
      for (int j = 0; j < n_blocks && ok; ++j) {
        if (j + 1 < n_blocks && !load_kv(&map_k, BAR_KF, BAR_KE, L::OFF_K, j + 1)) { ok = false; break; }
        if (!load_kv(&map_v, BAR_VF, BAR_VE, L::OFF_V, j)) { ok = false; break; }
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        for (int id = 0; id < BAR_KE; ++id) {
          if (!(armed & (1u << id))) continue;
          while (!mbar_try_wait(&bar[id], (armed_phase >> id) & 1) && globaltimer_ns() - t0 < wait_budget_ns()) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------- MMA issuer ------------------------------------------------
    // (all lanes walk the loop; one elected lane issues: see elect_one)
    constexpr uint32_t idesc_s = make_idesc_bf16(ATT_BM, BN, 0, 0);
    constexpr uint32_t idesc_pv = make_idesc_bf16(ATT_BM, D, 0, 1);
    const SmemDesc dq_ = make_smem_desc2(smem_u32(smem + L::OFF_Q), 16, 1024);
    const SmemDesc dk_ = make_smem_desc2(smem_u32(smem + L::OFF_K), 16, 1024);
    const SmemDesc dv_ = make_smem_desc2(smem_u32(smem + L::OFF_V), L::TILE, 1024);  // MN-major, 64-wide d blocks
    constexpr uint32_t T16 = L::T_BYTES >> 4;
    constexpr uint32_t KV_HALF = 64 * 128 >> 4;   // 64 kv rows further in a swizzled block of K or V
    // S of tile t, block j.  HALVES: of half t, into one of two buffers.
    auto issue_s = [&](int t, int j) {
      const uint32_t q_lo = dq_.lo + (HALVES ? 0 : t * T16), k_lo = dk_.lo + (j % NS) * T16 + (HALVES ? t * KV_HALF : 0);
      const int buf = HALVES ? (j & 1) : 0;
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        const uint32_t off = ((k >> 2) * L::TILE + (k & 3) * 32) >> 4;
        umma_bf16_ss2(tmem_base + t * ATT_BN + buf * 64, q_lo + off, dq_.hi, k_lo + off, dk_.hi, idesc_s, k != 0);
      }
      umma_commit(&bar[BAR_SF + t + 2 * buf]);
    };
    auto issue_pv = [&](int t, int j) {
      const uint32_t p_col = tmem_base + t * ATT_BN + (HALVES ? (j & 1) * 64 : 0);
      const uint32_t v_lo = dv_.lo + (j % NS) * T16 + (HALVES ? t * KV_HALF : 0);
#pragma unroll
      for (int k = 0; k < BN / 16; ++k)   // 16 kv rows = 8 packed columns of P per step
        umma_bf16_ts2(tmem_o + t * D, p_col + k * 8, v_lo + k * 128, dv_.hi, idesc_pv, (j | k) != 0);
    };
    auto wait = [&](int id, uint32_t phase) -> bool {
      const bool done = mbar_wait_bounded_warp(&bar[id], phase & 1, abort_flag, p.status);
      tc_fence_after();
      return done;
    };
    bool ok = wait(BAR_Q, 0) && wait(BAR_KF, 0);
    if constexpr (HALVES) {
      // S runs up to two blocks ahead of P V, so that a half's next scores are there when its softmax asks for them
      for (int j = 0; j < 2 && j < n_blocks && ok; ++j) {
        if (j > 0 && !wait(BAR_KF + j % NS, j / NS)) { ok = false; break; }
        if (elect_one()) {
          issue_s(0, j);
          issue_s(1, j);
          umma_commit(&bar[BAR_KE + j % NS]);
        }
        __syncwarp();
      }
      for (int j = 0; j < n_blocks && ok; ++j) {
        if (!wait(BAR_VF + j % NS, j / NS)) { ok = false; break; }
        const bool more = j + 2 < n_blocks;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (!wait(BAR_PF + t + 2 * (j & 1), j >> 1)) { ok = false; break; }
          if (elect_one()) {
            issue_pv(t, j);
            umma_commit(&bar[BAR_PV + t]);
            if (j + 1 == n_blocks) umma_commit(&bar[BAR_O + t]);
            if (t == 1) umma_commit(&bar[BAR_VE + j % NS]);
          }
          __syncwarp();
          if (!more) continue;
          if (t == 0 && !wait(BAR_KF + (j + 2) % NS, (j + 2) / NS)) { ok = false; break; }
          if (elect_one()) {
            issue_s(t, j + 2);   // over the P that P V of this block reads: the tensor core runs them in the order of issue
            if (t == 1) umma_commit(&bar[BAR_KE + (j + 2) % NS]);
          }
          __syncwarp();
        }
      }
    } else {
      if (ok) {
        if (elect_one()) issue_s(0, 0);
        __syncwarp();
        if (n1 > 0) {
          ok = wait(BAR_Q + 1, 0);
          if (ok && elect_one()) issue_s(1, 0);
          __syncwarp();
        }
        if (elect_one()) umma_commit(&bar[BAR_KE]);
        __syncwarp();
      }
      for (int j = 0; j < n_blocks && ok; ++j) {
        if (!wait(BAR_VF + j % NS, j / NS)) { ok = false; break; }
        if (j + 1 < n_blocks && !wait(BAR_KF + (j + 1) % NS, (j + 1) / NS)) { ok = false; break; }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int n = t ? n1 : n0;
          if (j >= n) continue;
          if (!wait(BAR_PF + t, j)) { ok = false; break; }
          if (elect_one()) {
            issue_pv(t, j);
            // The next S overwrites the P that this product reads: the tensor core runs them in the order of issue.
            if (j + 1 < n) issue_s(t, j + 1);
            else umma_commit(&bar[BAR_O + t]);
          }
          __syncwarp();
        }
        if (!ok) break;
        if (elect_one()) {
          umma_commit(&bar[BAR_VE + j % NS]);
          if (j + 1 < n_blocks) umma_commit(&bar[BAR_KE + (j + 1) % NS]);
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------- softmax / correction / epilogue -----------------------------
    const int t = (warp - 2) >> 2;              // tile, or half of every kv block
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;          // row within the tile == TMEM lane
    const int mt = m0 + (HALVES ? 0 : t * ATT_BM);
    const int qi = mt + r;                      // query index
    const int n = t ? n1 : n0;
    const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
    const uint32_t t_s0 = tmem_base + t * ATT_BN + lane_addr, t_o = tmem_o + t * D + lane_addr;
    const float sl2 = p.scale * 1.4426950408889634f;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n && ok; ++j) {
      const int buf = HALVES ? (j & 1) : 0;
      const uint32_t t_s = t_s0 + buf * 64;
      if (!mbar_wait_bounded_warp(&bar[BAR_SF + t + 2 * buf], (HALVES ? j >> 1 : j) & 1, abort_flag, p.status)) { ok = false; break; }
      tc_fence_after();
      float sv[BN];
      {
        uint32_t a[BN / 32][32];
#pragma unroll
        for (int c = 0; c < BN / 32; ++c) tmem_ld_32x32(t_s + c * 32, a[c]);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < BN; ++i) sv[i] = __uint_as_float(a[i >> 5][i & 31]);
      }
      const int kv0 = j * ATT_BN + (HALVES ? t * BN : 0);
      const bool need_mask = (p.causal && kv0 + BN - 1 > mt + (p.Sk - p.Sq)) || (kv0 + BN > p.Sk);
      if (need_mask) {
        const int limit = (p.causal ? min(qi + (p.Sk - p.Sq), p.Sk - 1) : p.Sk - 1) - kv0;  // last visible column
#pragma unroll
        for (int i = 0; i < BN; ++i)
          if (i > limit) sv[i] = -INFINITY;
      }
      float mx4[4] = {sv[0], sv[1], sv[2], sv[3]};
#pragma unroll
      for (int i = 4; i < BN; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], sv[i]);
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // Lazy rescaling: the reference maximum of a row only moves when the new maximum exceeds it by more than
      // 8 in log2 units (P then stays below 2^8, harmless in fp32 sums and bf16 P), so the read-scale-write
      // pass over O in TMEM, a chain of TMEM round trips, runs in a few blocks instead of nearly all of them.
      const float m_cand = fmaxf(m_run, mx);
      const bool bump = (m_cand - m_run) * sl2 > 8.f;   // also true for the first finite maximum (m_run = -inf)
      const float m_new = bump ? m_cand : m_run;
      const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
      const float neg = -m_use * sl2;
      if (__any_sync(0xffffffffu, bump)) {
        const float alpha = bump ? exp2f((m_run - m_use) * sl2) : 1.f;  // 0 when m_run = -inf
        l_run *= alpha;
        // Without HALVES, S of this block was issued after P V of the last one, so O is complete up to there; with it, only
        // up to the one before (P V of this block waits for this thread).
        if (HALVES && j > 0) {
          if (!mbar_wait_bounded_warp(&bar[BAR_PV + t], (j - 1) & 1, abort_flag, p.status)) { ok = false; break; }
          tc_fence_after();
        }
        if (j > 0) {
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t w[16];
            tmem_ld_32x16(t_o + c * 16, w);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * alpha);
            tmem_st_32x16(t_o + c * 16, w);
          }
        }
      }
      m_run = m_new;
      float rs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float x = exp2f(fmaf(sv[c * 32 + i], sl2, neg)), y = exp2f(fmaf(sv[c * 32 + i + 1], sl2, neg));
          rs[(i >> 1) & 3] += x + y;
          w[i >> 1] = pack_bf16(x, y);
        }
        tmem_st_32x16(t_s + c * 16, w);   // row r is lane r, kv columns (2c, 2c+1) share the 32-bit column c
      }
      l_run += (rs[0] + rs[1]) + (rs[2] + rs[3]);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar[BAR_PF + t + 2 * buf]);
    }
    const bool row_ok = qi < p.Sq;
    __nv_bfloat16* orow = p.o + ((size_t(b) * p.Sq + qi) * p.H + h) * D;
    auto store8 = [&](__nv_bfloat16* dst, const float (&x)[8]) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
    };
    if constexpr (HALVES) {
      // The two halves of a row: (m, l) meet in shared memory, O of both is in the tensor memory lanes that either thread
      // can read; half t writes columns [t * D / 2, (t + 1) * D / 2).
      // (all 256 threads come to the barrier, whether their waits ran out or not; by then nothing reads Q any more)
      ok = ok && n > 0 && mbar_wait_bounded_warp(&bar[BAR_O], 0, abort_flag, p.status) &&
           mbar_wait_bounded_warp(&bar[BAR_O + 1], 0, abort_flag, p.status);
      if (ok) row_ml[t * 128 + r] = make_float2(m_run, l_run);
      softmax_sync();
      if (ok) {
        tc_fence_after();
        const float2 ml0 = row_ml[r], ml1 = row_ml[128 + r];
        const float m = fmaxf(ml0.x, ml1.x);
        // a half without a maximum was summed against the reference 0, and is empty where the other half has one
        const float a0 = m == -INFINITY ? 1.f : ml0.x == -INFINITY ? 0.f : exp2f((ml0.x - m) * sl2);
        const float a1 = m == -INFINITY ? 1.f : ml1.x == -INFINITY ? 0.f : exp2f((ml1.x - m) * sl2);
        const float l = a0 * ml0.y + a1 * ml1.y;
        const float inv = l > 0.f ? 1.f / l : 0.f;
        const float f0 = a0 * inv, f1 = a1 * inv;
        const uint32_t t_o0 = tmem_o + lane_addr + t * (D / 2);
#pragma unroll
        for (int c = 0; c < D / 2; c += 32) {
          uint32_t w0[32], w1[32];
          tmem_ld_32x32(t_o0 + c, w0);
          tmem_ld_32x32(t_o0 + D + c, w1);
          tc_wait_ld();
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              float x[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) x[e] = fmaf(__uint_as_float(w0[i + e]), f0, __uint_as_float(w1[i + e]) * f1);
              store8(orow + t * (D / 2) + c + i, x);
            }
          }
        }
        if (row_ok && t == 0) p.lse[(size_t(b) * p.H + h) * p.Sq + qi] = l > 0.f ? m * p.scale + logf(l) : -INFINITY;
      }
    } else if (ok && n > 0 && mbar_wait_bounded_warp(&bar[BAR_O + t], 0, abort_flag, p.status)) {
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t w[32];
        tmem_ld_32x32(t_o + c * 32, w);
        tc_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(w[i + e]) * inv;
            store8(orow + c * 32 + i, x);
          }
        }
      }
      if (row_ok) p.lse[(size_t(b) * p.H + h) * p.Sq + qi] = (l_run > 0.f) ? m_run * p.scale + logf(l_run) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// 4-D map over a [B, S, Hn, D] bf16 tensor with a box of [128 rows of S] x [64 elements of D]
static int make_bshd_map(CUtensorMap* out, const void* base, int B, int S, int Hn, int D) {
  uint64_t dims[4] = {uint64_t(D), uint64_t(Hn), uint64_t(S), uint64_t(B)};
  uint64_t strides[3] = {uint64_t(D) * 2, uint64_t(Hn) * D * 2, uint64_t(S) * Hn * D * 2};
  uint32_t box[4] = {64, 1, 128, 1};
  return jpb_make_tensor_map(out, base, 2, 4, dims, strides, box, 1);
}

template <int D, bool HALVES>
static int launch_attn_fwd(const void* q, const void* k, const void* v, const AttnParams& p, cudaStream_t stream) {
  using L = AttnSmem<D, HALVES>;
  CUtensorMap mq, mk, mv;
  int rc = make_bshd_map(&mq, q, p.B, p.Sq, p.H, D);
  if (rc) return rc;
  rc = make_bshd_map(&mk, k, p.B, p.Sk, p.Hkv, D);
  if (rc) return rc;
  rc = make_bshd_map(&mv, v, p.B, p.Sk, p.Hkv, D);
  if (rc) return rc;
  auto kernel = attention_fwd_kernel<D, HALVES>;
  static const cudaError_t configured = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
  if (configured != cudaSuccess) return int(configured);
  kernel<<<p.items * p.H * p.B, ATT_THREADS, L::TOTAL, stream>>>(mq, mk, mv, p);
  return int(cudaGetLastError());
}

// Which of the two forms?  Estimated times: two tiles in turn take 1.93 us a block at head_dim 128 (1.78 at 64), the halves of
// one tile 1.36 (1.08), and a CTA 4 us to start and end.  Where tiles differ in length (causal), the long ones start first and
// the short ones fill the gaps but for 5 %; else the CTAs run in whole rounds.  Of 179 grids measured in both forms (head_dim
// 64 and 128, 1 to 64 heads, 1 to 16384 rows) the estimate's choice is more than 3 % slower than the other in two, by 5 %.
// Two rounds of halves are slower than one of pairs: 25 heads of 128, 1024 rows, all keys: 32 against 25 us; causal 19 against
// 24; 16 x 8 heads of 512 causal rows 32 against 26.
// With a single block and tile there is nothing to overlap; which form is faster goes by 0.4 us either way.
static bool halves_are_faster(const AttnParams& p, int D) {
  if (p.Sk <= ATT_BN && p.Sq <= ATT_BM) return false;
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    return cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 148;
  }();
  auto time = [&](int rows, double step) {
    const long long heads = (long long)p.B * p.H;
    long long ctas = 0, total = 0;
    int most = 0, least = 1 << 30;
    for (int m0 = 0; m0 < p.Sq; m0 += rows, ++ctas) {
      const int a = att_blocks(p, m0), b = rows > ATT_BM ? att_blocks(p, m0 + ATT_BM) : 0, n = a > b ? a : b;
      total += n;
      most = n > most ? n : most;
      least = n < least ? n : least;
    }
    const double ends = 4.0, longest = most * step + ends;
    if (least == most) return double((ctas * heads + sms - 1) / sms) * longest;
    const double shared = 1.05 * heads * (total * step + ends * ctas) / sms;
    return shared > longest ? shared : longest;
  };
  return time(ATT_BM, D == 128 ? 1.36 : 1.08) < time(2 * ATT_BM, D == 128 ? 1.93 : 1.78);
}

}  // namespace jpb

// Does this call take halves of one tile per CTA (1) or two tiles (0)?
JPB_API int jpb_attention_fwd_halves(int B, int Sq, int Sk, int H, int D, int causal) {
  jpb::AttnParams p = {};
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.H = H; p.causal = causal;
  return jpb::halves_are_faster(p, D);
}

// q: [B,Sq,H,D], k/v: [B,Sk,Hkv,D] contiguous bf16; o like q; lse: [B,H,Sq] fp32 (natural log).
JPB_API int jpb_attention_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Sq, int Sk, int H,
                              int Hkv, int D, int causal, float scale, void* stream) {
  using namespace jpb;
  if (H % Hkv != 0 || (D != 64 && D != 128)) return -JPB_ERR_BAD_ARGUMENT;
  AttnParams p;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.H = H; p.Hkv = Hkv; p.causal = causal; p.scale = scale;
  p.o = static_cast<__nv_bfloat16*>(o); p.lse = lse; p.status = jpb_status_device_ptr();
  const bool halves = halves_are_faster(p, D);
  p.items = halves ? (Sq + ATT_BM - 1) / ATT_BM : (Sq + 2 * ATT_BM - 1) / (2 * ATT_BM);
  // Longest tiles of all heads first balances the last wave; once K and V of all heads no longer fit in half of the L2
  // cache the CTAs in flight should share theirs, so a head's tiles go together.
  p.head_major = (long long)B * Sk * Hkv * D * 4 > 64ll * 1024 * 1024;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (halves) return D == 128 ? launch_attn_fwd<128, true>(q, k, v, p, s) : launch_attn_fwd<64, true>(q, k, v, p, s);
  return D == 128 ? launch_attn_fwd<128, false>(q, k, v, p, s) : launch_attn_fwd<64, false>(q, k, v, p, s);
}
