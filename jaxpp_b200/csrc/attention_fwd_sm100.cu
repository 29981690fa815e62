// Flash attention forward for sm_100a (causal or full, MHA/GQA, head_dim 64 or 128, bf16 in/out).
//
// One CTA handles two tiles of 128 query rows of one (batch, head).  Warp 0 streams both Q tiles once and K/V blocks of
// 128 rows through a shared-memory ring with TMA; warp 1 issues tcgen05.mma; warps 2-5 and 6-9 are the softmax of one
// tile each: a thread owns one query row, reads its 128 columns of S = Q K^T from TMEM, and writes the probabilities
// back over them as bf16, from where O += P V takes its A operand.  S, P and O never leave tensor memory.
//
// What bounds it: a block of 128 x 128 scores costs 16384 exponentials (1024 cycles of the SM's special-function
// units) and two products (1024 cycles of the tensor cores at head_dim 128).  Both would be busy all the time if a
// tile's softmax could overlap its own products, which depend on it; with two tiles in turn the tensor cores work on
// one while the exponentials of the other are taken.  A thread per row needs no exchange of maxima between warps.
// O is rescaled in TMEM only when some row's maximum has moved by enough to matter.
// Causal, 32 heads of 128: 4096 rows 148 us (927 TFLOP/s), 16384 rows 2.02 ms (1089); with one tile per CTA and its
// columns split among four warp groups, all in step with each other, 226 us and 2.63 ms.
// All waits are bounded and report through the status word.
#include "common.cuh"

namespace jpb {

constexpr int ATT_BM = 128;   // query rows per tile, two tiles per CTA
constexpr int ATT_BN = 128;   // kv rows per block
constexpr int ATT_THREADS = 64 + 2 * 128;

struct AttnParams {
  int B, Sq, Sk, H, Hkv;
  int causal;
  int pairs;          // CTAs per (batch, head)
  int head_major;     // order of the CTAs: all of a head first, or the longest of every head first
  float scale;
  __nv_bfloat16* o;   // [B, Sq, H, D]
  float* lse;         // [B, H, Sq]
  int* status;
};

template <int D>
struct AttnSmem {
  static constexpr int TILE = 128 * 64 * 2;           // one [128 rows x 64 elements] swizzled block, 16 KiB
  static constexpr int DB = D / 64;                   // 64-element blocks along head_dim
  static constexpr int NS = D == 128 ? 2 : 4;         // K/V stages
  static constexpr int T_BYTES = DB * TILE;           // a tile of Q, K or V
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = OFF_Q + 2 * T_BYTES;
  static constexpr int OFF_V = OFF_K + NS * T_BYTES;
  static constexpr int OFF_BAR = OFF_V + NS * T_BYTES;
  static constexpr int TOTAL = OFF_BAR + 256 + 1024;
};

// barriers: Q per tile, K/V full and empty per stage, S ready / P ready / O complete per tile
enum { BAR_Q = 0, BAR_KF = 2, BAR_VF = 6, BAR_KE = 10, BAR_VE = 14, BAR_SF = 18, BAR_PF = 20, BAR_O = 22, BAR_N = 24 };

__device__ __forceinline__ int att_blocks(const AttnParams& p, int m0) {  // kv blocks that tile m0 sees
  if (m0 >= p.Sq) return 0;
  int n = (p.Sk + ATT_BN - 1) / ATT_BN;
  if (p.causal) {
    const int last = (m0 + ATT_BM - 1 + (p.Sk - p.Sq)) / ATT_BN + 1;
    n = last < n ? last : n;
    if (n < 1) n = 1;
  }
  return n;
}

template <int D>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attention_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  using L = AttnSmem<D>;
  constexpr int NS = L::NS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + BAR_N);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int heads = p.H * p.B;
  const int bh = p.head_major ? blockIdx.x / p.pairs : blockIdx.x % heads;
  const int pair = p.pairs - 1 - (p.head_major ? blockIdx.x % p.pairs : blockIdx.x / heads);  // longest causal tiles first
  const int h = bh % p.H, b = bh / p.H;
  const int hk = h / (p.H / p.Hkv);
  const int m0 = pair * 2 * ATT_BM;
  const int n0 = att_blocks(p, m0), n1 = att_blocks(p, m0 + ATT_BM);  // n1 is 0 or at least n0
  const int n_blocks = n0 > n1 ? n0 : n1;

  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&bar[BAR_Q + t], 1);
      mbar_init(&bar[BAR_SF + t], 1);
      mbar_init(&bar[BAR_PF + t], 4);   // one arrival per softmax warp of the tile
      mbar_init(&bar[BAR_O + t], 1);
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
  // columns: S of tile 0 and 1 (P, packed bf16, over the first 64 of each), O of tile 0 and 1
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
      if (n1 > 0) load_q(1);
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
    if (lane == 0) {
      // ------------------------------------- MMA issuer ------------------------------------------------
      constexpr uint32_t idesc_s = make_idesc_bf16(ATT_BM, ATT_BN, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc_bf16(ATT_BM, D, 0, 1);
      const SmemDesc dq_ = make_smem_desc2(smem_u32(smem + L::OFF_Q), 16, 1024);
      const SmemDesc dk_ = make_smem_desc2(smem_u32(smem + L::OFF_K), 16, 1024);
      const SmemDesc dv_ = make_smem_desc2(smem_u32(smem + L::OFF_V), L::TILE, 1024);  // MN-major, 64-wide d blocks
      constexpr uint32_t T16 = L::T_BYTES >> 4;
      auto issue_s = [&](int t, int j) {   // S of tile t, block j
        const uint32_t q_lo = dq_.lo + t * T16, k_lo = dk_.lo + (j % NS) * T16;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = ((k >> 2) * L::TILE + (k & 3) * 32) >> 4;
          umma_bf16_ss2(tmem_base + t * ATT_BN, q_lo + off, dq_.hi, k_lo + off, dk_.hi, idesc_s, k != 0);
        }
        umma_commit(&bar[BAR_SF + t]);
      };
      bool ok = mbar_wait_bounded(&bar[BAR_Q], 0, abort_flag, p.status) && mbar_wait_bounded(&bar[BAR_KF], 0, abort_flag, p.status);
      if (ok) {
        tc_fence_after();
        issue_s(0, 0);
        if (n1 > 0) {
          ok = mbar_wait_bounded(&bar[BAR_Q + 1], 0, abort_flag, p.status);
          if (ok) { tc_fence_after(); issue_s(1, 0); }
        }
        umma_commit(&bar[BAR_KE]);
      }
      for (int j = 0; j < n_blocks && ok; ++j) {
        const int s = j % NS;
        if (!mbar_wait_bounded(&bar[BAR_VF + s], (j / NS) & 1, abort_flag, p.status)) { ok = false; break; }
        if (j + 1 < n_blocks && !mbar_wait_bounded(&bar[BAR_KF + (j + 1) % NS], ((j + 1) / NS) & 1, abort_flag, p.status)) { ok = false; break; }
        const uint32_t v_lo = dv_.lo + s * T16;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int n = t ? n1 : n0;
          if (j >= n) continue;
          if (!mbar_wait_bounded(&bar[BAR_PF + t], j & 1, abort_flag, p.status)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < ATT_BN / 16; ++k)   // 16 kv rows = 8 packed columns of P per step
            umma_bf16_ts2(tmem_o + t * D, tmem_base + t * ATT_BN + k * 8, v_lo + k * 128, dv_.hi, idesc_pv, (j | k) != 0);
          // The next S overwrites the P that this product reads: the tensor core runs them in the order of issue.
          if (j + 1 < n) issue_s(t, j + 1);
          else umma_commit(&bar[BAR_O + t]);
        }
        if (!ok) break;
        umma_commit(&bar[BAR_VE + s]);
        if (j + 1 < n_blocks) umma_commit(&bar[BAR_KE + (j + 1) % NS]);
      }
    }
  } else {
    // ------------------------------------- softmax / correction / epilogue -----------------------------
    const int t = (warp - 2) >> 2;              // tile
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;          // row within the tile == TMEM lane
    const int mt = m0 + t * ATT_BM;
    const int qi = mt + r;                      // query index
    const int n = t ? n1 : n0;
    const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
    const uint32_t t_s = tmem_base + t * ATT_BN + lane_addr, t_o = tmem_o + t * D + lane_addr;
    const float sl2 = p.scale * 1.4426950408889634f;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n && ok; ++j) {
      if (!mbar_wait_bounded_warp(&bar[BAR_SF + t], j & 1, abort_flag, p.status)) { ok = false; break; }
      tc_fence_after();
      float sv[ATT_BN];
      {
        uint32_t a[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, a[c]);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < ATT_BN; ++i) sv[i] = __uint_as_float(a[i >> 5][i & 31]);
      }
      const int kv0 = j * ATT_BN;
      const bool need_mask = (p.causal && kv0 + ATT_BN - 1 > mt + (p.Sk - p.Sq)) || (kv0 + ATT_BN > p.Sk);
      if (need_mask) {
        const int limit = (p.causal ? min(qi + (p.Sk - p.Sq), p.Sk - 1) : p.Sk - 1) - kv0;  // last visible column
#pragma unroll
        for (int i = 0; i < ATT_BN; ++i)
          if (i > limit) sv[i] = -INFINITY;
      }
      float mx4[4] = {sv[0], sv[1], sv[2], sv[3]};
#pragma unroll
      for (int i = 4; i < ATT_BN; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], sv[i]);
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
        if (j > 0) {   // S of this block was issued after P V of the last one, so O is complete up to there
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
      for (int c = 0; c < 4; ++c) {
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
      if (lane == 0) mbar_arrive(&bar[BAR_PF + t]);
    }
    if (ok && n > 0 && mbar_wait_bounded_warp(&bar[BAR_O + t], 0, abort_flag, p.status)) {
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const bool row_ok = qi < p.Sq;
      __nv_bfloat16* orow = p.o + ((size_t(b) * p.Sq + qi) * p.H + h) * D;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t w[32];
        tmem_ld_32x32(t_o + c * 32, w);
        tc_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(w[i]) * inv, __uint_as_float(w[i + 1]) * inv);
            v.y = pack_bf16(__uint_as_float(w[i + 2]) * inv, __uint_as_float(w[i + 3]) * inv);
            v.z = pack_bf16(__uint_as_float(w[i + 4]) * inv, __uint_as_float(w[i + 5]) * inv);
            v.w = pack_bf16(__uint_as_float(w[i + 6]) * inv, __uint_as_float(w[i + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + i) = v;
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

template <int D>
static int launch_attn_fwd(const void* q, const void* k, const void* v, const AttnParams& p, cudaStream_t stream) {
  using L = AttnSmem<D>;
  CUtensorMap mq, mk, mv;
  int rc = make_bshd_map(&mq, q, p.B, p.Sq, p.H, D);
  if (rc) return rc;
  rc = make_bshd_map(&mk, k, p.B, p.Sk, p.Hkv, D);
  if (rc) return rc;
  rc = make_bshd_map(&mv, v, p.B, p.Sk, p.Hkv, D);
  if (rc) return rc;
  auto kernel = attention_fwd_kernel<D>;
  static const cudaError_t configured = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
  if (configured != cudaSuccess) return int(configured);
  kernel<<<p.pairs * p.H * p.B, ATT_THREADS, L::TOTAL, stream>>>(mq, mk, mv, p);
  return int(cudaGetLastError());
}

}  // namespace jpb

// q: [B,Sq,H,D], k/v: [B,Sk,Hkv,D] contiguous bf16; o like q; lse: [B,H,Sq] fp32 (natural log).
JPB_API int jpb_attention_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Sq, int Sk, int H,
                              int Hkv, int D, int causal, float scale, void* stream) {
  using namespace jpb;
  if (H % Hkv != 0 || (D != 64 && D != 128)) return -JPB_ERR_BAD_ARGUMENT;
  AttnParams p;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.H = H; p.Hkv = Hkv; p.causal = causal; p.scale = scale;
  p.o = static_cast<__nv_bfloat16*>(o); p.lse = lse; p.status = jpb_status_device_ptr();
  p.pairs = (Sq + 2 * ATT_BM - 1) / (2 * ATT_BM);
  // Longest tiles of all heads first balances the last wave; once K and V of all heads no longer fit in half of the L2
  // cache the CTAs in flight should share theirs, so a head's tiles go together.
  p.head_major = (long long)B * Sk * Hkv * D * 4 > 64ll * 1024 * 1024;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return D == 128 ? launch_attn_fwd<128>(q, k, v, p, s) : launch_attn_fwd<64>(q, k, v, p, s);
}
