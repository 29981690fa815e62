// Mixture-of-experts layer on one GPU, around its expert GEMMs: routing (forward and backward), the slot of every
// (token, pick), and the movement of rows between token order and expert slots with its transposes.
//
// What bounds them: HBM for the row movement, one pass each -- a slot's row is read (or zeros written) and stored once,
// a token's picks are summed while they are read, and the gradient of the combination reads the expert output and the
// token gradient once for both of its results.  The routing kernels touch a few hundred kilobytes and are bound by
// latency: registers instead of local arrays, shuffles instead of shared-memory atomics.
#include "common.cuh"

namespace jpb {

constexpr int MOE_MAX_E = 64, MOE_MAX_K = 8;

template <typename T> struct Row;  // 16 bytes of a row as floats
template <> struct Row<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void load(const float* p, float (&f)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&f)[4]) { *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]); }
};
template <> struct Row<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&f)[8]) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 u = unpack_bf16(w[i]); f[2 * i] = u.x; f[2 * i + 1] = u.y; }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&f)[8]) {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
  }
};
__device__ __forceinline__ float as_float(float v) { return v; }
__device__ __forceinline__ float as_float(__nv_bfloat16 v) { return __bfloat162float(v); }

// ---------------------------------------------------------------------------------------------------------
// Router: softmax over the expert logits, top-k pick, weights renormalised over the picks, and the two
// per-expert statistics of the load-balancing loss (sum of probabilities, number of picks) in one pass.
// One thread per token, its probabilities in registers: EP is E rounded up to a power of two.  A CTA leaves the sums of
// its tokens' probabilities in its own row of `part` (may be absent), so that the loss is a sum in a fixed order: the same
// bits on every run.  The picks are counted in whole numbers, whose order does not matter.
// ---------------------------------------------------------------------------------------------------------
constexpr int ROUTER_THREADS = 64;
template <typename T, int EP>
__global__ void __launch_bounds__(ROUTER_THREADS)
router_kernel(const T* __restrict__ logits, float* __restrict__ probs, long long* __restrict__ top_i, float* __restrict__ weights,
              float* __restrict__ part, float* __restrict__ hits, int n_tok, int E, int k, int* status) {
  __shared__ float sums[ROUTER_THREADS / 32][EP];
  __shared__ int counts[ROUTER_THREADS / 32][EP];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = t < n_tok;
  float p[EP];
  float mx = -INFINITY;
#pragma unroll
  for (int e = 0; e < EP; ++e) {
    p[e] = in && e < E ? as_float(logits[size_t(t) * E + e]) : -INFINITY;
    mx = fmaxf(mx, p[e]);
  }
  float sum = 0.f;
#pragma unroll
  for (int e = 0; e < EP; ++e) {
    p[e] = e < E ? __expf(p[e] - mx) : 0.f;
    sum += p[e];
  }
  const float inv = 1.f / sum;
#pragma unroll
  for (int e = 0; e < EP; ++e) {
    p[e] = in ? p[e] * inv : 0.f;
    if (in && e < E) probs[size_t(t) * E + e] = p[e];
  }
  unsigned long long taken = 0ull;
  int idx[MOE_MAX_K];
  float val[MOE_MAX_K];
  float picked = 0.f;
#pragma unroll
  for (int j = 0; j < MOE_MAX_K; ++j) {
    if (j >= k) break;
    int best = -1;
    float bv = -1.f;
#pragma unroll
    for (int e = 0; e < EP; ++e)
      if (e < E && !((taken >> e) & 1ull) && p[e] > bv) { bv = p[e]; best = e; }   // ties: lowest index, like torch.topk
    if (best < 0) {
      // no comparison succeeded: the probabilities are not finite (NaN logits of a diverged step).  Take the
      // lowest expert not yet picked, so that every index stays in range, and report through the status word.
      best = __ffsll(static_cast<long long>(~taken)) - 1;
      bv = 0.f;
      if (in) report_status(status, JPB_ERR_BAD_ARGUMENT);
    }
    taken |= 1ull << best;
    idx[j] = best; val[j] = bv; picked += bv;
  }
  const float pinv = 1.f / picked;
#pragma unroll
  for (int j = 0; j < MOE_MAX_K; ++j) {
    if (j >= k || !in) break;
    top_i[size_t(t) * k + j] = idx[j];
    weights[size_t(t) * k + j] = val[j] * pinv;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!in) taken = 0ull;
#pragma unroll
  for (int e = 0; e < EP; ++e) {
    if (e >= E) break;
    const float s = warp_sum(p[e]);
    const int c = __popc(__ballot_sync(0xffffffffu, (taken >> e) & 1ull));
    if (lane == 0) { sums[warp][e] = s; counts[warp][e] = c; }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += ROUTER_THREADS) {
    float s = 0.f;
    int c = 0;
#pragma unroll
    for (int w = 0; w < ROUTER_THREADS / 32; ++w) { s += sums[w][e]; c += counts[w][e]; }
    if (part) part[size_t(blockIdx.x) * E + e] = s;
    if (c) atomicAdd(hits + e, float(c));
  }
}

// aux = scale * sum_e hits[e] * (sum of column e of part).  AUX_THREADS / EP threads share a column, EP being E rounded up
// to a power of two; their sums, and then the experts', meet in trees.  Bound by the latency of a thread's chain of loads,
// of which four are in flight: 8192 tokens of 8 experts are 128 rows, one load a thread.
constexpr int AUX_THREADS = 1024;
__global__ void __launch_bounds__(AUX_THREADS) router_aux_kernel(const float* __restrict__ part, const float* __restrict__ hits,
                                                                 float* __restrict__ aux, int rows, int E, int EP, float scale) {
  __shared__ float red[AUX_THREADS];
  const int e = threadIdx.x & (EP - 1), slice = threadIdx.x / EP, slices = AUX_THREADS / EP;
  float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
  if (e < E) {
    int r = slice;
    for (; r + 3 * slices < rows; r += 4 * slices) {
      a0 += part[size_t(r) * E + e];
      a1 += part[size_t(r + slices) * E + e];
      a2 += part[size_t(r + 2 * slices) * E + e];
      a3 += part[size_t(r + 3 * slices) * E + e];
    }
    for (; r < rows; r += slices) a0 += part[size_t(r) * E + e];
  }
  red[threadIdx.x] = (a0 + a1) + (a2 + a3);
  __syncthreads();
  for (int n = AUX_THREADS / 2; n >= EP; n >>= 1) {
    if (threadIdx.x < n) red[threadIdx.x] += red[threadIdx.x + n];
    __syncthreads();
  }
  if (threadIdx.x < EP) red[threadIdx.x] *= e < E ? hits[e] : 0.f;
  __syncthreads();
  for (int n = EP / 2; n >= 1; n >>= 1) {
    if (threadIdx.x < n) red[threadIdx.x] += red[threadIdx.x + n];
    __syncthreads();
  }
  if (threadIdx.x == 0) *aux = red[0] * scale;
}

// Gradient of the logits from those of the weights (w_j = p_{i_j} / S, S the sum of the picked probabilities), of the
// probabilities and of the load-balancing loss (each may be absent).
template <typename T>
__global__ void router_bwd_kernel(const long long* __restrict__ top_i, const float* __restrict__ probs, const float* __restrict__ g_w,
                                  const float* __restrict__ g_probs, const float* __restrict__ g_aux, const float* __restrict__ hits,
                                  T* __restrict__ dlogits, int n_tok, int E, int k, float aux_scale) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tok) return;
  const float* pr = probs + size_t(t) * E;
  int idx[MOE_MAX_K];
  float d_pv[MOE_MAX_K];
  float s = 0.f, dot = 0.f;
#pragma unroll
  for (int j = 0; j < MOE_MAX_K; ++j) {
    idx[j] = j < k ? int(top_i[size_t(t) * k + j]) : -1;
    const float pv = j < k ? pr[idx[j]] : 0.f, g = j < k && g_w ? g_w[size_t(t) * k + j] : 0.f;
    s += pv;
    dot += g * pv;
    d_pv[j] = g;
  }
#pragma unroll
  for (int j = 0; j < MOE_MAX_K; ++j) d_pv[j] = g_w ? d_pv[j] / s - dot / (s * s) : 0.f;
  const float ga = g_aux ? *g_aux * aux_scale : 0.f;
  auto grad = [&](int e) {
    float d = g_probs ? g_probs[size_t(t) * E + e] : 0.f;
    if (g_aux) d += ga * hits[e];
#pragma unroll
    for (int j = 0; j < MOE_MAX_K; ++j) if (idx[j] == e) d += d_pv[j];
    return d;
  };
  float all = 0.f;
  for (int e = 0; e < E; ++e) all += grad(e) * pr[e];
  for (int e = 0; e < E; ++e) dlogits[size_t(t) * E + e] = T(pr[e] * (grad(e) - all));
}

// ---------------------------------------------------------------------------------------------------------
// Slots: pick i (token-major) of expert e goes to slot e * C + (number of earlier picks of e), or to E * C when the
// expert is full.  One CTA walks the picks 1024 at a time: ranks within a warp come from match, ranks between warps from
// a scan of the warps' counts, the running count of each expert from shared memory.
// ---------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) slots_kernel(const long long* __restrict__ top_i, long long* __restrict__ dest,
                                                     int* __restrict__ inv, int* __restrict__ counts, int n, int E, int C) {
  __shared__ int hist[32][MOE_MAX_E + 1];
  __shared__ int before[MOE_MAX_E];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < E; e += blockDim.x) before[e] = 0;
  for (int base = 0; base < n; base += 1024) {
    for (int e = lane; e < E; e += 32) hist[warp][e] = 0;
    __syncwarp();
    const int i = base + threadIdx.x;
    int e = i < n ? int(top_i[i]) : -1;
    if (e >= E) e = -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (e >= 0 && rank == 0) hist[warp][e] = __popc(same);
    __syncthreads();
    for (int x = warp; x < E; x += 32) {   // warp `warp` turns the counts of expert x into positions
      const int c = hist[lane][x];
      int run = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
      }
      const int b = before[x];
      __syncwarp();
      hist[lane][x] = b + run - c;
      if (lane == 31) before[x] = b + run;
    }
    __syncthreads();
    if (i < n) {
      const int pos = e >= 0 ? hist[warp][e] + rank : C;
      const bool keep = pos < C;
      dest[i] = keep ? (long long)e * C + pos : (long long)E * C;
      if (keep) inv[e * C + pos] = i;
    }
    __syncthreads();
  }
  __syncthreads();
  for (int e = warp; e < E; e += 32) {
    const int c = min(before[e], C);
    if (lane == 0) counts[e] = c;
    for (int s = c + lane; s < C; s += 32) inv[e * C + s] = -1;
  }
}

// out[slot] = x[inv[slot] / k], zeros where the slot is empty
template <typename T>
__global__ void dispatch_rows_kernel(const T* __restrict__ x, const int* __restrict__ inv, T* __restrict__ out, int slots, int d, int k) {
  constexpr int N = Row<T>::N;
  for (int s = blockIdx.x; s < slots; s += gridDim.x) {
    const int pick = inv[s];
    const T* src = x + size_t(pick < 0 ? 0 : pick / k) * d;
    T* dst = out + size_t(s) * d;
    for (int v = threadIdx.x * N; v < d; v += blockDim.x * N) {
      uint4 r = make_uint4(0, 0, 0, 0);
      if (pick >= 0) r = *reinterpret_cast<const uint4*>(src + v);
      *reinterpret_cast<uint4*>(dst + v) = r;
    }
  }
}

// out[t] = sum_j w[t, j] * y[dest[t, j]] (w absent: 1); a dropped pick (dest == slots) adds nothing
template <typename T>
__global__ void combine_rows_kernel(const T* __restrict__ y, const long long* __restrict__ dest, const float* __restrict__ w,
                                    T* __restrict__ out, int n_tok, int d, int k, int slots) {
  constexpr int N = Row<T>::N;
  for (int t = blockIdx.x; t < n_tok; t += gridDim.x) {
    for (int v = threadIdx.x * N; v < d; v += blockDim.x * N) {
      float acc[N];
#pragma unroll
      for (int i = 0; i < N; ++i) acc[i] = 0.f;
      for (int j = 0; j < k; ++j) {
        const long long s = dest[size_t(t) * k + j];
        if (s < 0 || s >= slots) continue;
        const float wj = w ? w[size_t(t) * k + j] : 1.f;
        float f[N];
        Row<T>::load(y + size_t(s) * d + v, f);
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] += f[i] * wj;
      }
      Row<T>::store(out + size_t(t) * d + v, acc);
    }
  }
}

// The transpose of the combination: dy[slot] = w[pick] * g[token], dw[pick] = <y[slot], g[token]>; zeros in empty slots.
// dw of dropped picks is zeroed by the caller.
template <typename T>
__global__ void combine_rows_bwd_kernel(const T* __restrict__ g, const T* __restrict__ y, const int* __restrict__ inv,
                                        const float* __restrict__ w, T* __restrict__ dy, float* __restrict__ dw, int slots, int d, int k) {
  constexpr int N = Row<T>::N;
  __shared__ float part[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int s = blockIdx.x; s < slots; s += gridDim.x) {
    const int pick = inv[s];           // the same in the whole CTA
    T* dst = dy + size_t(s) * d;
    if (pick < 0) {
      for (int v = threadIdx.x * N; v < d; v += blockDim.x * N) *reinterpret_cast<uint4*>(dst + v) = make_uint4(0, 0, 0, 0);
      continue;
    }
    const float wp = w[pick];
    const T* gr = g + size_t(pick / k) * d;
    const T* yr = y + size_t(s) * d;
    float dot = 0.f;
    for (int v = threadIdx.x * N; v < d; v += blockDim.x * N) {
      float a[N], b[N];
      Row<T>::load(gr + v, a);
      Row<T>::load(yr + v, b);
#pragma unroll
      for (int i = 0; i < N; ++i) { dot += a[i] * b[i]; a[i] *= wp; }
      Row<T>::store(dst + v, a);
    }
    dot = warp_sum(dot);
    __syncthreads();                   // `part` may still be read from the previous slot
    if (lane == 0) part[warp] = dot;
    __syncthreads();
    if (warp == 0) {
      const float all = warp_sum(lane < int(blockDim.x >> 5) ? part[lane] : 0.f);
      if (lane == 0) dw[pick] = all;
    }
  }
}

static int row_threads(int d, int n) {   // whole warps, one 16-byte piece per thread up to 512 threads
  int t = (d / n + 31) / 32 * 32;
  return t < 32 ? 32 : t > 512 ? 512 : t;
}
static int row_grid(int rows) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return rows < sms * 16 ? rows : sms * 16;
}
template <typename F>
static int by_dtype(int dt, F&& f) {
  if (dt == 0) return f(float{});
  if (dt == 1) return f(__nv_bfloat16{});
  return -JPB_ERR_BAD_ARGUMENT;
}
static bool aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace jpb

// fp32 elements of scratch that the loss of jpb_router needs: one row of E sums per CTA.
JPB_API long long jpb_router_scratch_elems(int n_tok, int E) {
  return (long long)((n_tok + jpb::ROUTER_THREADS - 1) / jpb::ROUTER_THREADS) * E;
}

// logits [n_tok, E] (fp32 dtype 0 or bf16 dtype 1) -> probs [n_tok, E] fp32, top_i [n_tok, k] int64, weights [n_tok, k]
// fp32, hits [E] fp32 (zeroed here), aux (one fp32, may be absent) = aux_scale * sum_e hits[e] * sum_t probs[t][e], which
// needs `part`, jpb_router_scratch_elems() of scratch.  E <= 64, k <= 8.  A token whose probabilities are not
// finite gets the lowest-numbered experts (indices stay in range) and the status word is set to JPB_ERR_BAD_ARGUMENT.
JPB_API int jpb_router(int dtype, const void* logits, float* probs, long long* top_i, float* weights, float* part,
                       float* hits, float* aux, float aux_scale, int n_tok, int E, int k, void* stream) {
  using namespace jpb;
  if (E < 1 || E > MOE_MAX_E || k < 1 || k > MOE_MAX_K || k > E || (aux && n_tok > 0 && !part)) return -JPB_ERR_BAD_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaMemsetAsync(hits, 0, sizeof(float) * E, s);
  const int threads = ROUTER_THREADS, blocks = n_tok > 0 ? (n_tok + threads - 1) / threads : 0;
  if (blocks) {
    float* sums = aux ? part : nullptr;
    int* status = jpb_status_device_ptr();
    const int rc = by_dtype(dtype, [&](auto tag) {
      using T = decltype(tag);
      const T* lg = static_cast<const T*>(logits);
      if (E <= 8) router_kernel<T, 8><<<blocks, threads, 0, s>>>(lg, probs, top_i, weights, sums, hits, n_tok, E, k, status);
      else if (E <= 16) router_kernel<T, 16><<<blocks, threads, 0, s>>>(lg, probs, top_i, weights, sums, hits, n_tok, E, k, status);
      else if (E <= 32) router_kernel<T, 32><<<blocks, threads, 0, s>>>(lg, probs, top_i, weights, sums, hits, n_tok, E, k, status);
      else router_kernel<T, 64><<<blocks, threads, 0, s>>>(lg, probs, top_i, weights, sums, hits, n_tok, E, k, status);
      return 0;
    });
    if (rc) return rc;
  }
  if (aux) {
    int ep = 1;
    while (ep < E) ep *= 2;
    router_aux_kernel<<<1, AUX_THREADS, 0, s>>>(part, hits, aux, blocks, E, ep, aux_scale);
  }
  return int(cudaGetLastError());
}

// dlogits [n_tok, E] of type `dtype` from g_w [n_tok, k], g_probs [n_tok, E] and g_aux (one value), all fp32, any may be absent.
JPB_API int jpb_router_bwd(int dtype, const long long* top_i, const float* probs, const float* g_w, const float* g_probs, const float* g_aux,
                           const float* hits, void* dlogits, int n_tok, int E, int k, float aux_scale, void* stream) {
  using namespace jpb;
  if (E < 1 || E > MOE_MAX_E || k < 1 || k > MOE_MAX_K || k > E) return -JPB_ERR_BAD_ARGUMENT;
  if (n_tok <= 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    router_bwd_kernel<T><<<(n_tok + 63) / 64, 64, 0, s>>>(top_i, probs, g_w, g_probs, g_aux, hits, static_cast<T*>(dlogits), n_tok, E, k,
                                                          aux_scale);
    return int(cudaGetLastError());
  });
}

// top_i [n] int64 in [0, E) -> dest [n] int64, inv [E * C] (pick of each slot, or -1), counts [E] (filled slots).  E <= 64.
JPB_API int jpb_moe_slots(const long long* top_i, long long* dest, int* inv, int* counts, int n, int E, int C, void* stream) {
  using namespace jpb;
  if (E < 1 || E > MOE_MAX_E || C < 0 || n < 0 || (long long)E * C > 0x7fffffffll) return -JPB_ERR_BAD_ARGUMENT;
  slots_kernel<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(top_i, dest, inv, counts, n, E, C);
  return int(cudaGetLastError());
}

// Rows of d elements (fp32 dtype 0, bf16 dtype 1), contiguous, on 16-byte boundaries.
JPB_API int jpb_moe_dispatch_rows(int dtype, const void* x, const int* inv, void* out, int slots, int d, int k, void* stream) {
  using namespace jpb;
  if (slots <= 0 || d <= 0) return 0;
  return by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    if (d % Row<T>::N || !aligned(x) || !aligned(out)) return -int(JPB_ERR_BAD_ARGUMENT);
    dispatch_rows_kernel<T><<<row_grid(slots), row_threads(d, Row<T>::N), 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const T*>(x), inv, static_cast<T*>(out), slots, d, k);
    return int(cudaGetLastError());
  });
}
JPB_API int jpb_moe_combine_rows(int dtype, const void* y, const long long* dest, const float* w, void* out, int n_tok, int d, int k, int slots,
                            void* stream) {
  using namespace jpb;
  if (n_tok <= 0 || d <= 0) return 0;
  return by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    if (d % Row<T>::N || !aligned(y) || !aligned(out)) return -int(JPB_ERR_BAD_ARGUMENT);
    combine_rows_kernel<T><<<row_grid(n_tok), row_threads(d, Row<T>::N), 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const T*>(y), dest, w, static_cast<T*>(out), n_tok, d, k, slots);
    return int(cudaGetLastError());
  });
}
JPB_API int jpb_moe_combine_rows_bwd(int dtype, const void* g, const void* y, const int* inv, const float* w, void* dy, float* dw, int slots,
                                int d, int k, void* stream) {
  using namespace jpb;
  if (slots <= 0 || d <= 0) return 0;
  return by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    if (d % Row<T>::N || !aligned(g) || !aligned(y) || !aligned(dy)) return -int(JPB_ERR_BAD_ARGUMENT);
    combine_rows_bwd_kernel<T><<<row_grid(slots), row_threads(d, Row<T>::N), 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const T*>(g), static_cast<const T*>(y), inv, w, static_cast<T*>(dy), dw, slots, d, k);
    return int(cudaGetLastError());
  });
}
