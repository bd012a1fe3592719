// Fused router (score function + bias + top-k + normalisation in one pass, one warp per token) and the
// softmax cross-entropy forward+backward that turns a chunk of logits into its gradient in place.
//
// Reference analogues: fused router with aux score (notes/2026-04/2026-04-25_gptoss_22_*:118-127),
// fused cross entropy (notes/2026-04/2026-04-19_gptoss_01_mlperf_best_e2e_run.md:85).
#include "common.cuh"

namespace slab {

constexpr int ROUTER_MAX_PER_LANE = 16;   // up to 512 experts

// logits: [T, E] fp32.  score: 0 softmax, 1 sigmoid.  bias (optional, [E]) only affects selection.
// Outputs: weights [T, K] fp32 (normalised over the selected experts if norm, times scaling), idx [T, K].
__global__ void router_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias,
                                   float* __restrict__ weights, int* __restrict__ idx, int T, int E, int K,
                                   int score, int norm, float scaling) {
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (int t = blockIdx.x * warps + (threadIdx.x >> 5); t < T; t += gridDim.x * warps) {
    float s[ROUTER_MAX_PER_LANE], sel[ROUTER_MAX_PER_LANE];
    const float* row = logits + (size_t)t * E;
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < ROUTER_MAX_PER_LANE; ++i) {
      int e = lane + i * 32;
      s[i] = e < E ? row[e] : -INFINITY;
      mx = fmaxf(mx, s[i]);
    }
    if (score == 0) {
      mx = warp_max(mx);
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < ROUTER_MAX_PER_LANE; ++i) {
        int e = lane + i * 32;
        s[i] = e < E ? __expf(s[i] - mx) : 0.f;
        sum += s[i];
      }
      sum = warp_sum(sum);
      const float inv = 1.f / sum;
#pragma unroll
      for (int i = 0; i < ROUTER_MAX_PER_LANE; ++i) s[i] *= inv;
    } else {
#pragma unroll
      for (int i = 0; i < ROUTER_MAX_PER_LANE; ++i) {
        int e = lane + i * 32;
        s[i] = e < E ? 1.f / (1.f + __expf(-s[i])) : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < ROUTER_MAX_PER_LANE; ++i) {
      int e = lane + i * 32;
      sel[i] = e < E ? (s[i] + (bias ? bias[e] : 0.f)) : -INFINITY;
    }
    float wsum = 0.f;
    float my_w = 0.f;     // lane k keeps the k-th selection
    int my_i = 0;
    for (int k = 0; k < K; ++k) {
      float best = -INFINITY;
      int bi = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < ROUTER_MAX_PER_LANE; ++i) {
        int e = lane + i * 32;
        if (sel[i] > best) { best = sel[i]; bi = e; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        float ob = __shfl_xor_sync(0xffffffffu, best, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      // owner lane publishes the (unbiased) score and retires the expert
      float sc = 0.f;
#pragma unroll
      for (int i = 0; i < ROUTER_MAX_PER_LANE; ++i) {
        if (lane + i * 32 == bi) { sc = s[i]; sel[i] = -INFINITY; }
      }
      sc = __shfl_sync(0xffffffffu, sc, bi & 31);
      wsum += sc;
      if (lane == k) { my_w = sc; my_i = bi; }
    }
    if (lane < K) {
      float w = norm ? my_w / (wsum + 1e-20f) : my_w;
      weights[(size_t)t * K + lane] = w * scaling;
      idx[(size_t)t * K + lane] = my_i;
    }
  }
}

// ---------------------------------------------------------------- fused router with load statistics + aux loss
// Scores of one token (softmax or sigmoid of its fp32 logits), spread over the warp: lane l holds experts
// l, l + 32, ... (PL of them, the smallest of 4, 8 and 16 that covers E: what a token costs is proportional to it; 8192 tokens x 256
// experts, top-8, forward 30 -> 20 us against 16 for every E).
template <int PL>
__device__ __forceinline__ void router_scores(const float* __restrict__ row, int E, int score, int lane, float (&s)[PL]) {
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    const int e = lane + i * 32;
    s[i] = e < E ? row[e] : -INFINITY;
    mx = fmaxf(mx, s[i]);
  }
  if (score == 0) {
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      const int e = lane + i * 32;
      s[i] = e < E ? __expf(s[i] - mx) : 0.f;
      sum += s[i];
    }
    sum = warp_sum(sum);
    const float inv = 1.f / sum;
#pragma unroll
    for (int i = 0; i < PL; ++i) s[i] *= inv;
  } else {
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      const int e = lane + i * 32;
      s[i] = e < E ? 1.f / (1.f + __expf(-s[i])) : 0.f;
    }
  }
}

constexpr float ROUTER_FIX = 1099511627776.f;      // 2^40: scores in [0, 1] as fixed point, exact integer sums

// Same selection as router_topk_kernel, plus in the same pass the statistics the load-balancing loss needs:
//   counts[e]  = pairs routed to expert e               (int)
//   p_fix[e]   = sum over tokens of score[t, e] * 2^40  (unsigned 64-bit fixed point: the sum does not depend on
//                the order in which blocks arrive, so the loss is reproducible bit for bit)
// and the loss itself, written by the last block to finish:
//   aux = aux_coeff * E * sum_e (counts[e] / (T K)) * (p_sum[e] / T)
// counts, p_fix and ticket must be zero on entry.
template <int PL>
__global__ void __launch_bounds__(256)
router_fused_fwd_kernel(const float* __restrict__ logits, const float* __restrict__ bias, float* __restrict__ weights,
                        int* __restrict__ idx, int T, int E, int K, int score, int norm, float scaling,
                        int* __restrict__ counts, unsigned long long* __restrict__ p_fix, int* __restrict__ ticket,
                        float aux_coeff, float* __restrict__ aux_out) {
  __shared__ unsigned long long p_s[32 * PL];
  __shared__ int c_s[32 * PL];
  __shared__ float red[8];
  __shared__ int last;
  for (int e = threadIdx.x; e < E; e += blockDim.x) { p_s[e] = 0ull; c_s[e] = 0; }
  __syncthreads();
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  unsigned long long pacc[PL];     // this lane's experts, summed over the warp's tokens
#pragma unroll
  for (int i = 0; i < PL; ++i) pacc[i] = 0ull;
  for (int t = blockIdx.x * warps + (threadIdx.x >> 5); t < T; t += gridDim.x * warps) {
    float s[PL], sel[PL];
    router_scores(logits + (size_t)t * E, E, score, lane, s);
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      const int e = lane + i * 32;
      sel[i] = e < E ? (s[i] + (bias ? bias[e] : 0.f)) : -INFINITY;
      pacc[i] += (unsigned long long)(s[i] * ROUTER_FIX);      // padding lanes hold score 0
    }
    float wsum = 0.f, my_w = 0.f;
    int my_i = 0;
    for (int k = 0; k < K; ++k) {
      float best = -INFINITY;
      int bi = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < PL; ++i) {
        const int e = lane + i * 32;
        if (sel[i] > best) { best = sel[i]; bi = e; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      float sc = 0.f;
#pragma unroll
      for (int i = 0; i < PL; ++i) {
        if (lane + i * 32 == bi) { sc = s[i]; sel[i] = -INFINITY; }
      }
      sc = __shfl_sync(0xffffffffu, sc, bi & 31);
      wsum += sc;
      if (lane == k) { my_w = sc; my_i = bi; }
    }
    if (lane < K) {
      const float w = norm ? my_w / (wsum + 1e-20f) : my_w;
      weights[(size_t)t * K + lane] = w * scaling;
      idx[(size_t)t * K + lane] = my_i;
      if (my_i >= 0 && my_i < E) atomicAdd(&c_s[my_i], 1);
    }
  }
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    const int e = lane + i * 32;
    if (e < E && pacc[i]) atomicAdd(&p_s[e], pacc[i]);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    if (c_s[e]) atomicAdd(&counts[e], c_s[e]);
    if (p_s[e]) atomicAdd(&p_fix[e], p_s[e]);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(ticket, 1) == (int)gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  float acc = 0.f;                                  // fixed order: thread i sums experts i, i + 256, ...
  for (int e = threadIdx.x; e < E && T > 0; e += blockDim.x) {
    const float f = (float)__ldcg(&counts[e]) / ((float)T * (float)K);
    const float pm = (float)((double)__ldcg(&p_fix[e]) / (double)ROUTER_FIX) / (float)T;
    acc += f * pm;
  }
  acc = warp_sum(acc);
  if (lane == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < warps; ++w) tot += red[w];
    *aux_out = aux_coeff * (float)E * tot;
  }
}

// Gradient of the fused router with respect to the logits, one warp per token: the scores are recomputed from
// the logits (cheaper than storing [T, E] of them), then
//   G[e]      = g_aux * aux_coeff * E * counts[e] / (T^2 K)                      (dense: the load-balancing loss)
//             + for the selected experts, the gate-weight path: with W = sum of the selected scores,
//               norm:  (scaling / W) * (gw[k] - sum_j gw[j] * s_j / W),   else  scaling * gw[k]
//   softmax:  dlogit[e] = s[e] * (G[e] - sum_j s[j] G[j]);     sigmoid:  dlogit[e] = G[e] * s[e] * (1 - s[e]).
// counts / g_aux may be null (no auxiliary loss).
template <int PL>
__global__ void __launch_bounds__(256)
router_fused_bwd_kernel(const float* __restrict__ logits, const int* __restrict__ idx, const float* __restrict__ gw,
                        const int* __restrict__ counts, const float* __restrict__ g_aux, float aux_coeff,
                        float* __restrict__ dlogits, int T, int E, int K, int score, int norm, float scaling) {
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const float ga = (g_aux && counts) ? *g_aux * aux_coeff * (float)E / ((float)T * (float)T * (float)K) : 0.f;
  for (int t = blockIdx.x * warps + (threadIdx.x >> 5); t < T; t += gridDim.x * warps) {
    float s[PL], G[PL];
    router_scores(logits + (size_t)t * E, E, score, lane, s);
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      const int e = lane + i * 32;
      G[i] = (ga != 0.f && e < E) ? ga * (float)counts[e] : 0.f;
    }
    // lane k < K holds selection k
    const int my_i = lane < K ? idx[(size_t)t * K + lane] : -1;
    const float my_g = lane < K ? gw[(size_t)t * K + lane] : 0.f;
    float my_s = 0.f;
    for (int k = 0; k < K; ++k) {
      const int e = __shfl_sync(0xffffffffu, my_i, k);
      float sc = 0.f;
#pragma unroll
      for (int i = 0; i < PL; ++i)
        if (lane + i * 32 == e) sc = s[i];
      sc = __shfl_sync(0xffffffffu, sc, e & 31);
      if (lane == k) my_s = sc;
    }
    const float W = warp_sum(my_s) + 1e-20f;
    const float gdot = warp_sum(my_g * my_s) / W;          // sum_j gw[j] * s_j / W
    const float my_G = lane < K ? (norm ? (scaling / W) * (my_g - gdot) : scaling * my_g) : 0.f;
    for (int k = 0; k < K; ++k) {
      const int e = __shfl_sync(0xffffffffu, my_i, k);
      const float add = __shfl_sync(0xffffffffu, my_G, k);
#pragma unroll
      for (int i = 0; i < PL; ++i)
        if (lane + i * 32 == e) G[i] += add;
    }
    float* out = dlogits + (size_t)t * E;
    if (score == 0) {
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < PL; ++i) dot += s[i] * G[i];
      dot = warp_sum(dot);
#pragma unroll
      for (int i = 0; i < PL; ++i) {
        const int e = lane + i * 32;
        if (e < E) out[e] = s[i] * (G[i] - dot);
      }
    } else {
#pragma unroll
      for (int i = 0; i < PL; ++i) {
        const int e = lane + i * 32;
        if (e < E) out[e] = G[i] * s[i] * (1.f - s[i]);
      }
    }
  }
}

// CTAS blocks (a cluster) per row: loss_row = logsumexp(logits) - logits[target]; logits <- (softmax - onehot) * gscale
// (GRAD).  `loss_sum` accumulates sum of row losses (fp32 atomics).  V % 8 == 0.
//
// Bound by memory and the exponentials (two per element on a pipe of 16 lanes per clock).  A row is 2 V bytes (300 - 400 KB
// at the vocabularies in use), too long for one SM's shared memory, so it is read twice.  The maximum and the sum come
// from ONE pass (running maximum, rescaled sum), and few rows are in flight at a time, so the second read and the write
// find the row in the 126 MB L2 and memory sees one read and one write.  Long rows are shared by the two blocks of a
// cluster: 148 rows of at most 400 KB = 60 MB in flight, and every SM has blocks of two rows, one of which computes while
// the other waits at a row's end.  The next piece is requested before the current one is worked on.  [1021, 201088] 297 ->
// 227 us (3.6 TB/s of one read and one write), the loss alone 105; [8192, 151936] 1553 -> 1292 us, 573; three reads before.
constexpr int CE_UNROLL = 2;

template <int CTAS>
__device__ __forceinline__ void ce_row_sync() {
  if (CTAS > 1)
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  else
    __syncthreads();
}
// the other block's copy of a shared variable
__device__ __forceinline__ float ce_peer(const float* v, uint32_t peer) {
  uint32_t a;
  float f;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(v)), "r"(peer));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(a) : "memory");
  return f;
}

// Calls f(vector, index) for the vectors lo + threadIdx.x, + THREADS, ... below hi.
template <int THREADS, typename F>
__device__ __forceinline__ void ce_walk(const bf16x8* row, int lo, int hi, F f) {
  bf16x8 next[CE_UNROLL];
#pragma unroll
  for (int u = 0; u < CE_UNROLL; ++u)
    if (lo + (int)threadIdx.x + u * THREADS < hi) next[u] = row[lo + threadIdx.x + u * THREADS];
  for (int c0 = lo + threadIdx.x; c0 < hi; c0 += THREADS * CE_UNROLL) {
    bf16x8 v[CE_UNROLL];
#pragma unroll
    for (int u = 0; u < CE_UNROLL; ++u) {
      v[u] = next[u];
      const int c = c0 + (CE_UNROLL + u) * THREADS;
      if (c < hi) next[u] = row[c];
    }
#pragma unroll
    for (int u = 0; u < CE_UNROLL; ++u)
      if (c0 + u * THREADS < hi) f(v[u], c0 + u * THREADS);
  }
}

template <int THREADS, int CTAS, bool GRAD>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(THREADS, 1024 / THREADS)
ce_kernel(__nv_bfloat16* __restrict__ logits, const long* __restrict__ targets, float* __restrict__ loss_sum, int rows,
          int V, float gscale) {
  __shared__ float red_m[2][THREADS / 32], red_s[2][THREADS / 32];   // by parity of the row: one barrier per row
  __shared__ float all_m[2], all_s[2];
  constexpr int WARPS = THREADS / 32;
  const int nvec = V >> 3;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CTAS > 1 ? (int)(blockIdx.x % CTAS) : 0;
  const int half = (nvec + CTAS - 1) / CTAS;
  const int lo = rank * half, hi = min(nvec, lo + half);
  int par = 0;
  for (int r = blockIdx.x / CTAS; r < rows; r += gridDim.x / CTAS, par ^= 1) {
    bf16x8* row = reinterpret_cast<bf16x8*>(logits + (size_t)r * V);
    const long tgt = targets[r];
    const float lt = threadIdx.x == 0 ? __bfloat162float(logits[(size_t)r * V + tgt]) : 0.f;
    float m = -INFINITY, s = 0.f;
    ce_walk<THREADS>(row, lo, hi, [&](const bf16x8& v, int) {
      float f[8];
      unpack8(v, f);
      float vm = f[0];
#pragma unroll
      for (int j = 1; j < 8; ++j) vm = fmaxf(vm, f[j]);
      if (vm > m) {
        s *= __expf(m - vm);               // the first time m is -inf and s is 0
        m = vm;
      }
      // columns masked with -inf: while nothing finite was seen the reference point is 0, and they add exp(-inf) = 0
      const float ref = m == -INFINITY ? 0.f : m;
#pragma unroll
      for (int j = 0; j < 8; ++j) s += __expf(f[j] - ref);
    });
    const float wm = warp_max(m);
    s = warp_sum(m == -INFINITY ? s : s * __expf(m - wm));
    if (lane == 0) { red_m[par][warp] = wm; red_s[par][warp] = s; }
    __syncthreads();
    const float bm = lane < WARPS ? red_m[par][lane] : -INFINITY;
    const float bs = lane < WARPS ? red_s[par][lane] : 0.f;
    float mx = warp_max(bm);
    float sum = warp_sum(bm == -INFINITY ? bs : bs * __expf(bm - mx));
    if (CTAS > 1) {
      if (threadIdx.x == 0) { all_m[par] = mx; all_s[par] = sum; }
      ce_row_sync<CTAS>();                 // both parts have been read and summed
      const float pm = ce_peer(&all_m[par], rank ^ 1), ps = ce_peer(&all_s[par], rank ^ 1);
      const float top = fmaxf(mx, pm);
      sum = (mx == -INFINITY ? sum : sum * __expf(mx - top)) + (pm == -INFINITY ? ps : ps * __expf(pm - top));
      mx = top;
    }
    if (rank == 0 && threadIdx.x == 0) atomicAdd(loss_sum, logf(sum) + mx - lt);
    if (!GRAD) continue;
    const float inv = gscale / sum;
    ce_walk<THREADS>(row, lo, hi, [&](const bf16x8& v, int c) {
      float f[8];
      unpack8(v, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        f[j] = __expf(f[j] - mx) * inv;
        if ((long)c * 8 + j == tgt) f[j] -= gscale;
      }
      row[c] = pack8(f);
    });
  }
  if (CTAS > 1) ce_row_sync<CTAS>();       // the other block may still be reading this one's sums
}

}  // namespace slab

using namespace slab;

extern "C" int slab_router_topk(const float* logits, const float* bias, float* weights, int* idx, int T, int E,
                                int K, int score, int norm, float scaling, cudaStream_t st) {
  if (E > 32 * ROUTER_MAX_PER_LANE || K > 32 || K > E) return -100;
  if (T == 0) return 0;
  int blocks = (T + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  router_topk_kernel<<<blocks, 256, 0, st>>>(logits, bias, weights, idx, T, E, K, score, norm, scaling);
  return (int)cudaGetLastError();
}

// Router forward with load statistics and the load-balancing loss in one launch.  stats: int32 [3 * E + 2], zero on
// entry, laid out as counts [E] | p_fix [E] as unsigned 64-bit (2 ints each, 8-byte aligned because E is rounded to
// even by the caller's layout: offset (E + E % 2) ints) | ticket.  aux_out: fp32 [1].
extern "C" int slab_router_fused_fwd(const float* logits, const float* bias, float* weights, int* idx, int T, int E,
                                     int K, int score, int norm, float scaling, int* stats, float aux_coeff,
                                     float* aux_out, cudaStream_t st) {
  if (E > 32 * ROUTER_MAX_PER_LANE || K > 32 || K > E) return -100;
  if ((uintptr_t)stats & 7) return -101;
  int blocks = (T + 7) / 8;
  if (blocks > 148 * 4) blocks = 148 * 4;
  if (blocks < 1) blocks = 1;
  const int e2 = E + (E & 1);
  auto kern = E <= 128 ? router_fused_fwd_kernel<4> : E <= 256 ? router_fused_fwd_kernel<8> : router_fused_fwd_kernel<16>;
  kern<<<blocks, 256, 0, st>>>(logits, bias, weights, idx, T, E, K, score, norm, scaling, stats,
                               reinterpret_cast<unsigned long long*>(stats + e2), stats + e2 + 2 * E, aux_coeff, aux_out);
  return (int)cudaGetLastError();
}

extern "C" int slab_router_fused_bwd(const float* logits, const int* idx, const float* gw, const int* counts,
                                     const float* g_aux, float aux_coeff, float* dlogits, int T, int E, int K,
                                     int score, int norm, float scaling, cudaStream_t st) {
  if (E > 32 * ROUTER_MAX_PER_LANE || K > 32 || K > E) return -100;
  if (T == 0) return 0;
  int blocks = (T + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  auto kern = E <= 128 ? router_fused_bwd_kernel<4> : E <= 256 ? router_fused_bwd_kernel<8> : router_fused_bwd_kernel<16>;
  kern<<<blocks, 256, 0, st>>>(logits, idx, gw, counts, g_aux, aux_coeff, dlogits, T, E, K, score, norm, scaling);
  return (int)cudaGetLastError();
}

template <bool GRAD>
static int launch_ce(void* logits, const long* targets, float* loss_sum, int rows, int V, float gscale, cudaStream_t st) {
  if (V % 8) return -100;
  if (rows == 0) return 0;
  // Two blocks per row pay where a row is long, or where there are not enough rows to give every SM two: 3095 rows of 33024 / 64000 /
  // 80000 / 96000 / 129280 columns 145 / 225 / 276 / 316 / 409 us, four small blocks per SM 95 / 206 / 262 / 319 / 426; 200 rows 13.2 /
  // 18.3 / 21.9 / 24.7 / 34.3 against 12.2 / 19.9 / 24.1 / 28.3 / 41.8.
  if (V > 90112 || (V > 49152 && rows <= 2 * 148))
    ce_kernel<512, 2, GRAD><<<2 * (rows < 148 ? rows : 148), 512, 0, st>>>((__nv_bfloat16*)logits, targets, loss_sum, rows, V, gscale);
  else
    ce_kernel<256, 1, GRAD><<<rows < 148 * 4 ? rows : 148 * 4, 256, 0, st>>>((__nv_bfloat16*)logits, targets, loss_sum, rows, V, gscale);
  return (int)cudaGetLastError();
}

extern "C" int slab_ce_fwd_bwd(void* logits, const long* targets, float* loss_sum, int rows, int V, float gscale,
                               cudaStream_t st) {
  return launch_ce<true>(logits, targets, loss_sum, rows, V, gscale, st);
}

// The loss alone: the logits are left as they are.
extern "C" int slab_ce_fwd(const void* logits, const long* targets, float* loss_sum, int rows, int V, cudaStream_t st) {
  return launch_ce<false>(const_cast<void*>(logits), targets, loss_sum, rows, V, 0.f, st);
}
