// Block-scaled fp8 (e4m3) grouped expert GEMM, forward:  C[r, n] = sum_k A[r, k] * B[e, n, k]  with
//   A: [R, K] e4m3, scales sa [R, K/128] fp32 (1x128 blocks along K, as written by the fused dispatch or the
//      quantising SwiGLU), B: [E, N, K] e4m3, scales sb [E, N/128, K/128] fp32 (128x128 blocks), C bf16.
//
// tcgen05.mma kind::f8f6f4 (128x128x32 per instruction) accumulates one 128-wide K block into a TMEM buffer;
// because the scale changes every K block the partial sum is promoted outside the tensor core: the four
// epilogue warps read the 128x128 fp32 partial with tcgen05.ld, multiply by sa[row, kb] * sb[e, nb, kb] and
// add into register accumulators while the MMA warp already fills the next TMEM buffer (4 buffers of 128
// columns).  Operands arrive by TMA (128-byte swizzle: one 128-element fp8 row per swizzle row), 6 stages,
// no cluster multicast.  The output goes through swizzled shared staging and a TMA store.
//
// Bound by the read-out and scaling of a partial tile per K block (two columns per multiply-add).  Copies and MMAs are
// issued by an elected lane of a converged warp; before, issuing them was what a K block waited for: 32 experts, 16384 rows,
// 7168 -> 4096 782 -> 588 us (1230 -> 1637 TFLOP/s), 2048 -> 7168 408 -> 313 us, the same bits.
//
// Reference analogues: the fused fp8 grouped GEMM with dequantising epilogue (`acc *= sa*sb`,
// summary/fp8_expert_gemm_optimization.md:84-116) and the blockwise recipe that was the slowest variant there
// (notes/2026-04/2026-04-21_gptoss_10_moe_fp8_grouped_gemm_diagnosis.md:74-85).
#include "common.cuh"
#include "tma_host.cuh"

namespace slab {

constexpr int F8_BM = 128, F8_BN = 128, F8_BK = 128, F8_UK = 32, F8_STAGES = 6, F8_TBUF = 4;
constexpr int F8_THREADS = 320;          // TMA warp, MMA warp, 2 x 4 epilogue warps (each group owns 64 columns)
constexpr int F8_CTRL = 3072, F8_PREFIX_OFF = 256;
constexpr int F8_A_BYTES = F8_BM * F8_BK, F8_B_BYTES = F8_BN * F8_BK, F8_STAGE = F8_A_BYTES + F8_B_BYTES;
constexpr int F8_STORE_OFF = F8_CTRL + F8_STAGES * F8_STAGE;
constexpr int F8_STORE_BYTES = F8_BM * 64 * 2;
constexpr int F8_SMEM = F8_STORE_OFF + 2 * F8_STORE_BYTES;
static_assert(F8_SMEM <= 232448, "shared memory budget");

constexpr int F8_AHEAD = 4;              // K blocks whose scales are requested ahead

// two fp32 values side by side: one instruction multiplies and adds both
__device__ __forceinline__ unsigned long long f32x2(uint32_t lo, uint32_t hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

struct Fp8Params {
  const int* seg_offsets;
  const int* seg_counts;
  const float* sa;       // [R, K/128]
  const float* sb;       // [E, N/128, K/128]
  int E, R, N, K;
  int* status;
};

__device__ __forceinline__ int f8_seg_rows(const Fp8Params& p, int e) {
  const int off = p.seg_offsets[e], cnt = p.seg_counts[e];
  if (off < 0 || off >= p.R || cnt <= 0) return 0;
  return cnt < p.R - off ? cnt : p.R - off;
}

struct F8Tile {
  int e, m_idx, n_idx, row0;
};

__device__ __forceinline__ bool f8_get_tile(int t, const int* prefix, const Fp8Params& p, F8Tile& ti) {
  if (t >= prefix[p.E]) return false;
  int lo = 0, hi = p.E;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (prefix[mid] <= t) lo = mid; else hi = mid;
  }
  const int local = t - prefix[lo];
  const int m_tiles = (f8_seg_rows(p, lo) + F8_BM - 1) / F8_BM;
  ti.e = lo;
  ti.m_idx = local % m_tiles;
  ti.n_idx = local / m_tiles;
  ti.row0 = p.seg_offsets[lo] + ti.m_idx * F8_BM;
  return true;
}

__global__ void __launch_bounds__(F8_THREADS, 1)
grouped_gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                        const __grid_constant__ CUtensorMap tmap_c, const Fp8Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) atomicCAS(p.status, 0, ST_BAD_INDEX);
    return;
  }
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty_bar = full_bar + F8_STAGES;
  uint64_t* tfull_bar = empty_bar + F8_STAGES;
  uint64_t* tempty_bar = tfull_bar + F8_TBUF;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + F8_TBUF);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* prefix = reinterpret_cast<int*>(smem + F8_PREFIX_OFF);
  uint8_t* ring = smem + F8_CTRL;
  uint8_t* store_buf = smem + F8_STORE_OFF;
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int n_tiles = (p.N + F8_BN - 1) / F8_BN;
  const int kblocks = p.K / F8_BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < F8_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < F8_TBUF; ++b) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 8); }
    *abort_flag = 0;
    fence_mbar_init();
    int acc = 0;
    for (int e = 0; e < p.E; ++e) {
      prefix[e] = acc;
      acc += ((f8_seg_rows(p, e) + F8_BM - 1) / F8_BM) * n_tiles;
    }
    prefix[p.E] = acc;
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
    prefetch_tmap(&tmap_c);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, F8_TBUF * F8_BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const int tiles = warp_uniform(prefix[p.E]);

  if (warp == 0) {
    // ---------------- TMA producer (the whole warp, see elect_one)
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
      F8Tile ti;
      f8_get_tile(t, prefix, p, ti);
      const int a_row = warp_uniform(ti.row0), b_row = warp_uniform(ti.e * p.N + ti.n_idx * F8_BN);
      for (int kb = 0; kb < kblocks; ++kb) {
        ok = mbar_wait_warp(&empty_bar[s], ph ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY);
        if (!ok) break;
        uint8_t* a_dst = ring + s * F8_STAGE;
        if (elect_one()) {
          mbar_arrive_expect_tx(&full_bar[s], F8_STAGE);
          tma_load_2d(a_dst, &tmap_a, &full_bar[s], kb * F8_BK, a_row);
          tma_load_2d(a_dst + F8_A_BYTES, &tmap_b, &full_bar[s], kb * F8_BK, b_row);
        }
        if (++s == F8_STAGES) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: one TMEM buffer per K block
    constexpr uint32_t idesc = make_idesc(0, 0, 0, 0, F8_BM, F8_BN);     // e4m3 x e4m3, K-major both
    const uint64_t a0 = make_smem_desc(smem_u32(ring), 16, 1024, 2);
    const uint64_t b0 = make_smem_desc(smem_u32(ring) + F8_A_BYTES, 16, 1024, 2);
    int s = 0;
    uint32_t ph = 0;
    uint32_t it = 0;                                   // K blocks issued so far (selects the TMEM buffer)
    bool ok = true;
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
      for (int kb = 0; kb < kblocks; ++kb, ++it) {
        const uint32_t buf = it % F8_TBUF;
        ok = __all_sync(0xffffffffu,
                        mbar_wait(&tempty_bar[buf], ((it / F8_TBUF) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY) &&
                            mbar_wait(&full_bar[s], ph, abort_flag, p.status, ST_TIMEOUT_FULL));
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k4 = 0; k4 < F8_BK / F8_UK; ++k4)
            umma_f8(tmem_base + buf * F8_BN, a0 + (uint32_t)(s * (F8_STAGE >> 4)) + k4 * 2,
                    b0 + (uint32_t)(s * (F8_STAGE >> 4)) + k4 * 2, idesc, k4 != 0 ? 1u : 0u);
          umma_commit(&empty_bar[s]);
          umma_commit(&tfull_bar[buf]);
        }
        if (++s == F8_STAGES) { s = 0; ph ^= 1; }
      }
    }
  } else {
    // ---------------- epilogue warps: promote every K block with its scales, then store the tile.
    // Two groups of four warps; group `half` owns output columns [64*half, 64*half + 64) of the tile.
    const int lg = warp & 3;
    const int half = (warp - 2) >> 2;
    const bool store_thread = ((warp == 2 || warp == 6) && lane == 0);
    const int r_in_tile = lg * 32 + lane;
    const int nb_total = p.N / 128;
    uint8_t* sbuf = store_buf + half * F8_STORE_BYTES;
    uint32_t it = 0;
    F8Tile ti;
    bool ok = true;                                      // no wait of this warp has run out (see mbar_wait_warp)
    for (int t = blockIdx.x; f8_get_tile(t, prefix, p, ti); t += gridDim.x) {
      unsigned long long acc[32];                        // two fp32 columns each
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = 0ull;
      const int row = ti.row0 + r_in_tile;
      const float* sa_row = p.sa + (size_t)(row < p.R ? row : 0) * kblocks;
      const float* sb_row = p.sb + ((size_t)ti.e * nb_total + ti.n_idx) * kblocks;
      auto scale_at = [&](int kb) {
        return kb < kblocks ? (row < p.R ? __ldg(sa_row + kb) : 0.f) * __ldg(sb_row + kb) : 0.f;
      };
      // The lanes' activation scales lie a row apart, 32 cache lines per load, and the operand ring leaves the L1 too small
      // to keep them: every load goes to L2.  They are requested F8_AHEAD K blocks ahead.
      float sc[F8_AHEAD];
#pragma unroll
      for (int i = 0; i < F8_AHEAD; ++i) sc[i] = scale_at(i);
      for (int kb = 0; ok && kb < kblocks; ++kb, ++it) {
        const uint32_t buf = it % F8_TBUF;
        const float now = sc[0];
#pragma unroll
        for (int i = 0; i + 1 < F8_AHEAD; ++i) sc[i] = sc[i + 1];
        sc[F8_AHEAD - 1] = scale_at(kb + F8_AHEAD);
        ok = mbar_wait_warp(&tfull_bar[buf], (it / F8_TBUF) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + (uint32_t(lg * 32) << 16) + buf * F8_BN + half * 64;
        uint32_t v0[32], v1[32];
        tmem_ld_32x32(taddr, v0);
        tmem_ld_32x32(taddr + 32, v1);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[buf]);     // the MMA warp may refill this buffer during the FMAs
        const unsigned long long s2 = f32x2(__float_as_uint(now), __float_as_uint(now));
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          acc[i] = fma_f32x2(f32x2(v0[2 * i], v0[2 * i + 1]), s2, acc[i]);
          acc[16 + i] = fma_f32x2(f32x2(v1[2 * i], v1[2 * i + 1]), s2, acc[16 + i]);
        }
      }
      // this group's 64 columns: swizzled staging (one buffer per group) -> TMA store
      if (store_thread) tma_store_wait_read<0>();
      if (half == 0) asm volatile("bar.sync 1, 128;" ::: "memory"); else asm volatile("bar.sync 2, 128;" ::: "memory");
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        float f[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          f[2 * i] = __uint_as_float((uint32_t)acc[g * 4 + i]);
          f[2 * i + 1] = __uint_as_float((uint32_t)(acc[g * 4 + i] >> 32));
        }
        *reinterpret_cast<bf16x8*>(sbuf + r_in_tile * 128 + ((g ^ (r_in_tile & 7)) << 4)) = pack8(f);
      }
      fence_proxy_async();
      if (half == 0) asm volatile("bar.sync 1, 128;" ::: "memory"); else asm volatile("bar.sync 2, 128;" ::: "memory");
      if (ok && store_thread) {
        tma_store_2d(&tmap_c, sbuf, ti.n_idx * F8_BN + half * 64, ti.row0);
        tma_store_commit();
      }
    }
    if (store_thread) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 100000) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, F8_TBUF * F8_BN);
  }
}

}  // namespace slab

// ---------------------------------------------------------------- host side (tensor maps: tma_host.cuh)
// Forward only.  Requires K % 128 == 0, N % 128 == 0, E <= 512; expert segments start on multiples of 128 rows.
extern "C" int slab_grouped_gemm_fp8(const void* A, const float* sa, const void* B, const float* sb, void* C,
                                     const int* seg_offsets, const int* seg_counts, int E, int R, int N, int K,
                                     int max_ctas, int* status, cudaStream_t stream) {
  using namespace slab;
  if (E > 512 || K % 128 || N % 128) return -100;
  Fp8Params p{seg_offsets, seg_counts, sa, sb, E, R, N, K, status};
  CUtensorMap ma, mb, mc;
  int rc;
  if ((rc = tma_make_map_2d(&ma, A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, R, K, K, F8_BM, F8_BK))) return rc;
  if ((rc = tma_make_map_2d(&mb, B, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)E * N, K, K, F8_BN, F8_BK))) return rc;
  if ((rc = tma_make_map_2d(&mc, C, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, R, N, N, F8_BM, 64))) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    SLAB_CUDA_CHECK(cudaFuncSetAttribute(grouped_gemm_fp8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F8_SMEM));
    attr_set = true;
  }
  int dev = 0, grid = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&grid, cudaDevAttrMultiProcessorCount, dev);
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  grouped_gemm_fp8_kernel<<<grid, F8_THREADS, F8_SMEM, stream>>>(ma, mb, mc, p);
  return (int)cudaGetLastError();
}
