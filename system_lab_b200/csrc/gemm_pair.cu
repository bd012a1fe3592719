// Grouped expert GEMM on pairs of SMs (tcgen05.mma.cta_group::2), bf16 or row-scaled e4m3.
//
// Rows are grouped by expert, every segment starts at a multiple of 128 rows and padding rows are zero:
//   FWD    C[r, n]    = sum_k A[r, k] * B[e, n, k]     A: acts [R, K]   B: weights [E, N, K]
//   DGRAD  C[r, k]    = sum_n A[r, n] * B[e, n, k]     A: dY   [R, N]   B: weights [E, N, K] (MN-major operand)
//   WGRAD  C[e, n, k] = sum_r A[r, n] * B[r, k]        A: dY   [R, N]   B: acts    [R, K]    (both MN-major)
//   row-scaled e4m3 (FWD only): the same product times sa[r] * sb[e, n]
//   WGRAD_T  WGRAD with the operands' sides exchanged (the tile is computed transposed), for N just over a multiple of 256
//
// Bound by the tensor pipe, its operand feed and, on long runs, the power cap.  What follows from that:
//  * Two CTAs share one instruction (256 x n): each stages 128 rows of the M operand and half of the N operand, so a CTA
//    fills 32 KB of shared memory per 64-deep step of a 256 x 256 tile where one CTA alone fills 48 KB for 128 x 256.
//  * FWD and DGRAD put the weights on the M side and the rows on the N side (the tile is computed transposed).  M is
//    fixed at 256, but n can be any multiple of 32: an expert's rows are cut into equal chunks of at most 256, so an
//    expert of 520 rows costs 544 columns of MMA time, not five 128-row tiles = 640.
//  * One TMA copy per operand and stage (MN-major operands are mapped as panels of 64 columns), issued like the MMAs by an
//    elected lane of a converged warp (elect_one): 640 -> 398 ns for a 64-deep step of 256 x 256 when both were done.
// The transposed accumulator is read with 16x256b loads, whose registers are 8x8 matrix fragments, and turned around by
// stmatrix.trans on its way to the swizzled staging buffer, so output rows still leave as 128-byte TMA stores.
//
// Measured against one CTA per 128 x 256 tile (cold L2, TFLOP/s without padding): [8192, 2048] x [5120, 2048]^T forward
// 1412 -> 1526, input gradient 1233 -> 1398, weight gradient 1104 -> 1261; 32 experts, 16384 rows, 7168 -> 4096: 1198 ->
// 1271, 1194 -> 1329, 1085 -> 1169; the same weight gradient added to an old one 5.7 -> 0.95 ms; 128 experts, 65536 rows,
// 768 -> 2048: 987 -> 1071; 7168 -> 4096 in e4m3: 2003 -> 2343.
//
// Roles per CTA (320 threads): warp 0 TMA producer, warp 1 MMA issuer (first CTA of the pair) and TMEM owner, warps 2..9
// epilogue, in two groups that take the 32-row steps (WGRAD: 64-column chunks) of a tile in turn: with short reductions
// (K = 768) one group alone is slower than the main loop.  Two 256-column accumulators overlap the epilogue of one tile
// with the main loop of the next.  Every wait is bounded (common.cuh); TMA loads carry no multicast: each CTA loads its
// own part.
#include "common.cuh"
#include "tma_host.cuh"

namespace slab {

constexpr int PG_THREADS = 320;
constexpr int PG_MAX_STAGES = 8;
constexpr int PG_OPERAND = 128 * 128;            // bytes of a whole operand in one stage: 128 rows of 128 bytes
constexpr int PG_PREFIX_OFF = 256;               // FWD / DGRAD: tiles before every expert, int [513]

// Shared memory: barriers, the tile prefix, {first row, rows} of every expert (every role looks one up per tile, and the
// ring leaves the L1 too small to keep them: 1000 cycles per tile from L2), operand ring, staging of the output.
template <int MODE>
struct PairSmem {
  static constexpr bool WGRAD = MODE == 2;
  static constexpr int SEG_OFF = WGRAD ? 256 : 2312;
  static constexpr int SEG_MAX = WGRAD ? 352 : 512;        // experts with an entry; the others' are read from memory
  static constexpr int CTRL = WGRAD ? 3072 : 7168;
  static constexpr int RING = WGRAD ? 5 * 2 * PG_OPERAND : 172 * 1024;     // what the rest leaves of the SM's 227 KB
  static constexpr int STORE_OFF = CTRL + RING;
  static constexpr int STORE_BUF = WGRAD ? 16384 : 8192;   // 128 rows x 64 columns, or 32 rows x 128 columns
  static constexpr int STORE_BUFS = WGRAD ? 2 : 3;         // per epilogue group
  static constexpr int STORE = STORE_BUF * STORE_BUFS;
  static constexpr int TOTAL = STORE_OFF + 2 * STORE;
  static_assert(SEG_OFF + SEG_MAX * 8 <= CTRL && CTRL % 1024 == 0 && TOTAL <= 232448, "shared memory budget");
};

// A stage holds 128 rows of the M operand and, for every chunk of rows up to `units` long, half of it in boxes of 32 rows.
// Short chunks leave room for more stages: 8 of 20 KB up to 64 rows, 7 up to 128, 6 up to 192, 5 of 32 KB.  With few rows per
// expert the product is bound by streaming the weights, and so by what is in flight: 32 experts x 37 rows, 2880 -> 2880, 104 us
// with 5 stages for every length, 97 with these.
__device__ __forceinline__ int pg_stage_bytes(int units) { return PG_OPERAND + (units + 1) / 2 * 4096; }
__device__ __forceinline__ int pg_stages(int units) { return 9 - (units + 1) / 2; }
static_assert(PG_MAX_STAGES * (PG_OPERAND + 4096) <= 172 * 1024 && 7 * (PG_OPERAND + 8192) <= 172 * 1024 &&
              6 * (PG_OPERAND + 12288) <= 172 * 1024 && 5 * 2 * PG_OPERAND <= 172 * 1024, "ring");

constexpr int PG_UNIT = 32;                      // rows per unit of an expert's chunk (the MMA's step in n)
constexpr int PG_MAX_UNITS = 8;
constexpr int PG_TILE_UNITS = 3;                 // what a tile costs beside its rows, in units (see pg_plan_tiles)

enum { PG_FWD = 0, PG_DGRAD = 1, PG_WGRAD = 2, PG_WGRAD_T = 3 };
__host__ __device__ constexpr bool pg_over_rows(int mode) { return mode >= PG_WGRAD; }      // the reduction runs over an expert's rows

// WGRAD: a group of epilogue warps stores a 16 KB chunk every PG_STORE_NS at most (one may come early), a little less than all of
// them together get from memory (5.9 TB/s).  With short reductions the launch is bound by writing its result.  The groups can
// produce it at twice that rate, and memory serves the SMs unevenly: those it favours end at 67 us of 92 and the others go on
// alone (8 experts x 25 rows into [4096, 7168], 470 MB).  Paced, all end together: 98 -> 86 us; 32 experts x 37 rows 410 -> 325,
// into [5760, 2880] 236 -> 198.  780 ns gives 84 there but 396 and 242, 840 ns with four chunks early 88, 332 and 234.
constexpr uint64_t PG_STORE_NS = 820;

struct PairParams {
  const int* seg_offsets;
  const int* seg_counts;
  int E, R, N, K;
  int width;                // WGRAD: columns of a tile on the N side, 256 or 128
  __nv_bfloat16* C;
  const float* sa;          // e4m3: [R]
  const float* sb;          // e4m3: [E, N]
  int* status;
  const int* ready;         // per-(source, expert) arrival flags of the rows (FWD / DGRAD), or null
  int ready_world, ready_epoch;
  unsigned long long ready_limit_ns;
};

// ---------------------------------------------------------------- PTX of the pair
__device__ __forceinline__ uint32_t pg_cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pg_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the first CTA's copy of a shared variable
__device__ __forceinline__ uint32_t pg_leader_addr(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
// What the waiter goes on to overwrite is tensor memory, whose reads tcgen05.wait::ld has completed: no order over other
// memory is needed.  A release at cluster scope waits for all the warp's stores first (2500 cycles per tile measured).
__device__ __forceinline__ void pg_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Load into this CTA's shared memory, bytes counted on a barrier of either CTA of the pair.
__device__ __forceinline__ void pg_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(dst),
      "l"(map), "r"(bar_cluster), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void pg_load_panels(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int row,
                                               int panel) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];" ::"r"(dst),
      "l"(map), "r"(bar_cluster), "r"(0), "r"(row), "r"(panel)
      : "memory");
}
template <bool FP8>
__device__ __forceinline__ void pg_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  if (FP8)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive on both CTAs' copy of a barrier once every MMA issued so far has completed.
__device__ __forceinline__ void pg_commit_both(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
// 16 lanes x 32 fp32 columns.  Registers 4j .. 4j+3 of thread i: row i / 4, columns 8j + 2 (i % 4) and the next, then
// the same columns of row i / 4 + 8: the fragment of two 8x8 matrices.
__device__ __forceinline__ void pg_tmem_ld_16x32(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void pg_stmatrix_trans(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(a), "r"(b),
               "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ void pg_group_sync(int grp) {
  asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory");
}
__device__ __forceinline__ uint32_t pg_pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// ---------------------------------------------------------------- tile walk
// FWD / DGRAD: experts in order, inside an expert the row chunk runs fastest (pairs that run together share the weight
// tile in L2).  WGRAD: experts in order, the 256-row block of the output runs fastest.
struct PairTile {
  int e, ob, cb;            // expert, 256-wide block on the M side, (WGRAD) block of columns on the N side
  int row0, n;              // first row of the chunk; n of the MMA
  int width;                // WGRAD: columns of a tile
  int zero_steps;           // FWD / DGRAD: 32-row steps behind the chunk up to the segment's 128-row boundary
  int ksteps, mmas;         // stages, and MMAs over all of them
};

// {first row, rows} of an expert's segment: a corrupt plan must not turn into a runaway tile walk
__device__ __forceinline__ int2 pg_clip(const PairParams& p, int2 s) {
  if (s.x < 0 || s.x >= p.R || s.y <= 0) return make_int2(0, 0);
  return make_int2(s.x, s.y < p.R - s.x ? s.y : p.R - s.x);
}
__device__ __forceinline__ int2 pg_segment(const PairParams& p, int e) {
  return pg_clip(p, make_int2(p.seg_offsets[e], p.seg_counts[e]));
}

// On entry ti.e holds the expert of the tile visited before (0 at first).
template <int MODE, bool FP8>
__device__ __forceinline__ void pg_get_tile(int t, const int* prefix, const int2* segs, int max_units, const PairParams& p,
                                            PairTile& ti) {
  constexpr int BKE = FP8 ? 128 : 64;
  if (pg_over_rows(MODE)) {
    const int side_m = MODE == PG_WGRAD_T ? p.K : p.N, side_n = MODE == PG_WGRAD_T ? p.N : p.K;
    const int obs = (side_m + 255) >> 8, per = obs * ((side_n + p.width - 1) / p.width);
    ti.e = t / per;
    ti.zero_steps = 0;
    const int local = t - ti.e * per;
    ti.cb = local / obs;
    ti.ob = local - ti.cb * obs;
    const int2 seg = ti.e < PairSmem<MODE>::SEG_MAX ? segs[ti.e] : pg_segment(p, ti.e);
    const int rows = seg.y;
    ti.row0 = seg.x;
    ti.width = p.width;
    ti.n = side_n - ti.cb * p.width > 128 ? p.width : 128;       // half of it is whole 64-column panels; what lies beyond reads as zero
    ti.ksteps = (rows + BKE - 1) / BKE;
    ti.mmas = (rows + 15) >> 4;                          // rows behind the last valid one are zero: whole MMAs of them are left out
    return;
  }
  int lo = ti.e;                                         // tiles are visited in ascending order: at or behind the last expert
  while (prefix[lo + 1] <= t) ++lo;
  const int local = t - prefix[lo];
  const int2 seg = segs[lo];
  const int units = (seg.y + PG_UNIT - 1) / PG_UNIT;
  const int chunks = (units + max_units - 1) / max_units;
  const int ci = local % chunks;
  const int base = units / chunks, rem = units - base * chunks;
  ti.e = lo;
  ti.cb = ti.width = 0;
  ti.ob = local / chunks;
  ti.row0 = seg.x + (ci * base + min(ci, rem)) * PG_UNIT;
  ti.n = (base + (ci < rem ? 1 : 0)) * PG_UNIT;
  ti.zero_steps = ci == chunks - 1 ? ((units + 3) & ~3) - units : 0;
  ti.ksteps = ((MODE == PG_FWD) ? p.K : p.N) / BKE;
  ti.mmas = ti.ksteps * 4;
}

// The same in all lanes, visibly (see elect_one).
__device__ __forceinline__ void pg_uniform(PairTile& ti) {
  ti.e = warp_uniform(ti.e);
  ti.ob = warp_uniform(ti.ob);
  ti.cb = warp_uniform(ti.cb);
  ti.row0 = warp_uniform(ti.row0);
  ti.n = warp_uniform(ti.n);
  ti.ksteps = warp_uniform(ti.ksteps);
  ti.mmas = warp_uniform(ti.mmas);
}

// Largest chunk (in 32-row units): the one whose waves of tiles cost least, the mean tile of n columns taken as n + 96: a
// 64-deep step of n columns takes 249 ns at 128 and 398 ns at 256, because the weights' half of the operands is staged
// whatever n is.  Over 166 products (13 dense and 11 grouped shapes of 128 to 20000 rows, forward and input gradient) the choice is
// within 0.3 % of the best of all eight in the mean and 5 % at worst; with n + 32 it was 2.1 % and 26 % (input gradient of
// [4096, 7168] x [2048, 7168] 108.8 us in chunks of 160 where 256 take 90.3).
// One warp; writes the segments and the tile prefix over experts, and returns the choice and a bound on the chunks it makes.
__device__ __forceinline__ int2 pg_plan_tiles(const PairParams& p, int obs, int pairs, int* prefix, const int2* segs) {
  const int lane = threadIdx.x & 31;
  int tiles[PG_MAX_UNITS - 1], total = 0, longest = 0;
#pragma unroll
  for (int j = 0; j < PG_MAX_UNITS - 1; ++j) tiles[j] = 0;
  // Small loops: a launch finds its instructions in no cache, and unrolled for 512 experts this took 3000 cycles of 4500 before the
  // first copy (a launch without rows: 4.3 us for 1 expert, 5.0 for 128; 2.6 and 3.3 now).  A lane has neighbouring experts,
  // so that one scan over the warp gives the prefix.
  const int per = (p.E + 31) >> 5, e0 = lane * per, e1 = min(p.E, e0 + per);
#pragma unroll 1
  for (int e = e0; e < e1; ++e) {
    const int u = (segs[e].y + PG_UNIT - 1) / PG_UNIT;
    total += u;
    longest = max(longest, u);
#pragma unroll
    for (int j = 0; j < PG_MAX_UNITS - 1; ++j) tiles[j] += (u + j + 1) / (j + 2);
  }
  total = __reduce_add_sync(0xffffffffu, total);
  longest = __reduce_max_sync(0xffffffffu, longest);
  int best = PG_MAX_UNITS;
  float best_cost = INFINITY;
#pragma unroll
  for (int mu = PG_MAX_UNITS; mu >= 2; --mu) {
    const int t = __reduce_add_sync(0xffffffffu, tiles[mu - 2]);
    // (single precision throughout: 64-bit divisions here cost a microsecond per launch)
    const float waves = ceilf(__fdividef((float)t * (float)obs, (float)pairs));
    const float cost = __fdividef(waves * (float)(total + PG_TILE_UNITS * t), (float)max(t, 1));
    if (cost < best_cost) { best_cost = cost; best = mu; }
  }
  // ceil(units / best) without a division: exact below 2^29
  const uint32_t inverse = 0xffffffffu / (uint32_t)best + 1;
  auto tiles_of = [&](int e) { return (int)__umulhi((segs[e].y + PG_UNIT - 1) / PG_UNIT + best - 1, inverse) * obs; };
  int mine = 0;
#pragma unroll 1
  for (int e = e0; e < e1; ++e) mine += tiles_of(e);
  int acc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, acc, o);
    if (lane >= o) acc += v;
  }
  if (lane == 31) prefix[p.E] = acc;
  acc -= mine;
#pragma unroll 1
  for (int e = e0; e < e1; ++e) {
    prefix[e] = acc;
    acc += tiles_of(e);
  }
  return make_int2(best, max(min(longest, best), 1));
}

// Tensor maps.  w: M-side operand (weights; WGRAD: dY), x: N-side operand in boxes of 32, 64, 96 and 128 rows (WGRAD: x[2]
// one panel, x[3] two), c: result.  MN-major operands are mapped as panels of 64 columns.
struct PairMaps {
  CUtensorMap w, c, x[4];
};

// ACC: WGRAD adds to the old result.
template <int MODE, bool FP8, bool ACC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PG_THREADS, 1)
pair_gemm_kernel(const __grid_constant__ PairMaps maps, const PairParams p) {
  using L = PairSmem<MODE>;
  constexpr bool RED = pg_over_rows(MODE);
  constexpr bool W_MN = MODE != PG_FWD, X_MN = RED;
  constexpr int BKE = FP8 ? 128 : 64;
  extern __shared__ __align__(1024) uint8_t smem[];
  // (24 barriers side by side, see the initialisation)
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);           // first CTA's copy counts both CTAs' bytes
  uint64_t* empty_bar = full_bar + PG_MAX_STAGES;
  uint64_t* tfull_bar = empty_bar + PG_MAX_STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;                             // first CTA's copy counts both CTAs' epilogue warps
  uint64_t* old_bar = tempty_bar + 2;                               // WGRAD, accumulate: a chunk of the old result is here (two per group)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(old_bar + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int2* units_slot = reinterpret_cast<int2*>(tmem_slot + 2);        // largest chunk allowed, and none is longer than
  int* prefix = reinterpret_cast<int*>(smem + PG_PREFIX_OFF);
  int2* segs = reinterpret_cast<int2*>(smem + L::SEG_OFF);
  uint8_t* ring = smem + L::CTRL;
  uint8_t* store_buf = smem + L::STORE_OFF;
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t cta = pg_cta_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int out_cols = MODE == PG_FWD ? p.N : p.K;

  if (warp == 0) {
    if (lane < 2 * PG_MAX_STAGES + 8) {
      mbar_init(&full_bar[lane], &full_bar[lane] == &tempty_bar[0] || &full_bar[lane] == &tempty_bar[1] ? 16 : 1);
      fence_mbar_init();
    }
    if (lane == 0) {
      if (smem_u32(smem) & 1023u) atomicCAS(p.status, 0, ST_BAD_INDEX);   // the runtime aligns it; swizzled tiles rely on it
      *abort_flag = 0;
      prefetch_tmap(&maps.w);
      prefetch_tmap(&maps.x[3]);
      prefetch_tmap(&maps.c);
    }
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (warp >= 2)
    for (int e = threadIdx.x - 64; e < p.E && e < L::SEG_MAX; e += PG_THREADS - 64) segs[e] = pg_segment(p, e);
  if (!RED && warp >= 2) asm volatile("bar.sync 3, 256;" ::: "memory");
  if (!RED && warp == 2) {
    const int2 mu = pg_plan_tiles(p, (out_cols + 255) >> 8, pairs, prefix, segs);
    if (lane == 0) *units_slot = mu;
  }
  tc_fence_before();
  __syncwarp();
  pg_cluster_sync();                              // this CTA's set-up is done, and the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const int max_units = RED ? 0 : units_slot->x;
  const int side_m = MODE == PG_WGRAD ? p.N : p.K, side_n = MODE == PG_WGRAD ? p.K : p.N;
  const int tiles = warp_uniform(RED ? ((side_m + 255) >> 8) * ((side_n + p.width - 1) / p.width) * p.E : prefix[p.E]);
  const int stage_bytes = RED ? 2 * PG_OPERAND : warp_uniform(pg_stage_bytes(units_slot->y));
  // A pair with fewer tiles than others takes its share of the ring only: with few rows the launch is bound by memory, and the
  // pairs that have most to fetch should have most in flight (8 experts x 25 rows, 224 tiles of 4096 x 256: 87 -> 80 us; 96
  // tiles of 5760 x 256: 65 -> 55).
  const float waves = __fdividef((float)tiles, (float)pairs);
  int stages = RED ? 5 : pg_stages(units_slot->y);
  const int each = (int)waves;                    // (both CTAs and all roles get the same, whatever it is rounded to)
  if (pair >= tiles - each * pairs && tiles > each * pairs)
    stages = max((int)ceilf(__fdividef((float)(stages * each), (float)(each + 1))), 2);
  stages = warp_uniform(stages);

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    int s = 0;
    uint32_t ph = 0;
    int last_e = -1;
    bool ok = true;
    const uint32_t ring_addr = smem_u32(ring);
    const uint32_t bar0 = (uint32_t)warp_uniform((int)pg_leader_addr(full_bar));
    PairTile ti;
    ti.e = 0;
    for (int t = pair; ok && t < tiles; t += pairs) {
      pg_get_tile<MODE, FP8>(t, prefix, segs, max_units, p, ti);
      pg_uniform(ti);
      if (!RED && p.ready != nullptr && ti.e != last_e) {
        // rows arrive expert by expert from the sources: one flag per lane; the proxy fence orders the TMA reads
        // behind the acquired generic-proxy stores
        bool mine = true;
        if (lane < p.ready_world)
          mine = wait_flag_ge(p.ready + lane * p.E + ti.e, p.ready_epoch, p.status, p.ready_limit_ns);
        ok = __all_sync(0xffffffffu, mine);
        if (!ok) {
          if (lane == 0) *abort_flag = 1;
          break;
        }
        asm volatile("fence.proxy.async.global;" ::: "memory");
        last_e = ti.e;
      }
      const int half = ti.n >> 1;
      const int units = X_MN ? 4 : (half + 31) >> 5;
      const uint32_t bytes = 2u * (PG_OPERAND + (X_MN ? half * 128 : units * 4096));      // of both CTAs
      const int w_row = ti.e * p.N, m0 = ti.ob * 256 + (int)cta * 128;
      const int x0 = RED ? ti.cb * p.width + (int)cta * half : ti.row0 + (int)cta * half;
      const CUtensorMap* x_map = &maps.x[X_MN ? (half == 128 ? 3 : 2) : units - 1];
      for (int ks = 0; ks < ti.ksteps; ++ks) {
        ok = mbar_wait_warp(&empty_bar[s], ph ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY);
        if (!ok) break;
        const uint32_t w_dst = ring_addr + s * stage_bytes, x_dst = w_dst + PG_OPERAND, bar = bar0 + s * 8;
        if (elect_one()) {
          if (cta == 0) mbar_arrive_expect_tx(&full_bar[s], bytes);
          if (W_MN) pg_load_panels(w_dst, &maps.w, bar, (RED ? ti.row0 : w_row) + ks * BKE, m0 >> 6);
          else pg_load_2d(w_dst, &maps.w, bar, ks * BKE, w_row + m0);
          if (X_MN) pg_load_panels(x_dst, x_map, bar, ti.row0 + ks * BKE, x0 >> 6);
          else pg_load_2d(x_dst, x_map, bar, ks * BKE, x0);
        }
        if (++s == stages) { s = 0; ph ^= 1; }
      }
    }
    // the first CTA's commits arrive on both CTAs: all of them have before this CTA may leave
    for (int i = 0; ok && pair < tiles && i < stages; ++i) {
      ok = mbar_wait(&empty_bar[s], ph ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY);
      if (++s == stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (first CTA, for both)
    if (cta == 0) {
      // K-major: 32 bytes per MMA inside the 128-byte swizzle row; MN-major: 16 reduction rows of 128 bytes
      constexpr uint32_t W_STEP = W_MN ? 2048 >> 4 : 32 >> 4, X_STEP = X_MN ? 2048 >> 4 : 32 >> 4;
      const uint32_t ring_addr = smem_u32(ring);
      const uint64_t wd0 = W_MN ? make_smem_desc(ring_addr, 8192, 1024, 2) : make_smem_desc(ring_addr, 16, 1024, 2);
      const uint64_t xd0 = X_MN ? make_smem_desc(ring_addr + PG_OPERAND, 8192, 1024, 2)
                                : make_smem_desc(ring_addr + PG_OPERAND, 16, 1024, 2);
      int s = 0;
      uint32_t ph = 0;
      int it = 0;
      bool ok = true;
      PairTile ti;
      ti.e = 0;
      for (int t = pair; ok && t < tiles; t += pairs) {
        pg_get_tile<MODE, FP8>(t, prefix, segs, max_units, p, ti);
        pg_uniform(ti);
        if (ti.ksteps == 0) continue;
        const int buf = it & 1;
        ok = mbar_wait_warp(&tempty_bar[buf], ((it >> 1) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem_base + buf * 256;
        const uint32_t idesc = make_idesc(FP8 ? 0 : 1, FP8 ? 0 : 1, W_MN ? 1 : 0, X_MN ? 1 : 0, 256, ti.n);
        int left = ti.mmas;
        for (int ks = 0; ks < ti.ksteps; ++ks) {
          ok = mbar_wait_warp(&full_bar[s], ph, abort_flag, p.status, ST_TIMEOUT_FULL);
          if (!ok) break;
          tc_fence_after();
          const uint64_t wd = wd0 + (uint32_t)(s * (stage_bytes >> 4)), xd = xd0 + (uint32_t)(s * (stage_bytes >> 4));
          if (elect_one()) {
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4)
              if (!RED || k4 < left)
                pg_mma<FP8>(d, wd + k4 * W_STEP, xd + k4 * X_STEP, idesc, (ks | k4) != 0 ? 1u : 0u);
            pg_commit_both(&empty_bar[s]);
            if (ks == ti.ksteps - 1) pg_commit_both(&tfull_bar[buf]);
          }
          left -= 4;
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        ++it;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9 of both CTAs)
    const int lg = warp & 3;                      // TMEM lane group this warp may read
    const int grp = (warp - 2) >> 2;
    const bool store_thread = (warp == 2 || warp == 6) && lane == 0;
    uint8_t* const stage = store_buf + grp * L::STORE;
    uint64_t* const old_g = old_bar + 2 * grp;
    int it = 0, ctr = 0;
    int slot = 0;                                 // FWD / DGRAD: staging buffer in turn
    uint64_t due = 0;                             // WGRAD: when this group's next chunk may be stored
    bool ok = true;                               // no wait of this warp has run out (see mbar_wait_warp)
    PairTile ti;
    ti.e = 0;
    for (int t = pair; t < tiles; t += pairs) {
      pg_get_tile<MODE, FP8>(t, prefix, segs, max_units, p, ti);
      const bool empty = RED && ti.ksteps == 0;   // an expert without rows: its weight gradient is zero
      const int m0 = ti.ob * 256 + (int)cta * 128;
      const int buf = it & 1;
      const uint32_t taddr = tmem_base + (uint32_t(lg * 32) << 16) + buf * 256;
      // WGRAD: 64-column chunks of this CTA's 128 rows (none beyond the expert's N; the output map clips a block that hangs over
      // it).  A sum onto the old result has that brought in by TMA too (a thread's own row is a line per access when read from
      // global memory), one chunk ahead.
      const int col0 = ti.cb * ti.width;
      const int chunks = m0 >= p.N || (ACC && empty) ? 0 : min(ti.width, p.K - col0) >> 6;
      if (ACC && grp < chunks && ok && store_thread) {
        tma_store_wait_read<0>();
        mbar_arrive_expect_tx(&old_g[ctr & 1], 16384);
        tma_load_3d(stage + (ctr & 1) * 16384, &maps.c, &old_g[ctr & 1], col0 + grp * 64, m0, ti.e);
      }
      // e4m3: channel scales (channels lane / 4 + 0, 8, 16, 24 of this warp's 32) and the scale of row `lane` of the group's
      // first step are requested before the accumulator is waited for
      float sb[4] = {1.f, 1.f, 1.f, 1.f}, sa_next = 0.f;
      if (FP8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int ch = m0 + lg * 32 + i * 8 + (lane >> 2);
          sb[i] = ch < p.N ? __ldg(p.sb + (size_t)ti.e * p.N + ch) : 0.f;
        }
        const int r = ti.row0 + grp * PG_UNIT + lane;
        sa_next = r < p.R ? __ldg(p.sa + r) : 0.f;
      }
      if (!empty) {
        ok = ok && mbar_wait_warp(&tfull_bar[buf], (it >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
        tc_fence_after();
      }
      if (MODE != PG_WGRAD) {
        const int first = MODE == PG_WGRAD_T ? ti.cb * ti.width : ti.row0;
        const int all = MODE == PG_WGRAD_T ? min(ti.width, p.N - first) / PG_UNIT : ti.n / PG_UNIT + ti.zero_steps;
        const int steps = MODE != PG_WGRAD_T ? ti.n / PG_UNIT : empty ? 0 : all;
        bool held = !empty;                       // this warp has not handed the accumulator back yet
#pragma unroll 1
        for (int st = grp; st < all; st += 2) {
          // rows 8j + 2 (lane % 4) and the next one of this step's 32
          const int row = first + st * PG_UNIT;
          uint32_t v[2][16];
          float sa[4][2];
          if (st < steps) {
            pg_tmem_ld_16x32(taddr + st * PG_UNIT, v[0]);
            pg_tmem_ld_16x32(taddr + st * PG_UNIT + (16u << 16), v[1]);
            if (FP8) {
              const float sa_now = sa_next;
              const int r = row + 2 * PG_UNIT + lane;         // the group's next step
              sa_next = r < p.R && st + 2 < steps ? __ldg(p.sa + r) : 0.f;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                sa[j][0] = __shfl_sync(0xffffffffu, sa_now, 8 * j + 2 * (lane & 3));
                sa[j][1] = __shfl_sync(0xffffffffu, sa_now, 8 * j + 2 * (lane & 3) + 1);
              }
            }
            tmem_ld_wait();
            if (st + 2 >= steps) {                // this warp's last read: the MMA issuer may refill what all have read
              held = false;
              tc_fence_before();
              __syncwarp();
              if (lane == 0) pg_arrive_remote(pg_leader_addr(&tempty_bar[buf]));
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[0][i] = v[1][i] = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) sa[j][0] = sa[j][1] = 0.f;
          }
          uint8_t* sbuf = stage + slot * L::STORE_BUF + (lg >> 1) * 4096;
          const int chunk = (lg & 1) * 4 + (lane >> 3);          // 16-byte chunk (8 channels) this lane addresses
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t m[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float f0 = __uint_as_float(v[i >> 1][4 * j + 2 * (i & 1)]);
              float f1 = __uint_as_float(v[i >> 1][4 * j + 2 * (i & 1) + 1]);
              if (FP8) {
                f0 = f0 * sa[j][0] * sb[i];
                f1 = f1 * sa[j][1] * sb[i];
              }
              m[i] = pg_pack(f0, f1);
            }
            const int r = 8 * j + (lane & 7);
            pg_stmatrix_trans(smem_u32(sbuf) + r * 128 + ((chunk ^ (r & 7)) << 4), m[0], m[1], m[2], m[3]);
          }
          fence_proxy_async();
          // three buffers in turn: all but the last store have been read, so the next buffer is free
          if (store_thread) tma_store_wait_read<1>();
          pg_group_sync(grp);
          if (ok && store_thread) {
            const uint8_t* b = stage + slot * L::STORE_BUF;
            if (MODE == PG_WGRAD_T) {
              if (m0 < out_cols) tma_store_3d(&maps.c, b, m0, row, ti.e);
              if (m0 + 64 < out_cols) tma_store_3d(&maps.c, b + 4096, m0 + 64, row, ti.e);
            } else {
              if (m0 < out_cols && row < p.R) tma_store_2d(&maps.c, b, m0, row);
              if (m0 + 64 < out_cols && row < p.R) tma_store_2d(&maps.c, b + 4096, m0 + 64, row);
            }
            tma_store_commit();
          }
          if (++slot == L::STORE_BUFS) slot = 0;
        }
        if (held) {                               // a tile of one step has none for the second group
          tc_fence_before();
          __syncwarp();
          if (lane == 0) pg_arrive_remote(pg_leader_addr(&tempty_bar[buf]));
        }
      } else {
        const int r_in_tile = lg * 32 + lane;
#pragma unroll 1
        for (int c = grp; c < chunks; c += 2) {
          uint32_t lo[32], hi[32];
          if (!empty) {
            tmem_ld_32x32(taddr + c * 64, lo);
            tmem_ld_32x32(taddr + c * 64 + 32, hi);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) lo[i] = hi[i] = 0u;
          }
          uint8_t* sbuf = stage + (ctr & 1) * 16384;
          if (ACC) {
            ok = ok && mbar_wait_warp(&old_g[ctr & 1], (ctr >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL);
            if (ok && store_thread && c + 2 < chunks) {   // the group's next chunk, into the buffer whose store came before this one
              tma_store_wait_read<0>();
              mbar_arrive_expect_tx(&old_g[(ctr + 1) & 1], 16384);
              tma_load_3d(stage + ((ctr + 1) & 1) * 16384, &maps.c, &old_g[(ctr + 1) & 1], col0 + c * 64 + 128, m0, ti.e);
            }
          } else {
            if (store_thread) tma_store_wait_read<1>();
            pg_group_sync(grp);
          }
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const uint32_t* v = g < 4 ? lo + g * 8 : hi + (g - 4) * 8;
            bf16x8* dst = reinterpret_cast<bf16x8*>(sbuf + r_in_tile * 128 + ((g ^ (r_in_tile & 7)) << 4));
            float f[8], o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(v[i]);
            if (ACC) {
              unpack8(*dst, o);
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i] += o[i];
            }
            *dst = pack8(f);
          }
          fence_proxy_async();
          pg_group_sync(grp);
          if (store_thread) {                     // see PG_STORE_NS
            uint64_t now = globaltimer_ns();
            for (int spins = 0; now < due && spins < 1000; ++spins) now = globaltimer_ns();
            due = max(due + PG_STORE_NS, now);
          }
          if (ok && store_thread) {
            tma_store_3d(&maps.c, sbuf, col0 + c * 64, m0, ti.e);
            tma_store_commit();
          }
          ++ctr;
        }
        if (!empty) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) pg_arrive_remote(pg_leader_addr(&tempty_bar[buf]));
        }
      }
      if (!empty) ++it;
    }
    if (store_thread) tma_store_wait<0>();
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // give copies that are still in flight time to land before shared memory is handed on
    uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 100000) __nanosleep(1000);
    __syncthreads();
  }
  __syncwarp();
  pg_cluster_sync();                              // the peer still counts bytes and arrivals in this CTA until here
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

template <int MODE, bool FP8, bool ACC = false>
static int pg_launch(const void* A, const void* B, const PairParams& p, int max_ctas, cudaStream_t stream) {
  constexpr CUtensorMapDataType DT = FP8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  constexpr int ES = FP8 ? 1 : 2, BKE = FP8 ? 128 : 64;
  PairMaps m;
  const uint64_t wrows = (uint64_t)p.E * p.N;
  int rc;
  if (pg_over_rows(MODE)) {
    const bool t = MODE == PG_WGRAD_T;
    const void *w = t ? B : A, *x = t ? A : B;
    const int side_m = t ? p.K : p.N, side_n = t ? p.N : p.K;
    if ((rc = tma_make_map_2d(&m.w, w, DT, ES, p.R, side_m, side_m, 64, 64, 2))) return rc;
    if ((rc = tma_make_map_2d(&m.x[3], x, DT, ES, p.R, side_n, side_n, 64, 64, 2))) return rc;
    if ((rc = tma_make_map_2d(&m.x[2], x, DT, ES, p.R, side_n, side_n, 64, 64, 1))) return rc;
    m.x[0] = m.x[1] = m.x[2];
    if ((rc = tma_make_map_2d(&m.c, p.C, DT, ES, p.N, p.K, p.K, t ? 32 : 128, 64, -p.E))) return rc;
  } else {
    const int red = MODE == PG_FWD ? p.K : p.N;
    if (MODE == PG_FWD) rc = tma_make_map_2d(&m.w, B, DT, ES, wrows, p.K, p.K, 128, BKE);
    else rc = tma_make_map_2d(&m.w, B, DT, ES, wrows, p.K, p.K, 64, 64, 2);
    if (rc) return rc;
    for (int i = 0; i < 4; ++i)
      if ((rc = tma_make_map_2d(&m.x[i], A, DT, ES, p.R, red, red, 32 * (i + 1), BKE))) return rc;
    if ((rc = tma_make_map_bf16(&m.c, p.C, p.R, MODE == PG_FWD ? p.N : p.K, 32, 64))) return rc;
  }
  auto kern = pair_gemm_kernel<MODE, FP8, ACC>;
  static bool attr_set = false;
  if (!attr_set) {
    SLAB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem<MODE>::TOTAL));
    attr_set = true;
  }
  int grid = sm_count();
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  grid = grid < 2 ? 2 : grid & ~1;
  kern<<<grid, PG_THREADS, PairSmem<MODE>::TOTAL, stream>>>(m, p);
  return (int)cudaGetLastError();
}

// What the waves of tiles cost with `side_m` on the M side: a tile of 128 columns takes 0.62 of one of 256 (249 against 398 ns per
// 64-deep step), and so does a last tile of at most 128.
static float pg_wgrad_cost(int E, int side_m, int side_n, int width, int pairs) {
  const int cbs = (side_n + width - 1) / width, last = side_n - (cbs - 1) * width;
  const long tiles = (long)E * ((side_m + 255) / 256) * cbs;
  const float mean = ((cbs - 1) * (width == 256 ? 1.f : 0.62f) + (last > 128 ? 1.f : 0.62f)) / cbs;
  return (float)((tiles + pairs - 1) / pairs) * mean;
}

}  // namespace slab

extern "C" unsigned long long slab_moe_wait_limit_ns();

// mode: 0 fwd, 1 dgrad, 2 wgrad.  Shapes: see the header comment.  Requires K % 64 == 0, N % 64 == 0, at most 512
// experts.  `status` is a device int the kernel sets on a bounded-wait timeout (0 = ok).  Returns a CUDA/driver error code
// (0 = launched).  `max_ctas` > 0 bounds the CTAs (rounded down to pairs, at least one pair).
// `ready` (optional, modes 0 and 1): per-(source, expert) arrival flags of the row operand, int [ready_world][E] in
// this GPU's memory; the kernel waits (bounded) for all `ready_world` flags of an expert to reach `ready_epoch`
// before it loads that expert's rows.  Null: the operand is complete when the kernel starts.
extern "C" int slab_grouped_gemm_bf16(int mode, const void* A, const void* B, void* C, const int* seg_offsets,
                                      const int* seg_counts, int E, int R, int N, int K, int accumulate,
                                      int max_ctas, const int* ready, int ready_world, int ready_epoch, int* status,
                                      cudaStream_t stream) {
  using namespace slab;
  if (E > 512 || K % 64 || N % 64) return -100;
  if (ready && (ready_world < 1 || ready_world > 32 || mode == PG_WGRAD)) return -102;
  // WGRAD: the width of tiles, and the side of the operands, whose waves cost least.  Exchanged sides have to be a tenth better: they
  // are where N is just over a multiple of 256 (4096 rows into [576, 7168]: 52 us as three blocks of which 0.75 are empty, 37 us
  // exchanged, 38 on one CTA per 128 x 256).  They do not add to an old result, which would have to come in transposed.
  const int pairs = (max_ctas > 1 && max_ctas < sm_count() ? max_ctas : sm_count()) / 2;
  const float c256 = pg_wgrad_cost(E, N, K, 256, pairs), c128 = pg_wgrad_cost(E, N, K, 128, pairs);
  const float t256 = pg_wgrad_cost(E, K, N, 256, pairs), t128 = pg_wgrad_cost(E, K, N, 128, pairs);
  const bool exchange = mode == PG_WGRAD && !accumulate && fminf(t256, t128) < 0.9f * fminf(c256, c128);
  const int width = (exchange ? t128 < t256 : c128 < c256) ? 128 : 256;
  PairParams p{seg_offsets, seg_counts, E, R, N, K, width, static_cast<__nv_bfloat16*>(C), nullptr, nullptr, status, ready, ready_world, ready_epoch, slab_moe_wait_limit_ns()};
  switch (mode) {
    case PG_FWD: return pg_launch<PG_FWD, false>(A, B, p, max_ctas, stream);
    case PG_DGRAD: return pg_launch<PG_DGRAD, false>(A, B, p, max_ctas, stream);
    case PG_WGRAD:
      if (exchange) return pg_launch<PG_WGRAD_T, false>(A, B, p, max_ctas, stream);
      return accumulate ? pg_launch<PG_WGRAD, false, true>(A, B, p, max_ctas, stream)
                        : pg_launch<PG_WGRAD, false>(A, B, p, max_ctas, stream);
  }
  return -101;
}

// Row-scaled e4m3 forward: sa [R], sb [E, N].  Requires K % 128 == 0, N % 64 == 0, at most 512 experts.
extern "C" int slab_grouped_gemm_fp8_rowwise(const void* A, const float* sa, const void* B, const float* sb, void* C,
                                             const int* seg_offsets, const int* seg_counts, int E, int R, int N,
                                             int K, int max_ctas, int* status, cudaStream_t stream) {
  using namespace slab;
  if (E > 512 || K % 128 || N % 64) return -100;
  PairParams p{seg_offsets, seg_counts, E, R, N, K, 256, static_cast<__nv_bfloat16*>(C), sa, sb, status,
               nullptr, 0, 0, 0};
  return pg_launch<PG_FWD, true>(A, B, p, max_ctas, stream);
}
