// bf16 GEMM for few activation rows: C[M, N] = X[M, K] * W^T, M from a batch of decoding sequences to some hundred rows
// of a prompt.  Such a product has too few 128- or 256-row tiles to occupy the chip (48 x 2560 is ten tiles of 128 x 256) and is
// bound by how many SMs stream the weights, so
//   * the weights take the 128-row side of the MMA and the activation rows its N side: a tile is 128 weight rows by
//     `bt` activation rows (a multiple of 16 up to 256), and nothing is staged or multiplied for absent rows;
//   * K is split over the `split` CTAs of a cluster (1, 2, 4 or 8).  Each leaves its fp32 partial tile in its shared
//     memory, and the cluster adds the parts in rank order (the same order every time) through distributed shared
//     memory, each CTA a share of the rows: no workspace, no atomics, no second launch.
// Measured against 128 x 256 tiles on single CTAs (weights from memory): 48 rows x 2560 x 9728 58.5 -> 18.1 us, 333 rows 61.1 ->
// 28.9, 48 rows x 6144 x 2560 20.1 -> 14.1; with the activation, 48 rows x 19456 x 2560 36.2 -> 23.1 (two launches -> one).
// The weights alone take 7.6, 7.6, 4.8 and 15.2 us at the copy bandwidth.  Row-major weights whose rows start on 128-byte lines go to
// csrc/gemm_tall.cu where that gives no CTA too many of them (13.2 us for the first of these; ksa_gemm_tall_plan), [K, N] weights of any number of rows
// and the rest stay here, most from 257 rows on, as that kernel reads the activations again for every tile.
// Roles per CTA (192 threads): warp 0 TMA producer, warp 1 MMA issuer, warps 2..5 move the accumulator to shared
// memory, and all of them write the result.  One tile per CTA.  No TMA load uses multicast; every wait is bounded.
//
// kGlu: W holds F gate rows followed by F up rows, a tile is 64 features (64 gate rows and the matching 64 up rows) and
// C[M, F] = silu(gate) * up, with gate and up rounded to bf16 first as separate projection and activation kernels do.
#include "common.cuh"
#include "host.h"

namespace ksa {

constexpr int kNwThreads = 192;
constexpr int kNwBK = 64;
constexpr int kNwWBytes = 128 * kNwBK * 2;
constexpr int kNwMaxStages = 8;

struct NarrowArgs {
  bf16* c;
  long long ldc;
  int M, N, K;               // N: rows of W
  int bt, split, stages, tiles_m, tmem_cols;
  float alpha;
  int beside;                // launch_beside()
};

__device__ __forceinline__ uint32_t nw_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void nw_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 nw_ld_cluster(uint32_t local_addr, uint32_t rank) {
  float4 v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\t"
               "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(local_addr), "r"(rank)
               : "memory");
  return v;
}

template <bool W_MN, bool kGlu>
__global__ void __launch_bounds__(kNwThreads)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const NarrowArgs p,
                   int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[kNwMaxStages], empty[kNwMaxStages], acc_full;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)nw_cluster_rank();
  const int tile = (int)blockIdx.x / p.split;
  const int mb = tile % p.tiles_m, nb = tile / p.tiles_m;   // tiles that share weights are neighbours
  const int m0 = mb * p.bt;
  const int num_kb = (p.K + kNwBK - 1) / kNwBK;
  const int kb0 = (int)((long long)num_kb * rank / p.split), kb1 = (int)((long long)num_kb * (rank + 1) / p.split);
  const int stage_bytes = kNwWBytes + p.bt * kNwBK * 2;
  const int n_out = kGlu ? p.N / 2 : p.N;
  const int row0 = nb * (kGlu ? 64 : 128);                  // first weight rows of the two halves of the tile
  const int row1 = kGlu ? n_out + row0 : row0 + 64;
  const WaitGuard guard{&abort_word, status};

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(&acc_full, 1);
    abort_word = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 2) { tmem_alloc(&tmem_slot, p.tmem_cols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  grid_dependency_enter(p.beside);

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, guard, kTimeoutStageEmpty)) break;
        uint8_t* sw = smem + stage * stage_bytes;
        mbar_expect_tx(&full[stage], stage_bytes);
        if (!W_MN) {
          tma_load_2d(sw, &tmW, kb * kNwBK, row0, &full[stage]);
          tma_load_2d(sw + 8192, &tmW, kb * kNwBK, row1, &full[stage]);
        } else {
          tma_load_2d(sw, &tmW, row0, kb * kNwBK, &full[stage]);
          tma_load_2d(sw + 8192, &tmW, row1, kb * kNwBK, &full[stage]);
        }
        tma_load_2d(sw + kNwWBytes, &tmX, kb * kNwBK, m0, &full[stage]);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(128, p.bt, W_MN ? 1 : 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full[stage], phase, guard, kTimeoutTmaFull)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sw = smem_u32(smem + stage * stage_bytes), sx = sw + kNwWBytes;
#pragma unroll
        for (int k = 0; k < kNwBK / 16; ++k) {
          const uint64_t dw = W_MN ? smem_desc_mnmajor_sw128(sw + k * 2048, 8192) : smem_desc_kmajor_sw128(sw + k * 32);
          umma_ss(tmem_base, dw, smem_desc_kmajor_sw128(sx + k * 32), idesc, (kb != kb0 || k != 0) ? 1u : 0u);
        }
        umma_commit(&empty[stage]);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(&acc_full);
    }
    __syncwarp();
  } else {
    // every MMA has read its operands once acc_full completes, so the ring can hold the partial tile [bt][128]
    const int quad = warp & 3;
    if (mbar_wait(&acc_full, 0, guard, kTimeoutAccFull)) {
      __syncwarp();
      tc_fence_after();
      float* part = reinterpret_cast<float*>(smem) + quad * 32 + lane;
      const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16);
      for (int c = 0; c < p.bt; c += 16) {
        uint32_t r[16];
        tmem_ld16(t_row + c, r);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) part[(c + j) * 128] = __uint_as_float(r[j]);
      }
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  nw_cluster_sync();

  // this CTA's share of the rows, the parts added in rank order
  const int share = (p.bt + p.split - 1) / p.split;
  const int r_lo = rank * share, r_hi = min(min(r_lo + share, p.bt), p.M - m0);
  constexpr int kPerRow = kGlu ? 8 : 16;                    // 8 outputs per thread
  const uint32_t part0 = smem_u32(smem);
  for (int i = r_lo * kPerRow + (int)threadIdx.x; i < r_hi * kPerRow; i += kNwThreads) {
    const int m = i / kPerRow, n8 = (i % kPerRow) * 8;
    if (row0 + n8 >= n_out) continue;
    constexpr int kVecs = kGlu ? 4 : 2;
    float4 s[kVecs];
#pragma unroll
    for (int v = 0; v < kVecs; ++v) s[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < p.split; ++r) {
#pragma unroll
      for (int v = 0; v < kVecs; ++v) {
        const float4 x = nw_ld_cluster(part0 + (m * 128 + n8 + (v >> 1) * 64 + (v & 1) * 4) * 4, r);
        s[v].x += x.x; s[v].y += x.y; s[v].z += x.z; s[v].w += x.w;
      }
    }
    float o[8] = {s[0].x, s[0].y, s[0].z, s[0].w, s[1].x, s[1].y, s[1].z, s[1].w};
    if (kGlu) {
      const float u[8] = {s[kVecs - 2].x, s[kVecs - 2].y, s[kVecs - 2].z, s[kVecs - 2].w,
                          s[kVecs - 1].x, s[kVecs - 1].y, s[kVecs - 1].z, s[kVecs - 1].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float g = __bfloat162float(__float2bfloat16(o[j])), up = __bfloat162float(__float2bfloat16(u[j]));
        o[j] = g / (1.f + __expf(-g)) * up;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] *= p.alpha;
    }
    uint4 v;
    v.x = pack_bf16x2(o[0], o[1]); v.y = pack_bf16x2(o[2], o[3]);
    v.z = pack_bf16x2(o[4], o[5]); v.w = pack_bf16x2(o[6], o[7]);
    *reinterpret_cast<uint4*>(p.c + (long long)(m0 + m) * p.ldc + row0 + n8) = v;
  }
  __syncwarp();               // lanes leave the loop after different numbers of rows, and the barrier takes whole warps
  nw_cluster_sync();          // nobody leaves while its part may still be read
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
  grid_dependency_leave(p.beside);
}

// Tile height and split for a product, and its time in microseconds as modelled.  The figures were fitted to 10551 measured (shape, height,
// split) triples of 1650 products of 2 to 2048 rows with 64 to 24000 x 64 to 12288 weights in both layouts, 74 % of them with
// rows off the 128-byte lines:
//   * one 64-wide step of K takes a CTA that has an SM to itself 1.05 us over the stages of its ring (the latency of its loads), and CTAs
//     that share an SM 0.078 + 0.00102 bt each, so a grid should fill both slots of every SM; a ring for more than 160 rows leaves room for
//     one CTA only, but has five stages again;
//   * operands of all CTAs come through the L2 at 23 TB/s, the weights from memory at 5, at 5.7 in a single wave;
//   * a wave of CTAs costs 3.2 us to start and drain, and 0.0175 + 0.0035 split per activation row to write and add up; with the activation
//     0.012 more where nothing else on the SM covers it and 0.002 split (3200 measured triples, 8 %; 471 x 2 x 3888 x 2048 18.3 us in two
//     launches, 20.6 with 240 rows a tile);
//   * clusters of 4 and 8 do not fill every SM: narrow_first and narrow_slots below;
//   * less than eight steps are not split from 65 rows on, so that their sums are those of the tiled kernels whatever the number of rows (512
//     x 512 x 256 5.7 us on tiles, 5.0 here, 4.5 in two parts);
//   * rows that do not start on a 128-byte line take a second line for every box row, weights and activations 1.82 and 1.87 times their
//     bytes: in full through the L2, for three quarters of it in what CTAs that share an SM take, for a fifth in the latency.
// The model's standard deviation is 9 %; over the 1650 products the choice (tiled kernels included) is 1.0 % above the best on average, 4 % faster
// than the first one, fitted to 17 to 1411 rows of the presets' widths, and one product in a hundred more than 5 % slower than that; figures fitted to
// 288 to 2048 rows alone, with the tiled kernels at 128 x 256 throughout, were 2.7 % above the best and slower in one of twenty-two: 62 x
// 1704 x 416 4.3 us on tiles and 5.4 here, 1151 x 1184 x 8472 39.5 with 192 rows and 45.7 with 240, 310 x 3840 x 4096 17.4 and 19.4.
constexpr int kNwSms = 148;
constexpr int kNwMaxRows = 2048;   // the model holds near the range that it was fitted to (8000 x 128 x 2048: 27.4 against 15.3 us)
static constexpr bool narrow_two_per_sm(int bt) { return 3 * (kNwWBytes + bt * kNwBK * 2) <= 110 * 1024; }
static constexpr int narrow_stages(int bt) {
  const int stages = (narrow_two_per_sm(bt) ? 110 : 220) * 1024 / (kNwWBytes + bt * kNwBK * 2);
  return stages < kNwMaxStages ? stages : kNwMaxStages;
}
// the ring, or the partial tile that takes its place
static constexpr int narrow_smem(int bt) {
  const int ring = narrow_stages(bt) * (kNwWBytes + bt * kNwBK * 2), part = bt * 128 * 4;
  return (ring > part ? ring : part) + 1024;
}
static constexpr int narrow_least_smem() {
  int least = narrow_smem(16);
  for (int bt = 32; bt <= 256; bt += 16) least = narrow_smem(bt) < least ? narrow_smem(bt) : least;
  return least;
}
static_assert(narrow_least_smem() >= kTmemClusterLeast, "a smaller block would share an SM with clusters that count on its size");
// CTAs that run with an SM to themselves, and CTAs resident at once.  A cluster stays within one group of SMs, and the groups' sizes
// are no multiples of 4 and 8: 33 clusters of 4 and 15 of 8 with one CTA per SM (the occupancy query's answer and the
// grids at which the time jumps), 70 and 33 with two (the grids at which it jumps).
static int narrow_first(int split) { return split <= 2 ? kNwSms : split == 4 ? 132 : 120; }
static int narrow_slots(int bt, int split) {
  if (!narrow_two_per_sm(bt)) return narrow_first(split);
  return split <= 2 ? 2 * kNwSms : split == 4 ? 280 : 264;
}
static double narrow_plan(int M, int N, long long n_tiles, int K, bool gated, bool ragged_x, bool ragged_w, int* bt_out, int* split_out) {
  const int num_kb = (K + kNwBK - 1) / kNwBK, fewest = (M + 255) / 256;
  const double weights = (double)N * K * 2e-6;
  double best = 1e30, best_t = 1e30;
  for (int tm = fewest; tm < fewest + 9; ++tm) {
    const int bt = ((M + tm - 1) / tm + 15) / 16 * 16;
    if (tm > fewest && bt < 48) break;
    const int per_sm_most = narrow_two_per_sm(bt) ? 2 : 1;
    const double bytes = kNwWBytes + bt * kNwBK * 2;
    const double lines = (kNwWBytes * (ragged_w ? 1.82 : 1.0) + bt * kNwBK * 2 * (ragged_x ? 1.87 : 1.0)) / bytes - 1.0;
    for (int split = 1; split <= 8 && split <= num_kb; split *= 2) {
      if (split > 1 && M > 64 && num_kb < 8) break;
      const long long ctas = (long long)((M + bt - 1) / bt) * n_tiles * split;
      const double steps = (num_kb + split - 1) / split;
      const double row = 0.0175 + (gated && per_sm_most == 1 ? 0.012 : 0.0) + (split > 1 ? (gated ? 0.0055 : 0.0035) * split : 0.0);
      const int slots = narrow_slots(bt, split), first = narrow_first(split);
      auto wave = [&](long long n) {
        if (n == 0) return 0.0;
        const long long rounds = (n + first - 1) / first;
        const double per_sm = (double)(rounds < per_sm_most ? rounds : per_sm_most);
        const double shared = per_sm * (0.078 + 0.00102 * bt) * (1 + 0.76 * lines), alone = 1.05 / narrow_stages(bt) * (1 + 0.21 * lines);
        const double l2 = n * bytes * (1 + lines) / 23.2e6;
        const double step = shared > alone ? (shared > l2 ? shared : l2) : (alone > l2 ? alone : l2);
        return 3.2 + steps * step + per_sm * bt * row;
      };
      const double t = (double)(ctas / slots) * wave(slots) + wave(ctas % slots), memory = 4.0 + weights / (ctas <= slots ? 5.7 : 5.0);
      const double all = t > memory ? t : memory;
      if (all < best || (all == best && t < best_t)) { best = all; best_t = t; *bt_out = bt; *split_out = split; }
    }
  }
  return best;
}
static long long tiled_waves(int M, int N, int rows, int slots) {
  return ((long long)((M + rows - 1) / rows) * ((N + 255) / 256) + slots - 1) / slots;
}
static bool enough_for_pairs(int M, int N, int pair_min_tiles) {
  return pair_min_tiles > 0 && (long long)((M + 255) / 256) * ((N + 255) / 256) >= pair_min_tiles;
}
static bool on_pairs(int M, int N, int pair_min_tiles) {
  return enough_for_pairs(M, N, pair_min_tiles) && 2 * tiled_waves(M, N, 256, kNwSms / 2) < 3 * tiled_waves(M, N, 128, kNwSms);
}
// The time of the tiled kernel that serves the same product otherwise, fitted to the same products (12 %).  74 CTA pairs with 256 x 256 tiles take
// 0.3 us a 64-wide step, 2.1 a wave and 3.6 around them, a last wave of halves 0.7 of that.  Single CTAs with 128 x 256 tiles take 0.31 to 0.47 a
// step, the more of the SMs have a tile, 4.5 around them and 2.4 between waves, those with 128 x 128 tiles 0.18 to 0.26, 3.1 and 1.2.
// Weights come from memory at 5.2 and 5 TB/s.
// glu: 1, and of the separate activation kernel, 3 us and the way of what it reads; 2, on pairs that apply it themselves, a microsecond more a wave and no halves.
static double tiled_time(int M, int N, int K, int glu, int pair_min_tiles, bool ragged_x, bool ragged_w) {
  const double num_kb = (double)((K + 63) / 64), weights = (double)N * K * 2e-6, act = glu == 1 ? 3.0 + 2.5e-7 * M * N : 0.0;
  if (on_pairs(M, N, pair_min_tiles)) {
    const long long tiles = (long long)((M + 255) / 256) * ((N + 255) / 256), last = tiles % (kNwSms / 2);
    const double waves = (double)(tiles / (kNwSms / 2)) + (last == 0 ? 0.0 : 2 * last <= kNwSms / 2 && glu != 2 ? 0.7 : 1.0);
    const double step = 0.3 * (1 + (ragged_x ? 0.1 : 0.0) + (ragged_w ? 0.04 : 0.0));
    const double t = 3.6 + waves * (step * num_kb + (glu == 2 ? 3.1 : 2.1));
    return act + (t > weights / 5.2 ? t : weights / 5.2);
  }
  const bool wide = gemm_wide_tiles(M, N);
  const int bn = wide ? 256 : 128;
  const long long tiles = (long long)((M + 127) / 128) * ((N + bn - 1) / bn);
  const double waves = (double)((tiles + kNwSms - 1) / kNwSms), busy = tiles < kNwSms ? tiles / (double)kNwSms : 1.0;
  const double step = (wide ? 0.31 + 0.16 * busy : 0.18 + 0.083 * busy) * (1 + (ragged_x ? 0.16 : 0.0) + (ragged_w ? 0.34 : 0.0));
  const double t = (wide ? 4.5 : 3.1) + waves * step * num_kb + (waves - 1) * (wide ? 2.4 : 1.2), memory = 3.5 + weights / 5.0;
  return act + (t > memory ? t : memory);
}
double few_rows_time(int M, int N, int K) {
  int bt = 0, split = 0;
  const double narrow = narrow_plan(M, N, (N + 127) / 128, K, false, false, false, &bt, &split), tiled = tiled_time(M, N, K, 0, 0, false, false);
  return narrow < tiled ? narrow : tiled;
}

template <bool W_MN, bool kGlu>
static int launch_narrow(const void* x, const void* w, NarrowArgs p, long long ldx, long long ldw, cudaStream_t st) {
  CUtensorMap tmX, tmW;
  int rc;
  {
    uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)p.M};
    uint64_t str[2] = {2, (uint64_t)ldx * 2};
    uint32_t box[2] = {kNwBK, (uint32_t)p.bt};
    if ((rc = make_tmap(&tmX, x, 2, 2, dims, str, box, true))) return rc;
  }
  {
    uint64_t dims[2] = {(uint64_t)(W_MN ? p.N : p.K), (uint64_t)(W_MN ? p.K : p.N)};
    uint64_t str[2] = {2, (uint64_t)ldw * 2};
    uint32_t box[2] = {64, 64};
    if ((rc = make_tmap(&tmW, w, 2, 2, dims, str, box, true))) return rc;
  }
  // two CTAs per SM while a ring of three stages fits half of its shared memory, else one with a deeper ring
  p.stages = narrow_stages(p.bt);
  const int smem = narrow_smem(p.bt);
  p.tmem_cols = 32;
  while (p.tmem_cols < p.bt) p.tmem_cols *= 2;
  p.tiles_m = (p.M + p.bt - 1) / p.bt;
  const int n_tile = kGlu ? 64 : 128, n_out = kGlu ? p.N / 2 : p.N;
  const int tiles = p.tiles_m * ((n_out + n_tile - 1) / n_tile);
  auto kern = gemm_narrow_kernel<W_MN, kGlu>;
  static PerDevice raised;
  KSA_CHECK_CUDA(raise_smem_limit(raised, kern, 222 * 1024));
  int* status = status_word();
  KSA_REQUIRE(status != nullptr, "could not allocate the status word");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.split);
  cfg.blockDim = dim3(kNwThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.split;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent_launches() ? 2 : 1;
  KSA_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, tmW, tmX, p, status));
  return 0;
}

}  // namespace ksa

// C[M, N] (bf16) = alpha * X[M, K] * W^T; W is [N, K] row-major, or [K, N] with w_mn_major.  glu: W holds N/2 gate and N/2 up
// rows (row-major only) and C[M, N/2] = silu(X gate^T) * (X up^T).  bt: activation rows per tile (multiple of 16 up to
// 256), split: CTAs that share the reduction of a tile (1, 2, 4 or 8, at most one per 64 elements of K).
KSA_API int ksa_gemm_narrow_bf16(const void* x, const void* w, void* c, int M, int N, int K, long long ldx, long long ldw,
                                 long long ldc, int w_mn_major, int glu, int bt, int split, float alpha, void* stream) {
  KSA_ENTER(x);
  using namespace ksa;
  KSA_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_narrow: empty problem %d x %d x %d", M, N, K);
  KSA_REQUIRE(ldx % 8 == 0 && ldw % 8 == 0, "gemm_narrow: ldx/ldw must be multiples of 8 elements (got %lld, %lld)", ldx, ldw);
  KSA_REQUIRE(N % (glu ? 16 : 8) == 0 && ldc % 8 == 0, "gemm_narrow: N and ldc must keep 16-byte row alignment (N=%d ldc=%lld)", N, ldc);
  KSA_REQUIRE((reinterpret_cast<uintptr_t>(c) & 15) == 0, "gemm_narrow: C must be 16-byte aligned");
  KSA_REQUIRE(!(glu && w_mn_major), "gemm_narrow: the gated form takes row-major weights");
  KSA_REQUIRE(bt >= 16 && bt <= 256 && bt % 16 == 0, "gemm_narrow: tile of %d rows (16 to 256, in steps of 16)", bt);
  KSA_REQUIRE((split == 1 || split == 2 || split == 4 || split == 8) && split <= (K + kNwBK - 1) / kNwBK,
              "gemm_narrow: K = %d in %d parts", K, split);
  NarrowArgs p{};
  p.c = static_cast<bf16*>(c); p.ldc = ldc; p.M = M; p.N = N; p.K = K; p.bt = bt; p.split = split; p.alpha = alpha;
  p.beside = launch_beside();
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (glu) return launch_narrow<false, true>(x, w, p, ldx, ldw, st);
  return w_mn_major ? launch_narrow<true, false>(x, w, p, ldx, ldw, st) : launch_narrow<false, false>(x, w, p, ldx, ldw, st);
}

// Whether the CTA pairs of ksa_gemm2_bf16 serve an M x N product (from `pair_min_tiles` 256 x 256 tiles on, 0: never) or the single CTAs of
// ksa_gemm_bf16: a tile of 256 rows on a pair takes 0.75 to 0.95 of the time of two tiles of 128 rows, but rows that end
// in the first half of a tile and a last wave of a few tiles can cost pairs a whole wave more.  Pairs unless they take half as many waves
// again: 333 x 19456 x 2560 3 waves against 2, 44.0 us on pairs and 41.0 on single CTAs; 333 x 12288 x 2048 2 against 1, 28.7 and 21.9;
// 1152 x 4096 x 2048 2 against 1, 26.0 and 18.0 (fp32 from transposed operands 29.1 and 22.5).  At 4 against 3 both are within 6 %
// (513 x 19456 x 2560 59.3 and 57.5, fp32 at 1152 x 12288 x 2048 53.3 and 61.1), at 6 against 5 pairs are 5 to 15 % faster.
// Waves count 128 x 256 tiles; the 128 x 128 tiles that ksa_gemm_bf16 takes for a ragged N of few tiles take about as long together
// (100 x 19320 x 2560 34.5 us on pairs and 32.5 there).
KSA_API int ksa_gemm_on_pairs(int M, int N, int pair_min_tiles) {
  return ksa::on_pairs(M, N, pair_min_tiles);
}

// Whether this kernel is expected to beat the tiled ones (of which CTA pairs are taken from `pair_min_tiles` 256 x 256 tiles on, 0:
// never): bt * 16 + split for ksa_gemm_narrow_bf16, or 0, as for weights of less than 64 KB, where nothing but the launch takes time.  By 5 % at
// least, but up to 64 rows with weights wide enough for pairs, whose tiled kernels take the longer the fewer of a tile's rows are there, which the
// model does not know, also where it is modelled slower (112 such products: always faster here; 32 x 15856 x 9728 49.5 us and 56.3 on
// pairs, 5 x 18408 x 6144 35.3 and 55.6, 4 x 19456 x 1024 10.3 and 15.2 on single CTAs, with the activation 18 x 2 x 9472 x 2560 21.3 and 29.0).
// glu: 1, the gated form, one launch against the tiled kernels' two (then small weights of more than one step are worth it as well: 96 x 2 x 88 x 168 4.8 us and 5.5);
// 2, the plain form and a separate activation, 2 us, against CTA pairs, which apply it themselves (77 x 2 x 4864 x 2048 15.2 us and 16.8, 429 x 2 x
// 4864 x 4096 39.4 and 45.7; over 118 products the choice is 2.5 % above the better of both on average, always pairs 9 %, never pairs 16 %).
// ragged: bit 0, the activations' rows do not all start on a 128-byte line (their pitch is no multiple of 64 elements); bit 1, those of
// the weights as they lie in memory.
KSA_API int ksa_gemm_narrow_plan(int M, int N, int K, int glu, int pair_min_tiles, int ragged) {
  using namespace ksa;
  if (M <= 0 || M > kNwMaxRows || N <= 0 || K <= 0 || (glu == 1 ? K <= kNwBK : (long long)N * K < 32768)) return 0;
  int bt = 0, split = 0;
  const bool rx = (ragged & 1) != 0, rw = (ragged & 2) != 0;
  const double t = narrow_plan(M, N, glu == 1 ? (N / 2 + 63) / 64 : (N + 127) / 128, K, glu == 1, rx, rw, &bt, &split) + (glu == 2 ? 2.0 : 0.0);
  return t < (M <= 64 && enough_for_pairs(M, N, pair_min_tiles) ? 1.4 : 0.95) * tiled_time(M, N, K, glu, pair_min_tiles, rx, rw) ? bt * 16 + split : 0;
}
