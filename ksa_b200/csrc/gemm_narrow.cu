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
// The weights alone take 7.6, 7.6, 4.8 and 15.2 us at the copy bandwidth.  Row-major weights of up to 256 rows go to csrc/gemm_tall.cu now (13.2
// us for the first of these), which reads the activations again for every tile; from there on this one has the better balance.
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

// Tile height and split for a product, and its time in microseconds as modelled.  The figures were fitted to 4176 measured (shape, height,
// split) triples of 288 to 2048 rows against 512 x 4096 .. 9728 x 2560 weights in both layouts, the last two items to 900 shapes of
// 17 to 2048 rows and 64 to 19456 x 64 to 12288 weights:
//   * one 64-wide step of K takes a CTA that has an SM to itself 0.241 + 0.00054 bt us (the latency of its loads) and two that share
//     one 2 x (0.093 + 0.00094 bt), so a grid should fill both slots of every SM; a ring for more than 160 rows leaves
//     room for one CTA only;
//   * the weights of all CTAs come through the L2 at 16 TB/s, with the activations at 21.9;
//   * a launch costs 1.4 us, a wave of CTAs 3.6 us to start and drain, and 0.013 + 0.0043 split per activation row to write
//     and add up;
//   * clusters of 4 and 8 do not fill every SM: narrow_first and narrow_slots below;
//   * rows that do not start on a 128-byte line take a second line for every box row: weights and activations then come
//     through the L2 at 21 TB/s as 1.86 and 1.55 times their bytes.
// The model's standard deviation is 8 %; over those 270 products the choice (tiled kernels included) is 1.2 % above the best on average,
// against 3.3 % with the figures of before the issuing threads were elected, and 2 % faster: 333 x 2560 x 4096 19.8 -> 15.6 us, 576 x 2560 x 9728
// 37.9 -> 31.2, 700 x 2048 x 12288 40.7 -> 34.9.  Without the last two items 21 of the 900 shapes were up to 30 % slower (779 x 3552 x 6008:
// 62.5 us on tiles of 160 rows in two parts, 42.9 on CTA pairs; 193 x 4256 x 3352 30.2 on 208 rows in four parts, 21.0).
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
static double narrow_plan(int M, long long n_tiles, int K, bool ragged_x, bool ragged_w, int* bt_out, int* split_out) {
  const int num_kb = (K + kNwBK - 1) / kNwBK, fewest = (M + 255) / 256;
  double best = 1e30;
  for (int tm = fewest; tm < fewest + 9; ++tm) {
    const int bt = ((M + tm - 1) / tm + 15) / 16 * 16;
    if (tm > fewest && bt < 48) break;
    const int per_sm_most = narrow_two_per_sm(bt) ? 2 : 1;
    for (int split = 1; split <= 8 && split <= num_kb; split *= 2) {
      const long long ctas = (long long)((M + bt - 1) / bt) * n_tiles * split;
      const double steps = (num_kb + split - 1) / split;
      const int slots = narrow_slots(bt, split), first = narrow_first(split);
      auto wave = [&](long long n) {
        if (n == 0) return 0.0;
        const long long rounds = (n + first - 1) / first;
        const double per_sm = (double)(rounds < per_sm_most ? rounds : per_sm_most);
        double step = per_sm * (0.093 + 0.00094 * bt);
        if (step < 0.241 + 0.00054 * bt) step = 0.241 + 0.00054 * bt;
        if (step < n * 0.00102) step = n * 0.00102;
        const double all = n * (kNwWBytes + bt * kNwBK * 2.0) / 21.9e6;
        if (step < all) step = all;
        if (ragged_x || ragged_w) {
          const double bytes = kNwWBytes * (ragged_w ? 1.86 : 1.0) + bt * kNwBK * 2 * (ragged_x ? 1.55 : 1.0);
          if (step < n * bytes / 21e6) step = n * bytes / 21e6;
        }
        return 3.6 + steps * step + per_sm * bt * (0.013 + (split > 1 ? 0.0043 * split : 0.0)) + (split == 8 ? 0.26 : 0.0);
      };
      const double t = 1.36 + (double)(ctas / slots) * wave(slots) + wave(ctas % slots);
      if (t < best) { best = t; *bt_out = bt; *split_out = split; }
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
// The time of the tiled kernel that serves the same product otherwise: 0.327 us a 64-wide step and wave of 74 CTA pairs with 256 x 256
// tiles, 6.7 us around them.  Single CTAs with 128 x 256 tiles take 0.352 a step and wave and 5.6 around them where there are too few tiles for
// pairs (16.4 us measured for 900 x 2048 x 2048, 60.5 for 576 x 2560 x 9728).  Where they are taken for their fewer waves, most SMs have a
// tile: 5.7 us and, a step and wave, 0.364 and 0.057 for every megabyte of weights that the step's tiles read: 333 x 4096 x 2048 16.4 us
// (0.5 MB), 333 x 12288 x 2048 21.2 (1.6 MB), 128 x 19456 x 2560 26.2 (2.5 MB).
// glu: and of the separate activation kernel, 2 us and more, 2.8 to 3.7 behind the products of the last kind.
static double tiled_time(int M, int N, int K, bool glu, int pair_min_tiles) {
  const long long num_kb = (K + 63) / 64;
  const double act = glu ? 2.0 : 0.0;
  if (on_pairs(M, N, pair_min_tiles)) return act + 6.7 + 0.327 * num_kb * tiled_waves(M, N, 256, kNwSms / 2);
  const double steps = (double)(num_kb * tiled_waves(M, N, 128, kNwSms));
  if (!enough_for_pairs(M, N, pair_min_tiles)) return act + 5.6 + 0.352 * steps;
  const long long tm = (M + 127) / 128, tn = (N + 255) / 256, abreast = (kNwSms + tm - 1) / tm;      // tiles of a row in one wave
  return (glu ? 3.5 : 0.0) + 5.7 + (0.364 + 0.057 * (tn < abreast ? tn : abreast) * 256 * kNwBK * 2 / 1e6) * steps;
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
// never), by more than 4 %, with K in one part by more than 8 (900 x 2048 x 2048 16.4 us on tiles and 17.5 here): bt * 16 + split for
// ksa_gemm_narrow_bf16, or 0, as for weights of less than 64 KB, where nothing but the launch takes time.  glu: the separate activation
// kernel counts on the other side; 2: it counts on this side, as CTA pairs apply it themselves.  ragged: bit 0, the activations' rows do not all start on a 128-byte line (their
// pitch is no multiple of 64 elements); bit 1, those of the weights as they lie in memory.
KSA_API int ksa_gemm_narrow_plan(int M, int N, int K, int glu, int pair_min_tiles, int ragged) {
  using namespace ksa;
  if (M <= 0 || M > kNwMaxRows || N <= 0 || K <= 0 || (long long)N * K < 32768) return 0;
  int bt = 0, split = 0;
  const bool gated = glu == 1;
  double t = narrow_plan(M, gated ? (N / 2 + 63) / 64 : (N + 127) / 128, K, (ragged & 1) != 0, (ragged & 2) != 0, &bt, &split);
  if (glu == 2) t += 3.0;
  return t < (split == 1 ? 0.92 : 0.96) * tiled_time(M, N, K, gated, pair_min_tiles) ? bt * 16 + split : 0;
}
