// bf16 GEMM for 17 to some hundred rows: C[M, N] = X[M, K] W[N, K]^T, optionally with SwiGLU, M <= 384.
//
// A tile holds ALL rows and as many columns as give every SM one tile, so the weights cross the L2 once, whole, and no last wave is
// left over; the few activation rows are read again by every CTA.  Up to three blocks of 128 rows take products with the same weights of a
// stage, each into columns of tensor memory of its own.  (Tiles of 128 x 256 read the weights once per 128 rows, at the L2's 12 TB/s, and
// 228 of them on 148 SMs take two waves; tiles of 128 weight rows, which csrc/gemm_narrow.cu takes, are too few or too many for the SMs.)
// Where N leaves the SMs too little, K is split over a cluster (without SwiGLU): the tiles get wider by the same factor, so that the
// activations are read as often as before, and the parts are sent straight from tensor memory to the CTA that adds them up, in rank order.
// Bound by the weights' way from memory up to 128 rows (5.6 TB/s) and by what a CTA can take in above (some 150 GB/s with its ring full).
// us, before (split-K or 128-row tiles, from 190 rows on with the activation in a launch of its own) and here:
//   SwiGLU, 2 x 9728 x 2560 weights: 48 rows 21.2 -> 20.4, 128 29.7 -> 21.5, 256 40.3 -> 27.9, 317 51.6 -> 38.4; 2 x 6144 x 2048: 48 rows 15.3 ->
//   12.3, 128 19.8 -> 12.2, 256 20.5 -> 16.8; the output head 151936 x 2560: 17 rows 134 -> 119, 128 rows 195 -> 154;
//   in four parts, 2560 x 9728: 48 rows 17.7 -> 13.3, 128 19.6 -> 14.5, 256 26.7 -> 19.5; 2560 x 4096: 48 rows 10.7 -> 8.7, 256 18.2 -> 12.8;
//   2048 x 6144: 48 rows 12.7 -> 9.6; in two, 6144 x 2560: 48 rows 13.2 -> 10.0, 256 17.1 -> 14.2.
#include "common.cuh"
#include "host.h"

namespace ksa {

constexpr int kTlBK = 64;
constexpr int kTlThreads = 320;      // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue, two for each quarter of the lanes
constexpr int kTlMaxStages = 8;
constexpr int kTlRing = 222 * 1024;

struct TallArgs {
  bf16* c;
  long long ldc;
  int M, N, K;               // N: columns of C
  int bn;                    // weight rows of a tile: as many columns of C, or kGlu bn / 2 gate and bn / 2 up rows
  int last_rows;             // rows of the last row block that are loaded (the rest of its operand is whatever the ring held)
  int stages;
  int split;                 // CTAs of a cluster that share the reduction of a tile
  int beside;                // launch_beside()
};
enum TallForm { kTlPlain, kTlGlu, kTlSplit };
// accumulator columns of a row block, and the most that row blocks leave room for in tensor memory
__host__ __device__ constexpr int tall_columns(int bn) { return (bn + 31) / 32 * 32; }
constexpr int tall_most_columns(int mt) { return mt <= 2 ? 256 : 160; }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}

__device__ __forceinline__ uint32_t tl_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void tl_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t tl_map(uint32_t local_addr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  return a;
}
__device__ __forceinline__ void tl_st_cluster(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

template <int MT, TallForm F>            // row blocks of 128
__global__ void __launch_bounds__(kTlThreads, 1)
gemm_tall_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmXl, const __grid_constant__ CUtensorMap tmW,
                 const TallArgs p, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[kTlMaxStages], empty[kTlMaxStages], acc_full, acc_empty;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const WaitGuard guard{&abort_word, status};
  constexpr bool kGlu = F == kTlGlu, kSplit = F == kTlSplit;
  const int per_tile = kGlu ? p.bn / 2 : p.bn;               // columns of C
  const int tiles = (p.N + per_tile - 1) / per_tile, num_kb = (p.K + kTlBK - 1) / kTlBK;
  // the weights of a stage follow its activations; the last row block's operand reaches into them where its rows are not loaded
  const int x_bytes = (MT - 1) * 16384 + p.last_rows * 128, half_bytes = per_tile * 128, stage_bytes = x_bytes + p.bn * 128;
  const int cols = tall_columns(p.bn);
  const int rank = kSplit ? (int)tl_cluster_rank() : 0;
  const int first = kSplit ? (int)blockIdx.x / p.split : (int)blockIdx.x, step = kSplit ? tiles : (int)gridDim.x;
  const int kb0 = kSplit ? num_kb * rank / p.split : 0, kb1 = kSplit ? num_kb * (rank + 1) / p.split : num_kb;
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, 8);
    abort_word = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmXl);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 2) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  grid_dependency_enter(p.beside);

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int tile = first; tile < tiles && ok; tile += step) {
        const int n0 = tile * per_tile;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty[stage], phase, guard, kTimeoutStageEmpty)) { ok = false; break; }
          uint8_t* sx = smem + stage * stage_bytes;
          mbar_expect_tx(&full[stage], stage_bytes);
          tma_load_2d(sx + x_bytes, &tmW, kb * kTlBK, n0, &full[stage]);
          if (kGlu) tma_load_2d(sx + x_bytes + half_bytes, &tmW, kb * kTlBK, p.N + n0, &full[stage]);
#pragma unroll
          for (int m = 0; m < MT - 1; ++m) tma_load_2d(sx + m * 16384, &tmX, kb * kTlBK, m * 128, &full[stage]);
          tma_load_2d(sx + (MT - 1) * 16384, &tmXl, kb * kTlBK, (MT - 1) * 128, &full[stage]);
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(128, p.bn, 0, 0);
      int stage = 0, local = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < tiles && ok; tile += step, ++local) {
        if (local > 0 && !mbar_wait(&acc_empty, (local - 1) & 1, guard, kTimeoutAccEmpty)) break;
        tc_fence_after();
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full[stage], phase, guard, kTimeoutTmaFull)) { ok = false; break; }
          tc_fence_after();
          const uint64_t xd = smem_desc_kmajor_sw128(smem_u32(smem + stage * stage_bytes)), wd = xd + (x_bytes >> 4);
#pragma unroll
          for (int k = 0; k < kTlBK / 16; ++k)
#pragma unroll
            for (int m = 0; m < MT; ++m)
              umma_ss(tmem_base + m * cols, xd + m * 1024 + k * 2, wd + k * 2, idesc, kb != kb0 || k != 0 ? 1u : 0u);
          umma_commit(&empty[stage]);
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit(&acc_full);
      }
    }
    __syncwarp();
  } else if (!kSplit) {
    const int quad = warp & 3, half = (warp - 2) >> 2;
    int local = 0;
    for (int tile = first; tile < tiles; tile += step, ++local) {
      if (!mbar_wait(&acc_full, local & 1, guard, kTimeoutAccFull)) break;
      tc_fence_after();
      const int n0 = tile * per_tile, n = min(per_tile, p.N - n0);
#pragma unroll 1
      for (int m = 0; m < MT; ++m) {
        const int row = m * 128 + quad * 32 + lane;
        const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + m * cols;
        bf16* dst = p.c + (long long)row * p.ldc + n0;
#pragma unroll 2
        for (int f = half * 8; f < n; f += 16) {
          uint32_t g[8], o[4];
          tmem_ld8(t_row + f, g);
          if (kGlu) {
            uint32_t u[8];
            tmem_ld8(t_row + per_tile + f, u);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              // gate and up are rounded to bf16 first, as the separate projection + SwiGLU kernels do
              float v[2];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const float gt = __bfloat162float(__float2bfloat16(__uint_as_float(g[2 * i + e])));
                v[e] = gt / (1.f + __expf(-gt)) * __bfloat162float(__float2bfloat16(__uint_as_float(u[2 * i + e])));
              }
              o[i] = pack_bf16x2(v[0], v[1]);
            }
          } else {
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = pack_bf16x2(__uint_as_float(g[2 * i]), __uint_as_float(g[2 * i + 1]));
          }
          if (row < p.M) *reinterpret_cast<uint4*>(dst + f) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty);
    }
  }
  if (kSplit) {
    // Every CTA sends the columns of its partial tile to the CTA of the cluster that adds them up, into what was the ring: [part][8 columns]
    // [4 of them][row][4].  The first barrier says that all products have read their operands, the second that all parts are there.
    const int slots = (p.bn / 8 + p.split - 1) / p.split, rows = (MT - 1) * 128 + p.last_rows, n0 = first * p.bn;
    bool ok = true;
    if (warp >= 2) ok = mbar_wait(&acc_full, 0, guard, kTimeoutAccFull);
    __syncwarp();
    tl_cluster_sync();
    if (warp >= 2 && ok) {
      tc_fence_after();
      const int quad = warp & 3, half = (warp - 2) >> 2, n = min(p.bn, p.N - n0);
#pragma unroll 1
      for (int m = 0; m < MT; ++m) {
        const int row = m * 128 + quad * 32 + lane;
        if (m * 128 + quad * 32 >= rows) break;
        const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + m * cols;
#pragma unroll 2
        for (int c = half; c < n / 8; c += 2) {
          uint32_t g[8];
          tmem_ld8(t_row + c * 8, g);
          const uint32_t at = smem_u32(smem) + (uint32_t)((((rank * slots + c % slots) * 2) * rows + row) * 16);
          const uint32_t to = tl_map(at, c / slots);
          tmem_wait_ld();
          if (row < rows) {
            tl_st_cluster(to, g[0], g[1], g[2], g[3]);
            tl_st_cluster(to + rows * 16, g[4], g[5], g[6], g[7]);
          }
        }
      }
    }
    __syncwarp();
    tl_cluster_sync();
    const float4* part = reinterpret_cast<const float4*>(smem);
    const int mine = min(slots, (min(p.bn, p.N - n0)) / 8 - rank * slots);
    for (int i = (int)threadIdx.x; i < mine * rows; i += kTlThreads) {
      const int c = i / rows, row = i - c * rows;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
      for (int r = 0; r < p.split; ++r) {
        const float4 u = part[((r * slots + c) * 2) * rows + row], v = part[((r * slots + c) * 2 + 1) * rows + row];
        a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
        b.x += v.x; b.y += v.y; b.z += v.z; b.w += v.w;
      }
      if (row < p.M)
        *reinterpret_cast<uint4*>(p.c + (long long)row * p.ldc + n0 + (rank * slots + c) * 8) =
            make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  grid_dependency_leave(p.beside);
}

template <int MT, TallForm F>
static int launch_tall(const void* x, const void* w, TallArgs p, long long ldx, long long ldw, cudaStream_t st) {
  constexpr bool kGlu = F == kTlGlu;
  CUtensorMap tmX, tmXl, tmW;
  int rc;
  p.last_rows = (p.M - (MT - 1) * 128 + 7) / 8 * 8;
  for (int rows : {p.last_rows, 128}) {
    uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)p.M};
    uint64_t str[2] = {2, (uint64_t)ldx * 2};
    uint32_t box[2] = {kTlBK, (uint32_t)rows};
    if ((rc = make_tmap(&tmX, x, 2, 2, dims, str, box, true))) return rc;
    if (rows == p.last_rows) tmXl = tmX;
    if (MT == 1 || p.last_rows == 128) break;           // one map serves
  }
  {
    uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)(kGlu ? 2 : 1) * p.N};
    uint64_t str[2] = {2, (uint64_t)ldw * 2};
    uint32_t box[2] = {kTlBK, (uint32_t)(kGlu ? p.bn / 2 : p.bn)};
    if ((rc = make_tmap(&tmW, w, 2, 2, dims, str, box, true))) return rc;
  }
  const int stage_bytes = (MT - 1) * 16384 + p.last_rows * 128 + p.bn * 128;
  // behind the last stage there is room for the rows that its last row block does not load
  const int slack = 16384 - p.last_rows * 128 - p.bn * 128 > 0 ? 16384 - p.last_rows * 128 - p.bn * 128 : 0;
  p.stages = (kTlRing - slack) / stage_bytes;
  if (p.stages > kTlMaxStages) p.stages = kTlMaxStages;
  auto kern = gemm_tall_kernel<MT, F>;
  static PerDevice raised;
  KSA_CHECK_CUDA(raise_smem_limit(raised, kern, kTlRing + 1024));
  const int per_tile = kGlu ? p.bn / 2 : p.bn;
  const int sms = sm_count(), tiles = (p.N + per_tile - 1) / per_tile;
  KSA_REQUIRE(sms > 0, "no device");
  int* status = status_word();
  KSA_REQUIRE(status != nullptr, "could not allocate the status word");
  const int ring = p.stages * stage_bytes + slack, parts = p.split * ((p.bn / 8 + p.split - 1) / p.split) * ((MT - 1) * 128 + p.last_rows) * 32;
  if (F != kTlSplit) {
    KSA_CHECK_CUDA(launch_kernel(kern, dim3(tiles < sms ? tiles : sms), dim3(kTlThreads), (size_t)(ring + 1024), st, tmX, tmXl, tmW, p, status));
    return 0;
  }
  KSA_REQUIRE(parts <= kTlRing, "gemm_tall: %d parts of %d rows of %d columns", p.split, p.M, p.bn);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.split);
  cfg.blockDim = dim3(kTlThreads);
  // all of the tensor memory: no room for a block of another cluster that holds some (host.h)
  const int held = (ring > parts ? ring : parts) + 1024;
  cfg.dynamicSmemBytes = (size_t)(held > kTmemClusterAlone ? held : kTmemClusterAlone);
  static_assert(kTlRing + 1024 >= kTmemClusterAlone, "the limit raised above covers it");
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
  KSA_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, tmX, tmXl, tmW, p, status));
  return 0;
}

}  // namespace ksa

// C[M, N] (bf16) = X W^T, X [M, K], W [N, K] row-major; glu: W holds N gate rows, then N up rows, and C = silu(gate) * up with both products
// rounded to bf16 first.  M <= 384; columns: weight rows of a tile, a multiple of 16 up to 256 (M <= 256) or 160; split: CTAs of a cluster that share
// the reduction of a tile (1 with glu).
KSA_API int ksa_gemm_tall_bf16(const void* x, const void* w, void* c, int M, int N, int K, long long ldx, long long ldw, long long ldc, int glu,
                               int columns, int split, void* stream) {
  KSA_ENTER(x);
  using namespace ksa;
  KSA_REQUIRE(M > 0 && N > 0 && K > 0 && M <= 384, "gemm_tall: %d rows, %d columns of %d", M, N, K);
  KSA_REQUIRE(ldx % 8 == 0 && ldw % 8 == 0, "gemm_tall: ldx/ldw must be multiples of 8 elements (got %lld, %lld)", ldx, ldw);
  KSA_REQUIRE(N % 8 == 0 && ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0, "gemm_tall: rows of C must keep 16-byte alignment");
  const int mt = (M + 127) / 128;
  KSA_REQUIRE(columns >= 16 && columns % 16 == 0 && columns <= tall_most_columns(mt), "gemm_tall: tiles of %d columns for %d rows", columns, M);
  KSA_REQUIRE(split >= 1 && split <= 8 && split <= (K + kTlBK - 1) / kTlBK && (split == 1 || !glu), "gemm_tall: K = %d in %d parts", K, split);
  TallArgs p{static_cast<bf16*>(c), ldc, M, N, K, columns, 0, 0, split, launch_beside()};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define KSA_TALL(MT)                                                            \
  return glu          ? launch_tall<MT, kTlGlu>(x, w, p, ldx, ldw, st)          \
         : split == 1 ? launch_tall<MT, kTlPlain>(x, w, p, ldx, ldw, st)        \
                      : launch_tall<MT, kTlSplit>(x, w, p, ldx, ldw, st)
  if (mt <= 1) KSA_TALL(1);
  if (mt == 2) KSA_TALL(2);
  KSA_TALL(3);
#undef KSA_TALL
}

// Without SwiGLU the reduction may be split as well: tiles as wide as the clusters that fit at once allow (33 of four CTAs, 15 of eight), the
// parts added in shared memory.  Modelled time in us, fitted to 1100 measured (shape, tile, split) triples of 17 to 384 rows against 128 x
// 2560 .. 12288 x 2048 and 5120 x 13824 weights (6 % standard deviation; the choice 0.6 % above the best of the splits on average).  A 64-wide step
// of K takes the longest of: a trip to memory over the stages in flight, and 0.06 for each further block of rows; all CTAs' bytes through the L2 at
// 20.6 TB/s; the weights from memory at 6; this CTA's bytes at 151 GB/s; the products, which read 128 + columns rows of operands at 128 bytes a
// cycle.
namespace ksa {
constexpr int kTlSms = 148;
static double tall_time(int rows, int blocks, int steps, int columns, int split, int ctas) {
  const double bytes = (rows + columns) * 128.0, terms[5] = {0.19 + 0.06 * (blocks - 1), ctas * bytes / 20.6e6, ctas * columns * 128.0 / 6e6,
                                                             bytes / 151e3, blocks * (32 + columns / 4) * 4 * 6.76e-4};
  double step = 0;
  for (double t : terms) step = t > step ? t : step;
  return 2.1 + steps * step + (split > 1 ? 1.7 + 2.2e-4 * rows * columns : 2.6e-4 * rows * columns);
}
static int tall_split_plan(int M, int N, int K, double* time) {
  const int blocks = (M + 127) / 128, rows = (M + 7) / 8 * 8, num_kb = (K + kTlBK - 1) / kTlBK;
  double best = 1e30;
  int plan = 0;
  for (int split = 1; split <= 8 && split <= num_kb; split *= 2) {
    const int most = split == 4 ? 33 : split == 8 ? 15 : kTlSms / split;
    const int columns = ((N + most - 1) / most + 15) / 16 * 16, tiles = (N + columns - 1) / columns;
    if (columns > tall_most_columns(blocks) || (split > 1 && split * ((columns / 8 + split - 1) / split) * rows * 32 > kTlRing)) continue;
    const double t = tall_time(rows, blocks, (num_kb + split - 1) / split, columns, split, tiles * split);
    if (t < best) { best = t; plan = columns * 16 + split; }
  }
  *time = best;
  return plan;
}
}  // namespace ksa

// Weight rows of a tile * 16 + split for ksa_gemm_tall_bf16 where that kernel is taken, else 0 (then the split-K kernel or tiles of 128 rows
// are).  Where the lines lie, in us of the others and here:
//   * plain, up to 128 rows: always (2560 x 9728 48 rows 17.7 -> 13.3, 128 rows 19.6 -> 14.5; 2560 x 4096 48 rows 10.7 -> 8.7; 6144 x 2560 48 rows
//     13.2 -> 10.0; 128 x 2560 7.5 -> 6.8; 10240 x 2560 128 rows 19.8 -> 13.1) to 96 columns a CTA without a split, and the output head, several
//     tiles to an SM from 160 columns on, as nothing covers the time between them (151936 x 2560 128 rows 195 -> 154; with 128 columns, 2 x 18944 x
//     3584 48 rows 47.3 -> 48.3).  What lies between stays where it was, gate and up rows without SwiGLU for the most part, though it would
//     gain here too: 22 x 15080 x 2560 15.9 -> 14.3, 40 x 19456 x 3840 27.5 -> 25.8, 84 x 19456 x 1280 14.7 -> 11.0, 81 x 19456 x 9728 76 -> 62.
//   * plain, up to 256 rows: to 80 columns (2560 x 9728 256 rows 26.7 -> 19.5; 10240 x 2560 19.8 -> 18.2; 12288 x 2048 17.9 -> 18.0)
//   * plain, up to 384 rows: to 112 columns a CTA with K in four parts, where the model above is at most 8 % over those of the other kernels, from
//     300 columns and a longer K on up to 20 %, as it is itself high there, the more the longer K (9 % over 233 such products of up to 6000 x
//     12288): 333 x 2560 x 9728 28.8 -> 24.5, 328 x 2048 x 6144 16.9 -> 16.0, 290 x 640 x 4096 10.0 -> 9.2; but 357 x 152 x 512 4.5 -> 5.8,
//     334 x 152 x 12288 11.2 -> 13.5, 346 x 1024 x 1024 6.2 -> 6.8, 333 x 2560 x 4096 14.2 -> 15.7.  3.6 % above the best on average, one in forty
//     more than 5 % slower than without this kernel.  Weights of fewer than eight tiles of 16 are nobody's case.
//   * SwiGLU: the smallest tile that gives no SM more tiles than another, from 48 columns on (2 x 3072 x 1024, 48: 48 rows 8.5 -> 7.2, 256 rows 18.9 ->
//     9.3; 2 x 1536 x 2048, 32: 130 rows 9.7 -> 11.5); with fewer than 64 rows and a long K from 80 on (2 x 4608 x 4096, 64: 48 rows 17.5 -> 17.8),
//     as with more than 128 rows and K above 2560 (2 x 3072 x 4096, 48: 132 rows 16.1 -> 19.7, 256 rows x 6144 27.9 -> 29.3; 2 x 3072 x 2048 200 rows
//     13.4 -> 11.9; 2 x 5920 x 4096, 80: 132 rows 25.3 -> 24.1); up to 224, with 256 there are too few stages (2 x 18944 x 3584 17 rows 46.1 -> 48.0, 2 x 14336 x 4096, 208: 48 rows 44.6 -> 43.5); above 128 rows up
//     to 160 (2 x 14336 x 4096, 208: 130 rows 54.1 -> 61.4), up to 384 rows from 144 (2 x 9728 x 2560 384 rows 48.4 -> 39.5; 2 x 8960 x 1536, 128: 264
//     rows 21.6 -> 23.0); four blocks of rows never (2 x 9728 x 2560 479 rows 55.7 -> 66.0).
// ragged: rows off the 128-byte lines, which the split-K kernel's model knows about.
KSA_API int ksa_gemm_tall_plan(int M, int N, int K, int glu, int ragged) {
  using namespace ksa;
  if (M <= 16 || M > 384 || N < 128 || K <= 0 || ragged || N % 8 != 0) return 0;
  const int blocks = (M + 127) / 128, most = blocks == 1 ? 224 : 160;
  const long long rows = (glu ? 2LL : 1LL) * N, waves = (rows + (long long)kTlSms * most - 1) / ((long long)kTlSms * most);
  const int columns = (int)(((rows + kTlSms * waves - 1) / (kTlSms * waves) + 15) / 16 * 16);
  if (!glu && waves == 1) {
    if (blocks == 1 ? columns > 96 : blocks == 2 ? columns > 80 : N > 33 * 112) return 0;
    double time = 0;
    const int plan = tall_split_plan(M, N, K, &time);
    const double over = 1.08 + (N < 300 || K <= 3456 ? 0.0 : 4.3e-5 * ((K < 6144 ? K : 6144) - 3456));
    return blocks <= 2 || time < over * few_rows_time(M, N, K) ? plan : 0;
  }
  if (waves > 1 && blocks > 1) return 0;
  const int least = blocks == 3 ? 144 : waves > 1 ? 160 : (M < 64 && K > 3072) || (blocks == 2 && K > 2560) ? 80 : 48;
  return columns >= least ? columns * 16 + 1 : 0;
}
