// bf16 GEMM for 17 to some hundred rows and wide weights: C[M, N] = X[M, K] W[N, K]^T, optionally with SwiGLU, M <= 384.
//
// A tile holds ALL rows and as many columns as give every SM one tile, so the weights cross the L2 once, whole, and no last wave is
// left over; the few activation rows are read again by every CTA.  Up to three blocks of 128 rows take products with the same
// weights of a stage, each into columns of tensor memory of its own.  (Tiles of 128 x 256 read the weights once per 128 rows, at the L2's 12
// TB/s, and 228 of them on 148 SMs take two waves; a K split over clusters reads them once per 256 rows and adds up in shared memory.)
// Bound by the weights' way from memory up to 128 rows (5.6 TB/s), by the L2 above.  us, before (split-K or 128-row tiles, from 190 rows on
// with the activation in a launch of its own) and here: SwiGLU with 2 x 9728 x 2560 weights: 48 rows 21.2 -> 20.4, 128 29.7 -> 21.5, 160 31.7 ->
// 26.2, 256 40.3 -> 27.9, 317 51.6 -> 38.4; with 2 x 6144 x 2048: 48 rows 15.3 -> 12.3, 128 19.8 -> 12.2, 256 20.5 -> 16.8; the output head
// 151936 x 2560: 17 rows 134 -> 119, 48 rows 139 -> 122, 128 rows 195 -> 154.
#include "common.cuh"
#include "host.h"

namespace ksa {

constexpr int kTlBK = 64;
constexpr int kTlThreads = 192;      // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue
constexpr int kTlMaxStages = 8;
constexpr int kTlRing = 222 * 1024;

struct TallArgs {
  bf16* c;
  long long ldc;
  int M, N, K;               // N: columns of C
  int bn;                    // weight rows of a tile: as many columns of C, or kGlu bn / 2 gate and bn / 2 up rows
  int last_rows;             // rows of the last row block that are loaded (the rest of its operand is whatever the ring held)
  int stages;
  int beside;                // launch_beside()
};
// accumulator columns of a row block, and the most that row blocks leave room for in tensor memory
__host__ __device__ constexpr int tall_columns(int bn) { return (bn + 31) / 32 * 32; }
constexpr int tall_most_columns(int mt) { return mt <= 2 ? 256 : 160; }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}

template <int MT, bool kGlu>            // row blocks of 128
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
  const int per_tile = kGlu ? p.bn / 2 : p.bn;               // columns of C
  const int tiles = (p.N + per_tile - 1) / per_tile, num_kb = (p.K + kTlBK - 1) / kTlBK;
  // the weights of a stage follow its activations; the last row block's operand reaches into them where its rows are not loaded
  const int x_bytes = (MT - 1) * 16384 + p.last_rows * 128, half_bytes = per_tile * 128, stage_bytes = x_bytes + p.bn * 128;
  const int cols = tall_columns(p.bn);
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, 4);
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
      for (int tile = (int)blockIdx.x; tile < tiles && ok; tile += (int)gridDim.x) {
        const int n0 = tile * per_tile;
        for (int kb = 0; kb < num_kb; ++kb) {
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
      for (int tile = (int)blockIdx.x; tile < tiles && ok; tile += (int)gridDim.x, ++local) {
        if (local > 0 && !mbar_wait(&acc_empty, (local - 1) & 1, guard, kTimeoutAccEmpty)) break;
        tc_fence_after();
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&full[stage], phase, guard, kTimeoutTmaFull)) { ok = false; break; }
          tc_fence_after();
          const uint64_t xd = smem_desc_kmajor_sw128(smem_u32(smem + stage * stage_bytes)), wd = xd + (x_bytes >> 4);
#pragma unroll
          for (int k = 0; k < kTlBK / 16; ++k)
#pragma unroll
            for (int m = 0; m < MT; ++m)
              umma_ss(tmem_base + m * cols, xd + m * 1024 + k * 2, wd + k * 2, idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit(&empty[stage]);
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit(&acc_full);
      }
    }
    __syncwarp();
  } else {
    const int quad = warp & 3;
    int local = 0;
    for (int tile = (int)blockIdx.x; tile < tiles; tile += (int)gridDim.x, ++local) {
      if (!mbar_wait(&acc_full, local & 1, guard, kTimeoutAccFull)) break;
      tc_fence_after();
      const int n0 = tile * per_tile, n = min(per_tile, p.N - n0);
#pragma unroll 1
      for (int m = 0; m < MT; ++m) {
        const int row = m * 128 + quad * 32 + lane;
        const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + m * cols;
        bf16* dst = p.c + (long long)row * p.ldc + n0;
#pragma unroll 2
        for (int f = 0; f < n; f += 8) {
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
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  grid_dependency_leave(p.beside);
}

template <int MT, bool kGlu>
static int launch_tall(const void* x, const void* w, TallArgs p, long long ldx, long long ldw, cudaStream_t st) {
  CUtensorMap tmX, tmXl, tmW;
  int rc;
  p.last_rows = (p.M - (MT - 1) * 128 + 7) / 8 * 8;
  for (int last = 0; last < 2; ++last) {
    uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)p.M};
    uint64_t str[2] = {2, (uint64_t)ldx * 2};
    uint32_t box[2] = {kTlBK, (uint32_t)(last ? p.last_rows : 128)};
    if ((rc = make_tmap(last ? &tmXl : &tmX, x, 2, 2, dims, str, box, true))) return rc;
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
  auto kern = gemm_tall_kernel<MT, kGlu>;
  static PerDevice raised;
  KSA_CHECK_CUDA(raise_smem_limit(raised, kern, kTlRing + 1024));
  const int per_tile = kGlu ? p.bn / 2 : p.bn;
  const int sms = sm_count(), tiles = (p.N + per_tile - 1) / per_tile;
  KSA_REQUIRE(sms > 0, "no device");
  int* status = status_word();
  KSA_REQUIRE(status != nullptr, "could not allocate the status word");
  KSA_CHECK_CUDA(launch_kernel(kern, dim3(tiles < sms ? tiles : sms), dim3(kTlThreads), (size_t)(p.stages * stage_bytes + slack + 1024), st, tmX,
                               tmXl, tmW, p, status));
  return 0;
}

}  // namespace ksa

// C[M, N] (bf16) = X W^T, X [M, K], W [N, K] row-major; glu: W holds N gate rows, then N up rows, and C = silu(gate) * up with both products
// rounded to bf16 first.  M <= 384; columns: weight rows of a tile, a multiple of 16 up to 256 (M <= 256) or 160.
KSA_API int ksa_gemm_tall_bf16(const void* x, const void* w, void* c, int M, int N, int K, long long ldx, long long ldw, long long ldc, int glu,
                               int columns, void* stream) {
  KSA_ENTER(x);
  using namespace ksa;
  KSA_REQUIRE(M > 0 && N > 0 && K > 0 && M <= 384, "gemm_tall: %d rows, %d columns of %d", M, N, K);
  KSA_REQUIRE(ldx % 8 == 0 && ldw % 8 == 0, "gemm_tall: ldx/ldw must be multiples of 8 elements (got %lld, %lld)", ldx, ldw);
  KSA_REQUIRE(N % 8 == 0 && ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0, "gemm_tall: rows of C must keep 16-byte alignment");
  const int mt = (M + 127) / 128;
  KSA_REQUIRE(columns >= 16 && columns % 16 == 0 && columns <= tall_most_columns(mt), "gemm_tall: tiles of %d columns for %d rows", columns, M);
  TallArgs p{static_cast<bf16*>(c), ldc, M, N, K, columns, 0, 0, launch_beside()};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define KSA_TALL(MT) return glu ? launch_tall<MT, true>(x, w, p, ldx, ldw, st) : launch_tall<MT, false>(x, w, p, ldx, ldw, st)
  if (mt <= 1) KSA_TALL(1);
  if (mt == 2) KSA_TALL(2);
  KSA_TALL(3);
#undef KSA_TALL
}

// Weight rows of a tile of ksa_gemm_tall_bf16 where that kernel is taken, else 0 (then the split-K kernel or tiles of 128 rows are).
// The tile is the smallest that gives no SM more tiles than another, and it must be wide enough: a 64-wide step of K takes 0.17 us at least
// (one trip to memory over the stages in flight), 0.1 more for each further block of rows.  us of the others and here where the lines lie:
//   * up to 128 rows from 48 columns on: 6144 x 2560 (48 columns) 48 rows 13.5 -> 10.4, but 2560 x 4096 (32) 128 rows 13.3 -> 14.5; with
//     fewer than 64 rows and a long K from 80 on, where a K split reads as fast: 9216 x 4096 (64) 48 rows 17.5 -> 17.8;
//   * up to 224 columns, with 256 there are too few stages: 2 x 18944 x 3584 17 rows 46.1 -> 48.0, 2 x 14336 x 4096 (208) 48 rows 44.6 -> 43.5;
//   * several tiles to an SM from 160 columns on, as nothing covers the time between them: 151936 x 2560 (208) 128 rows 195 -> 154,
//     2 x 18944 x 3584 (128) 48 rows 47.3 -> 48.3; one only above 128 rows (151936 x 2560 256 rows 164 -> 238);
//   * more rows with SwiGLU only, which the others leave to a launch of its own from some 200 rows on (12288 x 2048 without it, 256 rows
//     17.9 -> 18.0; 16384 x 4096 34.6 -> 38.0): up to 256 rows to 160 columns (2 x 14336 x 4096, 208: 130 rows 54.1 -> 61.4; 2 x 3072 x 1024, 48:
//     256 rows 18.9 -> 9.3; 2 x 1536 x 2048, 32: 130 rows 9.7 -> 11.5), up to 384 from 144 (2 x 9728 x 2560 384 rows 48.4 -> 39.5; 2 x 8960 x 1536,
//     128: 264 rows 21.6 -> 23.0); four blocks of rows never (2 x 9728 x 2560 479 rows 55.7 -> 66.0);
//   * projections to 96 columns and the output head without it: what lies between is gate and up rows, which come with SwiGLU.
// ragged: rows off the 128-byte lines, which the split-K kernel's model knows about.
KSA_API int ksa_gemm_tall_plan(int M, int N, int K, int glu, int ragged) {
  if (M <= 16 || M > (glu ? 384 : 128) || N <= 0 || K <= 0 || ragged || N % 8 != 0) return 0;
  constexpr int kSms = 148;
  const int mt = (M + 127) / 128, most = mt == 1 ? 224 : 160;
  const long long rows = (glu ? 2LL : 1LL) * N, waves = (rows + (long long)kSms * most - 1) / ((long long)kSms * most);
  if (waves > 1 && mt > 1) return 0;
  const int columns = (int)(((rows + kSms * waves - 1) / (kSms * waves) + 15) / 16 * 16);
  const int least = mt == 3 ? 144 : mt == 2 ? 48 : waves > 1 ? 160 : M < 64 && K > 3072 ? 80 : 48;
  return columns >= least && (glu || waves > 1 || columns <= 96) ? columns : 0;
}
