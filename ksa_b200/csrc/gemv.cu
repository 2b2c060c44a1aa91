// Skinny GEMM for decoding: C[M, N] = A[M, K] * B[N, K]^T with M <= 16 rows (one token per sequence of the batch).
// The work is a stream of the weight matrix B, and what bounds it is how early and how steadily every SM asks for its share:
//   * one CTA per SM, and each owns the same number of weight rows (+-1) whatever N is, so no last wave is left over;
//   * a producer thread brings the rows in as TMA boxes of 64 columns through a ring of some 90 KB of shared memory, so a CTA keeps
//     its share of the memory system busy from its first cycle to its last; the activations of the same columns travel in
//     the same stages;
//   * eight warps split the 16-wide steps of K of a stage among themselves and multiply with mma.sync m16n8k16 (16 weight rows by
//     8 or 16 activation rows; a 128-row tcgen05 tile would leave most SMs without a tile), and their partial sums meet in shared
//     memory once per group of at most 32 rows.
// (Untiled bulk copies of whole row segments to rows padded by 16 bytes reached 11 GB/s an SM, a quarter of its share: a destination
// off the 128-byte lines is written 16 bytes at a time.  The boxes' 128-byte swizzle serves ldmatrix as well.)
//
// Measured against scalar products (up to 4 rows with a norm) and mma.sync on register tiles with a barrier every 1024 columns,
// weights from memory, us: 4 rows x 2560 x 9728 21.5 -> 12.5 (the weights alone take 7.6 at the copy bandwidth), 16 rows 24.5 -> 12.3,
// 16 x 6144 x 2560 15.1 -> 9.3, 16 x 151936 x 2560 208 -> 118; with the norm, 4 x 6144 x 2560 25.4 -> 10.8, 4 x 19456 x 2560 with
// SwiGLU 41.6 -> 22.7.  Integer divisions by the number of stages in the producer's loop alone had cost 0.4 us a stage.
//
// A decode step is a chain of such kernels, each a few microseconds long, so the engine switches early weights on for its
// thread (host.h): a CTA that starts beside the CTA of the previous kernel of the stream (both fit one SM) then fills its whole ring
// with weights, which no earlier kernel writes, and only after that waits for the previous kernel (griddepcontrol.wait) and
// reads the activations.  The gate/up projection can apply SwiGLU itself (kGlu): a group then holds matching gate and up
// rows and the CTA writes silu(gate) * up.  Every wait is bounded; no TMA load uses multicast.
#include "common.cuh"
#include "host.h"

namespace ksa {

constexpr int kStWarps = 8;                        // warps that multiply
constexpr int kStThreads = kStWarps * 32;
constexpr int kStMaxStages = 16;
constexpr int kStBlocks = 2;                       // 16-row blocks of a group
constexpr int kStBarrierBytes = 2 * kStMaxStages * 8 + 64;
constexpr int kStBoxes = 8;                        // boxes of 64 columns a stage at most
constexpr int kStSmemMost = 225 * 1024;

// kGlu: B holds N/2 gate rows followed by N/2 up rows; C[m, f] = silu(gate) * up has N/2 columns.
// Optional residual add + RMSNorm in front of the projection (a decode step's `x + delta -> norm -> projection`): the
// activation rows are then A = bf16(rms_norm(bf16(A + delta)) * w), computed by every CTA and kept in its shared memory (the
// rows are a few kilobytes), and CTA 0 also writes the new residual stream bf16(A + delta) to `res_out`.
struct GemvNorm {
  const bf16* delta;     // [delta_rows, K] or null
  const bf16* w;         // [K] norm weight; null: no norm, A is used as it is
  bf16* res_out;         // [M, K] or null
  long long ld_delta, ld_res;
  float eps;
  int delta_rows;
};

struct StreamArgs {
  const bf16* A;         // read directly for the norm only
  bf16* C;
  long long lda, ldc;
  int M, N, K;
  int groups, per_group; // row groups of a CTA, and their output columns
  int boxes;             // boxes of 64 columns of a stage
  int ragged;            // K is no multiple of 64: one load per box, which fills the columns past K with zeros
  int w_rows, x_rows;    // rows of a box in shared memory (weights, activations): those loaded, for `ragged` in whole swizzle atoms
  int stages, stage_bytes;
  GemvNorm nrm;
};

__device__ __forceinline__ void mma_bf16_16x8x16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                 uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void multiply_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kStThreads) : "memory"); }

// byte offset of columns 8 q .. 8 q + 7 (q < 8) of row r in a box of 128-byte rows with the 128-byte swizzle
__device__ __forceinline__ uint32_t swizzled(int r, int q) { return (uint32_t)(r * 128 + ((q ^ (r & 7)) << 4)); }

// When the kernel waits for the one before it, and when it lets the one after it start.  Known to the compiler: with the conditions in the
// kernels that a decode step launches, a step of four sequences took 442 us instead of 420.
enum StreamMode {
  kStWaits,      // before it reads anything; the successor of a block's first product (a norm, SwiGLU) starts behind that, and so may
                 // take weights to be as they are for good (ops.linear_of_block: a feed-forward block of one row 32.3 -> 31.4 us)
  kStEarly,      // weights_early(): the weights are read before the previous kernel has ended, and the successor starts at once
  kStBeside,     // launch_beside(): before it ends; all that it reads of global memory goes through the producer
};
// NB: batch blocks of 8 rows, 1 (M <= 8) or 2 (M <= 16)
template <int NB, bool kGlu, bool kNorm, StreamMode kMode>
__global__ void __launch_bounds__(kStThreads + 32, 2)
stream_gemm_kernel(const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA, const StreamArgs p,
                   int* status) {
  extern __shared__ uint8_t st_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(st_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + p.stages * p.stage_bytes);
  uint64_t* empty = full + kStMaxStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + kStMaxStages);
  float* part = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(full) + kStBarrierBytes);   // [warps][NB * 8][part_pitch]
  const int half_rows = (p.per_group + 15) / 16 * 16;               // rows of a half (gate, up), in whole blocks
  const int part_pitch = half_rows * (kGlu ? 2 : 1) + 4;     // 4 modulo 16: the fragments' stores and the sums' loads both miss no bank twice
  uint8_t* xres = reinterpret_cast<uint8_t*>(part + kStWarps * NB * 8 * part_pitch);    // kNorm: [M][K] + 16 to 32 bytes a row
  const int xpitch = (p.K + 15) / 16 * 32 + 16;
  __shared__ float s_red[kStWarps][4], s_rstd[4];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const WaitGuard guard{abort_flag, status};
  const int n_out = kGlu ? p.N / 2 : p.N;
  const int c0 = (int)blockIdx.x * p.groups * p.per_group;           // first output column of this CTA
  const int groups = min(p.groups, (n_out - c0 + p.per_group - 1) / p.per_group);
  const int num_kb = (p.K + 63) / 64, nk = (num_kb + p.boxes - 1) / p.boxes;
  const int n_items = groups * nk;
  const int w_bytes = (p.boxes * p.w_rows + 7) / 8 * 1024;        // a box of weights (of the gate or the up half)
  const int x_off = w_bytes * (kGlu ? 2 : 1);                        // the activations' box follows the weights'

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], kStWarps); }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmB);
    if (!kNorm) tma_prefetch_desc(&tmA);
  }
  __syncthreads();
  // the plain product's successor starts at once in every mode (16 x 6144 x 2560 7.7 us in a row of them, 7.9 with the later start)
  constexpr bool kAtOnce = kMode != kStWaits || (!kGlu && !kNorm);
  if (kAtOnce) grid_dependency_launch();

  if (warp == kStWarps) {
    // ------------------------------------------------------------ producer: lane 0, or for `ragged` a lane per box
    // position in the ring and in the matrix, carried along: a division a stage costs more than its loads
    struct Cursor {
      int stage = 0, kb = 0, row;
      uint32_t phase = 1;
    } w, x;
    w.row = c0;
    auto next = [&](Cursor& c) {
      if (++c.stage == p.stages) { c.stage = 0; c.phase ^= 1; }
      if ((c.kb += p.boxes) >= num_kb) { c.kb = 0; c.row += p.per_group; }
    };
    const uint32_t bytes = p.boxes * 128 * (p.per_group * (kGlu ? 2 : 1) + (kNorm ? 0 : p.M));     // also past the matrix's edges
    auto load_weights = [&]() {
      uint8_t* dst = ring + w.stage * p.stage_bytes;
      if (lane == 0) mbar_expect_tx(&full[w.stage], bytes);
      __syncwarp();
      if (lane < (p.ragged ? p.boxes : 1)) {
        const int col = p.ragged ? (w.kb + lane) * 64 : 0, kb = p.ragged ? 0 : w.kb;
        dst += lane * p.w_rows * 128;
        tma_load_3d(dst, &tmB, col, w.row, kb, &full[w.stage]);
        if (kGlu) tma_load_3d(dst + w_bytes, &tmB, col, n_out + w.row, kb, &full[w.stage]);
      }
      next(w);
    };
    auto load_acts = [&]() {
      if (kNorm) return;
      if (lane < (p.ragged ? p.boxes : 1))
        tma_load_3d(ring + x.stage * p.stage_bytes + x_off + lane * p.x_rows * 128, &tmA, p.ragged ? (x.kb + lane) * 64 : 0, 0,
                    p.ragged ? 0 : x.kb, &full[x.stage]);
      next(x);
    };
    // in a decode step weights do not depend on the previous kernel; the activations do
    if (kMode == kStWaits) grid_dependency_wait();
    if (kMode == kStBeside) grid_dependency_observe();
    if (!kAtOnce) grid_dependency_launch();
    const int ahead = min(p.stages, n_items);
    for (int it = 0; it < ahead; ++it) load_weights();
    if (kMode == kStEarly) grid_dependency_wait();
    for (int it = 0; it < ahead; ++it) load_acts();
    for (int it = ahead; it < n_items; ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait(&empty[w.stage], w.phase, guard, kTimeoutStageEmpty))) break;
      load_weights();
      load_acts();
    }
    return;
  }

  // -------------------------------------------------------------- the eight warps that multiply
  if (kMode != kStBeside) grid_dependency_wait();     // also for the outputs: an earlier kernel may still read their memory
  if (kNorm) {
    float ss[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = threadIdx.x * 8; c < p.K; c += kStThreads * 8) {
      uint4 xv[4], dv[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        xv[m] = dv[m] = make_uint4(0, 0, 0, 0);
        if (m < p.M) {
          xv[m] = *reinterpret_cast<const uint4*>(p.A + m * p.lda + c);
          if (m < p.nrm.delta_rows) dv[m] = *reinterpret_cast<const uint4*>(p.nrm.delta + m * p.nrm.ld_delta + c);
        }
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (m >= p.M) break;
        const uint32_t xu[4] = {xv[m].x, xv[m].y, xv[m].z, xv[m].w}, du[4] = {dv[m].x, dv[m].y, dv[m].z, dv[m].w};
        uint32_t o[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float2 f = unpack_bf16x2(xu[q]);
          if (m < p.nrm.delta_rows) {
            const float2 d = unpack_bf16x2(du[q]);
            f.x = __bfloat162float(__float2bfloat16(f.x + d.x));
            f.y = __bfloat162float(__float2bfloat16(f.y + d.y));
          }
          ss[m] += f.x * f.x + f.y * f.y;
          o[q] = pack_bf16x2(f.x, f.y);
        }
        const uint4 r = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(xres + m * xpitch + c * 2) = r;
        if (blockIdx.x == 0 && p.nrm.res_out != nullptr)
          *reinterpret_cast<uint4*>(p.nrm.res_out + m * p.nrm.ld_res + c) = r;
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      ss[m] = warp_sum(ss[m]);
      if (lane == 0) s_red[warp][m] = ss[m];
    }
    if (p.K % 16 != 0 && threadIdx.x < p.M)               // columns K .. K + 7 take part in the last step, against zeros
      *reinterpret_cast<uint4*>(xres + threadIdx.x * xpitch + p.K * 2) = make_uint4(0, 0, 0, 0);
    multiply_sync();
    if (threadIdx.x < 4) {
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < kStWarps; ++k) t += s_red[k][threadIdx.x];
      s_rstd[threadIdx.x] = rsqrtf(t / (float)p.K + p.nrm.eps);
    }
    multiply_sync();
    for (int c = threadIdx.x * 8; c < p.K; c += kStThreads * 8) {      // a thread's own columns again
      const uint4 wv = *reinterpret_cast<const uint4*>(p.nrm.w + c);
      const uint32_t wu[4] = {wv.x, wv.y, wv.z, wv.w};
      for (int m = 0; m < p.M; ++m) {
        uint4* at = reinterpret_cast<uint4*>(xres + m * xpitch + c * 2);
        const uint4 xv = *at;
        const uint32_t xu[4] = {xv.x, xv.y, xv.z, xv.w};
        const float rstd = s_rstd[m];
        uint32_t o[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 x = unpack_bf16x2(xu[q]), f = unpack_bf16x2(wu[q]);
          o[q] = pack_bf16x2(x.x * rstd * f.x, x.y * rstd * f.y);
        }
        *at = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
    multiply_sync();
  }

  bool ok = true;
  int stage = 0;
  uint32_t phase = 0;
  for (int g = 0; g < groups; ++g) {
    const int f0 = c0 + g * p.per_group, nf = min(p.per_group, n_out - f0);
    const int nblk = (nf + 15) / 16;                 // blocks in use: of the gate and of the up half each for kGlu
    constexpr int kHalf = kGlu ? kStBlocks / 2 : kStBlocks;
    // this lane's row of every block (rows past the end repeat the last one; their sums are dropped) ..
    int row[kStBlocks];
#pragma unroll
    for (int b = 0; b < kStBlocks; ++b) row[b] = min((b % kHalf) * 16 + (lane & 15), nf - 1);
    // .. and of the activations: lanes 0-7 / 8-15 rows 0-7 at k and k + 8, lanes 16-31 the same of rows 8-15
    const int xrow = min((lane & 7) + (NB == 2 ? (lane >> 4) * 8 : 0), p.M - 1), xq = (lane >> 3) & 1;
    float acc[kStBlocks][NB][4];
#pragma unroll
    for (int b = 0; b < kStBlocks; ++b)
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[b][n][i] = 0.f;

    for (int kb = 0; kb < num_kb; kb += p.boxes) {
      if (ok) ok = mbar_wait(&full[stage], phase, guard, kTimeoutTmaFull);
      if (ok) {
        // steps of 16 columns, four to a box; columns past K are zeros in both operands
        const int steps = min(p.boxes * 4, (p.K - kb * 64 + 15) / 16);
        const uint32_t sw = smem_u32(ring + stage * p.stage_bytes);
        const uint32_t sx = kNorm ? smem_u32(xres) + xrow * xpitch + kb * 128 + xq * 16 : sw + x_off;
#pragma unroll
        for (int u = 0; u < kStBoxes * 4 / kStWarps; ++u) {
          const int s = u * kStWarps + warp, box = s >> 2, q = (s & 3) * 2;
          if (s >= steps) break;
          uint32_t x[4];                              // NB == 1: lanes 16-31 repeat lanes 0-15, x[2] and x[3] are not used
          ldmatrix4(x, kNorm ? sx + s * 32 : sx + swizzled(box * p.x_rows + xrow, q + xq));
#pragma unroll
          for (int b = 0; b < kStBlocks; ++b) {
            if (b % kHalf >= nblk) continue;
            uint32_t w[4];
            ldmatrix4(w, sw + (b >= kHalf ? w_bytes : 0) + swizzled(box * p.w_rows + row[b], q + (lane >> 4)));
#pragma unroll
            for (int n = 0; n < NB; ++n) mma_bf16_16x8x16(acc[b][n], w[0], w[1], w[2], w[3], x[2 * n], x[2 * n + 1]);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    // acc[b][n] = {D[gr][2t], D[gr][2t + 1], D[gr + 8][2t], D[gr + 8][2t + 1]}: rows of the block by activation rows 8 n + ..
    {
      const int gr = lane >> 2, t = lane & 3;
      float* dst = part + warp * NB * 8 * part_pitch;
#pragma unroll
      for (int b = 0; b < kStBlocks; ++b) {
        if (b % kHalf >= nblk) continue;
        const int r = (b % kHalf) * 16 + gr + (b >= kHalf ? half_rows : 0);
#pragma unroll
        for (int n = 0; n < NB; ++n) {
          float* at = dst + (n * 8 + 2 * t) * part_pitch + r;
          at[0] = acc[b][n][0];
          at[part_pitch] = acc[b][n][1];
          at[8] = acc[b][n][2];
          at[part_pitch + 8] = acc[b][n][3];
        }
      }
      multiply_sync();
      if (ok) {
        for (int i = threadIdx.x; i < nf * p.M; i += kStThreads) {
          const int f = i % nf, m = i / nf;            // consecutive threads -> consecutive outputs
          float v = 0.f, u = 0.f;
#pragma unroll
          for (int w = 0; w < kStWarps; ++w) {
            const float* src = part + (w * NB * 8 + m) * part_pitch + f;
            v += src[0];
            if (kGlu) u += src[half_rows];
          }
          if (kGlu) {
            // gate and up are rounded to bf16 first, as the separate projection + SwiGLU kernels do
            const float gt = __bfloat162float(__float2bfloat16(v)), up = __bfloat162float(__float2bfloat16(u));
            v = gt / (1.f + __expf(-gt)) * up;
          }
          p.C[(long long)m * p.ldc + f0 + f] = __float2bfloat16(v);
        }
      }
      multiply_sync();        // the next group's partial sums overwrite these
    }
  }
  if (kMode == kStBeside) grid_dependency_leave(1);
}

template <int NB, bool kGlu, bool kNorm, StreamMode kMode>
static int launch_stream(StreamArgs p, const void* b, long long ldb, cudaStream_t st) {
  const int sms = sm_count();
  KSA_REQUIRE(sms > 0, "gemv: no device");
  int* status = status_word();
  KSA_REQUIRE(status != nullptr, "could not allocate the status word");
  const int n_out = kGlu ? p.N / 2 : p.N;
  const int most = (n_out + sms - 1) / sms;                       // output columns of a CTA
  constexpr int kCap = kStBlocks * 16 / (kGlu ? 2 : 1);
  p.groups = (most + kCap - 1) / kCap;
  p.per_group = (most + p.groups - 1) / p.groups;
  const int grid = (n_out + p.groups * p.per_group - 1) / (p.groups * p.per_group);
  const int num_kb = (p.K + 63) / 64;
  p.ragged = p.K % 64 != 0;
  p.w_rows = p.ragged ? (p.per_group + 7) / 8 * 8 : p.per_group;
  p.x_rows = p.ragged ? NB * 8 : p.M;
  p.boxes = kStBoxes;
  if (p.boxes > num_kb) p.boxes = num_kb;
  p.stage_bytes = (p.boxes * p.w_rows + 7) / 8 * 1024 * (kGlu ? 2 : 1) + (kNorm ? 0 : (p.boxes * p.x_rows + 7) / 8 * 1024);
  const int part_pitch = (p.per_group + 15) / 16 * 16 * (kGlu ? 2 : 1) + 4;
  const int fixed = 1024 + kStBarrierBytes + kStWarps * NB * 8 * part_pitch * 4 + (kNorm ? p.M * ((p.K + 15) / 16 * 32 + 16) : 0);
  const int n_items = p.groups * ((num_kb + p.boxes - 1) / p.boxes);
  // Both limits together leave room for this kernel and its neighbour in a decode step on one SM.  A ring of two stages, or of
  // less than 64 KB, does not hide the memory's latency: the ring is then as large as it can be (4 x 151936 x 2560 with two stages of
  // 36 KB 132 us, with five 117).
  const int beside = (kNorm ? 130 : 96) * 1024, ring = beside - fixed;
  const int limit = ring < 3 * p.stage_bytes || ring < 64 * 1024 ? kStSmemMost : beside;
  p.stages = (limit - fixed) / p.stage_bytes;
  if (p.stages > kStMaxStages) p.stages = kStMaxStages;
  if (p.stages > n_items) p.stages = n_items;
  KSA_REQUIRE(p.stages >= 1, "gemv: %d rows of %d columns do not fit shared memory", p.M, p.K);
  const int smem = fixed + p.stages * p.stage_bytes;
  CUtensorMap tmB, tmA;
  int rc;
  {
    uint64_t dims[3] = {(uint64_t)(p.ragged ? p.K : 64), (uint64_t)p.N, (uint64_t)(p.ragged ? 1 : num_kb)};
    uint64_t str[3] = {2, (uint64_t)(p.N == 1 ? p.K : ldb) * 2, 128};       // one row: its pitch may be anything
    uint32_t box[3] = {64, (uint32_t)p.per_group, (uint32_t)(p.ragged ? 1 : p.boxes)};
    if ((rc = make_tmap(&tmB, b, 2, 3, dims, str, box, true))) return rc;
  }
  if (kNorm) {
    tmA = tmB;       // not used
  } else {
    uint64_t dims[3] = {(uint64_t)(p.ragged ? p.K : 64), (uint64_t)p.M, (uint64_t)(p.ragged ? 1 : num_kb)};
    uint64_t str[3] = {2, (uint64_t)(p.M == 1 ? p.K : p.lda) * 2, 128};
    uint32_t box[3] = {64, (uint32_t)p.M, (uint32_t)(p.ragged ? 1 : p.boxes)};
    if ((rc = make_tmap(&tmA, p.A, 2, 3, dims, str, box, true))) return rc;
  }
  auto kern = stream_gemm_kernel<NB, kGlu, kNorm, kMode>;
  static PerDevice raised;
  KSA_CHECK_CUDA(raise_smem_limit(raised, kern, kStSmemMost));
  KSA_CHECK_CUDA(launch_kernel(kern, dim3(grid), dim3(kStThreads + 32), (size_t)smem, st, tmB, tmA,
                              p, status));
  return 0;
}

// ------------------------------------------------------------------------------------------ one and two rows
// Each warp streams whole weight rows with 16-byte loads and multiplies on the FMA units; the activation rows sit in shared memory.
// No ring to set up and as many CTAs as there are rows for, which the hardware deals out as SMs become free: launched by itself it
// starts 0.7 us earlier than the ring and ends more evenly (one row x 2560 x 4096 6.4 against 7.1 us, x 151936 x 2560 108 against 115).
// kGlu: weight row r of a warp is gate row f for even r and up row f for odd r (f = first feature + r / 2).
constexpr int kGemvThreads = 256;
constexpr int kGemvKTile = 2048;   // activation columns staged in shared memory per pass

// 16-byte load that does not pollute L1: every weight byte is used once per step
__device__ __forceinline__ uint4 ld_stream_16(const void* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

template <int MT, int R, bool kGlu, bool kBeside>
__global__ void __launch_bounds__(kGemvThreads)
gemv_kernel(const bf16* A, const bf16* B, bf16* C, int M, int N, int K,
            long long lda, long long ldb, long long ldc, int early) {
  extern __shared__ __align__(16) uint8_t gemv_smem[];
  bf16* sA = reinterpret_cast<bf16*>(gemv_smem);           // [MT][kGemvKTile]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * (kGemvThreads / 32) + warp) * (kGlu ? R / 2 : R);   // first row / first feature
  const int n_out = kGlu ? N / 2 : N;
  long long row_of[R];       // weight row of slot r, or -1 past the end
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int f = kGlu ? n0 + r / 2 : n0 + r;
    row_of[r] = f < n_out ? (long long)(kGlu && (r & 1) ? n_out + f : f) : -1;
  }
  float acc[R][MT];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[r][m] = 0.f;

  // U chunks of every row are requested before any is used, so that enough loads are in flight per SM
  constexpr int U = (R >= 4) ? 2 : (R == 2 ? 4 : 8);
  uint4 w[U][R];
  auto load_w = [&](int k0, int kt, int c0) {
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int c = c0 + u * 256;
        w[u][r] = make_uint4(0, 0, 0, 0);
        if (c < kt && row_of[r] >= 0) w[u][r] = ld_stream_16(B + row_of[r] * ldb + k0 + c);
      }
  };
  // in a decode step weights are not written by an earlier kernel of the stream: ask for the first chunks, then wait for the
  // kernel that produces the activations
  if (kBeside) grid_dependency_enter(1);
  else if (!early) grid_dependency_wait();
  load_w(0, min(kGemvKTile, K), lane * 8);
  if (!kBeside) grid_dependency_enter();

  for (int k0 = 0; k0 < K; k0 += kGemvKTile) {
    const int kt = min(kGemvKTile, K - k0);          // multiple of 8
    __syncthreads();
    for (int i = threadIdx.x; i < MT * (kGemvKTile / 8); i += kGemvThreads) {
      const int m = i / (kGemvKTile / 8), c = (i % (kGemvKTile / 8)) * 8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (m < M && c < kt) v = *reinterpret_cast<const uint4*>(A + (long long)m * lda + k0 + c);
      *reinterpret_cast<uint4*>(sA + m * kGemvKTile + c) = v;
    }
    __syncthreads();
    for (int c0 = lane * 8; c0 < kt; c0 += 256 * U) {
      if (k0 != 0 || c0 != lane * 8) load_w(k0, kt, c0);      // the very first chunks are already on their way
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = c0 + u * 256;
        if (c >= kt) break;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const uint4 a = *reinterpret_cast<const uint4*>(sA + m * kGemvKTile + c);
          const uint32_t au[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const uint32_t wu[4] = {w[u][r].x, w[u][r].y, w[u][r].z, w[u][r].w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float2 x = unpack_bf16x2(au[q]), y = unpack_bf16x2(wu[q]);
              acc[r][m] = fmaf(x.x, y.x, acc[r][m]);
              acc[r][m] = fmaf(x.y, y.y, acc[r][m]);
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[r][m] = warp_sum(acc[r][m]);
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < R; r += (kGlu ? 2 : 1)) {
      const int f = kGlu ? n0 + r / 2 : n0 + r;
      if (f >= n_out) break;
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        if (m >= M) break;
        float v = acc[r][m];
        if (kGlu) {
          // gate and up are rounded to bf16 first, as the separate projection + SwiGLU kernels do
          const float g = __bfloat162float(__float2bfloat16(v));
          const float u = __bfloat162float(__float2bfloat16(acc[r + (kGlu ? 1 : 0)][m]));
          v = g / (1.f + __expf(-g)) * u;
        }
        C[(long long)m * ldc + f] = __float2bfloat16(v);
      }
    }
  }
  if (kBeside) grid_dependency_leave(1);
}

template <int MT, int R, bool kGlu, bool kBeside = false>
static int launch_gemv(const void* a, const void* b, void* c, int M, int N, int K, long long lda, long long ldb,
                       long long ldc, cudaStream_t st) {
  const int per_cta = (kGemvThreads / 32) * (kGlu ? R / 2 : R);      // output columns per CTA
  const int n_out = kGlu ? N / 2 : N;
  const size_t smem = (size_t)MT * kGemvKTile * sizeof(bf16);
  auto kern = gemv_kernel<MT, R, kGlu, kBeside>;
  KSA_CHECK_CUDA(launch_kernel(kern, dim3((n_out + per_cta - 1) / per_cta),
                              dim3(kGemvThreads), smem, st, (const bf16*)a, (const bf16*)b, (bf16*)c, M, N, K, lda, ldb,
                              ldc, (int)weights_early()));
  return 0;
}

template <bool kGlu>
static int gemv_dispatch(const void* a, const void* b, void* c, int M, int N, int K, long long lda, long long ldb,
                         long long ldc, cudaStream_t st, const GemvNorm& nrm = GemvNorm{}) {
  KSA_REQUIRE(((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(nrm.delta) |
                reinterpret_cast<uintptr_t>(nrm.w) | reinterpret_cast<uintptr_t>(nrm.res_out)) & 15) == 0,
              "gemv: the operands must be 16-byte aligned");
  StreamArgs p{};
  p.A = (const bf16*)a; p.C = (bf16*)c;
  p.lda = lda; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
  p.nrm = nrm;
  const bool early = weights_early();
  if (nrm.w != nullptr) return early ? launch_stream<1, kGlu, true, kStEarly>(p, b, ldb, st) : launch_stream<1, kGlu, true, kStWaits>(p, b, ldb, st);
  if (!kGlu && launch_beside()) {          // the summary rows of a short prompt: the same kernels as below
    if (M > 8) return launch_stream<2, false, false, kStBeside>(p, b, ldb, st);
    if (M > 2) return launch_stream<1, false, false, kStBeside>(p, b, ldb, st);
    if (M == 1) return N <= 8192 ? launch_gemv<1, 1, false, true>(a, b, c, M, N, K, lda, ldb, ldc, st)
                                 : launch_gemv<1, 4, false, true>(a, b, c, M, N, K, lda, ldb, ldc, st);
    return N <= 8192 ? launch_gemv<2, 1, false, true>(a, b, c, M, N, K, lda, ldb, ldc, st)
                     : launch_gemv<2, 4, false, true>(a, b, c, M, N, K, lda, ldb, ldc, st);
  }
  // In a decode step the ring is filled while the previous kernel runs (one row x 2560 x 9728 10.4 against 11.9 us, x
  // 4096 x 2048 4.4 against 5.4, x 2560 x 4096 6.2 both); the output head is long enough not to need that.
  if (M <= 2 && !(early && N <= 32768)) {
    // rows per warp: fewer for narrow outputs so that the grid still covers every SM a few times (with SwiGLU a warp
    // needs at least one gate row and one up row)
    constexpr int R1 = kGlu ? 2 : 1;
    if (M == 1) return N <= 8192 ? launch_gemv<1, R1, kGlu>(a, b, c, M, N, K, lda, ldb, ldc, st)
                                 : launch_gemv<1, 4, kGlu>(a, b, c, M, N, K, lda, ldb, ldc, st);
    return N <= 8192 ? launch_gemv<2, R1, kGlu>(a, b, c, M, N, K, lda, ldb, ldc, st)
                     : launch_gemv<2, 4, kGlu>(a, b, c, M, N, K, lda, ldb, ldc, st);
  }
  if (early) return M <= 8 ? launch_stream<1, kGlu, false, kStEarly>(p, b, ldb, st) : launch_stream<2, kGlu, false, kStEarly>(p, b, ldb, st);
  return M <= 8 ? launch_stream<1, kGlu, false, kStWaits>(p, b, ldb, st) : launch_stream<2, kGlu, false, kStWaits>(p, b, ldb, st);
}
}  // namespace ksa

// C[M, N] (bf16, ldc) = A[M, K] (bf16, lda) * B[N, K]^T (bf16, ldb) for 1 <= M <= 16; K, lda, ldb multiples of 8.
KSA_API int ksa_gemv_bf16(const void* a, const void* b, void* c, int M, int N, int K, long long lda, long long ldb,
                          long long ldc, void* stream) {
  KSA_ENTER(a);
  using namespace ksa;
  KSA_REQUIRE(M >= 1 && M <= 16, "gemv: M=%d out of range (1..16)", M);
  KSA_REQUIRE(N > 0 && K > 0 && K % 8 == 0 && lda % 8 == 0 && ldb % 8 == 0, "gemv: K, lda, ldb must be multiples of 8");
  return gemv_dispatch<false>(a, b, c, M, N, K, lda, ldb, ldc, reinterpret_cast<cudaStream_t>(stream));
}

// The gate/up projection of a SwiGLU feed-forward block with its activation: B holds N/2 gate rows followed by N/2
// up rows, C[M, N/2] = silu(A * gate^T) * (A * up^T), gate and up rounded to bf16 before the activation.
KSA_API int ksa_gemv_swiglu_bf16(const void* a, const void* b, void* c, int M, int N, int K, long long lda,
                                 long long ldb, long long ldc, void* stream) {
  KSA_ENTER(a);
  using namespace ksa;
  KSA_REQUIRE(M >= 1 && M <= 16, "gemv_swiglu: M=%d out of range (1..16)", M);
  KSA_REQUIRE(N > 0 && N % 2 == 0 && K > 0 && K % 8 == 0 && lda % 8 == 0 && ldb % 8 == 0,
              "gemv_swiglu: N must be even and K, lda, ldb multiples of 8");
  return gemv_dispatch<true>(a, b, c, M, N, K, lda, ldb, ldc, reinterpret_cast<cudaStream_t>(stream));
}

// A decode step's `residual add -> RMSNorm -> projection` in one launch, for at most 4 rows:
//   res = bf16(x + delta)  (delta may be null or have fewer rows; written to res_out by one CTA when res_out is given)
//   C   = rms_norm(res, norm_w, eps) * B^T          (glu = 0; C is [M, N])
//   C   = silu(. * gate^T) * (. * up^T)             (glu = 1; B = gate rows then up rows, C is [M, N/2])
KSA_API int ksa_gemv_norm_bf16(const void* x, const void* delta, const void* norm_w, void* res_out, const void* b, void* c,
                               int M, int N, int K, long long ldx, long long ld_delta, long long ld_res, long long ldb,
                               long long ldc, float eps, int delta_rows, int glu, void* stream) {
  KSA_ENTER(x);
  using namespace ksa;
  KSA_REQUIRE(M >= 1 && M <= 4, "gemv_norm: M=%d out of range (1..4)", M);
  KSA_REQUIRE(norm_w != nullptr, "gemv_norm: the norm weight is required");
  KSA_REQUIRE(N > 0 && K > 0 && K % 8 == 0 && ldx % 8 == 0 && ldb % 8 == 0 && ld_delta % 8 == 0 && ld_res % 8 == 0,
              "gemv_norm: K and the leading dimensions must be multiples of 8");
  KSA_REQUIRE(!glu || N % 2 == 0, "gemv_norm: N must be even with glu");
  GemvNorm nrm{(const bf16*)delta, (const bf16*)norm_w, (bf16*)res_out, ld_delta, ld_res, eps, delta ? delta_rows : 0};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return glu ? gemv_dispatch<true>(x, b, c, M, N, K, ldx, ldb, ldc, st, nrm)
             : gemv_dispatch<false>(x, b, c, M, N, K, ldx, ldb, ldc, st, nrm);
}
