// Cross entropy over a chunk of bf16 logits, in place: per-row loss, and the logits become d(loss) / d(logits).
//
// Bound: the logits are read once and written once, 1.24 GB for 2048 x 151936.  A row (304 KB) fits no SM, and a CTA per row that reads
// it again for the sum and for the gradient reads it from memory each time, since the rows in flight are more than the L2 holds:
// 391 us, the whole copy bandwidth for three reads and a write.  Here a cluster of 1, 2, 4 or 8 CTAs keeps a row in its shared memory
// (at most 80 KB a CTA, two or three CTAs an SM, so that one loads while the others compute or store); the CTAs' maxima and sums meet
// through distributed shared memory: 296 us (100 rows 25 -> 17, 2048 x 32000 62 -> 59, 4096 x 4096 27 -> 23).  With 512 threads a CTA 327,
// with 1024 409; with parts of 40 KB 389.  Wider rows (above 327680 columns) go to the CTA per row.
#include "common.cuh"
#include "host.h"
#include "vec.cuh"

namespace ksa {

constexpr int kCeThreads = 256;
constexpr int kCePieces = 4;                        // loads of a CTA's part of the row
constexpr int kCeMostBytes = 80 * 1024;

// One CTA per row.  Writes per-row loss (0 for ignored rows) and turns the logits into d(loss)/d(logits) * (*grad_scale) in place.
__global__ void __launch_bounds__(kCeThreads)
cross_entropy_kernel(bf16* logits, const long long* labels, float* row_loss,
                     const float* grad_scale, int V, long long ld, int ignore_index, int write_grad) {
  grid_dependency_enter();
  __shared__ float red[32];
  const long long row = blockIdx.x;
  bf16* lg = logits + row * ld;
  const long long label = labels[row];
  const bool ignored = (label == ignore_index) || label < 0 || label >= V;
  const int nvec = V / 8;
  if (ignored) {
    if (threadIdx.x == 0) row_loss[row] = 0.f;
    if (write_grad) {
      BF8 z{{0, 0, 0, 0}};
      for (int i = threadIdx.x; i < nvec; i += kCeThreads) *reinterpret_cast<BF8*>(lg + i * 8) = z;
    }
    return;
  }
  float mx = -INFINITY;
  for (int i = threadIdx.x; i < nvec; i += kCeThreads) {
    float f[8];
    load8(lg + i * 8, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) mx = fmaxf(mx, f[j]);
  }
  mx = block_max<kCeThreads>(mx, red);
  float sum = 0.f;
  for (int i = threadIdx.x; i < nvec; i += kCeThreads) {
    float f[8];
    load8(lg + i * 8, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += __expf(f[j] - mx);
  }
  sum = block_sum<kCeThreads>(sum, red);
  const float lse = mx + __logf(sum);
  if (threadIdx.x == 0) row_loss[row] = lse - __bfloat162float(lg[label]);
  if (!write_grad) return;
  __syncthreads();
  const float gs = *grad_scale;
  const float inv = 1.f / sum;
  for (int i = threadIdx.x; i < nvec; i += kCeThreads) {
    float f[8];
    load8(lg + i * 8, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __expf(f[j] - mx) * inv;
      if ((long long)i * 8 + j == label) p -= 1.f;
      f[j] = p * gs;
    }
    store8(lg + i * 8, f);
  }
}

__device__ __forceinline__ float2 ce_ld_cluster(uint32_t local_addr, uint32_t rank) {
  float2 v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %2, %3;\n\tld.shared::cluster.v2.f32 {%0, %1}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y) : "r"(local_addr), "r"(rank) : "memory");
  return v;
}

// The same with the row in the shared memory of a cluster: CTA `rank` holds `part` vectors of 8 columns from rank * part on.
__global__ void __launch_bounds__(kCeThreads, 2)
cross_entropy_cluster_kernel(bf16* logits, const long long* labels, float* row_loss,
                             const float* grad_scale, int V, long long ld, int ignore_index, int write_grad, int ctas,
                             int part, int* status) {
  extern __shared__ __align__(128) uint8_t ce_smem[];
  __shared__ uint64_t full[kCePieces];
  __shared__ float red[32];
  __shared__ float2 s_mine;                          // maximum and sum of this CTA's columns
  __shared__ int abort_word;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const long long row = blockIdx.x / ctas;
  const int nvec = V / 8, v0 = (int)rank * part, n = max(0, min(part, nvec - v0));
  bf16* lg = logits + row * ld + (long long)v0 * 8;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kCePieces; ++i) mbar_init(&full[i], 1);
    abort_word = 0;
    fence_mbar_init();
  }
  __syncthreads();
  grid_dependency_enter();
  const long long label = labels[row];
  if (label == ignore_index || label < 0 || label >= V) {              // the same for the whole cluster
    if (threadIdx.x == 0 && rank == 0) row_loss[row] = 0.f;
    if (write_grad) {
      BF8 z{{0, 0, 0, 0}};
      for (int i = threadIdx.x; i < n; i += kCeThreads) *reinterpret_cast<BF8*>(lg + i * 8) = z;
    }
    return;
  }
  const int step = (n + kCePieces - 1) / kCePieces;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kCePieces; ++i) {
      const int lo = min(i * step, n), m = min(step, n - lo);
      if (m <= 0) { mbar_arrive(&full[i]); continue; }
      mbar_expect_tx(&full[i], m * 16);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(smem_u32(ce_smem) + lo * 16), "l"(lg + lo * 8), "r"(m * 16), "r"(smem_u32(&full[i])) : "memory");
    }
  }
  const WaitGuard guard{&abort_word, status};
  const bf16* sl = reinterpret_cast<const bf16*>(ce_smem);
  float mx = -INFINITY;
  bool ok = true;
  for (int p = 0; p < kCePieces; ++p) {
    ok = ok && mbar_wait(&full[p], 0, guard, kTimeoutTmaFull);
    if (!ok) break;
    const int hi = min((p + 1) * step, n);
    for (int i = p * step + threadIdx.x; i < hi; i += kCeThreads) {
      float f[8];
      load8(sl + i * 8, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) mx = fmaxf(mx, f[j]);
    }
  }
  mx = block_max<kCeThreads>(mx, red);
  const float m_use = mx == -INFINITY ? 0.f : mx;    // a CTA without columns, or with masked ones only
  float sum = 0.f;
  if (ok)
    for (int i = threadIdx.x; i < n; i += kCeThreads) {
      float f[8];
      load8(sl + i * 8, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += __expf(f[j] - m_use);
    }
  __syncthreads();
  sum = block_sum<kCeThreads>(sum, red);
  if (threadIdx.x == 0) s_mine = make_float2(mx, sum);
  __syncthreads();
  if (ctas > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    float all = -INFINITY, total = 0.f;
    float2 part_of[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c >= ctas) break;
      part_of[c] = ce_ld_cluster(smem_u32(&s_mine), c);
      all = fmaxf(all, part_of[c].x);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c >= ctas) break;
      total += part_of[c].x == -INFINITY ? part_of[c].y : part_of[c].y * __expf(part_of[c].x - all);    // (0, or what is no number)
    }
    mx = all;
    sum = total;
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");       // this CTA has read the others' parts
  }
  if (ok) {
    const long long at = label - (long long)v0 * 8;
    if (threadIdx.x == 0 && at >= 0 && at < n * 8) row_loss[row] = mx + __logf(sum) - __bfloat162float(sl[at]);
    if (write_grad) {
      const float gs = *grad_scale;
      const float inv = 1.f / sum;
      for (int i = threadIdx.x; i < n; i += kCeThreads) {
        float f[8];
        load8(sl + i * 8, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float p = __expf(f[j] - mx) * inv;
          if ((long long)i * 8 + j == at) p -= 1.f;
          f[j] = p * gs;
        }
        store8(lg + i * 8, f);
      }
    }
  }
  __syncwarp();               // lanes leave the loop after different numbers of columns, and the barrier takes whole warps
  if (ctas > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");     // nobody leaves before it has been read
}

}  // namespace ksa

using namespace ksa;

KSA_API int ksa_cross_entropy(void* logits, const void* labels, void* row_loss, const void* grad_scale, long long rows,
                              int V, long long ld, int ignore_index, int write_grad, void* stream) {
  KSA_ENTER(logits);
  KSA_REQUIRE(V % 8 == 0 && ld % 8 == 0, "cross_entropy: V=%d and ld=%lld must be multiples of 8", V, ld);
  KSA_REQUIRE((reinterpret_cast<uintptr_t>(logits) & 15) == 0, "cross_entropy: the logits must be 16-byte aligned");
  if (rows == 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int ctas = 1;
  while (ctas < 8 && ((V / 8 + ctas - 1) / ctas) * 16 > kCeMostBytes) ctas *= 2;
  const int part = (V / 8 + ctas - 1) / ctas;
  if (V > 0 && part * 16 <= kCeMostBytes) {
    static PerDevice raised;
    KSA_CHECK_CUDA(raise_smem_limit(raised, cross_entropy_cluster_kernel, kCeMostBytes));
    int* status = status_word();
    KSA_REQUIRE(status != nullptr, "could not allocate the status word");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(rows * ctas));
    cfg.blockDim = dim3(kCeThreads);
    cfg.dynamicSmemBytes = (size_t)part * 16;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = dependent_launches() ? 2 : 1;
    KSA_CHECK_CUDA(cudaLaunchKernelEx(&cfg, cross_entropy_cluster_kernel, (bf16*)logits, (const long long*)labels, (float*)row_loss,
                                      (const float*)grad_scale, V, ld, ignore_index, write_grad, ctas, part, status));
    return 0;
  }
  KSA_CHECK_CUDA(launch_stream_kernel(6LL * rows * V, cross_entropy_kernel, dim3((unsigned)rows), dim3(kCeThreads), 0, st,
                                      (bf16*)logits, (const long long*)labels, (float*)row_loss, (const float*)grad_scale, V, ld,
                                      ignore_index, write_grad));
  return 0;
}
