// Host-side helpers shared by the launchers: TMA descriptor encoding through the
// driver entry point (no link-time dependency on libcuda), error reporting, and
// the per-device status word that bounded waits write to.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <stdint.h>
#include <stdio.h>

#define KSA_API extern "C" __attribute__((visibility("default")))

namespace ksa {

// Error codes returned by the C entry points (0 = success).
enum HostError : int {
  kErrNone = 0,
  kErrCuda = -1,       // a CUDA runtime/driver call failed; see ksa_last_error()
  kErrArgument = -2,   // unsupported shape / alignment / size
  kErrNoDriver = -3,   // cuTensorMapEncodeTiled could not be resolved
};

void set_last_error(const char* fmt, ...);

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_tiled();

// Encode a bf16 (elem_bytes = 2) or fp32 (4) tiled tensor map with a 128-byte swizzle.
// dims / strides are innermost-first; strides[0] is implied (element size) and strides[i>0] are bytes.
int make_tmap(CUtensorMap* out, const void* base, int elem_bytes, int rank, const uint64_t* dims,
              const uint64_t* strides_bytes, const uint32_t* box, bool swizzle128);

// Device status word for the current device (allocated once per device on first use).
int* status_word();

// SMs of the current device, or 0.
int sm_count();

// What has been done once on every device (a process may use several, from several threads).
struct PerDevice {
  std::atomic<uint64_t> done{0};
};
// The limit of a kernel's dynamic shared memory belongs to the kernel on one device.
template <typename Kern>
inline cudaError_t raise_smem_limit(PerDevice& raised, Kern kern, size_t bytes) {
  int dev = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (raised.done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) raised.done.fetch_or(bit, std::memory_order_release);
  return e;
}

// Make the device that owns `device_ptr` current on the calling thread.  Callers may arrive on threads that have
// never touched CUDA through this library's runtime (autograd worker threads): without this, descriptor encoding
// fails for lack of a context and launches would go to device 0.  Cached per thread; returns 0 on success.
int ensure_device(const void* device_ptr);

#define KSA_ENTER(ptr)                                   \
  do {                                                   \
    int _rc = ksa::ensure_device(ptr);                   \
    if (_rc) return _rc;                                 \
  } while (0)

#define KSA_CHECK_CUDA(expr)                                                              \
  do {                                                                                    \
    cudaError_t _e = (expr);                                                              \
    if (_e != cudaSuccess) {                                                              \
      ksa::set_last_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, __LINE__); \
      return ksa::kErrCuda;                                                               \
    }                                                                                     \
  } while (0)

// Dependent launches (programmatic stream serialization).  Most kernels are launched so that each may start while its predecessor on the
// stream still runs, and wait for it on the device before they touch memory (grid_dependency_enter): the launch and the set-up of
// one kernel lie under the end of the one before.  Kernels that write weights (the optimizer) are launched the ordinary way.
// A thread launches in one of three modes (ksa_set_dependent_launch): as described, or with early weights (the inference engine's
// decode step), in which the weight-streaming products also read their weights before they wait, since no kernel of such a chain
// writes weights, or the ordinary way (KSA_DEPENDENT_LAUNCH=0).
enum LaunchMode : int { kLaunchOrdinary = -1, kLaunchDependent = 0, kLaunchEarlyWeights = 1 };
int launch_mode();
inline bool dependent_launches() { return launch_mode() != kLaunchOrdinary; }
inline bool weights_early() { return launch_mode() == kLaunchEarlyWeights; }

// Clusters whose blocks hold tensor memory: a block that finds none left on its SM waits without a limit, while the rest of its cluster waits
// for it.  Two clusters from two streams could so wait for one another's blocks, for good, unless no two blocks of theirs
// that might want more tensor memory than there is find room in an SM's shared memory.  So every such block takes at least kTmemClusterLeast
// (the least is split-K, csrc/gemm_narrow.cu: tiles of 96 rows), which leaves room for two, and one that takes more than half of the
// tensor memory also takes kTmemClusterAlone, which leaves none for another.
constexpr int kSmSharedBytes = 228 * 1024;           // of which every block costs 1024 besides its own
constexpr int kTmemClusterLeast = 85 * 1024;
constexpr int kTmemClusterAlone = kSmSharedBytes - kTmemClusterLeast;
static_assert(3 * (kTmemClusterLeast + 1024) > kSmSharedBytes && kTmemClusterLeast + kTmemClusterAlone + 2 * 1024 > kSmSharedBytes,
              "two blocks of half the tensor memory each, or one alone");

// Two kernels of one call that do not depend on one another (text rows and summary rows: other inputs' rows, other outputs) need not
// run one after the other.  After ksa_set_launch_beside(1), products and summary attention are launched to start as soon as every block of the
// kernel before them has begun its work, and wait for its end only before their own.  That is sound because a kernel begins its
// work when its own predecessors have ended (grid_dependency_enter), so what the second kernel reads and overwrites has to be
// finished before the FIRST one begins, and the first one has to be such a kernel: not one that lets successors start before it waits
// (the weight-streaming products) or lets none start.  What may come between the two from another thread is no exception: it, too, starts
// after the first has begun, and ends after it.  No effect with early weights, whose chains hold such products.
// PTX promises less than this rests on: a grid sees its prerequisites' writes through its own griddepcontrol.wait, and the second kernel
// has not executed one when it reads.  Two things are assumed: blocks of the second kernel start only after every block of the first has
// executed launch_dependents or ended (PTX says that it is what lets them be scheduled, not that it orders memory), and what the
// first kernel's wait has made visible to it is by then complete in the L2, where all SMs meet.  A block of the second kernel therefore
// reads nothing ahead of grid_dependency_observe(), which keeps its loads from lines that its SM may have held from before.
// A layer on 333 tokens 158.7 -> 142.9 us (the projection and the attention of two summary rows lie under those of the text rows), a
// training layer on 2 x 700 632 -> 615, on 8192 2840 -> 2800, attention over 32768 tokens 811 -> 794.
bool launch_beside();
template <typename Kern, typename... Args>
inline cudaError_t launch_kernel_if(bool dependent, Kern kern, dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent && dependent_launches() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}
// Kernels that bring their data in by TMA, and short ones.
template <typename Kern, typename... Args>
inline cudaError_t launch_kernel(Kern kern, dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  return launch_kernel_if(true, kern, grid, block, smem, st, args...);
}
// Kernels that stream `bytes` through registers: dependent only while the start weighs more than the streaming.  A kernel that starts
// beside a GEMM runs with the little L1 that the GEMM's shared memory leaves, and with it fewer loads in flight: with every launch
// dependent the output head over 4096 tokens took 7.14 ms instead of 6.91 (two cross entropies over 0.6 GB each), a training layer on
// 8192 tokens 2.98 ms instead of 2.93, summary attention on 32768 tokens 931 us instead of 912.  What the short ones gain: a layer on
// 333 tokens 185 -> 164 us, a feed-forward block of 48 rows 51 -> 43, a training layer on 1400 tokens 666 -> 646.
constexpr long long kStreamedDependent = 32LL << 20;
template <typename Kern, typename... Args>
inline cudaError_t launch_stream_kernel(long long bytes, Kern kern, dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  return launch_kernel_if(bytes <= kStreamedDependent, kern, grid, block, smem, st, args...);
}

// Whether the single-CTA kernel (csrc/gemm.cu) takes tiles of 128 x 256 for an M x N product, or of 128 x 128.
inline bool gemm_wide_tiles(int M, int N) {
  return N >= 256 && ((long long)((M + 127) / 128) * ((N + 255) / 256) >= 96 || N % 256 == 0);
}
// Modelled time in us of a row-major product on the split-K kernel or the single-CTA kernel, whichever is the faster (csrc/gemm_narrow.cu).
double few_rows_time(int M, int N, int K);

#define KSA_REQUIRE(cond, ...)                  \
  do {                                          \
    if (!(cond)) {                              \
      ksa::set_last_error(__VA_ARGS__);         \
      return ksa::kErrArgument;                 \
    }                                           \
  } while (0)

}  // namespace ksa
