// Host-side runtime of the kernel library: last-error string, TMA descriptor
// encoding, the device status word written by bounded waits.
#include "host.h"

#include <mutex>
#include <stdarg.h>
#include <stdlib.h>
#include <string.h>

namespace ksa {

static thread_local char g_last_error[512] = "";

void set_last_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
}

EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
    }
  });
  return fn;
}

int make_tmap(CUtensorMap* out, const void* base, int elem_bytes, int rank, const uint64_t* dims,
              const uint64_t* strides_bytes, const uint32_t* box, bool swizzle128) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) {
    set_last_error("cuTensorMapEncodeTiled is not available from the driver");
    return kErrNoDriver;
  }
  cuuint64_t gdim[5];
  cuuint64_t gstr[4];
  cuuint32_t bdim[5];
  cuuint32_t estr[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bdim[i] = box[i];
    estr[i] = 1;
    if (i > 0) gstr[i - 1] = strides_bytes[i];
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) {
    set_last_error("TMA base address %p is not 16-byte aligned", base);
    return kErrArgument;
  }
  for (int i = 1; i < rank; ++i) {
    if (strides_bytes[i] % 16 != 0) {
      set_last_error("TMA stride %d = %llu bytes is not a multiple of 16", i, (unsigned long long)strides_bytes[i]);
      return kErrArgument;
    }
  }
  CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = enc(out, dt, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstr, bdim, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("cuTensorMapEncodeTiled failed with CUresult %d (rank %d, dims %llu x %llu, box %u x %u)", (int)r,
                   rank, (unsigned long long)dims[0], (unsigned long long)(rank > 1 ? dims[1] : 0), box[0],
                   rank > 1 ? box[1] : 0);
    return kErrCuda;
  }
  return kErrNone;
}

int ensure_device(const void* device_ptr) {
  static thread_local int bound_device = -1;
  if (bound_device >= 0 || device_ptr == nullptr) return kErrNone;
  cudaPointerAttributes attr;
  cudaError_t e = cudaPointerGetAttributes(&attr, device_ptr);
  if (e != cudaSuccess || (attr.type != cudaMemoryTypeDevice && attr.type != cudaMemoryTypeManaged)) {
    cudaGetLastError();
    set_last_error("pointer %p is not device memory (%s)", device_ptr, e == cudaSuccess ? "host pointer" : cudaGetErrorString(e));
    return kErrArgument;
  }
  e = cudaSetDevice(attr.device);
  if (e != cudaSuccess) {
    set_last_error("cudaSetDevice(%d) failed: %s", attr.device, cudaGetErrorString(e));
    return kErrCuda;
  }
  cudaFree(0);  // force the primary context to be current on this thread
  bound_device = attr.device;
  return kErrNone;
}

int sm_count() {
  static std::atomic<int> counts[64];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (dev < 64 && (n = counts[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (dev < 64) counts[dev].store(n, std::memory_order_relaxed);
  return n;
}

constexpr long long kDefaultPeerWaitMs = 10000;   // 10 s
static int* g_status[64] = {nullptr};
static std::mutex g_status_mu;

int* status_word() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(g_status_mu);
  if (!g_status[dev]) {
    int* p = nullptr;
    // the first kernel of a process may be launched into a capture: the word is then set up beside it, on a stream of its own
    struct Relaxed {
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      cudaStream_t st = nullptr;
      Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
      ~Relaxed() {
        if (st) cudaStreamDestroy(st);
        cudaThreadExchangeStreamCaptureMode(&mode);
      }
    } relaxed;
    if (cudaMalloc(&p, 256) != cudaSuccess) return nullptr;
    if (cudaStreamCreateWithFlags(&relaxed.st, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    // word 1: limit of waits on flags written by OTHER GPUs, in units of 2^20 clock cycles (0 = the built-in limit).
    // Ranks drift apart on the host (graph capture, a slow data loader), so this limit is longer than the one of the
    // waits inside a kernel; KSA_PEER_WAIT_MS overrides it, ksa_set_peer_wait_ms changes it at run time.
    int units = (int)(kDefaultPeerWaitMs * 2000LL / 1049);      // ~2 GHz: 2e6 cycles per ms
    if (const char* e = getenv("KSA_PEER_WAIT_MS")) {
      const long long ms = atoll(e);
      if (ms > 0) units = (int)(ms * 2000LL / 1049 + 1);
    }
    int words[64] = {0, units};
    if (cudaMemcpyAsync(p, words, sizeof(words), cudaMemcpyHostToDevice, relaxed.st) != cudaSuccess ||
        cudaStreamSynchronize(relaxed.st) != cudaSuccess)
      return nullptr;
    g_status[dev] = p;
  }
  return g_status[dev];
}

}  // namespace ksa

KSA_API const char* ksa_last_error() { return ksa::g_last_error; }

// Address of the status word of the current device (for torch to wrap / read).
KSA_API void* ksa_status_ptr() { return ksa::status_word(); }

// Read and clear the status word (synchronises the device).  Returns the status, or -1 on a CUDA error.
KSA_API int ksa_read_status(int clear) {
  int* p = ksa::status_word();
  if (!p) return -1;
  int v = 0;
  if (cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (clear && v != 0) cudaMemset(p, 0, sizeof(int));
  return v;
}

// Limit (milliseconds at ~2 GHz) of device-side waits on flags written by other GPUs, for the current device.
KSA_API int ksa_set_peer_wait_ms(int ms) {
  int* p = ksa::status_word();
  if (!p || ms <= 0) return -1;
  const int units = (int)((long long)ms * 2000LL / 1049 + 1);
  return cudaMemcpy(p + 1, &units, sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -1;
}

namespace ksa {
// How the calling thread launches (host.h).  Of the thread alone: a product that another thread issues meanwhile must not read its
// weights early, and two threads that each save and restore the setting would leave it on.
static int first_launch_mode() {
  static const int mode = [] {
    const char* e = getenv("KSA_DEPENDENT_LAUNCH");
    return e != nullptr && strcmp(e, "0") == 0 ? kLaunchOrdinary : kLaunchDependent;
  }();
  return mode;
}
static thread_local int t_launch_mode = first_launch_mode();
int launch_mode() { return t_launch_mode; }
static thread_local bool t_beside = false;
bool launch_beside() { return t_beside && t_launch_mode == kLaunchDependent; }
}  // namespace ksa

// Sets the calling thread's launch mode (below zero: ordinary, 0: dependent, above: dependent with early weights) and returns the
// one it had.
KSA_API int ksa_set_dependent_launch(int mode) {
  const int before = ksa::t_launch_mode;
  ksa::t_launch_mode = mode < 0 ? ksa::kLaunchOrdinary : mode > 0 ? ksa::kLaunchEarlyWeights : ksa::kLaunchDependent;
  return before;
}

// Whether the calling thread's launches may run beside the kernel before them (host.h: launch_beside); returns the setting before.
KSA_API int ksa_set_launch_beside(int on) {
  const int before = ksa::t_beside;
  ksa::t_beside = on != 0;
  return before;
}

KSA_API int ksa_abi_version() { return 1; }
