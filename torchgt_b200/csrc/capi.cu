// Error reporting, version and layout validation shared by every entry point of the C ABI.
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "attn_common.cuh"

namespace tgt {

namespace {
thread_local char g_error[512] = "";
std::atomic<int> g_forced_ge{0};
std::atomic<int> g_lane_mode{0};
// Every link is chained.  The walks release their dependents when their edges are done, so what is launched early takes no slots
// from them.  Measured on B200, us with ordinary launches | links 1 and 4 | all: 64,000 nodes 8 x 8 fp32 forward 34.5 | 34.6 | 33.2,
// backward 98.1 | 96.8 | 94.5, with dbias 111.6 | 108.3 | 105.5; bf16 31.1 | 30.9 | 29.8 and 81.7 | 79.9 | 77.0; one head 17.3 | 17.4
// | 16.1 and 41.4 | 39.5 | 37.2; 4,096 nodes 8 x 8 fp32 9.8 | 10.0 | 9.2 and 24.8 | 23.9 | 21.6.
std::atomic<int> g_dependent_launch{kLinkWalk | kLinkStitch | kLinkAfterStitch};
}  // namespace

int lane_mode() { return g_lane_mode.load(std::memory_order_relaxed); }
int dependent_launch_mask() { return g_dependent_launch.load(std::memory_order_relaxed); }

int set_error(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
  return code;
}

int forced_ge() { return g_forced_ge.load(std::memory_order_relaxed); }

int current_device() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    set_error(TGT_ERR_UNSUPPORTED, "no current CUDA device with an ordinal below %d", kMaxDevices);
    return -1;
  }
  return dev;
}

int sm_count() {
  static std::atomic<int> cache[kMaxDevices] = {};
  const int dev = current_device();
  if (dev < 0) return 148;
  int n = cache[dev].load(std::memory_order_relaxed);
  if (n <= 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = 148;
    }
    cache[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

int expired_wait_word(int** word) {
  static std::atomic<int*> words{nullptr};     // of all devices, for good
  static std::mutex mutex;
  const int dev = current_device();
  if (dev < 0) return TGT_ERR_UNSUPPORTED;
  int* all = words.load(std::memory_order_acquire);
  if (all == nullptr) {
    const std::lock_guard<std::mutex> lock(mutex);
    all = words.load(std::memory_order_relaxed);
    if (all == nullptr) {
      // the allocation is not part of a graph that this thread may be capturing
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      TGT_CHECK_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
      const cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&all), kMaxDevices * sizeof(int), cudaHostAllocPortable);
      TGT_CHECK_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
      TGT_CHECK_CUDA(e);
      memset(all, 0, kMaxDevices * sizeof(int));
      words.store(all, std::memory_order_release);
    }
  }
  *word = all + dev;
  if (__atomic_load_n(*word, __ATOMIC_RELAXED) != 0 && __atomic_exchange_n(*word, 0, __ATOMIC_RELAXED) != 0)
    return set_error(TGT_ERR_CUDA, "a product launched before waited in vain for the tensor cores; its results are NaN");
  return TGT_OK;
}

int check_layout(const tgt_layout* L, const char* name) {
  if (L == nullptr) return set_error(TGT_ERR_INVALID, "%s is null", name);
  if (L->n_rows < 0 || L->n_edges < 0 || L->n_rows >= (int64_t(1) << 31) - 1 ||
      L->n_edges >= (int64_t(1) << 31) - 1)
    return set_error(TGT_ERR_INVALID, "%s: n_rows/n_edges out of range", name);
  if (L->n_edges > 0 && L->n_rows == 0)
    return set_error(TGT_ERR_INVALID, "%s: edges without rows", name);
  if (L->n_rows > 0 && L->ptr == nullptr) return set_error(TGT_ERR_INVALID, "%s: ptr is null", name);
  if (L->n_edges > 0 && (L->other == nullptr || L->perm == nullptr || L->seg == nullptr))
    return set_error(TGT_ERR_INVALID, "%s: other/perm/seg is null", name);
  return TGT_OK;
}

}  // namespace tgt

extern "C" int tgt_version(void) { return 101; }

extern "C" const char* tgt_last_error(void) { return tgt::g_error; }

extern "C" int tgt_products_status(void) {
  int* word = nullptr;
  return tgt::expired_wait_word(&word);
}

extern "C" int tgt_debug_set_tile_edges(int edges_per_lane_group) {
  TGT_CHECK_ARG(edges_per_lane_group >= 0, "edges_per_lane_group must be >= 0");
  tgt::g_forced_ge.store(edges_per_lane_group, std::memory_order_relaxed);
  return TGT_OK;
}

extern "C" int tgt_debug_set_lane_mode(int mode) {
  TGT_CHECK_ARG(mode >= 0 && mode <= 2, "mode must be 0 (library's choice), 1 (16-byte lanes) or 2 (32-byte lanes)");
  tgt::g_lane_mode.store(mode, std::memory_order_relaxed);
  return TGT_OK;
}

extern "C" int tgt_debug_set_dependent_launch(int links) {
  TGT_CHECK_ARG(links >= 0 && links <= 7, "links is a bit mask of 1, 2 and 4");
  tgt::g_dependent_launch.store(links, std::memory_order_relaxed);
  return TGT_OK;
}
