// common.cu -- error state, scratch allocation, version.
#include <cstdarg>
#include <cstring>
#include <mutex>
#include "common.cuh"

namespace cageo {

static thread_local char g_last_error[512] = "no error";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
}

cageo_status cuda_fail(cudaError_t e, const char* what) {
  set_error("CUDA error %d (%s) in %s", (int)e, cudaGetErrorString(e), what);
  return CAGEO_ERR_CUDA;
}

// Scratch of stage calls without a workspace comes from a pool of the library's
// own, one per device, that keeps up to kPoolKeeps bytes between calls.  (The
// device's default pool, whose setting is the program's, gives everything back
// at each synchronization: a stage call then mapped and unmapped its
// scratch, ~170 us of a stream burning's 220.)  The driver orders its reuse on
// streams and threads.
constexpr unsigned long long kPoolKeeps = 256ull << 20;

static std::mutex g_pool_mutex;
static cudaMemPool_t g_pools[kMaxDevices];
static bool g_pool_tried[kMaxDevices];

static cudaMemPool_t scratch_pool(bool make) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (!g_pool_tried[dev] && make) {
    g_pool_tried[dev] = true;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    unsigned long long keeps = kPoolKeeps;
    if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
      if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keeps) == cudaSuccess)
        g_pools[dev] = pool;
      else
        cudaMemPoolDestroy(pool);
    }
    cudaGetLastError();
  }
  return g_pools[dev];
}

void scratch_trim() {
  if (cudaMemPool_t pool = scratch_pool(false)) cudaMemPoolTrimTo(pool, 0);
  cudaGetLastError();
}

cageo_status Scratch::acquire(void* given, size_t given_bytes, size_t need,
                              cudaStream_t s) {
  stream = s;
  if (given) {
    if (given_bytes < need) {
      set_error("workspace of %zu bytes is smaller than the %zu bytes needed",
                given_bytes, need);
      return CAGEO_ERR_ARGUMENT;
    }
    if ((uintptr_t)given % 256 != 0) {
      set_error("workspace must start on a 256-byte boundary (as cudaMalloc returns)");
      return CAGEO_ERR_ARGUMENT;
    }
    ptr = given;
    owned = false;
    return CAGEO_OK;
  }
  // (While a stream is captured: the default pool, whose allocations become
  // nodes of the graph.)
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(s, &capture);
  cudaMemPool_t pool =
      e == cudaSuccess && capture == cudaStreamCaptureStatusNone ? scratch_pool(true) : nullptr;
  if (pool) {
    e = cudaMallocFromPoolAsync(&ptr, need ? need : 16, pool, s);
    if (e == cudaSuccess) {
      owned = true;
      return CAGEO_OK;
    }
    cudaGetLastError();
    scratch_trim();
  }
  e = cudaMallocAsync(&ptr, need ? need : 16, s);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync(workspace)");
  owned = true;
  return CAGEO_OK;
}

Scratch::~Scratch() {
  if (owned && ptr) cudaFreeAsync(ptr, stream);
}

}  // namespace cageo

extern "C" const char* cageo_version(void) { return "cageo-gb300 0.1 (sm_103a)"; }

extern "C" const char* cageo_last_error_string(void) {
  return cageo::g_last_error;
}
