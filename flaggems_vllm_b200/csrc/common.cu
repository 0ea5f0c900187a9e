// Host-side error bookkeeping of the C ABI.
#include <cstdarg>
#include <cstdio>

#include <atomic>
#include <mutex>
#include <set>
#include <utility>

#include "moe_common.cuh"

namespace moe {

int allow_smem(const void* kernel, int bytes, bool large_cluster) {
  int dev = 0;
  cudaGetDevice(&dev);
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;  // one entry per kernel and device
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({kernel, dev})) return 0;
  const cudaError_t ce = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (ce != cudaSuccess) return fail((int)ce, "shared memory attribute (%d bytes): %s", bytes, cudaGetErrorString(ce));
  if (large_cluster) {
    const cudaError_t cl = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (cl != cudaSuccess) return fail((int)cl, "cluster size attribute: %s", cudaGetErrorString(cl));
  }
  done.insert({kernel, dev});
  return 0;
}

int max_clusters(const void* kernel, int ctas, int threads, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess) return n;
  cudaGetLastError();
  return -1;
}

int sm_count() {
  static std::atomic<int> cached[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}
static thread_local char g_err[512] = "";
static unsigned long long g_wait_limit_ns = 2000000000ull;
unsigned long long wait_limit_ns() { return g_wait_limit_ns; }

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

static std::atomic<unsigned long long> g_launches{0};

int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    snprintf(g_err, sizeof(g_err), "%s: %s", what, cudaGetErrorString(e));
    return (int)e;
  }
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return 0;
}
}  // namespace moe

extern "C" int moe_abi_version(void) { return 1; }
extern "C" unsigned long long moe_set_wait_limit_ns(unsigned long long ns) {
  const unsigned long long old = moe::g_wait_limit_ns;
  if (ns != 0) moe::g_wait_limit_ns = ns;
  return old;
}
extern "C" unsigned long long moe_launch_count(void) { return moe::g_launches.load(std::memory_order_relaxed); }
extern "C" const char* moe_last_error(void) { return moe::g_err; }
