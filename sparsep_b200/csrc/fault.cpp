// fault.cpp -- device allocations and failure injection for tests.
//
// No counterpart in the reference, whose failures abort (DPU_ASSERT,
// spmv/1D/CSR-row/host/app.c:91-93).  Here every failure is a status, and
// these switches let tests make the two kinds of failure happen on purpose
// without faulting a GPU: a device allocation that fails (SPARSEP_ENOMEM) and
// a bounded device wait that runs out (SPARSEP_ETIMEDOUT).
#include <atomic>
#include <mutex>

#include "fault.hpp"
#include "sparsep.h"

namespace sparsep {

static std::atomic<long long> g_live{0};  // live device allocations
static std::atomic<int> g_fail_in{0};     // the g_fail_in-th allocation from now fails (0: none)
static std::atomic<int> g_wait_fault{0};

// The allocation that the tests asked to fail is this one.
static bool fails_now() {
  int n = g_fail_in.load();
  while (n > 0 && !g_fail_in.compare_exchange_weak(n, n - 1)) {
  }
  return n == 1;
}

// The current device's pool, made on first use; null where the device has none.
static std::mutex g_pool_mu;
static cudaMemPool_t g_pool[64];
static std::atomic<size_t> g_pool_used[64];  // bytes of the pool's memory in use
static cudaMemPool_t pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p = nullptr;
    uint64_t keep = POOL_KEEP;
    if (cudaMemPoolCreate(&p, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
      if (p) cudaMemPoolDestroy(p);
      cudaGetLastError();
      return nullptr;
    }
    g_pool[dev] = p;
  }
  return g_pool[dev];
}
// What the current device's pool keeps and nobody uses, back to the device.
static cudaError_t trim_pool() {
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  if (dev < 0 || dev >= 64) return cudaSuccess;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_pool[dev]) return cudaSuccess;
  // what is given back on a stream counts once the stream has come to that
  if (cudaError_t e = cudaDeviceSynchronize()) return e;
  return cudaMemPoolTrimTo(g_pool[dev], 0);
}

cudaError_t dev_malloc(void **p, size_t bytes) {
  *p = nullptr;
  if (fails_now()) return cudaErrorMemoryAllocation;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    trim_pool();
    e = cudaMalloc(p, bytes);
  }
  if (e == cudaSuccess) ++g_live;
  return e;
}

void dev_free(void *p) {
  if (!p) return;
  cudaFree(p);
  --g_live;
}

cudaError_t ws_malloc(Scratch *m, size_t bytes, cudaStream_t s) {
  *m = Scratch();
  if (fails_now()) return cudaErrorMemoryAllocation;
  cudaMemPool_t pl = pool();
  if (pl) {
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return e;
    if (g_pool_used[dev].fetch_add(bytes) + bytes <= POOL_KEEP) m->pool = dev;
    else g_pool_used[dev].fetch_sub(bytes);
  }
  auto get = [&] { return m->pool >= 0 ? cudaMallocFromPoolAsync(&m->p, bytes, pl, s) : cudaMalloc(&m->p, bytes); };
  cudaError_t e = get();
  if (e == cudaErrorMemoryAllocation) {
    trim_pool();
    e = get();
  }
  if (e == cudaSuccess) {
    m->bytes = bytes;
    ++g_live;
  } else {
    if (m->pool >= 0) g_pool_used[m->pool].fetch_sub(bytes);
    *m = Scratch();
  }
  cudaGetLastError();  // a failure is in e: no later launch is to report it
  return e;
}

void ws_free(Scratch *m, cudaStream_t s) {
  if (!m->p) return;
  if (m->pool >= 0) {
    cudaFreeAsync(m->p, s);
    g_pool_used[m->pool].fetch_sub(m->bytes);
  } else {
    cudaStreamSynchronize(s);  // the work that uses it
    cudaFree(m->p);
  }
  *m = Scratch();
  --g_live;
}

int wait_fault() { return g_wait_fault.load(); }

}  // namespace sparsep

extern "C" {

int sparsep_trim_scratch(void) { return sparsep::trim_pool() == cudaSuccess ? SPARSEP_OK : SPARSEP_EIO; }

int sparsep_test_fail_alloc(int nth) {
  if (nth < 0) return SPARSEP_EINVAL;
  sparsep::g_fail_in.store(nth);
  return SPARSEP_OK;
}

long long sparsep_test_live_allocations(void) { return sparsep::g_live.load(); }

int sparsep_test_wait_fault(int on) {
  sparsep::g_wait_fault.store(on ? 1 : 0);
  return SPARSEP_OK;
}

}  // extern "C"
