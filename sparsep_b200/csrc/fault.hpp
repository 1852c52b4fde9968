// fault.hpp -- device allocations of the library and the test-support fault
// switches (fault.cpp).
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace sparsep {

// Every device allocation of the library goes through dev_malloc / dev_free:
// test support can make the n-th allocation fail (as cudaMalloc does when the
// device is full), and the count of live allocations shows leaks.
cudaError_t dev_malloc(void **p, size_t bytes);
void dev_free(void *p);

// Scratch memory that a call takes and gives back, ordered on its stream: from a
// pool of the library's own per device, which keeps up to POOL_KEEP bytes between
// calls (a quarter gigabyte from cudaMalloc and back costs a call milliseconds and
// two device-wide synchronisations) until sparsep_trim_scratch or an allocation of the
// library's own that finds the device full.  What does not fit into POOL_KEEP bytes
// with the scratch in use comes from cudaMalloc and goes back: a pool that maps and
// unmaps memory in every call is slower than that (COO -> CSR of 60 M nonzeros, FP32:
// 16.4 ms from the pool, 3.6 from cudaMalloc; inside POOL_KEEP, 15 M nonzeros: 0.5
// against 2.5 ms).  Counted and failed on request like dev_malloc.
constexpr size_t POOL_KEEP = (size_t)512 << 20;
struct Scratch {
  void *p = nullptr;
  size_t bytes = 0;
  int pool = -1;  // the device whose pool it is from, -1: cudaMalloc
};
cudaError_t ws_malloc(Scratch *m, size_t bytes, cudaStream_t s);
void ws_free(Scratch *m, cudaStream_t s);  // nothing where m holds none

// Nonzero while test support asks the kernels with bounded staging waits to
// add one wait that nothing completes (after their own copies have landed).
int wait_fault();

}  // namespace sparsep
