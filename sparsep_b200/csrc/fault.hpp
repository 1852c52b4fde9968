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
// library's own that finds the device full.  POOL_KEEP holds what converting some 30 M
// nonzeros takes; scratch beyond it goes back to the device after every call, as all
// of it did from cudaMalloc.  Counted and failed on request like dev_malloc.
constexpr size_t POOL_KEEP = (size_t)512 << 20;
cudaError_t ws_malloc(void **p, size_t bytes, cudaStream_t s);
void ws_free(void *p, cudaStream_t s);

// Nonzero while test support asks the kernels with bounded staging waits to
// add one wait that nothing completes (after their own copies have landed).
int wait_fault();

}  // namespace sparsep
