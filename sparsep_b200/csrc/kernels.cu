// kernels.cu -- host launchers of the sm_100a SpMV kernels (kernels_impl.cuh).
#include <atomic>

#include "kernels_impl.cuh"
#include "kernels.hpp"

namespace sparsep {

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
// Lets kernel k use `smem` bytes of dynamic shared memory.  The default limit
// is 48 KB minus the kernel's static shared memory; the largest size set so
// far is kept per device (host threads may plan concurrently, on different
// devices).
template <typename K>
static cudaError_t allow_smem(K *k, std::atomic<int> (&configured)[64], size_t smem) {
  if (smem == 0) return cudaSuccess;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::atomic<int> &c = configured[dev & 63];
  if ((int)smem <= c.load()) return cudaSuccess;
  e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int cur = c.load();
  while ((int)smem > cur && !c.compare_exchange_weak(cur, (int)smem)) {
  }
  return cudaSuccess;
}

template <typename T, int FMT, int RB, int CB, int CAP = 0>
static cudaError_t launch_t(const Params<T> &P, uint32_t carry_w, int threads, size_t smem, cudaStream_t st) {
  static std::atomic<int> configured[64];
  if (cudaError_t e = allow_smem(spmv_items<T, FMT, RB, CB, CAP>, configured, smem)) return e;
  spmv_items<T, FMT, RB, CB, CAP><<<P.nitems, threads, smem, st>>>(P, carry_w);
  return cudaGetLastError();
}

// BCSR blocks: the chunk kernel where it takes the block size and type.
template <typename T, int RB, int CB>
static cudaError_t launch_bcsr(const Params<T> &P, int threads, size_t smem, cudaStream_t st) {
  if constexpr (bcsr_chunk_blocks(RB, CB, sizeof(T)) == 0) {
    return launch_t<T, SPARSEP_FMT_BCSR, RB, CB>(P, 1, threads, smem, st);
  } else {
    static std::atomic<int> configured[64];
    smem = (smem + 127) / 128 * 128 + BlockStage<T, RB, CB>::SMEM;  // a tile's staged x first
    if (cudaError_t e = allow_smem(bcsr_chunks<T, RB, CB>, configured, smem)) return e;
    bcsr_chunks<T, RB, CB><<<P.nitems, threads, smem, st>>>(P);
    return cudaGetLastError();
  }
}

template <typename T, int RB, int CB>
static cudaError_t launch_bcoo(const Params<T> &P, int threads, size_t smem, cudaStream_t st) {
  static std::atomic<int> configured[64];
  smem = (smem + 127) / 128 * 128 + BcooStage<T, RB, CB>::SMEM;
  if (cudaError_t e = allow_smem(bcoo_chunks<T, RB, CB>, configured, smem)) return e;
  bcoo_chunks<T, RB, CB><<<P.nitems, threads, smem, st>>>(P);
  return cudaGetLastError();
}
template <typename T, bool ATOMIC>
static cudaError_t launch_coo(const Params<T> &P, int threads, size_t smem, cudaStream_t st) {
  static std::atomic<int> configured[64];
  if (cudaError_t e = allow_smem(coo_items<T, ATOMIC>, configured, smem)) return e;
  coo_items<T, ATOMIC><<<P.nitems, threads, smem, st>>>(P);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_items(const Params<T> &P, int fmt, uint32_t carry_w, int threads, size_t smem, bool slim,
                         cudaStream_t st) {
  if (P.nitems == 0) return cudaSuccess;
  const uint32_t rb = P.rb, cb = P.cb;
  switch (fmt) {
    case SPARSEP_FMT_CSR:
      if (slim) return launch_t<T, SPARSEP_FMT_CSR, 0, 0, csr_chunk_nnz(sizeof(T), true)>(P, carry_w, threads, smem, st);
      // 16 warps take 2048 nonzeros per pass: 8-byte types in 32 KB then (FP64, 16 warps,
      // 400,000 rows of 12, power-law: 52 us in 16 KB, 42)
      return threads > 256
                 ? launch_t<T, SPARSEP_FMT_CSR, 0, 0, 4096>(P, carry_w, threads, smem, st)
                 : launch_t<T, SPARSEP_FMT_CSR, 0, 0, csr_chunk_nnz(sizeof(T), false)>(P, carry_w, threads, smem, st);
    case SPARSEP_FMT_COO:
      return P.out_mode == OUT_ATOMIC ? launch_coo<T, true>(P, threads, smem, st)
                                      : launch_coo<T, false>(P, threads, smem, st);
    case SPARSEP_FMT_BCSR:
      if (rb == 4 && cb == 4) return launch_bcsr<T, 4, 4>(P, threads, smem, st);
      if (rb == 8 && cb == 8) return launch_bcsr<T, 8, 8>(P, threads, smem, st);
      if (rb == 2 && cb == 2) return launch_bcsr<T, 2, 2>(P, threads, smem, st);
      return launch_t<T, SPARSEP_FMT_BCSR, 0, 0>(P, carry_w, threads, smem, st);
    case SPARSEP_FMT_BCOO:
      if (rb == 4 && cb == 4) return launch_bcoo<T, 4, 4>(P, threads, smem, st);
      if (rb == 8 && cb == 8) return launch_bcoo<T, 8, 8>(P, threads, smem, st);
      if (rb == 2 && cb == 2) return launch_bcoo<T, 2, 2>(P, threads, smem, st);
      return launch_t<T, SPARSEP_FMT_BCOO, 0, 0>(P, carry_w, threads, smem, st);
  }
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_merge(const T *part, T *y, uint32_t nrows, uint32_t V, int sms, cudaStream_t st) {
  if (nrows == 0) return cudaSuccess;
  uint32_t blocks = (nrows + 255) / 256;
  uint32_t cap = (uint32_t)sms * 8;
  if (blocks > cap) blocks = cap;
  merge_partials<T><<<blocks, 256, 0, st>>>(part, y, nrows, V);
  return cudaGetLastError();
}

// The build compiles this file once per element type (-DSPARSEP_KT=<type>) so
// the instantiations build in parallel.
#ifndef SPARSEP_KT
#define SPARSEP_KT float
#endif
template cudaError_t launch_items<SPARSEP_KT>(const Params<SPARSEP_KT> &, int, uint32_t, int, size_t, bool, cudaStream_t);
template cudaError_t launch_merge<SPARSEP_KT>(const SPARSEP_KT *, SPARSEP_KT *, uint32_t, uint32_t, int, cudaStream_t);

}  // namespace sparsep
