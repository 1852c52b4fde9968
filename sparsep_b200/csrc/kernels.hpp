// kernels.hpp -- host-side declarations of the kernel launchers (kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"

namespace sparsep {

// Launch the work-item kernel for format `fmt` (sparsep_format) with one CTA
// per item.  carry_w = carry slots per item (1 for CSR/COO, rb for BCOO); slim:
// CSR items of at most csr_chunk_nnz(.., true) nonzeros.
template <typename T>
cudaError_t launch_items(const Params<T> &P, int fmt, uint32_t carry_w, int threads, size_t smem, bool slim,
                         cudaStream_t st);

// y[r] = sum over the V partial slices of row r, in slice order.
template <typename T>
cudaError_t launch_merge(const T *part, T *y, uint32_t nrows, uint32_t V, int sms, cudaStream_t st);

// Blocks per chunk (32 KB of values) of the BCSR kernel bcsr_chunks for rb x cb
// blocks of es-byte elements, 0 for those that spmv_items runs: other block
// sizes, and 2x2 blocks of 8-byte types, whose 64-byte groups of lanes meet in
// the same shared-memory banks (FP64, 1M rows, 12 blocks per block row: 73 us
// in chunks, 62 us there).
constexpr uint32_t bcsr_chunk_blocks(uint32_t rb, uint32_t cb, size_t es) {
  return rb == cb && ((rb == 2 && es < 8) || rb == 4 || rb == 8)
             ? (uint32_t)(32768 / (rb * cb * es) < 2048 ? 32768 / (rb * cb * es) : 2048)
             : 0;
}
// block rows per chunk
constexpr uint32_t BCSR_CHUNK_ROWS = 512;

// Nonzeros whose products the CSR row kernel holds in shared memory at a time (and
// a quarter as many rows): 8 KB of them in the slim form, 16 KB in the wide one.
// A gather of x holds a line of L1 while it is under way, and shared memory is
// taken from L1: with 32 KB of FP64 products per CTA the gathers stood in line
// (1M-row power-law matrix, FP64 188 us; 16 KB 107 us; 8 KB and 4 warps per CTA 93
// us; FP32 with 16 KB 87 us, 8 KB and 4 warps 83.5 us).  Automatic items, parts and
// tiles are slim; wide are those of a given size (item_nnz), of tiles whose x is staged,
// and where the planner finds that better (wide_items in plan.cu: more than 8 warps, most
// nonzeros in long rows).
constexpr int csr_chunk_nnz(size_t es, bool slim) { return (slim ? 8192 : 16384) / (es == 8 ? 8 : 4); }

// Nonzeros per automatic COO item: 4096, fewer where that leaves less than six
// items per SM of a B200's 148 (1.5 M nonzeros, FP32: 20 us in 366 items, 16.5 us in 733; 16.7 M:
// 94 us in items of 2048, 91 us of 4096).
constexpr uint32_t coo_item_elems(uint64_t nnz) {
  return nnz >= 4096 * 888ull ? 4096 : nnz <= 512 * 888ull ? 512 : (uint32_t)((nnz / 888 + 3) & ~3ull);
}
// Blocks per BCOO chunk (bcoo_chunks, 32 KB of values at most), 0 for the block
// sizes that spmv_items runs.
constexpr uint32_t bcoo_chunk_blocks(uint32_t rb, uint32_t cb, size_t es) {
  return rb == cb && (rb == 2 || rb == 4 || rb == 8)
             ? (uint32_t)(32768 / (rb * cb * es) < 1024 ? 32768 / (rb * cb * es) : 1024)
             : 0;
}

// Persistent TMA-pipelined CSR kernel (csr_pipe.cu) for 1D items built by the
// automatic planner; grid = SMs x resident CTAs (capped at the item count).
template <typename T>
cudaError_t launch_csr_pipe(const Params<T> &P, int sms, cudaStream_t st, int *grid_out, uint32_t max_item_nnz);

// Split CSR plans (csr_stripes.cu).  stripe_geometry gives, for element type
// T, the stripe width (columns), the kernel's dynamic shared memory, the
// nonzeros of a heavy and of a light chunk and the rows of a chunk;
// launch_stripes runs `ctas` persistent CTAs over their chunk lists;
// launch_heavy_merge writes y[hrow[k]] = sum over stripes of the partials.
template <typename T>
void stripe_geometry(uint32_t *width, size_t *smem, uint32_t *chunk_nnz, uint32_t *light_nnz, uint32_t *chunk_rows);
template <typename T>
cudaError_t launch_stripes(const StripeParams<T> &P, uint32_t ctas, cudaStream_t st);
template <typename T>
cudaError_t launch_heavy_merge(const T *part, const uint32_t *hrow, uint32_t nH, uint32_t nS, T *y, int sms,
                               cudaStream_t st);

}  // namespace sparsep
