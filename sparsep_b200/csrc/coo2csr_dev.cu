// coo2csr_dev.cu -- COO -> CSR on the device, with the arrays the host
// converter coo2csr (formats.cpp; the reference's counting sort,
// spmv/1D/CSR-row/support/matrix.h:113-152) produces: rows in order, and
// inside a row the input order kept (a stable sort by row).
//
// Stable LSD radix sort (radix.cuh) of (row, column, value) records, only as many
// passes as the row count needs (20 bits -> 3 passes for 1M rows); the last pass
// writes the columns and values where they belong, so nothing is gathered
// afterwards.  Then rowptr[r] = first sorted position with row >= r (a binary
// search per row).
//
// Scratch: the outputs hold the columns and values of every second pass, so that one
// more set of them and two of keys do: 12 bytes per nonzero and a value (4 bytes with
// one pass).  Where the device has no room for that, values of 8 bytes, for which it is
// more than the 16 bytes of a sort of indices, are sorted by their indices, which lie
// in the outputs until a gather replaces them: 8 bytes per nonzero.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <initializer_list>
#include <new>

#include "fault.hpp"
#include "internal.hpp"
#include "radix.cuh"
#include "sparsep.h"

namespace sparsep {
namespace c2c {

// rowptr[r] = number of sorted rows < r (lower bound), r = 0 .. nrows
__global__ void rowptr_kernel(const uint32_t *__restrict__ key, uint32_t n, uint32_t nrows,
                              uint32_t *__restrict__ rowptr) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r > nrows) return;
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (key[mid] < r) lo = mid + 1;
    else hi = mid;
  }
  rowptr[r] = lo;
}

// colind holds the nonzeros' indices in order: their columns and values instead
template <typename V>
__global__ void gather(uint32_t n, const uint32_t *__restrict__ cols, const V *__restrict__ vals, uint32_t *colind,
                       V *__restrict__ vals_out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t k = colind[i];
    colind[i] = cols[k];
    vals_out[i] = vals[k];
  }
}

}  // namespace c2c
}  // namespace sparsep

using namespace sparsep::c2c;

template <size_t N> struct UintOf;
template <> struct UintOf<1> { using type = uint8_t; };
template <> struct UintOf<2> { using type = uint16_t; };
template <> struct UintOf<4> { using type = uint32_t; };
template <> struct UintOf<8> { using type = unsigned long long; };

static int c2c_err(cudaError_t e) {
  if (e == cudaSuccess) return SPARSEP_OK;
  char msg[160];
  std::snprintf(msg, sizeof msg, "%s (%d)", cudaGetErrorString(e), (int)e);
  sparsep::record_error(msg);
  return e == cudaErrorMemoryAllocation ? SPARSEP_ENOMEM : SPARSEP_EIO;
}

// Device COO (rows, cols, vals) -> device CSR, V an unsigned type of the values' size.
template <typename V>
static int coo2csr_device(const uint32_t *rows, const uint32_t *cols, const V *vals, uint32_t nnz, uint32_t nrows,
                          uint32_t *rowptr, uint32_t *colind, V *vals_out, cudaStream_t s) {
  using namespace sparsep::radix;
  if (!rowptr || nrows == 0xFFFFFFFFu || (nnz && (!rows || !cols || !vals || !colind || !vals_out)))
    return SPARSEP_EINVAL;
  int bits = 0;
  while (bits < 32 && (nrows - 1) >> bits) ++bits;  // bits of the largest row index
  if (nrows <= 1) bits = 0;
  const int np = passes(bits);
  const size_t n = nnz, vb = ((n * sizeof(V)) + 15) & ~(size_t)15, kb = ((n * 4) + 15) & ~(size_t)15;
  // Outputs that overlap the inputs are written by the last pass alone (the inputs are
  // read by the first alone), with two more sets between.
  auto meet = [](const void *a, size_t an, const void *b, size_t bn) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return x < y + bn && y < x + an;
  };
  bool in_place = false;
  for (const void *in : {(const void *)rows, (const void *)cols, (const void *)vals}) {
    const size_t bytes = n * (in == (const void *)vals ? sizeof(V) : 4);
    in_place |= meet(colind, n * 4, in, bytes) || meet(vals_out, n * sizeof(V), in, bytes);
  }
  const size_t keys = np > 1 ? 2 * kb : kb, one = np > 1 ? kb + vb : 0, set = in_place && np > 2 ? 2 * one : one,
               rest = count_words(nnz) * 4 + 64;
  sparsep::Scratch mem;
  bool by_index = false;
  cudaError_t e = sparsep::ws_malloc(&mem, keys + set + rest, s);
  if (e == cudaErrorMemoryAllocation && sizeof(V) == 8 && np > 1 && !in_place) {
    by_index = true;
    e = sparsep::ws_malloc(&mem, keys + rest, s);
  }
  int st = c2c_err(e);
  if (st) return st;
  unsigned char *buf = static_cast<unsigned char *>(mem.p);
  uint32_t *key_buf[2] = {reinterpret_cast<uint32_t *>(buf), reinterpret_cast<uint32_t *>(buf + keys - kb)};
  auto col_set = [&](int p) { return reinterpret_cast<uint32_t *>(buf + keys + (in_place && p % 2 ? one : 0)); };
  auto val_set = [&](int p) { return reinterpret_cast<V *>(buf + keys + (in_place && p % 2 ? one : 0) + kb); };
  uint32_t *counts = reinterpret_cast<uint32_t *>(buf + keys + (by_index ? 0 : set));
  int *bad = reinterpret_cast<int *>(counts + count_words(nnz));
  const uint32_t *key = rows, *col = by_index ? nullptr : cols;
  const V *val = vals;
  if (nnz) {
    int h_bad = 0;
    st = c2c_err(cudaMemsetAsync(bad, 0, sizeof(int), s));
    for (int p = 0, shift = 0; !st && p < np; shift += pass_bits(bits, p, np), ++p) {
      const int b = pass_bits(bits, p, np);
      const bool out = in_place ? p == np - 1 : (np - 1 - p) % 2 == 0;  // the last pass writes the outputs
      st = c2c_err(count_pass<uint32_t>(key, nnz, shift, b, counts, s, p ? nullptr : bad, nrows));
      if (!st && p == 0) {  // nothing of the outputs is written for a row index >= nrows
        st = c2c_err(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
        if (!st) st = c2c_err(cudaStreamSynchronize(s));
        if (!st && h_bad) st = SPARSEP_EINVAL;
      }
      uint32_t *ko = key_buf[p % 2], *co = out ? colind : by_index ? reinterpret_cast<uint32_t *>(vals_out) : col_set(p);
      if (!st && by_index)
        st = c2c_err(scatter_pass<uint32_t, NoValue>(key, col, nullptr, nnz, shift, b, counts, ko, co, nullptr, s));
      V *vo = out ? vals_out : val_set(p);
      if (!st && !by_index) {
        st = c2c_err(scatter_pass<uint32_t, V>(key, col, val, nnz, shift, b, counts, ko, co, vo, s));
        val = vo;
      }
      key = ko, col = co;
    }
    if (!st && by_index) {  // the indices are in colind now
      gather<V><<<(unsigned)std::min<uint64_t>(16384, (n + 255) / 256), 256, 0, s>>>(nnz, cols, vals, colind, vals_out);
      st = c2c_err(cudaGetLastError());
    }
  }
  if (!st) {
    rowptr_kernel<<<(nrows + 1 + 255) / 256, 256, 0, s>>>(key, nnz, nrows, rowptr);
    st = c2c_err(cudaGetLastError());
  }
  sparsep::ws_free(&mem, s);
  if (!st) st = c2c_err(cudaStreamSynchronize(s));
  return st;
}

#define SPARSEP_C2C_ENTRY(T, S)                                                                                 \
  int sparsep_coo2csr_device_##S(const uint32_t *d_rows, const uint32_t *d_cols, const T *d_vals, uint32_t nnz, \
                                 uint32_t nrows, uint32_t *d_rowptr, uint32_t *d_colind, T *d_vals_out,         \
                                 void *stream) {                                                                \
    using V = UintOf<sizeof(T)>::type;                                                                          \
    return coo2csr_device<V>(d_rows, d_cols, reinterpret_cast<const V *>(d_vals), nnz, nrows, d_rowptr,         \
                             d_colind, reinterpret_cast<V *>(d_vals_out), static_cast<cudaStream_t>(stream));   \
  }

extern "C" {
SPARSEP_C2C_ENTRY(int8_t, i8)
SPARSEP_C2C_ENTRY(int16_t, i16)
SPARSEP_C2C_ENTRY(int32_t, i32)
SPARSEP_C2C_ENTRY(int64_t, i64)
SPARSEP_C2C_ENTRY(float, f32)
SPARSEP_C2C_ENTRY(double, f64)
}
