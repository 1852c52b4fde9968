// kernels_impl.cuh -- the sm_100a SpMV kernels of sparsep_b200 (device code,
// included by kernels.cu and by the allocation-free entry point).
//
// One kernel template executes a list of work items (device.cuh: Item); one
// CTA runs one item.  The item kinds cover every reference kernel family:
//   CSR rows  (spmv/1D/CSR-*/dpu/task.c:31-215, spmv/2D/*DCSR/dpu/task.c)
//       -> products of a chunk of rows through shared memory (csr_stream), or
//          L lanes per row (L = 1..32); 128-bit loads of colind / values
//   CSR long-row chunks (no reference counterpart; the nnz balance remedy of
//       partition_by_nnz pushed below row granularity) -> CTA-wide reduction
//   COO elements (spmv/1D/COO-nnz/dpu/task.c lf :21-679, lb-fg :686-1338)
//       -> a stream of elements per warp, summed per row by segmented scans
//          (coo_items); rows that items share: lock-free, by the last item to
//          arrive, in item order, or red.global
//   BCSR block rows (spmv/1D/BCSR-nnz/dpu/task.c:231-380) -> chunks of blocks in
//       shared memory (bcsr_chunks), or for the block sizes without a template
//       the block in registers, L lanes per block row (bcsr_rows)
//   BCOO blocks (spmv/1D/BCOO-nnz/dpu/task.c:22-894) -> chunks likewise
//       (bcoo_chunks), or a block segmented scan with a row-block-wide payload
//       and carries added by the last CTA (bcoo_lf)
// 2D tiles are items whose x-segment is staged into shared memory by bulk
// (TMA) copies; their partial y goes to per-stripe slices merged on the device.
#pragma once
#include <cstdio>
#include <cstring>

#include "device.cuh"
#include "kernels.hpp"

namespace sparsep {

constexpr unsigned long long NO_CARRY = ~0ull;

// ---------------------------------------------------------------------------
// output helpers
// ---------------------------------------------------------------------------
// Carry targets are indices into the mode's output array: y, or the partial
// slices (slot * nrows + row).
template <typename T>
__device__ __forceinline__ uint64_t out_index(const Params<T> &P, const Item &it, uint64_t row) {
  return P.out_mode == OUT_PARTIAL ? (uint64_t)it.slot * P.nrows + row : row;
}

// x element: the staged segment lives in shared memory and must be read with
// generic loads; the non-coherent read-only path (ld.global.nc) is for x in
// global memory only.
template <typename T>
__device__ __forceinline__ T xload(const T *__restrict__ xb, uint64_t i, bool staged) {
  return staged ? xb[i] : __ldg(xb + i);
}

// checked build: x index valid for the staged segment or the whole vector
template <typename T>
__device__ __forceinline__ bool x_ok(const Params<T> &P, const Item &it, uint64_t col) {
  return it.xw > 0 ? (col >= it.xlo && col - it.xlo < it.xw) : col < P.n_x;
}

template <typename T>
__device__ __forceinline__ void put(const Params<T> &P, T *out, uint64_t r, Acc<T> v) {
  if (SP_BAD(P, r < P.nrows, -1004)) return;
  if (P.out_mode == OUT_ATOMIC) atomic_add_out<T>(out + r, v);
  else out[r] = from_acc<T>(v);
}

// ---------------------------------------------------------------------------
// CSR rows, L lanes per row
// ---------------------------------------------------------------------------
template <typename T, int L>
__device__ void csr_rows(const Params<T> &P, const Item &it, const T *__restrict__ xb) {
  using A = Acc<T>;
  constexpr int G = 32 / L;
  T *out = out_base(P, it);
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane / L, gl = lane % L;
  const uint32_t *rp = P.rowptr + it.ptr_base;
  const uint64_t r0 = it.a0, r1 = it.a1;
  const uint32_t xoff = it.col_off;

  auto do_row = [&](uint64_t r, bool valid_in) {
    bool valid = valid_in;
    A acc = A(0);
    if (valid && SP_BAD(P, it.ptr_base + r + 1 < P.n_rowptr, -1001)) valid = false;
    if (valid) {
      const uint64_t s = (uint64_t)rp[r] + it.nnz_base, e = (uint64_t)rp[r + 1] + it.nnz_base;
#pragma unroll 2
      for (uint64_t j = (s & ~3ull) + 4 * gl; j < e; j += 4 * L) {
        if (SP_BAD(P, j + 3 < P.n_idx && j + 3 < P.n_val, -1002)) break;
        const uint4 c4 = ld_stream4(P.colind + j);
        const Vec4<T> v4 = ld_vals4<T>(P.val + j);
        const uint32_t cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (j + k >= s && j + k < e && !SP_BAD(P, x_ok(P, it, (uint64_t)xoff + cc[k]), -1003))
            acc += mul<T>(v4.v[k], xload(xb, (uint64_t)xoff + cc[k], it.xw > 0));
      }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (valid && gl == 0) put<T>(P, out, it.row_off + r, acc);
  };

  if (it.worker_bal == SPARSEP_BAL_INTERLEAVE) {
    for (uint64_t k = 0;; ++k) {
      uint64_t base = r0 + (k * nw + warp) * G;
      if (base >= r1) break;
      do_row(base + g, base + g < r1);
    }
    return;
  }
  // contiguous row range per warp (reference tasklet split, partition_tsklt_by_row /
  // partition_tsklt_by_nnz, spmv/1D/CSR-row/support/partition.h:66-131)
  uint64_t wb, we;
  if (it.worker_bal == SPARSEP_BAL_NNZ) {
    const uint64_t lo = rp[r0], hi = rp[r1];
    auto find = [&](uint64_t target) {  // first row whose start >= target
      uint64_t a = r0, b = r1;
      while (a < b) {
        uint64_t m = (a + b) >> 1;
        if (rp[m] < target) a = m + 1; else b = m;
      }
      return a;
    };
    wb = warp == 0 ? r0 : find(lo + (hi - lo) * warp / nw);
    we = warp == nw - 1 ? r1 : find(lo + (hi - lo) * (warp + 1) / nw);
  } else {
    const uint64_t n = r1 - r0, q = n / nw, rem = n % nw;
    wb = r0 + q * warp + (warp < (int)rem ? warp : rem);
    we = wb + q + (warp < (int)rem ? 1 : 0);
  }
  for (uint64_t base = wb; base < we; base += G) do_row(base + g, base + g < we);
}

// ---------------------------------------------------------------------------
// Sums of the rows in a warp's stream of products (CSR rows, COO nonzeros), in
// windows of 32 lanes x K consecutive products.  A lane writes the rows that
// begin and end with it, a segmented scan over the lanes gives the others; a
// window inside one row only adds to the lanes' sums.  The part of the warp's
// first row and of its last one are left to the caller, since other warps may
// have parts of them too.
// ---------------------------------------------------------------------------
template <typename A> __device__ __forceinline__ A warp_sum(A v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename A> struct RowStream {
  A acc = A(0), osum = A(0);  // the open row's sum: a part per lane (windows inside the row) and the rest
  uint32_t open;              // the open row
  bool heads = false;         // a row began inside the stream: the first row's sum is in *first
  bool pend = false;          // acc holds something
};

// One window: products v, bit j of `hb` set where a row begins with the lane's
// product j, the row in rk[j].  put(row, sum) writes a row; *first takes the sum
// of the stream's first row once it has ended.
template <int K, typename A, typename Put>
__device__ __forceinline__ void row_window(RowStream<A> &S, const A (&v)[K], uint32_t hb, const uint32_t (&rk)[K],
                                           A *first, Put put) {
  constexpr uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool h0 = hb & 1u, brk = hb > 1u;
  const uint32_t mh = __ballot_sync(FULL, h0), mb = __ballot_sync(FULL, brk), m = mh | mb;
  A run = v[0];
  if (m == 0) {  // the window lies inside the open row
#pragma unroll
    for (int j = 1; j < K; ++j) run += v[j];
    S.acc += run;
    S.pend = true;
    return;
  }
  // the lane's products: its first row's part, rows of its own, its last row's part
  A hd = A(0);
  uint32_t row = rk[0];
  bool one = true;  // still in the first row
#pragma unroll
  for (int j = 1; j < K; ++j) {
    const bool h = (hb >> j) & 1u;
    if (h && !one) put(row, run);
    hd = h && one ? run : hd;
    one = one && !h;
    run = h ? v[j] : run + v[j];
    row = h ? rk[j] : row;
  }
  // the row that a lane goes on with is the last that began before it
  const uint32_t upto = FULL >> (31 - lane), below = m & (upto >> 1);
  const uint32_t from = __shfl_sync(FULL, row, below ? 31 - __clz(below) : 0);
  const uint32_t in = below ? from : S.open;
  const uint32_t row0 = h0 ? rk[0] : in;  // the lane's first row
  if (!h0 && !brk) row = in;              // and its last one
  // sums over the lanes since the last row began
  const int s = m & upto ? 31 - __clz(m & upto) : 0;
  A sc = run;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const A o = __shfl_up_sync(FULL, sc, d);
    if (lane - d >= s) sc += o;
  }
  const A up = __shfl_up_sync(FULL, sc, 1);
  if (lane > 0 && !h0) hd += up;  // the first row's part with what lanes before have of it
  // The open row ends before lane 0's products (c < 0), or in lane c: in its first
  // row (brk) or with its last.
  if (S.pend) S.osum += warp_sum<A>(S.acc);
  const int cb = mb ? __ffs(mb) - 1 : 32, ch = mh ? __ffs(mh) - 2 : 32, c = cb < ch ? cb : ch;
  const bool ends = lane < 31 && ((mh >> (lane + 1)) & 1u);  // the lane's last row ends with it
  if (S.heads) {
    const A add = lane == c ? S.osum : A(0);
    if (c < 0 && lane == 0) put(S.open, S.osum);
    if (brk) put(row0, hd + add);
    if (ends) put(row, brk ? sc : sc + add);
  } else {
    const bool mine = lane == c;
    if (mine || (c < 0 && lane == 0)) *first = S.osum + (c < 0 ? A(0) : brk ? hd : sc);
    if (brk && !mine) put(row0, hd);
    if (ends && (brk || !mine)) put(row, sc);
  }
  S.heads = true;
  S.pend = false;
  S.acc = A(0);
  S.osum = __shfl_sync(FULL, sc, 31);
  S.open = __shfl_sync(FULL, row, 31);
}

// What a CTA's warps leave of their streams: warp w's first row k0 with its
// part, and where a row began inside (heads) its last row k1 with its part.
template <typename A> struct StreamEnds {
  A first[16], last[16];
  uint32_t k0[16], k1[16], heads[16];
};
template <typename A> __device__ __forceinline__ void leave_ends(StreamEnds<A> &E, int w, RowStream<A> &S) {
  const A rest = S.osum + (S.pend ? warp_sum<A>(S.acc) : A(0));
  if ((threadIdx.x & 31) == 0) {
    if (S.heads) E.last[w] = rest;
    else E.first[w] = rest;
    E.k1[w] = S.open;
    E.heads[w] = S.heads;
  }
}

// ---------------------------------------------------------------------------
// CSR rows, staged ("stream") form used when lanes = auto.  A chunk of up to
// CSR_CAP nonzeros and a quarter as many rows is moved in three coalesced sweeps:
// its rowptr slice into shared memory, then every nonzero (128-bit loads of colind
// and values) times its gathered x into a shared product array; rows are then
// summed from shared memory (a thread per short row, a warp per long row) and
// written with consecutive threads on consecutive rows.  A row longer than the
// chunk capacity is reduced by the whole CTA straight from global memory.
// Bound by the gathers (see csr_chunk_nnz for what CSR_CAP costs them).
// ---------------------------------------------------------------------------
constexpr int CSR_SHORT = 48;  // rows up to this length are summed by one thread

// sum of a[s, e) x over the whole CTA (thread 0 gets the total)
template <typename T>
__device__ Acc<T> cta_range_sum(const Params<T> &P, const Item &it, const T *__restrict__ xb, uint64_t s,
                                uint64_t e, Acc<T> *red) {
  using A = Acc<T>;
  A acc = A(0);
#pragma unroll 2
  for (uint64_t j = (s & ~3ull) + 4 * threadIdx.x; j < e; j += 4 * blockDim.x) {
    if (SP_BAD(P, j + 3 < P.n_idx && j + 3 < P.n_val, -1005)) break;
    const uint4 c4 = ld_stream4(P.colind + j);
    const Vec4<T> v4 = ld_vals4<T>(P.val + j);
    const uint32_t cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j + k >= s && j + k < e && !SP_BAD(P, x_ok(P, it, (uint64_t)it.col_off + cc[k]), -1006))
        acc += mul<T>(v4.v[k], xload(xb, (uint64_t)it.col_off + cc[k], it.xw > 0));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __syncthreads();  // red may still be read from a previous call
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  A tot = A(0);
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
  return tot;
}

template <typename T, int CSR_CAP>
__device__ void csr_stream(const Params<T> &P, const Item &it, const T *__restrict__ xb) {
  using A = Acc<T>;
  constexpr int CSR_RCAP = CSR_CAP / 4;  // rows per chunk
  __shared__ A prods[CSR_CAP];
  __shared__ uint32_t srp[CSR_RCAP + 1];
  __shared__ uint16_t longs[CSR_RCAP];
  __shared__ uint32_t nlong;
  __shared__ A red[32];
  T *out = out_base(P, it);
  const uint32_t *rp = P.rowptr + it.ptr_base;
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool staged = it.xw > 0;
  uint64_t r = it.a0;
  while (r < it.a1) {
    const uint32_t nr = (uint32_t)((it.a1 - r) < CSR_RCAP ? (it.a1 - r) : CSR_RCAP);
    if (SP_BAD(P, it.ptr_base + r + nr < P.n_rowptr, -1001)) return;
    for (uint32_t i = threadIdx.x; i <= nr; i += blockDim.x) srp[i] = __ldcs(rp + r + i);
    if (threadIdx.x == 0) nlong = 0;
    __syncthreads();
    // rows [r, r+k) form the chunk: the longest prefix within CSR_CAP nonzeros
    const uint32_t base = srp[0];
    uint32_t k = nr;
    if (srp[nr] - base > (uint32_t)CSR_CAP) {
      uint32_t lo = 0, hi = nr;  // largest k with srp[k] - base <= CAP
      while (lo < hi) {
        const uint32_t m = (lo + hi + 1) >> 1;
        if (srp[m] - base <= (uint32_t)CSR_CAP) lo = m; else hi = m - 1;
      }
      k = lo;
    }
    if (k == 0) {  // one row longer than the chunk: whole-CTA reduction from global
      const A tot = cta_range_sum<T>(P, it, xb, (uint64_t)base + it.nnz_base, (uint64_t)srp[1] + it.nnz_base, red);
      if (threadIdx.x == 0) put<T>(P, out, it.row_off + r, tot);
      __syncthreads();
      r += 1;
      continue;
    }
    const uint64_t s0 = (uint64_t)base + it.nnz_base, e0 = (uint64_t)srp[k] + it.nnz_base;
    // per thread and pass 4 nonzeros: their index and value loads, then all x
    // gathers in flight at once, then the products
    for (uint64_t j = (s0 & ~3ull) + 4 * threadIdx.x; j < e0; j += 4 * blockDim.x) {
      if (SP_BAD(P, j + 3 < P.n_idx && j + 3 < P.n_val, -1002)) break;
      const uint4 c4 = ld_stream4(P.colind + j);
      const Vec4<T> v4 = ld_vals4<T>(P.val + j);
      const uint32_t cc[4] = {c4.x, c4.y, c4.z, c4.w};
      T xv[4];
      uint32_t bad = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (j + q >= s0 && j + q < e0) {
          const uint64_t col = (uint64_t)it.col_off + cc[q];
          if (SP_BAD(P, x_ok(P, it, col), -1003)) bad |= 1u << q;
          else xv[q] = xload(xb, col, staged);
        }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (j + q >= s0 && j + q < e0) prods[j + q - s0] = (bad >> q) & 1u ? A(0) : mul<T>(v4.v[q], xv[q]);
    }
    __syncthreads();
    // short rows: one thread each; long rows are queued for the warps
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
      const uint32_t a = srp[i] - base, b = srp[i + 1] - base;
      if (b - a <= (uint32_t)CSR_SHORT) {
        A acc = A(0);
        for (uint32_t q = a; q < b; ++q) acc += prods[q];
        put<T>(P, out, it.row_off + r + i, acc);
      } else {
        longs[atomicAdd(&nlong, 1u)] = (uint16_t)i;
      }
    }
    __syncthreads();
    for (uint32_t li = warp; li < nlong; li += nw) {
      const uint32_t i = longs[li];
      const uint32_t a = srp[i] - base, b = srp[i + 1] - base;
      A acc = A(0);
      for (uint32_t q = a + lane; q < b; q += 32) acc += prods[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) put<T>(P, out, it.row_off + r + i, acc);
    }
    __syncthreads();
    r += k;
  }
}

// ---------------------------------------------------------------------------
// CSR long-row chunk: all threads reduce elements [a0, a1) of row crow.
// ---------------------------------------------------------------------------
template <typename T>
__device__ void csr_long(const Params<T> &P, const Item &it, const T *__restrict__ xb, uint32_t item_id) {
  using A = Acc<T>;
  __shared__ A red[32];
  const uint64_t s = it.a0, e = it.a1;
  A acc = A(0);
#pragma unroll 2
  for (uint64_t j = (s & ~3ull) + 4 * threadIdx.x; j < e; j += 4 * blockDim.x) {
    if (SP_BAD(P, j + 3 < P.n_idx && j + 3 < P.n_val, -1005)) break;
    const uint4 c4 = ld_stream4(P.colind + j);
    const Vec4<T> v4 = ld_vals4<T>(P.val + j);
    const uint32_t cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j + k >= s && j + k < e && !SP_BAD(P, x_ok(P, it, (uint64_t)it.col_off + cc[k]), -1006))
        acc += mul<T>(v4.v[k], xload(xb, (uint64_t)it.col_off + cc[k], it.xw > 0));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    A tot = A(0);
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
    T *out = out_base(P, it);
    if (SP_BAD(P, it.crow < P.nrows && (P.out_mode == OUT_ATOMIC || item_id < P.n_carry), -1007)) return;
    if (P.out_mode == OUT_ATOMIC) {
      atomic_add_out<T>(out + it.crow, tot);
    } else {
      // the last chunk of the row to arrive sums the row's partials in chunk order
      P.carry_val[item_id] = acc_bits(tot);
      __threadfence();
      const unsigned int prev = atomicAdd(P.row_cnt + it.cslot, 1u);
      if (prev == it.nchunk - 1) {
        __threadfence();
        A sum = A(0);
        for (uint32_t c = 0; c < it.nchunk; ++c) sum += bits_acc<A>(__ldcg(P.carry_val + it.first + c));
        out[it.crow] = from_acc<T>(sum);
        P.row_cnt[it.cslot] = 0;  // ready for the next launch
      }
    }
  }
}

// the reference's AoS nonzero for element type T
template <typename T> struct ElemOf;
template <> struct ElemOf<int8_t> { using type = sparsep_elem_i8; };
template <> struct ElemOf<int16_t> { using type = sparsep_elem_i16; };
template <> struct ElemOf<int32_t> { using type = sparsep_elem_i32; };
template <> struct ElemOf<int64_t> { using type = sparsep_elem_i64; };
template <> struct ElemOf<float> { using type = sparsep_elem_f32; };
template <> struct ElemOf<double> { using type = sparsep_elem_f64; };

// Row-vector of CB elements of a dense block row, at an address aligned to CB*sizeof(T).
template <typename T, int CB>
__device__ __forceinline__ void load_brow(const T *p, T (&v)[CB]) {
  constexpr int BYTES = CB * (int)sizeof(T);
  if constexpr (BYTES >= 16) {
#pragma unroll
    for (int q = 0; q < BYTES / 16; ++q) {
      uint4 w = ld_stream4(reinterpret_cast<const char *>(p) + 16 * q);
      const T *t = reinterpret_cast<const T *>(&w);
#pragma unroll
      for (int i = 0; i < 16 / (int)sizeof(T); ++i) v[q * (16 / sizeof(T)) + i] = t[i];
    }
  } else if constexpr (BYTES == 8) {
    uint2 w = __ldcs(reinterpret_cast<const uint2 *>(p));
    const T *t = reinterpret_cast<const T *>(&w);
#pragma unroll
    for (int i = 0; i < CB; ++i) v[i] = t[i];
  } else if constexpr (BYTES == 4) {
    unsigned int w = __ldcs(reinterpret_cast<const unsigned int *>(p));
    const T *t = reinterpret_cast<const T *>(&w);
#pragma unroll
    for (int i = 0; i < CB; ++i) v[i] = t[i];
  } else {
#pragma unroll
    for (int i = 0; i < CB; ++i) v[i] = p[i];
  }
}

// One dense RB x CB block times its x-segment, accumulated into acc[RB].
// RB = CB = 0 selects the runtime-size path (rb <= 16).
template <typename T, int RB, int CB>
__device__ __forceinline__ void block_mv(const Params<T> &P, const T *__restrict__ xb, uint64_t b, uint32_t J,
                                         uint32_t col_off, Acc<T> *acc, const Item &it) {
  if (SP_BAD(P, (b + 1) * P.rb * P.cb <= P.n_val, -1010)) return;
  if constexpr (RB > 0) {
    const uint64_t c0 = (uint64_t)col_off + (uint64_t)J * CB;
    T xv[CB];
#pragma unroll
    for (int c = 0; c < CB; ++c)
      xv[c] = (c0 + c < P.ncols && !SP_BAD(P, x_ok(P, it, c0 + c), -1011)) ? xload(xb, c0 + c, it.xw > 0) : T(0);
    const T *bp = P.bval + b * (RB * CB);
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      T v[CB];
      load_brow<T, CB>(bp + r * CB, v);
#pragma unroll
      for (int c = 0; c < CB; ++c) acc[r] += mul<T>(v[c], xv[c]);
    }
  } else {
    const uint32_t rb = P.rb, cb = P.cb;
    const uint64_t c0 = (uint64_t)col_off + (uint64_t)J * cb;
    const T *bp = P.bval + b * rb * cb;
    for (uint32_t c = 0; c < cb; ++c) {
      if (c0 + c >= P.ncols) break;
      if (SP_BAD(P, x_ok(P, it, c0 + c), -1011)) break;
      T xv = xload(xb, c0 + c, it.xw > 0);
      for (uint32_t r = 0; r < rb; ++r) acc[r] += mul<T>(bp[r * cb + c], xv);
    }
  }
}

// ---------------------------------------------------------------------------
// Dense blocks of 2x2, 4x4 and 8x8, read as the 16-byte pieces they are made
// of: consecutive lanes take consecutive pieces, so a warp reads 512
// contiguous bytes of block values whatever the type and the block size.  A
// block of B bytes is spread over LPB = B / 16 lanes (one lane for blocks of
// up to 16 bytes); a piece is RPC whole rows of the block, or a CPR-th of one.
// ---------------------------------------------------------------------------
template <typename T, int RB, int CB> struct Pieces {
  static constexpr int B = RB * CB * (int)sizeof(T);
  static constexpr int BYTES = B < 16 ? B : 16;     // of a piece
  static constexpr int E = BYTES / (int)sizeof(T);  // elements of a piece
  static constexpr int LPB = B / BYTES;             // lanes per block
  static constexpr int RPC = E >= CB ? E / CB : 1;  // rows in a piece
  static constexpr int CPR = E >= CB ? 1 : CB / E;  // pieces of a row
  static constexpr int NX = E >= CB ? CB : E;       // x elements a piece meets
  static constexpr int XB = NX * (int)sizeof(T);    // their bytes
  static constexpr int W = (BYTES + 3) / 4, XW = (XB + 3) / 4;
};

// N bytes (2, 4, 8 or 16) at an address aligned to them, as 32-bit words.
template <int N> __device__ __forceinline__ void load_words(const void *p, uint32_t *w) {
  if constexpr (N == 16) {
    const uint4 q = *reinterpret_cast<const uint4 *>(p);
    w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
  } else if constexpr (N == 8) {
    const uint2 q = *reinterpret_cast<const uint2 *>(p);
    w[0] = q.x, w[1] = q.y;
  } else if constexpr (N == 4) {
    w[0] = *reinterpret_cast<const uint32_t *>(p);
  } else {
    w[0] = *reinterpret_cast<const uint16_t *>(p);
  }
}

// Element i of packed words.
template <typename T> __device__ __forceinline__ T word_elem(const uint32_t *w, int i) {
  if constexpr (sizeof(T) == 1) return (T)(int8_t)(w[i >> 2] >> (8 * (i & 3)));
  else if constexpr (sizeof(T) == 2) return (T)(int16_t)(w[i >> 1] >> (16 * (i & 1)));
  else {
    T v;
    if constexpr (sizeof(T) == 4) {
      memcpy(&v, &w[i], 4);
    } else {
      const unsigned long long u = ((unsigned long long)w[2 * i + 1] << 32) | w[2 * i];
      memcpy(&v, &u, 8);
    }
    return v;
  }
}

// The NX elements of x that a piece of a block in block column J meets (xt: x
// from the tile's first column), packed.  FULL: the block column lies inside
// the matrix and x is aligned to the NX elements, so one load brings them.
// Otherwise one by one, zeros past the last column.
template <typename T, int RB, int CB, bool FULL>
__device__ __forceinline__ void load_xpiece(const Params<T> &P, const Item &it, const T *__restrict__ xt, uint32_t J,
                                            uint32_t xcol, uint32_t (&w)[Pieces<T, RB, CB>::XW]) {
  using G = Pieces<T, RB, CB>;
  const uint64_t c = (uint64_t)J * CB + xcol;
  if constexpr (FULL) {
    if (!SP_BAD(P, x_ok(P, it, it.col_off + c) && x_ok(P, it, it.col_off + c + G::NX - 1), -1011))
      load_words<G::XB>(xt + c, w);
  } else {
#pragma unroll
    for (int i = 0; i < G::XW; ++i) w[i] = 0;
#pragma unroll
    for (int i = 0; i < G::NX; ++i) {
      T v = T(0);
      if (it.col_off + c + i < P.ncols && !SP_BAD(P, x_ok(P, it, it.col_off + c + i), -1011)) v = xt[c + i];
      if constexpr (sizeof(T) == 8) {
        unsigned long long u;
        memcpy(&u, &v, 8);
        w[2 * i] = (uint32_t)u, w[2 * i + 1] = (uint32_t)(u >> 32);
      } else if constexpr (sizeof(T) == 4) {
        memcpy(&w[i], &v, 4);
      } else {
        constexpr int PER = 4 / (int)sizeof(T), SH = 8 * (int)sizeof(T);
        w[i / PER] |= ((uint32_t)v & ((1u << SH) - 1u)) << (SH * (i % PER));
      }
    }
  }
}

// A lane's sum of a block row's row.  Floating point: with what the additions rounded
// off beside it (the fast two-sum; exact while the sum is the larger of the two, and
// no worse than plain addition otherwise).  A lane adds the pieces of an eighth to all
// of a block row's blocks one after the other, where bcsr_rows spread them over 16 or
// 32 lanes: FP32 4x4 / 8x8, root mean square error in units of the last place of a
// row's norm, 20 blocks per block row 0.60 / 0.70 with bcsr_rows, 0.98 / 1.01 added up
// plainly, 0.55 / 0.57 like this; 200 blocks 0.92 / 1.20, 1.56 / 3.0, 0.60 / 0.69.  It
// costs FP32 1 to 2 % and FP64 3 to 4 % (1M rows 4x4, FP64: 116 -> 120 us; two plain sums
// in turn 118.5 us, but 200 blocks 8x8 no better than bcsr_rows).
template <typename T> struct RowSum {
  Acc<T> s = Acc<T>(0), off = Acc<T>(0);  // off: floating point only
  __device__ __forceinline__ void add(Acc<T> x) {
    const Acc<T> t = s + x;
    off += x - (t - s);
    s = t;
  }
  // off is not a number once a sum is infinite
  __device__ __forceinline__ Acc<T> get() const {
    if constexpr (std::is_floating_point<T>::value) return off - off == Acc<T>(0) ? s + off : s;
    else return s;
  }
};

// N pieces times their x, added to the sums of their rows.
template <typename T, int RB, int CB, int N>
__device__ __forceinline__ void pieces_mv(const uint32_t (&v)[N][Pieces<T, RB, CB>::W],
                                          const uint32_t (&x)[N][Pieces<T, RB, CB>::XW],
                                          RowSum<T> (&acc)[Pieces<T, RB, CB>::RPC]) {
  using G = Pieces<T, RB, CB>;
#pragma unroll
  for (int r = 0; r < G::RPC; ++r) {
    if constexpr (sizeof(T) == 1 && G::NX % 4 == 0) {  // four products and their sum in one instruction, exact
#pragma unroll
      for (int n = 0; n < N; ++n)
#pragma unroll
        for (int q = 0; q < G::NX / 4; ++q)
          acc[r].s = (uint32_t)__dp4a((int)v[n][r * (G::NX / 4) + q], (int)x[n][q], (int)acc[r].s);
    } else if constexpr (!std::is_floating_point<T>::value) {
#pragma unroll
      for (int n = 0; n < N; ++n)
#pragma unroll
        for (int c = 0; c < G::NX; ++c) acc[r].s += mul<T>(word_elem<T>(v[n], r * G::NX + c), word_elem<T>(x[n], c));
    } else {
      Acc<T> sum = Acc<T>(0);
#pragma unroll
      for (int n = 0; n < N; ++n) {
        Acc<T> p = mul<T>(word_elem<T>(v[n], r * G::NX), word_elem<T>(x[n], 0));
#pragma unroll
        for (int c = 1; c < G::NX; ++c) p += mul<T>(word_elem<T>(v[n], r * G::NX + c), word_elem<T>(x[n], c));
        sum = n ? sum + p : p;
      }
      acc[r].add(sum);
    }
  }
}

// Sums over the lanes of a group that hold other blocks (strides LPB, 2 LPB,
// ..., L / 2), or other pieces of the same block row's row (strides below CPR).
template <typename T, int RB, int CB, int L>
__device__ __forceinline__ void sum_pieces(Acc<T> (&acc)[Pieces<T, RB, CB>::RPC]) {
  using G = Pieces<T, RB, CB>;
#pragma unroll
  for (int w = 0; w < G::RPC; ++w) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1)
      if (o >= G::LPB || o < G::CPR) acc[w] += __shfl_xor_sync(0xffffffffu, acc[w], o);
  }
}

// ---------------------------------------------------------------------------
// BCSR in chunks: a work item is a chunk of whole block rows (at most S blocks
// and ROWS block rows, or one longer block row).  Its values and block columns
// come into shared memory by bulk copies; then LPB * BK lanes take a block
// row, BK blocks at a time, and only x is read from memory by loads.
//
// Bound by HBM, the block values.  A lane per whole block, as every block size
// ran before (bcsr_rows), asked for each 32-byte sector twice (lanes 64 bytes
// apart) with 100 M instructions.  Block-banded matrices, 20 blocks per block
// row, before -> now: FP32 4x4, 2M rows (732 MB) 191 -> 119 us, 6.1 TB/s, 94 % of
// the measured copy rate; INT8 8x8, 2M rows (362 MB) 149 -> 62 us; INT16 4x4,
// 1M rows 71 -> 43 us; FP64 4x4, 1M rows 229 -> 124 us.
// What was tried on the way, FP32 4x4: the same lanes reading values straight
// from memory 200 us (the latency of one step after another); a ring of copies
// per warp over contiguous block rows 185 us (143 M instructions at the block
// rows' ends); persistent CTAs with two chunks in flight 176 us and with x
// gathered a chunk ahead 160 us (24 warps per SM cannot hide the x loads).
// Chunks of 24 / 28 / 40 KB: 133 / 125 / 127 us against 119 us for 32 KB, six
// CTAs per SM; 46 instead of 40 registers (five CTAs) 126 us.
// ---------------------------------------------------------------------------
template <typename T, int RB, int CB> struct BlockStage {
  using G = Pieces<T, RB, CB>;
  static constexpr int S = (int)bcsr_chunk_blocks(RB, CB, sizeof(T)), ROWS = (int)BCSR_CHUNK_ROWS;
  // 4-block (16-byte) alignment at both ends of the copies
  static constexpr int COL = (S + 8) * G::B, PTR = COL + (S + 8) * 4;
  static constexpr int SMEM = (PTR + (ROWS + 1) * 4 + 127) / 128 * 128;
};

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void expect_bytes(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Bounded wait of the CTA for a barrier phase; false (for all) when it ran out:
// the error word is set, and the copies get one more bounded wait.  The first
// warp polls, suspended up to ~20 us per try, and the others wait for it at the
// CTA's barrier, out of the way of the other CTAs (5 % of a COO kernel that staged
// its nonzeros this way).
__device__ __forceinline__ bool cta_wait(uint64_t *bar, uint32_t parity, int *err) {
  auto poll = [&]() {
    uint32_t done = 0;
    for (uint32_t i = 0; i < (1u << 18) && !done; ++i)
      asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
                   : "=r"(done)
                   : "r"(smem_u32(bar)), "r"(parity), "r"(20000u)
                   : "memory");
    return done != 0;
  };
  if (!__syncthreads_or(threadIdx.x < 32 && !poll())) return true;
  if (threadIdx.x == 0 && err) atomicExch(err, SPARSEP_ETIMEDOUT);
  if (threadIdx.x < 32) poll();
  return false;
}

// k block rows whose blocks are staged from sval on, block columns from scol on
// (CS apart), block row i at [srp[i], srp[i + 1]) - srp[0].  put_row(i, r, sum)
// takes row r of block row i from the lane that holds its sum.
template <typename T, int RB, int CB, int BK, bool FULL, int CS, typename Put>
__device__ __forceinline__ void block_rows_staged(const Params<T> &P, const Item &it, const T *__restrict__ xt,
                                                  uint32_t k, const uint32_t *srp, const unsigned char *sval,
                                                  const uint32_t *scol, Put put_row) {
  using G = Pieces<T, RB, CB>;
  using A = Acc<T>;
  constexpr int L = G::LPB * BK, GN = 32 / L;  // lanes per block row, block rows per warp
  const uint32_t b0 = srp[0];
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane / L, gl = lane % L, q = gl % G::LPB, bi = gl / G::LPB;
  const uint32_t xcol = (uint32_t)(q % G::CPR) * G::NX;
  sval += q * G::BYTES;
  for (uint32_t base = warp * GN; base < k; base += nw * GN) {
    const uint32_t i = base + g;
    RowSum<T> sums[G::RPC];
    if (i < k) {
      const uint32_t e = srp[i + 1] - b0;
      uint32_t b = srp[i] - b0 + bi;
      // two blocks a step: their x on the way together
      for (; b + BK < e; b += 2 * BK) {
        uint32_t v[2][G::W], x[2][G::XW];
        const uint32_t J0 = scol[b * CS], J1 = scol[(b + BK) * CS];
        load_xpiece<T, RB, CB, FULL>(P, it, xt, J0, xcol, x[0]);
        load_xpiece<T, RB, CB, FULL>(P, it, xt, J1, xcol, x[1]);
        load_words<G::BYTES>(sval + b * G::B, v[0]);
        load_words<G::BYTES>(sval + (b + BK) * G::B, v[1]);
        pieces_mv<T, RB, CB, 2>(v, x, sums);
      }
      if (b < e) {
        uint32_t v[1][G::W], x[1][G::XW];
        load_xpiece<T, RB, CB, FULL>(P, it, xt, scol[b * CS], xcol, x[0]);
        load_words<G::BYTES>(sval + b * G::B, v[0]);
        pieces_mv<T, RB, CB, 1>(v, x, sums);
      }
    }
    __syncwarp();
    A acc[G::RPC];
#pragma unroll
    for (int w = 0; w < G::RPC; ++w) acc[w] = sums[w].get();
    sum_pieces<T, RB, CB, L>(acc);
    if (i < k && bi == 0 && q % G::CPR == 0) {
#pragma unroll
      for (int w = 0; w < G::RPC; ++w) put_row(i, (q / G::CPR) * G::RPC + w, acc[w]);
    }
  }
}

// The same for the item's number of blocks at a time, as far as a warp holds them.
template <typename T, int RB, int CB, int CS, typename Put>
__device__ __forceinline__ void block_rows_any(const Params<T> &P, const Item &it, const T *__restrict__ xt,
                                               uint32_t k, const uint32_t *srp, const unsigned char *sval,
                                               const uint32_t *scol, uint32_t lanes, bool whole, Put put_row) {
  constexpr uint32_t M = 32 / Pieces<T, RB, CB>::LPB;
  auto go = [&](auto n) {
    constexpr int BK = decltype(n)::value;
    if (whole) block_rows_staged<T, RB, CB, BK, true, CS>(P, it, xt, k, srp, sval, scol, put_row);
    else block_rows_staged<T, RB, CB, BK, false, CS>(P, it, xt, k, srp, sval, scol, put_row);
  };
  const uint32_t bk = lanes < M ? lanes : M;
  if constexpr (M >= 8) if (bk >= 8) go(std::integral_constant<int, 8>());
  if constexpr (M >= 4) if (bk == 4) go(std::integral_constant<int, 4>());
  if constexpr (M >= 2) if (bk == 2) go(std::integral_constant<int, 2>());
  if (bk == 1) go(std::integral_constant<int, 1>());
}

// Whether x can be read piece by piece: it is aligned to the pieces and the
// chunk's n block columns (CS apart) lie inside the matrix.  A barrier where the
// tile's last block column is ragged.
template <typename T, int RB, int CB, int CS>
__device__ __forceinline__ bool x_whole(const Params<T> &P, const Item &it, const T *xt, const uint32_t *scol,
                                        uint32_t n) {
  if (reinterpret_cast<uintptr_t>(xt) & (Pieces<T, RB, CB>::XB - 1)) return false;
  const uint32_t jfull = it.col_off < P.ncols ? (P.ncols - it.col_off) / CB : 0;
  if (it.col_off + (uint64_t)jfull * CB >= P.ncols) return true;
  bool in = true;
  for (uint32_t b = threadIdx.x; b < n; b += blockDim.x) in &= scol[b * CS] < jfull;
  return !__syncthreads_or(!in);
}

// A block row of more blocks than a chunk holds: the CTA's warps share its
// blocks and read them straight from memory; warp sums added in warp order.
template <typename T, int RB, int CB>
__device__ void bcsr_long_row(const Params<T> &P, const Item &it, const T *__restrict__ xt, Acc<T> *red) {
  using G = Pieces<T, RB, CB>;
  using A = Acc<T>;
  constexpr int STEP = 32 / G::LPB;
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = lane % G::LPB, bi = lane / G::LPB;
  const uint32_t xcol = (uint32_t)(q % G::CPR) * G::NX;
  RowSum<T> sums[G::RPC];
#pragma unroll 2
  for (uint64_t b = it.n0 + warp * STEP + bi; b < it.n1; b += nw * STEP) {
    uint32_t v[1][G::W], x[1][G::XW];
    load_words<G::BYTES>(reinterpret_cast<const char *>(P.bval) + b * G::B + q * G::BYTES, v[0]);
    load_xpiece<T, RB, CB, false>(P, it, xt, P.bcolind[b], xcol, x[0]);
    pieces_mv<T, RB, CB, 1>(v, x, sums);
  }
  A acc[G::RPC];
#pragma unroll
  for (int w = 0; w < G::RPC; ++w) acc[w] = sums[w].get();
  __syncwarp();
  sum_pieces<T, RB, CB, 32>(acc);
#pragma unroll
  for (int w = 0; w < G::RPC; ++w)
    if (bi == 0 && q % G::CPR == 0) red[warp * RB + (q / G::CPR) * G::RPC + w] = acc[w];
  __syncthreads();
  const uint64_t row = (uint64_t)it.row_off + it.a0 * RB + threadIdx.x;
  if (threadIdx.x < RB && row < it.row_end) {
    A t = A(0);
    for (int w = 0; w < nw; ++w) t += red[w * RB + threadIdx.x];
    put<T>(P, out_base(P, it), row, t);
  }
}

template <typename T, int RB, int CB>
__global__ void __launch_bounds__(512, 3) bcsr_chunks(Params<T> P) {
  using G = Pieces<T, RB, CB>;
  using St = BlockStage<T, RB, CB>;
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  __shared__ uint64_t bar, xbar;
  unsigned char *sm = dyn_smem + (P.smem_bytes + 127) / 128 * 128;  // behind a tile's staged x
  uint32_t *srp = reinterpret_cast<uint32_t *>(sm + St::PTR);
  const Item it = P.items[blockIdx.x];
  const uint64_t A0 = it.n0 & ~3ull, A1 = (it.n1 + 3) & ~3ull;  // the arrays are padded past their end
  const bool longer = it.n1 - it.n0 > (uint64_t)St::S, stage = it.n0 < it.n1 && !longer;
  if (SP_BAD(P, A1 <= P.n_idx && A1 * (RB * CB) <= P.n_val, -1013)) return;
  if (SP_BAD(P, it.ptr_base + it.a1 < P.n_rowptr && it.a1 - it.a0 <= St::ROWS, -1012)) return;
  mbar_init(&bar);
  if (threadIdx.x == 0 && stage) {
    const uint32_t n = (uint32_t)(A1 - A0);
    expect_bytes(&bar, n * (uint32_t)(G::B + 4));
    bulk_load(sm + St::COL, P.bcolind + A0, n * 4, &bar);
    bulk_load(sm, reinterpret_cast<const char *>(P.bval) + A0 * G::B, n * G::B, &bar);
  }
  for (uint32_t i = threadIdx.x; i <= (uint32_t)(it.a1 - it.a0); i += blockDim.x)
    srp[i] = __ldcs(P.rowptr + it.ptr_base + it.a0 + i);
  const T *xb = P.x;
  if (it.xw > 0) {
    uint32_t phase = 0;
    mbar_init(&xbar);
    xb = stage_x<T>(P.x, it.xlo, it.xw, dyn_smem, &xbar, phase, P.err, P.smem_bytes,
                    reinterpret_cast<uintptr_t>(P.x + P.n_xalloc), P.fault_wait);
  }
  const T *xt = xb + it.col_off;
  T *out = out_base(P, it);
  if (longer) {
    bcsr_long_row<T, RB, CB>(P, it, xt, reinterpret_cast<Acc<T> *>(sm));
    return;
  }
  if (stage) {
    if (!cta_wait(&bar, 0, P.err)) return;
  } else {
    __syncthreads();
  }
  const uint32_t lead = (uint32_t)(it.n0 - A0);
  const uint32_t *scol = reinterpret_cast<const uint32_t *>(sm + St::COL) + lead;
  const bool whole = x_whole<T, RB, CB, 1>(P, it, xt, scol, (uint32_t)(it.n1 - it.n0));
  block_rows_any<T, RB, CB, 1>(P, it, xt, (uint32_t)(it.a1 - it.a0), srp, sm + lead * G::B, scol, it.lanes, whole,
                               [&](uint32_t i, uint32_t r, Acc<T> sum) {
                                 const uint64_t row = (uint64_t)it.row_off + (it.a0 + i) * RB + r;
                                 if (row < it.row_end) put<T>(P, out, row, sum);
                               });
}

// ---------------------------------------------------------------------------
// BCSR block rows of the other block sizes, L lanes per block row
// ---------------------------------------------------------------------------
template <typename T, int RB, int CB, int L>
__device__ void bcsr_rows(const Params<T> &P, const Item &it, const T *__restrict__ xb) {
  using A = Acc<T>;
  constexpr int RMAX = RB > 0 ? RB : 16;
  constexpr int G = 32 / L;
  T *out = out_base(P, it);
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane / L, gl = lane % L;
  const uint32_t rb = RB > 0 ? RB : P.rb;
  const uint32_t *bp = P.rowptr + it.ptr_base;  // browptr
  for (uint64_t k = 0;; ++k) {
    const uint64_t base = it.a0 + (k * nw + warp) * G;
    if (base >= it.a1) break;
    const uint64_t br = base + g;
    const bool valid = br < it.a1;
    A acc[RMAX];
#pragma unroll
    for (int r = 0; r < RMAX; ++r) acc[r] = A(0);
    if (valid && !SP_BAD(P, it.ptr_base + br + 1 < P.n_rowptr, -1012)) {
      const uint64_t s = (uint64_t)bp[br] + it.nnz_base, e = (uint64_t)bp[br + 1] + it.nnz_base;
      for (uint64_t b = s + gl; b < e; b += L) {
        if (SP_BAD(P, b < P.n_idx, -1013)) break;
        block_mv<T, RB, CB>(P, xb, b, __ldcs(P.bcolind + b), it.col_off, acc, it);
      }
    }
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
    }
    if (valid) {
#pragma unroll
      for (int r = 0; r < RMAX; ++r) {
        if (r < (int)rb && gl == (r % L)) {
          const uint64_t row = (uint64_t)it.row_off + br * rb + r;
          if (row < it.row_end) put<T>(P, out, row, acc[r]);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Rows shared by several element items.  A COO item is a range of nonzeros (a
// BCOO item of blocks), so its first and its last row may go on in its
// neighbours.  The planner numbers those rows: each has a counter and knows
// its items [f, f + n), consecutive ones.  Every item of the row leaves its part
// in its slots (2 item: as the row's last item, 2 item + 1: as an earlier one)
// and counts itself; the last to arrive adds the parts in item order, the row's
// last item's part last, writes the row and clears the counter.  Every item
// arrives, also after a failed wait (with zeros), so the counters are zero
// between launches.
// ---------------------------------------------------------------------------
struct RowGroup {
  uint32_t cnt, f, n;  // counter, first item, items (0: the row is the item's own)
};
__device__ __forceinline__ RowGroup first_row_group(const Item &it) { return {it.cslot, it.first, it.nchunk}; }
__device__ __forceinline__ RowGroup last_row_group(const Item &it) { return {it.chunk, it.crow, (uint32_t)it.n1}; }

// An item's part of a shared row (of the W rows of a shared block row): lane r < W
// of the warp holds row r, which belongs at out[row0 + r].
template <typename T> struct SharedPart {
  RowGroup g{0, 0, 0};  // n = 0: none
  uint64_t row0 = 0;
  Acc<T> part = Acc<T>(0);
};

// One warp leaves the parts of the item's first and last row, counts the item
// in for both at once, and adds up the rows that are complete by that.  Rows from
// `row_end` on are dropped.
template <typename T, int W>
__device__ void arrive(const Params<T> &P, T *out, uint32_t item, uint64_t row_end, const SharedPart<T> &first,
                       const SharedPart<T> &last) {
  using A = Acc<T>;
  const uint32_t lane = threadIdx.x & 31;
  auto slot = [](const RowGroup &g, uint32_t i) {
    return (uint64_t)(2 * (uint64_t)i + (i == g.f + g.n - 1 ? 0 : 1)) * W;
  };
  if (SP_BAD(P, (2 * (uint64_t)item + 2) * W <= P.n_carry, -1018)) return;
  if (lane < W) {
    if (first.g.n) P.carry_val[slot(first.g, item) + lane] = acc_bits(first.part);
    if (last.g.n) P.carry_val[slot(last.g, item) + lane] = acc_bits(last.part);
  }
  __threadfence();  // the parts are visible before the arrival
  __syncwarp();
  unsigned int prev = 0;
  if (lane == 0 && first.g.n) prev = atomicAdd(P.row_cnt + first.g.cnt, 1u);
  if (lane == 1 && last.g.n) prev = atomicAdd(P.row_cnt + last.g.cnt, 1u);
  for (int which = 0; which < 2; ++which) {
    const SharedPart<T> &s = which ? last : first;
    if (s.g.n == 0 || __shfl_sync(0xffffffffu, prev, which) != s.g.n - 1) continue;
    __threadfence();
    const RowGroup g = s.g;
    A sum = A(0);
    constexpr uint32_t N = 32 / W;  // items whose parts come in one round trip, added one after the other
    for (uint32_t c0 = 0; c0 + 1 < g.n; c0 += N) {
      const uint32_t c = c0 + lane / W;
      const A v = c + 1 < g.n ? bits_acc<A>(__ldcg(P.carry_val + slot(g, g.f + c) + lane % W)) : A(0);
      for (uint32_t j = 0; j < N && c0 + j + 1 < g.n; ++j) {
        const A t = __shfl_sync(0xffffffffu, v, j * W + lane % W);
        sum = c0 + j ? sum + t : t;
      }
    }
    if (lane < W) {
      sum = bits_acc<A>(__ldcg(P.carry_val + slot(g, g.f + g.n - 1) + lane)) + sum;
      if (s.row0 + lane < row_end && !SP_BAD(P, s.row0 + lane < P.nrows, -1015))
        out[s.row0 + lane] = from_acc<T>(sum);
    }
    if (lane == 0) P.row_cnt[g.cnt] = 0;  // ready for the next launch
  }
}

// ---------------------------------------------------------------------------
// COO nonzeros (AoS, sorted by row) as a stream of products: each warp takes an
// even share of the item's nonzeros, K consecutive ones per lane and window
// (128-bit loads, the next window's under way); a row begins where the row index
// changes.  One barrier, then warp 0 joins the rows cut by the warps' boundaries.
//
// Bound by the gathers of x, each a line that L1 has to hold while it is under
// way: 16.7 M of them at random columns take 67 us by themselves, and what the
// kernel takes of L1 as shared memory it loses in gathers in flight.  FP32 on the
// 1M-row power-law matrix (210 MB): block-wide segmented scans, 4 nonzeros per
// thread, and a last CTA that added all carries 172 us; this 90 us.  The same
// stream over chunks brought into shared memory by bulk copies 116 us, with
// windows dealt out through 1.5 KB of it per warp 112 us, 8 warps per CTA 100 us,
// x a window ahead (64 registers) 107 us.  FP64 203 -> 102 us; equal tiles 16 x 16
// of the 524,309-row matrix, most of whose rows are empty, 116 -> 76 us (94 while
// each lane zeroed the rows before its own nonzeros one by one).
//
// GROUPS: the planner numbered the rows that items share; otherwise the item's
// first row goes to y as far as the item has it, and a last row that goes on in
// the next item to the item's carry slot (carry_fixup adds the carries).
// ---------------------------------------------------------------------------
template <typename T, bool GROUPS, bool ATOMIC>
__device__ __forceinline__ void coo_stream(const Params<T> &P, const Item &it, const T *__restrict__ xb,
                                           uint32_t item_id) {
  using A = Acc<T>;
  constexpr int EB = (int)sizeof(typename ElemOf<T>::type);
  constexpr int K = sizeof(T) <= 4 ? 4 : 2;  // elements per lane, in whole 16-byte units
  constexpr int W = K * EB / 4;
  constexpr uint32_t FULL = 0xffffffffu, WIN = 32 * K;
  __shared__ StreamEnds<A> ends;
  T *out = out_base(P, it);
  const bool staged = it.xw > 0;
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t row_end = it.row_end, row_off = it.row_off;
  auto write = [&](uint32_t row, A sum) {
    if (row >= row_end || SP_BAD(P, row < P.nrows, -1015)) return;
    if constexpr (ATOMIC) atomic_add_out<T>(out + row, sum);
    else out[row] = from_acc<T>(sum);
  };
  // rows r0 + from, r0 + from + step, ... below r1, which have no nonzeros
  auto zeros = [&](uint32_t r0, uint32_t r1, uint32_t from, uint32_t step) {
    if (r1 > row_end) r1 = row_end;
    for (uint64_t r = (uint64_t)r0 + from; r < r1; r += step) write((uint32_t)r, A(0));
  };
  if (it.a0 >= it.a1) {  // a tile without nonzeros
    if (!ATOMIC) zeros(it.own0, it.own1, threadIdx.x, blockDim.x);
    if (!GROUPS && !ATOMIC && threadIdx.x == 0) P.carry_idx[item_id] = NO_CARRY;
    return;
  }
  // Positions count from the multiple of 4 elements at or before the item's: the
  // item's are [lead, tn), what lies around them in whole windows counts as
  // zeros of the rows beside.
  const uint64_t e0 = it.a0 & ~3ull;
  const uint64_t lead = it.a0 - e0, tn = it.a1 - e0;
  const uint64_t per = (tn + nw * WIN - 1) / (nw * WIN) * WIN;
  const uint64_t begin = warp * per < tn ? warp * per : tn, end = begin + per < tn ? begin + per : tn;
  const char *el = static_cast<const char *>(P.elems) + e0 * EB;
  const T *xt = xb + it.col_off;
  if (begin < end && !SP_BAD(P, it.a1 <= P.n_elems, -1009)) {
    auto key_at = [&](uint64_t i) { return *reinterpret_cast<const uint32_t *>(el + i * EB); };
    uint32_t w[W];
    auto fetch = [&](uint64_t b) {
      const uint64_t i = b + lane * K;
      if (i >= tn) return;
      if (e0 + i + K <= P.n_elems) {
#pragma unroll
        for (int q = 0; q < W / 4; ++q) {
          const uint4 v = ld_stream4(el + i * EB + 16 * q);
          w[4 * q] = v.x, w[4 * q + 1] = v.y, w[4 * q + 2] = v.z, w[4 * q + 3] = v.w;
        }
      } else {  // the last elements of an array without padding
#pragma unroll
        for (int q = 0; q < W; ++q)
          if (i + q * 4 / EB < tn) w[q] = *reinterpret_cast<const uint32_t *>(el + i * EB + 4 * q);
      }
    };
    RowStream<A> S;
    S.open = key_at(begin > lead ? begin : lead) + row_off;
    if (lane == 0) ends.k0[warp] = S.open;
    uint32_t last = S.open;  // the row of the nonzero before the window
    fetch(begin);
    for (uint64_t b = begin; b < end; b += WIN) {
      uint32_t k[K];
      A v[K];
      {
        T x[K], vx[K];
        const bool edge = b < lead || b + WIN > tn;
#pragma unroll
        for (int j = 0; j < K; ++j) {
          const uint64_t i = b + lane * K + j;
          bool in = !edge || (i >= lead && i < tn);
          k[j] = in ? w[j * EB / 4] + row_off : FULL;
          const uint32_t col = w[j * EB / 4 + 1];
          vx[j] = in ? word_elem<T>(w + j * EB / 4 + 2, 0) : T(0);
          if (SP_BAD(P, !in || x_ok(P, it, (uint64_t)it.col_off + col), -1009)) in = false;
          x[j] = in ? xload(xt, col, staged) : T(0);
        }
        if (b + WIN < end) fetch(b + WIN);
#pragma unroll
        for (int j = 0; j < K; ++j) v[j] = mul<T>(vx[j], x[j]);
      }
      if (b < lead || b + WIN > tn) {
        const uint32_t tail = key_at(tn - 1) + row_off;
#pragma unroll
        for (int j = 0; j < K; ++j)
          if (k[j] == FULL) k[j] = b + lane * K + j < lead ? last : tail;
      }
      uint32_t prev = __shfl_up_sync(FULL, k[K - 1], 1);
      if (lane == 0) prev = last;
      uint32_t hb = k[0] != prev ? 1u : 0u, gap = k[0] - prev;
#pragma unroll
      for (int j = 1; j < K; ++j) {
        const uint32_t d = k[j] - k[j - 1];
        hb |= (d ? 1u : 0u) << j;
        gap = d > gap ? d : gap;
      }
      const uint32_t before = last;
      last = __shfl_sync(FULL, k[K - 1], 31);
      if constexpr (!ATOMIC) {
        // Rows without nonzeros in between: all rows between the window's first and
        // last are zeroed side by side, and those with nonzeros written after that.
        if (__any_sync(FULL, gap > 1)) {
          zeros(before, last, lane + 1, 32);
          __syncwarp();
        }
      }
      row_window<K, A>(S, v, hb, k, &ends.first[warp], write);
    }
    leave_ends<A>(ends, warp, S);
  }
  __syncthreads();
  if (warp != 0 || SP_BAD(P, it.a1 <= P.n_elems, -1009)) return;
  // rows cut by the warps' boundaries, in order (the whole warp follows, lane 0 writes)
  SharedPart<T> first_part, last_part;
  if constexpr (GROUPS) {
    first_part.g = first_row_group(it);
    last_part.g = last_row_group(it);
  }
  uint32_t cur = ends.k0[0];
  A sum = ends.first[0];
  bool first = true;  // `cur` is the item's first row
  auto close = [&]() {
    if (first && first_part.g.n) {
      first_part.row0 = cur;
      first_part.part = sum;
    } else if (lane == 0) {
      write(cur, sum);
    }
    first = false;
  };
  if (!ATOMIC) zeros(it.own0, cur, lane, 32);
  for (int w = 0; w < nw && w * per < tn; ++w) {
    if (w) {
      if (ends.k0[w] == cur) {
        sum += ends.first[w];
      } else {
        close();
        if (!ATOMIC) zeros(cur, ends.k0[w], lane + 1, 32);
        cur = ends.k0[w];
        sum = ends.first[w];
      }
    }
    if (ends.heads[w]) {
      close();
      cur = ends.k1[w];
      sum = ends.last[w];
    }
  }
  if constexpr (GROUPS) {
    if (last_part.g.n) {  // goes on in the next item
      if (first) first_part.g.n = 0;  // and came from the one before
      last_part.row0 = cur;
      last_part.part = sum;
    } else {
      close();
      if (!ATOMIC) zeros(cur, it.own1, lane + 1, 32);
    }
    if (first_part.g.n + last_part.g.n) arrive<T, 1>(P, out, item_id, row_end, first_part, last_part);
  } else if (ATOMIC || cur < it.own1) {
    if (lane == 0) {
      write(cur, sum);
      if (!ATOMIC) P.carry_idx[item_id] = NO_CARRY;
    }
    if (!ATOMIC) zeros(cur, it.own1, lane + 1, 32);
  } else if (lane == 0) {
    P.carry_idx[item_id] = cur < row_end ? out_index(P, it, cur) : NO_CARRY;
    P.carry_val[item_id] = acc_bits(sum);
  }
}

template <typename T, bool ATOMIC> __global__ void __launch_bounds__(512) coo_items(Params<T> P) {
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  __shared__ uint64_t xbar;
  const Item it = P.items[blockIdx.x];
  const T *xb = P.x;
  if (it.xw > 0 && it.a0 < it.a1) {
    uint32_t phase = 0;
    mbar_init(&xbar);
    xb = stage_x<T>(P.x, it.xlo, it.xw, dyn_smem, &xbar, phase, P.err, P.smem_bytes,
                    reinterpret_cast<uintptr_t>(P.x + P.n_xalloc), P.fault_wait);
  }
  coo_stream<T, !ATOMIC, ATOMIC>(P, it, xb, blockIdx.x);
}

// ---------------------------------------------------------------------------
// BCOO in chunks of up to S blocks (sorted by block row), 2x2, 4x4 and 8x8:
// values and block indices come into shared memory by bulk copies, the block
// rows' starts are found there (a ballot per 32 blocks and a scan of the
// ballots), and then the block rows are summed as BCSR's are.  INT16 4x4, 1M rows,
// 20 blocks per block row (204 MB): a block per thread and block-wide scans of
// 4-wide sums 291 us, this 76 us.
// ---------------------------------------------------------------------------
template <typename T, int RB, int CB> struct BcooStage {
  using G = Pieces<T, RB, CB>;
  static constexpr int S = (int)bcoo_chunk_blocks(RB, CB, sizeof(T));
  static constexpr int IND = (S + 8) * G::B, RUN = IND + (S + 8) * (int)sizeof(sparsep_bind);
  static constexpr int SMEM = (RUN + (S + 1) * 4 + 127) / 128 * 128;
  static_assert(S <= 1024, "a warp scans the chunk's ballots");
};

template <typename T, int RB, int CB>
__global__ void __launch_bounds__(512, 3) bcoo_chunks(Params<T> P) {
  using A = Acc<T>;
  using G = Pieces<T, RB, CB>;
  using St = BcooStage<T, RB, CB>;
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  __shared__ uint64_t bar, xbar;
  __shared__ uint32_t ballots[St::S / 32 + 1];
  __shared__ A s_first[RB], s_last[RB];
  unsigned char *sm = dyn_smem + (P.smem_bytes + 127) / 128 * 128;  // behind a tile's staged x
  const Item it = P.items[blockIdx.x];
  T *out = out_base(P, it);
  const bool atomic = P.out_mode == OUT_ATOMIC;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t n = (uint32_t)(it.a1 - it.a0);
  const uint64_t A0 = it.a0 & ~3ull, A1 = (it.a1 + 3) & ~3ull;  // the arrays are padded past their end
  const RowGroup ga = first_row_group(it), gb = last_row_group(it);
  auto row_of = [&](uint64_t key) { return (uint64_t)it.row_off + key * RB; };
  auto zero_rows = [&](uint64_t r0, uint64_t r1) {  // by the whole CTA
    if (!atomic)
      for (uint64_t r = r0 + threadIdx.x; r < r1 && r < it.row_end; r += blockDim.x) put<T>(P, out, r, A(0));
  };
  if (n == 0) {
    zero_rows(row_of(it.own0), row_of(it.own1));
    return;
  }
  bool good = !SP_BAD(P, A1 <= P.n_elems && A1 * (RB * CB) <= P.n_val && n <= St::S, -1014);
  mbar_init(&bar);
  if (threadIdx.x == 0 && good) {
    const uint32_t m = (uint32_t)(A1 - A0);
    expect_bytes(&bar, m * (uint32_t)(G::B + sizeof(sparsep_bind)));
    bulk_load(sm + St::IND, P.bind + A0, m * (uint32_t)sizeof(sparsep_bind), &bar);
    bulk_load(sm, reinterpret_cast<const char *>(P.bval) + A0 * G::B, m * G::B, &bar);
  }
  const T *xb = P.x;
  if (it.xw > 0) {
    uint32_t phase = 0;
    mbar_init(&xbar);
    xb = stage_x<T>(P.x, it.xlo, it.xw, dyn_smem, &xbar, phase, P.err, P.smem_bytes,
                    reinterpret_cast<uintptr_t>(P.x + P.n_xalloc), P.fault_wait);
  }
  if (good) good = cta_wait(&bar, 0, P.err);
  // parts of the first and last block row that other items share (one and the
  // same block row counts as the last)
  SharedPart<T> first_part{ga, 0, A(0)}, last_part{gb, 0, A(0)};
  if (gb.n && ga.cnt == gb.cnt) first_part.g.n = 0;
  if (!good) {  // give the item up, but arrive
    first_part.row0 = row_of(it.own0);
    last_part.row0 = row_of(it.own1);
    if (warp == 0 && ga.n + gb.n) arrive<T, RB>(P, out, blockIdx.x, it.row_end, first_part, last_part);
    return;
  }
  const uint32_t lead = (uint32_t)(it.a0 - A0);
  const sparsep_bind *ind = reinterpret_cast<const sparsep_bind *>(sm + St::IND) + lead;
  uint32_t *run = reinterpret_cast<uint32_t *>(sm + St::RUN);
  // block rows' first blocks, in order
  const uint32_t words = (n + 31) / 32;
  bool gap = false;  // a block row without blocks before this thread's
  for (uint32_t b = threadIdx.x; b < words * 32; b += blockDim.x) {
    const uint32_t step = b == 0 ? 1u : b < n ? ind[b].rowind - ind[b - 1].rowind : 0u;
    gap |= step > 1;
    const uint32_t m = __ballot_sync(0xffffffffu, step != 0);
    if (lane == 0) ballots[b / 32] = m;
  }
  // Rows without blocks between the chunk's first and last block row: the CTA zeroes
  // all rows in between side by side, and those with blocks are written after the next
  // barrier.  A thread per gap took 2.3 ms for 40 block rows 20,000 rows apart (FP32 4x4).
  if (__syncthreads_or(gap)) zero_rows(row_of((uint64_t)ind[0].rowind + 1), row_of(ind[n - 1].rowind));
  const uint32_t mine = lane < words ? ballots[lane] : 0u;
  uint32_t before = __popc(mine);  // inclusive, then exclusive
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, before, d);
    if (lane >= d) before += o;
  }
  const uint32_t k = __shfl_sync(0xffffffffu, before, 31);  // block rows
  before -= __popc(mine);
  for (uint32_t b = threadIdx.x; b < words * 32; b += blockDim.x) {
    const uint32_t m = __shfl_sync(0xffffffffu, mine, b / 32);
    const uint32_t at = __shfl_sync(0xffffffffu, before, b / 32);
    if ((m >> lane) & 1u) run[at + __popc(m & ((1u << lane) - 1u))] = b;
  }
  if (threadIdx.x == 0) run[k] = n;
  __syncthreads();
  // and rows of no block before the first and after the last block row
  zero_rows(row_of(it.own0), row_of(ind[0].rowind));
  if (!gb.n) zero_rows(row_of((uint64_t)ind[n - 1].rowind + 1), row_of(it.own1));
  const T *xt = xb + it.col_off;
  const uint32_t *scol = &ind[0].colind;
  const bool whole = x_whole<T, RB, CB, 2>(P, it, xt, scol, n);
  block_rows_any<T, RB, CB, 2>(P, it, xt, k, run, sm + lead * G::B, scol, it.lanes, whole,
                               [&](uint32_t i, uint32_t r, A sum) {
                                 if (i + 1 == k && gb.n) {
                                   s_last[r] = sum;
                                 } else if (i == 0 && ga.n) {
                                   s_first[r] = sum;
                                 } else {
                                   const uint64_t row = row_of(ind[run[i]].rowind) + r;
                                   if (row < it.row_end) put<T>(P, out, row, sum);
                                 }
                               });
  if (!ga.n && !gb.n) return;
  __syncthreads();
  if (warp != 0) return;
  first_part.row0 = row_of(ind[0].rowind);
  last_part.row0 = row_of(ind[n - 1].rowind);
  if (lane < RB) first_part.part = s_first[lane], last_part.part = s_last[lane];
  arrive<T, RB>(P, out, blockIdx.x, it.row_end, first_part, last_part);
}

// ---------------------------------------------------------------------------
// BCOO blocks of the other sizes (rb <= BCOO_W): block segmented scan, a block
// per thread.  Keys are tile-local block rows (row = row_off + key * rb + r).
// The item writes every row of block rows [own0, own1): sums of complete runs,
// zeros for block rows without blocks; a run reaching own1 is a carry for the
// fix-up.
// ---------------------------------------------------------------------------
constexpr int BCOO_W = 16;

template <typename T>
__device__ __forceinline__ void zero_block_rows(const Params<T> &P, const Item &it, T *out, long long k0,
                                                long long k1) {
  // keys strictly inside (k0, k1)
  for (long long k = k0 + 1; k < k1; ++k)
    for (uint32_t r = 0; r < P.rb; ++r) {
      const uint64_t row = (uint64_t)it.row_off + (uint64_t)k * P.rb + r;
      if (row < it.row_end && !SP_BAD(P, row < P.nrows, -1015)) out[row] = T(0);
    }
}

template <typename T>
__device__ __forceinline__ void write_run(const Params<T> &P, const Item &it, T *out, long long key,
                                          const Acc<T> (&v)[BCOO_W], bool atomic) {
#pragma unroll
  for (int r = 0; r < BCOO_W; ++r) {
    if (r >= (int)P.rb) break;
    const uint64_t row = (uint64_t)it.row_off + (uint64_t)key * P.rb + r;
    if (row >= it.row_end) continue;
    if (SP_BAD(P, row < P.nrows, -1015)) continue;
    if (atomic) atomic_add_out<T>(out + row, v[r]);
    else out[row] = from_acc<T>(v[r]);
  }
}

template <typename T>
__device__ void bcoo_lf(const Params<T> &P, const Item &it, const T *__restrict__ xb, uint32_t item_id, uint32_t cw) {
  // cw = carry slots per item (rb), the scratch stride
  using A = Acc<T>;
  constexpr int W = BCOO_W;
  using KVT = KV<A, W>;
  __shared__ KVT scan_smem[32];
  __shared__ KVT tail_smem;
  __shared__ long long keys_smem[512];
  T *out = out_base(P, it);
  const uint64_t lo = it.a0, hi = it.a1;
  const bool atomic = P.out_mode == OUT_ATOMIC;

  if (SP_BAD(P, (uint64_t)(item_id + 1) * cw <= P.n_carry || atomic, -1018)) return;
  if (lo >= hi) {  // empty: only zero the owned rows
    if (!atomic && threadIdx.x == 0) zero_block_rows<T>(P, it, out, (long long)it.own0 - 1, it.own1);
    if (!atomic && threadIdx.x < cw) P.carry_idx[(uint64_t)item_id * cw + threadIdx.x] = NO_CARRY;
    return;
  }
  KVT carry;
  carry.k = (long long)it.own0 - 1;
#pragma unroll
  for (int i = 0; i < W; ++i) carry.v[i] = A(0);

  for (uint64_t cg = lo; cg < hi; cg += blockDim.x) {
    const uint64_t g = cg + threadIdx.x;
    KVT mine;
    mine.k = LLONG_MAX;
#pragma unroll
    for (int i = 0; i < W; ++i) mine.v[i] = A(0);
    if (g < hi && !SP_BAD(P, g < P.n_elems, -1014)) {
      const sparsep_bind bi = P.bind[g];
      mine.k = (long long)bi.rowind;
      block_mv<T, 0, 0>(P, xb, g, bi.colind, it.col_off, mine.v, it);
    }
    const bool any = mine.k != LLONG_MAX;
    keys_smem[threadIdx.x] = mine.k;  // read after the scan's barriers
    KVT ex, in;
    block_seg_scan<A, W>(mine, carry, ex, in, scan_smem);
    const uint64_t last_g = (hi < cg + blockDim.x ? hi : cg + blockDim.x) - 1;
    // a run is complete when the next thread starts another key; the chunk's
    // last thread hands its run on instead
    if (any && g != last_g && keys_smem[threadIdx.x + 1] != mine.k) write_run<T>(P, it, out, mine.k, in.v, atomic);
    // likewise the run handed over by the previous chunk
    if (threadIdx.x == 0 && carry.k >= (long long)it.own0 && mine.k != carry.k)
      write_run<T>(P, it, out, carry.k, carry.v, atomic);
    if (any && !atomic) zero_block_rows<T>(P, it, out, ex.k, mine.k);
    // the chunk's last thread with a block hands its run to the next chunk
    if (g == last_g) tail_smem = in;
    __syncthreads();
    carry = tail_smem;
    __syncthreads();
  }
  // final run of the item
  if (threadIdx.x == 0) {
    if (atomic) {
      write_run<T>(P, it, out, carry.k, carry.v, true);
    } else if (carry.k < (long long)it.own1) {
      write_run<T>(P, it, out, carry.k, carry.v, false);
      zero_block_rows<T>(P, it, out, carry.k, it.own1);
      for (uint32_t i = 0; i < cw; ++i) P.carry_idx[(uint64_t)item_id * cw + i] = NO_CARRY;
    } else {
      for (uint32_t i = 0; i < cw && i < (uint32_t)W; ++i) {
        const uint64_t row = (uint64_t)it.row_off + (uint64_t)carry.k * P.rb + i;
        const bool ok = i < P.rb && row < it.row_end;
        P.carry_idx[(uint64_t)item_id * cw + i] = ok ? out_index(P, it, row) : NO_CARRY;
        P.carry_val[(uint64_t)item_id * cw + i] = acc_bits(carry.v[i]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Carry fix-up, run by the last CTA to finish: slot runs with the same target
// are summed in item order, then added once (deterministic).
// ---------------------------------------------------------------------------
template <typename T>
__device__ void carry_fixup(const Params<T> &P, uint32_t nslots, uint32_t W) {
  using A = Acc<T>;
  constexpr int U = 4;  // slots a thread reads in one round trip
  for (uint32_t s0 = threadIdx.x; s0 < nslots; s0 += U * blockDim.x) {
    unsigned long long idx[U], prev[U], val[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t s = s0 + u * blockDim.x;
      const bool in = s < nslots;
      idx[u] = in ? __ldcg(P.carry_idx + s) : NO_CARRY;
      prev[u] = in && s >= W ? __ldcg(P.carry_idx + s - W) : NO_CARRY;
      val[u] = in ? __ldcg(P.carry_val + s) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t s = s0 + u * blockDim.x;
      if (idx[u] == NO_CARRY || prev[u] == idx[u]) continue;  // none, or not the first of its run
      if (SP_BAD(P, idx[u] < (uint64_t)P.nslots * P.nrows, -1016)) continue;
      A sum = bits_acc<A>(val[u]);
      for (uint32_t t = s + W; t < nslots && __ldcg(P.carry_idx + t) == idx[u]; t += W)
        sum += bits_acc<A>(__ldcg(P.carry_val + t));
      T *p = (P.out_mode == OUT_PARTIAL ? P.part : P.y) + idx[u];
      T cur = __ldcg(p);
      *p = from_acc<T>(to_acc<T>(cur) + sum);
    }
  }
}

// ---------------------------------------------------------------------------
// The item kernel
// ---------------------------------------------------------------------------
template <typename T, int FMT, int RB, int CB, int CAP>
__global__ void __launch_bounds__(512) spmv_items(Params<T> P, uint32_t carry_w) {
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  __shared__ uint64_t mbar;
  __shared__ uint32_t is_last;
  const uint32_t item_id = blockIdx.x;
  const Item it = P.items[item_id];
  const T *xb = P.x;
  if (it.xw > 0) {
    uint32_t phase = 0;
    mbar_init(&mbar);
    xb = stage_x<T>(P.x, it.xlo, it.xw, dyn_smem, &mbar, phase, P.err, P.smem_bytes,
                    reinterpret_cast<uintptr_t>(P.x + P.n_xalloc), P.fault_wait);
  }

  if constexpr (FMT == SPARSEP_FMT_CSR) {
    if (it.kind == ITEM_LONG) {
      csr_long<T>(P, it, xb, item_id);
    } else {
      switch (it.lanes) {
        case 0: csr_stream<T, CAP>(P, it, xb); break;
        case 1: csr_rows<T, 1>(P, it, xb); break;
        case 2: csr_rows<T, 2>(P, it, xb); break;
        case 4: csr_rows<T, 4>(P, it, xb); break;
        case 8: csr_rows<T, 8>(P, it, xb); break;
        case 16: csr_rows<T, 16>(P, it, xb); break;
        default: csr_rows<T, 32>(P, it, xb); break;
      }
    }
  } else if constexpr (FMT == SPARSEP_FMT_BCSR) {
    switch (it.lanes) {
      case 1: bcsr_rows<T, RB, CB, 1>(P, it, xb); break;
      case 2: bcsr_rows<T, RB, CB, 2>(P, it, xb); break;
      case 4: bcsr_rows<T, RB, CB, 4>(P, it, xb); break;
      case 8: bcsr_rows<T, RB, CB, 8>(P, it, xb); break;
      case 16: bcsr_rows<T, RB, CB, 16>(P, it, xb); break;
      default: bcsr_rows<T, RB, CB, 32>(P, it, xb); break;
    }
  } else {
    bcoo_lf<T>(P, it, xb, item_id, carry_w);
  }

  // lock-free carries: the last CTA to finish adds them (threadfence reduction)
  if (P.carry_idx != nullptr && P.out_mode != OUT_ATOMIC) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned int ticket = atomicAdd(P.done, 1u);
      is_last = (ticket == P.nitems - 1);
    }
    __syncthreads();
    if (is_last) {
      __threadfence();
      carry_fixup<T>(P, P.nitems * carry_w, carry_w);
      if (threadIdx.x == 0) *P.done = 0;
    }
  }

  // Host-buffer path: the item is counted in its row band once all of its
  // writes to y are visible device-wide (barrier, then one fence before the
  // count: the fence is cumulative over the writes the barrier ordered before
  // it); a copy stream waiting on the band's count moves those rows to the
  // host while later items still run.
  if (P.band_cnt != nullptr) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(P.band_cnt + P.items[item_id].band, 1u);  // re-read: keeps the band out of the body's registers
    }
  }
}

// ---------------------------------------------------------------------------
// 2D merge of per-stripe partial y, in stripe order like the reference's host
// merge (spmv/2D/BDCSR/host/app.c:437-447, spmv/2D/DCSR/host/app.c:340-351).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void merge_partials(const T *__restrict__ part, T *__restrict__ y, uint32_t nrows, uint32_t V) {
  for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += (uint64_t)gridDim.x * blockDim.x) {
    Acc<T> s = to_acc<T>(__ldcs(part + r));
    for (uint32_t c = 1; c < V; ++c) {
      if constexpr (std::is_floating_point<T>::value) s = (T)(s + __ldcs(part + (uint64_t)c * nrows + r));
      else s += to_acc<T>(__ldcs(part + (uint64_t)c * nrows + r));
    }
    y[r] = from_acc<T>(s);
  }
}


}  // namespace sparsep
