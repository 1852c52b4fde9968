// csr2bcsr_dev.cu -- CSR -> BCSR on the device, with the arrays the host
// converter csr2bcsr produces (formats.cpp; the reference's csr2bcsr +
// sortBCSRMatrix + countNNZperBlockBCSRMatrix,
// spmv/1D/BCSR-nnz/support/matrix.h:202-485): per block row the blocks sorted
// by block column, each block a row-major rb x cb array in which a later
// duplicate entry of a position overwrites an earlier one, and
// nnz_per_block[b] = the block's entries != 0.
//
// A block row's nonzeros are consecutive in the CSR, so nothing is sorted
// globally: a warp takes a block row and finds its block columns with a hash table
// in shared memory.
// layout (type-independent, sparsep_bcsr_layout_device):
//   count  per block row, its distinct block columns; rowptr and columns checked
//   scan   of the counts -> browptr
// fill (per element type, sparsep_csr2bcsr_device_<t>):
//   the block columns again, ranked; the blocks put together in shared memory
//   where they fit (else in place), 32 nonzeros at a time in input order, so that
//   a later duplicate of a position overwrites an earlier one; the nonzero values
//   of each block counted.
// Matrices with a block row of more than LIM nonzeros go through a sort of
// all nonzeros by (block row, block column) instead (radix.cuh):
//   keys   per nonzero k: its row r (binary search in rowptr) and the key
//          (r / rb) << jbits | colind[k] / cb
//   sort   stable, carrying k, so that the entries of one block stay in input order
//   heads  a block starts where the sorted key changes: exclusive scan of the
//          head flags -> block start positions and block keys
//   fill   browptr by lower bound among the block keys, one thread per block
// FP32, 10.5 M nonzeros in 1 M blocks of 4x4 (COO -> CSR -> BCSR as one ingest): 8.1
// ms with the sort for every matrix and scratch from cudaMalloc, of which 1.9 ms in
// kernels; 0.67 ms now, of which layout 0.12 and fill 0.16 ms (fill_rows 134 us, bound
// by its instructions: 850 for a block row of 80 nonzeros).  With longer block rows, by
// the sort: 98 M nonzeros (2 M rows, banded, block rows around 190 and up to more than
// 256) 13.7 ms, 20.6 with the earlier sort.
#include <algorithm>
#include <cstdio>
#include <new>

#include "fault.hpp"
#include "internal.hpp"
#include "radix.cuh"
#include "sparsep.h"

namespace sparsep {
namespace c2b {

constexpr int NT = 256;

// rowptr[0] == 0, non-decreasing, rowptr[nrows] == nnz
__global__ void check_rowptr(const uint32_t *__restrict__ rowptr, uint32_t nrows, uint32_t nnz, int *__restrict__ bad) {
  for (uint64_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += gridDim.x * blockDim.x)
    if (rowptr[r] > rowptr[r + 1]) atomicExch(bad, 1);
  if (blockIdx.x == 0 && threadIdx.x == 0 && (rowptr[0] != 0 || rowptr[nrows] != nnz)) atomicExch(bad, 1);
}

// ---------------------------------------------------------------------------
// A block row per warp
// ---------------------------------------------------------------------------
// Nonzeros of a block row that go through a table.  Layout and fill of 4 M nonzeros,
// 4x4, block rows of 250: 665 us with scattered columns (250 blocks each), 172 with
// 32 blocks each; by the sort, block rows of 260: 840 and 550 us.  A table for up to
// 2048, a warp per block row with its block columns ranked pair by pair, was slower than
// the sort at once: 3.5 ms at 260 scattered nonzeros, 70 at 2000.
constexpr int LIM = 256;
constexpr uint32_t EMPTY = 0xFFFFFFFFu;  // no block column: columns are below 2^32 - 1
constexpr int SLOTS = 2 * LIM;
constexpr int WARPS = 4;      // block rows per CTA
constexpr int BLOCKS = 2048;  // bytes for a block row's blocks

struct BlockRow {
  uint32_t r0, k0, k1;  // first row, nonzeros [k0, k1)
};
// Block row I of a CSR whose rowptr may be malformed (checked elsewhere): ranges
// stay inside the arrays.
__device__ __forceinline__ BlockRow block_row(const uint32_t *__restrict__ rowptr, uint32_t nrows, uint32_t nnz,
                                              uint32_t rb, uint32_t I) {
  const uint64_t r0 = (uint64_t)I * rb, r1 = r0 + rb < nrows ? r0 + rb : nrows;
  BlockRow b;
  b.r0 = (uint32_t)r0;
  b.k0 = rowptr[r0] < nnz ? rowptr[r0] : nnz;
  b.k1 = rowptr[r1] < nnz ? rowptr[r1] : nnz;
  if (b.k1 < b.k0) b.k1 = b.k0;
  return b;
}
__device__ __forceinline__ uint32_t block_col(uint32_t c, uint32_t cb, int cshift) {
  return cshift >= 0 ? c >> cshift : c / cb;
}
// Slots used of a table for m nonzeros (a power of two, at least 2 m), as a shift
// of the 32-bit hash.
__device__ __forceinline__ int table_shift(uint32_t m) { return m <= 16 ? 27 : __clz(2 * m - 1); }
__device__ __forceinline__ uint32_t hash(uint32_t J, int shift) { return (J * 0x9E3779B1u) >> shift; }
// The slot of J; *fresh: it was not there before.
__device__ __forceinline__ uint32_t insert(uint32_t *t, uint32_t J, int shift, bool *fresh) {
  const uint32_t mask = (1u << (32 - shift)) - 1u;
  for (uint32_t s = hash(J, shift);; s = (s + 1) & mask) {  // at least half of the slots stay empty
    uint32_t old = *(volatile uint32_t *)(t + s);
    if (old == EMPTY) old = atomicCAS(t + s, EMPTY, J);
    if (old == EMPTY || old == J) {
      *fresh = old == EMPTY;
      return s;
    }
  }
}
__device__ __forceinline__ uint32_t find(const uint32_t *t, uint32_t J, int shift) {  // J is in the table
  const uint32_t mask = (1u << (32 - shift)) - 1u;
  uint32_t s = hash(J, shift);
  for (uint32_t i = 0; i < mask && t[s] != J; ++i) s = (s + 1) & mask;
  return s;
}
// Calls f(I) with the whole warp for every block row I.
template <typename F> __device__ __forceinline__ void each_block_row(uint32_t nbr, F f) {
  for (uint64_t I = (uint64_t)blockIdx.x * WARPS + (threadIdx.x >> 5); I < nbr; I += (uint64_t)gridDim.x * WARPS)
    f((uint32_t)I);
}

// cnt[I] = blocks of block row I, for block rows of up to LIM nonzeros; flag[0]: a
// bad column among these, flag[1]: a longer block row.
__global__ void __launch_bounds__(32 * WARPS)
    count_blocks(const uint32_t *__restrict__ rowptr, uint32_t nrows, const uint32_t *__restrict__ colind, uint32_t nnz,
                 uint32_t ncols, uint32_t rb, uint32_t cb, int cshift, uint32_t nbr, uint32_t *__restrict__ cnt,
                 int *__restrict__ flag) {
  __shared__ uint32_t table[WARPS][SLOTS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  each_block_row(nbr, [&](uint32_t I) {
    const BlockRow br = block_row(rowptr, nrows, nnz, rb, I);
    const uint32_t m = br.k1 - br.k0;
    if (m > LIM && lane == 0) flag[1] = 1;
    if (m == 0 && lane == 0) cnt[I] = 0;
    if (m == 0 || m > LIM) return;
    const int shift = table_shift(m);
    uint32_t *t = table[warp];
    for (uint32_t i = lane; i < 1u << (32 - shift); i += 32) t[i] = EMPTY;
    __syncwarp();
    uint32_t mine = 0;
    for (uint32_t i = lane; i < m; i += 32) {  // k0 + i of a lane past the end may pass 2^32: compare i
      uint32_t c = colind[br.k0 + i];
      if (c >= ncols) {
        flag[0] = 1;
        c = 0;
      }
      bool fresh;
      insert(t, block_col(c, cb, cshift), shift, &fresh);
      mine += fresh;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) cnt[I] = mine;
    __syncwarp();
  });
}

template <typename T>
__global__ void __launch_bounds__(32 * WARPS)
    fill_rows(const uint32_t *__restrict__ rowptr, uint32_t nrows, const uint32_t *__restrict__ colind, uint32_t nnz,
              uint32_t ncols, const T *__restrict__ values, uint32_t rb, uint32_t cb, int cshift, uint32_t nbr,
              const uint32_t *__restrict__ browptr, uint32_t *__restrict__ bcolind, T *__restrict__ bval,
              uint32_t *__restrict__ nnz_per_block) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ uint32_t table[WARPS][SLOTS];
  __shared__ uint16_t rank_of[WARPS][SLOTS];
  __shared__ uint32_t list[WARPS][LIM];
  __shared__ uint32_t count[WARPS];
  __shared__ __align__(16) unsigned char blocks[WARPS][BLOCKS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t *t = table[warp], *l = list[warp];
  uint16_t *rk = rank_of[warp];
  const uint64_t bs = (uint64_t)rb * cb;
  each_block_row(nbr, [&](uint32_t I) {
    const BlockRow br = block_row(rowptr, nrows, nnz, rb, I);
    const uint32_t m = br.k1 - br.k0;
    if (m == 0 || m > LIM) return;
    const int shift = table_shift(m);
    // all that memory has to give, at once: the first nonzeros, the rows' ends and the blocks' place
    constexpr int PRE = 4;
    uint32_t pc[PRE];
    T pv[PRE];
#pragma unroll
    for (int q = 0; q < PRE; ++q) {
      const uint32_t i = q * 32 + lane;
      pc[q] = 0;
      pv[q] = T(0);
      if (i < m) {
        pc[q] = colind[br.k0 + i];
        pv[q] = values[br.k0 + i];
      }
    }
    const uint32_t rend = lane < rb && br.r0 + lane + 1 <= nrows ? rowptr[br.r0 + lane + 1] : 0xFFFFFFFFu;
    const uint32_t b0 = browptr[I], room = browptr[I + 1] - b0;
    for (uint32_t i = lane; i < 1u << (32 - shift); i += 32) t[i] = EMPTY;
    if (lane == 0) count[warp] = 0;
    __syncwarp();
    auto enter = [&](uint32_t c) {
      const uint32_t J = block_col(c < ncols ? c : 0, cb, cshift);
      bool fresh;
      const uint32_t slot = insert(t, J, shift, &fresh);
      if (fresh) l[atomicAdd(&count[warp], 1u)] = J;
      return slot;
    };
    uint32_t ps[PRE];
#pragma unroll
    for (int q = 0; q < PRE; ++q) {
      ps[q] = 0;
      if (q * 32 + lane < m) ps[q] = enter(pc[q]);
    }
    for (uint32_t i = PRE * 32 + lane; i < m; i += 32) enter(colind[br.k0 + i]);
    __syncwarp();
    const uint32_t D = count[warp] < room ? count[warp] : room;  // equal, while colind is as it was counted
    for (uint32_t d = lane; d < D; d += 32) {
      const uint32_t J = l[d];
      uint32_t r = 0;
#pragma unroll 4
      for (uint32_t e = 0; e < D; ++e) r += l[e] < J;
      rk[find(t, J, shift)] = (uint16_t)r;
      if (r < room) bcolind[b0 + r] = J;
    }
    __syncwarp();
    // the blocks: in shared memory where they fit, else where they belong
    T *gout = bval + b0 * bs;
    const uint64_t ne = D * bs;
    const bool in_smem = ne * sizeof(T) <= (uint64_t)BLOCKS;
    T *blk = in_smem ? reinterpret_cast<T *>(blocks[warp]) : gout;
    for (uint64_t e = lane; e < ne; e += 32) blk[e] = T(0);
    __syncwarp();
    // The list is done with: which lane came to a position.  Matching 64-bit positions
    // in every group of 32 cost FP32 4x4 65 us of 222 (10.5 M nonzeros).
    unsigned char *tag = reinterpret_cast<unsigned char *>(l);
    auto place_all = [&](auto zero) {  // positions as wide as this
      using P = decltype(zero);
      const P nel = (P)ne, bsz = (P)bs;
      auto place = [&](uint32_t i, uint32_t c, T v, auto slot_of) {  // nonzeros [k0 + i, k0 + i + 32)
        const bool in = i + lane < m;
        const uint32_t k = br.k0 + i + lane;
        uint32_t rl = 0;  // row in the block: the block row's rows that end at or before this nonzero
        if (rb <= 32) {
          for (uint32_t q = 0; q + 1 < rb; ++q) rl += __shfl_sync(FULL, rend, q) <= k;
        } else if (in) {
          uint32_t a = 0, b = rb - 1;
          while (a < b) {
            const uint32_t mid = (a + b) >> 1;
            const uint64_t r = (uint64_t)br.r0 + mid + 1;
            if (r <= nrows && rowptr[r] <= k) a = mid + 1; else b = mid;
          }
          rl = a;
        }
        P pos = ~(P)lane;  // its own, for lanes without a nonzero
        if (in) {
          if (c >= ncols) c = 0;
          const uint32_t J = block_col(c, cb, cshift);
          pos = rk[slot_of(J)] * bsz + (P)rl * cb + (c - J * cb);
        }
        bool last = in && pos < nel;  // of the lanes with this position, the last
        bool twice = true;            // there may be two lanes with one position
        if (nel <= sizeof(list[warp])) {
          if (last) tag[pos] = (unsigned char)lane;
          __syncwarp();
          twice = __any_sync(FULL, last && tag[pos] != lane);
        }
        if (twice) last &= lane == 31 - __clz(__match_any_sync(FULL, pos));
        if (last) blk[pos] = v;
        __syncwarp();
      };
      // input order: a later duplicate wins
#pragma unroll
      for (int q = 0; q < PRE; ++q)
        if (q * 32 < m) place(q * 32, pc[q], pv[q], [&](uint32_t) { return ps[q]; });
      for (uint32_t i = PRE * 32; i < m; i += 32) {
        const bool in = i + lane < m;
        place(i, in ? colind[br.k0 + i + lane] : 0, in ? values[br.k0 + i + lane] : T(0),
              [&](uint32_t J) { return find(t, J, shift); });
      }
    };
    if (in_smem) place_all(0u); else place_all(0ull);
    if (bs <= 32 && (bs & (bs - 1)) == 0 && in_smem) {  // 32 / bs blocks at a time
      const uint32_t nel = (uint32_t)ne, b32 = (uint32_t)bs, s32 = __ffs(b32) - 1;
      for (uint32_t e = lane; e - lane < nel; e += 32) {
        const uint32_t some = __ballot_sync(FULL, e < nel && blk[e] != T(0));
        if (e < nel && (e & (b32 - 1)) == 0)
          nnz_per_block[b0 + (e >> s32)] = __popc(some >> lane & (0xFFFFFFFFu >> (32 - b32)));
      }
    } else for (uint32_t d = lane; d < D; d += 32) {
      uint32_t nz = 0;
      for (uint32_t q = 0, e = d % (uint32_t)bs; q < bs; ++q) {  // lanes start apart: other banks
        nz += blk[d * bs + e] != T(0);
        e = e + 1 == bs ? 0 : e + 1;
      }
      nnz_per_block[b0 + d] = nz;
    }
    if (in_smem) {
      const uint64_t bytes = ne * sizeof(T);
      if (((reinterpret_cast<uintptr_t>(gout) | bytes) & 15) == 0) {
        const uint4 *src = reinterpret_cast<const uint4 *>(blk);
        for (uint64_t e = lane; e < bytes / 16; e += 32) reinterpret_cast<uint4 *>(gout)[e] = src[e];
      } else {
        for (uint64_t e = lane; e < ne; e += 32) gout[e] = blk[e];
      }
    }
    __syncwarp();
  });
}

// ---------------------------------------------------------------------------
// All nonzeros sorted by block
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(NT) keys(const uint32_t *__restrict__ rowptr, uint32_t nrows,
                                           const uint32_t *__restrict__ colind, uint32_t nnz, uint32_t ncols,
                                           uint32_t rb, uint32_t cb, int jbits, uint64_t *__restrict__ key,
                                           uint32_t *__restrict__ row, int *__restrict__ bad) {
  for (uint32_t k = blockIdx.x * NT + threadIdx.x; k < nnz; k += gridDim.x * NT) {
    uint32_t lo = 0, hi = nrows - 1;  // last row whose start is <= k
    while (lo < hi) {
      const uint32_t mid = lo + ((hi - lo + 1) >> 1);
      if (rowptr[mid] <= k) lo = mid;
      else hi = mid - 1;
    }
    uint32_t c = colind[k];
    if (c >= ncols) {
      atomicExch(bad, 1);
      c = 0;
    }
    row[k] = lo;
    key[k] = ((uint64_t)(lo / rb) << jbits) | (c / cb);
  }
}

__global__ void __launch_bounds__(NT) head_flags(const uint64_t *__restrict__ skey, uint32_t n,
                                                 uint32_t *__restrict__ flag) {
  for (uint32_t i = blockIdx.x * NT + threadIdx.x; i < n; i += gridDim.x * NT)
    flag[i] = (i == 0 || skey[i] != skey[i - 1]) ? 1u : 0u;
}

// excl = exclusive scan of the head flags: block excl[i] starts at sorted position i
__global__ void __launch_bounds__(NT) block_starts(const uint64_t *__restrict__ skey, uint32_t n,
                                                   const uint32_t *__restrict__ excl, uint32_t *__restrict__ bstart,
                                                   uint64_t *__restrict__ bkey, uint32_t *__restrict__ nblocks) {
  for (uint32_t i = blockIdx.x * NT + threadIdx.x; i < n; i += gridDim.x * NT) {
    const bool head = i == 0 || skey[i] != skey[i - 1];
    if (head) {
      bstart[excl[i]] = i;
      bkey[excl[i]] = skey[i];
    }
    if (i == n - 1) {
      const uint32_t nb = excl[i] + (head ? 1u : 0u);
      bstart[nb] = n;
      *nblocks = nb;
    }
  }
}

// browptr[I] = number of blocks in block rows < I, I = 0 .. nbr
__global__ void browptr_kernel(const uint64_t *__restrict__ bkey, uint32_t nblocks, uint32_t nbr, int jbits,
                               uint32_t *__restrict__ browptr) {
  const uint32_t I = blockIdx.x * blockDim.x + threadIdx.x;
  if (I > nbr) return;
  const uint64_t want = (uint64_t)I << jbits;
  uint32_t lo = 0, hi = nblocks;
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (bkey[mid] < want) lo = mid + 1;
    else hi = mid;
  }
  browptr[I] = lo;
}

template <typename T>
__global__ void __launch_bounds__(NT) fill_blocks(const uint64_t *__restrict__ bkey,
                                                  const uint32_t *__restrict__ bstart, uint32_t nblocks,
                                                  const uint32_t *__restrict__ sidx, const uint32_t *__restrict__ row,
                                                  const uint32_t *__restrict__ colind, const T *__restrict__ values,
                                                  uint32_t rb, uint32_t cb, int jbits, uint32_t *__restrict__ bcolind,
                                                  T *__restrict__ bval, uint32_t *__restrict__ nnz_per_block) {
  const uint64_t jmask = (1ull << jbits) - 1;
  const size_t bs = (size_t)rb * cb;
  for (uint32_t b = blockIdx.x * NT + threadIdx.x; b < nblocks; b += gridDim.x * NT) {
    const uint64_t k = bkey[b];
    const uint32_t J = (uint32_t)(k & jmask), r0 = (uint32_t)(k >> jbits) * rb, c0 = J * cb;
    bcolind[b] = J;
    T *blk = bval + (size_t)b * bs;
    for (size_t q = 0; q < bs; ++q) blk[q] = T(0);
    for (uint32_t i = bstart[b]; i < bstart[b + 1]; ++i) {  // input order: a later duplicate wins
      const uint32_t e = sidx[i], dc = colind[e] - c0;
      if (dc < cb) blk[(size_t)(row[e] - r0) * cb + dc] = values[e];  // columns as checked by the layout
    }
    uint32_t cnt = 0;
    for (size_t q = 0; q < bs; ++q) cnt += blk[q] != T(0);
    nnz_per_block[b] = cnt;
  }
}

}  // namespace c2b
}  // namespace sparsep

using namespace sparsep::c2b;

struct sparsep_bcsr_layout {
  uint32_t nrows = 0, ncols = 0, nnz = 0, rb = 0, cb = 0, nbr = 0, nblocks = 0;
  int dev = 0;
  const uint32_t *colind = nullptr;  // the caller's column indices (read again by the fill)
  // block rows in shared memory
  uint32_t *rowptr = nullptr;   // the row pointers
  uint32_t *browptr = nullptr;  // nbr + 1
  // the sort
  int jbits = 0;
  uint32_t *row = nullptr;     // row of each nonzero
  uint32_t *sidx = nullptr;    // nonzeros in block order (input order inside a block)
  uint32_t *bstart = nullptr;  // nblocks + 1 start positions in sidx
  uint64_t *bkey = nullptr;    // block keys (block row << jbits | block column)
  sparsep::Scratch mem[4];     // where these lie
  int nmem = 0;
};

static int c2b_err(cudaError_t e) {
  if (e == cudaSuccess) return SPARSEP_OK;
  char msg[160];
  std::snprintf(msg, sizeof msg, "%s (%d)", cudaGetErrorString(e), (int)e);
  sparsep::record_error(msg);
  return e == cudaErrorMemoryAllocation ? SPARSEP_ENOMEM : SPARSEP_EIO;
}

static int bits_for(uint64_t v) {  // bits of the largest value < v
  int b = 0;
  while (b < 64 && v > 1 && ((v - 1) >> b)) ++b;
  return b;
}

static unsigned grid_for(uint64_t n) { return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(16384, (n + NT - 1) / NT)); }

static int col_shift(uint32_t cb) {  // log2 of a power of two, else -1
  if (cb & (cb - 1)) return -1;
  int s = 0;
  while ((1u << s) < cb) ++s;
  return s;
}

// Memory of the layout's own.
template <typename T>
static cudaError_t take(sparsep_bcsr_layout *L, T **p, size_t bytes, cudaStream_t s) {
  const cudaError_t e = sparsep::ws_malloc(&L->mem[L->nmem], bytes, s);
  if (e == cudaSuccess) *p = static_cast<T *>(L->mem[L->nmem++].p);
  return e;
}

static void give_back(sparsep_bcsr_layout *L, cudaStream_t s) {
  while (L->nmem) sparsep::ws_free(&L->mem[--L->nmem], s);
  L->rowptr = L->browptr = L->row = L->sidx = L->bstart = nullptr;
  L->bkey = nullptr;
}

// Block rows in shared memory; *fits false where one is too long for that.
static int layout_rows(const uint32_t *rowptr, sparsep_bcsr_layout *L, bool *fits, cudaStream_t s) {
  using sparsep::radix::SCAN_CHUNK;
  const uint32_t m = L->nbr + 1, nb = (m + SCAN_CHUNK - 1) / SCAN_CHUNK;
  sparsep::Scratch sums;
  int h_flag[2] = {0, 0};
  int st = c2b_err(take(L, &L->rowptr, ((size_t)L->nrows + 1) * 4, s));
  if (!st) st = c2b_err(take(L, &L->browptr, (size_t)m * 4, s));
  if (!st) st = c2b_err(sparsep::ws_malloc(&sums, ((size_t)nb + 4) * 4, s));
  if (!st) {
    uint32_t *buf = static_cast<uint32_t *>(sums.p);
    int *flag = reinterpret_cast<int *>(buf + nb);
    st = c2b_err(cudaMemsetAsync(flag, 0, 2 * sizeof(int), s));
    if (!st) st = c2b_err(cudaMemsetAsync(L->browptr, 0, (size_t)m * 4, s));
    if (!st)
      st = c2b_err(cudaMemcpyAsync(L->rowptr, rowptr, ((size_t)L->nrows + 1) * 4, cudaMemcpyDeviceToDevice, s));
    if (!st) {
      const int cs = col_shift(L->cb);
      if (L->nrows) check_rowptr<<<grid_for(L->nrows), NT, 0, s>>>(rowptr, L->nrows, L->nnz, flag);
      if (L->nnz) {
        const unsigned grid = (unsigned)std::min<uint64_t>(16384, ((uint64_t)L->nbr + WARPS - 1) / WARPS);
        count_blocks<<<grid, 32 * WARPS, 0, s>>>(rowptr, L->nrows, L->colind, L->nnz, L->ncols, L->rb, L->cb, cs,
                                                 L->nbr, L->browptr, flag);
        sparsep::radix::scan_reduce<<<nb, sparsep::radix::NT, 0, s>>>(L->browptr, m, buf);
        sparsep::radix::scan_top<<<1, sparsep::radix::NT, 0, s>>>(buf, nb);
        sparsep::radix::scan_down<<<nb, sparsep::radix::NT, 0, s>>>(L->browptr, m, buf);
      }
      st = c2b_err(cudaGetLastError());
    }
    if (!st) st = c2b_err(cudaMemcpyAsync(h_flag, flag, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    if (!st)
      st = c2b_err(cudaMemcpyAsync(&L->nblocks, L->browptr + L->nbr, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    if (!st) st = c2b_err(cudaStreamSynchronize(s));
    if (!st && h_flag[0]) st = SPARSEP_EINVAL;
  }
  sparsep::ws_free(&sums, s);
  *fits = !h_flag[1];
  return st;
}

static int layout_sorted(const uint32_t *rowptr, const uint32_t *colind, uint32_t nrows, uint32_t ncols, uint32_t nnz,
                         uint32_t rb, uint32_t cb, sparsep_bcsr_layout *L, cudaStream_t s);

static int layout(const uint32_t *rowptr, const uint32_t *colind, uint32_t nrows, uint32_t ncols, uint32_t nnz,
                  uint32_t rb, uint32_t cb, sparsep_bcsr_layout *L, cudaStream_t s) {
  L->nrows = nrows;
  L->ncols = ncols;
  L->nnz = nnz;
  L->rb = rb;
  L->cb = cb;
  L->colind = colind;
  L->nbr = (uint32_t)(((uint64_t)nrows + rb - 1) / rb);
  int st = c2b_err(cudaGetDevice(&L->dev));
  bool fits = true;
  if (!st) st = layout_rows(rowptr, L, &fits, s);
  if (st || fits) return st;
  give_back(L, s);
  return layout_sorted(rowptr, colind, nrows, ncols, nnz, rb, cb, L, s);
}

static int layout_sorted(const uint32_t *rowptr, const uint32_t *colind, uint32_t nrows, uint32_t ncols, uint32_t nnz,
                         uint32_t rb, uint32_t cb, sparsep_bcsr_layout *L, cudaStream_t s) {
  using sparsep::radix::radix_scratch_words;
  const uint64_t nbc = ((uint64_t)ncols + cb - 1) / cb;
  L->jbits = bits_for(nbc);
  const int bits = L->jbits + bits_for(L->nbr);
  sparsep::Scratch flags, work;
  int st = c2b_err(sparsep::ws_malloc(&flags, 2 * sizeof(int), s));
  if (st) return st;
  int *bad = static_cast<int *>(flags.p);
  uint32_t *dnb = reinterpret_cast<uint32_t *>(bad + 1);
  int h_bad = 0;
  st = c2b_err(cudaMemsetAsync(bad, 0, 2 * sizeof(int), s));
  // scratch, in 32-bit words: input keys (2n), two key buffers (2n each), the
  // radix scratch, the head flags (n) with their scan sums (nbs + 8), and
  // the block starts (n + 1).  After the sort the input-key buffer holds the
  // block keys.
  const uint32_t nbs = (nnz + sparsep::radix::SCAN_CHUNK - 1) / sparsep::radix::SCAN_CHUNK;
  const size_t rsw = (radix_scratch_words(nnz) + 1) & ~(size_t)1;
  const size_t words = 6 * (size_t)nnz + rsw + ((size_t)nnz + nbs + 8) + ((size_t)nnz + 1) + 8;
  if (!st) st = c2b_err(sparsep::ws_malloc(&work, words * 4, s));
  if (!st) st = c2b_err(take(L, &L->row, (size_t)nnz * 4, s));
  if (!st) {
    uint64_t *key = static_cast<uint64_t *>(work.p), *k0 = key + nnz, *k1 = k0 + nnz;
    uint32_t *scratch = reinterpret_cast<uint32_t *>(k1 + nnz);
    uint32_t *flag = scratch + rsw, *sums = flag + nnz, *bstart_tmp = sums + nbs + 8;
    uint64_t *bkey_tmp = key;
    keys<<<grid_for(nnz), NT, 0, s>>>(rowptr, nrows, colind, nnz, ncols, rb, cb, L->jbits, key, L->row, bad);
    const uint64_t *skey = nullptr;
    const uint32_t *sidx = nullptr;
    st = c2b_err(sparsep::radix::radix_sort<uint64_t>(key, nnz, bits, k0, k1, scratch, &skey, &sidx, s));
    if (!st) {
      head_flags<<<grid_for(nnz), NT, 0, s>>>(skey, nnz, flag);
      sparsep::radix::scan_reduce<<<nbs, sparsep::radix::NT, 0, s>>>(flag, nnz, sums);
      sparsep::radix::scan_top<<<1, sparsep::radix::NT, 0, s>>>(sums, nbs);
      sparsep::radix::scan_down<<<nbs, sparsep::radix::NT, 0, s>>>(flag, nnz, sums);
      block_starts<<<grid_for(nnz), NT, 0, s>>>(skey, nnz, flag, bstart_tmp, bkey_tmp, dnb);
      st = c2b_err(cudaGetLastError());
    }
    // the columns of the longer block rows are looked at here for the first time
    if (!st) st = c2b_err(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
    if (!st) st = c2b_err(cudaMemcpyAsync(&L->nblocks, dnb, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    if (!st) st = c2b_err(cudaStreamSynchronize(s));
    if (!st && h_bad) st = SPARSEP_EINVAL;
    if (!st) st = c2b_err(take(L, &L->sidx, (size_t)nnz * 4, s));
    if (!st) st = c2b_err(take(L, &L->bstart, ((size_t)L->nblocks + 1) * 4, s));
    if (!st) st = c2b_err(take(L, &L->bkey, (size_t)std::max<uint32_t>(L->nblocks, 1) * 8, s));
    if (!st) st = c2b_err(cudaMemcpyAsync(L->sidx, sidx, (size_t)nnz * 4, cudaMemcpyDeviceToDevice, s));
    if (!st)
      st = c2b_err(cudaMemcpyAsync(L->bstart, bstart_tmp, ((size_t)L->nblocks + 1) * 4, cudaMemcpyDeviceToDevice, s));
    if (!st) st = c2b_err(cudaMemcpyAsync(L->bkey, bkey_tmp, (size_t)L->nblocks * 8, cudaMemcpyDeviceToDevice, s));
    if (!st) st = c2b_err(cudaStreamSynchronize(s));
  }
  sparsep::ws_free(&work, s);
  sparsep::ws_free(&flags, s);
  return st;
}

template <typename T>
static int fill(const sparsep_bcsr_layout *L, const T *values, uint32_t *browptr, uint32_t *bcolind, T *bval,
                uint32_t *nnz_per_block, cudaStream_t s) {
  if (!L || !browptr || (L->nblocks && (!values || !bcolind || !bval || !nnz_per_block))) return SPARSEP_EINVAL;
  if (L->browptr) {
    int st = c2b_err(cudaMemcpyAsync(browptr, L->browptr, ((size_t)L->nbr + 1) * 4, cudaMemcpyDeviceToDevice, s));
    if (!st && L->nblocks) {
      const int cs = col_shift(L->cb);
      const unsigned grid = (unsigned)std::min<uint64_t>(16384, ((uint64_t)L->nbr + WARPS - 1) / WARPS);
      fill_rows<T><<<grid, 32 * WARPS, 0, s>>>(L->rowptr, L->nrows, L->colind, L->nnz, L->ncols, values, L->rb, L->cb,
                                               cs, L->nbr, L->browptr, bcolind, bval, nnz_per_block);
      st = c2b_err(cudaGetLastError());
    }
    if (!st) st = c2b_err(cudaStreamSynchronize(s));
    return st;
  }
  browptr_kernel<<<(L->nbr + 1 + 255) / 256, 256, 0, s>>>(L->bkey, L->nblocks, L->nbr, L->jbits, browptr);
  if (L->nblocks)
    fill_blocks<T><<<grid_for(L->nblocks), NT, 0, s>>>(L->bkey, L->bstart, L->nblocks, L->sidx, L->row, L->colind,
                                                        values, L->rb, L->cb, L->jbits, bcolind, bval, nnz_per_block);
  int st = c2b_err(cudaGetLastError());
  if (!st) st = c2b_err(cudaStreamSynchronize(s));
  return st;
}

extern "C" {

int sparsep_bcsr_layout_device(const uint32_t *d_rowptr, const uint32_t *d_colind, uint32_t nrows, uint32_t ncols,
                               uint32_t nnz, uint32_t rb, uint32_t cb, sparsep_bcsr_layout **out, uint64_t *nblocks,
                               void *stream) {
  if (!out) return SPARSEP_EINVAL;
  *out = nullptr;
  if (!d_rowptr || (nnz && !d_colind) || rb == 0 || cb == 0 || (nnz && nrows == 0)) return SPARSEP_EINVAL;
  auto *L = new (std::nothrow) sparsep_bcsr_layout();
  if (!L) return SPARSEP_ENOMEM;
  const int st = layout(d_rowptr, d_colind, nrows, ncols, nnz, rb, cb, L, static_cast<cudaStream_t>(stream));
  if (st) {
    sparsep_bcsr_layout_free(L);
    return st;
  }
  if (nblocks) *nblocks = L->nblocks;
  *out = L;
  return SPARSEP_OK;
}

void sparsep_bcsr_layout_free(sparsep_bcsr_layout *L) {
  if (!L) return;
  // layout and fill have synchronised their streams: nothing uses these any more
  int dev = L->dev;
  cudaGetDevice(&dev);
  if (dev != L->dev) cudaSetDevice(L->dev);
  give_back(L, nullptr);
  if (dev != L->dev) cudaSetDevice(dev);
  delete L;
}

#define SPARSEP_C2B_ENTRY(T, S)                                                                                   \
  int sparsep_csr2bcsr_device_##S(const sparsep_bcsr_layout *L, const T *d_values, uint32_t *d_browptr,          \
                                  uint32_t *d_bcolind, T *d_bval, uint32_t *d_nnz_per_block, void *stream) {      \
    return fill<T>(L, d_values, d_browptr, d_bcolind, d_bval, d_nnz_per_block, static_cast<cudaStream_t>(stream)); \
  }
SPARSEP_C2B_ENTRY(int8_t, i8)
SPARSEP_C2B_ENTRY(int16_t, i16)
SPARSEP_C2B_ENTRY(int32_t, i32)
SPARSEP_C2B_ENTRY(int64_t, i64)
SPARSEP_C2B_ENTRY(float, f32)
SPARSEP_C2B_ENTRY(double, f64)

}  // extern "C"
