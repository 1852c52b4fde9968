// radix.cuh -- stable LSD radix sort on the device, up to 7 bits per pass, used by
// the device format builders: COO -> CSR sorts (row, column, value) records by
// row; CSR -> BCSR, where a block row is too long for shared memory, (key, index)
// pairs by (block row, block column).
//   hist     per 4096-element tile, counts of each digit  -> hist[d][tile]
//   scan     exclusive scan of hist in digit-major order (three launches)
//   scatter  each element to scan[d][tile] + (earlier elements of its tile with
//            digit d).  A warp takes 256 consecutive elements, 32 at a time;
//            a vote per digit bit gives the rank among the lanes with the same digit
//            and the warp's own counter per digit the rank before that, so the
//            warps meet only twice.  Keys, payloads and values then go through
//            shared memory, so that a digit's elements leave as runs of
//            consecutive addresses.
// Bound by HBM in the limit (a record is read and written once per pass: 38 us for
// 10.5 M records of 12 bytes); a pass takes 12 us (hist) + 10 (scan) + 80 (scatter),
// the scatter issuing in 40 % of the cycles for its ranking and address arithmetic.
// 512 threads and two CTAs per SM: 1024 threads are 8 to 20 % slower, 3 CTAs at 42
// registers no faster.  With 256 threads of 16 elements and __match_any_sync the
// scatter took 236 us; with 4-bit digits, 1024-element tiles and three barriers per
// 256 elements, keys and indices alone 107 us per pass and 5 passes for 19 bits.
#pragma once
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

namespace sparsep {
namespace radix {
namespace {  // internal linkage: every translation unit that sorts gets its own kernels

constexpr int NT = 256;            // threads per CTA
constexpr int TILE = 4096;         // elements per tile
constexpr int SNT = 512;           // threads of the scatter: 8 elements each, 64 registers
constexpr int MAX_BITS = 7;        // bits of a digit
constexpr int MAX_RADIX = 1 << MAX_BITS;
constexpr unsigned FULL = 0xffffffffu;

template <typename K>
__global__ void __launch_bounds__(NT) hist(const K *__restrict__ key, uint32_t n, int shift, int bits, uint32_t nt,
                                           uint32_t *__restrict__ h, K bound, int *__restrict__ bad) {
  __shared__ uint32_t c[NT / 32][MAX_RADIX];  // per warp: fewer lanes meet at one counter
  const int warp = threadIdx.x >> 5, radix = 1 << bits;
  for (int i = threadIdx.x; i < NT / 32 * MAX_RADIX; i += NT) (&c[0][0])[i] = 0;
  __syncthreads();
  constexpr int IPT = TILE / NT;
  const uint32_t base = blockIdx.x * TILE;
  // all loads first: left to the compiler, each waited for the counter before it
  // (28 instead of 12 us for 10.5 M keys)
  K k[IPT];
#pragma unroll
  for (int r = 0; r < IPT; ++r) {
    const uint32_t i = base + r * NT + threadIdx.x;
    k[r] = i < n ? key[i] : K(0);
  }
  bool out = false;
#pragma unroll
  for (int r = 0; r < IPT; ++r)
    if (base + r * NT + threadIdx.x < n) {
      out |= k[r] >= bound;
      atomicAdd(&c[warp][(uint32_t)(k[r] >> shift) & (radix - 1)], 1u);
    }
  if (bad && out) atomicExch(bad, 1);  // first pass only: keys must be < bound
  __syncthreads();
  if (threadIdx.x < radix) {
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) t += c[w][threadIdx.x];
    h[(size_t)threadIdx.x * nt + blockIdx.x] = t;
  }
}

// Exclusive scan of the m digit counts in place, in three launches:
//   scan_reduce  CTA b sums its chunk h[b*SCAN_CHUNK, ...)        -> sums[b]
//   scan_top     one CTA scans sums[0, nb) (exclusive), in chunks
//   scan_down    CTA b scans its chunk and adds sums[b]
// A chunk is SCAN_CHUNK = 4 counts per thread; a thread scans its 4 serially
// and the CTA scans the thread totals with warp shuffles.
constexpr int SCAN_CHUNK = 4 * NT;

// exclusive scan of v over the CTA; *total gets the sum of all v
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *total) {
  __shared__ uint32_t ws[NT / 32 + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < NT / 32 ? ws[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < NT / 32) ws[lane] = wi - w;
    if (lane == NT / 32 - 1) ws[NT / 32] = wi;
  }
  __syncthreads();
  const uint32_t r = ws[warp] + inc - v;
  *total = ws[NT / 32];
  __syncthreads();  // ws is reused by the next call
  return r;
}

// exclusive scan of a[base, base + SCAN_CHUNK) (clipped to m) plus offset; returns the chunk's sum
__device__ __forceinline__ uint32_t scan_chunk(uint32_t *__restrict__ a, uint32_t m, uint32_t base, uint32_t offset) {
  const uint32_t i0 = base + 4 * threadIdx.x;
  uint32_t v[4], t = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = i0 + k < m ? a[i0 + k] : 0u;
    t += v[k];
  }
  uint32_t total;
  uint32_t run = offset + block_scan(t, &total);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i0 + k < m) a[i0 + k] = run;
    run += v[k];
  }
  return total;
}

__global__ void __launch_bounds__(NT) scan_reduce(const uint32_t *__restrict__ h, uint32_t m,
                                                  uint32_t *__restrict__ sums) {
  const uint32_t i0 = blockIdx.x * SCAN_CHUNK + 4 * threadIdx.x;
  uint32_t t = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) t += i0 + k < m ? h[i0 + k] : 0u;
  uint32_t total;
  block_scan(t, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(NT) scan_top(uint32_t *__restrict__ sums, uint32_t nb) {
  uint32_t carry = 0;
  for (uint32_t b = 0; b < nb; b += SCAN_CHUNK) carry += scan_chunk(sums, nb, b, carry);
}

__global__ void __launch_bounds__(NT) scan_down(uint32_t *__restrict__ h, uint32_t m,
                                                const uint32_t *__restrict__ sums) {
  scan_chunk(h, m, blockIdx.x * SCAN_CHUNK, sums[blockIdx.x]);
}

// One pass.  The payload of an element is a 32-bit word (its index where w_in is
// null) and, unless V is NoValue, a value.
struct NoValue {};

// The lanes of the warp that have this lane's digit d, a vote per bit:
// __match_any_sync takes as many steps as the warp has different digits (142 instead
// of 92 us per pass over 10.5 M records).
__device__ __forceinline__ uint32_t same_digit(uint32_t d) {
  uint32_t same = FULL;
#pragma unroll
  for (int b = 0; b < MAX_BITS; ++b) {
    const int32_t mine = (int32_t)(d << (31 - b)) >> 31;  // the bit in all places
    same &= ~(__ballot_sync(FULL, mine) ^ mine);
  }
  return same;
}

template <typename K, typename V> struct Stage {  // a tile's records in shared memory
  static constexpr size_t VALUES = TILE * sizeof(K);
  static constexpr size_t WORDS = VALUES + (std::is_same<V, NoValue>::value ? 0 : TILE * sizeof(V));
  static constexpr size_t BYTES = WORDS + TILE * 4;
};

template <typename K, typename V>
__global__ void __launch_bounds__(SNT, 2) scatter(const K *__restrict__ key, const uint32_t *__restrict__ w_in,
                                              const V *__restrict__ v_in, uint32_t n, int shift, int bits, uint32_t nt,
                                              const uint32_t *__restrict__ off, K *__restrict__ key_out,
                                              uint32_t *__restrict__ w_out, V *__restrict__ v_out) {
  constexpr bool VALUE = !std::is_same<V, NoValue>::value;
  constexpr int IPT = TILE / SNT, WARPS = SNT / 32;
  extern __shared__ __align__(16) unsigned char stage[];  // Stage<K, V>::BYTES: keys, values, words
  K *sk = reinterpret_cast<K *>(stage);
  V *sv = reinterpret_cast<V *>(stage + Stage<K, V>::VALUES);
  uint32_t *sw = reinterpret_cast<uint32_t *>(stage + Stage<K, V>::WORDS);
  __shared__ uint32_t cnt[WARPS][MAX_RADIX];
  __shared__ uint32_t first[MAX_RADIX];  // of the tile's elements, the first of each digit
  __shared__ uint32_t dst[MAX_RADIX];    // its place in the output less that
  __shared__ uint32_t sums[4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, radix = 1 << bits;
  const uint32_t base = blockIdx.x * TILE, here = n - base < TILE ? n - base : TILE;
  for (int i = threadIdx.x; i < WARPS * MAX_RADIX; i += SNT) (&cnt[0][0])[i] = 0;
  __syncthreads();
  // this thread's elements: 32 apart, in the warp's share
  const uint32_t mine = warp * (32 * IPT) + lane;
  auto tile = [&](auto whole) {  // whole: TILE elements
    constexpr bool WHOLE = decltype(whole)::value;
    auto in = [&](int r) { return WHOLE || mine + r * 32 < here; };
    auto digit = [&](K x) { return (uint32_t)(x >> shift) & (radix - 1); };
    const K *kp = key + base + mine;
    K k[IPT];
    uint32_t w[IPT], pos[IPT];
#pragma unroll
    for (int r = 0; r < IPT; ++r) k[r] = in(r) ? kp[r * 32] : K(0);
    if (w_in) {
      const uint32_t *wp = w_in + base + mine;
#pragma unroll
      for (int r = 0; r < IPT; ++r) w[r] = in(r) ? wp[r * 32] : 0u;
    } else {
#pragma unroll
      for (int r = 0; r < IPT; ++r) w[r] = base + mine + r * 32;
    }
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
      uint32_t same = same_digit(digit(k[r]));
      if constexpr (!WHOLE) same &= __ballot_sync(FULL, in(r));
      const int leader = __ffs(same) - 1;
      uint32_t before = 0;
      if (in(r) && lane == leader) {
        before = cnt[warp][digit(k[r])];
        cnt[warp][digit(k[r])] = before + __popc(same);
      }
      pos[r] = __shfl_sync(FULL, before, leader < 0 ? 0 : leader) + __popc(same & ((1u << lane) - 1u));
      __syncwarp();
    }
    [[maybe_unused]] V v[IPT];
    if constexpr (VALUE) {
      const V *vp = v_in + base + mine;
#pragma unroll
      for (int r = 0; r < IPT; ++r)
        if (in(r)) v[r] = vp[r * 32];
    }
    __syncthreads();
    uint32_t all = 0, inc = 0;
    if (threadIdx.x < MAX_RADIX) {
      if (threadIdx.x < radix)
#pragma unroll
        for (int q = 0; q < WARPS; ++q) {
          const uint32_t c = cnt[q][threadIdx.x];
          cnt[q][threadIdx.x] = all;
          all += c;
        }
      inc = all;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += t;
      }
      if (lane == 31) sums[warp] = inc;
    }
    __syncthreads();
    if (threadIdx.x < radix) {
      uint32_t f = inc - all;
      for (int q = 0; q < warp; ++q) f += sums[q];
      first[threadIdx.x] = f;
      dst[threadIdx.x] = off[(size_t)threadIdx.x * nt + blockIdx.x] - f;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < IPT; ++r)
      if (in(r)) {
        const uint32_t p = pos[r] + first[digit(k[r])] + cnt[warp][digit(k[r])];
        sk[p] = k[r];
        sw[p] = w[r];
        if constexpr (VALUE) sv[p] = v[r];
      }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      const uint32_t q = threadIdx.x + j * SNT;
      if (WHOLE || q < here) {
        const K kk = sk[q];
        const uint32_t to = dst[digit(kk)] + q;
        key_out[to] = kk;
        w_out[to] = sw[q];
        if constexpr (VALUE) v_out[to] = sv[q];
      }
    }
  };
  if (here == TILE) tile(std::true_type{}); else tile(std::false_type{});
}

// Passes for `bits` bits (at least one, so that the outputs are produced even for
// none), and the bits of each.
inline int passes(int bits) { return bits <= MAX_BITS ? 1 : (bits + MAX_BITS - 1) / MAX_BITS; }
inline int pass_bits(int bits, int pass, int np) { return bits / np + (pass < bits % np ? 1 : 0); }

// Scratch words (32-bit) of the digit counts of n elements and their scan.
inline size_t count_words(uint32_t n) {
  const size_t nt = ((size_t)n + TILE - 1) / TILE, m = MAX_RADIX * nt, nb = (m + SCAN_CHUNK - 1) / SCAN_CHUNK;
  return m + nb + 8;
}

// One pass over n elements from `shift` on; counts: count_words(n) words.
template <typename K>
cudaError_t count_pass(const K *key, uint32_t n, int shift, int bits, uint32_t *counts, cudaStream_t s,
                       int *bad = nullptr, K bound = K(0)) {
  const uint32_t nt = (uint32_t)(((uint64_t)n + TILE - 1) / TILE), m = nt << bits,
                 nb = (m + SCAN_CHUNK - 1) / SCAN_CHUNK;
  uint32_t *sums = counts + m;
  hist<K><<<nt, NT, 0, s>>>(key, n, shift, bits, nt, counts, bound, bad);
  scan_reduce<<<nb, NT, 0, s>>>(counts, m, sums);
  scan_top<<<1, NT, 0, s>>>(sums, nb);
  scan_down<<<nb, NT, 0, s>>>(counts, m, sums);
  return cudaGetLastError();
}
template <typename K, typename V>
cudaError_t scatter_pass(const K *key, const uint32_t *w_in, const V *v_in, uint32_t n, int shift, int bits,
                         const uint32_t *counts, K *key_out, uint32_t *w_out, V *v_out, cudaStream_t s) {
  const uint32_t nt = (uint32_t)(((uint64_t)n + TILE - 1) / TILE);
  constexpr size_t bytes = Stage<K, V>::BYTES;
  if (cudaError_t e = cudaFuncSetAttribute(scatter<K, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes))
    return e;
  scatter<K, V><<<nt, SNT, bytes, s>>>(key, w_in, v_in, n, shift, bits, nt, counts, key_out, w_out, v_out);
  return cudaGetLastError();
}

// Scratch words (32-bit) radix_sort needs for n elements besides the key buffers.
inline size_t radix_scratch_words(uint32_t n) { return 2 * (size_t)n + count_words(n); }

// Stable sort of keys[0, n) by their low `bits` bits, carrying the input index.
// k0/k1: two key buffers of n; scratch: radix_scratch_words(n) words.  On return
// *ks / *is point at the sorted keys and input indices (inside k0/k1 and scratch).
template <typename K>
cudaError_t radix_sort(const K *keys, uint32_t n, int bits, K *k0, K *k1, uint32_t *scratch, const K **ks,
                       const uint32_t **is, cudaStream_t s) {
  uint32_t *i0 = scratch, *i1 = i0 + n, *counts = i1 + n;
  const K *key = keys;
  const uint32_t *idx = nullptr;
  const int np = passes(bits);
  for (int p = 0, shift = 0; n && p < np; shift += pass_bits(bits, p, np), ++p) {
    K *ko = p % 2 ? k1 : k0;
    uint32_t *io = p % 2 ? i1 : i0;
    const int b = pass_bits(bits, p, np);
    if (cudaError_t e = count_pass<K>(key, n, shift, b, counts, s)) return e;
    if (cudaError_t e = scatter_pass<K, NoValue>(key, idx, nullptr, n, shift, b, counts, ko, io, nullptr, s)) return e;
    key = ko;
    idx = io;
  }
  *ks = key;
  *is = idx;
  return cudaSuccess;
}

}  // namespace
}  // namespace radix
}  // namespace sparsep
