// Mask / index construction kernels (integer and byte work, HBM-bound):
//   block_scores      column sums -> per-KV-block scores (fixed summation order)
//   build_block_mask  always-kept blocks U top-k remaining blocks by score -> uint8 mask (+ lists)
//   topk              exact, deterministic top-k of fp32 rows -> int32 index lists (+ counts)
//   mask_to_indices   bool mask rows -> padded index lists in the reference kernel's order
//   bitpack/bitunpack little-endian bit packing of bool tensors
// Ordering rule used everywhere a selection is made: descending by value, equal values in
// ascending index order; -0.0 equals +0.0; NaNs with the sign bit clear sort above +inf.
#include <math.h>

#include "common.cuh"

namespace lvar {

namespace {

// Monotone map float -> uint32: a > b  <=>  key(a) > key(b)  (for non-NaN; -0 folded onto +0).
__device__ __forceinline__ uint32_t ordered_key(float x) {
  const uint32_t u = __float_as_uint(x + 0.0f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  return v;
}

// ------------------------------------------------------------------------------------------------
// block scores
// ------------------------------------------------------------------------------------------------
// One warp per (row, kv block).  Lane partials are summed sequentially, then a fixed xor tree.
__global__ void block_scores_kernel(const float* __restrict__ cs, float* __restrict__ out, int64_t rows, int Lkv,
                                    int nk, int block, int64_t cs_row_stride) {
  const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= rows * nk) return;
  const int64_t row = w / nk;
  const int kb = (int)(w % nk);
  const float* src = cs + row * cs_row_stride + (int64_t)kb * block;
  const int valid = min(block, Lkv - kb * block);
  float acc = 0.f;
  for (int c = lane; c < block; c += 32) acc += (c < valid) ? src[c] : 0.f;
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if (lane == 0) out[row * nk + kb] = acc;
}

// ------------------------------------------------------------------------------------------------
// block mask: always U top-(k_total - |always|) of the rest
// ------------------------------------------------------------------------------------------------
// How many blocks come before block j among those that are not always kept: a larger key, or the same key at a lower
// index.  Always-kept blocks have key 0, which precedes nothing but another 0 (a NaN's key): those look at the flags.  Past
// the block's own 32 the index order is fixed, so that a comparison is all that is left: bound by issue where the rows
// fill the chip (8192 rows of 192 blocks: 112 us with flag, key and index looked at in every step and a branch, 125 us
// without the branch).
__device__ __forceinline__ int rank_of(const uint32_t* keys, const uint8_t* flag, int nk, int j) {
  const uint32_t kj = keys[j];
  int rank = 0;
  if (kj == 0u) {
    for (int i = 0; i < nk; ++i) rank += !flag[i] && (keys[i] > 0u || i < j);
    return rank;
  }
  const int j0 = j & ~31, j1 = min(nk, j0 + 32);
#pragma unroll 8
  for (int i = 0; i < j0; ++i) rank += keys[i] >= kj;
#pragma unroll 4
  for (int i = j0; i < j1; ++i) {
    const uint32_t ki = keys[i];
    rank += ki > kj || (ki == kj && i < j);
  }
#pragma unroll 8
  for (int i = j1; i < nk; ++i) rank += keys[i] > kj;
  return rank;
}

// One CTA (128 threads) per (b, h, q-block row).  Rank counting over the row held in shared memory.
__global__ void build_block_mask_kernel(const float* __restrict__ scores, const uint8_t* __restrict__ always,
                                        uint8_t* __restrict__ mask, int32_t* __restrict__ lists,
                                        int32_t* __restrict__ counts, int nq, int nk, int k_total) {
  extern __shared__ uint32_t sh[];
  uint32_t* keys = sh;                                      // [nk]
  uint8_t* flag = reinterpret_cast<uint8_t*>(keys + nk);    // [nk] 1 = always, then final selection
  __shared__ int n_always;
  const int64_t row = blockIdx.x;  // over B*H*nq
  const int qi = (int)(row % nq);
  const float* s = scores + row * nk;
  if (threadIdx.x == 0) n_always = 0;
  __syncthreads();
  int local = 0;
  for (int j = threadIdx.x; j < nk; j += blockDim.x) {
    const uint8_t a = always ? (always[(int64_t)qi * nk + j] != 0) : 0;
    keys[j] = a ? 0u : ordered_key(s[j]);
    flag[j] = a;
    local += a;
  }
  if (local) atomicAdd(&n_always, local);
  __syncthreads();
  const int need = max(0, k_total - n_always);
  uint8_t* mrow = mask + row * nk;
  for (int j = threadIdx.x; j < nk; j += blockDim.x) {
    uint8_t sel = flag[j];
    if (!sel && need > 0) {
      sel = rank_of(keys, flag, nk, j) < need;
    }
    mrow[j] = sel;
  }
  if (lists != nullptr) {
    __syncthreads();  // mrow visible to the CTA (global writes by this CTA; read back below)
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      int n = 0;
      for (int base = 0; base < nk; base += 32) {
        const int j = base + lane;
        const bool on = (j < nk) && mrow[j];
        const uint32_t vote = __ballot_sync(0xffffffffu, on);
        if (on) lists[row * nk + n + __popc(vote & ((1u << lane) - 1u))] = j;
        n += __popc(vote);
      }
      for (int j = n + lane; j < nk; j += 32) lists[row * nk + j] = -1;
      if (lane == 0 && counts) counts[row] = n;
    }
  }
}

// Column sums -> block mask in one pass: one CTA (256 threads) per (b, h, q-block row) reads its row of column
// sums once, forms the per-KV-block scores with block_scores_kernel's summation order (one warp per block: the
// same bits) and selects as build_block_mask_kernel does.  Scores, lists and counts are optional outputs.
// Bound by the latency of its loads: a warp has those of four 128-key blocks in flight.  1024 rows x 10521:
// 10.8 us (17.1 us with one block's four and a branch per rank step).
__global__ void __launch_bounds__(256)
block_mask_from_colsums_kernel(const float* __restrict__ cs, int64_t cs_row_stride, const uint8_t* __restrict__ always,
                               uint8_t* __restrict__ mask, float* __restrict__ scores_out, int32_t* __restrict__ lists,
                               int32_t* __restrict__ counts, int nq, int nk, int Lkv, int block, int k_total) {
  extern __shared__ uint32_t sh[];
  uint32_t* keys = sh;                                      // [nk]
  uint8_t* flag = reinterpret_cast<uint8_t*>(keys + nk);    // [nk]
  __shared__ int n_always;
  const int64_t row = blockIdx.x;
  const int qi = (int)(row % nq);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  if (threadIdx.x == 0) n_always = 0;
  const float* src_row = cs + row * cs_row_stride;
  if (block == 128) {
    constexpr int U = 4;  // blocks per warp at a time: sixteen loads in flight
    for (int kb = warp; kb < nk; kb += U * n_warps) {
      float v[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k0 = (kb + u * n_warps) * 128;
#pragma unroll
        for (int i = 0; i < 4; ++i) v[u][i] = (k0 + lane + 32 * i < Lkv) ? src_row[k0 + lane + 32 * i] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc += v[u][i];
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
        const int k = kb + u * n_warps;
        if (lane == 0 && k < nk) {
          keys[k] = ordered_key(acc);
          if (scores_out) scores_out[row * nk + k] = acc;
        }
      }
    }
  } else {
    for (int kb = warp; kb < nk; kb += n_warps) {
      const float* src = src_row + (int64_t)kb * block;
      const int valid = min(block, Lkv - kb * block);
      float acc = 0.f;
      for (int c = lane; c < block; c += 32) acc += (c < valid) ? src[c] : 0.f;
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
      if (lane == 0) {
        keys[kb] = ordered_key(acc);
        if (scores_out) scores_out[row * nk + kb] = acc;
      }
    }
  }
  __syncthreads();
  int local = 0;
  for (int j = threadIdx.x; j < nk; j += blockDim.x) {
    const uint8_t a = always ? (always[(int64_t)qi * nk + j] != 0) : 0;
    flag[j] = a;
    if (a) keys[j] = 0u;
    local += a;
  }
  if (local) atomicAdd(&n_always, local);
  __syncthreads();
  const int need = max(0, k_total - n_always);
  uint8_t* mrow = mask + row * nk;
  for (int j = threadIdx.x; j < nk; j += blockDim.x) {
    uint8_t sel = flag[j];
    if (!sel && need > 0) {
      sel = rank_of(keys, flag, nk, j) < need;
    }
    mrow[j] = sel;
  }
  if (lists != nullptr) {
    __syncthreads();
    if (threadIdx.x < 32) {
      int n = 0;
      for (int base = 0; base < nk; base += 32) {
        const int j = base + lane;
        const bool on = (j < nk) && mrow[j];
        const uint32_t vote = __ballot_sync(0xffffffffu, on);
        if (on) lists[row * nk + n + __popc(vote & ((1u << lane) - 1u))] = j;
        n += __popc(vote);
      }
      for (int j = n + lane; j < nk; j += 32) lists[row * nk + j] = -1;
      if (lane == 0 && counts) counts[row] = n;
    }
  }
}

// ------------------------------------------------------------------------------------------------
// exact top-k
// ------------------------------------------------------------------------------------------------
constexpr int kHistCopies = 8, kHistStride = 257;
constexpr int kRankCap = 256;   // candidates that are ranked against each other instead of another histogram pass
constexpr int kSortRun = 64;    // pairs a warp sorts in registers, two per lane

// One merge step of the bitonic network on a run of 64 pairs held by a warp (element lane in x, lane + 32 in y): all
// exchanges at distances first, first / 2, ..., 1.
__device__ __forceinline__ void bitonic_run(unsigned long long& x, unsigned long long& y, int lane, int base, int size,
                                            int first) {
  for (int d = first; d >= 1; d >>= 1) {
    if (d == 32) {
      const bool desc = ((base + lane) & size) == 0;
      if ((x < y) == desc) {
        const unsigned long long t = x;
        x = y;
        y = t;
      }
    } else {
      const bool low = (lane & d) == 0;
      const unsigned long long ox = __shfl_xor_sync(0xffffffffu, x, d), oy = __shfl_xor_sync(0xffffffffu, y, d);
      const bool dx = (((base + lane) & size) == 0) == low, dy = (((base + lane + 32) & size) == 0) == low;
      x = dx ? (x > ox ? x : ox) : (x < ox ? x : ox);
      y = dy ? (y > oy ? y : oy) : (y < oy ? y : oy);
    }
  }
}

// One CTA per row.  Shared: keys[n] | pairs[K2] (descending-value order only).
// A row of a few thousand scores is bound by latency: block-wide steps (histogram passes, sorting steps) and the rows
// in flight per SM, not by the 40 KB it reads.
//  * Radix select starts below the leading bits that all keys share and stops as soon as the bin that holds the k-th
//    largest key has few enough members to rank them against each other: one or two passes instead of four.
//    Scores of one row share most of their leading bits (attention column sums span a few binades), so a pass puts
//    most keys into a handful of bins: the histogram is kept in eight copies (one per lane modulo 8, 257 words apart so
//    that equal bins of different copies sit in different banks), which cuts the serialisation of same-address atomics
//    eightfold; the copies are added up when the bins are scanned.
//  * Compaction by ballots over coalesced reads; a warp owns a contiguous range.
//  * The sort of the descending order keeps the steps at distances up to 32 in a warp's registers: 28 block-wide steps
//    for 4096 pairs instead of 78, 6 instead of 36 for 256.
//  * 512 threads where the rows fill the chip (up to four rows per SM; 256 threads measured 10 to 20 % slower on long
//    rows, 1024 leave one row per SM), 1024 for fewer rows and for rows so long that an SM holds one (1024 x 24576, k =
//    2000 descending: 218 us with 1024 threads, 274 with 512).
// rows x n, k: 224 x 4121, 256 descending 25.8 -> 15.1 us; 512 x 10521, 2176 descending 186 -> 135 us; 960 x 2500, 320
// descending 94 -> 45 us; 32 x 10521, 1052 ascending 11.7 -> 10.8 us; 32 x 121, 12 ascending 6.1 -> 3.9 us (before: four
// 8-bit passes always, every sorting step block-wide, 1024 threads always).
template <int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 512 ? 4 : 1)
topk_kernel(const float* __restrict__ scores, int64_t row_stride, int n, int k, int ascending_index,
            int32_t* __restrict__ out, int64_t out_stride, int out_cols, int32_t* __restrict__ counts,
            int count_value, int K2) {
  constexpr int WARPS = THREADS / 32;
  extern __shared__ __align__(16) uint8_t sh_raw[];
  uint32_t* keys = reinterpret_cast<uint32_t*>(sh_raw);
  unsigned long long* pairs = reinterpret_cast<unsigned long long*>(sh_raw + (((size_t)n * 4 + 15) & ~(size_t)15));
  __shared__ int hist[kHistCopies * kHistStride];
  __shared__ __align__(16) uint32_t cand[kRankCap];
  __shared__ int wsum_gt[WARPS], wsum_eq[WARPS];
  __shared__ uint32_t wmin[WARPS], wmax[WARPS];
  __shared__ uint32_t sh_prefix;
  __shared__ int sh_remaining, sh_bin, n_cand;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row = blockIdx.x;
  const float* src = scores + row * row_stride;
  int32_t* dst = out + row * out_stride;

  uint32_t kmin = 0xffffffffu, kmax = 0u;
#pragma unroll 4
  for (int i = tid; i < n; i += THREADS) {
    const uint32_t key = ordered_key(src[i]);
    keys[i] = key;
    kmin = min(kmin, key);
    kmax = max(kmax, key);
  }
  // the tail of the output row: zeros, 16 bytes at a time from the first aligned column on
  {
    const int first = min(out_cols, k + (int)((4 - ((reinterpret_cast<uintptr_t>(dst + k) >> 2) & 3)) & 3));
    const int quads = (out_cols - first) >> 2, rest = first + 4 * quads;
    int4* d4 = reinterpret_cast<int4*>(dst + first);
    for (int i = tid; i < quads; i += THREADS) d4[i] = make_int4(0, 0, 0, 0);
    if (tid < first - k) dst[k + tid] = 0;
    if (tid < out_cols - rest) dst[rest + tid] = 0;
  }
  if (counts != nullptr && tid == 0) counts[row] = count_value;
  if (k <= 0) return;

  kmin = __reduce_min_sync(0xffffffffu, kmin);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  if (lane == 0) {
    wmin[warp] = kmin;
    wmax[warp] = kmax;
  }
  for (int i = tid; i < kHistCopies * kHistStride; i += THREADS) hist[i] = 0;
  __syncthreads();
  kmin = __reduce_min_sync(0xffffffffu, wmin[lane & (WARPS - 1)]);
  kmax = __reduce_max_sync(0xffffffffu, wmax[lane & (WARPS - 1)]);

  uint32_t T = kmin;  // the k-th largest key
  int need_eq = k;    // keys equal to it that belong to the selection
  if (kmin != kmax) {
    // digits of 8 bits, the first one right below the common leading bits
    int top = 32 - __clz(kmin ^ kmax);          // bits [0, top) are still open
    uint32_t prefix = top < 32 ? (kmin >> top) << top : 0u;
    while (true) {
      const int shift = max(0, top - 8);
      const uint32_t dmask = (1u << (top - shift)) - 1u;
      const uint32_t above = top < 32 ? ~0u << top : 0u;
      int* myhist = hist + (lane & (kHistCopies - 1)) * kHistStride;
      for (int i = tid; i < n; i += THREADS) {
        const uint32_t key = keys[i];
        if ((key & above) == prefix) atomicAdd(&myhist[(key >> shift) & dmask], 1);
      }
      __syncthreads();
      if (warp == 0) {
        // bins from the top: the bin that holds the need_eq-th largest candidate.  Lane l owns bins 8l .. 8l+7.
        int binc[8];  // this lane's eight bins, summed over the copies
        int own = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          int c = 0;
#pragma unroll
          for (int k2 = 0; k2 < kHistCopies; ++k2) c += hist[k2 * kHistStride + 8 * lane + j];
          binc[j] = c;
          own += c;
        }
        int suffix = own;  // candidates in this lane's bins and all higher ones
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int t = __shfl_down_sync(0xffffffffu, suffix, d);
          if (lane + d < 32) suffix += t;
        }
        const uint32_t reach = __ballot_sync(0xffffffffu, suffix >= need_eq);  // never empty: all candidates >= need_eq
        const int L = 31 - __clz(reach);
        if (lane == L) {
          int r = need_eq - (suffix - own);  // still to find inside this lane's bins
          int j = 7, size = binc[7];
#pragma unroll
          for (int t = 7; t > 0; --t) {
            if (j == t && binc[t] < r) {
              r -= binc[t];
              j = t - 1;
              size = binc[t - 1];
            }
          }
          sh_prefix = prefix | ((uint32_t)(8 * lane + j) << shift);
          sh_remaining = r;
          sh_bin = size;
          n_cand = 0;
        }
      } else {
        for (int i = tid - 32; i < kRankCap; i += THREADS - 32) cand[i] = 0u;
      }
      __syncthreads();
      prefix = sh_prefix;
      need_eq = sh_remaining;
      top = shift;
      const int size = sh_bin;
      if (top == 0 || size == need_eq) break;
      if (size <= kRankCap) break;
      for (int i = tid; i < kHistCopies * kHistStride; i += THREADS) hist[i] = 0;
      __syncthreads();
    }
    T = prefix;
    if (top > 0) {
      // the bin's members in shared memory, in any order: the k-th largest has fewer than need_eq greater ones and at
      // least need_eq not smaller ones
      const uint32_t above = ~0u << top;
      const int size = sh_bin;
      if (size > kRankCap) {
        // all of a large bin is selected: its smallest member
        uint32_t least = 0xffffffffu;
        for (int i = tid; i < n; i += THREADS) {
          const uint32_t key = keys[i];
          if ((key & above) == prefix) least = min(least, key);
        }
        least = __reduce_min_sync(0xffffffffu, least);
        if (lane == 0) wmin[warp] = least;
        __syncthreads();
        T = __reduce_min_sync(0xffffffffu, wmin[lane & (WARPS - 1)]);
        // how many equal ones: all of them
        need_eq = n;
      } else {
        for (int i = tid; i < n; i += THREADS) {
          const uint32_t key = keys[i];
          if ((key & above) == prefix) cand[atomicAdd(&n_cand, 1)] = key;
        }
        __syncthreads();
        if (tid < size) {
          const uint32_t mine = cand[tid];
          // four at a time; the zeros behind the last one are never greater, and equal only to the smallest key there
          // is, for which the test below holds either way
          int greater = 0, equal = 0;
#pragma unroll 4
          for (int i = 0; i < size; i += 4) {
            const uint4 c = *reinterpret_cast<const uint4*>(cand + i);
            greater += (c.x > mine) + (c.y > mine) + (c.z > mine) + (c.w > mine);
            equal += (c.x == mine) + (c.y == mine) + (c.z == mine) + (c.w == mine);
          }
          if (greater < need_eq && greater + equal >= need_eq) {  // equal members write equal values
            sh_prefix = mine;
            sh_remaining = need_eq - greater;
          }
        }
        __syncthreads();
        T = sh_prefix;
        need_eq = sh_remaining;
      }
    }
  }

  // ordered compaction: warp w owns the contiguous range [w*per, (w+1)*per), 32 keys at a time
  const int per = (((n + 31) / 32 + WARPS - 1) / WARPS) * 32;
  const int lo = min(n, warp * per), hi = min(n, lo + per);
  int gt = 0, eq = 0;
  for (int i = lo; i < hi; i += 32) {
    const uint32_t key = i + lane < hi ? keys[i + lane] : 0u;
    const bool in = i + lane < hi;
    gt += __popc(__ballot_sync(0xffffffffu, in && key > T));
    eq += __popc(__ballot_sync(0xffffffffu, in && key == T));
  }
  if (lane == 0) {
    wsum_gt[warp] = gt;
    wsum_eq[warp] = eq;
  }
  __syncthreads();
  int gt_b = 0, eq_b = 0;  // keys above T / equal to T before this warp's range
  {
    const int a = lane < warp ? wsum_gt[lane & (WARPS - 1)] : 0, b = lane < warp ? wsum_eq[lane & (WARPS - 1)] : 0;
    gt_b = __reduce_add_sync(0xffffffffu, a);
    eq_b = __reduce_add_sync(0xffffffffu, b);
  }
  const uint32_t lt = (1u << lane) - 1u;
  for (int i = lo; i < hi; i += 32) {
    const bool in = i + lane < hi;
    const uint32_t key = in ? keys[i + lane] : 0u;
    const uint32_t vg = __ballot_sync(0xffffffffu, in && key > T), ve = __ballot_sync(0xffffffffu, in && key == T);
    const int g_before = gt_b + __popc(vg & lt), e_before = eq_b + __popc(ve & lt);
    if (in && (key > T || (key == T && e_before < need_eq))) {
      const int pos = g_before + min(e_before, need_eq);
      if (ascending_index) dst[pos] = i + lane;
      else pairs[pos] = ((unsigned long long)key << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)(i + lane));
    }
    gt_b += __popc(vg);
    eq_b += __popc(ve);
  }
  if (ascending_index) return;

  for (int i = k + tid; i < K2; i += THREADS) pairs[i] = 0ull;  // sorts last
  __syncthreads();
  // bitonic sort, descending on (key, ~index): equal keys come out in ascending index order
  for (int run = warp * kSortRun; run < K2; run += WARPS * kSortRun) {
    unsigned long long x = pairs[run + lane], y = pairs[run + lane + 32];
    for (int size = 2; size <= kSortRun; size <<= 1) bitonic_run(x, y, lane, run, size, size >> 1);
    pairs[run + lane] = x;
    pairs[run + lane + 32] = y;
  }
  for (int size = 2 * kSortRun; size <= K2; size <<= 1) {
    __syncthreads();
    for (int stride = size >> 1; stride >= kSortRun; stride >>= 1) {
      for (int t = tid; t < (K2 >> 1); t += THREADS) {
        const int i = 2 * t - (t & (stride - 1));
        const int j = i + stride;
        const bool desc = ((i & size) == 0);
        const unsigned long long a = pairs[i], b = pairs[j];
        if ((a < b) == desc) {
          pairs[i] = b;
          pairs[j] = a;
        }
      }
      __syncthreads();
    }
    for (int run = warp * kSortRun; run < K2; run += WARPS * kSortRun) {
      unsigned long long x = pairs[run + lane], y = pairs[run + lane + 32];
      bitonic_run(x, y, lane, run, size, kSortRun >> 1);
      pairs[run + lane] = x;
      pairs[run + lane + 32] = y;
    }
  }
  __syncthreads();
  for (int i = tid; i < k; i += THREADS) dst[i] = (int32_t)(0xFFFFFFFFu - (uint32_t)(pairs[i] & 0xFFFFFFFFull));
}

// ------------------------------------------------------------------------------------------------
// mask_to_indices
// ------------------------------------------------------------------------------------------------
// One warp per row, row staged in shared memory with coalesced loads.  Output order: lane t owns
// columns t, t+32, ...; lanes write their set columns at the exclusive prefix of the lane counts.
// The count is rounded up to multiple_of using the first unset columns.
__global__ void mask_to_indices_kernel(const uint8_t* __restrict__ mask, int32_t* __restrict__ indices,
                                       int32_t* __restrict__ counts, int n, int pad_n, int multiple_of) {
  extern __shared__ uint8_t row_s[];
  const int64_t row = blockIdx.x;
  const int lane = threadIdx.x;
  const uint8_t* src = mask + row * n;
  for (int c = lane; c < n; c += 32) row_s[c] = src[c];
  __syncwarp();
  int local = 0;
  for (int c = lane; c < n; c += 32) local += row_s[c] != 0;
  const int incl = warp_incl_scan(local, lane);
  int offset = incl - local;
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  const int padded = (total + multiple_of - 1) / multiple_of * multiple_of;
  int32_t* dst = indices + row * pad_n;
  for (int c = lane; c < n; c += 32)
    if (row_s[c]) dst[offset++] = c;
  int filled = total;
  for (int base = 0; base < n && filled < padded; base += 32) {
    const int c = base + lane;
    const bool off = (c < n) && (row_s[c] == 0);
    const uint32_t vote = __ballot_sync(0xffffffffu, off);
    const int pos = filled + __popc(vote & ((1u << lane) - 1u));
    if (off && pos < padded && pos < pad_n) dst[pos] = c;
    filled += __popc(vote);
  }
  if (lane == 0) counts[row] = padded;
}

// ------------------------------------------------------------------------------------------------
// bitpack / bitunpack
// ------------------------------------------------------------------------------------------------
__global__ void bitpack_kernel(const uint8_t* __restrict__ mask, uint8_t* __restrict__ packed, int64_t n_bits,
                               int64_t n_bytes) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_bytes) return;
  const int64_t base = i * 8;
  uint32_t v = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (base + j < n_bits && mask[base + j]) v |= 1u << j;
  packed[i] = (uint8_t)v;
}

__global__ void bitunpack_kernel(const uint8_t* __restrict__ packed, uint8_t* __restrict__ mask, int64_t n_bits) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_bits) return;
  mask[i] = (packed[i >> 3] >> (i & 7)) & 1u;
}

// ------------------------------------------------------------------------------------------------
// index lists of a sparse step: remapped decision-scale lists followed by the scale's local band
// ------------------------------------------------------------------------------------------------
// out[bh, g, c] = clamp(src[bh, remap[g], c / rep], 0, k_len - 1)   for c <  cnt
//               = band[g, c - cnt]                                  for cnt <= c < cnt + band_count
//               = 0                                                 beyond;   counts[bh, g] = count_value
// Bound by the writes, which are nearly all zeros (the list rows have k_len columns): one block per list row, so that
// no element pays for index divisions, and the tail in 16-byte stores from the first aligned column on.
// 512 rows x 10521 columns: 5.6 us (3.8 TB/s of writes); 23.3 us with one flat index and its two 64-bit divisions per
// element.  Where there are fewer rows than SMs several blocks share a row (one row x 32768, all listed: 7.6 us by one
// block).
__global__ void __launch_bounds__(256)
sparse_step_lists_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ remap,
                         const int32_t* __restrict__ band, int32_t* __restrict__ out, int32_t* __restrict__ counts,
                         int64_t rows, int64_t src_g_stride, int64_t src_bh_stride, int Gk, int cnt, int rep,
                         int band_count, int k_len, int out_cols, int count_value) {
  const int tid = blockIdx.y * 256 + threadIdx.x, step = gridDim.y * 256;
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const int64_t bh = row / Gk;
    const int g = (int)(row - bh * Gk);
    const int32_t* s = src + bh * src_bh_stride + (int64_t)remap[g] * src_g_stride;
    const int32_t* bd = band + (int64_t)g * band_count;
    int32_t* dst = out + row * out_cols;
    for (int c = tid; c < cnt; c += step) dst[c] = max(0, min(s[rep == 1 ? c : c / rep], k_len - 1));
    for (int c = tid; c < band_count; c += step) dst[cnt + c] = bd[c];
    const int used = cnt + band_count;
    const int first = min(out_cols, used + (int)((4 - ((reinterpret_cast<uintptr_t>(dst + used) >> 2) & 3)) & 3));
    const int quads = (out_cols - first) >> 2;
    int4* d4 = reinterpret_cast<int4*>(dst + first);
    for (int i = tid; i < quads; i += step) d4[i] = make_int4(0, 0, 0, 0);
    if (tid < first - used) dst[used + tid] = 0;
    const int rest = first + 4 * quads;
    if (tid < out_cols - rest) dst[rest + tid] = 0;
    if (tid == 0) counts[row] = count_value;
  }
}

}  // namespace

int launch_sparse_step_lists(const int32_t* src, const int32_t* remap, const int32_t* band, int32_t* out,
                             int32_t* counts, int64_t BH, int Gs, int src_cols, int64_t src_g_stride,
                             int64_t src_bh_stride, int Gk, int cnt, int band_count, int k_len, int out_cols,
                             int count_value, cudaStream_t stream) {
  LVAR_REQUIRE(src && remap && out && counts, LVAR_ERR_ARG, "src, remap, out and counts must be non-null");
  LVAR_REQUIRE(band != nullptr || band_count == 0, LVAR_ERR_ARG, "band is null but band_count > 0");
  LVAR_REQUIRE(BH >= 1 && Gs >= 1 && Gk >= 1 && src_cols >= 1 && k_len >= 1, LVAR_ERR_ARG, "bad sizes");
  LVAR_REQUIRE(cnt >= 0 && band_count >= 0 && cnt + band_count <= out_cols, LVAR_ERR_ARG,
               "cnt + band_count = %d does not fit in %d output columns", cnt + band_count, out_cols);
  // lists shorter than cnt are stretched by repeating every entry `rep` times (repeat_interleave)
  const int rep = src_cols >= cnt ? 1 : (cnt + src_cols - 1) / src_cols;
  const int64_t rows = BH * Gk;
  const unsigned blocks = (unsigned)(rows < (1ll << 30) ? rows : (1ll << 30));
  // parts of at least four stores per thread
  const int64_t parts = rows >= 148 ? 1 : (296 + rows - 1) / rows, most = (out_cols + 1023) / 1024;
  const dim3 grid(blocks, (unsigned)(parts < most ? parts : most));
  sparse_step_lists_kernel<<<grid, 256, 0, stream>>>(src, remap, band, out, counts, rows, src_g_stride, src_bh_stride,
                                                       Gk, cnt, rep, band_count, k_len, out_cols, count_value);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_block_scores(const float* cs, float* out, int64_t rows, int Lkv, int block, int64_t cs_row_stride,
                        cudaStream_t stream) {
  LVAR_REQUIRE(cs && out, LVAR_ERR_ARG, "cs and out must be non-null");
  LVAR_REQUIRE(rows >= 1 && Lkv >= 1, LVAR_ERR_ARG, "rows and Lkv must be >= 1");
  LVAR_REQUIRE(block >= 32 && block % 32 == 0, LVAR_ERR_ARG, "block must be a multiple of 32");
  const int nk = (Lkv + block - 1) / block;
  const int64_t warps = rows * nk;
  const int wpb = 8;
  const int64_t blocks = (warps + wpb - 1) / wpb;
  LVAR_REQUIRE(blocks < (1ll << 31), LVAR_ERR_LIMIT, "too many rows");
  block_scores_kernel<<<(unsigned)blocks, wpb * 32, 0, stream>>>(cs, out, rows, Lkv, nk, block, cs_row_stride);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_build_block_mask(const float* scores, const uint8_t* always, uint8_t* mask, int32_t* lists,
                            int32_t* counts, int64_t BH, int nq, int nk, int k_total, cudaStream_t stream) {
  LVAR_REQUIRE(scores && mask, LVAR_ERR_ARG, "scores and mask must be non-null");
  LVAR_REQUIRE(BH >= 1 && nq >= 1 && nk >= 1, LVAR_ERR_ARG, "BH, nq, nk must be >= 1");
  LVAR_REQUIRE(nk <= 8192, LVAR_ERR_LIMIT, "at most 8192 KV blocks per row (got %d)", nk);
  LVAR_REQUIRE(BH * nq < (1ll << 31), LVAR_ERR_LIMIT, "too many rows");
  const size_t smem = (size_t)nk * 5;
  build_block_mask_kernel<<<(unsigned)(BH * nq), 128, smem, stream>>>(scores, always, mask, lists, counts, nq, nk,
                                                                      k_total);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_block_mask_from_colsums(const float* cs, int64_t cs_row_stride, const uint8_t* always, uint8_t* mask,
                                   float* scores_out, int32_t* lists, int32_t* counts, int64_t BH, int nq, int Lkv,
                                   int block, int k_total, cudaStream_t stream) {
  LVAR_REQUIRE(cs && mask, LVAR_ERR_ARG, "cs and mask must be non-null");
  LVAR_REQUIRE(BH >= 1 && nq >= 1 && Lkv >= 1 && block >= 1, LVAR_ERR_ARG, "BH, nq, Lkv, block must be >= 1");
  const int nk = (Lkv + block - 1) / block;
  LVAR_REQUIRE(nk <= 8192, LVAR_ERR_LIMIT, "at most 8192 KV blocks per row (got %d)", nk);
  LVAR_REQUIRE(BH * nq < (1ll << 31), LVAR_ERR_LIMIT, "too many rows");
  const size_t smem = (size_t)nk * 5;
  block_mask_from_colsums_kernel<<<(unsigned)(BH * nq), 256, smem, stream>>>(cs, cs_row_stride, always, mask, scores_out,
                                                                             lists, counts, nq, nk, Lkv, block, k_total);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_topk(const float* scores, int64_t rows, int n, int64_t row_stride, int k, int ascending_index,
                int32_t* out, int64_t out_stride, int out_cols, int32_t* counts, int count_value,
                cudaStream_t stream) {
  LVAR_REQUIRE(scores && out, LVAR_ERR_ARG, "scores and out must be non-null");
  LVAR_REQUIRE(rows >= 1 && n >= 1, LVAR_ERR_ARG, "rows and n must be >= 1");
  LVAR_REQUIRE(k >= 0 && k <= n, LVAR_ERR_ARG, "k must be in [0, n] (k=%d, n=%d)", k, n);
  LVAR_REQUIRE(out_cols >= k && out_stride >= out_cols, LVAR_ERR_ARG, "output row too short for k entries");
  LVAR_REQUIRE(rows < (1ll << 31), LVAR_ERR_LIMIT, "too many rows");
  size_t smem = (((size_t)n * 4 + 15) & ~(size_t)15);
  int K2 = 0;
  if (!ascending_index && k > 0) {
    K2 = 2;
    while (K2 < k) K2 <<= 1;
    LVAR_REQUIRE(smem + (size_t)K2 * 8 <= 200 * 1024, LVAR_ERR_LIMIT,
                 "row of %d scores with k=%d needs %zu bytes of shared memory (limit 204800)", n, k, smem + (size_t)K2 * 8);
    if (K2 < kSortRun) K2 = kSortRun;
  }
  LVAR_REQUIRE(smem <= 200 * 1024, LVAR_ERR_LIMIT,
               "row of %d scores with k=%d needs %zu bytes of shared memory (limit 204800)", n, k, smem);
  smem += (size_t)K2 * 8;
  int dev = 0, sms = 0;
  LVAR_CUDA_OK(cudaGetDevice(&dev));
  LVAR_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // 512 threads where more than one row per SM is in flight: enough rows, and shared memory for two (of an SM's 228 KB a
  // block takes 9.3 static and 1 reserved)
  const bool half = rows > sms && 2 * (smem + 10752) <= 228 * 1024;
  auto kern = half ? topk_kernel<512> : topk_kernel<1024>;
  LVAR_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024 + kSortRun * 8));
  kern<<<(unsigned)rows, half ? 512 : 1024, smem, stream>>>(scores, row_stride, n, k, ascending_index, out,
                                                                  out_stride, out_cols, counts, count_value, K2);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_mask_to_indices(const uint8_t* mask, int32_t* indices, int32_t* counts, int64_t rows, int n, int pad_n,
                           int multiple_of, cudaStream_t stream) {
  LVAR_REQUIRE(mask && indices && counts, LVAR_ERR_ARG, "mask, indices and counts must be non-null");
  LVAR_REQUIRE(rows >= 1 && n >= 1 && pad_n >= n && multiple_of >= 1, LVAR_ERR_ARG, "bad sizes");
  LVAR_REQUIRE(n <= 200 * 1024, LVAR_ERR_LIMIT, "rows longer than 204800 columns are not supported");
  LVAR_REQUIRE(rows < (1ll << 31), LVAR_ERR_LIMIT, "too many rows");
  if (n > 48 * 1024)
    LVAR_CUDA_OK(cudaFuncSetAttribute(mask_to_indices_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, n));
  mask_to_indices_kernel<<<(unsigned)rows, 32, n, stream>>>(mask, indices, counts, n, pad_n, multiple_of);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_bitpack(const uint8_t* mask, uint8_t* packed, int64_t n_bits, cudaStream_t stream) {
  LVAR_REQUIRE(mask && packed && n_bits >= 1, LVAR_ERR_ARG, "bad arguments");
  const int64_t n_bytes = (n_bits + 7) / 8;
  bitpack_kernel<<<(unsigned)((n_bytes + 255) / 256), 256, 0, stream>>>(mask, packed, n_bits, n_bytes);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_bitunpack(const uint8_t* packed, uint8_t* mask, int64_t n_bits, cudaStream_t stream) {
  LVAR_REQUIRE(mask && packed && n_bits >= 1, LVAR_ERR_ARG, "bad arguments");
  bitunpack_kernel<<<(unsigned)((n_bits + 255) / 256), 256, 0, stream>>>(packed, mask, n_bits);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

}  // namespace lvar
