// Stable in-cell order of the grid build for crowded cells.
//
// The grid build sorts particles by cell key with a counting sort whose
// scatter leaves each cell's ids in atomic arrival order; the reference's
// stable radix sort (wp.HashGrid.build) leaves them ascending.  Cells of up
// to kSmallCell particles take their rank by counting smaller ids (at most
// kSmallCell loads per particle).  The ids of a more crowded cell are sorted
// by one thread block, either by comparisons in shared memory (bitonic) or, as
// they are distinct numbers below n, through a bitmap: a bit per id, set in any
// order and read off in order, a window of 2^18 ids at a time.  Where n is many
// windows, the ids are first put in the order of their windows.
// Work stays O(N) per build whatever the occupancy: a blown-up state, whose
// non-finite particles share one bucket, or a grid far coarser than the
// particles costs a few passes over the ids instead of k^2 comparisons.
#pragma once

#include <stdint.h>

namespace fs {

constexpr int kSmallCell = 64;        // cells up to this size rank in place
constexpr int kSortThreads = 1024;    // most threads of a sorting block
constexpr int kBitonicMax = 4096;     // largest set that is sorted by comparisons
constexpr int kBitWords = 8192;       // words of the bitmap
constexpr int kWindowBits = 18;
constexpr int kWindow = 1 << kWindowBits;
constexpr int kSortLoads = 8;         // loads a thread has in flight
// Where the lines lie: a bitonic sort's time grows with log^2 of its ids, the
// bitmap's with its windows, each of which is cleared and read off whatever it
// holds.  Whole builds (B200, us), with one choice and the other:
//   kBitonicFew     cells of 1,000 ids: n = 400,000 bitonic 69, bitmap 73;
//                   n = 1,000,000 146, 177; a cell of 1,000 alone 30, 28
//   kDirectWindows  one cell, each window looks at every id, or ordered first:
//                   n = 400,000 (2 windows) 506, 714; 1,000,000 (4) 1,471,
//                   1,724; 2,000,000 (8) 3,857, 3,355; 4,000,000 11,461, 6,629
//   kWindowsPerSort a bitonic sort instead of more than 4 windows, or than 8:
//                   cells of 10,000, n = 4,000,000 469, 523; of 40,000,
//                   n = 16,000,000 1,856, 2,148
// Against a bitonic sort up to 4,096 ids and a radix sort above that, both with
// 1,024 threads in a kernel of their own: one cell of 5,000 68 -> 30, of 200,000
// 1,512 -> 246, n = 400,000 in cells of 3,636 139 -> 102, of 10,000 203 -> 144,
// n = 4,000,000 in cells of 40,000 920 -> 912, n = 16,000,000 2,049 -> 1,952.
constexpr int kBitonicFew = 1024;     // up to here always by comparisons
constexpr int kDirectWindows = 4;     // up to here every window looks at all ids of the cell
constexpr int kWindowsPerSort = 4;    // ordered: a sort instead of more windows than this
// shared memory of a sorting block: the bitmap and a count per warp
constexpr int kSortSmemInts = kBitWords + kSortThreads / 32;
constexpr size_t kSortSmemBytes = sizeof(int32_t) * kSortSmemInts;
static_assert(kWindow == 32 * kBitWords && kBitonicMax <= kBitWords, "one buffer for both sorts");
static_assert((1ll << 31) >> kWindowBits <= kBitWords, "and for a counter per window");

// Ascending sort of in[0, len) (len <= kBitonicMax) into out; the whole block
// calls it.
__device__ inline void block_bitonic_sort(const int32_t* in, int32_t* out, int len, int32_t* s) {
  int p = 1;
  while (p < len) p <<= 1;
  for (int k = threadIdx.x; k < p; k += blockDim.x) s[k] = k < len ? in[k] : 0x7fffffff;
  __syncthreads();
  for (int k = 2; k <= p; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < p / 2; t += blockDim.x) {
        const int i = t + (t & -j), l = i + j;  // the t-th pair: i without bit j, l with it
        const int32_t a = s[i], b = s[l];
        const bool up = (i & k) == 0;
        if ((a > b) == up) {
          s[i] = b;
          s[l] = a;
        }
      }
      __syncthreads();
    }
  }
  for (int k = threadIdx.x; k < len; k += blockDim.x) out[k] = s[k];
  __syncthreads();
}

// f(id) for this thread's share of in[from, len), kSortLoads at a time;
// UNTIL_FALSE: after a batch whose last id f refuses nothing more is read.
template <bool UNTIL_FALSE, class F>
__device__ __forceinline__ void for_ids(const int32_t* in, int from, int len, F&& f) {
  const int nthr = blockDim.x;
  for (int64_t k = from + (int)threadIdx.x; k < len; k += (int64_t)kSortLoads * nthr) {
    int32_t id[kSortLoads];
#pragma unroll
    for (int q = 0; q < kSortLoads; ++q) id[q] = k + q * nthr < len ? in[k + q * nthr] : -1;
    bool more = true;
#pragma unroll
    for (int q = 0; q < kSortLoads; ++q) more = id[q] >= 0 && f(id[q]);
    if (UNTIL_FALSE && !more) return;
  }
}

// out[0, len) = in[0, len) in the order of their windows (in any order within
// one); the whole block calls it.  counter[nwindows] in shared memory.
__device__ inline void block_order_by_window(const int32_t* in, int32_t* out, int len, int nwindows, int32_t* counter) {
  for (int k = threadIdx.x; k < nwindows; k += blockDim.x) counter[k] = 0;
  __syncthreads();
  for_ids<false>(in, 0, len, [&](int32_t id) { return atomicAdd(&counter[id >> kWindowBits], 1) >= 0; });
  __syncthreads();
  if (threadIdx.x < 32) {  // exclusive prefix
    const int lane = threadIdx.x;
    int run = 0;
    for (int k = lane; k - lane < nwindows; k += 32) {
      const int c = k < nwindows ? counter[k] : 0;
      int inc = c;
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (k < nwindows) counter[k] = run + inc - c;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  __syncthreads();
  for_ids<false>(in, 0, len, [&](int32_t id) {
    out[atomicAdd(&counter[id >> kWindowBits], 1)] = id;
    return true;
  });
  __syncthreads();
}

// The distinct ids in[0, len), each in [0, n), in ascending order into out
// (another array); the whole block (whole warps) calls it.  smem holds
// kSortSmemInts ints.
__device__ inline void block_bitmap_sort(const int32_t* in, int32_t* out, int len, int64_t n, int32_t* smem) {
  uint32_t* const bits = reinterpret_cast<uint32_t*>(smem);
  int32_t* const warp_ids = smem + kBitWords;
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, w = tid >> 5, nw = nthr >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int nwindows = (int)((n + kWindow - 1) >> kWindowBits);
  const bool ordered = nwindows > kDirectWindows;
  if (ordered) block_order_by_window(in, out, len, nwindows, smem);
  int done = 0;  // ids in their places (the same in all threads)
  for (int window = 0; window < nwindows && done < len; ++window) {
    if (ordered) {
      window = out[done] >> kWindowBits;  // the next one that holds any
      // the windows from here whose ids one sort can hold (all threads read the same)
      int end = min(done + kBitonicMax, len);
      const int stop = end < len ? out[end] >> kWindowBits : nwindows;
      if (end < len) {
        int a = done, b = end;  // the first id of window `stop`
        while (a < b) {
          const int mid = (a + b) >> 1;
          if (out[mid] >> kWindowBits < stop)
            a = mid + 1;
          else
            b = mid;
        }
        end = a;
      }
      if (end > done && stop - window > kWindowsPerSort) {
        block_bitonic_sort(out + done, out + done, end - done, smem);
        done = end;
        window = stop - 1;
        continue;
      }
    }
    const int lo = window << kWindowBits;
    const int words = n - lo >= kWindow ? kBitWords : (int)(n - lo + 31) >> 5;
    for (int k = tid; k < words; k += nthr) bits[k] = 0;
    __syncthreads();
    auto set = [&](int32_t id) {
      if (id >> kWindowBits != window) return false;
      atomicOr(&bits[(id - lo) >> 5], 1u << (id & 31));
      return true;
    };
    if (ordered)
      for_ids<true>(out, done, len, set);
    else
      for_ids<false>(in, 0, len, set);
    __syncthreads();
    // each warp reads off its own run of words
    const int per = ((words + nw - 1) / nw + 31) & ~31;
    const int w0 = min(w * per, words), w1 = min(w0 + per, words);
    int count = 0;
    for (int q = w0 + lane; q < w1; q += 32) count += __popc(bits[q]);
    count = __reduce_add_sync(0xffffffffu, count);
    if (lane == 0) warp_ids[w] = count;
    __syncthreads();
    int base = done;
    for (int q = 0; q < nw; ++q) {
      const int c = warp_ids[q];
      if (q < w) base += c;
      done += c;
    }
    for (int q = w0; q < w1; q += 32) {
      const uint32_t m = q + lane < w1 ? bits[q + lane] : 0;
      unsigned left = __ballot_sync(0xffffffffu, m != 0);
      if (!left) continue;
      const int c = __popc(m);
      int inc = c;
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      int at = base + inc - c;
      if (__reduce_max_sync(0xffffffffu, (unsigned)c) < __popc(left)) {
        for (uint32_t r = m; r; r &= r - 1)  // sparse: a lane per word, one bit at a time
          out[at++] = lo + (q + lane) * 32 + __ffs(r) - 1;
      } else {
        for (; left; left &= left - 1) {  // dense: a lane per bit, one word at a time
          const int j = __ffs(left) - 1;
          const uint32_t word = __shfl_sync(0xffffffffu, m, j);
          const int to = __shfl_sync(0xffffffffu, at, j);
          if (word >> lane & 1) out[to + __popc(word & below)] = lo + (q + j) * 32 + lane;
        }
      }
      base += __shfl_sync(0xffffffffu, inc, 31);
    }
    __syncthreads();
  }
}

// The distinct ids in[0, len), each in [0, n), in ascending order into out
// (another array); the whole block calls it.
__device__ inline void block_sort_ids(const int32_t* in, int32_t* out, int len, int64_t n, int32_t* smem) {
  if (len <= kBitonicFew || (len <= kBitonicMax && n > (int64_t)kDirectWindows * kWindow))
    block_bitonic_sort(in, out, len, smem);
  else
    block_bitmap_sort(in, out, len, n, smem);
}

}  // namespace fs
