// Unsorted reducers: a stable sort of the edges by row id on the device, so that a Reducer whose index is not
// ascending can still be served by the CSR kernels.  The reference converts COO row ids to CSR offsets with
// bincount + cumsum and silently assumes the ids are already sorted
// (python_wrapper/dynamic_replace_submodule.py:20-41); here the permutation that sorts them is computed once,
// the per-edge arrays are permuted with it, and the CSR offsets come from the sorted ids.
//
// Least-significant-digit radix sort on the row ids, which are dense: ceil(log2(num_rows)) bits in as few passes as cover
// them, every pass the same width (21 bits: 3 x 7).  A pass is three launches: digit counts per tile of keys, one CTA per
// digit that scans that digit's counts over the tiles, and the stable scatter.  No block waits for another one.  Digits have
// up to 8 bits, or 9 and 10 where that saves a pass that costs more (flexspmv_sort_rows); every width is compiled by itself.  The first pass reads the caller's ids and takes the
// positions as values, so there is no separate initialisation; the passes alternate between two buffers so that the last one
// writes the caller's permutation.  Equal digits keep their input order in every pass (see sort_scatter_kernel), so the
// permutation equals a stable argsort (bit-exact against numpy.argsort(kind="stable")).
#include <cuda_runtime.h>

#include "flex_common.cuh"

namespace flex {

int device_sm_count();      // flex_core.cu

constexpr int kSortKeysPerThread = 16;
// One width of digit: bins, threads of a CTA, and with 16 keys a thread the tile.  A pass with 512 or 1024 bins has tiles of 8192
// keys, so that a digit's keys in a tile still leave in runs of 8 and more.
template <int BITS_, int THREADS_>
struct SortShape {
  static constexpr int kBits = BITS_, kBins = 1 << BITS_, kThreads = THREADS_, kWarps = THREADS_ / 32;
  static constexpr int kTile = THREADS_ * kSortKeysPerThread;
  static constexpr int kWordsPerThread = kBins / 2 > THREADS_ ? kBins / 2 / THREADS_ : 1;    // two 16-bit counters a word
  static constexpr int kCntPitch = kBins + 2;            // per warp; the bin behind the last takes the lanes behind the end
  // shared memory of the scatter: tile in digit order, global place of every digit, counters by warp
  static constexpr int kSmem = kTile * 8 + kBins * 4 + kWarps * kCntPitch * 2;
};
template <int BITS>
using SortNarrow = SortShape<BITS, 256>;
template <int BITS>
using SortWide = SortShape<BITS, 512>;

template <typename KeyT>
__device__ __forceinline__ unsigned digit_of(KeyT key, int shift, unsigned mask) { return ((unsigned)key >> shift) & mask; }

// Per tile: number of keys with each digit -> hist[digit * num_tiles + tile].  CHECK (first pass): flags ids outside
// [0, num_rows).
template <typename KeyT, bool CHECK, class S>
__global__ void __launch_bounds__(S::kThreads) sort_count_kernel(const KeyT* keys, long long n, long long num_rows,
                                                                 int shift, int num_tiles, unsigned* hist, int* status) {
  constexpr unsigned mask = S::kBins - 1;
  __shared__ unsigned s_cnt[S::kBins];
  const int tid = threadIdx.x;
  pdl_wait();
  pdl_launch_dependents();
  for (int d = tid; d < S::kBins; d += S::kThreads) s_cnt[d] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * S::kTile + tid;
  const int left = (int)(n - base < S::kTile ? n - base : S::kTile);      // key i of the thread lies inside the input: i * kThreads < left
  const KeyT* const in = keys + base;
  bool bad = false;
  KeyT k[kSortKeysPerThread];           // all loads before the first atomic
#pragma unroll
  for (int i = 0; i < kSortKeysPerThread; ++i) k[i] = i * S::kThreads < left ? in[i * S::kThreads] : KeyT(0);
#pragma unroll
  for (int i = 0; i < kSortKeysPerThread; ++i) {
    if (i * S::kThreads < left) {
      if (CHECK) bad |= (long long)k[i] < 0 || (long long)k[i] >= num_rows;
      atomicAdd(&s_cnt[digit_of(k[i], shift, mask)], 1u);     // integer counts: order does not matter
    }
  }
  if (CHECK && bad) atomicCAS(status, 0, FLEXSPMV_ERR_BAD_ARG);
  __syncthreads();
  for (int d = tid; d < S::kBins; d += S::kThreads) hist[(size_t)d * num_tiles + blockIdx.x] = s_cnt[d];
}

// Exclusive scan over the CTA's 32 * WARPS threads; `total` is the sum of all.  s_warp: WARPS words.
template <int WARPS>
__device__ __forceinline__ unsigned block_exclusive(unsigned v, unsigned* s_warp, unsigned& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  unsigned before = 0, sum = 0;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    const unsigned c = s_warp[w];
    if (w < warp) before += c;
    sum += c;
  }
  total = sum;
  __syncthreads();          // s_warp may be reused
  return before + x - v;
}

// One CTA per digit: exclusive scan of the digit's counts over the tiles, in place; the digit's total.
constexpr int kScanThreads = 512;
__global__ void __launch_bounds__(kScanThreads) sort_scan_kernel(unsigned* __restrict__ hist, int num_tiles, unsigned* __restrict__ totals) {
  __shared__ unsigned s_warp[kScanThreads / 32];
  pdl_wait();
  pdl_launch_dependents();
  unsigned* row = hist + (size_t)blockIdx.x * num_tiles;
  unsigned run = 0;
  constexpr int kPer = 4;
  for (int base = 0; base < num_tiles; base += kScanThreads * kPer) {
    unsigned v[kPer], sum = 0;
    const int i0 = base + threadIdx.x * kPer;
#pragma unroll
    for (int j = 0; j < kPer; ++j) { v[j] = i0 + j < num_tiles ? row[i0 + j] : 0u; sum += v[j]; }
    unsigned total;
    unsigned at = run + block_exclusive<kScanThreads / 32>(sum, s_warp, total);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (i0 + j < num_tiles) row[i0 + j] = at;
      at += v[j];
    }
    run += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = run;
}

// Stable scatter of one pass.  A warp ranks its 512 consecutive keys 32 at a time (lanes with the same digit find one another
// with one vote per bit of the digit -- __match_any_sync took four times as long, 80 us a pass; the rank counts the lanes
// below), the tile is put in digit order in shared memory and leaves from there, so that a digit's keys are stored side by
// side.  Storing straight from the ranks would touch a sector per key.  Order: warps own consecutive runs of keys, a warp's
// rounds follow one another and lanes are ranked in order, so equal digits never change places.  FIRST: the values are the
// positions.  Bound by the instructions of the ranking and the moves and by shared memory's wavefronts (52 %).  With the width and whole tiles
// known to the compiler a vote is four instructions, not seven, and no key asks whether it lies inside: 8.4 M ids in three
// passes of 7 bits 306 -> 283 us (265 with the launches overlapped) with the counts, offsets and a permutation.  Measured and left out: two passes of 11 bits in ranges of
// tiles a CTA, lanes meeting in shared memory instead of by votes (331: 2048 counters a warp, 48 wavefronts for 32 keys).
template <typename KeyT, bool FIRST, class S>
__global__ void __launch_bounds__(S::kThreads, 1024 / S::kThreads)
sort_scatter_kernel(const KeyT* keys_in, const int* vals_in, long long n, int shift,
                    int num_tiles, const unsigned* hist, const unsigned* totals, unsigned* keys_out, int* vals_out) {
  constexpr int KPT = kSortKeysPerThread, T = S::kThreads, W = S::kWarps, WPT = S::kWordsPerThread;
  constexpr unsigned mask = S::kBins - 1;
  extern __shared__ __align__(16) unsigned char s_sort[];
  uint2* const s_pair = reinterpret_cast<uint2*>(s_sort);                                  // [kTile] the tile in digit order
  unsigned* const s_out = reinterpret_cast<unsigned*>(s_pair + S::kTile);                  // [kBins] where the digit's run goes, less its place in the tile
  unsigned short* const s_cnt = reinterpret_cast<unsigned short*>(s_out + S::kBins);       // [W][kCntPitch]
  __shared__ unsigned s_warp[W];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long tile0 = (long long)blockIdx.x * S::kTile;
  const int count = (int)(n - tile0 < S::kTile ? n - tile0 : S::kTile);
  const int mine = warp * (32 * KPT) + lane;      // place of the lane's first key in the tile
  const int left = count - mine;                  // key i of the thread lies inside the input: i * 32 < left
  for (int i = tid; i < W * S::kCntPitch / 2; i += T) reinterpret_cast<unsigned*>(s_cnt)[i] = 0;
  pdl_wait();
  pdl_launch_dependents();
  unsigned k[KPT];
  const KeyT* const in = keys_in + tile0 + mine;
#pragma unroll
  for (int i = 0; i < KPT; ++i) k[i] = i * 32 < left ? (unsigned)in[i * 32] : 0u;
  __syncthreads();
  unsigned short* const cnt = s_cnt + warp * S::kCntPitch;
  const unsigned below_mask = (1u << lane) - 1u;
  unsigned rank[KPT / 2];                          // two 16-bit ranks a register
  auto rank_keys = [&](auto full) {
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      unsigned d = (k[i] >> shift) & mask, same = 0xffffffffu;
      bool inside = true;
      if constexpr (!full.value) {
        inside = i * 32 < left;
        same = __ballot_sync(0xffffffffu, inside);
        if (!inside) same = ~same;
      }
#pragma unroll
      for (int b = 0; b < S::kBits; ++b) {
        const bool bit = (d & (1u << b)) != 0;
        const unsigned set = __ballot_sync(0xffffffffu, bit);
        same &= set ^ (bit ? 0u : 0xffffffffu);
      }
      if constexpr (!full.value) if (!inside) d = (unsigned)S::kBins;
      const unsigned below = __popc(same & below_mask);
      const unsigned seen = cnt[d];
      __syncwarp();
      if (below == 0) cnt[d] = (unsigned short)(seen + __popc(same));
      __syncwarp();
      rank[i / 2] = i & 1 ? rank[i / 2] | (seen + below) << 16 : seen + below;
    }
  };
  if (count == S::kTile) rank_keys(IntC<1>{}); else rank_keys(IntC<0>{});
  __syncthreads();
  // values: needed last, requested now
  int v[KPT];
#pragma unroll
  for (int i = 0; i < KPT; ++i) v[i] = FIRST ? (int)(tile0 + mine + i * 32) : (i * 32 < left ? vals_in[tile0 + mine + i * 32] : 0);
  {
    // two digits a word: the warps' counts become places in the tile -- behind the digits before, behind the warps before
    unsigned* const words = reinterpret_cast<unsigned*>(s_cnt);
    constexpr int kPitch = S::kCntPitch / 2;
    const int w0 = tid * WPT;
    const bool has = w0 < S::kBins / 2;
    unsigned sum[WPT], tot[2 * WPT], digits = 0, global = 0;
#pragma unroll
    for (int j = 0; j < WPT; ++j) {
      sum[j] = 0;
      tot[2 * j] = tot[2 * j + 1] = 0;
      if (has) {
#pragma unroll
        for (int w = 0; w < W; ++w) sum[j] += words[w * kPitch + w0 + j];
        tot[2 * j] = totals[2 * (w0 + j)];
        tot[2 * j + 1] = totals[2 * (w0 + j) + 1];
      }
      digits += (sum[j] & 0xffffu) + (sum[j] >> 16);
      global += tot[2 * j] + tot[2 * j + 1];
    }
    unsigned all;
    unsigned place = block_exclusive<W>(digits, s_warp, all);
    unsigned to = block_exclusive<W>(global, s_warp, all);
    if (has) {
#pragma unroll
      for (int j = 0; j < WPT; ++j) {
        const int d = 2 * (w0 + j);
        const unsigned second = place + (sum[j] & 0xffffu);
        s_out[d] = to + hist[(size_t)d * num_tiles + blockIdx.x] - place;
        s_out[d + 1] = to + tot[2 * j] + hist[(size_t)(d + 1) * num_tiles + blockIdx.x] - second;
        unsigned at = place | second << 16;        // places are at most a tile: no carry between the halves
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const unsigned c = words[w * kPitch + w0 + j];
          words[w * kPitch + w0 + j] = at;
          at += c;
        }
        place = second + (sum[j] >> 16);
        to += tot[2 * j] + tot[2 * j + 1];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < KPT; ++i)
    if (i * 32 < left) {
      const unsigned at = cnt[(k[i] >> shift) & mask] + (i & 1 ? rank[i / 2] >> 16 : rank[i / 2] & 0xffffu);
      s_pair[at] = make_uint2(k[i], (unsigned)v[i]);
    }
  __syncthreads();
#pragma unroll 4
  for (int j = tid; j < count; j += T) {
    const uint2 q = s_pair[j];
    const unsigned to = s_out[(q.x >> shift) & mask] + (unsigned)j;
    keys_out[to] = q.x;
    vals_out[to] = (int)q.y;
  }
}

// one row: nothing to sort, the permutation is the identity
template <typename IdT>
__global__ void sort_identity_kernel(const IdT* __restrict__ ids, long long n, long long num_rows, unsigned* __restrict__ keys,
                                     int* __restrict__ vals, int* status) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  bool bad = false;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    const long long v = (long long)ids[e];
    bad |= v < 0 || v >= num_rows;
    keys[e] = (unsigned)v;
    vals[e] = (int)e;
  }
  if (bad) atomicCAS(status, 0, FLEXSPMV_ERR_BAD_ARG);
}

// First position of a key >= row in keys[0 .. n), found by a whole warp: 32 probes a round.
__device__ __forceinline__ long long warp_lower_bound(const unsigned* keys, long long n, long long row) {
  const int lane = threadIdx.x & 31;
  long long lo = 0, hi = n;
  while (lo < hi) {
    const long long step = (hi - lo + 31) / 32;
    const long long at = lo + lane * step;
    const bool less = at < hi && (long long)keys[at] < row;
    const int k = __popc(__ballot_sync(0xffffffffu, less));
    const long long next_hi = lo + k * step < hi ? lo + k * step : hi;
    if (k) lo += (k - 1) * step + 1;
    hi = next_hi;
  }
  return lo;
}
// CSR offsets of sorted ids: offsets[r] = number of ids < r.  A block owns ROWS consecutive rows: two warps find the
// run of ids of those rows (five rounds of 32 probes for 33 M ids).  Where the run is not much longer than the rows are many,
// it is read once, side by side: a place whose id differs from the one before it is where that row begins, and a row without
// ids begins where the next one does (a minimum from behind).  A longer run (few rows hold most edges) is bisected per row.
// Bound by round trips unless the rows are many.  The kernel alone, us, bisected in blocks of 256 rows / read once in blocks of 256 /
// of 1024:  8 ids a row, 10 007 rows 6.3 / 6.2 / 6.2, 100 003 6.3 / 6.2 / 7.3, 400 009 10.3 / 10.3 / 8.3, 1 M 19.5 / 16.5 / 12.4, 8 M rows
// of one id 95 / 84 / 39;  24 ids a row, 100 003 rows 7.3 / 7.2 / 10.8, 400 009 12.5 / 12.4 / 12.4;  48 ids, 100 003 rows 8.3 / 8.3 / 16.5,
// 400 009 16.6 / 18.6 / 18.5;  100 ids, 10 007 rows 6.3 / 10.3 / 28.  So: read once up to 24 ids a row, and blocks of 1024 rows where
// they are two an SM and more.
constexpr int kOffsetThreads = 256, kOffsetIdsARow = 24;
template <typename OffsetT, int ROWS>
__global__ void __launch_bounds__(kOffsetThreads) sorted_offsets_kernel(const unsigned* keys, long long n, long long num_rows, OffsetT* offsets) {
  constexpr int kPer = ROWS / kOffsetThreads;
  __shared__ long long s_run[2];
  __shared__ unsigned s_begin[ROWS];
  __shared__ unsigned s_warp[kOffsetThreads / 32];
  const long long r0 = (long long)blockIdx.x * ROWS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_launch_dependents();
  if (warp < 2) {
    const long long at = warp_lower_bound(keys, n, r0 + ROWS * warp);
    if (lane == 0) s_run[warp] = at;
  }
  for (int i = tid; i < ROWS; i += kOffsetThreads) s_begin[i] = 0xffffffffu;
  __syncthreads();
  const long long lo = s_run[0], hi = s_run[1];
  if (hi - lo > kOffsetIdsARow * ROWS) {
    // the thread's rows at once: one round trip a halving, whatever their number
    long long from[kPer], to[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) { from[j] = lo; to[j] = hi; }
    for (bool more = true; more;) {
      more = false;
#pragma unroll
      for (int j = 0; j < kPer; ++j)
        if (from[j] < to[j]) {
          const long long mid = (from[j] + to[j]) >> 1;
          if ((long long)keys[mid] < r0 + j * kOffsetThreads + tid) from[j] = mid + 1; else to[j] = mid;
          more = true;
        }
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const long long r = r0 + j * kOffsetThreads + tid;
      if (r <= num_rows) offsets[r] = (OffsetT)from[j];
    }
    return;
  }
#pragma unroll 4
  for (long long e = lo + tid; e < hi; e += kOffsetThreads) {
    const unsigned id = keys[e], row = id - (unsigned)r0;
    if ((e == lo || keys[e - 1] != id) && row < (unsigned)ROWS) s_begin[row] = (unsigned)e;    // (ids out of range are not in order)
  }
  __syncthreads();
  // a row without ids: the smallest beginning behind it, or the run's end
  unsigned b[kPer], least = 0xffffffffu;
#pragma unroll
  for (int j = kPer - 1; j >= 0; --j) {
    b[j] = s_begin[tid * kPer + j];
    least = min(least, b[j]);
  }
  unsigned behind = least;                     // smallest of this thread's rows and of the lanes behind
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_down_sync(0xffffffffu, behind, o);
    if (lane + o < 32) behind = min(behind, t);
  }
  if (lane == 0) s_warp[warp] = behind;
  __syncthreads();
  unsigned next = __shfl_down_sync(0xffffffffu, behind, 1);
  if (lane == 31) next = 0xffffffffu;
  for (int w = warp + 1; w < kOffsetThreads / 32; ++w) next = min(next, s_warp[w]);
  next = min(next, (unsigned)hi);
#pragma unroll
  for (int j = kPer - 1; j >= 0; --j) {
    next = min(next, b[j]);
    const long long r = r0 + tid * kPer + j;
    if (r <= num_rows) offsets[r] = (OffsetT)next;
  }
}

template <typename OffsetT, int ROWS>
static int sorted_offsets(const unsigned* keys, long long n, long long num_rows, void* offsets, cudaStream_t st) {
  // (the blocks cover offsets[0 .. num_rows])
  return launch_pdl(sorted_offsets_kernel<OffsetT, ROWS>, (unsigned)(num_rows / ROWS + 1), kOffsetThreads, 0, st, keys, n, num_rows, static_cast<OffsetT*>(offsets));
}

// dst[e] = src[perm[e]] for records of one machine word, read and written whole (T: the vector type of that width)
template <typename T>
__global__ void __launch_bounds__(256) permute_records_kernel(const T* __restrict__ src, T* __restrict__ dst, const int* __restrict__ perm,
                                                              long long n) {
  constexpr int kPer = 4;       // gathers in flight per thread: the records of a random permutation are L2 round trips
  const long long stride = (long long)gridDim.x * blockDim.x * kPer;
  for (long long base = (long long)blockIdx.x * blockDim.x * kPer + threadIdx.x; base < n; base += stride) {
    T r[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const long long e = base + (long long)j * blockDim.x;
      if (e < n) r[j] = src[perm[e]];
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const long long e = base + (long long)j * blockDim.x;
      if (e < n) dst[e] = r[j];
    }
  }
}
// records of any other width (a multiple of 4 bytes), or arrays whose addresses do not allow whole-record accesses
__global__ void permute_kernel(const unsigned* __restrict__ src, unsigned* __restrict__ dst, const int* __restrict__ perm,
                               long long n, int words) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n * words; i += stride) {
    const long long e = i / words;
    const int w = (int)(i - e * words);
    dst[i] = src[(long long)perm[e] * words + w];
  }
}

// One pass over `keys` (FIRST: the values are the positions, and the ids are checked).
template <typename KeyT, bool FIRST, class S>
static int sort_pass(const KeyT* keys, const int* vals, long long n, long long num_rows, int shift, unsigned* hist, unsigned* totals,
                     unsigned* keys_out, int* vals_out, int* status, cudaStream_t st) {
  const int tiles = (int)((n + S::kTile - 1) / S::kTile);
  auto scatter = sort_scatter_kernel<KeyT, FIRST, S>;
  if (S::kSmem > 48 * 1024)
    if (cudaError_t e = cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem); e != cudaSuccess) return (int)e;
  // Three kernels a pass, each a few to forty microseconds: programmatic dependent launches, so that a kernel's blocks are placed while
  // the one before drains.  Every thread waits for that kernel ahead of its first access to global memory, and the inputs are read by
  // plain loads (no __restrict__: what a pass reads was written while the kernel may already have been placed).  us, whole sort and a
  // permutation, before / after: 300 k ids of 10 007 rows 94 / 78, 3.2 M of 100 003 143 / 130, 8.4 M of 1.05 M 285 / 265, 30 M of 8 M 1172 / 1162.
  if (int e = launch_pdl(sort_count_kernel<KeyT, FIRST, S>, (unsigned)tiles, S::kThreads, 0, st, keys, n, num_rows, shift, tiles, hist, status)) return e;
  if (int e = launch_pdl(sort_scan_kernel, (unsigned)S::kBins, kScanThreads, 0, st, hist, tiles, totals)) return e;
  return launch_pdl(scatter, (unsigned)tiles, S::kThreads, S::kSmem, st, keys, vals, n, shift, tiles, hist, totals, keys_out, vals_out);
}

// All passes of S::kBits each (one alone may have fewer); `cur` says which of the two key buffers holds the sorted ids.
template <class S>
static int sort_passes(const void* ids, int id_bits, long long n, long long num_rows, int passes, int* perm, unsigned* const keys[2],
                       int* spare, unsigned* hist, unsigned* totals, int* status, cudaStream_t st, int& cur) {
  // the last pass writes the caller's permutation; the ones before it alternate with the spare buffer
  int* vals[2] = {(passes & 1) ? spare : perm, (passes & 1) ? perm : spare};
  for (int p = 0; p < passes; ++p) {
    const int to = cur ^ 1, shift = p * S::kBits;
    int e;
    if (p > 0)
      e = sort_pass<unsigned, false, S>(keys[cur], vals[cur], n, num_rows, shift, hist, totals, keys[to], vals[to], status, st);
    else if (id_bits == 32)
      e = sort_pass<int, true, S>(static_cast<const int*>(ids), nullptr, n, num_rows, 0, hist, totals, keys[to], vals[to], status, st);
    else
      e = sort_pass<long long, true, S>(static_cast<const long long*>(ids), nullptr, n, num_rows, 0, hist, totals, keys[to], vals[to], status, st);
    if (e) return e;
    cur = to;
  }
  return 0;
}

// Bytes of the counts and totals of a pass with digits of up to BITS bits.
template <class S>
static uint64_t sort_count_bytes(long long n) {
  return align_up((uint64_t)((n + S::kTile - 1) / S::kTile) * S::kBins * 4u, 256) + S::kBins * 4u;
}

static int grid_for(long long work, int block) {
  long long g = (work + block - 1) / block;
  const long long cap = 148ll * 16;
  if (g > cap) g = cap;
  return (int)(g < 1 ? 1 : g);
}

}  // namespace flex

extern "C" {

int flexspmv_sort_rows_bytes(int64_t num_edges, size_t* bytes) {
  if (!bytes || num_edges < 0) return FLEXSPMV_ERR_BAD_ARG;
  if (num_edges > 0x7fffffffLL) return FLEXSPMV_ERR_TOO_LARGE;
  // keys (2 buffers), values (1 extra buffer; the other is the caller's permutation array), digit x tile counts, digit totals
  const uint64_t wide = flex::sort_count_bytes<flex::SortWide<10>>(num_edges), narrow = flex::sort_count_bytes<flex::SortNarrow<8>>(num_edges);
  *bytes = (size_t)(flex::align_up((uint64_t)num_edges * 4u, 256) * 3 + (wide > narrow ? wide : narrow));
  return 0;
}

int flexspmv_sort_rows(const void* d_row_ids, int32_t id_bits, int64_t num_edges, int64_t num_rows, int32_t* d_perm,
                       void* d_row_offsets, int32_t offset_bits, void* d_scratch, size_t scratch_bytes, int32_t* d_status,
                       void* stream) {
  if (!d_perm || !d_row_offsets || !d_status || num_edges < 0 || num_rows < 0 || (num_edges > 0 && !d_row_ids))
    return FLEXSPMV_ERR_BAD_ARG;
  if ((id_bits != 32 && id_bits != 64) || (offset_bits != 32 && offset_bits != 64)) return FLEXSPMV_ERR_BAD_ARG;
  if (num_edges > 0x7fffffffLL || num_rows > 0x7fffffffLL) return FLEXSPMV_ERR_TOO_LARGE;
  const uint64_t seg = flex::align_up((uint64_t)num_edges * 4u, 256);
  // scratch for 8-bit digits is enough; with less than flexspmv_sort_rows_bytes says the wider ones are not taken
  const uint64_t narrow_bytes = 3 * seg + flex::sort_count_bytes<flex::SortNarrow<8>>(num_edges);
  const uint64_t wide_bytes = 3 * seg + flex::sort_count_bytes<flex::SortWide<10>>(num_edges);
  if (!d_scratch || scratch_bytes < narrow_bytes) return FLEXSPMV_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(d_scratch) & 15u) return FLEXSPMV_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaError_t e = cudaMemsetAsync(d_status, 0, sizeof(int32_t), st); e != cudaSuccess) return (int)e;
  char* base = static_cast<char*>(d_scratch);
  unsigned* const keys[2] = {reinterpret_cast<unsigned*>(base), reinterpret_cast<unsigned*>(base + seg)};
  int* spare = reinterpret_cast<int*>(base + 2 * seg);
  unsigned* hist = reinterpret_cast<unsigned*>(base + 3 * seg);
  int cur = 0;
  if (num_edges > 0) {
    int bits = 0;
    while (bits < 31 && (1ll << bits) < num_rows) ++bits;
    // 9- and 10-bit digits where one of them is enough, and two of 9 bits for three of 6 from 3 M to 5 M ids.  us, the whole sort and a
    // permutation, wide / narrow digits.  9 and 10 bits: 0.3 M ids 75 / 77, 85 / 87; 5 M 122 / 120, 132 / 133; 30 M 749 / 750, 822 / 822.  17 bits: 0.5 M 110 / 97, 2 M
    // 123 / 115, 3.2 M 141 / 146, 4 M 153 / 156, 5 M 176 / 179, 5.6 M 188 / 188, 6.5 M 208 / 204, 8.4 M 247 / 253, 30 M 1009 / 1024; 18 bits: 1 M 103 / 96, 3.2 M 130 / 133, 4 M
    // 147 / 154, 5 M 173 / 176, 6.5 M 207 / 205, 30 M 1030 / 1035.  Pairs of 10 bits (19 and 20) lose at every size: 1 M 118 / 102, 2 M 121 / 118, 4 M 170 / 154, 8.4 M 282 / 265,
    // 12 M 438 / 396; three of 9 bits for four of 7: 26 bits 4 M 320 / 312, 12 M 599 / 594, 28 bits 5 M 1081 / 985.
    const bool wide = scratch_bytes >= wide_bytes &&
        (bits == 9 || bits == 10 || ((bits == 17 || bits == 18) && num_edges >= 3'000'000 && num_edges <= 5ll << 20));
    // the totals are the last words of the scratch that the shape takes
    unsigned* totals = reinterpret_cast<unsigned*>(base + (wide ? wide_bytes : narrow_bytes)) - (wide ? flex::SortWide<10>::kBins : flex::SortNarrow<8>::kBins);
    if (bits == 0) {
      const int g = flex::grid_for(num_edges, 256);
      if (id_bits == 32)
        flex::sort_identity_kernel<int><<<g, 256, 0, st>>>(static_cast<const int*>(d_row_ids), num_edges, num_rows, keys[0], d_perm, d_status);
      else
        flex::sort_identity_kernel<long long><<<g, 256, 0, st>>>(static_cast<const long long*>(d_row_ids), num_edges, num_rows, keys[0],
                                                                 d_perm, d_status);
    } else {
      const int passes = (bits + (wide ? 9 : 7)) / (wide ? 10 : 8), width = (bits + passes - 1) / passes;
      auto sort = flex::sort_passes<flex::SortNarrow<4>>;             // 1 to 4 bits
      switch (width) {
        case 5: sort = flex::sort_passes<flex::SortNarrow<5>>; break;
        case 6: sort = flex::sort_passes<flex::SortNarrow<6>>; break;
        case 7: sort = flex::sort_passes<flex::SortNarrow<7>>; break;
        case 8: sort = flex::sort_passes<flex::SortNarrow<8>>; break;
        case 9: sort = flex::sort_passes<flex::SortWide<9>>; break;
        case 10: sort = flex::sort_passes<flex::SortWide<10>>; break;
        default: break;
      }
      if (int e = sort(d_row_ids, id_bits, num_edges, num_rows, passes, d_perm, keys, spare, hist, totals, d_status, st, cur)) return e;
    }
  }
  if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) return (int)e;
  const bool many = num_rows >= 2048ll * flex::device_sm_count() && num_edges <= flex::kOffsetIdsARow * num_rows;
  if (offset_bits == 32)
    return (many ? flex::sorted_offsets<int, 1024> : flex::sorted_offsets<int, 256>)(keys[cur], num_edges, num_rows, d_row_offsets, st);
  return (many ? flex::sorted_offsets<long long, 1024> : flex::sorted_offsets<long long, 256>)(keys[cur], num_edges, num_rows, d_row_offsets, st);
}

int flexspmv_permute_edges(const void* d_src, void* d_dst, const int32_t* d_perm, int64_t num_edges, int32_t record_bytes,
                           void* stream) {
  if (num_edges < 0 || record_bytes <= 0 || (record_bytes & 3)) return FLEXSPMV_ERR_BAD_ARG;
  if (num_edges == 0) return 0;
  if (!d_src || !d_dst || !d_perm || d_src == d_dst) return FLEXSPMV_ERR_BAD_ARG;
  const int words = record_bytes / 4;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // whole-record accesses where the width is a machine word and both addresses are multiples of it
  const uintptr_t at = reinterpret_cast<uintptr_t>(d_src) | reinterpret_cast<uintptr_t>(d_dst);
  const int g = flex::grid_for((num_edges + 3) / 4, 256);
  if (words == 1)
    flex::permute_records_kernel<unsigned><<<g, 256, 0, st>>>(static_cast<const unsigned*>(d_src), static_cast<unsigned*>(d_dst), d_perm, num_edges);
  else if (words == 2 && at % 8 == 0)
    flex::permute_records_kernel<uint2><<<g, 256, 0, st>>>(static_cast<const uint2*>(d_src), static_cast<uint2*>(d_dst), d_perm, num_edges);
  else if (words == 4 && at % 16 == 0)
    flex::permute_records_kernel<uint4><<<g, 256, 0, st>>>(static_cast<const uint4*>(d_src), static_cast<uint4*>(d_dst), d_perm, num_edges);
  else
    flex::permute_kernel<<<flex::grid_for(num_edges * words, 256), 256, 0, st>>>(static_cast<const unsigned*>(d_src), static_cast<unsigned*>(d_dst),
                                                                                 d_perm, num_edges, words);
  return (int)cudaGetLastError();
}

}  // extern "C"
