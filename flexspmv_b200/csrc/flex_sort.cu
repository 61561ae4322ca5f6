// Unsorted reducers: a stable sort of the edges by row id on the device, so that a Reducer whose index is not
// ascending can still be served by the CSR kernels.  The reference converts COO row ids to CSR offsets with
// bincount + cumsum and silently assumes the ids are already sorted
// (python_wrapper/dynamic_replace_submodule.py:20-41); here the permutation that sorts them is computed once,
// the per-edge arrays are permuted with it, and the CSR offsets come from the sorted ids.
//
// Least-significant-digit radix sort on the row ids, which are dense: ceil(log2(num_rows)) bits in as few passes of at
// most 8 bits as cover them, every pass the same width (20 bits: 3 x 7).  A pass is three launches: digit counts per
// tile of 4096 keys, one CTA per digit that scans that digit's counts over the tiles, and the stable scatter.  No block
// waits for another one.  The first pass reads the caller's ids and takes the positions as values, so there is no
// separate initialisation; the passes alternate between two buffers so that the last one writes the caller's
// permutation.  Equal digits keep their input order in every pass (see sort_scatter_kernel), so the permutation equals
// a stable argsort (bit-exact against numpy.argsort(kind="stable")).
#include <cuda_runtime.h>

#include "flex_common.cuh"

namespace flex {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortKeysPerThread = 16;
constexpr int kSortTile = kSortThreads * kSortKeysPerThread;
constexpr int kMaxRadix = 256;                // bins of the widest digit

template <typename KeyT>
__device__ __forceinline__ unsigned digit_of(KeyT key, int shift, unsigned mask) { return ((unsigned)key >> shift) & mask; }

// Per tile: number of keys with each digit -> hist[digit * num_tiles + tile].  CHECK (first pass): flags ids outside
// [0, num_rows).
template <typename KeyT, bool CHECK>
__global__ void __launch_bounds__(kSortThreads) sort_count_kernel(const KeyT* __restrict__ keys, long long n, long long num_rows,
                                                                  int shift, unsigned mask, int num_tiles,
                                                                  unsigned* __restrict__ hist, int* status) {
  __shared__ unsigned s_cnt[kMaxRadix];
  const int tid = threadIdx.x;
  s_cnt[tid] = 0;
  static_assert(kMaxRadix == kSortThreads, "one bin per thread");
  __syncthreads();
  const long long base = (long long)blockIdx.x * kSortTile + tid;
  bool bad = false;
  KeyT k[kSortKeysPerThread];           // all loads before the first atomic
#pragma unroll
  for (int i = 0; i < kSortKeysPerThread; ++i) {
    const long long e = base + i * kSortThreads;
    k[i] = e < n ? keys[e] : KeyT(0);
  }
#pragma unroll
  for (int i = 0; i < kSortKeysPerThread; ++i) {
    if (base + i * kSortThreads < n) {
      if (CHECK) bad |= (long long)k[i] < 0 || (long long)k[i] >= num_rows;
      atomicAdd(&s_cnt[digit_of(k[i], shift, mask)], 1u);     // integer counts: order does not matter
    }
  }
  if (CHECK && bad) atomicCAS(status, 0, FLEXSPMV_ERR_BAD_ARG);
  __syncthreads();
  if (tid <= (int)mask) hist[(size_t)tid * num_tiles + blockIdx.x] = s_cnt[tid];
}

// Exclusive scan over the CTA's kSortThreads threads; `total` is the sum of all.  s_warp: kSortWarps words.
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
  for (int w = 0; w < kSortWarps; ++w) {
    const unsigned c = s_warp[w];
    if (w < warp) before += c;
    sum += c;
  }
  total = sum;
  __syncthreads();          // s_warp may be reused
  return before + x - v;
}

// One CTA per digit: exclusive scan of the digit's counts over the tiles, in place; the digit's total.
__global__ void __launch_bounds__(kSortThreads) sort_scan_kernel(unsigned* __restrict__ hist, int num_tiles, unsigned* __restrict__ totals) {
  __shared__ unsigned s_warp[kSortWarps];
  unsigned* row = hist + (size_t)blockIdx.x * num_tiles;
  unsigned run = 0;
  constexpr int kPer = 4;
  for (int base = 0; base < num_tiles; base += kSortThreads * kPer) {
    unsigned v[kPer], sum = 0;
    const int i0 = base + threadIdx.x * kPer;
#pragma unroll
    for (int j = 0; j < kPer; ++j) { v[j] = i0 + j < num_tiles ? row[i0 + j] : 0u; sum += v[j]; }
    unsigned total;
    unsigned at = run + block_exclusive(sum, s_warp, total);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (i0 + j < num_tiles) row[i0 + j] = at;
      at += v[j];
    }
    run += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = run;
}

// Stable scatter of one pass.  Bound by memory traffic (8 bytes in and 8 out per key) once the stores leave in runs:
// a warp ranks its 512 consecutive keys 32 at a time (lanes with the same digit find one another with one vote per bit
// of the digit -- __match_any_sync took four times as long, 80 us a pass; the rank counts the lanes below), the tile is put in digit order in shared memory and leaves from there, so that a digit's
// keys are stored side by side.  Storing straight from the ranks would touch a sector per key.  Order: warps own
// consecutive runs of keys, a warp's rounds follow one another and lanes are ranked in order, so equal digits never
// change places.  FIRST: the values are the positions.
// Measured (8.4 M 64-bit ids, 1 M rows, B200): the whole sort with offsets and one permuted tensor 1106 us with 4-bit
// digits, a one-CTA scan of all counts and stores straight from the ranks; 334 us like this (a pass 70 us).
template <typename KeyT, bool FIRST>
__global__ void __launch_bounds__(kSortThreads, 4) sort_scatter_kernel(const KeyT* __restrict__ keys_in, const int* __restrict__ vals_in,
                                                                    long long n, int shift, unsigned mask, int num_tiles,
                                                                    const unsigned* __restrict__ hist,
                                                                    const unsigned* __restrict__ totals,
                                                                    unsigned* __restrict__ keys_out, int* __restrict__ vals_out) {
  __shared__ unsigned short s_cnt[kSortWarps][kMaxRadix + 1];    // the last bin takes the lanes behind the end
  __shared__ unsigned s_out[kMaxRadix];                          // where the digit's run goes, less its place in the tile
  __shared__ unsigned short s_first[kMaxRadix];                  // the digit's place in the tile
  __shared__ unsigned s_warp[kSortWarps];
  __shared__ unsigned s_key[kSortTile];
  __shared__ int s_val[kSortTile];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long tile0 = (long long)blockIdx.x * kSortTile;
  const int count = (int)(n - tile0 < kSortTile ? n - tile0 : kSortTile);
  for (int i = tid; i < kSortWarps * (kMaxRadix + 1); i += kSortThreads) (&s_cnt[0][0])[i] = 0;
  unsigned k[kSortKeysPerThread];
  int v[kSortKeysPerThread];
  const int mine = warp * (32 * kSortKeysPerThread) + lane;      // place of the lane's first key in the tile
#pragma unroll
  for (int i = 0; i < kSortKeysPerThread; ++i) {
    const int at = mine + i * 32;
    k[i] = 0; v[i] = 0;
    if (at < count) {
      k[i] = (unsigned)keys_in[tile0 + at];
      v[i] = FIRST ? (int)(tile0 + at) : vals_in[tile0 + at];
    }
  }
  __syncthreads();
  unsigned rank[kSortKeysPerThread];
#pragma unroll
  for (int i = 0; i < kSortKeysPerThread; ++i) {
    const bool in = mine + i * 32 < count;
    const unsigned d = in ? digit_of(k[i], shift, mask) : (unsigned)kMaxRadix;
    unsigned same = __ballot_sync(0xffffffffu, in);
    if (!in) same = ~same;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if ((mask >> b) == 0) break;                              // the same for every lane
      const unsigned set = __ballot_sync(0xffffffffu, (d >> b) & 1u);
      same &= (d >> b) & 1u ? set : ~set;
    }
    const unsigned below = __popc(same & ((1u << lane) - 1u));
    const unsigned seen = s_cnt[warp][d];
    __syncwarp();
    if (below == 0) s_cnt[warp][d] = (unsigned short)(seen + __popc(same));
    __syncwarp();
    rank[i] = seen + below;
  }
  __syncthreads();
  {
    // thread = digit: the warps' counts become places behind the warps before; the digits' places follow one another
    unsigned mine_d = 0;
    for (int w = 0; w < kSortWarps; ++w) {
      const unsigned c = s_cnt[w][tid];
      s_cnt[w][tid] = (unsigned short)mine_d;
      mine_d += c;
    }
    const bool real = tid <= (int)mask;
    unsigned sum;
    const unsigned place = block_exclusive(mine_d, s_warp, sum);
    const unsigned global = block_exclusive(real ? totals[tid] : 0u, s_warp, sum);
    s_first[tid] = (unsigned short)place;
    if (real) s_out[tid] = global + hist[(size_t)tid * num_tiles + blockIdx.x] - place;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSortKeysPerThread; ++i)
    if (mine + i * 32 < count) {
      const unsigned d = digit_of(k[i], shift, mask);
      const unsigned at = s_first[d] + s_cnt[warp][d] + rank[i];
      s_key[at] = k[i];
      s_val[at] = v[i];
    }
  __syncthreads();
  for (int j = tid; j < count; j += kSortThreads) {
    const unsigned key = s_key[j];
    const unsigned to = s_out[digit_of(key, shift, mask)] + (unsigned)j;
    keys_out[to] = key;
    vals_out[to] = s_val[j];
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
__device__ __forceinline__ long long warp_lower_bound(const unsigned* __restrict__ keys, long long n, long long row) {
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
// CSR offsets of sorted ids: offsets[r] = number of ids < r.  A block owns 256 consecutive rows: two warps find the run
// of ids of those rows (five rounds of 32 probes for 33 M ids), then every row bisects inside that run, which is a few
// kilobytes on average and stays in L1 -- against a bisection over all ids per row (1 M rows, 8.4 M ids: 48 us).
template <typename OffsetT>
__global__ void __launch_bounds__(256) sorted_offsets_kernel(const unsigned* __restrict__ keys, long long n, long long num_rows,
                                                             OffsetT* __restrict__ offsets) {
  __shared__ long long s_run[2];
  const long long r0 = (long long)blockIdx.x * 256;
  const int warp = threadIdx.x >> 5;
  if (warp < 2) {
    const long long at = warp_lower_bound(keys, n, r0 + 256 * warp);
    if ((threadIdx.x & 31) == 0) s_run[warp] = at;
  }
  __syncthreads();
  const long long r = r0 + threadIdx.x;
  if (r > num_rows) return;
  long long lo = s_run[0], hi = s_run[1];
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if ((long long)keys[mid] < r) lo = mid + 1; else hi = mid;
  }
  offsets[r] = (OffsetT)lo;
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

template <typename IdT>
static void sort_first_pass(const IdT* ids, long long n, long long num_rows, unsigned mask, int tiles, unsigned* hist, unsigned* totals,
                            unsigned* keys_out, int* vals_out, int* status, cudaStream_t st) {
  sort_count_kernel<IdT, true><<<tiles, kSortThreads, 0, st>>>(ids, n, num_rows, 0, mask, tiles, hist, status);
  sort_scan_kernel<<<mask + 1, kSortThreads, 0, st>>>(hist, tiles, totals);
  sort_scatter_kernel<IdT, true><<<tiles, kSortThreads, 0, st>>>(ids, nullptr, n, 0, mask, tiles, hist, totals, keys_out, vals_out);
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
  const uint64_t blocks = (uint64_t)(num_edges + flex::kSortTile - 1) / flex::kSortTile;
  // keys (2 buffers), values (1 extra buffer; the other is the caller's permutation array), digit x tile counts, digit totals
  *bytes = (size_t)(flex::align_up((uint64_t)num_edges * 4u, 256) * 3 + flex::align_up(blocks * flex::kMaxRadix * 4u, 256) +
                    flex::kMaxRadix * 4u);
  return 0;
}

int flexspmv_sort_rows(const void* d_row_ids, int32_t id_bits, int64_t num_edges, int64_t num_rows, int32_t* d_perm,
                       void* d_row_offsets, int32_t offset_bits, void* d_scratch, size_t scratch_bytes, int32_t* d_status,
                       void* stream) {
  if (!d_perm || !d_row_offsets || !d_status || num_edges < 0 || num_rows < 0 || (num_edges > 0 && !d_row_ids))
    return FLEXSPMV_ERR_BAD_ARG;
  if ((id_bits != 32 && id_bits != 64) || (offset_bits != 32 && offset_bits != 64)) return FLEXSPMV_ERR_BAD_ARG;
  if (num_edges > 0x7fffffffLL || num_rows > 0x7fffffffLL) return FLEXSPMV_ERR_TOO_LARGE;
  size_t need = 0;
  if (int e = flexspmv_sort_rows_bytes(num_edges, &need)) return e;
  if (!d_scratch || scratch_bytes < need) return FLEXSPMV_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(d_scratch) & 15u) return FLEXSPMV_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaError_t e = cudaMemsetAsync(d_status, 0, sizeof(int32_t), st); e != cudaSuccess) return (int)e;
  const uint64_t seg = flex::align_up((uint64_t)num_edges * 4u, 256);
  char* base = static_cast<char*>(d_scratch);
  unsigned* keys[2] = {reinterpret_cast<unsigned*>(base), reinterpret_cast<unsigned*>(base + seg)};
  int* spare = reinterpret_cast<int*>(base + 2 * seg);
  unsigned* hist = reinterpret_cast<unsigned*>(base + 3 * seg);
  const int tiles = (int)((num_edges + flex::kSortTile - 1) / flex::kSortTile);
  char* behind = base + 3 * seg + flex::align_up((uint64_t)tiles * flex::kMaxRadix * 4u, 256);
  unsigned* totals = reinterpret_cast<unsigned*>(behind);
  int cur = 0;
  if (num_edges > 0) {
    int bits = 0;
    while (bits < 31 && (1ll << bits) < num_rows) ++bits;
    const int passes = (bits + 7) / 8;
    if (passes == 0) {
      const int g = flex::grid_for(num_edges, 256);
      if (id_bits == 32)
        flex::sort_identity_kernel<int><<<g, 256, 0, st>>>(static_cast<const int*>(d_row_ids), num_edges, num_rows, keys[0], d_perm, d_status);
      else
        flex::sort_identity_kernel<long long><<<g, 256, 0, st>>>(static_cast<const long long*>(d_row_ids), num_edges, num_rows, keys[0],
                                                                 d_perm, d_status);
    } else {
      const int width = (bits + passes - 1) / passes;
      const unsigned mask = (1u << width) - 1u;
      // the last pass writes the caller's permutation; the ones before it alternate with the spare buffer
      int* vals[2] = {(passes & 1) ? spare : d_perm, (passes & 1) ? d_perm : spare};
      for (int p = 0; p < passes; ++p) {
        const int shift = p * width, to = cur ^ 1;
        if (p == 0 && id_bits == 32)
          flex::sort_first_pass<int>(static_cast<const int*>(d_row_ids), num_edges, num_rows, mask, tiles, hist, totals, keys[to], vals[to], d_status, st);
        else if (p == 0)
          flex::sort_first_pass<long long>(static_cast<const long long*>(d_row_ids), num_edges, num_rows, mask, tiles, hist, totals, keys[to],
                                           vals[to], d_status, st);
        else {
          flex::sort_count_kernel<unsigned, false><<<tiles, flex::kSortThreads, 0, st>>>(keys[cur], num_edges, num_rows, shift, mask, tiles, hist, d_status);
          flex::sort_scan_kernel<<<mask + 1, flex::kSortThreads, 0, st>>>(hist, tiles, totals);
          flex::sort_scatter_kernel<unsigned, false><<<tiles, flex::kSortThreads, 0, st>>>(keys[cur], vals[cur], num_edges, shift, mask, tiles,
                                                                                           hist, totals, keys[to], vals[to]);
        }
        cur = to;
      }
    }
  }
  if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) return (int)e;
  const unsigned g = (unsigned)((num_rows + 256) / 256);
  if (offset_bits == 32)
    flex::sorted_offsets_kernel<int><<<g, 256, 0, st>>>(keys[cur], num_edges, num_rows, static_cast<int*>(d_row_offsets));
  else
    flex::sorted_offsets_kernel<long long><<<g, 256, 0, st>>>(keys[cur], num_edges, num_rows, static_cast<long long*>(d_row_offsets));
  return (int)cudaGetLastError();
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
