// Destination-sorted edge order, CSR offsets and the source-sorted view, built on the device.
//
// The required order is the total order (dst, src, original position); the source view orders
// sorted-edge ids by (src, sorted id).  Both are total orders without ties, so any algorithm
// gives the same arrays bit for bit: bucket the edges by node with atomics (arbitrary order
// inside a bucket), then order every bucket by itself.  Buckets are the in-/out-neighbourhoods (tens
// of edges), so a warp sorts one in its registers: up to 64 edges into a node, 128 out of one; larger
// buckets are ranked by comparison of all pairs.  Edges that come grouped by rising destination, as
// neighbour lists do, are in their buckets already: their first bucketing is skipped.  3 M edges of
// 100 000 nodes take 110 us, in any other order 252 (295 for both with every edge counted and bucketed
// twice); 2.7 M edges of 30 000 nodes, 90 each way, 121 and 367 (510).  What is left are the atomics and
// scattered words of the source view.  Up to 4 096 edges of 128 nodes are sorted by one block.
#include <algorithm>
#include <mutex>

#include "zp_common.cuh"

// Scratch of zp_csr_build_static: one fixed array per GPU that loads the library.  In host code
// this name is only a handle for cudaGetSymbolAddress, never a pointer a kernel can be given.
static __device__ __align__(256) unsigned char g_csr_static_scratch[ZP_CSR_STATIC_BYTES];

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;                          // counters per thread and scan step
constexpr int kScanSpan = kScanThreads * kScanItems;   // counters per block of a multi-block scan
constexpr int64_t kScanOneBlock = 2 * kScanSpan;       // up to here one block per array does it all

enum { kFlagEdges = 1, kFlagElements = 2 };

// Node indices come from the caller.  One outside [0, N) is never used as an address: the edge
// is left out, the flag word is raised, and zp_csr_status reports it (the arrays of such a call
// are not a valid sort).  Both views are counted in one pass; the slot that an omitted edge leaves
// in the sorted list reads as an edge 0 -> 0, so it counts for source 0.  Element numbers, when
// given, are only range-checked.
//
// A run of equal destinations within a warp is counted by one atomic.  flag[1] is raised where the
// destinations do not rise from edge to edge.
__global__ void count_kernel(int64_t E, int64_t N, const int64_t *__restrict__ src,
                             const int64_t *__restrict__ dst, const int64_t *__restrict__ z,
                             int n_elements, int32_t *cnt_dst, int32_t *cnt_src, int32_t *flag) {
  zp_after_previous();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  if (z && i < N && (uint64_t)z[i] >= (uint64_t)n_elements) atomicOr(flag, kFlagElements);
  const int64_t d = i < E ? dst[i] : -1, s = i < E ? src[i] : -1;
  const bool valid = (uint64_t)d < (uint64_t)N && (uint64_t)s < (uint64_t)N;
  if (i < E && !valid) {
    atomicOr(flag, kFlagEdges);
    if (N > 0) atomicAdd(&cnt_src[0], 1);
  }
  if (valid) atomicAdd(&cnt_src[s], 1);
  const int64_t key = valid ? d : -1;
  const int64_t before = __shfl_up_sync(0xffffffffu, key, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || before != key);
  if (valid && (heads >> lane & 1)) {
    const unsigned later = heads & ~((2u << lane) - 1u);
    atomicAdd(&cnt_dst[d], (later ? __ffs(later) - 1 : 32) - lane);
  }
  const bool falls = i < E && (!valid || (lane ? before > d : i > 0 && dst[i - 1] > d));
  if (__any_sync(0xffffffffu, falls) && lane == 0) flag[1] = 1;
}

// Exclusive scan of the two counter arrays (blockIdx.y), in place, the offsets also going to
// row_ptr / row_ptr_src with the total behind them: the counters become the fill cursors of the
// buckets.  One block walks a whole array up to kScanOneBlock counters; beyond that each block takes
// kScanSpan of them and adds up the totals of the blocks before it (written by scan_totals_kernel).
struct ScanArgs {
  int32_t *cnt[2], *ptr[2];
  int32_t *totals;                       // [2][gridDim.x], multi-block scans only
};
__device__ __forceinline__ int32_t block_exclusive_scan(int32_t v, int32_t *warp_sums, int32_t &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int32_t w = warp_sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  total = warp_sums[31];
  const int32_t before = warp ? warp_sums[warp - 1] : 0;
  __syncthreads();
  return before + inc - v;
}
__global__ void __launch_bounds__(kScanThreads) scan_totals_kernel(int64_t n, const ScanArgs a) {
  zp_after_previous();
  __shared__ int32_t sums[32];
  const int32_t *cnt = a.cnt[blockIdx.y];
  const int64_t base = (int64_t)blockIdx.x * kScanSpan + threadIdx.x * kScanItems;
  int32_t v = 0, total;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) v += base + k < n ? cnt[base + k] : 0;
  block_exclusive_scan(v, sums, total);
  if (threadIdx.x == 0) a.totals[blockIdx.y * gridDim.x + blockIdx.x] = total;
}
__global__ void __launch_bounds__(kScanThreads) scan_kernel(int64_t n, const ScanArgs a) {
  zp_after_previous();
  __shared__ int32_t sums[32];
  int32_t *cnt = a.cnt[blockIdx.y], *ptr = a.ptr[blockIdx.y];
  int64_t lo = 0, hi = n;
  int32_t carry = 0, total;
  if (gridDim.x > 1) {
    lo = (int64_t)blockIdx.x * kScanSpan;
    hi = min(n, lo + kScanSpan);
    for (int b0 = 0; b0 < (int)blockIdx.x; b0 += kScanThreads) {     // totals of the blocks before
      const int b = b0 + threadIdx.x;
      block_exclusive_scan(b < (int)blockIdx.x ? a.totals[blockIdx.y * gridDim.x + b] : 0, sums, total);
      carry += total;
    }
  }
  for (int64_t s0 = lo; s0 < hi || s0 == lo; s0 += kScanSpan) {
    const int64_t base = s0 + threadIdx.x * kScanItems;
    int32_t v[kScanItems], sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      v[k] = base + k < hi ? cnt[base + k] : 0;
      sum += v[k];
    }
    int32_t run = carry + block_exclusive_scan(sum, sums, total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (base + k < hi) {
        ptr[base + k] = run;
        cnt[base + k] = run;
      }
      run += v[k];
    }
    carry += total;
  }
  // ptr[n] = the number of elements COUNTED (edges left out for an invalid node index are not among
  // them), so that no offset range ever covers a slot nothing was written to
  if (hi == n && threadIdx.x == 0) ptr[n] = carry;
}

__global__ void bucket_kernel(int64_t E, int64_t N, const int64_t *__restrict__ src,
                              const int64_t *__restrict__ dst, const int32_t *__restrict__ flag,
                              int32_t *cursor, int32_t *tmp) {
  zp_after_previous();
  if (!flag[1]) return;                  // edge i is in place i
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = dst[i];
    if ((uint64_t)k >= (uint64_t)N || (uint64_t)src[i] >= (uint64_t)N) continue;   // flagged above
    tmp[atomicAdd(&cursor[k], 1)] = (int32_t)i;
  }
}

// 32 R keys in rising order, key r of a lane standing at 32 r + lane
template <int R, typename Key>
__device__ __forceinline__ void warp_sort(Key (&key)[R], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int p = r ^ (j / 32);
          if (p > r && (key[r] > key[p]) == ((32 * r & k) == 0)) {
            const Key t = key[r];
            key[r] = key[p];
            key[p] = t;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const Key other = __shfl_xor_sync(0xffffffffu, key[r], j);
          const bool low = ((lane & j) == 0) == (((32 * r + lane) & k) == 0);
          key[r] = low ? min(key[r], other) : max(key[r], other);
        }
      }
    }
  }
}

// whether the n keys of a bucket come in rising order
template <int R>
__device__ __forceinline__ bool bucket_rises(int n, int lane, unsigned long long (&key)[R]) {
  bool rising = true;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    unsigned long long next = __shfl_down_sync(0xffffffffu, key[r], 1);
    if (r + 1 < R) {
      const unsigned long long first = __shfl_sync(0xffffffffu, key[r + 1 < R ? r + 1 : r], 0);
      if (lane == 31) next = first;
    }
    rising = rising && (32 * r + lane + 1 >= n || key[r] < next);
  }
  return __all_sync(0xffffffffu, rising);
}
// One warp per destination node: order its edges by (src, original position), and bucket the sorted
// edges by source (into perm_src, which rank_src_kernel orders in place).  The slots past the
// kept edges read as an edge 0 -> 0 at position 0: a caller that launches per-edge kernels over all
// E slots without looking at the flag (a recorded graph replay) still indexes inside its arrays.
__global__ void rank_dst_kernel(int64_t N, int64_t E, const int64_t *__restrict__ src64,
                                const int32_t *__restrict__ row_ptr,
                                const int32_t *__restrict__ flag, const int32_t *__restrict__ tmp,
                                int32_t *perm, int32_t *src_sorted, int32_t *dst_sorted,
                                int32_t *cursor_src, int32_t *perm_src) {
  zp_after_previous();
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = row_ptr[N] + tid; i < E; i += (int64_t)gridDim.x * blockDim.x) {
    perm[i] = src_sorted[i] = dst_sorted[i] = 0;
    if (N > 0) perm_src[atomicAdd(&cursor_src[0], 1)] = (int32_t)i;      // counted for source 0
  }
  const int64_t n = tid / 32;
  const int lane = threadIdx.x % 32;
  if (n >= N) return;
  const int beg = row_ptr[n], end = row_ptr[n + 1];
  const bool bucketed = flag[1] != 0;
  // every slot of a bucket was filled by bucket_kernel with an edge id; the range test only keeps
  // a broken invariant from turning into a wild read
  auto load = [&](int i) -> unsigned long long {
    const int32_t id = bucketed ? tmp[i] : i;
    if ((uint32_t)id >= (uint64_t)E) return ~0ull;
    return ((unsigned long long)src64[id] << 32) | (uint32_t)id;
  };
  auto put = [&](unsigned long long key, int at) {
    if (key == ~0ull) return;
    const int32_t s = (int32_t)(key >> 32);
    perm[at] = (int32_t)(uint32_t)key;
    src_sorted[at] = s;
    dst_sorted[at] = (int32_t)n;
    perm_src[atomicAdd(&cursor_src[s], 1)] = at;
  };
  if (end - beg <= 64) {
    constexpr int R = 2;
    unsigned long long key[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
      key[r] = beg + 32 * r + lane < end ? load(beg + 32 * r + lane) : ~0ull;
    if (!bucket_rises(end - beg, lane, key)) warp_sort(key, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) put(key[r], beg + 32 * r + lane);
    return;
  }
  bool rising = true;
  for (int i = beg + lane; i < end; i += 32) rising = rising && (i + 1 >= end || load(i) < load(i + 1));
  rising = __all_sync(0xffffffffu, rising);
  for (int i = beg + lane; i < end; i += 32) {
    const unsigned long long key = load(i);
    int at = i;
    if (!rising) {
      at = beg;
      for (int j = beg; j < end; ++j) at += load(j) < key;
    }
    put(key, at);
  }
}

// One warp per source node: order the sorted-edge ids of its outgoing edges increasingly, in place:
// up to 128 of them in registers, more with `tmp` holding the bucket as it was.
template <int R>
__device__ __forceinline__ void sort_src_bucket(int beg, int end, int lane, const int32_t *bucket,
                                                int32_t *perm_src) {
  uint32_t key[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    key[r] = beg + 32 * r + lane < end ? (uint32_t)bucket[beg + 32 * r + lane] : ~0u;
  warp_sort(key, lane);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (beg + 32 * r + lane < end) perm_src[beg + 32 * r + lane] = (int32_t)key[r];
}
__global__ void rank_src_kernel(int64_t N, int64_t E, const int32_t *__restrict__ row_ptr_src,
                                int32_t *tmp, int32_t *perm_src) {
  zp_after_previous();
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = row_ptr_src[N] + tid; i < E; i += (int64_t)gridDim.x * blockDim.x) perm_src[i] = 0;
  const int64_t n = tid / 32;
  const int lane = threadIdx.x % 32;
  if (n >= N) return;
  const int beg = row_ptr_src[n], end = row_ptr_src[n + 1];
  if (end - beg <= 32) return sort_src_bucket<1>(beg, end, lane, perm_src, perm_src);
  if (end - beg <= 64) return sort_src_bucket<2>(beg, end, lane, perm_src, perm_src);
  if (end - beg <= 128) return sort_src_bucket<4>(beg, end, lane, perm_src, perm_src);
  for (int i = beg + lane; i < end; i += 32) tmp[i] = perm_src[i];
  __syncwarp();
  for (int i = beg + lane; i < end; i += 32) {
    const int32_t id = tmp[i];
    int rank = 0;
    for (int j = beg; j < end; ++j) rank += tmp[j] < id;
    perm_src[beg + rank] = id;          // ids are positions 0 .. E-1 written by rank_dst_kernel
  }
}

// The whole sort of a small graph by one block, everything between its arrays in shared memory: one launch for
// six.  Calls of this size are the host's to bound: EdgeGraph.build of 64 to 128 nodes and 500 to 4 096 edges in the
// order of a neighbour list 58-61 -> 44-51 us, in any other 60-72 -> 54-64; inference of 64 atoms (1 920 edges)
// 199 -> 195, forces of 100 at lmax 4 613 -> 607.  One SM takes 17 to 22 us on the device for 6 000 to 10 000 edges, where the
// five kernels take 13 once they are queued, and no pass of that size got faster; a thousand nodes are 31 buckets
// for each warp, and their 4 000 edges in any order took 159 us for 65.
constexpr int kSmallThreads = 1024, kSmallEdges = 4096, kSmallNodes = 128, kSmallReplayed = 64;
struct SmallSort {
  const int64_t *src, *dst, *z;
  int n_elements;
  int32_t *perm, *src_sorted, *dst_sorted, *row_ptr, *perm_src, *row_ptr_src, *flag;
};
// words of shared memory: offsets and cursors of both views, the buckets of both, the sources
constexpr size_t small_sort_bytes(int64_t E, int64_t N) { return sizeof(int32_t) * (4 * (size_t)(N + 1) + 3 * (size_t)E); }

__global__ void __launch_bounds__(kSmallThreads)
small_sort_kernel(int E, int N, const SmallSort a) {
  zp_after_previous();
  extern __shared__ int32_t small_s[];
  __shared__ int32_t sums[32], bits, falling;
  int32_t *const row[2] = {small_s, small_s + N + 1};
  int32_t *const cursor[2] = {row[1] + N + 1, row[1] + 2 * (N + 1)};
  int32_t *const tmp = row[1] + 3 * (N + 1), *const out = tmp + E, *const source = out + E;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = kSmallThreads / 32;
  if (threadIdx.x == 0) bits = falling = 0;
  for (int i = threadIdx.x; i < 2 * (N + 1); i += kSmallThreads) cursor[0][i] = 0;
  __syncthreads();
  // counts, as count_kernel
  for (int i0 = 0; i0 < E; i0 += kSmallThreads) {
    const int i = i0 + threadIdx.x;
    const int64_t d = i < E ? a.dst[i] : -1, s = i < E ? a.src[i] : -1;
    const bool valid = (uint64_t)d < (uint64_t)N && (uint64_t)s < (uint64_t)N;
    if (i < E && !valid) {
      atomicOr(&bits, kFlagEdges);
      if (N > 0) atomicAdd(&cursor[1][0], 1);
    }
    if (valid) {
      atomicAdd(&cursor[0][d], 1);
      atomicAdd(&cursor[1][s], 1);
    }
    if (i < E) source[i] = valid ? (int32_t)s : -1;
    const int64_t before = __shfl_up_sync(0xffffffffu, d, 1);
    if (i < E && (!valid || (lane ? before > d : i > 0 && a.dst[i - 1] > d))) falling = 1;
  }
  if (a.z)
    for (int i = threadIdx.x; i < N; i += kSmallThreads)
      if ((uint64_t)a.z[i] >= (uint64_t)a.n_elements) atomicOr(&bits, kFlagElements);
  __syncthreads();
  // offsets: every thread takes a stretch of the counters
  const int per = (N + kSmallThreads - 1) / kSmallThreads;
  for (int v = 0; v < 2; ++v) {
    const int lo = min(N, (int)threadIdx.x * per), hi = min(N, lo + per);
    int32_t sum = 0, total;
    for (int i = lo; i < hi; ++i) sum += cursor[v][i];
    int32_t run = block_exclusive_scan(sum, sums, total);
    int32_t *const ptr = v ? a.row_ptr_src : a.row_ptr;
    for (int i = lo; i < hi; ++i) {
      const int32_t n = cursor[v][i];
      ptr[i] = row[v][i] = cursor[v][i] = run;
      run += n;
    }
    if (threadIdx.x == 0) ptr[N] = row[v][N] = total;      // edges counted
  }
  if (threadIdx.x == 0) {
    a.flag[0] = bits;
    a.flag[1] = falling;
  }
  __syncthreads();
  const bool bucketed = falling != 0;
  if (bucketed) {
    for (int i = threadIdx.x; i < E; i += kSmallThreads) {
      if (source[i] >= 0) tmp[atomicAdd(&cursor[0][a.dst[i]], 1)] = i;
    }
    __syncthreads();
  }
  // destinations, as rank_dst_kernel
  for (int i = row[0][N] + threadIdx.x; i < E; i += kSmallThreads) {
    a.perm[i] = a.src_sorted[i] = a.dst_sorted[i] = 0;
    if (N > 0) out[atomicAdd(&cursor[1][0], 1)] = i;
  }
  for (int n = warp; n < N; n += warps) {
    const int beg = row[0][n], end = row[0][n + 1];
    auto load = [&](int i) -> unsigned long long {
      const int32_t id = bucketed ? tmp[i] : i;
      return ((unsigned long long)(uint32_t)source[id] << 32) | (uint32_t)id;
    };
    auto put = [&](unsigned long long key, int at) {
      const int32_t s = (int32_t)(key >> 32);
      a.perm[at] = (int32_t)(uint32_t)key;
      a.src_sorted[at] = s;
      a.dst_sorted[at] = n;
      out[atomicAdd(&cursor[1][s], 1)] = at;
    };
    if (end - beg <= 64) {
      constexpr int R = 2;
      unsigned long long key[R];
#pragma unroll
      for (int r = 0; r < R; ++r) key[r] = beg + 32 * r + lane < end ? load(beg + 32 * r + lane) : ~0ull;
      if (!bucket_rises(end - beg, lane, key)) warp_sort(key, lane);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (beg + 32 * r + lane < end) put(key[r], beg + 32 * r + lane);
    } else {
      bool rising = true;
      for (int i = beg + lane; i < end; i += 32) rising = rising && (i + 1 >= end || load(i) < load(i + 1));
      rising = __all_sync(0xffffffffu, rising);
      for (int i = beg + lane; i < end; i += 32) {
        const unsigned long long key = load(i);
        int at = i;
        if (!rising) {
          at = beg;
          for (int j = beg; j < end; ++j) at += load(j) < key;
        }
        put(key, at);
      }
    }
  }
  __syncthreads();
  // sources, as rank_src_kernel
  for (int i = row[1][N] + threadIdx.x; i < E; i += kSmallThreads) a.perm_src[i] = 0;
  for (int n = warp; n < N; n += warps) {
    const int beg = row[1][n], end = row[1][n + 1];
    if (end - beg <= 32) sort_src_bucket<1>(beg, end, lane, out, a.perm_src);
    else if (end - beg <= 64) sort_src_bucket<2>(beg, end, lane, out, a.perm_src);
    else if (end - beg <= 128) sort_src_bucket<4>(beg, end, lane, out, a.perm_src);
    else
      for (int i = beg + lane; i < end; i += 32) {
        const int32_t id = out[i];
        int rank = 0;
        for (int j = beg; j < end; ++j) rank += out[j] < id;
        a.perm_src[beg + rank] = id;
      }
  }
}

struct CsrWork {
  int32_t *flag, *cnt_dst, *cnt_src, *tmp, *totals;   // two flags and the counters side by side
  size_t bytes;
};

CsrWork carve_csr(int64_t E, int64_t N, void *base) {
  CsrWork w;
  size_t off = 0;
  auto take = [&](size_t n) {
    int32_t *p = base ? reinterpret_cast<int32_t *>(static_cast<char *>(base) + off) : nullptr;
    off += zp_align_up(n * sizeof(int32_t), 256);
    return p;
  };
  w.flag = take(2);
  w.cnt_dst = take((size_t)N + 1);
  w.cnt_src = take((size_t)N + 1);
  w.tmp = take((size_t)(E > 0 ? E : 1));
  w.totals = take((size_t)zp_ceil_div(N + 1, 1024) + 1);   // >= two per kScanSpan counters
  w.bytes = off;
  return w;
}

}  // namespace

extern "C" {

size_t zp_csr_work_bytes(int64_t n_edges, int64_t n_nodes) {
  if (n_edges < 0 || n_nodes < 0) return 0;
  return carve_csr(n_edges, n_nodes, nullptr).bytes;
}

static int csr_build(const int64_t *edge_index, int64_t E, int64_t N, int32_t *perm,
                     int32_t *src_sorted, int32_t *dst_sorted, int32_t *row_ptr, int32_t *perm_src,
                     int32_t *row_ptr_src, const int64_t *atomic_numbers, int n_elements,
                     void *work, size_t work_bytes, cudaStream_t st) {
  if (E < 0 || N < 0 || E > INT32_MAX || N >= INT32_MAX) return ZP_ERR_INVALID_ARG;
  if (!row_ptr || !row_ptr_src || !work) return ZP_ERR_INVALID_ARG;
  if (E && (!edge_index || !perm || !src_sorted || !dst_sorted || !perm_src))
    return ZP_ERR_INVALID_ARG;
  const CsrWork w = carve_csr(E, N, work);
  if (work_bytes < w.bytes) return ZP_ERR_WORKSPACE;
  const int64_t *src64 = edge_index, *dst64 = edge_index + E;
  // (in a recorded graph launches cost the host nothing, and above 64 nodes one SM is no longer the faster: 100 to 128
  // nodes, 1 000 to 4 096 edges in any order 19 to 24 us a replay, 14 to 15 with the five kernels; 64 nodes 13 to 17 and
  // 14 to 16, 32 and fewer 5 to 13 and 12 to 25)
  int64_t most = kSmallNodes;
  if (E > 0 && E <= kSmallEdges && N > kSmallReplayed && N <= most) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) cudaGetLastError();
    if (capture != cudaStreamCaptureStatusNone) most = kSmallReplayed;
  }
  if (E > 0 && E <= kSmallEdges && N > 0 && N <= most) {
    static ZpSmemOptIn opt_in;
    const size_t smem = small_sort_bytes(E, N);
    if (int rc = zp_ensure_smem(small_sort_kernel, small_sort_bytes(kSmallEdges, kSmallNodes), opt_in)) return rc;
    zp_launch(small_sort_kernel, 1, kSmallThreads, smem, st, (int)E, (int)N,
              SmallSort{src64, dst64, atomic_numbers, n_elements, perm, src_sorted, dst_sorted, row_ptr,
                        perm_src, row_ptr_src, w.flag});
    ZP_LAUNCH_CHECK("small_sort_kernel");
    return ZP_OK;
  }
  // one wave: on edges that need no bucketing it only looks at the flag
  const unsigned eb = (unsigned)std::min<int64_t>(zp_ceil_div(E > 0 ? E : 1, 256), 148 * 8);
  const unsigned nbw = (unsigned)zp_ceil_div((N > 0 ? N : 1) * 32, 256);

  ZP_CUDA(cudaMemsetAsync(w.flag, 0, (char *)w.tmp - (char *)w.flag, st));
  if (E || atomic_numbers) {
    const int64_t items = atomic_numbers && N > E ? N : E;
    zp_launch(count_kernel, (unsigned)zp_ceil_div(items > 0 ? items : 1, 256), 256, 0, st, E, N, src64,
              dst64, atomic_numbers, n_elements, w.cnt_dst, w.cnt_src, w.flag);
    ZP_LAUNCH_CHECK("count_kernel");
  }
  const ScanArgs a{{w.cnt_dst, w.cnt_src}, {row_ptr, row_ptr_src}, w.totals};
  const unsigned sb = N <= kScanOneBlock ? 1u : (unsigned)zp_ceil_div(N, kScanSpan);
  if (sb > 1) {
    zp_launch(scan_totals_kernel, dim3(sb, 2), kScanThreads, 0, st, N, a);
    ZP_LAUNCH_CHECK("scan_totals_kernel");
  }
  zp_launch(scan_kernel, dim3(sb, 2), kScanThreads, 0, st, N, a);
  ZP_LAUNCH_CHECK("scan_kernel");
  if (E) {
    zp_launch(bucket_kernel, eb, 256, 0, st, E, N, src64, dst64, w.flag, w.cnt_dst, w.tmp);
    ZP_LAUNCH_CHECK("bucket_kernel");
    zp_launch(rank_dst_kernel, nbw, 256, 0, st, N, E, src64, row_ptr, w.flag, w.tmp, perm, src_sorted,
              dst_sorted, w.cnt_src, perm_src);
    ZP_LAUNCH_CHECK("rank_dst_kernel");
    zp_launch(rank_src_kernel, nbw, 256, 0, st, N, E, row_ptr_src, w.tmp, perm_src);
    ZP_LAUNCH_CHECK("rank_src_kernel");
  }
  return ZP_OK;
}

int zp_csr_build(const int64_t *edge_index, int64_t E, int64_t N, int32_t *perm,
                 int32_t *src_sorted, int32_t *dst_sorted, int32_t *row_ptr, int32_t *perm_src,
                 int32_t *row_ptr_src, void *work, size_t work_bytes, void *stream) {
  return csr_build(edge_index, E, N, perm, src_sorted, dst_sorted, row_ptr, perm_src, row_ptr_src,
                   nullptr, 0, work, work_bytes, (cudaStream_t)stream);
}

int zp_csr_build_checked(const int64_t *edge_index, int64_t E, int64_t N,
                         const int64_t *atomic_numbers, int n_elements, int32_t *perm,
                         int32_t *src_sorted, int32_t *dst_sorted, int32_t *row_ptr,
                         int32_t *perm_src, int32_t *row_ptr_src, int32_t *flags_host, void *done,
                         void *work, size_t work_bytes, void *stream) {
  if (!flags_host || (N && !atomic_numbers)) return ZP_ERR_INVALID_ARG;
  const int rc = csr_build(edge_index, E, N, perm, src_sorted, dst_sorted, row_ptr, perm_src,
                           row_ptr_src, atomic_numbers, n_elements, work, work_bytes,
                           (cudaStream_t)stream);
  if (rc) return rc;
  ZP_CUDA(cudaMemcpyAsync(flags_host, carve_csr(E, N, work).flag, sizeof(int32_t),
                          cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  if (done) ZP_CUDA(cudaEventRecord((cudaEvent_t)done, (cudaStream_t)stream));
  return ZP_OK;
}

int zp_csr_status(const void *work, void *stream, int *status_out) {
  if (!work || !status_out) return ZP_ERR_INVALID_ARG;
  int32_t flag = 0;
  cudaStream_t st = (cudaStream_t)stream;
  ZP_CUDA(cudaMemcpyAsync(&flag, carve_csr(0, 0, const_cast<void *>(work)).flag, sizeof(flag),
                          cudaMemcpyDeviceToHost, st));
  ZP_CUDA(cudaStreamSynchronize(st));
  *status_out = flag ? ZP_ERR_INVALID_ARG : ZP_OK;
  return ZP_OK;
}

// The sort without a caller-provided work buffer and without any allocation: the scratch is the
// file-scope device array above.  Its device address is looked up once per device (first call on
// that device, with that device current) and cached; the sort itself is zp_csr_build unchanged,
// which clears the counters it needs at the start of every call.
static int static_scratch(void **out) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static void *scratch_of_device[kMaxDevices] = {nullptr};
  int dev = -1;
  ZP_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return ZP_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(mu);
  if (!scratch_of_device[dev]) {
    void *ptr = nullptr;
    ZP_CUDA(cudaGetSymbolAddress(&ptr, g_csr_static_scratch));
    scratch_of_device[dev] = ptr;
  }
  *out = scratch_of_device[dev];
  return ZP_OK;
}

int zp_csr_build_static(const int64_t *edge_index, int64_t E, int64_t N, int32_t *perm,
                        int32_t *src_sorted, int32_t *dst_sorted, int32_t *row_ptr,
                        int32_t *perm_src, int32_t *row_ptr_src, void *stream) {
  if (E < 0 || N < 0) return ZP_ERR_INVALID_ARG;
  if (E > ZP_CSR_STATIC_MAX_EDGES || N > ZP_CSR_STATIC_MAX_NODES ||
      carve_csr(E, N, nullptr).bytes > (size_t)ZP_CSR_STATIC_BYTES)
    return ZP_ERR_TOO_LARGE;
  void *scratch = nullptr;
  const int rc = static_scratch(&scratch);
  if (rc) return rc;
  return zp_csr_build(edge_index, E, N, perm, src_sorted, dst_sorted, row_ptr, perm_src,
                      row_ptr_src, scratch, (size_t)ZP_CSR_STATIC_BYTES, stream);
}

int zp_csr_static_status(void *stream, int *status_out) {
  void *scratch = nullptr;
  const int rc = static_scratch(&scratch);
  if (rc) return rc;
  return zp_csr_status(scratch, stream, status_out);
}

}  // extern "C"
