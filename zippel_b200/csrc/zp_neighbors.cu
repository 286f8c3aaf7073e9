// Periodic neighbour list with the per-destination cap, built on the device.
//
// The graph front end of the block: all directed edges src -> dst with
//     d2 = |pos[dst] - pos[src] + shift|^2 < cutoff^2,   shift = image * box,
// in a cubic periodic box, without the self pair at zero shift, keeping per destination the
// `max_neighbors` edges of smallest (d2, src, shift_x, shift_y, shift_z).  The reference builds
// its edge lists on the host with an external neighbour-list package and applies no cap
// (fixtures/make_fixtures.py:13-15, 78-100); the cap and the order are defined by this library.
//
// Output order is (dst, src, shift_x, shift_y, shift_z), i.e. already the destination-sorted form,
// with row_ptr.  Everything is a function of exact fp64 arithmetic written without contraction
//     dx = (pos[dst].x - pos[src].x) + shift_x;   d2 = (dx*dx + dy*dy) + dz*dz
// and of total orders without ties, so the arrays are reproducible bit for bit and equal to the
// host statement of the same rule.
//
// Method: uniform cells of edge >= cutoff / w (w = 2, or 1 where atoms are sparse, or more where
// the box is smaller than the cutoff); one warp per destination walks the (2w+1)^2 columns of cells
// around it in unwrapped cell coordinates, each cut to the stretch that the cutoff can reach; the
// unwrapped coordinate gives both the wrapped cell and the periodic image, so every
// (source, image) pair is visited at most once.  The atoms are copied in cell order with their own
// image numbers, so the walk reads them with whole-line loads and divides nothing, and the
// columns of a walk are laid end to end so that no lane waits at a column's end.  Pass 1 collects the
// hits of an atom and, when the cap binds, selects the nearest by closing in on a distance that
// parts off exactly `cap` of them (ranking all when equal distances stand in the way); the survivors
// are placed by counting the smaller (src, image) keys and kept in the workspace.  A scan of their
// numbers gives row_ptr, and pass 2 writes the edges out.  Atoms of more than 192 hits are only counted
// in pass 1 (up to the cap); pass 2 walks them again and selects by a bitonic sort on (d2, src, image)
// in shared memory.
#include <algorithm>
#include <cmath>

#include "zp_common.cuh"
#include "zippel_b200.h"

namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kHitCap = ZP_NEIGHBORS_MAX_HITS;     // hits held per destination in shared memory
constexpr int kFewHits = 192;                      // ... in registers, six per lane
constexpr int kKept = 128;                         // edges per destination kept from pass 1 to 2
constexpr int kScanBlock = 1024;

struct Grid {
  double box, per_cell;            // per_cell: cells per unit of length
  int nc;          // cells per dimension
  int w;           // search half-width in cells
  int reach;       // largest |image| component that can occur
  struct Sphere {
    double r2;     // pairs closer than its root
    float reach2;  // (radius / cell)^2 and a margin for working in fp32
    int w;         // half-width in cells
  } all, near;     // the cutoff; where a cap binds, what most probably holds that many (else all again)
};

// words of the workspace's head: error bits, whether an atom lies outside the box, crowded atoms
enum { kFlagBits = 0, kUnwrapped = 1, kCrowdedList = 3 };

struct Hit {
  double d2;
  unsigned long long tie;      // src << 32 | image code (ascending = ascending shift tuple)
};

__device__ __forceinline__ bool hit_less(const Hit &a, const Hit &b) {
  return a.d2 < b.d2 || (a.d2 == b.d2 && a.tie < b.tie);
}

// Positions may lie outside [0, box): o = floor(p / box) is the atom's own image offset and
// p - o * box its wrapped coordinate, used only to pick the cell.  Distances are always taken
// between the positions as given.
__device__ __forceinline__ int own_image(double p, const Grid &g) { return (int)floor(p / g.box); }
__device__ __forceinline__ int clamp_cell(double p, const Grid &g) {
  const int c = (int)floor(p);
  return c < 0 ? 0 : (c >= g.nc ? g.nc - 1 : c);
}
__device__ __forceinline__ int cell_coord(double p, const Grid &g) {
  return clamp_cell((p - floor(p / g.box) * g.box) * g.per_cell, g);
}

__device__ __forceinline__ int floor_div(int a, int n) {
  int q = a / n;
  if ((a % n) < 0) --q;
  return q;
}
// image that the unwrapped cell coordinate a, at most w outside [0, nc), lies in
__device__ __forceinline__ int cell_image(int a, const Grid &g) {
  return g.w > g.nc ? floor_div(a, g.nc) : a < 0 ? -1 : a >= g.nc;
}

// Image code.  The shift of a hit is (o_src - o_dst - k) * box with k the image found in wrapped
// coordinates (|k| <= reach) and o the atoms' own offsets.  For one (dst, src) pair the offsets
// are fixed, so ordering by -k orders by shift: the code holds -k only, and the writer adds the
// offsets back.
__device__ __forceinline__ unsigned image_code(int nkx, int nky, int nkz, int reach) {
  const unsigned s = 2u * reach + 1u;
  return ((unsigned)(nkx + reach) * s + (unsigned)(nky + reach)) * s + (unsigned)(nkz + reach);
}

__global__ void cell_count_kernel(int64_t N, const double *__restrict__ pos, Grid g,
                                  int32_t *__restrict__ atom_cell, int4 *__restrict__ own,
                                  int32_t *cell_count, int32_t *flags) {
  zp_after_previous();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
  const double far = 1.0e6 * g.box;
  if (!(fabs(x) < far && fabs(y) < far && fabs(z) < far))
    atomicOr(flags, 1);                               // not finite, or absurdly far from the box
  const int c = (cell_coord(x, g) * g.nc + cell_coord(y, g)) * g.nc + cell_coord(z, g);
  atom_cell[i] = c;
  const int4 mine = make_int4(own_image(x, g), own_image(y, g), own_image(z, g), (int)i);
  own[i] = mine;
  if (mine.x | mine.y | mine.z) flags[kUnwrapped] = 1;
  atomicAdd(&cell_count[c], 1);
}

// atoms in cell order: coordinates and {own image, index}
struct Sorted {
  double *x, *y, *z;
  int4 *who;
};
__global__ void cell_fill_kernel(int64_t N, const double *__restrict__ pos, Grid g,
                                 const int32_t *__restrict__ atom_cell,
                                 const int4 *__restrict__ own, const int32_t *__restrict__ cell_start, int32_t *cell_cursor,
                                 const Sorted out) {
  zp_after_previous();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int c = atom_cell[i];
  const int at = cell_start[c] + atomicAdd(&cell_cursor[c], 1);
  out.x[at] = pos[3 * i];
  out.y[at] = pos[3 * i + 1];
  out.z[at] = pos[3 * i + 2];
  out.who[at] = own[i];
}

// exclusive scan of n ints (n + 1 outputs, the last is the total): block scans, then each
// block adds the totals of those before it
__global__ void scan_block_kernel(int64_t n, const int32_t *__restrict__ in, int32_t *out,
                                  int32_t *block_sums) {
  zp_after_previous();
  __shared__ int32_t s[kScanBlock];
  const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  const int32_t mine = i < n ? in[i] : 0;
  s[threadIdx.x] = mine;
  __syncthreads();
  for (int off = 1; off < kScanBlock; off <<= 1) {
    const int32_t v = threadIdx.x >= off ? s[threadIdx.x - off] : 0;
    __syncthreads();
    s[threadIdx.x] += v;
    __syncthreads();
  }
  if (i <= n) out[i] = s[threadIdx.x] - mine;
  if (threadIdx.x == kScanBlock - 1) block_sums[blockIdx.x] = s[threadIdx.x];
}
__global__ void __launch_bounds__(kScanBlock)
scan_add_kernel(int64_t n, int32_t *out, const int32_t *__restrict__ block_sums) {
  zp_after_previous();
  __shared__ int32_t before;             // totals of the blocks before this one
  if (threadIdx.x == 0) before = 0;
  __syncthreads();
  int32_t sum = 0;
  for (unsigned b = threadIdx.x; b < blockIdx.x; b += kScanBlock) sum += block_sums[b];
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (threadIdx.x % 32 == 0 && sum) atomicAdd(&before, sum);
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  if (i <= n) out[i] += before;
}

int exclusive_scan(int64_t n, const int32_t *in, int32_t *out, int32_t *block_sums,
                   cudaStream_t st) {
  const int64_t nb = zp_ceil_div(n + 1, kScanBlock);
  zp_launch(scan_block_kernel, (unsigned)nb, kScanBlock, 0, st, n, in, out, block_sums);
  ZP_LAUNCH_CHECK("scan_block_kernel");
  zp_launch(scan_add_kernel, (unsigned)nb, kScanBlock, 0, st, n, out, block_sums);
  ZP_LAUNCH_CHECK("scan_add_kernel");
  return ZP_OK;
}

// Calls f(hit, src, image code, d2) on all 32 lanes together for every batch of candidate
// (source, image) pairs around destination j; `hit` marks the lanes whose candidate lies within
// the sphere.  The walk goes on while f returns true (the same on all lanes).  Bound by instruction
// issue: what hangs on images alone is formed once per column, and the conversions and products
// of a shift are left out where it is zero (in a large cell, for most atoms).
constexpr int kNoImage = 512 | 512 << 10 | 512 << 20;
template <typename F>
__device__ __forceinline__ void for_each_hit(const Grid &g, const Grid::Sphere &ball,
                                             const int32_t *__restrict__ cell_start,
                                             const Sorted &atoms, int64_t at, int lane, F &&f) {
  const double xj = atoms.x[at], yj = atoms.y[at], zj = atoms.z[at];
  const int4 own = atoms.who[at];
  // cell, and where in it (in cells)
  const double wx = (xj - own.x * g.box) * g.per_cell, wy = (yj - own.y * g.box) * g.per_cell,
               wz = (zj - own.z * g.box) * g.per_cell;
  const int cx = clamp_cell(wx, g), cy = clamp_cell(wy, g), cz = clamp_cell(wz, g);
  const float fx = (float)(wx - cx), fy = (float)(wy - cy), fz = (float)(wz - cz);
  const int w = ball.w, side = 2 * w + 1, columns = side * side;
  const int kz1 = cell_image(cz + w, g);
  for (int q0 = 0; q0 < columns; q0 += 32) {
    // a lane per column of cells along z, cut to what the cutoff can reach
    const int q = q0 + lane;
    const int ox = q / side - w, oy = q % side - w;
    const float ax = ox > 0 ? ox - fx : ox < 0 ? fx - (ox + 1) : 0.f;
    const float ay = oy > 0 ? oy - fy : oy < 0 ? fy - (oy + 1) : 0.f;
    const float r2 = ball.reach2 - (ax * ax + ay * ay);
    const bool in = q < columns && r2 > 0.f;
    const float r = in ? sqrtf(r2) : 0.f;
    const int u0 = max(cz - w, cz + (int)floorf(fz - r)), u1 = min(cz + w, cz + (int)floorf(fz + r));
    const int kx = cell_image(cx + ox, g), ky = cell_image(cy + oy, g);
    const int column = ((cx + ox - kx * g.nc) * g.nc + (cy + oy - ky * g.nc)) * g.nc;
    for (int kz = cell_image(cz - w, g); kz <= kz1; ++kz) {
      const int z0 = max(u0 - kz * g.nc, 0), z1 = min(u1 - kz * g.nc, g.nc - 1);
      int off = 0, len = 0;
      const int image = (512 - kx) | (512 - ky) << 10 | (512 - kz) << 20;
      const unsigned image_place = image_code(-kx, -ky, -kz, g.reach);
      if (in && z0 <= z1) {
        off = cell_start[column + z0];
        len = cell_start[column + z1 + 1] - off;
      }
      int upto = len;                              // candidates of the columns up to this one
  #pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += u;
      }
      const int total = __shfl_sync(0xffffffffu, upto, 31);
      off -= upto - len;
      for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        int cell = 0;                              // the column candidate t belongs to
  #pragma unroll
        for (int b = 16; b > 0; b >>= 1) {
          const int v = __shfl_sync(0xffffffffu, upto, cell + b - 1);
          if (v <= t) cell += b;
        }
        const int a = __shfl_sync(0xffffffffu, off, cell) + t;
        const int im = __shfl_sync(0xffffffffu, image, cell);
        const unsigned code = __shfl_sync(0xffffffffu, image_place, cell);
        bool hit = false;
        int i = 0;
        double d2 = 0.0;
        if (t < total) {
          const int4 who = atoms.who[a];
          i = who.w;
          // the source's wrapped copy sits k boxes away in wrapped coordinates:
          // pos[j] - (pos[i] - o_i box + k box) stays as (pos[j] - pos[i]) + (o_i - o_j - k) box
          // once the destination's own offset o_j is taken out of the search origin
          double dx = __dsub_rn(xj, atoms.x[a]), dy = __dsub_rn(yj, atoms.y[a]),
                 dz = __dsub_rn(zj, atoms.z[a]);
          const bool shifted = im != kNoImage || who.x != own.x || who.y != own.y || who.z != own.z;
          bool self = i == own.w;
          if (shifted) {
            const int mx = who.x - own.x + (im & 1023) - 512, my = who.y - own.y + (im >> 10 & 1023) - 512,
                      mz = who.z - own.z + (im >> 20 & 1023) - 512;
            dx = __dadd_rn(dx, __dmul_rn((double)mx, g.box));
            dy = __dadd_rn(dy, __dmul_rn((double)my, g.box));
            dz = __dadd_rn(dz, __dmul_rn((double)mz, g.box));
            self = self && mx == 0 && my == 0 && mz == 0;
          }
          d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
          hit = d2 < ball.r2 && !self;
        }
        if (!f(hit, i, code, d2)) return;
      }
    }
  }
}

// bitonic sort of the first n2 (a power of two) entries of h by `less`, one warp
template <typename Less>
__device__ __forceinline__ void warp_bitonic(Hit *h, int n2, int lane, Less less) {
  for (int k = 2; k <= n2; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = lane; i < n2; i += 32) {
        const int p = i ^ j;
        if (p > i) {
          const Hit a = h[i], b = h[p];
          const bool up = (i & k) == 0;
          if (up ? less(b, a) : less(a, b)) { h[i] = b; h[p] = a; }
        }
      }
      __syncwarp();
    }
  }
}

__device__ __forceinline__ int pow2_at_least(int n) {
  int p = 1;
  while (p < n) p <<= 1;
  return p;
}

// Writes edge `place` of destination j, whose source and image are in `tie`.
struct Writer {
  const int4 *own;
  const Grid &g;
  bool unwrapped;          // atoms have images of their own
  int64_t E, j, base;
  int64_t *edge_index;
  double *shifts;
  __device__ __forceinline__ void put_pair(unsigned long long tie, int place) const {
    edge_index[base + place] = (int64_t)(tie >> 32);
    edge_index[E + base + place] = j;
  }
  // component `v % 3` of the shift of edge `v / 3`
  __device__ __forceinline__ void put_shift(unsigned long long tie, int v) const {
    const unsigned code = (unsigned)(tie & 0xffffffffu);
    double shift = 0.0;
    if (unwrapped || code != image_code(0, 0, 0, g.reach)) {
      const unsigned s = 2u * g.reach + 1u, axis = v % 3;
      int m = (int)((axis == 0 ? code / (s * s) : axis == 1 ? code / s : code) % s) - g.reach;
      if (unwrapped) {
        const int *image = reinterpret_cast<const int *>(own);
        m += image[4 * (int64_t)(tie >> 32) + axis] - image[4 * j + axis];
      }
      shift = (double)m * g.box;
    }
    shifts[3 * base + v] = shift;
  }
};

// Moves the ties of the `cap` nearest of the n <= 32 R hits to the front, n > cap > 0.
template <int R>
__device__ __forceinline__ void keep_nearest(Hit *h, int n, int cap, float radius2, int lane) {
      float near[R];                // rounding to fp32 keeps the order, or makes equals
#pragma unroll
      for (int k = 0; k < R; ++k) near[k] = lane + 32 * k < n ? (float)h[lane + 32 * k].d2 : INFINITY;
      // close in on a distance that exactly `cap` hits do not exceed: by interpolation and by halves
      float lo = 0.f, hi = radius2;
      int below_lo = 0, below_hi = n;
      unsigned alive[R];            // survivors, a bit per lane
      bool found = false;
      for (int step = 0; step < 32 && !found; ++step) {
        const float part = step & 1 ? 0.5f : (cap - below_lo) / (float)(below_hi - below_lo);
        const float mid = lo + (hi - lo) * part;
        int below = 0;
#pragma unroll
        for (int k = 0; k < R; ++k) {
          alive[k] = __ballot_sync(0xffffffffu, near[k] <= mid);
          below += __popc(alive[k]);
        }
        found = below == cap;
        if (below < cap) {
          lo = mid;
          below_lo = below;
        } else {
          hi = mid;
          below_hi = below;
        }
      }
      if (!found) {                 // equal distances at the cap: rank by (d2, src, image)
        for (int k = 0; k < R; ++k) {
          const int own_t = lane + 32 * k;
          const Hit mine = h[own_t < n ? own_t : 0];
          int rank = 0;
          for (int t = 0; t < n; ++t) rank += hit_less(h[t], mine);
          alive[k] = __ballot_sync(0xffffffffu, own_t < n && rank < cap);
        }
      }
      // survivors to the front
      unsigned long long tie[R];
#pragma unroll
      for (int k = 0; k < R; ++k) tie[k] = h[lane + 32 * k].tie;
      __syncwarp();
      int slot = 0;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        if (alive[k] >> lane & 1) h[slot + __popc(alive[k] & ((1u << lane) - 1u))].tie = tie[k];
        slot += __popc(alive[k]);
      }
      __syncwarp();
}

// Pass 1, a warp per destination, its hits compacted in 3 KB of shared memory so that an SM holds its
// full count of warps: the survivors of destination j go to kept[j][0 ...] in their final order.  One
// with more than kFewHits hits or kKept survivors goes on the list `crowded` instead, its row of
// `kept` marked: 192 hits because a warp walking again alone costs as much as a third of all others
// (57 us for the few atoms in 100 000 that have more than 128 where the mean is 90).  Bound by
// instruction issue: 175 us for 100 000 atoms, 90 hits each, cap 30, where a count of 90 us came before
// 235 us of this; 186 with four blocks per SM instead of five (48 registers, no spills).
constexpr int kSelectWarps = 8;
constexpr unsigned long long kCrowded = ~0ull;
__global__ void __launch_bounds__(32 * kSelectWarps, 5)
select_kernel(int64_t N, Grid g, const int32_t *__restrict__ cell_start, const Sorted atoms, int cap,
              int32_t *__restrict__ counts, unsigned long long *__restrict__ kept, int stride, int32_t *flags,
              int32_t *__restrict__ crowded) {
  zp_after_previous();
  __shared__ Hit hits[kSelectWarps][kFewHits];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int64_t at = (int64_t)blockIdx.x * kSelectWarps + warp;
  if (at >= N) return;
  const int64_t j = atoms.who[at].w;           // in cell order: neighbours read the same cells
  Hit *h = hits[warp];
  int n = 0;                      // hits seen (warp-uniform)
  bool everything = g.near.r2 == g.all.r2;
  for (;;) {
    for_each_hit(g, everything ? g.all : g.near, cell_start, atoms, at, lane,
                 [&](bool hit, int i, unsigned code, double d2) {
                   const unsigned m = __ballot_sync(0xffffffffu, hit);
                   const int slot = n + __popc(m & ((1u << lane) - 1u));
                   if (hit && slot < kFewHits) {
                     h[slot].d2 = d2;
                     h[slot].tie = ((unsigned long long)(unsigned)i << 32) | code;
                   }
                   n += __popc(m);
                   return n <= kFewHits || cap <= 0 || n < cap;    // past both the count is known
                 });
    if (everything || n >= cap) break;
    everything = true;            // fewer than the cap so near: all within the cutoff
    n = 0;
    __syncwarp();
  }
  kept += j * stride;
  if (n > kFewHits || (n > kKept && (cap <= 0 || cap > kKept))) {             // left to fill_many_kernel
    if (lane == 0) {
      if (cap <= 0 && n > kHitCap) atomicOr(flags, 2);     // uncapped list too long for it
      counts[j] = cap > 0 && n > cap ? cap : n;
      kept[0] = kCrowded;
      crowded[1 + atomicAdd(&crowded[0], 1)] = (int32_t)at;
    }
    return;
  }
  __syncwarp();
  if (cap > 0 && n > cap) {
    if (n <= 64)
      keep_nearest<2>(h, n, cap, (float)(everything ? g.all : g.near).r2, lane);
    else if (n <= 128)
      keep_nearest<4>(h, n, cap, (float)(everything ? g.all : g.near).r2, lane);
    else
      keep_nearest<kFewHits / 32>(h, n, cap, (float)(everything ? g.all : g.near).r2, lane);
    n = cap;
  }
  if (lane == 0) counts[j] = n;
  // place of a survivor = number of survivors with a smaller (src, image)
  for (int t = lane; t < n; t += 32) {
    const unsigned long long mine = h[t].tie;
    int rank = 0;
#pragma unroll 4
    for (int q = 0; q < n; ++q) rank += h[q].tie < mine;
    kept[rank] = mine;
  }
}

// Pass 2, a warp per destination: the survivors of pass 1 to their edges.  Bound by the 40 bytes that an
// edge is written in; a lane takes one component of a shift, so that stores are whole lines, and an edge
// inside the box needs neither a division nor its atoms' images.  Two passes that each walked the cells,
// and a read of flags behind them, took 760 us with the edge sort that follows them, this 440 (100 000
// atoms, 3 M edges).
constexpr int kFillWarps = 8;
__global__ void __launch_bounds__(32 * kFillWarps)
fill_kernel(int64_t N, const int4 *__restrict__ own, Grid g,
            const unsigned long long *__restrict__ kept, int stride,
            const int32_t *__restrict__ row_ptr,
            int64_t E, int64_t *__restrict__ edge_index, double *__restrict__ shifts,
            const int32_t *__restrict__ flags) {
  zp_after_previous();
  const int lane = threadIdx.x % 32;
  const int64_t j = (int64_t)blockIdx.x * kFillWarps + threadIdx.x / 32;
  if (j >= N) return;
  const int64_t base = row_ptr[j];
  const int n = (int)(row_ptr[j + 1] - base);
  kept += j * stride;
  if (n <= 0 || kept[0] == kCrowded) return;
  const Writer out{own, g, flags[kUnwrapped] != 0, E, j, base, edge_index, shifts};
  for (int t = lane; t < n; t += 32) out.put_pair(kept[t], t);
  for (int v = lane; v < 3 * n; v += 32) out.put_shift(kept[v / 3], v);
}

// The destinations listed in `crowded` (more than kFewHits hits).
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
fill_many_kernel(const int32_t *__restrict__ crowded, const int4 *__restrict__ own, Grid g,
                 const int32_t *__restrict__ cell_start, const Sorted atoms, int cap,
                 const int32_t *__restrict__ row_ptr, int64_t E, int64_t *__restrict__ edge_index,
                 double *__restrict__ shifts, int32_t *flags) {
  zp_after_previous();
  extern __shared__ unsigned char smem_raw[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  Hit *h = reinterpret_cast<Hit *>(smem_raw) + (size_t)warp * kHitCap;
  for (int c = blockIdx.x * kWarpsPerBlock + warp; c < crowded[0]; c += gridDim.x * kWarpsPerBlock) {
    const int64_t at = crowded[1 + c], j = atoms.who[at].w;
    const Hit inf{INFINITY, ~0ull};
    int n = 0;                      // hits held (warp-uniform)
    bool overflow = false;
    for_each_hit(g, g.all, cell_start, atoms, at, lane,
                 [&](bool hit, int i, unsigned code, double d2) {
                   const unsigned m = __ballot_sync(0xffffffffu, hit);
                   const int add = __popc(m);
                   if (n + add > kHitCap) {
                     if (cap > 0) {          // keep the best `cap` so far, drop the rest
                       const int n2 = pow2_at_least(n);
                       for (int t = n + lane; t < n2; t += 32) h[t] = inf;
                       __syncwarp();
                       warp_bitonic(h, n2, lane, hit_less);
                       n = n < cap ? n : cap;
                     } else {
                       overflow = true;
                     }
                   }
                   if (hit && !overflow) {
                     const int slot = n + __popc(m & ((1u << lane) - 1u));
                     h[slot].d2 = d2;
                     h[slot].tie = ((unsigned long long)(unsigned)i << 32) | code;
                   }
                   if (!overflow) n += add;
                   __syncwarp();
                   return !overflow;
                 });
    if (overflow) {
      if (lane == 0) atomicOr(flags, 2);
      continue;
    }
    if (cap > 0 && n > cap) {
      const int n2 = pow2_at_least(n);
      for (int t = n + lane; t < n2; t += 32) h[t] = inf;
      __syncwarp();
      warp_bitonic(h, n2, lane, hit_less);
      n = cap;
    }
    // survivors in (src, image) order
    {
      const int n2 = pow2_at_least(n);
      for (int t = n + lane; t < n2; t += 32) h[t] = inf;
      __syncwarp();
      warp_bitonic(h, n2, lane, [](const Hit &a, const Hit &b) { return a.tie < b.tie; });
    }
    const int64_t base = row_ptr[j];
    if (row_ptr[j + 1] - base != n) {          // not seen: both read the same copies; nothing is written past the row
      if (lane == 0) atomicOr(flags, 4);
      n = min(n, (int)(row_ptr[j + 1] - base));
    }
    const Writer out{own, g, flags[kUnwrapped] != 0, E, j, base, edge_index, shifts};
    for (int t = lane; t < n; t += 32) out.put_pair(h[t].tie, t);
    for (int v = lane; v < 3 * n; v += 32) out.put_shift(h[v / 3].tie, v);
    __syncwarp();
  }
}

struct NbWork {
  int32_t *flags, *cell_count, *cell_start, *cell_cursor, *atom_cell, *counts, *crowded,
      *block_sums;
  int4 *own;       // own image and index of each atom
  unsigned long long *kept;     // [N][kept_stride] survivors of pass 1
  Sorted atoms;
  size_t bytes;
};

// Radius that the `cap` nearest of an atom most probably lie within: a uniform gas has that many 3.5
// standard deviations below its mean there (one atom in 4 000 has not, and is walked again).  The cutoff, if that
// leaves less than a fifth of the sphere out.  100 000 atoms of 90 hits, cap 30: a sphere of 56.
double near_radius(int64_t N, double box, double cutoff, int cap) {
  if (cap <= 0) return cutoff;
  const double held = (double)N / (box * box * box) * (4.0 / 3.0 * 3.14159265358979) * cutoff * cutoff * cutoff;
  const double want = cap + 4.0 * std::sqrt((double)cap) + 4.0;
  return want < 0.8 * held ? cutoff * std::cbrt(want / held) : cutoff;
}

constexpr int kMaxCells = 256;           // per dimension

int make_grid(int64_t N, double box, double cutoff, int cap, Grid *g) {
  if (!(box > 0.0) || !(cutoff > 0.0) || !std::isfinite(box) || !std::isfinite(cutoff))
    return ZP_ERR_INVALID_ARG;
  // Cells a hair wider than the radius, so that a last-bit rounding of a cell coordinate can
  // never put a pair within it more than w cells apart.  Half-radius cells leave 2.4 times
  // as few candidates outside the sphere and still give a warp one column per lane (25); they
  // are taken when they are no more than the atoms, so that clearing and scanning them is cheap.
  constexpr double kHair = 1.0 + 1e-9;
  const double wide = cutoff * kHair;
  auto halves = [&](double radius) {
    const double cells = std::floor(box / (0.5 * radius * kHair));
    const bool fit = cells >= 1 && cells <= kMaxCells && cells * cells * cells <= (double)N;
    return fit ? (int)cells : 0;
  };
  double near = near_radius(N, box, cutoff, cap);
  int nc = halves(near);
  if (nc == 0 && near < cutoff) nc = halves(near = cutoff);
  if (nc == 0) {
    near = cutoff;
    const double cells = std::floor(box / wide);
    nc = cells < 1 ? 1 : cells > kMaxCells ? kMaxCells : (int)cells;
  }
  g->box = box;
  g->nc = nc;
  const double cell = box / nc;
  g->per_cell = nc / box;
  auto sphere = [&](double radius) {
    const int w = (int)std::ceil(radius * kHair / cell);
    return Grid::Sphere{radius * radius, (float)(1.0001 * (radius / cell) * (radius / cell)), w < 1 ? 1 : w};
  };
  g->all = sphere(cutoff);
  g->near = sphere(near);
  g->w = g->all.w;
  g->reach = (int)std::ceil(cutoff / box);
  if (g->reach < 1) g->reach = 1;
  if (g->reach > 8) return ZP_ERR_UNSUPPORTED;         // box far smaller than the cutoff
  return ZP_OK;
}

// edges per destination kept from pass 1 to pass 2
int kept_stride(int cap) { return cap > 0 && cap < kKept ? cap : kKept; }

// most: room for the grid of any cap
NbWork carve_nb(int64_t N, const Grid &g, int cap, void *base, bool most = false) {
  NbWork w;
  size_t off = 0;
  auto take = [&](size_t n) {
    int32_t *p = base ? reinterpret_cast<int32_t *>(static_cast<unsigned char *>(base) + off)
                      : nullptr;
    off += zp_align_up(n * sizeof(int32_t), 256);
    return p;
  };
  size_t cells = (size_t)g.nc * g.nc * g.nc;
  if (most) cells = std::max(cells, std::min<size_t>((size_t)N, (size_t)kMaxCells * kMaxCells * kMaxCells));
  w.flags = take((size_t)N + 4);
  w.crowded = w.flags + kCrowdedList;      // how many, then which
  w.cell_count = take(cells + 1);
  w.cell_cursor = take(cells + 1);
  w.cell_start = take(cells + 1);
  w.atom_cell = take((size_t)N);
  w.own = reinterpret_cast<int4 *>(take((size_t)4 * N));
  w.atoms.x = reinterpret_cast<double *>(take((size_t)2 * N));
  w.atoms.y = reinterpret_cast<double *>(take((size_t)2 * N));
  w.atoms.z = reinterpret_cast<double *>(take((size_t)2 * N));
  w.atoms.who = reinterpret_cast<int4 *>(take((size_t)4 * N));
  w.kept = reinterpret_cast<unsigned long long *>(take((size_t)2 * kept_stride(cap) * N));
  w.counts = take((size_t)N + 1);
  w.block_sums = take((size_t)zp_ceil_div((int64_t)std::max<size_t>(cells, (size_t)N) + 2, kScanBlock) + 1);
  w.bytes = off;
  return w;
}

}  // namespace

extern "C" {

size_t zp_neighbors_work_bytes(int64_t n_atoms, double box, double cutoff) {
  Grid g;
  if (n_atoms < 0 || make_grid(n_atoms, box, cutoff, 0, &g)) return 0;
  return carve_nb(n_atoms, g, 0, nullptr, true).bytes;
}

size_t zp_neighbors_work_bytes_capped(int64_t n_atoms, double box, double cutoff, int max_neighbors) {
  Grid g;
  if (n_atoms < 0 || make_grid(n_atoms, box, cutoff, max_neighbors, &g)) return 0;
  return carve_nb(n_atoms, g, max_neighbors, nullptr, true).bytes;      // a smaller cap may have finer cells
}

int zp_neighbors_count(const double *pos, int64_t N, double box, double cutoff, int max_neighbors,
                       int32_t *row_ptr, int32_t *flags_out, void *work, size_t work_bytes,
                       void *stream) {
  Grid g;
  int rc = make_grid(N, box, cutoff, max_neighbors, &g);
  if (rc) return rc;
  if (N < 0 || N > 2000000000ll || !row_ptr || !flags_out || !work || (N && !pos))
    return ZP_ERR_INVALID_ARG;
  if (max_neighbors > ZP_NEIGHBORS_MAX_CAP) return ZP_ERR_TOO_LARGE;
  const NbWork w = carve_nb(N, g, max_neighbors, work);
  if (work_bytes < w.bytes) return ZP_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t cells = (size_t)g.nc * g.nc * g.nc;
  ZP_CUDA(cudaMemsetAsync(w.flags, 0, 4 * sizeof(int32_t), st));
  ZP_CUDA(cudaMemsetAsync(w.cell_count, 0, (w.cell_start - w.cell_count) * sizeof(int32_t), st));
  if (N > 0) {
    zp_launch(cell_count_kernel, (unsigned)zp_ceil_div(N, 256), 256, 0, st, N, pos, g, w.atom_cell,
              w.own, w.cell_count, w.flags);
    ZP_LAUNCH_CHECK("cell_count_kernel");
  }
  if ((rc = exclusive_scan((int64_t)cells, w.cell_count, w.cell_start, w.block_sums, st))) return rc;
  if (N > 0) {
    zp_launch(cell_fill_kernel, (unsigned)zp_ceil_div(N, 256), 256, 0, st, N, pos, g, w.atom_cell,
              w.own, w.cell_start, w.cell_cursor, w.atoms);
    ZP_LAUNCH_CHECK("cell_fill_kernel");
    zp_launch(select_kernel, (unsigned)zp_ceil_div(N, kSelectWarps), 32 * kSelectWarps, 0, st, N, g,
              w.cell_start, w.atoms, max_neighbors, w.counts, w.kept, kept_stride(max_neighbors),
              w.flags, w.crowded);
    ZP_LAUNCH_CHECK("select_kernel");
  }
  if ((rc = exclusive_scan(N, w.counts, row_ptr, w.block_sums, st))) return rc;
  ZP_CUDA(cudaMemcpyAsync(flags_out, w.flags, sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
  return ZP_OK;
}

int zp_neighbors_fill(const double *pos, int64_t N, double box, double cutoff, int max_neighbors,
                      const int32_t *row_ptr, int64_t E, int64_t *edge_index, double *shifts,
                      int32_t *flags_out, void *work, size_t work_bytes, void *stream) {
  Grid g;
  int rc = make_grid(N, box, cutoff, max_neighbors, &g);
  if (rc) return rc;
  if (N < 0 || E < 0 || !row_ptr || !flags_out || !work || (N && !pos) ||
      (E && (!edge_index || !shifts)))
    return ZP_ERR_INVALID_ARG;
  if (max_neighbors > ZP_NEIGHBORS_MAX_CAP) return ZP_ERR_TOO_LARGE;
  const NbWork w = carve_nb(N, g, max_neighbors, work);
  if (work_bytes < w.bytes) return ZP_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  if (N > 0) {
    zp_launch(fill_kernel, (unsigned)zp_ceil_div(N, kFillWarps), 32 * kFillWarps, 0, st, N, w.own, g,
              w.kept, kept_stride(max_neighbors), row_ptr, E, edge_index, shifts, w.flags);
    ZP_LAUNCH_CHECK("fill_kernel");
    const size_t smem = sizeof(Hit) * kHitCap * kWarpsPerBlock;
    static ZpSmemOptIn opt_in;
    if (int rc_ = zp_ensure_smem(fill_many_kernel, smem, opt_in)) return rc_;
    const unsigned blocks = (unsigned)std::min<int64_t>(zp_ceil_div(N, kWarpsPerBlock), 148);
    zp_launch(fill_many_kernel, blocks, 32 * kWarpsPerBlock, smem, st, w.crowded, w.own, g,
              w.cell_start, w.atoms, max_neighbors, row_ptr, E, edge_index, shifts, w.flags);
    ZP_LAUNCH_CHECK("fill_many_kernel");
  }
  ZP_CUDA(cudaMemcpyAsync(flags_out, w.flags, sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
  return ZP_OK;
}

}  // extern "C"
