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
// Method: uniform cells of edge >= cutoff / w (w = 1 unless the box is smaller than the cutoff);
// one warp per destination walks the (2w+1)^3 cells around it in unwrapped cell coordinates; the
// unwrapped coordinate gives both the wrapped cell and the periodic image, so every
// (source, image) pair is visited exactly once.  The atoms are copied in cell order with their own
// image numbers, so the walk reads them with whole-line loads and divides nothing, and the cells
// of a walk are laid end to end so that no lane waits at a cell's end.  Pass 1 counts, a scan gives
// row_ptr, pass 2 collects the hits and, when the cap binds, selects the nearest: up to 128 hits
// in registers by bisecting the distance until it parts off exactly `cap` of them (ranking all
// when equal distances stand in the way), more by a bitonic sort on (d2, src, image) in shared
// memory.  The survivors are placed by counting the smaller (src, image) keys.
#include <algorithm>
#include <cmath>

#include "zp_common.cuh"
#include "zippel_b200.h"

namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kHitCap = ZP_NEIGHBORS_MAX_HITS;     // hits held per destination in shared memory
constexpr int kFewHits = 128;                      // ... in registers, four per lane
constexpr int kScanBlock = 1024;

struct Grid {
  double box, cell, cutoff2;
  int nc;          // cells per dimension
  int w;           // search half-width in cells
  int reach;       // largest |image| component that can occur
};

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
__device__ __forceinline__ int cell_coord(double p, const Grid &g) {
  const double pw = p - floor(p / g.box) * g.box;
  int c = (int)floor(pw / g.cell);
  return c < 0 ? 0 : (c >= g.nc ? g.nc - 1 : c);
}

__device__ __forceinline__ int floor_div(int a, int n) {
  int q = a / n;
  if ((a % n) < 0) --q;
  return q;
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
                                  int32_t *__restrict__ atom_cell, int32_t *cell_count,
                                  int32_t *flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
  const double far = 1.0e6 * g.box;
  if (!(fabs(x) < far && fabs(y) < far && fabs(z) < far))
    atomicOr(flags, 1);                               // not finite, or absurdly far from the box
  const int c = (cell_coord(x, g) * g.nc + cell_coord(y, g)) * g.nc + cell_coord(z, g);
  atom_cell[i] = c;
  atomicAdd(&cell_count[c], 1);
}

// atoms in cell order: coordinates and {own image, index}
struct Sorted {
  double *x, *y, *z;
  int4 *who;
};
__global__ void cell_fill_kernel(int64_t N, const double *__restrict__ pos, Grid g,
                                 const int32_t *__restrict__ atom_cell,
                                 const int32_t *__restrict__ cell_start, int32_t *cell_cursor,
                                 const Sorted out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int c = atom_cell[i];
  const int at = cell_start[c] + atomicAdd(&cell_cursor[c], 1);
  const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
  out.x[at] = x;
  out.y[at] = y;
  out.z[at] = z;
  out.who[at] = make_int4(own_image(x, g), own_image(y, g), own_image(z, g), (int)i);
}

// exclusive scan of n ints (n + 1 outputs, the last is the total): block scans, serial scan of
// the block totals, add back
__global__ void scan_block_kernel(int64_t n, const int32_t *__restrict__ in, int32_t *out,
                                  int32_t *block_sums) {
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
__global__ void scan_sums_kernel(int64_t nb, int32_t *block_sums) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    int32_t run = 0;
    for (int64_t b = 0; b < nb; ++b) {
      const int32_t v = block_sums[b];
      block_sums[b] = run;
      run += v;
    }
  }
}
__global__ void scan_add_kernel(int64_t n, int32_t *out, const int32_t *__restrict__ block_sums) {
  const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  if (i <= n) out[i] += block_sums[blockIdx.x];
}

int exclusive_scan(int64_t n, const int32_t *in, int32_t *out, int32_t *block_sums,
                   cudaStream_t st) {
  const int64_t nb = zp_ceil_div(n + 1, kScanBlock);
  scan_block_kernel<<<(unsigned)nb, kScanBlock, 0, st>>>(n, in, out, block_sums);
  ZP_LAUNCH_CHECK("scan_block_kernel");
  scan_sums_kernel<<<1, 32, 0, st>>>(nb, block_sums);
  ZP_LAUNCH_CHECK("scan_sums_kernel");
  scan_add_kernel<<<(unsigned)nb, kScanBlock, 0, st>>>(n, out, block_sums);
  ZP_LAUNCH_CHECK("scan_add_kernel");
  return ZP_OK;
}

// Calls f(hit, src, -kx, -ky, -kz, d2) on all 32 lanes together for every batch of candidate
// (source, image) pairs around destination j; `hit` marks the lanes whose candidate lies within
// the cutoff, k is its image in wrapped coordinates.
template <typename F>
__device__ __forceinline__ void for_each_hit(const Grid &g, const double *__restrict__ pos,
                                             const int32_t *__restrict__ cell_start,
                                             const Sorted &atoms, int64_t j, int lane, F &&f) {
  const double xj = pos[3 * j], yj = pos[3 * j + 1], zj = pos[3 * j + 2];
  const int cx = cell_coord(xj, g), cy = cell_coord(yj, g), cz = cell_coord(zj, g);
  const int ojx = own_image(xj, g), ojy = own_image(yj, g), ojz = own_image(zj, g);
  const int side = 2 * g.w + 1, cells = side * side * side;
  for (int q0 = 0; q0 < cells; q0 += 32) {
    // a lane per cell: where its atoms stand, and its image
    const int q = q0 + lane;
    int off = 0, len = 0, image = 0;
    if (q < cells) {
      const int ux = cx - g.w + q / (side * side), uy = cy - g.w + q / side % side, uz = cz - g.w + q % side;
      const int kx = floor_div(ux, g.nc), ky = floor_div(uy, g.nc), kz = floor_div(uz, g.nc);
      const int c = ((ux - kx * g.nc) * g.nc + (uy - ky * g.nc)) * g.nc + (uz - kz * g.nc);
      off = cell_start[c];
      len = cell_start[c + 1] - off;
      image = (kx + 512) | (ky + 512) << 10 | (kz + 512) << 20;
    }
    int upto = len;                              // candidates of the cells up to this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += u;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31);
    off -= upto - len;
    for (int t0 = 0; t0 < total; t0 += 32) {
      const int t = t0 + lane;
      int cell = 0;                              // the cell candidate t belongs to
#pragma unroll
      for (int b = 16; b > 0; b >>= 1) {
        const int v = __shfl_sync(0xffffffffu, upto, cell + b - 1);
        if (v <= t) cell += b;
      }
      const int a = __shfl_sync(0xffffffffu, off, cell) + t;
      const int im = __shfl_sync(0xffffffffu, image, cell);
      bool hit = false;
      int i = 0, nkx = 0, nky = 0, nkz = 0;
      double d2 = 0.0;
      if (t < total) {
        const int4 who = atoms.who[a];
        i = who.w;
        nkx = 512 - (im & 1023);
        nky = 512 - (im >> 10 & 1023);
        nkz = 512 - (im >> 20 & 1023);
        // the source's wrapped copy sits k boxes away in wrapped coordinates:
        // pos[j] - (pos[i] - o_i box + k box) stays as (pos[j] - pos[i]) + (o_i - o_j - k) box
        // once the destination's own offset o_j is taken out of the search origin
        const int mx = who.x - ojx + nkx, my = who.y - ojy + nky, mz = who.z - ojz + nkz;
        const double dx = __dadd_rn(__dsub_rn(xj, atoms.x[a]), __dmul_rn((double)mx, g.box));
        const double dy = __dadd_rn(__dsub_rn(yj, atoms.y[a]), __dmul_rn((double)my, g.box));
        const double dz = __dadd_rn(__dsub_rn(zj, atoms.z[a]), __dmul_rn((double)mz, g.box));
        d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        hit = d2 < g.cutoff2 && !(i == j && mx == 0 && my == 0 && mz == 0);
      }
      f(hit, i, nkx, nky, nkz, d2);
    }
  }
}

__global__ void __launch_bounds__(32 * kWarpsPerBlock)
count_kernel(int64_t N, const double *__restrict__ pos, Grid g,
             const int32_t *__restrict__ cell_start, const Sorted atoms, int cap,
             int32_t *__restrict__ counts, int32_t *flags, int32_t *__restrict__ crowded) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int64_t at = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  if (at >= N) return;
  const int64_t j = atoms.who[at].w;           // in cell order: neighbours read the same cells
  int n = 0;
  for_each_hit(g, pos, cell_start, atoms, j, lane,
               [&](bool hit, int, int, int, int, double) {
                 n += __popc(__ballot_sync(0xffffffffu, hit));
               });
  if (lane == 0) {
    if (cap <= 0 && n > kHitCap) atomicOr(flags, 2);       // uncapped list too long for pass 2
    counts[j] = cap > 0 && n > cap ? cap : n;
    if (n > kFewHits) crowded[1 + atomicAdd(&crowded[0], 1)] = (int32_t)j;
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

// Writes the edges of destination j: survivor `tie` at place `rank` of its list.
struct Writer {
  const double *pos;
  const Grid &g;
  int64_t E, j, base;
  int64_t *edge_index;
  double *shifts;
  int ojx, ojy, ojz;
  __device__ Writer(const double *p, const Grid &grid, int64_t n_edges, int64_t dst, int64_t first,
                    int64_t *edges, double *sh)
      : pos(p), g(grid), E(n_edges), j(dst), base(first), edge_index(edges), shifts(sh),
        ojx(own_image(p[3 * dst], grid)), ojy(own_image(p[3 * dst + 1], grid)),
        ojz(own_image(p[3 * dst + 2], grid)) {}
  __device__ __forceinline__ void put(unsigned long long tie, int rank) const {
    const unsigned s = 2u * g.reach + 1u;
    const unsigned code = (unsigned)(tie & 0xffffffffu);
    const int64_t i = (int64_t)(tie >> 32);
    const int nkz = (int)(code % s) - g.reach, nky = (int)((code / s) % s) - g.reach,
              nkx = (int)(code / (s * s)) - g.reach;
    edge_index[base + rank] = i;
    edge_index[E + base + rank] = j;
    shifts[3 * (base + rank)] = (double)(own_image(pos[3 * i], g) - ojx + nkx) * g.box;
    shifts[3 * (base + rank) + 1] = (double)(own_image(pos[3 * i + 1], g) - ojy + nky) * g.box;
    shifts[3 * (base + rank) + 2] = (double)(own_image(pos[3 * i + 2], g) - ojz + nkz) * g.box;
  }
};

// Destinations with at most kFewHits hits.  The hits are compacted through 2 KB of shared memory per
// warp and then live in registers, four per lane.
constexpr int kFillWarps = 8;
__global__ void __launch_bounds__(32 * kFillWarps)
fill_few_kernel(int64_t N, const double *__restrict__ pos, Grid g,
                const int32_t *__restrict__ cell_start, const Sorted atoms, int cap,
                const int32_t *__restrict__ row_ptr, int64_t E, int64_t *__restrict__ edge_index,
                double *__restrict__ shifts, int32_t *flags) {
  __shared__ Hit hits[kFillWarps][kFewHits];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int64_t at = (int64_t)blockIdx.x * kFillWarps + warp;
  if (at >= N) return;
  const int64_t j = atoms.who[at].w;
  Hit *h = hits[warp];
  int n = 0;                      // hits seen (warp-uniform)
  for_each_hit(g, pos, cell_start, atoms, j, lane,
               [&](bool hit, int i, int nkx, int nky, int nkz, double d2) {
                 const unsigned m = __ballot_sync(0xffffffffu, hit);
                 const int slot = n + __popc(m & ((1u << lane) - 1u));
                 if (hit && slot < kFewHits) {
                   h[slot].d2 = d2;
                   h[slot].tie = ((unsigned long long)(unsigned)i << 32) | image_code(nkx, nky, nkz, g.reach);
                 }
                 n += __popc(m);
               });
  if (n > kFewHits) return;       // left to fill_many_kernel
  __syncwarp();
  constexpr int R = kFewHits / 32;
  double d2[R];
  unsigned long long tie[R];
  unsigned alive = 0;             // which of this lane's hits survive
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int t = lane + 32 * k;
    d2[k] = t < n ? h[t].d2 : INFINITY;
    tie[k] = t < n ? h[t].tie : ~0ull;
    if (t < n) alive |= 1u << k;
  }
  if (cap > 0 && n > cap) {
    // bisect the distance; every step counts the hits up to the middle
    double lo = 0.0, hi = g.cutoff2;
    bool found = false;
    for (int step = 0; step < 40 && !found; ++step) {
      const double mid = 0.5 * (lo + hi);
      int below = 0;
#pragma unroll
      for (int k = 0; k < R; ++k) below += __popc(__ballot_sync(0xffffffffu, d2[k] <= mid));
      if (below == cap) {
        found = true;
#pragma unroll
        for (int k = 0; k < R; ++k)
          if (!(d2[k] <= mid)) alive &= ~(1u << k);
      } else if (below < cap) {
        lo = mid;
      } else {
        hi = mid;
      }
    }
    if (!found) {                 // equal distances at the cap: rank by (d2, src, image)
      int rank[R];
#pragma unroll
      for (int k = 0; k < R; ++k) rank[k] = 0;
      for (int t = 0; t < n; ++t) {
        const Hit o = h[t];
#pragma unroll
        for (int k = 0; k < R; ++k) rank[k] += o.d2 < d2[k] || (o.d2 == d2[k] && o.tie < tie[k]);
      }
#pragma unroll
      for (int k = 0; k < R; ++k)
        if (rank[k] >= cap) alive &= ~(1u << k);
    }
    n = cap;
  }
  // place of a survivor = number of survivors with a smaller (src, image)
  int rank[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    rank[k] = 0;
    if (!(alive >> k & 1)) tie[k] = ~0ull;
  }
#pragma unroll
  for (int k = 0; k < R; ++k) {
    for (unsigned m = __ballot_sync(0xffffffffu, alive >> k & 1); m; m &= m - 1) {
      const unsigned long long o = __shfl_sync(0xffffffffu, tie[k], __ffs(m) - 1);
#pragma unroll
      for (int q = 0; q < R; ++q) rank[q] += o < tie[q];
    }
  }
  const int64_t base = row_ptr[j];
  if (lane == 0 && row_ptr[j + 1] - base != n) atomicOr(flags, 4);     // passes disagree
  const Writer out(pos, g, E, j, base, edge_index, shifts);
#pragma unroll
  for (int k = 0; k < R; ++k)
    if (alive >> k & 1) out.put(tie[k], rank[k]);
}

// The destinations listed in `crowded` (more than kFewHits hits).
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
fill_many_kernel(const int32_t *__restrict__ crowded, const double *__restrict__ pos, Grid g,
                 const int32_t *__restrict__ cell_start, const Sorted atoms, int cap,
                 const int32_t *__restrict__ row_ptr, int64_t E, int64_t *__restrict__ edge_index,
                 double *__restrict__ shifts, int32_t *flags) {
  extern __shared__ unsigned char smem_raw[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  Hit *h = reinterpret_cast<Hit *>(smem_raw) + (size_t)warp * kHitCap;
  for (int c = blockIdx.x * kWarpsPerBlock + warp; c < crowded[0]; c += gridDim.x * kWarpsPerBlock) {
    const int64_t j = crowded[1 + c];
    const Hit inf{INFINITY, ~0ull};
    int n = 0;                      // hits held (warp-uniform)
    bool overflow = false;
    for_each_hit(g, pos, cell_start, atoms, j, lane,
                 [&](bool hit, int i, int nkx, int nky, int nkz, double d2) {
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
                     h[slot].tie = ((unsigned long long)(unsigned)i << 32) |
                                   image_code(nkx, nky, nkz, g.reach);
                   }
                   if (!overflow) n += add;
                   __syncwarp();
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
    if (lane == 0 && row_ptr[j + 1] - base != n) atomicOr(flags, 4);     // passes disagree
    const Writer out(pos, g, E, j, base, edge_index, shifts);
    for (int t = lane; t < n; t += 32) out.put(h[t].tie, t);
    __syncwarp();
  }
}

struct NbWork {
  int32_t *flags, *cell_count, *cell_start, *cell_cursor, *atom_cell, *counts, *crowded,
      *block_sums;
  Sorted atoms;
  size_t bytes;
};

int make_grid(double box, double cutoff, Grid *g) {
  if (!(box > 0.0) || !(cutoff > 0.0) || !std::isfinite(box) || !std::isfinite(cutoff))
    return ZP_ERR_INVALID_ARG;
  // cells a hair wider than the cutoff, so that a last-bit rounding of a cell coordinate can
  // never put a pair within the cutoff more than w cells apart
  int nc = (int)std::floor(box / (cutoff * (1.0 + 1e-9)));
  if (nc < 1) nc = 1;
  if (nc > 256) nc = 256;
  g->box = box;
  g->nc = nc;
  g->cell = box / nc;
  g->cutoff2 = cutoff * cutoff;
  g->w = (int)std::ceil(cutoff * (1.0 + 1e-9) / g->cell);
  if (g->w < 1) g->w = 1;
  g->reach = (int)std::ceil(cutoff / box);
  if (g->reach < 1) g->reach = 1;
  if (g->reach > 8) return ZP_ERR_UNSUPPORTED;         // box far smaller than the cutoff
  return ZP_OK;
}

NbWork carve_nb(int64_t N, const Grid &g, void *base) {
  NbWork w;
  size_t off = 0;
  auto take = [&](size_t n) {
    int32_t *p = base ? reinterpret_cast<int32_t *>(static_cast<unsigned char *>(base) + off)
                      : nullptr;
    off += zp_align_up(n * sizeof(int32_t), 256);
    return p;
  };
  const size_t cells = (size_t)g.nc * g.nc * g.nc;
  w.flags = take((size_t)N + 4);
  w.crowded = w.flags + 3;                 // how many, then which: cleared with the flags
  w.cell_count = take(cells + 1);
  w.cell_cursor = take(cells + 1);
  w.cell_start = take(cells + 1);
  w.atom_cell = take((size_t)N);
  w.atoms.x = reinterpret_cast<double *>(take((size_t)2 * N));
  w.atoms.y = reinterpret_cast<double *>(take((size_t)2 * N));
  w.atoms.z = reinterpret_cast<double *>(take((size_t)2 * N));
  w.atoms.who = reinterpret_cast<int4 *>(take((size_t)4 * N));
  w.counts = take((size_t)N + 1);
  w.block_sums = take((size_t)zp_ceil_div((int64_t)std::max<size_t>(cells, (size_t)N) + 2, kScanBlock) + 1);
  w.bytes = off;
  return w;
}

}  // namespace

extern "C" {

size_t zp_neighbors_work_bytes(int64_t n_atoms, double box, double cutoff) {
  Grid g;
  if (n_atoms < 0 || make_grid(box, cutoff, &g)) return 0;
  return carve_nb(n_atoms, g, nullptr).bytes;
}

int zp_neighbors_count(const double *pos, int64_t N, double box, double cutoff, int max_neighbors,
                       int32_t *row_ptr, int32_t *flags_out, void *work, size_t work_bytes,
                       void *stream) {
  Grid g;
  int rc = make_grid(box, cutoff, &g);
  if (rc) return rc;
  if (N < 0 || N > 2000000000ll || !row_ptr || !flags_out || !work || (N && !pos))
    return ZP_ERR_INVALID_ARG;
  if (max_neighbors > ZP_NEIGHBORS_MAX_CAP) return ZP_ERR_TOO_LARGE;
  const NbWork w = carve_nb(N, g, work);
  if (work_bytes < w.bytes) return ZP_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t cells = (size_t)g.nc * g.nc * g.nc;
  ZP_CUDA(cudaMemsetAsync(w.flags, 0, 4 * sizeof(int32_t), st));
  ZP_CUDA(cudaMemsetAsync(w.cell_count, 0, (w.cell_start - w.cell_count) * sizeof(int32_t), st));
  if (N > 0) {
    cell_count_kernel<<<(unsigned)zp_ceil_div(N, 256), 256, 0, st>>>(N, pos, g, w.atom_cell,
                                                                     w.cell_count, w.flags);
    ZP_LAUNCH_CHECK("cell_count_kernel");
  }
  if ((rc = exclusive_scan((int64_t)cells, w.cell_count, w.cell_start, w.block_sums, st))) return rc;
  if (N > 0) {
    cell_fill_kernel<<<(unsigned)zp_ceil_div(N, 256), 256, 0, st>>>(N, pos, g, w.atom_cell,
                                                                    w.cell_start, w.cell_cursor, w.atoms);
    ZP_LAUNCH_CHECK("cell_fill_kernel");
    count_kernel<<<(unsigned)zp_ceil_div(N, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, st>>>(
        N, pos, g, w.cell_start, w.atoms, max_neighbors, w.counts, w.flags, w.crowded);
    ZP_LAUNCH_CHECK("count_kernel");
  }
  if ((rc = exclusive_scan(N, w.counts, row_ptr, w.block_sums, st))) return rc;
  ZP_CUDA(cudaMemcpyAsync(flags_out, w.flags, sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
  return ZP_OK;
}

int zp_neighbors_fill(const double *pos, int64_t N, double box, double cutoff, int max_neighbors,
                      const int32_t *row_ptr, int64_t E, int64_t *edge_index, double *shifts,
                      int32_t *flags_out, void *work, size_t work_bytes, void *stream) {
  Grid g;
  int rc = make_grid(box, cutoff, &g);
  if (rc) return rc;
  if (N < 0 || E < 0 || !row_ptr || !flags_out || !work || (N && !pos) ||
      (E && (!edge_index || !shifts)))
    return ZP_ERR_INVALID_ARG;
  if (max_neighbors > ZP_NEIGHBORS_MAX_CAP) return ZP_ERR_TOO_LARGE;
  const NbWork w = carve_nb(N, g, work);
  if (work_bytes < w.bytes) return ZP_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  if (N > 0) {
    fill_few_kernel<<<(unsigned)zp_ceil_div(N, kFillWarps), 32 * kFillWarps, 0, st>>>(
        N, pos, g, w.cell_start, w.atoms, max_neighbors, row_ptr, E, edge_index, shifts, w.flags);
    ZP_LAUNCH_CHECK("fill_few_kernel");
    const size_t smem = sizeof(Hit) * kHitCap * kWarpsPerBlock;
    static ZpSmemOptIn opt_in;
    if (int rc_ = zp_ensure_smem(fill_many_kernel, smem, opt_in)) return rc_;
    const unsigned blocks = (unsigned)std::min<int64_t>(zp_ceil_div(N, kWarpsPerBlock), 148 * 3);
    fill_many_kernel<<<blocks, 32 * kWarpsPerBlock, smem, st>>>(w.crowded, pos, g, w.cell_start, w.atoms,
                                                                max_neighbors, row_ptr, E, edge_index,
                                                                shifts, w.flags);
    ZP_LAUNCH_CHECK("fill_many_kernel");
  }
  ZP_CUDA(cudaMemcpyAsync(flags_out, w.flags, sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
  return ZP_OK;
}

}  // extern "C"
