// Shared pieces of the rotate kernels, by edge and by node: packed arithmetic, staging, plane stores, and how a
// kernel by node deals a graph's edges out.
#pragma once

#include <algorithm>

#include "zp_common.cuh"
#include "zp_planes.cuh"

// Four channels as two packed fp32 pairs.  One packed multiply-add does two channels, so a kernel
// spends half as many issue slots on its sums; each half rounds as fmaf does.
using u64 = unsigned long long;
struct __align__(16) F4 {
  u64 a, b;
};
__device__ __forceinline__ u64 fma2(u64 x, u64 y, u64 z) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(x), "l"(y), "l"(z));
  return d;
}
__device__ __forceinline__ u64 mul2(u64 x, u64 y) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return d;
}
__device__ __forceinline__ u64 sub2(u64 x, u64 y) {
  u64 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return d;
}
__device__ __forceinline__ u64 pack2(float lo, float hi) {
  u64 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 unpack2(u64 x) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(x));
  return v;
}
__device__ __forceinline__ float sum2(u64 v) {
  const float2 f = unpack2(v);
  return f.x + f.y;
}
__device__ __forceinline__ F4 load4(const float *p) { return *reinterpret_cast<const F4 *>(p); }
__device__ __forceinline__ F4 zero4() { return F4{0ull, 0ull}; }
__device__ __forceinline__ void store4(float *p, const F4 &v) { *reinterpret_cast<F4 *>(p) = v; }
// acc += w v with a duplicated weight
__device__ __forceinline__ void axpy4(F4 &acc, u64 w, const F4 &v) {
  acc.a = fma2(w, v.a, acc.a);
  acc.b = fma2(w, v.b, acc.b);
}
__device__ __forceinline__ F4 mul4(const F4 &x, const F4 &y) { return F4{mul2(x.a, y.a), mul2(x.b, y.b)}; }
// acc += x . y, two partial sums side by side
__device__ __forceinline__ u64 dot4(u64 acc, const F4 &x, const F4 &y) {
  return fma2(x.a, y.a, fma2(x.b, y.b, acc));
}
// Two channels, for the degrees whose rows would not fit the registers four at a time
struct __align__(8) F2 {
  u64 a;
};
template <typename V> struct VecOf;
template <> struct VecOf<F4> { static constexpr int n = 4; };
template <> struct VecOf<F2> { static constexpr int n = 2; };
template <typename V>
__device__ __forceinline__ V load_vec(const float *p) { return *reinterpret_cast<const V *>(p); }
template <typename V>
__device__ __forceinline__ void store_vec(float *p, const V &v) { *reinterpret_cast<V *>(p) = v; }
template <typename V>
__device__ __forceinline__ V zero_vec() { return V{}; }
__device__ __forceinline__ u64 add2(u64 x, u64 y) {
  u64 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return d;
}
__device__ __forceinline__ F4 add4(const F4 &x, const F4 &y) { return F4{add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ F2 add4(const F2 &x, const F2 &y) { return F2{add2(x.a, y.a)}; }
__device__ __forceinline__ void axpy4(F2 &acc, u64 w, const F2 &v) { acc.a = fma2(w, v.a, acc.a); }
__device__ __forceinline__ F2 mul4(const F2 &x, const F2 &y) { return F2{mul2(x.a, y.a)}; }
__device__ __forceinline__ u64 dot4(u64 acc, const F2 &x, const F2 &y) { return fma2(x.a, y.a, acc); }
// x y + z w
__device__ __forceinline__ F4 mul_add4(const F4 &x, const F4 &y, const F4 &z, const F4 &w) {
  return F4{fma2(x.a, y.a, mul2(z.a, w.a)), fma2(x.b, y.b, mul2(z.b, w.b))};
}
__device__ __forceinline__ F2 mul_add4(const F2 &x, const F2 &y, const F2 &z, const F2 &w) {
  return F2{fma2(x.a, y.a, mul2(z.a, w.a))};
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Operand formats the kernels are instantiated for: fp32 rows, one or three bf16 terms, two scaled
// fp16 terms (the branches of a run-time format were a tenth of these kernels' instructions).
enum { kFmtFp32 = 0, kFmtBf16 = 1, kFmtFp16x2 = 2, kFmtBf16x3 = 3 };
inline int zp_plane_format(const ZpPlanes &p) { return p.planes; }      // planes 1, 2, 3 as above

// One quad into every plane (or, kFmtFp32, the fp32 row); `at`: the quad in plane 0; inv: duplicated
// inverse scale (fp16 only)
template <int FMT>
__device__ __forceinline__ void put4(void *at, int64_t plane_bytes, const F4 &v, u64 inv) {
  char *dst = static_cast<char *>(at);
  if constexpr (FMT == kFmtFp32) {
    *reinterpret_cast<F4 *>(dst) = v;
  } else if constexpr (FMT == kFmtFp16x2) {
    const u64 xa = mul2(v.a, inv), xb = mul2(v.b, inv);
    const float2 lo = unpack2(xa), hi = unpack2(xb);
    const __half2 h0 = __floats2half2_rn(lo.x, lo.y), h1 = __floats2half2_rn(hi.x, hi.y);
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    const float2 r0 = unpack2(sub2(xa, pack2(f0.x, f0.y))), r1 = unpack2(sub2(xb, pack2(f1.x, f1.y)));
    const __half2 g0 = __floats2half2_rn(r0.x, r0.y), g1 = __floats2half2_rn(r1.x, r1.y);
    *reinterpret_cast<uint2 *>(dst) =
        make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1));
    *reinterpret_cast<uint2 *>(dst + plane_bytes) =
        make_uint2(*reinterpret_cast<const uint32_t *>(&g0), *reinterpret_cast<const uint32_t *>(&g1));
  } else {
    u64 xa = v.a, xb = v.b;
#pragma unroll
    for (int pl = 0; pl < (FMT == kFmtBf16 ? 1 : 3); ++pl) {
      const float2 lo = unpack2(xa), hi = unpack2(xb);
      const __nv_bfloat162 h0 = __floats2bfloat162_rn(lo.x, lo.y), h1 = __floats2bfloat162_rn(hi.x, hi.y);
      *reinterpret_cast<uint2 *>(dst + pl * plane_bytes) =
          make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1));
      const float2 f0 = __bfloat1622float2(h0), f1 = __bfloat1622float2(h1);
      xa = sub2(xa, pack2(f0.x, f0.y));
      xb = sub2(xb, pack2(f1.x, f1.y));
    }
  }
}

// ... and one pair
template <int FMT>
__device__ __forceinline__ void put4(void *at, int64_t plane_bytes, const F2 &v, u64 inv) {
  char *dst = static_cast<char *>(at);
  if constexpr (FMT == kFmtFp32) {
    *reinterpret_cast<F2 *>(dst) = v;
  } else if constexpr (FMT == kFmtFp16x2) {
    const u64 x = mul2(v.a, inv);
    const float2 f = unpack2(x);
    const __half2 h = __floats2half2_rn(f.x, f.y);
    const float2 b = __half22float2(h), r = unpack2(sub2(x, pack2(b.x, b.y)));
    *reinterpret_cast<__half2 *>(dst) = h;
    *reinterpret_cast<__half2 *>(dst + plane_bytes) = __floats2half2_rn(r.x, r.y);
  } else {
    u64 x = v.a;
#pragma unroll
    for (int pl = 0; pl < (FMT == kFmtBf16 ? 1 : 3); ++pl) {
      const float2 f = unpack2(x);
      const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
      *reinterpret_cast<__nv_bfloat162 *>(dst + pl * plane_bytes) = h;
      const float2 b = __bfloat1622float2(h);
      x = sub2(x, pack2(b.x, b.y));
    }
  }
}

template <int BYTES>
__device__ __forceinline__ void cp_async(float *smem_dst, const float *gmem_src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The rows of one edge put in flight together, degree by degree (one commit group each), every
// thread fetching its own four channels: a kernel that loads its rows as it comes to them waits for
// HBM once per row, one step of prefetch or not.  In shared memory the rows stand in degree order
// (m = 0, +1, -1, ..), `ls` floats apart; in global memory m'-major, `stride` floats apart.
//   ROWS  rows |m| <= mmax of a degree     RAD  its radial gains |m| <= mmax, 2C floats apart
template <int L, int LMAX, bool ROWS, bool RAD>
struct StageEdge {
  static __device__ __forceinline__ void run(const ZpTables &t, const float *rows, int stride,
                                             float *row_s, const float *rad, float *rad_s, int ls) {
    StageEdge<L - 1, LMAX, ROWS, RAD>::run(t, rows, stride, row_s, rad, rad_s, ls);
    const int mm = t.mmax < L ? t.mmax : L;
    float *rs = row_s + (ROWS ? t.deg_row[L] * ls : 0), *gs = rad_s + (RAD ? t.deg_rad[L] * ls : 0);
    int r = L, k = L;                            // row m = 0, gain |m| = 0 of this degree
    if (ROWS) cp_async<16>(rs, rows + r * stride);
    if (RAD) cp_async<16>(gs, rad + k * 2 * t.C);
#pragma unroll 1
    for (int am = 1; am <= mm; ++am) {
      const int km = LMAX + 1 - am;              // rows of +am
      r += (am == 1 ? 1 : 2) * (km + 1) - 1;
      k += km;                                   // (km + 1) - 1
      if (ROWS) {
        rs += 2 * ls;
        cp_async<16>(rs - ls, rows + r * stride);
        cp_async<16>(rs, rows + (r + km) * stride);
      }
      if (RAD) {
        gs += ls;
        cp_async<16>(gs, rad + k * 2 * t.C);
      }
    }
    cp_async_commit();
  }
};
template <int LMAX, bool ROWS, bool RAD>
struct StageEdge<-1, LMAX, ROWS, RAD> {
  static __device__ __forceinline__ void run(const ZpTables &, const float *, int, float *,
                                             const float *, float *, int) {}
};

// n rotation entries of one row, duplicated in shared memory (row start 16-byte aligned): entry j
// of a pair of channels costs half a 16-byte load.  f(j, weight pair)
template <int N, typename F>
__device__ __forceinline__ void for_row(const float2 *row, F f) {
#pragma unroll
  for (int j = 0; j < N; j += 2) {
    const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(row + j);
    f(j, w.x);
    if (j + 1 < N) f(j + 1, w.y);
  }
}
// ... of a row as it stands in global memory (row start 8-byte aligned)
template <int N, typename F>
__device__ __forceinline__ void for_row_plain(const float *row, F f) {
#pragma unroll
  for (int j = 0; j < N; j += 2) {
    const float2 w = *reinterpret_cast<const float2 *>(row + j);
    f(j, pack2(w.x, w.x));
    if (j + 1 < N) f(j + 1, pack2(w.y, w.y));
  }
}
// rotation entries of `edges` consecutive edges duplicated into shared memory
__device__ __forceinline__ void stage_dup(const float *__restrict__ rot, float2 *rot_s, int ld, int edges) {
  for (int i = threadIdx.x; i < ld * edges; i += blockDim.x) {
    const float v = rot[i];
    rot_s[i] = make_float2(v, v);
  }
}

// ---- kernels by node ---------------------------------------------------------------------------
// A block owns one node, whose rows of x (or of the upstream gradient) stand in shared memory, and goes through
// the node's edges: by edge, a thread fetches them from L2 again and again, and those fetches were between a
// third and a half of all that L2 has to deliver, which is what bounds these kernels (60 000 edges at lmax 4 / C 128:
// 57 KB an edge in 389 us going in, 95 KB in 810 coming back, 8.9 and 7.0 TB/s).  G lanes are a worker, which has
// an edge to itself, each lane one vector of channels; the node's edges are dealt to the workers in turn.
// A degree's rows of the worker's next edge are requested as soon as those of the current one have been used,
// so that one edge is always on its way.  All copies into a worker's rows are its lanes' own, but the rotation's.
struct NodeShape {
  int vec, groups, quads, G;             // channels a lane; blocks per node; lanes with channels, lanes of a worker
};
inline NodeShape zp_node_shape(int channels, int vec) {
  NodeShape s;
  s.vec = vec;
  const int lanes = channels / vec;
  s.groups = (lanes + 31) / 32;
  s.quads = (lanes + s.groups - 1) / s.groups;
  s.G = s.quads <= 4 ? 4 : s.quads <= 8 ? 8 : s.quads <= 16 ? 16 : 32;
  return s;
}
// How a kernel by node is launched: a block for each of `parts` stretches of a node's edges.  What decides is how
// often the SMs have to take a new set of blocks, times how long a block takes: its edges, and the start (row
// offsets, first rotation, first rows, one after the other, as long as some three edges).  From 12 edges a node on four
// warps and eight, whole nodes and halves are within 5 % of each other and two warps up to 10 % behind; 216 nodes of 90
// edges took 739 us a training step with eight warps, 799 with four and 952 with two.  Nodes of few edges leave wide
// blocks idle: the VJP of rotate_in over 60 000 edges (lmax 4, C 128) of nodes that have 1, 2, 4 and 8 each way took
// 2.95, 1.72, 1.12 and 0.79 ms with four warps and the node's rows loaded before the first edge's were asked for; 0.90,
// 0.74, 0.66 and 0.63 with one or two and all of them asked for at once (edge by edge 1.79, 1.38, 1.23 and 1.18).  One
// or two are taken only where they promise a fifth: they lose that where a few nodes have most of the edges.
constexpr int kNodeMaxWarps = 8;
struct NodeLaunch {
  int warps, parts;
  size_t smem;
};
// blocks: nodes times channel groups; items: edges of a node on average; rows: vectors a lane holds of an edge;
// sm_warps: warps of the kernel that an SM's registers hold; max_parts: 1 where a node's edges belong together
inline NodeLaunch zp_node_launch(int64_t blocks, double items, const NodeShape &s, const ZpTables &t, int rows,
                                 int sm_warps, int max_parts) {
  NodeLaunch best{1, 1, 0}, few{1, 1, 0};
  double best_cost = 1e300, few_cost = 1e300;
  for (int warps = 1; warps <= kNodeMaxWarps; warps *= 2) {
    const size_t workers = 32 * warps / s.G;
    const size_t smem = sizeof(float) * ((size_t)s.G * s.vec * (t.K + workers * rows) + workers * 2 * t.rot_ld);
    if (warps > 1 && smem > 220 * 1024) break;
    if (warps == 4) {
      few = best;
      few_cost = best_cost;
      best_cost = 1e300;
    }
    const int64_t resident = 148 * std::max<int64_t>(1, std::min<int64_t>(sm_warps / warps, (int64_t)(225 * 1024 / (smem + 1024))));
    for (int parts = 1; parts <= max_parts; parts *= 2) {
      const double rounds = std::max(1.0, (double)(blocks * parts) / (double)resident + 0.5);
      const double cost = rounds * (items / (double)(parts * workers) + 3.0);
      if (cost < 0.98 * best_cost) {
        best_cost = cost;
        best = NodeLaunch{warps, parts, smem};
      }
    }
  }
  return few_cost < 0.8 * best_cost ? few : best;
}

// The node's edges, numbered: those into it, then (with a source view) those out of it.  Block N of a launch
// has the slots that the sort has left out (edges of indices out of range): they stand behind all others and read
// as edges 0 -> 0, but are edges into no node.
//
// A node of very many edges is cut: all nodes' edges stand in one row, and it has a cut wherever that row reaches a
// multiple of `step`.  The blocks of node n have what comes before the first cut, block k behind all nodes' what
// follows cut k; those whose cut falls into no such node, in most graphs all of them, end where they begin.  A
// step is half of an SM's share of the edges, so that a node by itself keeps its blocks busy as long as the others
// take at most, and a node is left whole whose blocks (two at least) have no more than that each.  Nodes of up to
// four times the mean are whole, or graphs of even nodes would be cut (those of up to 74 nodes are: one and two of 90
// edges took 10 and 7 % longer a training step than edge by edge).  Lines of eight times the mean cost 200 nodes
// of 30 edges and one of 600 more 11 % of a force evaluation, and gain nothing elsewhere.  2 000 nodes of 30 edges
// and one of 20 000 more, lmax 4 / C 128: a training step of 22.4 ms edge by edge took 52.5 with every node one
// block's, and takes 21.6; inference 12.1, 20.7 and 12.2.
struct NodeCut {
  int nodes, parts;                      // N; blocks of a node
  uint32_t step, cuts, whole;            // whole: edges of a node that is not cut, at most
  __host__ __device__ __forceinline__ int ends() const { return (nodes + 1) * parts; }    // blocks before the cuts'
  unsigned blocks() const { return (unsigned)ends() + cuts; }
};
inline NodeCut zp_node_cut(int64_t N, int64_t E, bool both, int parts) {
  const int64_t total = both ? 2 * E : E, pieces = std::max(parts, 2);
  int64_t step = std::max<int64_t>(zp_ceil_div(total, kZpNodeCuts), 64);
  if (N > kZpNodeCuts / 4) step = std::max<int64_t>(step, zp_ceil_div(4 * zp_ceil_div(total, N), pieces));
  return NodeCut{(int)N, parts, (uint32_t)step, total ? (uint32_t)((total - 1) / step) : 0u, (uint32_t)(pieces * step)};
}
struct NodeEdges {
  int n, beg, own, sbeg, total;          // node; first and number of the edges into it; first edge out; of both
  const int32_t *perm_src;
  int first, last;                       // this block's stretch of them
  uint32_t cut0, cut1;                   // first and last cut of the node (a cut node: cut0 <= cut1)
  __host__ __device__ __forceinline__ NodeEdges(int block, const NodeCut &cut, int64_t E, const int32_t *row_ptr,
                                                const int32_t *view, const int32_t *row_ptr_src) {
    const int N = cut.nodes;
    auto before = [&](int k) { return (uint32_t)row_ptr[k] + (view ? (uint32_t)row_ptr_src[k] : 0u); };
    const bool tail = block >= cut.ends();
    uint32_t at = 0;
    int part = 0, parts = 1;
    if (!tail) {
      parts = cut.parts;
      n = block / parts;
      part = block - n * parts;
    } else {                             // the node that the cut falls into: the last that begins at it or before
      at = (uint32_t)(block - cut.ends() + 1) * cut.step;
      int lo = 0, hi = N;                // before(lo) <= at; by halves it took 3 us of a block with nothing to do
      while (lo < hi) {
#ifdef __CUDA_ARCH__
        const int stride = (hi - lo + blockDim.x - 1) / blockDim.x, k = lo + ((int)threadIdx.x + 1) * stride;
        const int below = __syncthreads_count(k <= hi && before(k) <= at);
        lo += below * stride;
        hi = min(hi, lo + stride - 1);
#else
        const int mid = (lo + hi + 1) / 2;
        if (before(mid) <= at) lo = mid;
        else hi = mid - 1;
#endif
      }
      n = lo;
    }
    beg = row_ptr[n];
    total = own = (n < N ? row_ptr[n + 1] : (int)E) - beg;
    sbeg = 0;
    perm_src = view;
    if (view && n < N) {
      sbeg = row_ptr_src[n];
      total += row_ptr_src[n + 1] - sbeg;
    }
    int lo = 0, hi = total;
    cut0 = 1;
    cut1 = 0;
    if ((uint32_t)total > cut.whole) {
      const uint32_t begin = before(n);
      cut0 = begin / cut.step + 1;
      cut1 = (begin + (uint32_t)total - 1) / cut.step;
      if (!tail) {
        hi = (int)(cut0 * cut.step - begin);
      } else if (at > begin && at - begin < (uint32_t)total) {
        lo = (int)(at - begin);
        hi = total - lo < (int)cut.step ? total : lo + (int)cut.step;
      } else {
        hi = 0;
      }
    } else if (tail) {
      hi = 0;
    }
    first = lo + (int)((int64_t)(hi - lo) * part / parts);
    last = lo + (int)((int64_t)(hi - lo) * (part + 1) / parts);
  }
  __host__ __device__ __forceinline__ int64_t row(const NodeCut &cut) const { return n < cut.nodes ? n : 0; }
  // -1: past this block's
  __host__ __device__ __forceinline__ int edge(int i) const {
    if (i >= last) return -1;
    return i < own ? beg + i : perm_src[sbeg + i - own];
  }
};

// Puts one degree's rows of an edge on their way: ROWS |m| <= mmax (m'-major, `stride` floats apart), RAD its
// radial gains (2C floats apart); in shared memory as StageEdge.
template <int L, int LMAX, typename V, bool ROWS, bool RAD>
__device__ __forceinline__ void stage_degree(const ZpTables &t, const float *rows, int stride, const float *rad,
                                             float *row_s, float *rad_s, int ls) {
  constexpr int B = 4 * VecOf<V>::n;
  const int mm = t.mmax < L ? t.mmax : L, C2 = 2 * t.C;
  float *rs = row_s + (ROWS ? t.deg_row[L] * ls : 0), *gs = rad_s + (RAD ? t.deg_rad[L] * ls : 0);
  int r = L, k = L;                              // row m = 0, gain |m| = 0 of this degree
  if (ROWS) cp_async<B>(rs, rows + r * stride);
  if (RAD) cp_async<B>(gs, rad + k * C2);
#pragma unroll 1
  for (int am = 1; am <= mm; ++am) {
    const int km = LMAX + 1 - am;                // rows of +am
    r += (am == 1 ? 1 : 2) * (km + 1) - 1;
    k += km;
    if (ROWS) {
      rs += 2 * ls;
      cp_async<B>(rs - ls, rows + r * stride);
      cp_async<B>(rs, rows + (r + km) * stride);
    }
    if (RAD) {
      gs += ls;
      cp_async<B>(gs, rad + k * C2);
    }
  }
}
// all degrees of a first edge, a commit group each; what the caller has requested goes with the first
template <int L, int LMAX, typename V, bool ROWS, bool RAD>
struct StageAll {
  static __device__ __forceinline__ void run(const ZpTables &t, const float *rows, int stride, const float *rad,
                                             float *row_s, float *rad_s, int ls, bool live) {
    if constexpr (L > 0) StageAll<L - 1, LMAX, V, ROWS, RAD>::run(t, rows, stride, rad, row_s, rad_s, ls, live);
    if (live) stage_degree<L, LMAX, V, ROWS, RAD>(t, rows, stride, rad, row_s, rad_s, ls);
    cp_async_commit();
  }
};
// A worker's lanes request an edge's rotation.  Its entries are made into pairs where they are used, 300
// instructions of 2400 an edge; copied into pairs, four bytes at a time, they took a tenth longer at lmax 4 and half
// as long again at lmax 6, where their room costs blocks too.
__device__ __forceinline__ void stage_rot(const float *rot, float *rot_s, int ld, int li, int G) {
  for (int i = 4 * li; i < ld; i += 4 * G) cp_async<16>(rot_s + i, rot + i);
}
// Puts the node's K rows on their way into shared memory, ls floats a row: every lane its channels (at x, x_s) of
// its worker's share of the rows.  For all workers, so a block meets once they have landed.
template <typename V>
__device__ __forceinline__ void stage_node(const float *x, int C, int K, int w, int workers, float *x_s, int ls) {
  for (int k = w; k < K; k += workers) cp_async<4 * VecOf<V>::n>(x_s + k * ls, x + (size_t)k * C);
}
