// Gather / rotate / scatter kernels around the SO(2) contraction.
//
//   rotate_in            a[e, r, c2] = radial[e, .] * sum_j rot[e, r, j] * [x_src ; x_dst][l_r^2 + j, c2]
//   rotate_back_scatter  node_out[n, l^2 + j, c] = sum_{e -> n} env_e * sum_r rot[e, r, j] * y[e, r, c]
//
// They take over blocks/eso2_ref.py:334-335 (gather + rotate in, with the radial gain of
// :269-271, :284-285 applied while the row is in registers) and :343-349 (envelope, rotate
// back, index_add_).  The rotation is block diagonal in the degree l, so each thread keeps
// one degree's 2l+1 input rows of its channel group in registers and forms only the rows with
// |m| <= mmax.  Channels are the fastest axis everywhere: a thread owns four consecutive
// channels (two in rotate_back_scatter at lmax 5 and 6) and moves them with one vector load/store.  No atomics: every output element is
// produced by exactly one thread, in an order fixed by the CSR offsets.
#include <algorithm>

#include "zp_rotate.cuh"

namespace {

// ------------------------------------------------------------------------------------------
// rotate_in: one (edge, channel quad) per thread
// ------------------------------------------------------------------------------------------
// Moves 31.8 KB of HBM per edge at lmax 4 / mmax 2 / C 128 (radial rows in, planes out; the node rows
// come from L2).  What kept it from that rate was waiting (a radial row requested one step before
// its use) and address arithmetic: the radial rows are put in flight together at the start, and
// rows are walked with fixed steps.
constexpr int kRotInThreads = 256;
constexpr int kRotInMaxEdges = 16;       // narrow rows: bounds the rotations held in shared memory

template <int L, int LMAX, int FMT>
struct RotIn {
  // rot_s: the edge's rotation; rad_s: this thread's radial gains; out: this thread's quad in row 0
  static __device__ __forceinline__ void run(const ZpTables &t, const float *xrow,
                                             const float2 *rot_s, const float *rad_s, int ls,
                                             uint16_t *out, int64_t plane_bytes, u64 inv) {
    RotIn<L - 1, LMAX, FMT>::run(t, xrow, rot_s, rad_s, ls, out, plane_bytes, inv);
    constexpr int n = 2 * L + 1;
    const int C2 = 2 * t.C;
    F4 u[n];
    const float *xl = xrow + L * L * t.C;
#pragma unroll
    for (int j = 0; j < n; ++j) u[j] = load4(xl + j * t.C);
    const int mm = t.mmax < L ? t.mmax : L;
    const float2 *w = rot_s + t.deg_rot[L];
    const float *g = rad_s + t.deg_rad[L] * ls;
    uint16_t *o = out + L * C2;
    cp_async_wait<LMAX - L>();             // the radial gains of degrees 0..L have landed
    {
      F4 acc = zero4();
      for_row<n>(w, [&](int j, u64 c) { axpy4(acc, c, u[j]); });
      put4<FMT>(o, plane_bytes, mul4(acc, load4(g)), inv);
    }
    // a real loop over |m| (one copy of the body per degree keeps the kernel's code inside the
    // instruction cache)
#pragma unroll 1
    for (int am = 1; am <= mm; ++am) {
      const int km = LMAX + 1 - am;
      w += 2 * (n + 1);
      g += ls;
      o += ((am == 1 ? 1 : 2) * (km + 1) - 1) * C2;
      const F4 gain = load4(g);
      F4 ap = zero4(), an = zero4();
      for_row<n>(w - (n + 1), [&](int j, u64 c) { axpy4(ap, c, u[j]); });
      for_row<n>(w, [&](int j, u64 c) { axpy4(an, c, u[j]); });
      put4<FMT>(o, plane_bytes, mul4(ap, gain), inv);
      put4<FMT>(o + km * C2, plane_bytes, mul4(an, gain), inv);
    }
  }
};
template <int LMAX, int FMT>
struct RotIn<-1, LMAX, FMT> {
  static __device__ __forceinline__ void run(const ZpTables &, const float *, const float2 *,
                                             const float *, int, uint16_t *, int64_t, u64) {}
};

template <int LMAX, int FMT>
__global__ void __launch_bounds__(kRotInThreads, (LMAX <= 3 ? 4 : 3))
rotate_in_kernel(const __grid_constant__ ZpTables t, int64_t E, int epb,
                 const float *__restrict__ x, const int32_t *__restrict__ src,
                 const int32_t *__restrict__ dst, const float *__restrict__ rot,
                 const float *__restrict__ radial, const ZpPlanes a1, const ZpScale scale) {
  zp_after_previous();
  extern __shared__ __align__(16) float rot_in_s[];  // radial [rad_rows][blockDim] x 4 | rot [epb][rot_ld] dup.
  const int ls = 4 * blockDim.x;
  float *rad_s = rot_in_s + 4 * threadIdx.x;
  float2 *rot_s = reinterpret_cast<float2 *>(rot_in_s + (size_t)t.rad_rows * ls);
  const int Q = t.C / 2;                                 // channel quads of the 2C-wide message
  const int64_t e0 = (int64_t)blockIdx.x * epb;
  const int n_e = (int)min((int64_t)epb, E - e0);
  const int le = threadIdx.x / Q, c2 = 4 * (threadIdx.x - le * Q);
  const int64_t e = e0 + le;
  if (le < n_e)
    StageEdge<LMAX, LMAX, false, true>::run(t, nullptr, 0, nullptr, radial + (size_t)e * t.R + c2, rad_s, ls);
  stage_dup(rot + e0 * t.rot_ld, rot_s, t.rot_ld, n_e);
  const float inv = zp_publish_scale(a1, scale, blockIdx.x == 0 && threadIdx.x == 0);
  __syncthreads();
  if (le >= n_e) return;
  const bool second = c2 >= t.C;
  const int64_t node = second ? dst[e] : src[e];
  const float *xrow = x + (size_t)node * t.K * t.C + (second ? c2 - t.C : c2);
  RotIn<LMAX, LMAX, FMT>::run(t, xrow, rot_s + le * t.rot_ld, rad_s, ls,
                              static_cast<uint16_t *>(a1.base) + e * a1.ld + c2, 2 * a1.plane_stride,
                              pack2(inv, inv));
}

// The same by node (zp_rotate.cuh), for callers with a source view.  Four channels a lane.  In a training step at
// lmax 4 / C 128, 60 000 edges in two planes 571 -> 510 us, 384 000 in one 3.39 -> 2.45 ms.
template <int L, int LMAX, int FMT>
struct RotInN {
  static __device__ __forceinline__ void run(const ZpTables &t, const float *x_s, const float *rot, float *rad_s, int ls,
                                             uint16_t *out, int64_t plane_bytes, u64 inv, bool live, const float *next,
                                             bool more) {
    if constexpr (L > 0) RotInN<L - 1, LMAX, FMT>::run(t, x_s, rot, rad_s, ls, out, plane_bytes, inv, live, next, more);
    constexpr int n = 2 * L + 1;
    const int C2 = 2 * t.C;
    const int mm = t.mmax < L ? t.mmax : L;
    if (L > 0) cp_async_wait<LMAX>();    // (degree 0: the caller)
    if (live) {
      F4 u[n];
#pragma unroll
      for (int j = 0; j < n; ++j) u[j] = load4(x_s + (L * L + j) * ls);
      const float *w = rot + t.deg_rot[L];
      const float *g = rad_s + t.deg_rad[L] * ls;
      uint16_t *o = out + L * C2;
      {
        F4 acc = zero4();
        for_row_plain<n>(w, [&](int j, u64 c) { axpy4(acc, c, u[j]); });
        put4<FMT>(o, plane_bytes, mul4(acc, load4(g)), inv);
      }
#pragma unroll 1
      for (int am = 1; am <= mm; ++am) {
        const int km = LMAX + 1 - am;
        w += 2 * (n + 1);
        g += ls;
        o += ((am == 1 ? 1 : 2) * (km + 1) - 1) * C2;
        const F4 gain = load4(g);
        F4 ap = zero4(), an = zero4();
        for_row_plain<n>(w - (n + 1), [&](int j, u64 c) { axpy4(ap, c, u[j]); });
        for_row_plain<n>(w, [&](int j, u64 c) { axpy4(an, c, u[j]); });
        put4<FMT>(o, plane_bytes, mul4(ap, gain), inv);
        put4<FMT>(o + km * C2, plane_bytes, mul4(an, gain), inv);
      }
    }
    if (more) stage_degree<L, LMAX, F4, false, true>(t, nullptr, 0, next, nullptr, rad_s, ls);
    cp_async_commit();                   // (with degree 0 goes the rotation, requested before)
  }
};

// shared memory: x [K][G] vectors | per worker: radial gains [rad_rows][G] | per worker: two rotations [rot_ld]
template <int LMAX, int FMT>
__global__ void __launch_bounds__(32 * kNodeMaxWarps, 2)
node_rotate_in_kernel(const __grid_constant__ ZpTables t, const NodeCut cut, int64_t E, int G, int quads,
                      const float *__restrict__ x, const int32_t *__restrict__ row_ptr,
                      const int32_t *__restrict__ perm_src, const int32_t *__restrict__ row_ptr_src,
                      const float *__restrict__ rot, const float *__restrict__ radial, const ZpPlanes a1,
                      const ZpScale scale) {
  zp_after_previous();
  constexpr int K = (LMAX + 1) * (LMAX + 1);
  extern __shared__ __align__(16) float node_s[];
  const int workers = blockDim.x / G, w = threadIdx.x / G, li = threadIdx.x % G, ls = 4 * G;
  const int c0 = blockIdx.y * quads * 4, mine = min(quads, (t.C - c0) / 4);
  const bool active = li < mine;
  const int c = c0 + 4 * li;
  float *x_s = node_s, *stage = node_s + (size_t)K * ls, *rad_s = stage + (size_t)w * t.rad_rows * ls + 4 * li;
  float *rot_s = stage + (size_t)workers * t.rad_rows * ls + (size_t)w * 2 * t.rot_ld;
  const float inv = zp_publish_scale(a1, scale, blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0);
  const u64 inv2 = pack2(inv, inv);
  const NodeEdges edges(blockIdx.x, cut, E, row_ptr, perm_src, row_ptr_src);
  if (edges.first == edges.last) return;
  auto column = [&](int i) { return (i < edges.own ? t.C : 0) + c; };
  auto gains = [&](int e, int i) { return radial + (size_t)(e < 0 ? 0 : e) * t.R + column(i); };
  auto rotation = [&](int64_t e, int buffer) {
    stage_rot(rot + (size_t)e * t.rot_ld, rot_s + buffer * t.rot_ld, t.rot_ld, li, G);
  };
  const int i0 = edges.first + w;
  if (active) stage_node<F4>(x + (size_t)edges.row(cut) * t.K * t.C + c, t.C, K, w, workers, x_s + 4 * li, ls);
  int e = edges.edge(i0), e_next = edges.edge(i0 + workers);
  if (e >= 0) rotation(e, 0);
  StageAll<LMAX, LMAX, F4, false, true>::run(t, nullptr, 0, gains(e, i0), nullptr, rad_s, ls, e >= 0 && active);
  cp_async_wait<LMAX>();                 // the node's rows went with degree 0
  __syncthreads();
  for (int i = i0, buffer = 0; i - w < edges.last; i += workers, buffer ^= 1) {      // as often on all lanes
    const int e_after = edges.edge(i + 2 * workers);
    cp_async_wait<LMAX>();               // degree 0 and the rotation have landed
    __syncwarp();                        // ... the other lanes' part of it, and all are done with the last
    if (e_next >= 0) rotation(e_next, buffer ^ 1);
    RotInN<LMAX, LMAX, FMT>::run(t, x_s + 4 * li, rot_s + buffer * t.rot_ld, rad_s, ls,
                                 static_cast<uint16_t *>(a1.base) + (e < 0 ? 0 : e) * a1.ld + column(i),
                                 2 * a1.plane_stride, inv2, e >= 0 && active, gains(e_next, i + workers),
                                 e_next >= 0 && active);
    e = e_next;
    e_next = e_after;
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------------------------------
// per-destination-node kernel (forward scatter)
// ------------------------------------------------------------------------------------------


// P channel pairs of a lane: y_e is the edge's rows in shared memory ([Km][row_stride], this lane's
// channels at c), acc the node's rows
template <int L, int LMAX, int P>
struct RotBack {
  static __device__ __forceinline__ void run(const ZpTables &t, const float *y_e, int row_stride,
                                             const float2 *rot_s, u64 env,
                                             u64 (&acc)[(LMAX + 1) * (LMAX + 1)][P], int c) {
    RotBack<L - 1, LMAX, P>::run(t, y_e, row_stride, rot_s, env, acc, c);
    constexpr int n = 2 * L + 1;
    const int mm = t.mmax < L ? t.mmax : L;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const int am = i > L ? i - L : L - i;
      if (am <= mm) {
        const int r = t.row_of[L][i];
        const u64 *yp = reinterpret_cast<const u64 *>(y_e + (size_t)r * row_stride + c);
        u64 y[P];
        if constexpr (P == 2) {
          const F4 v = load4(reinterpret_cast<const float *>(yp));
          y[0] = mul2(v.a, env);
          y[1] = mul2(v.b, env);
        } else {
          y[0] = mul2(yp[0], env);
        }
        for_row<n>(rot_s + t.row_off[r], [&](int k, u64 w) {
#pragma unroll
          for (int v = 0; v < P; ++v) acc[L * L + k][v] = fma2(w, y[v], acc[L * L + k][v]);
        });
      }
    }
  }
};
template <int LMAX, int P>
struct RotBack<-1, LMAX, P> {
  static __device__ __forceinline__ void run(const ZpTables &, const float *, int, const float2 *,
                                             u64, u64 (&)[(LMAX + 1) * (LMAX + 1)][P], int) {}
};

// One block (four warps) owns 32 x VEC channels of one destination node.  The node's edges are
// dealt round-robin to the warps (warp w takes edges w, w + 4, ... of the CSR segment), which cuts
// the serial chain per node by four; the four partial sums are then added in warp order through
// shared memory, so the result does not depend on timing.
// Each warp keeps the rows of its NEXT edge in flight while it rotates the current one: every lane
// copies its own channels of the Km rows into a two-stage shared buffer with cp.async (16 or 8
// bytes per row), so the memory latency is paid once per edge, not once per row.
constexpr int kBackWarps = 4;

template <int LMAX, int VEC>
__global__ void __launch_bounds__(32 * kBackWarps, (LMAX >= 5 && VEC == 2 ? 3 : 1))
rotate_back_scatter_kernel(const __grid_constant__ ZpTables t, int64_t N,
                           const float *__restrict__ y, const float *__restrict__ env,
                           const float *__restrict__ rot, const int32_t *__restrict__ row_ptr,
                           float *__restrict__ node_out) {
  zp_after_previous();
  constexpr int K = (LMAX + 1) * (LMAX + 1);
  constexpr int W = 32 * VEC;              // channels of this block
  constexpr int P = VEC / 2;
  // rotation entries per lane of a staging warp: sum over l of (2l+1)(2l+2) at most
  constexpr int kRotMax = (LMAX + 1) * (LMAX + 2) * (4 * LMAX + 3) / 3;    // mmax = lmax: the most
  constexpr int NR = (kRotMax + 3 + 31) / 32;
  // rot [4][rot_main] duplicated | y stages [4 warps][2][Km][W], reused as partial [4][K][W] at the end
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  float2 *rot_s = reinterpret_cast<float2 *>(smem) + warp * t.rot_ld;
  float *region = smem + 2 * kBackWarps * t.rot_ld;
  float *ybuf = region + (size_t)warp * 2 * t.Km * W;
  float *part = region;
  const int64_t n = blockIdx.x;
  const int c0 = blockIdx.y * W;
  const int c = c0 + lane * VEC;
  const bool active = c < t.C;
  u64 acc[K][P];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int v = 0; v < P; ++v) acc[k][v] = 0ull;
  const int e_beg = row_ptr[n], e_end = row_ptr[n + 1];
  // the next edge's packed rotation is fetched into registers while the current one is used
  float nxt[NR];
  auto fetch = [&](int e) {
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int k = lane + 32 * i;
      nxt[i] = (e < e_end && k < t.rot_ld) ? rot[(size_t)e * t.rot_ld + k] : 0.f;
    }
  };
  auto stage_rows = [&](int e, int stage) {          // this lane's channels of edge e's Km rows
    if (e < e_end && active) {
      const float *src = y + (size_t)e * t.Km * t.C + c;
      float *dst = ybuf + (size_t)stage * t.Km * W + lane * VEC;
      for (int r = 0; r < t.Km; ++r) cp_async<4 * VEC>(dst + r * W, src + (size_t)r * t.C);
    }
    cp_async_commit();
  };
  fetch(e_beg + warp);
  stage_rows(e_beg + warp, 0);
  int stage = 0;
  for (int e = e_beg + warp; e < e_end; e += kBackWarps, stage ^= 1) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NR; ++i)
      if (lane + 32 * i < t.rot_ld) rot_s[lane + 32 * i] = make_float2(nxt[i], nxt[i]);
    const float env_e = env[e];
    fetch(e + kBackWarps);
    stage_rows(e + kBackWarps, stage ^ 1);
    cp_async_wait<1>();                  // everything but the group just committed has landed
    __syncwarp();
    if (active)
      RotBack<LMAX, LMAX, P>::run(t, ybuf + (size_t)stage * t.Km * W, W, rot_s, pack2(env_e, env_e),
                                  acc, lane * VEC);
  }
  cp_async_wait<0>();
  __syncthreads();                       // all warps are done with their stages: reuse as partials
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int v = 0; v < P; ++v)
      *reinterpret_cast<u64 *>(part + (warp * K + k) * W + lane * VEC + 2 * v) = acc[k][v];
  __syncthreads();
  for (int i = threadIdx.x; i < K * W; i += blockDim.x) {
    const int k = i / W, cc = i % W;
    if (c0 + cc < t.C) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < kBackWarps; ++w) s += part[(w * K + k) * W + cc];
      node_out[((size_t)n * K + k) * t.C + c0 + cc] = s;
    }
  }
}

// Final sums after the rotate-back epilogue of conv2.  The epilogue leaves, per m' row r, the
// partial sums of a node's edges: head[n] for the run that starts at the node's first edge and
// cont[b] for the run that enters 32-edge block b from the block before.  One block per node adds,
// per output row (l, j), the rows r of that degree in table order and, within a row, head first and
// then the continuation blocks in ascending order: a fixed order, so results repeat bit for bit.
__global__ void __launch_bounds__(128)
node_sum_kernel(const __grid_constant__ ZpTables t, int64_t N, const float *__restrict__ head,
                const float *__restrict__ cont, const int32_t *__restrict__ row_ptr,
                float *__restrict__ node_out) {
  zp_after_previous();
  const int64_t n = blockIdx.x;
  const int C4 = t.C / 4;
  const int beg = row_ptr[n], end = row_ptr[n + 1];
  const int b_first = beg >> 5, b_last = end > beg ? (end - 1) >> 5 : b_first;
  const size_t slab = (size_t)t.nnz * t.C;
  const float *hn = head + (size_t)n * slab;
  for (int i = threadIdx.x; i < t.K * C4; i += blockDim.x) {
    const int k = i / C4, c = (i - k * C4) * 4;
    int l = 0;
    while ((l + 1) * (l + 1) <= k) ++l;
    const int j = k - l * l;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (end > beg) {
      const int mm = t.mmax < l ? t.mmax : l;
      for (int q = l - mm; q <= l + mm; ++q) {
        const size_t o = (size_t)(t.rot_off[t.row_of[l][q]] + j) * t.C + c;
        float4 v = *reinterpret_cast<const float4 *>(hn + o);
        for (int b = b_first + 1; b <= b_last; ++b) {
          const float4 w = *reinterpret_cast<const float4 *>(cont + (size_t)b * slab + o);
          v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
    }
    *reinterpret_cast<float4 *>(node_out + ((size_t)n * t.K + k) * t.C + c) = acc;
  }
}

}  // namespace

int zp_launch_node_sum(const zp_plan *p, int64_t N, const float *head, const float *cont,
                       const int32_t *row_ptr, float *node_out, cudaStream_t st) {
  if (N == 0) return ZP_OK;
  zp_launch(node_sum_kernel, (unsigned)N, 128, 0, st, p->t, N, head, cont, row_ptr, node_out);
  ZP_LAUNCH_CHECK("node_sum_kernel");
  return ZP_OK;
}

int zp_launch_rotate_in(const zp_plan *p, int64_t E, const float *x, const int32_t *src,
                        const int32_t *dst, const ZpNodeView &view, const float *rot, const float *radial,
                        const ZpPlanes &a1, const ZpScale &scale, cudaStream_t st) {
  if (E == 0) return ZP_OK;
  const ZpTables &t = p->t;
  const int Q = t.C / 2;
  if (Q < 1 || Q > kRotInThreads) return ZP_ERR_UNSUPPORTED;
  // By node where it is the faster one.  Lanes without channels: 30 000 edges, by edge / by node, lmax 4, 64, 72,
  // 96, 112 and 128 channels 152 / 135, 175 / 263, 212 / 220, 250 / 265 and 262 / 244 us, lmax 6, 72, 96, 112 and 128 347 / 431,
  // 425 / 367, 411 / 355 and 520 / 392.  Half rows of other than whole 32-byte sectors are written twice: 56 and
  // 104 channels 144 / 222 and 202 / 289 at lmax 4, 290 / 360 and 390 / 464 at lmax 6.  Narrow rows at low degrees: lmax 2,
  // 257 000 edges of 32, 64 and 128 channels 287 / 378, 522 / 505 and 1 063 / 945.  And not where most nodes have
  // no edge (60 000 among 2 000 nodes of 100 000: 2 % of an inference).
  const NodeShape ns = zp_node_shape(t.C, 4);
  const bool full = t.lmax >= 5 ? t.C % 16 == 0 && 10 * ns.quads >= 7 * ns.G : ns.quads == ns.G;
  if (view.perm_src && full && (t.lmax >= 3 || t.C >= 64) && E >= view.nodes) {
    const int64_t N = view.nodes;
    const NodeLaunch nl = zp_node_launch(N * ns.groups, 2.0 * (double)E / (double)N, ns, t, t.rad_rows, 16, 4);
    const NodeCut cut = zp_node_cut(N, E, true, nl.parts);
    const dim3 grid(cut.blocks(), (unsigned)ns.groups);
#define CALL_FMT(LM, FMT)                                                                         \
  {                                                                                               \
    static ZpSmemOptIn opt_in;               /* per instantiation and device */                   \
    if (int rc_ = zp_ensure_smem(node_rotate_in_kernel<LM, FMT>, nl.smem, opt_in)) return rc_;    \
    zp_launch(node_rotate_in_kernel<LM, FMT>, grid, 32 * nl.warps, nl.smem, st, t, cut, E, ns.G, ns.quads, x, \
              view.row_ptr, view.perm_src, view.row_ptr_src, rot, radial, a1, scale);             \
    break;                                                                                        \
  }
#define CALL(LM)                                               \
  switch (zp_plane_format(a1)) {                               \
    case kFmtBf16: CALL_FMT(LM, kFmtBf16)                      \
    case kFmtFp16x2: CALL_FMT(LM, kFmtFp16x2)                  \
    default: CALL_FMT(LM, kFmtBf16x3)                          \
  }
    ZP_DISPATCH_LMAX(t.lmax, CALL)
#undef CALL
#undef CALL_FMT
    ZP_LAUNCH_CHECK("node_rotate_in_kernel");
    return ZP_OK;
  }
  int epb = kRotInThreads / Q;
  if (epb > kRotInMaxEdges) epb = kRotInMaxEdges;
  const dim3 grid((unsigned)zp_ceil_div(E, epb)), block(epb * Q);
  const size_t smem = (size_t)epb * (t.rot_ld * sizeof(float2) + Q * t.rad_rows * sizeof(float4));
#define CALL_FMT(LM, FMT)                                                                         \
  {                                                                                               \
    static ZpSmemOptIn opt_in;               /* per instantiation and device */                   \
    if (int rc_ = zp_ensure_smem(rotate_in_kernel<LM, FMT>, smem, opt_in)) return rc_;            \
    zp_launch(rotate_in_kernel<LM, FMT>, grid, block, smem, st, t, E, epb, x, src, dst, rot,      \
              radial, a1, scale);                                                                 \
    break;                                                                                        \
  }
#define CALL(LM)                                               \
  switch (zp_plane_format(a1)) {                               \
    case kFmtBf16: CALL_FMT(LM, kFmtBf16)                      \
    case kFmtFp16x2: CALL_FMT(LM, kFmtFp16x2)                  \
    default: CALL_FMT(LM, kFmtBf16x3)                          \
  }
  ZP_DISPATCH_LMAX(t.lmax, CALL)
#undef CALL
#undef CALL_FMT
  ZP_LAUNCH_CHECK("rotate_in_kernel");
  return ZP_OK;
}

int zp_launch_rotate_back_scatter(const zp_plan *p, int64_t N, const float *y, const float *env,
                                  const float *rot, const int32_t *row_ptr, float *node_out,
                                  cudaStream_t st) {
  if (N == 0) return ZP_OK;
  const ZpTables &t = p->t;
  const int vec = t.lmax <= 4 ? 4 : 2;     // K x VEC accumulators must fit in registers
  const dim3 grid((unsigned)N, (unsigned)zp_ceil_div(t.C, 32 * vec));
  const size_t rows = std::max<size_t>((size_t)t.K, 2 * (size_t)t.Km);   // partials | two y stages
  const size_t smem = (size_t)kBackWarps * (2 * t.rot_ld + rows * 32 * vec) * sizeof(float);
#define CALL(LM)                                                                               \
  {                                                                                            \
    auto kern = vec == 4 ? rotate_back_scatter_kernel<LM, 4> : rotate_back_scatter_kernel<LM, 2>; \
    static ZpSmemOptIn opt_in;             /* per instantiation and device */                    \
    if (int rc_ = zp_ensure_smem(kern, smem, opt_in)) return rc_;                              \
    zp_launch(kern, grid, 32 * kBackWarps, smem, st, t, N, y, env, rot, row_ptr, node_out);           \
  }
  ZP_DISPATCH_LMAX(t.lmax, CALL)
#undef CALL
  ZP_LAUNCH_CHECK("rotate_back_scatter_kernel");
  return ZP_OK;
}
