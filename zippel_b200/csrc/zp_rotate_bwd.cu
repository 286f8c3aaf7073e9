// The VJPs of the rotate kernels.
//
//   rotate_grad_out      the VJP of rotate_back_scatter (needs y), by edge or by node
//   rotate_in_bwd        the VJP of rotate_in by node, with the gradient of x_node
//
// (autograd through blocks/eso2_ref.py:334-349).  By edge, one (edge, channel quad) per thread; by node
// see zp_rotate.cuh, for the forward kernels zp_rotate.cu.
#include <algorithm>

#include "zp_rotate.cuh"

namespace {

// ------------------------------------------------------------------------------------------
// rotate_grad_out by edge: one (edge, channel quad) per thread
// ------------------------------------------------------------------------------------------
// Gradient of the rotation.  Both kernels hold, for every row (l, m) of an edge, its rotated value
// b[m] (a in the edge frame, or the rotated upstream gradient) and the factor p[m] it is multiplied
// with.  The edge's rotation enters the loss through sum_{rows, channels} p . b only, and every
// derivative of a rotation is a rotation generator times it, so the derivatives under turns of the
// edge frame about its own axis (T0) and the two perpendicular ones (T1, T2) are
//     T0 = sum m (p[m] b[-m] - p[-m] b[m])
//     T1 = sum c_lm [ p[m] b[m+1] - p[m+1] b[m]  +  p[-m] b[-m-1] - p[-m-1] b[-m] ]
//     T2 = sum c_lm [ p[-m-1] b[m] - p[m] b[-m-1]  +  p[-m] b[m+1] - p[m+1] b[-m] ]
// (terms with -m only for m > 0; c_lm: ZpTables::couple).  p is zero beyond |m| = mmax, b is needed
// up to mmax + 1.  Three sums per edge instead of one per rotation entry (115 at lmax 4 / mmax 2):
// the channel reductions of those were half of these kernels' instructions, and the array of
// gradients and the kernel that walked back through the construction of the matrices are gone.
constexpr int kEdgeThreads = 128;
constexpr int kEdgesPerBlock = 16;       // narrow rows: bounds the rotations held in shared memory

struct Torque {
  u64 t0, t1, t2;
  template <typename V>
  __device__ __forceinline__ void own(int m, const V &pp, const V &pm, const V &bp, const V &bm) {
    const u64 f = pack2((float)m, (float)m);
    t0 = fma2(f, sub2(dot4(0ull, pp, bm), dot4(0ull, pm, bp)), t0);
  }
  // (m, m + 1): q, s = p and b of m; y, t = those of m + 1
  template <typename V>
  __device__ __forceinline__ void pair(float c, const V &qp, const V &qm, const V &sp, const V &sm,
                                       const V &yp, const V &ym, const V &tp, const V &tm) {
    const u64 cc = pack2(c, c);
    t1 = fma2(cc, sub2(dot4(dot4(0ull, qp, tp), qm, tm), dot4(dot4(0ull, yp, sp), ym, sm)), t1);
    t2 = fma2(cc, sub2(dot4(dot4(0ull, ym, sp), qm, tp), dot4(dot4(0ull, qp, tm), yp, sm)), t2);
  }
  // (mmax, mmax + 1): p of the outer row is zero
  template <typename V>
  __device__ __forceinline__ void outer(float c, const V &qp, const V &qm, const V &tp, const V &tm) {
    const u64 cc = pack2(c, c);
    t1 = fma2(cc, dot4(dot4(0ull, qp, tp), qm, tm), t1);
    t2 = fma2(cc, sub2(dot4(0ull, qm, tp), dot4(0ull, qp, tm)), t2);
  }
};
// Sums a float4 per thread over the Q threads of every edge of the block, in a fixed order: a warp
// per edge, its lanes stepping through the edge's threads.  put(edge slot, sum) on one lane.
template <typename Put>
__device__ __forceinline__ void reduce_edges(float4 *part_s, const float4 &mine, int Q, int n_e, Put put) {
  part_s[threadIdx.x] = mine;
  __syncthreads();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, warps = blockDim.x / 32;
  for (int s = warp; s < n_e; s += warps) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = lane; q < Q; q += 32) {
      const float4 o = part_s[s * Q + q];
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    v.x = warp_sum(v.x); v.y = warp_sum(v.y); v.z = warp_sum(v.z); v.w = warp_sum(v.w);
    if (lane == 0) put(s, v);
  }
}

// ---- VJP of rotate_back_scatter -----------------------------------------------------------
//   t[r]        = sum_j rot[r, j] g[dst, l^2 + j]        (g = grad of node_out)
//   dy[e, r]    = env_e * t[r]                            (written as operand planes)
//   grad_env[e] = sum_{r, c} y[e, r, c] t[r, c]
//   torque[e]   = env_e * (sums above with p = y, b = t)
template <int L, int LMAX, int FMT>
struct GradOutE {
  // y_s: this thread's rows of y; out: this thread's quad in row 0 of dy
  static __device__ __forceinline__ void run(const ZpTables &t, const float *g_row, const float *y_s,
                                             int ls, uint16_t *out, int64_t plane_bytes, u64 inv,
                                             const float2 *rot_s, u64 env, u64 &genv, Torque &T) {
    GradOutE<L - 1, LMAX, FMT>::run(t, g_row, y_s, ls, out, plane_bytes, inv, rot_s, env, genv, T);
    constexpr int n = 2 * L + 1;
    const int mm = t.mmax < L ? t.mmax : L;
    F4 g[n];
    const float *gl = g_row + L * L * t.C;
#pragma unroll
    for (int j = 0; j < n; ++j) g[j] = load4(gl + j * t.C);
    const float2 *w = rot_s + t.deg_rot[L];
    const float *yr = y_s + t.deg_row[L] * ls;
    uint16_t *o = out + L * t.C;
    cp_async_wait<LMAX - L>();             // the rows of y of degrees 0..L have landed
    F4 qp = load4(yr), qm = zero4(), sp = zero4(), sm = zero4();          // row m = 0
    for_row<n>(w, [&](int j, u64 c) { axpy4(sp, c, g[j]); });
    genv = dot4(genv, qp, sp);
    put4<FMT>(o, plane_bytes, F4{mul2(sp.a, env), mul2(sp.b, env)}, inv);
    // a real loop over |m| (one copy of the body per degree: the unrolled form spent more time
    // waiting for instructions than for data)
#pragma unroll 1
    for (int am = 1; am <= mm; ++am) {
      const int km = LMAX + 1 - am;
      w += 2 * (n + 1);
      yr += 2 * ls;
      o += ((am == 1 ? 1 : 2) * (km + 1) - 1) * t.C;
      const F4 yp = load4(yr - ls), ym = load4(yr);
      F4 tp = zero4(), tm = zero4();
      for_row<n>(w - (n + 1), [&](int j, u64 c) { axpy4(tp, c, g[j]); });
      for_row<n>(w, [&](int j, u64 c) { axpy4(tm, c, g[j]); });
      genv = dot4(dot4(genv, yp, tp), ym, tm);
      put4<FMT>(o, plane_bytes, F4{mul2(tp.a, env), mul2(tp.b, env)}, inv);
      put4<FMT>(o + km * t.C, plane_bytes, F4{mul2(tm.a, env), mul2(tm.b, env)}, inv);
      T.own(am, yp, ym, tp, tm);
      T.pair(t.couple[L][am - 1], qp, qm, sp, sm, yp, ym, tp, tm);
      qp = yp; qm = ym; sp = tp; sm = tm;
    }
    if (L > t.mmax) {
      w += 2 * (n + 1);
      F4 tp = zero4(), tm = zero4();
      for_row<n>(w - (n + 1), [&](int j, u64 c) { axpy4(tp, c, g[j]); });
      for_row<n>(w, [&](int j, u64 c) { axpy4(tm, c, g[j]); });
      T.outer(t.couple[L][mm], qp, qm, tp, tm);
    }
  }
};
template <int LMAX, int FMT>
struct GradOutE<-1, LMAX, FMT> {
  static __device__ __forceinline__ void run(const ZpTables &, const float *, const float *, int,
                                             uint16_t *, int64_t, u64, const float2 *, u64, u64 &,
                                             Torque &) {}
};

// shared memory: partial sums [blockDim] float4 | y [Km][blockDim] float4 | rot [epb][rot_ld] dup.
template <int LMAX, int FMT>
__global__ void __launch_bounds__(kEdgeThreads, (LMAX <= 1 ? 6 : 4))
rotate_grad_out_kernel(const __grid_constant__ ZpTables t, int64_t E, int epb,
                       const float *__restrict__ g_out, const float *__restrict__ y,
                       const float *__restrict__ env, const float *__restrict__ rot,
                       const int32_t *__restrict__ dst, const ZpPlanes dy, const ZpScale scale,
                       float *__restrict__ grad_env, float4 *__restrict__ torque) {
  zp_after_previous();
  extern __shared__ __align__(16) float4 edge_s[];
  float *y_s = reinterpret_cast<float *>(edge_s + blockDim.x) + 4 * threadIdx.x;
  const int ls = 4 * blockDim.x;
  float2 *rot_s = reinterpret_cast<float2 *>(edge_s + (size_t)blockDim.x * (1 + t.Km));
  const int Q = t.C / 4;
  const int64_t e0 = (int64_t)blockIdx.x * epb;
  const int n_e = (int)min((int64_t)epb, E - e0);
  const int le = threadIdx.x / Q, c = 4 * (threadIdx.x - le * Q);
  const int64_t e = e0 + le;
  if (le < n_e)
    StageEdge<LMAX, LMAX, true, false>::run(t, y + (size_t)e * t.Km * t.C + c, t.C, y_s, nullptr, nullptr, ls);
  stage_dup(rot + e0 * t.rot_ld, rot_s, t.rot_ld, n_e);
  const float inv = zp_publish_scale(dy, scale, blockIdx.x == 0 && threadIdx.x == 0);
  __syncthreads();
  float4 sums = make_float4(0.f, 0.f, 0.f, 0.f);
  if (le < n_e) {
    const float env_e = env[e];
    Torque T{0ull, 0ull, 0ull};
    u64 genv = 0ull;
    GradOutE<LMAX, LMAX, FMT>::run(t, g_out + (size_t)dst[e] * t.K * t.C + c, y_s, ls,
                                   static_cast<uint16_t *>(dy.base) + e * dy.ld + c, 2 * dy.plane_stride,
                                   pack2(inv, inv), rot_s + le * t.rot_ld, pack2(env_e, env_e), genv, T);
    sums = make_float4(sum2(T.t0) * env_e, sum2(T.t1) * env_e, sum2(T.t2) * env_e, sum2(genv));
  }
  reduce_edges(edge_s, sums, Q, n_e, [&](int s, const float4 &v) {
    torque[e0 + s] = make_float4(v.x, v.y, v.z, 0.f);
    grad_env[e0 + s] = v.w;
  });
}

// The same by node (zp_rotate.cuh): a block for the edges into one node, whose rows of g are read once.  60 000
// edges at lmax 4 / mmax 2 / C 128: 32 KB an edge from L2 by edge, 19 here, 321 -> 207 us in a training step; 384 000
// in one plane 1.98 -> 1.22 ms.
template <int L, int LMAX, int FMT>
struct GradOutN {
  static __device__ __forceinline__ void run(const ZpTables &t, const float *g_s, float *y_s, int ls, uint16_t *out,
                                             int64_t plane_bytes, u64 inv, const float *rot, u64 env, bool live,
                                             const float *next, bool more, u64 &genv, Torque &T) {
    if constexpr (L > 0)
      GradOutN<L - 1, LMAX, FMT>::run(t, g_s, y_s, ls, out, plane_bytes, inv, rot, env, live, next, more, genv, T);
    constexpr int n = 2 * L + 1;
    const int mm = t.mmax < L ? t.mmax : L;
    if (L > 0) cp_async_wait<LMAX>();    // (degree 0: the caller)
    if (live) {
      F4 g[n];
#pragma unroll
      for (int j = 0; j < n; ++j) g[j] = load4(g_s + (L * L + j) * ls);
      const float *w = rot + t.deg_rot[L];
      const float *yr = y_s + t.deg_row[L] * ls;
      uint16_t *o = out + L * t.C;
      F4 qp = load4(yr), qm = zero4(), sp = zero4(), sm = zero4();          // row m = 0
      for_row_plain<n>(w, [&](int j, u64 c) { axpy4(sp, c, g[j]); });
      genv = dot4(genv, qp, sp);
      put4<FMT>(o, plane_bytes, F4{mul2(sp.a, env), mul2(sp.b, env)}, inv);
#pragma unroll 1
      for (int am = 1; am <= mm; ++am) {
        const int km = LMAX + 1 - am;
        w += 2 * (n + 1);
        yr += 2 * ls;
        o += ((am == 1 ? 1 : 2) * (km + 1) - 1) * t.C;
        const F4 yp = load4(yr - ls), ym = load4(yr);
        F4 tp = zero4(), tm = zero4();
        for_row_plain<n>(w - (n + 1), [&](int j, u64 c) { axpy4(tp, c, g[j]); });
        for_row_plain<n>(w, [&](int j, u64 c) { axpy4(tm, c, g[j]); });
        genv = dot4(dot4(genv, yp, tp), ym, tm);
        put4<FMT>(o, plane_bytes, F4{mul2(tp.a, env), mul2(tp.b, env)}, inv);
        put4<FMT>(o + km * t.C, plane_bytes, F4{mul2(tm.a, env), mul2(tm.b, env)}, inv);
        T.own(am, yp, ym, tp, tm);
        T.pair(t.couple[L][am - 1], qp, qm, sp, sm, yp, ym, tp, tm);
        qp = yp; qm = ym; sp = tp; sm = tm;
      }
      if (L > t.mmax) {
        w += 2 * (n + 1);
        F4 tp = zero4(), tm = zero4();
        for_row_plain<n>(w - (n + 1), [&](int j, u64 c) { axpy4(tp, c, g[j]); });
        for_row_plain<n>(w, [&](int j, u64 c) { axpy4(tm, c, g[j]); });
        T.outer(t.couple[L][mm], qp, qm, tp, tm);
      }
    }
    if (more) stage_degree<L, LMAX, F4, true, false>(t, next, t.C, nullptr, y_s, nullptr, ls);
    cp_async_commit();                   // (with degree 0 goes the rotation, requested before)
  }
};

// shared memory: g [K][G] vectors | per worker: rows of y [Km][G] | per worker: two rotations [rot_ld]
template <int LMAX, int FMT>
__global__ void __launch_bounds__(32 * kNodeMaxWarps, 2)
node_rotate_grad_out_kernel(const __grid_constant__ ZpTables t, const NodeCut cut, int64_t E, int G, int quads,
                            const float *__restrict__ g_out, const float *__restrict__ y,
                            const float *__restrict__ env, const float *__restrict__ rot,
                            const int32_t *__restrict__ row_ptr, const ZpPlanes dy, const ZpScale scale,
                            float *__restrict__ grad_env, float4 *__restrict__ torque) {
  zp_after_previous();
  constexpr int K = (LMAX + 1) * (LMAX + 1);
  extern __shared__ __align__(16) float node_s[];
  const int workers = blockDim.x / G, w = threadIdx.x / G, li = threadIdx.x % G, ls = 4 * G;
  const bool active = li < quads;
  const int c = 4 * li;
  float *g_s = node_s, *stage = node_s + (size_t)K * ls, *y_s = stage + (size_t)w * t.Km * ls + c;
  float *rot_s = stage + (size_t)workers * t.Km * ls + (size_t)w * 2 * t.rot_ld;
  const float inv = zp_publish_scale(dy, scale, blockIdx.x == 0 && threadIdx.x == 0);
  const u64 inv2 = pack2(inv, inv);
  const NodeEdges edges(blockIdx.x, cut, E, row_ptr, nullptr, nullptr);
  if (edges.first == edges.last) return;
  auto rows = [&](int e) { return y + (size_t)(e < 0 ? 0 : e) * t.Km * t.C + c; };
  auto rotation = [&](int64_t e, int buffer) {
    stage_rot(rot + (size_t)e * t.rot_ld, rot_s + buffer * t.rot_ld, t.rot_ld, li, G);
  };
  const int i0 = edges.first + w;
  if (active) stage_node<F4>(g_out + (size_t)edges.row(cut) * t.K * t.C + c, t.C, K, w, workers, g_s + c, ls);
  int e = edges.edge(i0), e_next = edges.edge(i0 + workers);
  if (e >= 0) rotation(e, 0);
  StageAll<LMAX, LMAX, F4, true, false>::run(t, rows(e), t.C, nullptr, y_s, nullptr, ls, e >= 0 && active);
  cp_async_wait<LMAX>();                 // the node's rows went with degree 0
  __syncthreads();
  for (int i = i0, buffer = 0; i - w < edges.last; i += workers, buffer ^= 1) {      // as often on all lanes
    const int e_after = edges.edge(i + 2 * workers);
    const float env_e = e >= 0 ? env[e] : 0.f;
    Torque T{0ull, 0ull, 0ull};
    u64 genv = 0ull;
    cp_async_wait<LMAX>();               // degree 0 and the rotation have landed
    __syncwarp();                        // ... the other lanes' part of it, and all are done with the last
    if (e_next >= 0) rotation(e_next, buffer ^ 1);
    GradOutN<LMAX, LMAX, FMT>::run(t, g_s + c, y_s, ls, static_cast<uint16_t *>(dy.base) + (e < 0 ? 0 : e) * dy.ld + c,
                                   2 * dy.plane_stride, inv2, rot_s + buffer * t.rot_ld, pack2(env_e, env_e),
                                   e >= 0 && active, rows(e_next), e_next >= 0 && active, genv, T);
    float t0 = sum2(T.t0), t1 = sum2(T.t1), t2 = sum2(T.t2), ge = sum2(genv);
    for (int o = G / 2; o > 0; o >>= 1) {
      t0 += __shfl_xor_sync(0xffffffffu, t0, o);
      t1 += __shfl_xor_sync(0xffffffffu, t1, o);
      t2 += __shfl_xor_sync(0xffffffffu, t2, o);
      ge += __shfl_xor_sync(0xffffffffu, ge, o);
    }
    if (li == 0 && e >= 0) {
      torque[e] = make_float4(t0 * env_e, t1 * env_e, t2 * env_e, 0.f);
      grad_env[e] = ge;
    }
    e = e_next;
    e_next = e_after;
  }
  cp_async_wait<0>();
}

// ---- VJP of rotate_in over the 2C message channels -----------------------------------------------
//   a[r]   = sum_j rot[r, j] u[l^2 + j]            (formed again; u = x_src | x_dst half)
//   ga[r]  = da[e, r] * radial
//   grad_radial[e, col] = sum over the +m / -m rows sharing the column of  da[r] * a[r]
//                         (fp32 rows, or operand planes of the radial layer's VJP)
//   torque[e] += sums above with p = ga, b = a
//   grad_x[node, l^2 + j] = sum over the node's edges and their rows  rot[r, j] ga[r]
template <int FMT> struct Elem { using type = uint16_t; };
template <> struct Elem<kFmtFp32> { using type = float; };

// By node (zp_rotate.cuh).  What an edge adds to the node's gradient stays in registers: written per
// edge and summed afterwards it was half of all bytes (2 x 25.6 KB of 95 KB an edge at lmax 4, C 128).  Four
// channels a lane, two from lmax 5 on: 36 rows of four do not fit the registers.  In a training step 60 000 edges in
// two planes, sums included, 1 121 -> 523 us, 384 000 in one 7.13 -> 3.43 ms; bound by fixed latencies and instruction
// issue (2 330 a worker and edge half, eight warps to an SM at 240 registers), HBM at half its rate.
// SUMS: the gradient of x_node is wanted (not in a force evaluation; the others are the same to the last bit).
// what a lane needs of an edge: its channels in row 0 of da1, in column 0 of radial
struct EdgeAt {
  const float *da, *rad;
};
template <int L, int LMAX, int FMT, typename V, bool SUMS>
struct NodeRot {
  using T_ = typename Elem<FMT>::type;
  // rot: the current edge's rotation; next: the worker's next edge, staged as this one is used up
  static __device__ __forceinline__ void run(const ZpTables &t, const float *x_s, float *da_s, float *rad_s, int ls,
                                             T_ *out, int64_t plane_bytes, u64 inv, const float *rot, bool live,
                                             const EdgeAt &next, bool more,
                                             V (&acc)[SUMS ? (LMAX + 1) * (LMAX + 1) : 1], Torque &T) {
    if constexpr (L > 0)
      NodeRot<L - 1, LMAX, FMT, V, SUMS>::run(t, x_s, da_s, rad_s, ls, out, plane_bytes, inv, rot, live, next, more, acc, T);
    constexpr int n = 2 * L + 1;
    const int C2 = 2 * t.C;
    const int mm = t.mmax < L ? t.mmax : L;
    if (L > 0) cp_async_wait<LMAX>();    // (degree 0: the caller)
    if (live) {
      V u[n];
#pragma unroll
      for (int j = 0; j < n; ++j) u[j] = load_vec<V>(x_s + (L * L + j) * ls);
      const float *w = rot + t.deg_rot[L];
      const float *dr = da_s + t.deg_row[L] * ls, *gr = rad_s + t.deg_rad[L] * ls;
      T_ *o = out + L * C2;
      V qp, qm = zero_vec<V>(), sp = zero_vec<V>(), sm = zero_vec<V>();
      {
        const V da = load_vec<V>(dr);
        qp = mul4(da, load_vec<V>(gr));
        for_row_plain<n>(w, [&](int j, u64 c) {
          axpy4(sp, c, u[j]);
          if constexpr (SUMS) axpy4(acc[L * L + j], c, qp);
        });
        put4<FMT>(o, plane_bytes, mul4(da, sp), inv);
      }
#pragma unroll 1
      for (int am = 1; am <= mm; ++am) {
        w += 2 * (n + 1);
        dr += 2 * ls;
        gr += ls;
        o += (LMAX + 1 - am) * C2;
        const V rad = load_vec<V>(gr), dp = load_vec<V>(dr - ls), dm = load_vec<V>(dr);
        const V yp = mul4(dp, rad), ym = mul4(dm, rad);
        V ap = zero_vec<V>(), an = zero_vec<V>();
        for_row_plain<n>(w - (n + 1), [&](int j, u64 c) {
          axpy4(ap, c, u[j]);
          if constexpr (SUMS) axpy4(acc[L * L + j], c, yp);
        });
        for_row_plain<n>(w, [&](int j, u64 c) {
          axpy4(an, c, u[j]);
          if constexpr (SUMS) axpy4(acc[L * L + j], c, ym);
        });
        put4<FMT>(o, plane_bytes, mul_add4(dp, ap, dm, an), inv);
        T.own(am, yp, ym, ap, an);
        T.pair(t.couple[L][am - 1], qp, qm, sp, sm, yp, ym, ap, an);
        qp = yp; qm = ym; sp = ap; sm = an;
      }
      if (L > t.mmax) {
        w += 2 * (n + 1);
        V ap = zero_vec<V>(), an = zero_vec<V>();
        for_row_plain<n>(w - (n + 1), [&](int j, u64 c) { axpy4(ap, c, u[j]); });
        for_row_plain<n>(w, [&](int j, u64 c) { axpy4(an, c, u[j]); });
        T.outer(t.couple[L][mm], qp, qm, ap, an);
      }
    }
    if (more) stage_degree<L, LMAX, V, true, true>(t, next.da, C2, next.rad, da_s, rad_s, ls);
    cp_async_commit();                   // (with degree 0 goes the rotation, requested before)
  }
};

struct NodeArgs {
  const float *da1, *radial, *x, *rot;
  const int32_t *row_ptr, *perm_src, *row_ptr_src;
  float *grad_radial, *grad_x;
  float4 *torque;                        // [slots][E]; slot 1 + 2 group + half is written here
  float *cuts;                           // [cut][K][C]: sums of what follows a cut
  int *arrived;
};
constexpr int kNodeQuadMaxL = 4;         // four channels a lane up to here
template <bool PAIR> struct NodeVecOf { using type = F4; };
template <> struct NodeVecOf<true> { using type = F2; };
template <int LMAX> using NodeVec = typename NodeVecOf<(LMAX > kNodeQuadMaxL)>::type;
inline NodeShape node_shape(const ZpTables &t) { return zp_node_shape(t.C, t.lmax <= kNodeQuadMaxL ? 4 : 2); }
// shared memory: x [K][G] vectors | per worker: staged rows [Km + rad_rows][G] vectors, later its sums [K][G] |
// per worker: two rotations [rot_ld]
template <int LMAX, int FMT, bool SUMS>
__global__ void __launch_bounds__(32 * kNodeMaxWarps, (SUMS && LMAX > 2 ? 1 : 2))
node_rotate_in_bwd_kernel(const __grid_constant__ ZpTables t, const NodeCut cut, int64_t E, int G, int quads, const NodeArgs a,
                          const ZpPlanes grad_radial_planes, const ZpScale scale) {
  zp_after_previous();
  using T_ = typename Elem<FMT>::type;
  using V = NodeVec<LMAX>;
  constexpr int K = (LMAX + 1) * (LMAX + 1), VN = VecOf<V>::n;
  extern __shared__ __align__(16) float node_s[];
  const int workers = blockDim.x / G, w = threadIdx.x / G, li = threadIdx.x % G;
  const int ls = G * VN;                                    // floats between two rows
  const int rows = SUMS ? max(t.Km + t.rad_rows, K) : t.Km + t.rad_rows;
  const int c0 = blockIdx.y * quads * VN, mine = min(quads, (t.C - c0) / VN);
  const bool active = li < mine;
  const int c = c0 + li * VN;
  float *x_s = node_s, *stage = node_s + (size_t)K * ls, *da_s = stage + (size_t)w * rows * ls + li * VN;
  float *rad_s = da_s + t.Km * ls;
  float *rot_s = stage + (size_t)workers * rows * ls + (size_t)w * 2 * t.rot_ld;
  const NodeEdges node(blockIdx.x, cut, E, a.row_ptr, a.perm_src, a.row_ptr_src);
  float inv = 1.f;
  if constexpr (FMT == kFmtFp16x2)
    inv = zp_publish_scale(grad_radial_planes, scale, blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0);
  const u64 inv2 = pack2(inv, inv);
  const int64_t plane_bytes = 2 * grad_radial_planes.plane_stride;
  V acc[SUMS ? K : 1];
#pragma unroll
  for (int k = 0; k < (SUMS ? K : 1); ++k) acc[k] = zero_vec<V>();
  if (node.first == node.last) {
    if (SUMS && blockIdx.x < cut.nodes && active)
      for (int k = w; k < K; k += workers) store_vec<V>(a.grad_x + ((size_t)blockIdx.x * K + k) * t.C + c, zero_vec<V>());
    return;
  }
  // with sums the loop has every register in use
  __shared__ __align__(16) unsigned char edges_s[sizeof(NodeEdges)];
  if (SUMS && threadIdx.x == 0) *reinterpret_cast<NodeEdges *>(edges_s) = node;
  if (SUMS) __syncthreads();
  const NodeEdges &edges = SUMS ? *reinterpret_cast<NodeEdges *>(edges_s) : node;

  // (edge -1 reads as edge 0)
  auto column = [&](int i) { return (i < edges.own ? t.C : 0) + c; };
  auto at = [&](int e, int i) {
    const size_t row = max(e, 0);
    return EdgeAt{a.da1 + row * t.Km * 2 * t.C + column(i), a.radial + row * t.R + column(i)};
  };
  auto out_at = [&](int e, int i) {
    const size_t row = max(e, 0);
    if constexpr (FMT == kFmtFp32) return a.grad_radial + row * t.R + column(i);
    else return static_cast<uint16_t *>(grad_radial_planes.base) + row * grad_radial_planes.ld + column(i);
  };
  auto rotation = [&](int64_t e, int buffer) {
    stage_rot(a.rot + (size_t)e * t.rot_ld, rot_s + buffer * t.rot_ld, t.rot_ld, li, G);
  };
  const int i0 = edges.first + w;
  if (active) stage_node<V>(a.x + (size_t)edges.row(cut) * t.K * t.C + c, t.C, K, w, workers, x_s + li * VN, ls);
  int e = edges.edge(i0), e_next = edges.edge(i0 + workers);
  if (e >= 0) rotation(e, 0);
  StageAll<LMAX, LMAX, V, true, true>::run(t, at(e, i0).da, 2 * t.C, at(e, i0).rad, da_s, rad_s, ls, e >= 0 && active);
  cp_async_wait<LMAX>();                 // the node's rows went with degree 0
  __syncthreads();
  for (int i = i0, buffer = 0; i - w < edges.last; i += workers, buffer ^= 1) {      // as often on all lanes
    const int e_after = edges.edge(i + 2 * workers);
    const EdgeAt next = at(e_next, i + workers);
    Torque T{0ull, 0ull, 0ull};
    cp_async_wait<LMAX>();               // degree 0 and the rotation have landed
    __syncwarp();                        // ... the other lanes' part of it, and all are done with the last
    if (e_next >= 0) rotation(e_next, buffer ^ 1);
    NodeRot<LMAX, LMAX, FMT, V, SUMS>::run(t, x_s + li * VN, da_s, rad_s, ls, out_at(e, i), plane_bytes, inv2,
                                     rot_s + buffer * t.rot_ld, e >= 0 && active, next, e_next >= 0 && active,
                                     acc, T);
    float t0 = sum2(T.t0), t1 = sum2(T.t1), t2 = sum2(T.t2);
    for (int o = G / 2; o > 0; o >>= 1) {
      t0 += __shfl_xor_sync(0xffffffffu, t0, o);
      t1 += __shfl_xor_sync(0xffffffffu, t1, o);
      t2 += __shfl_xor_sync(0xffffffffu, t2, o);
    }
    if (li == 0 && e >= 0)
      a.torque[(size_t)(1 + 2 * blockIdx.y + (i < edges.own ? 1 : 0)) * E + e] = make_float4(t0, t1, t2, 0.f);
    e = e_next;
    e_next = e_after;
  }
  cp_async_wait<0>();
  if (!SUMS) return;
  const int n = edges.n;
  if (n == cut.nodes) return;            // left-out slots
  // this lane's place in the rows that the sums go to
  float *const to = (blockIdx.x >= cut.ends() ? a.cuts + (size_t)(blockIdx.x - cut.ends()) * K * t.C
                                            : a.grad_x + (size_t)n * K * t.C) + c0 + li * VN;
  __syncthreads();                       // all are done with their rows: the sums take their place
  float *const sums = stage + li * VN;
#pragma unroll
  for (int k = 0; k < K; ++k) store_vec<V>(sums + ((size_t)w * rows + k) * ls, acc[SUMS ? k : 0]);
  __syncthreads();
  if (active)
    for (int k = w; k < K; k += workers) {
      V s = load_vec<V>(sums + k * ls);
      for (int v = 1; v < workers; ++v) s = add4(s, load_vec<V>(sums + ((size_t)v * rows + k) * ls));
      store_vec<V>(to + (size_t)k * t.C, s);
    }
  const int cut0 = edges.cut0, cut1 = edges.cut1;
  if (cut0 > cut1) return;
  // a cut node: whoever gets done last adds up, in the order of the stretches
  __shared__ int all_here;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
    all_here = atomicAdd(a.arrived + blockIdx.y * kZpNodeCuts + cut0, 1) == cut1 - cut0 + 1;
  __syncthreads();
  if (!all_here || !active) return;
  __threadfence();
  for (int k = w; k < K; k += workers) {
    const size_t at = (size_t)k * t.C + c0 + li * VN;
    float *const gx = a.grad_x + (size_t)n * K * t.C + at;
    for (int v = 0; v < VN; ++v) {
      float s = __ldcg(gx + v);
      for (int i = cut0; i <= cut1; ++i) s += __ldcg(a.cuts + (size_t)(i - 1) * K * t.C + at + v);
      gx[v] = s;
    }
  }
}

}  // namespace

int zp_launch_rotate_grad_out(const zp_plan *p, int64_t first, int64_t N, int64_t E, const float *g, const float *y,
                              const float *env, const float *rot, const int32_t *dst, const int32_t *row_ptr,
                              const ZpPlanes &dy, const ZpScale &scale, float *grad_env,
                              float *torque, cudaStream_t st) {
  if (E == 0) return ZP_OK;
  const ZpTables &t = p->t;
  const NodeShape ns = zp_node_shape(t.C, 4);
  // By node the sums over an edge's channels are one worker's; nodes of fewer than three edges are over before
  // they have paid for their start.  By edge / by node at one, two and three edges a node: lmax 4, C 128, 60 000 edges
  // 363 / 370, 346 / 298 and 336 / 265 us; lmax 6, 20 000 edges 255 / 298, 222 / 225; lmax 2, C 32, 20 000 21 / 42, 20 / 30.
  // At lmax 1 a worker's idle lanes weigh more than the rows of g: 72 of 128 channels, 30 000 edges 19 / 24 us.
  if (ns.groups == 1 && E >= 3 * N && (t.lmax >= 2 || 10 * ns.quads >= 7 * ns.G)) {
    const NodeLaunch nl = zp_node_launch(N, (double)E / (double)N, ns, t, t.Km, 16, 4);
    const NodeCut cut = zp_node_cut(N, E, false, nl.parts);
#define CALL_FMT(LM, FMT)                                                                         \
  {                                                                                               \
    static ZpSmemOptIn opt_in;               /* per instantiation and device */                   \
    if (int rc_ = zp_ensure_smem(node_rotate_grad_out_kernel<LM, FMT>, nl.smem, opt_in)) return rc_; \
    zp_launch(node_rotate_grad_out_kernel<LM, FMT>, dim3(cut.blocks()), 32 * nl.warps, nl.smem, st, t, cut, E, ns.G, ns.quads, \
              g + (size_t)first * t.K * t.C, y, env, rot, row_ptr + first, dy, scale, grad_env, reinterpret_cast<float4 *>(torque));  \
    break;                                                                                        \
  }
#define CALL(LM)                                               \
  switch (zp_plane_format(dy)) {                               \
    case kFmtBf16: CALL_FMT(LM, kFmtBf16)                      \
    case kFmtFp16x2: CALL_FMT(LM, kFmtFp16x2)                  \
    default: CALL_FMT(LM, kFmtBf16x3)                          \
  }
    ZP_DISPATCH_LMAX(t.lmax, CALL)
#undef CALL
#undef CALL_FMT
    ZP_LAUNCH_CHECK("node_rotate_grad_out_kernel");
    return ZP_OK;
  }
  const int Q = t.C / 4;
  if (Q < 1 || Q > kEdgeThreads) return ZP_ERR_UNSUPPORTED;
  const int epb = std::min(kEdgeThreads / Q, kEdgesPerBlock), threads = (epb * Q + 31) / 32 * 32;
  const unsigned grid = (unsigned)zp_ceil_div(E, epb);
  const size_t smem = (size_t)threads * (1 + t.Km) * sizeof(float4) + (size_t)epb * t.rot_ld * sizeof(float2);
#define CALL_FMT(LM, FMT)                                                                         \
  {                                                                                               \
    static ZpSmemOptIn opt_in;               /* per instantiation and device */                   \
    if (int rc_ = zp_ensure_smem(rotate_grad_out_kernel<LM, FMT>, smem, opt_in)) return rc_;      \
    zp_launch(rotate_grad_out_kernel<LM, FMT>, grid, threads, smem, st,                           \
        t, E, epb, g, y, env, rot, dst, dy, scale, grad_env, reinterpret_cast<float4 *>(torque)); \
    break;                                                                                        \
  }
#define CALL(LM)                                               \
  switch (zp_plane_format(dy)) {                               \
    case kFmtBf16: CALL_FMT(LM, kFmtBf16)                      \
    case kFmtFp16x2: CALL_FMT(LM, kFmtFp16x2)                  \
    default: CALL_FMT(LM, kFmtBf16x3)                          \
  }
  ZP_DISPATCH_LMAX(t.lmax, CALL)
#undef CALL
#undef CALL_FMT
  ZP_LAUNCH_CHECK("rotate_grad_out_kernel");
  return ZP_OK;
}

int zp_launch_rotate_in_bwd(const zp_plan *p, int64_t N, int64_t E, const float *da1, const float *radial,
                            const float *x, const int32_t *row_ptr, const int32_t *perm_src,
                            const int32_t *row_ptr_src, const float *rot, float *grad_radial, float *grad_x,
                            float *torque, float *cuts, int *arrived, cudaStream_t st,
                            const ZpPlanes *grad_radial_planes, const ZpScale &scale) {
  const ZpPlanes gp = grad_radial_planes ? *grad_radial_planes : ZpPlanes{nullptr, 0, 0, 0, 0, nullptr};
  const ZpTables &t = p->t;
  if (grad_x ? N == 0 : E == 0) return ZP_OK;
  if (t.C > 256) {
    if (E) return ZP_ERR_UNSUPPORTED;
    ZP_CUDA(cudaMemsetAsync(grad_x, 0, sizeof(float) * (size_t)N * t.K * t.C, st));
    return ZP_OK;
  }
  const bool sums = grad_x != nullptr;
  const NodeShape ns = node_shape(t);
  const int rows = t.Km + t.rad_rows;
  const NodeLaunch nl = zp_node_launch(N * ns.groups, 2.0 * (double)E / (double)N, ns, t,
                                       sums ? std::max(rows, t.K) : rows, sums && t.lmax > 2 ? 8 : 16, sums ? 1 : 4);
  const NodeArgs a{da1, radial, x, rot, row_ptr, perm_src, row_ptr_src, grad_radial, grad_x,
                   reinterpret_cast<float4 *>(torque), cuts, arrived};
  const NodeCut cut = zp_node_cut(N, E, true, nl.parts);
  const dim3 grid(cut.blocks(), (unsigned)ns.groups);
#define CALL_S(LM, FMT, S)                                                                        \
  {                                                                                               \
    static ZpSmemOptIn opt_in;               /* per instantiation and device */                   \
    if (int rc_ = zp_ensure_smem(node_rotate_in_bwd_kernel<LM, FMT, S>, nl.smem, opt_in)) return rc_; \
    zp_launch(node_rotate_in_bwd_kernel<LM, FMT, S>, grid, 32 * nl.warps, nl.smem, st, t, cut, E, ns.G, ns.quads, a, \
              gp, scale);                                                                         \
  }
#define CALL_FMT(LM, FMT)                        \
  {                                              \
    if (sums) CALL_S(LM, FMT, true)              \
    else CALL_S(LM, FMT, false)                  \
    break;                                       \
  }
#define CALL(LM)                                               \
  switch (zp_plane_format(gp)) {                               \
    case kFmtFp32: CALL_FMT(LM, kFmtFp32)                      \
    case kFmtBf16: CALL_FMT(LM, kFmtBf16)                      \
    case kFmtFp16x2: CALL_FMT(LM, kFmtFp16x2)                  \
    default: CALL_FMT(LM, kFmtBf16x3)                          \
  }
  ZP_DISPATCH_LMAX(t.lmax, CALL)
#undef CALL
#undef CALL_FMT
#undef CALL_S
  ZP_LAUNCH_CHECK("node_rotate_in_bwd_kernel");
  return ZP_OK;
}

int zp_node_groups(const ZpTables &t) { return node_shape(t).groups; }
int zp_torque_slots(const ZpTables &t) { return 1 + 2 * zp_node_groups(t); }
int64_t zp_node_cuts_most(int64_t E) { return zp_node_cut(1, E, true, 1).cuts; }
