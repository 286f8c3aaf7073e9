// The VJPs of the per-edge rotate kernels.
//
//   rotate_grad_out      the VJP of rotate_back_scatter (needs y)
//   rotate_in_bwd        the VJP of rotate_in, per-edge node contributions
//
// (autograd through blocks/eso2_ref.py:334-349).  One (edge, channel quad) per thread; see
// zp_rotate.cu for the forward kernels.
#include <algorithm>

#include "zp_rotate.cuh"

namespace {

// ------------------------------------------------------------------------------------------
// per-edge backward kernels: one (edge, channel quad) per thread
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
  __device__ __forceinline__ void own(int m, const F4 &pp, const F4 &pm, const F4 &bp, const F4 &bm) {
    const u64 f = pack2((float)m, (float)m);
    t0 = fma2(f, sub2(dot4(0ull, pp, bm), dot4(0ull, pm, bp)), t0);
  }
  // (m, m + 1): q, s = p and b of m; y, t = those of m + 1
  __device__ __forceinline__ void pair(float c, const F4 &qp, const F4 &qm, const F4 &sp, const F4 &sm,
                                       const F4 &yp, const F4 &ym, const F4 &tp, const F4 &tm) {
    const u64 cc = pack2(c, c);
    t1 = fma2(cc, sub2(dot4(dot4(0ull, qp, tp), qm, tm), dot4(dot4(0ull, yp, sp), ym, sm)), t1);
    t2 = fma2(cc, sub2(dot4(dot4(0ull, ym, sp), qm, tp), dot4(dot4(0ull, qp, tm), yp, sm)), t2);
  }
  // (mmax, mmax + 1): p of the outer row is zero
  __device__ __forceinline__ void outer(float c, const F4 &qp, const F4 &qm, const F4 &tp, const F4 &tm) {
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

// ---- VJP of rotate_in over the 2C message channels -----------------------------------------------
//   a[r]   = sum_j rot[r, j] u[l^2 + j]            (formed again; u = x_src | x_dst half)
//   ga[r]  = da[e, r] * radial
//   grad_radial[e, col] = sum over the +m / -m rows sharing the column of  da[r] * a[r]
//                         (fp32 rows, or operand planes of the radial layer's VJP)
//   du[e, half, l^2 + j] = sum_r rot[r, j] ga[r]   (summed per node afterwards)
//   torque[e] += sums above with p = ga, b = a
template <int FMT> struct Elem { using type = uint16_t; };
template <> struct Elem<kFmtFp32> { using type = float; };

template <int L, int LMAX, int FMT>
struct RotInBwdE {
  using T_ = typename Elem<FMT>::type;
  // da_s, rad_s: this thread's channels of the edge's gradient rows and radial gains; out: its quad
  // in column 0 of grad_radial
  static __device__ __forceinline__ void run(const ZpTables &t, const float *xrow, const float *da_s,
                                             const float *rad_s, int ls, T_ *out, int64_t plane_bytes,
                                             u64 inv, const float2 *rot_s, float *du_row, Torque &T) {
    RotInBwdE<L - 1, LMAX, FMT>::run(t, xrow, da_s, rad_s, ls, out, plane_bytes, inv, rot_s, du_row, T);
    constexpr int n = 2 * L + 1;
    const int C2 = 2 * t.C;
    const int mm = t.mmax < L ? t.mmax : L;
    F4 u[n], du[n];
    const float *xl = xrow + L * L * t.C;
#pragma unroll
    for (int j = 0; j < n; ++j) u[j] = load4(xl + j * t.C);
    const float2 *w = rot_s + t.deg_rot[L];
    const float *dr = da_s + t.deg_row[L] * ls, *gr = rad_s + t.deg_rad[L] * ls;
    T_ *o = out + L * C2;
    cp_async_wait<LMAX - L>();             // what degrees 0..L need has landed
    F4 qp, qm = zero4(), sp = zero4(), sm = zero4();
    {
      const F4 da = load4(dr);
      qp = mul4(da, load4(gr));
      for_row<n>(w, [&](int j, u64 c) {
        axpy4(sp, c, u[j]);
        du[j] = F4{mul2(c, qp.a), mul2(c, qp.b)};
      });
      put4<FMT>(o, plane_bytes, mul4(da, sp), inv);
    }
    // a real loop over |m| (one copy of the body per degree keeps the code in the instruction cache)
#pragma unroll 1
    for (int am = 1; am <= mm; ++am) {
      w += 2 * (n + 1);
      dr += 2 * ls;
      gr += ls;
      o += (LMAX + 1 - am) * C2;
      const F4 rad = load4(gr), dp = load4(dr - ls), dm = load4(dr);
      const F4 yp = mul4(dp, rad), ym = mul4(dm, rad);
      F4 ap = zero4(), an = zero4();
      for_row<n>(w - (n + 1), [&](int j, u64 c) {
        axpy4(ap, c, u[j]);
        axpy4(du[j], c, yp);
      });
      for_row<n>(w, [&](int j, u64 c) {
        axpy4(an, c, u[j]);
        axpy4(du[j], c, ym);
      });
      put4<FMT>(o, plane_bytes, F4{fma2(dp.a, ap.a, mul2(dm.a, an.a)), fma2(dp.b, ap.b, mul2(dm.b, an.b))}, inv);
      T.own(am, yp, ym, ap, an);
      T.pair(t.couple[L][am - 1], qp, qm, sp, sm, yp, ym, ap, an);
      qp = yp; qm = ym; sp = ap; sm = an;
    }
    if (du_row) {                        // no du_both: the caller wants no gradient of x_node
      float *dl = du_row + L * L * t.C;
#pragma unroll
      for (int j = 0; j < n; ++j) store4(dl + j * t.C, du[j]);
    }
    if (L > t.mmax) {
      w += 2 * (n + 1);
      F4 ap = zero4(), an = zero4();
      for_row<n>(w - (n + 1), [&](int j, u64 c) { axpy4(ap, c, u[j]); });
      for_row<n>(w, [&](int j, u64 c) { axpy4(an, c, u[j]); });
      T.outer(t.couple[L][mm], qp, qm, ap, an);
    }
  }
};
template <int LMAX, int FMT>
struct RotInBwdE<-1, LMAX, FMT> {
  static __device__ __forceinline__ void run(const ZpTables &, const float *, const float *,
                                             const float *, int, typename Elem<FMT>::type *, int64_t,
                                             u64, const float2 *, float *, Torque &) {}
};

// du_both [E][2][K][C]: half 0 = contribution to the source node, half 1 = to the destination.
// shared memory: partial sums [blockDim] float4 | da [Km][blockDim] float4 | radial
// [rad_rows][blockDim] float4 | rot [epb][rot_ld] dup.
template <int LMAX, int FMT>
__global__ void __launch_bounds__(kEdgeThreads, (LMAX <= 2 ? 4 : LMAX <= 4 ? 3 : 2))
rotate_in_bwd_kernel(const __grid_constant__ ZpTables t, int64_t E, int epb,
                     const float *__restrict__ da1, const float *__restrict__ radial,
                     const float *__restrict__ x, const int32_t *__restrict__ src,
                     const int32_t *__restrict__ dst, const float *__restrict__ rot,
                     float *__restrict__ grad_radial, const ZpPlanes grad_radial_planes,
                     const ZpScale scale, float *__restrict__ du_both, float4 *__restrict__ torque) {
  zp_after_previous();
  extern __shared__ __align__(16) float4 edge_s[];
  const int ls = 4 * blockDim.x;
  float *da_s = reinterpret_cast<float *>(edge_s + blockDim.x) + 4 * threadIdx.x;
  float *rad_s = da_s + t.Km * ls;
  float2 *rot_s = reinterpret_cast<float2 *>(edge_s + (size_t)blockDim.x * (1 + t.Km + t.rad_rows));
  const int Q = t.C / 2;
  const int64_t e0 = (int64_t)blockIdx.x * epb;
  const int n_e = (int)min((int64_t)epb, E - e0);
  const int le = threadIdx.x / Q, c2 = 4 * (threadIdx.x - le * Q);
  const int64_t e = e0 + le;
  if (le < n_e)
    StageEdge<LMAX, LMAX, true, true>::run(t, da1 + (size_t)e * t.Km * 2 * t.C + c2, 2 * t.C, da_s,
                                           radial + (size_t)e * t.R + c2, rad_s, ls);
  stage_dup(rot + e0 * t.rot_ld, rot_s, t.rot_ld, n_e);
  float inv = 1.f;
  if constexpr (FMT == kFmtFp16x2)
    inv = zp_publish_scale(grad_radial_planes, scale, blockIdx.x == 0 && threadIdx.x == 0);
  __syncthreads();
  float4 sums = make_float4(0.f, 0.f, 0.f, 0.f);
  if (le < n_e) {
    const int half = c2 >= t.C ? 1 : 0;
    const int c = c2 - half * t.C;
    const int64_t node = half ? dst[e] : src[e];
    typename Elem<FMT>::type *out;
    if constexpr (FMT == kFmtFp32) out = grad_radial + (size_t)e * t.R + c2;
    else out = static_cast<uint16_t *>(grad_radial_planes.base) + e * grad_radial_planes.ld + c2;
    Torque T{0ull, 0ull, 0ull};
    RotInBwdE<LMAX, LMAX, FMT>::run(t, x + (size_t)node * t.K * t.C + c, da_s, rad_s, ls, out,
                                    2 * grad_radial_planes.plane_stride, pack2(inv, inv),
                                    rot_s + le * t.rot_ld,
                                    du_both ? du_both + ((size_t)e * 2 + half) * t.K * t.C + c : nullptr, T);
    sums = make_float4(sum2(T.t0), sum2(T.t1), sum2(T.t2), 0.f);
  }
  cp_async_wait<0>();
  reduce_edges(edge_s, sums, Q, n_e, [&](int s, const float4 &v) {
    float4 o = torque[e0 + s];
    o.x += v.x; o.y += v.y; o.z += v.z;
    torque[e0 + s] = o;
  });
}

}  // namespace

int zp_launch_rotate_grad_out(const zp_plan *p, int64_t E, const float *g, const float *y,
                              const float *env, const float *rot, const int32_t *dst,
                              const ZpPlanes &dy, const ZpScale &scale, float *grad_env,
                              float *torque, cudaStream_t st) {
  if (E == 0) return ZP_OK;
  const ZpTables &t = p->t;
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

int zp_launch_rotate_in_bwd(const zp_plan *p, int64_t E, const float *da1, const float *radial,
                            const float *x, const int32_t *src, const int32_t *dst,
                            const float *rot, float *grad_radial, float *du_both, float *torque,
                            cudaStream_t st, const ZpPlanes *grad_radial_planes,
                            const ZpScale &scale) {
  const ZpPlanes gp = grad_radial_planes ? *grad_radial_planes : ZpPlanes{nullptr, 0, 0, 0, 0, nullptr};
  if (E == 0) return ZP_OK;
  const ZpTables &t = p->t;
  const int Q = t.C / 2;
  if (Q < 1 || Q > kEdgeThreads) return ZP_ERR_UNSUPPORTED;
  const int epb = std::min(kEdgeThreads / Q, kEdgesPerBlock), threads = (epb * Q + 31) / 32 * 32;
  const unsigned grid = (unsigned)zp_ceil_div(E, epb);
  const size_t smem = (size_t)threads * (1 + t.Km + t.rad_rows) * sizeof(float4) +
                      (size_t)epb * t.rot_ld * sizeof(float2);
#define CALL_FMT(LM, FMT)                                                                         \
  {                                                                                               \
    static ZpSmemOptIn opt_in;               /* per instantiation and device */                   \
    if (int rc_ = zp_ensure_smem(rotate_in_bwd_kernel<LM, FMT>, smem, opt_in)) return rc_;        \
    zp_launch(rotate_in_bwd_kernel<LM, FMT>, grid, threads, smem, st,                             \
        t, E, epb, da1, radial, x, src, dst, rot, grad_radial, gp, scale, du_both,                \
        reinterpret_cast<float4 *>(torque));                                                      \
    break;                                                                                        \
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
  ZP_LAUNCH_CHECK("rotate_in_bwd_kernel");
  return ZP_OK;
}
