// Per-edge rational Wigner-D rotation and its VJP with respect to the edge vector.
//
// Follows the construction of the reference's blocks/wigner.py:60-160: normalise the edge,
// cos/sin(k beta) from Chebyshev polynomials of y, cos/sin(k alpha) by de Moivre from
// (z, x) / sqrt(x^2 + z^2), then per degree l
//     D_l = Xa(-gamma) J_l Xb(-beta) J_l Xc(-alpha)
// with X(theta) carrying cos on the diagonal and signed sin on the anti-diagonal.  Only the
// rows with |m| <= mmax are formed and they are written straight into the packed m'-major
// layout (the reference's `to_m @ wigner`, blocks/eso2_ref.py:330-331).
//
// Arithmetic in fp64 (a few thousand flops per edge, far below the cost of the SO(2) contraction),
// result rounded once to fp32.  The sparse X factors are applied as two-term updates; only the product
// with J in the middle is dense.  Forward: a block per 32 edges, its warps taking columns.  VJP: a thread
// per edge from the gradient of the entries (zp_wigner_backward), or, in the block, from three torques.
#include "zp_common.cuh"

namespace {

constexpr double kS2Floor = 1e-12;   // blocks/wigner.py:57

template <int LMAX>
struct Frame {
  double v[3];
  double n2_raw, inv_norm, xh, yh, zh, s2_raw, s2, inv_r, r, ca1, sa1;
  double cb[LMAX + 1], sb[LMAX + 1], u[LMAX + 1], ca[LMAX + 1], sa[LMAX + 1];
};

template <int LMAX>
__device__ __forceinline__ void frame_forward(Frame<LMAX> &f, const float *ev) {
  f.v[0] = ev[0]; f.v[1] = ev[1]; f.v[2] = ev[2];
  f.n2_raw = f.v[0] * f.v[0] + f.v[1] * f.v[1] + f.v[2] * f.v[2];
  f.inv_norm = rsqrt(fmax(f.n2_raw, kS2Floor));
  f.xh = f.v[0] * f.inv_norm; f.yh = f.v[1] * f.inv_norm; f.zh = f.v[2] * f.inv_norm;
  f.s2_raw = f.xh * f.xh + f.zh * f.zh;
  f.s2 = fmax(f.s2_raw, kS2Floor);
  f.inv_r = rsqrt(f.s2);
  f.r = f.s2 * f.inv_r;
  f.cb[0] = 1.0; f.u[0] = 1.0; f.sb[0] = 0.0; f.ca[0] = 1.0; f.sa[0] = 0.0;
  f.ca1 = f.zh * f.inv_r; f.sa1 = f.xh * f.inv_r;
  if constexpr (LMAX >= 1) {
    f.cb[1] = f.yh; f.u[1] = 2.0 * f.yh; f.ca[1] = f.ca1; f.sa[1] = f.sa1;
  }
#pragma unroll
  for (int k = 2; k <= LMAX; ++k) {
    f.cb[k] = 2.0 * f.yh * f.cb[k - 1] - f.cb[k - 2];
    f.u[k] = 2.0 * f.yh * f.u[k - 1] - f.u[k - 2];
    f.ca[k] = f.ca1 * f.ca[k - 1] - f.sa1 * f.sa[k - 1];
    f.sa[k] = f.sa1 * f.ca[k - 1] + f.ca1 * f.sa[k - 1];
  }
#pragma unroll
  for (int k = 1; k <= LMAX; ++k) f.sb[k] = f.r * f.u[k - 1];
}

// signed anti-diagonal entry of X(-theta) on row i of the degree-L block (0 on the centre row)
template <int L>
__device__ __forceinline__ double anti(const double *sn, int i) {
  const int f = L - i;
  return f > 0 ? -sn[f] : (f < 0 ? sn[-f] : 0.0);
}

// Column j of the degree-L block: the rows |m| <= rows_m, written through put(i, value).
// frame: cos/sin(k beta), cos/sin(k alpha), cos/sin(k gamma) at frame[(6 * k + which) * 32].
template <int L, typename Put>
__device__ __forceinline__ void block_column(const double *__restrict__ J, const double *frame, int j,
                                             int rows_m, Put put) {
  constexpr int n = 2 * L + 1;
  auto fr = [&](int k, int which) { return frame[(6 * k + which) * 32]; };
  // column j of  Xb J Xc
  const int dj = j > L ? j - L : L - j;
  const double c1 = fr(dj, 2);
  const double s1 = j > L ? -fr(dj, 3) : (j < L ? fr(dj, 3) : 0.0);       // Xc[n-1-j, j]
  double P[n], Nn[n];
#pragma unroll
  for (int i = 0; i < n; ++i) P[i] = J[i * n + j] * c1 + J[i * n + (n - 1 - j)] * s1;
#pragma unroll
  for (int i = 0; i < n; ++i) {
    const int di = i > L ? i - L : L - i;
    const double sb = i < L ? -fr(di, 1) : (i > L ? fr(di, 1) : 0.0);
    Nn[i] = fr(di, 0) * P[i] + sb * P[n - 1 - i];
  }
  // rows |m| <= rows_m of J (Xb J Xc), then the Xa mix of row i with its partner n-1-i
#pragma unroll
  for (int d = 0; d <= L; ++d) {
    if (d > rows_m) break;
    double mp = 0.0, mn = 0.0;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      mp += J[(L + d) * n + k] * Nn[k];
      if (d) mn += J[(L - d) * n + k] * Nn[k];
    }
    if (d == 0) {
      put(L, mp);
    } else {
      const double cg = fr(d, 4), sg = fr(d, 5);
      put(L + d, cg * mp + sg * mn);
      put(L - d, cg * mn - sg * mp);
    }
  }
}

template <int L, int LMAX>
struct ForEachL {
  static __device__ __forceinline__ void bwd(const ZpTables &t, const double *J,
                                             const Frame<LMAX> &f, const double *cg,
                                             const double *sg, const float *g_e, double *dcb,
                                             double *dsb, double *dca, double *dsa);
};
template <int LMAX>
struct ForEachL<-1, LMAX> {
  static __device__ __forceinline__ void bwd(const ZpTables &, const double *,
                                             const Frame<LMAX> &, const double *, const double *,
                                             const float *, double *, double *, double *,
                                             double *) {}
};

// Reverse of block_column: adds column j's cotangents of cos/sin(k beta), cos/sin(k alpha).
template <int L, int LMAX>
__device__ __forceinline__ void column_backward(const ZpTables &t, const double *__restrict__ J,
                                               const Frame<LMAX> &f, const double *cg,
                                               const double *sg, const float *g_e, int j,
                                                double *dcb, double *dsb, double *dca, double *dsa) {
  constexpr int n = 2 * L + 1;
  const int mm = t.mmax < L ? t.mmax : L;
  const int dj = j > L ? j - L : L - j;
  const double c1 = f.ca[dj];
  const double s1 = j > L ? -f.sa[dj] : (j < L ? f.sa[dj] : 0.0);
  double P[n];
#pragma unroll
  for (int i = 0; i < n; ++i) P[i] = J[i * n + j] * c1 + J[i * n + (n - 1 - j)] * s1;
  // G = dL/dD column j (zero outside the kept rows);  dM = Xa^T G
  double G[n], dM[n];
#pragma unroll
  for (int i = 0; i < n; ++i) {
    const int di = i > L ? i - L : L - i;
    G[i] = di <= mm ? (double)g_e[t.rot_off[t.row_of[L][i]] + j] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < n; ++k) {
    const int dk = k > L ? k - L : L - k;
    // Xa[n-1-k, k] is the anti-diagonal entry of row n-1-k
    dM[k] = dk <= mm ? cg[dk] * G[k] + anti<L>(sg, n - 1 - k) * G[n - 1 - k] : 0.0;
  }
  // dN = J^T dM (J symmetric in exact arithmetic; transpose written out regardless)
  double dN[n];
#pragma unroll
  for (int k = 0; k < n; ++k) {
    double acc = 0.0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const int di = i > L ? i - L : L - i;
      if (di <= mm) acc += J[i * n + k] * dM[i];
    }
    dN[k] = acc;
  }
  // N = Xb P:  cotangents of the beta harmonics, and dP = Xb^T dN
  double dP[n];
#pragma unroll
  for (int i = 0; i < n; ++i) {
    const int di = i > L ? i - L : L - i;
    dcb[di] += dN[i] * P[i];
    if (i < L) dsb[di] -= dN[i] * P[n - 1 - i];
    if (i > L) dsb[di] += dN[i] * P[n - 1 - i];
    dP[i] = f.cb[di] * dN[i] + anti<L>(f.sb, n - 1 - i) * dN[n - 1 - i];
  }
  // P = J Xc:  column j of Xc holds cos at row j and the signed sin at row n-1-j
  double acc_c = 0.0, acc_s = 0.0;
#pragma unroll
  for (int i = 0; i < n; ++i) {
    acc_c += J[i * n + j] * dP[i];
    acc_s += J[i * n + (n - 1 - j)] * dP[i];
  }
  dca[dj] += acc_c;
  if (j > L) dsa[dj] -= acc_s;
  if (j < L) dsa[dj] += acc_s;
}

template <int L, int LMAX>
__device__ __forceinline__ void ForEachL<L, LMAX>::bwd(const ZpTables &t, const double *J,
                                                       const Frame<LMAX> &f, const double *cg,
                                                       const double *sg, const float *g_e,
                                                       double *dcb, double *dsb, double *dca,
                                                       double *dsa) {
  ForEachL<L - 1, LMAX>::bwd(t, J, f, cg, sg, g_e, dcb, dsb, dca, dsa);
#pragma unroll 1
  for (int j = 0; j < 2 * L + 1; ++j)
    column_backward<L, LMAX>(t, J + t.jd_off[L], f, cg, sg, g_e, j, dcb, dsb, dca, dsa);
}

template <int L, int LMAX>
struct ColumnOf {
  template <typename Put>
  static __device__ __forceinline__ void run(const ZpTables &t, const double *J, const double *frame,
                                             int l, int j, int extra, Put put) {
    if (l == L) {
      const int rows = t.mmax + extra < L ? t.mmax + extra : L;
      block_column<L>(J + t.jd_off[L], frame, j, rows, put);
    } else {
      ColumnOf<L - 1, LMAX>::run(t, J, frame, l, j, extra, put);
    }
  }
};
template <int LMAX>
struct ColumnOf<-1, LMAX> {
  template <typename Put>
  static __device__ __forceinline__ void run(const ZpTables &, const double *, const double *, int, int,
                                             int, Put) {}
};

// A block turns 32 edges: one warp forms their frames, then every warp takes columns (l, j) of the
// rotation in turn, its lanes being the edges, so all lanes read the same J entries and run the same
// code.  The entries are collected in shared memory and leave as whole rows.  (One thread per edge
// wrote them one by one, 32 sectors per store, and had too few warps to hide the fp64 latency:
// 87 us for 60 000 edges at lmax 4, against 42 us.)  packed: the public layout, else the kernels' own
// with the rows m = +-(mmax + 1).
constexpr int kFwdThreads = 256;
template <int LMAX>
__global__ void __launch_bounds__(kFwdThreads)
wigner_fwd_kernel(const __grid_constant__ ZpTables t, const double *__restrict__ J, int64_t E,
                  const float *__restrict__ ev, const float *__restrict__ cgam,
                  const float *__restrict__ sgam, float *__restrict__ rot, int packed) {
  zp_after_previous();
  extern __shared__ __align__(16) double smem_d[];       // frames [LMAX + 1][6][32] | out [32][ld + 1]
  double *frames = smem_d;
  float *out = reinterpret_cast<float *>(smem_d + (LMAX + 1) * 6 * 32);
  const int ld = packed ? t.nnz_pad : t.rot_ld, lds = ld | 1;
  const int64_t e0 = (int64_t)blockIdx.x * 32;
  const int n_e = (int)min((int64_t)32, E - e0);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (warp == 0) {
    const int64_t e = e0 + min(lane, n_e - 1);
    Frame<LMAX> f;
    frame_forward<LMAX>(f, ev + 3 * e);
#pragma unroll
    for (int k = 0; k <= LMAX; ++k) {
      double *q = frames + 6 * k * 32 + lane;
      q[0] = f.cb[k]; q[32] = f.sb[k]; q[64] = f.ca[k]; q[96] = f.sa[k];
      q[128] = cgam[e * (LMAX + 1) + k];
      q[160] = sgam[e * (LMAX + 1) + k];
    }
  } else {
    for (int i = threadIdx.x - 32; i < 32 * lds; i += kFwdThreads - 32) out[i] = 0.f;   // padding entries
  }
  __syncthreads();
  float *mine = out + lane * lds;
  for (int col = warp; col < t.K; col += kFwdThreads / 32) {
    int l = 0;
    while ((l + 1) * (l + 1) <= col) ++l;
    const int j = col - l * l;
    ColumnOf<LMAX, LMAX>::run(t, J, frames + lane, l, j, packed ? 0 : 1, [&](int i, double v) {
      const int am = i > l ? i - l : l - i;
      int off;
      if (am > t.mmax) off = t.ext_off[l][i > l ? 0 : 1];
      else off = packed ? t.rot_off[t.row_of[l][i]] : t.row_off[t.row_of[l][i]];
      mine[off + j] = (float)v;
    });
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n_e * ld; i += kFwdThreads) {
    const int le = i / ld, k = i - le * ld;
    rot[e0 * ld + i] = out[le * lds + k];
  }
}

// What an edge's cotangents of the harmonics add up to in its vector.
template <int LMAX>
__device__ __forceinline__ void frame_backward(const Frame<LMAX> &f, double *dcb, const double *dsb,
                                               double *dca, double *dsa, float *gev) {
  double du[LMAX + 1];
#pragma unroll
  for (int k = 0; k <= LMAX; ++k) du[k] = 0.0;
  // sin(k beta) = r * U_{k-1}(y)
  double dr = 0.0, dy = 0.0;
#pragma unroll
  for (int k = 1; k <= LMAX; ++k) {
    dr += dsb[k] * f.u[k - 1];
    du[k - 1] += dsb[k] * f.r;
  }
  // Chebyshev recursions, reversed
#pragma unroll
  for (int k = LMAX; k >= 2; --k) {
    dy += 2.0 * (f.cb[k - 1] * dcb[k] + f.u[k - 1] * du[k]);
    dcb[k - 1] += 2.0 * f.yh * dcb[k]; dcb[k - 2] -= dcb[k];
    du[k - 1] += 2.0 * f.yh * du[k];   du[k - 2] -= du[k];
  }
  double dca1 = 0.0, dsa1 = 0.0;
  if constexpr (LMAX >= 1) dy += dcb[1] + 2.0 * du[1];
  // de Moivre recursion, reversed
#pragma unroll
  for (int k = LMAX; k >= 2; --k) {
    dca1 += dca[k] * f.ca[k - 1] + dsa[k] * f.sa[k - 1];
    dsa1 += -dca[k] * f.sa[k - 1] + dsa[k] * f.ca[k - 1];
    dca[k - 1] += dca[k] * f.ca1 + dsa[k] * f.sa1;
    dsa[k - 1] += -dca[k] * f.sa1 + dsa[k] * f.ca1;
  }
  if constexpr (LMAX >= 1) { dca1 += dca[1]; dsa1 += dsa[1]; }

  double dz = dca1 * f.inv_r, dx = dsa1 * f.inv_r;
  const double dinv_r = dca1 * f.zh + dsa1 * f.xh + dr * f.s2;
  double ds2 = dr * f.inv_r - 0.5 * dinv_r * f.inv_r / f.s2;
  if (!(f.s2_raw >= kS2Floor)) ds2 = 0.0;             // clamp_min passes no gradient below the floor
  dx += 2.0 * f.xh * ds2;
  dz += 2.0 * f.zh * ds2;
  const double dinv_norm = dx * f.v[0] + dy * f.v[1] + dz * f.v[2];
  double dn2 = -0.5 * dinv_norm * f.inv_norm / fmax(f.n2_raw, kS2Floor);
  if (!(f.n2_raw >= kS2Floor)) dn2 = 0.0;
  gev[0] = (float)(dx * f.inv_norm + 2.0 * f.v[0] * dn2);
  gev[1] = (float)(dy * f.inv_norm + 2.0 * f.v[1] * dn2);
  gev[2] = (float)(dz * f.inv_norm + 2.0 * f.v[2] * dn2);
}

// VJP of one edge's rotation, step by step through the construction above.  g_e: packed layout.
template <int LMAX>
__device__ __noinline__ void chain_backward(const ZpTables &t, const double *__restrict__ J,
                                            const float *ev, const float *cgam, const float *sgam,
                                            const float *g_e, float *gev) {
  Frame<LMAX> f;
  frame_forward<LMAX>(f, ev);
  double cg[LMAX + 1], sg[LMAX + 1];
  double dcb[LMAX + 1], dsb[LMAX + 1], dca[LMAX + 1], dsa[LMAX + 1];
#pragma unroll
  for (int k = 0; k <= LMAX; ++k) {
    cg[k] = cgam[k];
    sg[k] = sgam[k];
    dcb[k] = dsb[k] = dca[k] = dsa[k] = 0.0;
  }
  ForEachL<LMAX, LMAX>::bwd(t, J, f, cg, sg, g_e, dcb, dsb, dca, dsa);
  frame_backward<LMAX>(f, dcb, dsb, dca, dsa, gev);
}
// The same by a warp, its lanes taking the columns (l, j).
template <int L, int LMAX>
struct ColumnBackward {
  static __device__ __forceinline__ void run(const ZpTables &t, const double *J, const Frame<LMAX> &f,
                                             const double *cg, const double *sg, const float *g_e, int l,
                                             int j, double *dcb, double *dsb, double *dca, double *dsa) {
    if (l == L) column_backward<L, LMAX>(t, J + t.jd_off[L], f, cg, sg, g_e, j, dcb, dsb, dca, dsa);
    else ColumnBackward<L - 1, LMAX>::run(t, J, f, cg, sg, g_e, l, j, dcb, dsb, dca, dsa);
  }
};
template <int LMAX>
struct ColumnBackward<-1, LMAX> {
  static __device__ __forceinline__ void run(const ZpTables &, const double *, const Frame<LMAX> &,
                                             const double *, const double *, const float *, int, int,
                                             double *, double *, double *, double *) {}
};
template <int LMAX>
__device__ __noinline__ void chain_backward_warp(const ZpTables &t, const double *__restrict__ J,
                                                 const float *ev, const float *cgam, const float *sgam,
                                                 const float *g_e, float *gev) {
  const int lane = threadIdx.x % 32;
  Frame<LMAX> f;
  frame_forward<LMAX>(f, ev);
  double cg[LMAX + 1], sg[LMAX + 1];
  double dcb[LMAX + 1], dsb[LMAX + 1], dca[LMAX + 1], dsa[LMAX + 1];
#pragma unroll
  for (int k = 0; k <= LMAX; ++k) {
    cg[k] = cgam[k];
    sg[k] = sgam[k];
    dcb[k] = dsb[k] = dca[k] = dsa[k] = 0.0;
  }
#pragma unroll 1
  for (int col = lane; col < t.K; col += 32) {
    int l = 0;
    while ((l + 1) * (l + 1) <= col) ++l;
    ColumnBackward<LMAX, LMAX>::run(t, J, f, cg, sg, g_e, l, col - l * l, dcb, dsb, dca, dsa);
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k <= LMAX; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dcb[k] += __shfl_xor_sync(0xffffffffu, dcb[k], o);
      dsb[k] += __shfl_xor_sync(0xffffffffu, dsb[k], o);
      dca[k] += __shfl_xor_sync(0xffffffffu, dca[k], o);
      dsa[k] += __shfl_xor_sync(0xffffffffu, dsa[k], o);
    }
  if (lane == 0) frame_backward<LMAX>(f, dcb, dsb, dca, dsa, gev);
}

template <int LMAX>
__global__ void __launch_bounds__(128)
wigner_bwd_kernel(const __grid_constant__ ZpTables t, const double *__restrict__ J, int64_t E,
                  const float *__restrict__ ev, const float *__restrict__ cgam,
                  const float *__restrict__ sgam, const float *__restrict__ grot,
                  float *__restrict__ gev) {
  zp_after_previous();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  chain_backward<LMAX>(t, J, ev + 3 * e, cgam + e * (LMAX + 1), sgam + e * (LMAX + 1),
                       grot + e * t.nnz_pad, gev + 3 * e);
}

// The rotation of an edge frame depends on the edge's direction only, so its VJP needs no more than
// the three derivatives under rotations of the frame, which the kernels that hold the rows form on
// the way (torque; zp_rotate_bwd.cu):  with v = |v| (sin b sin a, cos b, sin b cos a), roll angle g,
//   dL/db = cos g T1 + sin g T2,    dL/da = sin b (sin g T1 - cos g T2) + cos b T0,
//   grad v = ( dL/db e_b + dL/da / sin b  e_a ) / |v|.
// Two kinds of edges have no proper rotation and go through the construction step by step, from the
// gradient of every rotation entry: those along the polar axis (sin^2 b below the floor of the
// construction; a few per atom in a crystal without displacements) and those whose roll-angle
// harmonics are not cos(k g), sin(k g) of one angle, k up to mmax + 1 (rounded to 16 bits, say).
// A block lists its own such edges and its warps form the entries of one each, row by row.  A few of them
// then run the construction by a warp, its lanes taking the columns; from kFewSteps on by a thread each, all
// at the same time.  Forces of 256 fcc atoms (19 968 edges, lmax 4, 2.40 ms): undisplaced 2.49 ms (2.60
// with one lane taking one edge after the other), every edge's harmonics rounded 3.98 (4.70 with a warp
// per edge throughout).
constexpr int kFewSteps = 8;
constexpr double kHarmonicSlack = 4e-6;      // 32 units in the last place of 1: fp32 recurrences pass
template <int LMAX>
__device__ __forceinline__ bool one_angle(const float *cgam, const float *sgam, int top) {
  if constexpr (LMAX == 0) return true;
  const double c1 = cgam[1], s1 = sgam[1];
  double worst = fabs(c1 * c1 + s1 * s1 - 1.0), c = c1, s = s1;
#pragma unroll
  for (int k = 2; k <= LMAX; ++k) {
    const double cn = c1 * c - s1 * s;
    s = s1 * c + c1 * s;
    c = cn;
    if (k <= top) worst = fmax(worst, fmax(fabs(cgam[k] - c), fabs(sgam[k] - s)));
  }
  return worst <= kHarmonicSlack;
}
// The gradient of the 2l + 1 entries of one row, by a warp: unrolled per degree, so that the rows of the
// nodes are requested together.
template <int L>
struct RowEntries {
  static __device__ __forceinline__ void run(int l, int C, int lane, float env, const float *da,
                                             const float *rad, const float *y, const float *xs,
                                             const float *xd, const float *g, float *out) {
    if (l != L) return RowEntries<L - 1>::run(l, C, lane, env, da, rad, y, xs, xd, g, out);
    constexpr int n = 2 * L + 1;
    float in[n];
#pragma unroll
    for (int j = 0; j < n; ++j) in[j] = 0.f;
    for (int c = 4 * lane; c < C; c += 128) {            // channel counts are multiples of 8
      auto at = [&](const float *p) { return *reinterpret_cast<const float4 *>(p + c); };
      auto mul = [](const float4 &u, const float4 &v) { return make_float4(u.x * v.x, u.y * v.y, u.z * v.z, u.w * v.w); };
      auto dot = [](const float4 &u, const float4 &v) { return (u.x * v.x + u.y * v.y) + (u.z * v.z + u.w * v.w); };
      const float4 ps = mul(at(da), at(rad)), pd = mul(at(da + C), at(rad + C));
      const float4 py = mul(at(y), make_float4(env, env, env, env));
      float4 u[n];
      const float4 *const p[3] = {&ps, &pd, &py};
      const float *const rows[3] = {xs, xd, g};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int j = 0; j < n; ++j) u[j] = at(rows[k] + (L * L + j) * C);
#pragma unroll
        for (int j = 0; j < n; ++j) in[j] += dot(*p[k], u[j]);
      }
    }
#pragma unroll
    for (int k = 16; k > 0; k >>= 1)
#pragma unroll
      for (int j = 0; j < n; ++j) in[j] += __shfl_xor_sync(0xffffffffu, in[j], k);
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < n; ++j) out[j] = in[j];
    }
  }
};
template <>
struct RowEntries<-1> {
  static __device__ __forceinline__ void run(int, int, int, float, const float *, const float *, const float *,
                                             const float *, const float *, const float *, float *) {}
};
template <int LMAX>
__global__ void __launch_bounds__(128)
edge_vec_grad_kernel(const __grid_constant__ ZpTables t, const double *__restrict__ J, int64_t E,
                     const float *__restrict__ ev, const float *__restrict__ cgam,
                     const float *__restrict__ sgam, const float4 *__restrict__ torque, int slots,
                     const ZpTorqueArgs a, float *__restrict__ gev) {
  zp_after_previous();
  __shared__ int steps[128], found[4];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int64_t e0 = (int64_t)blockIdx.x * 128, e = e0 + threadIdx.x;
  bool step = false;
  if (e < E) {
    const double x = ev[3 * e], y = ev[3 * e + 1], z = ev[3 * e + 2];
    const double n2 = x * x + y * y + z * z;
    const double inv = rsqrt(fmax(n2, kS2Floor));
    const double xh = x * inv, yh = y * inv, zh = z * inv, s2 = xh * xh + zh * zh;
    const int top = t.mmax + 1;
    step = LMAX >= 1 && !(n2 >= kS2Floor && s2 >= kS2Floor &&
                          one_angle<LMAX>(cgam + e * (LMAX + 1), sgam + e * (LMAX + 1), top));
    if (!step) {
      double gx = 0.0, gy = 0.0, gz = 0.0;
      if constexpr (LMAX >= 1) {
        float4 T = torque[e];
        for (int s = 1; s < slots; ++s) {
          const float4 more = torque[s * E + e];
          T.x += more.x; T.y += more.y; T.z += more.z;
        }
        const double inv_r = rsqrt(s2), r = s2 * inv_r, ca = zh * inv_r, sa = xh * inv_r;
        const double c1 = cgam[e * (LMAX + 1) + 1], s1 = sgam[e * (LMAX + 1) + 1];
        const double gb = c1 * T.y + s1 * T.z, ga = s1 * T.y - c1 * T.z + yh * inv_r * T.x;
        gx = inv * (gb * yh * sa + ga * ca);
        gy = -inv * gb * r;
        gz = inv * (gb * yh * ca - ga * sa);
      }
      gev[3 * e] = (float)gx;
      gev[3 * e + 1] = (float)gy;
      gev[3 * e + 2] = (float)gz;
    }
  }
  const int total = __syncthreads_count(step);
  if (total == 0) return;
  const unsigned mine = __ballot_sync(0xffffffffu, step);
  if (lane == 0) found[warp] = __popc(mine);
  __syncthreads();
  int before = __popc(mine & ((1u << lane) - 1u));
  for (int w = 0; w < warp; ++w) before += found[w];
  if (step) steps[before] = threadIdx.x;
  __syncthreads();
  const int C = t.C, C2 = 2 * t.C;
  for (int q = warp; q < total; q += 4) {
    const int64_t i = e0 + steps[q];
    const float *xs = a.x + (size_t)a.src[i] * t.K * C, *xd = a.x + (size_t)a.dst[i] * t.K * C;
    const float *g = a.g_out + (size_t)a.dst[i] * t.K * C;
    float *entries = a.entries + (size_t)i * t.nnz_pad;
    const float env = a.env[i];
    for (int r = 0; r < t.Km; ++r) {
      const int l = t.row_l[r], m = t.row_m[r], am = m < 0 ? -m : m;
      RowEntries<LMAX>::run(l, C, lane, env, a.da1 + ((size_t)i * t.Km + r) * C2,
                            a.radial + (size_t)i * t.R + t.rad_off[am] + (l - am) * C2,
                            a.y + ((size_t)i * t.Km + r) * C, xs, xd, g, entries + t.rot_off[r]);
    }
    if (total <= kFewSteps) {
      __syncwarp();
      chain_backward_warp<LMAX>(t, J, ev + 3 * i, cgam + i * (LMAX + 1), sgam + i * (LMAX + 1), entries, gev + 3 * i);
    }
  }
  if (total <= kFewSteps) return;
  __syncthreads();
  if (step)
    chain_backward<LMAX>(t, J, ev + 3 * e, cgam + e * (LMAX + 1), sgam + e * (LMAX + 1),
                         a.entries + (size_t)e * t.nnz_pad, gev + 3 * e);
}

}  // namespace

int zp_launch_wigner_fwd(const zp_plan *p, int64_t E, const float *ev, const float *cg,
                         const float *sg, float *rot, int packed, cudaStream_t st) {
  if (E == 0) return ZP_OK;
  const unsigned grid = (unsigned)zp_ceil_div(E, 32);
  const int ld = packed ? p->t.nnz_pad : p->t.rot_ld;
  const size_t smem = (size_t)(p->t.lmax + 1) * 6 * 32 * sizeof(double) + (size_t)32 * (ld | 1) * sizeof(float);
#define CALL(LM)                                                                                  \
  {                                                                                               \
    static ZpSmemOptIn opt_in;                                                                    \
    if (int rc_ = zp_ensure_smem(wigner_fwd_kernel<LM>, smem, opt_in)) return rc_;                \
    zp_launch(wigner_fwd_kernel<LM>, grid, kFwdThreads, smem, st, p->t,                             \
              p->jd_dev, E, ev, cg, sg, rot, packed);                                               \
  }
  ZP_DISPATCH_LMAX(p->t.lmax, CALL)
#undef CALL
  ZP_LAUNCH_CHECK("wigner_fwd_kernel");
  return ZP_OK;
}

int zp_launch_wigner_bwd(const zp_plan *p, int64_t E, const float *ev, const float *cg,
                         const float *sg, const float *grot, float *gev, cudaStream_t st) {
  if (E == 0) return ZP_OK;
  const dim3 grid((unsigned)zp_ceil_div(E, 128)), block(128);
#define CALL(LM) \
  zp_launch(wigner_bwd_kernel<LM>, grid, block, 0, st, p->t, p->jd_dev, E, ev, cg, sg, grot, gev);
  ZP_DISPATCH_LMAX(p->t.lmax, CALL)
#undef CALL
  ZP_LAUNCH_CHECK("wigner_bwd_kernel");
  return ZP_OK;
}

int zp_launch_edge_vec_grad(const zp_plan *p, int64_t E, const float *ev, const float *cg,
                            const float *sg, const float *torque, int slots, const ZpTorqueArgs &a, float *gev,
                            cudaStream_t st) {
  if (E == 0) return ZP_OK;
  const dim3 grid((unsigned)zp_ceil_div(E, 128)), block(128);
#define CALL(LM)                                                                                  \
  zp_launch(edge_vec_grad_kernel<LM>, grid, block, 0, st, p->t, p->jd_dev, E, ev, cg, sg,             \
                                                      reinterpret_cast<const float4 *>(torque), slots, a, gev)
  ZP_DISPATCH_LMAX(p->t.lmax, CALL)
#undef CALL
  ZP_LAUNCH_CHECK("edge_vec_grad_kernel");
  return ZP_OK;
}
