// LayerNorm followed by SiLU, forward and backward, for the hidden layers of the radial MLP
// (reference blocks/eso2_ref.py:170-180: Linear, LayerNorm, SiLU, Linear, LayerNorm, SiLU, Linear).
//
//   forward   z = (x - mean) * rstd;  u = z * gamma + beta;  y = u * sigmoid(u)
//   backward  du = dy * s * (1 + u * (1 - s)),  s = sigmoid(u)
//             dgamma = sum_rows du * z,  dbeta = sum_rows du
//             dz = du * gamma;  dx = rstd * (dz - mean(dz) - z * mean(dz * z))
//
// One warp owns a row (width <= 1024, a multiple of 4; lane i holds columns 4i..4i+3 of every
// 128-column group).  Rows are streamed once; mean and rstd are saved by the forward.  Both
// directions are bound by HBM latency: a row is 512 bytes per warp and array, and two dozen warps of
// them do not fill the pipe.  So a warp has its next row on the way while it works on one (up to 256
// columns; wider rows are enough by themselves), and no more blocks are launched than are resident.
// 264 000 rows of 128: forward 85 -> 74 us, backward without parameter gradients
// 140 -> 85 (a third of it was two blocks per SM), with them 190 -> 132 for 384 000 rows in one plane.  The
// parameter gradients are reduced in a fixed order: every lane sums its columns over the rows of
// its warp, the warps of a block are added in warp order through shared memory, each block writes
// one partial row, and a second kernel adds the partial rows in block order.
#include <algorithm>

#include "zp_common.cuh"
#include "zippel_b200.h"

namespace {

constexpr int kWarps = 8;
constexpr int kMaxGroups = 8;              // 128-column groups per row: width <= 1024

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// a lane's columns of row r; zeros past the end of the row or the last row
template <int G>
__device__ __forceinline__ void load_row(float4 (&v)[G], const float *__restrict__ x, int64_t r,
                                         int64_t rows, int width, int lane) {
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int c = 128 * i + 4 * lane;
    v[i] = r < rows && c < width ? *reinterpret_cast<const float4 *>(x + (size_t)r * width + c)
                                 : make_float4(0, 0, 0, 0);
  }
}

template <int G>
__global__ void __launch_bounds__(32 * kWarps)
ln_silu_fwd_kernel(int64_t rows, int width, const float *__restrict__ x,
                   const float *__restrict__ gamma, const float *__restrict__ beta, float eps,
                   float *__restrict__ y, const ZpPlanes yp, const ZpScale scale,
                   float *__restrict__ mean_out, float *__restrict__ rstd_out, float *rstd_max) {
  zp_after_previous();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const float inv = yp.planes ? zp_publish_scale(yp, scale, blockIdx.x == 0 && threadIdx.x == 0) : 1.f;
  float seen = 0.f;
  float4 g[G], b[G];
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int c = 128 * i + 4 * lane;
    g[i] = c < width ? *reinterpret_cast<const float4 *>(gamma + c) : make_float4(0, 0, 0, 0);
    b[i] = c < width ? *reinterpret_cast<const float4 *>(beta + c) : make_float4(0, 0, 0, 0);
  }
  const float inv_w = 1.f / (float)width;
  const int64_t step = (int64_t)gridDim.x * kWarps, first = (int64_t)blockIdx.x * kWarps + warp;
  constexpr bool kAhead = G <= 2;
  float4 next[G];
  if (kAhead) load_row(next, x, first, rows, width, lane);
  for (int64_t r = first; r < rows; r += step) {
    float4 v[G];
    if (kAhead) {
#pragma unroll
      for (int i = 0; i < G; ++i) v[i] = next[i];
      load_row(next, x, r + step, rows, width, lane);
    } else {
      load_row(v, x, r, rows, width, lane);
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < G; ++i) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    const float mean = warp_sum(s) * inv_w;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int c = 128 * i + 4 * lane;
      if (c < width) {
        const float a0 = v[i].x - mean, a1 = v[i].y - mean, a2 = v[i].z - mean, a3 = v[i].w - mean;
        q += (a0 * a0 + a1 * a1) + (a2 * a2 + a3 * a3);
      }
    }
    const float rstd = rsqrtf(warp_sum(q) * inv_w + eps);
    seen = fmaxf(seen, rstd);
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int c = 128 * i + 4 * lane;
      if (c < width) {
        float4 o;
        float u;
        u = (v[i].x - mean) * rstd * g[i].x + b[i].x; o.x = u / (1.f + expf(-u));
        u = (v[i].y - mean) * rstd * g[i].y + b[i].y; o.y = u / (1.f + expf(-u));
        u = (v[i].z - mean) * rstd * g[i].z + b[i].z; o.z = u / (1.f + expf(-u));
        u = (v[i].w - mean) * rstd * g[i].w + b[i].w; o.w = u / (1.f + expf(-u));
        if (yp.planes) {
          const float ov[4] = {o.x, o.y, o.z, o.w};
          zp_store_planes<4>(yp, r * yp.ld + c, ov, inv);
        } else {
          *reinterpret_cast<float4 *>(y + (size_t)r * width + c) = o;
        }
      } else if (yp.planes && c < yp.ld) {         // zero padding up to the row stride
        const float zero[4] = {0.f, 0.f, 0.f, 0.f};
        zp_store_planes<4>(yp, r * yp.ld + c, zero, 1.f);
      }
    }
    if (lane == 0) { mean_out[r] = mean; rstd_out[r] = rstd; }
  }
  if (rstd_max && lane == 0 && seen > *reinterpret_cast<volatile float *>(rstd_max))
    zp_atomic_absmax(rstd_max, seen);
}

__device__ __forceinline__ void bwd_elem(float xv, float mean, float rstd, float g, float b,
                                         float dyv, float &z, float &du) {
  z = (xv - mean) * rstd;
  const float u = z * g + b;
  const float s = 1.f / (1.f + expf(-u));
  du = dyv * s * (1.f + u * (1.f - s));
}

// NP: partial rows per block, 2 = {dgamma, dbeta}, 3 = those and the column sums of dx (the bias
// gradient of the dense layer in front), 0 = no parameter gradients
template <int G, int NP>
__global__ void __launch_bounds__(32 * kWarps)
ln_silu_bwd_kernel(int64_t rows, int width, const float *__restrict__ x,
                   const float *__restrict__ gamma, const float *__restrict__ beta,
                   const float *__restrict__ mean_in, const float *__restrict__ rstd_in,
                   const float *__restrict__ dy, float *__restrict__ dx, const ZpPlanes dxp,
                   const ZpScale scale, float *__restrict__ partial) {
  zp_after_previous();   // [gridDim.x][NP][width]
  extern __shared__ float red[];                              // [kWarps][NP][width]
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const float inv = dxp.planes ? zp_publish_scale(dxp, scale, blockIdx.x == 0 && threadIdx.x == 0) : 1.f;
  float4 g[G], b[G], dg[G], db[G], dd[G];
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int c = 128 * i + 4 * lane;
    g[i] = c < width ? *reinterpret_cast<const float4 *>(gamma + c) : make_float4(0, 0, 0, 0);
    b[i] = c < width ? *reinterpret_cast<const float4 *>(beta + c) : make_float4(0, 0, 0, 0);
    dg[i] = make_float4(0, 0, 0, 0);
    db[i] = make_float4(0, 0, 0, 0);
    dd[i] = make_float4(0, 0, 0, 0);
  }
  const float inv_w = 1.f / (float)width;
  const int64_t step = (int64_t)gridDim.x * kWarps, first = (int64_t)blockIdx.x * kWarps + warp;
  constexpr bool kAhead = G <= 2;
  float4 next_x[G], next_dy[G];
  float next_mean = 0.f, next_rstd = 0.f;
  auto load = [&](int64_t r) {
    load_row(next_x, x, r, rows, width, lane);
    load_row(next_dy, dy, r, rows, width, lane);
    next_mean = r < rows ? mean_in[r] : 0.f;
    next_rstd = r < rows ? rstd_in[r] : 0.f;
  };
  if (kAhead) load(first);
  for (int64_t r = first; r < rows; r += step) {
    if (!kAhead) load(r);
    float4 x_row[G], dy_row[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      x_row[i] = next_x[i];
      dy_row[i] = next_dy[i];
    }
    const float mean = next_mean, rstd = next_rstd;
    if (kAhead) load(r + step);
    float4 z[G], dz[G];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int c = 128 * i + 4 * lane;
      z[i] = make_float4(0, 0, 0, 0);
      dz[i] = make_float4(0, 0, 0, 0);
      if (c < width) {
        const float4 xv = x_row[i], dv = dy_row[i];
        float du;
        bwd_elem(xv.x, mean, rstd, g[i].x, b[i].x, dv.x, z[i].x, du);
        dg[i].x += du * z[i].x; db[i].x += du; dz[i].x = du * g[i].x;
        bwd_elem(xv.y, mean, rstd, g[i].y, b[i].y, dv.y, z[i].y, du);
        dg[i].y += du * z[i].y; db[i].y += du; dz[i].y = du * g[i].y;
        bwd_elem(xv.z, mean, rstd, g[i].z, b[i].z, dv.z, z[i].z, du);
        dg[i].z += du * z[i].z; db[i].z += du; dz[i].z = du * g[i].z;
        bwd_elem(xv.w, mean, rstd, g[i].w, b[i].w, dv.w, z[i].w, du);
        dg[i].w += du * z[i].w; db[i].w += du; dz[i].w = du * g[i].w;
        s1 += (dz[i].x + dz[i].y) + (dz[i].z + dz[i].w);
        s2 += (dz[i].x * z[i].x + dz[i].y * z[i].y) + (dz[i].z * z[i].z + dz[i].w * z[i].w);
      }
    }
    const float m1 = warp_sum(s1) * inv_w, m2 = warp_sum(s2) * inv_w;
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int c = 128 * i + 4 * lane;
      if (c < width) {
        float4 o;
        o.x = rstd * (dz[i].x - m1 - z[i].x * m2);
        o.y = rstd * (dz[i].y - m1 - z[i].y * m2);
        o.z = rstd * (dz[i].z - m1 - z[i].z * m2);
        o.w = rstd * (dz[i].w - m1 - z[i].w * m2);
        if (NP == 3) { dd[i].x += o.x; dd[i].y += o.y; dd[i].z += o.z; dd[i].w += o.w; }
        if (dxp.planes) {
          const float ov[4] = {o.x, o.y, o.z, o.w};
          zp_store_planes<4>(dxp, r * dxp.ld + c, ov, inv);
        } else {
          *reinterpret_cast<float4 *>(dx + (size_t)r * width + c) = o;
        }
      } else if (dxp.planes && c < dxp.ld) {
        const float zero[4] = {0.f, 0.f, 0.f, 0.f};
        zp_store_planes<4>(dxp, r * dxp.ld + c, zero, 1.f);
      }
    }
  }
  if constexpr (NP != 0) {
  // block partial of (dgamma, dbeta): warps added in warp order
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int c = 128 * i + 4 * lane;
    if (c < width) {
      *reinterpret_cast<float4 *>(red + (size_t)(warp * NP + 0) * width + c) = dg[i];
      *reinterpret_cast<float4 *>(red + (size_t)(warp * NP + 1) * width + c) = db[i];
      if (NP == 3) *reinterpret_cast<float4 *>(red + (size_t)(warp * NP + 2) * width + c) = dd[i];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < NP * width; i += blockDim.x) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s += red[(size_t)w * NP * width + i];
    partial[(size_t)blockIdx.x * NP * width + i] = s;
  }
  }
}

int check_shape(int64_t rows, int width) {
  if (rows < 0 || width < 4 || width > 128 * kMaxGroups || (width % 4)) return ZP_ERR_UNSUPPORTED;
  return ZP_OK;
}

#define ZP_DISPATCH_GROUPS(groups, CALL) \
  switch (groups) {                      \
    case 1: { CALL(1); break; }          \
    case 2: { CALL(2); break; }          \
    case 3: case 4: { CALL(4); break; }  \
    default: { CALL(8); break; }         \
  }

}  // namespace

int zp_launch_ln_silu_fwd(int64_t rows, int width, const float *x, const float *gamma,
                          const float *beta, float eps, float *y, const ZpPlanes *y_planes,
                          const ZpScale &scale, float *mean, float *rstd, float *rstd_max,
                          cudaStream_t st) {
  if (rows == 0) return ZP_OK;
  const ZpPlanes yp = y_planes ? *y_planes : ZpPlanes{nullptr, 0, 0, 0, 0, nullptr};
  const int groups = (width + 127) / 128;
  const unsigned grid = (unsigned)std::min<int64_t>(zp_ceil_div(rows, kWarps), 148 * 4);
#define CALL(G)                                                                                   \
  zp_launch(ln_silu_fwd_kernel<G>, grid, 32 * kWarps, 0, st, rows, width, x, gamma, beta, eps, y, yp, scale, \
                                                      mean, rstd, rstd_max)
  ZP_DISPATCH_GROUPS(groups, CALL);
#undef CALL
  ZP_LAUNCH_CHECK("ln_silu_fwd_kernel");
  return ZP_OK;
}

int zp_launch_ln_silu_bwd(int64_t rows, int width, const float *x, const float *gamma,
                          const float *beta, const float *mean, const float *rstd, const float *dy,
                          float *dx, const ZpPlanes *dx_planes, const ZpScale &scale,
                          float *dgamma, float *dbeta, float *dbias, float *partial,
                          ZpFinalList &list, cudaStream_t st) {
  if (rows == 0) return ZP_OK;
  const ZpPlanes dxp = dx_planes ? *dx_planes : ZpPlanes{nullptr, 0, 0, 0, 0, nullptr};
  const int groups = (width + 127) / 128;
  const int np = !dgamma ? 0 : dbias ? 3 : 2;
  const int blocks = (int)std::min<int64_t>(zp_ceil_div(rows, kWarps), np ? ZP_LN_PARTIALS : 148 * 4);
  const size_t smem = sizeof(float) * kWarps * np * (size_t)width;     // <= 96 KB
#define CALL_NP(G, NP)                                                                          \
  do {                                                                                          \
    static ZpSmemOptIn opt_in;                                                                  \
    if (int rc_ = zp_ensure_smem(ln_silu_bwd_kernel<G, NP>, smem, opt_in)) return rc_;          \
    zp_launch(ln_silu_bwd_kernel<G, NP>, blocks, 32 * kWarps, smem, st, \
        rows, width, x, gamma, beta, mean, rstd, dy, dx, dxp, scale, partial);                  \
  } while (0)
#define CALL(G)                      \
  do {                               \
    if (np == 3) CALL_NP(G, 3);      \
    else if (np == 2) CALL_NP(G, 2); \
    else CALL_NP(G, 0);              \
  } while (0)
  ZP_DISPATCH_GROUPS(groups, CALL);
#undef CALL
#undef CALL_NP
  ZP_LAUNCH_CHECK("ln_silu_bwd_kernel");
  float *const dst[3] = {dgamma, dbeta, dbias};
  for (int k = 0; k < np; ++k)
    list.add(partial + (size_t)k * width, dst[k], (int64_t)np * width, 1, width, blocks,
             ZP_FIN_COLUMN);
  return ZP_OK;
}

extern "C" {

size_t zp_layernorm_work_bytes(int width) {
  return sizeof(float) * (size_t)ZP_LN_PARTIALS * 2 * (size_t)(width > 0 ? width : 0);
}

int zp_layernorm_silu_forward(int64_t rows, int width, const float *x, const float *gamma,
                              const float *beta, float eps, float *y, float *mean, float *rstd,
                              void *stream) {
  int rc = check_shape(rows, width);
  if (rc) return rc;
  if (rows == 0) return ZP_OK;
  if (!x || !gamma || !beta || !y || !mean || !rstd) return ZP_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  return zp_launch_ln_silu_fwd(rows, width, x, gamma, beta, eps, y, nullptr, ZpScale{}, mean, rstd,
                               nullptr, st);
}

int zp_layernorm_silu_backward(int64_t rows, int width, const float *x, const float *gamma,
                               const float *beta, const float *mean, const float *rstd,
                               const float *dy, float *dx, float *dgamma, float *dbeta,
                               void *work, size_t work_bytes, void *stream) {
  int rc = check_shape(rows, width);
  if (rc) return rc;
  if (!dgamma || !dbeta) return ZP_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (rows == 0) {
    ZP_CUDA(cudaMemsetAsync(dgamma, 0, sizeof(float) * width, st));
    ZP_CUDA(cudaMemsetAsync(dbeta, 0, sizeof(float) * width, st));
    return ZP_OK;
  }
  if (!x || !gamma || !beta || !mean || !rstd || !dy || !dx || !work) return ZP_ERR_INVALID_ARG;
  if (work_bytes < zp_layernorm_work_bytes(width)) return ZP_ERR_WORKSPACE;
  ZpFinalList list;
  if ((rc = zp_launch_ln_silu_bwd(rows, width, x, gamma, beta, mean, rstd, dy, dx, nullptr, ZpScale{},
                                  dgamma, dbeta, nullptr, static_cast<float *>(work), list, st)))
    return rc;
  return zp_launch_finalize(list, st);
}

}  // extern "C"
