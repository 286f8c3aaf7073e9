// Per-edge front end of the block: geometry, Gaussian distance basis, element embeddings,
// envelope, and the re-ordering of the per-edge inputs into the destination-sorted order, in one
// pass; and its VJP (position and embedding gradients) with fixed-order node sums.
//
//   forward (reference blocks/eso2_ref.py:320-327, :164-168, :242-246)
//     v      = pos[dst] - pos[src] + shift                     edge_vec [E,3]
//     d      = sqrt(max(|v|^2, 1e-24))
//     x_edge = [ exp(coeff * (d - offset_b)^2)  |  emb[Z[src]]  |  emb[Z[dst]] ]      [E, NB + 2 EC]
//     env    = 1 + s^p (a + s (b + c s)) for s = d / cutoff < 1, else 0
//     cos/sin gamma rows copied to the sorted order
//   backward
//     d_d    = sum_b gx[b] gauss_b 2 coeff (d - offset_b)  +  g_env env'(s) / cutoff
//     g_v    = g_edge_vec + d_d v / d                          (0 through the clamp)
//     g_pos[n] = sum_{e into n} g_v[e] - sum_{e out of n} g_v[e]          (fixed order, no atomics)
//     g_emb[z] = sum over atoms n of element z, in index order, of
//                ( sum_{e out of n} gx[e, src part] + sum_{e into n} gx[e, dst part] )
//
// One warp per edge in the forward (lanes run over basis functions / channels), or eight edges.
#include "zp_common.cuh"
#include "zippel_b200.h"

namespace {

constexpr int kWarps = 8;

__device__ __forceinline__ float ipow(float s, int p) {
  float r = 1.f;
  for (int i = 0; i < p; ++i) r *= s;
  return r;
}

struct EnvCoef {
  float a, b, c;
  int p;
};
__host__ __device__ inline EnvCoef env_coef(int p) {
  EnvCoef k;
  k.p = p;
  k.a = -(float)((p + 1) * (p + 2)) / 2.f;
  k.b = (float)(p * (p + 2));
  k.c = -(float)(p * (p + 1)) / 2.f;
  return k;
}

__global__ void __launch_bounds__(32 * kWarps)
edge_features_fwd_kernel(int64_t E, zp_front_config cfg, const float *__restrict__ pos,
                         const float *__restrict__ shifts, const int64_t *__restrict__ z,
                         const float *__restrict__ emb, const float *__restrict__ offsets,
                         const float *__restrict__ cos_g, const float *__restrict__ sin_g,
                         const int32_t *__restrict__ perm, const int32_t *__restrict__ src,
                         const int32_t *__restrict__ dst, float *__restrict__ edge_vec,
                         float *__restrict__ dist_out, float *__restrict__ x_edge,
                         const ZpPlanes xp, const ZpScale scale, float *__restrict__ env_out, float *__restrict__ cos_s,
                         float *__restrict__ sin_s) {
  zp_after_previous();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int64_t e = (int64_t)blockIdx.x * kWarps + warp;
  const float inv = xp.planes ? zp_publish_scale(xp, scale, blockIdx.x == 0 && threadIdx.x == 0) : 1.f;
  if (e >= E) return;
  const int64_t o = perm[e], i = src[e], j = dst[e];
  const float vx = pos[3 * j] - pos[3 * i] + shifts[3 * o];
  const float vy = pos[3 * j + 1] - pos[3 * i + 1] + shifts[3 * o + 1];
  const float vz = pos[3 * j + 2] - pos[3 * i + 2] + shifts[3 * o + 2];
  const float d = sqrtf(fmaxf((vx * vx + vy * vy) + vz * vz, 1e-24f));
  const int NB = cfg.num_basis, EC = cfg.edge_channels, W = NB + 2 * EC;
  // element numbers come from the caller: one outside the table never becomes an address (it is
  // clamped to the nearest row; the Python layer rejects such input before it gets here, as
  // nn.Embedding does in the reference)
  const int64_t zi = min(max(z[i], (int64_t)0), (int64_t)cfg.n_elements - 1);
  const int64_t zj = min(max(z[j], (int64_t)0), (int64_t)cfg.n_elements - 1);
  const float *es = emb + (size_t)zi * EC, *ed = emb + (size_t)zj * EC;
  if (xp.planes) {
    // operand planes of the radial MLP's first layer, a quad of columns per lane; a quad may
    // straddle the parts of the row (num_basis need not be a multiple of 4), and the columns up
    // to the row stride are zero
    for (int c = 4 * lane; c < xp.ld; c += 128) {
      float v[4];
      if (c >= NB && (NB & 3) == 0 && c < W) {
        const float4 q = *reinterpret_cast<const float4 *>(c < NB + EC ? es + (c - NB) : ed + (c - NB - EC));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int b = c + k;
          if (b < NB) {
            const float t = d - offsets[b];
            v[k] = expf(cfg.gauss_coeff * t * t);
          } else {
            v[k] = b < NB + EC ? es[b - NB] : b < W ? ed[b - NB - EC] : 0.f;
          }
        }
      }
      zp_store_planes<4>(xp, e * xp.ld + c, v, inv);
    }
  } else {
    float *row = x_edge + (size_t)e * W;
    for (int b = lane; b < NB; b += 32) {
      const float t = d - offsets[b];
      row[b] = expf(cfg.gauss_coeff * t * t);
    }
    for (int c = lane; c < EC / 4; c += 32) {
      const float4 a = reinterpret_cast<const float4 *>(es)[c], b = reinterpret_cast<const float4 *>(ed)[c];
      float *ps = row + NB + 4 * c, *pd = row + NB + EC + 4 * c;
      ps[0] = a.x; ps[1] = a.y; ps[2] = a.z; ps[3] = a.w;        // NB need not be a multiple of 4
      pd[0] = b.x; pd[1] = b.y; pd[2] = b.z; pd[3] = b.w;
    }
  }
  const int nl = cfg.lmax + 1;
  for (int k = lane; k < nl; k += 32) {
    cos_s[e * nl + k] = cos_g[o * nl + k];
    sin_s[e * nl + k] = sin_g[o * nl + k];
  }
  if (lane == 0) {
    edge_vec[3 * e] = vx; edge_vec[3 * e + 1] = vy; edge_vec[3 * e + 2] = vz;
    dist_out[e] = d;
    const EnvCoef k = env_coef(cfg.envelope_exponent);
    const float s = d / cfg.cutoff;
    env_out[e] = s < 1.f ? 1.f + ipow(s, k.p) * (k.a + s * (k.b + k.c * s)) : 0.f;
  }
}

// The same for many edges, rows as planes only: a warp takes kManyEdges edges, a lane each for their
// geometry, all lanes together for their rows.  Bound by the planes it writes (1280 bytes an edge at 64
// basis functions, 128 channels, two planes).  With an edge per warp its reads are a chain of four behind
// which 31 lanes wait: 190 us for 264 000 edges, here 82 (232 and 105 for 384 000 edges and one plane).
constexpr int kManyEdges = 8;
__global__ void __launch_bounds__(32 * kWarps)
edge_features_fwd_many_kernel(int64_t E, zp_front_config cfg, const float *__restrict__ pos,
                              const float *__restrict__ shifts, const int64_t *__restrict__ z,
                              const float *__restrict__ emb, const float *__restrict__ offsets,
                              const float *__restrict__ cos_g, const float *__restrict__ sin_g,
                              const int32_t *__restrict__ perm, const int32_t *__restrict__ src,
                              const int32_t *__restrict__ dst, float *__restrict__ edge_vec,
                              float *__restrict__ dist_out, const ZpPlanes xp, const ZpScale scale,
                              float *__restrict__ env_out, float *__restrict__ cos_s,
                              float *__restrict__ sin_s) {
  zp_after_previous();
  constexpr int G = kManyEdges;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int64_t e0 = ((int64_t)blockIdx.x * kWarps + warp) * G;
  const float inv = zp_publish_scale(xp, scale, blockIdx.x == 0 && threadIdx.x == 0);
  if (e0 >= E) return;
  const int n = G < E - e0 ? G : (int)(E - e0);
  const int NB = cfg.num_basis, EC = cfg.edge_channels, W = NB + 2 * EC;
  int order = 0, elem_s = 0, elem_d = 0;
  float dist = 0.f;
  if (lane < n) {
    const int64_t e = e0 + lane, o = perm[e], i = src[e], j = dst[e];
    const float vx = pos[3 * j] - pos[3 * i] + shifts[3 * o];
    const float vy = pos[3 * j + 1] - pos[3 * i + 1] + shifts[3 * o + 1];
    const float vz = pos[3 * j + 2] - pos[3 * i + 2] + shifts[3 * o + 2];
    const float d = sqrtf(fmaxf((vx * vx + vy * vy) + vz * vz, 1e-24f));
    elem_s = (int)min(max(z[i], (int64_t)0), (int64_t)cfg.n_elements - 1);
    elem_d = (int)min(max(z[j], (int64_t)0), (int64_t)cfg.n_elements - 1);
    order = (int)o;
    dist = d;
    edge_vec[3 * e] = vx; edge_vec[3 * e + 1] = vy; edge_vec[3 * e + 2] = vz;
    dist_out[e] = d;
    const EnvCoef k = env_coef(cfg.envelope_exponent);
    const float s = d / cfg.cutoff;
    env_out[e] = s < 1.f ? 1.f + ipow(s, k.p) * (k.a + s * (k.b + k.c * s)) : 0.f;
  }
  const int nl = cfg.lmax + 1;
  for (int t0 = 0; t0 < n * nl; t0 += 32) {
    const int t = t0 + lane, q = t / nl;
    const int64_t o = __shfl_sync(0xffffffffu, order, q < G ? q : 0);
    if (t < n * nl) {
      cos_s[e0 * nl + t] = cos_g[o * nl + t - q * nl];
      sin_s[e0 * nl + t] = sin_g[o * nl + t - q * nl];
    }
  }
  // the quads with basis functions (the last may reach into the source's embedding), of as many edges
  // at a time as the lanes reach
  const int quads = (NB + 3) / 4, shift = quads <= 8 ? 3 : quads <= 16 ? 4 : 5;
  const int sub = lane & ((1 << shift) - 1);
  for (int q0 = 0; q0 < n; q0 += 32 >> shift) {
    const int q = q0 + (lane >> shift), from = q < G ? q : 0;
    const float d = __shfl_sync(0xffffffffu, dist, from);
    const float *es = emb + (size_t)__shfl_sync(0xffffffffu, elem_s, from) * EC;
    if (q < n) {
      for (int k = sub; k < quads; k += 1 << shift) {
        float v[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int b = 4 * k + r;
          const float t = d - (b < NB ? offsets[b] : 0.f);
          v[r] = b < NB ? expf(cfg.gauss_coeff * t * t) : es[b - NB];
        }
        zp_store_planes<4>(xp, (e0 + q) * xp.ld + 4 * k, v, inv);
      }
    }
  }
  // the embeddings, edge by edge
#pragma unroll 2
  for (int q = 0; q < n; ++q) {
    const float *es = emb + (size_t)__shfl_sync(0xffffffffu, elem_s, q) * EC,
                *ed = emb + (size_t)__shfl_sync(0xffffffffu, elem_d, q) * EC;
    for (int c = 4 * (quads + lane); c < xp.ld; c += 128) {
      float v[4];
      if ((NB & 3) == 0 && c < W) {
        const float4 r = *reinterpret_cast<const float4 *>(c < NB + EC ? es + (c - NB) : ed + (c - NB - EC));
        v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
      } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int b = c + r;
          v[r] = b < NB + EC ? es[b - NB] : b < W ? ed[b - NB - EC] : 0.f;
        }
      }
      zp_store_planes<4>(xp, (e0 + q) * xp.ld + c, v, inv);
    }
  }
}

// g_v[e] = g_edge_vec[e] + d_d v / d.  The basis values are formed again from the distance: cheaper
// than reading them back.  gx [E, ldg]: at least the num_basis leading columns.  Eight lanes per edge, a
// sector of its row at a time; a warp per edge left 31 lanes waiting for one that closes the edge:
// 76 us for 264 000 edges, now 29 (107 and 41 for 384 000 and rows of 320 columns).
constexpr int kBwdLanes = 8, kBwdEdges = 32 / kBwdLanes * kWarps;
__global__ void __launch_bounds__(32 * kWarps)
edge_features_bwd_edge_kernel(int64_t E, zp_front_config cfg, const float *__restrict__ edge_vec,
                              const float *__restrict__ dist, const float *__restrict__ offsets,
                              const float *__restrict__ gx, int64_t ldg,
                              const float *__restrict__ g_env, const float *__restrict__ g_vec_in,
                              float *__restrict__ g_vec) {
  zp_after_previous();
  const int sub = threadIdx.x % kBwdLanes;
  const int64_t e = (int64_t)blockIdx.x * kBwdEdges + threadIdx.x / kBwdLanes;
  const bool live = e < E;
  const float d = live ? dist[e] : 1.f;
  float acc = 0.f;
  if (gx && live) {
    const float *gr = gx + (size_t)e * ldg;
#pragma unroll 4
    for (int b = sub; b < cfg.num_basis; b += kBwdLanes) {
      const float t = d - offsets[b];
      acc += gr[b] * expf(cfg.gauss_coeff * t * t) * (2.f * cfg.gauss_coeff * t);
    }
  }
#pragma unroll
  for (int o = kBwdLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (sub == 0 && live) {
    if (g_env) {
      const EnvCoef k = env_coef(cfg.envelope_exponent);
      const float s = d / cfg.cutoff;
      if (s < 1.f) {
        // d/ds [ s^p (a + b s + c s^2) ] = s^(p-1) (p a + (p+1) b s + (p+2) c s^2)
        const float ds = ipow(s, k.p - 1) * (k.p * k.a + s * ((k.p + 1) * k.b + (k.p + 2) * k.c * s));
        acc += g_env[e] * ds / cfg.cutoff;
      }
    }
    const float vx = edge_vec[3 * e], vy = edge_vec[3 * e + 1], vz = edge_vec[3 * e + 2];
    const bool clamped = (vx * vx + vy * vy) + vz * vz < 1e-24f;
    const float f = clamped ? 0.f : acc / d;
    g_vec[3 * e] = (g_vec_in ? g_vec_in[3 * e] : 0.f) + f * vx;
    g_vec[3 * e + 1] = (g_vec_in ? g_vec_in[3 * e + 1] : 0.f) + f * vy;
    g_vec[3 * e + 2] = (g_vec_in ? g_vec_in[3 * e + 2] : 0.f) + f * vz;
  }
}

// one block per atom: the last warp forms the position gradient, a lane per edge, the warps before it (if
// the embedding gradient is wanted) the atom's row of that, eight edges on their way.  Bound by the latency
// of its gathers where atoms are few: 26 -> 16 us for 216 atoms of 42 edges each way; positions alone,
// which three threads added edge by edge before, 16 -> 9 us for 5 832 atoms.
constexpr int kEmbThreads = 128;
__global__ void __launch_bounds__(kEmbThreads + 32)
edge_features_bwd_node_kernel(int64_t N, zp_front_config cfg, const float *__restrict__ g_vec,
                              const float *__restrict__ gx, int64_t ldg,
                              const int32_t *__restrict__ row_ptr,
                              const int32_t *__restrict__ perm_src,
                              const int32_t *__restrict__ row_ptr_src, float *__restrict__ g_pos,
                              float *__restrict__ node_emb) {
  zp_after_previous();
  const int64_t n = blockIdx.x;
  const int beg = row_ptr[n], end = row_ptr[n + 1];
  const int sbeg = row_ptr_src[n], send = row_ptr_src[n + 1];
  const int emb_threads = blockDim.x - 32;
  if (threadIdx.x >= emb_threads) {
    if (!g_pos) return;
    const int lane = threadIdx.x - emb_threads;
    float acc[3] = {0.f, 0.f, 0.f};
    for (int e = beg + lane; e < end; e += 32)
#pragma unroll
      for (int k = 0; k < 3; ++k) acc[k] += g_vec[3 * (int64_t)e + k];
    for (int t = sbeg + lane; t < send; t += 32) {
      const int64_t e = perm_src[t];
#pragma unroll
      for (int k = 0; k < 3; ++k) acc[k] -= g_vec[3 * e + k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (lane < 3) g_pos[3 * n + lane] = lane == 0 ? acc[0] : lane == 1 ? acc[1] : acc[2];
    return;
  }
  const int NB = cfg.num_basis, EC = cfg.edge_channels;
  for (int c = threadIdx.x; c < EC; c += emb_threads) {
    float acc = 0.f;
    if (gx) {
      for (int k = sbeg; k < send; k += 8) {
        float v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r)
          v[r] = k + r < send ? gx[(size_t)perm_src[k + r] * ldg + NB + c] : 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) acc += v[r];
      }
      for (int e = beg; e < end; e += 8) {
        float v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r)
          v[r] = e + r < end ? gx[(size_t)(e + r) * ldg + NB + EC + c] : 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) acc += v[r];
      }
    }
    node_emb[(size_t)n * EC + c] = acc;
  }
}

// one block per (element, slice of the atoms): rows of the slice's atoms of that element, in
// index order, into partial[slice][element]; the slices are then added in slice order.  The block
// lists the atoms of its element among 1024 at a time, then its threads add their rows, eight loads on
// their way: 105 us for 12 800 atoms when they were tested and added one by one, now 19.
constexpr int kElemSlices = 8;           // the rows of one element are a serial chain of additions
constexpr int kElemPerThread = 8;
__global__ void __launch_bounds__(128)
edge_features_bwd_elem_kernel(int64_t N, int EC, const int64_t *__restrict__ z,
                              const float *__restrict__ node_emb, float *__restrict__ partial) {
  zp_after_previous();
  __shared__ int list[128 * kElemPerThread];
  __shared__ int found[kElemPerThread * 4];          // atoms per 32 consecutive ones
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t elem = blockIdx.x;
  const int64_t per = (N + kElemSlices - 1) / kElemSlices;
  const int64_t lo = blockIdx.y * per, hi = min(N, lo + per);
  float *g_emb = partial + (size_t)blockIdx.y * gridDim.x * EC;
  float acc[8];                                   // channels c = threadIdx.x + k * blockDim.x
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  for (int64_t n0 = lo; n0 < hi; n0 += 128 * kElemPerThread) {
    unsigned hits[kElemPerThread];
#pragma unroll
    for (int r = 0; r < kElemPerThread; ++r) {
      const int64_t n = n0 + 128 * r + threadIdx.x;
      hits[r] = __ballot_sync(0xffffffffu, n < hi && z[n] == elem);
      if (lane == 0) found[4 * r + warp] = __popc(hits[r]);
    }
    __syncthreads();
    int upto = found[lane];                       // 32 groups of 32 atoms, a lane each
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += u;
    }
    const int count = __shfl_sync(0xffffffffu, upto, 31), before = upto - found[lane];
#pragma unroll
    for (int r = 0; r < kElemPerThread; ++r) {
      const int at = __shfl_sync(0xffffffffu, before, 4 * r + warp);
      if (hits[r] >> lane & 1)
        list[at + __popc(hits[r] & ((1u << lane) - 1u))] = 128 * r + threadIdx.x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int c = threadIdx.x + k * 128;
      if (c < EC) {
#pragma unroll 8
        for (int t = 0; t < count; ++t) acc[k] += node_emb[(size_t)(n0 + list[t]) * EC + c];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int c = threadIdx.x + k * 128;
    if (c < EC) g_emb[(size_t)elem * EC + c] = acc[k];
  }
}
static_assert(kElemPerThread * 4 == 32, "a lane per group");

__global__ void edge_features_elem_sum_kernel(int64_t total, const float *__restrict__ partial,
                                             float *__restrict__ g_emb) {
  zp_after_previous();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  float s = 0.f;
  for (int k = 0; k < kElemSlices; ++k) s += partial[(size_t)k * total + i];
  g_emb[i] = s;
}

int check_cfg(const zp_front_config *cfg) {
  if (!cfg) return ZP_ERR_INVALID_ARG;
  if (cfg->num_basis < 1 || cfg->edge_channels < 4 || (cfg->edge_channels % 4) ||
      cfg->n_elements < 1 || cfg->lmax < 0 || cfg->lmax > ZP_MAX_L || !(cfg->cutoff > 0.f) ||
      cfg->edge_channels > 1024 || cfg->envelope_exponent < 1 || cfg->envelope_exponent > 16)
    return ZP_ERR_UNSUPPORTED;
  return ZP_OK;
}

}  // namespace

int zp_launch_edge_features_fwd(const zp_front_config &cfg, int64_t E, const float *pos,
                                const float *shifts, const int64_t *atomic_numbers, const float *emb,
                                const float *gauss_offsets, const float *cos_g, const float *sin_g,
                                const int32_t *perm, const int32_t *src, const int32_t *dst,
                                float *edge_vec, float *dist, float *x_edge,
                                const ZpPlanes *x_planes, const ZpScale &scale, float *env,
                                float *cos_sorted, float *sin_sorted, cudaStream_t st) {
  if (E == 0) return ZP_OK;
  const ZpPlanes xp = x_planes ? *x_planes : ZpPlanes{nullptr, 0, 0, 0, 0, nullptr};
  // several edges per warp where that leaves every SM half its warps; below that latency is all that
  // counts, and a warp per edge is 2 us faster at 6 000 edges
  if (x_planes && E >= (int64_t)148 * 32 * kManyEdges)
    zp_launch(edge_features_fwd_many_kernel, (unsigned)zp_ceil_div(E, kWarps * kManyEdges), 32 * kWarps,
              0, st, E, cfg, pos, shifts, atomic_numbers, emb, gauss_offsets, cos_g, sin_g, perm, src,
              dst, edge_vec, dist, xp, scale, env, cos_sorted, sin_sorted);
  else
    zp_launch(edge_features_fwd_kernel, (unsigned)zp_ceil_div(E, kWarps), 32 * kWarps, 0, st, E, cfg,
              pos, shifts, atomic_numbers, emb, gauss_offsets, cos_g, sin_g, perm, src, dst, edge_vec,
              dist, x_edge, xp, scale, env, cos_sorted, sin_sorted);
  ZP_LAUNCH_CHECK("edge_features_fwd_kernel");
  return ZP_OK;
}

int zp_launch_edge_features_bwd(const zp_front_config &cfg, int64_t N, int64_t E,
                                const float *edge_vec, const float *dist,
                                const float *gauss_offsets, const int64_t *atomic_numbers,
                                const float *grad_edge_vec, const float *grad_x_edge, int64_t ldg,
                                const float *grad_env, const int32_t *row_ptr,
                                const int32_t *perm_src, const int32_t *row_ptr_src,
                                float *grad_pos, float *grad_emb, void *work, cudaStream_t st) {
  float *g_vec = static_cast<float *>(work);
  float *node_emb = reinterpret_cast<float *>(static_cast<unsigned char *>(work) +
                                              zp_align_up(sizeof(float) * 3 * (size_t)E, 256));
  if (E && grad_pos) {
    zp_launch(edge_features_bwd_edge_kernel, (unsigned)zp_ceil_div(E, kBwdEdges), 32 * kWarps, 0, st, E,
              cfg, edge_vec, dist, gauss_offsets, grad_x_edge, ldg, grad_env, grad_edge_vec, g_vec);
    ZP_LAUNCH_CHECK("edge_features_bwd_edge_kernel");
  }
  zp_launch(edge_features_bwd_node_kernel, (unsigned)N, grad_emb ? kEmbThreads + 32 : 32, 0, st, N, cfg, g_vec, grad_x_edge, ldg,
            row_ptr, perm_src, row_ptr_src, grad_pos, grad_emb ? node_emb : nullptr);
  ZP_LAUNCH_CHECK("edge_features_bwd_node_kernel");
  if (grad_emb) {
    float *partial = reinterpret_cast<float *>(
        reinterpret_cast<unsigned char *>(node_emb) +
        zp_align_up(sizeof(float) * (size_t)N * cfg.edge_channels, 256));
    const int64_t total = (int64_t)cfg.n_elements * cfg.edge_channels;
    zp_launch(edge_features_bwd_elem_kernel, dim3((unsigned)cfg.n_elements, kElemSlices), 128, 0, st,
              N, cfg.edge_channels, atomic_numbers, node_emb, partial);
    ZP_LAUNCH_CHECK("edge_features_bwd_elem_kernel");
    zp_launch(edge_features_elem_sum_kernel, (unsigned)zp_ceil_div(total, 256), 256, 0, st, total,
              partial, grad_emb);
    ZP_LAUNCH_CHECK("edge_features_elem_sum_kernel");
  }
  return ZP_OK;
}

extern "C" {

size_t zp_edge_features_work_bytes(const zp_front_config *cfg, int64_t n_nodes, int64_t n_edges) {
  if (check_cfg(cfg) || n_nodes < 0 || n_edges < 0) return 0;
  return zp_align_up(sizeof(float) * 3 * (size_t)n_edges, 256) +
         zp_align_up(sizeof(float) * (size_t)n_nodes * cfg->edge_channels, 256) +
         zp_align_up(sizeof(float) * (size_t)kElemSlices * cfg->n_elements * cfg->edge_channels, 256) +
         256;
}

int zp_edge_features_forward(const zp_front_config *cfg, int64_t N, int64_t E, const float *pos,
                             const float *shifts, const int64_t *atomic_numbers, const float *emb,
                             const float *gauss_offsets, const float *cos_g, const float *sin_g,
                             const int32_t *perm, const int32_t *src, const int32_t *dst,
                             float *edge_vec, float *dist, float *x_edge, float *env,
                             float *cos_sorted, float *sin_sorted, void *stream) {
  int rc = check_cfg(cfg);
  if (rc) return rc;
  if (N < 0 || E < 0) return ZP_ERR_INVALID_ARG;
  if (E == 0) return ZP_OK;
  if (!pos || !shifts || !atomic_numbers || !emb || !gauss_offsets || !cos_g || !sin_g || !perm ||
      !src || !dst || !edge_vec || !dist || !x_edge || !env || !cos_sorted || !sin_sorted)
    return ZP_ERR_INVALID_ARG;
  if (reinterpret_cast<uintptr_t>(emb) & 15) return ZP_ERR_INVALID_ARG;
  return zp_launch_edge_features_fwd(*cfg, E, pos, shifts, atomic_numbers, emb, gauss_offsets, cos_g,
                                     sin_g, perm, src, dst, edge_vec, dist, x_edge, nullptr,
                                     ZpScale{}, env, cos_sorted, sin_sorted, (cudaStream_t)stream);
}

int zp_edge_features_backward(const zp_front_config *cfg, int64_t N, int64_t E,
                              const float *edge_vec, const float *dist, const float *x_edge,
                              const float *gauss_offsets, const int64_t *atomic_numbers,
                              const float *grad_edge_vec, const float *grad_x_edge,
                              const float *grad_env, const int32_t *row_ptr,
                              const int32_t *perm_src, const int32_t *row_ptr_src,
                              float *grad_pos, float *grad_emb, void *work, size_t work_bytes,
                              void *stream) {
  int rc = check_cfg(cfg);
  if (rc) return rc;
  if (N < 0 || E < 0 || !grad_pos) return ZP_ERR_INVALID_ARG;
  if (N == 0) return E == 0 ? ZP_OK : ZP_ERR_INVALID_ARG;
  if (!atomic_numbers || !row_ptr || !row_ptr_src || !work) return ZP_ERR_INVALID_ARG;
  if (E && (!edge_vec || !dist || !x_edge || !gauss_offsets || !perm_src)) return ZP_ERR_INVALID_ARG;
  if (work_bytes < zp_edge_features_work_bytes(cfg, N, E)) return ZP_ERR_WORKSPACE;
  return zp_launch_edge_features_bwd(*cfg, N, E, edge_vec, dist, gauss_offsets, atomic_numbers,
                                     grad_edge_vec, grad_x_edge,
                                     cfg->num_basis + 2 * cfg->edge_channels, grad_env, row_ptr,
                                     perm_src, row_ptr_src, grad_pos, grad_emb, work,
                                     (cudaStream_t)stream);
}

}  // extern "C"
