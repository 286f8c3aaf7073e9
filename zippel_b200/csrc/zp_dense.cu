// Elementwise and layout pieces around the SO(2) contraction: the gate activation and its VJP,
// weight folding into bf16 planes (and the transpose of that for the weight gradients), and
// column sums for the bias gradients.  The contraction itself runs on the tensor cores.
//
// Weight folding.  For m > 0 the reference applies one Linear to the real and the imaginary
// rows and recombines the halves of its output (blocks/eso2_ref.py:282-291):
//     out_re = Wa x_re - Wb x_im,   out_im = Wb x_re + Wa x_im,   W = [Wa ; Wb].
// With the m'-major row order (real rows, then imaginary rows) that is ONE product with
//     W_fold = [ Wa  -Wb ]
//              [ Wb   Wa ]            of shape [2 km Cout, 2 km Cin],
// the same number of multiply-adds as the reference's two-row form, and no recombination.
// Every m-block of conv1 and conv2 is therefore a plain  Y[E, out] = X[E, in] W_fold^T.
#include <cuda_bf16.h>

#include <algorithm>

#include "zp_rotate.cuh"

namespace {

// fp32 matrices (blockIdx.z) -> planes (bf16, or fp16 with the tensor's scale), zero padding up to ld_out.
// threadIdx.x walks the quads of a row, threadIdx.y / blockIdx.x the rows (no division anywhere).
__global__ void split_planes_kernel(const __grid_constant__ ZpSplitList d) {
  zp_after_previous();
  const int b = blockIdx.z;
  const float *__restrict__ in = d.in[b];
  const int64_t rows = d.rows[b], cols = d.cols[b], ld_in = d.ld_in[b];
  const ZpPlanes out = d.out[b];
  const int64_t c = 4 * ((int64_t)blockIdx.y * blockDim.x + threadIdx.x);
  const float inv =
      zp_publish_scale(out, d.scale[b], blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 &&
                                            threadIdx.y == 0);
  if (c >= out.ld) return;
  const bool vec = (ld_in & 3) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0 && c + 3 < cols;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.y + threadIdx.y; r < rows;
       r += (int64_t)gridDim.x * blockDim.y) {
    float v[4];
    if (vec) {
      const float4 q = *reinterpret_cast<const float4 *>(in + r * ld_in + c);
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = c + k < cols ? in[r * ld_in + c + k] : 0.f;
    }
    zp_store_planes<4>(out, r * out.ld + c, v, inv);
  }
}

// largest node index the edge list names (the caller zeroed *out)
__global__ void max_index_kernel(int64_t E, const int32_t *__restrict__ src,
                                 const int32_t *__restrict__ dst, int *out) {
  zp_after_previous();
  int m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E;
       i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, max(src[i], dst[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(out, m);
}

// max |x| over rows [r0, r1) of a contiguous [*, cols] matrix (cols a multiple of 4, 16-byte
// aligned rows), the row numbers read from device memory:
//   r0 = first ? *first : 0,   r1 = max(min_rows, last ? *last + 1 : 0)
__global__ void absmax_row_range_kernel(const float *__restrict__ in, int64_t cols,
                                        const int32_t *first, const int32_t *last,
                                        int64_t min_rows, float *out) {
  zp_after_previous();
  const int64_t r0 = first ? *first : 0;
  int64_t r1 = last ? (int64_t)*last + 1 : 0;
  if (r1 < min_rows) r1 = min_rows;
  float m = 0.f;
  const float4 *in4 = reinterpret_cast<const float4 *>(in + r0 * cols);
  const int64_t n4 = (r1 > r0 ? r1 - r0 : 0) * cols / 4;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float4 v = in4[i];
    m = fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.f) zp_atomic_absmax(out, m);
}

// ------------------------------------------------------------------------------------------
// gate activation (blocks/eso2_ref.py:295-301): conv1 output row h1[e] = [gate (lmax*H) | y (Km*H)]
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float sigmoidf(float x) { return 1.f / (1.f + __expf(-x)); }

// Both directions: one thread per (edge, hidden-channel quad) goes through the degrees.  A degree's gate is read
// and its sigmoid formed once for its 2 mmax + 1 rows, and the rows of up to |m| = 2 are requested before any is
// used.  Bound by HBM (forward 21.5 KB, backward 33 KB an edge at lmax 4 / mmax 2 / H 128 in two planes: 60 000 edges in
// 193 and 291 us, 6.7 and 6.9 TB/s; 261 and 372 with a gate read for every row and chosen at run time).
//
// With `gate_max` set the forward also records the largest sigmoid'(gate) it sees: max|dht| * rows(l) * max|h1| *
// that value bounds the gate part of the backward's dh1, which fixes the scale of its fp16 planes before they
// are written (the bound follows the gates into saturation, where a constant 1/4 would be orders of magnitude
// loose).
constexpr int kGateThreads = 128;
struct GateItem {
  int64_t e;
  int h;
  bool live;
  // 32-bit arithmetic within a block: a 64-bit division per thread would cost more than the rest
  __device__ __forceinline__ GateItem(int64_t E, int H4, int per_block) {
    const int le = threadIdx.x / H4;
    e = (int64_t)blockIdx.x * per_block + le;
    h = ((int)threadIdx.x - le * H4 + (int)blockIdx.y * (int)blockDim.x) * 4;
    live = le < per_block && e < E && h < 4 * H4;
    if (gridDim.y > 1) {                 // rows wider than a block: a block per part of one edge
      e = blockIdx.x;
      h = ((int)blockIdx.y * (int)blockDim.x + (int)threadIdx.x) * 4;
      live = h < 4 * H4;
    }
    if (!live) { e = 0; h = 0; }         // recomputes edge 0
  }
};
__device__ __forceinline__ F4 sigmoid4(const F4 &x) {
  const float2 a = unpack2(x.a), b = unpack2(x.b);
  return F4{pack2(sigmoidf(a.x), sigmoidf(a.y)), pack2(sigmoidf(b.x), sigmoidf(b.y))};
}
// s (1 - s)
__device__ __forceinline__ F4 slope4(const F4 &s) {
  const u64 one = pack2(1.f, 1.f);
  return F4{mul2(s.a, sub2(one, s.a)), mul2(s.b, sub2(one, s.b))};
}
__device__ __forceinline__ float most4(const F4 &v) {
  const float2 a = unpack2(v.a), b = unpack2(v.b);
  return fmaxf(fmaxf(a.x, a.y), fmaxf(b.x, b.y));
}

template <int LM, int FMT>
__global__ void __launch_bounds__(kGateThreads)
gate_fwd_kernel(const __grid_constant__ ZpTables t, int64_t E, int per_block, const float *__restrict__ h1,
                const ZpPlanes ht, const ZpScale scale, float *gate_max) {
  zp_after_previous();
  const GateItem it(E, t.H / 4, per_block);
  const float inv = zp_publish_scale(ht, scale, blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0);
  const float *gates = h1 + (size_t)it.e * t.w1_cols + it.h, *x = gates + t.n_gate;
  uint16_t *const out = static_cast<uint16_t *>(ht.base) + it.e * ht.ld + it.h;
  const int64_t plane_bytes = 2 * ht.plane_stride;
  const u64 inv2 = pack2(inv, inv);
  const int H = t.H;
  float seen = 0.f;
  auto row = [&](int r, const F4 &v, const F4 &s) {
    if (it.live) put4<FMT>(out + r * H, plane_bytes, mul4(v, s), inv2);
  };
#pragma unroll
  for (int l = 0; l <= LM; ++l) {
    const int mm = t.mmax < l ? t.mmax : l;
    // rows of the degree in the m'-major order: l, then +m and -m, LM + 1 - m rows apart
    const int p1 = l + LM, m1 = p1 + LM, p2 = p1 + 2 * LM - 1, m2 = p2 + LM - 1;
    const F4 x0 = load4(x + l * H);
    F4 g, a1, b1, a2, b2;
    if (l > 0) g = load4(gates + (l - 1) * H);
    if (mm >= 1) { a1 = load4(x + p1 * H); b1 = load4(x + m1 * H); }
    if (mm >= 2) { a2 = load4(x + p2 * H); b2 = load4(x + m2 * H); }
    const F4 s = sigmoid4(l > 0 ? g : x0);      // l = 0: x sigmoid(x)
    if (l > 0) seen = fmaxf(seen, most4(slope4(s)));
    row(l, x0, s);
    if (mm >= 1) { row(p1, a1, s); row(m1, b1, s); }
    if (mm >= 2) { row(p2, a2, s); row(m2, b2, s); }
    for (int m = 3, p = p2; m <= mm; ++m) {
      const int km = LM + 1 - m;
      p += 2 * (km + 1) - 1;
      const F4 a = load4(x + p * H), b = load4(x + (p + km) * H);
      row(p, a, s);
      row(p + km, b, s);
    }
  }
  if (gate_max) {
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) seen = fmaxf(seen, __shfl_xor_sync(0xffffffffu, seen, k));
    // one address for the whole grid: only warps that would raise the maximum touch it atomically
    if ((threadIdx.x & 31) == 0 && seen > *reinterpret_cast<volatile float *>(gate_max))
      zp_atomic_absmax(gate_max, seen);
  }
}

// Also sums the lmax gate gradients.  The scale of the fp16 planes is fixed beforehand from max |dht| and the
// forward's gate bound:
//   |dh1 row| <= 1.1 max|dht|  (sigmoid <= 1, silu' <= 1.1),
//   |dh1 gate_l| = sigmoid'(g_l) |sum_rows dht h1| <= max|dht| * rows(l) * max|h1| * max sigmoid'.
template <int LM, int FMT>
__global__ void __launch_bounds__(kGateThreads)
gate_bwd_kernel(const __grid_constant__ ZpTables t, int64_t E, int per_block, const float *__restrict__ h1,
                const float *__restrict__ dht, const ZpPlanes dh1, const ZpScale scale) {
  zp_after_previous();
  const GateItem it(E, t.H / 4, per_block);
  const float inv = zp_publish_scale(dh1, scale, blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0);
  const float *gates = h1 + (size_t)it.e * t.w1_cols + it.h, *x = gates + t.n_gate;
  const float *d = dht + (size_t)it.e * t.Km * t.H + it.h;
  uint16_t *const out = static_cast<uint16_t *>(dh1.base) + it.e * dh1.ld + it.h;
  const int64_t plane_bytes = 2 * dh1.plane_stride;
  const u64 inv2 = pack2(inv, inv);
  const int H = t.H;
  auto put = [&](int column, const F4 &v) {
    if (it.live) put4<FMT>(out + column, plane_bytes, v, inv2);
  };
#pragma unroll
  for (int l = 0; l <= LM; ++l) {
    const int mm = t.mmax < l ? t.mmax : l;
    const int p1 = l + LM, m1 = p1 + LM, p2 = p1 + 2 * LM - 1, m2 = p2 + LM - 1;
    const F4 x0 = load4(x + l * H), d0 = load4(d + l * H);
    F4 g, a1, b1, a2, b2, c1, e1, c2, e2;
    if (l > 0) g = load4(gates + (l - 1) * H);
    if (mm >= 1) { a1 = load4(x + p1 * H); b1 = load4(x + m1 * H); c1 = load4(d + p1 * H); e1 = load4(d + m1 * H); }
    if (mm >= 2) { a2 = load4(x + p2 * H); b2 = load4(x + m2 * H); c2 = load4(d + p2 * H); e2 = load4(d + m2 * H); }
    const F4 s = sigmoid4(l > 0 ? g : x0), slope = slope4(s);
    if (l == 0) {                        // d (s + x s (1 - s))
      put(t.n_gate, mul4(d0, F4{fma2(x0.a, slope.a, s.a), fma2(x0.b, slope.b, s.b)}));
      continue;
    }
    F4 dg = zero4();
    auto row = [&](int r, const F4 &xv, const F4 &dv) {
      put(t.n_gate + r * H, mul4(dv, s));
      dg.a = fma2(dv.a, xv.a, dg.a);
      dg.b = fma2(dv.b, xv.b, dg.b);
    };
    row(l, x0, d0);
    if (mm >= 1) { row(p1, a1, c1); row(m1, b1, e1); }
    if (mm >= 2) { row(p2, a2, c2); row(m2, b2, e2); }
    for (int m = 3, p = p2; m <= mm; ++m) {
      const int km = LM + 1 - m;
      p += 2 * (km + 1) - 1;
      row(p, load4(x + p * H), load4(d + p * H));
      row(p + km, load4(x + (p + km) * H), load4(d + (p + km) * H));
    }
    put((l - 1) * H, mul4(dg, slope));
  }
}

// ------------------------------------------------------------------------------------------
// weight folding and its transpose
// ------------------------------------------------------------------------------------------
// Maxima of up to ZP_MAX_ITEMS arrays in one launch (the caller zeroed the slots): every weight block,
// and whatever else a call needs the magnitude of before its first product.  A block takes a stretch
// of neighbouring tiles of 4096 values and leaves one atomic per warp and array.
constexpr int kMaxTile = 4096;
__global__ void __launch_bounds__(256)
max_list_kernel(const __grid_constant__ ZpMaxList d, const __grid_constant__ ZpTileRow row) {
  zp_after_previous();
  const int total = row.first[row.n];
  int t = (int)((int64_t)total * blockIdx.x / gridDim.x);
  const int end = (int)((int64_t)total * (blockIdx.x + 1) / gridDim.x);
  for (int b = 0; t < end;) {
    b = row.entry(t, b);
    const float *x = d.x[b];
    const int last = min(end, row.first[b + 1]);
    const int64_t i0 = (int64_t)(t - row.first[b]) * kMaxTile;
    const int64_t i1 = min(d.count[b], (int64_t)(last - row.first[b]) * kMaxTile);
    float m = 0.f;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
      const float4 *x4 = reinterpret_cast<const float4 *>(x);
#pragma unroll 4
      for (int64_t i = i0 / 4 + threadIdx.x; i < i1 / 4; i += 256) {
        const float4 v = x4[i];
        m = fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
      }
      if ((int)threadIdx.x < (int)(i1 & 3)) m = fmaxf(m, fabsf(x[(i1 & ~3ll) + threadIdx.x]));
    } else {
      for (int64_t i = i0 + threadIdx.x; i < i1; i += 256) m = fmaxf(m, fabsf(x[i]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.f) zp_atomic_absmax(d.out[b], m);
    t = last;
  }
}

// Writes every weight matrix as 16-bit planes, all of them in one launch (blockIdx.y = matrix).
//   plain          W [out, in] -> planes [out, ld], zero padded
//   kept / folded  W_fold [out, in] and its transpose [in, out];  m = 0 (kept): W_fold = W,
//                  m > 0 (folded): W = [Wa ; Wb] (rows), W_fold = [Wa -Wb ; Wb Wa]
// slot = {max |W|, scale}: the scale follows from the maximum here (fp16 planes).
// Bound by instruction issue, so a thread takes V = 4 neighbouring columns where the widths allow (every
// width in use): a value at a time took 115 instructions per value (38 us for the weights of lmax 4 /
// mmax 2 / C 128 as one plane; now 12).  Tiles of 32 rows and 32 V columns; the planes of W_fold go
// out row-major as they are formed, the transpose from a shared copy of the tile so that both
// stores run along the fastest axis.
constexpr int kPrepPitch = 130;
template <int V>
__device__ __forceinline__ void prep_tile(const ZpPrepList &d, int b, int tl, uint16_t (*tile)[kPrepPitch]) {
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;          // 32 x 8
  const int out = d.out[b], in = d.in[b], kind = d.kind[b], planes = d.planes[b], ld = d.ld[b];
  const bool fp16 = d.fp16[b];
  const int64_t stride = d.plane_stride[b];
  float inv = 1.f;
  if (fp16) {
    const float s = zp_scale_for_bound(d.slot[b][0]);
    inv = 1.f / s;
    if (tl == 0 && threadIdx.x == 0) d.slot[b][1] = s;
  }
  const int cols = kind == ZP_PREP_PLAIN ? ld : in;
  const int tiles_c = (cols + 32 * V - 1) / (32 * V);
  const int r0 = (tl / tiles_c) * 32, c0 = (tl % tiles_c) * 32 * V, c = c0 + tx * V;
  const int half = out / 2, kin = in / 2;
  const bool right = kind == ZP_PREP_FOLDED && c >= kin;
  const float *__restrict__ w = d.w[b] + (right ? c - kin : c);
  const int ld_w = kind == ZP_PREP_FOLDED ? kin : in;
  float v[4][V];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int row = r0 + ty + 8 * k;
#pragma unroll
    for (int q = 0; q < V; ++q) v[k][q] = 0.f;
    if (row >= out || c >= in) continue;
    // the upper right quarter is -Wb, the lower right Wa
    const int o = !right ? row : row < half ? row + half : row - half;
    const float *from = w + (size_t)o * ld_w;
    if (V == 4) {
      const float4 x = *reinterpret_cast<const float4 *>(from);
      v[k][0] = x.x; v[k][V / 4] = x.y; v[k][V / 2] = x.z; v[k][V - 1] = x.w;
    } else {
      v[k][0] = *from;
    }
    const float f = right && row < half ? -inv : inv;
#pragma unroll
    for (int q = 0; q < V; ++q) v[k][q] *= f;
  }
  const bool transpose = kind != ZP_PREP_PLAIN && d.transposes;
  uint16_t *wp = d.dst[b], *wtp = wp + (size_t)planes * stride;
  for (int p = 0; p < planes; ++p) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int row = r0 + ty + 8 * k;
      uint16_t h[V];
#pragma unroll
      for (int q = 0; q < V; ++q) {
        if (fp16) {
          const __half x = __float2half_rn(v[k][q]);
          h[q] = __half_as_ushort(x);
          v[k][q] -= __half2float(x);
        } else {
          const __nv_bfloat16 x = __float2bfloat16_rn(v[k][q]);
          h[q] = __bfloat16_as_ushort(x);
          v[k][q] -= __bfloat162float(x);
        }
      }
      uint16_t *to = wp + (size_t)p * stride + (size_t)row * ld + c;
      const bool inside = row < out && c < cols;
      if (V == 4) {
        const uint2 x = make_uint2(h[0] | (uint32_t)h[V / 4] << 16, h[V / 2] | (uint32_t)h[V - 1] << 16);
        if (inside) *reinterpret_cast<uint2 *>(to) = x;
        uint32_t *copy = reinterpret_cast<uint32_t *>(&tile[ty + 8 * k][tx * V]);
        if (transpose) copy[0] = x.x, copy[1] = x.y;
      } else {
        if (inside) *to = h[0];
        if (transpose) tile[ty + 8 * k][tx] = h[0];
      }
    }
    if (!transpose) continue;                    // uniform over the block
    __syncthreads();
    uint16_t *wt = wtp + (size_t)p * stride;
    if (V == 4) {                                // two rows per lane: the height is even
      const int rr = 2 * (threadIdx.x & 15), row = r0 + rr;
#pragma unroll
      for (int q = 0; q < 2 * V; ++q) {
        const int cc = (threadIdx.x >> 4) + 16 * q, col = c0 + cc;
        if (row < out && col < in)
          *reinterpret_cast<uint32_t *>(wt + (size_t)col * out + row) =
              tile[rr][cc] | (uint32_t)tile[rr + 1][cc] << 16;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int col = c0 + ty + 8 * k, row = r0 + tx;
        if (row < out && col < in) wt[(size_t)col * out + row] = tile[tx][ty + 8 * k];
      }
    }
    __syncthreads();
  }
}
__global__ void __launch_bounds__(256)
prep_weights_kernel(const __grid_constant__ ZpPrepList d, const __grid_constant__ ZpTileRow tiles) {
  zp_after_previous();
  __shared__ __align__(16) uint16_t tile[32][kPrepPitch];
  int b = 0;
  for (int t = blockIdx.x; t < tiles.first[tiles.n]; t += gridDim.x) {
    b = tiles.entry(t, b);
    if (d.quads[b]) prep_tile<4>(d, b, t - tiles.first[b], tile);
    else prep_tile<1>(d, b, t - tiles.first[b], tile);
  }
}

// The last step of every parameter gradient, all of them in one launch.
//   ZP_FIN_SUM     sum of `parts` partial matrices (K splits of a product), in order
//   ZP_FIN_UNFOLD  the same, mapped from the folded layout back to the reference's:
//                  dWa = F[0,0] + F[1,1], dWb = F[1,0] - F[0,1]
//   ZP_FIN_COLUMN  sum of `parts` partial rows: eight columns per tile, 32 threads per column take
//                  every 32nd row, and their sums are added in order
// Bound by the partials it reads.  A tile of the matrices has 256 groups of V neighbouring entries.
template <int V, bool folded>
__device__ __forceinline__ void finalize_entries(const float *__restrict__ f, float *__restrict__ dst,
                                                 int64_t stride, int rows, int cols, int parts, int ld,
                                                 int64_t tile) {
  const int kin = folded ? cols / 2 : cols, half = rows / 2;
  const int64_t idx = (tile * 256 + threadIdx.x) * V;
  if (idx >= (int64_t)rows * kin) return;
  const int c = (int)(idx % kin), row = (int)(idx / kin);
  const bool upper = row < half;
  const float *p = f + (size_t)row * ld + c;
  const float *q = f + (size_t)(upper ? half + row : row - half) * ld + kin + c;
  const float sign = upper ? 1.f : -1.f;
  constexpr int kBatch = folded ? 4 : 8;           // loads of eight groups on their way at a time
  float acc[V], v[kBatch][V], u[kBatch][V];
#pragma unroll
  for (int k = 0; k < V; ++k) acc[k] = 0.f;
  auto load = [](const float *from, float (&to)[V]) {
    if (V == 4) {
      const float4 x = *reinterpret_cast<const float4 *>(from);
      to[0] = x.x; to[V / 4] = x.y; to[V / 2] = x.z; to[V - 1] = x.w;
    } else {
      to[0] = *from;
    }
  };
  for (int s0 = 0; s0 < parts; s0 += kBatch) {
#pragma unroll
    for (int b = 0; b < kBatch; ++b)
      if (s0 + b < parts) {
        load(p + (size_t)(s0 + b) * stride, v[b]);
        if (folded) load(q + (size_t)(s0 + b) * stride, u[b]);
      }
#pragma unroll
    for (int b = 0; b < kBatch; ++b)
      if (s0 + b < parts) {
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] += folded ? v[b][k] + sign * u[b][k] : v[b][k];
      }
  }
  if (V == 4) *reinterpret_cast<float4 *>(dst + idx) = make_float4(acc[0], acc[V / 4], acc[V / 2], acc[V - 1]);
  else dst[idx] = acc[0];
}
__global__ void __launch_bounds__(256)
finalize_kernel(const __grid_constant__ ZpFinalList d, const __grid_constant__ ZpTileRow tiles) {
  zp_after_previous();
  __shared__ float red[32][9];
  int b = 0;
  for (int t = blockIdx.x; t < tiles.first[tiles.n]; t += gridDim.x) {
    b = tiles.entry(t, b);
    const float *f = d.src[b];
    float *dst = d.dst[b];
    const int64_t stride = d.stride[b];
    const int cols = d.cols[b], parts = d.parts[b], kind = d.kind[b], tile = t - tiles.first[b];
    if (kind != ZP_FIN_COLUMN) {
      const bool quads = d.quads[b];
      const int rows = d.rows[b], ld = d.ld[b];
      if (kind == ZP_FIN_UNFOLD) {
        if (quads) finalize_entries<4, true>(f, dst, stride, rows, cols, parts, ld, tile);
        else finalize_entries<1, true>(f, dst, stride, rows, cols, parts, ld, tile);
      } else {
        if (quads) finalize_entries<4, false>(f, dst, stride, rows, cols, parts, ld, tile);
        else finalize_entries<1, false>(f, dst, stride, rows, cols, parts, ld, tile);
      }
      continue;
    }
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    const int c = tile * 8 + tx;
    float s = 0.f;
    if (c < cols)
      for (int p0 = ty; p0 < parts; p0 += 32 * 8) {
        float v[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) v[b] = p0 + 32 * b < parts ? f[(size_t)(p0 + 32 * b) * stride + c] : 0.f;
#pragma unroll
        for (int b = 0; b < 8; ++b) s += v[b];
      }
    red[ty][tx] = s;
    __syncthreads();
    if (ty == 0 && c < cols) {
      float acc = 0.f;
#pragma unroll
      for (int g = 0; g < 32; ++g) acc += red[g][tx];
      dst[c] = acc;
    }
    __syncthreads();
  }
}

// column sums in two fixed-order stages.  Stage one: a block of 32 x 8 threads sums `per_block` rows of
// 256 columns; a thread owns 8 consecutive columns (one 16-byte load per row and plane) and every
// eighth row, the eight row groups are then added in order through shared memory.
__global__ void __launch_bounds__(256)
colsum_part_kernel(int64_t rows, int64_t cols, int64_t per_block, const ZpPlanes a,
                   float *__restrict__ part) {
  zp_after_previous();
  __shared__ float red[8][32][9];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int64_t c0 = ((int64_t)blockIdx.x * 32 + tx) * 8;
  const int64_t r0 = (int64_t)blockIdx.y * per_block;
  const int64_t r1 = min(rows, r0 + per_block);
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c0 < cols) {
#pragma unroll 4
    for (int64_t r = r0 + ty; r < r1; r += 8) {
      for (int pl = a.planes - 1; pl >= 0; --pl) {
        const uint4 v = *reinterpret_cast<const uint4 *>(
            static_cast<const uint16_t *>(a.base) + (size_t)pl * a.plane_stride + r * a.ld + c0);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          s[2 * k] += zp_plane_value(a, (uint16_t)(w[k] & 0xffffu));
          s[2 * k + 1] += zp_plane_value(a, (uint16_t)(w[k] >> 16));
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) red[ty][tx][k] = s[k];
  __syncthreads();
  if (ty == 0 && c0 < cols) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float acc = 0.f;
      for (int g = 0; g < 8; ++g) acc += red[g][tx][k];
      if (c0 + k < cols) part[(size_t)blockIdx.y * cols + c0 + k] = acc * zp_scale(a);
    }
  }
}
// scale of conv1's activated output from an a-priori bound (one block):
//   |h1| <= max_m(in_m * A * max|W_m|) + max|b|,  A = 2^15 * a1_scale >= max|a1|
struct BoundDesc {
  int n;
  int in[ZP_MAX_L + 1];
  int n_bias;
};
__global__ void __launch_bounds__(256)
conv1_bound_kernel(const BoundDesc d, const float *a1_scale, const float *wscales,
                   const float *__restrict__ bias, float *ht_scale) {
  zp_after_previous();
  __shared__ float red[8];
  float m = 0.f;
  for (int i = threadIdx.x; i < d.n_bias; i += blockDim.x) m = fmaxf(m, fabsf(bias[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float bmax = 0.f;
    for (int i = 0; i < 8; ++i) bmax = fmaxf(bmax, red[i]);
    const float a = 32768.f * *a1_scale;
    float bound = 0.f;
    for (int b = 0; b < d.n; ++b) bound = fmaxf(bound, (float)d.in[b] * a * wscales[2 * b]);
    *ht_scale = zp_scale_for_bound(1.001f * (bound + bmax));
  }
}

}  // namespace

int zp_launch_conv1_bound(const zp_plan *p, const float *a1_scale, const float *wscales,
                          const float *bias, float *ht_scale, cudaStream_t st) {
  BoundDesc d;
  d.n = p->n_blocks;
  for (int m = 0; m < p->n_blocks; ++m) d.in[m] = p->c1_in[m];
  d.n_bias = p->c1_out[0];
  zp_launch(conv1_bound_kernel, 1, 256, 0, st, d, a1_scale, wscales, bias, ht_scale);
  ZP_LAUNCH_CHECK("conv1_bound_kernel");
  return ZP_OK;
}

int zp_launch_split_list(const ZpSplitList &list, cudaStream_t st) {
  int64_t rows = 0, quads = 0;
  for (int i = 0; i < list.n; ++i) {
    rows = list.rows[i] > rows ? list.rows[i] : rows;
    quads = list.out[i].ld / 4 > quads ? list.out[i].ld / 4 : quads;
  }
  if (rows == 0 || quads == 0) return ZP_OK;
  int bx = 32;
  while (bx < quads && bx < 256) bx <<= 1;
  const int by = 256 / bx;
  int64_t gx = zp_ceil_div(rows, by);
  if (gx > 148 * 32) gx = 148 * 32;
  zp_launch(split_planes_kernel, dim3((unsigned)gx, (unsigned)zp_ceil_div(quads, bx), list.n),
            dim3(bx, by), 0, st, list);
  ZP_LAUNCH_CHECK("split_planes_kernel");
  return ZP_OK;
}

int zp_launch_split_planes(int64_t rows, int64_t cols, const float *in, int64_t ld_in,
                           const ZpPlanes &out, const ZpScale &scale, cudaStream_t st) {
  ZpSplitList list;
  list.add(rows, cols, in, ld_in, out, scale);
  return zp_launch_split_list(list, st);
}

int zp_launch_max_list(const ZpMaxList &list, cudaStream_t st) {
  if (list.n == 0) return ZP_OK;
  ZpTileRow row;
  for (int i = 0; i < list.n; ++i) row.add(zp_ceil_div(list.count[i], kMaxTile));
  if (row.total() == 0) return ZP_OK;
  zp_launch(max_list_kernel, (unsigned)std::min(row.total(), 148 * 8), 256, 0, st, list, row);
  ZP_LAUNCH_CHECK("max_list_kernel");
  return ZP_OK;
}

int zp_launch_prep_weights(ZpPrepList &list, cudaStream_t st) {
  ZpTileRow row;
  for (int i = 0; i < list.n; ++i) {
    const bool plain = list.kind[i] == ZP_PREP_PLAIN;
    list.quads[i] = list.in[i] % (plain ? 4 : 8) == 0 && (plain || list.out[i] % 2 == 0) &&
                    list.plane_stride[i] % 4 == 0 && (uintptr_t)list.w[i] % 16 == 0;
    row.add(zp_ceil_div(list.out[i], 32) *
            zp_ceil_div(plain ? list.ld[i] : list.in[i], list.quads[i] ? 128 : 32));
  }
  if (row.total() == 0) return ZP_OK;
  zp_launch(prep_weights_kernel, (unsigned)std::min(row.total(), 148 * 16), 256, 0, st, list, row);
  ZP_LAUNCH_CHECK("prep_weights_kernel");
  return ZP_OK;
}

int zp_launch_finalize(ZpFinalList &list, cudaStream_t st) {
  ZpTileRow row;
  for (int i = 0; i < list.n; ++i) {
    const int kin = list.kind[i] == ZP_FIN_UNFOLD ? list.cols[i] / 2 : list.cols[i];
    list.quads[i] = (kin | list.ld[i] | (int)(list.stride[i] & 3)) % 4 == 0 && ((uintptr_t)list.src[i] | (uintptr_t)list.dst[i]) % 16 == 0;
    row.add(list.kind[i] == ZP_FIN_COLUMN ? zp_ceil_div(list.cols[i], 8)
                                          : zp_ceil_div((int64_t)list.rows[i] * kin, list.quads[i] ? 1024 : 256));
  }
  if (row.total() == 0) return ZP_OK;
  zp_launch(finalize_kernel, (unsigned)std::min(row.total(), 148 * 16), 256, 0, st, list, row);
  ZP_LAUNCH_CHECK("finalize_kernel");
  return ZP_OK;
}

int zp_launch_max_index(int64_t E, const int32_t *src, const int32_t *dst, int *out,
                        cudaStream_t st) {
  if (E == 0) return ZP_OK;
  int64_t blocks = zp_ceil_div(E, 256 * 4);
  if (blocks > 592) blocks = 592;
  zp_launch(max_index_kernel, (unsigned)blocks, 256, 0, st, E, src, dst, out);
  ZP_LAUNCH_CHECK("max_index_kernel");
  return ZP_OK;
}

int zp_launch_absmax_row_range(const float *in, int64_t cols, const int32_t *first,
                               const int32_t *last, int64_t min_rows, float *out,
                               cudaStream_t st) {
  if (cols == 0 || (cols & 3)) return cols ? ZP_ERR_INVALID_ARG : ZP_OK;
  zp_launch(absmax_row_range_kernel, 1184, 256, 0, st, in, cols, first, last, min_rows, out);
  ZP_LAUNCH_CHECK("absmax_row_range_kernel");
  return ZP_OK;
}

// blocks of whole edges; of parts of one edge where its row is wider than a block
static dim3 gate_grid(int64_t E, int H4, int *per_block, int *threads) {
  *per_block = H4 <= kGateThreads ? kGateThreads / H4 : 1;
  *threads = H4 <= kGateThreads ? (*per_block * H4 + 31) / 32 * 32 : kGateThreads;
  return dim3((unsigned)zp_ceil_div(E, *per_block), (unsigned)zp_ceil_div(H4, H4 <= kGateThreads ? H4 : kGateThreads));
}

int zp_launch_gate_fwd(const zp_plan *p, int64_t E, const float *h1, const ZpPlanes &ht,
                       const ZpScale &scale, float *gate_max, cudaStream_t st) {
  if (E == 0) return ZP_OK;
  int per_block, threads;
  const dim3 grid = gate_grid(E, p->t.H / 4, &per_block, &threads);
#define CALL_FMT(LM, FMT) zp_launch(gate_fwd_kernel<LM, FMT>, grid, threads, 0, st, p->t, E, per_block, h1, ht, scale, gate_max)
#define CALL(LM)                                               \
  switch (zp_plane_format(ht)) {                               \
    case kFmtBf16: CALL_FMT(LM, kFmtBf16); break;              \
    case kFmtFp16x2: CALL_FMT(LM, kFmtFp16x2); break;          \
    default: CALL_FMT(LM, kFmtBf16x3); break;                  \
  }
  ZP_DISPATCH_LMAX(p->t.lmax, CALL)
#undef CALL
#undef CALL_FMT
  ZP_LAUNCH_CHECK("gate_fwd_kernel");
  return ZP_OK;
}

int zp_launch_gate_bwd(const zp_plan *p, int64_t E, const float *h1, const float *dht,
                       const ZpPlanes &dh1, const ZpScale &scale, cudaStream_t st) {
  if (E == 0) return ZP_OK;
  int per_block, threads;
  const dim3 grid = gate_grid(E, p->t.H / 4, &per_block, &threads);
#define CALL_FMT(LM, FMT) zp_launch(gate_bwd_kernel<LM, FMT>, grid, threads, 0, st, p->t, E, per_block, h1, dht, dh1, scale)
#define CALL(LM)                                               \
  switch (zp_plane_format(dh1)) {                               \
    case kFmtBf16: CALL_FMT(LM, kFmtBf16); break;              \
    case kFmtFp16x2: CALL_FMT(LM, kFmtFp16x2); break;          \
    default: CALL_FMT(LM, kFmtBf16x3); break;                  \
  }
  ZP_DISPATCH_LMAX(p->t.lmax, CALL)
#undef CALL
#undef CALL_FMT
  ZP_LAUNCH_CHECK("gate_bwd_kernel");
  return ZP_OK;
}

static const float *block_weight(const zp_weights *w, int conv, int m) {
  if (m == 0) return conv ? w->c2_w0 : w->c1_w0;
  return conv ? w->c2_wm[m - 1] : w->c1_wm[m - 1];
}

void zp_add_so2_weights(const zp_plan *p, const zp_weights *w, void *packed, float *scales,
                        ZpMaxList &maxima, ZpPrepList &prep, bool transposes) {
  prep.transposes = transposes;
  for (int conv = 0; conv < 2; ++conv)
    for (int m = 0; m < p->n_blocks; ++m) {
      const int out = conv ? p->c2_out[m] : p->c1_out[m], in = conv ? p->c2_in[m] : p->c1_in[m];
      const float *src = block_weight(w, conv, m);
      float *slot = scales + 2 * (conv * (ZP_MAX_L + 1) + m);
      // one power-of-two scale per weight block from its largest magnitude
      if (p->fp16) maxima.add(src, (int64_t)out * (m ? in / 2 : in), slot);
      prep.add(src, static_cast<uint16_t *>(packed) + (conv ? p->c2_woff[m] : p->c1_woff[m]), slot,
               (int64_t)out * in, out, in, in, m ? ZP_PREP_FOLDED : ZP_PREP_KEPT, p->planes, p->fp16);
    }
}

void zp_add_so2_grads(const zp_plan *p, const float *partials, int64_t split_stride,
                      const int *splits_c1, const int *splits_c2, const zp_weight_grads *gw,
                      ZpFinalList &list) {
  for (int conv = 0; conv < 2; ++conv)
    for (int m = 0; m < p->n_blocks; ++m) {
      float *dst = m == 0 ? (conv ? gw->c2_w0 : gw->c1_w0)
                          : (conv ? gw->c2_wm[m - 1] : gw->c1_wm[m - 1]);
      list.add(partials + (conv ? p->c2_goff[m] : p->c1_goff[m]), dst, split_stride,
               conv ? p->c2_out[m] : p->c1_out[m], conv ? p->c2_in[m] : p->c1_in[m],
               (conv ? splits_c2 : splits_c1)[m], m ? ZP_FIN_UNFOLD : ZP_FIN_SUM);
    }
}

int zp_launch_colsum(int64_t rows, int64_t cols, const ZpPlanes &a, float *out, float *scratch,
                     ZpFinalList &list, cudaStream_t st) {
  if (cols == 0) return ZP_OK;
  const int64_t nparts = zp_colsum_parts(rows, cols);
  if (nparts > 0) {
    const dim3 grid((unsigned)zp_ceil_div(cols, 256), (unsigned)nparts), block(32, 8);
    zp_launch(colsum_part_kernel, grid, block, 0, st, rows, cols, zp_colsum_rows(rows, cols), a,
              scratch);
    ZP_LAUNCH_CHECK("colsum_part_kernel");
  }
  list.add(scratch, out, cols, 1, (int)cols, (int)nparts, ZP_FIN_COLUMN);
  return ZP_OK;
}
