// Shared pieces of the per-edge rotate kernels: packed arithmetic, staging, plane stores.
#pragma once

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
// rotation entries of `edges` consecutive edges duplicated into shared memory
__device__ __forceinline__ void stage_dup(const float *__restrict__ rot, float2 *rot_s, int ld, int edges) {
  for (int i = threadIdx.x; i < ld * edges; i += blockDim.x) {
    const float v = rot[i];
    rot_s[i] = make_float2(v, v);
  }
}
