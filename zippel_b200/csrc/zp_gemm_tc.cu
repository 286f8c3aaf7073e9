// The SO(2) contraction on the Blackwell tensor cores (tcgen05 + TMEM + TMA), sm_100a only.
//
//     C[M, N] (fp32) = sum over plane pairs (pa, pb) of  A_pa[M, K] * B_pb[N, K]^T   (+ bias[n])
//
// Operands are bf16 "planes".  With one plane per operand this is a plain bf16 GEMM with fp32
// accumulation.  With three planes an fp32 value x is carried as x = x0 + x1 + x2 (each a
// bf16, x0 = rn(x), x1 = rn(x - x0), x2 = rn(x - x0 - x1)), and the six products
//     A0B0, A0B1, A1B0, A1B1, A0B2, A2B0
// (everything down to 2^-16 of the leading term) reproduce the fp32 product to ~2^-22 while
// staying on the bf16 pipe and keeping fp32's exponent range.  All planes of a k-block are
// loaded once and reused by the six MMAs.
//
// Accumulation accuracy.  The tensor core adds each k = 16 step into the fp32 accumulator with
// truncation, a bias of about 3e-8 of the accumulator per step (measured: relative error
// ~1e-9 * K for one product, 6.5e-9 * K when all six share an accumulator).  Two measures keep
// that below the fp32 budget: (1) the leading product A0B0 has its own TMEM accumulator and the
// five small products share a second one, whose truncation is 2^-8 smaller in absolute terms;
// (2) the contraction is cut into chunks of at most `kc` k-blocks, each accumulated in TMEM
// from zero and then added up in fp32 in the epilogue's registers (a tile is stored once), so
// the bias never grows beyond one chunk's length.  Long contractions (the weight
// gradients, which run over all edges) can also be split over CTAs: split s writes its own
// partial matrix C + s * split_stride, reduced afterwards in a fixed order.
//
// Structure: persistent CTAs (one per SM), 320 threads.
//   warp 0      TMA producer: one elected lane streams A/B plane tiles into a ring of stages
//   warp 1      allocates TMEM, then one elected lane issues tcgen05.mma and commits
//   warps 2..9  epilogue: tcgen05.ld the 128 x BN accumulator into registers, release TMEM,
//               then scale, add bias and store fp32 rows
// With one plane two TMEM accumulators (2 x 256 columns) let the epilogue of one tile overlap
// the main loop of the next; with three planes the 512 columns hold the leading and the small
// accumulator of one tile.  Tiles are ordered n-fastest so CTAs running side by side share one A row block
// (read from HBM once, then L2) while the weights stay L2 resident.
//
// Operand layouts in global memory (element strides, all multiples of 8 so TMA rows are 16-byte
// aligned):  K-major   X[p*plane + r*ld + k]   (rows r = m or n, contraction index fastest)
//            MN-major  X[p*plane + k*ld + r]   (used by the weight-gradient products, whose
//                                               contraction runs over edges)
// Shared-memory tiles use the 128-byte (BK = 64) or 64-byte (BK = 32) swizzle that TMA writes
// and the matrix descriptors name.  Every mbarrier wait is bounded: after ~2 s it records
// ZP_ERR_DEVICE_TIMEOUT in the status word, raises the CTA's abort flag and the CTA drains.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>

#include <cuda.h>
#include <cuda_bf16.h>

#include "zp_common.cuh"
#include "zp_share.cuh"

namespace {

constexpr int BM = 128;
constexpr int kTmemBuf = 256;          // TMEM columns per accumulator buffer
constexpr int kThreads = 320;            // producer warp, MMA warp, eight epilogue warps
constexpr uint64_t kWaitLimitNs = 2000000000ull;   // default bound of every device-side wait

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n"
      ".reg .pred px;\n"
      "elect.sync _|px, 0xFFFFFFFF;\n"
      "@px mov.s32 %0, 1;\n"
      "}\n"
      : "+r"(pred));
  return pred != 0;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  Returns false when the CTA is aborting (this wait or another one timed out).
// The clock is only looked at every 1024 failed polls (the first look starts the interval), so a
// wait that is satisfied quickly never pays for reading the global timer.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                          int *status, uint64_t limit_ns = kWaitLimitNs) {
  if (mbar_try_wait(bar, parity)) return true;
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 0x3ff) == 0) {
      if (*abort_flag) return false;
      const uint64_t now = globaltimer_ns();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > limit_ns) {
        *abort_flag = 1;
        atomicExch(status, (int)ZP_ERR_DEVICE_TIMEOUT);
        return false;
      }
    }
  }
  return true;
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0,
                                            int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0),
        "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void tcgen05_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor.
//   K-major tile  [rows][BK] with a BK*2-byte swizzle: 8-row groups are 8*BK*2 bytes apart (SBO).
//   MN-major tile [BK][64] with the 128-byte swizzle: 8 k-rows are 1024 bytes apart (SBO) and the
//   next 64 elements along M/N start `lbo_bytes` later (LBO).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes,
                                              uint32_t layout_type) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3fff);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;                       // descriptor version of this architecture
  d |= (uint64_t)layout_type << 61;             // 2 = 128-byte swizzle, 4 = 64-byte swizzle
  return d;
}

// One product of a launch.
struct GemmProb {
  CUtensorMap map_a, map_b, map_c;
  int M, N;
  int BN;                 // tile width, multiple of 16, <= 256
  int num_n, num_k;
  int ksplit, kb_per_split, kc;   // CTAs-level split of K; k-blocks per TMEM accumulation chunk
  int a_mn, b_mn;         // operand is MN-major
  const float *scale_a, *scale_b;   // device scalars multiplying the result (null = 1)
  float *absmax_out;      // device scalar: running max |C| of what this launch stores (or null)
  const float *bias;
};
// The products of one launch.  Independent products (the orders m of a convolution, input and weight
// gradients) share a launch when each alone would leave the device's last wave half empty: their
// tiles form one list that the persistent CTAs walk.
//
// Which units (CTAs, or CTA pairs) take which tiles is laid down by the host (share_out): units of one
// class, consecutive ones, take the same number of tiles of each product, side by side through the
// product's list.
struct GemmGroup {
  GemmProb p[ZP_GEMM_GROUP];
  int n, total;           // products, work items of all of them
  int classes;
  int unit0[kMaxClasses + 1];                  // first unit of each class, and the number of units
  int first[kMaxClasses][ZP_GEMM_GROUP];       // first tile of the class in the product's list
  int16_t count[kMaxClasses][ZP_GEMM_GROUP];   // tiles per unit
  int stages, stage_bytes;                     // ring of operand stages
  int b_tile;                                  // bytes of one plane of B in a stage
  int acc_bufs, small_off;                     // accumulators in flight; TMEM columns to the small one
  int fp16;               // operand planes are fp16 (else bf16)
  int *status;
  uint64_t wait_limit_ns; // bound of every mbarrier wait
  int unarmed;            // self-test: the producers load nothing, so the first wait runs out
  int rows_apart;         // short contractions: row tiles between two of a CTA (0: stretches)
  ZpEpilogue epi;         // work of the fused epilogues (mode 0: none; one product only)
};

// plane pairs; for three planes pair 0 is the leading product, pairs 1..5 the small ones
template <int P> struct Pairs;
template <> struct Pairs<1> {
  static constexpr int n = 1;
  __device__ static constexpr int a(int) { return 0; }
  __device__ static constexpr int b(int) { return 0; }
};
template <> struct Pairs<2> {
  static constexpr int n = 3;          // fp16 pair: h0 h0 | h0 h1, h1 h0
  __device__ static constexpr int a(int i) { return i == 2 ? 1 : 0; }
  __device__ static constexpr int b(int i) { return i == 1 ? 1 : 0; }
};
template <> struct Pairs<3> {
  static constexpr int n = 6;
  __device__ static constexpr int a(int i) { return i == 0 ? 0 : i == 1 ? 2 : i == 2 ? 0 : i == 3 ? 1 : i == 4 ? 1 : 0; }
  __device__ static constexpr int b(int i) { return i == 0 ? 0 : i == 1 ? 0 : i == 2 ? 2 : i == 3 ? 1 : i == 4 ? 0 : 1; }
};

// ---- epilogue through TMA stores ------------------------------------------------------------
// In TMEM a lane owns a row, so storing straight from the registers sends every lane of an
// instruction to a different output row: 32 separate 16-byte pieces per instruction, and the
// epilogue of a 128 x 256 tile costs ~8 000 store wavefronts.  Instead each epilogue warp writes
// 32 x 32 blocks into its own 4 KB of shared memory (128-byte rows under the 128-byte swizzle, the
// layout the tensor map names) and one lane hands the block to the TMA unit, which writes full
// lines and clips rows / columns beyond the matrix.  The accumulation chunks of a long contraction
// are added up in the epilogue's registers, so a tile is stored once.
constexpr int kEpiBlockBytes = 32 * 32 * 4;
constexpr int kEpiBytes = 8 * kEpiBlockBytes;                 // eight epilogue warps

__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, const void *src, int c0, int c1,
                                             int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() {            // shared source may be overwritten
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_all() {             // the writes themselves are done
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// One 32 x 32 block of the result on its way out.  v[j]: value at row `row0 + lane`, column n + j (scaled,
// no bias yet); `bias`: of column n + lane.  Columns past N are zero, since the operand rows they
// come from were filled with zeros; the TMA unit leaves them out, and rows past M.
__device__ __forceinline__ void store_block(const GemmProb &p, float (&v)[32], uint8_t *stage, int lane,
                                            int row0, int n, int split, bool has_bias, float bias,
                                            float &seen_max) {
  if (row0 >= p.M || n >= p.N) return;            // warp-uniform
  if (has_bias) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] += __shfl_sync(0xffffffffu, bias, j);
  }
  if (p.absmax_out && row0 + lane < p.M) {
    float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 32; ++j) m[j & 3] = fmaxf(m[j & 3], fabsf(v[j]));
    seen_max = fmaxf(seen_max, fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])));
  }
  if (lane == 0) bulk_wait_read();                // the block buffer is free again
  __syncwarp();
  // 128-byte swizzle: 16-byte chunk k of row r sits at chunk k ^ (r & 7)
#pragma unroll
  for (int k = 0; k < 8; ++k)
    *reinterpret_cast<float4 *>(stage + lane * 128 + ((k ^ (lane & 7)) << 4)) =
        make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    tma_store_3d(&p.map_c, stage, n, row0, split);
    bulk_commit();
  }
}

// ---- fused epilogues ------------------------------------------------------------------------
// A finished 32 x 32 block of the result sits in the warp's shared-memory stage in the layout
// above (row = edge, 16-byte chunk k of row r at chunk k ^ (r & 7)).  The fused epilogues read
// it back in a second assignment of lanes and consume it there, so the values never have to come
// back from HBM: the gate activation walks it row-wise (eight lanes share a row, coalesced
// loads of the gate scalars and 8-byte plane stores), the rotation back walks it column-wise
// (a lane owns one channel and runs over the block's edges in order).
__device__ __forceinline__ float fast_sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }

__device__ __forceinline__ void gate_block(const ZpEpilogue &f, const uint8_t *stage, int lane,
                                           int row0, int n, int M, int N, float inv,
                                           float &slope_max) {
  // Pass 1: request the gate scalars of all eight row groups (independent loads, one memory round
  // trip for the block).  Pass 2: activate and store.
  const int k = lane & 7, col = n + 4 * k;
  const int rq = col / f.width;
  const int r = f.row_first + rq, h = col - rq * f.width;
  const bool col_ok = col < N;
  const bool gated = r != 0;                      // row 0 (l = 0): x * sigmoid(x)
  const float *gcol = f.gate + (gated ? (f.row_l[r] - 1) * f.width + h : 0);
  float4 g[8];
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int row = row0 + it * 4 + (lane >> 3);
    g[it] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (gated && col_ok && row < M)
      g[it] = *reinterpret_cast<const float4 *>(gcol + (size_t)row * f.ld_gate);
  }
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int rr = it * 4 + (lane >> 3);
    const int row = row0 + rr;
    if (row < M && col_ok) {
      const float4 x = *reinterpret_cast<const float4 *>(stage + rr * 128 + ((k ^ (rr & 7)) << 4));
      const float4 q = gated ? g[it] : x;
      const float s0 = fast_sigmoid(q.x), s1 = fast_sigmoid(q.y), s2 = fast_sigmoid(q.z),
                  s3 = fast_sigmoid(q.w);
      const float o[4] = {x.x * s0, x.y * s1, x.z * s2, x.w * s3};
      if (gated)
        slope_max = fmaxf(slope_max, fmaxf(fmaxf(s0 * (1.f - s0), s1 * (1.f - s1)),
                                           fmaxf(s2 * (1.f - s2), s3 * (1.f - s3))));
      zp_store_planes<4>(f.out, (int64_t)row * f.out.ld + col, o, inv);
    }
  }
}

// row_ptr[idx] for the rotate-back epilogue: lane d of the warp holds row_ptr[node0 + d] (fetched
// once per tile), anything further away comes from memory.  idx is warp-uniform.
__device__ __forceinline__ int row_ptr_at(const ZpEpilogue &f, int idx, int node0, int rp_l) {
  const int d = idx - node0;
  return (d >= 0 && d < 32) ? __shfl_sync(0xffffffffu, rp_l, d) : f.row_ptr[idx];
}

constexpr int kMaxNj = 2 * ZP_MAX_L + 1;

// node: the node of edge row0 (from find_node)
__device__ __forceinline__ void rotate_back_block(const ZpEpilogue &f, const uint8_t *stage, int lane,
                                                  int row0, int n, int M, int N, int node,
                                                  const int node0, const int rp_l) {
  const int col = n + lane;
  const bool col_ok = col < N;
  const int cq = col_ok ? col : n;               // lanes beyond the matrix shadow column n
  const int rq = cq / f.width;
  const int r = f.row_first + rq, c = cq - rq * f.width;
  const int off = f.rot_off[r];
  const int nj = 2 * f.row_l[r] + 1;
  const int njmax = __reduce_max_sync(0xffffffffu, nj);
  const int row_end = min(row0 + 32, M);
  const size_t slab = (size_t)f.nnz * f.width;
  // Usual case: the block's 32 columns lie in one m' row, so every lane needs the same rotation
  // entries.  Lane i then fetches the envelope and the row's 2l+1 entries of EDGE row0 + i (all
  // requests in flight together: one memory round trip per block) and the edge loop broadcasts
  // them with shuffles.  Otherwise every lane reads its own row's entries edge by edge.
  const bool one_row = __all_sync(0xffffffffu, r == __shfl_sync(0xffffffffu, r, 0));
  float env_l = 0.f, rot_l[kMaxNj];
#pragma unroll
  for (int j = 0; j < kMaxNj; ++j) rot_l[j] = 0.f;
  if (one_row && row0 + lane < row_end) {
    const int ei = row0 + lane;
    env_l = f.env[ei];
    const float *re = f.rot + (size_t)ei * f.rot_ld + f.row_off[r];
#pragma unroll
    for (int j = 0; j < kMaxNj; ++j)
      if (j < nj) rot_l[j] = re[j];
  }
  int e = row0;
  while (e < row_end) {
    int next = row_ptr_at(f, node + 1, node0, rp_l);
    while (node + 1 < f.n_nodes && next <= e) {  // nodes without edges
      ++node;
      next = row_ptr_at(f, node + 1, node0, rp_l);
    }
    const bool is_head = row_ptr_at(f, node, node0, rp_l) == e;
    int stop = min(next, row_end);
    if (stop <= e) stop = row_end;               // offsets that do not cover the edges: never spin
    float acc[kMaxNj];
#pragma unroll
    for (int j = 0; j < kMaxNj; ++j) acc[j] = 0.f;
    if (one_row) {
#pragma unroll 4
      for (; e < stop; ++e) {
        const int i = e - row0;
        const float yv = __shfl_sync(0xffffffffu, env_l, i) *
                         *reinterpret_cast<const float *>(stage + i * 128 + (((lane >> 2) ^ (i & 7)) << 4) +
                                                          ((lane & 3) << 2));
#pragma unroll
        for (int j = 0; j < kMaxNj; ++j) {
          if (j >= njmax) break;                 // warp-uniform
          acc[j] = fmaf(__shfl_sync(0xffffffffu, rot_l[j], i), yv, acc[j]);
        }
      }
    } else {
#pragma unroll 2
      for (; e < stop; ++e) {
        const int i = e - row0;
        const float yv = f.env[e] * *reinterpret_cast<const float *>(
                                        stage + i * 128 + (((lane >> 2) ^ (i & 7)) << 4) + ((lane & 3) << 2));
        const float *re = f.rot + (size_t)e * f.rot_ld + f.row_off[r];
#pragma unroll
        for (int j = 0; j < kMaxNj; ++j) {
          if (j >= njmax) break;                 // warp-uniform
          if (j < nj) acc[j] = fmaf(re[j], yv, acc[j]);
        }
      }
    }
    float *out = (is_head ? f.head + (size_t)node * slab : f.cont + (size_t)(row0 >> 5) * slab) +
                 (size_t)off * f.width + c;
    if (col_ok) {
#pragma unroll
      for (int j = 0; j < kMaxNj; ++j)
        if (j < nj) out[(size_t)j * f.width] = acc[j];
    }
  }
}

// v[b][j]: value at row `row0 + lane`, column `n0 + col_lo + 32 b + j` (scaled, no bias yet).
template <int EPI>
__device__ __forceinline__ void epilogue_fused(const GemmProb &p, const ZpEpilogue &epi,
                                               float (&v)[4][32], uint8_t *stage, int lane, int row0,
                                               int n0, int col_lo, int col_hi, const float *bias,
                                               float &seen_max, float &slope_max, int node,
                                               int rp_l) {
  if (row0 >= p.M) return;
  const bool row_ok = row0 + lane < p.M;
  const float inv = EPI == ZP_EPI_GATE ? zp_inv_scale(epi.out) : 1.f;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const int cc = col_lo + 32 * b;
    if (cc >= col_hi) continue;                   // warp-uniform
    const int n = n0 + cc;
    if (n >= p.N) continue;
    if (epi.store_c && lane == 0) bulk_wait_read();   // the TMA store of the previous block
    __syncwarp();                                 // ... and every lane's reads of it are done
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float4 o = make_float4(v[b][4 * k], v[b][4 * k + 1], v[b][4 * k + 2], v[b][4 * k + 3]);
      const int c = n + 4 * k;
      if (bias) {
        o.x += c < p.N ? bias[c] : 0.f;
        o.y += c + 1 < p.N ? bias[c + 1] : 0.f;
        o.z += c + 2 < p.N ? bias[c + 2] : 0.f;
        o.w += c + 3 < p.N ? bias[c + 3] : 0.f;
      }
      if (row_ok) {
        float m = c < p.N ? fabsf(o.x) : 0.f;
        m = fmaxf(m, c + 1 < p.N ? fabsf(o.y) : 0.f);
        m = fmaxf(m, c + 2 < p.N ? fabsf(o.z) : 0.f);
        m = fmaxf(m, c + 3 < p.N ? fabsf(o.w) : 0.f);
        seen_max = fmaxf(seen_max, m);
      }
      *reinterpret_cast<float4 *>(stage + lane * 128 + ((k ^ (lane & 7)) << 4)) = o;
    }
    if (epi.store_c) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        tma_store_3d(&p.map_c, stage, n, row0, 0);
        bulk_commit();
      }
    } else {
      __syncwarp();
    }
    if (EPI == ZP_EPI_GATE) gate_block(epi, stage, lane, row0, n, p.M, p.N, inv, slope_max);
    else rotate_back_block(epi, stage, lane, row0, n, p.M, p.N, node, node, rp_l);
  }
}

// Shared memory of the general kernels: operand stages, control words (barriers, TMEM slot, abort
// flag), store blocks of the epilogue, and 1 KB of alignment slack.  A launch cuts the operand space into
// as many stages as its widest tile leaves room for: 160-wide tiles of three planes have three instead of the
// two that 256-wide ones have.
constexpr int kMaxStages = 8;
constexpr int kSmemTotal = 232448;
constexpr int kTileBytes = kSmemTotal - 2048 - kEpiBytes;
constexpr int kEpiOffset = kTileBytes + 1024;
static_assert(kTileBytes % 1024 == 0 && 8 * (2 * kMaxStages + 4) + 16 <= 1024, "control words fit in one KB");

// place in the ring of stages
struct Ring {
  int s = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next(int stages) {
    if (++s == stages) { s = 0; phase ^= 1; }
  }
};

// Accumulation unit `n` of a CTA: which of the accumulators it has, and the parity of its round.
struct AccUnit {
  int buf;
  uint32_t parity;
  __device__ __forceinline__ AccUnit(uint32_t n, bool two) : buf(two ? n & 1 : 0), parity((two ? n >> 1 : n) & 1) {}
};

// One unit of work of a CTA (or CTA pair): a product, an output tile of it, a K split and its
// k-block range.
struct Work {
  int prob, m0, n0, split, kb0, kb1;
};
// A unit's way through its share of the tiles.
struct Walk {
  int cls = 0, prob = 0, j = -1, unit;
  __device__ __forceinline__ Walk(const GemmGroup &g, int u) {
    while (cls + 1 < g.classes && u >= g.unit0[cls + 1]) ++cls;
    unit = u - g.unit0[cls];
  }
  __device__ __forceinline__ bool next(const GemmGroup &g) {
    ++j;
    while (prob < g.n && j >= g.count[cls][prob]) { ++prob; j = 0; }
    return prob < g.n;
  }
  template <int TM>
  __device__ __forceinline__ Work tile(const GemmGroup &g) const {
    Work x;
    x.prob = prob;
    const GemmProb &p = g.p[prob];
    const int w = g.first[cls][prob] + j * (g.unit0[cls + 1] - g.unit0[cls]) + unit;
    x.split = w % p.ksplit;
    const int tile = w / p.ksplit;
    x.m0 = (tile / p.num_n) * TM;
    x.n0 = (tile % p.num_n) * p.BN;
    x.kb0 = x.split * p.kb_per_split;
    x.kb1 = min(p.num_k, x.kb0 + p.kb_per_split);
    return x;
  }
};
// Columns of a tile that an epilogue warp drains: the tile's 32-column blocks are dealt to two warps
__device__ __forceinline__ int half_columns(int BN) { return (BN / 2 + 31) & ~31; }
__device__ __forceinline__ void prefetch_maps(const GemmGroup &g) {
  for (int i = 0; i < g.n; ++i) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&g.p[i].map_a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&g.p[i].map_b)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&g.p[i].map_c)) : "memory");
  }
}
// instruction descriptor: fp32 accumulators, operand format and majorness, tile shape
__device__ __forceinline__ uint32_t instr_desc(const GemmGroup &g, const GemmProb &p, int tile_m) {
  const uint32_t fmt = g.fp16 ? 0u : 1u;      // operand format field: 0 = f16, 1 = bf16
  return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.a_mn ? 1 : 0) << 15) |
         ((uint32_t)(p.b_mn ? 1 : 0) << 16) | ((uint32_t)(p.BN >> 3) << 17) | ((uint32_t)(tile_m >> 4) << 24);
}

// What an epilogue warp carries from tile to tile: the largest magnitude it stored of the current
// product, handed over when the product changes.
struct MaxTracker {
  float *out = nullptr;
  float seen = 0.f;
  __device__ __forceinline__ void flush(int lane) {
    if (out) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) seen = fmaxf(seen, __shfl_xor_sync(0xffffffffu, seen, o));
      if (lane == 0 && seen > 0.f) zp_atomic_absmax(out, seen);
    }
    seen = 0.f;
  }
  __device__ __forceinline__ void follow(float *next, int lane) {
    if (next != out) {
      flush(lane);
      out = next;
    }
  }
};

// 32 columns of the accumulator(s) at `taddr` into v: sixteen of them at a time (a slice of 128 values
// per thread leaves little room), both accumulators' loads in flight before one wait
template <int P>
__device__ __forceinline__ void read_block(float (&v)[32], uint32_t taddr, int small_off, float out_scale) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t r[16], r2[16];
    tmem_ld16(taddr + 16 * h, r);
    if (P != 1) tmem_ld16(taddr + small_off + 16 * h, r2);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float a = __uint_as_float(r[j]);
      if (P != 1) a += __uint_as_float(r2[j]);
      v[16 * h + j] = a * out_scale;
    }
  }
}
// The accumulator slice of a tile's first chunk (this warp's 32 rows, columns col_lo .. col_hi) into v
template <int P>
__device__ __forceinline__ void read_accumulator(float (&v)[4][32], uint32_t t_row, int small_off,
                                                 int col_lo, int col_hi, float out_scale) {
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if (col_lo + 32 * b < col_hi)         // warp-uniform
      read_block<P>(v[b], t_row + col_lo + 32 * b, small_off, out_scale);
}
// ... and of a later chunk, added to it (all of v is live here: eight columns at a time)
template <int P>
__device__ __forceinline__ void add_accumulator(float (&v)[4][32], uint32_t t_row, int small_off,
                                                int col_lo, int col_hi, float out_scale) {
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const int cc = col_lo + 32 * b;
    if (cc < col_hi) {
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        uint32_t r[8], r2[8];
        tmem_ld8(t_row + cc + 8 * h, r);
        if (P != 1) tmem_ld8(t_row + small_off + cc + 8 * h, r2);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float a = __uint_as_float(r[j]);
          if (P != 1) a += __uint_as_float(r2[j]);
          v[b][8 * h + j] = fmaf(a, out_scale, v[b][8 * h + j]);
        }
      }
    }
  }
}

template <int P, int BK, int EPI>
__device__ __forceinline__ void gemm_tc_body(const GemmGroup &g) {
  constexpr int kATile = BM * BK * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~(uintptr_t)1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + kTileBytes);
  uint64_t *empty = full + kMaxStages;
  uint64_t *tmem_full = empty + kMaxStages;
  uint64_t *tmem_empty = tmem_full + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  if (threadIdx.x == 0) {
    prefetch_maps(g);
    for (int s = 0; s < g.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], 8); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  zp_after_previous();                  // all of the above ran beside the kernel before
  const int stages = g.stages;
  const bool two_accs = P == 1 || g.acc_bufs == 2;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (!g.unarmed && elect_one()) {
      Ring ring;
      bool ok = true;
      for (Walk walk(g, blockIdx.x); ok && walk.next(g);) {
        const Work x = walk.tile<BM>(g);
        const GemmProb &p = g.p[x.prob];
        const uint32_t b_bytes = (uint32_t)p.BN * BK * 2;
        for (int kb = x.kb0; kb < x.kb1 && ok; ++kb, ring.next(stages)) {
          const int s = ring.s;
          ok = mbar_wait(&empty[s], ring.phase ^ 1, abort_flag, g.status, g.wait_limit_ns);
          if (!ok) break;
          uint8_t *st = smem + (size_t)s * g.stage_bytes;
          mbar_expect_tx(&full[s], P * (kATile + b_bytes));
          const int k0 = kb * BK;
#pragma unroll
          for (int pl = 0; pl < P; ++pl) {
            uint8_t *ta = st + pl * kATile, *tb = st + P * kATile + pl * g.b_tile;
            if (!p.a_mn) {
              tma_load_3d(ta, &p.map_a, &full[s], k0, x.m0, pl);
            } else {                      // two 64-wide column blocks of [BK][64]
              tma_load_3d(ta, &p.map_a, &full[s], x.m0, k0, pl);
              tma_load_3d(ta + BK * 128, &p.map_a, &full[s], x.m0 + 64, k0, pl);
            }
            if (!p.b_mn) {
              tma_load_3d(tb, &p.map_b, &full[s], k0, x.n0, pl);
            } else {
              for (int nb = 0; nb < p.BN; nb += 64)
                tma_load_3d(tb + (nb / 64) * BK * 128, &p.map_b, &full[s], x.n0 + nb, k0, pl);
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      constexpr uint32_t kLayout = BK == 64 ? 2u : 4u;
      const int b_tile = g.b_tile;
      uint32_t unit = 0;
      Ring ring;
      bool ok = true;
      for (Walk walk(g, blockIdx.x); ok && walk.next(g);) {
        const Work x = walk.tile<BM>(g);
        const GemmProb &p = g.p[x.prob];
        const uint32_t idesc = instr_desc(g, p, BM);
        for (int c0 = x.kb0; c0 < x.kb1 && ok; c0 += p.kc, ++unit) {
          const int c1 = min(x.kb1, c0 + p.kc);
          const AccUnit acc(unit, two_accs);
          const int buf = acc.buf;
          ok = mbar_wait(&tmem_empty[buf], acc.parity ^ 1, abort_flag, g.status, g.wait_limit_ns);
          if (!ok) break;
          tcgen05_fence_after();
          const uint32_t d_main = tmem_base + (uint32_t)buf * kTmemBuf;
          const uint32_t d_small = d_main + g.small_off;
          for (int kb = c0; kb < c1 && ok; ++kb, ring.next(stages)) {
            const int s = ring.s;
            ok = mbar_wait(&full[s], ring.phase, abort_flag, g.status, g.wait_limit_ns);
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t sa = smem_u32(smem + (size_t)s * g.stage_bytes);
            const uint32_t sb = sa + P * kATile;
#pragma unroll
            for (int ks = 0; ks < BK / 16; ++ks) {
#pragma unroll
              for (int q = 0; q < Pairs<P>::n; ++q) {
                const uint32_t ta = sa + Pairs<P>::a(q) * kATile;
                const uint32_t tb = sb + Pairs<P>::b(q) * b_tile;
                // K-major: 32 bytes along the swizzled row per k-step of 16
                // MN-major: 16 k-rows of 128 bytes per k-step
                const uint64_t da = p.a_mn ? make_desc(ta + ks * 2048, BK * 128, 1024, 2u)
                                           : make_desc(ta + ks * 32, 16, 8 * BK * 2, kLayout);
                const uint64_t db = p.b_mn ? make_desc(tb + ks * 2048, BK * 128, 1024, 2u)
                                           : make_desc(tb + ks * 32, 16, 8 * BK * 2, kLayout);
                const bool first_step = kb == c0 && ks == 0;
                if (q == 0) umma_bf16(d_main, da, db, idesc, first_step ? 0u : 1u);
                else umma_bf16(d_small, da, db, idesc, (first_step && q == 1) ? 0u : 1u);
              }
            }
            tcgen05_commit(&empty[s]);          // stage reusable once these MMAs have read it
          }
          if (ok) tcgen05_commit(&tmem_full[buf]);
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (warps 2..9)
    // Eight warps: warp w reads TMEM lane quarter w % 4 (the only one it may access) and column
    // half (w - 2) / 4.  A warp first pulls its whole 32 x 128 slice of the accumulator(s) into
    // registers and releases TMEM, so the next tile's MMAs start while it scales and stores.
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    uint8_t *epi_stage = smem + kEpiOffset + (warp - 2) * kEpiBlockBytes;
    uint32_t unit = 0;
    bool ok = true;
    float slope_max = 0.f;
    MaxTracker maxima;
    for (Walk walk(g, blockIdx.x); ok && walk.next(g);) {
      const Work x = walk.tile<BM>(g);
      const GemmProb &p = g.p[x.prob];
      const int row0 = x.m0 + q * 32;
      const int hc = half_columns(p.BN), col_lo = half * hc, col_hi = half ? p.BN : hc;
      const float *bias = x.split == 0 ? p.bias : nullptr;
      const float out_scale = (p.scale_a ? *p.scale_a : 1.f) * (p.scale_b ? *p.scale_b : 1.f);
      maxima.follow(p.absmax_out, lane);
      // the node of the warp's first edge and the offsets of the 32 nodes from there on, fetched
      // while the tile is still being formed
      int node = 0, rp_l = 0;
      if (EPI == ZP_EPI_ROTATE_BACK && row0 < p.M) {
        node = g.epi.block_node[row0 >> 5];
        rp_l = g.epi.row_ptr[min(node + lane, g.epi.n_nodes)];
      }
      float bias_l[4];
      if constexpr (EPI == ZP_EPI_NONE) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int c = x.n0 + col_lo + 32 * b + lane;
          bias_l[b] = bias && c < p.N ? bias[c] : 0.f;
        }
      }
      // wait for accumulation unit `unit`; where its columns stand
      auto finished = [&](int buf) {
        ok = mbar_wait(&tmem_full[buf], AccUnit(unit, two_accs).parity, abort_flag, g.status, g.wait_limit_ns);
        ok = __all_sync(0xffffffffu, ok);
        tcgen05_fence_after();
        return tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)buf * kTmemBuf;
      };
      auto release = [&](int buf) {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[buf]);
        ++unit;
      };
      float v[4][32];
      if constexpr (EPI == ZP_EPI_NONE && P == 1) {
        // One plane: the next tile has the other buffer, so the slice leaves block by block.  This is what
        // bounds the short contractions (256 x 256 tiles of K = 1024: 9.0 us, of them 5.8 MMAs; 10.2
        // with the whole slice read first and every column checked against N).
        if (x.kb1 - x.kb0 <= p.kc) {
          const int buf = AccUnit(unit, two_accs).buf;
          const uint32_t t_row = finished(buf);
          if (!ok) break;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int cc = col_lo + 32 * b;
            if (cc < col_hi) read_block<P>(v[0], t_row + cc, 0, out_scale);
            if (b == 3) release(buf);
            if (cc < col_hi)
              store_block(p, v[0], epi_stage, lane, row0, x.n0 + cc, x.split, bias != nullptr, bias_l[b],
                          maxima.seen);
          }
          continue;
        }
      }
      for (int c0 = x.kb0; c0 < x.kb1 && ok; c0 += p.kc) {
        const int buf = AccUnit(unit, two_accs).buf;
        const uint32_t t_row = finished(buf);
        if (!ok) break;
        if (c0 == x.kb0) read_accumulator<P>(v, t_row, g.small_off, col_lo, col_hi, out_scale);
        else add_accumulator<P>(v, t_row, g.small_off, col_lo, col_hi, out_scale);
        release(buf);                       // the slice is in registers now
      }
      if (!ok) break;
      if constexpr (EPI != ZP_EPI_NONE) {
        epilogue_fused<EPI>(p, g.epi, v, epi_stage, lane, row0, x.n0, col_lo, col_hi, bias, maxima.seen,
                            slope_max, node, rp_l);
      } else {
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (col_lo + 32 * b < col_hi)
            store_block(p, v[b], epi_stage, lane, row0, x.n0 + col_lo + 32 * b, x.split, bias != nullptr,
                        bias_l[b], maxima.seen);
      }
    }
    if (lane == 0) bulk_wait_all();                        // this warp's stores are done
    maxima.flush(lane);
    if (EPI == ZP_EPI_GATE && g.epi.slope_max) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) slope_max = fmaxf(slope_max, __shfl_xor_sync(0xffffffffu, slope_max, o));
      if (lane == 0 && slope_max > 0.f) zp_atomic_absmax(g.epi.slope_max, slope_max);
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                 : "memory");
  }
}

template <int P, int BK>
__global__ void __launch_bounds__(kThreads, 1) gemm_tc_kernel(const __grid_constant__ GemmGroup g) {
  gemm_tc_body<P, BK, ZP_EPI_NONE>(g);
}
// the same contraction with a fused epilogue (the epilogue warps hold more live values)
template <int P, int BK, int EPI>
__global__ void __launch_bounds__(kThreads, 1) gemm_tc_fused_kernel(const __grid_constant__ GemmGroup g) {
  gemm_tc_body<P, BK, EPI>(g);
}

// ---- short contractions -------------------------------------------------------------------
//
// With at most 256 / P operand columns a product is bound by its output stores (the last layer of the
// radial MLP writes 12 KB per edge and reads 0.5), and a tile's main loop is over before a pipeline
// of k-blocks has filled.  Here a CTA keeps the whole K x 128 block of B in shared memory and
// walks the row tiles under it: only A streams (1.5 tiles ahead), two accumulators alternate in
// TMEM, and sixteen epilogue warps take one 32 x 32 block of a tile each (eight with two blocks
// took 6 % longer: the way through TMEM, registers and shared memory is a chain of latencies).
// All columns of the same rows are walked at the same time, by CTAs that keep to one column, so
// that whole rows of C leave L2 together; where that would leave more than a tenth of the SMs out, CTAs
// take contiguous stretches of the (column, row) tiles, columns slowest, and change their B on the way.
// 60 000 x 128 -> 3072, two fp16 planes: 183 us, 302 with both operands streamed in 128 x 256 tiles.
constexpr int kShortBN = 128, kShortBK = 64;
constexpr int kShortEpiWarps = 16, kShortThreads = 64 + 32 * kShortEpiWarps;
template <int P>
struct ShortLayout {
  static constexpr int kTile = 128 * kShortBK * 2;             // one plane of a k-block of A or B
  static constexpr int kMaxBlocks = 4 / P;                     // k-blocks of B that fit
  static constexpr int kStages = 6 / P;
  static constexpr int kB = 0, kA = kMaxBlocks * P * kTile;
  static constexpr int kControl = kA + kStages * P * kTile;
  static constexpr int kEpiOffset = kControl + 1024;
  static constexpr int kTotal = kEpiOffset + kShortEpiWarps * kEpiBlockBytes + 1024;
};

template <int P>
__global__ void __launch_bounds__(kShortThreads, 1)
gemm_tc_short_kernel(const __grid_constant__ GemmGroup g) {
  using L = ShortLayout<P>;
  constexpr int STAGES = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~(uintptr_t)1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::kControl);
  uint64_t *empty = full + STAGES;
  uint64_t *b_full = empty + STAGES, *b_empty = b_full + 1;
  uint64_t *tmem_full = b_empty + 1, *tmem_empty = tmem_full + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const GemmProb &p = g.p[0];
  const int num_m = (p.M + BM - 1) / BM, num_k = p.num_k;
  const int step = g.rows_apart ? g.rows_apart : 1;
  int w0 = (int)((int64_t)g.total * blockIdx.x / gridDim.x);
  int w1 = (int)((int64_t)g.total * (blockIdx.x + 1) / gridDim.x);
  if (g.rows_apart) {
    const int first = blockIdx.x % p.num_n * num_m;
    w0 = first + blockIdx.x / p.num_n;
    w1 = first + num_m;
  }

  if (threadIdx.x == 0) {
    prefetch_maps(g);
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(b_full, 1);
    mbar_init(b_empty, 1);
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], kShortEpiWarps); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  zp_after_previous();                  // all of the above ran beside the kernel before

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (!g.unarmed && elect_one()) {
      const uint32_t b_bytes = (uint32_t)p.BN * kShortBK * 2;
      uint32_t it = 0, columns = 0;
      int col = -1;
      bool ok = true;
      for (int w = w0; w < w1 && ok; w += step) {
        if (w / num_m != col) {
          col = w / num_m;
          ok = mbar_wait(b_empty, (columns & 1) ^ 1, abort_flag, g.status, g.wait_limit_ns);
          if (!ok) break;
          ++columns;
          mbar_expect_tx(b_full, (uint32_t)(num_k * P) * b_bytes);
          for (int kb = 0; kb < num_k; ++kb)
#pragma unroll
            for (int pl = 0; pl < P; ++pl)
              tma_load_3d(smem + L::kB + (kb * P + pl) * L::kTile, &p.map_b, b_full, kb * kShortBK,
                          col * p.BN, pl);
        }
        const int m0 = (w - col * num_m) * BM;
        for (int kb = 0; kb < num_k; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, abort_flag, g.status, g.wait_limit_ns);
          if (!ok) break;
          mbar_expect_tx(&full[s], P * L::kTile);
#pragma unroll
          for (int pl = 0; pl < P; ++pl)
            tma_load_3d(smem + L::kA + (s * P + pl) * L::kTile, &p.map_a, &full[s], kb * kShortBK, m0, pl);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      const uint32_t idesc = instr_desc(g, p, BM);
      uint32_t it = 0, columns = 0, unit = 0;
      int col = -1;
      bool ok = true;
      for (int w = w0; w < w1 && ok; w += step, ++unit) {
        if (w / num_m != col) {
          col = w / num_m;
          ok = mbar_wait(b_full, columns & 1, abort_flag, g.status, g.wait_limit_ns);
          if (!ok) break;
          ++columns;
        }
        const uint32_t buf = unit & 1;
        ok = mbar_wait(&tmem_empty[buf], ((unit / 2) & 1) ^ 1, abort_flag, g.status, g.wait_limit_ns);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t d_main = tmem_base + buf * 256u, d_small = d_main + 128u;
        for (int kb = 0; kb < num_k; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(&full[s], (it / STAGES) & 1, abort_flag, g.status, g.wait_limit_ns);
          if (!ok) break;
          tcgen05_fence_after();
          const uint32_t sa = smem_u32(smem + L::kA + s * P * L::kTile);
          const uint32_t sb = smem_u32(smem + L::kB + kb * P * L::kTile);
#pragma unroll
          for (int ks = 0; ks < kShortBK / 16; ++ks) {
#pragma unroll
            for (int q = 0; q < Pairs<P>::n; ++q) {
              const uint64_t da = make_desc(sa + Pairs<P>::a(q) * L::kTile + ks * 32, 16, 1024, 2u);
              const uint64_t db = make_desc(sb + Pairs<P>::b(q) * L::kTile + ks * 32, 16, 1024, 2u);
              const bool first_step = kb == 0 && ks == 0;
              if (q == 0) umma_bf16(d_main, da, db, idesc, first_step ? 0u : 1u);
              else umma_bf16(d_small, da, db, idesc, (first_step && q == 1) ? 0u : 1u);
            }
          }
          tcgen05_commit(&empty[s]);
        }
        if (!ok) break;
        if (w + step < w1 && (w + step) / num_m != col) tcgen05_commit(b_empty);    // B has been read
        tcgen05_commit(&tmem_full[buf]);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (warps 2..17)
    // warp w: TMEM lane quarter w % 4, columns 32 ((w - 2) / 4) and on
    const int q = warp & 3, first = (warp - 2) / 4 * 32;
    uint8_t *stage = smem + L::kEpiOffset + (warp - 2) * kEpiBlockBytes;
    const float out_scale = (p.scale_a ? *p.scale_a : 1.f) * (p.scale_b ? *p.scale_b : 1.f);
    float bias = 0.f;                    // of column `lane` of the block
    MaxTracker maxima;
    maxima.follow(p.absmax_out, lane);
    uint32_t unit = 0;
    int col = -1;
    for (int w = w0; w < w1; w += step, ++unit) {
      if (w / num_m != col) {
        col = w / num_m;
        const int c = col * p.BN + first + lane;
        bias = p.bias && c < p.N ? p.bias[c] : 0.f;
      }
      const uint32_t buf = unit & 1;
      bool ok = mbar_wait(&tmem_full[buf], (unit / 2) & 1, abort_flag, g.status, g.wait_limit_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256u + first;
      float v[32];
      {
        uint32_t r[2][16], r2[2][16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tmem_ld16(t_row + 16 * h, r[h]);
          if (P != 1) tmem_ld16(t_row + 128 + 16 * h, r2[h]);
        }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          float a = __uint_as_float(r[j / 16][j % 16]);
          if (P != 1) a += __uint_as_float(r2[j / 16][j % 16]);
          v[j] = a * out_scale;
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[buf]);
      if (first < p.BN)                                   // warp-uniform
        store_block(p, v, stage, lane, (w - col * num_m) * BM + q * 32, col * p.BN + first, 0,
                    p.bias != nullptr, bias, maxima.seen);
    }
    if (lane == 0) bulk_wait_all();
    maxima.flush(lane);
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                 : "memory");
  }
}

// ---- CTA-pair variant ---------------------------------------------------------------------
//
// Two CTAs of a cluster (an SM pair) work on one 256 x BN tile with tcgen05.mma.cta_group::2:
// each CTA stages its own 128 rows of A and HALF of the B tile, and the pair's tensor cores read
// both halves, so a CTA pulls (128 + BN/2) operand rows per k-block from L2 instead of
// (128 + BN).  With two fp16 planes and three MMA passes per k-block the single-CTA kernel is
// limited by that operand feed; the pair is not.
//
// Roles per CTA are as above, except that only the even CTA of the pair (the leader) issues MMAs.
//   full[s]       leader's barrier; the leader's producer announces the bytes of BOTH CTAs and
//                 both producers' TMA loads complete on it (cta_group::2 loads)
//   empty[s]      one per CTA; the leader's tcgen05.commit releases the stage in both CTAs
//   tmem_full     one per CTA, signalled by the same kind of commit
//   tmem_empty    leader's barrier, 16 arrivals: the eight epilogue warps of each CTA
// TMEM holds rows 0..127 of the tile in the leader and rows 128..255 in its peer; each CTA's
// epilogue reads its own half.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\n"
               "barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}
// load into this CTA's shared memory, completing on a barrier of the pair's leader
__device__ __forceinline__ void tma_load_3d_pair(void *dst, const CUtensorMap *map,
                                                 uint32_t bar_cluster_addr, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0),
        "r"(c1), "r"(c2)
      : "memory");
}
// arrive on the barrier at this offset in both CTAs of the pair once the MMAs issued so far finish
__device__ __forceinline__ void tcgen05_commit_pair(uint64_t *bar) {
  const uint16_t both = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
      " [%0], %1;" ::"r"(smem_u32(bar)),
      "h"(both)
      : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

constexpr int BM2 = 256;               // rows of a pair's tile

template <int P, int BK, int EPI>
__device__ __forceinline__ void gemm_tc_pair_body(const GemmGroup &g) {
  constexpr int kATile = BM * BK * 2;                 // this CTA's 128 rows
  extern __shared__ uint8_t smem_raw[];
  // the dynamic shared window starts at the same offset in both CTAs, so does everything below
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~(uintptr_t)1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + kTileBytes);
  uint64_t *empty = full + kMaxStages;
  uint64_t *tmem_full = empty + kMaxStages;
  uint64_t *tmem_empty = tmem_full + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint32_t rank = cluster_ctarank();          // 0 = leader
  const int pair = blockIdx.x >> 1;

  if (threadIdx.x == 0) {
    prefetch_maps(g);
    for (int s = 0; s < g.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], 16); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  cluster_sync_all();                   // both CTAs' barriers exist before anything signals them
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();                   // both allocations exist before the leader's first MMA
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  zp_after_previous();                  // all of the above ran beside the kernel before
  const int stages = g.stages;
  const bool two_accs = P == 1 || g.acc_bufs == 2;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer (both CTAs)
    if (!g.unarmed && elect_one()) {
      Ring ring;
      bool ok = true;
      for (Walk walk(g, pair); ok && walk.next(g);) {
        const Work x = walk.tile<BM2>(g);
        const GemmProb &p = g.p[x.prob];
        const int half_n = p.BN >> 1;
        const uint32_t b_bytes = (uint32_t)half_n * BK * 2;
        const int m0 = x.m0 + (int)rank * BM, n0 = x.n0 + (int)rank * half_n;
        for (int kb = x.kb0; kb < x.kb1 && ok; ++kb, ring.next(stages)) {
          const int s = ring.s;
          ok = mbar_wait(&empty[s], ring.phase ^ 1, abort_flag, g.status, g.wait_limit_ns);
          if (!ok) break;
          uint8_t *st = smem + (size_t)s * g.stage_bytes;
          if (rank == 0) mbar_expect_tx(&full[s], 2 * P * (kATile + b_bytes));
          const uint32_t bar = map_to_cta(smem_u32(&full[s]), 0);
          const int k0 = kb * BK;
#pragma unroll
          for (int pl = 0; pl < P; ++pl) {
            uint8_t *ta = st + pl * kATile, *tb = st + P * kATile + pl * g.b_tile;
            if (!p.a_mn) {
              tma_load_3d_pair(ta, &p.map_a, bar, k0, m0, pl);
            } else {
              tma_load_3d_pair(ta, &p.map_a, bar, m0, k0, pl);
              tma_load_3d_pair(ta + BK * 128, &p.map_a, bar, m0 + 64, k0, pl);
            }
            if (!p.b_mn) {
              tma_load_3d_pair(tb, &p.map_b, bar, k0, n0, pl);
            } else {
              for (int nb = 0; nb < half_n; nb += 64)
                tma_load_3d_pair(tb + (nb / 64) * BK * 128, &p.map_b, bar, n0 + nb, k0, pl);
            }
          }
        }
      }
      // the leader's last stage releases must have landed here before this CTA may exit
      for (int j = 0; j < stages && ok; ++j, ring.next(stages))
        ok = mbar_wait(&empty[ring.s], ring.phase ^ 1, abort_flag, g.status, g.wait_limit_ns);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (leader only)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t kLayout = BK == 64 ? 2u : 4u;
      const int b_tile = g.b_tile;
      uint32_t unit = 0;
      Ring ring;
      bool ok = true;
      for (Walk walk(g, pair); ok && walk.next(g);) {
        const Work x = walk.tile<BM2>(g);
        const GemmProb &p = g.p[x.prob];
        const uint32_t idesc = instr_desc(g, p, BM2);
        for (int c0 = x.kb0; c0 < x.kb1 && ok; c0 += p.kc, ++unit) {
          const int c1 = min(x.kb1, c0 + p.kc);
          const AccUnit acc(unit, two_accs);
          const int buf = acc.buf;
          ok = mbar_wait(&tmem_empty[buf], acc.parity ^ 1, abort_flag, g.status, g.wait_limit_ns);
          if (!ok) break;
          tcgen05_fence_after();
          const uint32_t d_main = tmem_base + (uint32_t)buf * kTmemBuf;
          const uint32_t d_small = d_main + g.small_off;
          for (int kb = c0; kb < c1 && ok; ++kb, ring.next(stages)) {
            const int s = ring.s;
            ok = mbar_wait(&full[s], ring.phase, abort_flag, g.status, g.wait_limit_ns);
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t sa = smem_u32(smem + (size_t)s * g.stage_bytes);
            const uint32_t sb = sa + P * kATile;
#pragma unroll
            for (int ks = 0; ks < BK / 16; ++ks) {
#pragma unroll
              for (int q = 0; q < Pairs<P>::n; ++q) {
                const uint32_t ta = sa + Pairs<P>::a(q) * kATile;
                const uint32_t tb = sb + Pairs<P>::b(q) * b_tile;
                const uint64_t da = p.a_mn ? make_desc(ta + ks * 2048, BK * 128, 1024, 2u)
                                           : make_desc(ta + ks * 32, 16, 8 * BK * 2, kLayout);
                const uint64_t db = p.b_mn ? make_desc(tb + ks * 2048, BK * 128, 1024, 2u)
                                           : make_desc(tb + ks * 32, 16, 8 * BK * 2, kLayout);
                const bool first_step = kb == c0 && ks == 0;
                if (q == 0 || P == 1) umma_pair(d_main, da, db, idesc, first_step ? 0u : 1u);
                else umma_pair(d_small, da, db, idesc, (first_step && q == 1) ? 0u : 1u);
              }
            }
            tcgen05_commit_pair(&empty[s]);
          }
          if (ok) tcgen05_commit_pair(&tmem_full[buf]);
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (both CTAs)
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    uint8_t *epi_stage = smem + kEpiOffset + (warp - 2) * kEpiBlockBytes;
    uint32_t unit = 0;
    bool ok = true;
    float slope_max = 0.f;
    MaxTracker maxima;
    const uint32_t release_bar0 = map_to_cta(smem_u32(&tmem_empty[0]), 0);
    const uint32_t release_bar1 = map_to_cta(smem_u32(&tmem_empty[1]), 0);
    for (Walk walk(g, pair); ok && walk.next(g);) {
      const Work x = walk.tile<BM2>(g);
      const GemmProb &p = g.p[x.prob];
      const int row0 = x.m0 + (int)rank * BM + q * 32;
      const int hc = half_columns(p.BN), col_lo = half * hc, col_hi = half ? p.BN : hc;
      const float *bias = x.split == 0 ? p.bias : nullptr;
      const float out_scale = (p.scale_a ? *p.scale_a : 1.f) * (p.scale_b ? *p.scale_b : 1.f);
      maxima.follow(p.absmax_out, lane);
      // the node of the warp's first edge and the offsets of the 32 nodes from there on, fetched
      // while the tile is still being formed
      int node = 0, rp_l = 0;
      if (EPI == ZP_EPI_ROTATE_BACK && row0 < p.M) {
        node = g.epi.block_node[row0 >> 5];
        rp_l = g.epi.row_ptr[min(node + lane, g.epi.n_nodes)];
      }
      float bias_l[4];
      if constexpr (EPI == ZP_EPI_NONE) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int c = x.n0 + col_lo + 32 * b + lane;
          bias_l[b] = bias && c < p.N ? bias[c] : 0.f;
        }
      }
      // wait for accumulation unit `unit`; where its columns stand
      auto finished = [&](int buf) {
        ok = mbar_wait(&tmem_full[buf], AccUnit(unit, two_accs).parity, abort_flag, g.status, g.wait_limit_ns);
        ok = __all_sync(0xffffffffu, ok);
        tcgen05_fence_after();
        return tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)buf * kTmemBuf;
      };
      auto release = [&](int buf) {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(buf ? release_bar1 : release_bar0);
        ++unit;
      };
      float v[4][32];
      if constexpr (EPI == ZP_EPI_NONE && P == 1) {
        // One plane: the next tile has the other buffer, so the slice leaves block by block.  This is what
        // bounds the short contractions (256 x 256 tiles of K = 1024: 9.0 us, of them 5.8 MMAs; 10.2
        // with the whole slice read first and every column checked against N).
        if (x.kb1 - x.kb0 <= p.kc) {
          const int buf = AccUnit(unit, two_accs).buf;
          const uint32_t t_row = finished(buf);
          if (!ok) break;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int cc = col_lo + 32 * b;
            if (cc < col_hi) read_block<P>(v[0], t_row + cc, 0, out_scale);
            if (b == 3) release(buf);
            if (cc < col_hi)
              store_block(p, v[0], epi_stage, lane, row0, x.n0 + cc, x.split, bias != nullptr, bias_l[b],
                          maxima.seen);
          }
          continue;
        }
      }
      for (int c0 = x.kb0; c0 < x.kb1 && ok; c0 += p.kc) {
        const int buf = AccUnit(unit, two_accs).buf;
        const uint32_t t_row = finished(buf);
        if (!ok) break;
        if (c0 == x.kb0) read_accumulator<P>(v, t_row, g.small_off, col_lo, col_hi, out_scale);
        else add_accumulator<P>(v, t_row, g.small_off, col_lo, col_hi, out_scale);
        release(buf);                       // the slice is in registers now
      }
      if (!ok) break;
      if constexpr (EPI != ZP_EPI_NONE) {
        epilogue_fused<EPI>(p, g.epi, v, epi_stage, lane, row0, x.n0, col_lo, col_hi, bias, maxima.seen,
                            slope_max, node, rp_l);
      } else {
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (col_lo + 32 * b < col_hi)
            store_block(p, v[b], epi_stage, lane, row0, x.n0 + col_lo + 32 * b, x.split, bias != nullptr,
                        bias_l[b], maxima.seen);
      }
    }
    if (lane == 0) bulk_wait_all();                        // this warp's stores are done
    maxima.flush(lane);
    if (EPI == ZP_EPI_GATE && g.epi.slope_max) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) slope_max = fmaxf(slope_max, __shfl_xor_sync(0xffffffffu, slope_max, o));
      if (lane == 0 && slope_max > 0.f) zp_atomic_absmax(g.epi.slope_max, slope_max);
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();                   // neither CTA frees TMEM or exits while its peer still works
  if (warp == 1) {
    __syncwarp();
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                 : "memory");
  }
}

template <int P, int BK>
__global__ void __launch_bounds__(kThreads, 1) gemm_tc_pair_kernel(const __grid_constant__ GemmGroup g) {
  gemm_tc_pair_body<P, BK, ZP_EPI_NONE>(g);
}
template <int P, int BK, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_pair_fused_kernel(const __grid_constant__ GemmGroup g) {
  gemm_tc_pair_body<P, BK, EPI>(g);
}

// block_node[b] = the last node n with row_ptr[n] <= 32 b: the node of the first edge of 32-edge
// block b (row_ptr[0] = 0 and row_ptr[n_nodes] = E > 32 b)
__global__ void block_node_kernel(int64_t n_blocks, int n_nodes, const int32_t *__restrict__ row_ptr,
                                  int32_t *__restrict__ block_node) {
  zp_after_previous();
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_blocks) return;
  const int e = (int)(b * 32);
  int lo = 0, hi = n_nodes;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (row_ptr[mid] <= e) lo = mid; else hi = mid;
  }
  block_node[b] = lo;
}

// ---- host side ---------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// 3-d map over (inner, outer, plane) of a bf16 operand
int make_map(CUtensorMap *map, const void *base, uint64_t inner, uint64_t outer, uint64_t planes,
             uint64_t ld, uint64_t plane_stride, uint32_t box_inner, uint32_t box_outer,
             CUtensorMapSwizzle swz, int fp16) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return ZP_ERR_CUDA;
  const cuuint64_t dims[3] = {inner, outer, planes};
  const cuuint64_t strides[2] = {ld * 2, plane_stride * 2};
  const cuuint32_t box[3] = {box_inner, box_outer, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    zp_set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
    return ZP_ERR_CUDA;
  }
  return ZP_OK;
}

// 3-d map over (column, row, split) of the fp32 output, 32 x 32 boxes under the 128-byte swizzle
int make_map_c(CUtensorMap *map, float *C, uint64_t N, uint64_t M, uint64_t splits, uint64_t ldc,
               uint64_t split_stride) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return ZP_ERR_CUDA;
  const cuuint64_t dims[3] = {N, M, splits};
  const cuuint64_t strides[2] = {ldc * 4, (splits > 1 ? split_stride : ldc * M) * 4};
  const cuuint32_t box[3] = {32, 32, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, C, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    zp_set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled (output)");
    return ZP_ERR_CUDA;
  }
  return ZP_OK;
}

// Tile width: the multiple of `step` in [cap/2, cap] that wastes the fewest padded columns
// (ties: the widest); problems narrower than cap/2 get one tile.
int pick_bn(int64_t N, int cap, int step = 16) {
  if (N <= cap / 2) return (int)(zp_ceil_div(N, step) * step);
  int best = cap;
  int64_t best_pad = zp_ceil_div(N, cap) * cap;
  for (int bn = cap - step; bn >= cap / 2; bn -= step) {
    const int64_t pad = zp_ceil_div(N, bn) * bn;
    if (pad < best_pad) { best_pad = pad; best = bn; }
  }
  return best;
}

// The CTA-pair kernel serves all three formats unless the caller forces a kernel: variant 2 = single-CTA kernel,
// variant 3 = pair kernel, and of three planes variant 1, which only the single-CTA kernel has.
bool pair_enabled() {
  static int on = -1;
  if (on < 0) {
    const char *e = getenv("ZP_GEMM_PAIR");
    on = (e && e[0] == '0') ? 0 : 1;
  }
  return on == 1;
}
// whole 32-column store blocks; each CTA's share of an MN-major B tile comes in 64-wide blocks
int bn_step(const ZpGemmTc &g, int halves) { return g.b_mn ? 64 * halves : 32; }
int device_sms() {
  static std::atomic<int> known[64];               // asked for several times per launch
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && known[dev].load(std::memory_order_relaxed))
    return known[dev].load(std::memory_order_relaxed);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (dev >= 0 && dev < 64) known[dev].store(sms, std::memory_order_relaxed);
  return sms;
}
// Expected utilisation of the tensor pipes for one kernel choice and K split: padded-tile waste
// times the evenness of the last wave, with the pair's lighter operand feed counted as a gain.
double launch_score(const ZpGemmTc &g, bool pair, int splits) {
  const int64_t units = pair ? device_sms() / 2 : device_sms();
  const int tm = pair ? 256 : BM;
  const int bn = pair ? pick_bn(g.N, 256, g.b_mn ? 128 : 32) : pick_bn(g.N, 256, g.b_mn ? 64 : 32);
  const int64_t tiles_m = zp_ceil_div(g.M, tm), tiles_n = zp_ceil_div(g.N, bn);
  const double pad = (double)(g.M * g.N) / (double)(tiles_m * tm * tiles_n * bn);
  const int64_t items = tiles_m * tiles_n * splits;
  const double wave = (double)items / (double)(zp_ceil_div(items, units) * units);
  // one plane (one MMA pass per k-block) leans on the operand feed harder than two planes do
  const double feed = !pair ? 1.0 : g.planes == 1 ? 1.25 : 1.12;
  return pad * wave * feed * (1.0 - 0.004 * splits);
}
bool use_pair(const ZpGemmTc &g) {
  if (g.planes == 3 && g.variant == 1) return false;
  if (g.variant == 2) return false;
  if (g.variant == 3) return true;
  if (!pair_enabled()) return false;
  // short contractions leave the pair's cross-SM hand-offs exposed on every tile
  if (g.K < 512) return false;
  int s = g.ksplit < 1 ? 1 : g.ksplit;
  return launch_score(g, true, s) >= launch_score(g, false, s);
}

int pair_block_k(int planes) { return planes == 3 ? 32 : 64; }
int single_block_k(int planes, int variant) { return ((planes == 3 && variant != 1) || planes == 2) ? 32 : 64; }
int block_k(const ZpGemmTc &g) {
  return use_pair(g) ? pair_block_k(g.planes) : single_block_k(g.planes, g.variant);
}

// Split of the contraction in whole 64-deep steps, so that it does not depend on the kernel's k-block
void split_plan(const ZpGemmTc &g, int bk, int *ksplit, int *kbs, int *num_k) {
  const int steps = (int)zp_ceil_div(g.K, 64);
  int req = g.ksplit < 1 ? 1 : g.ksplit;
  if (req > steps) req = steps;
  const int per = (int)zp_ceil_div(steps, req);
  *ksplit = (int)zp_ceil_div(steps, per);
  *kbs = per * (64 / bk);
  *num_k = (int)zp_ceil_div(g.K, bk);
}

// One-time set-up of a kernel is per device (the raised dynamic shared-memory limit is an
// attribute of the function ON a device): remembered per device ordinal under a lock, since a
// plan may be used from several host threads.
constexpr int kMaxDevices = 64;
struct PerDevice {
  std::mutex lock;
  int value[kMaxDevices];
  bool done[kMaxDevices];
  PerDevice() { for (int i = 0; i < kMaxDevices; ++i) { value[i] = 0; done[i] = false; } }
};

bool fused_mode_ok(const ZpGemmTc &g, int bk) {
  if (!g.epi || g.epi->mode == ZP_EPI_NONE) return true;
  if (g.a_mn || g.b_mn || (g.planes != 1 && g.planes != 2)) return false;
  int ksplit, kbs, num_k;
  split_plan(g, bk, &ksplit, &kbs, &num_k);
  const int kc_elems = g.kc_elems > 0 ? g.kc_elems : 2048;
  const int kc = kc_elems / bk < 1 ? 1 : kc_elems / bk;
  return ksplit == 1 && kbs <= kc && (g.epi->width % 4) == 0;
}

// Time of a tile: its MMAs or its operands' way from L2 (38 bytes per clock and SM), whichever is longer, and what
// its epilogue adds.  It only has to rank shapes: 60 000 x 1280 -> 1152 in two planes takes 422 us in the pair
// kernel and 453 in the single one, in one plane 157 and 174.
double tile_cost(int planes, int halves, int bn, int steps, bool two_accs) {
  const int passes = planes == 1 ? 1 : planes == 2 ? 3 : 6;
  const double mma = 2.5 * passes * bn, feed = planes * 128.0 * (BM + bn / halves) / 38.0;
  const double main = steps * std::max(mma, feed), drain = 24.0 * bn;
  return (two_accs ? std::max(main, drain) + 0.1 * drain : main + 0.35 * drain) + (halves == 2 ? 900.0 : 600.0);
}

// bk: depth of a k-block; cap: widest tile
void plan_group(GroupPlan &pl, const ZpGemmTc *const *g, int n, bool pair, int bk, int cap, int units) {
  Shape shape[ZP_GEMM_GROUP];
  const int P = g[0]->planes, halves = pair ? 2 : 1, tile_m = pair ? 256 : BM;
  pl.pair = pair;
  pl.bk = bk;
  pl.halves = halves;
  pl.max_bn = 0;
  for (int i = 0; i < n; ++i) {
    const int step = bn_step(*g[i], halves);
    shape[i].bn = pick_bn(g[i]->N, std::max(cap / step, 1) * step, step);
    pl.max_bn = std::max(pl.max_bn, shape[i].bn);
  }
  const bool two_accs = P == 1 || pl.max_bn <= kTmemBuf / 2;
  for (int i = 0; i < n; ++i) {
    Shape &s = shape[i];
    split_plan(*g[i], bk, &s.ksplit, &s.kbs, &s.num_k);
    s.num_n = (int)zp_ceil_div(g[i]->N, s.bn);
    s.tiles = zp_ceil_div(g[i]->M, tile_m) * s.num_n * s.ksplit;
    s.cost = tile_cost(P, halves, s.bn, s.kbs * bk / 64, two_accs);
    int k = i;
    for (; k > 0 && shape[pl.order[k - 1]].cost < s.cost; --k) pl.order[k] = pl.order[k - 1];
    pl.order[k] = i;
  }
  for (int k = 0; k < n; ++k) pl.shape[k] = shape[pl.order[k]];
  share_out(pl, n, units);
}

// The plan of a launch.  `kernel`: 0 the single-CTA kernel, 1 the pair kernel, 2 whichever gets done first.
// Wide tiles live on fewer operand bytes and are taken wherever they go round: whole passes of 6 000 to 18 000
// edges took 4 to 7 % longer with tiles of at most 192 columns and 3 to 7 % with 128.  Where there are fewer tiles
// than units, narrower ones share the work out.
void plan_launch(GroupPlan &pl, const ZpGemmTc *const *g, int n, int kernel) {
  const int P = g[0]->planes, sms = device_sms();
  const bool narrow = P == 3 && g[0]->variant == 1;
  const int bk = single_block_k(P, g[0]->variant), widest = narrow ? 128 : 256;
  if (kernel == 1) {
    plan_group(pl, g, n, true, pair_block_k(P), widest, sms / 2);
  } else {
    plan_group(pl, g, n, false, bk, widest, sms);
    if (kernel == 2) {
      GroupPlan other;
      plan_group(other, g, n, true, pair_block_k(P), widest, sms / 2);
      if (other.makespan <= pl.makespan) pl = other;
    }
  }
  int64_t tiles = 0;
  for (int k = 0; k < n; ++k) tiles += pl.shape[k].tiles;
  const int units = pl.pair ? sms / 2 : sms;
  if (narrow || tiles >= units) return;
  const int cap = 4 * tiles <= units ? 64 : 2 * tiles <= units ? 128 : 192;
  GroupPlan other;
  plan_group(other, g, n, pl.pair, pl.bk, cap, units);
  if (other.makespan < 0.97 * pl.makespan) pl = other;
}

// Describes a launch to the kernel.
int fill_group(GemmGroup &grp, const GroupPlan &pl, const ZpGemmTc *const *g, int n) {
  const int P = g[0]->planes, bk = pl.bk, halves = pl.halves;
  grp.n = n;
  grp.fp16 = g[0]->fp16;
  grp.status = g[0]->status;
  grp.wait_limit_ns = g[0]->wait_limit_ns > 0 ? (uint64_t)g[0]->wait_limit_ns : kWaitLimitNs;
  grp.unarmed = g[0]->unarmed;
  const ZpEpilogue *epi = g[0]->epi;
  if (epi) grp.epi = *epi;
  else grp.epi.mode = ZP_EPI_NONE;
  grp.classes = pl.classes;
  std::copy(pl.unit0, pl.unit0 + pl.classes + 1, grp.unit0);
  for (int c = 0; c < pl.classes; ++c) {
    if (*std::max_element(pl.count[c], pl.count[c] + n) > INT16_MAX) return ZP_ERR_TOO_LARGE;
    std::copy(pl.first[c], pl.first[c] + n, grp.first[c]);
    std::copy(pl.count[c], pl.count[c] + n, grp.count[c]);
  }
  grp.b_tile = pl.max_bn / halves * bk * 2;
  grp.stage_bytes = P * (BM * bk * 2 + grp.b_tile);
  grp.stages = std::min(kMaxStages, kTileBytes / grp.stage_bytes);
  // one plane: one accumulator, alternating between two of 256 columns; two or three: the leading product's
  // and the small ones', twice side by side where both fit 256 columns
  grp.acc_bufs = P == 1 || pl.max_bn <= kTmemBuf / 2 ? 2 : 1;
  grp.small_off = pl.max_bn <= kTmemBuf / 2 ? kTmemBuf / 2 : kTmemBuf;
  const CUtensorMapSwizzle kswz = bk == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  grp.total = 0;
  for (int k = 0; k < n; ++k) {
    const ZpGemmTc &q = *g[pl.order[k]];
    const Shape &s = pl.shape[k];
    GemmProb &p = grp.p[k];
    p.M = (int)q.M; p.N = (int)q.N;
    p.ksplit = s.ksplit; p.kb_per_split = s.kbs; p.num_k = s.num_k;
    const int kc_elems = q.kc_elems > 0 ? q.kc_elems : 2048;
    p.kc = kc_elems / bk < 1 ? 1 : kc_elems / bk;
    p.a_mn = q.a_mn; p.b_mn = q.b_mn;
    p.scale_a = q.scale_a; p.scale_b = q.scale_b; p.absmax_out = q.absmax_out; p.bias = q.bias;
    p.BN = s.bn;
    p.num_n = s.num_n;
    grp.total += (int)s.tiles;
    int rc;
    if (!q.a_mn) rc = make_map(&p.map_a, q.A, q.K, q.M, P, q.lda, q.a_plane, bk, BM, kswz, q.fp16);
    else rc = make_map(&p.map_a, q.A, q.M, q.K, P, q.lda, q.a_plane, 64, bk, CU_TENSOR_MAP_SWIZZLE_128B, q.fp16);
    if (rc) return rc;
    if (!q.b_mn) rc = make_map(&p.map_b, q.B, q.K, q.N, P, q.ldb, q.b_plane, bk, p.BN / halves, kswz, q.fp16);
    else rc = make_map(&p.map_b, q.B, q.N, q.K, P, q.ldb, q.b_plane, 64, bk, CU_TENSOR_MAP_SWIZZLE_128B, q.fp16);
    if (rc) return rc;
    if (epi && epi->mode != ZP_EPI_NONE && !epi->store_c) p.map_c = p.map_a;      // never used
    else if ((rc = make_map_c(&p.map_c, q.C, q.N, q.M, p.ksplit, q.ldc, q.split_stride))) return rc;
  }
  return ZP_OK;
}

template <int P, int BK, int EPI>
int launch_e(const ZpGemmTc *const *g, int n, const GroupPlan &pl, cudaStream_t st) {
  auto kernel = [] {
    if constexpr (EPI == ZP_EPI_NONE) return gemm_tc_kernel<P, BK>;
    else return gemm_tc_fused_kernel<P, BK, EPI>;
  }();
  static ZpSmemOptIn opt_in;
  int rc;
  if ((rc = zp_ensure_smem(kernel, (size_t)kSmemTotal, opt_in))) return rc;
  GemmGroup grp;
  if ((rc = fill_group(grp, pl, g, n))) return rc;
  zp_launch(kernel, (unsigned)pl.units, kThreads, kSmemTotal, st, grp);
  ZP_LAUNCH_CHECK("gemm_tc_kernel");
  return ZP_OK;
}

template <int P>
int launch_short(const ZpGemmTc &g, cudaStream_t st) {
  using L = ShortLayout<P>;
  static_assert(L::kTotal <= 232448, "shared memory budget of one CTA");
  static ZpSmemOptIn opt_in;
  int rc;
  if ((rc = zp_ensure_smem(gemm_tc_short_kernel<P>, (size_t)L::kTotal, opt_in))) return rc;
  GemmGroup grp;
  GroupPlan pl;
  const ZpGemmTc *one = &g;
  const int sms = device_sms();
  plan_group(pl, &one, 1, false, kShortBK, kShortBN, sms);
  if ((rc = fill_group(grp, pl, &one, 1))) return rc;
  const int columns = grp.p[0].num_n, rows = grp.total / columns;
  grp.rows_apart = columns <= sms ? std::min(sms / columns, rows) : 0;
  if (grp.rows_apart < rows && columns * grp.rows_apart * 10 < sms * 9) grp.rows_apart = 0;
  const int grid = grp.rows_apart ? columns * grp.rows_apart : std::min(grp.total, sms);
  zp_launch(gemm_tc_short_kernel<P>, grid, kShortThreads, L::kTotal, st, grp);
  ZP_LAUNCH_CHECK("gemm_tc_short_kernel");
  return ZP_OK;
}

template <int P, int BK>
int launch(const ZpGemmTc *const *g, int n, const GroupPlan &pl, cudaStream_t st) {
  const int mode = g[0]->epi ? g[0]->epi->mode : ZP_EPI_NONE;
  if constexpr (P == 1 || P == 2) {
    if (mode == ZP_EPI_GATE) return launch_e<P, BK, ZP_EPI_GATE>(g, n, pl, st);
    if (mode == ZP_EPI_ROTATE_BACK) return launch_e<P, BK, ZP_EPI_ROTATE_BACK>(g, n, pl, st);
  }
  if (mode != ZP_EPI_NONE) return ZP_ERR_UNSUPPORTED;
  return launch_e<P, BK, ZP_EPI_NONE>(g, n, pl, st);
}

// CTA pairs of a kernel that the device holds at a time
template <typename Kernel>
int resident_pairs(Kernel *kernel, PerDevice &pairs, int *count) {
  int dev = 0;
  ZP_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return ZP_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> hold(pairs.lock);
  if (!pairs.done[dev]) {
    ZP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemTotal));
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    const int sms = device_sms();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sms / 2 * 2)); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = kSmemTotal;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    int fit = 0;
    ZP_CUDA(cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg));
    pairs.value[dev] = fit < sms / 2 ? fit : sms / 2;
    pairs.done[dev] = true;
  }
  *count = pairs.value[dev];
  return *count < 1 ? ZP_ERR_UNSUPPORTED : ZP_OK;
}

template <int P, int BK, int EPI>
int launch_pair_e(const ZpGemmTc *const *g, int n, const GroupPlan &planned, cudaStream_t st) {
  auto kernel = [] {
    if constexpr (EPI == ZP_EPI_NONE) return gemm_tc_pair_kernel<P, BK>;
    else return gemm_tc_pair_fused_kernel<P, BK, EPI>;
  }();
  static PerDevice pairs;
  int rc, units;
  if ((rc = resident_pairs(kernel, pairs, &units))) return rc;
  GroupPlan pl = planned;
  if (pl.units > units) plan_group(pl, g, n, true, BK, 256, units);     // fewer than half the SMs
  GemmGroup grp;
  if ((rc = fill_group(grp, pl, g, n))) return rc;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pl.units)); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = kSmemTotal;
  cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = 2;
  ZP_CUDA(cudaLaunchKernelEx(&cfg, kernel, grp));
  ZP_LAUNCH_CHECK("gemm_tc_pair_kernel");
  return ZP_OK;
}

template <int P, int BK>
int launch_pair(const ZpGemmTc *const *g, int n, const GroupPlan &pl, cudaStream_t st) {
  const int mode = g[0]->epi ? g[0]->epi->mode : ZP_EPI_NONE;
  if constexpr (P == 1 || P == 2) {
    if (mode == ZP_EPI_GATE) return launch_pair_e<P, BK, ZP_EPI_GATE>(g, n, pl, st);
    if (mode == ZP_EPI_ROTATE_BACK) return launch_pair_e<P, BK, ZP_EPI_ROTATE_BACK>(g, n, pl, st);
  }
  if (mode != ZP_EPI_NONE) return ZP_ERR_UNSUPPORTED;
  return launch_pair_e<P, BK, ZP_EPI_NONE>(g, n, pl, st);
}

int check_product(const ZpGemmTc &g) {
  if (g.K <= 0) return ZP_ERR_INVALID_ARG;
  if (g.fp16 != (g.planes == 2)) return ZP_ERR_UNSUPPORTED;   // fp16 planes come in pairs
  if (!fused_mode_ok(g, block_k(g))) return ZP_ERR_UNSUPPORTED;
  if ((g.lda % 8) || (g.ldb % 8) || (g.a_plane % 8) || (g.b_plane % 8) || (g.ldc % 4) ||
      (g.split_stride % 4))
    return ZP_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B) |
       reinterpret_cast<uintptr_t>(g.C)) & 15)
    return ZP_ERR_INVALID_ARG;
  return ZP_OK;
}

// Whether a group may go to the pair kernel: not where most of the work has short contractions, which leave its
// cross-SM hand-offs exposed on every tile
bool group_may_pair(const ZpGemmTc *const *g, int n) {
  double work = 0.0, deep = 0.0;
  for (int i = 0; i < n; ++i) {
    const double w = (double)g[i]->M * (double)g[i]->N * (double)g[i]->K;
    work += w;
    if (g[i]->K >= 512) deep += w;
  }
  return pair_enabled() && deep > 0.5 * work;
}

// the launch for products of one format; `kernel` as for plan_launch
int dispatch(const ZpGemmTc *const *g, int n, int kernel, cudaStream_t st) {
  const int planes = g[0]->planes;
  if (planes < 1 || planes > 3) return ZP_ERR_UNSUPPORTED;
  const bool is_short = kernel == 0 && n == 1 && !g[0]->a_mn && !g[0]->b_mn && !(g[0]->epi && g[0]->epi->mode) &&
                        g[0]->ksplit <= 1 && g[0]->variant == 0 && g[0]->K * planes <= 256;
  if (is_short && planes <= 2) return planes == 2 ? launch_short<2>(*g[0], st) : launch_short<1>(*g[0], st);
  GroupPlan pl;
  plan_launch(pl, g, n, kernel);
  if (pl.pair)
    return planes == 2 ? launch_pair<2, 64>(g, n, pl, st) : planes == 1 ? launch_pair<1, 64>(g, n, pl, st)
                                                                        : launch_pair<3, 32>(g, n, pl, st);
  if (planes == 2) return launch<2, 32>(g, n, pl, st);
  if (planes == 1) return launch<1, 64>(g, n, pl, st);
  return pl.bk == 64 ? launch<3, 64>(g, n, pl, st) : launch<3, 32>(g, n, pl, st);
}

}  // namespace

int zp_gemm_tc_splits(const ZpGemmTc &g) {
  if (g.K <= 0) return 1;
  int ksplit, kbs, num_k;
  split_plan(g, 64, &ksplit, &kbs, &num_k);
  return ksplit;
}

int zp_gemm_tc_pick_splits(const ZpGemmTc &g, int max_splits) {
  ZpGemmTc t = g;
  int best = 1;
  double best_score = -1.0;
  for (int s = 1; s <= max_splits; ++s) {
    t.ksplit = s;
    const double score = launch_score(t, use_pair(t), s);
    if (score > best_score) { best_score = score; best = s; }
  }
  return best;
}

bool zp_gemm_tc_pairs(const ZpGemmTc &g) { return use_pair(g); }

// The K split of a group's products whose contraction runs over the edges (the last `nw` of n): of a few
// that cut their tiles to between a whole and a third of the launch's time, the one with which it gets done
// first, but no more partial results than that takes.
void zp_gemm_group_splits(ZpGemmTc *g, int n, int nw, int max_splits) {
  const ZpGemmTc *all[ZP_GEMM_GROUP];
  if (n > ZP_GEMM_GROUP) n = ZP_GEMM_GROUP;
  for (int i = 0; i < n; ++i) all[i] = &g[i];
  const bool pair = group_may_pair(all, n);
  const int units = pair ? device_sms() / 2 : device_sms();
  const int bk = pair ? pair_block_k(g[0].planes) : single_block_k(g[0].planes, 0);
  GroupPlan pl;
  auto split = [&](int s) {
    for (int i = n - nw; i < n; ++i) g[i].ksplit = s;
    plan_group(pl, all, n, pair, bk, 256, units);
  };
  split(1);
  double work = 0.0;
  for (int k = 0; k < n; ++k) work += pl.shape[k].cost * (double)pl.shape[k].tiles;
  const int whole = (int)std::ceil(pl.shape[0].cost / (work / units));     // the longest tile is one of theirs
  int best = 1;
  double best_cost = pl.makespan;
  for (int thirds = 2; thirds <= 9; thirds += thirds < 4 ? 1 : 2) {
    const int s = std::min(max_splits, (int)zp_ceil_div((int64_t)whole * thirds, 3));
    if (s <= 1) continue;
    split(s);
    const double cost = pl.makespan * (1.0 + 0.004 * s);
    if (cost < best_cost) { best_cost = cost; best = s; }
    if (s == max_splits) break;
  }
  for (int i = n - nw; i < n; ++i) g[i].ksplit = best;
}

int zp_launch_block_nodes(int64_t E, int64_t N, const int32_t *row_ptr, int32_t *block_node,
                          cudaStream_t st) {
  const int64_t nb = zp_ceil_div(E, 32);
  if (nb == 0 || N == 0) return ZP_OK;
  zp_launch(block_node_kernel, (unsigned)zp_ceil_div(nb, 256), 256, 0, st, nb, (int)N, row_ptr,
            block_node);
  ZP_LAUNCH_CHECK("block_node_kernel");
  return ZP_OK;
}

bool zp_gemm_tc_fusable(const ZpGemmTc &g) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return false;
  return fused_mode_ok(g, block_k(g));
}

int zp_launch_gemm_tc(const ZpGemmTc &g, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0) return ZP_OK;
  if (const int rc = check_product(g)) return rc;
  if (g.M > zp_rows_per_launch(g.N) && !g.a_mn && !(g.epi && g.epi->mode)) {      // in halves
    ZpGemmTc half[2] = {g, g};
    half[0].M = zp_ceil_div(g.M / 2, 256) * 256;
    half[1].M = g.M - half[0].M;
    half[1].A = static_cast<const uint16_t *>(g.A) + half[0].M * g.lda;
    half[1].C = g.C + half[0].M * g.ldc;
    const int rc = zp_launch_gemm_tc(half[0], st);
    return rc ? rc : zp_launch_gemm_tc(half[1], st);
  }
  const ZpGemmTc *one = &g;
  return dispatch(&one, 1, use_pair(g) ? 1 : 0, st);
}

// Several independent products of one format in one launch.
int zp_launch_gemm_group(const ZpGemmTc *g, int n, cudaStream_t st) {
  const ZpGemmTc *live[ZP_GEMM_GROUP];
  int k = 0;
  for (int i = 0; i < n; ++i) {
    if (g[i].M <= 0 || g[i].N <= 0) continue;
    if (const int rc = check_product(g[i])) return rc;
    if (k == ZP_GEMM_GROUP || (g[i].epi && g[i].epi->mode) || g[i].planes != g[0].planes) return ZP_ERR_INVALID_ARG;
    live[k++] = &g[i];
  }
  return k ? dispatch(live, k, group_may_pair(live, k) ? 2 : 0, st) : ZP_OK;
}
