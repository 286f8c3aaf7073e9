// Shared declarations of the zippel_b200 kernels: layout tables, the plan, launch helpers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <utility>

#include "zippel_b200.h"
#include "zp_planes.cuh"

#define ZP_MAX_L 6                              // largest supported lmax
#define ZP_MAX_KM ((ZP_MAX_L + 1) * (ZP_MAX_L + 1))
#define ZP_MAX_N (2 * ZP_MAX_L + 1)

// Index tables of one (lmax, mmax) layout, passed to kernels by value.
//   m'-major rows: m = 0 for l = 0..lmax, then for |m| = 1..mmax the +m rows (l = m..lmax)
//   followed by the -m rows.  Row r belongs to degree row_l[r]; its 2l+1 rotation entries sit
//   at rot_off[r] in the packed per-edge rotation.
struct ZpTables {
  int lmax, mmax, K, Km, nnz, nnz_pad;
  int C, H;
  int n_gate;                                   // lmax * H
  int w1_cols;                                  // n_gate + Km * H
  int R;                                        // 2C * sum_m km
  int8_t row_l[ZP_MAX_KM];
  int8_t row_m[ZP_MAX_KM];                      // signed m
  int16_t rot_off[ZP_MAX_KM];
  int8_t row_of[ZP_MAX_L + 1][ZP_MAX_N];        // m' row of (l, i = m + l), or -1
  int16_t m_row0[ZP_MAX_L + 1];                 // first m' row of m-block m
  int16_t m_rows[ZP_MAX_L + 1];                 // rows in m-block m (km or 2 km)
  int32_t rad_off[ZP_MAX_L + 1];                // first radial column of m-block m
  int16_t rad_rows;                             // R / 2C
  int16_t jd_off[ZP_MAX_L + 1];                 // offset of J_l in the packed J array
  // Rotation as the kernels keep it between themselves (rot_ld entries per edge): degree by degree,
  // within a degree the rows m = 0, +1, -1, +2, -2, .. up to mmax and, for l > mmax, the two rows
  // +-(mmax + 1) the VJP needs besides (see zp_rotate_bwd.cu); every row padded to an even number of
  // entries (two weights per 16-byte load once duplicated in shared memory).  A walk through a degree's
  // rows is then a fixed step in all the per-edge arrays in shared memory, which have the same order.
  int16_t deg_rot[ZP_MAX_L + 1];                // first entry of a degree
  int16_t deg_row[ZP_MAX_L + 1];                // rows |m| <= mmax of the degrees before it
  int16_t deg_rad[ZP_MAX_L + 1];                // ... radial gains (l, |m|)
  int16_t row_off[ZP_MAX_KM];                   // entry offset by m'-major row
  int16_t ext_off[ZP_MAX_L + 1][2];
  int16_t rot_ld;
  // generators of rotations about the axes perpendicular to the edge couple m and m + 1 of one
  // degree with these coefficients
  float couple[ZP_MAX_L + 1][ZP_MAX_L + 1];
};

struct ZpTimer;

struct zp_plan {
  ZpTimer *timer;                               // null unless timing is enabled
  zp_config cfg;
  ZpTables t;
  int device;
  double *jd_dev;                               // packed J_l, fp64
  int *status_dev;                              // device status word (0 = ok)
  // per-m GEMM shapes of the folded SO(2) weights
  int n_blocks;                                 // mmax + 1
  int c1_in[ZP_MAX_L + 1], c1_out[ZP_MAX_L + 1], c2_in[ZP_MAX_L + 1], c2_out[ZP_MAX_L + 1];
  int planes;                                   // 16-bit planes per operand: 3 bf16, 2 fp16 or 1 bf16
  int fp16;                                     // planes are fp16 with per-tensor scales
  int64_t c1_woff[ZP_MAX_L + 1], c2_woff[ZP_MAX_L + 1];   // bf16 offsets of the folded planes
  int64_t w_elems;                              // bf16 elements of all folded planes
  int64_t c1_goff[ZP_MAX_L + 1], c2_goff[ZP_MAX_L + 1];   // fp32 offsets of the folded gradients
  int64_t g_elems;                              // fp32 elements of one set of folded gradients
  // Two more streams for launches that do not depend on each other (the per-m products of one
  // convolution, input- and weight-gradient products): run side by side, the last partial wave
  // of one persistent kernel is filled by the next kernel's CTAs.  Forked from and joined back
  // into the caller's stream inside every call; `lane_lock` serialises the enqueueing of calls
  // that share the plan.
  cudaStream_t aux_stream[2];
  cudaEvent_t ev_fork, ev_join[2];
  void *lane_lock;                              // std::mutex
};

// thread-local text of the last CUDA error
void zp_set_cuda_error(cudaError_t e, const char *where);

#define ZP_CUDA(call)                                   \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) {                            \
      zp_set_cuda_error(e_, #call);                     \
      return ZP_ERR_CUDA;                               \
    }                                                   \
  } while (0)

// kernel launches issued by this thread (each launch is followed by one ZP_LAUNCH_CHECK)
int64_t &zp_launch_counter();

#define ZP_LAUNCH_CHECK(name)                           \
  do {                                                  \
    ++zp_launch_counter();                              \
    cudaError_t e_ = cudaGetLastError();                \
    if (e_ != cudaSuccess) {                            \
      zp_set_cuda_error(e_, name);                      \
      return ZP_ERR_CUDA;                               \
    }                                                   \
  } while (0)

// Every kernel is launched so that it may be put in place while its predecessor on the stream still runs
// (two to three microseconds of every launch, a tenth of a step of some hundred atoms), and begins by
// waiting for all of that predecessor's work.  A kernel started by zp_launch has to call
// zp_after_previous before it touches global memory.
__device__ __forceinline__ void zp_after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
void zp_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cfg.attrs = attr; cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...);      // errors: ZP_LAUNCH_CHECK
}

// A kernel's raised dynamic shared-memory limit is an attribute of the function ON a device, so
// "already raised" is remembered per device ordinal (one ZpSmemOptIn per call site, under a lock:
// plans on several devices and several host threads may share the process).
struct ZpSmemOptIn {
  std::mutex lock;
  size_t allowed[64];
  ZpSmemOptIn() { for (size_t &a : allowed) a = 48 * 1024; }
};
template <typename Kernel>
int zp_ensure_smem(Kernel kernel, size_t bytes, ZpSmemOptIn &state) {
  int dev = 0;
  ZP_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return ZP_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> hold(state.lock);
  if (bytes > state.allowed[dev]) {
    ZP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    state.allowed[dev] = bytes;
  }
  return ZP_OK;
}

// ---- lists of small jobs that share one launch ------------------------------------------------
// The tiles of all entries stand in one row, entry i's from first[i] on, and blocks walk the row: a
// block column for each entry, as long as the largest needs, started 18 000 blocks to find most of
// them without work.
#define ZP_MAX_ITEMS 32
struct ZpTileRow {
  int n = 0;
  int first[ZP_MAX_ITEMS + 1] = {0};
  void add(int64_t tiles) { first[n + 1] = first[n] + (int)tiles; ++n; }
  int total() const { return first[n]; }
  // entry that tile `t` belongs to, not before entry `from`
  __device__ __forceinline__ int entry(int t, int from = 0) const {
    while (t >= first[from + 1]) ++from;
    return from;
  }
};
struct ZpMaxList {                              // *out = max |x[0 .. count)|, out zeroed beforehand
  int n = 0;
  const float *x[ZP_MAX_ITEMS];
  int64_t count[ZP_MAX_ITEMS];
  float *out[ZP_MAX_ITEMS];
  void add(const float *src, int64_t cnt, float *slot) {
    x[n] = src; count[n] = cnt; out[n++] = slot;
  }
};
struct ZpSplitList {                            // fp32 matrices to 16-bit planes
  int n = 0;
  int64_t rows[3], cols[3], ld_in[3];
  const float *in[3];
  ZpPlanes out[3];
  ZpScale scale[3];
  void add(int64_t n_rows, int64_t n_cols, const float *src, int64_t ld, const ZpPlanes &to,
           const ZpScale &q) {
    rows[n] = n_rows; cols[n] = n_cols; ld_in[n] = ld; in[n] = src; out[n] = to; scale[n++] = q;
  }
};
enum { ZP_PREP_PLAIN = 0, ZP_PREP_KEPT = 1, ZP_PREP_FOLDED = 2 };
struct ZpPrepList {                             // weight matrices to 16-bit planes
  int n = 0;
  const float *w[ZP_MAX_ITEMS];
  uint16_t *dst[ZP_MAX_ITEMS];
  float *slot[ZP_MAX_ITEMS];                    // {max |W|, scale}
  int64_t plane_stride[ZP_MAX_ITEMS];
  int out[ZP_MAX_ITEMS], in[ZP_MAX_ITEMS], ld[ZP_MAX_ITEMS];
  int8_t kind[ZP_MAX_ITEMS], planes[ZP_MAX_ITEMS], fp16[ZP_MAX_ITEMS];
  int8_t quads[ZP_MAX_ITEMS];                   // set by the launch
  bool transposes = true;                       // of kept and folded matrices
  void add(const float *src, void *to, float *max_and_scale, int64_t stride, int rows, int cols,
           int row_stride, int what, int n_planes, int is_fp16) {
    w[n] = src; dst[n] = static_cast<uint16_t *>(to); slot[n] = max_and_scale;
    plane_stride[n] = stride; out[n] = rows; in[n] = cols; ld[n] = row_stride;
    kind[n] = (int8_t)what; planes[n] = (int8_t)n_planes; fp16[n++] = (int8_t)is_fp16;
  }
};
enum { ZP_FIN_SUM = 0, ZP_FIN_UNFOLD = 1, ZP_FIN_COLUMN = 2 };
struct ZpFinalList {                            // last sums of the parameter gradients
  int n = 0;
  const float *src[ZP_MAX_ITEMS];
  float *dst[ZP_MAX_ITEMS];
  int64_t stride[ZP_MAX_ITEMS];                 // elements between partials
  int rows[ZP_MAX_ITEMS], cols[ZP_MAX_ITEMS], parts[ZP_MAX_ITEMS];
  int ld[ZP_MAX_ITEMS];                         // row stride of a partial
  int8_t kind[ZP_MAX_ITEMS], quads[ZP_MAX_ITEMS];   // quads: set by the launch
  void add(const float *partials, float *to, int64_t between, int n_rows, int n_cols, int n_parts,
           int what, int row_stride = 0) {
    src[n] = partials; dst[n] = to; stride[n] = between; ld[n] = row_stride ? row_stride : n_cols;
    rows[n] = n_rows; cols[n] = n_cols; parts[n] = n_parts; kind[n++] = (int8_t)what;
  }
};

static inline int64_t zp_ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
static inline size_t zp_align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

#define ZP_DISPATCH_LMAX(lmax, CALL)          \
  switch (lmax) {                             \
    case 0: { CALL(0); break; }               \
    case 1: { CALL(1); break; }               \
    case 2: { CALL(2); break; }               \
    case 3: { CALL(3); break; }               \
    case 4: { CALL(4); break; }               \
    case 5: { CALL(5); break; }               \
    case 6: { CALL(6); break; }               \
    default: return ZP_ERR_UNSUPPORTED;       \
  }

// ---- kernels (each in its own translation unit) --------------------------------------------
// rot in the packed layout [E, nnz_pad] (packed != 0) or in the kernels' own [E, rot_ld]
int zp_launch_wigner_fwd(const zp_plan *p, int64_t E, const float *ev, const float *cg,
                         const float *sg, float *rot, int packed, cudaStream_t st);
int zp_launch_wigner_bwd(const zp_plan *p, int64_t E, const float *ev, const float *cg,
                         const float *sg, const float *grot, float *gev, cudaStream_t st);

// The arrays of one edge convolution's VJP that an edge's rotation gradient comes from.
// torque [slots][E, 4], to be summed over the slots: for each edge the derivative of the loss under a rotation of the edge frame about
// its own axis (entry 0) and the two axes perpendicular to it (1, 2).
struct ZpTorqueArgs {
  const float *da1, *radial, *x, *y, *g_out, *env;
  const int32_t *src, *dst;
  float *entries;                        // [E, nnz_pad] scratch: gradient of the rotation entries
};
// torque -> gradient of the edge vectors
int zp_launch_edge_vec_grad(const zp_plan *p, int64_t E, const float *ev, const float *cg,
                            const float *sg, const float *torque, int slots, const ZpTorqueArgs &a, float *gev,
                            cudaStream_t st);

// All nodes that the edges name, with the edges into and out of each; perm_src null: the caller has no view by source
struct ZpNodeView {
  int64_t nodes;
  const int32_t *row_ptr, *perm_src, *row_ptr_src;
};
int zp_launch_rotate_in(const zp_plan *p, int64_t E, const float *x, const int32_t *src,
                        const int32_t *dst, const ZpNodeView &view, const float *rot, const float *radial,
                        const ZpPlanes &a1, const ZpScale &scale, cudaStream_t st);
int zp_launch_rotate_back_scatter(const zp_plan *p, int64_t N, const float *y, const float *env,
                                  const float *rot, const int32_t *row_ptr, float *node_out,
                                  cudaStream_t st);
// N nodes from `first` on hold all edges' destinations
int zp_launch_rotate_grad_out(const zp_plan *p, int64_t first, int64_t N, int64_t E, const float *g, const float *y,
                              const float *env, const float *rot, const int32_t *dst, const int32_t *row_ptr,
                              const ZpPlanes &dy, const ZpScale &scale, float *grad_env,
                              float *torque, cudaStream_t st);
// grad_radial goes out as fp32 rows [E, R], or (grad_radial_planes given) as operand planes.  grad_x null:
// nobody wants the gradient of x_node.  Slot 0 of torque holds what rotate_grad_out has left; as many slots are
// written or added to as zp_torque_slots says.
int zp_launch_rotate_in_bwd(const zp_plan *p, int64_t N, int64_t E, const float *da1, const float *radial,
                            const float *x, const int32_t *row_ptr, const int32_t *perm_src,
                            const int32_t *row_ptr_src, const float *rot, float *grad_radial, float *grad_x,
                            float *torque, float *cuts, int *arrived, cudaStream_t st,
                            const ZpPlanes *grad_radial_planes, const ZpScale &scale);
int zp_torque_slots(const ZpTables &t);
// Nodes of many edges are cut into stretches (zp_rotate.cuh), at this many places at most.  A cut's part of the
// gradient of x_node stands in `cuts` [kZpNodeCuts][K][C] until the last stretch of its node to get done adds them up:
// `arrived`, zero before the launch, counts them, kZpNodeCuts words for each group of channels.
constexpr int kZpNodeCuts = 296;
int64_t zp_node_cuts_most(int64_t E);              // no more than this many of E edges
int zp_node_groups(const ZpTables &t);
// node_out[n, l^2 + j, c] = sum over the m' rows r of degree l, in table order, of
//   head[n][rot_off[r] + j][c] + the continuation partials of the 32-edge blocks n's edges reach
int zp_launch_node_sum(const zp_plan *p, int64_t N, const float *head, const float *cont,
                       const int32_t *row_ptr, float *node_out, cudaStream_t st);

int zp_launch_gate_fwd(const zp_plan *p, int64_t E, const float *h1, const ZpPlanes &ht,
                       const ZpScale &scale, float *gate_max, cudaStream_t st);
// gate_max (device scalar, may be null): largest sigmoid'(gate) seen by the forward
int zp_launch_gate_bwd(const zp_plan *p, int64_t E, const float *h1, const float *dht,
                       const ZpPlanes &dh1, const ZpScale &scale, cudaStream_t st);

// Work the contraction's epilogue does on a finished 32-row x 32-column block of the result
// while it is still on chip (staged in shared memory), besides or instead of storing it.
//   ZP_EPI_GATE         conv1 of the SO(2) block: column n is hidden channel (n % width) of m' row
//                       row_first + n / width; the block goes through the gate activation
//                       (blocks/eso2_ref.py:295-301: SiLU for row 0, x * sigmoid(gate[l-1]) for the
//                       others, the raw gate scalars read from `gate`) and is written as 16-bit
//                       operand planes for conv2.
//   ZP_EPI_ROTATE_BACK  conv2: column n is channel (n % width) of m' row row_first + n / width;
//                       every edge's value is scaled by its envelope, expanded by the edge's
//                       packed rotation row into the 2l+1 outputs of its degree and summed over
//                       the consecutive edges of a destination node (the edges are destination
//                       sorted).  A node's first run of edges inside a 32-row block goes to
//                       head[node], a run that continues from the previous block to cont[block];
//                       zp_launch_node_sum adds them up in a fixed order.
// Requires K-major operands, one accumulation chunk and no K split.
enum { ZP_EPI_NONE = 0, ZP_EPI_GATE = 1, ZP_EPI_ROTATE_BACK = 2 };
struct ZpEpilogue {
  int mode;
  int store_c;                                  // also store the fp32 result to C
  int width;                                    // channels per m' row (H or C)
  int row_first;                                // m' row of column 0
  int8_t row_l[ZP_MAX_KM];                      // degree of each m' row
  int16_t rot_off[ZP_MAX_KM];                   // offset of the row's partial sums in a slab
  // gate
  const float *gate;                            // [M, ld_gate] raw gate scalars, block l-1 at column (l-1)*width
  int64_t ld_gate;
  ZpPlanes out;                                 // activated rows: element (e, n) at e*out.ld + n
  float *slope_max;                             // running max of sigmoid'(gate), or null
  // rotate back
  const float *rot, *env;                       // [M, rot_ld], [M]
  int16_t row_off[ZP_MAX_KM];                   // offset of the row's entries in `rot`
  int rot_ld;
  const int32_t *row_ptr;                       // [n_nodes + 1] offsets of the nodes' edges
  const int32_t *block_node;                    // [ceil(M/32)] node of edge 32 b (zp_launch_block_nodes)
  int n_nodes, nnz;
  float *head, *cont;                           // [n_nodes][nnz][width], [ceil(M/32)][nnz][width]
};

// Tensor-core product over bf16 planes: C[M,N] = sum_pairs A_pa * B_pb^T (+ bias), fp32 out.
// K-major operand: X[p*plane + r*ld + k]; MN-major (x_mn = 1): X[p*plane + k*ld + r].
struct ZpGemmTc {
  int64_t M, N, K;
  int planes;                                   // 1 (bf16) or 3 (fp32 carried as three bf16)
  const void *A; int64_t lda, a_plane; int a_mn;
  const void *B; int64_t ldb, b_plane; int b_mn;
  const float *bias;
  float *C; int64_t ldc;
  int *status;                                  // device word, set on a device-side timeout
  int variant;                                  // tile-shape choice for the 3-plane K-major case
  int ksplit;                                   // requested split of K over CTAs (>= 1)
  int64_t split_stride;                         // elements between the partial outputs of splits
  int kc_elems;                                 // K per TMEM accumulation chunk (0 = 2048)
  int fp16;                                     // planes are fp16 (planes must be 2), else bf16
  const float *scale_a, *scale_b;               // device scalars multiplied into the result
  float *absmax_out;                            // device scalar updated with max |C| (or null)
  const ZpEpilogue *epi;                        // fused epilogue (null = store C)
  int64_t wait_limit_ns;                        // bound of the device-side waits (0 = 2 s)
  int unarmed;                                  // self-test: no operand is ever loaded
};
int zp_launch_gemm_tc(const ZpGemmTc &g, cudaStream_t st);
// up to ZP_GEMM_GROUP independent products of one format in one launch
#define ZP_GEMM_GROUP 8
int zp_launch_gemm_group(const ZpGemmTc *g, int n, cudaStream_t st);
// sets the K split (<= max_splits) of the last nw of n products that will share a launch
void zp_gemm_group_splits(ZpGemmTc *g, int n, int nw, int max_splits);
// block_node[b] = node of the first edge of 32-edge block b, for ZpEpilogue::block_node
int zp_launch_block_nodes(int64_t E, int64_t N, const int32_t *row_ptr, int32_t *block_node,
                          cudaStream_t st);
// whether zp_launch_gemm_tc accepts a fused epilogue for this problem
bool zp_gemm_tc_fusable(const ZpGemmTc &g);
// number of partial outputs the launch above will write for this problem (<= g.ksplit)
int zp_gemm_tc_splits(const ZpGemmTc &g);
// K split (<= max_splits) that fills the device's CTAs (or CTA pairs) most evenly for this problem
int zp_gemm_tc_pick_splits(const ZpGemmTc &g, int max_splits);
// whether a launch of the product alone goes to the CTA-pair kernel
bool zp_gemm_tc_pairs(const ZpGemmTc &g);
// fp32 [rows, cols] (row stride ld_in) -> planes [rows, out.ld], zero padded
int zp_launch_split_list(const ZpSplitList &list, cudaStream_t st);
int zp_launch_split_planes(int64_t rows, int64_t cols, const float *in, int64_t ld_in,
                           const ZpPlanes &out, const ZpScale &scale, cudaStream_t st);
int zp_launch_max_list(const ZpMaxList &list, cudaStream_t st);
int zp_launch_prep_weights(ZpPrepList &list, cudaStream_t st);
int zp_launch_finalize(ZpFinalList &list, cudaStream_t st);
// *out = largest node index in src / dst (device scalar, zeroed by the caller)
int zp_launch_max_index(int64_t E, const int32_t *src, const int32_t *dst, int *out,
                        cudaStream_t st);
// *out = max |in| over rows [first ? *first : 0, max(min_rows, last ? *last + 1 : 0)) of a
// contiguous [*, cols] matrix; first / last are device pointers to row numbers, *out was zeroed
int zp_launch_absmax_row_range(const float *in, int64_t cols, const int32_t *first,
                               const int32_t *last, int64_t min_rows, float *out,
                               cudaStream_t st);

// The SO(2) weight blocks of both convolutions, for zp_launch_max_list (fp16 planes) and
// zp_launch_prep_weights: per block W_fold [P][out][in] followed by its transpose [P][in][out], at
// element offset c{1,2}_woff[m] of `packed`; `scales`: per block (conv * (ZP_MAX_L+1) + m) two
// floats {max |W|, scale}.
// (the transpose only if a backward follows: `transposes`)
void zp_add_so2_weights(const zp_plan *p, const zp_weights *w, void *packed, float *scales,
                        ZpMaxList &maxima, ZpPrepList &prep, bool transposes);
// ... and their gradients, for zp_launch_finalize: per split s the folded fp32 gradients stand at
// partials + s*split_stride + c{1,2}_goff[m]
void zp_add_so2_grads(const zp_plan *p, const float *partials, int64_t split_stride,
                      const int *splits_c1, const int *splits_c2, const zp_weight_grads *gw,
                      ZpFinalList &list);
// *ht_scale = fp16-plane scale of conv1's activated output from an a-priori bound:
//   |h1| <= max_m(in_m * max|a1| * max|W1_m|) + max|b1|,  |gate_act(h1)| <= |h1|
// (a1_scale maps the bound of a1 to 2^15; wscales: {max, scale} pairs per weight block)
int zp_launch_conv1_bound(const zp_plan *p, const float *a1_scale, const float *wscales,
                          const float *bias, float *ht_scale, cudaStream_t st);
// LayerNorm + SiLU over rows of `width` floats.  The result goes out as fp32 rows (y / dx) or, with
// y_planes / dx_planes given, as operand planes of the next product; rstd_max: device scalar updated
// with the largest 1/std (or null).  Backward: dgamma null = no parameter gradients; dbias = column
// sums of dx (or null); `partial`: ZP_LN_PARTIALS * 3 * width floats.
#define ZP_LN_PARTIALS 296
int zp_launch_ln_silu_fwd(int64_t rows, int width, const float *x, const float *gamma,
                          const float *beta, float eps, float *y, const ZpPlanes *y_planes,
                          const ZpScale &scale, float *mean, float *rstd, float *rstd_max,
                          cudaStream_t st);
int zp_launch_ln_silu_bwd(int64_t rows, int width, const float *x, const float *gamma,
                          const float *beta, const float *mean, const float *rstd, const float *dy,
                          float *dx, const ZpPlanes *dx_planes, const ZpScale &scale,
                          float *dgamma, float *dbeta, float *dbias, float *partial,
                          ZpFinalList &list, cudaStream_t st);
// VJP of y = x W^T + b with all operands as planes (of one format); `partials`: max_splits * N *
// round4(K) floats, `colsum_scratch`: zp_colsum_parts(M, N) * N floats.  dw and db, formed on
// `side`, get their last sums from `list` (zp_launch_finalize); dx_absmax: device scalar updated with
// max |dx|, or null; dx_cols: how many leading columns of dx are wanted (0: all K)
int zp_linear_backward_planes(const zp_plan *plan, int64_t M, int64_t K, int64_t N,
                              const ZpPlanes &x, const ZpPlanes &w, const ZpPlanes &dy, float *dx,
                              float *dw, float *db, float *partials, int max_splits,
                              float *colsum_scratch, ZpFinalList &list, cudaStream_t st,
                              cudaStream_t side, float *dx_absmax = nullptr, int64_t dx_cols = 0);
// zp_linear_forward / zp_linear_backward_saved for a caller whose own kernels found the maxima.
// `slots` (the start of the work buffer): {max x, scale, max w, scale, max dy, scale, and two words
// for the caller's use}; with fp16 planes the maxima stand there when these are called.
constexpr int kLinSlotX = 0, kLinSlotW = 2, kLinSlotDy = 4, kLinSlotFree = 6, kLinSlots = 8;
int zp_linear_forward_maxima(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *x,
                             const float *w, const float *bias, float *y, void *work,
                             cudaStream_t st);
int zp_linear_backward_maxima(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *dy,
                              float *dx, float *dw, float *db, void *work, cudaStream_t st);
// column sums of `a`: partial sums into scratch (zp_colsum_parts(rows, cols) * cols floats), the rest by
// `list`.  A part has 512 rows, or fewer (64 at least) where that leaves less than eight blocks per SM.
inline int64_t zp_colsum_rows(int64_t rows, int64_t cols) {
  const int64_t each = zp_ceil_div(rows * zp_ceil_div(cols, 256), 148 * 8);
  return each <= 64 ? 64 : each >= 512 ? 512 : zp_ceil_div(each, 8) * 8;
}
inline int64_t zp_colsum_parts(int64_t rows, int64_t cols) {
  return rows > 0 ? zp_ceil_div(rows, zp_colsum_rows(rows, cols)) : 0;
}
int zp_launch_colsum(int64_t rows, int64_t cols, const ZpPlanes &a, float *out, float *scratch,
                     ZpFinalList &list, cudaStream_t st);

// The per-edge front end.  x_planes given: the input of the radial MLP goes out as operand planes
// (zero padded to their row stride) instead of fp32 rows.
int zp_launch_edge_features_fwd(const zp_front_config &cfg, int64_t E, const float *pos,
                                const float *shifts, const int64_t *atomic_numbers, const float *emb,
                                const float *gauss_offsets, const float *cos_g, const float *sin_g,
                                const int32_t *perm, const int32_t *src, const int32_t *dst,
                                float *edge_vec, float *dist, float *x_edge,
                                const ZpPlanes *x_planes, const ZpScale &scale, float *env,
                                float *cos_sorted, float *sin_sorted, cudaStream_t st);
// grad_x_edge [E, ldg]: all columns when grad_emb is wanted, at least the num_basis leading ones
// otherwise; grad_pos or grad_emb may be null
int zp_launch_edge_features_bwd(const zp_front_config &cfg, int64_t N, int64_t E,
                                const float *edge_vec, const float *dist,
                                const float *gauss_offsets, const int64_t *atomic_numbers,
                                const float *grad_edge_vec, const float *grad_x_edge, int64_t ldg,
                                const float *grad_env, const int32_t *row_ptr,
                                const int32_t *perm_src, const int32_t *row_ptr_src,
                                float *grad_pos, float *grad_emb, void *work, cudaStream_t st);
