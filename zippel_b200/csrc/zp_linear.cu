// A dense layer  y = x W^T + b  and its VJP on the tensor-core contraction engine, with the
// plan's operand format (fp32-accurate or bf16).  Used for the widest layer of the radial MLP
// (edge_channels -> R, the reference's rad_func[6], blocks/eso2_ref.py:169-182), which as an fp32
// library GEMM costs more than the whole SO(2) forward.
//
// No transposed copies are made: W [N, K] as stored is the K-major B operand of the forward, the
// MN-major B operand of the input gradient (contraction over N), and x / dy as stored are the
// MN-major operands of the weight gradient (contraction over the M rows).
#include "zp_core.cuh"

namespace {

struct LinWork {
  float *scales;          // kLinSlots
  ZpPlanes x, w, dy;
  float *partials;        // weight-gradient partial sums [splits][N*K]
  float *colsum;          // bias-gradient partials
  size_t bytes;
};

constexpr int kLinSplits = 8;

LinWork carve_lin(const zp_plan *p, int64_t M, int64_t K, int64_t N, void *base) {
  LinWork w;
  size_t off = 0;
  auto take = [&](size_t nbytes) {
    char *ptr = base ? static_cast<char *>(base) + off : nullptr;
    off += zp_align_up(nbytes, 256);
    return ptr;
  };
  auto planes = [&](int64_t rows, int64_t cols, float *scale) {
    ZpPlanes pl;
    pl.ld = (cols + 7) / 8 * 8;
    pl.planes = p->planes;
    pl.fp16 = p->fp16;
    pl.scale = p->fp16 ? scale : nullptr;
    pl.plane_stride = (int64_t)zp_align_up((size_t)rows * pl.ld, 128);
    pl.base = take((size_t)pl.planes * pl.plane_stride * 2);
    return pl;
  };
  w.scales = reinterpret_cast<float *>(take(kLinSlots * sizeof(float)));
  w.x = planes(M, K, w.scales + kLinSlotX + 1);
  w.w = planes(N, K, w.scales + kLinSlotW + 1);
  w.dy = planes(M, N, w.scales + kLinSlotDy + 1);
  w.partials = reinterpret_cast<float *>(take(sizeof(float) * kLinSplits * N * K));
  w.colsum = reinterpret_cast<float *>(take(sizeof(float) * (size_t)(zp_colsum_parts(M, N) * N)));
  w.bytes = off;
  return w;
}

// planes of up to three fp32 matrices, each with the scale of its own maximum (slot = {max, scale})
struct SplitJob {
  int64_t rows, cols;
  const float *in;
  const ZpPlanes *planes;
  float *slot;
};
int split_scaled(const zp_plan *p, const SplitJob *jobs, int n, cudaStream_t st,
                 bool maxima_known = false) {
  int rc;
  if (p->fp16 && !maxima_known) {
    ZpMaxList maxima;
    float *last = jobs[n - 1].slot;                       // slots in ascending order
    ZP_CUDA(cudaMemsetAsync(jobs[0].slot, 0, (last + 1 - jobs[0].slot) * sizeof(float), st));
    for (int i = 0; i < n; ++i) maxima.add(jobs[i].in, jobs[i].rows * jobs[i].cols, jobs[i].slot);
    if ((rc = zp_launch_max_list(maxima, st))) return rc;
  }
  ZpSplitList list;
  for (int i = 0; i < n; ++i) {
    const SplitJob &q = jobs[i];
    list.add(q.rows, q.cols, q.in, q.cols, *q.planes, zp_scale_of(1.f, q.slot, q.slot + 1));
  }
  return zp_launch_split_list(list, st);
}

}  // namespace

// The three products of a dense layer's VJP with every operand already in plane form.
//   dx[M, K] = dy[M, N] W[N, K]        (contraction over N: W as stored is the MN-major operand)
//   dw[N, K] = dy^T x                  (contraction over the M rows, both operands MN-major,
//                                       split over CTAs into `partials`, summed in order)
//   db[N]    = column sums of dy
int zp_linear_backward_planes(const zp_plan *plan, int64_t M, int64_t K, int64_t N,
                              const ZpPlanes &x, const ZpPlanes &w, const ZpPlanes &dy, float *dx,
                              float *dw, float *db, float *partials, int max_splits,
                              float *colsum_scratch, ZpFinalList &list, cudaStream_t st,
                              cudaStream_t side, float *dx_absmax, int64_t dx_cols) {
  int rc, n = 0;
  const int P = dy.planes, fp16 = dy.fp16;
  ZpGemmTc g[2];
  if (dx) {
    const int64_t cols = dx_cols > 0 ? dx_cols : K;
    g[n++] = ZpGemmTc{M, cols, N, P, dy.base, dy.ld, dy.plane_stride, 0,
                      w.base, w.ld, w.plane_stride, 1, nullptr, dx, (cols + 3) / 4 * 4,
                      plan->status_dev, 0, 1, 0, 0, fp16, dy.scale, w.scale, dx_absmax};
  }
  const int64_t ldk = (K + 3) / 4 * 4;           // rows of the partial sums start 16-byte aligned
  ZpGemmTc &wg = g[n];
  if (dw) {
    wg = ZpGemmTc{N, K, M, P, dy.base, dy.ld, dy.plane_stride, 1,
                  x.base, x.ld, x.plane_stride, 1, nullptr, partials, ldk, plan->status_dev,
                  0, 1, N * ldk, 0, fp16, dy.scale, x.scale, nullptr};
    ++n;
  }
  // One launch for both, but not where the weight gradient would leave the CTA pairs for it: with two planes
  // the other kernel takes its operands in k-blocks of half the depth, and they are all it has.  A call of the layer
  // and its VJP, apart / together, two planes: 128 x 128 at 25 000, 40 000 and 100 000 rows 188 / 202, 212 / 248 and
  // 332 / 387 us, 256 x 256 at 25 000 and 100 000 218 / 242 and 416 / 511 (15 000 rows of either the same within 5 %);
  // same kernel either way: 64 x 64 at 100 000 384 / 357, 128 x 1536 at 25 000 357 / 334.
  bool together = dx && dw && M <= kTogetherBackward;
  if (dw && (!together || (P == 2 && M > 20000))) {
    wg.ksplit = zp_gemm_tc_pick_splits(wg, max_splits);
    if (together) together = !zp_gemm_tc_pairs(wg) || zp_gemm_tc_pairs(g[0]);
  }
  if (together) {
    zp_gemm_group_splits(g, n, 1, max_splits);
    if ((rc = zp_launch_gemm_group(g, n, st))) return rc;
  } else {
    if (dx && (rc = zp_launch_gemm_tc(g[0], st))) return rc;
    if (dw && (rc = zp_launch_gemm_tc(wg, side))) return rc;
  }
  if (dw) list.add(partials, dw, N * ldk, (int)N, (int)K, zp_gemm_tc_splits(wg), ZP_FIN_SUM, (int)ldk);
  if (db) return zp_launch_colsum(M, N, dy, db, colsum_scratch, list, side);
  return ZP_OK;
}

namespace {

int check(const zp_plan *p, int64_t M, int64_t K, int64_t N) {
  if (!p || M < 0 || K <= 0 || N <= 0) return ZP_ERR_INVALID_ARG;
  if (K % 8 || N % 8) return ZP_ERR_UNSUPPORTED;
  return ZP_OK;
}

int forward(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *x, const float *w,
            const float *bias, float *y, const LinWork &lw, bool maxima_known, cudaStream_t st) {
  const SplitJob jobs[2] = {{M, K, x, &lw.x, lw.scales + kLinSlotX},
                            {N, K, w, &lw.w, lw.scales + kLinSlotW}};
  if (int rc = split_scaled(plan, jobs, 2, st, maxima_known)) return rc;
  const ZpGemmTc g{M, N, K, plan->planes, lw.x.base, lw.x.ld, lw.x.plane_stride, 0,
                   lw.w.base, lw.w.ld, lw.w.plane_stride, 0, bias, y, N, plan->status_dev,
                   0, 1, 0, 0, plan->fp16, lw.x.scale, lw.w.scale, nullptr};
  return zp_launch_gemm_tc(g, st);
}

// the planes of x and w and their scales are where the forward left them
int backward_saved(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *dy, float *dx,
                   float *dw, float *db, const LinWork &lw, bool maximum_known, cudaStream_t st) {
  const SplitJob job{M, N, dy, &lw.dy, lw.scales + kLinSlotDy};
  int rc = split_scaled(plan, &job, 1, st, maximum_known);
  if (rc) return rc;
  ZpFinalList list;
  if ((rc = zp_linear_backward_planes(plan, M, K, N, lw.x, lw.w, lw.dy, dx, dw, db, lw.partials,
                                      kLinSplits, lw.colsum, list, st, st)))
    return rc;
  return zp_launch_finalize(list, st);
}

}  // namespace

extern "C" {

size_t zp_linear_work_bytes(const zp_plan *plan, int64_t M, int64_t K, int64_t N) {
  if (check(plan, M, K, N)) return 0;
  return carve_lin(plan, M, K, N, nullptr).bytes;
}

int zp_linear_forward(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *x,
                      const float *w, const float *bias, float *y, void *work, size_t work_bytes,
                      void *stream) {
  int rc = check(plan, M, K, N);
  if (rc) return rc;
  if (M == 0) return ZP_OK;
  if (!x || !w || !y || !work) return ZP_ERR_INVALID_ARG;
  const LinWork lw = carve_lin(plan, M, K, N, work);
  if (work_bytes < lw.bytes) return ZP_ERR_WORKSPACE;
  return forward(plan, M, K, N, x, w, bias, y, lw, false, (cudaStream_t)stream);
}

int zp_linear_backward(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *x,
                       const float *w, const float *dy, float *dx, float *dw, float *db,
                       void *work, size_t work_bytes, void *stream) {
  int rc = check(plan, M, K, N);
  if (rc) return rc;
  if (!w || !work || (!dw && !dx) || (M && (!x || !dy))) return ZP_ERR_INVALID_ARG;
  const LinWork lw = carve_lin(plan, M, K, N, work);
  if (work_bytes < lw.bytes) return ZP_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  if (M == 0) {
    if (dw) ZP_CUDA(cudaMemsetAsync(dw, 0, sizeof(float) * N * K, st));
    if (db) ZP_CUDA(cudaMemsetAsync(db, 0, sizeof(float) * N, st));
    return ZP_OK;
  }
  // dw == NULL: frozen parameters, only the input gradient (and db if given) is formed
  SplitJob jobs[3];
  int n = 0;
  if (dw) jobs[n++] = {M, K, x, &lw.x, lw.scales};
  if (dx) jobs[n++] = {N, K, w, &lw.w, lw.scales + kLinSlotW};
  jobs[n++] = {M, N, dy, &lw.dy, lw.scales + kLinSlotDy};
  if ((rc = split_scaled(plan, jobs, n, st))) return rc;
  ZpFinalList list;
  if ((rc = zp_linear_backward_planes(plan, M, K, N, lw.x, lw.w, lw.dy, dx, dw, db, lw.partials,
                                      kLinSplits, lw.colsum, list, st, st)))
    return rc;
  return zp_launch_finalize(list, st);
}

int zp_linear_backward_saved(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *dy,
                             float *dx, float *dw, float *db, void *work, size_t work_bytes,
                             void *stream) {
  int rc = check(plan, M, K, N);
  if (rc) return rc;
  if (!work || (!dw && !dx) || (M && !dy)) return ZP_ERR_INVALID_ARG;
  const LinWork lw = carve_lin(plan, M, K, N, work);
  if (work_bytes < lw.bytes) return ZP_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  if (M == 0) {
    if (dw) ZP_CUDA(cudaMemsetAsync(dw, 0, sizeof(float) * N * K, st));
    if (db) ZP_CUDA(cudaMemsetAsync(db, 0, sizeof(float) * N, st));
    return ZP_OK;
  }
  return backward_saved(plan, M, K, N, dy, dx, dw, db, lw, false, st);
}

}  // extern "C"

int zp_linear_forward_maxima(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *x,
                             const float *w, const float *bias, float *y, void *work,
                             cudaStream_t st) {
  return forward(plan, M, K, N, x, w, bias, y, carve_lin(plan, M, K, N, work), true, st);
}

int zp_linear_backward_maxima(const zp_plan *plan, int64_t M, int64_t K, int64_t N, const float *dy,
                              float *dx, float *dw, float *db, void *work, cudaStream_t st) {
  return backward_saved(plan, M, K, N, dy, dx, dw, db, carve_lin(plan, M, K, N, work), true, st);
}
