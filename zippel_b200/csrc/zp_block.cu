// The whole block in two calls: positions to node output, and the VJP of that.
//
//   forward (reference blocks/eso2_ref.py:317-349): per-edge front end, radial MLP, edge convolution
//   backward: autograd through all of it
//
// The pieces are the ones the other entry points run one at a time.  Run together they need less:
// every activation and gradient of the radial MLP that only feeds a product is written once, as
// operand planes, by the kernel that forms it (scaled from an a-priori bound instead of a scan),
// the maxima and the planes of all weights are one launch each, and all parameter gradients share
// one last launch.  A block of 2 000 edges is bound by its launches: 110 for an energy and its
// forces when every piece was a call of its own, 37 here with its edge sort and head.
#include <cmath>

#include "zp_core.cuh"

namespace {

struct BlockWs {
  ZpWorkspace conv;
  float *edge_vec, *dist, *env, *cos_s, *sin_s;
  ZpPlanes xe, hid0, w0, w1;             // operands of the first two dense layers
  float *h0, *h1;                        // their outputs (LayerNorm inputs)
  float *stats;                          // mean0, rstd0, mean1, rstd1 [E] each
  // backward
  float *g_hid1, *g_hid0, *g_xe, *g_vec_rot, *g_env;
  ZpPlanes dz1, dz0;
  float *part0, *part1, *ln_part;        // weight-gradient partials of the two layers; LayerNorm's
  void *front;                           // work of the front end's backward
  size_t bytes;
};

// Narrow layers whose widths are not multiples of 8 keep fp32 accuracy (two fp16 planes) whatever
// the plan's operand format is: they cost next to nothing, the bf16 format is for the wide products.
ZpFormat layer_format(const zp_plan *p, int in, int out) {
  return (in % 8 || out % 8) ? ZpFormat{2, 1} : ZpFormat{p->planes, p->fp16};
}

struct Formats {
  ZpFormat f0, f1, f2;
};
Formats formats(const zp_plan *p, const zp_front_config &f) {
  const int ec = f.edge_channels, w0 = f.num_basis + 2 * ec;
  return {layer_format(p, w0, ec), layer_format(p, ec, ec), layer_format(p, ec, p->t.R)};
}

int64_t round4(int64_t x) { return (x + 3) / 4 * 4; }

// mode as zp_workspace_bytes
BlockWs carve_block(const zp_plan *p, const zp_front_config &f, int64_t N, int64_t rows, int64_t E,
                    int mode, void *base) {
  BlockWs w;
  const Formats fm = formats(p, f);
  const int ec = f.edge_channels, w0 = f.num_basis + 2 * ec, nl = f.lmax + 1;
  const size_t e = (size_t)E;
  w.conv = zp_carve(p, N, E, mode, base, ec, fm.f2);
  ZpCarver c(base);
  c.off = zp_align_up(w.conv.bytes, 256);
  float *sc = w.conv.scales;
  w.edge_vec = c.floats(3 * e);
  w.dist = c.floats(e);
  w.env = c.floats(e);
  w.cos_s = c.floats(e * nl);
  w.sin_s = c.floats(e * nl);
  w.xe = c.planes(E, w0, fm.f0, sc + kScXe);
  w.hid0 = c.planes(E, ec, fm.f1, sc + kScHid0);
  w.w0 = c.planes(ec, w0, fm.f0, sc + kScW0Scale);
  w.w1 = c.planes(ec, ec, fm.f1, sc + kScW1Scale);
  w.h0 = c.floats(e * ec);
  w.h1 = c.floats(e * ec);
  w.stats = c.floats(4 * e);
  if (mode == 1) {
    w.g_hid1 = c.floats(e * ec);
    w.g_hid0 = c.floats(e * ec);
    w.g_xe = c.floats(e * round4(w0));
    w.g_vec_rot = c.floats(3 * e);
    w.g_env = c.floats(e);
    w.dz1 = c.planes(E, ec, fm.f1, sc + kScDz1);
    w.dz0 = c.planes(E, ec, fm.f0, sc + kScDz0);
    w.part0 = c.floats((size_t)zp_radial_splits(ec, w0) * ec * round4(w0));
    w.part1 = c.floats((size_t)zp_radial_splits(ec, ec) * ec * round4(ec));
    w.ln_part = c.floats((size_t)2 * ZP_LN_PARTIALS * 3 * ec);
    w.front = c.bytes(zp_edge_features_work_bytes(&f, rows, E));
  }
  w.bytes = c.off;
  return w;
}

// what both directions read
int check_common(const zp_plan *plan, const zp_front_config *f, const zp_block_call *c,
                 const zp_block_params *p) {
  if (!plan || !f || !c || !p) return ZP_ERR_INVALID_ARG;
  if (f->lmax != plan->t.lmax || f->edge_channels < 4 || f->edge_channels % 4 ||
      f->edge_channels > 1024 || plan->t.R % 8)
    return ZP_ERR_UNSUPPORTED;
  if (c->n_nodes < 0 || c->n_edges < 0 || c->n_rows < c->n_nodes) return ZP_ERR_INVALID_ARG;
  if (c->n_nodes == 0) return c->n_edges == 0 ? ZP_OK : ZP_ERR_INVALID_ARG;
  if (!c->x_node || !c->row_ptr || !zp_aligned16(c->x_node)) return ZP_ERR_INVALID_ARG;
  if (c->n_edges && (!c->atomic_numbers || !c->src || !c->dst)) return ZP_ERR_INVALID_ARG;
  if (!p->gauss_offsets) return ZP_ERR_INVALID_ARG;
  for (int i = 0; i < 2; ++i)
    if (!p->ln_gamma[i] || !p->ln_beta[i] || !zp_aligned16(p->ln_gamma[i]) || !zp_aligned16(p->ln_beta[i]))
      return ZP_ERR_INVALID_ARG;
  return ZP_OK;
}
int check_forward(const zp_plan *plan, const zp_front_config *f, const zp_block_call *c,
                  const zp_block_params *p) {
  if (const int rc = check_common(plan, f, c, p)) return rc;
  if (c->n_nodes == 0) return ZP_OK;
  if (c->n_edges && (!c->pos || !c->shifts || !c->cos_g || !c->sin_g || !c->perm))
    return ZP_ERR_INVALID_ARG;
  if (!p->emb || !zp_aligned16(p->emb)) return ZP_ERR_INVALID_ARG;
  for (int i = 0; i < 3; ++i)
    if (!p->rad_w[i] || !p->rad_b[i]) return ZP_ERR_INVALID_ARG;
  return zp_check_weights(plan, &p->so2);
}

// silu(LayerNorm(x)) is at most sqrt(width) max|gamma| + max|beta| in magnitude
ZpScale ln_out_scale(int width, const float *gamma, const float *beta, float *out) {
  ZpScale s = zp_scale_of(std::sqrt((float)width), gamma, out);
  s.e = beta;
  s.e_factor = 1.f;
  return s;
}
// LayerNorm + SiLU backward: with |silu'| <= 1.1, rms(z) = 1 and |z| <= sqrt(width),
//   |dx| <= rstd (|dz| + |mean dz| + |z| |mean dz z|) <= rstd 1.1 max|dy| max|gamma| (2 + sqrt(width))
ZpScale ln_grad_scale(int width, const float *dy, const float *gamma, const float *rstd, float *out) {
  ZpScale s = zp_scale_of(1.1f * (2.f + std::sqrt((float)width)), dy, out, gamma);
  s.c = rstd;
  return s;
}

}  // namespace

extern "C" {

size_t zp_block_workspace_bytes(const zp_plan *plan, const zp_front_config *front, int64_t n_nodes,
                                int64_t n_rows, int64_t n_edges, int with_backward) {
  if (!plan || !front || n_nodes < 0 || n_rows < n_nodes || n_edges < 0 || with_backward < 0 ||
      with_backward > 2 || zp_edge_features_work_bytes(front, n_rows, n_edges) == 0)
    return 0;
  return carve_block(plan, *front, n_nodes, n_rows, n_edges, with_backward, nullptr).bytes;
}

int zp_block_forward(const zp_plan *plan, const zp_front_config *front, const zp_block_call *call,
                     const zp_block_params *params, float *node_out, void *workspace,
                     size_t workspace_bytes, int keep_for_backward, void *x_ready_event,
                     void *stream) {
  int rc = check_forward(plan, front, call, params);
  if (rc) return rc;
  const int64_t N = call->n_nodes, E = call->n_edges;
  if (N == 0) return ZP_OK;
  if (!node_out || !workspace || !zp_aligned16(node_out) || !zp_aligned16(workspace))
    return ZP_ERR_INVALID_ARG;
  const BlockWs b = carve_block(plan, *front, N, call->n_rows, E, keep_for_backward ? 1 : 2, workspace);
  if (workspace_bytes < b.bytes) return ZP_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const ZpTables &t = plan->t;
  const ZpWorkspace &ws = b.conv;
  const Formats fm = formats(plan, *front);
  const int ec = front->edge_channels, w0 = front->num_basis + 2 * ec;
  float *sc = ws.scales;
  const bool x_scale = plan->fp16 || fm.f2.fp16;

  // The convolutions' weights and the embeddings are first read after the radial MLP: their maxima
  // and planes are formed beside it, on a side stream, unless there are none (the two calls then
  // share their launches).
  ZpLanes lanes(plan, E, st);
  ZpMaxList maxima, late_maxima_;
  ZpPrepList prep, late_prep_;
  ZpMaxList &late_maxima = lanes.on ? late_maxima_ : maxima;
  ZpPrepList &late_prep = lanes.on ? late_prep_ : prep;
  zp_add_so2_weights(plan, &params->so2, ws.wfold, sc + kScWeights, late_maxima, late_prep,
                     keep_for_backward);
  if (E > 0) {
    prep.add(params->rad_w[0], b.w0.base, sc + kScW0, b.w0.plane_stride, ec, w0, (int)b.w0.ld,
             ZP_PREP_PLAIN, fm.f0.planes, fm.f0.fp16);
    prep.add(params->rad_w[1], b.w1.base, sc + kScW1, b.w1.plane_stride, ec, ec, (int)b.w1.ld,
             ZP_PREP_PLAIN, fm.f1.planes, fm.f1.fp16);
    prep.add(params->rad_w[2], ws.rw.base, sc + kScRw, ws.rw.plane_stride, t.R, ec, (int)ws.rw.ld,
             ZP_PREP_PLAIN, fm.f2.planes, fm.f2.fp16);
    if (fm.f0.fp16) {
      maxima.add(params->rad_w[0], (int64_t)ec * w0, sc + kScW0);
      maxima.add(params->emb, (int64_t)front->n_elements * ec, sc + kScEmb);
    }
    if (fm.f1.fp16) maxima.add(params->rad_w[1], (int64_t)ec * ec, sc + kScW1);
    if (fm.f2.fp16) maxima.add(params->rad_w[2], (int64_t)t.R * ec, sc + kScRw);
    const bool g0 = fm.f1.fp16 || fm.f0.fp16, g1 = fm.f2.fp16 || fm.f1.fp16;
    if (g0) maxima.add(params->ln_gamma[0], ec, sc + kScGamma0);
    if (g0) maxima.add(params->ln_beta[0], ec, sc + kScBeta0);
    if (g1) maxima.add(params->ln_gamma[1], ec, sc + kScGamma1);
    if (g1) maxima.add(params->ln_beta[1], ec, sc + kScBeta1);
    if (x_scale && !x_ready_event) late_maxima.add(call->x_node, call->n_rows * t.K * t.C, sc + kScX);
  }
  if (maxima.n || late_maxima.n) ZP_CUDA(cudaMemsetAsync(sc, 0, sizeof(float) * kScCount, st));
  if (lanes.on) {
    if ((rc = lanes.fork(1))) return rc;
    ZP_TIMED(ZP_K_FOLD, zp_launch_max_list(late_maxima, lanes.pick(1)));
    ZP_TIMED(ZP_K_FOLD, zp_launch_prep_weights(late_prep, lanes.pick(1)));
  }
  ZP_TIMED(ZP_K_FOLD, zp_launch_max_list(maxima, st));
  ZP_TIMED(ZP_K_FOLD, zp_launch_prep_weights(prep, st));
  if (E > 0) {
    float *mean0 = b.stats, *rstd0 = b.stats + E, *mean1 = b.stats + 2 * E, *rstd1 = b.stats + 3 * E;
    ZpScale xe_scale = zp_scale_of(1.f, nullptr, sc + kScXe);      // basis values are at most 1
    xe_scale.c = sc + kScEmb;
    xe_scale.offset = 1.f;
    if ((rc = zp_launch_edge_features_fwd(*front, E, call->pos, call->shifts, call->atomic_numbers,
                                          params->emb, params->gauss_offsets, call->cos_g,
                                          call->sin_g, call->perm, call->src, call->dst, b.edge_vec,
                                          b.dist, nullptr, &b.xe, xe_scale, b.env, b.cos_s, b.sin_s,
                                          st)))
      return rc;
    if ((rc = lanes.fork(1))) return rc;
    ZP_TIMED(ZP_K_WIGNER_FWD, zp_launch_wigner_fwd(plan, E, b.edge_vec, b.cos_s, b.sin_s, ws.rot, 0,
                                                   lanes.pick(1)));
    const ZpGemmTc g0{E, ec, w0, b.xe.planes, b.xe.base, b.xe.ld, b.xe.plane_stride, 0,
                      b.w0.base, b.w0.ld, b.w0.plane_stride, 0, params->rad_b[0], b.h0, ec,
                      plan->status_dev, 0, 1, 0, 0, b.xe.fp16, b.xe.scale, b.w0.scale, nullptr};
    if ((rc = zp_launch_gemm_tc(g0, st))) return rc;
    if ((rc = zp_launch_ln_silu_fwd(E, ec, b.h0, params->ln_gamma[0], params->ln_beta[0],
                                    params->ln_eps, nullptr, &b.hid0,
                                    ln_out_scale(ec, sc + kScGamma0, sc + kScBeta0, sc + kScHid0),
                                    mean0, rstd0, fm.f0.fp16 ? sc + kScRstd0 : nullptr, st)))
      return rc;
    const ZpGemmTc g1{E, ec, ec, b.hid0.planes, b.hid0.base, b.hid0.ld, b.hid0.plane_stride, 0,
                      b.w1.base, b.w1.ld, b.w1.plane_stride, 0, params->rad_b[1], b.h1, ec,
                      plan->status_dev, 0, 1, 0, 0, b.hid0.fp16, b.hid0.scale, b.w1.scale, nullptr};
    if ((rc = zp_launch_gemm_tc(g1, st))) return rc;
    if ((rc = zp_launch_ln_silu_fwd(E, ec, b.h1, params->ln_gamma[1], params->ln_beta[1],
                                    params->ln_eps, nullptr, &ws.hr,
                                    ln_out_scale(ec, sc + kScGamma1, sc + kScBeta1, sc + kScHrScale),
                                    mean1, rstd1, fm.f1.fp16 ? sc + kScRstd1 : nullptr, st)))
      return rc;
    if ((rc = zp_core_radial(plan, ws, E, ec, params->rad_b[2], st))) return rc;
  }
  if ((rc = lanes.join(1))) return rc;
  if (x_ready_event) {                   // x_node is first read from here on
    ZP_CUDA(cudaStreamWaitEvent(st, (cudaEvent_t)x_ready_event, 0));
    if (x_scale && E > 0) {
      ZpMaxList x_max;
      x_max.add(call->x_node, call->n_rows * t.K * t.C, sc + kScX);
      ZP_TIMED(ZP_K_FOLD, zp_launch_max_list(x_max, st));
    }
  }
  ZpConv c{N, E, call->x_node, b.edge_vec, b.cos_s, b.sin_s, ws.radial, b.env, call->src,
           call->dst, call->row_ptr + call->first_node, nullptr, nullptr, &params->so2};
  // (a piece of a graph has most of its edges at few of the nodes: 100 000 in pieces of 30 000 edges took 51 ms of
  // rotate_in by node, lmax 2 and 64 channels, 8.5 by edge)
  if (N == call->n_rows && call->perm_src && call->row_ptr_src)
    c.view = ZpNodeView{call->n_rows, call->row_ptr, call->perm_src, call->row_ptr_src};
  return zp_core_forward(plan, ws, c, node_out, keep_for_backward, lanes);
}

int zp_block_backward(const zp_plan *plan, const zp_front_config *front, const zp_block_call *call,
                      const zp_block_params *params, const float *grad_node_out,
                      float *grad_x_node, float *grad_pos, const zp_block_grads *grads,
                      void *workspace, size_t workspace_bytes, void *stream) {
  int rc = check_common(plan, front, call, params);
  if (rc) return rc;
  const int64_t N = call->n_nodes, E = call->n_edges, rows = call->n_rows;
  if (N == 0) return ZP_OK;
  if (!grad_node_out || !grads || !workspace || !call->row_ptr_src || (E && !call->perm_src) ||
      !zp_aligned16(grad_node_out) || !zp_aligned16(grad_x_node) || !zp_aligned16(workspace))
    return ZP_ERR_INVALID_ARG;
  const bool want_so2 = grads->so2.c1_w0 != nullptr, want_rad = grads->rad_w[0] != nullptr;
  if (want_so2) {
    if (!grads->so2.c1_b0 || !grads->so2.c2_w0 || !grads->so2.c2_b0) return ZP_ERR_INVALID_ARG;
    for (int m = 1; m < plan->n_blocks; ++m)
      if (!grads->so2.c1_wm || !grads->so2.c2_wm || !grads->so2.c1_wm[m - 1] || !grads->so2.c2_wm[m - 1])
        return ZP_ERR_INVALID_ARG;
  }
  if (want_rad) {
    for (int i = 0; i < 3; ++i)
      if (!grads->rad_w[i] || !grads->rad_b[i]) return ZP_ERR_INVALID_ARG;
    for (int i = 0; i < 2; ++i)
      if (!grads->ln_gamma[i] || !grads->ln_beta[i]) return ZP_ERR_INVALID_ARG;
  }
  const BlockWs b = carve_block(plan, *front, N, rows, E, 1, workspace);
  if (workspace_bytes < b.bytes) return ZP_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const ZpWorkspace &ws = b.conv;
  const Formats fm = formats(plan, *front);
  const int ec = front->edge_channels, w0 = front->num_basis + 2 * ec;
  float *sc = ws.scales;
  ZpFinalList list;

  // what the gradients of positions, embedding table and radial parameters all go through
  const bool chain = grad_pos || want_rad || grads->emb;
  ZpRadialLayer rl{nullptr, nullptr, nullptr, ec, chain && E > 0 ? b.g_hid1 : nullptr,
                   grads->rad_w[2], grads->rad_b[2], fm.f1.fp16 ? sc + kScGHid1 : nullptr, &list};
  const ZpConv c{rows, E, call->x_node, b.edge_vec, b.cos_s, b.sin_s, ws.radial, b.env, call->src,
                 call->dst, call->row_ptr, call->perm_src, call->row_ptr_src, &params->so2,
                 {0, nullptr, nullptr, nullptr}, call->first_node, N};
  ZpLanes lanes(plan, E, st);
  if ((rc = zp_core_backward(plan, ws, c, grad_node_out, grad_x_node, b.g_vec_rot, nullptr, b.g_env,
                             want_so2 ? &grads->so2 : nullptr, &rl, lanes)))
    return rc;
  if (E == 0) {
    auto zero = [&](float *p, size_t n) { return p ? cudaMemsetAsync(p, 0, n * sizeof(float), st) : cudaSuccess; };
    if (want_rad) {
      const size_t in[2] = {(size_t)w0, (size_t)ec};
      for (int i = 0; i < 2; ++i) {
        ZP_CUDA(zero(grads->rad_w[i], in[i] * ec));
        ZP_CUDA(zero(grads->rad_b[i], ec));
        ZP_CUDA(zero(grads->ln_gamma[i], ec));
        ZP_CUDA(zero(grads->ln_beta[i], ec));
      }
    }
    ZP_CUDA(zero(grads->emb, (size_t)front->n_elements * ec));
    ZP_CUDA(zero(grad_pos, 3 * (size_t)rows));
  } else if (chain) {
    const float *mean0 = b.stats, *rstd0 = b.stats + E, *mean1 = b.stats + 2 * E,
                *rstd1 = b.stats + 3 * E;
    float *ln0 = b.ln_part, *ln1 = b.ln_part + (size_t)ZP_LN_PARTIALS * 3 * ec;
    // the bias gradient of a layer is the column sum of what LayerNorm's backward passes on
    if ((rc = zp_launch_ln_silu_bwd(E, ec, b.h1, params->ln_gamma[1], params->ln_beta[1], mean1, rstd1,
                                    b.g_hid1, nullptr, &b.dz1,
                                    ln_grad_scale(ec, sc + kScGHid1, sc + kScGamma1, sc + kScRstd1,
                                                  sc + kScDz1),
                                    grads->ln_gamma[1], grads->ln_beta[1], grads->rad_b[1], ln1, list, st)))
      return rc;
    // their weight gradients on the side stream, if at all behind a fork after what they read: up to that line on
    // the caller's, in the input gradient's launch or (nobody wants the input's) one of their own
    const bool apart = want_rad && E > kTogetherBackward;
    const cudaStream_t side = apart ? lanes.pick(2) : st;
    if (apart && (rc = lanes.fork(2))) return rc;
    if ((rc = zp_linear_backward_planes(plan, E, ec, ec, b.hid0, b.w1, b.dz1, b.g_hid0,
                                        grads->rad_w[1], nullptr, b.part1, zp_radial_splits(ec, ec), nullptr,
                                        list, st, side, fm.f0.fp16 ? sc + kScGHid0 : nullptr)))
      return rc;
    if ((rc = zp_launch_ln_silu_bwd(E, ec, b.h0, params->ln_gamma[0], params->ln_beta[0], mean0, rstd0,
                                    b.g_hid0, nullptr, &b.dz0,
                                    ln_grad_scale(ec, sc + kScGHid0, sc + kScGamma0, sc + kScRstd0,
                                                  sc + kScDz0),
                                    grads->ln_gamma[0], grads->ln_beta[0], grads->rad_b[0], ln0, list, st)))
      return rc;
    // without an embedding gradient only the distance basis' columns of the input gradient are used
    const int64_t cols = grads->emb ? w0 : front->num_basis;
    const bool want_in = grad_pos || grads->emb;
    if (apart && (rc = lanes.fork(2))) return rc;
    if ((rc = zp_linear_backward_planes(plan, E, w0, ec, b.xe, b.w0, b.dz0, want_in ? b.g_xe : nullptr,
                                        grads->rad_w[0], nullptr, b.part0, zp_radial_splits(ec, w0), nullptr,
                                        list, st, side, nullptr, cols)))
      return rc;
    if (!apart && (rc = lanes.join(2))) return rc;         // the rotation's part of the edge vectors' gradient
    if (want_in &&
        (rc = zp_launch_edge_features_bwd(*front, rows, E, b.edge_vec, b.dist, params->gauss_offsets,
                                          call->atomic_numbers, b.g_vec_rot, b.g_xe, round4(cols),
                                          b.g_env, call->row_ptr, call->perm_src, call->row_ptr_src,
                                          grad_pos, grads->emb, b.front, st)))
      return rc;
  }
  if ((rc = lanes.join())) return rc;
  ZP_TIMED(ZP_K_FOLD, zp_launch_finalize(list, st));
  return ZP_OK;
}

}  // extern "C"
