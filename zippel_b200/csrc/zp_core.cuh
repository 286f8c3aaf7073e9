// The edge convolution's workspace and the launch sequences shared by the C-ABI entry points of
// the convolution alone (zp_api.cu) and of the whole block (zp_block.cu).
#pragma once

#include <cstring>
#include <mutex>
#include <vector>

#include "zp_common.cuh"

// Event pairs recorded around kernel classes while timing is on.
struct ZpTimer {
  struct Span { int cls; cudaEvent_t a, b; int64_t launches; };
  std::vector<Span> spans;      // pool; `used` of them hold live records
  size_t used = 0;
  Span *open(int cls, cudaStream_t st) {
    if (used == spans.size()) {
      Span s{cls, nullptr, nullptr, 0};
      if (cudaEventCreate(&s.a) != cudaSuccess || cudaEventCreate(&s.b) != cudaSuccess) return nullptr;
      spans.push_back(s);
    }
    Span *s = &spans[used++];
    s->cls = cls;
    s->launches = zp_launch_counter();
    cudaEventRecord(s->a, st);
    return s;
  }
  static void close(Span *s, cudaStream_t st) {
    if (!s) return;
    cudaEventRecord(s->b, st);
    s->launches = zp_launch_counter() - s->launches;
  }
};

// brackets one expression with a timing span when the plan has a timer
#define ZP_TIMED(cls, expr)                                                      \
  do {                                                                           \
    ZpTimer::Span *span_ = plan->timer ? plan->timer->open(cls, st) : nullptr;   \
    rc = (expr);                                                                 \
    ZpTimer::close(span_, st);                                                   \
    if (rc) return rc;                                                           \
  } while (0)

inline bool zp_aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline int64_t zp_round8(int64_t x) { return (x + 7) / 8 * 8; }

// 16-bit operand format of a product: number of planes and element type
struct ZpFormat {
  int planes, fp16;
};

// Carves regions out of one buffer (or, with a null base, measures them); each starts 256-byte
// aligned.
struct ZpCarver {
  char *base;
  size_t off = 0;
  explicit ZpCarver(void *b) : base(static_cast<char *>(b)) {}
  char *bytes(size_t n) {
    char *p = base ? base + off : nullptr;
    off += zp_align_up(n, 256);
    return p;
  }
  float *floats(size_t n) { return reinterpret_cast<float *>(bytes(n * sizeof(float))); }
  ZpPlanes planes(int64_t rows, int64_t cols, ZpFormat f, const float *scale) {
    ZpPlanes pl;
    pl.ld = zp_round8(cols);
    pl.planes = f.planes;
    pl.fp16 = f.fp16;
    pl.scale = base && f.fp16 ? scale : nullptr;
    pl.plane_stride = (int64_t)zp_align_up((size_t)rows * pl.ld, 128);
    pl.base = bytes((size_t)pl.planes * pl.plane_stride * 2);
    return pl;
  }
};

// Device-side scale array (fp16 planes): raw maxima, derived scales, and per weight block
// {max |W|, scale} from kScWeights on.  One memset at the start of a forward clears it; a backward
// clears the words from kScBwd on itself.
enum { kScX = 0, kScRad, kScH1, kScA1, kScHt, kScDy, kScDh1, kScGate, kScMaxNode /* an int */,
       // the radial layer run inside the call: {max, scale} of its input and of its weight, scale
       // of the planes of grad_radial
       kScHr, kScHrScale, kScRw, kScRwScale, kScGrScale,
       kScWeights = 24,
       // the rest of the radial MLP (whole-block calls): maxima of the embedding table, of the
       // LayerNorm parameters and of 1/std, {max, scale} of the two weights, scales of activations
       // and gradients
       kScEmb = kScWeights + 4 * (ZP_MAX_L + 1), kScGamma0, kScBeta0, kScGamma1, kScBeta1, kScRstd0,
       kScRstd1, kScW0, kScW0Scale, kScW1, kScW1Scale, kScXe, kScHid0, kScDz1, kScDz0,
       // what a backward clears at its start: maxima it accumulates (upstream gradient, conv2's and conv1's
       // input gradient, gradients of the radial MLP's two hidden activations); its counters follow
       kScBwd, kScG = kScBwd, kScDht, kScDa1, kScGHid1, kScGHid0,
       kScCount };

// Up to this many edges the products of a convolution share one launch, those of the forward and those of the
// backward with the radial layers'.  Beyond it each is a launch of its own on the plan's streams: the
// CTAs of a next launch start wherever an SM becomes free, and the tiles of one product keep to one operand in L2;
// below it the set-up and the draining of each launch cost more.  Whole passes at lmax 4 / C 128, apart and together:
// inference of 30 000 edges in fp32 1.70 / 1.67 ms, in bf16 0.93 / 0.91, of 60 000 3.19 / 3.20 to 3.23, of 105 000
// 5.48 / 5.46 to 5.60; a training step of 30 000 4.98 / 4.73 and 2.61 / 2.44, of 60 000 9.56 / 9.19 and 4.85 / 4.66, of
// 105 000 16.5 / 16.2 and 8.29 / 8.08, of 180 000 28.0 / 28.1.  lmax 2, 158 000 edges: 8.80 / 8.53; lmax 6, 60 000:
// 19.45 / 19.3, 120 000: 39.1 / 39.7.
constexpr int64_t kTogetherEdges = 40000, kTogetherBackward = 110000;

constexpr int kZpWgradSplits = 8;
// K splits of a radial layer's weight gradient [N, K], whose contraction runs over the edges: as many
// as it takes to give every SM a share of the few tiles (eight left 140 SMs idle for 100 us at
// 60 000 edges and 128 x 128), eight at least
inline int zp_radial_splits(int64_t N, int64_t K) {
  const int64_t tiles = zp_ceil_div(N, 128) * zp_ceil_div(K, 256), s = 148 / tiles;
  return (int)(s < 8 ? 8 : s > 64 ? 64 : s);
}

//   forward:  rot | a1 planes | h1 | ht planes | y | folded weight planes | head, cont partials
//   backward: dy planes | dht | dh1 planes | da1 | torque | cut nodes' sums | wgrad partials | scratch
// mode 0 / 1: forward that keeps what a backward reads (1: plus the backward's own regions);
// mode 2: forward alone with fused epilogues -- of h1 only the gate scalars exist, y does not.
struct ZpWorkspace {
  float *rot, *h1, *y, *dht, *da1, *torque, *cuts, *wgrad, *scales, *head, *cont;
  int *arrived;                          // behind the scales
  size_t arrived_words;
  float *rot_grad;                       // [E, nnz_pad], in dht's place where it fits: that is read by then
  float *col1, *col2, *col_rad;          // partial column sums: bias gradients of conv1, conv2, radial
  float *radial, *rad_partials;          // radial layer inside the call: its output, dW partials
  int64_t ld_h1;
  int32_t *block_node;
  ZpPlanes a1, ht, dy, dh1;
  ZpPlanes hr, rw, gr;                   // planes of the layer's input, weight, output gradient
  uint16_t *wfold;
  size_t bytes;
};
// ec > 0: the last layer of the radial MLP (ec -> R), with operands in format `rad`, runs inside
// the call
ZpWorkspace zp_carve(const zp_plan *p, int64_t N, int64_t E, int mode, void *base, int ec,
                     ZpFormat rad);

// The caller's stream plus the plan's two side streams for one forward / backward call.  Up to
// kZpLaneEdges edges everything stays on the caller's: the kernels are then shorter than the host
// takes to launch them, and every event makes it take longer.  Training steps without / with lanes: lmax 4,
// C 128, fp32 0.95 / 0.92 ms at 1 800 edges, 1.14 / 1.10 at 4 200, 1.38 / 1.32 at 6 000; bf16 within 5 % either
// way; lmax 2, C 64 0.64 / 0.80 at 1 800, 0.65 / 0.87 at 4 200, 0.72 / 0.86 at 8 400, 0.89 / 0.93 at 16 800.
// The line is a compromise between the two.  However a call ends, the caller's stream
// goes on behind whatever the side streams have been given: they work in the caller's memory.
constexpr int64_t kZpLaneEdges = 4096;
bool zp_lanes_enabled();
struct ZpLanes {
  const zp_plan *p;
  cudaStream_t main;
  bool on;
  int open = 0;                          // side streams forked and not joined yet, a bit each
  std::unique_lock<std::mutex> hold;
  ZpLanes(const zp_plan *plan, int64_t edges, cudaStream_t st)
      : p(plan), main(st),
        on(edges > kZpLaneEdges && zp_lanes_enabled() && !plan->timer && plan->aux_stream[0]) {
    if (on) hold = std::unique_lock<std::mutex>(*static_cast<std::mutex *>(plan->lane_lock));
  }
  cudaStream_t pick(int i) const { return (!on || i % 3 == 0) ? main : p->aux_stream[i % 3 - 1]; }
  // side streams (`which`: bit 0 the first, bit 1 the second) continue from what the caller's
  // stream has been given so far
  int fork(int which = 3) {
    if (!on) return ZP_OK;
    ZP_CUDA(cudaEventRecord(p->ev_fork, main));
    for (int i = 0; i < 2; ++i)
      if (which >> i & 1) {
        open |= 1 << i;
        ZP_CUDA(cudaStreamWaitEvent(p->aux_stream[i], p->ev_fork, 0));
      }
    return ZP_OK;
  }
  // the caller's stream continues after everything the side streams have been given
  int join(int which = 3) {
    if (!on) return ZP_OK;
    for (int i = 0; i < 2; ++i) {
      if (!(which >> i & 1)) continue;
      ZP_CUDA(cudaEventRecord(p->ev_join[i], p->aux_stream[i]));
      ZP_CUDA(cudaStreamWaitEvent(main, p->ev_join[i], 0));
      open &= ~(1 << i);
    }
    return ZP_OK;
  }
  ~ZpLanes() {                           // an error left the call between fork and join
    for (int i = 0; i < 2; ++i)
      if ((open >> i & 1) && (cudaEventRecord(p->ev_join[i], p->aux_stream[i]) != cudaSuccess ||
                              cudaStreamWaitEvent(main, p->ev_join[i], 0) != cudaSuccess))
        cudaGetLastError();              // the error that is reported is the first one
  }
};

// One convolution call.  Per-edge arrays are in the sorted order.
struct ZpConv {
  int64_t N, E;
  const float *x_node, *edge_vec, *cos_g, *sin_g, *radial, *env;
  const int32_t *src, *dst, *row_ptr, *perm_src, *row_ptr_src;
  const zp_weights *w;
  ZpNodeView view{0, nullptr, nullptr, nullptr};     // forward: all nodes, where the caller has the view by source
  int64_t first = 0, into = 0;                       // backward: all edges end in these `into` nodes from `first` on
};
// The last dense layer of the radial MLP (blocks/eso2_ref.py:169-182, rad_func[6]), when the call
// runs it itself: radial[E, R] = h[E, ec] w[R, ec]^T + b.
struct ZpRadialLayer {
  const float *h, *w, *b;
  int ec;
  float *grad_h, *grad_w, *grad_b;       // backward only
  float *grad_h_max;                     // device scalar updated with max |grad_h|, or null
  ZpFinalList *later;                    // takes the last sums of the layer's parameter gradients where
                                         // its products share a launch (null: they are formed at once)
};

int zp_check_weights(const zp_plan *p, const zp_weights *w);

// radial = hr rw^T + b into ws.radial, its largest magnitude into the scale array
int zp_core_radial(const zp_plan *plan, const ZpWorkspace &ws, int64_t E, int ec, const float *bias,
                   cudaStream_t st);
// Everything from the rotation into the edge frame to node_out; the rotation matrices, the maxima of
// x_node and radial and the weight planes are in place.  keep != 0: what a backward reads is left in
// the workspace.
int zp_core_forward(const zp_plan *plan, const ZpWorkspace &ws, const ZpConv &c, float *node_out,
                    int keep, ZpLanes &lanes);
// gw null: no weight gradients; grad_x_node null: no node contributions.  With rl the gradient of
// radial stays inside.  Both side streams are still to be joined.
int zp_core_backward(const zp_plan *plan, const ZpWorkspace &ws, const ZpConv &c,
                     const float *grad_node_out, float *grad_x_node, float *grad_edge_vec,
                     float *grad_radial, float *grad_env, const zp_weight_grads *gw,
                     const ZpRadialLayer *rl, ZpLanes &lanes);
