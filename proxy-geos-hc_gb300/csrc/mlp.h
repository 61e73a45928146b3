// mlp.h -- the boundary network of the learned absorbing boundary: 81 inputs (p at three time
// levels on the 3x3x3 node neighbourhood, divided by a per-node scale), two hidden layers of 64
// with GELU, one output.  BF16 weights and activations into FP32 accumulators on the tensor
// cores (mma.sync m16n8k16), FP32 master weights and Adam state for training.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "host_util.h"

namespace semgb {

constexpr int kMlpIn = 81;
constexpr int kMlpInPad = 96;  // K of layer 1 padded to whole 16-wide MMA steps
constexpr int kMlpHidden = 64;
// FP32 master layout: W1[64][81], b1[64], W2[64][64], b2[64], w3[64], b3
constexpr int kOffW1 = 0;
constexpr int kOffB1 = kOffW1 + kMlpHidden * kMlpIn;
constexpr int kOffW2 = kOffB1 + kMlpHidden;
constexpr int kOffB2 = kOffW2 + kMlpHidden * kMlpHidden;
constexpr int kOffW3 = kOffB2 + kMlpHidden;
constexpr int kOffB3 = kOffW3 + kMlpHidden;
constexpr int kMlpParams = kOffB3 + 1;
constexpr int kMlpTile = 128;  // rows (nodes or samples) per CTA

// Device copy of the network for the kernels: BF16 W1 as [64][96] (zero-padded K) and W2 as
// [64][64], FP32 biases and output layer.
struct MlpDev {
    const uint16_t *w1;  // [64][96] bf16 bits
    const uint16_t *w2;  // [64][64]
    const float *b1, *b2, *w3, *b3;
};

// Strip of nodes the network corrects, and the levels it reads.
struct AbcArgs {
    const int64_t *nodes;  // device-layout indices of the strip nodes
    int64_t n;
    const float *p_new;    // p^{n+1} (sponge applied)
    const float *p_cur;    // p^n stored without its last sponge factor (actual = s * stored)
    const float *hist;     // p^{n-1} (actual values) on the history shell, device layout [n_int]
    const float *sx, *sy, *sz;  // sponge factors (null: none)
    int64_t nx, nxp, ny, nz;
    float *corr;           // out: correction per strip node
    int absolute;          // 1: the network gives the node's value (scale * y), 0: a correction
};

// Face-tiled correction of the boundary nodes (strip layer 0): the six faces of the box are cut
// into tiles of kFaceTU x kFaceTV nodes (one CTA tile of kMlpTile rows), every boundary node on
// exactly one face.  A tile's three levels on the face plane and the plane inside it, with a
// one-node rim, are staged in shared memory once, and each node's 81 features come from there.
constexpr int kFaceTU = 16, kFaceTV = 8;
static_assert(kFaceTU * kFaceTV == kMlpTile, "one face tile is one network tile");
struct FaceDesc {
    int axis_n, axis_u, axis_v;  // axes (0: x, 1: y, 2: z) normal to the face and along its tiles
    int side;                    // node coordinate of the face along axis_n
    int inward;                  // +1 or -1: the direction into the box along axis_n
    int ulo, uhi, vlo, vhi;      // node ranges of the face along axis_u and axis_v
};
struct AbcFaceArgs {
    FaceDesc face[6];
    const int4 *tiles;     // (face, u0, v0, 0) per tile
    int64_t ntiles;
    float *p_new;          // p^{n+1} (sponge applied); out: the boundary nodes' new values
    const float *p_cur;    // p^n stored without its last sponge factor
    const float *hist;     // p^{n-1} (actual values) on the two-node shell, device layout
    float *hist_next;      // out: p^n (actual values) on the two-node shell, device layout
    const float *sx, *sy, *sz;  // sponge factors (null: none)
    int64_t nx, nxp, ny, nz;
};
// Face-tiled boundary values (the features, network, output and clipping of abc_correction with
// absolute values) written into p_new, and p^n into hist_next on the shell.  p^{n+1} of the
// boundary nodes is taken as s * hist (what the step leaves there), the rest from p_new.
cudaError_t abc_face(const MlpDev &net, const AbcFaceArgs &a, cudaStream_t s);

// ---- adjoint of the time loop with the network on the boundary nodes (k_bptt.cu) ----------
// Work arrays of one backward pass over a box (device layout, nb boundary nodes).
struct BpttFields {
    int nx, ny, nz;
    int64_t nxp, n_int;
    const float *sx, *sy, *sz;  // sponge factors (null: none)
    const int64_t *nodes;       // boundary nodes (device layout), nb of them
    int64_t nb;
    const int *sidx;            // [n_int]: index in `nodes`, -1 elsewhere
    const int64_t *shell;       // nodes within one of the boundary, n_shell of them
    int64_t n_shell;
    float *dx;                  // [81][dx_stride] feature gradient
    int64_t dx_stride;
    float *a[3];                // adjoints of out^m, out^{m-1}, out^{m-2}
    float *v;                   // [n_int] work field
    const int64_t *roi;         // region of interest (device layout), n_roi nodes
    int n_roi;
    const int *ridx;            // [n_int]: index in the region, -1 elsewhere (null: it lists a node twice)
};
// The stiffness operator of the stencil pass: 1-D table T[l][d + o] (direct form, diagonal
// included), assembled weights by local index, g for the x, z and y terms.
struct BpttOperator {
    int order;
    float T[kMaxOrder * (2 * kMaxOrder + 1)];
    float wa[kMaxOrder];
    float g[3];
};
// Feature gradients gathered into A0, A1, A2, and v = a s A0 on interior nodes (a_mass = dt^2 / M).
cudaError_t bptt_scatter(const BpttFields &f, const float *a_mass, cudaStream_t s);
// Interior leapfrog adjoint (v, A0 -> A1, A2; A0 cleared); with next_out the loss gradient of that
// level against next_ref is added to A1 (needs f.ridx).
cudaError_t bptt_interior(const BpttFields &f, const BpttOperator &op, const float *next_out, const float *next_ref,
                          cudaStream_t s);
// Loss gradient of one level into A0.
cudaError_t bptt_seed(const BpttFields &f, const float *out, const float *ref, cudaStream_t s);
// Loss over the region of interest at every step: loss[m] of levels + m * stride against row m of ref.
cudaError_t bptt_losses(const BpttFields &f, const float *levels, int64_t stride, const float *ref, int n_steps,
                        double *loss, cudaStream_t s);
// dst <- src, n floats (a multiple of 4), behind the preceding kernel of the stream.
cudaError_t bptt_copy_level(const float *src, float *dst, int64_t n, cudaStream_t s);

// bf16 conversion of the FP32 master weights into the device layout.
cudaError_t mlp_pack(const float *master, uint16_t *w1, uint16_t *w2, float *b1, float *b2, float *w3, float *b3,
                     cudaStream_t s);
// y[i] = net(x[i]) for x [n][81] (FP32, device).
cudaError_t mlp_forward(const MlpDev &net, const float *x, float *y, int64_t n, cudaStream_t s);
// Work arrays of a training pass (k_mlp_train.cu), rows of one round (mlp_work_rows).
constexpr int kMlpMaxSlots = 152 * 4;  // partial-sum slots: tile t of a pass adds to slot t % kMlpMaxSlots
constexpr int kMlpXbStride = 88;       // row stride (bf16) of the stored inputs
struct MlpWork {
    uint16_t *xb = nullptr;   // [rows][88] BF16 inputs
    uint16_t *h1 = nullptr;   // [rows][64] BF16 hidden activations
    float *dz1 = nullptr, *dz2 = nullptr, *g2 = nullptr;  // [rows][64] dZ of both layers, GELU(z2)
    float *err = nullptr, *dy = nullptr;                  // [rows] y - t, output gradient
    float *part = nullptr;    // [kMlpMaxSlots][kMlpParams] partial gradients
    double *lsum = nullptr;   // [kMlpMaxSlots][32] partial squared errors
};
// Rows of work arrays that a pass over n rows needs (at most kMlpMaxSlots tiles: longer passes run
// in rounds).
int64_t mlp_work_rows(int64_t n);
// Adam on the FP32 master parameters: moments, step count (from 1) and rate, and the kernels' form
// of the network, rewritten with the new parameters.
struct MlpAdam {
    float *master, *m, *v;
    int t;
    float lr;
    uint16_t *w1, *w2;
    float *b1, *b2, *w3, *b3;
};
// Shared-memory limits of the training kernels on the current device.
cudaError_t mlp_train_setup();
// Loss 1/n sum (net(x_i) - t_i)^2 accumulated into *loss (double), gradients with respect to the
// master parameters accumulated into grad (FP32 [kMlpParams]).  Deterministic: partial sums per
// tile, added in order.
cudaError_t mlp_loss_grad(const MlpDev &net, const float *x, const float *t, int64_t n, double *loss, float *grad,
                          const MlpWork &w, cudaStream_t s);
// One minibatch of Adam on samples idx[0..n): the loss before the step into *loss.  dependent: the
// preceding work of the stream is a step on the same network.
cudaError_t mlp_train_step(const MlpDev &net, const float *x, const float *t, const int64_t *idx, int64_t n,
                           double *loss, const MlpAdam &adam, const MlpWork &w, cudaStream_t s, bool dependent);
// The network in one step of the adjoint of the time loop, at the boundary nodes: features from the
// levels out^m, out^{m-1}, out^{m-2}, output gradient from A0, feature gradients into f.dx, and the
// rows' part of the parameter gradients into the work arrays' group `group` (the steps of one
// mlp_boundary_params call).  Boxes of more boundary nodes than mlp_work_rows(nb) run in rounds and
// add their parameter gradients to grad at once (mlp_boundary_groups returns 1).
int mlp_boundary_groups(int64_t nb);
cudaError_t mlp_boundary_rows(const MlpDev &net, const BpttFields &f, const float *lm, const float *lm1,
                              const float *lm2, int group, const MlpWork &w, float *grad, cudaStream_t s);
// Parameter gradients of groups 0..n-1 added to grad, group by group.
cudaError_t mlp_boundary_params(int64_t nb, int n, float *grad, const MlpWork &w, cudaStream_t s);
// One Adam step with a given gradient.
cudaError_t mlp_adam(const MlpAdam &adam, const float *grad, cudaStream_t s);
// Boundary correction: corr[i] = scale_i * net(features_i / scale_i) for the strip nodes.
cudaError_t abc_correction(const MlpDev &net, const AbcArgs &a, cudaStream_t s);
// p_new[node_i] += corr[i].
cudaError_t abc_apply(const AbcArgs &a, float *p_new, float *hist, cudaStream_t s);
// hist[q] <- p^n (actual: stored value times the node's sponge factor) on the history shell.
cudaError_t abc_history(const int64_t *shell, int64_t n, const float *p_cur, const float *sx, const float *sy,
                        const float *sz, int64_t nxp, int64_t nz, float *hist, cudaStream_t s);

}  // namespace semgb
