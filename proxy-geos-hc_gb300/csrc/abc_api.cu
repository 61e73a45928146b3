// abc_api.cu -- C ABI of the learned absorbing boundary: the boundary network (sem_mlp_*) and
// its attachment to a solver (sem_abc_*).
//
// After every solver step the network corrects the new level on the strip nodes -- the boundary
// nodes themselves (layer 0), or the interior nodes within `layer` elements of a face -- from
// p^{n+1}, p^n and p^{n-1} on each node's 3x3x3
// neighbourhood (81 features, divided by their largest magnitude; the output, clipped to [-1, 1],
// is multiplied back).  On the boundary nodes it is the node's new value (so it never exceeds
// the largest magnitude of its neighbourhood), on interior strip nodes a correction.
// p^{n-1} of the strip and of its inner neighbour layer is kept in a history array.  The
// sponge of the solver (if any) still applies; the network replaces most of its thickness.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

#include "abi.h"
#include "mlp.h"
#include "solver.h"

using namespace semgb;

struct sem_mlp {
    float *d_master = nullptr;  // FP32 parameters (mlp.h layout)
    float *d_m = nullptr, *d_v = nullptr, *d_grad = nullptr;
    MlpWork work;               // training work arrays for up to work_rows rows
    int64_t work_rows = 0;
    uint16_t *d_w1 = nullptr, *d_w2 = nullptr;
    float *d_b1 = nullptr, *d_b2 = nullptr, *d_w3 = nullptr, *d_b3 = nullptr;
    double *d_loss = nullptr;
    int adam_t = 0;
    cudaStream_t stream = nullptr;
    MlpDev dev() const { return MlpDev{d_w1, d_w2, d_b1, d_b2, d_w3, d_b3}; }
    MlpAdam adam(float lr) { return MlpAdam{d_master, d_m, d_v, ++adam_t, lr, d_w1, d_w2, d_b1, d_b2, d_w3, d_b3}; }
};

struct sem_abc {
    sem_solver *s = nullptr;
    sem_mlp *net = nullptr;
    int layer = 0;
    int64_t *d_nodes = nullptr;  // strip nodes (device layout)
    int64_t n = 0;
    int64_t *d_shell = nullptr;  // history nodes: strip and its inner neighbours
    int64_t n_shell = 0;
    float *d_hist = nullptr;     // [n_int]
    float *d_corr = nullptr;     // [n]
    // layer 0: face tiles (abc_face) and a second history buffer: a step reads p^{n-1} from
    // hbuf[hcur] and writes p^n into the other
    bool face = false;
    int4 *d_tiles = nullptr;
    int64_t ntiles = 0;
    float *d_hist_alt = nullptr;
    int hcur = 0;
    FaceDesc faces[6];
    // kGraphSteps corrected steps replayed as one CUDA graph, per (current level, history buffer)
    // parity; valid while the solver's captured parameters are (graph_gen)
    cudaGraphExec_t graph[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
    uint64_t graph_gen = 0;
    int plain_runs = 0;  // runs of kGraphSteps launched since the graphs were dropped
    float *hist_now() const { return face && hcur ? d_hist_alt : d_hist; }
    float *hist_next() const { return face && !hcur ? d_hist_alt : d_hist; }
};

namespace {

void free_work(sem_mlp *m)
{
    MlpWork &w = m->work;
    dfree(w.xb); dfree(w.h1); dfree(w.dz1); dfree(w.dz2); dfree(w.g2); dfree(w.err); dfree(w.dy); dfree(w.part);
    dfree(w.lsum);
    m->work_rows = 0;
}

// Training work arrays for a pass over n rows (kept with the network: at most 86 MB; passes over
// more rows run in rounds).  The caller's stream is idle or about to use them.
cudaError_t ensure_work(sem_mlp *m, int64_t n)
{
    const int64_t rows = mlp_work_rows(n);
    if (rows <= m->work_rows) return cudaSuccess;
    free_work(m);
    MlpWork &w = m->work;
    const size_t r = (size_t)rows, slots = r / kMlpTile;
    cudaError_t e = dalloc(&w.xb, r * kMlpXbStride);
    if (e == cudaSuccess) e = dalloc(&w.h1, r * kMlpHidden);
    for (float **p : {&w.dz1, &w.dz2, &w.g2})
        if (e == cudaSuccess) e = dalloc(p, r * kMlpHidden);
    if (e == cudaSuccess) e = dalloc(&w.err, r);
    if (e == cudaSuccess) e = dalloc(&w.dy, r);
    if (e == cudaSuccess) e = dalloc(&w.part, slots * kMlpParams);
    if (e == cudaSuccess) e = dalloc(&w.lsum, slots * 32);
    if (e != cudaSuccess) {
        free_work(m);
        return e;
    }
    m->work_rows = rows;
    return cudaSuccess;
}

int net_upload(sem_mlp *m)
{
    CUDA_TRY(mlp_pack(m->d_master, m->d_w1, m->d_w2, m->d_b1, m->d_b2, m->d_w3, m->d_b3, m->stream));
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    return SEM_OK;
}

AbcArgs abc_args(const sem_abc *a)
{
    const sem_solver *s = a->s;
    const Box &b = s->mesh->box;
    AbcArgs x{};
    x.nodes = a->d_nodes;
    x.n = a->n;
    x.p_new = s->d_p[s->cur];      // after a step the new level is the current one
    x.p_cur = s->d_p[1 - s->cur];  // and p^n the stored previous one
    x.hist = a->hist_now();
    x.sx = s->sponge ? s->d_sx : nullptr;
    x.sy = s->sponge ? s->d_sy : nullptr;
    x.sz = s->sponge ? s->d_sz : nullptr;
    x.nx = b.nx;
    x.nxp = b.nxp;
    x.ny = b.ny;
    x.nz = b.nz;
    x.corr = a->d_corr;
    x.absolute = a->layer == 0 ? 1 : 0;
    return x;
}

// correction after the step that just ran (levels as abc_args reads them)
cudaError_t enqueue_correction(sem_abc *a)
{
    sem_solver *s = a->s;
    const AbcArgs x = abc_args(a);
    if (a->face) {
        AbcFaceArgs f{};
        for (int k = 0; k < 6; k++) f.face[k] = a->faces[k];
        f.tiles = a->d_tiles;
        f.ntiles = a->ntiles;
        f.p_new = s->d_p[s->cur];
        f.p_cur = x.p_cur;
        f.hist = a->hist_now();
        f.hist_next = a->hist_next();
        f.sx = x.sx; f.sy = x.sy; f.sz = x.sz;
        f.nx = x.nx; f.nxp = x.nxp; f.ny = x.ny; f.nz = x.nz;
        cudaError_t e = abc_face(a->net->dev(), f, s->stream);  // writes the new values in place
        if (e != cudaSuccess) return e;
        a->hcur ^= 1;
        return cudaSuccess;
    }
    cudaError_t e = abc_correction(a->net->dev(), x, s->stream);
    if (e != cudaSuccess) return e;
    if ((e = abc_apply(x, s->d_p[s->cur], a->d_hist, s->stream)) != cudaSuccess) return e;
    const Box &b = s->mesh->box;
    return abc_history(a->d_shell, a->n_shell, s->d_p[1 - s->cur], x.sx, x.sy, x.sz, b.nxp, b.nz, a->d_hist,
                       s->stream);
}

// No source node is read or written by the corrections: those reach the strip nodes' neighbours.
// The passes of a run of steps can then add the next step's sources before the correction runs.
bool sources_clear_of_strip(const sem_abc *a)
{
    const Box &b = a->s->mesh->box;
    const int64_t reach = (int64_t)a->layer * b.order + 1;
    for (int64_t q : a->s->src_group) {
        const int64_t iy = q / (b.nxp * b.nz), r = q - iy * b.nxp * b.nz, iz = r / b.nxp, ix = r - iz * b.nxp;
        if (std::min({ix, b.nx - 1 - ix, iy, b.ny - 1 - iy, iz, b.nz - 1 - iz}) <= reach) return false;
    }
    return true;
}

// n corrected steps from the current level and history buffer
cudaError_t enqueue_corrected(sem_abc *a, int n)
{
    sem_solver *s = a->s;
    const bool run = sources_clear_of_strip(a);
    for (int k = 0; k < n; k++) {
        StepExtra x;
        if (run) {
            x.advance = k == 0 ? n : 0;
            x.step_off = k;
            x.inject = k + 1 < n;
        }
        x.after = k > 0;
        cudaError_t e = solver_enqueue_step(s, s->cur, nullptr, &x);
        s->cur ^= 1;
        if (e == cudaSuccess) e = enqueue_correction(a);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- network -------------------------------------------------------------------------------

int sem_mlp_destroy(sem_mlp *m)
{
    if (!m) return SEM_OK;
    if (m->stream) cudaStreamSynchronize(m->stream);
    dfree(m->d_master); dfree(m->d_m); dfree(m->d_v); dfree(m->d_grad);
    free_work(m);
    dfree(m->d_w1); dfree(m->d_w2); dfree(m->d_b1); dfree(m->d_b2); dfree(m->d_w3); dfree(m->d_b3);
    dfree(m->d_loss);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return SEM_OK;
}

int sem_mlp_create(uint64_t seed, sem_mlp **out)
{
    GUARD_BEGIN
    if (!out) return sem_fail(SEM_ERR_ARG, "NULL argument");
    *out = nullptr;
    sem_mlp *m = new sem_mlp();
    cudaError_t e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = dalloc(&m->d_master, kMlpParams);
    if (e == cudaSuccess) e = dalloc(&m->d_m, kMlpParams);
    if (e == cudaSuccess) e = dalloc(&m->d_v, kMlpParams);
    if (e == cudaSuccess) e = dalloc(&m->d_grad, kMlpParams);
    if (e == cudaSuccess) e = mlp_train_setup();
    if (e == cudaSuccess) e = dalloc(&m->d_w1, kMlpHidden * kMlpInPad);
    if (e == cudaSuccess) e = dalloc(&m->d_w2, kMlpHidden * kMlpHidden);
    if (e == cudaSuccess) e = dalloc(&m->d_b1, kMlpHidden);
    if (e == cudaSuccess) e = dalloc(&m->d_b2, kMlpHidden);
    if (e == cudaSuccess) e = dalloc(&m->d_w3, kMlpHidden);
    if (e == cudaSuccess) e = dalloc(&m->d_b3, 1);
    if (e == cudaSuccess) e = dalloc(&m->d_loss, 1);
    if (e != cudaSuccess) {
        sem_mlp_destroy(m);
        return sem_fail(SEM_ERR_OOM, cudaGetErrorString(e));
    }
    // He-normal hidden layers, a small output layer (the initial correction is close to zero)
    std::mt19937_64 rng(seed);
    std::normal_distribution<float> nd(0.f, 1.f);
    std::vector<float> p(kMlpParams, 0.f);
    for (int i = 0; i < kMlpHidden * kMlpIn; i++) p[kOffW1 + i] = nd(rng) * std::sqrt(2.f / kMlpIn);
    for (int i = 0; i < kMlpHidden * kMlpHidden; i++) p[kOffW2 + i] = nd(rng) * std::sqrt(2.f / kMlpHidden);
    for (int i = 0; i < kMlpHidden; i++) p[kOffW3 + i] = nd(rng) * 0.01f;
    int rc = sem_mlp_set_params(m, p.data());
    if (rc) {
        sem_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return SEM_OK;
    GUARD_END
}

int sem_mlp_n_params(void) { return kMlpParams; }

int sem_mlp_set_params(sem_mlp *m, const float *params)
{
    GUARD_BEGIN
    if (!m || !params) return sem_fail(SEM_ERR_ARG, "NULL argument");
    for (int i = 0; i < kMlpParams; i++)
        if (!std::isfinite(params[i])) return sem_fail(SEM_ERR_ARG, "non-finite parameter");
    CUDA_TRY(cudaMemcpyAsync(m->d_master, params, kMlpParams * 4, cudaMemcpyHostToDevice, m->stream));
    CUDA_TRY(cudaMemsetAsync(m->d_m, 0, kMlpParams * 4, m->stream));
    CUDA_TRY(cudaMemsetAsync(m->d_v, 0, kMlpParams * 4, m->stream));
    m->adam_t = 0;
    return net_upload(m);
    GUARD_END
}

int sem_mlp_get_params(sem_mlp *m, float *params)
{
    GUARD_BEGIN
    if (!m || !params) return sem_fail(SEM_ERR_ARG, "NULL argument");
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    CUDA_TRY(cudaMemcpy(params, m->d_master, kMlpParams * 4, cudaMemcpyDeviceToHost));
    return SEM_OK;
    GUARD_END
}

int sem_mlp_forward(sem_mlp *m, int64_t n, const float *x, float *y)
{
    GUARD_BEGIN
    if (!m || n < 0 || (n > 0 && (!x || !y))) return sem_fail(SEM_ERR_ARG, "bad arguments");
    if (n == 0) return SEM_OK;
    float *dx = nullptr, *dy = nullptr;
    CUDA_TRY(dalloc(&dx, (size_t)n * kMlpIn));
    cudaError_t e = dalloc(&dy, (size_t)n);
    if (e == cudaSuccess) e = upload(dx, x, (size_t)n * kMlpIn, m->stream);
    if (e == cudaSuccess) e = mlp_forward(m->dev(), dx, dy, n, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e == cudaSuccess) e = cudaMemcpy(y, dy, (size_t)n * 4, cudaMemcpyDeviceToHost);
    dfree(dx);
    dfree(dy);
    CUDA_TRY(e);
    return SEM_OK;
    GUARD_END
}

int sem_mlp_loss_grad(sem_mlp *m, int64_t n, const float *x, const float *t, double *loss, float *grad)
{
    GUARD_BEGIN
    if (!m || n < 1 || !x || !t) return sem_fail(SEM_ERR_ARG, "bad arguments");
    float *dx = nullptr, *dt = nullptr;
    CUDA_TRY(dalloc(&dx, (size_t)n * kMlpIn));
    cudaError_t e = dalloc(&dt, (size_t)n);
    if (e == cudaSuccess) e = upload(dx, x, (size_t)n * kMlpIn, m->stream);
    if (e == cudaSuccess) e = upload(dt, t, n, m->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->d_grad, 0, kMlpParams * 4, m->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->d_loss, 0, 8, m->stream);
    if (e == cudaSuccess) e = ensure_work(m, n);
    if (e == cudaSuccess) e = mlp_loss_grad(m->dev(), dx, dt, n, m->d_loss, m->d_grad, m->work, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e == cudaSuccess && loss) e = cudaMemcpy(loss, m->d_loss, 8, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && grad) e = cudaMemcpy(grad, m->d_grad, kMlpParams * 4, cudaMemcpyDeviceToHost);
    dfree(dx);
    dfree(dt);
    CUDA_TRY(e);
    return SEM_OK;
    GUARD_END
}

int sem_mlp_train(sem_mlp *m, int64_t n, const float *x, const float *t, int epochs, int batch, float lr,
                  uint64_t seed, double *losses)
{
    GUARD_BEGIN
    if (!m || n < 1 || !x || !t || epochs < 0 || batch < 1 || !(lr > 0))
        return sem_fail(SEM_ERR_ARG, "bad arguments");
    // samples resident on the device; their order is shuffled once per epoch on the host, while the
    // device still runs the epoch before: two index arrays in turn, each copied on its own stream
    const int64_t nb = std::min<int64_t>(batch, n), nbatch = n / nb;
    float *dx = nullptr, *dt = nullptr;
    int64_t *dperm[2] = {nullptr, nullptr};
    double *dl = nullptr;
    cudaStream_t copy = nullptr;
    cudaEvent_t done[2] = {nullptr, nullptr};
    cudaError_t e = dalloc(&dx, (size_t)n * kMlpIn);
    if (e == cudaSuccess) e = dalloc(&dt, (size_t)n);
    for (auto &p : dperm)
        if (e == cudaSuccess) e = dalloc(&p, (size_t)n);
    if (e == cudaSuccess) e = dalloc(&dl, (size_t)std::max(epochs, 1) * nbatch);
    if (e == cudaSuccess) e = ensure_work(m, nb);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&copy, cudaStreamNonBlocking);
    for (auto &v : done)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dx, x, (size_t)n * kMlpIn * 4, cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dt, t, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream);
    std::vector<int64_t> perm(n);
    for (int64_t i = 0; i < n; i++) perm[i] = i;
    std::mt19937_64 rng(seed);
    for (int ep = 0; ep < epochs && e == cudaSuccess; ep++) {
        std::shuffle(perm.begin(), perm.end(), rng);
        const int k = ep & 1;
        if (ep >= 2) e = cudaEventSynchronize(done[k]);  // the epoch that last read this index array
        if (e == cudaSuccess) e = cudaMemcpyAsync(dperm[k], perm.data(), (size_t)n * 8, cudaMemcpyHostToDevice, copy);
        if (e == cudaSuccess) e = cudaStreamSynchronize(copy);
        for (int64_t j = 0; j < nbatch && e == cudaSuccess; j++)
            e = mlp_train_step(m->dev(), dx, dt, dperm[k] + j * nb, nb, dl + ep * nbatch + j, m->adam(lr), m->work,
                               m->stream, j > 0);
        if (e == cudaSuccess) e = cudaEventRecord(done[k], m->stream);
    }
    const cudaError_t es = cudaStreamSynchronize(m->stream);
    if (e == cudaSuccess) e = es;
    if (e == cudaSuccess && losses && epochs > 0) {
        std::vector<double> l((size_t)epochs * nbatch);
        e = cudaMemcpy(l.data(), dl, l.size() * 8, cudaMemcpyDeviceToHost);
        for (int ep = 0; ep < epochs; ep++) {
            double lsum = 0.0;
            for (int64_t j = 0; j < nbatch; j++) lsum += l[ep * nbatch + j] * nb;
            losses[ep] = lsum / (nbatch * nb);
        }
    }
    dfree(dx); dfree(dt); dfree(dperm[0]); dfree(dperm[1]); dfree(dl);
    for (auto v : done)
        if (v) cudaEventDestroy(v);
    if (copy) cudaStreamDestroy(copy);
    CUDA_TRY(e);
    return SEM_OK;
    GUARD_END
}

int sem_mlp_adam_step(sem_mlp *m, const float *grad, float lr)
{
    GUARD_BEGIN
    if (!m || !grad || !(lr > 0)) return sem_fail(SEM_ERR_ARG, "bad arguments");
    CUDA_TRY(cudaMemcpyAsync(m->d_grad, grad, kMlpParams * 4, cudaMemcpyHostToDevice, m->stream));
    CUDA_TRY(mlp_adam(m->adam(lr), m->d_grad, m->stream));
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    return SEM_OK;
    GUARD_END
}

// ---- boundary ------------------------------------------------------------------------------

int sem_abc_destroy(sem_abc *a)
{
    if (!a) return SEM_OK;
    // the solver may already be gone (handles closed in any order): wait for the device instead
    // of the solver's stream
    cudaDeviceSynchronize();
    for (auto &row : a->graph)
        for (auto &g : row)
            if (g) cudaGraphExecDestroy(g);
    dfree(a->d_nodes);
    dfree(a->d_shell);
    dfree(a->d_hist);
    dfree(a->d_corr);
    dfree(a->d_tiles);
    dfree(a->d_hist_alt);
    delete a;
    return SEM_OK;
}

int sem_abc_create(sem_solver *s, sem_mlp *net, int layer_elems, sem_abc **out)
{
    GUARD_BEGIN
    if (!s || !net || !out) return sem_fail(SEM_ERR_ARG, "NULL argument");
    *out = nullptr;
    const Box &b = s->mesh->box;
    if (layer_elems < 0 || 2 * layer_elems > std::min({b.ex, b.ey, b.ez}))
        return sem_fail(SEM_ERR_ARG, "layer must be >= 0 elements and fit twice in every axis");
    // layer 0: the boundary nodes themselves (the network supplies the face values that the
    // Dirichlet update would hold fixed); layer w > 0: interior nodes within w elements of a face
    const int64_t w = (int64_t)layer_elems * b.order;
    std::vector<int64_t> nodes, shell;
    for (int64_t iy = 0; iy < b.ny; iy++)
        for (int64_t iz = 0; iz < b.nz; iz++)
            for (int64_t ix = 0; ix < b.nx; ix++) {
                const int64_t d = std::min({ix, b.nx - 1 - ix, iy, b.ny - 1 - iy, iz, b.nz - 1 - iz});
                const int64_t q = ix + iz * b.nxp + iy * b.nxp * b.nz;
                if (w == 0 ? d == 0 : (d >= 1 && d <= w)) nodes.push_back(q);
                if (d <= w + 1) shell.push_back(q);
            }
    sem_abc *a = new sem_abc();
    a->s = s;
    a->net = net;
    a->layer = layer_elems;
    a->n = (int64_t)nodes.size();
    a->n_shell = (int64_t)shell.size();
    cudaError_t e = dalloc(&a->d_nodes, nodes.size());
    if (e == cudaSuccess) e = dalloc(&a->d_shell, shell.size());
    if (e == cudaSuccess) e = dalloc(&a->d_hist, (size_t)b.n_int);
    if (e == cudaSuccess) e = dalloc(&a->d_corr, nodes.size());
    if (e == cudaSuccess) e = upload(a->d_nodes, nodes.data(), nodes.size(), s->stream);
    if (e == cudaSuccess) e = upload(a->d_shell, shell.data(), shell.size(), s->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(a->d_hist, 0, (size_t)b.n_int * 4, s->stream);
    if (e == cudaSuccess && layer_elems == 0) {
        // face tiles: y-faces whole, z-faces without the rows on y-faces, x-faces without the
        // rows on y- and z-faces, so every boundary node lies on one face
        const int64_t nx = b.nx, ny = b.ny, nz = b.nz;
        const int64_t dims[3] = {nx, ny, nz};
        struct Spec { int n, u, v; int64_t ulo, uhi, vlo, vhi; };
        const Spec spec[3] = {{1, 0, 2, 0, nx, 0, nz}, {2, 0, 1, 0, nx, 1, ny - 1}, {0, 2, 1, 1, nz - 1, 1, ny - 1}};
        std::vector<int4> tiles;
        for (int k = 0; k < 6; k++) {
            const Spec &sp = spec[k / 2];
            FaceDesc &f = a->faces[k];
            f.axis_n = sp.n; f.axis_u = sp.u; f.axis_v = sp.v;
            f.side = (k % 2 == 0) ? 0 : (int)(dims[sp.n] - 1);
            f.inward = (k % 2 == 0) ? 1 : -1;
            f.ulo = (int)sp.ulo; f.uhi = (int)sp.uhi; f.vlo = (int)sp.vlo; f.vhi = (int)sp.vhi;
            // a tile row is a node of the face where it lies within [ulo, uhi) x [vlo, vhi); every
            // such node is a boundary node (the strip of layer 0)
            for (int64_t v0 = sp.vlo; v0 < sp.vhi; v0 += kFaceTV)
                for (int64_t u0 = sp.ulo; u0 < sp.uhi; u0 += kFaceTU) tiles.push_back(make_int4(k, (int)u0, (int)v0, 0));
        }
        a->face = true;
        a->ntiles = (int64_t)tiles.size();
        e = dalloc(&a->d_tiles, tiles.size());
        if (e == cudaSuccess) e = dalloc(&a->d_hist_alt, (size_t)b.n_int);
        if (e == cudaSuccess) e = upload(a->d_tiles, tiles.data(), tiles.size(), s->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(a->d_hist_alt, 0, (size_t)b.n_int * 4, s->stream);
    }
    if (e != cudaSuccess) {
        sem_abc_destroy(a);
        return sem_fail(SEM_ERR_OOM, cudaGetErrorString(e));
    }
    *out = a;
    return SEM_OK;
    GUARD_END
}

int sem_abc_info(const sem_abc *a, int64_t *n_nodes, int64_t *n_history)
{
    if (!a) return sem_fail(SEM_ERR_ARG, "NULL boundary");
    if (n_nodes) *n_nodes = a->n;
    if (n_history) *n_history = a->n_shell;
    return SEM_OK;
}

int sem_abc_nodes(const sem_abc *a, int64_t *nodes)
{
    GUARD_BEGIN
    if (!a || !nodes) return sem_fail(SEM_ERR_ARG, "NULL argument");
    std::vector<int64_t> q(a->n);
    CUDA_TRY(cudaMemcpy(q.data(), a->d_nodes, a->n * 8, cudaMemcpyDeviceToHost));
    for (int64_t i = 0; i < a->n; i++) nodes[i] = to_reference(a->s->mesh->box, q[i]);
    return SEM_OK;
    GUARD_END
}

int sem_abc_reset(sem_abc *a)
{
    GUARD_BEGIN
    if (!a) return sem_fail(SEM_ERR_ARG, "NULL boundary");
    // on the solver's stream, ordered with the steps (see sem_solver_reset)
    cudaStream_t st = a->s->stream;
    CUDA_TRY(cudaMemsetAsync(a->d_hist, 0, (size_t)a->s->mesh->box.n_int * 4, st));
    if (a->d_hist_alt) CUDA_TRY(cudaMemsetAsync(a->d_hist_alt, 0, (size_t)a->s->mesh->box.n_int * 4, st));
    a->hcur = 0;
    return SEM_OK;
    GUARD_END
}

int sem_abc_set_history(sem_abc *a, const float *p_prev)
{
    GUARD_BEGIN
    if (!a || !p_prev) return sem_fail(SEM_ERR_ARG, "NULL argument");
    const Box &b = a->s->mesh->box;
    CUDA_TRY(cudaStreamSynchronize(a->s->stream));
    CUDA_TRY(field_from_host(a->hist_now(), p_prev, b.nx, b.nxp, b.nz * b.ny, a->s->stream));
    return SEM_OK;
    GUARD_END
}

int sem_abc_step(sem_abc *a, int n_steps)
{
    GUARD_BEGIN
    if (!a || n_steps < 0) return sem_fail(SEM_ERR_ARG, "bad arguments");
    if (n_steps == 0) return SEM_OK;
    sem_solver *s = a->s;
    if (s->kernel == SEM_KERNEL_ELEMENT) return sem_fail(SEM_ERR_STATE, "the learned boundary runs with the stencil pass");
    int rc = solver_prepare(s, n_steps);
    if (rc) return rc;
    if (a->graph_gen != s->graph_gen) {
        for (auto &row : a->graph)
            for (auto &g : row)
                if (g) { cudaGraphExecDestroy(g); g = nullptr; }
        a->graph_gen = s->graph_gen;
        a->plain_runs = 0;
    }
    int done = 0;
    for (; n_steps - done >= kGraphSteps; done += kGraphSteps) {
        cudaGraphExec_t &ge = a->graph[s->cur][a->hcur];
        if (!ge && a->plain_runs + (n_steps - done) / kGraphSteps <= kPlainRuns) {
            // (first 16 steps, graph -> launches: 8^3 elements of order 4 357 -> 240 us, 24^3 514 -> 386; 128 steps
            // 1703 -> 1728, 2932 -> 2897)
            CUDA_TRY(enqueue_corrected(a, kGraphSteps));
            a->plain_runs++;
            continue;
        }
        if (!ge) {
            // an even number of steps: the level and history parities come back to where they
            // started
            cudaGraph_t g = nullptr;
            CUDA_TRY(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
            const cudaError_t e = enqueue_corrected(a, kGraphSteps);
            const cudaError_t e2 = cudaStreamEndCapture(s->stream, &g);
            if (e != cudaSuccess || e2 != cudaSuccess) {
                if (g) cudaGraphDestroy(g);
                return sem_fail(SEM_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e != cudaSuccess ? e : e2));
            }
            const cudaError_t e3 = cudaGraphInstantiate(&ge, g, 0);
            cudaGraphDestroy(g);
            if (e3 != cudaSuccess) return sem_fail(SEM_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e3));
        }
        CUDA_TRY(cudaGraphLaunch(ge, s->stream));
    }
    CUDA_TRY(enqueue_corrected(a, n_steps - done));
    s->steps_done += n_steps;
    return SEM_OK;
    GUARD_END
}

int sem_abc_bptt(sem_abc *a, int n_steps, int n_roi, const int64_t *roi_nodes, const float *ref, double *loss,
                 float *grad)
{
    GUARD_BEGIN
    if (!a || n_steps < 1 || n_roi < 0 || (n_roi > 0 && (!roi_nodes || !ref)) || !loss)
        return sem_fail(SEM_ERR_ARG, "bad arguments");
    if (!a->face) return sem_fail(SEM_ERR_STATE, "the adjoint runs with the network on the boundary nodes (layer 0)");
    sem_solver *s = a->s;
    const Box &b = s->mesh->box;
    // sources must lie outside every boundary node's neighbourhood: the recorded levels do not
    // hold the source term a step adds before it reads them
    for (int64_t q : s->src_node) {
        const int64_t iy = q / (b.nxp * b.nz), r = q - iy * b.nxp * b.nz, iz = r / b.nxp, ix = r - iz * b.nxp;
        if (ix < 2 || ix > b.nx - 3 || iy < 2 || iy > b.ny - 3 || iz < 2 || iz > b.nz - 3)
            return sem_fail(SEM_ERR_ARG, "a source lies within two nodes of the boundary");
    }
    std::vector<int64_t> roi(n_roi);
    for (int r = 0; r < n_roi; r++) {
        if (roi_nodes[r] < 0 || roi_nodes[r] >= b.n_nodes) return sem_fail(SEM_ERR_ARG, "region node out of range");
        roi[r] = to_internal(b, roi_nodes[r]);
    }
    int rc = sem_solver_reset(s);
    if (rc) return rc;
    if ((rc = sem_abc_reset(a))) return rc;
    if ((rc = solver_prepare(s, n_steps))) return rc;
    const int64_t n_int = b.n_int, nb = a->n;
    cudaStream_t st = s->stream;

    // work arrays (freed on every exit path)
    float *rec = nullptr, *dx = nullptr;
    float *A[3] = {nullptr, nullptr, nullptr}, *v = nullptr, *dref = nullptr;
    int *sidx = nullptr, *ridx = nullptr;
    int64_t *droi = nullptr;
    double *dloss = nullptr;
    const int64_t dx_stride = (nb + 31) / 32 * 32;
    auto release = [&]() {
        cudaStreamSynchronize(st);
        dfree(rec); dfree(dx);
        for (auto &p : A) dfree(p);
        dfree(v); dfree(dref); dfree(sidx); dfree(ridx); dfree(droi); dfree(dloss);
    };
    cudaError_t e = dalloc(&rec, (size_t)(n_steps + 2) * n_int);
    if (e == cudaSuccess && n_roi > 0) e = dalloc(&dref, (size_t)n_steps * n_roi);
    if (e == cudaSuccess && n_roi > 0) e = dalloc(&droi, (size_t)n_roi);
    if (e == cudaSuccess) e = dalloc(&dloss, (size_t)n_steps);
    if (grad) {
        if (e == cudaSuccess) e = dalloc(&dx, (size_t)dx_stride * kMlpIn);
        if (e == cudaSuccess) e = ensure_work(a->net, mlp_boundary_groups(nb) * mlp_work_rows(nb));
        for (auto &p : A)
            if (e == cudaSuccess) e = dalloc(&p, (size_t)n_int);
        if (e == cudaSuccess) e = dalloc(&v, (size_t)n_int);
        if (e == cudaSuccess) e = dalloc(&sidx, (size_t)n_int);
        std::vector<int64_t> nodes(nb);
        if (e == cudaSuccess) e = cudaMemcpy(nodes.data(), a->d_nodes, nb * 8, cudaMemcpyDeviceToHost);
        std::vector<int> map(n_int, -1);
        for (int64_t i = 0; i < nb; i++) map[nodes[i]] = (int)i;
        if (e == cudaSuccess) e = upload(sidx, map.data(), n_int, st);
        std::fill(map.begin(), map.end(), -1);
        bool twice = false;
        for (int r = 0; r < n_roi; r++) {
            twice = twice || map[roi[r]] >= 0;
            map[roi[r]] = r;
        }
        if (!twice && n_roi > 0) {
            if (e == cudaSuccess) e = dalloc(&ridx, (size_t)n_int);
            if (e == cudaSuccess) e = upload(ridx, map.data(), n_int, st);
        }
    }
    // (both outlive the copies: the call waits for its stream before it returns)
    if (e == cudaSuccess && n_roi > 0) e = cudaMemcpyAsync(droi, roi.data(), (size_t)n_roi * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && n_roi > 0)
        e = cudaMemcpyAsync(dref, ref, (size_t)n_steps * n_roi * 4, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(rec, 0, 2 * n_int * 4, st);  // p^{-1} = p^0 = 0: from rest
    // forward, the levels after every step recorded (by a kernel: the chain of dependent launches
    // goes on)
    for (int m = 1; m <= n_steps && e == cudaSuccess; m++) {
        StepExtra x;
        x.after = m > 1;
        e = solver_enqueue_step(s, s->cur, nullptr, &x);
        s->cur ^= 1;
        if (e == cudaSuccess) e = enqueue_correction(a);
        if (e == cudaSuccess) e = bptt_copy_level(s->d_p[s->cur], rec + (size_t)(m + 1) * n_int, n_int, st);
    }
    s->steps_done += n_steps;
    BpttFields f{};
    f.nx = (int)b.nx; f.ny = (int)b.ny; f.nz = (int)b.nz;
    f.nxp = b.nxp; f.n_int = n_int;
    f.sx = s->sponge ? s->d_sx : nullptr;
    f.sy = s->sponge ? s->d_sy : nullptr;
    f.sz = s->sponge ? s->d_sz : nullptr;
    f.nodes = a->d_nodes; f.nb = nb; f.sidx = sidx;
    f.shell = a->d_shell; f.n_shell = a->n_shell;
    f.dx = dx; f.dx_stride = dx_stride; f.ridx = ridx;
    for (int k = 0; k < 3; k++) f.a[k] = A[k];
    f.v = v; f.roi = droi; f.n_roi = n_roi;
    if (e == cudaSuccess && n_roi > 0) e = bptt_losses(f, rec + 2 * n_int, n_int, dref, n_steps, dloss, st);
    if (grad) {
        for (auto p : A)
            if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, n_int * 4, st);
        BpttOperator op{};
        op.order = b.order;
        Gll gl;
        gll_tables(b.order, gl);
        stencil_table(gl, op.T);
        const int W = 2 * b.order + 1;
        for (int l = 0; l < b.order; l++) {
            // the direct form's diagonal: minus the rounded row sum, as the stencil pass uses it
            double sum = 0;
            for (int d = -b.order; d <= b.order; d++)
                if (d != 0) sum += op.T[l * W + d + b.order];
            op.T[l * W + b.order] = (float)-sum;
            op.wa[l] = s->stencil->wa[l];
        }
        for (int k = 0; k < 3; k++) op.g[k] = s->stencil->g[k];
        sem_mlp *net = a->net;
        if (e == cudaSuccess) e = cudaMemsetAsync(net->d_grad, 0, kMlpParams * 4, st);
        auto level = [&](int m) { return rec + (size_t)(m + 1) * n_int; };
        auto ref_of = [&](int m) { return dref + (size_t)(m - 1) * n_roi; };
        const int groups = mlp_boundary_groups(nb);
        int group = 0;
        if (e == cudaSuccess) e = bptt_seed(f, level(n_steps), ref_of(n_steps), st);
        for (int m = n_steps; m >= 1 && e == cudaSuccess; m--) {
            e = mlp_boundary_rows(net->dev(), f, level(m), level(m - 1), level(m - 2), group++, net->work, net->d_grad, st);
            if (e == cudaSuccess && (group == groups || m == 1)) {
                e = mlp_boundary_params(nb, group, net->d_grad, net->work, st);
                group = 0;
            }
            if (e == cudaSuccess) e = bptt_scatter(f, s->d_a, st);
            const bool fused = ridx && m > 1;
            if (e == cudaSuccess)
                e = bptt_interior(f, op, fused ? level(m - 1) : nullptr, fused ? ref_of(m - 1) : nullptr, st);
            // the adjoints move one level back: out^{m-1} becomes the newest
            std::swap(f.a[0], f.a[1]);
            std::swap(f.a[1], f.a[2]);
            if (e == cudaSuccess && !ridx && m > 1) e = bptt_seed(f, level(m - 1), ref_of(m - 1), st);
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(grad, net->d_grad, kMlpParams * 4, cudaMemcpyDeviceToHost, st);
    }
    std::vector<double> step_loss(n_steps, 0.0);
    if (e == cudaSuccess && n_roi > 0)
        e = cudaMemcpyAsync(step_loss.data(), dloss, (size_t)n_steps * 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (grad) std::reverse(step_loss.begin(), step_loss.end());  // (summed newest step first, as the sweep runs)
    double sum = 0.0;
    for (double l : step_loss) sum += l;
    if (e == cudaSuccess) *loss = sum;
    release();
    CUDA_TRY(e);
    return SEM_OK;
    GUARD_END
}

int sem_abc_correct(sem_abc *a)
{
    GUARD_BEGIN
    if (!a) return sem_fail(SEM_ERR_ARG, "NULL boundary");
    CUDA_TRY(enqueue_correction(a));
    return SEM_OK;
    GUARD_END
}

int sem_abc_features(sem_abc *a, float *x, float *scale)
{
    GUARD_BEGIN
    if (!a || !x) return sem_fail(SEM_ERR_ARG, "NULL argument");
    // the features exactly as k_abc_correction gathers them (same order, sponge product and
    // scaling), from host copies of the levels: training sets are built from these
    sem_solver *s = a->s;
    const Box &b = s->mesh->box;
    CUDA_TRY(cudaStreamSynchronize(s->stream));
    std::vector<float> pn(b.n_int), pc(b.n_int), ph(b.n_int);
    CUDA_TRY(cudaMemcpy(pn.data(), s->d_p[s->cur], b.n_int * 4, cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemcpy(pc.data(), s->d_p[1 - s->cur], b.n_int * 4, cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemcpy(ph.data(), a->hist_now(), b.n_int * 4, cudaMemcpyDeviceToHost));
    std::vector<float> sx(b.nx, 1.f), sy(b.ny, 1.f), sz(b.nz, 1.f);
    if (s->sponge) {
        CUDA_TRY(cudaMemcpy(sx.data(), s->d_sx, b.nx * 4, cudaMemcpyDeviceToHost));
        CUDA_TRY(cudaMemcpy(sy.data(), s->d_sy, b.ny * 4, cudaMemcpyDeviceToHost));
        CUDA_TRY(cudaMemcpy(sz.data(), s->d_sz, b.nz * 4, cudaMemcpyDeviceToHost));
    }
    std::vector<int64_t> q(a->n);
    CUDA_TRY(cudaMemcpy(q.data(), a->d_nodes, a->n * 8, cudaMemcpyDeviceToHost));
    const int64_t plane = b.nxp * b.nz;
    for (int64_t i = 0; i < a->n; i++) {
        const int64_t iy = q[i] / plane, rr = q[i] - iy * plane, iz = rr / b.nxp, ix = rr - iz * b.nxp;
        float m = 0.f;
        float *f = x + i * kMlpIn;
        for (int l = 0; l < 3; l++)
            for (int nb = 0; nb < 27; nb++) {
                const int dz = nb / 9 - 1, dy = (nb / 3) % 3 - 1, dx = nb % 3 - 1;
                const int64_t jx = ix + dx, jy = iy + dy, jz = iz + dz;
                float v = 0.f;
                if (jx >= 0 && jx < b.nx && jy >= 0 && jy < b.ny && jz >= 0 && jz < b.nz) {
                    const int64_t qj = jx + jz * b.nxp + jy * plane;
                    v = l == 0 ? pn[qj] : l == 1 ? pc[qj] * ((sx[jx] * sy[jy]) * sz[jz]) : ph[qj];
                }
                f[l * 27 + nb] = v;
                m = std::max(m, std::fabs(v));
            }
        const float sc = m + 1e-30f;
        for (int k = 0; k < kMlpIn; k++) f[k] /= sc;
        if (scale) scale[i] = sc;
    }
    return SEM_OK;
    GUARD_END
}

}  // extern "C"
