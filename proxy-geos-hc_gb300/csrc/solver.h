// solver.h -- the solver handle (struct sem_solver) and the internal step interface shared by
// the C-ABI translation units (api.cu: plain solver; adjoint_api.cu: checkpointed adjoint).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <functional>
#include <vector>

#include "abi.h"
#include "stencil.h"

// Steps per captured graph (even: the level parity returns).  Inside one, passes follow each other
// as programmatic dependents and only the first step has a source launch; between graphs the
// launch gap is that of an ordinary kernel boundary.  Per step, against two steps (four kernels) per
// graph: 40^3 elements of order 2 7.3 -> 4.7 us, 61 x 70 x 53 of order 4 52.5 -> 49.0, 80 x 77 x 83
// of order 5 304.7 -> 291.9, 200^3 of order 4 1394.6 -> 1392.2, a group of 32 small boxes 36.7 -> 34.1.
constexpr int kGraphSteps = 16;

// Runs of kGraphSteps launched after a change (sources, receivers, model) before their graph is made: capturing
// and instantiating one costs more than replaying saves over few steps.  The first 16 steps after a change,
// graph -> launches: 12^3 elements of order 2 160 -> 103 us, 24^3 of order 4 231 -> 176, 40^3 400 -> 346; 128
// steps 638 -> 597, 1200 -> 1173, 2550 -> 2514; beyond, the host's time counts.
constexpr int kPlainRuns = 8;

struct sem_solver {
    sem_mesh *mesh = nullptr;
    float dt = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int kernel = SEM_KERNEL_AUTO;
    int form = SEM_FORM_DIRECT;  // operator form of the stencil pass
    int rounding = SEM_ROUNDING_DEFAULT;  // SEM_ROUNDING_REFERENCE: the reference's rounded rows
    int64_t n_int = 0;               // nodes of the device layout
    float *d_p[2] = {nullptr, nullptr};
    int cur = 0;                 // index of the current level
    float *d_y = nullptr;        // element path accumulator
    float *d_a = nullptr;        // dt^2 / M
    uint64_t a_version = 0;
    float *d_tab = nullptr;      // element coefficient table
    float *d_rtab = nullptr;     // SEM_ROUNDING_REFERENCE: the reference's element rows (element path)
    float *d_mref = nullptr;     // SEM_ROUNDING_REFERENCE: the reference's float mass (element path)
    uint64_t mref_version = 0;
    double *d_w = nullptr;       // GLL weights (double) for the mass kernel
    semgb::StencilTables *stencil = nullptr;
    int tile_shape = -1;  // stencil tile shape: -1 chosen per box, or a semgb::StencilTileShape
    // sponge
    bool sponge = false;
    float *d_sx = nullptr, *d_sy = nullptr, *d_sz = nullptr;
    std::vector<float> h_sx, h_sy, h_sz;  // the same on the host
    float *pin = nullptr, *d_pin = nullptr;  // pinned staging of receiver rows (sem_solver_step_host)
    // sources
    int nsrc = 0, nsamples = 0;
    int64_t *d_src_node = nullptr;
    int *d_src_off = nullptr, *d_src_perm = nullptr;  // sources grouped by node (SourceTable)
    std::vector<int64_t> src_group;                   // node of each group
    uint64_t src_version = 1;
    float *d_src_coef = nullptr;
    float *d_wavelet = nullptr;
    std::vector<int64_t> src_node;
    std::vector<float> src_coef;
    // receivers
    int nrec = 0;
    int64_t *d_rec_node = nullptr;  // sorted by node
    int *d_rec_perm = nullptr;      // sorted position -> caller's receiver index
    std::vector<int64_t> rec_sorted;
    uint64_t rec_version = 1;
    float *d_traces = nullptr;      // [trace_cap][nrec]
    int64_t trace_cap = 0;
    int64_t traces_checked = 0;
    int *d_ctr = nullptr;           // [0] next step, [1] step in flight
    int *d_status = nullptr;        // non-zero after a bounded device wait gave up
    int *d_upd_rec_off = nullptr;   // receivers grouped by update-kernel block
    uint64_t upd_rec_version = 0;
    int64_t steps_done = 0;
    // graphs: [parity] kGraphSteps steps starting at level `parity`
    cudaGraphExec_t graph[2] = {nullptr, nullptr};
    cudaGraphExec_t pair[2] = {nullptr, nullptr};  // two steps of the element path
    int plain_runs = 0;  // runs of kGraphSteps enqueued without their graph since the last change
    uint64_t graph_gen = 0;  // bumped whenever captured launch parameters may have changed
};

// Side buffers of one stencil pass (modes of k_stencil.cu: record K p, or accumulate a gradient).
struct StepExtra {
    int mode = semgb::STENCIL_PLAIN;
    float *kp = nullptr;
    float *grad = nullptr;
    // place in a run of steps: steps the source launch covers (0: the pass before added this
    // step's sources), steps since it, whether this pass adds the next step's, and whether the
    // preceding kernel on the stream belongs to the run
    int advance = 1, step_off = 0;
    bool inject = false, after = false;
    const semgb::HostSamples *samples = nullptr;  // this step's source samples, by value (advance 1)
};

// Device resources for stepping n_new more steps (mass, stencil tables, receiver CSR, trace
// storage).  Returns a SEM_* status.
int solver_prepare(sem_solver *s, int64_t n_new);
// One step from level c (source, stiffness + update, receivers) enqueued on the solver stream.
cudaError_t solver_enqueue_step(sem_solver *s, int c, cudaEvent_t *ev = nullptr, const StepExtra *extra = nullptr);
// n steps from level c with nothing between them.  side(k) (may be empty) gives step k's side buffers.
cudaError_t solver_enqueue_run(sem_solver *s, int c, int n, const std::function<StepExtra(int)> &side = nullptr);
void solver_invalidate_graphs(sem_solver *s);
// The source table that the solver's launches read.
semgb::SourceTable solver_sources(const sem_solver *s);
// Sources by device-layout node with explicit coefficients: p^n[node_k] += coef_k * wavelet_k[n].
int solver_set_raw_sources(sem_solver *s, int n_src, const int64_t *nodes, const float *coef, const float *wavelet,
                           int n_samples);
// A field between the device layout (rows of nxp floats) and a host array in the reference
// layout (rows of nx floats), `rows` rows, through two pinned staging buffers: the copy engine
// gathers (scatters) one chunk of rows while the host moves the previous one, so the caller's
// pageable array is not crossed row by row.  Ordered on and synchronous with stream s.
cudaError_t field_to_host(float *dst, const float *src, int64_t nx, int64_t nxp, int64_t rows, cudaStream_t s);
cudaError_t field_from_host(float *dst, const float *src, int64_t nx, int64_t nxp, int64_t rows, cudaStream_t s);
