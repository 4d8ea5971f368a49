// Internal structures of libglgpu: instance descriptors, device-side loop state,
// the handle, and the host-side launch helpers shared by the translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <string>
#include <vector>

#include "glgpu_common.cuh"
#include "../../include/glgpu.h"

namespace glgpu {

// Temporal blocking of the FP32 psi Jacobi loop: a round (a launch, for the bulk-copy
// kernel) does kFuse consecutive sweeps, and the loop can stop after any of them exactly
// where a loop of single sweeps stops: the bulk-copy kernel stores every sweep, a round of
// k_psi_loop_f32 (tdl.cu) its last, or all, or is repeated up to the sweep that it lacks.
#ifndef GLGPU_FUSE
#define GLGPU_FUSE 3
#endif
constexpr int kFuse = GLGPU_FUSE;
static_assert(kFuse >= 1 && kFuse <= 4, "1 <= GLGPU_FUSE <= 4");
constexpr int kPsiBufs = kFuse + 2;  // right-hand side, input, the kFuse outputs
// TD graphs cached per handle / batch: eqn mode (3) x any finite kappa (2) x any
// fixed vortices (2)
constexpr int kTDGraphs = 12;

// Device-resident state of one instance's Jacobi loops (updated by the kernels
// themselves so that a whole TD run needs no host round trip).
struct InstState {
    unsigned long long res;   // A loop: max residual of the current sweep, as IEEE bits
    unsigned long long resp[4];  // psi loop: max residual of each sweep of the current launch
    int nanlv;                // psi loop: bit l set if sweep l of the current launch saw a NaN residual
    unsigned blocks_done;     // CTAs (A) / strips (psi) of this instance finished in the current launch
    int sweep;                // sweeps done in the current Jacobi loop
    int done;                 // current Jacobi loop finished
    int rhs;                  // buffer index (0..kPsiBufs-1) of psi^(0) = right-hand side of the psi loop
    int rhsA;                 // same for the A loop (0..2)
    uint32_t rand_t;          // Langevin time seed (svirl/solvers/td.py:35-37,204,313)
    int nan_seen;             // a NaN residual was seen (the reference counts it as converged)
    int last_sweeps_psi, last_sweeps_A, max_sweeps_psi, max_sweeps_A;
    long long total_sweeps_psi, total_sweeps_A;
    int steps;                // time steps done in the current call
    int redo, keep;           // cooperative loops (tdl.cu): what the next round repeats the last one for (0: it
                              // does not), which sweeps the round keeps
    int commitA;              // FP32 A loop: 1 + the buffer of A^(0) to add to the final offsets (0: none)
};

// Device-resident state of one instance in the batched device CG.
struct CGState {
    double beta_psi, beta_A;
    double c[17];             // line-search coefficients of the current iteration
    double alpha_psi, alpha_A;
    double E, E_prev;         // energy after the last / the previous update
    double g2, g2_0;          // |gradient|^2 now and at the first iteration
    int iter, done, gi, di;   // iterations done, finished, current gradient / direction buffer
    int status;               // 0 ok, 1 gradient-norm stop, 2 energy stop, 3 n_iter, 4 energy target,
                              // 5 energy window (stagnation), -1 no step found
    int pi;                   // buffer (psi[pi], ab[pi]) holding the current state during a CG call
    int ticket;               // CTAs of this instance finished in the running launch
    int it_mark;              // iteration of the last energy-window mark
    double E_mark;            // energy at that mark
};

// Everything a kernel needs to process one instance.  Lives in device memory,
// one entry per instance of a batch (a single GLSolver is a batch of one).
struct Inst {
    Geo g;
    double dt, epsilon, kappa2, rho, H;
    double lang_psi, lang_A;
    double stop_psi, stop_A;
    float fdt, fepsilon, fkappa2, frho, fH, flang_psi, flang_A, pad_f;  // the same, rounded to float
    int lang_psi_on, lang_A_on;  // Langevin coefficient (in the solver's precision) > 1e-32 (td.h:147,451)
    void* psi[kPsiBufs];      // rotating TD buffers, psi[0] holds the state at rest
    void* ab[3];              // rotating TD buffers, ab[0] holds the state at rest
    const void* abei;         // external+irregular vector potential or NULL
    const uint8_t* mt;        // material tiling (cells) or NULL
    const void* eps_sp;       // spatial linear coefficient (nodes) or NULL
    void* U;                  // link factors of the psi loop (Nab complex); during the A loop the
                              // fixed parts of the FP64 link updates (k_A_sweep), Nab reals
    uint8_t* code;            // per-node link-weight bits of the psi loop, N bytes
    void* dinv;               // per-node reciprocal of the psi step's diagonal, N reals (FP32: bits ^ kDead, tdl.cu)
    uint8_t* cbits;           // per-node cell bits (cell_bits) for the batched CG, N bytes (NULL until CG)
    void* vpi;                // irregular vector potential of fixed vortices, Nab, or NULL
    const int32_t* lock;      // phase-lock node list or NULL
    int lock_n, pad_lock;
    InstState* st;
    CGState* cg;              // batched device CG state (set in a batch's descriptors for a CG call)
    void* gpsi[2];            // CG gradient buffers (psi part, A part) and directions
    void* gA[2];
    void* dpsi[2];
    void* dA[2];
    int tile0, ntiles;        // this instance's range in the tile table
    int natiles;              // its A-sweep tiles (ATile)
    int nitems;               // number of warp-strip items of this instance
    int solveA;               // finite kappa
    int cg_exact;             // batched device CG: exact dF/dA on boundary links
    double cg_target;         // batched device CG: stop once E <= cg_target + cg_target_tol |cg_target| (NaN: off)
    double cg_target_tol;
    unsigned long long thr_psi, thr_A;  // largest residual that meets the stop rule, as IEEE bits (res_threshold)
};

// Global state of one batched Jacobi/time loop.
struct LoopState {
    int active;               // instances whose current Jacobi loop is not done
    unsigned blocks_done;     // CTAs finished in the current launch
    int launches;             // sweeps launched in the current Jacobi loop
    int cont;                 // last decision of the Jacobi while loop
    int step, Nt;             // time loop position / length
    int err;                  // error bits (kErr*)
    int ninst;
    long long total_launches;  // sweep kernel launches (psi and A) in the current call
    int guard;                // launches after which a Jacobi loop is stopped with kErrLoopGuard
    unsigned arrived, round;  // cooperative Jacobi loop (end_round): CTAs arrived; 2 x finished rounds + go on
    unsigned spins;           // polls of a barrier between CTAs before one gives up (kErrBarrier)
};

constexpr int kErrLoopGuard = 1;
constexpr int kErrCopyWait = 2;  // a wait for a bulk copy into shared memory ran out (psi sweep)
constexpr int kErrBarrier = 4;   // a wait at a barrier between CTAs ran out (cooperative loops)

// LoopState::spins by default (a poll takes about a microsecond: seconds).
constexpr unsigned kBarrierSpins = 1u << 22;

// Resident time loop (tdr.cu).  An instance's barrier: CTAs arrived so far in the
// call, and the residual maxima and NaN bits of the last three rounds.
constexpr int kResSweeps = 8;    // at most this many sweeps per round
struct ResGroup {
    unsigned arrived, pad;
    unsigned long long res[3][kResSweeps];
    int nan[3], pad2;
};
// One CTA's tile of an instance: origin of its own nodes, the instance's CTAs, where
// the instance's tiles start in the owner table, tiles per row.
struct ResTile {
    int inst, x0, y0, ncta, own0, ntx;
};
// Schedule of a call: CTA c works on tiles[first[c]] .. tiles[first[c + 1] - 1];
// owner: the CTA of every tile of every instance.
struct ResPlan {
    void* fn = nullptr;
    int threads = 0, smem = 0;
    size_t scratch = 0;  // exchange slots of a CTA, bytes
    std::vector<ResTile> tiles;
    std::vector<int> first, owner;
};
// A handle's or batch's schedule and its device copies.
struct ResState {
    int ready = 0;  // 0: not made, 1: made, -1: the domain does not fit on chip
    ResPlan plan;
    ResTile* tiles = nullptr;
    int *first = nullptr, *owner = nullptr;
    ResGroup* groups = nullptr;
    void* scratch = nullptr;
};

// A tile = 256 consecutive nodes of one instance.
struct Tile {
    int inst, n0;
};

// A tile of the FP64 A sweep: kATX x kATY nodes of one instance from node (i0, j0)
// (a CTA of 256 threads covers 256 / kATX rows of the tile per pass).  64 x 32:
// 0.65 ms per sweep at 2049^2 and kappa = 4; 32 x 32, 64 x 16 and 128 x 8 tiles
// 0.70-0.71 ms, 32 x 64 0.65, 128 x 16 0.67.
#ifndef GLGPU_ATX
#define GLGPU_ATX 64
#endif
#ifndef GLGPU_ATY
#define GLGPU_ATY 32
#endif
constexpr int kATX = GLGPU_ATX, kATY = GLGPU_ATY;
static_assert(256 % kATX == 0 && kATY % (256 / kATX) == 0, "A tile: whole rows per pass, whole passes per tile");
struct ATile {
    int inst, i0, j0, pad;
};
inline int atiles_of(int Nx, int Ny) { return ((Nx + kATX - 1) / kATX) * ((Ny + kATY - 1) / kATY); }

// Work item of a warp in a psi sweep: a strip of columns (x0..) by rows (j0..) of one
// instance.  Bulk-copy sweep: kStripCols columns and one of the heights of kStripRowsSet
// (chosen by choose_strip_rows, td.cu), the warp's 32 lanes also covering kFuse halo
// columns on each side.  Loop of tdl.cu: kWideCols columns and `pad` rows.
#ifdef GLGPU_STRIP_ROWS
constexpr int kStripRowsSet[] = {GLGPU_STRIP_ROWS};
#else
constexpr int kStripRowsSet[] = {8, 12, 17};
#endif
constexpr int kNumStripRows = (int)(sizeof(kStripRowsSet) / sizeof(kStripRowsSet[0]));
constexpr int kStripCols = 32 - 2 * kFuse;
inline int strip_items(int Nx, int Ny, int rows) {
    return ((Nx + kStripCols - 1) / kStripCols) * ((Ny + rows - 1) / rows);
}
// The bulk-copy sweep runs kPsiGroup adjacent strips of one row band per CTA (they
// share one ring of rows in shared memory), so the item table lists each band's
// strips in groups of kPsiGroup, the last group of a band padded with empty
// items (inst = -1).  strip_table_len: entries of one instance's table.
constexpr int kPsiGroup = 4;
inline int strip_table_len(int Nx, int Ny, int rows) {
    const int nstrips = (Nx + kStripCols - 1) / kStripCols;
    return (nstrips + kPsiGroup - 1) / kPsiGroup * kPsiGroup * ((Ny + rows - 1) / rows);
}
struct Item {
    int inst, x0, j0, pad;  // inst = -1: an empty item (group padding of the bulk-copy sweep)
};

}  // namespace glgpu

// The opaque handle behind glgpu_handle*: one instance with its buffers.
struct glgpu_handle {
    int dtype;                   // 4 or 8
    glgpu::Geo g;
    glgpu_params p;
    cudaStream_t stream = nullptr;
    int device = 0;
    // device buffers
    void* psi[glgpu::kPsiBufs] = {};
    void* ab[3] = {nullptr, nullptr, nullptr};
    void* abei = nullptr;
    uint8_t* mt = nullptr;
    void* eps_sp = nullptr;
    void* U = nullptr;
    uint8_t* code = nullptr;
    void* dinv = nullptr;
    glgpu::InstState* st = nullptr;
    glgpu::Inst* inst = nullptr;        // device copy of the descriptor
    glgpu::Inst inst_h;                 // host copy of the descriptor
    glgpu::Tile* tiles = nullptr;
    glgpu::ATile* atiles = nullptr;     // A-sweep tiles
    int natiles = 0;
    glgpu::Item* items = nullptr;
    int nitems = 0;
    int strip_rows = 0;                 // strip height of the psi sweep items
    glgpu::Item* litems = nullptr;      // FP32: items of the cooperative psi loop
    int nlitems = 0;
    int loop_rows = 0;                  // their strip height
    glgpu::Item* aitems = nullptr;      // FP32: items of the cooperative A loop
    int naitems = 0;
    int psi_grid = 0;                   // CTAs of the persistent psi sweep
    glgpu::LoopState* loop = nullptr;
    int ntiles = 0;
    // reductions / outputs
    double* partials = nullptr;         // nblocks * 17 doubles
    unsigned* counter = nullptr;        // ticket counter for grid_sum_finish
    double* dscal = nullptr;            // device scalars: [0..16] coefficients, [20] energy, [24..27] beta sums, [28] beta_psi, [29] beta_A
    void* out = nullptr;                // staging buffer for observables (Nab reals, Nc reals)
    void* vort = nullptr;               // vortex candidates
    int* vort_n = nullptr;
    int vort_cap = 0;
    // CG buffers (allocated on first use)
    void* g_psi[2] = {nullptr, nullptr};
    void* g_A[2] = {nullptr, nullptr};
    void* dir_psi[2] = {nullptr, nullptr};
    void* dir_A[2] = {nullptr, nullptr};
    int cg_g = 0, cg_dir = 0;           // current index of g / dir
    void* vpi = nullptr;                // irregular vector potential (fixed vortices), Nab, or NULL (the TD step's copy)
    int32_t* lock = nullptr;            // phase-lock node list (fixed vortices) or NULL
    int lock_n = 0;
    uint8_t* cbits = nullptr;           // batched CG: cell bits per node, written at the start of a call
    // TD graphs, one per (equation mode, kappa finite)
    cudaGraphExec_t td_exec[glgpu::kTDGraphs] = {};
    bool td_graph_failed = false;
    bool use_graphs = true;
    int loop_guard = 0;                 // Jacobi loop guard in sweep launches (0: kLoopGuard)
    int wait_limit = 0;                 // polls of a barrier between CTAs (0: kBarrierSpins)
    int psi_select = 0;                 // psi sweep kernel (bulk_selected)
    int psi_scheme = 0;                 // psi time stepping: 0 backward Euler, 1 Crank-Nicolson, 2 as written
    std::string last_error;
    void* flush = nullptr;              // L2 flush buffer for kernel timing
    // host pinned staging for small results
    double* hscal = nullptr;
    void* pin = nullptr;                // PinStage (pinned host memory)
    glgpu::ResState res;                // resident time loop
};

// A batch: several handles (instances of any sizes and parameters, one dtype,
// one device) advanced together.  Their descriptors, item and tile tables are
// concatenated, so one sweep launch covers every instance and each instance
// keeps its own Jacobi stop rule.
// Pinned host staging of a handle's calls (descriptor up, loop state and statistics down).
struct PinStage {
    glgpu::Inst inst;
    glgpu::InstState st;
    glgpu::LoopState loop;
};

struct glgpu_batch {
    int dtype = 4, device = 0, ninst = 0;
    std::vector<glgpu_handle*> hs;
    cudaStream_t stream = nullptr;
    glgpu::Inst* insts = nullptr;
    glgpu::Tile* tiles = nullptr;
    glgpu::ATile* atiles = nullptr;     // A-sweep tiles
    int natiles = 0;
    glgpu::LoopState* loop = nullptr;
    std::vector<glgpu::InstState> gather_h;
    glgpu::InstState* gather_pin = nullptr;  // pinned host copies of the per-call transfers
    glgpu::LoopState* loop_pin = nullptr;
    glgpu::Inst* insts_pin = nullptr;
    int ntiles = 0;
    glgpu::Item* litems = nullptr;       // FP32: items of the cooperative psi loop
    int nlitems = 0;
    glgpu::Item* aitems = nullptr;      // FP32: items of the cooperative A loop
    int naitems = 0;
    cudaGraphExec_t td_exec[glgpu::kTDGraphs] = {};
    bool td_graph_failed = false, use_graphs = true;
    int loop_guard = 0;                  // Jacobi loop guard in sweep launches (0: kLoopGuard)
    int wait_limit = 0;                  // polls of a barrier between CTAs (0: kBarrierSpins)
    // batched device CG (allocated on first use)
    void* cg_tiles = nullptr;            // CG tile table (larger tiles than the TD one)
    int cg_ntiles = 0;
    double* cg_partials = nullptr;       // cg_ntiles * 17 doubles
    void* cg_loop = nullptr;             // CGLoop
    glgpu::CGState* cg_states = nullptr; // one per instance
    std::vector<glgpu::CGState> cg_states_h;
    cudaGraphExec_t cg_exec = nullptr;
    bool cg_graph_failed = false;
    std::vector<double> cg_targets;      // per-instance energy targets (empty: none)
    double cg_target_tol = 0.0;
    int cg_window = 0;                   // energy-window stop: iterations (0: off) and relative decrease
    double cg_window_tol = 0.0;
    glgpu::ResState res;                 // resident time loop
    std::string last_error;
};

namespace glgpu {

int batch_error(glgpu_batch* b, int code, const std::string& msg);
int batch_td(glgpu_batch* b, double dt, int Nt, int eqn, glgpu_td_stats* stats, double* elapsed_ms);
int set_error(glgpu_handle* h, int code, const std::string& msg);
int cuda_check(glgpu_handle* h, cudaError_t e, const char* what);
void upload_inst(glgpu_handle* h);
size_t real_size(const glgpu_handle* h);

// td.cu
int td_run(glgpu_handle* h, double dt, int Nt, int eqn, glgpu_td_stats* stats, double* elapsed_ms);
int time_sweeps(glgpu_handle* h, int which, int nrep, double* avg_ms);
bool td_resident(glgpu_handle* h);  // its TD calls run as one resident launch (unless the bulk-copy sweep is selected)
int choose_strip_rows(const Geo& g);
// the FP32 bulk-copy psi sweep is selected (glgpu_set_psi_sweep_kernel)
inline bool bulk_selected(const glgpu_handle* h) { return h->dtype == 4 && h->psi_select == 1; }
int bulk_sweep_grid(int rows, int nitems);
std::vector<Item> make_items(const Geo& g, int inst, int rows);
// tdl.cu: the cooperative psi loop's kernel, its CTA size, its CTAs over n tiles (FP64) or items (FP32)
const void* psi_loop_fn(int dtype);
int psi_loop_threads(int dtype);
int psi_loop_grid(int dtype, int n);
constexpr int kWideCols = 56, kACols = 60;  // output columns of an FP32 item of the psi loop, of the A loop
int choose_loop_rows(const Geo* const* geos, int n);
int choose_A_rows(const Geo* const* geos, int n);
double loops_step_us(const Geo* const* geos, int n, bool any_A);
void add_loop_items(std::vector<Item>& items, const Geo& g, int inst, int rows, int cols);
const void* A_loop_fn();  // the cooperative A loop (FP32), its CTAs over n items
int A_loop_grid(int n);
// tdr.cu
bool res_prepare(ResState* r, glgpu_handle* const* hs, int n);
void res_free(ResState* r);
cudaError_t res_launch(const ResState& r, const Inst* insts, int ninst, LoopState* loop, int Nt, int eqn, cudaStream_t s);
unsigned long long res_threshold(int dtype, double stop);
// obs.cu
int obs_free_energy(glgpu_handle* h, double* out);
int obs_magnetic_field(glgpu_handle* h, void* host_out);
int obs_current_density(glgpu_handle* h, void* host_out);
int obs_supercurrent_density(glgpu_handle* h, void* host_out);
int obs_vortex_candidates(glgpu_handle* h, int cap, int* n_out, int32_t* cells, void* corners);
int reduce_sum(glgpu_handle* h, const double* x, long long n, int nv, double* out);
int free_energy_noalloc(const glgpu_grid* grid, const glgpu_params* p, const void* psi, const void* ab,
                        const void* abei, const uint8_t* mt, double* energy, cudaStream_t stream);
// cg.cu
int cg_ensure(glgpu_handle* h);
int cg_reset_direction(glgpu_handle* h);
int cg_gradient(glgpu_handle* h, int compute_beta);
int cg_coefficients(glgpu_handle* h, double* c_out);
int cg_update(glgpu_handle* h, double alpha_psi, double alpha_A, double* energy_out);
int cg_read_gradient(glgpu_handle* h, void* gpsi_host, void* gA_host);
int cg_coef_for(glgpu_handle* h, const void* dpsi_host, const void* dab_host, double* c_out);
// cgb.cu
int batch_set_energy_targets(glgpu_batch* b, const double* targets, double rel_tol);
int batch_set_cg_window(glgpu_batch* b, int window, double rel_tol);
int batch_cg(glgpu_batch* b, int n_iter, double rtol, double gtol, int flags, int32_t* iters, double* energies, double* grad_rel,
             int32_t* status, double* elapsed_ms);
// td.cu graph helpers
cudaError_t add_kernel(cudaGraph_t g, cudaGraphNode_t* node, const cudaGraphNode_t* deps, int ndeps, void* fn, dim3 grid,
                       dim3 block, void** args, unsigned smem_bytes = 0);
cudaError_t add_while(cudaGraph_t g, cudaGraphNode_t* node, const cudaGraphNode_t* deps, int ndeps,
                      cudaGraphConditionalHandle h, cudaGraph_t* body);

inline int blocks_for(long long n) { return (int)((n + kThreads - 1) / kThreads); }

}  // namespace glgpu
