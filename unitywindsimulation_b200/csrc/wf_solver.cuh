// wf_solver.cuh - the solver handle behind the C ABI (private).
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <string>
#include <tuple>

#include "wf_common.cuh"
#include "wf_resident.cuh"

namespace wf {
struct LoopRecorder;
}

struct wf_solver {
    wf_config cfg{};
    wf::Params P{};
    wf::Bnd B{};
    int device = 0;
    cudaStream_t st = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;

    // ---- device fields (see wf_common.cuh for the layout) ----
    uint8_t* fl = nullptr;
    uint8_t* nbm = nullptr;   // neighbour masks (Params::nbm)
    // Three velocity buffers rotated by role like the reference's
    // velField / velFieldLastTime / velFieldLastIter textures.  When
    // iter_alias is set, velFieldLastIter is logically equal to
    // velFieldLastTime and buffer vb[iI] holds no meaningful fluid values
    // (this replaces the end-of-step copy, FvmSolverGpu.cs:1106).
    // A fourth, spare buffer lets the multi-sweep kernels write iterates n
    // and n-1 while velFieldLastTime and the pass input stay intact.  Solid
    // cells hold the same values in all four (no kernel writes them).
    float* vb[4] = {nullptr, nullptr, nullptr, nullptr};
    int iT = 0, iF = 1, iI = 2;
    bool iter_alias = false;
    float *uc = nullptr, *Dv = nullptr, *bv = nullptr, *aodu = nullptr, *face = nullptr;
    float* pr = nullptr;
    // presCorrectField / presCorrectFieldLastIter.  When pc_zero is set both
    // are logically all-zero (replaces SetPresCorrectFieldtoZero,
    // FvmSolverGpu.cs:1545-1554; the first sweep then reads no input).
    // Three physical buffers: the multi-sweep kernels need a third one to
    // materialise iterate n-1 next to iterate n.
    float* pcb[3] = {nullptr, nullptr, nullptr};
    int iPC = 0, iPCL = 1;
    bool pc_zero = true;
    float *Dp = nullptr, *bp = nullptr, *eddy = nullptr;
    float* drag = nullptr;    // Brinkman drag per cell (allocated when first set)
    // non-uniform collocated grid (wf_nonuniform.cu): face positions
    // fx[nx+1], fy[ny+1], fz[nz+1] back to back, and the face-flux texture
    // (three planes of (nx+1)(ny+1)(nz+1)); nonuniform selects its kernels
    float* fpos = nullptr;
    float* flux = nullptr;
    float* nucoef = nullptr;  // the pressure sweeps' per-step coefficient planes (wf::kNuCoefPlanes)
    bool nonuniform = false;
    float* bnd[6] = {};
    // sweep coefficient caches of the fast path (wf_sweeps.cu)
    float* pcoef = nullptr;   // pressure: c_E, c_N, c_U, 1/Dp, PISO rhs (5 planes)
    float* vcoef = nullptr;   // momentum: A_E..A_D, 1/D (9 planes)
    float* grad = nullptr;    // cell-centre velocity gradient tensors (9 planes)
    // generation of DField (bumped by every write) and the generation the
    // cached pressure face coefficients c_E, c_N, c_U were built from: the
    // three pressure solves of a step share D, so they share the coefficients
    long long d_gen = 1, c3_gen = 0;
    long long id_gen = 0;     // generation of D the cached 1/D (vcoef + 6N) belongs to
    // the momentum pre-compute of the step in progress wrote vcoef (A and
    // 1/D) for the current D; the step's sweeps take them as they are
    bool vcoef_step = false;
    bool ainv_step = false;   // the same for 1/Dp (pcoef + 3N) and the pressure pre-compute
    // scratch
    double* part = nullptr;
    double* dsum = nullptr;   // 4 doubles
    float* dref = nullptr;
    int* dbad = nullptr;
    void* stage = nullptr;    // 4N floats of device staging for host I/O
    // inflow-plane upload: page-locked staging (3 * ny * nz floats) and the
    // event after which the staging may be rewritten
    float* in_stage = nullptr;
    cudaEvent_t ev_in = nullptr;
    // asynchronous readback: snapshot (4N + N floats), copy stream, events
    float* snap = nullptr;
    cudaStream_t cst = nullptr;
    cudaEvent_t ev_snap = nullptr, ev_done = nullptr;
    bool rb_pending = false;
    double* hsum = nullptr;   // pinned

    float wind = 0.f;
    int64_t step = 0;
    float res_vel = -1.f, res_pres = -1.f;
    float last_ms = 0.f;
    int fast = 1;             // use the fast Jacobi kernels (wf_sweeps.cu)
    int pres_k = 4;           // pressure sweeps per multi-sweep pass (1..4)
    int vel_k = 1;            // momentum sweeps per multi-sweep pass (1..2)
    int pres_ty = 32;         // tile rows of the pressure multi-sweep kernel (32 or 16)
    int pres_tma = 1;         // four-sweep passes with TMA-staged tiles where they apply
                              // (WF_TMA=0: the per-thread-staged kernel; same iterates)
    // sticky status of the bounded waits in the TMA-staged kernels and the loops on chip: page-locked
    // host word (hstat) and its device alias (dstat); nonzero = a wait ran out
    int* hstat = nullptr;
    int* dstat = nullptr;
    // loops that keep the whole grid on chip (wf_resident.cu) where it fits;
    // 0: the pass kernels (wf_set_loops, an explicit depth or tile, WF_RESIDENT=0)
    int resident = 1;
    wf::Resident res;
    // what the step being enqueued runs beside: nothing, other handles' steps on their
    // own streams, or the other cases of a batch
    enum Company { kAlone, kBeside, kBatch };
    Company company = kAlone;
    // steps enqueued and not waited for yet; how many other handles of the device had
    // such steps when they were enqueued, and up to when they were waited for
    // (steps_begin, steps_end)
    bool pending = false;
    int beside_begin = 0, beside_seen = 0;
    long long begin_ticket = 0;
    bool rb_stepped = false;  // a step was enqueued after the readback in flight
    int vel_blk[3] = {32, 4, 2};  // block of the four-cell momentum sweep (256 threads)
    int num_sms = 148;        // multiprocessors of the device
    int pdl = 1;              // programmatic dependent launch in the non-uniform grid's sweep chains
                              // (WF_PDL=0: plain stream order)
    int vec4 = 1;             // 4-cell vector momentum sweep when nx % 4 == 0 and the
                              // planes are 16-byte aligned (WF_VEC4=0: one cell per thread)
    bool in_step = false;     // inside wf_step: skip iterates no later kernel reads
    wf::LoopRecorder* rec = nullptr;  // set while a batch records the step in segments
    long long launches = 0;   // kernels launched by wf_step
    std::string err;

    // CUDA-graph cache of one step, keyed by the buffer roles before the step.
    using RoleKey = std::tuple<int, int, int, int, int>;
    struct GraphEntry {
        cudaGraph_t graph = nullptr;  // kept for composition into batch graphs
        cudaGraphExec_t exec = nullptr;
        RoleKey after{};
        long long kernels = 0;
    };
    std::map<RoleKey, GraphEntry> graphs;
    std::map<RoleKey, GraphEntry> batch_graphs;   // the same for steps in a batch (exec unused)
    std::map<RoleKey, GraphEntry> beside_graphs;  // and for steps beside other handles' steps
    std::map<RoleKey, GraphEntry>& step_graphs() {
        return company == kBatch ? batch_graphs : company == kBeside ? beside_graphs : graphs;
    }
};

namespace wf {
// Whether a loop of n sweeps runs on chip.
inline bool loops_on_chip(const wf_solver* h, const ResPlan& p, int n) {
    return h->resident && h->dstat && h->res.ok(p) && n >= p.least;
}
// Handles whose steps run at the same time (step_async on their own streams, one
// thread a handle, any mix): a loop on all multiprocessors waits until the other handles'
// loops have left, so beside others a handle takes splits that leave at least half of
// the multiprocessors to them, where there are such.  A handle knows its company by a
// count per device of the handles with steps in flight: those it sees when it enqueues,
// or those that its last steps ran beside (the first handle of a round sees none when it
// enqueues).  The fields do not depend on it.  Ms for one step of each of 2 / 4 / 16
// handles, passes, lone splits, now: 24 x 12 x 16 0.56 / 0.57 / 0.64, 0.29 / 0.57 / 2.22, 0.18 /
// 0.19 / 0.27; 64 x 32 x 48 0.61 / 0.76 / 2.80, 0.33 / 0.68 / 2.80, 0.33 / 0.48 / 1.42; 72 x 40 x 72
// 0.75 / 1.17 / 5.3, 0.47 / 0.97 / 4.0, 0.45 / 0.67 / 2.7; stretched 24 x 12 x 16 0.21 / 0.22 / 0.40,
// 0.23 / 0.46 / 1.82, 0.13 / 0.14 / 0.21, 64 x 32 x 48 0.27 / 0.38 / 1.61, 0.27 / 0.56 / 2.29, 0.27 / 0.33 /
// 1.24.  Larger grids keep the lone splits: 100 x 50 x 100 1.39 / 3.6 / - in passes, 0.85 / 1.81
// / -.
void steps_begin(wf_solver* h);
void steps_end(wf_solver* h);  // nothing of the handle's stream is in flight any more
bool beside_others(const wf_solver* h);
// Counts a handle of the device in or out; whether there are others that it may yet
// step beside (wf_prepare_graphs then captures both forms of its step).
void count_handle(const wf_solver* h, int by);
bool has_beside_splits(const wf_solver* h);
bool may_run_beside(const wf_solver* h);
inline bool shares(const wf_solver* h, const ResPlan& p) { return p.bz > 0 && 2 * p.boxes() <= h->num_sms; }

// The same between two residual checks, whose passes are eager launches of one sweep on
// either mesh: from the uniform loop's count on (100 x 50 x 100, 3 sweeps: -11 us of 150).
inline int least_between_checks(const wf_solver* h) { return h->res.pres_alone().least; }

// The loops' splits: the fastest alone; beside the other cases of a batch the
// one that holds the fewest multiprocessors for its time, where it leaves at
// least half of them to the others.  A larger case keeps its pressure split for
// a lone case and its momentum passes.  Us a batched step: 16 cases of 0.06-0.21 M
// cells 3370 in passes, 3770 with lone splits (one loop after another), 2061
// with shared ones (1920 now); 16 cases of 0.7-1.75 M cells 20600 in passes, 19600
// with this rule (18500 now), 28800 with shared splits whatever their size and 27900
// with lone momentum splits too (loops of more than half the GPU each wait for it
// to empty).
inline const ResPlan& pres_plan(const wf_solver* h) {
    if (h->company == wf_solver::kAlone) return h->res.pres_alone();
    if (h->company == wf_solver::kBeside) return h->res.pres_beside;
    return shares(h, h->res.pres_shared) ? h->res.pres_shared : h->res.pres;
}
inline const ResPlan& nupres_plan(const wf_solver* h) {
    return h->company == wf_solver::kBeside ? h->res.nupres_beside : h->res.nupres_alone();
}
inline const ResPlan& vel_plan(const wf_solver* h) {
    static const ResPlan none;
    if (h->company == wf_solver::kAlone) return h->res.vel;
    if (h->company == wf_solver::kBeside) return h->res.vel_beside;
    return shares(h, h->res.vel_shared) ? h->res.vel_shared : none;
}

// Step-graph plumbing shared by the single-handle and the batched step.
bool step_graphable(const wf_solver* h);
// Captures (once per buffer-role assignment and company) the graph of one step from
// the handle's current state without running it.
int ensure_step_graph(wf_solver* h, const wf_solver::GraphEntry** out);
// Applies the role rotation and counters of one replayed step.
void commit_graph_step(wf_solver* h, const wf_solver::GraphEntry& e);
// One step launched kernel by kernel on the handle's stream.
int run_step_eager(wf_solver* h);
// Captures one step from the handle's current state as segments around its
// Jacobi loops (rec), without running it; *after receives the roles after
// the step and *kernels the kernels in the segments.
int capture_step_segments(wf_solver* h, LoopRecorder* rec, wf_solver::RoleKey* after, long long* kernels);
void drop_graphs(wf_solver* h);
}  // namespace wf
