// wf_resident.cuh - Jacobi loops that keep the whole grid on chip
// (wf_resident.cu): plan, workspace and launchers.
#pragma once
#include <cuda_runtime.h>

#include "wf_common.cuh"

namespace wf {

// Split of a grid into px x py x pz boxes of bx x by x bz cells, one box per
// block and at most one block per multiprocessor.  bz is the number of cells
// a thread owns (a z column); bz == 0: the grid does not fit on chip.
struct ResPlan {
    int bx = 0, by = 0, bz = 0, px = 0, py = 0, pz = 0;
    bool pair = false;   // pressure loop that runs two sweeps a halo trip
    int least = 2;       // sweeps from which on the loop beats the passes
    int boxes() const { return px * py * pz; }
};

// Device workspace of the loops of one stream: the halo packets of both
// parities, the epoch words and streamed coefficients.  One loop at a time may use it.
// Limit of one wait, in polling rounds: a round is one trip to L2 (0.2 to
// 0.5 us), so a wait ends after one to two seconds.
constexpr int kWaitRounds = 1 << 22;
struct ResWork {
    void* pk = nullptr;    // the allocation; 64-bit packets of the pressure loops
    void* pk3 = nullptr;   // 128-bit packets of the momentum loop
    unsigned* ctl = nullptr;
    float* stream = nullptr;  // coefficients the momentum loop reads in every sweep
    int rounds = kWaitRounds;
    int silent = -1;          // block that sends nothing (the self-test of the waits)
};

// The plans of one handle's loops and their workspace.
struct Resident {
    ResPlan pres;      // uniform pressure loops
    ResPlan nupres;    // non-uniform pressure loop
    ResPlan pres2, nupres2;  // the same, two sweeps a halo trip, where that is faster
    ResPlan vel;       // momentum loop
    ResPlan pres_shared, vel_shared;  // the same beside the cases of a batch: fewest multiprocessors
    ResPlan pres_beside, nupres_beside, vel_beside;  // beside a few other handles' loops
    ResWork work;
    const ResPlan& pres_alone() const { return pres2.bz > 0 ? pres2 : pres; }
    const ResPlan& nupres_alone() const { return nupres2.bz > 0 ? nupres2 : nupres; }
    bool ok(const ResPlan& p) const { return p.bz > 0 && work.pk != nullptr; }
};

// Plans for the grid of P on a device of `sms` multiprocessors.
void resident_plan(const Params& P, int sms, Resident* r);
// Attributes of the plans' kernels; call on the device before the first
// launch.
int resident_setup(const Resident& r);
// Allocates / frees the workspace the plans need (stream-ordered zeroing on
// st).  Without memory the plans stay unused: the loops run as passes.
void resident_alloc(Resident* r, cudaStream_t st);
void resident_free(Resident* r);

// n >= 2 sweeps p = ainv (rhs - C p) of the uniform grid's pressure
// equations in one cooperative launch, from pin (nullptr: zero), with the
// iterates of k_pres_msweep / k_pres_tma4 bit for bit.  pout receives iterate
// n on fluid cells, pprev (nullable) iterate n - 1; stack (nullable) every
// iterate k = 1..n of every cell at stack + k N.  rhs nullptr: 0.  ordered
// (without a stack): the iterates of the one-sweep kernel launch_pres_sweep
// instead.  A bounded wait that runs out sets *status to 1.
cudaError_t launch_res_pres(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w, const float* c3,
                            const float* ainv, const float* rhs, const float* pin, float* pout, float* pprev,
                            float* stack, int n, int* status, bool ordered = false);
// The same for the non-uniform grid: six face coefficients and 1/Dp
// (coef, kNuCoefPlanes planes), right-hand side bp; the iterates of
// k_nu_pres_sweep bit for bit.
cudaError_t launch_res_nupres(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w,
                              const float* coef, const float* bp, const float* pin, float* pout, float* pprev, int n,
                              int* status);
// n >= 2 momentum sweeps u = (1/D) (sum_f A_f u_f + b) from uin in one
// launch: A holds A_E..A_D, iD the three components of 1/D.  The iterates of
// k_vel_sweep4 bit for bit; uout (uprev, nullable) receives iterate n (n - 1)
// on fluid cells and may not alias uin.  stack (nullable; uout may then be
// nullptr): every iterate k = 1..n of every cell at stack + k step, non-fluid cells
// with uin's value.  bv nullptr: 0.
cudaError_t launch_res_vel(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w, const float* A,
                           const float* iD, const float* bv, const float* uin, float* uout, float* uprev, int n,
                           int* status, float* stack = nullptr, long long step = 0);

}  // namespace wf
