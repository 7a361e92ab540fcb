// wf_resident.cu - Jacobi loops that keep the whole grid on chip.
//
// A grid of up to about a million cells fits the register files and shared
// memories of the GPU's multiprocessors together.  One cooperative launch
// then runs a whole loop: every block owns a box of cells, reads its
// coefficients from memory once, holds them in registers for all sweeps, and
// keeps the iterate in a double-buffered shared box with a one-cell halo.  A
// sweep touches memory only for the cells on the faces between boxes.
//
// Halo exchange.  A face cell travels as one 64-bit packet {value, epoch}
// written with a relaxed 64-bit store and polled by the thread of the
// neighbour box that needs it.  A 64-bit access is single-copy atomic, so a
// packet with the sweep's epoch carries the sweep's value: no fence, no flag,
// one trip through L2 per sweep.  Packets alternate between two buffers: a
// block may write sweep k + 2's packets only after it has received its
// neighbours' packets of sweep k + 1, which they send after reading sweep
// k's, so a slot is never overwritten before it is read.  Epochs continue
// from launch to launch: every block reads the base when it starts, and the
// last block to finish (an atomic ticket) advances it.
//
// What bounds it: the trip of the packets (470 cycles within a die, 900 across,
// measured SM to SM) and the instructions of a column, one warp after another;
// not memory.  Measured, us a pressure sweep: 0.75 on 64 x 32 x 48 and 0.80 on 80 x
// 40 x 40 (two sweeps a trip, k_res_pair; 1.10 and 1.16 with one), 1.69 on 100 x 50 x
// 100, 2.3 on 128 x 64 x 96, 3.6 on 149 x 61 x 103; a momentum sweep: 1.35, 1.44,
// 2.9, 4.7 and 6.7.  With one launch for every one to four sweeps: 4.7, 4.7, 5.2, 5.2,
// 6.3 and 2.1, 3.0, 5.6, 6.1, 11.6.
//
// The launch is cooperative, so all blocks are resident and every packet
// that is waited for will be sent.  The waits are bounded all the same
// (kWaitRounds): a wait that runs out sets *status and the block returns, its
// neighbours' waits then run out as well.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <iterator>

#include "wf_kernels.cuh"
#include "wf_resident.cuh"

namespace wf {
namespace {

constexpr int NT = 512;                               // threads of a block, one z column each
constexpr int kMaxBoxes = 256;
constexpr size_t kSmemMax = 232448 - 1024;

__device__ __forceinline__ void put(unsigned long long* p, float v, unsigned ep) {
    const unsigned long long w = ((unsigned long long)ep << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w));
}
__device__ __forceinline__ unsigned long long get(const unsigned long long* p) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p));
    return w;
}

// Three components and the epoch in one 128-bit packet (a scalar 128-bit
// access is single-copy atomic as well).
struct Packet3 {
    unsigned long long lo, hi;   // x, y | z, epoch
};
__device__ __forceinline__ void put3(Packet3* p, float x, float y, float z, unsigned ep) {
    const unsigned long long lo = ((unsigned long long)__float_as_uint(y) << 32) | __float_as_uint(x);
    const unsigned long long hi = ((unsigned long long)ep << 32) | __float_as_uint(z);
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                 "l"(lo), "l"(hi));
}
__device__ __forceinline__ Packet3 get3(const Packet3* p) {
    Packet3 w;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(w.lo), "=l"(w.hi)
                 : "l"(p));
    return w;
}

// One block's box and its threads.  The columns on the box's x and y edges
// (the rim) come first, in whole warps of their own, then the inner columns
// row by row: the rim warps compute and send their cells and then only wait
// for the halo, while the other warps still compute.
// Shared layout: R planes of (by + 2) rows with the x / y halo in place and a
// row pitch of bx + 30 words.  The pitch equals the length of a row of inner
// columns modulo the 32 banks, so a warp's 32 columns, whatever rows they lie
// in, read and write 32 different banks.  The z halo belongs to the column's
// own thread and stays in registers.
// The plane size is a compile-time constant, so every shared access of a
// column is an immediate offset from one of three addresses.
// Packets of a box and parity: r * rim + thread for the rim cells of plane r,
// then the top and the bottom plane in thread order.
struct Box {
    int id, x0, y0, z0;
    int rim;              // rim columns
    int inner0;           // first thread of the inner columns
    int sx;               // shared row pitch
    int slots;            // packets of one box and parity
};
constexpr int kPad = 30;
// Words of a shared plane for R cells a thread: what two boxes of R planes
// (and, above kRegR, 1/Dp and the right-hand side) leave room for.
constexpr int kRegR = 8;
__host__ __device__ constexpr int plane_of(int R) {
    return R <= 8 ? 1536 : R <= 10 ? 1472 : R <= 12 ? 1408 : R <= 14 ? 1344 : 1248;
}
__host__ __device__ constexpr int rim_of(const ResPlan& p) { return 2 * (p.bx + p.by) - 4; }
__host__ __device__ constexpr int inner0_of(const ResPlan& p) { return (rim_of(p) + 4 + 31) / 32 * 32; }
__host__ __device__ constexpr int inner_of(const ResPlan& p) { return (p.bx - 2) * (p.by - 2); }
// Halo cells the busiest thread fetches: the rim + 4 halo cells of a plane go
// to as many threads, NT / (rim + 4) planes at a time.
__host__ __device__ constexpr int fetches_of(const ResPlan& p) {
    const int G = NT / (rim_of(p) + 4);
    return (p.bz + G - 1) / G;
}
__host__ __device__ constexpr int slots_of(const ResPlan& p) {
    return p.bz * rim_of(p) + 2 * (inner0_of(p) + inner_of(p));
}
__device__ __forceinline__ Box make_box(const ResPlan& pl) {
    Box b;
    b.id = blockIdx.x;
    const int ix = b.id % pl.px, iy = (b.id / pl.px) % pl.py, iz = b.id / (pl.px * pl.py);
    b.x0 = ix * pl.bx;
    b.y0 = iy * pl.by;
    b.z0 = iz * pl.bz;
    b.rim = rim_of(pl);
    b.inner0 = inner0_of(pl);
    b.sx = pl.bx + kPad;
    b.slots = slots_of(pl);
    return b;
}
// The column of a thread; false: the thread owns none.
__device__ __forceinline__ bool column_of(const Box& b, const ResPlan& pl, int tid, int& lx, int& ly) {
    lx = ly = 0;
    if (tid >= b.inner0) {
        const int q = tid - b.inner0, w = pl.bx - 2;
        if (q >= inner_of(pl)) return false;
        lx = 1 + q % w;
        ly = 1 + q / w;
        return true;
    }
    if (tid < 2 * pl.by) {
        lx = tid < pl.by ? pl.bx - 1 : 0;
        ly = tid < pl.by ? tid : tid - pl.by;
        return true;
    }
    const int q = tid - 2 * pl.by, w = pl.bx - 2;
    if (q >= 2 * w) return false;
    lx = 1 + (q < w ? q : q - w);
    ly = q < w ? pl.by - 1 : 0;
    return true;
}

// One thread's packets (offsets of plane 0 where a plane is meant; -1: none).
struct Links {
    int se;       // its cell on the rim
    int su, sd;   // its top and bottom cell
    int ru, rd;   // the cells above and below its column
    // the halo cells it fetches, of planes g, g + G, ...: packet and shared
    // offset of the first (re -1: outside the domain), their steps, how many
    int re, he, rstep, hstep, rn;
};
// Halo cells a thread fetches at most in the momentum loop of R cells a thread.
__host__ __device__ constexpr int fetch_max(int R) { return R <= 4 ? 1 : 2; }
// Halo cell e of the E, W, N, S side: its box coordinates, the box that owns it
// (-1: outside the domain) and its place t on that box's rim.
__device__ __forceinline__ int halo_cell(const Box& b, const ResPlan& pl, int e, int& t, int& hx, int& hy) {
    const int bx = pl.bx, by = pl.by, ix = b.id % pl.px, iy = (b.id / pl.px) % pl.py;
    if (e < by) {
        hx = bx; hy = e;
        t = by + e;
        return ix + 1 < pl.px ? b.id + 1 : -1;
    }
    if (e < 2 * by) {
        hx = -1; hy = e - by;
        t = hy;
        return ix > 0 ? b.id - 1 : -1;
    }
    if (e < 2 * by + bx) {
        hx = e - 2 * by; hy = by;
        t = hx == bx - 1 ? 0 : hx == 0 ? by : 2 * by + bx - 2 + hx - 1;
        return iy + 1 < pl.py ? b.id + pl.px : -1;
    }
    hx = e - 2 * by - bx; hy = -1;
    t = hx == bx - 1 ? by - 1 : hx == 0 ? 2 * by - 1 : 2 * by + hx - 1;
    return iy > 0 ? b.id - pl.px : -1;
}
// `groups`: planes whose halo cells are fetched by different threads.
__device__ __forceinline__ Links make_links(const Box& b, const ResPlan& pl, bool own, int groups) {
    Links l;
    const int tid = threadIdx.x, mine = b.id * b.slots;
    const int iz = b.id / (pl.px * pl.py);
    l.se = l.su = l.sd = l.ru = l.rd = l.re = -1;
    l.he = 0;
    const int G = groups, g = tid / (b.rim + 4), e = tid % (b.rim + 4);
    l.rstep = G * b.rim;
    l.hstep = G * plane_of(pl.bz);
    l.rn = g < G && g < pl.bz ? (pl.bz - 1 - g) / G + 1 : 0;
    const int top = pl.bz * b.rim, layer = pl.px * pl.py, half = b.inner0 + inner_of(pl);
    if (own) {
        if (tid < b.rim && layer > 1) l.se = mine + tid;
        if (iz + 1 < pl.pz) {
            l.su = mine + top + tid;
            l.ru = (b.id + layer) * b.slots + top + half + tid;
        }
        if (iz > 0) {
            l.sd = mine + top + half + tid;
            l.rd = (b.id - layer) * b.slots + top + tid;
        }
    }
    int t, hx, hy;
    const int from = halo_cell(b, pl, e, t, hx, hy);
    l.he = (hy + 1) * b.sx + hx + 1 + g * plane_of(pl.bz);
    if (from >= 0 && l.rn > 0) l.re = from * b.slots + t + g * b.rim;
    return l;
}

// Receives the halo of the iterate with epoch ep: the cells above and below
// the column into hu, hd and, in a rim warp (RIM), the thread's x / y halo
// cell of R planes into the shared box at v.  The whole warp polls until all
// its packets are there: one vote a round and loads without a condition of
// their own (a lane that waits for nothing reads a packet it ignores), so
// the loads leave back to back and the warp never diverges.  With a branch
// per packet and a clock in the loop an empty receive alone took 300 cycles.
// False where the rounds ran out.
template <int R, bool RIM>
__device__ __forceinline__ bool receive(const Links& l, int rim, float* v, const unsigned long long* pk, unsigned ep,
                                        int rounds, float& hu, float& hd) {
    const bool nu = l.ru >= 0, nd = l.rd >= 0, ne = RIM && l.re >= 0;
    const unsigned long long *pu = pk + (nu ? l.ru : 0), *pd = pk + (nd ? l.rd : 0), *pe = pk + (ne ? l.re : 0);
    constexpr int U = !RIM ? 0 : R <= 8 ? R : (R + 1) / 2;
#pragma unroll
    for (int r0 = 0; r0 < (RIM ? R : 1); r0 += RIM ? U : 1) {
        unsigned long long w[U + 1], wu = 0, wd = 0;
        int left = rounds;
        bool ok;
        do {
            if (r0 == 0) {
                wu = get(pu);
                wd = get(pd);
            }
#pragma unroll
            for (int q = 0; q < U; ++q) w[q] = get(pe + (r0 + q < R ? r0 + q : R - 1) * rim);
            ok = r0 != 0 || ((!nu || (unsigned)(wu >> 32) == ep) && (!nd || (unsigned)(wd >> 32) == ep));
            bool oke = true;
#pragma unroll
            for (int q = 0; q < U; ++q) oke = oke && (unsigned)(w[q] >> 32) == ep;
            ok = ok && (oke || !ne);
        } while (!__all_sync(0xffffffffu, ok) && --left);
        if (left == 0) return false;
        if (r0 == 0) {
            hu = nu ? __uint_as_float((unsigned)wu) : 0.f;
            hd = nd ? __uint_as_float((unsigned)wd) : 0.f;
        }
        if (ne) {
#pragma unroll
            for (int q = 0; q < U; ++q)
                if (r0 + q < R) v[l.he + (r0 + q) * plane_of(R)] = __uint_as_float((unsigned)w[q]);
        }
    }
    return true;
}

// Epoch base of this launch; the last block to leave advances it by `used`.
__device__ __forceinline__ unsigned epoch_begin(const unsigned* ctl) { return *(const volatile unsigned*)ctl; }
__device__ __forceinline__ void epoch_end(unsigned* ctl, unsigned base, unsigned used) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(ctl + 1, 1u) == gridDim.x - 1) {
            ctl[1] = 0;
            __threadfence();
            atomicExch(ctl, base + used);
        }
    }
}

// kPasses: the uniform grid with the rounding of the four-sweep passes (their
// compiled sum fuses the first product, not the second, into the add);
// kOrdered: with that of the one-sweep reference-form kernel; kStretched: six
// coefficients a cell, rounded as kOrdered.
enum class Form { kPasses, kOrdered, kStretched };

struct PresArgs {
    int nx, ny, nz, n;
    ResPlan pl;
    const float *c, *ainv, *rhs;   // c: c_E, c_N, c_U planes, or the six face planes
    const uint8_t* nbm;            // neighbour masks; bit 6: fluid
    const float* pin;
    float *pout, *pprev, *stack;
    unsigned long long* pk;
    size_t half;                   // packets of one parity
    unsigned* ctl;
    int* status;
    int rounds, silent;            // limit of a wait; block that sends nothing
};

// The loops read every neighbour, fluid or not, through a coefficient that is 0 on
// faces of non-fluid cells.  0 times an infinity or a NaN is NaN, and a fluid cell
// without fluid neighbours has 1/Dp = inf and the value NaN; so a cell whose 1/D is 0
// (not fluid, or beyond the domain) is 0 by selection, not by the product, and no NaN
// crosses a wall (the kernels of one sweep a launch skip non-fluid neighbours by the
// mask).  Up to kRegR cells a thread the column's cells to clear are bits of a word, and
// a warp without any skips them all (100 x 50 x 100, 400 sweeps: step 920 us, 942 with a
// select at every cell); above, the word costs spills (128 x 64 x 96 with its copies:
// 1092 us against 984) and every cell selects.  The pair kernel does not store such a
// cell and drops its packet: it stays 0.
template <int First, int Last, int M>
__device__ __forceinline__ void clear_walls(unsigned walls, float (&v)[M]) {
#pragma unroll
    for (int r = First; r <= Last; ++r)
        if (walls >> r & 1u) v[r] = 0.f;
}
template <bool kSelect>
__device__ __forceinline__ float scaled(float inv, float sum) {
    return !kSelect || inv != 0.f ? inv * sum : 0.f;
}
__device__ __forceinline__ bool fluid_bit(const PresArgs& a, int i) { return (__ldg(a.nbm + i) & 64u) != 0; }
// Cell i of the input iterate; where the mask decides, what a buffer holds on
// non-fluid cells is no iterate.
template <Form F>
__device__ __forceinline__ float input_of(const PresArgs& a, int i) {
    const float v = __ldg(a.pin + i);
    return F == Form::kPasses || fluid_bit(a, i) ? v : 0.f;
}
// Whether cell i of the result is stored: as in the kernel whose sums F are, those of
// the passes by 1/Dp, the others by the mask.
template <Form F>
__device__ __forceinline__ bool written(const PresArgs& a, int i, float inv) {
    return F == Form::kPasses ? inv != 0.f : fluid_bit(a, i);
}

// Above kRegR cells a thread 1/Dp and the right-hand side live in shared
// memory instead of registers.
constexpr size_t pres_smem(int R) {
    return 2 * (size_t)plane_of(R) * R * sizeof(float) + (R > kRegR ? 2 * (size_t)R * NT * sizeof(float) : 0);
}
static_assert(pres_smem(8) <= kSmemMax && pres_smem(10) <= kSmemMax && pres_smem(12) <= kSmemMax &&
              pres_smem(14) <= kSmemMax && pres_smem(16) <= kSmemMax, "boxes exceed the shared memory of one block");

// STACK: every iterate of every cell goes to a.stack.  The loop holds only
// what every sweep does (its code has to stay in the instruction cache: with
// the last sweep's and the optional stores inside, a sweep of an 11 x 8 x 8 box
// alone took 1980 cycles instead of 300); the last sweep follows it.
template <int R, Form F, bool STACK>
__global__ void __launch_bounds__(NT, 1) k_res_pres(const __grid_constant__ PresArgs a) {
    extern __shared__ __align__(16) float sm[];
    constexpr bool NU = F == Form::kStretched;
    constexpr bool kShared = R > kRegR;
    constexpr int PS = plane_of(R);
    const unsigned base = epoch_begin(a.ctl);
    const Box b = make_box(a.pl);
    float* sai = sm + 2 * R * PS;        // after the two boxes: [2][R][NT] 1/Dp, right-hand side
    const int tid = threadIdx.x;
    const int sxy = a.nx * a.ny;
    const size_t N = (size_t)sxy * a.nz;
    int lx, ly;
    const bool own = column_of(b, a.pl, tid, lx, ly), rim = tid < b.inner0;
    const int x = b.x0 + lx, y = b.y0 + ly;
    const bool inxy = own && x < a.nx && y < a.ny;
    const int i0 = inxy ? (b.z0 * a.ny + y) * a.nx + x : 0;
    const int o0 = (ly + 1) * b.sx + lx + 1;
    Links l = make_links(b, a.pl, own, 1);
    if (b.id == a.silent) l.se = l.su = l.sd = -1;
    // the input iterate with its halo, zero outside the domain
    for (int o = tid; o < 2 * R * PS; o += NT) sm[o] = 0.f;
    __syncthreads();
    float p[R], hu = 0.f, hd = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) p[r] = 0.f;
    if (a.pin) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (inxy && b.z0 + r < a.nz) p[r] = input_of<F>(a, i0 + r * sxy);
            if (own) sm[r * PS + o0] = p[r];
        }
        if (inxy && b.z0 > 0) hd = input_of<F>(a, i0 - sxy);
        if (inxy && b.z0 + R < a.nz) hu = input_of<F>(a, i0 + R * sxy);
        if (tid < b.rim + 4) {  // the threads that fetch from plane 0 on
            const int hy = b.y0 + l.he / b.sx - 1, hx = b.x0 + l.he % b.sx - 1;
            if (hx >= 0 && hx < a.nx && hy >= 0 && hy < a.ny) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (b.z0 + r < a.nz) sm[r * PS + l.he] = input_of<F>(a, (b.z0 + r) * sxy + hy * a.nx + hx);
            }
        }
    }
    // the column's coefficients
    float cE[R], cW[R], cN[R], cS[R], cU[R], cD[NU ? R : 1], ai[kShared ? 1 : R], rh[kShared ? 1 : R];
    unsigned walls = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = i0 + r * sxy;
        bool in = inxy && b.z0 + r < a.nz;
        if (NU && in) in = fluid_bit(a, i);  // solid cells hold no coefficients
        if (NU) {
            cE[r] = in ? __ldg(a.c + i) : 0.f;
            cW[r] = in ? __ldg(a.c + N + i) : 0.f;
            cN[r] = in ? __ldg(a.c + 2 * N + i) : 0.f;
            cS[r] = in ? __ldg(a.c + 3 * N + i) : 0.f;
            cU[r] = in ? __ldg(a.c + 4 * N + i) : 0.f;
            cD[NU ? r : 0] = in ? __ldg(a.c + 5 * N + i) : 0.f;
        } else {
            cE[r] = in ? __ldg(a.c + i) : 0.f;
            cW[r] = in && x > 0 ? __ldg(a.c + i - 1) : 0.f;
            cN[r] = in ? __ldg(a.c + N + i) : 0.f;
            cS[r] = in && y > 0 ? __ldg(a.c + N + i - a.nx) : 0.f;
            cU[r] = in ? __ldg(a.c + 2 * N + i) : 0.f;
            if (r == 0) cD[0] = in && b.z0 > 0 ? __ldg(a.c + 2 * N + i - sxy) : 0.f;
        }
        const float e_ai = in ? __ldg(a.ainv + i) : 0.f;
        if (!kShared && own && e_ai == 0.f) walls |= 1u << r;
        const float e_rh = in && a.rhs ? __ldg(a.rhs + i) : 0.f;
        if (kShared) {
            sai[r * NT + tid] = e_ai;
            sai[(R + r) * NT + tid] = e_rh;
        } else {
            ai[kShared ? 0 : r] = e_ai;
            rh[kShared ? 0 : r] = e_rh;
        }
    }
    // cell r of the column from the iterate at q (its own first cell)
    auto inv_of = [&](int r) { return kShared ? sai[r * NT + tid] : ai[kShared ? 0 : r]; };
    auto cell = [&](const float* q, int r, float up, float below) {
        const float *qn = q + b.sx, *qs = q - b.sx;
        float acc;
        if (F != Form::kPasses) {
            acc = __fmaf_rn(-cW[r], q[r * PS - 1], __fmul_rn(-cE[r], q[r * PS + 1]));
        } else {
            acc = -(cE[r] * q[r * PS + 1]);
            acc -= cW[r] * q[r * PS - 1];
        }
        acc -= cN[r] * qn[r * PS];
        acc -= cS[r] * qs[r * PS];
        acc -= cU[r] * up;
        acc -= (NU ? cD[NU ? r : 0] : (r > 0 ? cU[r > 0 ? r - 1 : 0] : cD[0])) * below;
        return scaled<kShared>(inv_of(r), acc + (kShared ? sai[(R + r) * NT + tid] : rh[kShared ? 0 : r]));
    };
    // one sweep of the column from the iterate at `cur`; the two end cells come
    // first, so that their packets can leave before the rest is computed
    auto keep = [&](int k) {
        float* s = a.stack + (size_t)k * N + i0;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (inxy && b.z0 + r < a.nz) s[(size_t)r * sxy] = p[r];
    };
    __syncthreads();
    float *cur = sm + o0, *nxt = sm + R * PS + o0;
    unsigned long long *pk = a.pk, *pk_next = a.pk + a.half;
    unsigned ep = base;
    bool bad = false;
    const bool has_halo = gridDim.x > 1 && (tid & ~31) < b.inner0 + inner_of(a.pl);
    const bool any_walls = !kShared && __any_sync(0xffffffffu, walls != 0);
    float v0, vT;
    auto ends = [&]() {
        v0 = cell(cur, 0, R > 1 ? p[R > 1 ? 1 : 0] : hu, hd);
        vT = R > 1 ? cell(cur, R - 1, hu, p[R > 1 ? R - 2 : 0]) : v0;
        if (any_walls) {
            if (walls & 1u) v0 = 0.f;
            if (walls >> (R - 1) & 1u) vT = 0.f;
        }
    };
    auto middle = [&]() {
        float below = p[0];
        const float top = p[R - 1];
#pragma unroll
        for (int r = 1; r < R - 1; ++r) {
            const float old = p[r];
            p[r] = cell(cur, r, r + 1 < R - 1 ? p[r + 1 < R ? r + 1 : 0] : top, below);
            below = old;
        }
        if (any_walls) clear_walls<1, R - 2>(walls, p);
        p[0] = v0;
        p[R - 1] = vT;
    };
    for (int k = 1; k < a.n; ++k) {
        ++ep;
        ends();
        if (l.sd >= 0) put(pk + l.sd, v0, ep);
        if (l.su >= 0) put(pk + l.su, vT, ep);
        middle();
        if (l.se >= 0) {
            unsigned long long* dst = pk + l.se;
#pragma unroll
            for (int r = 0; r < R; ++r) put(dst + r * b.rim, p[r], ep);
        }
        if (own) {
#pragma unroll
            for (int r = 0; r < R; ++r) nxt[r * PS] = p[r];
        }
        if (STACK) keep(k);
        if (has_halo)
            bad = rim ? !receive<R, true>(l, b.rim, nxt - o0, pk, ep, a.rounds, hu, hd)
                      : !receive<R, false>(l, b.rim, nxt - o0, pk, ep, a.rounds, hu, hd);
        if (__syncthreads_or(bad)) break;
        float* t = cur;
        cur = nxt;
        nxt = t;
        unsigned long long* u = pk;
        pk = pk_next;
        pk_next = u;
    }
    if (ep != base + (unsigned)a.n - 1u || __syncthreads_or(bad)) bad = true;
    if (bad) {
        if (tid == 0 && a.status) atomicExch(a.status, 1);
    } else {
        if (a.pprev) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (inxy && b.z0 + r < a.nz && written<F>(a, i0 + r * sxy, inv_of(r))) a.pprev[i0 + r * sxy] = p[r];
        }
        ends();
        middle();
        if (STACK) keep(a.n);
        if (a.pout) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (inxy && b.z0 + r < a.nz && written<F>(a, i0 + r * sxy, inv_of(r))) a.pout[i0 + r * sxy] = p[r];
        }
    }
    epoch_end(a.ctl, base, (unsigned)a.n + 1u);
}

// ---------------------------------------------- pressure, two sweeps a trip
// On small grids a sweep is mostly the packets' trip.  Here a box exchanges two
// layers of cells (and the edges between them) and runs two sweeps on them: the
// first also on the cells next to the box, which it computes as their owners do,
// the second on its own cells.
// A thread holds a column of the box or of the ring around it, with one cell above
// and below.  Rows of a plane: y = -2 .. by + 1 of bx + 2 words, then the cells two
// off the x faces; planes z = -2 .. R + 1.  A cell's packet has the cell's place in
// its box; the table lists the halo cells, their packets and places.
// Bound by the trip: a pair computes for 0.6 us and waits for 0.9.  Polling takes
// the bandwidth that the packets need (a round reads 2000 of them a box), so a box
// waits kPairWait cycles, about a trip, before the first round, and asks only for
// what is missing after it.  us a sweep, one sweep a trip / pairs polled at once /
// pairs that wait: 64 x 32 x 48 1.10 / 0.95 / 0.77, 80 x 40 x 40 1.16 / 0.98 / 0.81.
// It pays while one round fetches the halo (4 cells a thread): at 72 x 40 x 72,
// 2216 halo cells, 1.21 in either form; and up to 4 cells a thread (with 6 and 8
// the halo computed twice outgrows the trip: 1.2-1.6).
constexpr int kPairPlane = 736, kPairFetch = 4;  // words of a plane; halo cells a thread fetches at most
constexpr int kPairWait = 600;                     // cycles
constexpr int pair_plane_words(const ResPlan& p) { return (p.bx + 2) * (p.by + 4) + 2 * p.by; }
__host__ __device__ constexpr int pair_halo(const ResPlan& p) {
    return 4 * (p.bx * p.by + p.bx * p.bz + p.by * p.bz + p.bx + p.by + p.bz);
}
constexpr size_t pair_smem(const ResPlan& p) {
    return 2 * (size_t)(p.bz + 4) * kPairPlane * sizeof(float) + (size_t)pair_halo(p) * sizeof(int2);
}
// Box coordinates of halo cell e.
__device__ __forceinline__ void pair_cell(const ResPlan& p, int e, int& lx, int& ly, int& lz) {
    const int bx = p.bx, by = p.by, bz = p.bz;
    auto side = [](int q, int b) { return q == 0 ? -1 : q == 1 ? -2 : q == 2 ? b : b + 1; };
    int n = bx * by;
    if (e < 4 * n) {
        lz = side(e / n, bz);
        lx = e % n % bx;
        ly = e % n / bx;
        return;
    }
    e -= 4 * n;
    n = bx * bz;
    if (e < 4 * n) {
        ly = side(e / n, by);
        lx = e % n % bx;
        lz = e % n / bx;
        return;
    }
    e -= 4 * n;
    n = by * bz;
    if (e < 4 * n) {
        lx = side(e % 2 + e / (2 * n) * 2, bx);  // the two layers side by side: one sector
        ly = e / 2 % by;
        lz = e / 2 % n / by;
        return;
    }
    e -= 4 * n;
    auto lo = [](int q, int b) { return q ? b : -1; };
    if (e < 4 * bx) {
        lx = e % bx;
        ly = lo(e / bx & 1, by);
        lz = lo(e / bx >> 1, bz);
        return;
    }
    e -= 4 * bx;
    if (e < 4 * by) {
        ly = e % by;
        lx = lo(e / by & 1, bx);
        lz = lo(e / by >> 1, bz);
        return;
    }
    e -= 4 * by;
    lz = e % bz;
    lx = lo(e / bz & 1, bx);
    ly = lo(e / bz >> 1, by);
}

template <int R, Form F>
__global__ void __launch_bounds__(NT, 1) k_res_pair(const __grid_constant__ PresArgs a) {
    extern __shared__ __align__(16) float sm[];
    constexpr bool NU = F == Form::kStretched;
    constexpr int PS = kPairPlane, BUF = (R + 4) * PS, E = R + 2;
    const unsigned base = epoch_begin(a.ctl);
    const int bx = a.pl.bx, by = a.pl.by, px = a.pl.px, py = a.pl.py, id = blockIdx.x;
    const int x0 = id % px * bx, y0 = id / px % py * by, z0 = id / (px * py) * R;
    const int tid = threadIdx.x, w = bx + 2, cells = R * bx * by;
    const int sxy = a.nx * a.ny;
    const size_t N = (size_t)sxy * a.nz;
    float *s0 = sm, *s1 = sm + BUF;
    int2* tab = reinterpret_cast<int2*>(sm + 2 * BUF);
    const int H = gridDim.x > 1 ? pair_halo(a.pl) : 0;
    for (int o = tid; o < 2 * BUF; o += NT) sm[o] = 0.f;
    __syncthreads();
    for (int e = tid; e < H; e += NT) {
        int lx, ly, lz;
        pair_cell(a.pl, e, lx, ly, lz);
        const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
        const int row = lx == -2 ? w * (by + 4) + ly : lx == bx + 1 ? w * (by + 4) + by + ly : (ly + 2) * w + lx + 1;
        int2 t = make_int2(-1, (lz + 2) * PS + row);
        if (x >= 0 && x < a.nx && y >= 0 && y < a.ny && z >= 0 && z < a.nz) {
            // a non-fluid cell stays 0: its packet is waited for like any other (the
            // protocol needs both directions of a pair of boxes) and goes to the plane's
            // corner word, which no column reads
            const bool fluid = fluid_bit(a, (z * a.ny + y) * a.nx + x);
            if (!fluid) t.y = (lz + 2) * PS;
            const int ox = lx < 0 ? -1 : lx >= bx, oy = ly < 0 ? -1 : ly >= by, oz = lz < 0 ? -1 : lz >= R;
            t.x = (id + ox + px * (oy + py * oz)) * cells + (lx - ox * bx) + bx * ((ly - oy * by) + by * (lz - oz * R));
            if (a.pin && fluid) s0[t.y] = __ldg(a.pin + (z * a.ny + y) * a.nx + x);
        }
        tab[e] = t;
    }
    const int lx = tid % w - 1, ly = tid / w - 1;
    const bool ringx = lx < 0 || lx >= bx, ringy = ly < 0 || ly >= by, own = !ringx && !ringy;
    const int x = x0 + lx, y = y0 + ly;
    const bool col = ly <= by && !(ringx && ringy) && x >= 0 && x < a.nx && y >= 0 && y < a.ny;
    const int o = col ? tid + w : w;
    const int oE = col && lx == bx ? w * (by + 4) + by + ly : o + 1, oW = col && lx < 0 ? w * (by + 4) + ly : o - 1;
    const int i0 = col ? y * a.nx + x : 0;
    const int slot = id * cells + ly * bx + lx;
    const bool sends = H > 0 && id != a.silent;  // every cell: with 4 cells a thread at most few are not read
    const bool mine = own && col, lo = mine && z0 > 0, hi = mine && z0 + R < a.nz;
    // coefficients of the column's cells, j = 0 .. R + 1 for z = -1 .. R
    float cE[E], cW[E], cN[E], cS[E], cU[E], cD[NU ? E : 1], ai[E], rh[E];
    unsigned keep = 0;   // cells that are stored; the others stay 0
#pragma unroll
    for (int j = 0; j < E; ++j) {
        const int z = z0 + j - 1;
        const bool inz = col && z >= 0 && z < a.nz;
        bool in = inz && (own || (j > 0 && j <= R));
        const int i = inz ? z * sxy + i0 : 0;
        if (NU && in) in = fluid_bit(a, i);  // solid cells hold no coefficients
        if (NU) {
            cE[j] = in ? __ldg(a.c + i) : 0.f;
            cW[j] = in ? __ldg(a.c + N + i) : 0.f;
            cN[j] = in ? __ldg(a.c + 2 * N + i) : 0.f;
            cS[j] = in ? __ldg(a.c + 3 * N + i) : 0.f;
            cU[j] = in ? __ldg(a.c + 4 * N + i) : 0.f;
            cD[NU ? j : 0] = in ? __ldg(a.c + 5 * N + i) : 0.f;
        } else {
            cE[j] = in ? __ldg(a.c + i) : 0.f;
            cW[j] = in && x > 0 ? __ldg(a.c + i - 1) : 0.f;
            cN[j] = in ? __ldg(a.c + N + i) : 0.f;
            cS[j] = in && y > 0 ? __ldg(a.c + N + i - a.nx) : 0.f;
            cU[j] = inz ? __ldg(a.c + 2 * N + i) : 0.f;
            if (j == 0) cD[0] = in && z > 0 ? __ldg(a.c + 2 * N + i - sxy) : 0.f;
        }
        ai[j] = in ? __ldg(a.ainv + i) : 0.f;
        if ((j == 0 ? lo : j == R + 1 ? hi : col) && ai[j] != 0.f) keep |= 1u << j;
        if (mine && a.pin && j > 0 && j <= R && ai[j] != 0.f) s0[o + (j + 1) * PS] = __ldg(a.pin + i);
        rh[j] = in && a.rhs ? __ldg(a.rhs + i) : 0.f;
    }
    // cell j of the column from the iterate at s
    auto cell = [&](const float* s, int j, float up, float below) {
        const float* q = s + (j + 1) * PS;
        float acc = F == Form::kPasses ? __fmaf_rn(-cE[j], q[oE], __fmul_rn(-cW[j], q[oW]))
                                       : __fmaf_rn(-cW[j], q[oW], __fmul_rn(-cE[j], q[oE]));
        acc = __fmaf_rn(-cN[j], q[o + w], acc);
        acc = __fmaf_rn(-cS[j], q[o - w], acc);
        acc = __fmaf_rn(-cU[j], up, acc);
        acc = __fmaf_rn(-(NU ? cD[NU ? j : 0] : j > 0 ? cU[j > 0 ? j - 1 : 0] : cD[0]), below, acc);
        return ai[j] * (acc + rh[j]);
    };
    // cells first .. last from the iterate at s; all of them before the first
    // store, so that no load waits for one
    float v[E];
    auto sweep = [&](const float* s, int first, int last) {
        float below = s[o + first * PS], cen = s[o + (first + 1) * PS];
#pragma unroll
        for (int j = 0; j < E; ++j) {
            if (j < first || j > last) continue;
            const float up = s[o + (j + 2) * PS];
            v[j] = cell(s, j, up, below);
            below = cen;
            cen = up;
        }
    };
    auto outer = [&]() {
        sweep(s0, 0, R + 1);
#pragma unroll
        for (int j = 0; j < E; ++j)
            if (keep >> j & 1u) s1[o + (j + 1) * PS] = v[j];
    };
    __syncthreads();
    unsigned long long *pk = a.pk, *pk_next = a.pk + a.half;
    unsigned ep = base;
    bool bad = false;
    const int pairs = (a.n - 1) / 2;
    for (int k = 0; k < pairs; ++k) {
        ++ep;
        outer();
        __syncthreads();
        if (mine) {
            sweep(s1, 1, R);
            unsigned long long* dst = pk + slot;
#pragma unroll
            for (int j = 1; j <= R; ++j)
                if (sends) put(dst + (j - 1) * bx * by, v[j], ep);
#pragma unroll
            for (int j = 1; j <= R; ++j)
                if (keep >> j & 1u) s0[o + (j + 1) * PS] = v[j];
        }
        int left = a.rounds;
        if (H > 0) {
            const long long t0 = clock64();
            while (clock64() - t0 < kPairWait) {}
            int2 t[kPairFetch];
            unsigned long long g[kPairFetch];
#pragma unroll
            for (int u = 0; u < kPairFetch; ++u) {
                t[u] = tid + u * NT < H ? tab[tid + u * NT] : make_int2(-1, 0);
                g[u] = 0;
            }
            bool ok;
            do {
                ok = true;
#pragma unroll
                for (int u = 0; u < kPairFetch; ++u)
                    if (t[u].x >= 0 && (unsigned)(g[u] >> 32) != ep) g[u] = get(pk + t[u].x);
#pragma unroll
                for (int u = 0; u < kPairFetch; ++u) ok = ok && (t[u].x < 0 || (unsigned)(g[u] >> 32) == ep);
            } while (!__all_sync(0xffffffffu, ok) && --left > 0);
#pragma unroll
            for (int u = 0; u < kPairFetch; ++u)
                if (t[u].x >= 0) s0[t[u].y] = __uint_as_float((unsigned)g[u]);
        }
        if (__syncthreads_or(left <= 0)) {
            bad = true;
            break;
        }
        unsigned long long* t = pk;
        pk = pk_next;
        pk_next = t;
    }
    if (bad) {
        if (tid == 0 && a.status) atomicExch(a.status, 1);
    } else {
        const float* from = s0;
        if (a.n - 2 * pairs == 2) {
            outer();
            from = s1;
            __syncthreads();
        }
        if (mine) {
            sweep(from, 1, R);
#pragma unroll
            for (int j = 1; j <= R; ++j) {
                const int i = (z0 + j - 1) * sxy + i0;
                if (z0 + j - 1 < a.nz && written<F>(a, i, ai[j])) {
                    if (a.pprev) a.pprev[i] = from[o + (j + 1) * PS];
                    if (a.pout) a.pout[i] = v[j];
                }
            }
        }
    }
    epoch_end(a.ctl, base, (unsigned)a.n + 1u);
}

// ---------------------------------------------------------------- momentum
// Sweeps u = (1/D) (sum_f A_f u_f + b) of the three components.  One shared
// box (a second barrier a sweep separates its readers from its writers: two
// boxes of three components leave no room for the rest).  Above kVelRegR cells
// a thread b and the second and third component of 1/D live in shared memory.
constexpr int kVelRegR = 4;
constexpr size_t vel_smem(int R) {
    return 3 * (size_t)plane_of(R) * R * sizeof(float) + (R > kVelRegR ? 5 * (size_t)R * NT * sizeof(float) : 0);
}
static_assert(vel_smem(8) <= kSmemMax, "box exceeds the shared memory of one block");

struct VelArgs {
    int nx, ny, nz, n;
    ResPlan pl;
    const float *A, *iD, *bv, *uin;
    float *uout, *uprev;
    Packet3* pk;
    size_t half;
    unsigned* ctl;
    int* status;
    int rounds, silent;
    float* stream;   // k_res_vel_wide: the words read in every sweep
    float* stack;    // iterate k of every cell goes to stack + k step
    long long step;
};

// receive() for three components, CS floats apart in the shared box.  Every
// thread takes a share of the x / y halo, planes g, g + G, ..., so that one trip
// fetches it (a rim thread's R packets of four words do not fit beside the
// coefficients; the pressure loop, whose rim threads hold theirs, lost 5 % by it).
// The share's limit F is fixed at compile time (one packet up to R = 4 and two
// above in k_res_vel): shares of up to four behind a runtime count cost registers
// and a branch each.  us a sweep, rim threads alone / up to four / now: 64 x 32 x
// 48 1.58 / 1.38 / 1.30, 72 x 40 x 72 - / 1.61 / 1.55, 100 x 50 x 100 3.72 / 3.38 /
// 2.96.
template <int F, int CS>
__device__ __forceinline__ bool receive3(const Links& l, float* v, const Packet3* pk, unsigned ep, int rounds,
                                         float hu[3], float hd[3]) {
    const bool nu = l.ru >= 0, nd = l.rd >= 0;
    const Packet3 *pu = pk + (nu ? l.ru : 0), *pd = pk + (nd ? l.rd : 0);
    // (the exception saves registers where F is 4: 6.97 -> 6.67 us on 149 x 61 x 103)
    auto need = [&](int q) { return l.re >= 0 && ((F > 3 && q == 0) || q < l.rn); };
    Packet3 w[F], wu, wd;
    int left = rounds;
    bool ok;
    do {
        wu = get3(pu);
        wd = get3(pd);
#pragma unroll
        for (int q = 0; q < F; ++q) w[q] = get3(pk + (need(q) ? l.re + q * l.rstep : 0));
        ok = (!nu || (unsigned)(wu.hi >> 32) == ep) && (!nd || (unsigned)(wd.hi >> 32) == ep);
#pragma unroll
        for (int q = 0; q < F; ++q) ok = ok && (!need(q) || (unsigned)(w[q].hi >> 32) == ep);
    } while (!__all_sync(0xffffffffu, ok) && --left > 0);
    if (left <= 0) return false;
    hu[0] = nu ? __uint_as_float((unsigned)wu.lo) : 0.f;
    hu[1] = nu ? __uint_as_float((unsigned)(wu.lo >> 32)) : 0.f;
    hu[2] = nu ? __uint_as_float((unsigned)wu.hi) : 0.f;
    hd[0] = nd ? __uint_as_float((unsigned)wd.lo) : 0.f;
    hd[1] = nd ? __uint_as_float((unsigned)(wd.lo >> 32)) : 0.f;
    hd[2] = nd ? __uint_as_float((unsigned)wd.hi) : 0.f;
#pragma unroll
    for (int q = 0; q < F; ++q)
        if (need(q)) {
            float* o = v + l.he + q * l.hstep;
            o[0] = __uint_as_float((unsigned)w[q].lo);
            o[CS] = __uint_as_float((unsigned)(w[q].lo >> 32));
            o[2 * CS] = __uint_as_float((unsigned)w[q].hi);
        }
    return true;
}

// STACK: every iterate of every cell goes to a.stack (non-fluid cells keep the
// input's value); bv nullptr: 0.
template <int R, bool STACK>
__global__ void __launch_bounds__(NT, 1) k_res_vel(const __grid_constant__ VelArgs a) {
    extern __shared__ __align__(16) float sm[];
    constexpr bool kShared = R > kVelRegR;
    constexpr int PS = plane_of(R), CS = R * PS;  // plane, component
    const unsigned base = epoch_begin(a.ctl);
    const Box b = make_box(a.pl);
    float* priv = sm + 3 * CS;                    // [5][R][NT]: b, second and third component of 1/D
    const int tid = threadIdx.x;
    const int sxy = a.nx * a.ny;
    const size_t N = (size_t)sxy * a.nz;
    int lx, ly;
    const bool own = column_of(b, a.pl, tid, lx, ly);
    const int x = b.x0 + lx, y = b.y0 + ly;
    const bool inxy = own && x < a.nx && y < a.ny;
    const int i0 = inxy ? (b.z0 * a.ny + y) * a.nx + x : 0;
    const int o0 = (ly + 1) * b.sx + lx + 1;
    Links l = make_links(b, a.pl, own, NT / (b.rim + 4));
    if (b.id == a.silent) l.se = l.su = l.sd = -1;
    // the input iterate with its halo, zero outside the domain
    for (int o = tid; o < 3 * CS; o += NT) sm[o] = 0.f;
    __syncthreads();
    float u[3][R], hu[3] = {0.f, 0.f, 0.f}, hd[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            u[c][r] = inxy && b.z0 + r < a.nz ? __ldg(a.uin + c * N + i0 + r * sxy) : 0.f;
            if (own) sm[c * CS + r * PS + o0] = u[c][r];
        }
        if (inxy && b.z0 > 0) hd[c] = __ldg(a.uin + c * N + i0 - sxy);
        if (inxy && b.z0 + R < a.nz) hu[c] = __ldg(a.uin + c * N + i0 + R * sxy);
    }
    if (tid < b.rim + 4) {
        const int hy = b.y0 + l.he / b.sx - 1, hx = b.x0 + l.he % b.sx - 1;
        if (hx >= 0 && hx < a.nx && hy >= 0 && hy < a.ny)
            for (int c = 0; c < 3; ++c)
                for (int r = 0; r < R && b.z0 + r < a.nz; ++r)
                    sm[c * CS + r * PS + l.he] = __ldg(a.uin + c * N + (size_t)(b.z0 + r) * sxy + hy * a.nx + hx);
    }
    // the column's coefficients (1/D is 0 on solid cells, whose b is not
    // theirs)
    unsigned walls = 0;
    float A[6][R], d0[R], d12[kShared ? 1 : 2][kShared ? 1 : R], bb[kShared ? 1 : 3][kShared ? 1 : R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = i0 + r * sxy;
        const bool in = inxy && b.z0 + r < a.nz;
#pragma unroll
        for (int f = 0; f < 6; ++f) A[f][r] = in ? __ldg(a.A + f * N + i) : 0.f;
        d0[r] = in ? __ldg(a.iD + i) : 0.f;
        const bool fluid = d0[r] != 0.f;
        if (own && !fluid) walls |= 1u << r;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float v = fluid && a.bv ? __ldg(a.bv + c * N + i) : 0.f;
            if (kShared) priv[(c * R + r) * NT + tid] = v;
            else bb[kShared ? 0 : c][kShared ? 0 : r] = v;
            if (c > 0) {
                const float d = fluid ? __ldg(a.iD + c * N + i) : 0.f;
                if (kShared) priv[((2 + c) * R + r) * NT + tid] = d;
                else d12[kShared ? 0 : c - 1][kShared ? 0 : r] = d;
            }
        }
    }
    float* cur = sm + o0;
    // component c of cell r, in the order of k_vel_sweep4
    auto cell = [&](int c, int r, float up, float below) {
        const float* q = cur + c * CS + r * PS;
        float acc = A[0][r] * q[1];
        acc += A[1][r] * q[-1];
        acc += A[2][r] * cur[b.sx + c * CS + r * PS];
        acc += A[3][r] * (cur - b.sx)[c * CS + r * PS];
        acc += A[4][r] * up;
        acc += A[5][r] * below;
        const float rhs = kShared ? priv[(c * R + r) * NT + tid] : bb[kShared ? 0 : c][kShared ? 0 : r];
        const float d = c == 0 ? d0[r]
                      : kShared ? priv[((2 + c) * R + r) * NT + tid] : d12[kShared ? 0 : (c > 0 ? c - 1 : 0)][kShared ? 0 : r];
        return d * (acc + rhs);
    };
    const bool any_walls = __any_sync(0xffffffffu, walls != 0);
    float v0[3], vT[3];
    auto ends = [&]() {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v0[c] = cell(c, 0, u[c][1], hd[c]);
            vT[c] = cell(c, R - 1, hu[c], u[c][R - 2]);
        }
        if (any_walls) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (walls & 1u) v0[c] = 0.f;
                if (walls >> (R - 1) & 1u) vT[c] = 0.f;
            }
        }
    };
    auto middle = [&]() {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float below = u[c][0];
            const float top = u[c][R - 1];
#pragma unroll
            for (int r = 1; r < R - 1; ++r) {
                const float old = u[c][r];
                u[c][r] = cell(c, r, r + 1 < R - 1 ? u[c][r + 1 < R ? r + 1 : 0] : top, below);
                below = old;
            }
            u[c][0] = v0[c];
            u[c][R - 1] = vT[c];
        }
        if (any_walls) {
#pragma unroll
            for (int c = 0; c < 3; ++c) clear_walls<1, R - 2>(walls, u[c]);
        }
    };
    auto emit = [&](float* out) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (inxy && b.z0 + r < a.nz && d0[r] != 0.f) {
#pragma unroll
                for (int c = 0; c < 3; ++c) out[c * N + i0 + r * sxy] = u[c][r];
            }
    };
    auto keep = [&](int k) {
        float* s = a.stack + k * a.step;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (inxy && b.z0 + r < a.nz) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const size_t i = c * N + i0 + r * sxy;
                    s[i] = d0[r] != 0.f ? u[c][r] : __ldg(a.uin + i);
                }
            }
    };
    __syncthreads();
    Packet3 *pk = a.pk, *pk_next = a.pk + a.half;
    unsigned ep = base;
    bool bad = false;
    for (int k = 1; k < a.n; ++k) {
        ++ep;
        ends();
        if (l.sd >= 0) put3(pk + l.sd, v0[0], v0[1], v0[2], ep);
        if (l.su >= 0) put3(pk + l.su, vT[0], vT[1], vT[2], ep);
        middle();
        if (l.se >= 0) {
            Packet3* dst = pk + l.se;
#pragma unroll
            for (int r = 0; r < R; ++r) put3(dst + r * b.rim, u[0][r], u[1][r], u[2][r], ep);
        }
        __syncthreads();
        if (own) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int r = 0; r < R; ++r) cur[c * CS + r * PS] = u[c][r];
        }
        if (STACK) keep(k);
        if (gridDim.x > 1) bad = !receive3<fetch_max(R), CS>(l, sm, pk, ep, a.rounds, hu, hd);
        if (__syncthreads_or(bad)) break;
        Packet3* t = pk;
        pk = pk_next;
        pk_next = t;
    }
    if (ep != base + (unsigned)a.n - 1u || __syncthreads_or(bad)) bad = true;
    if (bad) {
        if (tid == 0 && a.status) atomicExch(a.status, 1);
    } else {
        if (a.uprev) emit(a.uprev);
        ends();
        middle();
        if (STACK) keep(a.n);
        if (a.uout) emit(a.uout);
    }
    epoch_end(a.ctl, base, (unsigned)a.n + 1u);
}

// ------------------------------------------- momentum, many cells a thread
// Above 8 cells a thread neither the registers nor the shared memory hold the
// twelve coefficient words and three values of a cell.  Here the six A_f stay in
// registers, the iterate in two compact boxes, and of the other six words (1/D and
// b) NR more in registers and NS in shared memory; the rest is read from L2 in
// every sweep, from a copy laid out by thread, a plane ahead of its use.
// Columns go to threads row by row.  A plane has by + 2 rows of bx words, its E
// and W halo columns behind them: a warp's columns are consecutive words whatever
// rows they lie in, and only the lanes on an x edge look elsewhere.
// What bounds it: the shared-memory reads (five a cell and component) and the
// streamed words while it computes, then a halo trip of 33 KB a box.  Measured,
// us a sweep: 4.7 on 128 x 64 x 96 (3.1 without the exchange, 4.1 without the
// streamed words), 6.6 on 149 x 61 x 103, against 6.1 and 11.6 for one sweep a
// launch, which moves all 82 bytes of a cell through L2.  Halo cells fetched
// while the planes are computed, with or without waiting, cost 0.2 us for each
// packet of a thread; all at the end is the fastest.  E and W halo columns
// packed without regard to banks cost 0.35 us on the first.
template <int R> struct Wide;
template <> struct Wide<10> { static constexpr int PS = 640, NR = 1, NS = 3; };
template <> struct Wide<12> { static constexpr int PS = 608, NR = 0, NS = 2; };
template <> struct Wide<14> { static constexpr int PS = 576, NR = 0, NS = 1; };
template <> struct Wide<15> { static constexpr int PS = 576, NR = 0, NS = 0; };
constexpr int wide_plane(int R) {
    return R == 10 ? Wide<10>::PS : R == 12 ? Wide<12>::PS : R == 14 ? Wide<14>::PS : Wide<15>::PS;
}
constexpr int wide_streamed(int R) {
    return 6 - (R == 10 ? Wide<10>::NR + Wide<10>::NS : R == 12 ? Wide<12>::NR + Wide<12>::NS
                : R == 14 ? Wide<14>::NR + Wide<14>::NS : Wide<15>::NR + Wide<15>::NS);
}
template <int R> constexpr size_t wide_smem() {
    return (6 * (size_t)Wide<R>::PS * R + (size_t)Wide<R>::NS * R * NT) * sizeof(float);
}
static_assert(wide_smem<10>() <= kSmemMax && wide_smem<12>() <= kSmemMax && wide_smem<14>() <= kSmemMax &&
              wide_smem<15>() <= kSmemMax, "boxes exceed the shared memory of one block");
// The x / y halo of kGroup planes is fetched at once, by as many threads.
constexpr int kGroup = 4;
// Places of the E and W halo cells of row ly: in the bank of the word that the
// lane would read if its row went on, so that a warp's 32 reads stay in 32
// banks.  The rows' banks repeat after 32 / gcd(bx, 32) rows; with an even bx the
// E cells lie in even banks and the W cells in odd ones.
struct Edges {
    int e, w, period, bx;
    __host__ __device__ explicit Edges(const ResPlan& p) : bx(p.bx) {
        const int low = p.bx & -p.bx;
        period = 32 / (low < 32 ? low : 32);
        e = (p.bx * (p.by + 2) + 31) / 32 * 32;
        w = e + (p.bx & 1 ? (p.by + period - 1) / period * 32 : 0);
    }
    __host__ __device__ int east(int ly) const { return e + ly / period * 32 + ((ly + 2) * bx & 31); }
    __host__ __device__ int west(int ly) const { return w + ly / period * 32 + ((ly + 1) * bx + 31 & 31); }
    __host__ __device__ int words(int by) const { return w + (by + period - 1) / period * 32; }
};

__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

template <int R, bool STACK>
__global__ void __launch_bounds__(NT, 1) k_res_vel_wide(const __grid_constant__ VelArgs a) {
    extern __shared__ __align__(16) float sm[];
    constexpr int PS = Wide<R>::PS, CS = R * PS, BUF = 3 * CS;      // plane, component, box
    constexpr int NR = Wide<R>::NR, NS = Wide<R>::NS, S = 6 - NR - NS;
    const unsigned base = epoch_begin(a.ctl);
    const Box b = make_box(a.pl);
    float* priv = sm + 2 * BUF;                                     // [NS][R][NT]
    const int tid = threadIdx.x, bx = a.pl.bx, by = a.pl.by, cols = bx * by;
    const int sxy = a.nx * a.ny;
    const size_t N = (size_t)sxy * a.nz;
    const bool own = tid < cols;
    const int lx = own ? tid % bx : 0, ly = own ? tid / bx : 0;
    const int x = b.x0 + lx, y = b.y0 + ly;
    const bool inxy = own && x < a.nx && y < a.ny;
    const int i0 = inxy ? (b.z0 * a.ny + y) * a.nx + x : 0;
    const Edges edges(a.pl);
    const int o0 = (ly + 1) * bx + lx;
    const int oE = lx == bx - 1 ? edges.east(ly) : o0 + 1, oW = lx == 0 ? edges.west(ly) : o0 - 1;
    // packets: as in make_links, with the columns in row order
    Links l;
    l.se = l.su = l.sd = l.ru = l.rd = l.re = -1;
    {
        const int iz = b.id / (a.pl.px * a.pl.py), layer = a.pl.px * a.pl.py;
        const int mine = b.id * b.slots, top = R * b.rim;
        if (own) {
            const bool rim = lx == 0 || lx == bx - 1 || ly == 0 || ly == by - 1;
            const int t = lx == bx - 1 ? ly : lx == 0 ? by + ly : 2 * by + (ly == by - 1 ? 0 : bx - 2) + lx - 1;
            if (rim && layer > 1) l.se = mine + t;
            if (iz + 1 < a.pl.pz) {
                l.su = mine + top + tid;
                l.ru = (b.id + layer) * b.slots + top + cols + tid;
            }
            if (iz > 0) {
                l.sd = mine + top + cols + tid;
                l.rd = (b.id - layer) * b.slots + top + tid;
            }
        }
        if (b.id == a.silent) l.se = l.su = l.sd = -1;
    }
    const int g = tid / (b.rim + 4), e = tid % (b.rim + 4);
    int ht, hx, hy;
    const int from = halo_cell(b, a.pl, e, ht, hx, hy);
    l.he = hx == bx ? edges.east(hy) : hx < 0 ? edges.west(hy) : (hy + 1) * bx + hx;
    hx += b.x0;
    hy += b.y0;
    // the input iterate with its halo, zero outside the domain
    for (int o = tid; o < 2 * BUF; o += NT) sm[o] = 0.f;
    __syncthreads();
    float hu[3] = {0.f, 0.f, 0.f}, hd[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (inxy && b.z0 + r < a.nz) sm[c * CS + r * PS + o0] = __ldg(a.uin + c * N + i0 + r * sxy);
        if (inxy && b.z0 > 0) hd[c] = __ldg(a.uin + c * N + i0 - sxy);
        if (inxy && b.z0 + R < a.nz) hu[c] = __ldg(a.uin + c * N + i0 + R * sxy);
    }
    if (g == 0 && hx >= 0 && hx < a.nx && hy >= 0 && hy < a.ny) {
        for (int c = 0; c < 3; ++c)
            for (int r = 0; r < R && b.z0 + r < a.nz; ++r)
                sm[c * CS + r * PS + l.he] = __ldg(a.uin + c * N + (size_t)(b.z0 + r) * sxy + hy * a.nx + hx);
    }
    l.rstep = kGroup * b.rim;
    l.hstep = kGroup * PS;
    l.rn = g < kGroup ? (R - 1 - g) / kGroup + 1 : 0;
    l.he += g * PS;
    if (from >= 0 && l.rn > 0) l.re = from * b.slots + ht + g * b.rim;
    // the column's coefficients: words 0..5 are 1/D_x, b_x, b_y, b_z, 1/D_y, 1/D_z
    // (1/D is 0 on solid cells, whose b is not theirs)
    float A[6][R], wr[NR > 0 ? NR : 1][R];
    float* str = a.stream + (size_t)b.id * (R * S * NT) + tid;      // [R][S][NT] of this box
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = i0 + r * sxy;
        const bool in = inxy && b.z0 + r < a.nz;
#pragma unroll
        for (int f = 0; f < 6; ++f) A[f][r] = in ? __ldg(a.A + f * N + i) : 0.f;
        const float d0 = in ? __ldg(a.iD + i) : 0.f;
        const bool fluid = d0 != 0.f;
#pragma unroll
        for (int w = 0; w < 6; ++w) {
            const float* src = w == 0 ? a.iD : w < 4 ? a.bv + (w - 1) * N : a.iD + (w - 3) * N;
            const float v = w == 0 ? d0 : fluid && (a.bv || w > 3) ? __ldg(src + i) : 0.f;
            if (w < NR) wr[w < NR ? w : 0][r] = v;
            else if (w < NR + NS) priv[((w - NR) * R + r) * NT + tid] = v;
            else str[(r * S + w - NR - NS) * NT] = v;
        }
    }
    float next[S > 0 ? S : 1];
    auto fetch = [&](int r) {
#pragma unroll
        for (int s = 0; s < S; ++s) next[s] = ld_stream(str + (r * S + s) * NT);
    };
    // One sweep from the box `cu`; plane(r, old, new, 1/D_x) takes the results of
    // plane r.
    auto sweep = [&](const float* cu, auto plane) {
        float cen[3], bel[3];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int r = j == 0 ? R - 1 : j - 1;
            float w[6];
#pragma unroll
            for (int s = 0; s < S; ++s) w[NR + NS + s < 6 ? NR + NS + s : 0] = next[s];
            if (j + 1 < R) fetch(j);
#pragma unroll
            for (int q = 0; q < NR + NS; ++q) w[q] = q < NR ? wr[q < NR ? q : 0][r] : priv[((q - NR) * R + r) * NT + tid];
            float v[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int k = c * CS + r * PS;
                if (j < 2) {
                    cen[c] = cu[o0 + k];
                    bel[c] = j == 0 ? cu[o0 + k - PS] : hd[c];
                }
                const float up = j == 0 ? hu[c] : cu[o0 + k + PS];
                // in the order of k_vel_sweep4
                float acc = A[0][r] * cu[oE + k];
                acc += A[1][r] * cu[oW + k];
                acc += A[2][r] * cu[o0 + bx + k];
                acc += A[3][r] * cu[o0 - bx + k];
                acc += A[4][r] * up;
                acc += A[5][r] * bel[c];
                v[c] = w[0] != 0.f ? w[c == 0 ? 0 : 3 + c] * (acc + w[1 + c]) : 0.f;
                bel[c] = cen[c];
                if (j > 0) cen[c] = up;
            }
            plane(r, bel, v, w[0]);
        }
    };
    auto keep = [&](int k, int r, const float* v, float d0) {
        if (!inxy || b.z0 + r >= a.nz) return;
        float* s = a.stack + k * a.step;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const size_t i = c * N + i0 + r * sxy;
            s[i] = d0 != 0.f ? v[c] : __ldg(a.uin + i);
        }
    };
    __syncthreads();
    fetch(R - 1);
    Packet3 *pk = a.pk, *pk_next = a.pk + a.half;
    unsigned ep = base;
    int at = 0;
    bool bad = false;
    for (int k = 1; k < a.n; ++k) {
        ++ep;
        const float* cu = sm + at;
        float* nb = sm + (BUF - at);
        sweep(cu, [&](int r, const float*, const float* v, float d0) {
            if (STACK) keep(k, r, v, d0);
            if (own) {
#pragma unroll
                for (int c = 0; c < 3; ++c) nb[o0 + c * CS + r * PS] = v[c];
            }
            if (l.se >= 0) put3(pk + l.se + r * b.rim, v[0], v[1], v[2], ep);
            if (r == 0 && l.sd >= 0) put3(pk + l.sd, v[0], v[1], v[2], ep);
            if (r == R - 1 && l.su >= 0) put3(pk + l.su, v[0], v[1], v[2], ep);
        });
        fetch(R - 1);
        if (gridDim.x > 1) bad = !receive3<(R + kGroup - 1) / kGroup, CS>(l, nb, pk, ep, a.rounds, hu, hd);
        if (__syncthreads_or(bad)) break;
        Packet3* t = pk;
        pk = pk_next;
        pk_next = t;
        at = BUF - at;
    }
    if (ep != base + (unsigned)a.n - 1u || __syncthreads_or(bad)) bad = true;
    if (bad) {
        if (tid == 0 && a.status) atomicExch(a.status, 1);
    } else {
        sweep(sm + at, [&](int r, const float* old, const float* v, float d0) {
            if (STACK) keep(a.n, r, v, d0);
            if (a.uout && inxy && b.z0 + r < a.nz && d0 != 0.f) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    a.uout[c * N + i0 + r * sxy] = v[c];
                    if (a.uprev) a.uprev[c * N + i0 + r * sxy] = old[c];
                }
            }
        });
    }
    epoch_end(a.ctl, base, (unsigned)a.n + 1u);
}

// Cells per thread the kernels are built for.
constexpr int kPresR[] = {2, 3, 4, 6, 8, 10, 12, 14, 16};
constexpr int kNuPresR[] = {2, 3, 4, 6, 8};
constexpr int kPairR[] = {2, 3, 4};
constexpr int kVelR[] = {2, 3, 4, 6, 8};
constexpr int kVelWideR[] = {10, 12, 14, 15};

using PresKernel = void (*)(const PresArgs);
template <Form F, bool STACK>
PresKernel pres_kernel(int R) {
    switch (R) {
        case 2: return k_res_pres<2, F, STACK>;
        case 3: return k_res_pres<3, F, STACK>;
        case 4: return k_res_pres<4, F, STACK>;
        case 6: return k_res_pres<6, F, STACK>;
        case 8: return k_res_pres<8, F, STACK>;
        default: break;
    }
    if constexpr (F != Form::kStretched) {
        switch (R) {
            case 10: return k_res_pres<10, F, STACK>;
            case 12: return k_res_pres<12, F, STACK>;
            case 14: return k_res_pres<14, F, STACK>;
            case 16: return k_res_pres<16, F, STACK>;
            default: break;
        }
    }
    return nullptr;
}

template <Form F>
PresKernel pair_kernel(int R) {
    switch (R) {
        case 2: return k_res_pair<2, F>;
        case 3: return k_res_pair<3, F>;
        case 4: return k_res_pair<4, F>;
        default: return nullptr;
    }
}

using VelKernel = void (*)(const VelArgs);
template <bool STACK>
VelKernel vel_kernel(int R) {
    switch (R) {
        case 2: return k_res_vel<2, STACK>;
        case 3: return k_res_vel<3, STACK>;
        case 4: return k_res_vel<4, STACK>;
        case 6: return k_res_vel<6, STACK>;
        case 8: return k_res_vel<8, STACK>;
        case 10: return k_res_vel_wide<10, STACK>;
        case 12: return k_res_vel_wide<12, STACK>;
        case 14: return k_res_vel_wide<14, STACK>;
        case 15: return k_res_vel_wide<15, STACK>;
        default: return nullptr;
    }
}

// The split with the least estimated time of a sweep.  Measured (us a sweep):
// 1.10 with 2 cells a thread, 1.13-1.23 with 3, 1.17 with 4, 1.3-1.4 with 6,
// 1.45-1.67 with 8 in 4 to 8 warps, 1.75 in 16 warps, 2.3 with 12, 2.6-2.9 with
// 14, 3.4 with 16: the cells of a thread weigh most (a warp works through
// them one after another), then the warps, then the halo.
// loop: whose limits the split has to keep.
// part > 0: beside other loops the product of a sweep's time and the
// multiprocessors it holds, `part` at least, counts instead, so that as many loops as
// possible run at once.
enum class Loop { kPres, kVel, kVelWide, kPair };
bool fits(const ResPlan& pl, Loop loop) {
    if (rim_of(pl) + 4 > NT) return false;
    if (loop == Loop::kPair)
        return (pl.bx + 2) * (pl.by + 2) <= NT && pair_plane_words(pl) <= kPairPlane &&
               pair_halo(pl) <= kPairFetch * NT;
    if (loop == Loop::kVelWide)
        return pl.bx * pl.by <= NT && Edges(pl).words(pl.by) <= wide_plane(pl.bz) && kGroup * (rim_of(pl) + 4) <= NT;
    return inner0_of(pl) + inner_of(pl) <= NT && (pl.bx + kPad) * (pl.by + 2) <= plane_of(pl.bz) &&
           (loop == Loop::kPres || fetches_of(pl) <= fetch_max(pl.bz));
}
template <size_t M>
ResPlan make_plan(const Params& P, int sms, const int (&Rs)[M], Loop loop = Loop::kPres, int part = 0) {
    ResPlan best;
    double cost = 1e30;
    sms = std::min(sms, kMaxBoxes);
    for (const int R : Rs) {
        const int pz = (P.nz + R - 1) / R;
        for (int px = 1; px <= P.nx && px * pz <= sms; ++px) {
            const int bx = (P.nx + px - 1) / px;
            if (bx < 2 || bx > NT || (P.nx + bx - 1) / bx != px) continue;
            for (int py = 1; py <= P.ny && px * py * pz <= sms; ++py) {
                const int by = (P.ny + py - 1) / py;
                if (by < 2 || (P.ny + by - 1) / by != py) continue;
                ResPlan pl;
                pl.bx = bx; pl.by = by; pl.bz = R;
                pl.pair = loop == Loop::kPair;
                pl.px = px; pl.py = py; pl.pz = pz;
                if (!fits(pl, loop)) continue;
                const double halo = 2.0 * ((px > 1 ? by * R : 0) + (py > 1 ? bx * R : 0) + (pz > 1 ? bx * by : 0));
                double c = R * (60.0 + 0.6 * (inner0_of(pl) / 32 + (inner_of(pl) + 31) / 32)) + 0.03 * halo;
                if (part > 0) c = (500.0 + c) * std::max(pl.boxes(), part);
                if (c < cost) {
                    cost = c;
                    best = pl;
                }
            }
        }
    }
    return best;
}
// A loop on chip first reads its coefficients, every box at once: 5 us with 2 cells a
// thread, 20 to 40 with 8 to 16, what a few sweeps in passes take.  The least number of
// sweeps that pay for it, from the times of loops of 2 to 48 sweeps on 75 grids of 27 to
// 1.1 M cells, cubes, sheets and needles.
// Pressure, by cells a thread.  Uniform: four sweeps a pass take 19 us on any of these
// grids, one or two little less; even at 1 to 2.6 sweeps with up to 8 cells a thread, 3 to 4.5
// above (two sweeps on 149 x 61 x 103 +8 us, five -1).  Stretched: a sweep in passes takes
// 1.2 to 2.4 us; even at 5 to 9 sweeps with 2 and 3 cells a thread, 5 to 12 with 4 and 6, 15
// with 8 (100 x 50 x 100: 8 sweeps +6 us, 24 -6).
int least_pres(const ResPlan& p, bool stretched) {
    const int R = p.bz;
    if (stretched) return R <= 3 ? 9 : R <= 6 ? 12 : 16;
    return R <= 6 ? 2 : R <= 8 ? 3 : R <= 12 ? 4 : 5;
}
// Momentum: the start and a sweep's time by cells a thread (a sweep of boxes with few
// columns takes less), against a sweep in passes: four cells a thread 1.8 us up to 0.1 M
// cells, 5.1 at 0.5 M, 6.3 at 0.86 M; one cell a thread (nx % 4 != 0) 2.4 + 9.3 a million.  Even
// (computed, measured): 64 x 32 x 48 15, 11; 72 x 40 x 72 8, 5; 100 x 50 x 100 11, 9; 128 x 64
// x 96 21, 20; 149 x 61 x 103 10, 8; 128 x 60 x 112 and needles such as 3 x 3 x 2000 never.
int least_vel(const Params& P, const ResPlan& p) {
    static constexpr struct { int R; double start, sweep; } kCost[] = {
        {2, 7, 1.40}, {3, 8.7, 1.45}, {4, 9.7, 1.55}, {6, 14, 2.2}, {8, 22, 2.95},
        {10, 20, 3.95}, {12, 26, 4.7}, {14, 35, 6.2}, {15, 39, 6.8}};
    const double m = 1e-6 * P.N, fill = (double)P.N / ((double)p.boxes() * NT * p.bz);
    const double pass = P.nx % 4 == 0 ? std::max(1.8, m < 0.5 ? 1.8 + 8.25 * (m - 0.1) : 5.1 + 3.3 * (m - 0.5))
                                      : 2.35 + 9.3 * m;
    for (const auto& c : kCost) {
        if (c.R != p.bz) continue;
        const double thin = 0.6 + 0.18 * c.R;
        const double gain = pass - (thin + (c.sweep - thin) * std::min(1.0, fill / 0.75));
        return gain > 0.0 ? std::max(2, (int)std::min(c.start / gain + 1.0, 1e9)) : INT_MAX;
    }
    return 2;
}
// Words of the momentum loop's streamed coefficients.
size_t streamed(const ResPlan& p) {
    return p.bz > kVelR[std::size(kVelR) - 1] ? (size_t)p.boxes() * p.bz * wide_streamed(p.bz) * NT : 0;
}
size_t vel_bytes(int R) {
    switch (R) {
        case 10: return wide_smem<10>();
        case 12: return wide_smem<12>();
        case 14: return wide_smem<14>();
        case 15: return wide_smem<15>();
        default: return vel_smem(R);
    }
}
size_t packets(const ResPlan& p) {
    if (p.pair) return (size_t)p.boxes() * p.bx * p.by * p.bz;
    return p.bz > 0 ? (size_t)p.boxes() * slots_of(p) : 0;
}

cudaError_t launch_coop(const void* fn, int blocks, size_t smem, cudaStream_t st, void* args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* argv[] = {args};
    return cudaLaunchKernelExC(&cfg, fn, argv);
}

}  // namespace

int resident_setup(const Resident& r) {
    cudaError_t e = cudaSuccess;
    auto opt_in = [&](auto k) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
    };
    if (r.pres.bz > 0) {
        opt_in(pres_kernel<Form::kPasses, false>(r.pres.bz));
        opt_in(pres_kernel<Form::kPasses, true>(r.pres.bz));
        opt_in(pres_kernel<Form::kOrdered, false>(r.pres.bz));
    }
    if (r.pres2.bz > 0) {
        opt_in(pair_kernel<Form::kPasses>(r.pres2.bz));
        opt_in(pair_kernel<Form::kOrdered>(r.pres2.bz));
        opt_in(pair_kernel<Form::kStretched>(r.pres2.bz));
    }
    if (r.nupres.bz > 0) opt_in(pres_kernel<Form::kStretched, false>(r.nupres.bz));
    if (r.pres_shared.bz > 0) opt_in(pres_kernel<Form::kPasses, false>(r.pres_shared.bz));
    if (r.pres_beside.bz > 0)
        opt_in(r.pres_beside.pair ? pair_kernel<Form::kPasses>(r.pres_beside.bz)
                                  : pres_kernel<Form::kPasses, false>(r.pres_beside.bz));
    if (r.nupres_beside.bz > 0)
        opt_in(r.nupres_beside.pair ? pair_kernel<Form::kStretched>(r.nupres_beside.bz)
                                    : pres_kernel<Form::kStretched, false>(r.nupres_beside.bz));
    if (r.vel.bz > 0) opt_in(vel_kernel<true>(r.vel.bz));
    for (const ResPlan& p : {r.vel, r.vel_shared, r.vel_beside})
        if (p.bz > 0) opt_in(vel_kernel<false>(p.bz));
    return e == cudaSuccess ? WF_OK : WF_ERR_CUDA;
}

void resident_plan(const Params& P, int sms, Resident* r) {
    r->pres = make_plan(P, sms, kPresR);
    r->nupres = make_plan(P, sms, kNuPresR);
    r->pres2 = make_plan(P, sms, kPairR, Loop::kPair);
    r->nupres2 = r->pres2;
    r->vel = make_plan(P, sms, kVelR, Loop::kVel);
    if (r->vel.bz == 0) r->vel = make_plan(P, sms, kVelWideR, Loop::kVelWide);
    for (ResPlan* p : {&r->pres, &r->pres2}) p->least = least_pres(*p, false);
    for (ResPlan* p : {&r->nupres, &r->nupres2}) p->least = least_pres(*p, true);
    r->vel.least = least_vel(P, r->vel);
    r->pres_shared = make_plan(P, sms, kPresR, Loop::kPres, 1);
    r->vel_shared = make_plan(P, sms, kVelR, Loop::kVel, 1);
    // Beside other handles: an eighth of the multiprocessors costs nothing yet.
    const int part = std::max(sms / 8, 1);
    const ResPlan pair = make_plan(P, sms, kPairR, Loop::kPair, part);
    auto better = [&](const ResPlan& p) { return pair.bz > 0 && pair.boxes() <= std::max(p.boxes(), part) ? pair : p; };
    r->pres_beside = better(make_plan(P, sms, kPresR, Loop::kPres, part));
    r->nupres_beside = better(make_plan(P, sms, kNuPresR, Loop::kPres, part));
    r->vel_beside = make_plan(P, sms, kVelR, Loop::kVel, part);
    // In company a loop counts by the multiprocessors it holds.  Steps of 2, 4 and 8 sweeps a
    // loop, passes / chip: 16 cases of 24 x 12 x 16 in a batch 102 / 135, 141 / 155, 207 / 187 us, of
    // 0.1 and 0.2 M cells 707 / 798, 874 / 886, 1199 / 1029; side by side 88 / 95, 128 / 101, 194
    // / 117 and 726 / 798, 979 / 887, 1370 / 1017.
    r->pres_shared.least = r->vel_shared.least = 6;
    r->pres_beside.least = r->vel_beside.least = 4;
    r->nupres_beside.least = least_pres(r->nupres_beside, true);
}

void resident_alloc(Resident* r, cudaStream_t st) {
    // both parities of the pressure packets, then of the momentum packets
    // (apart: a momentum packet's words must not be read as pressure
    // packets), then the epoch words
    const size_t np = 2 * std::max({packets(r->pres), packets(r->nupres), packets(r->pres2), packets(r->pres_shared),
                                    packets(r->pres_beside), packets(r->nupres_beside)}),
                 nv = 2 * std::max({packets(r->vel), packets(r->vel_shared), packets(r->vel_beside)});
    if (np + nv == 0 || r->work.pk) return;
    const size_t bytes = np * sizeof(unsigned long long) + nv * sizeof(Packet3) + 16 +
                         streamed(r->vel) * sizeof(float);
    void* pk = nullptr;
    if (cudaMalloc(&pk, bytes) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (cudaMemsetAsync(pk, 0, bytes - streamed(r->vel) * sizeof(float), st) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(pk);
        return;
    }
    r->work.pk = pk;
    r->work.pk3 = static_cast<unsigned long long*>(pk) + np;  // np is even: 16-byte aligned
    r->work.ctl = reinterpret_cast<unsigned*>(static_cast<Packet3*>(r->work.pk3) + nv);
    r->work.stream = reinterpret_cast<float*>(r->work.ctl + 4);
}

void resident_free(Resident* r) {
    if (r->work.pk) cudaFree(r->work.pk);
    r->work = ResWork();
}

namespace {
cudaError_t launch_pres(PresKernel k, const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w,
                        const float* c, const float* ainv, const float* rhs, const float* pin, float* pout,
                        float* pprev, float* stack, int n, int* status) {
    PresArgs a = {};
    a.nx = P.nx; a.ny = P.ny; a.nz = P.nz; a.n = n;
    a.pl = pl;
    a.c = c; a.ainv = ainv; a.rhs = rhs; a.nbm = P.nbm;
    a.pin = pin; a.pout = pout; a.pprev = pprev; a.stack = stack;
    a.pk = static_cast<unsigned long long*>(w.pk);
    a.half = packets(pl);
    a.ctl = w.ctl;
    a.status = status;
    a.rounds = w.rounds;
    a.silent = w.silent;
    const cudaError_t e = launch_coop((const void*)k, pl.boxes(), pl.pair ? pair_smem(pl) : pres_smem(pl.bz), st, &a);
    if (e == cudaSuccess) WF_COUNT_LAUNCH();
    else cudaGetLastError();
    return e;
}
}  // namespace

cudaError_t launch_res_pres(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w, const float* c3,
                            const float* ainv, const float* rhs, const float* pin, float* pout, float* pprev,
                            float* stack, int n, int* status, bool ordered) {
    const PresKernel k = pl.pair   ? ordered ? pair_kernel<Form::kOrdered>(pl.bz) : pair_kernel<Form::kPasses>(pl.bz)
                         : stack   ? pres_kernel<Form::kPasses, true>(pl.bz)
                         : ordered ? pres_kernel<Form::kOrdered, false>(pl.bz)
                                   : pres_kernel<Form::kPasses, false>(pl.bz);
    return launch_pres(k, P, st, pl, w, c3, ainv, rhs, pin, pout, pprev, stack, n, status);
}

cudaError_t launch_res_nupres(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w,
                              const float* coef, const float* bp, const float* pin, float* pout, float* pprev, int n,
                              int* status) {
    return launch_pres(pl.pair ? pair_kernel<Form::kStretched>(pl.bz) : pres_kernel<Form::kStretched, false>(pl.bz), P, st, pl, w, coef, coef + 6 * (size_t)P.N, bp, pin,
                       pout, pprev, nullptr, n, status);
}

cudaError_t launch_res_vel(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w, const float* A,
                           const float* iD, const float* bv, const float* uin, float* uout, float* uprev, int n,
                           int* status, float* stack, long long step) {
    VelArgs a = {};
    a.nx = P.nx; a.ny = P.ny; a.nz = P.nz; a.n = n;
    a.pl = pl;
    a.A = A; a.iD = iD; a.bv = bv; a.uin = uin;
    a.uout = uout; a.uprev = uprev;
    a.pk = static_cast<Packet3*>(w.pk3);
    a.half = packets(pl);
    a.ctl = w.ctl;
    a.status = status;
    a.rounds = w.rounds;
    a.silent = w.silent;
    a.stream = w.stream;
    a.stack = stack;
    a.step = step;
    const VelKernel k = stack ? vel_kernel<true>(pl.bz) : vel_kernel<false>(pl.bz);
    const cudaError_t e = launch_coop((const void*)k, pl.boxes(), vel_bytes(pl.bz), st, &a);
    if (e == cudaSuccess) WF_COUNT_LAUNCH();
    else cudaGetLastError();
    return e;
}

}  // namespace wf
