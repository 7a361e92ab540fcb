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
// not memory.  Measured, us a sweep: 1.1 on 64 x 32 x 48, 1.13 on 80 x 40 x 40,
// 1.75 on 100 x 50 x 100, 2.3 on 128 x 64 x 96, 3.5 on 149 x 61 x 103.  Whole
// steps, with the four-sweep passes before: 623 -> 310 us (64 x 32 x 48, PISO,
// 90 pressure sweeps), 5077 -> 1467 us (80 x 40 x 40, 1000), 2425 -> 1059 us (100 x 50 x
// 100, 400), 1278 -> 1027 us (128 x 64 x 96, 90), 1396 -> 1186 us (149 x 61 x 103, 90),
// 9761 -> 8258 us (100 x 50 x 100 stretched mesh, 2000).  With the momentum loop
// on chip too: 310 -> 269 us (64 x 32 x 48, 50 sweeps), 1467 -> 1399 us (80 x 40 x 40,
// 100), 1059 -> 982 us (100 x 50 x 100, 50), 8258 -> 6753 us (stretched mesh, 800).
//
// The launch is cooperative, so all blocks are resident and every packet
// that is waited for will be sent.  The waits are bounded all the same
// (kRounds): a wait that runs out sets *status and the block returns, its
// neighbours' waits then run out as well.
#include <cuda_runtime.h>

#include <algorithm>

#include "wf_kernels.cuh"
#include "wf_resident.cuh"

namespace wf {
namespace {

constexpr int NT = 512;                               // threads of a block, one z column each
// Limit of one wait, in polling rounds: a round is one trip to L2 (0.2 to
// 0.5 us), so a wait ends after one to two seconds.
constexpr int kRounds = 1 << 22;
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
// `groups`: planes whose halo cells are fetched by different threads.
__device__ __forceinline__ Links make_links(const Box& b, const ResPlan& pl, bool own, int groups) {
    Links l;
    const int tid = threadIdx.x, mine = b.id * b.slots;
    const int ix = b.id % pl.px, iy = (b.id / pl.px) % pl.py, iz = b.id / (pl.px * pl.py);
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
    // halo cell e of the E, W, N, S side and the rim thread of the neighbour
    // box that owns it
    const int bx = pl.bx, by = pl.by;
    int from = -1, t = 0, hx = 0, hy = 0;
    if (e < by) {
        if (ix + 1 < pl.px) from = b.id + 1;
        hx = bx; hy = e;
        t = by + e;
    } else if (e < 2 * by) {
        if (ix > 0) from = b.id - 1;
        hx = -1; hy = e - by;
        t = hy;
    } else if (e < 2 * by + bx) {
        if (iy + 1 < pl.py) from = b.id + pl.px;
        hx = e - 2 * by; hy = by;
        t = hx == bx - 1 ? 0 : hx == 0 ? by : 2 * by + bx - 2 + hx - 1;
    } else {
        if (iy > 0) from = b.id - pl.px;
        hx = e - 2 * by - bx; hy = -1;
        t = hx == bx - 1 ? by - 1 : hx == 0 ? 2 * by - 1 : 2 * by + hx - 1;
    }
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
                                        float& hu, float& hd) {
    const bool nu = l.ru >= 0, nd = l.rd >= 0, ne = RIM && l.re >= 0;
    const unsigned long long *pu = pk + (nu ? l.ru : 0), *pd = pk + (nd ? l.rd : 0), *pe = pk + (ne ? l.re : 0);
    constexpr int U = !RIM ? 0 : R <= 8 ? R : (R + 1) / 2;
#pragma unroll
    for (int r0 = 0; r0 < (RIM ? R : 1); r0 += RIM ? U : 1) {
        unsigned long long w[U + 1], wu = 0, wd = 0;
        int left = kRounds;
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
    const uint8_t* nbm;            // neighbour masks (non-uniform)
    const float* pin;
    float *pout, *pprev, *stack;
    unsigned long long* pk;
    size_t half;                   // packets of one parity
    unsigned* ctl;
    int* status;
};

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
    const Links l = make_links(b, a.pl, own, 1);
    // the input iterate with its halo, zero outside the domain
    for (int o = tid; o < 2 * R * PS; o += NT) sm[o] = 0.f;
    __syncthreads();
    float p[R], hu = 0.f, hd = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) p[r] = 0.f;
    if (a.pin) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (inxy && b.z0 + r < a.nz) p[r] = __ldg(a.pin + i0 + r * sxy);
            if (own) sm[r * PS + o0] = p[r];
        }
        if (inxy && b.z0 > 0) hd = __ldg(a.pin + i0 - sxy);
        if (inxy && b.z0 + R < a.nz) hu = __ldg(a.pin + i0 + R * sxy);
        if (tid < b.rim + 4) {  // the threads that fetch from plane 0 on
            const int hy = b.y0 + l.he / b.sx - 1, hx = b.x0 + l.he % b.sx - 1;
            if (hx >= 0 && hx < a.nx && hy >= 0 && hy < a.ny)
                for (int r = 0; r < R && b.z0 + r < a.nz; ++r)
                    sm[r * PS + l.he] = __ldg(a.pin + (size_t)(b.z0 + r) * sxy + hy * a.nx + hx);
        }
    }
    // the column's coefficients
    float cE[R], cW[R], cN[R], cS[R], cU[R], cD[NU ? R : 1], ai[kShared ? 1 : R], rh[kShared ? 1 : R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = i0 + r * sxy;
        bool in = inxy && b.z0 + r < a.nz;
        if (NU && in) in = (__ldg(a.nbm + i) & 64u) != 0;  // solid cells hold no coefficients
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
        return inv_of(r) * (acc + (kShared ? sai[(R + r) * NT + tid] : rh[kShared ? 0 : r]));
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
    float v0, vT;
    auto ends = [&]() {
        v0 = cell(cur, 0, R > 1 ? p[R > 1 ? 1 : 0] : hu, hd);
        vT = R > 1 ? cell(cur, R - 1, hu, p[R > 1 ? R - 2 : 0]) : v0;
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
            bad = rim ? !receive<R, true>(l, b.rim, nxt - o0, pk, ep, hu, hd)
                      : !receive<R, false>(l, b.rim, nxt - o0, pk, ep, hu, hd);
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
                if (inxy && b.z0 + r < a.nz && inv_of(r) != 0.f) a.pprev[i0 + r * sxy] = p[r];
        }
        ends();
        middle();
        if (STACK) keep(a.n);
        if (a.pout) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (inxy && b.z0 + r < a.nz && inv_of(r) != 0.f) a.pout[i0 + r * sxy] = p[r];
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
};

// receive() for three components, CS floats apart in the shared box.  Every
// thread takes a share of the x / y halo, so that one trip fetches it (a rim
// thread's R packets of four words do not fit beside the coefficients; the
// pressure loop, whose rim threads hold theirs, lost 5 % by it).  The share is
// one packet up to R = 4 and two above, fixed at compile time: shares of up to
// four behind a runtime count cost registers and a branch each.  us a sweep, rim
// threads alone / up to four / now: 64 x 32 x 48 1.58 / 1.38 / 1.30, 72 x 40 x 72
// - / 1.61 / 1.55, 100 x 50 x 100 3.72 / 3.38 / 2.96.
template <int R>
__device__ __forceinline__ bool receive3(const Links& l, float* v, const Packet3* pk, unsigned ep, float hu[3],
                                         float hd[3]) {
    constexpr int F = fetch_max(R), CS = R * plane_of(R);
    const bool nu = l.ru >= 0, nd = l.rd >= 0, ne = l.re >= 0;
    const Packet3 *pu = pk + (nu ? l.ru : 0), *pd = pk + (nd ? l.rd : 0), *pe = pk + (ne ? l.re : 0);
    const int second = F > 1 && l.rn > 1 ? l.rstep : 0;
    Packet3 w[F], wu, wd;
    int left = kRounds;
    bool ok;
    do {
        wu = get3(pu);
        wd = get3(pd);
        w[0] = get3(pe);
        if (F > 1) w[F - 1] = get3(pe + second);
        ok = (!nu || (unsigned)(wu.hi >> 32) == ep) && (!nd || (unsigned)(wd.hi >> 32) == ep);
        ok = ok && (!ne || ((unsigned)(w[0].hi >> 32) == ep && (unsigned)(w[F - 1].hi >> 32) == ep));
    } while (!__all_sync(0xffffffffu, ok) && --left);
    if (left == 0) return false;
    hu[0] = nu ? __uint_as_float((unsigned)wu.lo) : 0.f;
    hu[1] = nu ? __uint_as_float((unsigned)(wu.lo >> 32)) : 0.f;
    hu[2] = nu ? __uint_as_float((unsigned)wu.hi) : 0.f;
    hd[0] = nd ? __uint_as_float((unsigned)wd.lo) : 0.f;
    hd[1] = nd ? __uint_as_float((unsigned)(wd.lo >> 32)) : 0.f;
    hd[2] = nd ? __uint_as_float((unsigned)wd.hi) : 0.f;
    if (ne) {
        // a thread with one halo cell fetches and writes it twice
        const int at[2] = {l.he, l.he + (second ? l.hstep : 0)};
#pragma unroll
        for (int q = 0; q < F; ++q) {
            float* o = v + at[q];
            o[0] = __uint_as_float((unsigned)w[q].lo);
            o[CS] = __uint_as_float((unsigned)(w[q].lo >> 32));
            o[2 * CS] = __uint_as_float((unsigned)w[q].hi);
        }
    }
    return true;
}

template <int R>
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
    const Links l = make_links(b, a.pl, own, NT / (b.rim + 4));
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
    float A[6][R], d0[R], d12[kShared ? 1 : 2][kShared ? 1 : R], bb[kShared ? 1 : 3][kShared ? 1 : R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = i0 + r * sxy;
        const bool in = inxy && b.z0 + r < a.nz;
#pragma unroll
        for (int f = 0; f < 6; ++f) A[f][r] = in ? __ldg(a.A + f * N + i) : 0.f;
        d0[r] = in ? __ldg(a.iD + i) : 0.f;
        const bool fluid = d0[r] != 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float v = fluid ? __ldg(a.bv + c * N + i) : 0.f;
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
    float v0[3], vT[3];
    auto ends = [&]() {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v0[c] = cell(c, 0, u[c][1], hd[c]);
            vT[c] = cell(c, R - 1, hu[c], u[c][R - 2]);
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
    };
    auto emit = [&](float* out) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (inxy && b.z0 + r < a.nz && d0[r] != 0.f) {
#pragma unroll
                for (int c = 0; c < 3; ++c) out[c * N + i0 + r * sxy] = u[c][r];
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
        if (gridDim.x > 1) bad = !receive3<R>(l, sm, pk, ep, hu, hd);
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
        emit(a.uout);
    }
    epoch_end(a.ctl, base, (unsigned)a.n + 1u);
}

// Cells per thread the kernels are built for.
constexpr int kPresR[] = {2, 3, 4, 6, 8, 10, 12, 14, 16};
constexpr int kNuPresR[] = {2, 3, 4, 6, 8};
constexpr int kVelR[] = {2, 3, 4, 6, 8};

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

using VelKernel = void (*)(const VelArgs);
VelKernel vel_kernel(int R) {
    switch (R) {
        case 2: return k_res_vel<2>;
        case 3: return k_res_vel<3>;
        case 4: return k_res_vel<4>;
        case 6: return k_res_vel<6>;
        case 8: return k_res_vel<8>;
        default: return nullptr;
    }
}

// The split with the least estimated time of a sweep.  Measured (us a sweep):
// 1.10 with 2 cells a thread, 1.13-1.23 with 3, 1.17 with 4, 1.3-1.4 with 6,
// 1.45-1.67 with 8 in 4 to 8 warps, 1.75 in 16 warps, 2.3 with 12, 2.6-2.9 with
// 14, 3.4 with 16: the cells of a thread weigh most (a warp works through
// them one after another), then the warps, then the halo.
// shared: beside other cases' loops the product of a sweep's time and the
// multiprocessors it holds counts instead, so that as many loops as possible
// run at once.
template <size_t M>
ResPlan make_plan(const Params& P, int sms, const int (&Rs)[M], bool momentum = false, bool shared = false) {
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
                pl.px = px; pl.py = py; pl.pz = pz;
                if (inner0_of(pl) + inner_of(pl) > NT || (bx + kPad) * (by + 2) > plane_of(R) ||
                    rim_of(pl) + 4 > NT || (momentum && fetches_of(pl) > fetch_max(R)))
                    continue;
                const double halo = 2.0 * ((px > 1 ? by * R : 0) + (py > 1 ? bx * R : 0) + (pz > 1 ? bx * by : 0));
                double c = R * (60.0 + 0.6 * (inner0_of(pl) / 32 + (inner_of(pl) + 31) / 32)) + 0.03 * halo;
                if (shared) c = (500.0 + c) * pl.boxes();
                if (c < cost) {
                    cost = c;
                    best = pl;
                }
            }
        }
    }
    return best;
}
size_t packets(const ResPlan& p) {
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
    if (r.nupres.bz > 0) opt_in(pres_kernel<Form::kStretched, false>(r.nupres.bz));
    if (r.pres_shared.bz > 0) opt_in(pres_kernel<Form::kPasses, false>(r.pres_shared.bz));
    for (const ResPlan& p : {r.vel, r.vel_shared})
        if (p.bz > 0) opt_in(vel_kernel(p.bz));
    return e == cudaSuccess ? WF_OK : WF_ERR_CUDA;
}

void resident_plan(const Params& P, int sms, Resident* r) {
    r->pres = make_plan(P, sms, kPresR);
    r->nupres = make_plan(P, sms, kNuPresR);
    r->vel = make_plan(P, sms, kVelR, true);
    r->pres_shared = make_plan(P, sms, kPresR, false, true);
    r->vel_shared = make_plan(P, sms, kVelR, true, true);
}

void resident_alloc(Resident* r, cudaStream_t st) {
    // both parities of the pressure packets, then of the momentum packets
    // (apart: a momentum packet's words must not be read as pressure
    // packets), then the epoch words
    const size_t np = 2 * std::max({packets(r->pres), packets(r->nupres), packets(r->pres_shared)}),
                 nv = 2 * std::max(packets(r->vel), packets(r->vel_shared));
    if (np + nv == 0 || r->work.pk) return;
    const size_t bytes = np * sizeof(unsigned long long) + nv * sizeof(Packet3) + 16;
    void* pk = nullptr;
    if (cudaMalloc(&pk, bytes) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (cudaMemsetAsync(pk, 0, bytes, st) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(pk);
        return;
    }
    r->work.pk = pk;
    r->work.pk3 = static_cast<unsigned long long*>(pk) + np;  // np is even: 16-byte aligned
    r->work.ctl = reinterpret_cast<unsigned*>(static_cast<Packet3*>(r->work.pk3) + nv);
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
    const cudaError_t e = launch_coop((const void*)k, pl.boxes(), pres_smem(pl.bz), st, &a);
    if (e == cudaSuccess) WF_COUNT_LAUNCH();
    else cudaGetLastError();
    return e;
}
}  // namespace

cudaError_t launch_res_pres(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w, const float* c3,
                            const float* ainv, const float* rhs, const float* pin, float* pout, float* pprev,
                            float* stack, int n, int* status, bool ordered) {
    const PresKernel k = stack     ? pres_kernel<Form::kPasses, true>(pl.bz)
                         : ordered ? pres_kernel<Form::kOrdered, false>(pl.bz)
                                   : pres_kernel<Form::kPasses, false>(pl.bz);
    return launch_pres(k, P, st, pl, w, c3, ainv, rhs, pin, pout, pprev, stack, n, status);
}

cudaError_t launch_res_nupres(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w,
                              const float* coef, const float* bp, const float* pin, float* pout, float* pprev, int n,
                              int* status) {
    return launch_pres(pres_kernel<Form::kStretched, false>(pl.bz), P, st, pl, w, coef, coef + 6 * (size_t)P.N, bp, pin,
                       pout, pprev, nullptr, n, status);
}

cudaError_t launch_res_vel(const Params& P, cudaStream_t st, const ResPlan& pl, const ResWork& w, const float* A,
                           const float* iD, const float* bv, const float* uin, float* uout, float* uprev, int n,
                           int* status) {
    VelArgs a = {};
    a.nx = P.nx; a.ny = P.ny; a.nz = P.nz; a.n = n;
    a.pl = pl;
    a.A = A; a.iD = iD; a.bv = bv; a.uin = uin;
    a.uout = uout; a.uprev = uprev;
    a.pk = static_cast<Packet3*>(w.pk3);
    a.half = packets(pl);
    a.ctl = w.ctl;
    a.status = status;
    const cudaError_t e = launch_coop((const void*)vel_kernel(pl.bz), pl.boxes(), vel_smem(pl.bz), st, &a);
    if (e == cudaSuccess) WF_COUNT_LAUNCH();
    else cudaGetLastError();
    return e;
}

}  // namespace wf
