// ifc_persist2d.cuh -- the whole 2D SIMPLE loop in one cooperative launch.
//
// Every CTA owns one tile for the whole solve or, when the grid has more tiles
// than co-resident CTAs, a fixed set of tiles that it visits in turn inside
// every phase, and walks through the phases of each outer iteration
// (src/Solver.cu:160-289):
//   momentum passes (assembly + ks red-black sweeps of u and v on the tile's
//   region in registers, ifc_tile2d.cuh), Rhie-Chow faces + p' source, p'
//   passes, [p' mean removal], corrections + convergence test,
// separated by grid barriers instead of kernel boundaries.  After each barrier
// every CTA reads all CTAs' FP64 partial sums and reduces them in one fixed
// order, so every CTA takes the same early-exit and convergence decisions
// without another barrier.  The decisions are taken by two warps while the next
// pass (after the corrections: the first pass of the next outer iteration)
// already runs; a pass that the decision makes superfluous is not stored.
// Waiting for them first costs 3 us per pass of the 58 us that an outer
// iteration of the 512x128 channel takes.  Barrier waits are bounded: a CTA
// that waits longer than kBarrierTimeoutNs sets the error flag, every CTA leaves
// the loop, and the host reports IFC_TIMEOUT.  The launch is cooperative, so all
// CTAs are co-resident or the launch fails (the engine then uses the
// multi-kernel graph).
#pragma once

#include "ifc_fused2d.cuh"
#include "ifc_tile2d.cuh"

namespace ifc {

struct GridBarrier {
    unsigned int count;  // arrivals since the launch; barrier k completes at (k+1)*G
    unsigned int gen;    // unused, kept for layout
    int err;
};

constexpr unsigned long long kBarrierTimeoutNs = 2000000000ull;  // 2 s

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// The wait of a grid barrier: until `target` arrivals are in, or the limit.  One
// L2 round trip per poll; the error flag and the clock are read every 64 polls
// only, so they stay off the critical path.  A CTA that passes this barrier
// while another gave up meets the flag at the next barrier, which the other
// never reaches.
__device__ __forceinline__ int await_arrivals(GridBarrier *b, unsigned int target)
{
    const unsigned long long t0 = global_ns();
    unsigned int spins = 0;
    while (ld_acquire(&b->count) < target) {
        if ((++spins & 63u) == 0) {
            if (*(volatile int *)&b->err) return 0;
            if (global_ns() - t0 > kBarrierTimeoutNs) {
                atomicExch(&b->err, 1);
                return 0;
            }
        }
    }
    return 1;
}

// Grid barrier on a monotonically increasing arrival counter: each CTA adds
// one arrival and waits until all G arrivals of this barrier are in, so the
// critical path is one atomic plus the pollers' next read.  `epoch` counts
// the barriers this CTA has passed (same in every CTA).  Returns false in
// every thread of the CTA when the wait timed out or another CTA reported an
// error.  SINGLE: a launch of one CTA needs the block barrier only.  Not taken by
// k_csolve3d, which is bound by its two barriers per sweep and loses 2 to 4 % to
// the extra exit (67x39x25 cavity 564 -> 576 us per outer iteration).
template <bool SINGLE = true>
__device__ __forceinline__ bool grid_sync(GridBarrier *b, unsigned int nblocks, unsigned int &epoch)
{
    __shared__ int ok;
    __syncthreads();
    if (SINGLE && nblocks == 1) return true;  // the block barrier orders everything
    ++epoch;
    if (threadIdx.x == 0) {
        int good = 1;
        const unsigned int target = epoch * nblocks;
        // The arrival releases this CTA's writes (ordered before it by the
        // __syncthreads above) and, for the last CTA to arrive, acquires the
        // others'; the pollers acquire them through ld.acquire.  (An arrival
        // without a return value, polled at once, is slower: 2380 against 2110
        // cycles for 108 CTAs, the polls then queue before the arrivals.)
        unsigned int old;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(&b->count) : "memory");
        if (old + 1 < target) good = await_arrivals(b, target);
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// The two halves of grid_sync, with work of the CTA's own between them that no
// other CTA reads before a later barrier.  Every thread of a CTA of NT threads
// calls both.
template <int NT>
__device__ __forceinline__ void grid_arrive(GridBarrier *b, unsigned int nblocks, unsigned int &epoch)
{
    if (nblocks == 1) return;
    ++epoch;
    if (threadIdx.x < 32) {
        asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
        if (threadIdx.x == 0)
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&b->count) : "memory");
    } else {
        asm volatile("bar.arrive 1, %0;" ::"n"(NT) : "memory");
    }
}

__device__ __forceinline__ bool grid_wait(GridBarrier *b, unsigned int nblocks, unsigned int epoch)
{
    __shared__ int ok;
    if (nblocks > 1 && threadIdx.x == 0) ok = await_arrivals(b, epoch * nblocks);
    __syncthreads();
    return nblocks == 1 || ok != 0;
}

// Sum column r of partials (one value per CTA) for r < ncol in a fixed order;
// identical in every CTA (a single CTA has its totals in `out` already).  Warp w
// sums columns w, w + NT/32, ... (each lane-strided, then one shuffle tree), so
// the columns are reduced in parallel with one round trip to L2.  out: shared,
// ncol entries.
template <int NT>
static __device__ __noinline__ void reduce_partials(const double *partials, int ncol, int G, double *out)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = warp; r < ncol && G > 1; r += NT / 32) {
        const double *col = partials + (size_t)r * G;
        double x = 0.0;
#pragma unroll 4
        for (int b = lane; b < G; b += 32) x += __ldcg(&col[b]);
        x = warp_sum(x);
        if (lane == 0) out[r] = x;
    }
    __syncthreads();
}

constexpr int kMaxPassSweeps = 10;  // sweeps per pass of the single-launch solve, at most
// Columns of the partial sums: two sets used in turn (a set is rewritten only
// after the barrier of the other set's sums, which every CTA reaches after
// reading the first), then the mass imbalance.
constexpr int kSetColumns = 2 * kMaxPassSweeps;
constexpr int kMassColumn = 2 * kSetColumns;

// Block-uniform loop state, kept in shared memory.
struct LoopState {
    int it, it_begin, it_stop, act, log_level, log_n, status, done;
    int stop[4], sweeps[4];
    int ends;                   // the pass of the pending decision ends a group
    int hit[4];                 // the early-exit rule was met (it ends the sweeps where a group of passes ends)
    long long cell_updates[4];  // by equation, so that two warps can count at once
    double inner_max_sq[4];     // largest sum of squared changes of a sweep; negative: none yet
    double maxn[8];
};

struct PersistArgs {
    int n_iter[4];
    int pin;
    int one;               // one tile per CTA
    int ks;                // sweeps per pass
    int npass_m, npass_p;  // momentum and p' passes
    int group;             // passes per early-exit check: the sweeps end early after a multiple of ks * group only
    int tail_m, tail_p;    // the first pass of a phase's last group
    TileGrid tiles;  // tiles for a halo of 2*ks cells
    int stall_test;  // failure-detection test: CTA 0 leaves before its first barrier
};

// The early-exit rule of src/Solver.cu:955-962 evaluated after each sweep of a
// pass (ns <= 16), by one warp: lane s takes sweep s, the running maximum is a
// prefix maximum, and the first sweep that meets the rule ends the evaluation.
// Returns the sweep that met it or -1; mx: the largest sum up to there (the
// largest sum stands for the largest RMS: the root and the division by N keep
// the order; a NaN sum leaves the maximum).
// floor: a largest RMS from before this launch (-1e20: none).
static __device__ __noinline__ int exit_rule(double own, double before, double floor, int ns, int N, double tol,
                                             double *mx_out)
{
    const int lane = threadIdx.x & 31;
    double mx = own > before ? own : before;
#pragma unroll 1
    for (int o = 1; o < 16; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, mx, o);
        if (lane >= o && y > mx) mx = y;
    }
    const double rms = sqrt(own / (double)N);
    double top = mx >= 0.0 ? sqrt(mx / (double)N) : -1e20;
    if (floor > top) top = floor;
    const unsigned hit = __ballot_sync(0xffffffffu, lane < ns && rms / (top + 1e-20) < tol);
    const int at = hit ? __ffs(hit) - 1 : ns - 1;
    *mx_out = __shfl_sync(0xffffffffu, mx, at < 0 ? 0 : at);
    return hit ? at : -1;
}

// Inner bookkeeping for one equation after a pass, by one warp.  The rule
// itself (five FP64 roots and quotients, one after the other in one thread 3.5
// us per pass) is only evaluated when some sweep comes within a factor of the
// tolerance; otherwise the smallest and the largest sum show that none meets
// it.  Sums are not negative, so they order as their bits do.
// grouped: several passes per check; ends: the pass ends a group, so the sweeps
// may end here.
__device__ __forceinline__ void pass_done(LoopState &L, int e, const double *sq, int ns, int N, double tol,
                                          bool grouped, bool ends, double floor = -1e20)
{
    const int lane = threadIdx.x & 31;
    const double own = sq[lane < ns ? lane : 0], before = L.inner_max_sq[e];
    const unsigned hi = (unsigned)__double2hiint(own), lo = (unsigned)__double2loint(own);
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi), nhi = __reduce_min_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    double mx = __hiloint2double((int)mhi, (int)mlo);
    const double least = __hiloint2double((int)nhi, 0);
    if (before > mx) mx = before;
    bool stop = false;
    const double top = floor > 0.0 && floor * floor * N > mx ? floor * floor * N : mx;
    if (!(least > 1.001 * tol * tol * top && least > 1e-30 * N && mhi < 0x7ff00000u))
        stop = exit_rule(lane < ns ? own : 0.0, before, floor, ns, N, tol, &mx) >= 0;
    if (lane == 0) {
        L.inner_max_sq[e] = mx;
        L.sweeps[e] += ns;
        L.cell_updates[e] += (long long)ns * N;
        if (stop || (grouped && L.hit[e])) (ends ? L.stop : L.hit)[e] = 1;
    }
}

// Bookkeeping of the passes of a phase's last group: their sums could only set
// an early-exit flag for passes that do not follow (the flags are reset with
// every outer iteration), so they are not taken.
__device__ __forceinline__ void pass_count(LoopState &L, int e, int ns, int N)
{
    L.sweeps[e] += ns;
    L.cell_updates[e] += (long long)ns * N;
}

// The deferred correction of one cell, out of line (its scheme switch is
// large and only higher-order convection runs it).
template <typename T>
static __device__ __noinline__ T dc_call(const Geo<T> &g, const T *phi, int c, int i, int j, T uw, T ue, T vs, T vn)
{
    return dc_cell<T, 2>(g, phi, c, i, j, 0, uw, ue, vs, vn, (T)0, (T)0);
}

// End of an outer iteration, by one warp: norms, convergence test and log
// (src/Solver.cu:226-289), then the inner bookkeeping is reset for the next
// iteration.  tot: sums of p u v - uf vf -, mass.  Lane q < 8 holds norm q.
template <typename T>
static __device__ __noinline__ void finish_norms(const Geo<T> &g, LoopState &L, Ctl *ctl, const double *tot, double mass_sq)
{
    const int lane = threadIdx.x & 31, nx = g.nx, ny = g.ny, N = g.N;
    const bool field = lane < 7 && lane != 3 && lane != 6;
    const double cnt = lane == 4 ? (double)(nx - 1) * ny : lane == 5 ? (double)nx * (ny - 1) : (double)N;
    const double nq = field ? sqrt(tot[lane] / cnt) : lane == 7 ? sqrt(mass_sq / cnt) : 0.0;
    double mq = lane < 8 ? L.maxn[lane] : 0.0;
    const int it = L.it + 1;
    bool bad = __any_sync(0xffffffffu, !isfinite(nq));
    if (!bad && it - L.it_begin > 1) bad = __any_sync(0xffffffffu, lane < 7 && mq > 0.0 && nq > 1e6 * mq);
    double rel = 0.0;
    if (g.criterion == 0) {
        const double n0 = __shfl_sync(0xffffffffu, nq, 0), m0 = __shfl_sync(0xffffffffu, mq, 0);
        const double top = n0 > m0 ? n0 : m0;
        if (lane == 0) mq = top;
        if (lane < 7) rel = nq / top;
    } else if (field) {
        if (nq > mq) mq = nq;
        rel = mq > 0.0 ? nq / mq : 0.0;
    }
    const double tol = lane == 0 ? g.tol[EQ_P] : lane == 1 || lane == 4 ? g.tol[EQ_U] : g.tol[EQ_V];
    const double mass = __shfl_sync(0xffffffffu, nq, 7);
    bool conv = __all_sync(0xffffffffu, !field || rel < tol);
    conv = conv || mass < g.tol_mass;
    const int local = it - L.it_begin;
    const bool last = it >= L.it_stop || (L.act && conv) || bad;
    const bool rec = blockIdx.x == 0 && L.log_level > 0 && (local == 1 || local % 1000 == 0 || conv || last);
    const int slot = L.log_n < kLogCap ? L.log_n : kLogCap - 1;
    if (blockIdx.x == 0) {
        if (lane < 8) {
            ctl->norm[lane] = nq;
            ctl->maxn[lane] = mq;
        }
        if (lane < 7) {
            ctl->sq[lane] = field ? tot[lane] : 0.0;
            ctl->rel[lane] = rel;
            if (rec) ctl->log[slot].rel[lane] = rel;
        }
        if (lane < 4) ctl->it_sweeps[lane] = L.sweeps[lane];
    }
    __syncwarp();
    if (lane < 8) L.maxn[lane] = mq;
    if (lane < 4) {
        L.stop[lane] = 0;
        L.hit[lane] = 0;
        L.sweeps[lane] = 0;
        L.inner_max_sq[lane] = -1.0;
    }
    if (lane == 0) {
        L.it = it;
        if (bad) L.status = 2;
        if (blockIdx.x == 0) {
            ctl->sq[SQ_MASS] = mass_sq;
            ctl->it = it;
            ctl->converged = conv ? 1 : 0;
            if (bad) ctl->status = 2;
            ctl->cell_updates = L.cell_updates[0] + L.cell_updates[1] + L.cell_updates[2] + L.cell_updates[3];
            if (rec) {
                LogRec &R2 = ctl->log[slot];
                R2.it = local;
                R2.converged = conv;
                R2.mass = mass;
                if (L.log_n < kLogCap) L.log_n++;
                ctl->log_n = L.log_n;
            }
        }
        L.done = last;
    }
}

// A decision whose sums have been written (partials, `ncol` columns from `part`)
// but not yet taken; n0, n1: the sweeps of u (or p') and v that they cover.
enum { kPendNone = 0, kPendMomentum, kPendP, kPendNorms };

struct Pending {
    int kind, ncol, n0, n1;
    int part;  // offset of the first column in the partials
    __device__ __forceinline__ void set(int k, int p, int columns, int a, int b)
    {
        kind = k;
        ncol = columns;
        n0 = a;
        n1 = b;
        part = p;
    }
};

// The grid totals of a pending decision's columns into tot, by all warps
// (fixed order; a single CTA has them there already); the eighth column of the
// norms is the mass imbalance, its total goes to tot_mass.  Every
// warp reads at most ceil(ncol / NW) columns, all loads of one first.
template <int NW>
__device__ __forceinline__ void pending_totals(const Pending &pd, const double *partials, int G, double *tot,
                                               double *tot_mass)
{
    if (G == 1) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
    for (int c = warp; c < pd.ncol; c += NW) {
        const bool is_mass = pd.kind == kPendNorms && c == 7;
        const double *col = partials + (is_mass ? kMassColumn * G : pd.part + c * G);
        double x = 0.0;
#pragma unroll 1
        for (int b0 = 0; b0 < G; b0 += 160) {
            double y[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) y[k] = b0 + 32 * k + lane < G ? __ldcg(&col[b0 + 32 * k + lane]) : 0.0;
#pragma unroll
            for (int k = 0; k < 5; ++k) x += y[k];
        }
        x = warp_sum(x);
        if (lane == 0) *(is_mass ? tot_mass : tot + c) = x;
    }
}

// Takes the decision: warp 0 (u, p' or the norms) and warp 1 (v), after a
// block barrier; the outcome is in L after the next one.
template <typename T>
__device__ __forceinline__ void decide(const Geo<T> &g, LoopState &L, Ctl *ctl, const double *tot,
                                       const double &mass_sq, const Pending &pd, int ks, bool grouped)
{
    const int warp = threadIdx.x >> 5;
    if (warp > 1) return;
    if (pd.kind == kPendNorms) {
        if (warp == 0) finish_norms<T>(g, L, ctl, tot, mass_sq);
        return;
    }
    const int e = warp == 1 ? EQ_V : pd.kind == kPendP ? EQ_P : EQ_U;
    const int n = warp == 1 ? pd.n1 : pd.n0;
    if (n > 0) pass_done(L, e, tot + (warp == 1 ? ks : 0), n, g.N, g.tol[e], grouped, !grouped || L.ends);
}

// Faces whose loads one thread has in flight in the Rhie-Chow phase.
constexpr int kFaces = 2;

// The persistent kernel of one region shape.  One-tile CTAs keep the links,
// diagonals and sources of their region in registers through all passes of a
// phase and reload only the halo cells of the unknowns between passes.
template <typename T, int R_, int NW_>
__global__ void __launch_bounds__(32 * NW_, 1) k_simple2d(const __grid_constant__ Params<T> P,
                                                       const __grid_constant__ Fields<T> f, Ctl *ctl, double *partials,
                                                       GridBarrier *bar, const __grid_constant__ PersistArgs pa)
{
    using RT = RTile<T, R_, NW_>;
    constexpr int R = RT::R, NT = RT::NT, NW = RT::NW;
    const Geo<T> &g = P.g;
    const int nx = g.nx, ny = g.ny, N = g.N;
    const int G = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ntiles = pa.tiles.kx * pa.tiles.ky;
    const bool one = pa.one != 0;  // one tile per CTA
    const int ks = pa.ks;

    double *sred = reinterpret_cast<double *>(tile_smem<T>() + RT::END);  // per-thread sums of each sweep
    T *s_f = reinterpret_cast<T *>(sred);                                 // Rhie-Chow: the tile's faces
    __shared__ LoopState L;
    __shared__ double tot[2 * kMaxPassSweeps];
    __shared__ double tot_mass;

    if (tid == 0) {
        L.it = ctl->it;
        L.it_begin = ctl->it_begin;
        L.it_stop = ctl->it_stop;
        L.act = ctl->act;
        L.log_level = ctl->log_level;
        L.log_n = ctl->log_n;
        L.status = 0;
        L.done = L.it >= L.it_stop;
        for (int q = 0; q < 4; ++q) {
            L.cell_updates[q] = 0;
            L.stop[q] = 0;
            L.hit[q] = 0;
            L.sweeps[q] = 0;
            L.inner_max_sq[q] = -1.0;
        }
        for (int q = 0; q < 8; ++q) L.maxn[q] = ctl->maxn[q];
    }
    clear_guards<RT, T>();
    __syncthreads();

    bool failed = false;
    unsigned int epoch = 0;
    int set = 0;
    const int set_len = kSetColumns * G;
    // A pass stages halos from one buffer and writes its tile to the other, so
    // no tile reads a neighbour tile's values of the same pass; `mcur`/`pcur`
    // (the same in every CTA) say which buffer holds the current u, v / p'.
    auto bu = [&](int q) { return field_view(q ? (T *)f.tmp : (T *)f.u, N); };
    auto bv = [&](int q) { return field_view(q ? (T *)f.tmp + N : (T *)f.v, N); };
    auto bp = [&](int q) { return field_view(q ? (T *)f.tmp + 2 * (size_t)N : (T *)f.pc, N); };

    // The lane's place in the CTA's first tile, kept in FP64 only: in FP32 it is
    // cheaper to find anew in every pass than to hold (4096x2048 2.85 -> 2.73 ms per
    // outer iteration; FP64 500x190 104 -> 108 us).
    constexpr bool kKeepPlace = sizeof(T) == 8;
    const LanePlace<RT> place(tile_box(pa.tiles, blockIdx.x, nx, ny), ny);
    Pending pending;
    pending.kind = kPendNone;
    // Takes a pending decision at once: with several tiles per CTA (a
    // superfluous pass would read faces that the next phase of another CTA may
    // already be writing) and at the end of the call.
    auto resolve_now = [&]() {
        pending_totals<NW>(pending, partials, G, tot, &tot_mass);
        __syncthreads();
        decide<T>(g, L, ctl, tot, tot_mass, pending, ks, pa.group > 1);
        __syncthreads();
        pending.kind = kPendNone;
    };

#pragma unroll 1
    while (!L.done) {
        int mcur = 0, pcur = 0;

        // Failure-detection test (IFC_TEST_STALL_BARRIER=1 in the environment):
        // CTA 0 leaves without arriving, so every other CTA's bounded wait at the
        // next barrier runs out and the launch ends with the timeout status.
        if (pa.stall_test && blockIdx.x == 0) { failed = true; break; }

        // ---- deferred-correction sources (higher-order convection), from the
        // fields at the start of the outer iteration; the momentum passes read
        // them for their halos too, so a barrier follows ----
        if (g.conv != CONV_UPWIND) {
#pragma unroll 1
            for (int t = blockIdx.x; t < ntiles; t += G) {
                const TileBox tl = tile_box(pa.tiles, t, nx, ny);
                // one component of one cell per thread
                const int ow = tl.ox1 - tl.ox0, cells = ow * (tl.oy1 - tl.oy0);
                const SmallDiv dow(ow);
#pragma unroll 1
                for (int q = tid; q < 2 * cells; q += NT) {
                    const int e = q >= cells ? 1 : 0, q2 = q - e * cells, b = dow.div(q2);
                    const int i = tl.gx0 + tl.ox0 + q2 - b * ow, j = tl.gy0 + tl.oy0 + b, c = i + nx * j;
                    f.sdc[e * N + c] = dc_call<T>(g, e ? f.v : f.u, c, i, j, f.uf[i + (nx + 1) * j],
                                                  f.uf[i + 1 + (nx + 1) * j], f.vf[c], f.vf[c + nx]);
                }
            }
            if (!grid_sync(bar, G, epoch)) { failed = true; break; }
        }

        // ---------------- momentum passes ----------------
        {
            Links<RT, T> a;
            Cells<T, R> u, v;
            bool force = false;
#pragma unroll 1
            for (int pass = 0; pass < (pa.npass_m > 0 ? pa.npass_m : 1); ++pass) {
                const int ns0 = clamp_sweeps(pa.n_iter[0], pass, ks), ns1 = clamp_sweeps(pa.n_iter[1], pass, ks);
                // what is known of the early exits so far (the last pass's sums
                // may still be pending; the first pass starts a new iteration)
                const bool au = ns0 > 0 && (pass == 0 || !L.stop[EQ_U]);
                const bool av = ns1 > 0 && (pass == 0 || !L.stop[EQ_V]);
                if (!au && !av && pass > 0) break;
                const bool sums = pass < pa.tail_m;
                const bool keep = one && pass > 0;
                bool cu = au, cv = av;  // whether this pass's u, v count
#pragma unroll 1
                for (int t = blockIdx.x; t < ntiles; t += G) {
                    const LanePlace<RT> pl = kKeepPlace && one ? place : LanePlace<RT>(tile_box(pa.tiles, t, nx, ny), ny);
                    if (keep) {
                        load_cells<RT, T>(u, bu(mcur), pl, nx, ny, true, kOutside<T>);
                        load_cells<RT, T>(v, bv(mcur), pl, nx, ny, true, kOutside<T>);
                    } else {
                        load_cells<RT, T>(u, bu(mcur), pl, nx, ny, false, kOutside<T>);
                        load_cells<RT, T>(v, bv(mcur), pl, nx, ny, false, kOutside<T>);
                    }
                    if (pending.kind) pending_totals<NW>(pending, partials, G, tot, &tot_mass);
                    if (!keep) force = mom_links<RT, T>(P, f, pl, a);
                    publish<RT, T>(u, 0);
                    publish<RT, T>(v, 1);
                    __syncthreads();
                    if (pending.kind)
                        decide<T>(g, L, ctl, tot, tot_mass, pending, ks, pa.group > 1);
                    sweeps2<RT, T>(u, v, a, pl, g.relax[EQ_U], g.relax[EQ_V], force, au ? ns0 : 0,
                                   av ? ns1 : 0, ks, sums, t != (int)blockIdx.x, sred);
                    if (pending.kind) {
                        if (ns0 == 0 && ns1 == 0) __syncthreads();  // (the sweeps have barriers otherwise)
                        pending.kind = kPendNone;
                        if (L.done) break;
                        if (pass > 0) {
                            cu = au && !L.stop[EQ_U];
                            cv = av && !L.stop[EQ_V];
                            if (!cu && !cv) break;
                        }
                    }
                    // an unknown that had already stopped keeps its values
                    if (au && !cu) load_cells<RT, T>(u, bu(mcur), pl, nx, ny, false, kOutside<T>);
                    if (av && !cv) load_cells<RT, T>(v, bv(mcur), pl, nx, ny, false, kOutside<T>);
                    if (pass == 0) store_diagonal<RT, T>(a, f.ac, f.rac, pl, nx);
                    store_own<RT, T>(u, bu(mcur ^ 1), pl, nx);
                    store_own<RT, T>(v, bv(mcur ^ 1), pl, nx);
                }
                if (L.done || (pass > 0 && !cu && !cv)) break;
                mcur ^= 1;
                if (sums) column_partials<NT>(sred, 2 * ks, partials + set * set_len, G, tot);
                if (!grid_sync(bar, G, epoch)) { failed = true; break; }
                if (!sums) {
                    if (tid == 0) {
                        if (cu) pass_count(L, EQ_U, ns0, N);
                        if (cv) pass_count(L, EQ_V, ns1, N);
                    }
                    continue;
                }
                pending.set(kPendMomentum, set * set_len, 2 * ks, cu ? ns0 : 0, cv ? ns1 : 0);
                if (tid == 0 && pa.group > 1) L.ends = ((pass + 1) & (pa.group - 1)) == 0;
                set ^= 1;
                if (!one) resolve_now();
            }
        }
        if (failed || L.done) break;

        // ------------- Rhie-Chow faces, face BCs, p' source -------------
        Fields<T> fc = f;  // the current u, v
        fc.u = bu(mcur);
        fc.v = bv(mcur);
        {
            double m = 0.0;
            // The tile's x-faces and y-faces, spread over the threads, into
            // shared memory; then every cell's mass imbalance from its four
            // faces.  A face on the tile's east or north edge is also computed
            // by the next tile, which owns and stores it (same operations, same
            // value).
#pragma unroll 1
            for (int t = blockIdx.x; t < ntiles; t += G) {
                const TileBox tl = tile_box(pa.tiles, t, nx, ny);
                const int ow = tl.ox1 - tl.ox0, oh = tl.oy1 - tl.oy0, x0 = tl.gx0 + tl.ox0, y0 = tl.gy0 + tl.oy0;
                const int nfx = (ow + 1) * oh, nf = nfx + ow * (oh + 1);
                const SmallDiv dfx(ow + 1), dfy(ow);
                T *s_fy = s_f + nfx;
#pragma unroll 1
                for (int q0 = tid; q0 < nf; q0 += kFaces * NT) {
                    // the loads of kFaces faces first, then their arithmetic
                    T vL[kFaces], vR[kFaces], aL[kFaces], aR[kFaces], rL[kFaces], rR[kFaces];
                    T pLL[kFaces], pL[kFaces], pR[kFaces], pRR[kFaces];
#pragma unroll
                    for (int m_ = 0; m_ < kFaces; ++m_) {
                        const int q = q0 + m_ * NT;
                        if (q >= nf) continue;
                        const bool fx = q < nfx;
                        const int q2 = fx ? q : q - nfx, b = (fx ? dfx : dfy).div(q2), a = q2 - b * (fx ? ow + 1 : ow);
                        const int i = x0 + a, j = y0 + b;
                        const int k = fx ? i : j, n = fx ? nx : ny, st = fx ? 1 : nx;  // face k of n + 1 along its axis
                        const int cr = i + nx * j, cR = k < n ? cr : cr - st, cL = k > 0 ? cr - st : cr;
                        const T *vel = fx ? fc.u : fc.v;
                        vL[m_] = vel[cL];
                        vR[m_] = vel[cR];
                        aL[m_] = f.ac[cL];
                        aR[m_] = f.ac[cR];
                        rL[m_] = f.rac[cL];
                        rR[m_] = f.rac[cR];
                        pL[m_] = f.p[cL];
                        pR[m_] = f.p[cR];
                        pLL[m_] = k >= 2 ? f.p[cL - st] : (g.closed[fx ? WEST : SOUTH] ? pL[m_] : (T)0);
                        pRR[m_] = k <= n - 2 ? f.p[cR + st] : (g.closed[fx ? EAST : NORTH] ? pR[m_] : (T)0);
                    }
#pragma unroll
                    for (int m_ = 0; m_ < kFaces; ++m_) {
                        const int q = q0 + m_ * NT;
                        if (q >= nf) continue;
                        const bool fx = q < nfx;
                        const int q2 = fx ? q : q - nfx, b = (fx ? dfx : dfy).div(q2), a = q2 - b * (fx ? ow + 1 : ow);
                        const int i = x0 + a, j = y0 + b;
                        const int k = fx ? i : j, n = fx ? nx : ny;
                        T val;
                        if (k == 0) val = fx ? face_bc(g, WEST, 0, vR[m_], j) : face_bc(g, SOUTH, 1, vR[m_], 0);
                        else if (k == n) val = fx ? face_bc(g, EAST, 0, vL[m_], j) : face_bc(g, NORTH, 1, vL[m_], 0);
                        else val = rc_face_known(vL[m_], vR[m_], aL[m_], aR[m_], rL[m_], rR[m_], pLL[m_], pL[m_], pR[m_],
                                                 pRR[m_], fx ? g.Ax : g.Ay);
                        s_f[q] = val;
                        if (fx) {
                            if (a < ow || i == nx) f.uf[i + (nx + 1) * j] = val;
                        } else {
                            if (b < oh || j == ny) f.vf[i + nx * j] = val;
                        }
                    }
                }
                __syncthreads();
#pragma unroll 1
                for (int q = tid; q < ow * oh; q += NT) {
                    const int b = dfy.div(q), a = q - b * ow;
                    const T bm = mass_imbalance<T, 2>(g, s_f[a + (ow + 1) * b], s_f[a + 1 + (ow + 1) * b],
                                                      s_fy[a + ow * b], s_fy[a + ow * (b + 1)], (T)0, (T)0);
                    f.sp[x0 + a + nx * (y0 + b)] = bm;
                    m += (double)bm * (double)bm;
                }
                __syncthreads();  // the next tile's faces overwrite s_f
            }
            sred[tid] = m;  // the faces are no longer needed (barrier above)
            __syncthreads();
            column_partials<NT>(sred, 1, partials + kMassColumn * (size_t)G, G, &tot_mass);
            if (!grid_sync(bar, G, epoch)) break;
        }

        // ---------------- p' passes ----------------
        {
            Links<RT, T> a;
            Cells<T, R> x;
            bool force = false;
#pragma unroll 1
            for (int pass = 0; pass < pa.npass_p; ++pass) {
                const int ns = clamp_sweeps(pa.n_iter[3], pass, ks);
                if (pass > 0 && L.stop[EQ_P]) break;
                const bool sums = pass < pa.tail_p;
                const bool keep = one && pass > 0;
                bool stopped = false;
#pragma unroll 1
                for (int t = blockIdx.x; t < ntiles; t += G) {
                    const LanePlace<RT> pl = kKeepPlace && one ? place : LanePlace<RT>(tile_box(pa.tiles, t, nx, ny), ny);
                    if (pass == 0) zero_cells<RT, T>(x, pl, nx, ny);
                    else load_cells<RT, T>(x, bp(pcur), pl, nx, ny, keep, kOutside<T>);
                    if (pending.kind) pending_totals<NW>(pending, partials, G, tot, &tot_mass);
                    if (!keep) force = pc_links<RT, T>(P, f, pl, a);
                    publish<RT, T>(x, 0);
                    __syncthreads();
                    if (pending.kind)
                        decide<T>(g, L, ctl, tot, tot_mass, pending, ks, pa.group > 1);
                    sweeps1<RT, T>(x, a, pl, g.relax[EQ_P], force, ns, ks, sums, t != (int)blockIdx.x, sred);
                    if (pending.kind) {
                        pending.kind = kPendNone;
                        stopped = L.stop[EQ_P] != 0;
                        if (stopped) break;
                    }
                    store_own<RT, T>(x, bp(pcur ^ 1), pl, nx);
                }
                if (stopped) break;
                pcur ^= 1;
                if (sums) column_partials<NT>(sred, ks, partials + set * set_len, G, tot);
                if (!grid_sync(bar, G, epoch)) { failed = true; break; }
                if (!sums) {
                    if (tid == 0) pass_count(L, EQ_P, ns, N);
                    continue;
                }
                pending.set(kPendP, set * set_len, ks, ns, 0);
                if (tid == 0 && pa.group > 1) L.ends = ((pass + 1) & (pa.group - 1)) == 0;
                set ^= 1;
                if (!one) resolve_now();
            }
        }
        if (failed) break;

        const FieldArr<T> pcc = bp(pcur);  // the current p'
        if (pa.npass_p == 0) {       // no p' sweeps: p' = 0 (src/Solver.cu:193)
            // No p' pass takes a decision left over from the momentum passes; nothing
            // depends on it any more but the counts.
            if (pending.kind && tid == 0) {
                pass_count(L, EQ_U, pending.n0, N);
                pass_count(L, EQ_V, pending.n1, N);
            }
#pragma unroll 1
            for (int t = blockIdx.x; t < ntiles; t += G) {
                const TileBox tl = tile_box(pa.tiles, t, nx, ny);
#pragma unroll 1
                for (int b = tl.oy0 + warp; b < tl.oy1; b += NW)
#pragma unroll 1
                    for (int a = tl.ox0 + lane; a < tl.ox1; a += 32) pcc[tl.gx0 + a + nx * (tl.gy0 + b)] = (T)0;
            }
            if (!grid_sync(bar, G, epoch)) break;
        }

        // -------- optional p' mean removal (closed domains, FP64) --------
        if (pa.pin) {
            double m = 0.0;
#pragma unroll 1
            for (int t = blockIdx.x; t < ntiles; t += G) {
                const TileBox tl = tile_box(pa.tiles, t, nx, ny);
#pragma unroll 1
                for (int b = tl.oy0 + warp; b < tl.oy1; b += NW)
#pragma unroll 1
                    for (int a = tl.ox0 + lane; a < tl.ox1; a += 32) m += (double)pcc[tl.gx0 + a + nx * (tl.gy0 + b)];
            }
            sred[tid] = m;
            __syncthreads();
            column_partials<NT>(sred, 1, partials + set * set_len, G, tot);
            if (!grid_sync(bar, G, epoch)) break;
            reduce_partials<NT>(partials + set * set_len, 1, G, tot);
            set ^= 1;
            const double mean = tot[0] / (double)N;
#pragma unroll 1
            for (int t = blockIdx.x; t < ntiles; t += G) {
                const TileBox tl = tile_box(pa.tiles, t, nx, ny);
#pragma unroll 1
                for (int b = tl.oy0 + warp; b < tl.oy1; b += NW)
#pragma unroll 1
                    for (int a = tl.ox0 + lane; a < tl.ox1; a += 32) {
                        const int c = tl.gx0 + a + nx * (tl.gy0 + b);
                        pcc[c] = (T)((double)pcc[c] - mean);
                    }
            }
            if (!grid_sync(bar, G, epoch)) break;
        }

        // ---- corrections + next iteration's boundary faces, kernels.cuh:583-843 ----
        {
            double s[7] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
            for (int t = blockIdx.x; t < ntiles; t += G) {
                const TileBox tl = tile_box(pa.tiles, t, nx, ny);
                const int ow = tl.ox1 - tl.ox0;
                const SmallDiv dow(ow);
#pragma unroll 1
                for (int q = tid; q < ow * (tl.oy1 - tl.oy0); q += NT) {
                    const int b = dow.div(q), a = q - b * ow;
                    const int i = tl.gx0 + tl.ox0 + a, j = tl.gy0 + tl.oy0 + b;
                    const int c = i + nx * j;
                    const int fu = i + (nx + 1) * j;
                    // loads first
                    const T pc = pcc[c], aC = f.ac[c];
                    const T pcW = i > 0 ? pcc[c - 1] : (T)0, pcE = i < nx - 1 ? pcc[c + 1] : (T)0;
                    const T pcS = j > 0 ? pcc[c - nx] : (T)0, pcN = j < ny - 1 ? pcc[c + nx] : (T)0;
                    const T rC = f.rac[c], rW = i > 0 ? f.rac[c - 1] : (T)1, rS = j > 0 ? f.rac[c - nx] : (T)1;
                    const T p0 = f.p[c], u0 = fc.u[c], v0 = fc.v[c];
                    const T uf0 = i > 0 ? f.uf[fu] : (T)0, vf0 = j > 0 ? f.vf[c] : (T)0;
                    const T dp = g.relax[EQ_P] * pc;
                    const T lo = i > 0 ? pcW : (g.closed[WEST] ? pc : (T)0);
                    const T hi = i < nx - 1 ? pcE : (g.closed[EAST] ? pc : (T)0);
                    const T du = vel_corr(P.d.ru[0], lo, hi, g.Ax, aC);
                    const T so = j > 0 ? pcS : (g.closed[SOUTH] ? pc : (T)0);
                    const T no = j < ny - 1 ? pcN : (g.closed[NORTH] ? pc : (T)0);
                    const T dv = vel_corr(P.d.ru[1], so, no, g.Ay, aC);
                    const T un = u0 + du, vn = v0 + dv;
                    f.p[c] = p0 + dp;
                    f.u[c] = un;
                    f.v[c] = vn;
                    if (pcc != f.pc) f.pc[c] = pc;  // keep the p' field current for readers
                    s[0] += (double)dp * (double)dp;
                    s[1] += (double)du * (double)du;
                    s[2] += (double)dv * (double)dv;
                    if (i >= 1) {
                        const T d = face_corr_known(P.d.ru[0], rW, rC, pcW, pc, g.Ax);
                        f.uf[fu] = uf0 + d;
                        s[4] += (double)d * (double)d;
                    }
                    if (j >= 1) {
                        const T d = face_corr_known(P.d.ru[1], rS, rC, pcS, pc, g.Ay);
                        f.vf[c] = vf0 + d;
                        s[5] += (double)d * (double)d;
                    }
                    if (i == 0) f.uf[fu] = face_bc(g, WEST, 0, un, j);
                    if (i == nx - 1) f.uf[fu + 1] = face_bc(g, EAST, 0, un, j);
                    if (j == 0) f.vf[c] = face_bc(g, SOUTH, 1, vn, 0);
                    if (j == ny - 1) f.vf[c + nx] = face_bc(g, NORTH, 1, vn, 0);
                }
            }
#pragma unroll
            for (int q = 0; q < 7; ++q) sred[q * NT + tid] = s[q];
            __syncthreads();
            column_partials<NT>(sred, 7, partials + set * set_len, G, tot);
            if (!grid_sync(bar, G, epoch)) break;
            pending.set(kPendNorms, set * set_len, 8, 0, 0);
            set ^= 1;
        }
        // (the last iteration of the call has nothing to overlap with)
        if (!one || L.it + 1 >= L.it_stop) resolve_now();
    }
    if (tid == 0) {
        const bool to = failed || bar->err != 0;
        if (to) atomicExch(&ctl->status, 3);
        if (blockIdx.x == 0) {
            for (int q = 0; q < 4; ++q) {
                ctl->stop[q] = 0;
                ctl->sweeps[q] = 0;
                ctl->inner_max[q] = -1e20;
            }
        }
    }
}

}  // namespace ifc
