// ifc_energy.cuh -- steady temperature transport on the converged flow.
//
// The reference allocates the temperature, carries its boundary conditions
// (TempBCs, include/config.h:45-63) and thermal properties
// (include/config.h:19-23) and writes it to VTK, but never solves for it.
// Here the steady energy equation
//     div(rho u T) = div(Gamma grad T),   Gamma = thermalConductivity / specificHeatCapacity
// (so Gamma / rho is the reference's thermalDiffusivity) is discretised on the
// converged face mass fluxes exactly as the momentum equations are: first-order
// upwind convection and central diffusion links (kernels.cuh:97-134 with Gamma
// in place of mu), and the boundary fold-in of kernels.cuh:252-334 -- the
// wall/inlet form for a Dirichlet face (type 0, the given temperature) and
// the zero-gradient form for a Neumann face (type 1).  The linear system is
// solved with the library's red-black Gauss-Seidel sweep kernel, unrelaxed.
// With a higher-order convection scheme (ifc_convection.cuh) the links stay
// upwind and the deferred correction of the current temperature is added to
// the source at the start of every cycle of sweeps (k_temp_dc).
#pragma once

#include "ifc_persist2d.cuh"

namespace ifc {

template <typename T>
struct TempArgs {
    T Dx, Dy, Dz;  // Gamma * A / d per direction, evaluated in the scalar type
    int type[6];   // 0 Dirichlet, 1 Neumann (zero gradient)
    T val[6];
};

template <typename T, int DIM>
__device__ __forceinline__ void temp_fold(const Params<T> &P, const TempArgs<T> &ta, int face, int ex, int in,
                                          T (&a)[7], T &b)
{
    const T e = a[ex];
    if (ta.type[face] != 0) {
        a[AC] = a[AC] + e;
        a[ex] = (T)0;
        return;
    }
    a[AC] = a[AC] - (T)2 * e;
    a[in] = a[in] + e / (T)3;
    b = b - P.d.c83 * e * ta.val[face];
    a[ex] = (T)0;
}

// Coefficient planes (2*DIM+1, coef[cell + N*slot]) and source of the energy
// equation of every cell.
template <typename T, int DIM>
__global__ void k_temp_assemble(Params<T> P, Fields<T> f, TempArgs<T> ta, T *coef, T *src)
{
    const Geo<T> &g = P.g;
    const int N = g.N, nx = g.nx, ny = g.ny, nz = g.nz, pl = nx * ny;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
        const int i = c % nx, j = (c / nx) % ny, k = c / pl;
        const int fu = i + (nx + 1) * (j + ny * k), fv = i + nx * (j + (ny + 1) * k);
        const T ue = f.uf[fu + 1], uw = f.uf[fu], vn = f.vf[fv + nx], vs = f.vf[fv];
        T a[7];
        a[AE] = g.rho * min0(ue) * g.Ax - ta.Dx;
        a[AW] = g.rho * min0(-uw) * g.Ax - ta.Dx;
        a[AN] = g.rho * min0(vn) * g.Ay - ta.Dy;
        a[AS] = g.rho * min0(-vs) * g.Ay - ta.Dy;
        a[AC] = -(a[AE] + a[AW] + a[AN] + a[AS]);
        a[AT] = (T)0;
        a[AB] = (T)0;
        if (DIM == 3) {
            const T wt = f.wf[c + pl], wb = f.wf[c];
            a[AT] = g.rho * min0(wt) * g.Az - ta.Dz;
            a[AB] = g.rho * min0(-wb) * g.Az - ta.Dz;
            a[AC] += -(a[AT] + a[AB]);
        }
        T b = (T)0;
        if (i == nx - 1) temp_fold<T, DIM>(P, ta, EAST, AE, AW, a, b);
        if (i == 0) temp_fold<T, DIM>(P, ta, WEST, AW, AE, a, b);
        if (j == ny - 1) temp_fold<T, DIM>(P, ta, NORTH, AN, AS, a, b);
        if (j == 0) temp_fold<T, DIM>(P, ta, SOUTH, AS, AN, a, b);
        if (DIM == 3) {
            if (k == nz - 1) temp_fold<T, DIM>(P, ta, TOP, AT, AB, a, b);
            if (k == 0) temp_fold<T, DIM>(P, ta, BOTTOM, AB, AT, a, b);
        }
#pragma unroll
        for (int s = 0; s < 2 * DIM + 1; ++s) coef[c + (size_t)N * s] = a[s];
        src[c] = b;
    }
}

// src_eff = src + the deferred-correction source of the current temperature
// (same face fluxes and limiter as the momentum equations).
template <typename T, int DIM>
__global__ void k_temp_dc(Params<T> P, Fields<T> f, const T *src, T *src_eff)
{
    const Geo<T> &g = P.g;
    const int nx = g.nx, ny = g.ny, pl = nx * ny;
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), nw = (int)((gridDim.x * blockDim.x) >> 5);
    const int units = row_units(nx, ny * g.nz);
    for (int u = gw; u < units; u += nw) {
        const RowUnit w = row_unit(u, nx, ny);
        const int c0 = nx * w.r, f0 = (nx + 1) * w.r, v0 = nx * (w.j + (ny + 1) * w.k);
        for (int i = w.i0 + lane; i < w.i1; i += 32) {
            const int c = c0 + i;
            const T wb = DIM == 3 ? f.wf[c] : (T)0, wt = DIM == 3 ? f.wf[c + pl] : (T)0;
            const T d = dc_cell<T, DIM>(g, f.temp, c, i, w.j, w.k, f.uf[f0 + i], f.uf[f0 + i + 1], f.vf[v0 + i],
                                        f.vf[v0 + i + nx], wb, wt);
            src_eff[c] = src[c] + d;
        }
    }
}

static __global__ void k_clear_stop(Ctl *ctl, int eq) { ctl->stop[eq] = 0; }

// ---- 2D: a cycle of sweeps on stored coefficients in one cooperative launch --
// One tile per CTA, all CTAs co-resident: the region's coefficients are read
// into registers once per cycle (ifc_tile2d.cuh), the passes of kCoefSweeps
// sweeps are separated by the bounded grid barrier of ifc_persist2d.cuh, and the
// per-sweep FP64 sums of a pass are reduced and the inner early-exit rule is
// applied (as finish_sweeps does) while the next pass already runs; a pass that
// the rule makes superfluous is not stored.  The result is left in x0.  Values
// equal those of the per-pass launches.  400 sweeps of the 512x128 channel's
// temperature: 749 us with unknowns in shared memory and a 52x36 region per
// 32x16 tile, 471 us this way.
constexpr int kCoefSweeps = 5;

struct CoefArgs {
    TileGrid tiles;
    int eq, nsweeps, stall_test;
};

template <typename T, int R_, int NW_>
__global__ void __launch_bounds__(32 * NW_, 1)
    k_coef_solve2d(const __grid_constant__ Params<T> P, const T *coef, const T *src, Ctl *ctl, double *partials,
                   GridBarrier *bar, const CoefArgs ca, T *x0, T *x1)
{
    using RT = RTile<T, R_, NW_>;
    constexpr int R = RT::R, NT = RT::NT, KS = kCoefSweeps;
    const Geo<T> &g = P.g;
    const int nx = g.nx, ny = g.ny, N = g.N, G = gridDim.x, eq = ca.eq;
    const int tid = threadIdx.x, warp = tid >> 5;
    double *sred = reinterpret_cast<double *>(tile_smem<T>() + RT::END);  // per-thread sums of each sweep
    __shared__ LoopState L;
    __shared__ double tot[KS];
    __shared__ double last_sq;

    const double floor = ctl->inner_max[eq];
    if (tid == 0) {
        L.stop[eq] = ctl->stop[eq];
        L.hit[eq] = 0;
        L.sweeps[eq] = 0;
        L.cell_updates[eq] = 0;
        L.inner_max_sq[eq] = -1.0;
        last_sq = ctl->last_sweep_sq[eq];
    }
    clear_guards<RT, T>();
    const LanePlace<RT> pl(tile_box(ca.tiles, blockIdx.x, nx, ny), ny);
    Links<RT, T> a;
    Cells<T, R> x;
    {
        Cells<T, R> b;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int i = pl.gi + k, j = pl.gj + r;
                if (i < nx && j < ny) {
                    const size_t id = (size_t)i + (size_t)nx * j, n = (size_t)N;
                    // no neighbour beyond the domain: its value counts as 0
                    const T e = coef[id + n * AE], w = coef[id + n * AW], no = coef[id + n * AN], so = coef[id + n * AS];
                    a.set(r, k, i < nx - 1 ? e : e * (T)0, i > 0 ? w : w * (T)0, j < ny - 1 ? no : no * (T)0,
                          j > 0 ? so : so * (T)0, coef[id]);
                    b.at(r, k) = src[id];
                } else {
                    a.set(r, k, (T)0, (T)0, (T)0, (T)0, kOutside<T>);
                    b.at(r, k) = kOutside<T>;
                }
            }
        put_cells<RT, T>(b, RT::SRC);
    }
    const bool force = set_reciprocals<RT, T>(a);
    __syncthreads();

    bool failed = false;
    unsigned int epoch = 0;
    auto buf = [&](int q) { return field_view(q ? x1 : x0, N); };
    int cur = 0, set = 0;
    Pending pending;
    pending.kind = kPendNone;
    auto take = [&]() {  // by warp 0, after a block barrier
        if (warp != 0) return;
        pass_done(L, eq, tot, pending.n0, N, g.tol[eq], false, true, floor);
        if (tid == 0) last_sq = tot[pending.n0 - 1];
    };
#pragma unroll 1
    for (int pass = 0; pass * KS < ca.nsweeps && !L.stop[eq]; ++pass) {
        // Failure-detection test (stall_test = 1): CTA 0 leaves without
        // arriving, so every other CTA's bounded wait at this pass's barrier
        // runs out and the launch ends with the timeout status.
        if (ca.stall_test && blockIdx.x == 0) { failed = true; break; }
        const int ns = clamp_sweeps(ca.nsweeps, pass, KS);
        load_cells<RT, T>(x, buf(cur), pl, nx, ny, pass > 0, kOutside<T>);
        if (pending.kind) pending_totals<RT::NW>(pending, partials, G, tot, tot);
        publish<RT, T>(x, 0);
        __syncthreads();
        if (pending.kind) take();
        sweeps1<RT, T>(x, a, pl, g.relax[eq], force, ns, KS, true, false, sred);
        if (pending.kind) {
            pending.kind = kPendNone;
            if (L.stop[eq]) break;  // this pass was superfluous
        }
        store_own<RT, T>(x, buf(cur ^ 1), pl, nx);
        column_partials<NT>(sred, ns, partials + set * KS * G, G, tot);
        cur ^= 1;
        if (!grid_sync(bar, G, epoch)) { failed = true; break; }
        pending.set(kPendP, set * KS * G, ns, ns, 0);
        set ^= 1;
    }
    if (pending.kind && !failed) {
        pending_totals<RT::NW>(pending, partials, G, tot, tot);
        __syncthreads();
        take();
    }
    __syncthreads();
    // the last stored pass read x0, and every CTA has passed its barrier
    if (!failed && cur == 1) store_other<RT, T>(buf(0), buf(1), pl, nx);
    if (blockIdx.x == 0 && tid == 0 && !failed) {
        const double top = L.inner_max_sq[eq] >= 0.0 ? sqrt(L.inner_max_sq[eq] / (double)N) : -1e20;
        ctl->inner_max[eq] = top > floor ? top : floor;
        ctl->sweeps[eq] += L.sweeps[eq];
        ctl->cell_updates += L.cell_updates[eq];
        ctl->last_sweep_sq[eq] = last_sq;
        if (L.stop[eq]) ctl->stop[eq] = 1;
    }
    if (tid == 0 && (failed || bar->err)) atomicExch(&ctl->status, 3);
}

// ---- 2D: KS red-black sweeps on stored coefficients in one pass ------------
// The temporally blocked pass of ifc_fused2d.cuh for a linear system whose
// coefficient planes (coef[cell + N*slot], slots aC aE aW aN aS) and source
// are stored: the tile plus a halo of 2*KS cells is staged from x_in, every
// thread keeps its cells' coefficients in registers, and the tile after KS
// sweeps goes to x_out (a different buffer, so no tile reads a neighbour's
// values of the same pass).  Per-sweep FP64 sums of the owned cells feed the
// inner early-exit rule of equation eq after the pass (finish_sweeps).  Used
// by the energy solve; the values equal those of per-sweep red-black launches.
template <typename T, int TX, int TY, int KS, int NT>
__global__ void __launch_bounds__(NT) k_coef_pass2d(Params<T> P, const T *coef, const T *src, Ctl *ctl,
                                                    double *partials, int eq, int ns, const T *x_in, T *x_out)
{
    constexpr int H = 2 * KS;
    using R = Region<TX, TY, H>;
    constexpr int W = R::W, NR = R::NR;
    constexpr int CPT = (R::NHALF + NT - 1) / NT;
    const Geo<T> &g = P.g;
    const bool active = ns > 0 && !ctl->stop[eq];  // same in every block

    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *sx = reinterpret_cast<T *>(smem_raw);

    const int nx = g.nx, ny = g.ny, N = g.N;
    const int tiles_x = (nx + TX - 1) / TX;
    const int x0 = (blockIdx.x % tiles_x) * TX, y0 = (blockIdx.x / tiles_x) * TY;
    const int gx0 = x0 - H, gy0 = y0 - H;
    const int tid = threadIdx.x;

    for (int q = tid; q < NR; q += NT) {
        const int a = q % W, b = q / W;
        const int gi = gx0 + a, gj = gy0 + b;
        const bool in = gi >= 0 && gi < nx && gj >= 0 && gj < ny;
        sx[q] = in ? x_in[gi + nx * gj] : (T)0;
    }
    int cq[2][CPT], dq[2][CPT];
    own_cells<W, R::HH, R::NHALF, NT, CPT>(tid, gx0, gy0, nx, ny, cq);
    T cE[2][CPT], cW[2][CPT], cN[2][CPT], cS[2][CPT], cC[2][CPT], cb[2][CPT];
    bool own[2][CPT];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int q = cq[c][k];
            dq[c][k] = tile_distance<W, H, TX, TY>(q);
            own[c][k] = false;
            cE[c][k] = cW[c][k] = cN[c][k] = cS[c][k] = cb[c][k] = (T)0;
            cC[c][k] = (T)1;
            if (q < 0) continue;
            const int a = q % W, b = q / W;
            const int id = gx0 + a + nx * (gy0 + b);
            cC[c][k] = coef[id + (size_t)N * AC];
            cE[c][k] = coef[id + (size_t)N * AE];
            cW[c][k] = coef[id + (size_t)N * AW];
            cN[c][k] = coef[id + (size_t)N * AN];
            cS[c][k] = coef[id + (size_t)N * AS];
            cb[c][k] = src[id];
            own[c][k] = a >= H && a < H + TX && b >= H && b < H + TY;
        }
    __syncthreads();

    double acc[KS];
#pragma unroll
    for (int s = 0; s < KS; ++s) acc[s] = 0.0;
    const T relax = g.relax[eq];
#pragma unroll
    for (int s = 0; s < KS; ++s) {
        if (!active || s >= ns) break;
#pragma unroll
        for (int color = 0; color < 2; ++color) {
            const int reach = 2 * ns - 1 - (2 * s + color);
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                const int q = cq[color][k];
                if (q < 0 || dq[color][k] > reach) continue;
                T a7[7] = {cC[color][k], cE[color][k], cW[color][k], cN[color][k], cS[color][k], (T)0, (T)0};
                T d;
                sx[q] = point_update<T, 2>(a7, cb[color][k], sx[q], sx[q + 1], sx[q - 1], sx[q + W], sx[q - W],
                                           (T)0, (T)0, relax, d);
                if (own[color][k]) acc[s] += (double)d * (double)d;
            }
            __syncthreads();
        }
    }
    for (int q = tid; q < TX * TY; q += NT) {
        const int a = H + q % TX, b = H + q / TX;
        const int gi = gx0 + a, gj = gy0 + b;
        if (gi >= nx || gj >= ny) continue;
        x_out[gi + nx * gj] = sx[b * W + a];
    }
    if (!active) return;  // uniform: the copy above keeps the output buffer current

    __shared__ double tot[KS];
    if (grid_reduce<KS>(acc, partials, ctl, tot) && tid == 0) finish_sweeps(ctl, eq, tot, ns, N, g.tol[eq]);
}

}  // namespace ifc
