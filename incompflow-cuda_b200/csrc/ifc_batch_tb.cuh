// ifc_batch_tb.cuh -- temporally blocked form of the batched kernel (included
// by ifc_batch.cu inside its anonymous namespace, after the case queue, loop
// state and cluster-reduction helpers).
//
// A cluster of CL CTAs solves one case at a time, as k_batch2d does, but the
// linear sweeps run as temporally blocked passes on regions held in registers,
// the same passes as the single-case solve (ifc_tile2d.cuh): the case is cut
// into tiles, the cluster's CTAs take the tiles in turn, each tile's region (the
// tile and a halo of 2*ks cells) is loaded, swept ks times (momentum: u and v
// together, coefficients rebuilt on the fly; p': links from 1/aC) and written
// back -- to the other buffer of a ping-pong pair, so no tile reads a
// neighbour tile's values of the same pass.  Cluster barriers separate the
// passes and phases; every norm is reduced per CTA in a fixed order and across
// the cluster through distributed shared memory in rank order, so each CTA
// takes the same early-exit and convergence decisions.  The region shape, the
// cluster size and the sweeps per pass distinguish the variants; a batch picks
// them by its cases.  Against whole-row sweeps (a cluster barrier per half sweep,
// every coefficient rebuilt from L1/L2 in every half sweep) a batch of 48
// cavities of 32..256 squared takes 51 ms instead of 92 for 60 iterations each; a
// batch of hundreds of them keeps all of the whole-row form's 71 clusters busy
// and stays with it (256 cavities, 40 iterations: 134 ms, 184 in variant 2).

template <typename T>
struct TBPools {
    T *tu, *tv, *tpc;  // ping-pong partners of u, v and p' (same offsets as the pools)
};

// This CTA's column sums of sred into part (zeros when it had no tile); block
// barriers before and after.
template <int NT>
__device__ __forceinline__ void tb_part(const double *sred, int ncol, bool any, double *part)
{
    __syncthreads();
    if (any) column_partials<NT>(sred, ncol, nullptr, 1, part);
    else if ((int)threadIdx.x < ncol) part[threadIdx.x] = 0.0;
    __syncthreads();
}

// After a cluster barrier: the cluster-wide sums of the n slots `part` of every
// CTA, added in rank order (identical in every CTA).
template <int CL>
__device__ __forceinline__ void tb_cluster_total(cg::cluster_group &cl, double *part, int n, double *out)
{
    if ((int)threadIdx.x < n) {
        double t = 0.0;
        for (int r = 0; r < CL; ++r) t += cl.map_shared_rank(part, r)[threadIdx.x];
        out[threadIdx.x] = t;
    }
    __syncthreads();
}

// After a pass of ns sweeps of equation e from sweep `first`, with per-sweep
// sums sq[0..ns): the early-exit rule (not a second time when the pass was run
// `again`).
__device__ __forceinline__ void tb_pass_done(CaseLoop &L, int e, const double *sq, int first, int ns, int n, int check,
                                             int N, double tol, bool again)
{
    if (ns == 0) return;
    for (int s = 0; s < ns && !L.hit[e] && !again; ++s) inner_rule(L, e, sq[s], first + s, n, check, N, tol);
    L.sweeps[e] = first + ns;
}

// Sweeps of a pass that starts at sweep `first` of an inner solve of `limit`.
__device__ __forceinline__ int tb_sweeps(int limit, int first, int ks) { return max(0, min(limit - first, ks)); }

// Rhie-Chow velocity of interior face k of n along its axis (stride st; c: the
// cell above the face), with the reciprocals of the diagonals.
template <typename T>
__device__ __forceinline__ T tb_face(const Geo<T> &g, const T *vel, const Fields<T> &f, T A, int k, int n, int st, int c,
                                     int low, int high)
{
    const int L = c - st;
    const T pL = f.p[L], pR = f.p[c];
    const T pLL = k >= 2 ? f.p[L - st] : (g.closed[low] ? pL : (T)0);
    const T pRR = k <= n - 2 ? f.p[c + st] : (g.closed[high] ? pR : (T)0);
    return rc_face_known(vel[L], vel[c], f.ac[L], f.ac[c], f.rac[L], f.rac[c], pLL, pL, pR, pRR, A);
}

// Splits a case's grid into tiles (the rule of split_axis).
__device__ __forceinline__ bool tb_tiles(int nx, int ny, int rows, int ks, TileGrid &G)
{
    G.H = 2 * ks;
    return split_axis(nx, 64, G.H, &G.kx, &G.Ix) && split_axis(ny, rows, G.H, &G.ky, &G.Iy);
}

template <typename T, int R_, int NW_, int CL, int KS>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(32 * NW_, 1)
    k_batch_tb(const BCase<T> *cases, BState *states, BPools<T> pool, TBPools<T> tp, int ncases, BQueue *q,
               int chunk, cudaGraphConditionalHandle cond, int use_cond)
{
    using RT = RTile<T, R_, NW_>;
    constexpr int R = RT::R, NT = RT::NT;
    constexpr int NP = 2 * KS + 8;  // partial-sum slots per set
    cg::cluster_group cl = cg::this_cluster();
    const unsigned rank = cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31;
    const int gw = (int)rank * (NT / 32) + (tid >> 5);  // warp index within the cluster
    constexpr int TW = CL * NT / 32;                    // warps per cluster

    double *sred = reinterpret_cast<double *>(tile_smem<T>() + RT::END);  // per-thread sums
    clear_guards<RT, T>();
    __shared__ int s_case;
    __shared__ BCase<T> C;
    __shared__ CaseLoop L;
    __shared__ BState S;
    // Two sets of this CTA's partial sums, used alternately: a set is rewritten
    // only after a later cluster barrier that every CTA reaches after reading it.
    __shared__ double part[2][NP];
    __shared__ double tot[NP];
    int rs = 0;

    for (;;) {
        if (rank == 0 && tid == 0) s_case = (int)atomicAdd(&q->next, 1u);
        cl.sync();
        const int cid = *cl.map_shared_rank(&s_case, 0);
        if (cid >= ncases) break;
        if (tid == 0) {
            C = cases[cid];
            S = states[cid];
        }
        cl.sync();
        if (S.done) continue;

        const Params<T> &P = C.P;
        const Geo<T> &g = P.g;
        const int nx = g.nx, ny = g.ny, N = g.N;
        TileGrid tg;
        tb_tiles(nx, ny, RT::HR, KS, tg);
        const int ntiles = tg.kx * tg.ky;
        T *u = pool.u + C.off_c, *v = pool.v + C.off_c, *p = pool.p + C.off_c, *pc = pool.pc + C.off_c;
        T *ac = pool.ac + C.off_c, *rac = pool.rac + C.off_c, *sp = pool.sp + C.off_c;
        T *uf = pool.uf + C.off_uf, *vf = pool.vf + C.off_vf;
        T *bu[2] = {u, tp.tu + C.off_c}, *bv[2] = {v, tp.tv + C.off_c}, *bp[2] = {pc, tp.tpc + C.off_c};
        Fields<T> f;
        memset(&f, 0, sizeof(f));
        f.p = p;
        f.uf = uf;
        f.vf = vf;
        f.ac = ac;
        f.rac = rac;
        f.sp = sp;
#ifdef IFC_BOUNDS_CHECK
        f.p.n = f.ac.n = f.rac.n = f.sp.n = N;
        f.uf.n = (long long)(nx + 1) * ny;
        f.vf.n = (long long)nx * (ny + 1);
#endif

        // First iteration of the case: interior faces from cell means, then
        // the face boundary conditions (kernels.cuh:10-95).
        if (S.it == 0) {
            for (int j = gw; j < ny + 1; j += TW)
                for (int i = lane; i < nx + 1; i += 32) {
                    if (j < ny) {
                        const int c = i + nx * j;
                        T val;
                        if (i == 0) val = face_bc(g, WEST, 0, u[c], j);
                        else if (i == nx) val = face_bc(g, EAST, 0, u[c - 1], j);
                        else val = (u[c - 1] + u[c]) / (T)2;
                        uf[i + (nx + 1) * j] = val;
                    }
                    if (i < nx) {
                        const int c = i + nx * j;
                        T val;
                        if (j == 0) val = face_bc(g, SOUTH, 1, v[c], 0);
                        else if (j == ny) val = face_bc(g, NORTH, 1, v[c - nx], 0);
                        else val = (v[c - nx] + v[c]) / (T)2;
                        vf[c] = val;
                    }
                }
            cl.sync();
        }

        for (int it = 0; it < chunk && !S.done; ++it) {
            if (tid == 0)
                for (int e = 0; e < 4; ++e) {
                    L.limit[e] = C.n_iter[e];
                    L.hit[e] = 0;
                    L.inner_max[e] = -1e20;
                    L.sweeps[e] = 0;
                }
            __syncthreads();
            int mcur = 0, pcur = 0;

            // ---------------- momentum passes ----------------
            // (When the early-exit rule ends an inner solve before its pass does -- the
            // case is checked more often than KS sweeps -- the pass is run
            // again, from the same values, with fewer sweeps.)
            bool again = false;
            for (int first = 0;;) {
                const int ns0 = tb_sweeps(L.limit[EQ_U], first, KS), ns1 = tb_sweeps(L.limit[EQ_V], first, KS);
                if (ns0 == 0 && ns1 == 0 && first > 0) break;  // the same in every CTA
#pragma unroll 1
                for (int t = (int)rank; t < ntiles; t += CL) {
                    const LanePlace<RT> pl(tile_box(tg, t, nx, ny), ny);
                    Links<RT, T> a;
                    Cells<T, R> cu, cv;
                    load_cells<RT, T>(cu, field_view(bu[mcur], N), pl, nx, ny, false, kOutside<T>);
                    load_cells<RT, T>(cv, field_view(bv[mcur], N), pl, nx, ny, false, kOutside<T>);
                    const bool force = mom_links<RT, T>(P, f, pl, a);
                    if (first == 0) store_diagonal<RT, T>(a, field_view(ac, N), field_view(rac, N), pl, nx);
                    publish<RT, T>(cu, 0);
                    publish<RT, T>(cv, 1);
                    __syncthreads();
                    sweeps2<RT, T>(cu, cv, a, pl, g.relax[EQ_U], g.relax[EQ_V], force, ns0, ns1, KS, true,
                                   t != (int)rank, sred);
                    store_own<RT, T>(cu, field_view(bu[mcur ^ 1], N), pl, nx);
                    store_own<RT, T>(cv, field_view(bv[mcur ^ 1], N), pl, nx);
                }
                tb_part<NT>(sred, 2 * KS, ntiles > (int)rank, part[rs]);
                cl.sync();
                tb_cluster_total<CL>(cl, part[rs], 2 * KS, tot);
                rs ^= 1;
                if (tid == 0) {
                    tb_pass_done(L, EQ_U, tot, first, ns0, C.n_iter[0], C.check, N, g.tol[EQ_U], again);
                    tb_pass_done(L, EQ_V, tot + KS, first, ns1, C.n_iter[1], C.check, N, g.tol[EQ_V], again);
                }
                __syncthreads();
                again = (ns0 > 0 && first + ns0 > L.limit[EQ_U]) || (ns1 > 0 && first + ns1 > L.limit[EQ_V]);
                if (again) continue;
                mcur ^= 1;
                first += KS;
            }
            const T *const cu = bu[mcur], *const cv = bv[mcur];

            // ---- Rhie-Chow faces, face BCs, p' source, 1/aC (kernels.cuh:336-581)
            double mass_sq;
            {
                double m[1] = {0.0};
                for (int j = gw; j < ny; j += TW)
                    for (int i = lane; i < nx; i += 32) {
                        const int c = i + nx * j;
                        const T uw = i == 0 ? face_bc(g, WEST, 0, cu[c], j) : tb_face(g, cu, f, g.Ax, i, nx, 1, i + nx * j, WEST, EAST);
                        const T ue = i == nx - 1 ? face_bc(g, EAST, 0, cu[c], j) : tb_face(g, cu, f, g.Ax, i + 1, nx, 1, i + 1 + nx * j, WEST, EAST);
                        const T vs = j == 0 ? face_bc(g, SOUTH, 1, cv[c], 0) : tb_face(g, cv, f, g.Ay, j, ny, nx, i + nx * j, SOUTH, NORTH);
                        const T vn = j == ny - 1 ? face_bc(g, NORTH, 1, cv[c], 0) : tb_face(g, cv, f, g.Ay, j + 1, ny, nx, i + nx * (j + 1), SOUTH, NORTH);
                        const T bb = mass_imbalance<T, 2>(g, uw, ue, vs, vn, (T)0, (T)0);
                        uf[i + (nx + 1) * j] = uw;
                        if (i == nx - 1) uf[nx + (nx + 1) * j] = ue;
                        vf[c] = vs;
                        if (j == ny - 1) vf[c + nx] = vn;
                        sp[c] = bb;
                        m[0] += (double)bb * (double)bb;
                    }
                #pragma unroll
                for (int c = 0; c < 1; ++c) sred[c * NT + tid] = m[c];
                tb_part<NT>(sred, 1, true, part[rs]);
                cl.sync();
                tb_cluster_total<CL>(cl, part[rs], 1, tot);
                rs ^= 1;
                mass_sq = tot[0];
            }

            // ---------------- p' passes from p' = 0 ----------------
            again = false;
            for (int first = 0;;) {
                const int ns = tb_sweeps(L.limit[EQ_P], first, KS);
                if (ns == 0) break;  // the same in every CTA
#pragma unroll 1
                for (int t = (int)rank; t < ntiles; t += CL) {
                    const LanePlace<RT> pl(tile_box(tg, t, nx, ny), ny);
                    Links<RT, T> a;
                    Cells<T, R> x;
                    if (first == 0) zero_cells<RT, T>(x, pl, nx, ny);
                    else load_cells<RT, T>(x, field_view(bp[pcur], N), pl, nx, ny, false, kOutside<T>);
                    const bool force = pc_links<RT, T>(P, f, pl, a);
                    publish<RT, T>(x, 0);
                    __syncthreads();
                    sweeps1<RT, T>(x, a, pl, g.relax[EQ_P], force, ns, KS, true, t != (int)rank, sred);
                    store_own<RT, T>(x, field_view(bp[pcur ^ 1], N), pl, nx);
                }
                tb_part<NT>(sred, KS, ntiles > (int)rank, part[rs]);
                cl.sync();
                tb_cluster_total<CL>(cl, part[rs], KS, tot);
                rs ^= 1;
                if (tid == 0) tb_pass_done(L, EQ_P, tot, first, ns, C.n_iter[3], C.check, N, g.tol[EQ_P], again);
                __syncthreads();
                again = first + ns > L.limit[EQ_P];
                if (again) continue;
                pcur ^= 1;
                first += KS;
            }
            T *const pcc = bp[pcur];
            if (C.n_iter[3] <= 0) {
                for (int j = gw; j < ny; j += TW)
                    for (int i = lane; i < nx; i += 32) pcc[i + nx * j] = (T)0;
                cl.sync();
            }

            // ---- FP64 removal of the p' mean (closed cavities)
            if (C.pin) {
                double m[1] = {0.0};
                for (int j = gw; j < ny; j += TW)
                    for (int i = lane; i < nx; i += 32) m[0] += (double)pcc[i + nx * j];
                #pragma unroll
                for (int c = 0; c < 1; ++c) sred[c * NT + tid] = m[c];
                tb_part<NT>(sred, 1, true, part[rs]);
                cl.sync();
                tb_cluster_total<CL>(cl, part[rs], 1, tot);
                rs ^= 1;
                const double mean = tot[0] / (double)N;
                for (int j = gw; j < ny; j += TW)
                    for (int i = lane; i < nx; i += 32) pcc[i + nx * j] = (T)((double)pcc[i + nx * j] - mean);
                cl.sync();
            }

            // ---- corrections + next iteration's boundary faces (kernels.cuh:583-843)
            {
                double sq[5] = {0, 0, 0, 0, 0};
                for (int j = gw; j < ny; j += TW)
                    for (int i = lane; i < nx; i += 32) {
                        const int c = i + nx * j, fu = i + (nx + 1) * j;
                        const T x = pcc[c], aC = ac[c];
                        const T xW = i > 0 ? pcc[c - 1] : (T)0, xE = i < nx - 1 ? pcc[c + 1] : (T)0;
                        const T xS = j > 0 ? pcc[c - nx] : (T)0, xN = j < ny - 1 ? pcc[c + nx] : (T)0;
                        const T rC = rac[c], rW = i > 0 ? rac[c - 1] : (T)1, rS = j > 0 ? rac[c - nx] : (T)1;
                        const T p0 = p[c], u0 = cu[c], v0 = cv[c];
                        const T uf0 = i > 0 ? uf[fu] : (T)0, vf0 = j > 0 ? vf[c] : (T)0;
                        const T dp = g.relax[EQ_P] * x;
                        const T Lx = i > 0 ? xW : (g.closed[WEST] ? x : (T)0);
                        const T Rx = i < nx - 1 ? xE : (g.closed[EAST] ? x : (T)0);
                        const T dU = vel_corr(P.d.ru[0], Lx, Rx, g.Ax, aC);
                        const T Sy = j > 0 ? xS : (g.closed[SOUTH] ? x : (T)0);
                        const T Ny = j < ny - 1 ? xN : (g.closed[NORTH] ? x : (T)0);
                        const T dV = vel_corr(P.d.ru[1], Sy, Ny, g.Ay, aC);
                        const T un = u0 + dU, vn = v0 + dV;
                        p[c] = p0 + dp;
                        u[c] = un;
                        v[c] = vn;
                        sq[0] += (double)dp * (double)dp;
                        sq[1] += (double)dU * (double)dU;
                        sq[2] += (double)dV * (double)dV;
                        if (i >= 1) {
                            const T d = face_corr_known(P.d.ru[0], rW, rC, xW, x, g.Ax);
                            uf[fu] = uf0 + d;
                            sq[3] += (double)d * (double)d;
                        }
                        if (j >= 1) {
                            const T d = face_corr_known(P.d.ru[1], rS, rC, xS, x, g.Ay);
                            vf[c] = vf0 + d;
                            sq[4] += (double)d * (double)d;
                        }
                        if (i == 0) uf[fu] = face_bc(g, WEST, 0, un, j);
                        if (i == nx - 1) uf[fu + 1] = face_bc(g, EAST, 0, un, j);
                        if (j == 0) vf[c] = face_bc(g, SOUTH, 1, vn, 0);
                        if (j == ny - 1) vf[c + nx] = face_bc(g, NORTH, 1, vn, 0);
                    }
                #pragma unroll
                for (int c = 0; c < 5; ++c) sred[c * NT + tid] = sq[c];
                tb_part<NT>(sred, 5, true, part[rs]);
                cl.sync();
                tb_cluster_total<CL>(cl, part[rs], 5, tot);
                rs ^= 1;
            }

            // ---- norms and convergence test (src/Solver.cu:226-268)
            if (tid == 0) {
                double n[8];
                n[0] = sqrt(tot[0] / (double)N);
                n[1] = sqrt(tot[1] / (double)N);
                n[2] = sqrt(tot[2] / (double)N);
                n[3] = 0.0;
                n[4] = sqrt(tot[3] / ((double)(nx - 1) * ny));
                n[5] = sqrt(tot[4] / ((double)nx * (ny - 1)));
                n[6] = 0.0;
                n[7] = sqrt(mass_sq / (double)N);
                bool bad = false;
                for (int e = 0; e < 8; ++e) bad = bad || !isfinite(n[e]);
                double rel[7];
                if (g.criterion == 0) {
                    if (n[0] > S.maxn[0]) S.maxn[0] = n[0];
                    for (int e = 0; e < 7; ++e) rel[e] = n[e] / S.maxn[0];
                } else {
                    for (int e = 0; e < 7; ++e) {
                        if (e == 3 || e == 6) { rel[e] = 0.0; continue; }
                        if (n[e] > S.maxn[e]) S.maxn[e] = n[e];
                        rel[e] = S.maxn[e] > 0.0 ? n[e] / S.maxn[e] : 0.0;
                    }
                }
                bool conv = rel[0] < g.tol[EQ_P] && rel[1] < g.tol[EQ_U] && rel[2] < g.tol[EQ_V] &&
                            rel[4] < g.tol[EQ_U] && rel[5] < g.tol[EQ_V];
                conv = conv || n[7] < g.tol_mass;
                S.it += 1;
                S.converged = conv ? 1 : 0;
                if (bad) S.status = 2;
                S.done = conv || bad || S.it >= C.max_outer;
                for (int e = 0; e < 8; ++e) S.norm[e] = n[e];
                for (int e = 0; e < 7; ++e) S.rel[e] = rel[e];
                for (int e = 0; e < 4; ++e) S.sweeps[e] = L.sweeps[e];
            }
            __syncthreads();
        }
        if (rank == 0 && tid == 0) states[cid] = S;
        cl.sync();
    }
    cl.sync();
    if (tid == 0) {
        __threadfence();
        const unsigned int t = atomicAdd(&q->exited, 1u);
        if (t == gridDim.x - 1) {
            __threadfence();
            int left = 0;
            for (int c = 0; c < ncases; ++c) left |= !((volatile BState *)states)[c].done;
            q->next = 0;
            q->exited = 0;
            __threadfence();
            if (use_cond) cudaGraphSetConditional(cond, left ? 1u : 0u);
        }
    }
}
