// ifc_coop3d.cuh -- a 3D linear solve (the p' equation, or a system with
// stored coefficients such as the temperature) as one cooperative launch,
// with the unknown resident in shared memory and the links and source of
// every cell packed once per solve in sweep order.
//
// Work split: each CTA owns a rectangular block of x-rows (all i, j in
// [j0, j0+bj), k in [k0, k0+bk)) for the whole solve (PcBlocks, chosen on the
// host so that one CTA per SM holds its block).  Set-up: every cell of the
// block gets its six links -- for p' from 1/aC (kernels.cuh:518-537, FP64
// products as in k_pc_half3d), otherwise from the stored planes -- its
// diagonal and its source, written to a packed array in the order the sweeps
// consume them: per (row, colour) the cells of that colour, one 16-byte
// vector of four values per plane and cell slot.  A half sweep then reads
// each updated cell's coefficients with two coalesced 128-bit loads and its
// neighbours from shared memory (or, in the rows of a neighbouring block,
// from global memory, to which a CTA writes the cells of its edge rows as it
// updates them); a bounded grid barrier separates the half sweeps.  Rows
// inside the block take a path with every neighbour in shared memory.  The
// per-sweep FP64 sums are reduced by every CTA in one fixed order, so every
// CTA takes the same inner early-exit decision (src/Solver.cu:955-962).  The
// arithmetic of each update is that of point_update on the same
// coefficients, so the results equal the per-half-sweep kernels and the CPU
// oracle bit for bit.  Only the unknown takes shared memory (the source
// travels with the links), so FP64 grids of the size FP32 ones run at fit
// as well; each row keeps its even-i cells, then its odd-i cells, so the
// cells a warp updates and all their neighbours are consecutive words (no
// bank conflicts; FP64 solves 6 % faster, FP32 unchanged).
#pragma once

#include "ifc_fused3d.cuh"
#include "ifc_tile2d.cuh"

namespace ifc {

// Packed slots: per CTA rows_cap rows x 2 colours x hx cells, hx = (nx+1)/2;
// the cell (i, row r, colour c) sits in slot (2r + c) * hx + (i >> 1) of its
// CTA's range.  Two planes of 4 values per slot follow each other, each
// spanning all CTAs' slots.
__host__ __device__ inline long long coop3d_slots(const PcBlocks &B, int nx)
{
    return (long long)B.nbj * B.nbk * B.bj * B.bk * 2 * ((nx + 1) / 2);
}

// Shared memory: the row table (int4 per row), then the unknown of every
// cell of the block.
template <typename T>
__host__ __device__ inline size_t coop3d_smem_bytes(int rows, int nx)
{
    return (size_t)rows * 16 + (size_t)rows * 2 * ((nx + 1) / 2) * sizeof(T);
}

// The linear system a cooperative solve works on: the p' equation (coef null:
// links from 1/aC, start from p' = 0 without clearing the array, as the
// per-half-sweep kernel does) or a system with stored coefficient planes
// coef[cell + N*slot] (slots aC aE aW aN aS aT aB), e.g. the temperature.
// Unknown x, source src, equation slot eq of the control block (relaxation,
// tolerance, sweep bookkeeping).
template <typename T>
struct CSys {
    const T *coef;
    const T *src;
    T *x;
    int eq;
};

template <typename T, int NT>
__global__ void __launch_bounds__(NT, 1) k_csolve3d(Params<T> P, Fields<T> f, Ctl *ctl, double *partials,
                                                    GridBarrier *bar, PcBlocks B, int n_sweeps, T *pk, CSys<T> sys,
                                                    int stall_test)
{
    const Geo<T> &g = P.g;
    const int nx = g.nx, ny = g.ny, nz = g.nz, pl = nx * ny, N = g.N;
    const int G = gridDim.x, tid = threadIdx.x;
    const int j0 = (blockIdx.x % B.nbj) * B.bj, k0 = (blockIdx.x / B.nbj) * B.bk;
    const int nj = min(B.bj, ny - j0), nk = min(B.bk, nz - k0);
    const int rows_cap = B.bj * B.bk;
    const int nrow = nj * nk;
    const int warp = tid >> 5, lane = tid & 31;
    // shared layout: each local row holds its even-i cells, then its odd-i
    // cells (hx each), so a warp's cells of one colour and their neighbours
    // are consecutive words
    const int hx2 = 2 * ((nx + 1) / 2);
    const int ln = hx2, lt = hx2 * nj;  // local strides to the next row in j and in k
    const int hx = (nx + 1) / 2;
    const long long S = coop3d_slots(B, nx);
    const long long cbase = (long long)blockIdx.x * rows_cap * 2 * hx;
    T *pA = pk, *pB = pk + 4 * S;  // {aC, aE, aW, aN}, {aS, aT, aB, b}
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int4 *s_row = reinterpret_cast<int4 *>(smem_raw);
    T *s_x = reinterpret_cast<T *>(s_row + rows_cap);
    __shared__ double red[NT / 32];
    __shared__ double tot2[2];
    const int eq = sys.eq;
    const bool zero_start = sys.coef == nullptr;
    T *x = sys.x;

    // row table: x = global offset of the row, y = j, z = k, w = flags (1: row
    // j+1 in this block, 2: j-1, 4: k+1, 8: k-1)
    for (int r = tid; r < nrow; r += NT) {
        const int jj = r % nj, kk = r / nj;
        const int j = j0 + jj, k = k0 + kk;
        const int fl = (jj + 1 < nj ? 1 : 0) | (jj > 0 ? 2 : 0) | (kk + 1 < nk ? 4 : 0) | (kk > 0 ? 8 : 0);
        s_row[r] = make_int4(nx * (j + ny * k), j, k, fl);
    }
    __syncthreads();
    // packed links and sources of the CTA's cells, the unknown into shared memory
    for (int r = warp; r < nrow; r += NT / 32) {
        const int4 ri = s_row[r];
        const int j = ri.y, k = ri.z, crow = ri.x, lrow = hx2 * r;
        for (int i = lane; i < nx; i += 32) {
            const int c = crow + i;
            T a[7];
            if (zero_start) {
                const T rr = f.rac[c];
                a[AE] = i < nx - 1 ? (T)(P.d.Kx * (double)(T)(rr + f.rac[c + 1])) : (T)0;
                a[AW] = i > 0 ? (T)(P.d.Kx * (double)(T)(rr + f.rac[c - 1])) : (T)0;
                a[AN] = j < ny - 1 ? (T)(P.d.Ky * (double)(T)(rr + f.rac[c + nx])) : (T)0;
                a[AS] = j > 0 ? (T)(P.d.Ky * (double)(T)(rr + f.rac[c - nx])) : (T)0;
                a[AT] = k < nz - 1 ? (T)(P.d.Kz * (double)(T)(rr + f.rac[c + pl])) : (T)0;
                a[AB] = k > 0 ? (T)(P.d.Kz * (double)(T)(rr + f.rac[c - pl])) : (T)0;
                a[AC] = -(a[AE] + a[AW] + a[AN] + a[AS]);
                a[AC] += -(a[AT] + a[AB]);
            } else {
#pragma unroll
                for (int q = 0; q < 7; ++q) a[q] = sys.coef[c + (size_t)N * q];
            }
            const long long slot = cbase + (long long)(2 * r + ((i + j + k) & 1)) * hx + (i >> 1);
            st4(pA + 4 * slot, a[AC], a[AE], a[AW], a[AN]);
            st4(pB + 4 * slot, a[AS], a[AT], a[AB], sys.src[c]);
            s_x[lrow + (i & 1) * (hx2 >> 1) + (i >> 1)] = zero_start ? (T)0 : x[c];
        }
    }
    double mx = ctl->inner_max[eq];
    int sw = ctl->sweeps[eq];
    bool stop = ctl->stop[eq] != 0;
    double last_sq = 0.0;
    unsigned int epoch = 0;
    __syncthreads();  // the packed values are read back by the same CTA only

    // Failure-detection test (IFC_TEST_STALL_BARRIER=1): CTA 0 leaves before
    // its first grid barrier, so every other CTA's bounded wait runs out and
    // the launch ends with the timeout status.
    bool failed = stall_test && blockIdx.x == 0;
    for (int s = 0; s < n_sweeps && !stop && !failed; ++s) {
        for (int color = 0; color < 2; ++color) {
            const int zero_mode = (zero_start && s == 0) ? (color == 0 ? 1 : 2) : 0;
            const bool zn = zero_mode == 1;
            double sq = 0.0;
            for (int r = warp; r < nrow; r += NT / 32) {
                const int4 ri = s_row[r];
                const int j = ri.y, k = ri.z;
                const int lrow = hx2 * r, crow = ri.x;
                const bool inN = ri.w & 1, inS = ri.w & 2, inT = ri.w & 4, inB = ri.w & 8;
                const int off = (color + j + k) & 1;
                const long long sbase = cbase + (long long)(2 * r + color) * hx;
                // a row on the block's edge: its cells also go to global
                // memory at once, for the neighbouring blocks' next half sweep
                const bool edge_row = (ri.w & 15) != 15;
                if (!edge_row && !zero_mode) {
                    // all four off-row neighbours are rows of this block
                    for (int i = off + 2 * lane; i < nx; i += 64) {
                        const int l = lrow + off * (hx2 >> 1) + (i >> 1);
                        const int le = lrow + (1 - off) * (hx2 >> 1) + (i >> 1);  // i+1 is le + off, i-1 is le + off - 1
                        const long long slot = sbase + (i >> 1);
                        T q0[4], q1[4];
                        ld4(pA + 4 * slot, q0);
                        ld4(pB + 4 * slot, q1);
                        const T a[7] = {q0[0], q0[1], q0[2], q0[3], q1[0], q1[1], q1[2]};
                        const T pE = i != nx - 1 ? s_x[le + off] : (T)0;
                        const T pW = i != 0 ? s_x[le + off - 1] : (T)0;
                        T d;
                        s_x[l] = point_update<T, 3>(a, q1[3], s_x[l], pE, pW, s_x[l + ln], s_x[l - ln], s_x[l + lt],
                                                    s_x[l - lt], g.relax[eq], d);
                        sq += (double)d * (double)d;
                    }
                    continue;
                }
                for (int i = off + 2 * lane; i < nx; i += 64) {
                    const int l = lrow + off * (hx2 >> 1) + (i >> 1), c = crow + i;
                    const int le = lrow + (1 - off) * (hx2 >> 1) + (i >> 1);
                    const long long slot = sbase + (i >> 1);
                    T q0[4], q1[4];
                    ld4(pA + 4 * slot, q0);
                    ld4(pB + 4 * slot, q1);
                    const T a[7] = {q0[0], q0[1], q0[2], q0[3], q1[0], q1[1], q1[2]};
                    const T pE = (!zn && i != nx - 1) ? s_x[le + off] : (T)0;
                    const T pW = (!zn && i != 0) ? s_x[le + off - 1] : (T)0;
                    const T pN = (!zn && j != ny - 1) ? (inN ? s_x[l + ln] : __ldcg(&x[c + nx])) : (T)0;
                    const T pS = (!zn && j != 0) ? (inS ? s_x[l - ln] : __ldcg(&x[c - nx])) : (T)0;
                    const T pT = (!zn && k != nz - 1) ? (inT ? s_x[l + lt] : __ldcg(&x[c + pl])) : (T)0;
                    const T pB_ = (!zn && k != 0) ? (inB ? s_x[l - lt] : __ldcg(&x[c - pl])) : (T)0;
                    const T pc = zero_mode ? (T)0 : s_x[l];
                    T d;
                    const T v = point_update<T, 3>(a, q1[3], pc, pE, pW, pN, pS, pT, pB_, g.relax[eq], d);
                    s_x[l] = v;
                    if (edge_row) x[c] = v;
                    sq += (double)d * (double)d;
                }
            }
            sq = warp_sum(sq);
            if (lane == 0) red[warp] = sq;
            __syncthreads();
            if (tid == 0) {
                double t = 0.0;
                for (int w = 0; w < NT / 32; ++w) t += red[w];
                partials[(size_t)(2 * (s & 1) + color) * G + blockIdx.x] = t;
            }
            if (!grid_sync<false>(bar, G, epoch)) {
                failed = true;
                break;
            }
        }
        if (failed) break;
        // grid sums of both halves, fixed order, identical in every CTA
        if (tid < 64) {
            const int color = tid >> 5;
            double t = 0.0;
            for (int b = lane; b < G; b += 32) t += __ldcg(&partials[(size_t)(2 * (s & 1) + color) * G + b]);
            t = warp_sum(t);
            if (lane == 0) tot2[color] = t;
        }
        __syncthreads();
        const double ssq = tot2[0] + tot2[1];
        const double rms = sqrt(ssq / (double)N);
        if (rms > mx) mx = rms;
        if (rms / (mx + 1e-20) < g.tol[eq]) stop = true;
        ++sw;
        last_sq = ssq;
        __syncthreads();  // tot2 is rewritten only after the next sweep's barriers
    }
    for (int r = warp; r < nrow; r += NT / 32) {
        const int crow = s_row[r].x, lrow = hx2 * r;
        for (int i = lane; i < nx; i += 32) x[crow + i] = s_x[lrow + (i & 1) * (hx2 >> 1) + (i >> 1)];
    }
    if (blockIdx.x == 0 && tid == 0 && !failed) {
        const int done = sw - ctl->sweeps[eq];
        ctl->cell_updates += (long long)done * N;
        ctl->inner_max[eq] = mx;
        ctl->sweeps[eq] = sw;
        if (done > 0) ctl->last_sweep_sq[eq] = last_sq;
        if (stop) ctl->stop[eq] = 1;
    }
    if (tid == 0 && (failed || bar->err)) atomicExch(&ctl->status, 3);
}

// ---- the p' equation with its links across rows in shared memory -----------
//
// k_csolve3d streams 32 bytes per update (six links, diagonal, source) from L2
// and divides in every update.  The p' links are symmetric -- the link east of a
// cell is the link west of its neighbour -- so where there is room for them,
// this kernel keeps the links between rows (north and top, one value per face)
// in shared memory beside p', sums the diagonal from the links, and streams only
// the links along x, the source and 1/aC (16 bytes per update; the quotient is
// the corrected product of ifc_tile2d.cuh).  A lane updates two cells of a
// colour at a time, 2 columns apart in x and adjacent in memory, so each load,
// address and branch serves two updates.  It is bound by the instructions around
// the updates (235 per 64 updates, 90 of them the arithmetic; issue slots 52 %
// busy) and by the two grid barriers of a sweep; 24 warps of 72 registers, since
// with 64 the index arithmetic is recomputed for every row (317 instructions).
// p' solve of 50 sweeps: 128^3 FP32 849 -> 740 us, 97x89x101 FP64 991 -> 697 us.
// A record of 32 (FP64: 64) adjacent bytes per pair, flat pointers chosen per
// row instead of branches in the edge rows (780 us) and 16 warps (758 us) are
// slower.
//
// Layout: rows are colour-split as above, each half padded to an even number of
// cells (hp) whose pads stay zero.  The rows on a block's edge are written to
// `exch` in the same layout for the neighbouring blocks.

template <typename T>
__host__ __device__ inline int psolve3d_half(int nx)
{
    return 2 * (((nx + 1) / 2 + 1) / 2);
}

// Shared memory: the row table, p', the north faces (one row more per k) and the
// top faces (one layer more).
template <typename T>
__host__ __device__ inline size_t psolve3d_smem_bytes(const PcBlocks &B, int nx)
{
    const size_t rows = (size_t)B.bj * B.bk, faces = rows + B.bk + rows + B.bj;
    return rows * 16 + (rows + faces) * 2 * psolve3d_half<T>(nx) * sizeof(T);
}

template <typename T> struct Vec2;
template <> struct Vec2<float> { using V = float2; };
template <> struct Vec2<double> { using V = double2; };

// Diagonal of the p' equation from its links, in the order of k_csolve3d.
template <typename T>
__device__ __forceinline__ T p3_diagonal(T e, T w, T n, T s, T t, T b)
{
    T c = -(e + w + n + s);
    c += -(t + b);
    return c;
}

__device__ __forceinline__ Pair<float> pair(float2 v) { return Pair<float>(v); }
__device__ __forceinline__ Pair<double> pair(double2 v) { return Pair<double>(v.x, v.y); }
template <typename V>
__device__ __forceinline__ auto minus_products(V a, V x) -> decltype(pair(a))
{
    return {-a.x * x.x, -a.y * x.y};
}

// The streamed record of a cell slot m (aE, aW, source, 1/aC).  16-byte vectors
// whose lanes are adjacent: in FP32 two planes that hold two quantities of a
// pair each, in FP64 a plane per quantity (FP64 records of 64 adjacent bytes
// took 768 us where the planes take 682 us, 97x89x101).
__device__ __forceinline__ void store_record(float *rec, size_t slots, int m, float e, float w, float b, float z)
{
    float *q = rec + 4 * (m >> 1) + (m & 1);
    q[0] = e;
    q[2] = w;
    q[2 * slots] = b;
    q[2 * slots + 2] = z;
}
__device__ __forceinline__ void store_record(double *rec, size_t slots, int m, double e, double w, double b, double z)
{
    double *q = rec + m;
    q[0] = e;
    q[slots] = w;
    q[2 * slots] = b;
    q[3 * slots] = z;
}
__device__ __forceinline__ void load_record(const float *rec, size_t slots, int m, float2 &e, float2 &w, float2 &b, float2 &z)
{
    const float4 p = __ldcg(reinterpret_cast<const float4 *>(rec + 2 * m));
    const float4 q = __ldcg(reinterpret_cast<const float4 *>(rec + 2 * slots + 2 * m));
    e = make_float2(p.x, p.y);
    w = make_float2(p.z, p.w);
    b = make_float2(q.x, q.y);
    z = make_float2(q.z, q.w);
}
__device__ __forceinline__ void load_record(const double *rec, size_t slots, int m, double2 &e, double2 &w, double2 &b,
                                            double2 &z)
{
    const double *q = rec + m;
    e = __ldcg(reinterpret_cast<const double2 *>(q));
    w = __ldcg(reinterpret_cast<const double2 *>(q + slots));
    b = __ldcg(reinterpret_cast<const double2 *>(q + 2 * slots));
    z = __ldcg(reinterpret_cast<const double2 *>(q + 3 * slots));
}

template <typename T, int NT>
__global__ void __launch_bounds__(NT, 1) k_psolve3d(const __grid_constant__ Params<T> P, const __grid_constant__ Fields<T> f,
                                                    Ctl *ctl, double *partials, GridBarrier *bar, const PcBlocks B,
                                                    int n_sweeps, T *pk, int stall_test)
{
    using V = typename Vec2<T>::V;
    const Geo<T> &g = P.g;
    const int nx = g.nx, ny = g.ny, nz = g.nz, pl = nx * ny, N = g.N;
    const int G = gridDim.x, tid = threadIdx.x;
    const int j0 = (blockIdx.x % B.nbj) * B.bj, k0 = (blockIdx.x / B.nbj) * B.bk;
    const int nj = min(B.bj, ny - j0), nk = min(B.bk, nz - k0);
    const int rows_cap = B.bj * B.bk, nrow = nj * nk;
    const int warp = tid >> 5, lane = tid & 31;
    const int hp = psolve3d_half<T>(nx), rl = 2 * hp, lrl = nj * rl;  // half row, row, layer
    // streamed records of this CTA and the exchanged rows (by global row)
    const size_t slots = (size_t)G * rows_cap * rl;
    T *const rec = pk + (size_t)blockIdx.x * rows_cap * rl * (sizeof(T) == 4 ? 2 : 1);
    T *const exch = pk + 4 * slots;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int4 *s_row = reinterpret_cast<int4 *>(smem_raw);
    T *const s_x = reinterpret_cast<T *>(s_row + rows_cap);
    T *const s_n = s_x + rows_cap * rl;            // row kk*(nj+1) + jj+1 holds the faces north of (jj, kk)
    T *const s_t = s_n + (rows_cap + B.bk) * rl;   // row (kk+1)*nj + jj the faces on top of it
    __shared__ double red[NT / 32];
    __shared__ double tot1;
    __shared__ int s_edges;

    // row table: x = the row in s_x, y = its south faces in s_n, z = the row in
    // exch, w = flags (1 north, 2 south, 4 top, 8 bottom row in this block; 16,
    // 32, 64, 128: in another block; 256: j + k odd).  The rows that other
    // blocks read come first.
    if (warp == 0) {
        const bool hasS = j0 > 0, hasN = j0 + nj < ny, hasB = k0 > 0, hasT = k0 + nk < nz;
        const unsigned lower = (1u << lane) - 1u;
        auto is_edge = [&](int r) {
            const int jj = r % nj, kk = r / nj;
            return r < nrow && ((hasS && jj == 0) || (hasN && jj == nj - 1) || (hasB && kk == 0) || (hasT && kk == nk - 1));
        };
        int pe = 0, pi = 0;  // next place of an edge row and of an inner one
        for (int r = lane; r - lane < nrow; r += 32) pi += __popc(__ballot_sync(0xffffffffu, is_edge(r)));
        if (lane == 0) s_edges = pi;
        for (int r = lane; r - lane < nrow; r += 32) {
            const bool edge = is_edge(r);
            const unsigned me = __ballot_sync(0xffffffffu, edge), mi = __ballot_sync(0xffffffffu, !edge);
            const int jj = r % nj, kk = r / nj, j = j0 + jj, k = k0 + kk;
            const int fl = (jj + 1 < nj ? 1 : j + 1 < ny ? 16 : 0) | (jj > 0 ? 2 : j > 0 ? 32 : 0) |
                           (kk + 1 < nk ? 4 : k + 1 < nz ? 64 : 0) | (kk > 0 ? 8 : k > 0 ? 128 : 0) | ((j + k) & 1) << 8;
            if (r < nrow)
                s_row[edge ? pe + __popc(me & lower) : pi + __popc(mi & lower)] =
                    make_int4(r * rl, (kk * (nj + 1) + jj) * rl, (j + ny * k) * rl, fl);
            pe += __popc(me);
            pi += __popc(mi);
        }
    }
    __syncthreads();
    const int nedge = s_edges;
    for (int r = warp; r < (nj + 1) * nk; r += NT / 32) {
        const int j = j0 + r % (nj + 1), k = k0 + r / (nj + 1);  // the face below (j, k)
        for (int i = lane; i < rl; i += 32) {
            T a = (T)0;
            if (i < nx && j > 0 && j < ny) {
                const int c = i + nx * (j + ny * k);
                a = (T)(P.d.Ky * (double)(T)(f.rac[c] + f.rac[c - nx]));
            }
            s_n[r * rl + (i & 1) * hp + (i >> 1)] = a;
        }
    }
    for (int r = warp; r < nj * (nk + 1); r += NT / 32) {
        const int j = j0 + r % nj, k = k0 + r / nj;
        for (int i = lane; i < rl; i += 32) {
            T a = (T)0;
            if (i < nx && k > 0 && k < nz) {
                const int c = i + nx * (j + ny * k);
                a = (T)(P.d.Kz * (double)(T)(f.rac[c] + f.rac[c - pl]));
            }
            s_t[r * rl + (i & 1) * hp + (i >> 1)] = a;
        }
    }
    __syncthreads();
    for (int r = warp; r < nrow; r += NT / 32) {
        const int4 ri = s_row[r];
        const int crow = ri.z / rl * nx;
        for (int i = lane; i < rl; i += 32) {
            const int m = i >> 1, ps = (i & 1) * hp + m;
            s_x[ri.x + ps] = (T)0;
            T e = (T)1, w = (T)0, b = (T)1;  // the pad: an ordinary quotient, never stored
            if (i < nx) {
                const int c = crow + i;
                const T rr = f.rac[c];
                e = i < nx - 1 ? (T)(P.d.Kx * (double)(T)(rr + f.rac[c + 1])) : (T)0;
                if (i > 0) w = (T)(P.d.Kx * (double)(T)(rr + f.rac[c - 1]));
                b = f.sp[c];
            }
            const T y = p3_diagonal(e, w, s_n[ri.y + rl + ps], s_n[ri.y + ps], s_t[ri.x + lrl + ps], s_t[ri.x + ps]);
            store_record(rec, slots, ri.x + ((i + (ri.w >> 8)) & 1) * hp + m, e, w, b,
                         divisor_ok(y) ? (T)1 / y : (T)NAN);  // not a number: the division itself has to be taken
        }
    }
    const double mx = ctl->inner_max[EQ_P];
    const double near = 1.001 * g.tol[EQ_P] * g.tol[EQ_P], floor_sq = mx > 0.0 ? mx * mx * N : 0.0;
    double top_sq = -1.0;  // largest sum of this launch
    int sw = ctl->sweeps[EQ_P];
    bool stop = ctl->stop[EQ_P] != 0;
    double last_sq = 0.0;
    unsigned int epoch = 0;
    __syncthreads();  // the records are read back by the same CTA only

    const T relax = g.relax[EQ_P];
    const V zero = {(T)0, (T)0};
    // Failure-detection test (IFC_TEST_STALL_BARRIER=1): as in k_csolve3d.
    bool failed = stall_test && blockIdx.x == 0;
    for (int s = 0; s < n_sweeps && !stop && !failed; ++s) {
        double sq = 0.0;
        for (int color = 0; color < 2; ++color) {
            const bool first = s == 0 && color == 0;  // other blocks' rows are not written yet: all zero
            // After the even half only the rows that other blocks read have to be
            // there before the arrival; the inner rows are swept meanwhile.
            bool arrived = color == 1;
            for (int r = warp; r < nrow || !arrived; r += NT / 32) {
                if (!arrived && r >= nedge) {
                    grid_arrive<NT>(bar, G, epoch);
                    arrived = true;
                }
                if (r >= nrow) break;
                const int4 ri = s_row[r];
                const int fl = ri.w, off = (color ^ (fl >> 8)) & 1, oh = off ? hp : 0;
                for (int q = 2 * lane; 2 * q + off < nx; q += 64) {
                    T *const xo = s_x + ri.x + oh + q;         // the cells updated
                    const T *const xe = s_x + ri.x + hp - oh + q;  // the row's other cells
                    const T *const fn = s_n + ri.y + oh + q, *const ft = s_t + ri.x + oh + q;
                    V e, w, b, z;
                    load_record(rec, slots, ri.x + color * hp + q, e, w, b, z);
                    V xn, xs, xt, xb;
                    if ((fl & 15) == 15) {
                        xn = *reinterpret_cast<const V *>(xo + rl);
                        xs = *reinterpret_cast<const V *>(xo - rl);
                        xt = *reinterpret_cast<const V *>(xo + lrl);
                        xb = *reinterpret_cast<const V *>(xo - lrl);
                    } else {
                        const T *const ex = exch + (ri.z + oh + q);
                        xn = (fl & 1) ? *reinterpret_cast<const V *>(xo + rl)
                                      : (fl & 16) && !first ? __ldcg(reinterpret_cast<const V *>(ex + rl)) : zero;
                        xs = (fl & 2) ? *reinterpret_cast<const V *>(xo - rl)
                                      : (fl & 32) && !first ? __ldcg(reinterpret_cast<const V *>(ex - rl)) : zero;
                        xt = (fl & 4) ? *reinterpret_cast<const V *>(xo + lrl)
                                      : (fl & 64) && !first ? __ldcg(reinterpret_cast<const V *>(ex + ny * rl)) : zero;
                        xb = (fl & 8) ? *reinterpret_cast<const V *>(xo - lrl)
                                      : (fl & 128) && !first ? __ldcg(reinterpret_cast<const V *>(ex - ny * rl)) : zero;
                    }
                    const V o = *reinterpret_cast<const V *>(xe);
                    // the third cell of the other colour: west of the first cell
                    // or east of the second
                    T x3 = (T)0;
                    if (off ? 2 * q + 4 < nx : q > 0) x3 = xe[off ? 2 : -1];
                    const V n = *reinterpret_cast<const V *>(fn + rl), so = *reinterpret_cast<const V *>(fn);
                    const V t = *reinterpret_cast<const V *>(ft + lrl), bo = *reinterpret_cast<const V *>(ft);
                    const V c = *reinterpret_cast<const V *>(xo);
                    const V pe = off ? V{o.y, x3} : o, pw = off ? o : V{x3, o.x};
                    // minus the diagonal, the numerators (in the order of p3_diagonal
                    // and point_update)
                    const Pair<T> y = add2(add2(add2(add2(pair(e), pair(w)), pair(n)), pair(so)), add2(pair(t), pair(bo)));
                    Pair<T> np = add2(pair(b), minus_products(e, pe));
                    np = add2(np, minus_products(w, pw));
                    np = add2(np, minus_products(n, xn));
                    np = add2(np, minus_products(so, xs));
                    np = add2(np, add2(minus_products(t, xt), minus_products(bo, xb)));
                    const Pair<T> q0(np.lo() * z.x, np.hi() * z.y);
                    const Pair<T> qv = fma2(fma2(q0, y, np), pair(z), q0);
                    T v0 = qv.lo(), v1 = qv.hi();
                    if (max(quot_key(v0), quot_key(v1)) > KnownDiv<T>::kSpanQ) {
                        if (quot_key(v0) > KnownDiv<T>::kSpanQ && (np.lo() != (T)0 || z.x != z.x)) v0 = quot_far(np.lo(), -y.lo(), z.x);
                        if (quot_key(v1) > KnownDiv<T>::kSpanQ && (np.hi() != (T)0 || z.y != z.y)) v1 = quot_far(np.hi(), -y.hi(), z.y);
                    }
                    const T d0 = relax * (v0 - c.x);
                    T d1 = relax * (v1 - c.y);
                    V v = {c.x + d0, c.y + d1};
                    if (2 * q + 2 + off >= nx) v.y = d1 = (T)0;  // the pad
                    *reinterpret_cast<V *>(xo) = v;
                    if (fl & 240) __stcg(reinterpret_cast<V *>(exch + (ri.z + oh + q)), v);
                    sq += (double)d0 * (double)d0;
                    sq += (double)d1 * (double)d1;
                }
            }
            if (color == 1) {
                sq = warp_sum(sq);
                if (lane == 0) red[warp] = sq;
                __syncthreads();
                if (warp == 0) {
                    const double t = warp_sum(lane < NT / 32 ? red[lane] : 0.0);
                    if (lane == 0) partials[(size_t)(s & 1) * G + blockIdx.x] = t;
                }
            }
            if (!(color == 0 ? grid_wait(bar, G, epoch) : grid_sync(bar, G, epoch))) {
                failed = true;
                break;
            }
        }
        if (failed) break;
        // grid sum, fixed order, identical in every CTA
        if (tid < 32) {
            double t = 0.0;
#pragma unroll 5
            for (int b = lane; b < G; b += 32) t += __ldcg(&partials[(size_t)(s & 1) * G + b]);
            t = warp_sum(t);
            if (lane == 0) tot1 = t;
        }
        __syncthreads();
        // The early-exit rule (src/Solver.cu:955-962) on the sums: the root and
        // the division by N keep their order, so they are only taken when the
        // sweep comes close to the tolerance.
        const double ssq = tot1;
        if (ssq > top_sq) top_sq = ssq;
        if (!(ssq > near * top_sq && ssq > near * floor_sq && ssq > 1e-30 * N && ssq < 1e300)) {
            const double rms = sqrt(ssq / (double)N);
            double top = top_sq >= 0.0 ? sqrt(top_sq / (double)N) : mx;
            if (mx > top) top = mx;
            if (rms / (top + 1e-20) < g.tol[EQ_P]) stop = true;
        }
        ++sw;
        last_sq = ssq;
    }
    for (int r = warp; r < nrow; r += NT / 32) {
        const int crow = nx * (j0 + r % nj + ny * (k0 + r / nj));
        for (int i = lane; i < nx; i += 32) f.pc[crow + i] = s_x[r * rl + (i & 1) * hp + (i >> 1)];
    }
    if (blockIdx.x == 0 && tid == 0 && !failed) {
        const int done = sw - ctl->sweeps[EQ_P];
        ctl->cell_updates += (long long)done * N;
        const double top = top_sq >= 0.0 ? sqrt(top_sq / (double)N) : mx;
        ctl->inner_max[EQ_P] = top > mx ? top : mx;
        ctl->sweeps[EQ_P] = sw;
        if (done > 0) ctl->last_sweep_sq[EQ_P] = last_sq;
        if (stop) ctl->stop[EQ_P] = 1;
    }
    if (tid == 0 && (failed || bar->err)) atomicExch(&ctl->status, 3);
}

}  // namespace ifc
