// ifc_fused2d_impl.cuh -- host-side launch sequences of the fused 2D kernels.
#pragma once

#include <cstdlib>

namespace ifc {

// Source and destination buffers of one fused pass (u, v or p').
template <typename T>
struct PassBufs {
    const T *in[2];
    T *out[2];
};


template <typename T, int KS>
static int launch_mom_pass(Engine<T> &e, const PassArgs &pa, const PassBufs<T> &b, bool prepare = false)
{
    using S = TileShape2D<T>;
    using R = Region<S::TX, S::TY, 2 * KS>;
    const size_t smem = (size_t)3 * R::NR * sizeof(T);
    auto kern = k_mom_pass2d<T, S::TX, S::TY, KS, S::NT>;
    if (prepare) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
                               cudaSuccess ? IFC_OK : IFC_CUDA_ERROR;
    const int tiles = ((e.P.g.nx + S::TX - 1) / S::TX) * ((e.P.g.ny + S::TY - 1) / S::TY);
    kern<<<tiles, S::NT, smem, e.stream>>>(e.P, e.f, e.ctl, e.partials, pa, b.in[0], b.in[1], b.out[0], b.out[1]);
    ++e.launches;
    return IFC_OK;
}

template <typename T, int KS>
static int launch_pc_pass(Engine<T> &e, const PassArgs &pa, const PassBufs<T> &b, bool prepare = false)
{
    using S = TileShape2D<T>;
    using R = Region<S::TX, S::TY, 2 * KS>;
    const size_t smem = (size_t)2 * R::NR * sizeof(T);
    auto kern = k_pc_pass2d<T, S::TX, S::TY, KS, S::NT>;
    if (prepare) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
                               cudaSuccess ? IFC_OK : IFC_CUDA_ERROR;
    const int tiles = ((e.P.g.nx + S::TX - 1) / S::TX) * ((e.P.g.ny + S::TY - 1) / S::TY);
    kern<<<tiles, S::NT, smem, e.stream>>>(e.P, e.f, e.ctl, e.partials, pa, b.in[0], b.out[0]);
    ++e.launches;
    return IFC_OK;
}

// Supported sweeps per pass; other values round down to the nearest one.
static inline int fused_ks(int want)
{
    if (want >= 8) return 8;
    if (want >= 5) return want >= 6 ? 6 : 5;
    if (want >= 4) return 4;
    if (want >= 3) return 3;
    if (want >= 2) return 2;
    return 1;
}

template <typename T>
static int dispatch_mom(Engine<T> &e, int ks, const PassArgs &pa, const PassBufs<T> &b, bool prepare = false)
{
    switch (ks) {
    case 1: return launch_mom_pass<T, 1>(e, pa, b, prepare);
    case 2: return launch_mom_pass<T, 2>(e, pa, b, prepare);
    case 3: return launch_mom_pass<T, 3>(e, pa, b, prepare);
    case 4: return launch_mom_pass<T, 4>(e, pa, b, prepare);
    case 5: return launch_mom_pass<T, 5>(e, pa, b, prepare);
    case 6: return launch_mom_pass<T, 6>(e, pa, b, prepare);
    default: return launch_mom_pass<T, 8>(e, pa, b, prepare);
    }
}

template <typename T>
static int dispatch_pc(Engine<T> &e, int ks, const PassArgs &pa, const PassBufs<T> &b, bool prepare = false)
{
    switch (ks) {
    case 1: return launch_pc_pass<T, 1>(e, pa, b, prepare);
    case 2: return launch_pc_pass<T, 2>(e, pa, b, prepare);
    case 3: return launch_pc_pass<T, 3>(e, pa, b, prepare);
    case 4: return launch_pc_pass<T, 4>(e, pa, b, prepare);
    case 5: return launch_pc_pass<T, 5>(e, pa, b, prepare);
    case 6: return launch_pc_pass<T, 6>(e, pa, b, prepare);
    default: return launch_pc_pass<T, 8>(e, pa, b, prepare);
    }
}


// Raise the dynamic shared-memory limit of the kernels this handle launches
// (done once at creation, outside any stream capture).
template <typename T>
int Engine<T>::prepare_fused()
{
    PassArgs pa = {};
    PassBufs<T> b = {};
    int rc = dispatch_mom<T>(*this, fused_ks(spp_mom), pa, b, true);
    if (rc == IFC_OK) rc = dispatch_pc<T>(*this, fused_ks(spp_p), pa, b, true);
    if (rc != IFC_OK) err = "cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed";
    return rc;
}

template <typename T>
void Engine<T>::enq_fused_mom()
{
    const int ks = fused_ks(spp_mom);
    const int nu = cfg.n_iter_u, nv = cfg.n_iter_v;
    const int nmax = nu > nv ? nu : nv;
    int npass = (nmax + ks - 1) / ks;
    if (npass < 1) npass = 1;  // the first pass also stores aC
    // A pass stages halos from one buffer and writes its tiles to the other,
    // so no tile reads a neighbour tile's values of the same pass.
    const size_t N = (size_t)P.g.N;
    T *bu[2] = {f.u, f.tmp}, *bv[2] = {f.v, f.tmp + N};
    for (int pass = 0; pass < npass; ++pass) {
        PassArgs pa;
        pa.ns[0] = clamp_sweeps(nu, pass, ks);
        pa.ns[1] = clamp_sweeps(nv, pass, ks);
        pa.ns[2] = 0;
        pa.first = pass == 0;
        PassBufs<T> b = {{bu[pass & 1], bv[pass & 1]}, {bu[(pass + 1) & 1], bv[(pass + 1) & 1]}};
        dispatch_mom<T>(*this, ks, pa, b);
    }
    if (npass & 1) {
        cudaMemcpyAsync(f.u, f.tmp, N * sizeof(T), cudaMemcpyDeviceToDevice, stream);
        cudaMemcpyAsync(f.v, f.tmp + N, N * sizeof(T), cudaMemcpyDeviceToDevice, stream);
    }
}

template <typename T>
void Engine<T>::enq_fused_pcorr()
{
    const int ks = fused_ks(spp_p);
    const int np = cfg.n_iter_p;
    if (np == 0) {
        cudaMemsetAsync(f.pc, 0, (size_t)P.g.N * sizeof(T), stream);
        return;
    }
    const int npass = (np + ks - 1) / ks;
    // Ping-pong as for the momentum passes, ordered so that the last pass
    // writes f.pc (the first pass reads nothing: p' starts from 0).
    T *bp[2] = {f.pc, f.tmp + 2 * (size_t)P.g.N};
    for (int pass = 0; pass < npass; ++pass) {
        PassArgs pa;
        pa.ns[0] = clamp_sweeps(np, pass, ks);
        pa.ns[1] = pa.ns[2] = 0;
        pa.first = pass == 0;
        PassBufs<T> b = {{bp[(npass - pass) & 1], nullptr}, {bp[(npass - 1 - pass) & 1], nullptr}};
        dispatch_pc<T>(*this, ks, pa, b);
    }
}

template <typename T>
void Engine<T>::enq_fused_rc()
{
    k_rc_mass2d<T><<<grid(P.g.N), 256, 0, stream>>>(P, f, ctl, partials);
    ++launches;
}

}  // namespace ifc

namespace ifc {

// ---- the persistent single-launch 2D solve (ifc_persist2d.cuh) ----
// Region shapes: rows per lane and warps (a region is 64 x R*NW cells), and the
// relative time of an outer iteration with one tile per CTA (`one`) or with n in
// turn, whose links are rebuilt in every pass (base + n * each); the shape with
// the least is taken.  In us of the 5-sweep channel, FP32 / FP64, one tile: 24
// rows 50 / 68, 28 rows 54 / 76, 32 rows 57 / 84, 36 rows - / 101, 64 rows 105 /
// -.  Two tiles: 24 rows 90 FP32, 28 rows 106 FP32, 32 rows 111 / 175, 36 rows -
// / 211, 64 rows 228 FP32; eight of 28 rows 315 / 493, six of 32 268 / 437, four
// of 36 - / 374.  So small grids, which leave SMs idle, take the smallest region
// whose tiles fit one round, and the larger regions, which waste less on halos,
// win once they save rounds (1024x256: 106 us in one round of 64 rows).  FP64
// has half the registers per cell: 64 rows do not fit.  Its half sweeps take in
// proportion to their rows, so a single tile gains little from having no
// barriers (33x31: 79 us in one of 32 rows, 65 in three of 24), and 20 rows serve
// passes of up to four sweeps (33x31, 4 sweeps: 88 -> 70).
struct RegionShape {
    int R, NW;
    double one, base, each;
};
template <typename T>
struct RegionShapes;
template <>
struct RegionShapes<float> {
    static constexpr int n = 4;
    static constexpr RegionShape s[n] = {
        {2, 12, 0.87, 0.46, 0.56}, {2, 14, 0.95, 0.60, 0.61}, {2, 16, 1.0, 0.58, 0.68}, {4, 16, 1.85, 0.30, 1.80}};
    static constexpr double alone = 0.3;  // what a single tile gains without grid barriers
};
template <>
struct RegionShapes<double> {
    static constexpr int n = 5;
    static constexpr RegionShape s[n] = {{2, 10, 0.70, 0.45, 0.42},
                                         {2, 12, 0.80, 0.47, 0.50},
                                         {2, 14, 0.90, 0.54, 0.67},
                                         {2, 16, 1.0, 0.54, 0.77},
                                         {2, 18, 1.2, 0.56, 0.98}};
    static constexpr double alone = 0.1;
};

template <typename T, int I>
using ShapeTile = RTile<T, RegionShapes<T>::s[I].R, RegionShapes<T>::s[I].NW>;

// Dynamic shared memory of k_simple2d: exchange rows of two fields, then the
// per-thread sums of a pass or (Rhie-Chow) the faces of a tile.
template <typename RT, typename T>
static size_t persist_smem(int ks)
{
    const size_t sums = (size_t)(2 * ks > 7 ? 2 * ks : 7) * RT::NT * sizeof(double);
    const size_t faces = ((size_t)(RT::W + 1) * RT::HR + (size_t)RT::W * (RT::HR + 1)) * sizeof(T);
    return (size_t)RT::END * sizeof(T) + (sums > faces ? sums : faces);
}

// launch = false: set the kernel's shared-memory limit (one setting per process,
// so the device's maximum) and return in *capacity the CTAs that can be
// co-resident.  launch = true: launch it on e.persist_grid CTAs.
template <typename T, int I>
static int persist_kernel(Engine<T> &e, bool launch, int *capacity)
{
    using RT = ShapeTile<T, I>;
    auto kern = k_simple2d<T, RT::R, RT::NW>;
    const size_t smem = persist_smem<RT, T>(e.persist_args.ks);
    if (!launch) {
        int dev = 0, optin = 0;
        cudaFuncAttributes fa;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            cudaFuncGetAttributes(&fa, kern) != cudaSuccess)
            return IFC_CUDA_ERROR;
        const int dyn_max = optin - (int)fa.sharedSizeBytes;
        if ((long long)smem > dyn_max) return IFC_UNSUPPORTED;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn_max) != cudaSuccess)
            return IFC_CUDA_ERROR;
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, RT::NT, smem) != cudaSuccess)
            return IFC_CUDA_ERROR;
        *capacity = (per_sm < 2 ? per_sm : 2) * e.nsm;
        return IFC_OK;
    }
    PersistArgs &pa = e.persist_args;
    const char *stall = std::getenv("IFC_TEST_STALL_BARRIER");
    pa.stall_test = (stall && stall[0] == '1') ? 1 : 0;
    void *args[] = {&e.P, &e.f, &e.ctl, &e.partials, &e.barrier, &pa};
    return cudaLaunchCooperativeKernel((const void *)kern, dim3(e.persist_grid), dim3(RT::NT), args, smem, e.stream) ==
                   cudaSuccess
               ? IFC_OK
               : IFC_CUDA_ERROR;
}

template <typename T, int I = 0>
static int persist_dispatch(Engine<T> &e, int shape, bool launch, int *capacity)
{
    if constexpr (I + 1 < RegionShapes<T>::n) {
        if (shape > I) return persist_dispatch<T, I + 1>(e, shape, launch, capacity);
    }
    return persist_kernel<T, I>(e, launch, capacity);
}

static inline int persist_ks(int want)
{
    if (want >= 10) return 10;
    if (want >= 8) return 8;
    return want < 2 ? 2 : (want > 6 ? 6 : want);
}

// The whole 2D loop as one cooperative launch: one tile per CTA when all tiles'
// CTAs can be co-resident, otherwise every CTA visits ceil(tiles / CTAs) tiles
// in turn, on the fewest CTAs that give that count.  IFC_PERSIST_OFF=1 keeps
// the multi-kernel graph; IFC_PERSIST_MAX_CTAS caps the CTAs (used by the tests
// to run several tiles per CTA on small grids).
template <typename T>
int Engine<T>::prepare_persist()
{
    persist = false;
    if (dim != 2 || !fused || cfg.linear_solver != IFC_GAUSS_SEIDEL) return IFC_OK;
    // the residual rule needs the residual pass of the graph form
    if (P.g.criterion == 2) return IFC_OK;
    const char *off = std::getenv("IFC_PERSIST_OFF");  // the multi-kernel graph instead (A/B timing, tests)
    if (off && off[0] == '1') return IFC_OK;
    int coop = 0, dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return IFC_OK;
    PersistArgs &pa = persist_args;
    pa.n_iter[0] = cfg.n_iter_u;
    pa.n_iter[1] = cfg.n_iter_v;
    pa.n_iter[2] = 0;
    pa.n_iter[3] = cfg.n_iter_p;
    pa.pin = pin ? 1 : 0;
    pa.stall_test = 0;
    int cap_env = 0;
    if (const char *cap = std::getenv("IFC_PERSIST_MAX_CTAS")) cap_env = std::atoi(cap);
    // Passes of six and more sweeps need halos of 24 and more cells, which leave
    // little of a region (FP64 500x190, 8 sweeps: 433 us per outer iteration).  They
    // may be split into two each; the early exit is then checked after every
    // second pass, so the values are the same (same example: 103 us).
    const int check = persist_ks(spp_persist);
    const int n_m = cfg.n_iter_u > cfg.n_iter_v ? cfg.n_iter_u : cfg.n_iter_v;
    double best = 0.0;
    int best_ks = check;
    for (int group = 1; group <= (check >= 6 && check % 2 == 0 ? 2 : 1); ++group)
        for (int s = 0; s < RegionShapes<T>::n; ++s) {
            const RegionShape &sh = RegionShapes<T>::s[s];
            pa.ks = check / group;
            TileGrid tg;
            tg.H = 2 * pa.ks;
            if (!split_axis(P.g.nx, 64, tg.H, &tg.kx, &tg.Ix) || !split_axis(P.g.ny, sh.R * sh.NW, tg.H, &tg.ky, &tg.Iy))
                continue;
            int capacity = 0;
            if (persist_dispatch<T>(*this, s, false, &capacity) != IFC_OK) {
                cudaGetLastError();
                continue;
            }
            if (cap_env > 0 && capacity > cap_env) capacity = cap_env;
            if (capacity < 1) continue;
            const long long tiles = (long long)tg.kx * tg.ky;
            const long long per = (tiles + capacity - 1) / capacity;
            // Passes of an outer iteration times the cost of one: half of a
            // pass of five sweeps is its sweeps, half what comes with every
            // pass (64x64 FP32: 66 us per iteration with 3 sweeps, 50 with 5).
            const int passes = (n_m + pa.ks - 1) / pa.ks + (cfg.n_iter_p + pa.ks - 1) / pa.ks;
            // (a single tile runs without grid barriers)
            const double cost = (passes > 0 ? passes : 1) * (0.5 + 0.1 * pa.ks) *
                                (per > 1 ? sh.base + (double)per * sh.each : tiles > 1 ? sh.one : sh.one - RegionShapes<T>::alone);
            if (persist && cost >= best) continue;
            best = cost;
            best_ks = pa.ks;
            persist = true;
            persist_shape = s;
            persist_grid = (int)((tiles + per - 1) / per);
            pa.tiles = tg;
            pa.group = group;
        }
    pa.ks = best_ks;
    pa.one = persist && persist_grid == pa.tiles.kx * pa.tiles.ky;
    if (!persist) return IFC_OK;
    pa.npass_m = (n_m + pa.ks - 1) / pa.ks;
    pa.npass_p = (cfg.n_iter_p + pa.ks - 1) / pa.ks;
    pa.tail_m = pa.npass_m > 0 ? (pa.npass_m - 1) / pa.group * pa.group : 0;
    pa.tail_p = pa.npass_p > 0 ? (pa.npass_p - 1) / pa.group * pa.group : 0;
    // SMs that have no tile: narrower tiles, of twelve columns and more, share out
    // the phases between the sweeps (deferred correction, faces, corrections),
    // whose time follows a CTA's own cells; the sweeps cost the same, a region
    // each.  us per outer iteration, FP64 / FP32: 1169x18 QUICK 83 -> 73 / 62 -> 57,
    // 64x64 68 -> 63 / 50 -> 48.  A single tile only where these phases outweigh
    // its lack of barriers (64x22: FP64 QUICK 75 -> 73, FP64 upwind 64 -> 66, FP32
    // 42 -> 50).
    TileGrid &tg = pa.tiles;
    const int tiles = tg.kx * tg.ky, inner = P.g.nx - 2 * tg.H;
    int room = nsm;
    if (cap_env > 0 && room > cap_env) room = cap_env;
    if (persist_grid != tiles || inner <= 12 || (tiles == 1 && (sizeof(T) == 4 || cfg.convection_scheme == IFC_CONV_UPWIND)))
        return IFC_OK;
    const int most = room / tg.ky;
    if (most <= tg.kx) return IFC_OK;
    int w = (inner + most - 1) / most;
    w += w & 1;
    if (w < 12) w = 12;
    tg.Ix = w;
    tg.kx = (inner + w - 1) / w;
    persist_grid = tg.kx * tg.ky;
    pa.one = 1;
    return IFC_OK;
}

template <typename T>
int Engine<T>::launch_persist()
{
    if (cudaMemsetAsync(barrier, 0, sizeof(GridBarrier), stream) != cudaSuccess) return IFC_CUDA_ERROR;
    ++launches;
    return persist_dispatch<T>(*this, persist_shape, true, nullptr);
}

// ---- sweeps on stored 2D coefficients in one cooperative launch ----
// call = nullptr: prepare the kernel of shape I and return its co-resident CTAs.
template <typename T>
struct CoefCall {
    const Params<T> *P;
    const T *coef, *src;
    CoefArgs ca;
    T *x0, *x1;
};

template <typename T, int I>
static cudaError_t coef_kernel(Engine<T> &e, CoefCall<T> *call, int *capacity)
{
    using RT = ShapeTile<T, I>;
    auto kern = k_coef_solve2d<T, RT::R, RT::NW>;
    const size_t smem = (size_t)RT::END * sizeof(T) + (size_t)kCoefSweeps * RT::NT * sizeof(double);
    if (!call) {
        cudaError_t rc = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int per_sm = 0;
        if (rc == cudaSuccess) rc = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, RT::NT, smem);
        *capacity = (per_sm < 2 ? per_sm : 2) * e.nsm;
        return rc;
    }
    void *args[] = {(void *)call->P, &call->coef, &call->src, &e.ctl, &e.partials, &e.barrier, &call->ca, &call->x0, &call->x1};
    const TileGrid &tg = call->ca.tiles;
    return cudaLaunchCooperativeKernel((const void *)kern, dim3(tg.kx * tg.ky), dim3(RT::NT), args, smem, e.stream);
}

template <typename T, int I = 0>
static cudaError_t coef_dispatch(Engine<T> &e, int shape, CoefCall<T> *call, int *capacity)
{
    if constexpr (I + 1 < RegionShapes<T>::n) {
        if (shape > I) return coef_dispatch<T, I + 1>(e, shape, call, capacity);
    }
    return coef_kernel<T, I>(e, call, capacity);
}

template <typename T>
bool Engine<T>::coef_coop()
{
    if (coef_state >= 0) return coef_state == 1;
    coef_state = 0;
    int coop = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    const char *off = std::getenv("IFC_PERSIST_OFF");
    if (!coop || (off && off[0] == '1')) return false;
    double best = 0.0;
    for (int s = 0; s < RegionShapes<T>::n; ++s) {
        const RegionShape &sh = RegionShapes<T>::s[s];
        TileGrid tg;
        tg.H = 2 * kCoefSweeps;
        if (!split_axis(P.g.nx, 64, tg.H, &tg.kx, &tg.Ix) || !split_axis(P.g.ny, sh.R * sh.NW, tg.H, &tg.ky, &tg.Iy))
            continue;
        const long long tiles = (long long)tg.kx * tg.ky;
        const double cost = sh.one - (tiles == 1 ? RegionShapes<T>::alone : 0.0);
        int capacity = 0;
        if (coef_dispatch<T>(*this, s, nullptr, &capacity) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (tiles > capacity || (coef_state == 1 && cost >= best)) continue;
        best = cost;
        coef_state = 1;
        coef_shape = s;
        coef_tiles = tg;
    }
    return coef_state == 1;
}

template <typename T>
int Engine<T>::launch_coef(const Params<T> &PP, const T *coef, const T *src, int eq, int n, T *x0, T *x1, int stall)
{
    IFC_CK(cudaMemsetAsync(barrier, 0, sizeof(GridBarrier), stream));
    CoefCall<T> call = {&PP, coef, src, {coef_tiles, eq, n, stall}, x0, x1};
    IFC_CK(coef_dispatch<T>(*this, coef_shape, &call, nullptr));
    return IFC_OK;
}

}  // namespace ifc
