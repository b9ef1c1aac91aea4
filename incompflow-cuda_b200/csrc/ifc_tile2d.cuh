// ifc_tile2d.cuh -- red-black sweeps of a 2D region held in registers.
//
// One CTA of NW warps holds a region of 64 x (R*NW) cells for a whole pass of
// sweeps: lane l of warp w owns the columns 2l, 2l+1 of the rows w*R .. w*R+R-1,
// unknowns, links, diagonal and sources in registers.  In every row one of a
// lane's two cells is red and the other black (the region's origin is even in
// both directions), so every lane updates one cell per row and half sweep:
// its horizontal neighbours are the lane's other cell and one shuffle, its
// vertical neighbours the lane's own rows, and only the first and last row of
// a warp go through shared memory to the warps below and above, one block
// barrier per half sweep.  Rows are taken in pairs and the FP32 arithmetic
// that does not depend on the order of the rows' neighbours runs as packed
// pairs (half the issue slots).  What bounds it is the latency of a half sweep
// (barrier, exchange row, shuffle, a chain of eleven operations) and then the
// issue rate: 40 warp instructions for 64 updates; a half sweep of a 64x32 region
// takes about 500 cycles for p' and 800 for u and v together (512x128, counted
// inside the solve), against 640 for one unknown of 850 cells when unknowns sit
// in shared memory under a generic index map (about 80 instructions per 32
// updates: masks, addresses, the compiler's division).  The half sweeps are a
// third of an outer iteration; the rest is the grid barriers, the turn-round of
// a pass (halos, links, own cells and column sums) and the faces and corrections.
// Outer iteration of the 1024x256 channel 215 -> 103 us, 4096x2048 5.7 -> 2.7
// ms, 512x128 65.6 -> 58 us, 33x31 cavity 105 -> 84 us.
//
// The divisor of a point update, the equation's diagonal, does not change
// within a solve, so z = 1/aC is computed once (IEEE division) and a quotient
// costs one multiplication and two fused multiply-adds: q0 = RN(n z),
// r = RN(n - q0 y), q = RN(q0 + r z), which is n/y correctly rounded
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990; N. Brisebarre, J.-M.
// Muller, S. K. Raina, "Accelerating correctly rounded floating-point division
// when the divisor is known in advance", IEEE Trans. Comput. 53, 2004), away
// from overflow and underflow.  Tiny quotients are formed scaled up; those near
// overflow, and cells whose diagonal is outside the range of the reciprocal, take
// the division itself.
#pragma once

#include "ifc_kernels.cuh"

namespace ifc {

// Ranges in which the corrected quotient is exact: |y| in [ylo, yhi] and |n| in
// [2^-85, 2^80) (FP64: [2^-820, 2^800)) keep the residual n - q y (a multiple of
// ulp(q) ulp(y), at least 2^-47 |n|) and every intermediate normal.
// range_key(n) maps |n| to an unsigned number that is at most kSpan inside the
// range and larger for any other value, zero, infinity and NaN among them.
// Where z may be no number, quot_key looks at the quotient instead: |q| in
// [2^-62, 2^62) (FP64: [2^-700, 2^700)) does as well, for every y in its range.
template <typename T>
struct KnownDiv;
template <>
struct KnownDiv<float> {
    static constexpr float ylo = 0x1p-40f, yhi = 0x1p40f, small = 0x1p-20f, large = 0x1p120f;
    static constexpr float up = 0x1p64f, down = 0x1p-64f, tiny = 0x1p-126f, ulp = 0x1p-149f, half = 0x1p-86f;
    static constexpr unsigned kLow = (127u - 85u) << 24, kSpan = (165u << 24) - 1u;
    static constexpr unsigned kLowQ = (127u - 62u) << 24, kSpanQ = (124u << 24) - 1u;
};
template <>
struct KnownDiv<double> {
    static constexpr double ylo = 0x1p-200, yhi = 0x1p200, small = 0x1p-500, large = 0x1p1000;
    static constexpr double up = 0x1p400, down = 0x1p-400, tiny = 0x1p-1022, ulp = 0x1p-1074, half = 0x1p-675;
    static constexpr unsigned kLow = (1023u - 820u) << 21, kSpan = (1620u << 21) - 1u;
    static constexpr unsigned kLowQ = (1023u - 700u) << 21, kSpanQ = (1400u << 21) - 1u;
};

__device__ __forceinline__ unsigned magnitude(float a) { return __float_as_uint(a) * 2u; }
__device__ __forceinline__ unsigned magnitude(double a) { return (unsigned)__double2hiint(a) * 2u; }
template <typename T>
__device__ __forceinline__ unsigned range_key(T n)
{
    return magnitude(n) - KnownDiv<T>::kLow;
}
template <typename T>
__device__ __forceinline__ unsigned quot_key(T q)
{
    return magnitude(q) - KnownDiv<T>::kLowQ;
}
// Which of the two the sweeps look at: the numerator's range is wider (29x621
// channel, whose core holds tiny values for long, 69 -> 64 us per outer
// iteration), but with four rows per lane it costs registers (developed 2048x512
// 426 -> 436 us).
template <int R, typename T>
__device__ __forceinline__ unsigned far_key(T n, T q)
{
    return R == 2 ? range_key(n) : quot_key(q);
}
__device__ __forceinline__ float abs_t(float a) { return fabsf(a); }
__device__ __forceinline__ double abs_t(double a) { return fabs(a); }

// The division itself.  Written as volatile so that it stays behind the rarely
// taken branch: the compiler otherwise computes it always and selects (660
// against 530 cycles per half sweep of a 64x32 region).
__device__ __forceinline__ float quot_div(float n, float y)
{
    float q;
    asm volatile("div.rn.f32 %0, %1, %2;" : "=f"(q) : "f"(n), "f"(y));
    return q;
}
__device__ __forceinline__ double quot_div(double n, double y)
{
    double q;
    asm volatile("div.rn.f64 %0, %1, %2;" : "=d"(q) : "d"(n), "d"(y));
    return q;
}

// Whether divisor y may be used with a precomputed reciprocal.
template <typename T>
__device__ __forceinline__ bool divisor_ok(T y)
{
    return abs_t(y) >= KnownDiv<T>::ylo && abs_t(y) <= KnownDiv<T>::yhi;
}

__device__ __forceinline__ float fma1(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma1(double a, double b, double c) { return __fma_rn(a, b, c); }

// The quotient of n < small, given q = RN(m / y) of the numerator scaled up, m =
// up * n (exact): q scaled back.  That rounds a second time when the result is
// subnormal (or the smallest normal number, which can come from below): where q
// lies halfway between two subnormals -- `half` is half their distance, scaled
// up -- the sign of the exact residual tells on which side the quotient is.
template <typename T>
__device__ __forceinline__ T scaled_back(T q, T m, T y)
{
    using K = KnownDiv<T>;
    T d = q * K::down;
    if (abs_t(d) <= K::tiny) {
        const T diff = q - d * K::up, r = fma1(-q, y, m);
        if (abs_t(diff) == K::half && r != (T)0 && (diff > (T)0) == ((r > (T)0) == (y > (T)0)))
            d += diff > (T)0 ? K::ulp : -K::ulp;
    }
    return d;
}

// n / y for a divisor in [ylo, yhi] and z = RN(1/y), whatever the magnitude of
// n; `ok` tells whether it is (not where the quotient comes near overflow, nor
// where y or z is out of range or not a number).
template <typename T>
__device__ __forceinline__ T quot_scaled(T n, T y, T z, bool &ok)
{
    using K = KnownDiv<T>;
    const bool low = abs_t(n) < K::small;
    const T m = n * (low ? K::up : (T)1);
    T q = m * z;
    q = fma1(fma1(-q, y, m), z, q);
    ok = abs_t(q) <= K::large && divisor_ok(y);
    return low ? scaled_back(q, m, y) : q;
}

// The same in every case, out of line.
template <typename T>
static __device__ __noinline__ T quot_far(T n, T y, T z)
{
    bool ok;
    const T q = quot_scaled(n, y, z, ok);
    return ok ? q : quot_div(n, y);
}

// n / y given z = RN(1/y).
template <typename T>
__device__ __forceinline__ T quot_known(T n, T y, T z)
{
    T q = n * z;
    q = fma1(fma1(-q, y, n), z, q);
    if (range_key(n) > KnownDiv<T>::kSpan || !divisor_ok(y)) {
        if (n != (T)0 || !divisor_ok(y)) q = quot_far(n, y, z);
    }
    return q;
}

// ---- pairs -------------------------------------------------------------------
// Two values and the operations on them; in FP32 one packed instruction each.
// A packed sum must not take a packed product directly: the assembler contracts
// such a pair to one FMA, even under --fmad=false and with the rounding written
// out (tested: differences on 14 % of random operands), which would change the
// results.  Where a product is added, one of the two is done on the halves.
template <typename T>
struct Pair;
template <>
struct Pair<float> {
    float2 v;
    __device__ __forceinline__ Pair(float a, float b) : v(make_float2(a, b)) {}
    __device__ __forceinline__ explicit Pair(float2 q) : v(q) {}
    __device__ __forceinline__ float lo() const { return v.x; }
    __device__ __forceinline__ float hi() const { return v.y; }
};
template <>
struct Pair<double> {
    double a, b;
    __device__ __forceinline__ Pair(double x, double y) : a(x), b(y) {}
    __device__ __forceinline__ double lo() const { return a; }
    __device__ __forceinline__ double hi() const { return b; }
};
__device__ __forceinline__ Pair<float> mul2(Pair<float> a, Pair<float> b) { return Pair<float>(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ Pair<float> add2(Pair<float> a, Pair<float> b) { return Pair<float>(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ Pair<float> fma2(Pair<float> a, Pair<float> b, Pair<float> c)
{
    return Pair<float>(__ffma2_rn(a.v, b.v, c.v));
}
__device__ __forceinline__ Pair<double> mul2(Pair<double> a, Pair<double> b) { return {a.a * b.a, a.b * b.b}; }
__device__ __forceinline__ Pair<double> add2(Pair<double> a, Pair<double> b) { return {a.a + b.a, a.b + b.b}; }
__device__ __forceinline__ Pair<double> fma2(Pair<double> a, Pair<double> b, Pair<double> c)
{
    return {__fma_rn(a.a, b.a, c.a), __fma_rn(a.b, b.b, c.b)};
}

// Pairs in shared memory, 2 values at an address aligned to them.
__device__ __forceinline__ Pair<float> load_pair(const float *p) { return Pair<float>(*reinterpret_cast<const float2 *>(p)); }
__device__ __forceinline__ Pair<double> load_pair(const double *p)
{
    const double2 v = *reinterpret_cast<const double2 *>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ void store_pair(float *p, float a, float b) { *reinterpret_cast<float2 *>(p) = make_float2(a, b); }
__device__ __forceinline__ void store_pair(double *p, double a, double b) { *reinterpret_cast<double2 *>(p) = make_double2(a, b); }

// ---- tiles ------------------------------------------------------------------
// Along an axis of n cells, k tiles with interior width I and a halo of H = 2 *
// (sweeps per pass) cells: tile t's region starts at cell t*I, its own cells
// at H inside the region (at 0 for the first tile, whose region begins at the
// domain's edge, where no halo is needed) and end at H + I (at the domain's
// edge for the last).  I and H are even, so a region's origin is even and the
// colours fall on the same registers in every tile.
struct TileGrid {
    int H;
    int kx, Ix, ky, Iy;
};

struct TileBox {
    int gx0, gy0;              // region origin
    int ox0, ox1, oy0, oy1;    // own cells, in region coordinates
};

__device__ __forceinline__ TileBox tile_box(const TileGrid &G, int t, int nx, int ny)
{
    TileBox b;
    const int ty = t / G.kx, tx = t - ty * G.kx;
    b.gx0 = tx * G.Ix;
    b.gy0 = ty * G.Iy;
    b.ox0 = tx > 0 ? G.H : 0;
    b.ox1 = tx == G.kx - 1 ? nx - b.gx0 : G.H + G.Ix;
    b.oy0 = ty > 0 ? G.H : 0;
    b.oy1 = ty == G.ky - 1 ? ny - b.gy0 : G.H + G.Iy;
    return b;
}

// Splits n cells for regions of C cells; false when the halo leaves no room.
__host__ __device__ inline bool split_axis(int n, int C, int H, int *k, int *I)
{
    if (n <= C) {
        *k = 1;
        *I = 0;
        return true;
    }
    const int cap = C - 2 * H;
    if (cap < 2) return false;
    const int inner = n - 2 * H;
    int kk = (inner + cap - 1) / cap;
    int w = (inner + kk - 1) / kk;
    w += w & 1;
    *I = w;
    *k = (inner + w - 1) / w;
    return true;
}

// Shared memory of a CTA, in values of T from the start of the dynamic shared
// memory (addressed by 32-bit offsets from there: pointers would cost the
// sweeps two registers each):
//   sources of two unknowns: thread-private pairs, [colour][row pair][thread]
//     (in registers they would spill more of the sweeps: as it is, regions of 32
//     rows spill 34 values per thread, of 64 rows 183, FP64 77 to 144, and one
//     instruction in 80 is a spill at 512x128);
//   exchange rows of two unknowns: side 0 the warps' first rows, side 1 their
//     last, a row of zeros at either end, columns split by parity.
template <typename T, int R_, int NW_>
struct RTile {
    static constexpr int R = R_, NW = NW_, W = 64, HR = R * NW, NT = 32 * NW;
    static_assert(R % 2 == 0, "a warp's first row must be even");
    static constexpr int LEN = 2 * R * NT;  // values of one per-thread array
    static constexpr int SIDE = (NW + 2) * W;
    static constexpr int EX = 2 * SIDE;
    static constexpr int SRC = 0, XB = 2 * LEN;
    static constexpr int END = XB + 2 * EX;
};

template <typename T>
__device__ __forceinline__ T *tile_smem()
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    return reinterpret_cast<T *>(smem_raw);
}

// A lane's 2R values of a field, by colour: v[c][j][h] belongs to row 2j + h and
// to column (c + h) & 1, so a colour's values of a row pair are neighbours.
template <typename T, int R>
struct Cells {
    T v[2][R / 2][2];
    __device__ __forceinline__ T &at(int r, int k) { return v[(r + k) & 1][r >> 1][r & 1]; }
    __device__ __forceinline__ T at(int r, int k) const { return v[(r + k) & 1][r >> 1][r & 1]; }
    __device__ __forceinline__ Pair<T> pair(int c, int j) const { return Pair<T>(v[c][j][0], v[c][j][1]); }
};

// Offset of a lane's first column in its warp's first exchange row of unknown
// 0; the last row is SIDE further, the rows of the warps above and below one
// row width further on side 0 and back on side 1.
template <typename RT>
__device__ __forceinline__ int lane_row()
{
    return RT::XB + ((threadIdx.x >> 5) + 1) * RT::W + (threadIdx.x & 31);
}

// First and last row of x to the exchange rows of unknown f.
template <typename RT, typename T>
__device__ __forceinline__ void publish(const Cells<T, RT::R> &x, int f)
{
    T *p = tile_smem<T>() + lane_row<RT>() + f * RT::EX;
    p[0] = x.at(0, 0);
    p[32] = x.at(0, 1);
    p[RT::SIDE] = x.at(RT::R - 1, 0);
    p[RT::SIDE + 32] = x.at(RT::R - 1, 1);
}

// Thread-private pairs at offset `base` (SRC + f*LEN).
template <typename RT, typename T>
__device__ __forceinline__ void put_cells(const Cells<T, RT::R> &b, int base)
{
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < RT::R / 2; ++j)
            store_pair(tile_smem<T>() + base + 2 * (int)threadIdx.x + (c * (RT::R / 2) + j) * 2 * RT::NT, b.v[c][j][0],
                       b.v[c][j][1]);
}
template <typename RT, typename T>
__device__ __forceinline__ Pair<T> get_pair(int base, int c, int j)
{
    return load_pair(tile_smem<T>() + base + 2 * (int)threadIdx.x + (c * (RT::R / 2) + j) * 2 * RT::NT);
}

// Zeros in the rows beyond the region (once per launch).
template <typename RT, typename T>
__device__ __forceinline__ void clear_guards()
{
    T *ex = tile_smem<T>() + RT::XB;
    for (int q = threadIdx.x; q < 2 * 2 * 2 * RT::W; q += RT::NT) {
        const int c = q % RT::W, e = (q / RT::W) & 1, fs = q / (2 * RT::W);
        ex[fs * RT::SIDE + (e ? (RT::NW + 1) * RT::W : 0) + c] = (T)0;
    }
}

// Negated links, negated diagonal and the diagonal's reciprocal of a lane's
// cells (x - y is x + (-y) in every case, so the negation changes no result).
// O: the link to the lane's other cell of the row, H: to the neighbouring
// lane's cell.  Column 0 has its other cell in the east, column 1 in the west.
template <typename RT, typename T>
struct Links {
    static constexpr int R = RT::R;
    Cells<T, R> O, H, N, S, C, Z;
    __device__ __forceinline__ void set(int r, int k, T E, T W, T n, T s, T c)
    {
        O.at(r, k) = k == 0 ? -E : -W;
        H.at(r, k) = k == 0 ? -W : -E;
        N.at(r, k) = -n;
        S.at(r, k) = -s;
        C.at(r, k) = -c;
    }
};

// The quotients q = n / diagonal whose bit in `todo` is set (bit 2*J*f + 2*j + h),
// which lie outside the range of half_sweep's formula.  Fronts of a flow that
// develops from rest pass through all small magnitudes, down to zero, many warps
// at a time, and every CTA waits for the slowest: 1024x256 channel from rest,
// us per iteration over the first 20, with a division each (twice for subnormal
// quotients) 290 FP32 / 523 FP64, this way 138 / 428.  FP32 takes all values at
// once, scaled up where they are small; in FP64 that costs registers that the
// sweeps need (developed flow 308 -> 319), so one value at a time.
template <typename RT, typename T, int COLOR, int F>
__device__ __forceinline__ void far_quotients(const Links<RT, T> &a, const T (&n)[F][RT::R / 2][2],
                                              T (&q)[F][RT::R / 2][2], unsigned todo, bool force)
{
    using K = KnownDiv<T>;
    constexpr int J = RT::R / 2;
    constexpr bool at_once = sizeof(T) == 4;
    if (at_once && !force) {
        todo = 0;  // what is left: quotients near overflow
#pragma unroll
        for (int f = 0; f < F; ++f)
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const Pair<T> z = a.Z.pair(COLOR, j), c = a.C.pair(COLOR, j);
                const bool low0 = abs_t(n[f][j][0]) < K::small, low1 = abs_t(n[f][j][1]) < K::small;
                const Pair<T> m = mul2(Pair<T>(n[f][j][0], n[f][j][1]), Pair<T>(low0 ? K::up : (T)1, low1 ? K::up : (T)1));
                Pair<T> w = mul2(m, z);
                w = fma2(fma2(w, c, m), z, w);
                if (!(abs_t(w.lo()) <= K::large)) todo |= 1u << (2 * J * f + 2 * j);
                if (!(abs_t(w.hi()) <= K::large)) todo |= 2u << (2 * J * f + 2 * j);
                q[f][j][0] = low0 ? scaled_back(w.lo(), m.lo(), -c.lo()) : w.lo();
                q[f][j][1] = low1 ? scaled_back(w.hi(), m.hi(), -c.hi()) : w.hi();
            }
        if (!todo) return;
    }
    // In loops, so that they take little code.
    T tn[F * 2 * J], ty[2 * J];
#pragma unroll
    for (int i = 0; i < 2 * J; ++i) {
        ty[i] = -a.C.v[COLOR][i >> 1][i & 1];
#pragma unroll
        for (int f = 0; f < F; ++f) tn[2 * J * f + i] = n[f][i >> 1][i & 1];
    }
    if (at_once) {
#pragma unroll 1
        for (int i = 0; i < F * 2 * J; ++i)
            if (todo >> i & 1u) tn[i] = quot_div(tn[i], ty[i % (2 * J)]);
    } else {
#pragma unroll 1
        for (unsigned rest = todo; rest; rest &= rest - 1) {
            const int i = __ffs(rest) - 1;
            const T y = ty[i % (2 * J)];
            const bool low = abs_t(tn[i]) < K::small && divisor_ok(y);
            const T m = low ? tn[i] * K::up : tn[i], w = quot_div(m, y);
            tn[i] = low ? scaled_back(w, m, y) : w;
        }
    }
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
        for (int i = 0; i < 2 * J; ++i)
            if (todo >> (2 * J * f + i) & 1u) q[f][i >> 1][i & 1] = tn[2 * J * f + i];
}

// One half sweep of colour COLOR over the lane's rows for the F unknowns x[f]
// (one, or u and v with their common links: twice the independent work for
// the latency of one).  With SUM, acc[f][k] receives the squared changes of
// the lane's column k in the rows of `rown` (bit r set: row r belongs to the
// tile).  An unknown whose act[f] is false keeps its values.
template <typename RT, typename T, int COLOR, int F, bool SUM>
__device__ __forceinline__ void half_sweep(Cells<T, RT::R> *const (&xs)[F], const Links<RT, T> &a,
                                           const T (&relax)[F], const bool (&act)[F], bool force, unsigned rown,
                                           double (&acc)[F][2])
{
    constexpr int J = RT::R / 2, OC = 1 - COLOR;
    constexpr unsigned span = RT::R == 2 ? KnownDiv<T>::kSpan : KnownDiv<T>::kSpanQ;
    const Pair<T> minus(-(T)1, -(T)1);
    T n[F][J][2], q[F][J][2];
    T below[F], above[F];
    unsigned key = 0;
    T *const row = tile_smem<T>() + lane_row<RT>();
    // updated columns: COLOR in even rows, OC in odd ones
#pragma unroll
    for (int f = 0; f < F; ++f) {
        below[f] = row[f * RT::EX + RT::SIDE - RT::W + COLOR * 32];
        above[f] = row[f * RT::EX + RT::W + OC * 32];
    }
#pragma unroll
    for (int f = 0; f < F; ++f) {
        const Cells<T, RT::R> &x = *xs[f];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const Pair<T> b = get_pair<RT, T>(RT::SRC + f * RT::LEN, COLOR, j);
            const T olo = x.v[OC][j][0], ohi = x.v[OC][j][1];
            const T hlo = COLOR == 0 ? __shfl_up_sync(0xffffffffu, olo, 1) : __shfl_down_sync(0xffffffffu, olo, 1);
            const T hhi = COLOR == 0 ? __shfl_down_sync(0xffffffffu, ohi, 1) : __shfl_up_sync(0xffffffffu, ohi, 1);
            const Pair<T> pO = mul2(a.O.pair(COLOR, j), Pair<T>(olo, ohi));
            const Pair<T> pH = mul2(a.H.pair(COLOR, j), Pair<T>(hlo, hhi));
            const T nhi = j < J - 1 ? x.v[OC][j < J - 1 ? j + 1 : j][0] : above[f];
            const T slo = j > 0 ? x.v[OC][j > 0 ? j - 1 : 0][1] : below[f];
            const Pair<T> pN(a.N.v[COLOR][j][0] * ohi, a.N.v[COLOR][j][1] * nhi);
            const Pair<T> pS(a.S.v[COLOR][j][0] * slo, a.S.v[COLOR][j][1] * olo);
            // east first, then west
            const T t0 = COLOR == 0 ? (b.lo() + pO.lo()) + pH.lo() : (b.lo() + pH.lo()) + pO.lo();
            const T t1 = COLOR == 0 ? (b.hi() + pH.hi()) + pO.hi() : (b.hi() + pO.hi()) + pH.hi();
            const Pair<T> num = add2(add2(Pair<T>(t0, t1), pN), pS);
            const Pair<T> z = a.Z.pair(COLOR, j);
            Pair<T> quo = mul2(num, z);
            quo = fma2(fma2(quo, a.C.pair(COLOR, j), num), z, quo);
            n[f][j][0] = num.lo();
            n[f][j][1] = num.hi();
            q[f][j][0] = quo.lo();
            q[f][j][1] = quo.hi();
            key = max(key, max(far_key<RT::R>(n[f][j][0], q[f][j][0]), far_key<RT::R>(n[f][j][1], q[f][j][1])));
        }
    }
    if (force || key > span) {
        // A zero numerator needs nothing more: its quotient is a zero already
        // (only the sign may differ, which q - x and x + d erase).
        unsigned todo = 0;
#pragma unroll
        for (int f = 0; f < F; ++f)
#pragma unroll
            for (int i = 0; i < 2 * J; ++i)
                if (force || (far_key<RT::R>(n[f][i >> 1][i & 1], q[f][i >> 1][i & 1]) > span && n[f][i >> 1][i & 1] != (T)0))
                    todo |= 1u << (2 * J * f + i);
        if (todo) far_quotients<RT, T, COLOR, F>(a, n, q, todo, force);
    }
#pragma unroll
    for (int f = 0; f < F; ++f) {
        if (!act[f]) continue;  // uniform
        Cells<T, RT::R> &x = *xs[f];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const Pair<T> old = x.pair(COLOR, j);
            const Pair<T> e = fma2(old, minus, Pair<T>(q[f][j][0], q[f][j][1]));
            const Pair<T> d(relax[f] * e.lo(), relax[f] * e.hi());
            const Pair<T> nx = add2(old, d);
            x.v[COLOR][j][0] = nx.lo();
            x.v[COLOR][j][1] = nx.hi();
            if (SUM) {
                if (rown >> (2 * j) & 1u) acc[f][COLOR] += (double)d.lo() * (double)d.lo();
                if (rown >> (2 * j + 1) & 1u) acc[f][OC] += (double)d.hi() * (double)d.hi();
            }
        }
        row[f * RT::EX + COLOR * 32] = x.v[COLOR][0][0];
        row[f * RT::EX + RT::SIDE + OC * 32] = x.v[COLOR][J - 1][1];
    }
}

// What a lane knows of its place in a tile.
template <typename RT>
struct LanePlace {
    int gi, gj;            // global column of the lane's first cell, global row of its first row
    bool own0, own1;       // the lane's columns belong to the tile
    unsigned rown;         // rows that do
    int dist;              // rows between the warp's nearest row and the tile; large beyond the domain
    __device__ __forceinline__ LanePlace(const TileBox &t, int ny)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int a = 2 * lane, b = warp * RT::R;
        gi = t.gx0 + a;
        gj = t.gy0 + b;
        own0 = a >= t.ox0 && a < t.ox1;
        own1 = a + 1 >= t.ox0 && a + 1 < t.ox1;
        rown = 0;
#pragma unroll
        for (int r = 0; r < RT::R; ++r)
            if (b + r >= t.oy0 && b + r < t.oy1) rown |= 1u << r;
        dist = b + RT::R - 1 < t.oy0 ? t.oy0 - (b + RT::R - 1) : (b >= t.oy1 ? b - t.oy1 + 1 : 0);
        if (gj >= ny) dist = 1 << 20;
    }
};

// x = field[cell] of the lane's cells (`outside` beyond the domain); with
// only_halo, the tile's own cells keep their values.
template <typename RT, typename T, typename A>
__device__ __forceinline__ void load_cells(Cells<T, RT::R> &x, const A &field, const LanePlace<RT> &pl, int nx, int ny,
                                           bool only_halo, T outside)
{
#pragma unroll
    for (int r = 0; r < RT::R; ++r) {
        const int j = pl.gj + r;
        const bool ro = only_halo && (pl.rown >> r & 1u);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (ro && (k == 0 ? pl.own0 : pl.own1)) continue;
            x.at(r, k) = (j < ny && pl.gi + k < nx) ? field[pl.gi + k + nx * j] : outside;
        }
    }
}

template <typename RT, typename T, typename A>
__device__ __forceinline__ void store_own(const Cells<T, RT::R> &x, const A &field, const LanePlace<RT> &pl, int nx)
{
#pragma unroll
    for (int r = 0; r < RT::R; ++r) {
        if (!(pl.rown >> r & 1u)) continue;
        const int c = pl.gi + nx * (pl.gj + r);
        if (pl.own0) field[c] = x.at(r, 0);
        if (pl.own1) field[c + 1] = x.at(r, 1);
    }
}

// to = from on the tile's own cells.
template <typename RT, typename T, typename A>
__device__ __forceinline__ void store_other(const A &to, const A &from, const LanePlace<RT> &pl, int nx)
{
#pragma unroll
    for (int r = 0; r < RT::R; ++r) {
        if (!(pl.rown >> r & 1u)) continue;
        const int c = pl.gi + nx * (pl.gj + r);
        if (pl.own0) to[c] = from[c];
        if (pl.own1) to[c + 1] = from[c + 1];
    }
}

// Neighbours of a lane's cell k in row r; below, above: the exchange rows.
template <int R, typename T>
__device__ __forceinline__ T east_of(const Cells<T, R> &x, int r, int k)
{
    return k == 0 ? x.at(r, 1) : __shfl_down_sync(0xffffffffu, x.at(r, 0), 1);
}
template <int R, typename T>
__device__ __forceinline__ T west_of(const Cells<T, R> &x, int r, int k)
{
    return k == 1 ? x.at(r, 0) : __shfl_up_sync(0xffffffffu, x.at(r, 1), 1);
}
template <int R, typename T>
__device__ __forceinline__ T north_of(const Cells<T, R> &x, int r, int k, const T (&above)[2])
{
    return r < R - 1 ? x.at(r < R - 1 ? r + 1 : r, k) : above[k];
}
template <int R, typename T>
__device__ __forceinline__ T south_of(const Cells<T, R> &x, int r, int k, const T (&below)[2])
{
    return r > 0 ? x.at(r > 0 ? r - 1 : 0, k) : below[k];
}

// Cells beyond the domain hold x = 1 with no links, diagonal 1 and source 1, so
// their update changes nothing and its quotient stays in the safe range.
template <typename T>
constexpr T kOutside = (T)1;

// Reciprocals of the diagonals; returns whether a diagonal is outside the
// range of a precomputed reciprocal.
template <typename RT, typename T>
__device__ __forceinline__ bool set_reciprocals(Links<RT, T> &a)
{
    bool force = false;
#pragma unroll
    for (int r = 0; r < RT::R; ++r)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const T c = -a.C.at(r, k);
            a.Z.at(r, k) = (T)1 / c;
            force = force || !divisor_ok(c);
        }
    return force;
}

// Links, diagonal and sources of one cell, as mom_cell leaves them.
template <typename T>
struct MomCell {
    T E, W, N, S, C, bu, bv;
};

// The boundary fold-in of mom_cell (kernels.cuh:252-334).
template <typename T>
__device__ __forceinline__ void mom_fold(const Params<T> &P, int i, int j, MomCell<T> &m)
{
    const Geo<T> &g = P.g;
    T a[7] = {m.C, m.E, m.W, m.N, m.S, (T)0, (T)0}, b[3] = {m.bu, m.bv, (T)0};
    if (i == g.nx - 1) fold_face<T, 2>(P, EAST, AE, AW, g.bcv[EAST][0], g.bcv[EAST][1], (T)0, a, b);
    if (i == 0) {
        const T uin = (g.inlet && g.bc[WEST] == INLET) ? g.inlet[j] : g.bcv[WEST][0];
        fold_face<T, 2>(P, WEST, AW, AE, uin, g.bcv[WEST][1], (T)0, a, b);
    }
    if (j == g.ny - 1) fold_face<T, 2>(P, NORTH, AN, AS, g.bcv[NORTH][0], g.bcv[NORTH][1], (T)0, a, b);
    if (j == 0) fold_face<T, 2>(P, SOUTH, AS, AN, g.bcv[SOUTH][0], g.bcv[SOUTH][1], (T)0, a, b);
    m = {a[AE], a[AW], a[AN], a[AS], a[AC], b[0], b[1]};
}

// Momentum links, diagonal and sources of the lane's cells (kernels.cuh:97-334)
// from the faces and the pressure; the sources go to shared memory.  Uses the
// exchange rows of unknown 0 (two block barriers).  Returns the `force` flag of half_sweep.
template <typename RT, typename T>
__device__ __forceinline__ bool mom_links(const Params<T> &P, const Fields<T> &f, const LanePlace<RT> &pl,
                                          Links<RT, T> &a)
{
    constexpr int R = RT::R;
    const Geo<T> &g = P.g;
    const int nx = g.nx, ny = g.ny;
    // every load first: the barrier below would hold later ones back
    Cells<T, R> p;
    T fx[R][3], fy[R + 1][2];  // the faces west of the lane's columns and east of the last, south of its rows and north
    load_cells<RT, T>(p, f.p, pl, nx, ny, false, (T)0);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            fx[r][k] = pl.gj + r < ny && pl.gi + k <= nx ? f.uf[pl.gi + k + (nx + 1) * (pl.gj + r)] : (T)0;
#pragma unroll
    for (int r = 0; r <= R; ++r)
#pragma unroll
        for (int k = 0; k < 2; ++k)
            fy[r][k] = pl.gj + r <= ny && pl.gi + k < nx ? f.vf[pl.gi + k + nx * (pl.gj + r)] : (T)0;
    publish<RT, T>(p, 0);
    __syncthreads();
    const T *row = tile_smem<T>() + lane_row<RT>();
    const T pb[2] = {row[RT::SIDE - RT::W], row[RT::SIDE - RT::W + 32]}, pt[2] = {row[RT::W], row[RT::W + 32]};
    MomCell<T> cell[2 * R];
    Cells<T, R> bu, bv;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = pl.gj + r;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = pl.gi + k;
            const T pE = east_of<R, T>(p, r, k), pW = west_of<R, T>(p, r, k);
            const T pN = north_of<R, T>(p, r, k, pt), pS = south_of<R, T>(p, r, k, pb);
            const T pC = p.at(r, k), uw = fx[r][k], ue = fx[r][k + 1], vs = fy[r][k], vn = fy[r + 1][k];
            MomCell<T> &m = cell[2 * r + k];
            m.E = g.rho * min0(ue) * g.Ax - P.d.Dx;
            m.W = g.rho * min0(-uw) * g.Ax - P.d.Dx;
            m.N = g.rho * min0(vn) * g.Ay - P.d.Dy;
            m.S = g.rho * min0(-vs) * g.Ay - P.d.Dy;
            m.C = -(m.E + m.W + m.N + m.S);
            T lo = i > 0 ? pW : (g.closed[WEST] ? pC : (T)0), hi = i < nx - 1 ? pE : (g.closed[EAST] ? pC : (T)0);
            m.bu = (T)(0.5 * (double)(T)(lo - hi) * (double)g.Ax);
            lo = j > 0 ? pS : (g.closed[SOUTH] ? pC : (T)0);
            hi = j < ny - 1 ? pN : (g.closed[NORTH] ? pC : (T)0);
            m.bv = (T)(0.5 * (double)(T)(lo - hi) * (double)g.Ay);
        }
    }
    if (pl.gi == 0 || pl.gi + 2 >= nx || pl.gj == 0 || pl.gj + R >= ny) {
        // the lane has cells on the domain's edge (or beyond it)
        MomCell<T> tmp[2 * R];
#pragma unroll
        for (int q = 0; q < 2 * R; ++q) tmp[q] = cell[q];
#pragma unroll 1
        for (int q = 0; q < 2 * R; ++q) {
            const int i = pl.gi + (q & 1), j = pl.gj + (q >> 1);
            if (i < nx && j < ny) mom_fold<T>(P, i, j, tmp[q]);
            else tmp[q] = {(T)0, (T)0, (T)0, (T)0, kOutside<T>, kOutside<T>, kOutside<T>};
        }
#pragma unroll
        for (int q = 0; q < 2 * R; ++q) cell[q] = tmp[q];
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const MomCell<T> &m = cell[2 * r + k];
            T b3[3] = {m.bu, m.bv, (T)0};
            if (pl.gi + k < nx && pl.gj + r < ny) add_dc<T, 2>(P, f, pl.gi + k + nx * (pl.gj + r), b3);
            a.set(r, k, m.E, m.W, m.N, m.S, m.C);
            bu.at(r, k) = b3[0];
            bv.at(r, k) = b3[1];
        }
    put_cells<RT, T>(bu, RT::SRC);
    put_cells<RT, T>(bv, RT::SRC + RT::LEN);
    __syncthreads();  // the exchange rows are free again
    return set_reciprocals<RT, T>(a);
}

// The momentum diagonal of the tile's own cells and its reciprocal to global
// memory (the reciprocals serve Rhie-Chow, the p' links and the corrections).
template <typename RT, typename T, typename A>
__device__ __forceinline__ void store_diagonal(const Links<RT, T> &a, const A &ac, const A &rac, const LanePlace<RT> &pl,
                                               int nx)
{
    Cells<T, RT::R> c;
#pragma unroll
    for (int r = 0; r < RT::R; ++r) {
        c.at(r, 0) = -a.C.at(r, 0);
        c.at(r, 1) = -a.C.at(r, 1);
    }
    store_own<RT, T>(c, ac, pl, nx);
    store_own<RT, T>(a.Z, rac, pl, nx);
}

// p' links, diagonal and source of the lane's cells from the reciprocals of the
// momentum diagonal (kernels.cuh:517-537: interior faces only); as mom_links.
template <typename RT, typename T>
__device__ __forceinline__ bool pc_links(const Params<T> &P, const Fields<T> &f, const LanePlace<RT> &pl,
                                         Links<RT, T> &a)
{
    constexpr int R = RT::R;
    const Geo<T> &g = P.g;
    const int nx = g.nx, ny = g.ny;
    Cells<T, R> rr, b;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = pl.gi + k, j = pl.gj + r;
            const bool in = i < nx && j < ny;
            const int c = i + nx * j;
            rr.at(r, k) = in ? f.rac[c] : (T)0;
            b.at(r, k) = in ? f.sp[c] : kOutside<T>;
        }
    put_cells<RT, T>(b, RT::SRC);
    publish<RT, T>(rr, 0);
    __syncthreads();
    const T *row = tile_smem<T>() + lane_row<RT>();
    const T rb[2] = {row[RT::SIDE - RT::W], row[RT::SIDE - RT::W + 32]}, rt[2] = {row[RT::W], row[RT::W + 32]};
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = pl.gj + r;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = pl.gi + k;
            const T rE = east_of<R, T>(rr, r, k), rW = west_of<R, T>(rr, r, k);
            const T rN = north_of<R, T>(rr, r, k, rt), rS = south_of<R, T>(rr, r, k, rb);
            const T rc = rr.at(r, k);
            const bool in = i < nx && j < ny;
            const T e = in && i < nx - 1 ? (T)(P.d.Kx * (double)(T)(rc + rE)) : (T)0;
            const T w = in && i > 0 ? (T)(P.d.Kx * (double)(T)(rc + rW)) : (T)0;
            const T n = in && j < ny - 1 ? (T)(P.d.Ky * (double)(T)(rc + rN)) : (T)0;
            const T s = in && j > 0 ? (T)(P.d.Ky * (double)(T)(rc + rS)) : (T)0;
            a.set(r, k, e, w, n, s, in ? -(e + w + n + s) : kOutside<T>);
        }
    }
    __syncthreads();
    return set_reciprocals<RT, T>(a);
}

// p' = 0 (outside cells as load_cells leaves them).
template <typename RT, typename T>
__device__ __forceinline__ void zero_cells(Cells<T, RT::R> &x, const LanePlace<RT> &pl, int nx, int ny)
{
#pragma unroll
    for (int r = 0; r < RT::R; ++r)
#pragma unroll
        for (int k = 0; k < 2; ++k) x.at(r, k) = (pl.gj + r < ny && pl.gi + k < nx) ? (T)0 : kOutside<T>;
}

// Runs ns[f] sweeps of the F unknowns x[f].  After half sweep h of 2*ns[f] only
// rows within 2*ns[f]-1-h of the tile can still reach it; warps farther out only
// wait.  With SUM, sred[(f*ks + s)*NT + tid] receives (add: is increased by) the
// thread's sum of squared changes of sweep s over the tile's own cells.
template <typename RT, typename T, int F, bool SUM>
__device__ __forceinline__ void sweeps(Cells<T, RT::R> *const (&x)[F], const Links<RT, T> &a,
                                       const LanePlace<RT> &pl, const T (&relax)[F], bool force, const int (&ns)[F],
                                       int ks, bool add, double *sred)
{
    const int nmax = F == 2 ? max(ns[0], ns[F - 1]) : ns[0];
#pragma unroll 1
    for (int s = 0; s < nmax; ++s) {
        double acc[F][2];
        bool act[F], any = false;
#pragma unroll
        for (int f = 0; f < F; ++f) {
            acc[f][0] = acc[f][1] = 0.0;
            act[f] = pl.dist <= 2 * (ns[f] - s) - 1;  // never when ns[f] <= s
            any = any || act[f];
        }
        if (any) half_sweep<RT, T, 0, F, SUM>(x, a, relax, act, force, pl.rown, acc);
        __syncthreads();
        any = false;
#pragma unroll
        for (int f = 0; f < F; ++f) {
            act[f] = pl.dist <= 2 * (ns[f] - s) - 2;
            any = any || act[f];
        }
        if (any) half_sweep<RT, T, 1, F, SUM>(x, a, relax, act, force, pl.rown, acc);
        if (SUM) {
#pragma unroll
            for (int f = 0; f < F; ++f) {
                double *p = sred + (f * ks + s) * RT::NT + threadIdx.x;
                const double t = (pl.own0 ? acc[f][0] : 0.0) + (pl.own1 ? acc[f][1] : 0.0);
                *p = add ? *p + t : t;
            }
        }
        __syncthreads();
    }
}

// ns sweeps of one unknown.
template <typename RT, typename T>
__device__ __forceinline__ void sweeps1(Cells<T, RT::R> &x, const Links<RT, T> &a, const LanePlace<RT> &pl, T relax, bool force, int ns,
                                        int ks, bool sum, bool add, double *sred)
{
    Cells<T, RT::R> *const xs[1] = {&x};
    const T rl[1] = {relax};
    const int n[1] = {ns};
    if (sum) sweeps<RT, T, 1, true>(xs, a, pl, rl, force, n, ks, add, sred);
    else sweeps<RT, T, 1, false>(xs, a, pl, rl, force, n, ks, add, sred);
}

// ns0 sweeps of u and ns1 of v, which share the links (the sums of v at
// sred + ks*NT).
template <typename RT, typename T>
__device__ __forceinline__ void sweeps2(Cells<T, RT::R> &u, Cells<T, RT::R> &v, const Links<RT, T> &a,
                                        const LanePlace<RT> &pl, T ru, T rv, bool force, int ns0, int ns1, int ks,
                                        bool sum, bool add, double *sred)
{
    Cells<T, RT::R> *const xs[2] = {&u, &v};
    const T rl[2] = {ru, rv};
    const int n[2] = {ns0, ns1};
    if (sum) sweeps<RT, T, 2, true>(xs, a, pl, rl, force, n, ks, add, sred);
    else sweeps<RT, T, 2, false>(xs, a, pl, rl, force, n, ks, add, sred);
}

// The Rhie-Chow face velocity of rc_face with the reciprocals of the diagonals
// given (1/(4a) is 1/a scaled, so the two quotients need no division either).
template <typename T>
__device__ __forceinline__ T rc_face_known(T uL, T uR, T aCL, T aCR, T rL, T rR, T pLL, T pL, T pR, T pRR, T A)
{
    const double t0 = 0.5 * (double)(T)(uL + uR);
    const T t1 = quot_known((pR - pLL) * A, (T)4 * aCL, (T)0.25 * rL);
    const T t2 = quot_known((pRR - pL) * A, (T)4 * aCR, (T)0.25 * rR);
    const T sr = rL + rR;
    const double t3 = 0.5 * (double)sr * (double)(T)(pL - pR) * (double)A;
    return (T)(t0 + (double)t1 + (double)t2 + t3);
}

// x / d for x < 65536 and 2 <= d < 65536.
struct SmallDiv {
    unsigned d, inv;
    __device__ __forceinline__ explicit SmallDiv(int n) : d((unsigned)n), inv(0xffffffffu / (unsigned)n + 1u) {}
    __device__ __forceinline__ int div(int x) const { return (int)__umulhi((unsigned)x, inv); }
};

// This CTA's column sums of sred (NT values per column, fixed order) into
// partials[col*G + blockIdx.x], or straight into tot when there is one CTA;
// call with every thread after a barrier.
template <int NT>
static __device__ __noinline__ void column_partials(const double *sred, int ncol, double *partials, int G, double *tot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = warp; c < ncol; c += NT / 32) {
        double x = 0.0;
#pragma unroll 8
        for (int q = 0; q < NT / 32; ++q) x += sred[c * NT + q * 32 + lane];
        x = warp_sum(x);
        if (lane == 0) {
            if (G == 1) tot[c] = x;
            else partials[(size_t)c * G + blockIdx.x] = x;
        }
    }
}

}  // namespace ifc
