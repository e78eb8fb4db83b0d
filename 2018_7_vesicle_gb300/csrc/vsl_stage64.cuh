// vsl_stage64.cuh -- stage kernels of the plain FP64 form on cheaper arithmetic with the
// same results as the per-node functions of vsl_fused.cuh: bit for bit but for the sign of a zero
// (a transport stage adds no zero of the side it does not evaluate).
//
// What bounds these kernels is the FP64 pipe: two lanes per SM and clock on GB300, 1/64 of
// the FP32 rate, so a warp's FP64 instruction occupies it for 16 cycles and everything else
// (loads, integer work, selects) is free beside it.  A node of the per-node form costs about
// 1100 FP64 instructions per stage: 24 quotients per axis as general divisions, and both
// one-sided derivatives of every axis.  Here:
//   * quotients are the short ones of vsl_short64.cuh: three instructions by the grid spacing,
//     one shared reciprocal per divisor in the WENO weights;
//   * multiplications by powers of two ride in an FMA, which rounds the same;
//   * transport evaluates only the upwind side of an axis (the other is multiplied by zero),
//     and the Godunov norm only the sides whose three candidate values do not all have the
//     sign that the maximum with zero discards (the weights are positive, so the
//     reconstruction lies between the candidates);
//   * nodes with an interface distance ("flagged", the classification's list) are updated by
//     band blocks at the front of the same launch, so that no warp of the others runs the
//     nonuniform stencils for a few of its lanes; the WENO kinds run them as tasks sorted by
//     stencil kind (vsl_band.cuh), on the same short quotients.
//   * scaled differences are formed once per tile and shared through shared memory.
// 288 / 370 FP64 instructions per node and stage (transport / norm, band included; ncu), the pipe
// 86% busy.  Per stage at 128^3 on GB300: advection 1.13 ms, extension 1.17 ms, reinitialization
// 1.40 ms (3.2, 3.7 and 3.7 ms one node per thread with general quotients).
//
// The sequences above need operands away from overflow and underflow.  A node whose stencil
// holds a value that is neither zero nor of magnitude 2^-400 .. 2^100 (infinities and NaN
// among them), and a reinitialization node that has a sign change but no distance flag, takes
// the general code.  Spacings outside 2^-60 .. 2^60 send every node there.
#pragma once

#include <algorithm>
#include <cmath>

#include "vsl_band.cuh"
#include "vsl_fused.cuh"
#include "vsl_short64.cuh"

namespace vsl {
namespace {

// zero, or of magnitude 2^-400 .. 2^100
__device__ __forceinline__ bool ordinary(double x) { return within64(x, -400, 100); }
__device__ __forceinline__ bool sign_bit(double x) { return __double2hiint(x) < 0; }
__device__ __forceinline__ double flip(double x, bool neg)
{
    return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
}

// ---------------------------------------------------------------------------------------
// WENO5 (weno5_plain, the same roundings)
// ---------------------------------------------------------------------------------------

// the three candidate values of the window v1..v5
__device__ __forceinline__ void candidates64(double v1, double v2, double v3, double v4, double v5, double q[3])
{
    q[0] = 1. / 3. * v1 - 7. / 6. * v2 + 11. / 6. * v3;
    q[1] = 5. / 6. * v3 - 1. / 6. * v2 + 1. / 3. * v4;
    q[2] = 1. / 3. * v3 + 5. / 6. * v4 - 1. / 6. * v5;
}

// the weighted value of the candidates q of the window v1..v5
__device__ __forceinline__ double weighted64(double v1, double v2, double v3, double v4, double v5, const double q[3])
{
    const double t3 = 3.0 * v3;
    const double s1 = __fma_rn(0.25, sqr(__fma_rn(-4.0, v2, v1) + t3), 13. / 12. * sqr(__fma_rn(-2.0, v2, v1) + v3));
    const double s2 = __fma_rn(0.25, sqr(v2 - v4), 13. / 12. * sqr(__fma_rn(-2.0, v3, v2) + v4));
    const double s3 = __fma_rn(0.25, sqr(__fma_rn(-4.0, v4, t3) + v5), 13. / 12. * sqr(__fma_rn(-2.0, v4, v3) + v5));
    const double b1 = sqr(s1 + 1e-6), b2 = sqr(s2 + 1e-6), b3 = sqr(s3 + 1e-6);
    const double a1 = quotient(0.1, b1, reciprocal(b1));
    const double a2 = quotient(0.6, b2, reciprocal(b2));
    const double a3 = quotient(0.3, b3, reciprocal(b3));
    const double tot = a1 + a2 + a3, r = reciprocal(tot);
    return quotient(a1, tot, r) * q[0] + quotient(a2, tot, r) * q[1] + quotient(a3, tot, r) * q[2];
}

// D- from the scaled differences v1..v5 of its window; with the mirrored window of the node's six
// differences u, upwind64(u[5], u[4], u[3], u[2], u[1]), D+
__device__ __forceinline__ double upwind64(double v1, double v2, double v3, double v4, double v5)
{
    double q[3];
    candidates64(v1, v2, v3, v4, v5, q);
    return weighted64(v1, v2, v3, v4, v5, q);
}

// max(0, D-, -D+) of the scaled differences u of a line, with both derivatives negated where neg
// (godunov_norm's term before the square)
__device__ __forceinline__ double godunov_side64(const double u[6], bool neg)
{
    double qb[3], qf[3];
    {
        const double s1 = 1. / 6. * u[1], s4 = 1. / 6. * u[4], h2 = 1. / 3. * u[2], h3 = 1. / 3. * u[3];
        const double f2 = 5. / 6. * u[2], f3 = 5. / 6. * u[3];
        qb[0] = 1. / 3. * u[0] - 7. / 6. * u[1] + 11. / 6. * u[2];
        qb[1] = f2 - s1 + h3;
        qb[2] = h2 + f3 - s4;
        qf[0] = 1. / 3. * u[5] - 7. / 6. * u[4] + 11. / 6. * u[3];
        qf[1] = f3 - s4 + h2;
        qf[2] = h3 + f2 - s1;
    }
    // D- counts where positive (neg: negative), D+ where negative (neg: positive)
    const bool b = neg ? sign_bit(qb[0]) || sign_bit(qb[1]) || sign_bit(qb[2])
                       : !(sign_bit(qb[0]) && sign_bit(qb[1]) && sign_bit(qb[2]));
    const bool f = neg ? !(sign_bit(qf[0]) && sign_bit(qf[1]) && sign_bit(qf[2]))
                       : sign_bit(qf[0]) || sign_bit(qf[1]) || sign_bit(qf[2]);
    const double q[3] = {b ? qb[0] : qf[0], b ? qb[1] : qf[1], b ? qb[2] : qf[2]};
    double e = weighted64(b ? u[0] : u[5], b ? u[1] : u[4], b ? u[2] : u[3], b ? u[3] : u[2], b ? u[4] : u[1], q);
    e = flip(e, neg == b);
    e = (b || f) && !sign_bit(e) ? e : 0.0;
    if (b && f) {
        const double g = flip(weighted64(u[5], u[4], u[3], u[2], u[1], qf), !neg);
        e = g > e ? g : e;
    }
    return e;
}

// ---------------------------------------------------------------------------------------
// quadratic ENO (eno2_pair with r1 = l1 = h, the same roundings)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ double minmod64(double x, double y)
{
    const long long a = __double_as_longlong(x), b = __double_as_longlong(y), m = 0x7fffffffffffffffLL;
    const double s = (a & m) < (b & m) ? x : y;
    return (a ^ b) < 0 ? 0.0 : s;  // of opposite sign (or one a zero)
}

// Backward quadratic-ENO derivative at t3 of the points t1, t2, t3 (t3 the node); the mirrored
// points give the forward one negated.  c: the second difference at the node (the same sum for
// both sides), h2 = h * h, rh2 its reciprocal.
__device__ __forceinline__ double eno2_back64(double t1, double t2, double t3, double c, double h, double rh,
                                              double h2, double rh2)
{
    const double l = __fma_rn(-2.0, t2, t3) + t1;
    return quotient(t3 - t2, h, rh) + (0.5 * h) * quotient(minmod64(c, l), h2, rh2);
}

// ---------------------------------------------------------------------------------------
// the stage kernel
// ---------------------------------------------------------------------------------------
__host__ __device__ constexpr bool band_kind64(int kind) { return kind != K64_ADVECT; }

struct Args64 {
    Stage64 st;
    Ptr3<double> w;  // VELOCITY: the velocity written
    int band_blocks;
    Grid g;
    double h[3], rh[3], h2[3], rh2[3];
    double dt_uniform;  // 0.3 * min spacing: the pseudo time step of a node without a flag
    double floor;       // VELOCITY: the floor of |grad phi|
    double tiny[3];     // 2^-80 h: the least gap of a stencil on short quotients
    bool ordinary;      // the spacings are within the range of the short sequences
};

// One node by the general code (vsl_fused.cuh): band nodes, and the nodes whose stencil the
// short sequences do not take.
template <int KIND, int STAGE, bool ENO3> __device__ __forceinline__ void general_node64(const Args64 &a, long long c)
{
    const Grid &g = a.g;
    int i, j, k;
    node_of(g, c, i, j, k);
    if constexpr (KIND == K64_REINIT) {
        reinit_node<double, ENO3, false>(a.st.phi_s, a.st.phi_n, a.st.out, a.st.flags, a.st.d, g, STAGE, i, j, k);
    } else if constexpr (KIND == K64_EXTEND) {
        extend_node<double, ENO3, false>(a.st.phi_s, a.st.phi_n, a.st.out, a.st.flags, a.st.d, a.st.cp, a.st.v, g, STAGE, i, j, k);
    } else if constexpr (KIND == K64_ADVECT) {
        advect_node<double, false>(a.st.phi_s, a.st.phi_n, a.st.out, a.st.v, a.st.speed, a.st.dt, g, STAGE, i, j, k);
    } else if constexpr (KIND == K64_VELOCITY) {
        Ptr3<double> w = a.w;
        extension_velocity_node<double, ENO3>(a.st.phi_s, a.st.flags, a.st.d, w, g, a.floor, i, j, k);
    } else if constexpr (KIND == K64_ENO2) {
        enork2_extend_node<double>(a.st.phi_s, a.st.phi_n, a.st.out, a.st.flags, a.st.d, a.st.cp, a.st.v, g, STAGE, i, j, k);
    } else {
        enork2_reinit_node<double>(a.st.phi_s, a.st.phi_n, a.st.out, a.st.flags, a.st.d, g, STAGE, i, j, k);
    }
}
template <int KIND, int STAGE, bool ENO3> __device__ __noinline__ void general_call64(const Args64 &a, long long c)
{
    general_node64<KIND, STAGE, ENO3>(a, c);
}

// ---------------------------------------------------------------------------------------
// the band of the WENO kinds as sorted tasks
// ---------------------------------------------------------------------------------------

// One side of weno_nonuniform_pair at xs[3].  R: double, or Short64 where every value is ordinary.
template <typename R> __device__ __forceinline__ double nonuniform_side64(const double xs[7], const double hs[7], bool back)
{
    R x[7], dd[6];
#pragma unroll
    for (int m = 0; m < 7; ++m) x[m] = R(xs[m]);
#pragma unroll
    for (int m = 0; m < 6; ++m) dd[m] = (R(hs[m + 1]) - R(hs[m])) / (x[m + 1] - x[m]);
    if constexpr (std::is_same<R, double>::value)
        return back ? weno_nonuniform_back(x, dd) : weno_nonuniform_fore(x, dd);
    else
        return back ? weno_nonuniform_back(x, dd).v : weno_nonuniform_fore(x, dd).v;
}
__device__ __noinline__ void nonuniform_general64(const double xs[7], const double hs[7], double &df, double &db)
{
    weno_nonuniform_pair(xs, hs, df, db);
}

constexpr int CHUNK64 = 64;  // nodes per chunk: 192 axes over 128 threads
constexpr int BY64 = 4;      // columns per block (128 threads)

// Ops of run_band for the reinitialization (NORM) and the extension.  The derivatives of both
// sides are stored where both were evaluated; the Godunov term of a uniform axis
// (godunov_side64) is stored as the side that the norm takes it from.
template <int STAGE, bool ENO3, bool NORM> struct Band64 {
    using Chunk = BandChunk<double, CHUNK64>;
    const Args64 &a;
    __device__ __forceinline__ unsigned node(unsigned t) const { return a.st.flagged.idx[t]; }
    __device__ __forceinline__ const Grid &grid() const { return a.g; }
    __device__ __forceinline__ uint8_t flags(unsigned c) const { return __ldg(a.st.flags + c); }
    __device__ __forceinline__ unsigned kinds(const Chunk &ch, int node, int ax) const
    {
        const unsigned c = ch.c[node];
        bool iface;
        if constexpr (NORM) {
            iface = sign_change(a.st.phi_s, band_line(ch, a.g, node, ax));
        } else {
            const uint8_t fl = ch.fl[node];
            const double h = a.h[ax];
            iface = flagged_distance(fl, 2 * ax, a.st.d, c, h) < h || flagged_distance(fl, 2 * ax + 1, a.st.d, c, h) < h;
        }
        if (!iface) return 1u << BT_UNIFORM;
        if (ENO3) return 1u << BT_FORE;  // the ENO3 pair is one task
        if (NORM) return (1u << BT_FORE) | (1u << BT_BACK);
        return sign_bit(__ldg(a.st.v.p[ax] + c)) ? 1u << BT_FORE : 1u << BT_BACK;
    }
    __device__ __forceinline__ void eval(Chunk &ch, int kind, int node, int ax) const
    {
        const unsigned c = ch.c[node];
        const uint8_t fl = ch.fl[node];
        const AxisLine L = band_line(ch, a.g, node, ax);
        double p[7];
        load_line7(a.st.phi_s, L, p);
        bool ok = a.ordinary;
#pragma unroll
        for (int m = 0; m < 7; ++m) ok = ok && ordinary(p[m]);
        const double h = a.h[ax];
        double &df = ch.df[ax][node], &db = ch.db[ax][node];
        if (kind == BT_UNIFORM) {
            double u[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) u[m] = quotient(p[m + 1] - p[m], h, a.rh[ax]);
            if (!ok) {
                weno5_pair_plain(p, h, df, db);
            } else if constexpr (NORM) {
                const bool neg = fl & MASK_BIT;
                (neg ? df : db) = godunov_side64(u, neg);
            } else {
                const bool fore = sign_bit(__ldg(a.st.v.p[ax] + c));
                (fore ? df : db) = upwind64(fore ? u[5] : u[0], fore ? u[4] : u[1], fore ? u[3] : u[2],
                                            fore ? u[2] : u[3], fore ? u[1] : u[4]);
            }
            return;
        }
        const double r1 = flagged_distance(fl, 2 * ax, a.st.d, c, h);
        const double l1 = flagged_distance(fl, 2 * ax + 1, a.st.d, c, h);
        double hf = 0.0, hb = 0.0;
        if constexpr (!NORM) {
            hf = r1 < h ? __ldg(a.st.cp.p[2 * ax] + c) : 0.0;
            hb = l1 < h ? __ldg(a.st.cp.p[2 * ax + 1] + c) : 0.0;
            ok = ok && ordinary(hf) && ordinary(hb);
        }
        double xs[7], hs[7];
        insert_interface(p, r1, l1, h, hf, hb, xs, hs);
        if constexpr (ENO3) {
            eno3_nonuniform_pair(xs, hs, df, db);
        } else {
            // gaps below 2^-80 h would leave the range of the short quotients
            const double tiny = a.tiny[ax];
            ok = ok && xs[4] > tiny && xs[5] - xs[4] > tiny && -xs[2] > tiny && xs[2] - xs[1] > tiny;
            const bool back = kind == BT_BACK;
            if (ok)
                (back ? db : df) = nonuniform_side64<Short64>(xs, hs, back);
            else if (NORM)
                (back ? db : df) = nonuniform_side64<double>(xs, hs, back);
            else
                nonuniform_general64(xs, hs, df, db);  // both sides, as the sum reads them
        }
    }
    __device__ __forceinline__ void finish(const Chunk &ch, int node) const
    {
        const unsigned c = ch.c[node];
        const uint8_t fl = ch.fl[node];
        double step = 0.0;
        if (!(fl & FIXED_BIT)) {
            const double dt = pseudo_dt(fl, a.st.d, c, a.h[0], a.h[1], a.h[2]);
            if constexpr (NORM) {
                const bool neg = fl & MASK_BIT;
                const double gn = godunov_norm(neg, ch.df[0][node], ch.db[0][node], ch.df[1][node], ch.db[1][node],
                                               ch.df[2][node], ch.db[2][node]);
                step = (gn - 1.0) * dt * (neg ? -1.0 : 1.0);
            } else {
                step = upwind_dot(__ldg(a.st.v.p[0] + c), __ldg(a.st.v.p[1] + c), __ldg(a.st.v.p[2] + c),
                                  ch.df[0][node], ch.db[0][node], ch.df[1][node], ch.db[1][node], ch.df[2][node],
                                  ch.db[2][node]) *
                       dt;
            }
        }
        const double pn = STAGE == 0 ? 0.0 : __ldg(a.st.phi_n + c);
        a.st.out[c] = rk3_combine(STAGE, pn, __ldg(a.st.phi_s + c) - step);
    }
};

// The band blocks at the front of a launch (their chains are the longest); false for a tile block,
// with b then the tile's number.
template <int KIND, int STAGE, bool ENO3> __device__ __forceinline__ bool band_block64(const Args64 &a, unsigned &b)
{
    if constexpr (!band_kind64(KIND)) return false;
    if (b >= (unsigned)a.band_blocks) {
        b -= (unsigned)a.band_blocks;
        return false;
    }
    const unsigned nt = BX * BY64, n = *a.st.flagged.count, tid = threadIdx.y * BX + threadIdx.x;
    if constexpr (KIND == K64_REINIT || KIND == K64_EXTEND) {
        using Ops = Band64<STAGE, ENO3, KIND == K64_REINIT>;
        __shared__ typename Ops::Chunk ch;
        run_band<BX * BY64>(Ops{a}, ch, n, b, (unsigned)a.band_blocks, (int)tid);
    } else {
        for (unsigned t = b * nt + tid; t < n; t += (unsigned)a.band_blocks * nt)
            general_node64<KIND, STAGE, ENO3>(a, a.st.flagged.idx[t]);
    }
    return true;
}

// The WENO kinds: a block of 32 x 4 threads owns a tile of 32 rows x 4 columns x KZ pages.  Each
// scaled difference of the tile is formed once, in shared memory (a thread per difference), and
// read by the five or six nodes whose windows hold it: 28 FP64 instructions per node at KZ = 2
// instead of 60 (transport) or 72 (norm).  If any value of the tile's stencils is not ordinary,
// its nodes take the general code.
template <int KIND, int STAGE, bool ENO3, int KZ>
__global__ void __launch_bounds__(BX *BY64, 4) k_weno64(const __grid_constant__ Args64 a)
{
    const Grid &g = a.g;
    unsigned b = blockIdx.x;
    if (band_block64<KIND, STAGE, ENO3>(a, b)) return;
    const unsigned nx = (unsigned)(g.rows + BX - 1) / BX, ny = (unsigned)(g.cols + BY64 - 1) / BY64;
    const unsigned bz = b / (nx * ny), by = (b - bz * nx * ny) / nx, bx = b - (bz * ny + by) * nx;
    const int i0 = (int)bx * BX, j0 = (int)by * BY64, k0 = (int)bz * KZ;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * BX + tx;
    // differences along x between columns j0 + q - 3 and j0 + q - 2, along y between rows
    // i0 + q - 3 and i0 + q - 2, along z between pages k0 + q - 3 and k0 + q - 2 (all clamped)
    constexpr int NX = BY64 + 5, NY = BX + 5, NZ = KZ + 5;
    __shared__ double ux[KZ][NX][BX], uy[KZ][BY64][NY], uz[NZ][BY64][BX];
    const unsigned rows = (unsigned)g.rows, plane = (unsigned)g.plane;
    auto at = [&](int i, int j, int k) {
        return __ldg(a.st.phi_s + ((unsigned)clampi(k, g.pges) * plane + (unsigned)clampi(j, g.cols) * rows +
                                   (unsigned)clampi(i, g.rows)));
    };
    bool ok = a.ordinary;
    auto scaled = [&](double lo, double hi, int ax) {
        ok = ok && ordinary(lo) && ordinary(hi);
        return quotient(hi - lo, a.h[ax], a.rh[ax]);
    };
#pragma unroll 1
    for (int r = ty; r < KZ * NX; r += BY64) {
        const int kk = r / NX, q = r - kk * NX;
        ux[kk][q][tx] = scaled(at(i0 + tx, j0 + q - 3, k0 + kk), at(i0 + tx, j0 + q - 2, k0 + kk), AX_X);
    }
#pragma unroll 1
    for (int e = tid; e < KZ * BY64 * NY; e += BX * BY64) {
        const int r = e / NY, q = e - r * NY, kk = r / BY64, jj = r - kk * BY64;
        uy[kk][jj][q] = scaled(at(i0 + q - 3, j0 + jj, k0 + kk), at(i0 + q - 2, j0 + jj, k0 + kk), AX_Y);
    }
#pragma unroll 1
    for (int q = 0; q < NZ; ++q)
        uz[q][ty][tx] = scaled(at(i0 + tx, j0 + ty, k0 + q - 3), at(i0 + tx, j0 + ty, k0 + q - 2), AX_Z);
    ok = __syncthreads_and(ok);
    const int i = i0 + tx, j = j0 + ty;
    if (i >= g.rows || j >= g.cols) return;
#pragma unroll 1
    for (int kk = 0; kk < KZ && k0 + kk < g.pges; ++kk) {
        const int k = k0 + kk;
        const long long c = node_index(g, i, j, k);
        uint8_t fl = 0;
        if constexpr (band_kind64(KIND)) {
            fl = __ldg(a.st.flags + c);
            if (fl & 0x3F) continue;  // a band node
        }
        bool general = !ok;
        const double ps = __ldg(a.st.phi_s + c);
        if constexpr (KIND == K64_REINIT) {
            // a sign change next to a node without a distance: the general code decides
            const int hi = __double2hiint(ps);
            general = general || (hi ^ __double2hiint(at(i - 1, j, k))) < 0 || (hi ^ __double2hiint(at(i + 1, j, k))) < 0 ||
                      (hi ^ __double2hiint(at(i, j - 1, k))) < 0 || (hi ^ __double2hiint(at(i, j + 1, k))) < 0 ||
                      (hi ^ __double2hiint(at(i, j, k - 1))) < 0 || (hi ^ __double2hiint(at(i, j, k + 1))) < 0;
        }
        if (general) {
            general_call64<KIND, STAGE, ENO3>(a, c);
            continue;
        }
        auto diff = [&](int ax, int m) {
            return ax == AX_X ? ux[kk][ty + m][tx] : (ax == AX_Y ? uy[kk][ty][tx + m] : uz[kk + m][ty][tx]);
        };
        const bool neg = fl & MASK_BIT;
        double step = 0.0;
        if constexpr (KIND == K64_REINIT) {
            double e[3];
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                double u[6];
#pragma unroll
                for (int m = 0; m < 6; ++m) u[m] = diff(ax, m);
                e[ax] = godunov_side64(u, neg);
            }
            const double gn = norm_root(add_rn(add_rn(sqr(e[0]), sqr(e[1])), sqr(e[2])));
            step = flip((gn - 1.0) * a.dt_uniform, neg);
        } else {
            // one side of each axis: the upwind one of a transport, sum_ax min(0, v) D+ + max(0, v) D-,
            // or the one toward the smaller neighbour of the extension velocity
            double tr = 0.0, n[3];
            const double sp = KIND == K64_ADVECT && a.st.speed ? __ldg(a.st.speed + c) : 1.0;
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                double v = 0.0;
                bool fore;
                if constexpr (KIND == K64_VELOCITY) {
                    const double pm = at(i - (ax == AX_Y), j - (ax == AX_X), k - (ax == AX_Z));
                    const double pp = at(i + (ax == AX_Y), j + (ax == AX_X), k + (ax == AX_Z));
                    fore = fabs(pp) < fabs(pm);
                } else {
                    v = __ldg(a.st.v.p[ax] + c);
                    if (KIND == K64_ADVECT && a.st.speed) v = sp * v;
                    fore = sign_bit(v);
                }
                // the window by index arithmetic: u[0..4], or u[5..1]
                const int o = fore ? 5 : 0, d = fore ? -1 : 1;
                n[ax] = upwind64(diff(ax, o), diff(ax, o + d), diff(ax, o + 2 * d), diff(ax, o + 3 * d), diff(ax, o + 4 * d));
                tr = tr + v * n[ax];
            }
            if constexpr (KIND == K64_VELOCITY) {
                const double grad = vmax(sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]), a.floor);
                const double s = ps > 0.0 ? 1.0 : (ps < 0.0 ? -1.0 : 0.0);
#pragma unroll
                for (int ax = 0; ax < 3; ++ax) a.w.p[ax][c] = s * (n[ax] / grad);
                continue;
            }
            step = KIND == K64_ADVECT ? __ldg(a.st.dt) * tr : tr * a.dt_uniform;
        }
        if (band_kind64(KIND) && (fl & FIXED_BIT)) step = 0.0;
        const double pn = STAGE == 0 ? 0.0 : __ldg(a.st.phi_n + c);
        a.st.out[c] = rk3_combine(STAGE, pn, ps - step);
    }
}

// The ENORK2 kinds: one node per thread.
template <int KIND, int STAGE>
__global__ void __launch_bounds__(BX *BY64, 4) k_eno64(const __grid_constant__ Args64 a)
{
    const Grid &g = a.g;
    unsigned b = blockIdx.x;
    if (band_block64<KIND, STAGE, false>(a, b)) return;
    const unsigned nx = (unsigned)(g.rows + BX - 1) / BX, ny = (unsigned)(g.cols + BY64 - 1) / BY64;
    const unsigned bz = b / (nx * ny), by = (b - bz * nx * ny) / nx, bx = b - (bz * ny + by) * nx;
    const int i = (int)(bx * BX + threadIdx.x), j = (int)(by * BY64 + threadIdx.y), k = (int)bz;
    if (i >= g.rows || j >= g.cols) return;
    const long long c = node_index(g, i, j, k);
    const uint8_t fl = __ldg(a.st.flags + c);
    if (fl & 0x3F) return;  // a band node
    const double ps = __ldg(a.st.phi_s + c);
    bool ok = a.ordinary && ordinary(ps);
    double p[3][7];  // of each line the points 1 .. 5
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const AxisLine L = axis_line(g, i, j, k, ax);
#pragma unroll
        for (int s = 1; s < 6; ++s) {
            p[ax][s] = s == 3 ? ps : __ldg(a.st.phi_s + L.base + (long long)clampi(L.c + s - 3, L.n) * L.stride);
            if (s != 3) ok = ok && ordinary(p[ax][s]);
        }
    }
    if (!ok) {
        general_call64<KIND, STAGE, false>(a, c);
        return;
    }
    double step;
    if constexpr (KIND == K64_ENO2) {
        // the upwind side alone
        double tr = 0.0;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const double v = __ldg(a.st.v.p[ax] + c);
            const bool fore = sign_bit(v);
            const double c2 = __fma_rn(-2.0, ps, p[ax][2]) + p[ax][4];
            const double D = eno2_back64(fore ? p[ax][5] : p[ax][1], fore ? p[ax][4] : p[ax][2], ps, c2, a.h[ax],
                                         a.rh[ax], a.h2[ax], a.rh2[ax]);
            tr = tr + v * flip(D, fore);
        }
        step = tr * a.dt_uniform;
    } else {
        const bool neg = fl & MASK_BIT;
        double e[3];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const double c2 = __fma_rn(-2.0, ps, p[ax][2]) + p[ax][4];
            const double db = eno2_back64(p[ax][1], p[ax][2], ps, c2, a.h[ax], a.rh[ax], a.h2[ax], a.rh2[ax]);
            const double mf = eno2_back64(p[ax][5], p[ax][4], ps, c2, a.h[ax], a.rh[ax], a.h2[ax], a.rh2[ax]);
            e[ax] = vmax(0.0, vmax(flip(db, neg), flip(mf, neg)));  // mf = -D+
        }
        const double gn = norm_root(add_rn(add_rn(sqr(e[0]), sqr(e[1])), sqr(e[2])));
        step = flip((gn - 1.0) * a.dt_uniform, neg);
    }
    const double pn = STAGE == 0 ? 0.0 : __ldg(a.st.phi_n + c);
    a.st.out[c] = rk2_combine(STAGE, pn, ps, step);
}

// ---------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------
Args64 args64(const Grid &g)
{
    Args64 a{};
    a.g = g;
    const double h[3] = {g.dx, g.dy, g.dz};
    a.ordinary = true;
    for (int q = 0; q < 3; ++q) {
        a.h[q] = h[q];
        a.rh[q] = 1.0 / h[q];
        a.h2[q] = h[q] * h[q];
        a.rh2[q] = 1.0 / a.h2[q];
        a.tiny[q] = std::ldexp(h[q], -80);
        a.ordinary = a.ordinary && ordinary_spacing(h[q]);
    }
    a.dt_uniform = 0.3 * std::min(std::min(h[0], h[1]), h[2]);
    return a;
}

template <int KIND, int STAGE, int KZ> cudaError_t launch64_weno(Args64 &a, bool eno3, unsigned blocks, cudaStream_t s)
{
    const dim3 bl(BX, BY64);
    if constexpr (KIND != K64_ADVECT) {
        if (eno3) {
            k_weno64<KIND, STAGE, true, KZ><<<blocks, bl, 0, s>>>(a);
            return cudaGetLastError();
        }
    }
    k_weno64<KIND, STAGE, false, KZ><<<blocks, bl, 0, s>>>(a);
    return cudaGetLastError();
}
template <int KIND, int STAGE> cudaError_t launch64_as(Args64 &a, bool eno3, cudaStream_t s)
{
    const Grid &g = a.g;
    const long long columns = (long long)((g.rows + BX - 1) / BX) * ((g.cols + BY64 - 1) / BY64);
    constexpr bool ENO2 = KIND == K64_ENO2 || KIND == K64_ENO2R;
    // band blocks: up to four per SM (ENORK2: sixteen, for the warps that its long divisions wait on;
    // with 90 % of 128^3 a band 20 stages of extension 26.9 -> 24.4 ms, reinitialization 27.2 -> 25.8,
    // thin bands as before), and no more than the grid has nodes for
    a.band_blocks = band_kind64(KIND) ? (int)std::min<long long>((ENO2 ? 4 : 1) * list_blocks(), columns * g.pges) : 0;
    if constexpr (ENO2) {
        k_eno64<KIND, STAGE><<<(unsigned)(columns * g.pges + a.band_blocks), dim3(BX, BY64), 0, s>>>(a);
        return cudaGetLastError();
    } else {
        // Two pages per block where that leaves twelve blocks per SM, else one (a whole-SM imbalance
        // then costs more than the z differences saved).  Measured on GB300, ms, one / two / four
        // pages: 10 WENO5 reinitialization pseudo-steps 32^3 2.02 / 2.15 / 3.03, 64^3 6.63 / 6.82 /
        // 7.67, 96^3 19.6 / 19.4 / 19.9, 128^3 43.8 / 42.9 / 43.0; 10 extension pseudo-steps 96^3
        // 16.5 / 16.2 / 16.0, 128^3 37.8 / 36.8 / 36.3 (each difference formed per node: 47.9, 40.6).
        const long long tall = columns * ((g.pges + 1) / 2);
        if (tall >= 3 * list_blocks()) return launch64_weno<KIND, STAGE, 2>(a, eno3, (unsigned)(tall + a.band_blocks), s);
        return launch64_weno<KIND, STAGE, 1>(a, eno3, (unsigned)(columns * g.pges + a.band_blocks), s);
    }
}
template <int KIND> cudaError_t launch64(Args64 &a, int stage, bool eno3, cudaStream_t s)
{
    if (stage == 0) return launch64_as<KIND, 0>(a, eno3, s);
    if (stage == 1) return launch64_as<KIND, 1>(a, eno3, s);
    return launch64_as<KIND, 2>(a, eno3, s);
}

}  // namespace

cudaError_t launch_stage64(Kind64 kind, bool eno3, const Stage64 &st, int stage, const Grid &g, cudaStream_t s)
{
    Args64 a = args64(g);
    a.st = st;
    switch (kind) {
    case K64_REINIT: return launch64<K64_REINIT>(a, stage, eno3, s);
    case K64_EXTEND: return launch64<K64_EXTEND>(a, stage, eno3, s);
    case K64_ADVECT: return launch64<K64_ADVECT>(a, stage, eno3, s);
    case K64_ENO2: return launch64<K64_ENO2>(a, stage, eno3, s);
    case K64_ENO2R: return launch64<K64_ENO2R>(a, stage, eno3, s);
    default: return cudaErrorInvalidValue;
    }
}

template <>
cudaError_t launch_extension_velocity<double>(const double *phi, const uint8_t *flags, Ptr6<const double> dist,
                                              Ptr3<double> v, const Grid &g, bool eno3, double floor, NodeList flagged,
                                              cudaStream_t s)
{
    Args64 a = args64(g);
    a.st.phi_s = phi;
    a.st.flags = flags;
    a.st.d = dist;
    a.st.flagged = flagged;
    a.w = v;
    a.floor = floor;
    return launch64_as<K64_VELOCITY, 0>(a, eno3, s);
}

}  // namespace vsl
