// vsl_adjoint.cu -- reverse-mode (adjoint) kernels of the WENO5 TVD-RK3 advection and
// reinitialization stages, and of the sub-cell distances the reinitialization reads.
//
// A fused stage writes  out = a * phi_n + b * (phi_s - step(phi_s)).  Its adjoint, given
// lam = dL/d out, is
//     dL/d phi_s = b * lam - J^T (b * lam),   dL/d phi_n += a * lam,
// with J the Jacobian of `step`.  Row c of J touches the 7 values of each axis line
// through c (clamped at the grid edge), so J^T is applied in two deterministic passes:
//   1. per node c, the local partials d step_c / d p_ax[o] (o = 0..6 along axis ax) are
//      evaluated -- by the closed-form gradient of the uniform WENO5 (weno5_grad), and by
//      running the forward per-node code on dual numbers where the interface is inserted
//      -- scaled by b * lam_c and stored in 21 slots W[ax*7 + o][c] (slot-major,
//      coalesced);
//   2. per node j, every (c, ax, o) whose clamped stencil position is j is summed in a
//      fixed order (no atomics), giving (J^T b lam)_j.
// Partials with respect to the other inputs of a stage (the velocity of advection, the
// six interface distances of reinitialization) are accumulated per node in the same
// pass.  The distance adjoints are carried back to the field the distances were computed
// from by the implicit-function derivative of each root (k_adj_dist_edges).
//
// Every update is differentiated exactly as evaluated: WENO weights including their
// epsilon, the upwind and Godunov switches, the interface insertion and the minimum over
// the six distances in the pseudo-time step.  At a switch, the branch taken is
// differentiated.  The mask (sign of the field when a reinitialization starts) and the
// fixed-node test are piecewise constant and carry no derivative.
#include <cmath>
#include <type_traits>

#include "vsl_dual.cuh"
#include "vsl_internal.h"
#include "vsl_short64.cuh"

namespace vsl {
namespace {

// classification byte of the fused kernels: bit 6 mask (phi < 0 at the start), bit 7
// fixed node (a distance below 1e-6 dx)
constexpr uint8_t CLS_MASK = 0x40;
constexpr uint8_t CLS_FIXED = 0x80;
constexpr int SLOTS = 21;

__device__ __forceinline__ bool adj_node(const Grid &g, int &i, int &j, int &k, long long &c)
{
    i = blockIdx.x * BX + threadIdx.x;
    j = blockIdx.y * BY + threadIdx.y;
    k = blockIdx.z;
    if (i >= g.rows || j >= g.cols) return false;
    c = node_index(g, i, j, k);
    return true;
}

__device__ __forceinline__ void adj_node_of(const Grid &g, long long c, int &i, int &j, int &k)
{
    k = (int)(c / g.plane);
    const long long r = c - (long long)k * g.plane;
    j = (int)(r / g.rows);
    i = (int)(r - (long long)j * g.rows);
}

// products rounded by themselves, as where the forward code kept them in arrays
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// the seven values of an axis line through node c; lines away from the faces take no clamps
template <typename T>
__device__ __forceinline__ void adj_line7(const T *__restrict__ f, const Grid &g, int i, int j, int k, long long c,
                                          int ax, T p[7])
{
    const int q = ax == AX_X ? j : (ax == AX_Y ? i : k), n = ax == AX_X ? g.cols : (ax == AX_Y ? g.rows : g.pges);
    const long long stride = ax == AX_X ? (long long)g.rows : (ax == AX_Y ? 1 : g.plane);
    const T *fc = f + c;
    if (q >= 3 && q + 3 < n) {
#pragma unroll
        for (int s = -3; s <= 3; ++s) p[s + 3] = __ldg(fc + s * stride);
    } else {
#pragma unroll
        for (int s = -3; s <= 3; ++s) p[s + 3] = __ldg(fc + (clampi(q + s, n) - q) * stride);
    }
}

// Number types of the uniform stencils: quotients as a shared reciprocal, a product and a
// remainder correction (vsl_short64.cuh), three to six instructions where a general quotient is
// about twenty; a node took 38 of them per axis.  FP32: a Newton step from the hardware reciprocal
// gives the correctly rounded one for every significand (an ulp's error would do but for the
// significand of ones; sm_103a has that one right, tests/test_gpu_quotient32.py), and the quotient
// is then the correctly rounded one (Markstein's theorems), +0 for -0.  Operands near overflow take
// the general quotients (uniform_range).  In FP64 those near underflow do as well; in FP32 a
// numerator below about 2^-100, whose remainder is no normal number, leaves an ulp's error.
struct Short32 {
    float v;
    __device__ __forceinline__ Short32() {}
    __device__ __forceinline__ Short32(float x) : v(x) {}
    __device__ __forceinline__ Short32(double x) : v((float)x) {}
    __device__ __forceinline__ Short32(int x) : v((float)x) {}
    friend __device__ __forceinline__ Short32 operator+(Short32 a, Short32 b) { return a.v + b.v; }
    friend __device__ __forceinline__ Short32 operator-(Short32 a, Short32 b) { return a.v - b.v; }
    friend __device__ __forceinline__ Short32 operator*(Short32 a, Short32 b) { return a.v * b.v; }
    friend __device__ __forceinline__ Short32 operator/(Short32 a, Short32 b)
    {
        const float y0 = rcp_ftz(b.v);
        const float y = __fmaf_rn(__fmaf_rn(-b.v, y0, 1.f), y0, y0);
        const float q = __fmul_rn(a.v, y);
        return __fmaf_rn(__fmaf_rn(-b.v, q, a.v), y, q);
    }
};
// FP64: as Short64, with sums and products that the compiler may fuse as it does in the general
// code of this file
struct Fused64 {
    double v;
    __device__ __forceinline__ Fused64() {}
    __device__ __forceinline__ Fused64(double x) : v(x) {}
    __device__ __forceinline__ Fused64(int x) : v((double)x) {}
    friend __device__ __forceinline__ Fused64 operator+(Fused64 a, Fused64 b) { return a.v + b.v; }
    friend __device__ __forceinline__ Fused64 operator-(Fused64 a, Fused64 b) { return a.v - b.v; }
    friend __device__ __forceinline__ Fused64 operator*(Fused64 a, Fused64 b) { return a.v * b.v; }
    friend __device__ __forceinline__ Fused64 operator/(Fused64 a, Fused64 b) { return quotient(a.v, b.v, reciprocal(b.v)); }
};
__device__ __forceinline__ float adj_raw(Short32 x) { return x.v; }
__device__ __forceinline__ double adj_raw(Fused64 x) { return x.v; }
__device__ __forceinline__ float adj_raw(float x) { return x; }
__device__ __forceinline__ double adj_raw(double x) { return x; }
template <typename T> using ShortOf = typename std::conditional<std::is_same<T, float>::value, Short32, Fused64>::type;

// do the scaled differences of a line allow the short quotients (NaN fails the comparison)
__device__ __forceinline__ float max3_nan(float a, float b, float c)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ bool uniform_range(const float v[6])
{
    const float m = max3_nan(fabsf(v[0]), fabsf(v[1]), fabsf(v[2])), n = max3_nan(fabsf(v[3]), fabsf(v[4]), fabsf(v[5]));
    return max3_nan(m, n, n) < 16384.f;
}
__device__ __forceinline__ bool uniform_range(const double v[6])
{
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 6; ++q) ok = ok && within64(v[q], -200, 100);
    return ok;
}

// Jiang-Shu WENO5 of five differences (the weno5_plain formula) and its gradient g[5]:
// with alpha_k = d_k / (s_k + eps)^2 and w_k = alpha_k / sum alpha,
//   dD/dv = sum_k w_k dq_k/dv + sum_k c_k ds_k/dv,   c_k = -2 w_k (q_k - D) / (s_k + eps),
// where the candidates q_k are linear and the smoothness indicators s_k quadratic in v.
// The candidates come in q (weno5_candidates).
template <typename T> __device__ __forceinline__ void weno5_candidates(T v1, T v2, T v3, T v4, T v5, T q[3])
{
    q[0] = T(1. / 3.) * v1 - T(7. / 6.) * v2 + T(11. / 6.) * v3;
    q[1] = T(-1. / 6.) * v2 + T(5. / 6.) * v3 + T(1. / 3.) * v4;
    q[2] = T(1. / 3.) * v3 + T(5. / 6.) * v4 - T(1. / 6.) * v5;
}
template <typename T>
__device__ __forceinline__ T weno5_grad(T v1, T v2, T v3, T v4, T v5, const T q[3], T g[5])
{
    const T q1 = q[0], q2 = q[1], q3 = q[2];
    const T a1 = v1 - 2 * v2 + v3, b1 = v1 - 4 * v2 + 3 * v3;
    const T a2 = v2 - 2 * v3 + v4, b2 = v2 - v4;
    const T a3 = v3 - 2 * v4 + v5, b3 = 3 * v3 - 4 * v4 + v5;
    const T eps = T(1e-6);
    const T e1 = T(13. / 12.) * a1 * a1 + T(1. / 4.) * b1 * b1 + eps;
    const T e2 = T(13. / 12.) * a2 * a2 + T(1. / 4.) * b2 * b2 + eps;
    const T e3 = T(13. / 12.) * a3 * a3 + T(1. / 4.) * b3 * b3 + eps;
    const T al1 = T(0.1) / (e1 * e1), al2 = T(0.6) / (e2 * e2), al3 = T(0.3) / (e3 * e3);
    const T inv = T(1) / (al1 + al2 + al3);
    const T w1 = al1 * inv, w2 = al2 * inv, w3 = al3 * inv;
    const T D = w1 * q1 + w2 * q2 + w3 * q3;
    const T c1 = T(-2) * w1 * (q1 - D) / e1;
    const T c2 = T(-2) * w2 * (q2 - D) / e2;
    const T c3 = T(-2) * w3 * (q3 - D) / e3;
    // ds_k/dv: s1 = 13/12 a1^2 + 1/4 b1^2 with a1 = (1,-2,1,0,0).v, b1 = (1,-4,3,0,0).v, etc.
    const T A1 = T(13. / 6.) * a1 * c1, B1 = T(0.5) * b1 * c1;
    const T A2 = T(13. / 6.) * a2 * c2, B2 = T(0.5) * b2 * c2;
    const T A3 = T(13. / 6.) * a3 * c3, B3 = T(0.5) * b3 * c3;
    g[0] = T(1. / 3.) * w1 + A1 + B1;
    g[1] = T(-7. / 6.) * w1 - T(1. / 6.) * w2 - 2 * A1 - 4 * B1 + A2 + B2;
    g[2] = T(11. / 6.) * w1 + T(5. / 6.) * w2 + T(1. / 3.) * w3 + A1 + 3 * B1 - 2 * A2 + A3 + 3 * B3;
    g[3] = T(1. / 3.) * w2 + T(5. / 6.) * w3 + A2 - B2 - 2 * A3 - 4 * B3;
    g[4] = T(-1. / 6.) * w3 + A3 + B3;
    return D;
}

// One side (back: D-, else D+) of the uniform WENO5 derivatives of an axis line with its partials
// with respect to the seven line values: jac[o] = d D / d p[o].  A stage's update depends on one
// side of an axis (the upwind one of a transport, the one that the Godunov norm took), so the other
// side's partials, which would be multiplied by zero, are not formed.
template <typename R, typename T>
__device__ __forceinline__ void weno5_side_grad_of(const T v[6], bool back, T ih, T &D, T jac[7])
{
    // the candidates of both sides: with one side's alone the compiler would fuse other products
    R g[5], qb[3], qf[3], q[3];
    weno5_candidates<R>(R(v[0]), R(v[1]), R(v[2]), R(v[3]), R(v[4]), qb);
    weno5_candidates<R>(R(v[5]), R(v[4]), R(v[3]), R(v[2]), R(v[1]), qf);
#pragma unroll
    for (int m = 0; m < 3; ++m) q[m] = R(back ? adj_raw(qb[m]) : adj_raw(qf[m]));
    D = adj_raw(weno5_grad<R>(R(back ? v[0] : v[5]), R(back ? v[1] : v[4]), R(back ? v[2] : v[3]),
                              R(back ? v[3] : v[2]), R(back ? v[4] : v[1]), q, g));
    // d D / d v[m], m = 0..5: g in the window's order
    T G[6];
    G[0] = back ? adj_raw(g[0]) : T(0);
#pragma unroll
    for (int m = 1; m < 5; ++m) G[m] = back ? adj_raw(g[m]) : adj_raw(g[5 - m]);
    G[5] = back ? T(0) : adj_raw(g[0]);
#pragma unroll
    for (int o = 0; o < 7; ++o) {
        const T l = o >= 1 ? G[o - 1] : T(0), r = o <= 5 ? G[o] : T(0);
        jac[o] = (l - r) * ih;
    }
}
template <typename T>
__device__ __noinline__ void weno5_side_grad_general(const T p[7], T h, bool back, T &D, T jac[7])
{
    T v[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) v[m] = (p[m + 1] - p[m]) / h;
    weno5_side_grad_of<T>(v, back, T(1) / h, D, jac);
}
template <typename T> __device__ __forceinline__ void weno5_side_grad(const T p[7], T h, bool back, T &D, T jac[7])
{
    using R = ShortOf<T>;
    T v[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) v[m] = adj_raw(R(p[m + 1] - p[m]) / R(h));
    if (uniform_range(v))
        weno5_side_grad_of<R>(v, back, adj_raw(R(T(1)) / R(h)), D, jac);
    else
        weno5_side_grad_general(p, h, back, D, jac);
}

// the uniform pair's values (weno5_pair_plain)
template <typename T> __device__ __noinline__ void weno5_pair_general(const T p[7], T h, T &df, T &db)
{
    weno5_pair_plain<T>(p, h, df, db);
}
template <typename T> __device__ __forceinline__ void weno5_pair_values(const T p[7], T h, T &df, T &db)
{
    using R = ShortOf<T>;
    T v[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) v[m] = adj_raw(R(p[m + 1] - p[m]) / R(h));
    if (uniform_range(v)) {
        db = adj_raw(weno5_plain<R>(v[0], v[1], v[2], v[3], v[4]));
        df = adj_raw(weno5_plain<R>(v[5], v[4], v[3], v[2], v[1]));
    } else {
        weno5_pair_general(p, h, df, db);
    }
}

// One side (back: D-, else D+) of the nonuniform WENO5 pair, out of line on dual numbers.
template <typename D> __device__ __noinline__ D nonuniform_side(const D xs[7], const D hs[7], bool back)
{
    D dd[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) dd[m] = (hs[m + 1] - hs[m]) / (xs[m + 1] - xs[m]);
    if (back) return weno_nonuniform_back<D>(xs, dd);
    return weno_nonuniform_fore<D>(xs, dd);
}

// One side of the interface-aware pair (nonuniform WENO5 with the interface inserted at r1 / l1,
// value 0): its partials with respect to the seven line values (0..6) and r1, l1 (7, 8), by dual
// numbers.
template <typename T>
__device__ __noinline__ void iface_side_jac(const T p[7], T h, T r1, T l1, bool back, T jac[9])
{
    using D = Dual<T, 9>;
    D P[7], xs[7], hs[7];
#pragma unroll
    for (int o = 0; o < 7; ++o) P[o] = D::var(p[o], o);
    insert_interface<D>(P, D::var(r1, 7), D::var(l1, 8), D((double)h), D(0.0), D(0.0), xs, hs);
    const D r = nonuniform_side<D>(xs, hs, back);
#pragma unroll
    for (int o = 0; o < 9; ++o) jac[o] = r.d[o];
}

// ---------------------------------------------------------------------------------------
// advection stage: step = dt * sum_ax (min(0, v) D+ + max(0, v) D-)  (uniform WENO5)
// Bound by its instructions (about 1000 per node, 60 % of the issue slots) and the 176 MB of slots
// that it writes at 128^3 (30 % of the memory rate).  The next axis' line and velocity adjoint are
// loaded while an axis is formed, and the slots' addresses advance by additions: 105 -> 93 us.
// FP32: five blocks to an SM; FP64, bound by its pipe, two (no spills; forward and adjoint of four
// steps at 96^3 30.3 ms, 30.5 at five blocks and 48 registers, with four or three between).
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(BX *BY, (sizeof(T) == 4 ? 5 : 2))
    k_adj_advect_jac(const T *__restrict__ ps, Ptr3<const T> v, const double *__restrict__ dt,
                     const T *__restrict__ lam, T coef, T *__restrict__ W, Ptr3<T> gv, Grid g)
{
    int i, j, k;
    long long c;
    if (!adj_node(g, i, j, k, c)) return;
    const T lc = coef * __ldg(lam + c) * (T)__ldg(dt);
    T p[7], va = __ldg(v.p[0] + c), ga = gv.p[0][c];
    T *w = W + c;
    adj_line7(ps, g, i, j, k, c, 0, p);
#pragma unroll 1
    for (int ax = 0; ax < 3; ++ax) {
        // the next axis is on its way while this one is formed
        T pn[7], vn, gn;
        if (ax < 2) {
            adj_line7(ps, g, i, j, k, c, ax + 1, pn);
            vn = __ldg(v.p[ax + 1] + c);
            gn = gv.p[ax + 1][c];
        }
        // min(0, v) D+ + max(0, v) D-: D- where v > 0, D+ otherwise
        T jac[7], D;
        weno5_side_grad<T>(p, (T)axis_h(g, ax), va > T(0), D, jac);
#pragma unroll
        for (int o = 0; o < 7; ++o, w += g.num) *w = lc * (va * jac[o]);
        gv.p[ax][c] = ga - lc * D;
#pragma unroll
        for (int o = 0; o < 7; ++o) p[o] = pn[o];
        va = vn;
        ga = gn;
    }
}

// ---------------------------------------------------------------------------------------
// reinitialization stage: step = (|grad|_Godunov - 1) * 0.3 min(dist) * (mask ? -1 : 1)
// ---------------------------------------------------------------------------------------
// the six distances (stored where flagged, the spacing elsewhere) and their minimum (the
// pseudo-time step is 0.3 times it), taken in the order of the forward kernel's vmin tree
template <typename T>
__device__ __forceinline__ int reinit_distances(uint8_t fl, const Ptr6<const T> &d, long long c, const Grid &g, T dist[6])
{
    const T h[3] = {(T)g.dx, (T)g.dy, (T)g.dz};
#pragma unroll
    for (int q = 0; q < 6; ++q) dist[q] = (fl & (1u << q)) ? __ldg(d.p[q] + c) : h[q / 2];
    const T d01 = dist[0] < dist[1] ? dist[0] : dist[1], d23 = dist[2] < dist[3] ? dist[2] : dist[3],
            d45 = dist[4] < dist[5] ? dist[4] : dist[5], d25 = d23 < d45 ? d23 : d45;
    const int i01 = dist[0] < dist[1] ? 0 : 1, i23 = dist[2] < dist[3] ? 2 : 3, i45 = dist[4] < dist[5] ? 4 : 5;
    return d01 < d25 ? i01 : (d23 < d45 ? i23 : i45);
}

// One axis of the Godunov norm G = sqrt(sum_ax max(A_ax, B_ax)), with the branch of the max as
// the forward took it: the squared term, the side taken (back: D-) and the derivative gs of the
// term with respect to that side.
template <typename T> __device__ __forceinline__ T godunov_axis(bool neg, T df, T db, T &gs, bool &back)
{
    const T z = T(0);
    const T A = neg ? sqr(vmin(z, db)) : sqr(vmax(z, db));
    const T B = neg ? sqr(vmax(z, df)) : sqr(vmin(z, df));
    back = !(A < B);
    gs = T(2) * (back ? (neg ? vmin(z, db) : vmax(z, db)) : (neg ? vmax(z, df) : vmin(z, df)));
    return back ? A : B;
}

// One axis of a uniform line p: the term of the Godunov norm with its derivative gs with respect
// to the side that the norm takes, and that side's partials.
template <typename T>
__device__ __forceinline__ T reinit_axis(const T p[7], T h, bool neg, T &gs, T jac[7])
{
    using R = ShortOf<T>;
    T v[6], D, df, db;
    bool back;
#pragma unroll
    for (int m = 0; m < 6; ++m) v[m] = adj_raw(R(p[m + 1] - p[m]) / R(h));
    const bool in_range = uniform_range(v);
    if (in_range) {
        db = adj_raw(weno5_plain<R>(v[0], v[1], v[2], v[3], v[4]));
        df = adj_raw(weno5_plain<R>(v[5], v[4], v[3], v[2], v[1]));
    } else {
        weno5_pair_general(p, h, df, db);
    }
    const T X = godunov_axis(neg, df, db, gs, back);
    if (in_range)
        weno5_side_grad_of<R>(v, back, adj_raw(R(T(1)) / R(h)), D, jac);
    else
        weno5_side_grad_general(p, h, back, D, jac);
    return X;
}

// One node of the reinitialization-stage Jacobian whose three axis lines are all uniform (no sign
// change next to the node).  An axis is visited once: its side's partials wait in shared memory
// (kept: this thread's column) for the norm that scales them.
template <typename T>
__device__ __forceinline__ void reinit_jac_node(const T *__restrict__ ps, const uint8_t fl, Ptr6<const T> d,
                                                const T lc, T *__restrict__ W, Ptr6<T> mu, const Grid &g, int i,
                                                int j, int k, long long c, T (*kept)[BX * BY])
{
    T dist[6];
    const int qmin = reinit_distances(fl, d, c, g, dist);
    T dmin = dist[0];
#pragma unroll
    for (int q = 1; q < 6; ++q) dmin = q == qmin ? dist[q] : dmin;
    const T dtv = T(0.3) * dmin;
    const bool neg = fl & CLS_MASK;
    const T sgn = neg ? T(-1) : T(1);
    const int tid = threadIdx.y * BX + threadIdx.x;

    T gq[3], S = T(0);
#pragma unroll 1
    for (int ax = 0; ax < 3; ++ax) {
        T p[7], jac[7], gs;
        adj_line7(ps, g, i, j, k, c, ax, p);
        S = add_rn(S, reinit_axis(p, (T)axis_h(g, ax), neg, gs, jac));
#pragma unroll
        for (int a = 0; a < 3; ++a) gq[a] = a == ax ? gs : gq[a];
#pragma unroll
        for (int o = 0; o < 7; ++o) kept[ax * 7 + o][tid] = jac[o];
    }
    const T G = sqrt(S);
    const T dG = G > T(0) ? T(0.5) / G : T(0);  // zero derivative of sqrt at 0
    const T s_dt = dtv * sgn;
    T *w = W + c;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const T gs = gq[ax] * dG * s_dt;
#pragma unroll
        for (int o = 0; o < 7; ++o, w += g.num) *w = lc * (gs * kept[ax * 7 + o][tid]);
    }
    // d step / d dist_q: through dt for the minimum
    if (fl & (1u << qmin)) mu.p[qmin][c] -= lc * ((G - T(1)) * sgn * T(0.3));
}

// warp-aggregated append of `value` where `pred` holds (all 32 lanes of the warp call it)
__device__ __forceinline__ void adj_append(bool pred, unsigned value, unsigned *list, unsigned *count)
{
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    const unsigned lane = (threadIdx.y * blockDim.x + threadIdx.x) & 31u;
    const int leader = __ffs(m) - 1;
    unsigned base = 0;
    if ((int)lane == leader) base = atomicAdd(count, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) list[base + __popc(m & ((1u << lane) - 1u))] = value;
}

// dense pass: fixed nodes get zero slots; nodes with a sign change next to them on any
// axis are listed for k_adj_reinit_jac_band; the rest are done here.  Bound by its instructions
// (77 % of the issue slots at two passes over the axes): 173 us at 128^3 with general quotients and
// both sides' partials, 142 on short quotients and one side, 120 with each axis visited once.
template <typename T>
__global__ void __launch_bounds__(BX *BY) k_adj_reinit_jac(const T *__restrict__ ps, const uint8_t *__restrict__ flags,
                                                             Ptr6<const T> d, const T *__restrict__ lam, T coef,
                                                             T *__restrict__ W, Ptr6<T> mu, NodeList band, Grid g)
{
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y, k = blockIdx.z;
    const bool in = i < g.rows && j < g.cols;
    const long long c = in ? node_index(g, i, j, k) : 0;
    const uint8_t fl = in ? __ldg(flags + c) : uint8_t(0);
    bool near = false;
    if (in && !(fl & CLS_FIXED)) {
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const AxisLine L = axis_line(g, i, j, k, ax);
            const T pm = __ldg(ps + L.base + (long long)clampi(L.c - 1, L.n) * L.stride);
            const T p0 = __ldg(ps + c);
            const T pp = __ldg(ps + L.base + (long long)clampi(L.c + 1, L.n) * L.stride);
            near |= pm * p0 < T(0) || p0 * pp < T(0);
        }
    }
    adj_append(near, (unsigned)c, band.idx, band.count);
    if (!in || near) return;
    if (fl & CLS_FIXED) {
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) W[(long long)s * g.num + c] = T(0);
        return;
    }
    __shared__ T kept[SLOTS][BX * BY];
    reinit_jac_node<T>(ps, fl, d, coef * __ldg(lam + c), W, mu, g, i, j, k, c, kept);
}

// The listed nodes (40,000 around a sphere of radius 38), BAND_NODES at a time, as (node, axis)
// tasks: the derivative pairs first, then,
// once the norm of each node is known, the partials, with the tasks in order of kind (uniform,
// interface-aware forward, interface-aware backward) so that a warp takes one path.  Bound by
// fetching the instructions of the dual-number code, eight warps to a multiprocessor (255
// registers).  A thread per node with both sides of three axes took 110 us, a task to a lane
// without the order 89, this 76 (42 nodes to a block of 128: 77).
constexpr int BAND_NODES = 85, BAND_THREADS = 256;
template <typename T>
__global__ void __launch_bounds__(BAND_THREADS) k_adj_reinit_jac_band(const T *__restrict__ ps,
                                                                        const uint8_t *__restrict__ flags,
                                                                        Ptr6<const T> d, const T *__restrict__ lam,
                                                                        T coef, T *__restrict__ W, Ptr6<T> mu,
                                                                        NodeList band, Grid g)
{
    __shared__ T sdf[BAND_NODES][3], sdb[BAND_NODES][3];
    __shared__ unsigned char order[3 * BAND_NODES];
    __shared__ int kinds[4];
    const int tid = threadIdx.x;
    const unsigned n = *band.count;
    for (unsigned t0 = blockIdx.x * BAND_NODES; t0 < n; t0 += gridDim.x * BAND_NODES) {
        const int nodes = min((unsigned)BAND_NODES, n - t0);
        const bool task = tid < 3 * nodes;
        if (tid < 4) kinds[tid] = 0;
        __syncthreads();
        int kind = 0, rank = 0;
        if (task) {
            const int q = tid / 3, ax = tid - 3 * q;
            const long long c = band.idx[t0 + q];
            int i, j, k;
            adj_node_of(g, c, i, j, k);
            const uint8_t fl = __ldg(flags + c);
            const T h = (T)axis_h(g, ax);
            T p[7], df, db, gs;
            bool back;
            adj_line7(ps, g, i, j, k, c, ax, p);
            const bool iface = p[2] * p[3] < T(0) || p[3] * p[4] < T(0);
            if (iface) {
                const T r1 = (fl & (1u << (2 * ax))) ? __ldg(d.p[2 * ax] + c) : h;
                const T l1 = (fl & (2u << (2 * ax))) ? __ldg(d.p[2 * ax + 1] + c) : h;
                interface_pair<T>(p, r1, l1, h, T(0), T(0), false, df, db);
            } else {
                weno5_pair_values<T>(p, h, df, db);
            }
            godunov_axis((fl & CLS_MASK) != 0, df, db, gs, back);
            sdf[q][ax] = df;
            sdb[q][ax] = db;
            kind = iface ? (back ? 2 : 1) : 0;
            rank = atomicAdd(kinds + kind, 1);
        }
        __syncthreads();
        if (task) order[rank + (kind > 0 ? kinds[0] : 0) + (kind > 1 ? kinds[1] : 0)] = (unsigned char)tid;
        __syncthreads();
        if (task) {
            const int q = order[tid] / 3, ax = order[tid] - 3 * q;
            const bool iface = tid >= kinds[0], back_side = tid >= kinds[0] + kinds[1];
            const long long c = band.idx[t0 + q];
            int i, j, k;
            adj_node_of(g, c, i, j, k);
            const uint8_t fl = __ldg(flags + c);
            const bool neg = fl & CLS_MASK;
            const T sgn = neg ? T(-1) : T(1), h = (T)axis_h(g, ax), lc = coef * __ldg(lam + c);
            T dist[6], p[7];
            const int qmin = reinit_distances(fl, d, c, g, dist);
            adj_line7(ps, g, i, j, k, c, ax, p);
            T dmin = dist[0], r1 = dist[0], l1 = dist[1];
#pragma unroll
            for (int m = 1; m < 6; ++m) dmin = m == qmin ? dist[m] : dmin;
#pragma unroll
            for (int a = 1; a < 3; ++a) {
                r1 = a == ax ? dist[2 * a] : r1;
                l1 = a == ax ? dist[2 * a + 1] : l1;
            }
            T S = T(0), gs = T(0);
            bool back = false;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                T ga;
                bool ba;
                S = add_rn(S, godunov_axis(neg, sdf[q][a], sdb[q][a], ga, ba));
                gs = a == ax ? ga : gs;
                back = a == ax ? ba : back;
            }
            const T G = sqrt(S);
            const T dG = G > T(0) ? T(0.5) / G : T(0);  // zero derivative of sqrt at 0
            gs = gs * dG * (T(0.3) * dmin * sgn);
            T jac[9];
            if (iface) {
                iface_side_jac<T>(p, h, r1, l1, back_side, jac);
            } else {
                T D;
                weno5_side_grad<T>(p, h, back, D, jac);
                jac[7] = jac[8] = T(0);
            }
            T *w = W + (long long)(ax * 7) * g.num + c;
#pragma unroll
            for (int o = 0; o < 7; ++o, w += g.num) *w = lc * (gs * jac[o]);
            // d step / d dist: through the interface insertion, and through dt for the minimum
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int m = 2 * ax + o;
                const T md = mul_rn(gs, jac[7 + o]);
                const T ds = md + (m == qmin ? (G - T(1)) * sgn * T(0.3) : T(0));
                if (fl & (1u << m)) mu.p[m][c] -= lc * ds;
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------
// transpose pass: out_j = alpha * lam_j - sum of W over the stencil positions equal to j
// (+ acc_j); the share of lam that the step's start takes is added up in the same pass
// Bound by memory: 185 MB of slots at 128^3, 42 us (4.4 TB/s beside the write-back of the slots);
// with clamped 64-bit index arithmetic and first pages first it took 54.
// ---------------------------------------------------------------------------------------
// offset of the source of slot ax*7+o from its node: its slot's array, o - 3 nodes back
struct GatherOffsets {
    long long at[SLOTS];
};
template <typename T>
__global__ void __launch_bounds__(BX *BY) k_adj_gather(const T *__restrict__ W, const T *lam, T alpha,
                                                         const T *acc, T *out, AdjShare<T> share, GatherOffsets from, Grid g)
{
    // last pages first: theirs are the slots that the pass before wrote last, still in L2
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y, k = gridDim.z - 1 - blockIdx.z;
    if (i >= g.rows || j >= g.cols) return;
    const long long c = node_index(g, i, j, k);
    // sources whose offset o lands exactly on the node (none beyond an edge), all on their way at once
    T w[3][7];
    const T *Wc = W + c;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int cj = ax == AX_X ? j : (ax == AX_Y ? i : k), n = ax == AX_X ? g.cols : (ax == AX_Y ? g.rows : g.pges);
#pragma unroll
        for (int o = 0; o < 7; ++o) {
            const bool in = o < 3 ? cj + (3 - o) < n : (o > 3 ? cj >= o - 3 : true);
            w[ax][o] = in ? __ldg(Wc + from.at[ax * 7 + o]) : T(0);
        }
    }
    const T l = lam[c], a = acc ? acc[c] : T(0);
    if (share.acc) share.acc[c] = (share.init ? T(0) : share.acc[c]) + (T)share.a * l;
    T s = T(0);
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int cj = ax == AX_X ? j : (ax == AX_Y ? i : k), n = ax == AX_X ? g.cols : (ax == AX_Y ? g.rows : g.pges);
        const long long stride = ax == AX_X ? (long long)g.rows : (ax == AX_Y ? 1 : g.plane);
        const T *Wa = W + (long long)(ax * 7) * g.num + c;
        s += w[ax][3];
#pragma unroll
        for (int o = 0; o < 7; ++o)
            if (o != 3) s += w[ax][o];
        // sources whose offset ran past an edge and was clamped onto cj
        if (cj == 0) {
#pragma unroll 1
            for (int ci = 0; ci < min(3, n); ++ci)
                for (int o = 0; o <= 2 - ci; ++o) s += Wa[(long long)o * g.num + ci * stride];
        }
        if (cj == n - 1) {
#pragma unroll 1
            for (int ci = max(0, n - 3); ci < n; ++ci)
                for (int o = n + 3 - ci; o <= 6; ++o) s += Wa[(long long)o * g.num + (ci - cj) * stride];
        }
    }
    out[c] = alpha * l - s + a;
}

// ---------------------------------------------------------------------------------------
// distances: d/dv of the root of each crossed edge
// ---------------------------------------------------------------------------------------

// the quadratic ENO distance next to a kink, on dual numbers (same formula as the double
// eno2_distance)
template <typename D> __device__ D eno2_distance_dual(D a, D b, D c, D d, double h)
{
    const double eps = 10e-10;
    const D d2 = minmod(c - 2.0 * b + a, d - 2.0 * c + b);
    if (d2 > D(eps) || d2 < D(-eps)) {
        const D disc = sqr(0.5 * d2 - b - c) - 4. * b * c;
        return h * (D(0.5) + (b - c - sgn1((b - c).v) * sqrt(disc)) / d2);
    }
    return h * b / (b - c);
}

// jd[s] = d dist / d v[s] of quintic_distance(v, h): the implicit-function derivative
// -L_s(t) / P'(t) of the fitted root t (zero where the root was clamped to the cell), or
// the quadratic ENO derivative where that formula was used
__device__ void quintic_distance_jac(const double v[6], double h, double jd[6])
{
#pragma unroll
    for (int s = 0; s < 6; ++s) jd[s] = 0.0;
    if (v[1] * v[2] < 0 || v[3] * v[4] < 0) {
        using D = Dual<double, 4>;
        const D r = eno2_distance_dual<D>(D::var(v[1], 0), D::var(v[2], 1), D::var(v[3], 2), D::var(v[4], 3), h);
        for (int s = 0; s < 4; ++s) jd[s + 1] = r.d[s];
        return;
    }
    const double dist = quintic_distance(v, h);
    if (!(dist > 0.0 && dist < h)) return;
    const double t = dist + 2 * h;
    double L[6], dP = 0.0;
    for (int s = 0; s < 6; ++s) {
        double num = 1.0, den = 1.0, dnum = 0.0;
        for (int m = 0; m < 6; ++m) {
            if (m == s) continue;
            // derivative of the running product by the product rule
            dnum = dnum * (t - m * h) + num;
            num *= t - m * h;
            den *= (s - m) * h;
        }
        L[s] = num / den;
        dP += v[s] * (dnum / den);
    }
    if (dP == 0.0) return;
    for (int s = 0; s < 6; ++s) jd[s] = -L[s] / dP;
}

// W[(ax*7 + o)][c] = -(mu_fore(c) - mu_back(c + stride)) * d dist / d v[o - 1] for every
// crossed edge (c, c + stride); W is zero elsewhere (cleared by the launcher)
template <typename T>
__global__ void __launch_bounds__(128) k_adj_dist_edges(const T *__restrict__ f, EdgeLists e, Ptr6<const T> mu,
                                                          T *__restrict__ W, Grid g)
{
    for (int ax = 0; ax < 3; ++ax) {
        const unsigned n = *(e.count + ax);
        const double h = axis_h(g, ax);
        for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
            const long long c = e.idx[ax][t];
            int i, j, k;
            adj_node_of(g, c, i, j, k);
            const AxisLine L = axis_line(g, i, j, k, ax);
            const double m = (double)__ldg(mu.p[2 * ax] + c) - (double)__ldg(mu.p[2 * ax + 1] + c + L.stride);
            double v[6], jd[6];
#pragma unroll
            for (int s = -2; s <= 3; ++s) v[s + 2] = (double)__ldg(f + L.base + (long long)clampi(L.c + s, L.n) * L.stride);
            quintic_distance_jac(v, h, jd);
#pragma unroll
            for (int s = 0; s < 6; ++s) W[(long long)(ax * 7 + s + 1) * g.num + c] = (T)(-m * jd[s]);
        }
    }
}

int adj_list_blocks()
{
    static int n = 0;
    if (n == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        n = (sms > 0 ? sms : 132) * 4;
    }
    return n;
}

}  // namespace

// ---------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------
template <typename T>
cudaError_t launch_adj_advect_jac(const T *ps, Ptr3<const T> v, const double *dt, const T *lam, double coef, T *W,
                                  Ptr3<T> gv, const Grid &g, cudaStream_t s)
{
    k_adj_advect_jac<T><<<node_grid(g), dim3(BX, BY), 0, s>>>(ps, v, dt, lam, (T)coef, W, gv, g);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adj_reinit_jac(const T *ps, const uint8_t *flags, Ptr6<const T> d, const T *lam, double coef, T *W,
                                  Ptr6<T> mu, NodeList band, const Grid &g, cudaStream_t s)
{
    cudaError_t err = cudaMemsetAsync(band.count, 0, sizeof(unsigned), s);
    if (err != cudaSuccess) return err;
    k_adj_reinit_jac<T><<<node_grid(g), dim3(BX, BY), 0, s>>>(ps, flags, d, lam, (T)coef, W, mu, band, g);
    k_adj_reinit_jac_band<T><<<adj_list_blocks(), BAND_THREADS, 0, s>>>(ps, flags, d, lam, (T)coef, W, mu, band, g);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adj_gather(const T *W, const T *lam, double alpha, const T *acc, T *out, AdjShare<T> share,
                              const Grid &g, cudaStream_t s)
{
    const long long stride[3] = {g.rows, 1, g.plane};
    GatherOffsets from;
    for (int q = 0; q < SLOTS; ++q) from.at[q] = q * g.num - (q % 7 - 3) * stride[q / 7];
    k_adj_gather<T><<<node_grid(g), dim3(BX, BY), 0, s>>>(W, lam, (T)alpha, acc, out, share, from, g);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adj_dist_edges(const T *f, EdgeLists e, Ptr6<const T> mu, T *W, const Grid &g, cudaStream_t s)
{
    cudaError_t err = cudaMemsetAsync(W, 0, sizeof(T) * (size_t)SLOTS * (size_t)g.num, s);
    if (err != cudaSuccess) return err;
    k_adj_dist_edges<T><<<adj_list_blocks(), 128, 0, s>>>(f, e, mu, W, g);
    return cudaGetLastError();
}

#define VSL_INSTANTIATE_ADJ(T)                                                                                     \
    template cudaError_t launch_adj_advect_jac<T>(const T *, Ptr3<const T>, const double *, const T *, double, T *, \
                                                  Ptr3<T>, const Grid &, cudaStream_t);                             \
    template cudaError_t launch_adj_reinit_jac<T>(const T *, const uint8_t *, Ptr6<const T>, const T *, double, T *, \
                                                  Ptr6<T>, NodeList, const Grid &, cudaStream_t);                   \
    template cudaError_t launch_adj_gather<T>(const T *, const T *, double, const T *, T *, AdjShare<T>,           \
                                              const Grid &, cudaStream_t);                                          \
    template cudaError_t launch_adj_dist_edges<T>(const T *, EdgeLists, Ptr6<const T>, T *, const Grid &,          \
                                                  cudaStream_t);

VSL_INSTANTIATE_ADJ(float)
VSL_INSTANTIATE_ADJ(double)

}  // namespace vsl
