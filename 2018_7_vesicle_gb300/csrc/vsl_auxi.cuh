// vsl_auxi.cuh -- the calculus toolbox of the auxiliary level set A that marks the
// domains of a multiphase vesicle on the surface F = 0 (auxi_set_calculus_toolbox.cu:10-199,
// GPUAsetCalculusToolBox.m:2-63) and the masked FP64 surface and line integrals of
// SDF3.m:82-85, 212-227.  Templated on the field type; included by vsl_auxi_f64.cu (no
// multiply-add contraction, the reference's rounding) and vsl_auxi_f32.cu (mixed form).
//
// The fused form reads only A and F: F's gradient, Hessian, normal and Heaviside are
// recomputed from F's stencil with the calculus toolbox's own expressions instead of
// being read back from 14 stored toolbox fields.  Pass 1 writes the requested fields of
// the kernel plus the Heaviside functions of A and F; pass 2 forms AFDiracDelta and
// ADiracDeltaDn with SD.GD3's periodic operators, as the MATLAB method does.
#pragma once

#include <cmath>
#include <limits>

#include <type_traits>

#include "vsl_internal.h"
#include "vsl_tool64.cuh"

namespace vsl {
namespace {

constexpr int ANT = BX * BY;
constexpr int ANW = ANT / 32;

// ---------------------------------------------------------------------------------------
// Number types of the per-node code.  The plain form takes Short64 (the reference's roundings
// on the short quotients of vsl_short64.cuh, the FP64 pipe being its bound) where a node's values
// are ordinary, else double.  The mixed form takes Fast32: quotients as products with the
// approximate reciprocal, which the compiler shares between equal divisors (a general FP32
// quotient is about eight instructions, and the kernel issued 900 per node with 60 of them).
// ---------------------------------------------------------------------------------------
struct Fast32 {
    float v;
    __device__ __forceinline__ Fast32() {}
    __device__ __forceinline__ Fast32(float x) : v(x) {}
    friend __device__ __forceinline__ Fast32 operator+(Fast32 a, Fast32 b) { return a.v + b.v; }
    friend __device__ __forceinline__ Fast32 operator-(Fast32 a, Fast32 b) { return a.v - b.v; }
    friend __device__ __forceinline__ Fast32 operator-(Fast32 a) { return -a.v; }
    friend __device__ __forceinline__ Fast32 operator*(Fast32 a, Fast32 b) { return a.v * b.v; }
    friend __device__ __forceinline__ Fast32 operator/(Fast32 a, Fast32 b) { return a.v * rcp_ftz(b.v); }
};
__device__ __forceinline__ float raw64(Fast32 x) { return x.v; }
struct Divisor32 {
    float d;
};
__device__ __forceinline__ Fast32 operator/(Fast32 a, const Divisor32 &c) { return a.v * rcp_ftz(c.d); }
template <typename T>
using AuxDivisors = ToolDivisors<typename std::conditional<std::is_same<T, float>::value, Divisor32, Divisor64>::type>;
// the mixed form's divisors are products of FP32 spacings
inline AuxDivisors<float> aux_divisors(const Grid &g, double ds, float)
{
    const float x = (float)g.dx, y = (float)g.dy, z = (float)g.dz, s = (float)ds;
    return AuxDivisors<float>{{{2 * x}, {2 * y}, {2 * z}}, {{x * x}, {y * y}, {z * z}}, {4 * s * s}, true};
}
inline AuxDivisors<double> aux_divisors(const Grid &g, double ds, double) { return tool64(g, ds); }
__device__ __forceinline__ Fast32 a_root(Fast32 x) { return sqrtf(x.v); }
__device__ __forceinline__ Short64 a_root(Short64 x) { return sqrt(x.v); }
__device__ __forceinline__ double a_root(double x) { return sqrt(x); }
template <typename R> __device__ __forceinline__ R a_atleast(R x, R lo)
{
    return raw64(x) < raw64(lo) ? lo : x;  // vmax
}
// x / g^3, x / g^4 (FP32: general quotients, since the powers leave the normal range where |grad|
// is near its floor)
template <typename R> __device__ __forceinline__ R a_over3(R x, R g) { return x / R(pow_cr<3>(raw64(g))); }
template <> __device__ __forceinline__ Fast32 a_over3(Fast32 x, Fast32 g) { return x.v / (g.v * g.v * g.v); }
template <typename R> __device__ __forceinline__ R a_over4(R x, R g) { return x / R(pow_cr<4>(raw64(g))); }
template <> __device__ __forceinline__ Fast32 a_over4(Fast32 x, Fast32 g)
{
    return x.v / ((g.v * g.v) * (g.v * g.v));
}

// the vector norm of shared_utilities.cup:8-12, floored at 1e-14
template <typename R> __device__ __forceinline__ R a_norm(R x, R y, R z)
{
    return a_atleast(a_root(x * x + y * y + z * z), R(1e-14));
}

__device__ __forceinline__ bool a_node(const Grid &g, int &i, int &j, int &k, long long &c)
{
    i = blockIdx.x * BX + threadIdx.x;
    j = blockIdx.y * BY + threadIdx.y;
    k = blockIdx.z;
    if (i >= g.rows || j >= g.cols) return false;
    c = node_index(g, i, j, k);
    return true;
}

// offsets of a node's neighbours in 32 bits (grids hold fewer than 2^31 nodes)
struct Around {
    int im, ip, jm, jp, km, kp;
};
__device__ __forceinline__ Around clamped_around(const Grid &g, int i, int j, int k)
{
    const int rows = g.rows, plane = (int)g.plane;
    return Around{i > 0 ? -1 : 0, i + 1 < g.rows ? 1 : 0, j > 0 ? -rows : 0, j + 1 < g.cols ? rows : 0,
                  k > 0 ? -plane : 0, k + 1 < g.pges ? plane : 0};
}

// a field's values around a node: the node, its six neighbours, its twelve edge neighbours
template <typename T> struct Near {
    T c, xp, xm, yp, ym, zp, zm, xy[4], yz[4], zx[4];  // (+,+), (-,-), then the two of minus sign
};
template <typename T>
__device__ __forceinline__ Near<T> load_near(const T *__restrict__ f, long long c, const Around &n, bool cross)
{
    const T *p = f + c;
    auto at = [&](int o) { return __ldg(p + o); };
    Near<T> r;
    r.c = at(0);
    r.xp = at(n.jp);
    r.xm = at(n.jm);
    r.yp = at(n.ip);
    r.ym = at(n.im);
    r.zp = at(n.kp);
    r.zm = at(n.km);
    if (cross) {
        r.xy[0] = at(n.ip + n.jp);
        r.xy[1] = at(n.im + n.jm);
        r.xy[2] = at(n.ip + n.jm);
        r.xy[3] = at(n.im + n.jp);
        r.yz[0] = at(n.ip + n.kp);
        r.yz[1] = at(n.im + n.km);
        r.yz[2] = at(n.ip + n.km);
        r.yz[3] = at(n.im + n.kp);
        r.zx[0] = at(n.jp + n.kp);
        r.zx[1] = at(n.jm + n.km);
        r.zx[2] = at(n.jp + n.km);
        r.zx[3] = at(n.jm + n.kp);
    }
    return r;
}
__device__ __forceinline__ bool ordinary_near(const Near<double> &r, bool cross)
{
    bool ok = ordinary_tool(r.c) && ordinary_tool(r.xp) && ordinary_tool(r.xm) && ordinary_tool(r.yp) &&
              ordinary_tool(r.ym) && ordinary_tool(r.zp) && ordinary_tool(r.zm);
    if (cross)
#pragma unroll
        for (int q = 0; q < 4; ++q) ok = ok && ordinary_tool(r.xy[q]) && ordinary_tool(r.yz[q]) && ordinary_tool(r.zx[q]);
    return ok;
}

// F's toolbox values at one node: gradient, |grad F| (floored), Hessian, normal, and the
// Heaviside function from the primal max(F, 0) -- tool64_node's expressions in its order
template <typename R> struct FPart {
    R fx, fy, fz, gm, nx, ny, nz, fxx, fyy, fzz, fxy, fyz, fzx, heav;
};
template <typename R, typename T>
__device__ __forceinline__ FPart<R> f_part(const Near<T> &f, const AuxDivisors<T> &t)
{
    FPart<R> r;
    auto pos = [](T x) { return R(vmax(x, T(0))); };
    r.fx = (R(f.xp) - R(f.xm)) / t.two[0];
    r.fy = (R(f.yp) - R(f.ym)) / t.two[1];
    r.fz = (R(f.zp) - R(f.zm)) / t.two[2];
    r.gm = a_norm(r.fx, r.fy, r.fz);
    r.nx = r.fx / r.gm;
    r.ny = r.fy / r.gm;
    r.nz = r.fz / r.gm;
    const R two(2), c(f.c);
    r.fxx = (R(f.xp) - two * c + R(f.xm)) / t.sq[0];
    r.fyy = (R(f.yp) - two * c + R(f.ym)) / t.sq[1];
    r.fzz = (R(f.zp) - two * c + R(f.zm)) / t.sq[2];
    r.fxy = (R(f.xy[0]) + R(f.xy[1]) - R(f.xy[2]) - R(f.xy[3])) / t.four;
    r.fyz = (R(f.yz[0]) + R(f.yz[1]) - R(f.yz[2]) - R(f.yz[3])) / t.four;
    r.fzx = (R(f.zx[0]) + R(f.zx[1]) - R(f.zx[2]) - R(f.zx[3])) / t.four;
    const R px = (pos(f.xp) - pos(f.xm)) / t.two[0];
    const R py = (pos(f.yp) - pos(f.ym)) / t.two[1];
    const R pz = (pos(f.zp) - pos(f.zm)) / t.two[2];
    r.heav = (px * r.fx + py * r.fy + pz * r.fz) / (r.gm * r.gm);
    return r;
}

// The 27 fields of auxi_set_calculus_toolbox at one node, in the kernel's argument order
enum AuxField {
    AU_AX, AU_AY, AU_AZ, AU_AGRADMAG, AU_CX, AU_CY, AU_CZ, AU_NORMCROSS, AU_TX, AU_TY, AU_TZ, AU_NX, AU_NY, AU_NZ,
    AU_AXX, AU_AYY, AU_AZZ, AU_AXY, AU_AYZ, AU_AZX, AU_ALAP, AU_GEODESIC, AU_NORMALCURV, AU_TORSION, AU_BPERP,
    AU_AHEAV, AU_ADELTA, AU_KERNEL_FIELDS
};

// auxi_set_calculus_toolbox.cu:27-197 at one node: A's values `a`, its primal's `p` (the node and
// its six neighbours), F's toolbox values.
template <typename R, typename T>
__device__ __forceinline__ void aux_core(const Near<T> &a, const Near<T> &p, const FPart<R> &fp, const AuxDivisors<T> &t,
                                         T v[AU_KERNEL_FIELDS])
{
    const R ax = (R(a.xp) - R(a.xm)) / t.two[0];
    const R ay = (R(a.yp) - R(a.ym)) / t.two[1];
    const R az = (R(a.zp) - R(a.zm)) / t.two[2];
    const R agm = a_norm(ax, ay, az);
    v[AU_AX] = raw64(ax);
    v[AU_AY] = raw64(ay);
    v[AU_AZ] = raw64(az);
    v[AU_AGRADMAG] = raw64(agm);
    const R fx = fp.fx, fy = fp.fy, fz = fp.fz;
    const R cx = fy * az - fz * ay, cy = fz * ax - fx * az, cz = fx * ay - fy * ax;
    const R ncr = a_norm(cx, cy, cz);
    v[AU_CX] = raw64(cx);
    v[AU_CY] = raw64(cy);
    v[AU_CZ] = raw64(cz);
    v[AU_NORMCROSS] = raw64(ncr);
    const R tx = cx / ncr, ty = cy / ncr, tz = cz / ncr;
    v[AU_TX] = raw64(tx);
    v[AU_TY] = raw64(ty);
    v[AU_TZ] = raw64(tz);
    const R nx = ty * fp.nz - tz * fp.ny, ny = tz * fp.nx - tx * fp.nz, nz = tx * fp.ny - ty * fp.nx;
    v[AU_NX] = raw64(nx);
    v[AU_NY] = raw64(ny);
    v[AU_NZ] = raw64(nz);
    const R two(2), ac(a.c);
    const R axx = (R(a.xp) - two * ac + R(a.xm)) / t.sq[0];
    const R ayy = (R(a.yp) - two * ac + R(a.ym)) / t.sq[1];
    const R azz = (R(a.zp) - two * ac + R(a.zm)) / t.sq[2];
    const R axy = (R(a.xy[0]) + R(a.xy[1]) - R(a.xy[2]) - R(a.xy[3])) / t.four;
    const R ayz = (R(a.yz[0]) + R(a.yz[1]) - R(a.yz[2]) - R(a.yz[3])) / t.four;
    const R azx = (R(a.zx[0]) + R(a.zx[1]) - R(a.zx[2]) - R(a.zx[3])) / t.four;
    const R alap = axx + ayy + azz;
    v[AU_AXX] = raw64(axx);
    v[AU_AYY] = raw64(ayy);
    v[AU_AZZ] = raw64(azz);
    v[AU_AXY] = raw64(axy);
    v[AU_AYZ] = raw64(ayz);
    v[AU_AZX] = raw64(azx);
    v[AU_ALAP] = raw64(alap);
    const R fxx = fp.fxx, fyy = fp.fyy, fzz = fp.fzz, fxy = fp.fxy, fyz = fp.fyz, fzx = fp.fzx, fgm = fp.gm;
    // geodesic curvature n . ((H_F t) x grad A + grad F x (H_A t)) / |grad F x grad A|
    R vx = tx * fxx + ty * fxy + tz * fzx;
    R vy = tx * fxy + ty * fyy + tz * fyz;
    R vz = tx * fzx + ty * fyz + tz * fzz;
    const R w1x = vy * az - vz * ay, w1y = vz * ax - vx * az, w1z = vx * ay - vy * ax;
    vx = tx * axx + ty * axy + tz * azx;
    vy = tx * axy + ty * ayy + tz * ayz;
    vz = tx * azx + ty * ayz + tz * azz;
    const R w2x = fy * vz - fz * vy, w2y = fz * vx - fx * vz, w2z = fx * vy - fy * vx;
    v[AU_GEODESIC] = raw64((nx * (w1x + w2x) + ny * (w1y + w2y) + nz * (w1z + w2z)) / ncr);
    // grad N = H_F / |grad F| - grad F (H_F grad F)^T / |grad F|^3
    const R r1 = fxx * fx + fxy * fy + fzx * fz;
    const R r2 = fxy * fx + fyy * fy + fyz * fz;
    const R r3 = fzx * fx + fyz * fy + fzz * fz;
    const R Nxx = fxx / fgm - a_over3(fx * r1, fgm), Nyx = fxy / fgm - a_over3(fy * r1, fgm),
            Nzx = fzx / fgm - a_over3(fz * r1, fgm);
    const R Nxy = fxy / fgm - a_over3(fx * r2, fgm), Nyy = fyy / fgm - a_over3(fy * r2, fgm),
            Nzy = fyz / fgm - a_over3(fz * r2, fgm);
    const R Nxz = fzx / fgm - a_over3(fx * r3, fgm), Nyz = fyz / fgm - a_over3(fy * r3, fgm),
            Nzz = fzz / fgm - a_over3(fz * r3, fgm);
    vx = Nxx * tx + Nxy * ty + Nxz * tz;
    vy = Nyx * tx + Nyy * ty + Nyz * tz;
    vz = Nzx * tx + Nzy * ty + Nzz * tz;
    v[AU_NORMALCURV] = raw64(-(tx * vx + ty * vy + tz * vz));
    vx = Nxx * nx + Nxy * ny + Nxz * nz;
    vy = Nyx * nx + Nyy * ny + Nyz * nz;
    vz = Nzx * nx + Nzy * ny + Nzz * nz;
    v[AU_TORSION] = raw64(-(tx * vx + ty * vy + tz * vz));
    v[AU_BPERP] = raw64(-(nx * vx + ny * vy + nz * vz));
    // Heaviside and Dirac functions of A from its primal
    const R px = (R(p.xp) - R(p.xm)) / t.two[0], py = (R(p.yp) - R(p.ym)) / t.two[1],
            pz = (R(p.zp) - R(p.zm)) / t.two[2];
    const R dot = px * ax + py * ay + pz * az;
    const R pc(p.c);
    v[AU_AHEAV] = raw64(dot / (agm * agm));
    const R pxx = (R(p.xp) - two * pc + R(p.xm)) / t.sq[0];
    const R pyy = (R(p.yp) - two * pc + R(p.ym)) / t.sq[1];
    const R pzz = (R(p.zp) - two * pc + R(p.zm)) / t.sq[2];
    const R plap = pxx + pyy + pzz;
    v[AU_ADELTA] = raw64(plap / (agm * agm) - a_over4(dot * alap, agm));
}

// pass 1 of the fused form: F recomputed, AHPrimal = max(A, 0) on the fly; writes the
// requested fields, and the values pass 2 needs into `keep` where they are not requested
// (null: not needed): C, |C|, |grad A|, ADiracDelta, AHeaviside and F's Heaviside
template <typename R, typename T>
__device__ __forceinline__ void aux_node(const Near<T> &a, const Near<T> &f, const AuxDivisors<T> &t, T v[AU_KERNEL_FIELDS],
                                         T &fheav)
{
    const FPart<R> fp = f_part<R>(f, t);
    Near<T> p;
    auto pos = [](T x) { return vmax(x, T(0)); };
    p.c = pos(a.c);
    p.xp = pos(a.xp);
    p.xm = pos(a.xm);
    p.yp = pos(a.yp);
    p.ym = pos(a.ym);
    p.zp = pos(a.zp);
    p.zm = pos(a.zm);
    aux_core<R>(a, p, fp, t, v);
    fheav = raw64(fp.heav);
}
template <typename T>
__global__ void __launch_bounds__(ANT) k_aux_pass1(const T *__restrict__ A, const T *__restrict__ F,
                                                   const __grid_constant__ AuxOut<T> o,
                                                   const __grid_constant__ AuxKeep<T> keep,
                                                   const __grid_constant__ Grid g, const __grid_constant__ AuxDivisors<T> t)
{
    int i, j, k;
    long long c;
    if (!a_node(g, i, j, k, c)) return;
    const Around n = clamped_around(g, i, j, k);
    const Near<T> a = load_near(A, c, n, true), f = load_near(F, c, n, true);
    T v[AU_KERNEL_FIELDS], fheav;
    if constexpr (std::is_same<T, float>::value) {
        aux_node<Fast32>(a, f, t, v, fheav);
    } else {
        if (t.ordinary && ordinary_near(a, true) && ordinary_near(f, true))
            aux_node<Short64>(a, f, t, v, fheav);
        else
            aux_node<double>(a, f, t, v, fheav);
    }
#pragma unroll
    for (int q = 0; q < AU_KERNEL_FIELDS; ++q)
        if (o.f[q]) o.f[q][c] = v[q];
    if (keep.cx) keep.cx[c] = v[AU_CX];
    if (keep.cy) keep.cy[c] = v[AU_CY];
    if (keep.cz) keep.cz[c] = v[AU_CZ];
    if (keep.ncr) keep.ncr[c] = v[AU_NORMCROSS];
    if (keep.agm) keep.agm[c] = v[AU_AGRADMAG];
    if (keep.adelta) keep.adelta[c] = v[AU_ADELTA];
    if (keep.aheav) keep.aheav[c] = v[AU_AHEAV];
    if (keep.fheav) keep.fheav[c] = fheav;
}

// periodic neighbours of SD.GD3 (circshift)
__device__ __forceinline__ Around periodic_around(const Grid &g, int i, int j, int k)
{
    const int rows = g.rows, plane = (int)g.plane;
    return Around{i > 0 ? -1 : g.rows - 1,          i + 1 < g.rows ? 1 : 1 - g.rows,
                  j > 0 ? -rows : (g.cols - 1) * rows, j + 1 < g.cols ? rows : (1 - g.cols) * rows,
                  k > 0 ? -plane : (g.pges - 1) * plane, k + 1 < g.pges ? plane : (1 - g.pges) * plane};
}

// pass 2: AFDiracDelta = (C . (grad H_F x grad H_A)) / |C|^2 with GD3.Gradient, and
// ADiracDeltaDn = (Laplacian(H_A) - ADiracDelta Laplacian(A)) / |grad A| with GD3.Laplacian
// (GPUAsetCalculusToolBox.m:56-61)
template <typename R, typename T>
__device__ __forceinline__ T aux_afd(const Near<T> &h1, const Near<T> &h2, T cx, T cy, T cz, T ncr, const AuxDivisors<T> &t)
{
    const R h1x = (R(h1.xp) - R(h1.xm)) / t.two[0], h1y = (R(h1.yp) - R(h1.ym)) / t.two[1],
            h1z = (R(h1.zp) - R(h1.zm)) / t.two[2];
    const R h2x = (R(h2.xp) - R(h2.xm)) / t.two[0], h2y = (R(h2.yp) - R(h2.ym)) / t.two[1],
            h2z = (R(h2.zp) - R(h2.zm)) / t.two[2];
    const R chx = h2y * h1z - h2z * h1y, chy = h2z * h1x - h2x * h1z, chz = h2x * h1y - h2y * h1x;
    const R dot = R(cx) * chx + R(cy) * chy + R(cz) * chz;
    return raw64(dot / (R(ncr) * R(ncr)));
}
template <typename R, typename T> __device__ __forceinline__ R aux_lap(const Near<T> &f, const AuxDivisors<T> &t)
{
    const R two(2), c(f.c);
    const R fxx = (R(f.xp) - two * c + R(f.xm)) / t.sq[0];
    const R fyy = (R(f.yp) - two * c + R(f.ym)) / t.sq[1];
    const R fzz = (R(f.zp) - two * c + R(f.zm)) / t.sq[2];
    return fxx + fyy + fzz;
}
template <typename R, typename T>
__device__ __forceinline__ T aux_ddn(const Near<T> &h, const Near<T> &a, T adelta, T agm, const AuxDivisors<T> &t)
{
    return raw64((aux_lap<R>(h, t) - R(adelta) * aux_lap<R>(a, t)) / R(agm));
}
template <typename T>
__global__ void __launch_bounds__(ANT) k_aux_pass2(const T *__restrict__ A, const __grid_constant__ AuxKeepC<T> keep,
                                                   T *__restrict__ afd, T *__restrict__ addn,
                                                   const __grid_constant__ Grid g, const __grid_constant__ AuxDivisors<T> t)
{
    int i, j, k;
    long long c;
    if (!a_node(g, i, j, k, c)) return;
    const Around n = periodic_around(g, i, j, k);
    const Near<T> h1 = load_near(keep.aheav, c, n, false);
    if (afd) {
        const Near<T> h2 = load_near(keep.fheav, c, n, false);
        const T cx = __ldg(keep.cx + c), cy = __ldg(keep.cy + c), cz = __ldg(keep.cz + c), ncr = __ldg(keep.ncr + c);
        if constexpr (std::is_same<T, float>::value)
            afd[c] = aux_afd<Fast32>(h1, h2, cx, cy, cz, ncr, t);
        else if (t.ordinary && ordinary_near(h1, false) && ordinary_near(h2, false) && ordinary_tool(cx) &&
                 ordinary_tool(cy) && ordinary_tool(cz) && ordinary_tool(ncr))
            afd[c] = aux_afd<Short64>(h1, h2, cx, cy, cz, ncr, t);
        else
            afd[c] = aux_afd<double>(h1, h2, cx, cy, cz, ncr, t);
    }
    if (addn) {
        const Near<T> a = load_near(A, c, n, false);
        const T adelta = __ldg(keep.adelta + c), agm = __ldg(keep.agm + c);
        if constexpr (std::is_same<T, float>::value)
            addn[c] = aux_ddn<Fast32>(h1, a, adelta, agm, t);
        else if (t.ordinary && ordinary_near(h1, false) && ordinary_near(a, false) && ordinary_tool(adelta) &&
                 ordinary_tool(agm))
            addn[c] = aux_ddn<Short64>(h1, a, adelta, agm, t);
        else
            addn[c] = aux_ddn<double>(h1, a, adelta, agm, t);
    }
}

// Masked FP64 integral (SDF3.m:82-85, 212-227): sum over |F| < 2Ds (and |A| < 2Ds where A
// is given) of ((f0 * f1) * f2) * (1 - om), absent factors skipped (an absent f0 is 1),
// the products in FP64 in MATLAB's left-to-right order; per-block partials in a fixed order.
template <typename T>
__global__ void __launch_bounds__(ANT) k_masked_sum(const T *__restrict__ F, const T *__restrict__ A,
                                                    const T *__restrict__ f0, const T *__restrict__ f1,
                                                    const T *__restrict__ f2, const T *__restrict__ om, T thr,
                                                    Grid g, double *__restrict__ partials)
{
    int i, j, k;
    long long c = 0;
    double v = 0.0;
    if (a_node(g, i, j, k, c) && fabs(__ldg(F + c)) < thr && (!A || fabs(__ldg(A + c)) < thr)) {
        v = f0 ? (double)__ldg(f0 + c) : 1.0;
        if (f1) v *= (double)__ldg(f1 + c);
        if (f2) v *= (double)__ldg(f2 + c);
        if (om) v *= 1.0 - (double)__ldg(om + c);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __shared__ double s[ANW];
    const int t = threadIdx.y * BX + threadIdx.x;
    if ((t & 31) == 0) s[t >> 5] = v;
    __syncthreads();
    if (t == 0) {
        double r = 0.0;
        for (int w = 0; w < ANW; ++w) r += s[w];
        partials[blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z)] = r;
    }
}

// the smallest T not below x: x < a_round_up<T>(x') in T  <=>  (double)x < x'
template <typename T> T a_round_up(double x);
template <> double a_round_up<double>(double x) { return x; }
template <> float a_round_up<float>(double x)
{
    float r = (float)x;
    if ((double)r < x) r = std::nextafter(r, std::numeric_limits<float>::infinity());
    return r;
}

}  // namespace

template <typename T>
cudaError_t launch_aux_toolbox(const T *A, const T *F, AuxOut<T> o, AuxKeep<T> keep, const Grid &g, double ds,
                               cudaStream_t s)
{
    const dim3 gr = node_grid(g), bl(BX, BY);
    const AuxDivisors<T> t = aux_divisors(g, ds, T(0));
    T *afd = o.f[AU_KERNEL_FIELDS], *addn = o.f[AU_KERNEL_FIELDS + 1];
    // pass 2 reads the caller's arrays where the caller asked for those fields; pass 1 stores in
    // `keep` what pass 2 needs of the others
    AuxKeepC<T> kc{keep.cx, keep.cy, keep.cz, keep.ncr, keep.agm, keep.adelta, keep.aheav, keep.fheav};
    auto from = [&](T *&k, const T *&r, int field, bool needed) {
        if (!needed) {
            k = nullptr;
        } else if (o.f[field]) {
            r = o.f[field];
            k = nullptr;
        }
    };
    from(keep.cx, kc.cx, AU_CX, afd);
    from(keep.cy, kc.cy, AU_CY, afd);
    from(keep.cz, kc.cz, AU_CZ, afd);
    from(keep.ncr, kc.ncr, AU_NORMCROSS, afd);
    from(keep.agm, kc.agm, AU_AGRADMAG, addn);
    from(keep.adelta, kc.adelta, AU_ADELTA, addn);
    from(keep.aheav, kc.aheav, AU_AHEAV, afd || addn);
    if (!afd) keep.fheav = nullptr;
    k_aux_pass1<T><<<gr, bl, 0, s>>>(A, F, o, keep, g, t);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (!afd && !addn) return cudaSuccess;
    k_aux_pass2<T><<<gr, bl, 0, s>>>(A, kc, afd, addn, g, t);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_masked_sum(const T *F, const T *A, const T *f0, const T *f1, const T *f2, const T *om,
                              const Grid &g, double ds, double *partials, int *nblocks, cudaStream_t s)
{
    if (nblocks) *nblocks = toolbox_partial_blocks(g);
    k_masked_sum<T><<<node_grid(g), dim3(BX, BY), 0, s>>>(F, A, f0, f1, f2, om, a_round_up<T>(2 * ds), g, partials);
    return cudaGetLastError();
}

#define VSL_INSTANTIATE_AUXI(T)                                                                                     \
    template cudaError_t launch_aux_toolbox<T>(const T *, const T *, AuxOut<T>, AuxKeep<T>, const Grid &, double,   \
                                               cudaStream_t);                                                       \
    template cudaError_t launch_masked_sum<T>(const T *, const T *, const T *, const T *, const T *, const T *,     \
                                              const Grid &, double, double *, int *, cudaStream_t);

}  // namespace vsl
