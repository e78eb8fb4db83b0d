// vsl_tool64.cuh -- one node of the plain FP64 calculus toolbox (set_calculus_toolbox.cu:9-107),
// the reference's expressions in its order, on a number type R: double, or Short64 (the same
// roundings on the short quotients of vsl_short64.cuh) where the node's values are ordinary.
// The kernels that take it are in files compiled without multiply-add contraction (vsl_toolbox.cu,
// vsl_plain.cu); vsl_auxi.cuh takes the divisors and the range test in both precisions.
//
// What bounds it is the FP64 pipe: with general divisions and every field formed at every node a
// node took about 560 FP64 instructions.  Here a field is formed only where it is wanted.
#pragma once

#include "vsl_internal.h"
#include "vsl_short64.cuh"

namespace vsl {
namespace {

// the divisors of a grid: 2 d, d d, (4 Ds) Ds
template <typename D> struct ToolDivisors {
    D two[3], sq[3], four;
    bool ordinary;  // the spacings are within the range of the short quotients
};
using Tool64 = ToolDivisors<Divisor64>;
inline Tool64 tool64(const Grid &g, double ds)
{
    return Tool64{{divisor64(2 * g.dx), divisor64(2 * g.dy), divisor64(2 * g.dz)},
                  {divisor64(g.dx * g.dx), divisor64(g.dy * g.dy), divisor64(g.dz * g.dz)},
                  divisor64(4 * ds * ds),
                  ordinary_spacing(g.dx) && ordinary_spacing(g.dy) && ordinary_spacing(g.dz) && ordinary_spacing(ds)};
}
__device__ __forceinline__ bool ordinary_tool(double x) { return within64(x, -200, 100); }

// fields of the toolbox by what they need: bit q of a mask is field q of TOOLBOX_FIELDS
constexpr unsigned TOOL_NORMALS = 0x70u, TOOL_CROSS = 0x1C00u | 0xC000u, TOOL_MEAN = 0x4000u, TOOL_GAUSS = 0x8000u,
                   TOOL_PRIMAL = 0x30000u, TOOL_ALL = 0x3FFFFu;

// The fields of `want` at one node into v[18].  F(a, b, e), H(a, b, e): the field and its primal
// at row a, column b, page e; the neighbour coordinates are clamped.
template <typename R, class Get, class GetH>
__device__ __forceinline__ void tool64_node(Get F, GetH H, int i, int j, int k, int im, int ip, int jm, int jp, int km,
                                            int kp, const Tool64 &t, unsigned want, double v[18])
{
    const R fc(F(i, j, k));
    const R fxp(F(i, jp, k)), fxm(F(i, jm, k)), fyp(F(ip, j, k)), fym(F(im, j, k)), fzp(F(i, j, kp)), fzm(F(i, j, km));
    const R fx = (fxp - fxm) / t.two[0];
    const R fy = (fyp - fym) / t.two[1];
    const R fz = (fzp - fzm) / t.two[2];
    const double g0 = sqrt(raw64(fx * fx + fy * fy + fz * fz));
    const R gm(vmax(g0, 1e-14));
    v[0] = raw64(fx);
    v[1] = raw64(fy);
    v[2] = raw64(fz);
    v[3] = raw64(gm);
    if (want & TOOL_NORMALS) {
        v[4] = raw64(fx / gm);
        v[5] = raw64(fy / gm);
        v[6] = raw64(fz / gm);
    }
    const R fxx = (fxp - R(2.0) * fc + fxm) / t.sq[0];
    const R fyy = (fyp - R(2.0) * fc + fym) / t.sq[1];
    const R fzz = (fzp - R(2.0) * fc + fzm) / t.sq[2];
    const R lap = fxx + fyy + fzz;
    v[7] = raw64(fxx);
    v[8] = raw64(fyy);
    v[9] = raw64(fzz);
    v[13] = raw64(lap);
    if (want & TOOL_CROSS) {
        const R fxy = (R(F(ip, jp, k)) + R(F(im, jm, k)) - R(F(ip, jm, k)) - R(F(im, jp, k))) / t.four;
        const R fyz = (R(F(ip, j, kp)) + R(F(im, j, km)) - R(F(ip, j, km)) - R(F(im, j, kp))) / t.four;
        const R fzx = (R(F(i, jp, kp)) + R(F(i, jm, km)) - R(F(i, jp, km)) - R(F(i, jm, kp))) / t.four;
        v[10] = raw64(fxy);
        v[11] = raw64(fyz);
        v[12] = raw64(fzx);
        if (want & TOOL_MEAN) {
            const R r1 = fxx * fx + fxy * fy + fzx * fz;
            const R r2 = fxy * fx + fyy * fy + fyz * fz;
            const R r3 = fzx * fx + fyz * fy + fzz * fz;
            v[14] = raw64(-lap / gm + (fx * r1 + fy * r2 + fz * r3) / R(pow_cr<3>(raw64(gm))));
        }
        if (want & TOOL_GAUSS) {
            const R q1 = (fyy * fzz - fyz * fyz) * fx + (fzx * fyz - fxy * fzz) * fy + (fxy * fyz - fzx * fyy) * fz;
            const R q2 = (fyz * fzx - fxy * fzz) * fx + (fxx * fzz - fzx * fzx) * fy + (fzx * fxy - fxx * fyz) * fz;
            const R q3 = (fxy * fyz - fyy * fzx) * fx + (fzx * fxy - fxx * fyz) * fy + (fxx * fyy - fxy * fxy) * fz;
            v[15] = raw64((fx * q1 + fy * q2 + fz * q3) / R(pow_cr<4>(raw64(gm))));
        }
    }
    if (want & TOOL_PRIMAL) {
        const R hc(H(i, j, k));
        const R hxp(H(i, jp, k)), hxm(H(i, jm, k)), hyp(H(ip, j, k)), hym(H(im, j, k)), hzp(H(i, j, kp)), hzm(H(i, j, km));
        const R px = (hxp - hxm) / t.two[0], py = (hyp - hym) / t.two[1], pz = (hzp - hzm) / t.two[2];
        const R dot = px * fx + py * fy + pz * fz;
        const R pxx = (hxp - R(2.0) * hc + hxm) / t.sq[0];
        const R pyy = (hyp - R(2.0) * hc + hym) / t.sq[1];
        const R pzz = (hzp - R(2.0) * hc + hzm) / t.sq[2];
        const R plap = pxx + pyy + pzz;
        const R gm2 = gm * gm;
        v[16] = raw64(dot / gm2);
        v[17] = raw64(plap / gm2 - dot * lap / R(pow_cr<4>(raw64(gm))));
    }
}

}  // namespace
}  // namespace vsl
