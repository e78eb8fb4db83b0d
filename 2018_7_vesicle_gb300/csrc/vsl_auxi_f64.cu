// vsl_auxi_f64.cu -- the FP64 instantiation of the auxiliary level set toolbox and the
// masked integrals (vsl_auxi.cuh), compiled without multiply-add contraction so that it
// rounds like the reference, and the drop-in of auxi_set_calculus_toolbox.
#include "vsl_auxi.cuh"

namespace vsl {
namespace {

// the reference kernel's own form: F's toolbox fields and AHPrimal read from arrays
template <typename R>
__device__ __forceinline__ void auxi_dropin_node(const Near<double> &a, const Near<double> &p, const double fin[13],
                                                 const Tool64 &t, double v[AU_KERNEL_FIELDS])
{
    FPart<R> fp;
    fp.fx = R(fin[0]);
    fp.fy = R(fin[1]);
    fp.fz = R(fin[2]);
    fp.gm = R(fin[3]);
    fp.nx = R(fin[4]);
    fp.ny = R(fin[5]);
    fp.nz = R(fin[6]);
    fp.fxx = R(fin[7]);
    fp.fyy = R(fin[8]);
    fp.fzz = R(fin[9]);
    fp.fxy = R(fin[10]);
    fp.fyz = R(fin[11]);
    fp.fzx = R(fin[12]);
    aux_core<R>(a, p, fp, t, v);
}
__global__ void __launch_bounds__(ANT) k_auxi_dropin(const __grid_constant__ AuxOut<double> o,
                                                     const double *__restrict__ lsf, const double *__restrict__ ahp,
                                                     const __grid_constant__ AuxFIn<double> fin,
                                                     const __grid_constant__ Grid g, const __grid_constant__ Tool64 t)
{
    int i, j, k;
    long long c;
    if (!a_node(g, i, j, k, c)) return;
    const Around n = clamped_around(g, i, j, k);
    const Near<double> a = load_near(lsf, c, n, true), p = load_near(ahp, c, n, false);
    double f[13], v[AU_KERNEL_FIELDS];
    // the caller's F fields are divided by too: |grad F| a normal divisor, the others as the values
    bool ok = t.ordinary && ordinary_near(a, true) && ordinary_near(p, false);
#pragma unroll
    for (int q = 0; q < 13; ++q) {
        f[q] = fin.f[q][c];
        ok = ok && ordinary_tool(f[q]);
    }
    ok = ok && f[3] >= 1e-14;
    if (ok)
        auxi_dropin_node<Short64>(a, p, f, t, v);
    else
        auxi_dropin_node<double>(a, p, f, t, v);
#pragma unroll
    for (int q = 0; q < AU_KERNEL_FIELDS; ++q) o.f[q][c] = v[q];
}

}  // namespace

VSL_INSTANTIATE_AUXI(double)

cudaError_t launch_auxi_dropin(AuxOut<double> o, const double *lsf, const double *ahp, AuxFIn<double> fin,
                               const Grid &g, double ds, cudaStream_t s)
{
    k_auxi_dropin<<<node_grid(g), dim3(BX, BY), 0, s>>>(o, lsf, ahp, fin, g, tool64(g, ds));
    return cudaGetLastError();
}

}  // namespace vsl
