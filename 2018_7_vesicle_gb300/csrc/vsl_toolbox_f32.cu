// vsl_toolbox_f32.cu -- the FP32 (mixed-form) instantiation of the toolbox and
// band-maximum kernels of vsl_toolbox.cuh, compiled with the FP32 form's fast division.
#include "vsl_toolbox.cuh"

namespace vsl {

template <>
cudaError_t launch_toolbox<float>(const float *phi, ToolboxOut<float> out, const Grid &g, double ds, double *partials,
                                  int *nblocks, cudaStream_t s)
{
    const double ds2 = ds * ds;
    const Recips rc{1 / (2 * g.dx),
                    1 / (2 * g.dy),
                    1 / (2 * g.dz),
                    1 / (g.dx * g.dx),
                    1 / (g.dy * g.dy),
                    1 / (g.dz * g.dz),
                    (float)(1 / (2 * g.dx)),
                    (float)(1 / (2 * g.dy)),
                    (float)(1 / (2 * g.dz)),
                    (float)(1 / (g.dx * g.dx)),
                    (float)(1 / (g.dy * g.dy)),
                    (float)(1 / (g.dz * g.dz)),
                    (float)(1 / (4 * ds2))};
    // pages per block: a function of the grid alone (the partials, and so the sums, do
    // not depend on the device), about 2400 blocks where the grid allows, 16 pages at most
    dim3 gr = node_grid(g);
    const long long tiles = (long long)gr.x * gr.y;
    const int kz = (int)std::min<long long>(16, std::max<long long>(1, tiles * g.pges / 2400));
    gr.z = (unsigned)((g.pges + kz - 1) / kz);
    if (nblocks) *nblocks = (int)(tiles * gr.z);
    k_toolbox_tiled<float><<<gr, dim3(BX, BY), 0, s>>>(phi, out, g, ds, round_up<float>(2 * ds), partials, rc, kz);
    return cudaGetLastError();
}

template cudaError_t launch_band_maxabs<float>(const float *, const float *, double, const Grid &, double *, int *,
                                               cudaStream_t);

}  // namespace vsl
