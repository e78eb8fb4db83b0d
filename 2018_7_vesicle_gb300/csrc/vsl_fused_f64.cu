// vsl_fused_f64.cu -- instantiation of the fused stage kernels for double.
// FP64 plain form: built with -fmad=false, every product and sum rounded on its own as in
// the reference's FP64 kernels.
#include "vsl_fused.cuh"
#include "vsl_stage64.cuh"

namespace vsl {
VSL_INSTANTIATE_FUSED(double)
template cudaError_t launch_crossing<double>(const double *, Ptr6<const double>, Ptr6<double>, NodeList, const Grid &,
                                             bool, cudaStream_t);
template cudaError_t launch_enork2_crossing<double>(const double *, Ptr6<const double>, Ptr6<double>, NodeList,
                                                    const Grid &, cudaStream_t);

cudaError_t launch_condition_reset(cudaGraphConditionalHandle handle, cudaStream_t s)
{
    k_condition_reset<<<1, 1, 0, s>>>(handle);
    return cudaGetLastError();
}
}  // namespace vsl
