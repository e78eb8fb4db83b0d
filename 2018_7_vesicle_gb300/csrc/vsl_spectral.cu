// vsl_spectral.cu -- the bi-Laplacian smoothing of SD.GD3 (GD3.m:434-485) by FFT.
//
// smoothGMRES solves (I + alpha Dt L^2) x = rhs, L the 7-point Laplacian with periodic
// neighbours (GD3.m:110-189), by GMRES preconditioned with FFTs.  That operator is
// circulant, so the DFT diagonalises it exactly: its symbol is
//   1 + alpha Dt lambda^2,  lambda = sum_axis (2 cos(2 pi m / n) - 2) / h^2,
// and x = real(ifftn(fftn(rhs) ./ symbol)) is the system's solution, which the GMRES
// iteration approaches to its tolerance (1e-12).  smoothFFT applies the continuous symbol
// 1 + alpha Dt (kx^2 + ky^2 + kz^2)^2 with the wave numbers of GD3.m:195-207 (the
// fftshifted grid -n/2 : n/2-1, half-integers for odd n) in the same way.
//
// The transforms are cuFFT's complex-to-complex ones (a library FFT, as a GEMM would be
// cuBLAS), in place on a complex copy of rhs held in the caller's workspace; the plans
// are created once per grid shape and precision (the first call for a shape, or
// vsl_workspace_bytes, creates them), with cuFFT's work area also taken from the caller's
// workspace.  The scaling by 1/N of the inverse transform and the real part are fused
// into the last kernel.
#include <cufft.h>

#include <mutex>

#include "vsl_internal.h"
#include "vsl_short64.cuh"

namespace vsl {
namespace {

template <typename T> struct Cx;
template <> struct Cx<double> {
    using type = cufftDoubleComplex;
    static constexpr cufftType kind = CUFFT_Z2Z;
};
template <> struct Cx<float> {
    using type = cufftComplex;
    static constexpr cufftType kind = CUFFT_C2C;
};

struct PlanEntry {
    int rows, cols, pges;
    bool fp64;
    cufftHandle plan;
    size_t work;
};
constexpr int MAX_PLANS = 64;
std::mutex plan_mutex;
PlanEntry plans[MAX_PLANS];
int n_plans = 0;

// the plan for a shape (created on first use, work area supplied per call)
template <typename T> int get_plan(const Grid &g, PlanEntry **out)
{
    const bool fp64 = sizeof(T) == 8;
    for (int e = 0; e < n_plans; ++e)
        if (plans[e].rows == g.rows && plans[e].cols == g.cols && plans[e].pges == g.pges && plans[e].fp64 == fp64) {
            *out = &plans[e];
            return VSL_OK;
        }
    if (n_plans == MAX_PLANS) return VSL_ERR_VALUE;
    PlanEntry p{g.rows, g.cols, g.pges, fp64, 0, 0};
    if (cufftCreate(&p.plan) != CUFFT_SUCCESS) return VSL_ERR_CUDA;
    if (cufftSetAutoAllocation(p.plan, 0) != CUFFT_SUCCESS ||
        cufftMakePlan3d(p.plan, g.pges, g.cols, g.rows, Cx<T>::kind, &p.work) != CUFFT_SUCCESS) {
        cufftDestroy(p.plan);
        return VSL_ERR_CUDA;
    }
    plans[n_plans] = p;
    *out = &plans[n_plans++];
    return VSL_OK;
}

template <typename T>
__global__ void k_to_complex(const T *__restrict__ in, typename Cx<T>::type *__restrict__ out, long long n)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        out[t].x = in[t];
        out[t].y = T(0);
    }
}

// MATLAB's fftshift of -n/2 : n/2-1 at transform index t (GD3.m:195-201)
__device__ __forceinline__ double shifted_wave(int t, int n)
{
    const int s = n / 2;
    const int u = ((t - s) % n + n) % n;
    return -0.5 * n + u;
}

// The part of an axis of n nodes and spacing h in the symbol: the eigenvalue of its second
// difference (exact) or its wave number, at transform index t.
__device__ __forceinline__ double symbol_part(int t, int n, double h, bool exact)
{
    const double two_pi = 6.283185307179586;
    return exact ? (2 * cos(two_pi * t / n) - 2) / (h * h) : two_pi * shifted_wave(t, n) / (n * h);
}

// spec ./= 1 + alpha Dt symbol, symbol = lambda^2 (exact) or |k|^4 (continuous).  The FP64 pipe
// is the bound (three cosines, nine quotients an element): the parts of the symbol are formed
// once per axis and block in shared memory (TABLE: where they fit 48 KB), by one block to an SM,
// and the two quotients share a reciprocal.  96^3: 251 -> 38 us.
constexpr int FILTER_THREADS = 1024, FILTER_TABLE = 6144;
template <typename T, bool TABLE>
__global__ void __launch_bounds__(FILTER_THREADS) k_spectral_filter(typename Cx<T>::type *__restrict__ spec, Grid g,
                                                                    const double *__restrict__ dt, double alpha,
                                                                    int exact)
{
    extern __shared__ double part[];
    double *px = part, *py = px + g.cols, *pz = py + g.rows;
    if (TABLE) {
        for (int t = threadIdx.x; t < g.cols + g.rows + g.pges; t += blockDim.x) {
            const int u = t - g.cols, w = u - g.rows;
            part[t] = u < 0 ? symbol_part(t, g.cols, g.dx, exact)
                            : (w < 0 ? symbol_part(u, g.rows, g.dy, exact) : symbol_part(w, g.pges, g.dz, exact));
        }
        __syncthreads();
    }
    const long long n = g.num;
    const double adt = alpha * __ldg(dt);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(e / g.plane);
        const int r = (int)(e - (long long)k * g.plane);
        const int j = r / g.rows, i = r - j * g.rows;
        const double x = TABLE ? px[j] : symbol_part(j, g.cols, g.dx, exact);
        const double y = TABLE ? py[i] : symbol_part(i, g.rows, g.dy, exact);
        const double z = TABLE ? pz[k] : symbol_part(k, g.pges, g.dz, exact);
        const double s = exact ? x + y + z : x * x + y * y + z * z;
        const double d = 1 + adt * (s * s);
        const double re = spec[e].x, im = spec[e].y;
        if (within64(d, -400, 400) && within64(re, -400, 400) && within64(im, -400, 400)) {
            const double q = reciprocal(d);
            spec[e].x = (T)quotient(re, d, q);
            spec[e].y = (T)quotient(im, d, q);
        } else {
            spec[e].x = (T)(re / d);
            spec[e].y = (T)(im / d);
        }
    }
}

template <typename T>
__global__ void k_real_scaled(const typename Cx<T>::type *__restrict__ spec, T *__restrict__ out, long long n)
{
    const double inv = 1.0 / (double)n;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        out[t] = (T)(spec[t].x * inv);
}

inline int spec_blocks()
{
    static int nb = 0;
    if (nb == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        nb = (sms > 0 ? sms : 132) * 8;
    }
    return nb;
}

}  // namespace

template <typename T> size_t spectral_work_bytes(const Grid &g)
{
    std::lock_guard<std::mutex> lock(plan_mutex);
    PlanEntry *p = nullptr;
    if (get_plan<T>(g, &p) != VSL_OK) return 0;
    return p->work;
}

template <typename T>
int launch_smooth_bilaplacian(const T *rhs, T *out, const double *dt, double alpha, bool exact, const Grid &g,
                              void *spectrum, void *work, size_t work_bytes, cudaStream_t s)
{
    using C = typename Cx<T>::type;
    C *spec = static_cast<C *>(spectrum);
    k_to_complex<T><<<spec_blocks(), 256, 0, s>>>(rhs, spec, g.num);
    if (cudaGetLastError() != cudaSuccess) return VSL_ERR_CUDA;
    {
        std::lock_guard<std::mutex> lock(plan_mutex);
        PlanEntry *p = nullptr;
        if (int st = get_plan<T>(g, &p)) return st;
        if (p->work > work_bytes) return VSL_ERR_WORKSPACE;
        if (cufftSetStream(p->plan, s) != CUFFT_SUCCESS || cufftSetWorkArea(p->plan, work) != CUFFT_SUCCESS)
            return VSL_ERR_CUDA;
        cufftResult r;
        if constexpr (sizeof(T) == 8)
            r = cufftExecZ2Z(p->plan, spec, spec, CUFFT_FORWARD);
        else
            r = cufftExecC2C(p->plan, spec, spec, CUFFT_FORWARD);
        if (r != CUFFT_SUCCESS) return VSL_ERR_CUDA;
        const int parts = g.rows + g.cols + g.pges;
        if (parts <= FILTER_TABLE)
            k_spectral_filter<T, true><<<spec_blocks() / 8, FILTER_THREADS, parts * sizeof(double), s>>>(spec, g, dt, alpha,
                                                                                                   exact ? 1 : 0);
        else
            k_spectral_filter<T, false><<<spec_blocks() / 8, FILTER_THREADS, 0, s>>>(spec, g, dt, alpha, exact ? 1 : 0);
        if (cudaGetLastError() != cudaSuccess) return VSL_ERR_CUDA;
        if constexpr (sizeof(T) == 8)
            r = cufftExecZ2Z(p->plan, spec, spec, CUFFT_INVERSE);
        else
            r = cufftExecC2C(p->plan, spec, spec, CUFFT_INVERSE);
        if (r != CUFFT_SUCCESS) return VSL_ERR_CUDA;
    }
    k_real_scaled<T><<<spec_blocks(), 256, 0, s>>>(spec, out, g.num);
    return cudaGetLastError() == cudaSuccess ? VSL_OK : VSL_ERR_CUDA;
}

template size_t spectral_work_bytes<double>(const Grid &);
template size_t spectral_work_bytes<float>(const Grid &);
template int launch_smooth_bilaplacian<double>(const double *, double *, const double *, double, bool, const Grid &,
                                               void *, void *, size_t, cudaStream_t);
template int launch_smooth_bilaplacian<float>(const float *, float *, const double *, double, bool, const Grid &,
                                              void *, void *, size_t, cudaStream_t);

}  // namespace vsl
