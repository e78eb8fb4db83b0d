// vsl_toolbox.cu -- the FP64 instantiation of the toolbox and band-maximum kernels
// (vsl_toolbox.cuh), the fixed-order sums of the block partials and the time step.
#include "vsl_toolbox.cuh"
#include "vsl_tool64.cuh"

namespace vsl {
namespace {

// The plain FP64 toolbox, one node per thread, the reference's expressions (tool64_node).  The
// area and volume terms need the Heaviside and Dirac functions, which are formed at every node
// only where an output asks for them; otherwise at the nodes that carry a term (F < 2 Ds with a
// positive value among the seven; without one the volume term is exactly 1 and the area term 0),
// listed per block in shared memory and evaluated in full warps: a warp with one such node would
// otherwise run the FP64 block for all its lanes.  Each term returns to its node's thread, so the
// sums keep their order: warp shuffle tree, then the block's warps.
// thr2ds: 2 Ds (the reference's band tests).
template <class Get>
__device__ __noinline__ void tool64_general(Get F, int i, int j, int k, int im, int ip, int jm, int jp, int km, int kp,
                                            const Tool64 &t, unsigned want, double v[18])
{
    tool64_node<double>(F, [&](int a, int b, int e) { return vmax(F(a, b, e), 0.0); }, i, j, k, im, ip, jm, jp, km, kp,
                        t, want, v);
}

__global__ void __launch_bounds__(NT) k_toolbox64(const double *__restrict__ f, const __grid_constant__ ToolboxOut<double> o,
                                                  const __grid_constant__ Grid g, double thr2ds,
                                                  double *__restrict__ partials, const __grid_constant__ Tool64 tc,
                                                  unsigned want)
{
    const int i0 = blockIdx.x * BX, j0 = blockIdx.y * BY, k = blockIdx.z;
    const int t = threadIdx.y * BX + threadIdx.x;
    const unsigned rows = (unsigned)g.rows, plane = (unsigned)g.plane;
    // node offsets in 32 bits (grids hold fewer than 2^31 nodes)
    auto F = [&](int a, int b, int e) { return __ldg(f + ((unsigned)e * plane + (unsigned)b * rows + (unsigned)a)); };
    const int km = clampi(k - 1, g.pges), kp = clampi(k + 1, g.pges);
    // the fields of `mask` at (i, j, k)
    auto node = [&](int i, int j, unsigned mask, double v[18]) {
        const int im = clampi(i - 1, g.rows), ip = clampi(i + 1, g.rows);
        const int jm = clampi(j - 1, g.cols), jp = clampi(j + 1, g.cols);
        bool ok = tc.ordinary && ordinary_tool(F(i, j, k)) && ordinary_tool(F(i, jp, k)) && ordinary_tool(F(i, jm, k)) &&
                  ordinary_tool(F(ip, j, k)) && ordinary_tool(F(im, j, k)) && ordinary_tool(F(i, j, kp)) &&
                  ordinary_tool(F(i, j, km));
        if (mask & TOOL_CROSS)
            ok = ok && ordinary_tool(F(ip, jp, k)) && ordinary_tool(F(im, jm, k)) && ordinary_tool(F(ip, jm, k)) &&
                 ordinary_tool(F(im, jp, k)) && ordinary_tool(F(ip, j, kp)) && ordinary_tool(F(im, j, km)) &&
                 ordinary_tool(F(ip, j, km)) && ordinary_tool(F(im, j, kp)) && ordinary_tool(F(i, jp, kp)) &&
                 ordinary_tool(F(i, jm, km)) && ordinary_tool(F(i, jp, km)) && ordinary_tool(F(i, jm, kp));
        if (ok)
            tool64_node<Short64>(F, [&](int a, int b, int e) { return vmax(F(a, b, e), 0.0); }, i, j, k, im, ip, jm, jp,
                                 km, kp, tc, mask, v);
        else
            tool64_general(F, i, j, k, im, ip, jm, jp, km, kp, tc, mask, v);
    };
    const int i = i0 + (int)threadIdx.x, j = j0 + (int)threadIdx.y;
    const bool in = i < g.rows && j < g.cols;
    double area = 0.0, vol = 0.0;
    int units = 0;  // volume terms equal to exactly 1
    // the terms of a node from its Heaviside and Dirac values
    auto terms = [&](double fc, double heav, double delta) {
        if (fabs(fc) < thr2ds) area += delta;
        if (fc < thr2ds) {
            const double v1 = 1 - heav;  // heav == 0 (no positive neighbour): exactly 1
            if (v1 == 1.0)
                units += 1;
            else
                vol += v1;
        }
    };
    const bool direct = want & TOOL_PRIMAL;
    if (in && want) {
        double v[18];
        node(i, j, want, v);
        const long long c = node_index(g, i, j, k);
#pragma unroll
        for (int q = 0; q < 18; ++q)
            if (o.f[q]) o.f[q][c] = v[q];
        if (direct) terms(F(i, j, k), v[16], v[17]);
    }
    if (!partials) return;
    if (!direct) {
        __shared__ unsigned count;
        __shared__ uint8_t list[NT];
        __shared__ double heav[NT], delta[NT];
        if (t == 0) count = 0u;
        __syncthreads();
        bool need = false;
        double fc = 0.0;
        if (in) {
            fc = F(i, j, k);
            if (fc < thr2ds) {
                const double w[7] = {fc,
                                     F(i, clampi(j + 1, g.cols), k),
                                     F(i, clampi(j - 1, g.cols), k),
                                     F(clampi(i + 1, g.rows), j, k),
                                     F(clampi(i - 1, g.rows), j, k),
                                     F(i, j, kp),
                                     F(i, j, km)};
#pragma unroll
                for (int q = 0; q < 7; ++q) need = need || w[q] > 0.0 || !ordinary_tool(w[q]);
                need = need || !tc.ordinary;
                if (!need) units = 1;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, need), lane = t & 31;
        unsigned base = 0;
        if (m && lane == 0) base = atomicAdd(&count, (unsigned)__popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (need) list[base + __popc(m & ((1u << lane) - 1u))] = (uint8_t)t;
        __syncthreads();
        const unsigned n = count;
        if (t < (int)n) {
            const int at = list[t];
            double v[18];
            node(i0 + at % BX, j0 + at / BX, TOOL_PRIMAL, v);
            heav[at] = v[16];
            delta[at] = v[17];
        }
        __syncthreads();
        if (need) terms(fc, heav[t], delta[t]);
    }
    // Volume terms equal to exactly 1 are counted as integers; only warps holding other terms run
    // the FP64 shuffle tree.  Per block: partial = (double)count + FP64 tree sum of the rest, in a
    // fixed order.
    __shared__ double sa[NW], sv[NW];
    __shared__ int sc[NW];
    const int ones = __reduce_add_sync(0xffffffffu, units);
    if (__any_sync(0xffffffffu, area != 0.0)) area = warp_sum(area);
    if (__any_sync(0xffffffffu, vol != 0.0)) vol = warp_sum(vol);
    if ((t & 31) == 0) {
        sa[t >> 5] = area;
        sv[t >> 5] = vol;
        sc[t >> 5] = ones;
    }
    __syncthreads();
    if (t == 0) {
        double a = 0.0, v = 0.0;
        int n = 0;
        for (int w = 0; w < NW; ++w) {
            a += sa[w];
            v += sv[w];
            n += sc[w];
        }
        const long long b = block_linear();
        partials[2 * b] = a;
        partials[2 * b + 1] = (double)n + v;
    }
}

// result[q] = scale * sum_b partials[NC*b + q] in a fixed order (one block of 1024): per thread, per
// warp by shuffles, then the warps.  One block has one SM's FP64 pipe, 16 cycles a warp's
// instruction, and that and the chain of additions are its time: warps past the last partial are
// left out (their sums are exact zeros), and the components go side by side, each summed over the
// warps by a thread of its own (48^3, 432 partials of 2: 7.3 -> 4.3 us).  With many partials it
// waits on their loads, eight rows of which are in flight (the component count is the compiler's,
// so that no branch parts them: SUMLINE).
template <int NC>
__global__ void __launch_bounds__(1024) k_sum_partials(const double *__restrict__ partials, int nblocks, double scale,
                                                       double *__restrict__ result)
{
    __shared__ double s[NC][32];
    const int warp = threadIdx.x >> 5, warps = min((int)(blockDim.x >> 5), (nblocks + 31) >> 5);
    if (warp < warps) {
        double acc[NC];
#pragma unroll
        for (int q = 0; q < NC; ++q) acc[q] = 0.0;
        // the additions keep their order
#pragma unroll 8
        for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
#pragma unroll
            for (int q = 0; q < NC; ++q) acc[q] += partials[(long long)NC * b + q];
        }
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            acc[q] = warp_sum(acc[q]);
            if ((threadIdx.x & 31) == 0) s[q][warp] = acc[q];
        }
    }
    __syncthreads();
    if (threadIdx.x < NC) {
        double tot = 0.0;
        for (int w = 0; w < warps; ++w) tot += s[threadIdx.x][w];
        result[threadIdx.x] = tot * scale;
    }
}

__global__ void __launch_bounds__(1024) k_time_step(const double *__restrict__ partials, int nblocks, double cfl_ds,
                                                    double *__restrict__ dt, double *__restrict__ vmax)
{
    __shared__ double s[32];
    double m = 0.0;
#pragma unroll 8
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) m = fmax(m, partials[b]);
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r = fmax(r, s[w]);
        if (vmax) *vmax = r;
        *dt = r > 0.0 ? cfl_ds / r : 0.0;
    }
}

}  // namespace

int toolbox_partial_blocks(const Grid &g)
{
    dim3 gr = node_grid(g);
    return (int)((long long)gr.x * gr.y * gr.z);
}

cudaError_t launch_sum_partials(const double *partials, int nblocks, int ncomp, double scale, double *result,
                                cudaStream_t s)
{
    switch (ncomp) {
    case 1: k_sum_partials<1><<<1, 1024, 0, s>>>(partials, nblocks, scale, result); break;
    case 2: k_sum_partials<2><<<1, 1024, 0, s>>>(partials, nblocks, scale, result); break;
    case 4: k_sum_partials<4><<<1, 1024, 0, s>>>(partials, nblocks, scale, result); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_time_step(const double *partials, int nblocks, double cfl_ds, double *dt, double *vmax,
                             cudaStream_t s)
{
    k_time_step<<<1, 1024, 0, s>>>(partials, nblocks, cfl_ds, dt, vmax);
    return cudaGetLastError();
}

template <>
cudaError_t launch_toolbox<double>(const double *phi, ToolboxOut<double> out, const Grid &g, double ds, double *partials,
                                   int *nblocks, cudaStream_t s)
{
    // one node per thread, the reference's summation blocks
    if (nblocks) *nblocks = toolbox_partial_blocks(g);
    unsigned want = 0u;
    for (int q = 0; q < 18; ++q)
        if (out.f[q]) want |= 1u << q;
    k_toolbox64<<<node_grid(g), dim3(BX, BY), 0, s>>>(phi, out, g, 2 * ds, partials, tool64(g, ds), want);
    return cudaGetLastError();
}
template cudaError_t launch_band_maxabs<double>(const double *, const double *, double, const Grid &, double *,
                                                int *, cudaStream_t);

}  // namespace vsl
