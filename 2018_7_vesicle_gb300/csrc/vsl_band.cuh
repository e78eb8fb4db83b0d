// vsl_band.cuh -- band nodes (next to the interface) as tasks sorted by stencil kind.
//
// A band node needs, on each axis, either the uniform one-sided derivatives or the nonuniform
// ones with the interface inserted, which cost about ten times as much.  With one thread per
// node a warp runs both kinds of all three axes for whichever of its lanes need them, one
// after the other, and that chain is the time of a launch on a small grid (an extension stage
// took 11 us on every grid up to 64^3).  Here a block takes a chunk of band nodes, lists the
// derivatives they need by kind in shared memory (forward nonuniform, backward nonuniform,
// uniform) and evaluates each list in full warps: no lane waits for another kind, one axis is
// one task, and a transport stage, which multiplies only the upwind side of an axis by a speed,
// takes only that side of the nonuniform ones.  A last pass combines each node's derivatives.
// The lists' order has no part in the results.
//
// The phases between barriers cost throughput, so the mixed form takes this on small grids and
// one node per thread on the others (and in batches).  Measured on GB300, ms, tasks against one
// node per thread: 30 WENO5 extension pseudo-steps 32^3 0.84 / 1.27, 64^3 1.03 / 1.41, 96^3
// 1.61 / 1.78, 128^3 2.86 / 2.85, 192^3 7.16 / 6.92; 30 reinitialization pseudo-steps 32^3
// 1.35 / 1.48, 64^3 1.56 / 1.73, 128^3 3.92 / 3.98; a stage of 160^3 68.0 / 65.3 us.
// So do dense bands (folded or many interfaces) on small grids: ten reinitialization pseudo-steps of
// 64^3 with 35,000 / 53,000 / 191,000 band nodes 0.715 / 0.725, 0.812 / 0.744, 1.43 / 1.05, of 128^3
// with 32,000 / 126,000 / 1,530,000 1.41 / 1.42, 2.03 / 1.79, 9.2 / 6.0 (10 shapes, 9 bands each).
#pragma once

#include <cstdint>

#include "vsl_fused.cuh"

namespace vsl {
namespace {

enum BandTask { BT_FORE = 0, BT_BACK = 1, BT_UNIFORM = 2, BT_KINDS = 3 };
// the largest grids (nodes) whose reinitialization and extension bands run as tasks in the mixed
// form, and the most band nodes that do
constexpr long long REINIT_TASKS_GRID = 128LL * 128 * 128, EXTEND_TASKS_GRID = 112LL * 112 * 112;
constexpr unsigned EXTEND_TASKS_MOST = 20000, REINIT_TASKS_MOST = 40000;

// the shared memory of a chunk of N nodes
template <typename T, int N> struct BandChunk {
    static constexpr int NODES = N;
    using Real = T;
    T df[3][N], db[3][N];  // the derivatives (0 where not evaluated)
    unsigned c[N];
    int i[N], j[N], k[N];
    uint8_t fl[N];
    unsigned count[BT_KINDS];
    uint16_t task[BT_KINDS][3 * N];  // axis * N + node
};

// Runs the `n` band nodes of a list over `nb` blocks of NT threads (this one is block b).
// Ops:
//   unsigned node(t), uint8_t flags(c), const Grid &grid()   the t-th node, its classification
//   unsigned kinds(ch, node, ax)       bits of the tasks that the axis needs
//   void eval(ch, kind, node, ax)      one task: writes ch.df / ch.db
//   void finish(ch, node)              the node's update
template <int NT, class Ops, class Chunk>
__device__ __forceinline__ void run_band(const Ops &ops, Chunk &ch, unsigned n, unsigned b, unsigned nb, int tid)
{
    constexpr int N = Chunk::NODES;
    static_assert(N <= NT, "one node per thread");
    const unsigned plane = (unsigned)ops.grid().plane, rows = (unsigned)ops.grid().rows;
    for (unsigned base = b * N; base < n; base += nb * N) {
        const int m = (int)min((unsigned)N, n - base);
        if (tid < BT_KINDS) ch.count[tid] = 0u;
        if (tid < m) {
            const unsigned c = ops.node(base + tid), k = c / plane, r = c - k * plane, j = r / rows;
            ch.c[tid] = c;
            ch.i[tid] = (int)(r - j * rows);
            ch.j[tid] = (int)j;
            ch.k[tid] = (int)k;
            ch.fl[tid] = ops.flags(c);
        }
        __syncthreads();
        for (int q = tid; q < 3 * N; q += NT) {
            const int node = q % N, ax = q / N;
            if (node >= m) continue;
            ch.df[ax][node] = typename Chunk::Real(0);
            ch.db[ax][node] = typename Chunk::Real(0);
            if (ch.fl[node] & FIXED_BIT) continue;
            const unsigned need = ops.kinds(ch, node, ax);
#pragma unroll
            for (int kind = 0; kind < BT_KINDS; ++kind)
                if (need & (1u << kind)) ch.task[kind][atomicAdd(&ch.count[kind], 1u)] = (uint16_t)q;
        }
        __syncthreads();
        // warps take groups of 32 tasks of one kind
        const int n0 = (int)ch.count[0], n1 = (int)ch.count[1], n2 = (int)ch.count[2];
        const int g0 = (n0 + 31) / 32, g1 = g0 + (n1 + 31) / 32, g2 = g1 + (n2 + 31) / 32;
        for (int w = tid / 32; w < g2; w += NT / 32) {
            const int kind = w < g0 ? BT_FORE : (w < g1 ? BT_BACK : BT_UNIFORM);
            const int at = (w - (kind == BT_FORE ? 0 : (kind == BT_BACK ? g0 : g1))) * 32 + (tid & 31);
            if (at < (kind == BT_FORE ? n0 : (kind == BT_BACK ? n1 : n2))) {
                const int q = ch.task[kind][at];
                ops.eval(ch, kind, q % N, q / N);
            }
        }
        __syncthreads();
        if (tid < m) ops.finish(ch, tid);
        __syncthreads();
    }
}

// the axis line of a chunk's node
template <class Chunk> __device__ __forceinline__ AxisLine band_line(const Chunk &ch, const Grid &g, int node, int ax)
{
    return axis_line(g, ch.i[node], ch.j[node], ch.k[node], ax);
}

// does the field change sign between the node and a neighbour on the line (the
// reinitialization's trigger)
template <typename T> __device__ __forceinline__ bool sign_change(const T *__restrict__ f, const AxisLine &L)
{
    const T a = __ldg(f + L.base + (long long)clampi(L.c - 1, L.n) * L.stride);
    const T b = __ldg(f + L.base + (long long)L.c * L.stride);
    const T c = __ldg(f + L.base + (long long)clampi(L.c + 1, L.n) * L.stride);
    return a * b < T(0) || b * c < T(0);
}

// one side of the interface-aware derivatives of the mixed form, out of line (the register
// cap of the kernels that call it)
template <typename T, bool ENO3> __device__ __noinline__ T nonuniform_side_dd(const T G[6], const T dd[6], bool back)
{
    if constexpr (ENO3) {
        T f, b;
        eno3_nonuniform_pair_dd(G, dd, f, b);
        return back ? b : f;
    } else {
        return back ? weno_nonuniform_back_dd(G, dd) : weno_nonuniform_fore_dd(G, dd);
    }
}

}  // namespace
}  // namespace vsl
