// sweep_chunks.cu -- all linear sweeps of a system in one launch, with the
// system on the chip (sm_100a).
//
// A sweep as a launch of its own costs about 2 us in the captured iteration on a
// mesh of a few thousand cells, whatever its size: launch latency and a chain of
// load latencies. Here each CTA keeps a compact piece of the mesh (SweepChunks:
// coefficients, right-hand sides and iterates of its rows) in shared memory for
// all sweeps, and a sweep takes 0.5-0.9 us: 20 FP64 Jacobi sweeps of 864 cells
// 39 -> 22 us an iteration, 20 two-colour Gauss-Seidel sweeps of 8,000 cells
// 98 -> 40 us.
// After a sweep, CTAs exchange only the rows that others read:
//   * one CTA: a CTA barrier;
//   * up to 16 CTAs: one cluster. A row goes straight into the halos of the CTAs
//     that read it (distributed shared memory), and the hardware barrier is split
//     into arrive and wait;
// The rows that others read are swept first, so their way overlaps the sweep of
// the rest. (Larger systems on one CTA per SM, exchanging through L2 with a flag
// per CTA, measured 1.5-2 us a sweep, no less than the launches of 218k cells.)
//
// The arithmetic and its order are those of the per-sweep kernels
// (k_jacobi_uv, k_gs_uv, k_jacobi1, k_gs1, k_jacobi_uv32;
// linear_solver.cu:9-72), so the results are the same bit for bit. An unused
// slot has the coefficient +0 and reads a zero cell: the sum less +0, or in the
// FP32 form -0 times 0 plus the sum, is the sum. Compiled with --fmad=false.
#include <algorithm>

#include <cooperative_groups.h>

#include "kernels.hpp"

namespace axisim {

namespace {

constexpr int kChunkThreads = 1024;  // at most: 512 where every row has a thread then

template <class T, int NV>
struct Vec;
template <>
struct Vec<double, 1> {
    using type = double;
};
template <>
struct Vec<double, 2> {
    using type = double2;
};
template <>
struct Vec<float, 2> {
    using type = float2;
};

__device__ __forceinline__ double mulSub(double acc, double a, double g) { return acc - a * g; }
__device__ __forceinline__ float mulSub(float acc, float a, float g) { return __fmaf_rn(-a, g, acc); }
__device__ __forceinline__ double comp(double v, int) { return v; }
__device__ __forceinline__ double comp(double2 v, int q) { return q ? v.y : v.x; }
__device__ __forceinline__ float comp(float2 v, int q) { return q ? v.y : v.x; }
__device__ __forceinline__ void setComp(double& v, int, double x) { v = x; }
__device__ __forceinline__ void setComp(double2& v, int q, double x) { (q ? v.y : v.x) = x; }
__device__ __forceinline__ void setComp(float2& v, int q, float x) { (q ? v.y : v.x) = x; }

enum { kOneCta = 0, kCluster = 1 };

template <class T, int NV, int MODE>
__global__ void __launch_bounds__(kChunkThreads, 1) k_sweep_chunks(const Ctl* ctl, SweepChunksDev d, SweepSystem<T, NV> a,
                                                                   int sweeps, int colors) {
    using V = typename Vec<T, NV>::type;
    extern __shared__ __align__(16) unsigned char sm[];
    const SweepChunkInfo I = d.info[blockIdx.x];
    const int rows = I.rows, cells = rows + I.halos + 1;
    // values: iterates (two of them for Jacobi), right-hand sides, inverse diagonals, coefficients, references
    V* x = reinterpret_cast<V*>(sm);
    V* y = colors ? x : x + d.cellsMax;
    V* b = y + d.cellsMax;
    V* inv = b + d.rowsMax;
    T* c = reinterpret_cast<T*>(inv + d.rowsMax);
    ushort4* ref = reinterpret_cast<ushort4*>(c + 4 * (size_t)d.rowsMax);
    int* pushAt = reinterpret_cast<int*>(ref + d.rowsMax);  // a row's run of `push`
    unsigned* push = reinterpret_cast<unsigned*>(pushAt + d.rowsMax + 1);
    const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    for (int i = threadIdx.x; i < rows; i += blockDim.x) ref[i] = d.ref[I.row0 + i];  // static
    if (MODE == kCluster) {
        for (int i = threadIdx.x; i <= rows; i += blockDim.x) pushAt[i] = d.pushAt[I.row0 + blockIdx.x + i] - I.push0;
        for (int q = threadIdx.x; q < I.pushes; q += blockDim.x) push[q] = d.push[I.push0 + q];
    }
    pdlEnter();
    if (ctl->done) return;  // the same on every CTA
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
        const int n = d.cells[I.row0 + i];
        const ushort4 r = ref[i];  // this thread's own store
        const int rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int j = 0; j < 4; j++)
            c[j * d.rowsMax + i] = rr[j] < cells - 1 ? a.AF[(size_t)j * a.N + n] : T(0);
#pragma unroll
        for (int q = 0; q < NV; q++) {
            setComp(b[i], q, a.b[q][n]);
            setComp(inv[i], q, a.inv[q][n]);
            setComp(x[i], q, a.x[q][n]);
        }
    }
    for (int h = threadIdx.x; h < I.halos; h += blockDim.x) {
        const int n = d.cells[d.halo[I.halo0 + h]];
#pragma unroll
        for (int q = 0; q < NV; q++) setComp(x[rows + h], q, a.x[q][n]);
    }
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            setComp(x[cells - 1], q, T(0));
            setComp(y[cells - 1], q, T(0));
        }
    }
    // no CTA writes into another's iterates before that one has read its start
    if (MODE == kCluster) cl.sync();
    else __syncthreads();

    // rows i0 .. i1; send: to the CTAs that read them
    auto sweepRows = [&](int i0, int i1, bool send) {
        for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
            const ushort4 r = ref[i];
            T w[4];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = c[j * d.rowsMax + i];
            const V g[4] = {x[r.x], x[r.y], x[r.z], x[r.w]};
            const V bi = b[i], ai = inv[i], xi = x[i];
            V v;
#pragma unroll
            for (int q = 0; q < NV; q++) {
                T s = comp(bi, q);
#pragma unroll
                for (int j = 0; j < 4; j++) s = mulSub(s, w[j], comp(g[j], q));
                const T inverse = comp(ai, q);
                setComp(v, q, inverse != T(0) ? s * inverse : comp(xi, q));
            }
            y[i] = v;
            if (MODE == kCluster && send)
                for (int q = pushAt[i]; q < pushAt[i + 1]; q++) {
                    const unsigned p = push[q];  // CTA << 16 | its halo cell
                    *cl.map_shared_rank(y + (p & 0xFFFFu), p >> 16) = v;
                }
        }
    };

    const int steps = colors ? sweeps * colors : sweeps;
    for (int s = 0; s < steps; s++) {
        const int k = colors ? s % colors : 0;
        const bool more = s + 1 < steps;
        // A CTA is at most one sweep ahead of a neighbour, whose later rows read
        // the other iterate and no halo; a colour's rows arrive in cells that
        // rows of the same colour do not read.
        sweepRows(I.start[k], I.boundary[k], MODE == kCluster && more);
        // a warp's lanes come from loops of different lengths: the barrier's unaligned form
        if (MODE == kCluster && more) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        sweepRows(I.boundary[k], I.start[k + 1], false);
        if (!colors) {
            V* t = x;
            x = y;
            y = t;
        }
        if (MODE == kCluster && more) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        __syncthreads();
    }
    // the result, in place of the start: two steps or more, so every CTA that
    // reads this one's rows has exchanged once, after it read its start. (A
    // cluster's last pushes ended with the barrier before the last step.)
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
        const int n = d.cells[I.row0 + i];
#pragma unroll
        for (int q = 0; q < NV; q++) {
            const T v = comp(x[i], q);
            if (a.addTo[q]) a.addTo[q][n] += (double)v;
            else a.x[q][n] = v;
        }
    }
}

template <class T, int NV>
size_t chunkShared(const SweepChunksDev& d, bool gaussSeidel) {
    const size_t rows = (size_t)d.rowsMax, cells = (size_t)d.cellsMax;
    const size_t lists = d.chunks > 1 ? rows + 1 + (size_t)d.pushMax : 0;
    return (gaussSeidel ? 1 : 2) * cells * sizeof(T) * NV + rows * (2 * sizeof(T) * NV + 4 * sizeof(T) + 8) +
           sizeof(int) * lists + 16;
}

template <class T, int NV, int MODE>
bool launchMode(const Ctl* ctl, const SweepChunksDev& d, const SweepSystem<T, NV>& a, int sweeps, int colors, cudaStream_t s) {
    const size_t smem = chunkShared<T, NV>(d, colors > 0);
    auto* f = k_sweep_chunks<T, NV, MODE>;
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepChunkShared) != cudaSuccess) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(d.chunks);
    cfg.blockDim = dim3(d.rowsMax <= 512 ? 512 : kChunkThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (MODE == kCluster) {
        if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return false;
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)d.chunks;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
        int runnable = 0;
        cfg.attrs = attr;
        cfg.numAttrs = n;
        if (cudaOccupancyMaxActiveClusters(&runnable, f, &cfg) != cudaSuccess || runnable < 1) return false;
    }
    if (!tNextLaunchPlain) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    tNextLaunchPlain = false;
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, f, ctl, d, a, sweeps, colors) == cudaSuccess;
}

template <class T, int NV>
bool fits(const SweepChunksDev& d, bool gaussSeidel) {
    if (d.chunks < 1 || d.chunks > kSweepClusterChunks) return false;
    return chunkShared<T, NV>(d, gaussSeidel) <= kSweepChunkShared;
}

}  // namespace

bool sweepChunksFit(const SweepChunksDev& d, bool fp32, bool gaussSeidel) {
    return fp32 ? fits<float, 2>(d, false) : fits<double, 2>(d, gaussSeidel);
}

template <class T, int NV>
bool launchSweepChunks(const Ctl* ctl, const SweepChunksDev& d, const SweepSystem<T, NV>& a, int sweeps, int colors,
                       cudaStream_t s) {
    if (!fits<T, NV>(d, colors > 0) || sweeps < 2) return false;
    if (d.chunks == 1) return launchMode<T, NV, kOneCta>(ctl, d, a, sweeps, colors, s);
    return launchMode<T, NV, kCluster>(ctl, d, a, sweeps, colors, s);
}

template bool launchSweepChunks<double, 1>(const Ctl*, const SweepChunksDev&, const SweepSystem<double, 1>&, int, int, cudaStream_t);
template bool launchSweepChunks<double, 2>(const Ctl*, const SweepChunksDev&, const SweepSystem<double, 2>&, int, int, cudaStream_t);
template bool launchSweepChunks<float, 2>(const Ctl*, const SweepChunksDev&, const SweepSystem<float, 2>&, int, int, cudaStream_t);

}  // namespace axisim
