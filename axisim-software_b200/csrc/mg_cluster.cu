// mg_cluster.cu -- the deep levels of the multigrid V-cycle in one launch of
// one thread-block cluster (sm_100a).
//
// What bounds these levels is not bandwidth but the chain of dependent
// phases: each phase on a few thousand rows is a handful of loads and an
// ordered sum, and as a launch of its own it costs 3-4 us in the captured
// iteration, whatever its size. Here one CTA of a 16-CTA cluster holds every
// level of at most kClusterSolo cells in shared memory, and the other fifteen
// hold the levels up to kClusterMaxCells, one contiguous chunk of rows each.
//   * A chunk's rows and its halo (the cells of other chunks that they refer
//     to) lie in shared memory, so a row reads local memory only. The chunks
//     exchange values through L2 (written by the owner, fetched into the halo
//     after the hardware cluster barrier): reading single values of other CTAs
//     through distributed shared memory measured two lanes a cycle, three
//     times the cost of a step.
//   * A restriction forms the halo's right-hand sides and first sweeps as well
//     as its own, and a prolongation corrects the halo too, so a level costs
//     two cluster barriers (about 500 cycles each) a cycle.
//   * The topology is packed on the host, ready for shared memory, and fetched
//     with the list of steps before the kernel waits for its predecessor; read
//     from the kernel's parameters, each step's look-ups were a chain of
//     constant-bank misses of about 1,000 cycles.
//   * A row has its slots in groups of eight and at least one group (the levels'
//     slices are padded), so its loads have constant offsets. An unused slot refers to the chunk's
//     zero cell, which holds -0.0, and has the coefficient +0: its product is
//     -0.0 and adding it leaves every sum as it is, bit for bit.
//
// Every row keeps the arithmetic and the order of sums of the per-phase
// kernels (mg.cu: jacobiRow, residualRow, prolongSmoothRow, gatherFinish;
// MultigridSolver, solver/source/multigrid.cu:398-662), so the results are the
// same bit for bit. Compiled with --fmad=false.
#include <algorithm>
#include <cmath>
#include <cstring>

#include <cooperative_groups.h>

#include "coarsest.cuh"
#include "host_prep.hpp"
#include "kernels.hpp"

namespace axisim {

namespace {

inline size_t align16(size_t n) { return (n + 15) & ~size_t(15); }

template <class T>
__device__ __forceinline__ T tinyOf();
template <>
__device__ __forceinline__ double tinyOf<double>() {
    return 1.0e-30;
}
template <>
__device__ __forceinline__ float tinyOf<float>() {
    return 1.0e-30f;
}

extern __shared__ __align__(16) unsigned char smraw[];

template <class U>
__device__ __forceinline__ U& at(uint32_t o) {
    return *reinterpret_cast<U*>(smraw + o);
}

__device__ __forceinline__ void copy16(uint32_t o, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smraw + o)),
                 "l"(src)
                 : "memory");
}
template <class T>
__device__ __forceinline__ void copyElem(uint32_t o, const T* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smraw + o)),
                 "l"(src), "n"(sizeof(T))
                 : "memory");
}
__device__ __forceinline__ void copyWait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One level on one CTA, as its packed block describes it. Values per level:
// two iterates of `cells` (rows, halo, zero cell), right-hand side of the
// rows, diagonal of rows and halo, off-diagonals.
template <class T>
struct View {
    ClusterRows l;
    uint32_t x0, x1, b, AC, AF;
    __device__ __forceinline__ uint32_t iterate(int which) const { return which ? x1 : x0; }
};
template <class T>
__device__ __forceinline__ View<T> viewOf(int i) {
    View<T> w;
    w.l = at<ClusterRows>((uint32_t)(i * sizeof(ClusterRows)));
    w.x0 = sizeof(T) == 8 ? w.l.value64 : w.l.value32;
    w.x1 = w.x0 + (uint32_t)w.l.cells * (uint32_t)sizeof(T);
    w.b = w.x1 + (uint32_t)w.l.cells * (uint32_t)sizeof(T);
    w.AC = w.b + (uint32_t)w.l.cells * (uint32_t)sizeof(T);
    w.AF = w.AC + (uint32_t)w.l.cells * (uint32_t)sizeof(T);
    return w;
}

// A x of row n in slot order from the diagonal's term (axEager, mg.cu): eight
// slots' references and coefficients, and then their values, are read before
// the ordered sum.
template <class T>
__device__ __forceinline__ T rowAx(const View<T>& L, int n, uint32_t x, T Ax) {
    uint32_t s0 = (uint32_t)((n & ~31) * 8 + (n & 31));
    int groups = 1;
    if (L.l.wide) {  // some slice has more than eight slots a row
        const uint32_t w = at<uint32_t>(L.l.so + 4 * (n >> 5));
        s0 = (w & 0xFFFFFFu) + (n & 31);
        groups = (int)(w >> 24);
    }
    for (int q = 0; q < groups; q++, s0 += 256) {
        const uint32_t ia = L.l.nb + 2 * s0, ca = L.AF + (uint32_t)sizeof(T) * s0;
        uint32_t k[8];
        T c[8], g[8];
#pragma unroll
        for (int j = 0; j < 8; j++) k[j] = at<uint16_t>(ia + 64 * j);
#pragma unroll
        for (int j = 0; j < 8; j++) c[j] = at<T>(ca + 32 * (uint32_t)sizeof(T) * j);
#pragma unroll
        for (int j = 0; j < 8; j++) g[j] = at<T>(x + k[j] * (uint32_t)sizeof(T));
#pragma unroll
        for (int j = 0; j < 8; j++) Ax += c[j] * g[j];
    }
    return Ax;
}

// y = x + w (b - A x) / A_C on this CTA's rows (jacobiRow), or y = b - A x
// (residualRow), into shared memory and, where another CTA may read it, L2.
template <class T>
__device__ __forceinline__ void rowsOf(const View<T>& L, uint32_t x, uint32_t y, T* out, T w, bool residual) {
    for (int n = threadIdx.x; n < L.l.rows; n += blockDim.x) {
        const uint32_t o = (uint32_t)n * (uint32_t)sizeof(T);
        const T ac = at<T>(L.AC + o), bn = at<T>(L.b + o), xn = at<T>(x + o);
        const T r = bn - rowAx<T>(L, n, x, ac * xn);
        T yn = r;
        if (!residual) yn = fabs(ac) < tinyOf<T>() ? xn : xn + w * r / ac;
        at<T>(y + o) = yn;
        if (out) out[L.l.row0 + n] = yn;
    }
}

// x + scale P xc of the rows and the halo, in place (the first half of
// prolongSmoothRow). xc: the coarser level's values, by global cell in L2 or by
// row in this CTA's shared memory.
template <class T>
__device__ __forceinline__ void correct(const View<T>& L, uint32_t x, const T* xc, uint32_t xcHere, T scale, T* out) {
    for (int n = threadIdx.x; n < L.l.live; n += blockDim.x) {
        const uint32_t o = (uint32_t)n * (uint32_t)sizeof(T);
        const int c = at<int>(L.l.c2c + 4 * n);
        const T e = xc ? __ldcg(xc + c) : at<T>(xcHere + (uint32_t)c * (uint32_t)sizeof(T));
        const T v = at<T>(x + o) + scale * e;
        at<T>(x + o) = v;
        if (out && n < L.l.rows) out[L.l.row0 + n] = v;
    }
}

// b = sum of the members' residuals on the finer level, in member order, and
// x = 0 or the first sweep from zero (gatherCell, gatherFinish), for the rows
// and the halo.
template <class T>
__device__ __forceinline__ void restrictTo(const View<T>& C, const T* r, uint32_t rHere, uint32_t x, bool first, T w) {
    for (int c = threadIdx.x; c < C.l.live; c += blockDim.x) {
        const uint32_t o = (uint32_t)c * (uint32_t)sizeof(T);
        const int q0 = at<int>(C.l.ms + 4 * c), q1 = at<int>(C.l.ms + 4 * c + 4);
        const T ac = at<T>(C.AC + o);
        T sum = T(0);
        for (int q = q0; q < q1; q += 4) {
            int m[4];
            T v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) m[u] = at<int>(C.l.ml + 4 * min(q + u, q1 - 1));
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = r ? __ldcg(r + m[u]) : at<T>(rHere + (uint32_t)m[u] * (uint32_t)sizeof(T));
#pragma unroll
            for (int u = 0; u < 4; u++) sum = q + u < q1 ? sum + v[u] : sum;
        }
        at<T>(C.b + o) = sum;
        at<T>(x + o) = !first || fabs(ac) < tinyOf<T>() ? T(0) : T(0) + w * (sum - ac * T(0)) / ac;
    }
}

// The halo of an iterate that its owners have written to L2.
template <class T>
__device__ __forceinline__ void fetchHalo(const View<T>& L, uint32_t x, const T* from) {
    for (int h = threadIdx.x; h < L.l.live - L.l.rows; h += blockDim.x)
        at<T>(x + (uint32_t)(L.l.rows + h) * (uint32_t)sizeof(T)) = __ldcg(from + at<int>(L.l.halo + 4 * h));
}

// Barrier of the CTA's first `threads` threads (a multiple of 32).
__device__ __forceinline__ void partSync(int threads) {
    if (threads <= 32) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// The coarsest level's sweeps (coarsest.cuh), a row a thread; only the warps that
// hold rows take part (`part` threads of at most the CTA's).
template <class T>
__device__ __forceinline__ void coarsestRows(const View<T>& L, uint32_t x, uint32_t y, T w, int sweeps, int part) {
    const int n = min((int)threadIdx.x, L.l.rows - 1);  // a surplus lane repeats the last row and stores nothing
    const bool live = (int)threadIdx.x < L.l.rows;
    const uint32_t s0 = (uint32_t)((n & ~31) * 8 + (n & 31)), o = (uint32_t)n * (uint32_t)sizeof(T);
    T c[8];
    uint32_t adr[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        c[j] = at<T>(L.AF + (uint32_t)sizeof(T) * (s0 + 32 * j));
        adr[j] = x + at<uint16_t>(L.l.nb + 2 * (s0 + 32 * j)) * (uint32_t)sizeof(T);
    }
    coarsestSweeps<T>(smraw, x, y, o, c, adr, at<T>(L.AC + o), at<T>(L.b + o), live, w, sweeps,
                      [&] { partSync(part); });
}

template <class T, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_mg_cluster(const Ctl* ctl,
                                                           const __grid_constant__ ClusterArgsT<T> a) {
    const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int rank = (int)cl.block_rank();
    // the packed block and the steps do not depend on earlier kernels
    {
        const unsigned char* src = a.plan.blob + (size_t)rank * a.plan.blobBytes;
        for (uint32_t i = threadIdx.x * 16; i < a.plan.blobBytes; i += blockDim.x * 16) copy16(i, src + i);
    }
    const uint32_t stepsAt = a.plan.blobBytes;
    for (int s = threadIdx.x; s < a.nSteps; s += blockDim.x)
        at<ClusterStep>(stepsAt + (uint32_t)(s * sizeof(ClusterStep))) = a.steps[s];
    copyWait();
    __syncthreads();
    if (threadIdx.x < 2 * a.plan.count) {  // the zero cells
        const View<T> L = viewOf<T>(threadIdx.x >> 1);
        if (L.l.rows > 0) at<T>(L.iterate(threadIdx.x & 1) + (uint32_t)(L.l.cells - 1) * (uint32_t)sizeof(T)) = T(-0.0);
    }
    pdlEnter();
    if (ctl->done || ctl->ppSkip) return;  // the same on every CTA: none of them reaches a cluster barrier
#pragma unroll
    for (int i = 0; i < kMaxClusterLevels; i++) {
        if (i >= a.plan.count) break;
        const View<T> L = viewOf<T>(i);
        for (int n = threadIdx.x; n < L.l.live; n += blockDim.x) {
            const uint32_t o = (uint32_t)n * (uint32_t)sizeof(T);
            const int cell = n < L.l.rows ? L.l.row0 + n : at<int>(L.l.halo + 4 * (n - L.l.rows));
            copyElem(L.AC + o, a.AC[i] + cell);
            if (i == 0) {
                copyElem(L.b + o, a.b + cell);
                copyElem(L.x0 + o, a.x[0][0] + cell);
            }
        }
        // this CTA's slices are one run of the level's slots (whole slices: 16-byte aligned)
        const unsigned char* af = reinterpret_cast<const unsigned char*>(a.AF[i] + L.l.slot0);
        const uint32_t bytes = (uint32_t)L.l.slots * (uint32_t)sizeof(T);
        for (uint32_t q = threadIdx.x * 16; q < bytes; q += blockDim.x * 16) copy16(L.AF + q, af + q);
    }
    copyWait();
    if (a.syncFirst) cl.sync();
    else __syncthreads();

    // Every CTA follows the same steps and has rows in the steps of its levels.
    for (int s = 0; s < a.nSteps; s++) {
        const ClusterStep st = at<ClusterStep>(stepsAt + (uint32_t)(s * sizeof(ClusterStep)));
        const View<T> L = viewOf<T>(st.level);
        if (L.l.rows > 0) {
            const uint32_t x = L.iterate(st.from), y = L.iterate(st.to);
            T* out = static_cast<T*>(st.global);
            switch (st.op) {
                case kClSweep:
                case kClResidual:
                    rowsOf<T>(L, x, y, out, a.w, st.op == kClResidual);
                    break;
                case kClRestrict:  // from the finer level's buffer st.from into this level's st.to
                    restrictTo<T>(L, out, out ? 0 : viewOf<T>(st.level - 1).iterate(st.from), y, st.flag != 0, a.w);
                    break;
                case kClCorrect:  // with the coarser level's st.to
                    correct<T>(L, x, out, out ? 0 : viewOf<T>(st.level + 1).iterate(st.to), a.scale,
                               static_cast<T*>(st.global2));
                    break;
                case kClHalo:
                    fetchHalo<T>(L, x, out);
                    break;
                case kClCoarsest: {
                    const int part = ((L.l.rows + 31) / 32) * 32;
                    if ((int)threadIdx.x < part) coarsestRows<T>(L, x, L.iterate(st.from ^ 1), a.w, st.flag, part);
                    break;
                }
                case kClStore:
                    for (int n = threadIdx.x; n < L.l.rows; n += blockDim.x)
                        out[L.l.row0 + n] = at<T>(x + (uint32_t)n * (uint32_t)sizeof(T));
                    break;
            }
            if (!st.clusterWide) __syncthreads();
        }
        if (st.clusterWide) cl.sync();
    }
}

}  // namespace

// ---- host: the plan of a hierarchy and its packed topology ----
static bool buildClusterPlan(const std::vector<GridLevel>& hier, int first, const std::vector<std::vector<int32_t>>& sliceOff,
                      const std::vector<std::vector<int32_t>>& mStart, const std::vector<std::vector<int32_t>>& mList,
                      MgClusterPlan& plan, std::vector<unsigned char>& blob) {
    plan = MgClusterPlan();
    plan.first = first;
    plan.count = (int)hier.size() - first;
    if (first < 1 || plan.count < 1 || plan.count > kMaxClusterLevels) return false;
    for (int i = 0; i < plan.count; i++) {
        const int N = hier[(size_t)(first + i)].nCells;
        if (N < 1 || N > kClusterMaxCells) return false;
        plan.solo[i] = N <= kClusterSolo;
        if (i > 0 && plan.solo[i - 1] && !plan.solo[i]) return false;
        int W = 0;
        const std::vector<int32_t>& so = sliceOff[(size_t)(first + i)];
        for (size_t k = 0; k + 1 < so.size(); k++) {
            const int w = (so[k + 1] - so[k]) / 32;
            if (w < 8 || w % 8 != 0) return false;  // the kernel takes whole groups of eight, and one of every row
            W = std::max(W, w);
        }
        plan.W[i] = W;
        plan.N[i] = N;
    }
    const int last = plan.count - 1;
    // A row a thread on a coarsest level of up to 1,024 rows (a batch's merged one):
    // 513 rows, 20 iterations of 16 cases 3.26 ms FP64 and 2.80 mixed, with 512
    // threads in strides 4.42 and 3.91, with the single-CTA tail 4.21 and 3.50.
    // Smaller ones keep 512 threads: 1,024 measured slower there.
    if (plan.solo[last] && plan.W[last] <= 8 && plan.N[last] > kClusterThreads) plan.threads = kClusterThreadsLarge;
    plan.ctas = plan.solo[0] ? 1 : kClusterSize;  // CTA 0: the solo levels; the others: the chunks
    const int chunks = kClusterSize - 1;
    // a level on a CTA: its rows, its halo in ascending order, its slices
    struct Part {
        int n0 = 0, n1 = 0, s0 = 0, s1 = 0;
        std::vector<int32_t> halo;
    };
    std::vector<std::vector<Part>> parts((size_t)plan.count, std::vector<Part>((size_t)plan.ctas));
    for (int i = 0; i < plan.count; i++) {
        const GridLevel& g = hier[(size_t)(first + i)];
        const int N = g.nCells, R = plan.solo[i] ? N : 32 * ((N + 32 * chunks - 1) / (32 * chunks));
        std::vector<int> seen((size_t)N, -1);  // the last CTA that has the cell in its halo
        for (int r = 0; r < plan.ctas; r++) {
            if (plan.solo[i] != (r == 0)) continue;
            Part& p = parts[(size_t)i][(size_t)r];
            p.n0 = plan.solo[i] ? 0 : std::min((r - 1) * R, N);
            p.n1 = std::min(p.n0 + R, N);
            p.s0 = p.n0 / 32;
            p.s1 = p.n1 > p.n0 ? (p.n1 + 31) / 32 : p.s0;
            for (int k = g.faceStart[(size_t)p.n0]; k < g.faceStart[(size_t)p.n1]; k++) {
                const int m = g.faceNeighbor[(size_t)k];
                if (m < 0 || (m >= p.n0 && m < p.n1) || seen[(size_t)m] == r) continue;
                seen[(size_t)m] = r;
                p.halo.push_back(m);
            }
            std::sort(p.halo.begin(), p.halo.end());
        }
    }
    // The solo levels and the chunks' levels share the same range of offsets:
    // no CTA holds both. The largest CTA's sizes count for all.
    const size_t table = align16(sizeof(ClusterRows) * (size_t)plan.count);
    std::vector<std::vector<ClusterRows>> rows((size_t)plan.ctas, std::vector<ClusterRows>((size_t)plan.count));
    std::vector<size_t> blobEnd((size_t)plan.ctas, table);
    for (int r = 0; r < plan.ctas; r++)
        for (int i = 0; i < plan.count; i++) {
            const Part& p = parts[(size_t)i][(size_t)r];
            ClusterRows& l = rows[(size_t)r][(size_t)i];
            l.cells = 1;
            if (p.n1 == p.n0) continue;
            const std::vector<int32_t>& so = sliceOff[(size_t)(first + i)];
            l.rows = p.n1 - p.n0;
            l.row0 = p.n0;
            l.live = l.rows + (int)p.halo.size();
            l.cells = l.live + 1;
            l.wide = plan.W[i] > 8 ? 1 : 0;
            l.slot0 = so[(size_t)p.s0];
            l.slots = so[(size_t)p.s1] - l.slot0;
            if (l.cells > 65536 || l.slots >= (1 << 24)) return false;
            auto take = [&](size_t bytes) {
                const size_t o = blobEnd[(size_t)r];
                blobEnd[(size_t)r] += align16(bytes);
                return (uint32_t)o;
            };
            l.nb = take(sizeof(uint16_t) * (size_t)l.slots);
            if (l.wide) l.so = take(sizeof(uint32_t) * (size_t)(p.s1 - p.s0));
            l.halo = take(sizeof(int32_t) * p.halo.size());
            if (i + 1 < plan.count) l.c2c = take(sizeof(int32_t) * (size_t)l.live);
            if (i > 0) {
                const std::vector<int32_t>& ms = mStart[(size_t)(first + i)];
                size_t members = (size_t)(ms[(size_t)p.n1] - ms[(size_t)p.n0]);
                for (int h : p.halo) members += (size_t)(ms[(size_t)h + 1] - ms[(size_t)h]);
                l.ms = take(sizeof(int32_t) * (size_t)(l.live + 1));
                l.ml = take(sizeof(int32_t) * std::max<size_t>(members, 1));
            }
        }
    plan.blobBytes = (uint32_t)*std::max_element(blobEnd.begin(), blobEnd.end());
    const size_t values = align16(plan.blobBytes + sizeof(ClusterStep) * kMaxClusterSteps);
    plan.shared64 = plan.shared32 = values;
    for (int r = 0; r < plan.ctas; r++) {
        size_t v64 = values, v32 = values;
        for (int i = 0; i < plan.count; i++) {
            ClusterRows& l = rows[(size_t)r][(size_t)i];
            l.cells = (l.cells + 3) & ~3;  // every array 16-byte aligned in FP32 too: the last cell is the zero cell
            l.value64 = (uint32_t)v64;
            l.value32 = (uint32_t)v32;
            if (l.rows == 0) continue;
            v64 += sizeof(double) * (size_t)(4 * l.cells + l.slots);
            v32 += sizeof(float) * (size_t)(4 * l.cells + l.slots);
        }
        plan.shared64 = std::max(plan.shared64, v64);
        plan.shared32 = std::max(plan.shared32, v32);
    }
    if (plan.shared64 > kClusterMaxShared) return false;
    blob.assign((size_t)plan.blobBytes * (size_t)plan.ctas, 0);
    std::vector<uint16_t> at(kClusterMaxCells);  // a halo cell's place on the CTA at hand
    for (int r = 0; r < plan.ctas; r++) {
        unsigned char* base = blob.data() + (size_t)r * plan.blobBytes;
        for (int i = 0; i < plan.count; i++) {
            const GridLevel& g = hier[(size_t)(first + i)];
            const Part& p = parts[(size_t)i][(size_t)r];
            const ClusterRows& l = rows[(size_t)r][(size_t)i];
            std::memcpy(base + sizeof(ClusterRows) * (size_t)i, &l, sizeof l);
            if (l.rows == 0) continue;
            const std::vector<int32_t>& so = sliceOff[(size_t)(first + i)];
            for (size_t k = 0; k < p.halo.size(); k++) at[(size_t)p.halo[k]] = (uint16_t)(l.rows + (int)k);
            auto local = [&](int m) { return m >= p.n0 && m < p.n1 ? m - p.n0 : (int)at[(size_t)m]; };
            uint16_t* nb = reinterpret_cast<uint16_t*>(base + l.nb);
            for (int k = 0; k < l.slots; k++) nb[k] = (uint16_t)(l.cells - 1);
            for (int n = p.n0; n < p.n1; n++)
                for (int k = g.faceStart[(size_t)n], j = 0; k < g.faceStart[(size_t)n + 1]; k++, j++)
                    if (g.faceNeighbor[(size_t)k] >= 0)
                        nb[so[(size_t)(n >> 5)] - l.slot0 + 32 * j + (n & 31)] =
                            (uint16_t)local(g.faceNeighbor[(size_t)k]);
            if (l.wide)
                for (int k = p.s0; k < p.s1; k++)
                    reinterpret_cast<uint32_t*>(base + l.so)[k - p.s0] =
                        (uint32_t)(so[(size_t)k] - l.slot0) | (uint32_t)((so[(size_t)k + 1] - so[(size_t)k]) / 256) << 24;
            std::memcpy(base + l.halo, p.halo.data(), sizeof(int32_t) * p.halo.size());
            std::vector<int32_t> cells;  // rows, halo
            cells.reserve((size_t)l.live);
            for (int n = p.n0; n < p.n1; n++) cells.push_back(n);
            cells.insert(cells.end(), p.halo.begin(), p.halo.end());
            if (i + 1 < plan.count)
                for (size_t k = 0; k < cells.size(); k++)
                    reinterpret_cast<int32_t*>(base + l.c2c)[k] = g.cellToCoarse[(size_t)cells[k]];
            if (i > 0) {
                const std::vector<int32_t>& ms = mStart[(size_t)(first + i)];
                const std::vector<int32_t>& ml = mList[(size_t)(first + i)];
                int32_t* lms = reinterpret_cast<int32_t*>(base + l.ms);
                int32_t* lml = reinterpret_cast<int32_t*>(base + l.ml);
                int q = 0;
                for (size_t k = 0; k < cells.size(); k++) {
                    lms[k] = q;
                    for (int t = ms[(size_t)cells[k]]; t < ms[(size_t)cells[k] + 1]; t++) lml[q++] = ml[(size_t)t];
                }
                lms[cells.size()] = q;
            }
        }
    }
    return true;
}

MgClusterPlan findClusterPlan(const std::vector<GridLevel>& hier, int lastTerminal,
                              const std::vector<std::vector<int32_t>>& sliceOff,
                              const std::vector<std::vector<int32_t>>& mStart,
                              const std::vector<std::vector<int32_t>>& mList, std::vector<unsigned char>& blob) {
    MgClusterPlan plan;
    for (int t = std::max(1, lastTerminal + 1); t < (int)hier.size(); t++)
        if (buildClusterPlan(hier, t, sliceOff, mStart, mList, plan, blob)) return plan;
    return MgClusterPlan();
}

template <class T>
static cudaLaunchConfig_t clusterConfig(const MgClusterPlan& plan, cudaLaunchAttribute (&attr)[2]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan.ctas);
    cfg.blockDim = dim3(plan.threads);
    cfg.dynamicSmemBytes = sizeof(T) == 8 ? plan.shared64 : plan.shared32;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = plan.ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Whether the current device can hold the cluster of either precision (a GPC
// with kClusterSize SMs free); also raises the kernels' limits on it.
template <class T>
static auto* clusterKernel(const MgClusterPlan& plan) {
    return plan.threads == kClusterThreads ? k_mg_cluster<T, kClusterThreads> : k_mg_cluster<T, kClusterThreadsLarge>;
}
template <class T>
static bool clusterFits(const MgClusterPlan& plan) {
    auto* f = clusterKernel<T>(plan);
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = clusterConfig<T>(plan, attr);
    int n = 0;
    const bool ok =
        cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterMaxShared) ==
            cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, f, &cfg) == cudaSuccess && n >= 1;
    cudaGetLastError();
    return ok;
}
bool clusterRunnable(const MgClusterPlan& plan) { return clusterFits<double>(plan) && clusterFits<float>(plan); }

// The cycle as a list of steps (the recursion of MultigridSolver::vCycle,
// multigrid.cu:607-662) with the buffer each level's iterate is in. One loop in
// the kernel runs them, so each kind of step is in its code once. A chunked
// level's iterates go to L2 alternately to xNew and x, so a CTA still reading
// one exchange never sees the next; the last one of a level lands in x (the
// cycle's result on level `first`). False when the list is too long.
template <class T>
static bool clusterSteps(ClusterArgsT<T>& a) {
    const MgClusterPlan& p = a.plan;
    int cur[kMaxClusterLevels] = {};
    a.nSteps = 0;
    auto add = [&](ClusterOp op, int level, int from, int to, void* global, void* global2, int flag, bool wide) {
        if (a.nSteps < kMaxClusterSteps) {
            ClusterStep& s = a.steps[a.nSteps];
            s.op = op;
            s.level = (uint8_t)level;
            s.from = (uint8_t)from;
            s.to = (uint8_t)to;
            s.clusterWide = wide ? 1 : 0;
            s.flag = flag;
            s.global = global;
            s.global2 = global2;
        }
        a.nSteps++;
    };
    // `sweeps` sweeps; publish: the last one's values are read by other CTAs.
    // haloDue: the next step on this level reads neighbours.
    auto smooth = [&](int i, int sweeps, bool publish, bool haloDue) {
        const bool solo = p.solo[i];
        for (int k = 0; k < sweeps; k++) {
            const bool more = k + 1 < sweeps;
            T* out = !solo && (more || publish || haloDue) ? a.x[i][(sweeps - 1 - k) & 1] : nullptr;
            add(kClSweep, i, cur[i], cur[i] ^ 1, out, nullptr, 0, out && (more || haloDue || i > 0));
            cur[i] ^= 1;
            if (out && (more || haloDue)) add(kClHalo, i, cur[i], 0, out, nullptr, 0, false);
        }
    };
    const int last = p.count - 1;
    bool firstDone = a.firstDone != 0;
    // level `first` starts with a sweep: no CTA writes its iterate before all have read theirs
    a.syncFirst = !p.solo[0] && (last == 0 ? a.coarse : a.pre) > (firstDone ? 1 : 0) ? 1 : 0;
    for (int i = 0; i < last; i++) {
        smooth(i, a.pre - (firstDone ? 1 : 0), false, true);
        T* r = p.solo[i] ? nullptr : a.res[i];
        add(kClResidual, i, cur[i], cur[i] ^ 1, r, nullptr, 0, r != nullptr);
        firstDone = (i + 1 == last ? a.coarse : a.pre) >= 1;
        add(kClRestrict, i + 1, cur[i] ^ 1, 0, r, nullptr, firstDone ? 1 : 0, false);
    }
    const int sweeps = a.coarse - (firstDone ? 1 : 0);
    if (p.solo[last] && p.N[last] <= p.threads && p.W[last] <= 8 && sweeps > 0) {
        add(kClCoarsest, last, cur[last], 0, nullptr, nullptr, sweeps, false);
        cur[last] ^= sweeps & 1;
    } else {
        smooth(last, sweeps, true, false);
        if (!p.solo[last] && sweeps <= 0) add(kClStore, last, cur[last], 0, a.x[last][0], nullptr, 0, true);
    }
    for (int i = last - 1; i >= 0; i--) {
        // a solo level's iterate goes to the chunks above it through L2
        if (!p.solo[i] && p.solo[i + 1]) add(kClStore, i + 1, cur[i + 1], 0, a.x[i + 1][0], nullptr, 0, true);
        T* xc = p.solo[i] ? nullptr : a.x[i + 1][0];
        T* keep = a.post < 1 && !p.solo[i] ? a.x[i][0] : nullptr;
        add(kClCorrect, i, cur[i], cur[i + 1], xc, keep, 0, keep != nullptr);
        smooth(i, a.post, true, false);
    }
    if (p.solo[0]) add(kClStore, 0, cur[0], 0, a.x[0][0], nullptr, 0, false);
    return a.nSteps <= kMaxClusterSteps;
}

std::vector<ClusterStep> clusterStepList(const MgClusterPlan& plan, int pre, int post, int coarse) {
    ClusterArgsT<double> a;
    a.plan = plan;
    a.pre = pre;
    a.post = post;
    a.coarse = coarse;
    a.firstDone = (plan.count == 1 ? coarse : pre) >= 1 ? 1 : 0;  // the restriction into level `first` ran it
    double anywhere = 0.0;  // a step reads or writes L2 where it has an address
    for (int i = 0; i < kMaxClusterLevels; i++) a.x[i][0] = a.x[i][1] = a.res[i] = &anywhere;
    if (!clusterSteps(a)) return {};
    return std::vector<ClusterStep>(a.steps, a.steps + a.nSteps);
}

template <class T>
bool launchMGCluster(const Ctl* ctl, ClusterArgsT<T> a, cudaStream_t s) {
    if (a.plan.count < 1 || !clusterSteps(a)) return false;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = clusterConfig<T>(a.plan, attr);
    cfg.stream = s;
    cfg.numAttrs = tNextLaunchPlain ? 1 : 2;
    tNextLaunchPlain = false;
    return cudaLaunchKernelEx(&cfg, clusterKernel<T>(a.plan), ctl, a) == cudaSuccess;
}

template bool launchMGCluster<double>(const Ctl*, ClusterArgsT<double>, cudaStream_t);
template bool launchMGCluster<float>(const Ctl*, ClusterArgsT<float>, cudaStream_t);

}  // namespace axisim
