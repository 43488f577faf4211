// residual_static.cu -- the SIMPLE residuals (momentum u, v and continuity) of
// caller-owned device arrays, computed without allocating any memory.
//
// What bounds it: three rounds of dependent loads a cell (slots, faces, other
// cells) and, below some 200k cells, the call itself. A quad's slots come in
// three 16-byte loads where the arrays lie on 16-byte boundaries, each round's
// loads go together, and a block takes as many groups of 256 cells as make one
// wave, for one arrival. A call: 829 cells 40 -> 29 us, 218,624 cells 45 -> 34,
// 874,496 cells 78 -> 63 (the kernel 50 -> 43, cold caches).
//
// Same arithmetic as the solver's residual kernel (residualAll +
// continuityResidual, residuals.cu:5-100): per cell |b - A x| for u and v,
// A_C x as the DIAGONAL scale, and the signed mass imbalance; then one block
// partial per 256 cells and a final pass in block order, so results do not
// depend on scheduling.
//
// Why: some callers cannot allocate device memory at the point where they want
// residuals -- a host that has handed the whole GPU to a caching allocator or
// runs under a hard memory cap, or a monitoring hook inside a time-critical
// loop where cudaMalloc/cudaFree would stall (cudaFree synchronises the whole
// device). This entry point therefore keeps its reduction scratch in a
// fixed-size file-scope device array instead of the solver's arena.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>

#include <cuda_runtime.h>

#include "axisim_b200.h"

namespace {

constexpr int kThreads = 256;
constexpr int kQ = 5;  // stat_u, scale_u, stat_v, scale_v, continuity
constexpr int kMaxBlocks = AXISIM_STATIC_MAX_CELLS / kThreads;
constexpr int kPartialDoubles = kMaxBlocks * kQ;
constexpr int kCallSlots = 256;         // calls take them in turn
constexpr int kWordDoubles = kCallSlots + 2;  // a slot's two counters (8 bytes) each, after the partials
constexpr int kMaxDevices = 64;
constexpr int kResident = 148 * 4;  // blocks that run at once (64 registers a thread)
constexpr int kMaxGroups = 28;      // groups a block: kMaxBlocks over kResident

static_assert(AXISIM_STATIC_MAX_CELLS % kThreads == 0, "limit must be whole blocks");
static_assert(kMaxGroups * kResident >= kMaxBlocks, "every group has a block");

// Partials of up to kMaxBlocks blocks, then two counters per call slot: the
// arrival ticket and the number of cells that met an out-of-range index. The
// last block of a call returns its slot's counters to zero, and only that
// call's blocks touch them, so calls that overlap in time, whose sums may be
// wrong, leave nothing behind. The last two words hold the count of the call
// that has no host word. 640 KiB + 2 KiB per device.
static __device__ __align__(256) double g_residualScratch[kPartialDoubles + kWordDoubles];

__device__ __forceinline__ double combine(double a, double b, int isMax) { return isMax ? fmax(a, b) : a + b; }

__global__ void __launch_bounds__(kThreads, 4)
k_residual_static(int N, int F, int S, const int32_t* __restrict__ cellFaceStart,
                  const int32_t* __restrict__ cellFaceIDs, const int32_t* __restrict__ faceOwner,
                  const int32_t* __restrict__ faceNeighbor, const double* __restrict__ AF,
                  const double* __restrict__ ACu, const double* __restrict__ ACv, const double* __restrict__ bu,
                  const double* __restrict__ bv, const double* __restrict__ u, const double* __restrict__ v,
                  const double* __restrict__ mDot, int normU, int normV, double* __restrict__ resU,
                  double* __restrict__ resV, double* __restrict__ resC, double* __restrict__ sums,
                  double* scratch, unsigned int* words, int wide, int groups, volatile unsigned int* status) {
    const int isMax[kQ] = {normU == 2, 0, normV == 2, 0, 0};
    // groups of 256 cells, several a block: one arrival for all of them
    __shared__ double sh[kMaxGroups][kThreads / 32][kQ];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nGroups = (N + kThreads - 1) / kThreads;
    const int first = blockIdx.x * groups, mine = min(groups, nGroups - first);
    double acc[kQ];
    for (int gi = 0; gi < mine; gi++) {
#pragma unroll
        for (int q = 0; q < kQ; q++) acc[q] = isMax[q] ? -INFINITY : 0.0;
        const int n = (first + gi) * kThreads + (int)threadIdx.x;
        if (n < N) {
            const int k0 = cellFaceStart[n], k1 = cellFaceStart[n + 1];
            const double rhsU = bu[n], rhsV = bv[n];
            double Axu = ACu[n] * u[n];
            double Axv = ACv[n] * v[n];
            const double su = Axu, sv = Axv;
            double imb = 0.0;
            int bad = 0;
            if (k0 < 0 || k1 < k0 || k1 > S) {
                bad = 1;
            } else {
                // KS slots: the faces' cells and fluxes, then the other cells' values,
                // each round of loads together (an index out of range loads a safe
                // element and is left out of the sums), and the sums in slot order
                auto slots = [&](auto count, const int* f, const double* a) {
                    constexpr int KS = decltype(count)::value;
                    int own[KS], nbr[KS];
                    bool ok[KS];
                    double md[KS], uc[KS], vc[KS];
#pragma unroll
                    for (int j = 0; j < KS; j++) {
                        ok[j] = f[j] >= 0 && f[j] < F;
                        const int g = ok[j] ? f[j] : 0;
                        own[j] = faceOwner[g];
                        nbr[j] = faceNeighbor[g];
                        md[j] = mDot[g];
                    }
#pragma unroll
                    for (int j = 0; j < KS; j++) {
                        ok[j] = ok[j] && own[j] >= 0 && own[j] < N && nbr[j] >= -1 && nbr[j] < N;
                        if (!ok[j]) bad = 1;
                        const int c = ok[j] && nbr[j] >= 0 ? (own[j] == n ? nbr[j] : own[j]) : n;
                        uc[j] = u[c];
                        vc[j] = v[c];
                    }
#pragma unroll
                    for (int j = 0; j < KS; j++) {
                        if (!ok[j]) continue;
                        if (nbr[j] >= 0) {
                            Axu += a[j] * uc[j];
                            Axv += a[j] * vc[j];
                        }
                        if (own[j] == n) imb += md[j];
                        else if (nbr[j] == n) imb -= md[j];
                    }
                };
                if (wide && k1 - k0 == 4 && (k0 & 3) == 0) {  // a quad: its slots in three 16-byte loads
                    const int4 f4 = *reinterpret_cast<const int4*>(cellFaceIDs + k0);
                    const double2 a0 = *reinterpret_cast<const double2*>(AF + k0);
                    const double2 a1 = *reinterpret_cast<const double2*>(AF + k0 + 2);
                    const int f[4] = {f4.x, f4.y, f4.z, f4.w};
                    const double a[4] = {a0.x, a0.y, a1.x, a1.y};
                    slots(std::integral_constant<int, 4>(), f, a);
                } else {
                    for (int k = k0; k < k1; k++) {
                        const int f[1] = {cellFaceIDs[k]};
                        const double a[1] = {AF[k]};
                        slots(std::integral_constant<int, 1>(), f, a);
                    }
                }
            }
            if (bad) atomicAdd(&words[1], 1u);
            const double ru = fabs(rhsU - Axu);
            const double rv = fabs(rhsV - Axv);
            resU[n] = ru;
            resV[n] = rv;
            resC[n] = imb;
            acc[0] = normU == 1 ? ru * ru : ru;
            acc[1] = fabs(su);
            acc[2] = normV == 1 ? rv * rv : rv;
            acc[3] = fabs(sv);
            acc[4] = fabs(imb);
        }
#pragma unroll
        for (int q = 0; q < kQ; q++) {
            double x = acc[q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x = combine(x, __shfl_down_sync(0xffffffffu, x, o), isMax[q]);
            if (lane == 0) sh[gi][warp][q] = x;
        }
    }
    __syncthreads();
    // each group's partial, its warps in order
    for (int i = threadIdx.x; i < mine * kQ; i += kThreads) {
        const int gi = i / kQ, q = i % kQ;
        const int most = (q == 0 && normU == 2) || (q == 2 && normV == 2);
        double x = sh[gi][0][q];
        for (int w = 1; w < kThreads / 32; w++) x = combine(x, sh[gi][w][q], most);
        scratch[(size_t)(first + gi) * kQ + q] = x;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&words[0], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    // the last block to arrive adds the partials in block order
    __threadfence();
    __shared__ double tr[kThreads][kQ];
#pragma unroll
    for (int q = 0; q < kQ; q++) acc[q] = isMax[q] ? -INFINITY : 0.0;
    constexpr int kAhead = 16;  // partials loaded ahead of their sums, one statistic at a time: few registers
#pragma unroll
    for (int q = 0; q < kQ; q++) {
        for (int i = threadIdx.x; i < nGroups; i += kAhead * kThreads) {
            double x[kAhead];
#pragma unroll
            for (int w = 0; w < kAhead; w++)
                x[w] = __ldcg(scratch + (size_t)min(i + w * kThreads, nGroups - 1) * kQ + q);
#pragma unroll
            for (int w = 0; w < kAhead; w++)
                if (i + w * kThreads < nGroups) acc[q] = combine(acc[q], x[w], isMax[q]);
        }
        tr[threadIdx.x][q] = acc[q];
    }
    __syncthreads();
    for (int st = kThreads / 2; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st)
#pragma unroll
            for (int q = 0; q < kQ; q++) tr[threadIdx.x][q] = combine(tr[threadIdx.x][q], tr[threadIdx.x + st][q], isMax[q]);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < kQ; q++) sums[q] = tr[0][q];
        // the counters return to zero for the slot's next call
        *status = words[1];
        words[1] = 0u;
        words[0] = 0u;
    }
}

// Per-device address of the scratch array, looked up once per device, and the
// calls' turns at its slots.
std::mutex g_setupMu;
double* g_scratchPtr[kMaxDevices] = {};
unsigned int g_calls[kMaxDevices] = {};
// A page-locked host word per call slot and device for a call's bad-index count,
// mapped into the device (host memory, taken on the first call): the kernel's own
// store saves the copy back, some 10 of 39 us of a small call. Null where it
// could not be had: the count is then copied from the scratch words.
volatile unsigned int* g_status = nullptr;
bool g_statusTried = false;
constexpr unsigned int kUnwritten = 0xFFFFFFFFu;  // no count: at most one a cell

void setError(char* err, size_t errLen, const char* msg) {
    if (!err || errLen == 0) return;
    std::snprintf(err, errLen, "%s", msg);
}

// Device memory of device `dev`, or managed memory (reachable from any device).
// A pointer into another GPU's memory is rejected: without peer access the
// kernel would fault on it.
bool isDevicePointerOn(const void* p, int dev) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type == cudaMemoryTypeManaged) return true;
    return a.type == cudaMemoryTypeDevice && a.device == dev;
}

}  // namespace

extern "C" int axisim_residual_static(int32_t nCells, int32_t nFaces, int32_t nSlots, const int32_t* cellFaceStart,
                                      const int32_t* cellFaceIDs, const int32_t* faceOwner,
                                      const int32_t* faceNeighbor, const double* AF, const double* ACu,
                                      const double* ACv, const double* bu, const double* bv, const double* u,
                                      const double* v, const double* mDot, int32_t normU, int32_t normV,
                                      double* resU, double* resV, double* resC, double* sums, void* stream,
                                      char* err, size_t errLen) {
    char msg[160];
    if (nCells <= 0 || nFaces <= 0 || nSlots <= 0) {
        setError(err, errLen, "nCells, nFaces and nSlots must be positive");
        return AXISIM_E_ARG;
    }
    if (nCells > AXISIM_STATIC_MAX_CELLS) {
        std::snprintf(msg, sizeof msg, "nCells %d exceeds the static scratch limit of %d cells", nCells,
                      AXISIM_STATIC_MAX_CELLS);
        setError(err, errLen, msg);
        return AXISIM_E_ARG;
    }
    if (normU < 0 || normU > 2 || normV < 0 || normV > 2) {
        setError(err, errLen, "norm type must be 0 (L1), 1 (L2) or 2 (LINF)");
        return AXISIM_E_ARG;
    }
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        setError(err, errLen, "no current CUDA device");
        return AXISIM_E_CUDA;
    }
    const void* ptrs[] = {cellFaceStart, cellFaceIDs, faceOwner, faceNeighbor, AF, ACu, ACv, bu, bv, u, v, mDot,
                          resU, resV, resC, sums};
    for (const void* p : ptrs)
        if (!p || !isDevicePointerOn(p, dev)) {
            setError(err, errLen, "every array must be a device pointer on the current device");
            return AXISIM_E_ARG;
        }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // every call ends with a blocking read-back of the bad-index count, which
    // a capturing stream cannot do: refuse before touching the stream
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(s, &cap);
    if (e != cudaSuccess) {
        std::snprintf(msg, sizeof msg, "cudaStreamIsCapturing: %s", cudaGetErrorString(e));
        setError(err, errLen, msg);
        return AXISIM_E_CUDA;
    }
    if (cap != cudaStreamCaptureStatusNone) {
        setError(err, errLen, "cannot be called while the stream is being captured (it reads its status back)");
        return AXISIM_E_ARG;
    }
    double* scratch = nullptr;
    volatile unsigned int* hostWord = nullptr;
    unsigned int slot = 0;
    {
        std::lock_guard<std::mutex> lk(g_setupMu);
        if (!g_scratchPtr[dev]) {
            e = cudaGetSymbolAddress(reinterpret_cast<void**>(&g_scratchPtr[dev]), g_residualScratch);
            if (e != cudaSuccess) {
                g_scratchPtr[dev] = nullptr;
                std::snprintf(msg, sizeof msg, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
                setError(err, errLen, msg);
                return AXISIM_E_CUDA;
            }
        }
        scratch = g_scratchPtr[dev];
        if (!g_statusTried) {
            g_statusTried = true;
            void* p = nullptr;
            if (cudaHostAlloc(&p, sizeof(unsigned int) * kCallSlots * kMaxDevices,
                              cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess)
                g_status = static_cast<volatile unsigned int*>(p);
            cudaGetLastError();
        }
        slot = g_calls[dev]++ % kCallSlots;
        if (g_status) hostWord = g_status + (size_t)dev * kCallSlots + slot;
    }
    unsigned int* words = reinterpret_cast<unsigned int*>(scratch + kPartialDoubles) + 2 * slot;
    unsigned int* devWord = reinterpret_cast<unsigned int*>(scratch + kPartialDoubles) + 2 * kCallSlots;
    if (hostWord) *hostWord = kUnwritten;
    {
        const int nGroups = (nCells + kThreads - 1) / kThreads;
        const int groups = std::min(kMaxGroups, (nGroups + kResident - 1) / kResident);
        const int blocks = (nGroups + groups - 1) / groups;
        // 16-byte slot loads need the arrays on 16-byte boundaries
        const int wide = ((reinterpret_cast<uintptr_t>(cellFaceIDs) | reinterpret_cast<uintptr_t>(AF)) & 15) == 0;
        k_residual_static<<<blocks, kThreads, 0, s>>>(nCells, nFaces, nSlots, cellFaceStart, cellFaceIDs, faceOwner,
                                                      faceNeighbor, AF, ACu, ACv, bu, bv, u, v, mDot, normU, normV,
                                                      resU, resV, resC, sums, scratch, words, wide, groups,
                                                      hostWord ? hostWord : devWord);
        e = cudaGetLastError();
    }
    unsigned int bad = 0;
    if (e == cudaSuccess && !hostWord) e = cudaMemcpyAsync(&bad, devWord, sizeof bad, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && hostWord) bad = *hostWord;
    if (e != cudaSuccess) {
        std::snprintf(msg, sizeof msg, "CUDA: %s", cudaGetErrorString(e));
        setError(err, errLen, msg);
        return AXISIM_E_CUDA;
    }
    if (bad == kUnwritten) {  // more calls at once than slots
        setError(err, errLen, "too many calls overlapped: the results were not written");
        return AXISIM_E_CUDA;
    }
    if (bad) {
        std::snprintf(msg, sizeof msg, "%u cells met an out-of-range slot, face or cell index (skipped)", bad);
        setError(err, errLen, msg);
        return AXISIM_E_MESH;
    }
    setError(err, errLen, "");
    return AXISIM_OK;
}
