// learned.cu -- forward, backward and Adam kernels of the learned p'
// preconditioner (network described in learned.hpp), its host driver, and the
// harvest of training samples from the captured SIMPLE iteration.
//
// Every layer is the same fused operation over the rows of one level:
//   Y = act(Z W + b [+ add]),  Z = [T_1(X_1), T_2(X_2)]
// where each input transform T is the identity, the mean over the cell's
// neighbours, the mean over an agglomerate's members (pool) or the copy from
// the cell's agglomerate (unpool). The backward pass of a layer is
//   G = dY * act'(Y);  dW = Z^T G;  db = sum G;  dZ = G W^T
// followed by the adjoint of each transform, which accumulates dZ into the
// gradient of its source tensor: identity, neighbour-mean transposed (a
// gather over the same symmetric graph), pool transposed (copy back to the
// members), unpool transposed (sum over the members). All reductions over
// rows (dW, db, the loss) run as per-block partials summed in a fixed order,
// so a training step is deterministic.
//
// The dense products are small (K <= 256 inputs, <= 128 outputs per row): at
// the finest level, where nearly all rows are, a layer moves ~130 bytes and
// does ~1 kFLOP per row, and the coarse levels have a few dozen to a few
// thousand rows. So the finest levels are bound by memory traffic and the
// coarse ones by the latency of one tile; the products run as mma.sync on
// operands that go from global memory straight into fragments
// (k_layer_mma, k_layer_dz_mma; predictions and input gradients with BF16
// weights) or through shared-memory tiles (k_layer_tile, k_layer_dz_tile; the
// solver's preconditioner, the training forward pass, and FP32 weights).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <random>
#include <stdexcept>
#include <string>

#include <cuda_bf16.h>
#include <type_traits>

#include "host_prep.hpp"
#include "learned.hpp"

namespace axisim {

namespace {

constexpr int kThreads = 256;
inline int blocksFor(size_t n, int t = kThreads) { return (int)((n + t - 1) / t); }

#define NCK(x)                                                                                                \
    do {                                                                                                      \
        cudaError_t e_ = (x);                                                                                 \
        if (e_ != cudaSuccess) throw std::runtime_error(std::string("CUDA: ") + cudaGetErrorString(e_));      \
    } while (0)

using bfloat = __nv_bfloat16;

// FP32 -> TF32 (round to nearest, ties away), as the tensor cores read it
__device__ __forceinline__ uint32_t toTf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// d += a b for one m16n8k8 block (A row-major 16 x 8, B column-major 8 x 8, FP32 accumulators)
__device__ __forceinline__ void mmaTf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float ldv(const float* p, size_t i) { return p[i]; }
__device__ __forceinline__ float ldv(const bfloat* p, size_t i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void stv(float* p, size_t i, float v) { p[i] = v; }
__device__ __forceinline__ void stv(bfloat* p, size_t i, float v) { p[i] = __float2bfloat16_rn(v); }

// Inference kernels run inside the captured p' solve: ungated they return while
// the solve is done or skipped (ppSkip != 0); gated they run only while
// ppSkip == 2, the state in which the solve uses the network's step.
__device__ __forceinline__ bool idle(const Ctl* ctl, int gated) {
    if (!ctl) return false;
    return ctl->done || (gated ? ctl->ppSkip != 2 : ctl->ppSkip != 0);
}

// Sums NQ doubles over the grid: block partials, then the last block to arrive
// adds them in block order. Returns true in thread 0 of that block.
template <int NQ>
__device__ bool gridSumD(const double (&v)[NQ], double* partial, unsigned int* counter, double* out) {
    __shared__ double sh[kThreads / 32][NQ];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = 0; q < NQ; q++) {
        double x = v[q];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sh[warp][q] = x;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q < NQ; q++) {
            double x = 0.0;
            for (int w = 0; w < kThreads / 32; w++) x += sh[w][q];
            partial[(size_t)blockIdx.x * NQ + q] = x;
        }
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    __shared__ double tr[kThreads][NQ];
    double acc[NQ];
    for (int q = 0; q < NQ; q++) acc[q] = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kThreads)
        for (int q = 0; q < NQ; q++) acc[q] += ((volatile double*)partial)[(size_t)i * NQ + q];
    for (int q = 0; q < NQ; q++) tr[threadIdx.x][q] = acc[q];
    __syncthreads();
    for (int st = kThreads / 2; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st)
            for (int q = 0; q < NQ; q++) tr[threadIdx.x][q] += tr[threadIdx.x + st][q];
        __syncthreads();
    }
    if (threadIdx.x != 0) return false;
    for (int q = 0; q < NQ; q++) out[q] = tr[0][q];
    *counter = 0u;
    return true;
}

// ---------------- features ----------------

// scal[0] = mean (r / AC)^2 (sigma^2)
template <class TR>
__global__ void __launch_bounds__(kThreads) k_sigma(const Ctl* ctl, int gated, int N, const TR* r, const TR* AC, double* partial,
                                                    unsigned int* counter, double* scal) {
    pdlEnter();
    if (idle(ctl, gated)) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[1] = {0.0};
    if (n < N) {
        const double ac = (double)AC[n];
        const double q = ac != 0.0 ? (double)r[n] / ac : 0.0;
        acc[0] = q * q;
    }
    if (gridSumD<1>(acc, partial, counter, scal)) scal[0] /= (double)N;
}

// feat[n] = [r / (AC sigma), deficit]; deficit from the ELL matrix (AF != null)
// or given.
template <class TA, class TR>
__global__ void __launch_bounds__(kThreads) k_features(const Ctl* ctl, int gated, int N, const TR* r, const TR* AC,
                                                       const double* AF, const int32_t* nb, int W,
                                                       const float* deficit, const double* scal, TA* feat) {
    pdlEnter();
    if (idle(ctl, gated)) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    const double sigma = sqrt(scal[0]);
    const double ac = (double)AC[n];
    const double x = (ac != 0.0 && sigma > 0.0) ? (double)r[n] / (ac * sigma) : 0.0;
    float d;
    if (AF) {
        double s = 0.0;
        for (int j = 0; j < W; j++) {
            const size_t sl = (size_t)j * N + n;
            if (nb[sl] >= 0) s += fabs(AF[sl]);
        }
        d = ac != 0.0 ? (float)(1.0 - s / ac) : 0.f;
    } else {
        d = deficit[n];
    }
    stv(feat, (size_t)n * 2, (float)x);
    stv(feat, (size_t)n * 2 + 1, d);
}

// ---------------- layer forward ----------------

template <class TA>
__device__ __forceinline__ void gatherInput(const NetIn& I, int n, float* z) {
    const TA* x = (const TA*)I.x;
    const int C = I.C;
    if (I.xf == NX_ID) {
        for (int c = 0; c < C; c++) z[c] = ldv(x, (size_t)n * C + c);
    } else if (I.xf == NX_UNPOOL) {
        const int k = I.map[n];
        for (int c = 0; c < C; c++) z[c] = ldv(x, (size_t)k * C + c);
    } else {  // NBMEAN or POOL: mean over a CSR list
        for (int c = 0; c < C; c++) z[c] = 0.f;
        for (int q = I.s[n]; q < I.s[n + 1]; q++) {
            const int k = I.list[q];
            for (int c = 0; c < C; c++) z[c] += ldv(x, (size_t)k * C + c);
        }
        const float w = I.inv[n];
        for (int c = 0; c < C; c++) z[c] *= w;
    }
}

// One row per thread; the row's concatenated input Z lives in shared memory
// (stride K + 1: conflict-free across the warp), weights are broadcast loads.
template <class TA, class TW, int OCH>
__global__ void k_layer_fwd(const Ctl* ctl, int gated, NetLayer L, const TW* __restrict__ P) {
    pdlEnter();
    if (idle(ctl, gated)) return;
    extern __shared__ float zsm[];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= L.N) return;
    const int K = L.K, Cout = L.Cout;
    float* z = zsm + (size_t)threadIdx.x * (K + 1);
    int off = 0;
    for (int i = 0; i < L.nIn; i++) {
        gatherInput<TA>(L.in[i], n, z + off);
        off += L.in[i].C;
    }
    if (L.Z) {
        TA* Z = (TA*)L.Z;
        for (int k = 0; k < K; k++) stv(Z, (size_t)n * K + k, z[k]);
    }
    const TW* W = P + L.wOff;
    const TW* B = W + (size_t)K * Cout;
    const TA* add = (const TA*)L.add;
    TA* Y = (TA*)L.Y;
    for (int o0 = 0; o0 < Cout; o0 += OCH) {
        float acc[OCH];
#pragma unroll
        for (int j = 0; j < OCH; j++) acc[j] = (o0 + j < Cout) ? ldv(B, o0 + j) : 0.f;
        for (int k = 0; k < K; k++) {
            const float zk = z[k];
            const TW* wr = W + (size_t)k * Cout + o0;
#pragma unroll
            for (int j = 0; j < OCH; j++)
                if (o0 + j < Cout) acc[j] = fmaf(zk, ldv(wr, j), acc[j]);
        }
#pragma unroll
        for (int j = 0; j < OCH; j++) {
            if (o0 + j >= Cout) break;
            float v = acc[j];
            if (add) v += ldv(add, (size_t)n * Cout + o0 + j);
            if (L.relu) v = fmaxf(v, 0.f);
            stv(Y, (size_t)n * Cout + o0 + j, v);
        }
    }
}

// Tiled layers: a block computes a 64-row tile of Y = act(Z W + b [+ add])
// for all Cout = 16 CPT outputs. The tile's Z (64 x K, FP32) is gathered into
// shared memory (lanes along the channels, so source rows load coalesced),
// W is staged in 32-row chunks, and each of the 256 threads accumulates a
// 4-row x CPT-column register block (columns tx + 16 j: conflict-free
// weight reads, broadcast Z reads).
constexpr int kTileRows = 64;
constexpr int kChunk = 32;

// Every channel count here divides 256, so thread t handles channel t % C of
// rows t / C, t / C + 256 / C, ... of each input (no per-element division).
// For a mean over a CSR list, the tile's list bounds are first staged in
// shared memory (idx: TR + 1 ints) so the C threads of a row do not each
// re-read them.
template <class TA, int TR>
__device__ __forceinline__ void gatherTile(const NetLayer& L, int row0, float* zs, int ldz, int* idx) {
    int off = 0;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        if (i >= L.nIn) break;
        const NetIn& I = L.in[i];
        const int C = I.C;
        const int c = threadIdx.x % C, rstep = blockDim.x / C;
        const TA* x = (const TA*)I.x;
        const bool mean = I.xf == NX_NBMEAN || I.xf == NX_POOL;
        if (mean) {
            __syncthreads();
            for (int r = threadIdx.x; r <= TR; r += blockDim.x) idx[r] = I.s[min(row0 + r, L.N)];
            __syncthreads();
        }
        for (int r = threadIdx.x / C; r < TR; r += rstep) {
            const int n = row0 + r;
            float v = 0.f;
            if (n < L.N) {
                if (I.xf == NX_ID) v = ldv(x, (size_t)n * C + c);
                else if (I.xf == NX_UNPOOL) v = ldv(x, (size_t)I.map[n] * C + c);
                else {
                    // four independent list loads, then four independent row
                    // loads: coarse levels have long lists and few rows, so
                    // the loop is bound by load latency, not bandwidth
                    int q = idx[r];
                    const int q1 = idx[r + 1];
                    for (; q + 4 <= q1; q += 4) {
                        const int k0 = __ldg(I.list + q), k1 = __ldg(I.list + q + 1);
                        const int k2 = __ldg(I.list + q + 2), k3 = __ldg(I.list + q + 3);
                        const float a0 = ldv(x, (size_t)k0 * C + c), a1 = ldv(x, (size_t)k1 * C + c);
                        const float a2 = ldv(x, (size_t)k2 * C + c), a3 = ldv(x, (size_t)k3 * C + c);
                        v += (a0 + a1) + (a2 + a3);
                    }
                    for (; q < q1; q++) v += ldv(x, (size_t)__ldg(I.list + q) * C + c);
                    v *= __ldg(I.inv + n);
                }
            }
            zs[r * ldz + off + c] = v;
        }
        off += C;
    }
}

template <class TA, class TW, int CPT, int RPT>
__global__ void __launch_bounds__(256) k_layer_tile(const Ctl* ctl, int gated, NetLayer L, const TW* __restrict__ P) {
    pdlEnter();
    if (idle(ctl, gated)) return;
    constexpr int COUT = 16 * CPT;
    constexpr int TR = 16 * RPT;  // rows per tile
    extern __shared__ float sm[];
    const int K = L.K;
    const int ldz = K + 1;
    float* zs = sm;                   // [TR][K + 1]
    float* ws = sm + TR * ldz;        // [32][COUT]
    const int row0 = blockIdx.x * TR;
    gatherTile<TA, TR>(L, row0, zs, ldz, (int*)(ws + kChunk * COUT));
    __syncthreads();
    if (L.Z) {
        TA* Z = (TA*)L.Z;
        const int k = threadIdx.x % K, rstep = blockDim.x / K;
        for (int r = threadIdx.x / K; r < TR; r += rstep)
            if (row0 + r < L.N) stv(Z, (size_t)(row0 + r) * K + k, zs[r * ldz + k]);
    }
    // Tensor cores: the TR x COUT tile is (TR/16) x (COUT/8) mma.sync
    // m16n8k8 TF32 blocks with FP32 accumulators, dealt round-robin to the 8
    // warps. The FP32 activations are split into a TF32 high part and the
    // TF32 rounding of the remainder, and both are multiplied: close to FP32
    // accuracy. BF16 weights are exact in TF32; FP32 weights (the gradient
    // check's mode) are split the same way, adding a third product.
    constexpr int NRB = RPT, NCB = 2 * CPT;
    constexpr int TPW = (NRB * NCB + 7) / 8;  // blocks per warp
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t4 = lane & 3;
    const TW* W = P + L.wOff;
    float acc[TPW][4];
#pragma unroll
    for (int q = 0; q < TPW; q++) {
        const int blk = warp + 8 * q;
        const int cb = blk % NCB;
        const float b0 = blk < NRB * NCB ? ldv(W + (size_t)K * COUT, cb * 8 + 2 * t4) : 0.f;
        const float b1 = blk < NRB * NCB ? ldv(W + (size_t)K * COUT, cb * 8 + 2 * t4 + 1) : 0.f;
        acc[q][0] = b0;
        acc[q][1] = b1;
        acc[q][2] = b0;
        acc[q][3] = b1;
    }
    for (int k0 = 0; k0 < K; k0 += kChunk) {
        const int kn = min(kChunk, K - k0);
        // the chunk's weights: all of a thread's loads issued before any
        // shared-memory store, so they are in flight together
        constexpr int PER = kChunk * COUT / 256;
        float wv[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int idx = threadIdx.x + 256 * u;
            wv[u] = idx < kn * COUT ? ldv(W, (size_t)k0 * COUT + idx) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < PER; u++) ws[threadIdx.x + 256 * u] = wv[u];
        __syncthreads();
        for (int kk = 0; kk < kn; kk += 8) {
            // columns past the chunk (K below 8) read as zero, never the next row
            const bool c0ok = kk + t4 < kn, c1ok = kk + t4 + 4 < kn;
#pragma unroll
            for (int q = 0; q < TPW; q++) {
                const int blk = warp + 8 * q;
                if (blk >= NRB * NCB) break;
                const int rb = blk / NCB, cb = blk % NCB;
                const float* zr0 = zs + (rb * 16 + g) * ldz + k0 + kk;
                const float* zr1 = zr0 + 8 * ldz;
                const float a[4] = {c0ok ? zr0[t4] : 0.f, c0ok ? zr1[t4] : 0.f, c1ok ? zr0[t4 + 4] : 0.f,
                                    c1ok ? zr1[t4 + 4] : 0.f};
                const float bw[2] = {ws[(kk + t4) * COUT + cb * 8 + g], ws[(kk + t4 + 4) * COUT + cb * 8 + g]};
                uint32_t ahi[4], alo[4], bhi[2];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    ahi[e] = toTf32(a[e]);
                    alo[e] = toTf32(a[e] - __uint_as_float(ahi[e]));
                }
#pragma unroll
                for (int e = 0; e < 2; e++) bhi[e] = toTf32(bw[e]);
                if constexpr (std::is_same<TW, float>::value) {
                    uint32_t blo[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) blo[e] = toTf32(bw[e] - __uint_as_float(bhi[e]));
                    mmaTf32(acc[q], ahi, blo);
                }
                mmaTf32(acc[q], alo, bhi);
                mmaTf32(acc[q], ahi, bhi);
            }
        }
    }
    const TA* add = (const TA*)L.add;
    TA* Y = (TA*)L.Y;
#pragma unroll
    for (int q = 0; q < TPW; q++) {
        const int blk = warp + 8 * q;
        if (blk >= NRB * NCB) break;
        const int rb = blk / NCB, cb = blk % NCB;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int n = row0 + rb * 16 + g + (e >= 2 ? 8 : 0);
            const int o = cb * 8 + 2 * t4 + (e & 1);
            if (n >= L.N) continue;
            float v = acc[q][e];
            if (add) v += ldv(add, (size_t)n * COUT + o);
            if (L.relu) v = fmaxf(v, 0.f);
            stv(Y, (size_t)n * COUT + o, v);
        }
    }
}

// Tiled backward: G = gY * act'(Y) for a 64-row tile (kept in shared memory
// and written out for the weight gradient), then dZ = G W^T for K = 16 KPT
// columns, W^T staged in 32-output chunks.
template <class TA, class TW, int KPT>
__global__ void __launch_bounds__(256) k_layer_dz_tile(NetLayer L, const TW* __restrict__ P, float* __restrict__ G,
                                                       float* __restrict__ dZ) {
    pdlEnter();
    constexpr int KD = 16 * KPT;
    extern __shared__ float sm[];
    const int Cout = L.Cout;
    const int ldg = Cout + 1;
    float* gs = sm;                       // [64][Cout + 1]
    float* wt = sm + kTileRows * ldg;     // [32][KD]: W^T chunk
    const int row0 = blockIdx.x * kTileRows;
    const TA* Y = (const TA*)L.Y;
    const int o = threadIdx.x % Cout, rstep = blockDim.x / Cout;  // Cout divides 256
    for (int r = threadIdx.x / Cout; r < kTileRows; r += rstep) {
        const int n = row0 + r;
        float v = 0.f;
        if (n < L.N) {
            v = L.gY[(size_t)n * Cout + o];
            if (L.relu && ldv(Y, (size_t)n * Cout + o) <= 0.f) v = 0.f;
            G[(size_t)n * Cout + o] = v;
        }
        gs[r * ldg + o] = v;
    }
    if (!dZ) return;
    // tensor cores: the 64 x KD tile of dZ is 4 x (KD/8) mma.sync m16n8k8
    // TF32 blocks dealt to the 8 warps; G split into TF32 high and low parts,
    // W exact (BF16) or split (FP32)
    constexpr int NCB = 2 * KPT, NBLK = 4 * NCB, TPW = (NBLK + 7) / 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const TW* W = P + L.wOff;
    float acc[TPW][4];
#pragma unroll
    for (int q = 0; q < TPW; q++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[q][e] = 0.f;
    for (int o0 = 0; o0 < Cout; o0 += kChunk) {
        const int on = min(kChunk, Cout - o0);
        constexpr int PER = kChunk * KD / 256;
        float wv[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int idx = threadIdx.x + 256 * u;
            const int oo = idx / KD, k = idx % KD;
            wv[u] = oo < on ? ldv(W, (size_t)k * Cout + o0 + oo) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < PER; u++) wt[threadIdx.x + 256 * u] = wv[u];
        __syncthreads();
        for (int oo = 0; oo < on; oo += 8) {
            const bool c0ok = oo + t4 < on, c1ok = oo + t4 + 4 < on;
#pragma unroll
            for (int q = 0; q < TPW; q++) {
                const int blk = warp + 8 * q;
                if (blk >= NBLK) break;
                const int rb = blk / NCB, cb = blk % NCB;
                const float* g0 = gs + (rb * 16 + g) * ldg + o0 + oo;
                const float* g1 = g0 + 8 * ldg;
                const float a[4] = {c0ok ? g0[t4] : 0.f, c0ok ? g1[t4] : 0.f, c1ok ? g0[t4 + 4] : 0.f,
                                    c1ok ? g1[t4 + 4] : 0.f};
                const float bw[2] = {wt[(oo + t4) * KD + cb * 8 + g], wt[(oo + t4 + 4) * KD + cb * 8 + g]};
                uint32_t ahi[4], alo[4], bhi[2];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    ahi[e] = toTf32(a[e]);
                    alo[e] = toTf32(a[e] - __uint_as_float(ahi[e]));
                }
#pragma unroll
                for (int e = 0; e < 2; e++) bhi[e] = toTf32(bw[e]);
                if constexpr (std::is_same<TW, float>::value) {
                    uint32_t blo[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) blo[e] = toTf32(bw[e] - __uint_as_float(bhi[e]));
                    mmaTf32(acc[q], ahi, blo);
                }
                mmaTf32(acc[q], alo, bhi);
                mmaTf32(acc[q], ahi, bhi);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < TPW; q++) {
        const int blk = warp + 8 * q;
        if (blk >= NBLK) break;
        const int rb = blk / NCB, cb = blk % NCB;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int n = row0 + rb * 16 + g + (e >= 2 ? 8 : 0);
            if (n < L.N) dZ[(size_t)n * KD + cb * 8 + 2 * t4 + (e & 1)] = acc[q][e];
        }
    }
}

// ---------------- BF16 weights: fragments straight from memory ----------------
//
// A warp computes 16 rows times 8 NB columns of A B with mma.sync m16n8k16
// (BF16 operands, FP32 accumulators) without staging A in shared memory. The
// order of the inner index is free as long as A and B agree, so the lane that
// holds k = 2t, 2t+1, 2t+8, 2t+9 of a fragment (t = lane % 4) takes the
// channels 4t .. 4t+3 of each 16-channel slab: one 16-byte load per row and
// slab, the four lanes of a row reading 64 consecutive bytes. B (the layer's
// weights) is packed in that order when the weights change (k_pack), so a CTA
// copies it as it is and a lane reads its four values of a column as 8 bytes.
//
// The FP32 operand A goes in as three BF16 parts, a = a1 + a2 + a3 with each
// part the rounding of what the parts before it leave: 24 bits, all that FP32
// holds, and every product with a BF16 weight is exact in FP32. (TF32 in two
// parts, which the tiles below use, keeps 22 bits and takes four instructions
// where this takes three.)
__device__ __forceinline__ void mmaBf16(float (&d)[4], const uint32_t (&a)[4], uint2 b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}
__device__ __forceinline__ uint32_t packBf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// the next part of (x, y), which is taken off them
__device__ __forceinline__ uint32_t nextPart(float& x, float& y) {
    const uint32_t p = packBf16(x, y);
    x -= __uint_as_float(p << 16);
    y -= __uint_as_float(p & 0xFFFF0000u);
    return p;
}
// the three parts of a lane's channels of rows g (r0) and g + 8 (r1), smallest first
__device__ __forceinline__ void splitRows(float4 r0, float4 r1, uint32_t (&a)[3][4]) {
#pragma unroll
    for (int q = 2; q >= 0; q--) {
        a[q][0] = nextPart(r0.x, r0.y);
        a[q][1] = nextPart(r1.x, r1.y);
        a[q][2] = nextPart(r0.z, r0.w);
        a[q][3] = nextPart(r1.z, r1.w);
    }
}
__device__ __forceinline__ float4 ldv4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ldv4(const bfloat* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xFFFF0000u));
}
__device__ __forceinline__ void stv4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void stv4(bfloat* p, float4 v) {
    *reinterpret_cast<uint2*>(p) = make_uint2(packBf16(v.x, v.y), packBf16(v.z, v.w));
}
__device__ __forceinline__ float2 ldv2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 ldv2(const bfloat* p) {
    const uint32_t u = *reinterpret_cast<const uint32_t*>(p);
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}
__device__ __forceinline__ void stv2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
__device__ __forceinline__ void stv2(bfloat* p, float2 v) { *reinterpret_cast<uint32_t*>(p) = packBf16(v.x, v.y); }
__device__ __forceinline__ void add4(float4& a, float4 b) {
    a.x += b.x;
    a.y += b.y;
    a.z += b.z;
    a.w += b.w;
}

// The weight groups [K][Cout] of the flat vector in fragment order, for the
// forward product (inner index K) and the input gradient's (inner index Cout).
constexpr int kMaxGroups = 24;
struct PackArgs {
    int n = 0;
    unsigned int off[kMaxGroups];
    short K[kMaxGroups], Cout[kMaxGroups];
};
__global__ void __launch_bounds__(kThreads) k_pack(PackArgs a, const bfloat* __restrict__ low, bfloat* __restrict__ fwd,
                                                   bfloat* __restrict__ bwd) {
    pdlEnter();
    const unsigned int off = a.off[blockIdx.y];
    const int K = a.K[blockIdx.y], Cout = a.Cout[blockIdx.y];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K * Cout; i += gridDim.x * blockDim.x) {
        const int e = i & 3, lane = (i >> 2) & 31, g = lane >> 2, t4 = lane & 3, blk = i >> 7;
        const int nf = Cout / 8, nbk = K / 8;  // column blocks
        fwd[off + i] = low[off + (16 * (blk / nf) + 4 * t4 + e) * Cout + (blk % nf) * 8 + g];
        bwd[off + i] = low[off + ((blk % nbk) * 8 + g) * Cout + 16 * (blk / nbk) + 4 * t4 + e];
    }
}

// The packed weights of `cols` columns and `inner` inner indices into shared memory.
__device__ __forceinline__ void stageWeights(uint2* ws, const bfloat* packed, int inner, int cols) {
    const uint4* src = reinterpret_cast<const uint4*>(packed);
    uint4* dst = reinterpret_cast<uint4*>(ws);
    for (int i = threadIdx.x; i < inner * cols / 8; i += blockDim.x) dst[i] = __ldg(src + i);
    __syncthreads();
}

// acc += the slab's three parts times its weights
template <int NB>
__device__ __forceinline__ void slabMma(float (&acc)[NB][4], float4 r0, float4 r1, const uint2* w) {
    uint32_t a[3][4];
    splitRows(r0, r1, a);
#pragma unroll
    for (int nb = 0; nb < NB; nb++) {
        const uint2 b = w[nb * 32];
#pragma unroll
        for (int q = 0; q < 3; q++) mmaBf16(acc[nb], a[q], b);
    }
}

// Sum over a list's rows of the lane's four channels. The first eight entries
// are in registers (k), further ones are read again for every slab.
template <class TA>
__device__ __forceinline__ float4 listSum(const TA* x, int C, const int (&k)[8], int len, const int32_t* more) {
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (u < len) v[u] = ldv4(x + (size_t)k[u] * C);
    }
    add4(v[0], v[1]);
    add4(v[2], v[3]);
    add4(v[0], v[2]);
    if (len > 4) {
        add4(v[4], v[5]);
        add4(v[6], v[7]);
        add4(v[4], v[6]);
        add4(v[0], v[4]);
    }
    for (int u = 8; u < len; u++) add4(v[0], ldv4(x + (size_t)__ldg(more + u) * C));
    return v[0];
}

constexpr int kMmaThreads = 128;

// What bounds it: the finest level's tiles, by L2 (each row's inputs are read
// about five times, its own and its neighbours'), the coarse levels' by the
// latency of one tile. With the tile kernel, an 874k-cell finest layer took
// 127 us and a 54-row layer 27; here 81 and 19 (cold caches).
// Y = act(Z W + b [+ add]): 16-row tiles, Cout / (8 NB) warps of a CTA on one
// tile's column groups. CTAs loop over tiles with the weights kept.
template <class TA, int NB>
__global__ void __launch_bounds__(kMmaThreads) k_layer_mma(const Ctl* ctl, int gated, NetLayer L,
                                                           const bfloat* __restrict__ P,
                                                           const bfloat* __restrict__ packed) {
    pdlEnter();
    if (idle(ctl, gated)) return;
    extern __shared__ __align__(16) uint2 wsm[];
    const int K = L.K, Cout = L.Cout;
    stageWeights(wsm, packed + L.wOff, K, Cout);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int groups = Cout / (8 * NB), perCta = (kMmaThreads / 32) / groups;
    const int col0 = (warp % groups) * 8 * NB;
    const uint2* w0 = wsm + (col0 / 8) * 32 + lane;
    const int slabW = (Cout / 8) * 32;  // weights of one slab
    const bfloat* bias = P + L.wOff + (size_t)K * Cout;
    const TA* add = (const TA*)L.add;
    TA* Y = (TA*)L.Y;
    const int tiles = (L.N + 15) / 16;
    for (int tile = blockIdx.x * perCta + warp / groups; tile < tiles; tile += gridDim.x * perCta) {
        const int r0 = tile * 16 + g, r1 = r0 + 8;
        const int n0 = min(r0, L.N - 1), n1 = min(r1, L.N - 1);  // a surplus row repeats the last one and stores nothing
        float acc[NB][4];
#pragma unroll
        for (int nb = 0; nb < NB; nb++) {
            const float2 b = ldv2(bias + col0 + nb * 8 + 2 * t4);
            acc[nb][0] = acc[nb][2] = b.x;
            acc[nb][1] = acc[nb][3] = b.y;
        }
        int k0 = 0;
#pragma unroll 1
        for (int i = 0; i < L.nIn; i++) {
            const NetIn& I = L.in[i];
            const int C = I.C;
            const TA* x = (const TA*)I.x + 4 * t4;
            const bool mean = I.xf == NX_NBMEAN || I.xf == NX_POOL;
            int ka[8], kb[8], la = 0, lb = 0;
            float ia = 1.f, ib = 1.f;
            const int32_t *ma = nullptr, *mb = nullptr;
            if (mean) {
                const int sa = I.s[n0], sb = I.s[n1];
                la = I.s[n0 + 1] - sa;
                lb = I.s[n1 + 1] - sb;
                ia = I.inv[n0];
                ib = I.inv[n1];
                ma = I.list + sa;
                mb = I.list + sb;
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    ka[u] = u < la ? __ldg(ma + u) : 0;
                    kb[u] = u < lb ? __ldg(mb + u) : 0;
                }
            } else {
                ka[0] = I.xf == NX_UNPOOL ? I.map[n0] : n0;
                kb[0] = I.xf == NX_UNPOOL ? I.map[n1] : n1;
            }
#pragma unroll 2
            for (int c = 0; c < C; c += 16, k0 += 16, x += 16) {
                float4 va, vb;
                if (mean) {
                    va = listSum(x, C, ka, la, ma);
                    vb = listSum(x, C, kb, lb, mb);
                    va.x *= ia; va.y *= ia; va.z *= ia; va.w *= ia;
                    vb.x *= ib; vb.y *= ib; vb.z *= ib; vb.w *= ib;
                } else {
                    va = ldv4(x + (size_t)ka[0] * C);
                    vb = ldv4(x + (size_t)kb[0] * C);
                }
                slabMma<NB>(acc, va, vb, w0 + (k0 / 16) * slabW);
            }
        }
#pragma unroll
        for (int nb = 0; nb < NB; nb++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int n = h ? r1 : r0;
                if (n >= L.N) continue;
                const size_t o = (size_t)n * Cout + col0 + nb * 8 + 2 * t4;
                float2 v = make_float2(acc[nb][2 * h], acc[nb][2 * h + 1]);
                if (add) {
                    const float2 d = ldv2(add + o);
                    v.x += d.x;
                    v.y += d.y;
                }
                if (L.relu) {
                    v.x = fmaxf(v.x, 0.f);
                    v.y = fmaxf(v.y, 0.f);
                }
                stv2(Y + o, v);
            }
    }
}

// G = gY act'(Y) (written for the weight gradient) and dZ = G W^T, the same way
// with Cout as the inner index and K columns.
template <class TA, int NB>
__global__ void __launch_bounds__(kMmaThreads) k_layer_dz_mma(NetLayer L, const bfloat* __restrict__ packed,
                                                              float* __restrict__ G, float* __restrict__ dZ) {
    pdlEnter();
    extern __shared__ __align__(16) uint2 wsm[];
    const int K = L.K, Cout = L.Cout;
    stageWeights(wsm, packed + L.wOff, Cout, K);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int groups = K / (8 * NB), perCta = (kMmaThreads / 32) / groups;
    const int col0 = (warp % groups) * 8 * NB;
    const uint2* w0 = wsm + (col0 / 8) * 32 + lane;
    const int slabW = (K / 8) * 32;
    const TA* Y = (const TA*)L.Y;
    const int tiles = (L.N + 15) / 16;
    auto masked = [&](int n, int c) {
        const size_t o = (size_t)n * Cout + c;
        float4 v = ldv4(L.gY + o);
        if (L.relu) {
            const float4 y = ldv4(Y + o);
            if (y.x <= 0.f) v.x = 0.f;
            if (y.y <= 0.f) v.y = 0.f;
            if (y.z <= 0.f) v.z = 0.f;
            if (y.w <= 0.f) v.w = 0.f;
        }
        return v;
    };
    for (int tile = blockIdx.x * perCta + warp / groups; tile < tiles; tile += gridDim.x * perCta) {
        const int r0 = tile * 16 + g, r1 = r0 + 8;
        const int n0 = min(r0, L.N - 1), n1 = min(r1, L.N - 1);
        float acc[NB][4];
#pragma unroll
        for (int nb = 0; nb < NB; nb++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[nb][e] = 0.f;
#pragma unroll 2
        for (int c = 0; c < Cout; c += 16) {
            const float4 va = masked(n0, c + 4 * t4), vb = masked(n1, c + 4 * t4);
            if (col0 == 0) {
                if (r0 < L.N) stv4(G + (size_t)r0 * Cout + c + 4 * t4, va);
                if (r1 < L.N) stv4(G + (size_t)r1 * Cout + c + 4 * t4, vb);
            }
            slabMma<NB>(acc, va, vb, w0 + (c / 16) * slabW);
        }
#pragma unroll
        for (int nb = 0; nb < NB; nb++) {
            const int o = col0 + nb * 8 + 2 * t4;
            if (r0 < L.N) stv2(dZ + (size_t)r0 * K + o, make_float2(acc[nb][0], acc[nb][1]));
            if (r1 < L.N) stv2(dZ + (size_t)r1 * K + o, make_float2(acc[nb][2], acc[nb][3]));
        }
    }
}

// The input layer (two features per row), four lanes a row.
template <class TA>
__global__ void __launch_bounds__(kThreads) k_layer_in(const Ctl* ctl, int gated, NetLayer L,
                                                       const bfloat* __restrict__ P) {
    pdlEnter();
    if (idle(ctl, gated)) return;
    const int per = L.Cout / 4;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = i / per;
    const int o = (int)(i % per) * 4;
    if (n >= (size_t)L.N) return;
    const bfloat* W = P + L.wOff;
    const float2 z = ldv2((const TA*)L.in[0].x + 2 * n);
    const float4 w0 = ldv4(W + o), w1 = ldv4(W + L.Cout + o), b = ldv4(W + 2 * L.Cout + o);
    float4 v = make_float4(fmaf(z.y, w1.x, fmaf(z.x, w0.x, b.x)), fmaf(z.y, w1.y, fmaf(z.x, w0.y, b.y)),
                           fmaf(z.y, w1.z, fmaf(z.x, w0.z, b.z)), fmaf(z.y, w1.w, fmaf(z.x, w0.w, b.w)));
    if (L.relu) v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
    stv4((TA*)L.Y + n * L.Cout + o, v);
}

// The output layer (16 channels to one value), four lanes a row.
template <class TA>
__global__ void __launch_bounds__(kThreads) k_layer_out(const Ctl* ctl, int gated, NetLayer L,
                                                        const bfloat* __restrict__ P) {
    pdlEnter();
    if (idle(ctl, gated)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = i >> 2, t4 = i & 3;
    const int m = min(n, L.N - 1);
    const float4 z = ldv4((const TA*)L.in[0].x + (size_t)m * 16 + 4 * t4), w = ldv4(P + L.wOff + 4 * t4);
    float v = fmaf(z.w, w.w, fmaf(z.z, w.z, fmaf(z.y, w.y, z.x * w.x)));
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
    if (t4 == 0 && n < L.N) stv((TA*)L.Y, n, v + ldv(P, L.wOff + 16));
}

// Its input gradient straight into the source's: gX[n][k] += g[n] w[k].
__global__ void __launch_bounds__(kThreads) k_adj_out(NetLayer L, const bfloat* __restrict__ P, float* __restrict__ gX) {
    pdlEnter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = i >> 2, t4 = i & 3;
    if (n >= L.N) return;
    const float g = L.gY[n];
    const float4 w = ldv4(P + L.wOff + 4 * t4);
    float* p = gX + (size_t)n * 16 + 4 * t4;
    float4 v = ldv4(p);
    add4(v, make_float4(g * w.x, g * w.y, g * w.z, g * w.w));
    stv4(p, v);
}

// G = gY act'(Y) alone (the input layer has no input gradient)
template <class TA>
__global__ void __launch_bounds__(kThreads) k_mask(size_t n4, const float* __restrict__ gY, const TA* __restrict__ Y,
                                                   float* __restrict__ G) {
    pdlEnter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    float4 v = ldv4(gY + 4 * i);
    const float4 y = ldv4(Y + 4 * i);
    if (y.x <= 0.f) v.x = 0.f;
    if (y.y <= 0.f) v.y = 0.f;
    if (y.z <= 0.f) v.z = 0.f;
    if (y.w <= 0.f) v.w = 0.f;
    stv4(G + 4 * i, v);
}

// e = sigma * y
template <class TA>
__global__ void __launch_bounds__(kThreads) k_scale_out(const Ctl* ctl, int gated, int N, const TA* y, const double* scal,
                                                        float* e) {
    pdlEnter();
    if (idle(ctl, gated)) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    e[n] = (float)(sqrt(scal[0]) * (double)ldv(y, n));
}

// ---------------- loss ----------------

// Loss: the A-norm (energy) error left after the best scaling of the output,
//   loss = min_a ||a y - t||_A^2 / ||t||_A^2 = 1 - (y.b)^2 / ((y.A y)(b.t)),
// with A t = b. The Krylov solve applies the network's output with its own
// line search, which minimises exactly this error, so only y's direction in
// the energy norm matters. scal[1..3] = y.b, y.Ay, b.t.
template <class TA>
__global__ void __launch_bounds__(kThreads) k_loss_spmv(int N, int W, const int32_t* __restrict__ nb,
                                                        const float* __restrict__ AF, const float* __restrict__ AC,
                                                        const TA* y, const float* b, const float* t, float* Ay,
                                                        double* partial, unsigned int* counter, double* scal) {
    pdlEnter();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[3] = {0.0, 0.0, 0.0};
    if (n < N) {
        const double yn = (double)ldv(y, n);
        double a = (double)AC[n] * yn;
        for (int j = 0; j < W; j++) {
            const size_t sl = (size_t)j * N + n;
            const int k = nb[sl];
            if (k >= 0) a += (double)AF[sl] * (double)ldv(y, k);
        }
        Ay[n] = (float)a;
        acc[0] = yn * (double)b[n];
        acc[1] = yn * a;
        acc[2] = (double)b[n] * (double)t[n];
    }
    gridSumD<3>(acc, partial, counter, scal + 1);
}

// d loss / d y = -2 c / (E_y E_t) b + 2 c^2 / (E_y^2 E_t) A y,  c = y.b,
// E_y = y.Ay, E_t = b.t (A symmetric)
__global__ void __launch_bounds__(kThreads) k_loss_grad(int N, const float* b, const float* Ay, const double* scal,
                                                        float* gy, float* lossOut) {
    pdlEnter();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const double c = scal[1], ey = scal[2] > 0.0 ? scal[2] : 1e-300, et = scal[3] > 0.0 ? scal[3] : 1.0;
    if (n == 0) *lossOut = (float)(1.0 - c * c / (ey * et));
    if (n >= N) return;
    gy[n] = (float)(-2.0 * c / (ey * et) * (double)b[n] + 2.0 * c * c / (ey * ey * et) * (double)Ay[n]);
}

// ---------------- layer backward ----------------

// G = gY * act'(Y) ; dZ = G W^T (dZ may be null)
template <class TA, class TW, int KCH>
__global__ void __launch_bounds__(kThreads) k_layer_dz(NetLayer L, const TW* __restrict__ P, float* __restrict__ G,
                                                       float* __restrict__ dZ) {
    pdlEnter();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= L.N) return;
    const int K = L.K, Cout = L.Cout;
    const TA* Y = (const TA*)L.Y;
    for (int o = 0; o < Cout; o++) {
        float g = L.gY[(size_t)n * Cout + o];
        if (L.relu && ldv(Y, (size_t)n * Cout + o) <= 0.f) g = 0.f;
        G[(size_t)n * Cout + o] = g;
    }
    if (!dZ) return;
    const TW* W = P + L.wOff;
    for (int k0 = 0; k0 < K; k0 += KCH) {
        float acc[KCH];
#pragma unroll
        for (int j = 0; j < KCH; j++) acc[j] = 0.f;
        for (int o = 0; o < Cout; o++) {
            const float g = G[(size_t)n * Cout + o];
#pragma unroll
            for (int j = 0; j < KCH; j++)
                if (k0 + j < K) acc[j] = fmaf(g, ldv(W, (size_t)(k0 + j) * Cout + o), acc[j]);
        }
#pragma unroll
        for (int j = 0; j < KCH; j++)
            if (k0 + j < K) dZ[(size_t)n * K + k0 + j] = acc[j];
    }
}

// partial[split][K*Cout + Cout] = (Z^T G, sum G) over the split's rows.
// Block: a 32 x 32 tile of (k, o), 64 rows at a time; the next rows' values are
// loaded into registers while the current ones are multiplied.
template <class TA>
__global__ void __launch_bounds__(kThreads) k_wgrad(int N, int K, int Cout, int tilesO, int rowsPerSplit,
                                                    const TA* __restrict__ Z, const float* __restrict__ G,
                                                    float* __restrict__ partial) {
    pdlEnter();
    __shared__ float zs[64][33];
    __shared__ float gs[64][33];
    const int tk = blockIdx.x / tilesO, to = blockIdx.x % tilesO;
    const int k0 = tk * 32, o0 = to * 32;
    const int split = blockIdx.y;
    const int r0 = split * rowsPerSplit;
    const int r1 = min(N, r0 + rowsPerSplit);
    // tensor cores: the 32 x 32 tile of dW = Z^T G is 2 x 4 mma.sync m16n8k8
    // TF32 blocks, one per warp, reduced over the rows 8 at a time; FP32
    // operands split into TF32 high and low parts (BF16 activations are exact)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int mb = warp >> 2, nb = warp & 3;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    float bacc = 0.f;  // this warp's rows of column o0 + lane
    float zr[8], gr[8];
    auto load = [&](int rc) {
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int n = rc + warp + 8 * u;
            zr[u] = (n < r1 && k0 + lane < K) ? ldv(Z, (size_t)n * K + k0 + lane) : 0.f;
            gr[u] = (n < r1 && o0 + lane < Cout) ? G[(size_t)n * Cout + o0 + lane] : 0.f;
        }
    };
    load(r0);
    for (int rc = r0; rc < r1; rc += 64) {
#pragma unroll
        for (int u = 0; u < 8; u++) {
            zs[warp + 8 * u][lane] = zr[u];
            gs[warp + 8 * u][lane] = gr[u];
            bacc += gr[u];
        }
        __syncthreads();
        if (rc + 64 < r1) load(rc + 64);
#pragma unroll 2
        for (int kk = 0; kk < 64; kk += 8) {
            const float a[4] = {zs[kk + t4][mb * 16 + g], zs[kk + t4][mb * 16 + g + 8], zs[kk + t4 + 4][mb * 16 + g],
                                zs[kk + t4 + 4][mb * 16 + g + 8]};
            const float b[2] = {gs[kk + t4][nb * 8 + g], gs[kk + t4 + 4][nb * 8 + g]};
            uint32_t ahi[4], bhi[2], blo[2];
#pragma unroll
            for (int e = 0; e < 4; e++) ahi[e] = toTf32(a[e]);
#pragma unroll
            for (int e = 0; e < 2; e++) {
                bhi[e] = toTf32(b[e]);
                blo[e] = toTf32(b[e] - __uint_as_float(bhi[e]));
            }
            if constexpr (std::is_same<TA, float>::value) {
                uint32_t alo[4];
#pragma unroll
                for (int e = 0; e < 4; e++) alo[e] = toTf32(a[e] - __uint_as_float(ahi[e]));
                mmaTf32(acc, alo, bhi);
            }
            mmaTf32(acc, ahi, blo);
            mmaTf32(acc, ahi, bhi);
        }
        __syncthreads();
    }
    const size_t stride = (size_t)K * Cout + Cout;
    float* out = partial + (size_t)split * stride;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int k = k0 + mb * 16 + g + (e >= 2 ? 8 : 0);
        const int o = o0 + nb * 8 + 2 * t4 + (e & 1);
        if (k < K && o < Cout) out[(size_t)k * Cout + o] = acc[e];
    }
    if (tk != 0) return;
    zs[warp][lane] = bacc;
    __syncthreads();
    if (warp == 0 && o0 + lane < Cout) {
        for (int w = 1; w < kThreads / 32; w++) bacc += zs[w][lane];
        out[(size_t)K * Cout + o0 + lane] = bacc;
    }
}

// grad += the sum of the splits: 32 entries a block, eight threads an entry
__global__ void __launch_bounds__(kThreads) k_wgrad_reduce(int entries, int splits, const float* __restrict__ partial,
                                                           float* __restrict__ grad) {
    pdlEnter();
    __shared__ float sh[8][32];
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (e < entries) {
#pragma unroll 8
        for (int i = part; i < splits; i += 8) s += partial[(size_t)i * entries + e];
    }
    sh[part][lane] = s;
    __syncthreads();
    if (part == 0 && e < entries) {
        for (int w = 1; w < 8; w++) s += sh[w][lane];
        grad[e] += s;
    }
}

// adjoints: accumulate segment [off, off + C) of dZ (row stride K) into gX,
// four channels a thread (every C, K and off is a multiple of four)
__device__ __forceinline__ void accumulate4(float* p, float4 v) {
    float4 x = ldv4(p);
    add4(x, v);
    stv4(p, x);
}
__device__ __forceinline__ float4 scaled(float4 v, float w) { return make_float4(v.x * w, v.y * w, v.z * w, v.w * w); }

__global__ void __launch_bounds__(kThreads) k_adj_id(int N, int C, int off, int K, const float* __restrict__ dZ,
                                                     float* __restrict__ gX) {
    pdlEnter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, per = (size_t)C / 4;
    if (i >= (size_t)N * per) return;
    accumulate4(gX + 4 * i, ldv4(dZ + (i / per) * K + off + 4 * (i % per)));
}

// the message-passing layer's two inputs in one pass: the identity, then the
// neighbour mean transposed, gX[k] += dZ[k] + sum_{n in nb(k)} invDeg[n] dZ[n]
__global__ void __launch_bounds__(kThreads) k_adj_mp(int N, int C, int K, const int32_t* __restrict__ s,
                                                     const int32_t* __restrict__ list, const float* __restrict__ inv,
                                                     const float* __restrict__ dZ, float* __restrict__ gX) {
    pdlEnter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, per = (size_t)C / 4;
    if (i >= (size_t)N * per) return;
    const int k = (int)(i / per), c = (int)(i % per) * 4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const int q1 = s[k + 1];
    for (int q = s[k]; q < q1; q += 4) {
        int n[4];
        float w[4];
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) n[u] = list[min(q + u, q1 - 1)];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            w[u] = inv[n[u]];
            v[u] = ldv4(dZ + (size_t)n[u] * K + C + c);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (q + u < q1) {
                acc.x = fmaf(w[u], v[u].x, acc.x);
                acc.y = fmaf(w[u], v[u].y, acc.y);
                acc.z = fmaf(w[u], v[u].z, acc.z);
                acc.w = fmaf(w[u], v[u].w, acc.w);
            }
    }
    float* p = gX + (size_t)k * C + c;
    float4 x = ldv4(p);
    add4(x, ldv4(dZ + (size_t)k * K + c));
    add4(x, acc);
    stv4(p, x);
}

// pool transposed: gX[m] += invCnt[c] dZ[c], c = c2c[m] (m over the fine rows)
__global__ void __launch_bounds__(kThreads) k_adj_pool(int Nf, int C, int off, int K, const int32_t* __restrict__ c2c,
                                                       const float* __restrict__ invCnt, const float* __restrict__ dZ,
                                                       float* __restrict__ gX) {
    pdlEnter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, per = (size_t)C / 4;
    if (i >= (size_t)Nf * per) return;
    const int cc = c2c[i / per];
    accumulate4(gX + 4 * i, scaled(ldv4(dZ + (size_t)cc * K + off + 4 * (i % per)), invCnt[cc]));
}

// unpool transposed: gX[c] += sum_{m in members(c)} dZ[m] (c over the coarse rows)
__global__ void __launch_bounds__(kThreads) k_adj_unpool(int Nc, int C, int off, int K, const int32_t* __restrict__ ms,
                                                         const int32_t* __restrict__ ml, const float* __restrict__ dZ,
                                                         float* __restrict__ gX) {
    pdlEnter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, per = (size_t)C / 4;
    if (i >= (size_t)Nc * per) return;
    const int c = (int)(i / per);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = ms[c]; q < ms[c + 1]; q++) add4(acc, ldv4(dZ + (size_t)ml[q] * K + off + 4 * (i % per)));
    accumulate4(gX + 4 * i, acc);
}

// ---------------- optimiser ----------------

template <class TW>
__global__ void __launch_bounds__(kThreads) k_adam(size_t n, float* __restrict__ p, const float* __restrict__ g,
                                                   float* __restrict__ m, float* __restrict__ v, TW* low, float lr,
                                                   float b1, float b2, float eps, float c1, float c2) {
    pdlEnter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    stv(low, i, pi);
}

template <class TW>
__global__ void __launch_bounds__(kThreads) k_to_low(size_t n, const float* __restrict__ p, TW* __restrict__ low) {
    pdlEnter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) stv(low, i, p[i]);
}

// Appends (b, x, A_C, deficit, A_F) of this iteration's p' system to the sample
// store (FP32, [4 + W][N] per sample, A_F as ELL [W][N]) when the iteration
// counter is a multiple of `every` and the store has room; fs (nullable) holds
// the Krylov solve's (b, b) and (r, r) for the sample's relative residual.
__global__ void __launch_bounds__(kThreads) k_harvest(const Ctl* ctl, int N, int every, int cap, const double* b,
                                                      const double* x, const double* AC, const double* AF,
                                                      const int32_t* nb, int W, const double* fs, float* store,
                                                      int* count, float* relres, unsigned int* counter) {
    pdlEnter();
    if (ctl->done || every <= 0 || (ctl->currentIteration % every) != 0) return;
    const int slot = *(volatile int*)count;
    if (slot >= cap) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < N) {
        float* base = store + (size_t)slot * (4 + W) * N;
        const double ac = AC[n];
        double sum = 0.0;
        for (int j = 0; j < W; j++) {
            const size_t sl = (size_t)j * N + n;
            const bool in = nb[sl] >= 0;
            if (in) sum += fabs(AF[sl]);
            base[(size_t)(4 + j) * N + n] = in ? (float)AF[sl] : 0.f;
        }
        base[n] = (float)b[n];
        base[(size_t)N + n] = (float)x[n];
        base[2 * (size_t)N + n] = (float)ac;
        base[3 * (size_t)N + n] = ac != 0.0 ? (float)(1.0 - sum / ac) : 0.f;
    }
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        relres[slot] = (fs && fs[4] > 0.0) ? (float)sqrt(fs[5] / fs[4]) : -1.f;
        *count = slot + 1;
        *counter = 0u;
    }
}

// ---------------- host helpers ----------------

// Opts a kernel into more than 48 KB of dynamic shared memory, once per device.
template <class F>
void allowSmem(F* f, size_t bytes) {
    if (bytes <= 48 * 1024) return;
    static std::mutex mu;
    static std::vector<std::pair<int, const void*>> done;
    int dev = 0;
    NCK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    for (auto& d : done)
        if (d.first == dev && d.second == (const void*)f) return;
    NCK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
    done.push_back({dev, (const void*)f});
}

template <class TA, class TW, int CPT, int RPT>
void launchTileR(const Ctl* ctl, int gated, const NetLayer& L, const void* P, cudaStream_t s) {
    const size_t smem =
        ((size_t)16 * RPT * (L.K + 1) + (size_t)kChunk * 16 * CPT + 16 * RPT + 1) * sizeof(float);
    allowSmem(k_layer_tile<TA, TW, CPT, RPT>, smem);
    launchPDL(k_layer_tile<TA, TW, CPT, RPT>, dim3(blocksFor(L.N, 16 * RPT)), dim3(256), smem, s, ctl, gated, L, (const TW*)P);
}

// 64-row tiles on large levels; 16-row tiles (4 x the blocks, 1/4 the work
// per thread) where a level has too few rows to fill the GPU.
template <class TA, class TW, int CPT>
void launchTile(const Ctl* ctl, int gated, const NetLayer& L, const void* P, cudaStream_t s) {
    if (L.N >= 148 * 64 * 4) launchTileR<TA, TW, CPT, 4>(ctl, gated, L, P, s);
    else launchTileR<TA, TW, CPT, 1>(ctl, gated, L, P, s);
}

template <class TA, class TW, int KPT>
void launchDzTile(const NetLayer& L, const void* P, float* G, float* dZ, cudaStream_t s) {
    const size_t smem = ((size_t)kTileRows * (L.Cout + 1) + (size_t)kChunk * 16 * KPT) * sizeof(float);
    allowSmem(k_layer_dz_tile<TA, TW, KPT>, smem);
    launchPDL(k_layer_dz_tile<TA, TW, KPT>, dim3(blocksFor(L.N, kTileRows)), dim3(256), smem, s, L, (const TW*)P, G, dZ);
}

// The tiled kernels assume every channel count divides their 256 threads.
inline bool tileable(const NetLayer& L) {
    if (L.K > 256 || 256 % L.K != 0 || L.Cout > 256 || 256 % L.Cout != 0) return false;
    for (int i = 0; i < L.nIn; i++)
        if (256 % L.in[i].C != 0) return false;
    return true;
}

// The fragment kernels take layers whose inputs and outputs come in whole
// 16-channel slabs of at most 256 and 128 channels: all but the first and the
// last layer.
inline bool slabs(const NetLayer& L) {
    const auto pow2 = [](int c, int most) { return c >= 16 && c <= most && (c & (c - 1)) == 0; };
    return pow2(L.K, 256) && pow2(L.Cout, 128);
}
// Column blocks of eight a warp: up to eight, so a tile's gather is done by as
// few warps as the registers allow (four on the coarse levels, for more warps a
// tile, measured no faster: 1.99 against 1.99 ms a prediction on 874k cells,
// and 2.08 with four on every level).
inline int mmaBlocks(int cols) { return std::min(cols / 8, 8); }

// CTAs that loop over the tiles: at most as many as shared memory (192 KB of
// weights an SM) and 48 warps an SM would hold. Their registers (127) let 16
// warps an SM run at once; a grid of just those measured the same.
inline int mmaCtas(const NetLayer& L, int tilesPerCta, size_t smem) {
    const int perSm = (int)std::min<size_t>(48 * 32 / kMmaThreads, 192 * 1024 / smem);
    return std::min((L.N + 16 * tilesPerCta - 1) / (16 * tilesPerCta), 148 * perSm);
}

template <class TA, int NB>
void launchMmaNB(const Ctl* ctl, int gated, const NetLayer& L, const bfloat* P, const bfloat* packed, cudaStream_t s) {
    const size_t smem = (size_t)L.K * L.Cout * sizeof(bfloat);
    allowSmem(k_layer_mma<TA, NB>, smem);
    const int perCta = (kMmaThreads / 32) / (L.Cout / (8 * NB));
    launchPDL(k_layer_mma<TA, NB>, dim3(mmaCtas(L, perCta, smem)), dim3(kMmaThreads), smem, s, ctl, gated, L, P, packed);
}
template <class TA>
void launchMma(const Ctl* ctl, int gated, const NetLayer& L, const bfloat* P, const bfloat* packed, cudaStream_t s) {
    switch (mmaBlocks(L.Cout)) {
        case 2: launchMmaNB<TA, 2>(ctl, gated, L, P, packed, s); return;
        case 4: launchMmaNB<TA, 4>(ctl, gated, L, P, packed, s); return;
        default: launchMmaNB<TA, 8>(ctl, gated, L, P, packed, s); return;
    }
}
template <class TA, int NB>
void launchDzMmaNB(const NetLayer& L, const bfloat* packed, float* G, float* dZ, cudaStream_t s) {
    const size_t smem = (size_t)L.K * L.Cout * sizeof(bfloat);
    allowSmem(k_layer_dz_mma<TA, NB>, smem);
    const int perCta = (kMmaThreads / 32) / (L.K / (8 * NB));
    launchPDL(k_layer_dz_mma<TA, NB>, dim3(mmaCtas(L, perCta, smem)), dim3(kMmaThreads), smem, s, L, packed, G, dZ);
}
template <class TA>
void launchDzMma(const NetLayer& L, const bfloat* packed, float* G, float* dZ, cudaStream_t s) {
    switch (mmaBlocks(L.K)) {
        case 2: launchDzMmaNB<TA, 2>(L, packed, G, dZ, s); return;
        case 4: launchDzMmaNB<TA, 4>(L, packed, G, dZ, s); return;
        default: launchDzMmaNB<TA, 8>(L, packed, G, dZ, s); return;
    }
}

// A layer with BF16 weights.
template <class TA>
void launchLayerLow(const Ctl* ctl, int gated, const NetLayer& L, const bfloat* P, const bfloat* packed,
                    cudaStream_t s) {
    if (slabs(L)) launchMma<TA>(ctl, gated, L, P, packed, s);
    else if (L.K == 2) launchPDL(k_layer_in<TA>, dim3(blocksFor((size_t)L.N * L.Cout / 4)), dim3(kThreads), 0, s, ctl, gated, L, P);
    else launchPDL(k_layer_out<TA>, dim3(blocksFor((size_t)L.N * 4)), dim3(kThreads), 0, s, ctl, gated, L, P);
}

template <class TA, class TW>
void launchLayerFwd(const Ctl* ctl, int gated, const NetLayer& L, const void* P, cudaStream_t s) {
    switch (tileable(L) ? L.Cout : 0) {
        case 16: launchTile<TA, TW, 1>(ctl, gated, L, P, s); return;
        case 32: launchTile<TA, TW, 2>(ctl, gated, L, P, s); return;
        case 64: launchTile<TA, TW, 4>(ctl, gated, L, P, s); return;
        case 128: launchTile<TA, TW, 8>(ctl, gated, L, P, s); return;
        default: break;
    }
    const int rows = L.K <= 64 ? 128 : 32;
    const size_t smem = (size_t)rows * (L.K + 1) * sizeof(float);
    const dim3 grid(blocksFor(L.N, rows));
    const TW* p = (const TW*)P;
    if (L.Cout >= 32) launchPDL(k_layer_fwd<TA, TW, 32>, dim3(grid), dim3(rows), smem, s, ctl, gated, L, p);
    else if (L.Cout >= 16) launchPDL(k_layer_fwd<TA, TW, 16>, dim3(grid), dim3(rows), smem, s, ctl, gated, L, p);
    else launchPDL(k_layer_fwd<TA, TW, 1>, dim3(grid), dim3(rows), smem, s, ctl, gated, L, p);
}

template <class TA, class TW>
void launchLayerDz(const NetLayer& L, const void* P, float* G, float* dZ, cudaStream_t s) {
    if (dZ && tileable(L)) {
        switch (L.K) {
            case 16: launchDzTile<TA, TW, 1>(L, P, G, dZ, s); return;
            case 32: launchDzTile<TA, TW, 2>(L, P, G, dZ, s); return;
            case 64: launchDzTile<TA, TW, 4>(L, P, G, dZ, s); return;
            case 128: launchDzTile<TA, TW, 8>(L, P, G, dZ, s); return;
            case 256: launchDzTile<TA, TW, 16>(L, P, G, dZ, s); return;
            default: break;
        }
    }
    launchPDL(k_layer_dz<TA, TW, 16>, dim3(blocksFor(L.N)), dim3(kThreads), 0, s, L, (const TW*)P, G, dZ);
}

template <class T>
T* devAlloc(std::vector<void*>& list, size_t n) {
    void* p = nullptr;
    NCK(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)));
    list.push_back(p);
    NCK(cudaMemset(p, 0, std::max<size_t>(n, 1) * sizeof(T)));
    return static_cast<T*>(p);
}

template <class T>
T* devUpload(std::vector<void*>& list, const std::vector<T>& h) {
    T* d = devAlloc<T>(list, h.size());
    if (!h.empty()) NCK(cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
    return d;
}

// Splits of a layer's rows for its weight gradient: enough blocks (with its
// 32 x 32 tiles) for eight on each of 148 SMs, and at least 128 rows in each.
inline int wgradSplits(const NetLayer& L) {
    const int tiles = ((L.K + 31) / 32) * ((L.Cout + 31) / 32);
    return std::max(1, std::min((L.N + 127) / 128, (1184 + tiles - 1) / tiles));
}

}  // namespace

void launchHarvest(const Ctl* ctl, int N, int every, int cap, const double* b, const double* x, const double* AC,
                   const double* AF, const int32_t* nb, int W, const double* fcgScalars, float* store, int* count,
                   float* relres, unsigned int* counter, cudaStream_t s) {
    launchPDL(k_harvest, dim3(blocksFor(N)), dim3(kThreads), 0, s, ctl, N, every, cap, b, x, AC, AF, nb, W, fcgScalars, store, count,
                                                relres, counter);
}

// ---------------- LearnedNet ----------------

LearnedNet::~LearnedNet() { release(); }

void LearnedNet::release() {
    for (void* p : allocs_) cudaFree(p);
    allocs_.clear();
    g_.clear();
    layers_.clear();
    N0_ = 0;
    L_ = 0;
    nParams_ = 0;
}

void LearnedNet::init(const std::vector<GridLevel>& hier, const int32_t* nb, int W, int precision, uint64_t seed,
                      cudaStream_t s) {
    release();
    if (hier.empty()) throw std::runtime_error("learned preconditioner needs the multigrid hierarchy");
    nb0_ = nb;
    W0_ = W;
    // precision: 0 FP32 throughout, 1 BF16 weights and activations, 2 BF16
    // weights with FP32 activations
    actBf16_ = precision == 1 ? 1 : 0;
    wBf16_ = precision == 1 || precision == 2 ? 1 : 0;
    L_ = std::min<int>((int)hier.size(), 16);
    N0_ = hier[0].nCells;
    g_.assign((size_t)L_, NetGraphLevel{});
    C_.assign((size_t)L_, 128);
    const int chan[3] = {16, 32, 64};
    for (int l = 0; l < L_ && l < 3; l++) C_[(size_t)l] = chan[l];
    for (int l = 0; l < L_; l++) {
        const GridLevel& h = hier[(size_t)l];
        NetGraphLevel& G = g_[(size_t)l];
        G.N = h.nCells;
        std::vector<int32_t> ns((size_t)h.nCells + 1, 0), nl;
        std::vector<float> inv((size_t)h.nCells, 0.f);
        for (int c = 0; c < h.nCells; c++) {
            for (int q = h.faceStart[(size_t)c]; q < h.faceStart[(size_t)c + 1]; q++) {
                const int k = h.faceNeighbor[(size_t)q];
                if (k >= 0 && k != c) nl.push_back(k);
            }
            ns[(size_t)c + 1] = (int32_t)nl.size();
            const int d = ns[(size_t)c + 1] - ns[(size_t)c];
            inv[(size_t)c] = d > 0 ? 1.f / (float)d : 0.f;
        }
        G.nStart = devUpload(allocs_, ns);
        G.nList = devUpload(allocs_, nl);
        G.invDeg = devUpload(allocs_, inv);
        if (l + 1 < L_) G.c2c = devUpload(allocs_, h.cellToCoarse);
        if (l > 0) {
            const GridLevel& f = hier[(size_t)l - 1];
            std::vector<int32_t> ms((size_t)h.nCells + 1, 0), ml((size_t)f.nCells);
            for (int m = 0; m < f.nCells; m++) ms[(size_t)f.cellToCoarse[(size_t)m] + 1]++;
            for (int c = 0; c < h.nCells; c++) ms[(size_t)c + 1] += ms[(size_t)c];
            std::vector<int32_t> fill(ms.begin(), ms.end() - 1);
            for (int m = 0; m < f.nCells; m++) ml[(size_t)fill[(size_t)f.cellToCoarse[(size_t)m]]++] = m;
            std::vector<float> ic((size_t)h.nCells, 0.f);
            for (int c = 0; c < h.nCells; c++) {
                const int d = ms[(size_t)c + 1] - ms[(size_t)c];
                ic[(size_t)c] = d > 0 ? 1.f / (float)d : 0.f;
            }
            G.mStart = devUpload(allocs_, ms);
            G.mList = devUpload(allocs_, ml);
            G.invCnt = devUpload(allocs_, ic);
        }
    }
    buildLayers();
    // He-uniform weights, zero biases, from a fixed seed
    std::vector<float> hp(nParams_, 0.f);
    std::mt19937_64 rng(seed);
    std::vector<char> done(nParams_, 0);
    for (const NetLayer& L : layers_) {
        if (done[L.wOff]) continue;
        done[L.wOff] = 1;
        const float a = L.relu ? std::sqrt(6.f / (float)L.K) : std::sqrt(3.f / (float)L.K);
        std::uniform_real_distribution<float> U(-a, a);
        for (size_t i = 0; i < (size_t)L.K * L.Cout; i++) hp[L.wOff + i] = U(rng);
    }
    NCK(cudaMemcpy(params_, hp.data(), nParams_ * sizeof(float), cudaMemcpyHostToDevice));
    syncLowPrecision(s);
    NCK(cudaStreamSynchronize(s));
}

void LearnedNet::buildLayers() {
    const size_t tsz = actBf16_ ? sizeof(bfloat) : sizeof(float);
    auto act = [&](size_t n) { return (void*)devAlloc<unsigned char>(allocs_, n * tsz); };
    auto grd = [&](size_t n) { return devAlloc<float>(allocs_, n); };
    const int L = L_;
    // the activations' gradients in one block, zeroed together before a backward pass
    gradActs_ = 0;
    for (int l = 0; l < L; l++) gradActs_ += 4 * (size_t)g_[(size_t)l].N * C_[(size_t)l];
    gActs_ = grd(gradActs_);
    size_t gUsed = 0;
    auto actGrd = [&](size_t n) {
        gUsed += n;
        return gActs_ + gUsed - n;
    };
    std::vector<void*> H((size_t)L), E((size_t)L), S((size_t)L), D((size_t)L);
    std::vector<float*> gH((size_t)L), gE((size_t)L), gS((size_t)L), gD((size_t)L);
    for (int l = 0; l < L; l++) {
        const size_t n = (size_t)g_[(size_t)l].N * C_[(size_t)l];
        H[(size_t)l] = act(n);
        E[(size_t)l] = act(n);
        S[(size_t)l] = act(n);
        D[(size_t)l] = act(n);
        gH[(size_t)l] = actGrd(n);
        gE[(size_t)l] = actGrd(n);
        gS[(size_t)l] = actGrd(n);
        gD[(size_t)l] = actGrd(n);
    }
    feat_ = act((size_t)N0_ * 2);
    out_ = act((size_t)N0_);
    gOut_ = grd((size_t)N0_);
    // weight groups, allocated in first-use order
    std::vector<std::pair<std::string, size_t>> groups;
    size_t total = 0;
    auto group = [&](const std::string& key, int K, int Cout) -> size_t {
        for (auto& g : groups)
            if (g.first == key) return g.second;
        const size_t off = total;
        total += (size_t)K * Cout + Cout;
        groups.push_back({key, off});
        return off;
    };
    auto idIn = [&](const void* x, int C, int rows) {
        NetIn I;
        I.x = x;
        I.C = C;
        I.xf = NX_ID;
        I.srcRows = rows;
        return I;
    };
    auto mp = [&](const std::string& key, int l, void* X, float* gX, void* Y, float* gY) {
        NetLayer Ly;
        Ly.N = g_[(size_t)l].N;
        Ly.K = 2 * C_[(size_t)l];
        Ly.Cout = C_[(size_t)l];
        Ly.wOff = group(key, Ly.K, Ly.Cout);
        Ly.in[0] = idIn(X, C_[(size_t)l], Ly.N);
        NetIn I;
        I.x = X;
        I.C = C_[(size_t)l];
        I.xf = NX_NBMEAN;
        I.s = g_[(size_t)l].nStart;
        I.list = g_[(size_t)l].nList;
        I.inv = g_[(size_t)l].invDeg;
        I.srcRows = Ly.N;
        Ly.in[1] = I;
        Ly.nIn = 2;
        Ly.Y = Y;
        Ly.gY = gY;
        Ly.gIn[0] = gX;
        Ly.gIn[1] = gX;
        return Ly;
    };
    layers_.clear();
    {  // input
        NetLayer Ly;
        Ly.N = N0_;
        Ly.K = 2;
        Ly.Cout = C_[0];
        Ly.wOff = group("in", 2, C_[0]);
        Ly.in[0] = idIn(feat_, 2, N0_);
        Ly.nIn = 1;
        Ly.Y = H[0];
        Ly.gY = gH[0];
        layers_.push_back(Ly);
    }
    layers_.push_back(mp("enc0", 0, H[0], gH[0], E[0], gE[0]));
    for (int l = 1; l < L; l++) {
        NetLayer Ly;
        Ly.N = g_[(size_t)l].N;
        Ly.K = C_[(size_t)l - 1];
        Ly.Cout = C_[(size_t)l];
        Ly.wOff = group("down" + std::to_string(std::min(l, 4)), Ly.K, Ly.Cout);
        NetIn I;
        I.x = E[(size_t)l - 1];
        I.C = C_[(size_t)l - 1];
        I.xf = NX_POOL;
        I.s = g_[(size_t)l].mStart;
        I.list = g_[(size_t)l].mList;
        I.inv = g_[(size_t)l].invCnt;
        I.map = g_[(size_t)l - 1].c2c;
        I.srcRows = g_[(size_t)l - 1].N;
        Ly.in[0] = I;
        Ly.nIn = 1;
        Ly.Y = H[(size_t)l];
        Ly.gY = gH[(size_t)l];
        Ly.gIn[0] = gE[(size_t)l - 1];
        layers_.push_back(Ly);
        layers_.push_back(mp("enc" + std::to_string(std::min(l, 3)), l, H[(size_t)l], gH[(size_t)l], E[(size_t)l],
                             gE[(size_t)l]));
    }
    layers_.push_back(mp("mid" + std::to_string(std::min(L - 1, 3)), L - 1, E[(size_t)L - 1], gE[(size_t)L - 1],
                         D[(size_t)L - 1], gD[(size_t)L - 1]));
    for (int l = L - 2; l >= 0; l--) {
        NetLayer Ly;
        Ly.N = g_[(size_t)l].N;
        Ly.K = C_[(size_t)l + 1];
        Ly.Cout = C_[(size_t)l];
        Ly.wOff = group("up" + std::to_string(std::min(l, 3)), Ly.K, Ly.Cout);
        NetIn I;
        I.x = D[(size_t)l + 1];
        I.C = C_[(size_t)l + 1];
        I.xf = NX_UNPOOL;
        I.map = g_[(size_t)l].c2c;
        I.s = g_[(size_t)l + 1].mStart;
        I.list = g_[(size_t)l + 1].mList;
        I.srcRows = g_[(size_t)l + 1].N;
        Ly.in[0] = I;
        Ly.nIn = 1;
        Ly.add = E[(size_t)l];
        Ly.gAdd = gE[(size_t)l];
        Ly.Y = S[(size_t)l];
        Ly.gY = gS[(size_t)l];
        Ly.gIn[0] = gD[(size_t)l + 1];
        layers_.push_back(Ly);
        layers_.push_back(mp("dec" + std::to_string(std::min(l, 3)), l, S[(size_t)l], gS[(size_t)l], D[(size_t)l],
                             gD[(size_t)l]));
    }
    {  // output
        NetLayer Ly;
        Ly.N = N0_;
        Ly.K = C_[0];
        Ly.Cout = 1;
        Ly.relu = 0;
        Ly.wOff = group("out", C_[0], 1);
        Ly.in[0] = idIn(D[0], C_[0], N0_);
        Ly.nIn = 1;
        Ly.Y = out_;
        Ly.gY = gOut_;
        Ly.gIn[0] = gD[0];
        layers_.push_back(Ly);
    }
    nParams_ = total;
    params_ = devAlloc<float>(allocs_, nParams_);
    paramsLow_ = wBf16_ ? (void*)devAlloc<bfloat>(allocs_, nParams_) : (void*)params_;
    if (wBf16_) {
        packF_ = devAlloc<bfloat>(allocs_, nParams_);
        packB_ = devAlloc<bfloat>(allocs_, nParams_);
    }
    grad_ = devAlloc<float>(allocs_, nParams_);
    adamM_ = devAlloc<float>(allocs_, nParams_);
    adamV_ = devAlloc<float>(allocs_, nParams_);
    // training buffers: Z per layer, scratch for G and dZ, wgrad partials
    size_t maxG = 0, maxZ = 0, maxPart = 0;
    for (NetLayer& Ly : layers_) {
        Ly.Z = act((size_t)Ly.N * Ly.K);
        maxG = std::max(maxG, (size_t)Ly.N * Ly.Cout);
        maxZ = std::max(maxZ, (size_t)Ly.N * Ly.K);
        maxPart = std::max(maxPart, (size_t)wgradSplits(Ly) * ((size_t)Ly.K * Ly.Cout + Ly.Cout));
    }
    gpre_ = grd(maxG);
    dZ_ = grd(maxZ);
    wgPartial_ = grd(maxPart);
    Ay_ = grd((size_t)N0_);
    scal_ = devAlloc<double>(allocs_, 8);
    red_ = devAlloc<double>(allocs_, 3 * (size_t)blocksFor(N0_) + 8);
    counter_ = devAlloc<unsigned int>(allocs_, 4);
}

void LearnedNet::syncLowPrecision(cudaStream_t s) {
    if (!wBf16_) return;
    launchPDL(k_to_low<bfloat>, dim3(blocksFor(nParams_)), dim3(kThreads), 0, s, nParams_, params_, (bfloat*)paramsLow_);
    packWeights(s);
    NCK(cudaGetLastError());
}

// The weights in fragment order, after every change of them.
void LearnedNet::packWeights(cudaStream_t s) {
    PackArgs a;
    a.n = 0;
    for (const NetLayer& L : layers_) {
        if (!slabs(L)) continue;
        bool seen = false;
        for (int i = 0; i < a.n; i++) seen |= a.off[i] == (unsigned)L.wOff;
        if (seen) continue;
        if (a.n == kMaxGroups) throw std::runtime_error("too many weight groups");
        a.off[a.n] = (unsigned)L.wOff;
        a.K[a.n] = (short)L.K;
        a.Cout[a.n] = (short)L.Cout;
        a.n++;
    }
    if (a.n) launchPDL(k_pack, dim3(dim3(16, a.n)), dim3(kThreads), 0, s, a, (const bfloat*)paramsLow_, (bfloat*)packF_, (bfloat*)packB_);
}

// Predictions run on fragments from memory (874k cells: 0.8 ms of device time
// against 1.76 with the tiles). The preconditioner inside a solve and the
// training pass keep the tiles' rounding: a solve's FP64 iterates carry the
// difference of two forward passes (1e-6) to 8e-6 of the fields, and the
// gradient, a small difference of large sums, to 2.7e-5 (1.2e-5 to 1.6e-5 with
// the tiles, from the weight gradient's shorter sums). Their price: a gradient
// on 218k cells 1.6 -> 1.9 ms.
void LearnedNet::forward(const Ctl* ctl, int gated, bool keepZ, cudaStream_t s) {
    const bool tiles = ctl || keepZ;
    for (NetLayer L : layers_) {
        if (!keepZ) L.Z = nullptr;
        if (tiles && actBf16_) launchLayerFwd<bfloat, bfloat>(ctl, gated, L, paramsLow_, s);
        else if (tiles && wBf16_) launchLayerFwd<float, bfloat>(ctl, gated, L, paramsLow_, s);
        else if (actBf16_) launchLayerLow<bfloat>(ctl, gated, L, (const bfloat*)paramsLow_, (const bfloat*)packF_, s);
        else if (wBf16_) launchLayerLow<float>(ctl, gated, L, (const bfloat*)paramsLow_, (const bfloat*)packF_, s);
        else launchLayerFwd<float, float>(ctl, gated, L, paramsLow_, s);
    }
}

void LearnedNet::infer(const Ctl* ctl, int gated, const double* r, const double* AC, const double* AF,
                       const int32_t* nb, int W, float* e, cudaStream_t s) {
    const int nb0 = blocksFor(N0_);
    launchPDL(k_sigma<double>, dim3(nb0), dim3(kThreads), 0, s, ctl, gated, N0_, r, AC, red_, counter_, scal_);
    if (actBf16_)
        launchPDL(k_features<bfloat, double>, dim3(nb0), dim3(kThreads), 0, s, ctl, gated, N0_, r, AC, AF, nb, W, nullptr, scal_,
                                                             (bfloat*)feat_);
    else
        launchPDL(k_features<float, double>, dim3(nb0), dim3(kThreads), 0, s, ctl, gated, N0_, r, AC, AF, nb, W, nullptr, scal_,
                                                            (float*)feat_);
    forward(ctl, gated, false, s);
    if (actBf16_) launchPDL(k_scale_out<bfloat>, dim3(nb0), dim3(kThreads), 0, s, ctl, gated, N0_, (const bfloat*)out_, scal_, e);
    else launchPDL(k_scale_out<float>, dim3(nb0), dim3(kThreads), 0, s, ctl, gated, N0_, (const float*)out_, scal_, e);
}

void LearnedNet::backward(cudaStream_t s) {
    for (int i = (int)layers_.size() - 1; i >= 0; i--) {
        const NetLayer& L = layers_[(size_t)i];
        const bool needDz = L.gIn[0] != nullptr;
        const float* G = gpre_;
        const bool direct = wBf16_ && needDz && !slabs(L);  // the output layer: its input gradient in one pass
        if (!wBf16_) {
            launchLayerDz<float, float>(L, paramsLow_, gpre_, needDz ? dZ_ : nullptr, s);
        } else if (direct) {
            G = L.gY;
            launchPDL(k_adj_out, dim3(blocksFor((size_t)L.N * 4)), dim3(kThreads), 0, s, L, (const bfloat*)paramsLow_, L.gIn[0]);
        } else if (!needDz) {
            const size_t n4 = (size_t)L.N * L.Cout / 4;
            if (actBf16_) launchPDL(k_mask<bfloat>, dim3(blocksFor(n4)), dim3(kThreads), 0, s, n4, L.gY, (const bfloat*)L.Y, gpre_);
            else launchPDL(k_mask<float>, dim3(blocksFor(n4)), dim3(kThreads), 0, s, n4, L.gY, (const float*)L.Y, gpre_);
        } else if (actBf16_) {
            launchDzMma<bfloat>(L, (const bfloat*)packB_, gpre_, dZ_, s);
        } else {
            launchDzMma<float>(L, (const bfloat*)packB_, gpre_, dZ_, s);
        }
        // dW, db; a layer with one untransformed input has that as its Z
        const void* Z = wBf16_ && L.nIn == 1 && L.in[0].xf == NX_ID ? L.in[0].x : L.Z;
        const int splits = wgradSplits(L);
        const int rowsPerSplit = (L.N + splits - 1) / splits;
        const int tilesK = (L.K + 31) / 32, tilesO = (L.Cout + 31) / 32;
        const dim3 grid((unsigned)(tilesK * tilesO), (unsigned)splits);
        if (actBf16_)
            launchPDL(k_wgrad<bfloat>, dim3(grid), dim3(kThreads), 0, s, L.N, L.K, L.Cout, tilesO, rowsPerSplit, (const bfloat*)Z, G,
                                                      wgPartial_);
        else
            launchPDL(k_wgrad<float>, dim3(grid), dim3(kThreads), 0, s, L.N, L.K, L.Cout, tilesO, rowsPerSplit, (const float*)Z, G,
                                                     wgPartial_);
        const int entries = L.K * L.Cout + L.Cout;
        launchPDL(k_wgrad_reduce, dim3(blocksFor(entries, 32)), dim3(kThreads), 0, s, entries, splits, wgPartial_, grad_ + L.wOff);
        // adjoints of the inputs
        int off = 0;
        if (L.nIn == 2) {  // message passing: both inputs are the same tensor
            const NetIn& I = L.in[1];
            launchPDL(k_adj_mp, dim3(blocksFor((size_t)L.N * I.C / 4)), dim3(kThreads), 0, s, L.N, I.C, L.K, I.s, I.list, I.inv, dZ_,
                                                                         L.gIn[1]);
        }
        for (int q = 0; q < L.nIn && L.nIn == 1 && !direct; q++) {
            const NetIn& I = L.in[q];
            float* gX = L.gIn[q];
            if (gX) {
                const size_t n = (size_t)I.srcRows * I.C / 4;
                switch (I.xf) {
                    case NX_ID:
                        launchPDL(k_adj_id, dim3(blocksFor(n)), dim3(kThreads), 0, s, I.srcRows, I.C, off, L.K, dZ_, gX);
                        break;
                    case NX_POOL:
                        launchPDL(k_adj_pool, dim3(blocksFor(n)), dim3(kThreads), 0, s, I.srcRows, I.C, off, L.K, I.map, I.inv, dZ_, gX);
                        break;
                    default:
                        launchPDL(k_adj_unpool, dim3(blocksFor(n)), dim3(kThreads), 0, s, I.srcRows, I.C, off, L.K, I.s, I.list, dZ_, gX);
                        break;
                }
            }
            off += I.C;
        }
        if (L.gAdd) {
            const size_t n = (size_t)L.N * L.Cout / 4;
            launchPDL(k_adj_id, dim3(blocksFor(n)), dim3(kThreads), 0, s, L.N, L.Cout, 0, L.Cout, gpre_, L.gAdd);
        }
    }
    NCK(cudaGetLastError());
}

void LearnedNet::lossAndGrad(const Sample& smp, float* lossOut, cudaStream_t s) {
    const int nb0 = blocksFor(N0_);
    launchPDL(k_sigma<float>, dim3(nb0), dim3(kThreads), 0, s, nullptr, 0, N0_, smp.b, smp.AC, red_, counter_, scal_);
    if (actBf16_)
        launchPDL(k_features<bfloat, float>, dim3(nb0), dim3(kThreads), 0, s, nullptr, 0, N0_, smp.b, smp.AC, nullptr, nullptr, 0,
                                                           smp.deficit, scal_, (bfloat*)feat_);
    else
        launchPDL(k_features<float, float>, dim3(nb0), dim3(kThreads), 0, s, nullptr, 0, N0_, smp.b, smp.AC, nullptr, nullptr, 0,
                                                          smp.deficit, scal_, (float*)feat_);
    forward(nullptr, 0, true, s);
    if (actBf16_)
        launchPDL(k_loss_spmv<bfloat>, dim3(nb0), dim3(kThreads), 0, s, N0_, W0_, nb0_, smp.AF, smp.AC, (const bfloat*)out_, smp.b,
                                                     smp.target, Ay_, red_, counter_, scal_);
    else
        launchPDL(k_loss_spmv<float>, dim3(nb0), dim3(kThreads), 0, s, N0_, W0_, nb0_, smp.AF, smp.AC, (const float*)out_, smp.b,
                                                    smp.target, Ay_, red_, counter_, scal_);
    launchPDL(k_loss_grad, dim3(nb0), dim3(kThreads), 0, s, N0_, smp.b, Ay_, scal_, gOut_, lossOut);
    // zero every activation gradient except the output's, and the parameter gradient
    NCK(cudaMemsetAsync(gActs_, 0, gradActs_ * sizeof(float), s));
    NCK(cudaMemsetAsync(grad_, 0, nParams_ * sizeof(float), s));
    backward(s);
}

void LearnedNet::predict(const float* r, const float* AC, const float* deficit, float* out, cudaStream_t s) {
    const int nb0 = blocksFor(N0_);
    launchPDL(k_sigma<float>, dim3(nb0), dim3(kThreads), 0, s, nullptr, 0, N0_, r, AC, red_, counter_, scal_);
    if (actBf16_) {
        launchPDL(k_features<bfloat, float>, dim3(nb0), dim3(kThreads), 0, s, nullptr, 0, N0_, r, AC, nullptr, nullptr, 0, deficit, scal_,
                                                           (bfloat*)feat_);
        forward(nullptr, 0, false, s);
        launchPDL(k_scale_out<bfloat>, dim3(nb0), dim3(kThreads), 0, s, nullptr, 0, N0_, (const bfloat*)out_, scal_, out);
    } else {
        launchPDL(k_features<float, float>, dim3(nb0), dim3(kThreads), 0, s, nullptr, 0, N0_, r, AC, nullptr, nullptr, 0, deficit, scal_,
                                                          (float*)feat_);
        forward(nullptr, 0, false, s);
        launchPDL(k_scale_out<float>, dim3(nb0), dim3(kThreads), 0, s, nullptr, 0, N0_, (const float*)out_, scal_, out);
    }
    NCK(cudaGetLastError());
}

void LearnedNet::trainStep(const Sample& smp, float lr, int t, float* lossOut, cudaStream_t s) {
    lossAndGrad(smp, lossOut, s);
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)t), c2 = 1.f - std::pow(b2, (float)t);
    const dim3 grid(blocksFor(nParams_)), block(kThreads);
    if (wBf16_) {
        launchPDL(k_adam<bfloat>, grid, block, 0, s, nParams_, params_, grad_, adamM_, adamV_, (bfloat*)paramsLow_, lr,
                  b1, b2, 1e-8f, c1, c2);
        packWeights(s);
    } else {
        launchPDL(k_adam<float>, grid, block, 0, s, nParams_, params_, grad_, adamM_, adamV_, params_, lr, b1, b2,
                  1e-8f, c1, c2);
    }
    NCK(cudaGetLastError());
}

}  // namespace axisim
