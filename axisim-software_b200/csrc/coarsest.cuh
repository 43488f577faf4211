// coarsest.cuh -- weighted-Jacobi sweeps of a small system, one row per thread.
//
// A coarsest level has a few dozen rows, so its (typically 30) sweeps are one
// dependent chain, and a sweep's latency is all that counts: the coefficients,
// the neighbours' addresses and the row's own value stay in registers, the
// iterate alternates between two shared-memory buffers, and the quotient by the
// diagonal comes from its reciprocal (exact_div.cuh). A sweep is then one
// round of shared-memory reads, the ordered sum and the quotient: 280 (FP32)
// to 350 (FP64) cycles, against 630 to 920 with the buffers' pointers in local
// memory, a test per slot and the division operator.
#pragma once

#include <cstdint>

#include "exact_div.cuh"

namespace axisim {

// Row arithmetic of jacobiRow (multigrid.cu:447-484). sm: the CTA's shared
// memory; from, to: byte offsets of the two iterates (the first one is read by
// the first sweep); o: the row's offset in them; adr: the slots' values in
// `from`. An unused slot has the coefficient +0 and reads a cell that holds
// -0.0 in both buffers, so its product leaves the sum as it is. Threads that
// are not live repeat a row and store nothing. sync: barrier of the rows' threads.
template <class T, class Sync>
__device__ __forceinline__ void coarsestSweeps(unsigned char* sm, uint32_t from, uint32_t to, uint32_t o,
                                               const T (&c)[8], const uint32_t (&adr)[8], T ac, T bn, bool live, T w,
                                               int sweeps, Sync sync) {
    auto at = [&](uint32_t k) -> T& { return *reinterpret_cast<T*>(sm + k); };
    T xn = at(from + o);
    const bool empty = fabs(ac) < (sizeof(T) == 8 ? T(1.0e-30) : T(1.0e-30f));
    const ExactDiv<T> byAc(empty ? T(1) : ac);
    const uint32_t flip = to - from;
    uint32_t d = 0;
    for (int it = 0; it < sweeps; it++) {
        T g[8];
#pragma unroll
        for (int j = 0; j < 8; j++) g[j] = at(adr[j] + d);
        T Ax = ac * xn;
#pragma unroll
        for (int j = 0; j < 8; j++) Ax += c[j] * g[j];
        xn = empty ? xn : xn + byAc(w * (bn - Ax));
        d = flip - d;
        if (live) at(from + o + d) = xn;
        sync();
    }
}

}  // namespace axisim
