"""The quotient by a precomputed reciprocal (csrc/exact_div.cuh) against the
division operator, bit for bit. The header is compiled for the host, where its
operations (IEEE multiplication, FMA and division) round as on the device:
random mantissas and the extreme ones at, and on both sides of, each exponent
limit of dividend and divisor, zeros of both signs, subnormals, infinities, NaN.
"""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>
#define __device__
#define __forceinline__ inline
using std::fma;
static inline int __double2hiint(double x) { uint64_t u; std::memcpy(&u, &x, 8); return (int)(u >> 32); }
static inline int __float_as_int(float x) { int u; std::memcpy(&u, &x, 4); return u; }
#include "exact_div.cuh"

template <class T, class U>
static int check(const std::vector<int>& ea, const std::vector<int>& eb, int mant, int bias, int each) {
    std::mt19937_64 rng(1);
    const U full = ((U)1 << mant) - 1;
    auto make = [&](int e, U m, bool neg) {
        const U u = (U)neg << (sizeof(U) * 8 - 1) | (U)(e + bias) << mant | (m & full);
        T x; std::memcpy(&x, &u, sizeof x); return x;
    };
    const U special[] = {0, 1, 2, full, full - 1, full >> 1, (full >> 1) + 1, full ^ 2};
    int bad = 0;
    long tried = 0;
    auto one = [&](T a, T b) {
        const volatile T va = a, vb = b;  // no folding
        const T want = va / vb, got = axisim::ExactDiv<T>(b)(a);
        tried++;
        if (std::isnan(want) && std::isnan(got)) return;
        if (std::memcmp(&want, &got, sizeof(T)) != 0 && bad++ < 5) std::printf("%a / %a: %a, not %a\n", (double)a, (double)b, (double)got, (double)want);
    };
    std::vector<T> as, bs;
    using L = std::numeric_limits<T>;
    for (T v : {T(0), T(-0.0), L::denorm_min(), L::min(), L::max(), L::infinity(), -L::infinity(), L::quiet_NaN()}) {
        as.push_back(v);
        bs.push_back(v);
    }
    for (int e : ea) for (U m : special) as.push_back(make(e, m, m & 1));
    for (int e : eb) for (U m : special) bs.push_back(make(e, m, m & 2));
    for (T a : as) for (T b : bs) one(a, b);
    for (int e : ea)
        for (int f : eb)
            for (int k = 0; k < each; k++) {
                const U s = rng();
                // every fourth pair with one mantissa at an end of its range
                const U ma = k % 8 == 0 ? special[s % 8] : (U)rng(), mb = k % 8 == 4 ? special[s % 8] : (U)rng();
                one(make(e, ma, s >> 1 & 1), make(f, mb, s >> 2 & 1));
            }
    std::printf("%ld quotients, %d differ\n", tried, bad);
    return bad;
}

int main() {
    const std::vector<int> a64 = {-1022, -1021, -902, -901, -900, -899, -1, 0, 1, 53, 799, 800, 801, 802, 1023};
    const std::vector<int> b64 = {-1022, -102, -101, -100, -99, -1, 0, 1, 99, 100, 101, 102, 1023};
    const std::vector<int> a32 = {-126, -125, -92, -91, -90, -89, -1, 0, 1, 24, 59, 60, 61, 62, 127};
    const std::vector<int> b32 = {-126, -62, -61, -60, -59, -1, 0, 1, 29, 30, 31, 32, 127};
    return (check<double, uint64_t>(a64, b64, 52, 1023, 4000) + check<float, uint32_t>(a32, b32, 23, 127, 4000)) != 0;
}
'''


def test_quotients_equal_the_division_operator(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text("")
    src = tmp_path / "q.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "q"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(tmp_path), "-I",
                        os.path.join(ROOT, "axisim-software_b200", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
