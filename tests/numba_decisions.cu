// Host check of the numba engine's decisions after the determinant (lyem_device.cuh): the exact FP32 sign and U > 1
// checks followed by numba_tail, which decides without FP64 where the outcome is certain, must give that engine's
// FP64 decision (F = 1 / A, U, V, t; lyceanem/raycasting/rayfunctions.py:55-100) on every input.  Compiled for the
// host by tests/test_numba_decisions.py with -ffp-contract=off.
//
//   numba_decisions <n_cases> <seed>   prints "cases mismatches hits"
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "lyem_device.cuh"

int main(int argc, char** argv) {
    const long long n = atoll(argv[1]);
    std::mt19937_64 g((uint64_t)atoll(argv[2]));
    auto uni = [&] { return (double)(g() >> 11) * 0x1p-53; };
    auto pick = [&](int k) { return (int)(g() % (uint64_t)k); };
    auto near = [&](double x) {  // x rounded, a few ulps away, or off by a relative 2^-14 .. 2^-28
        float y = (float)x;
        const int kind = pick(3);
        if (kind == 1)
            for (int i = pick(5); i > 0; --i) y = std::nextafter(y, pick(2) ? INFINITY : -INFINITY);
        if (kind == 2) y = (float)(x * (1.0 + std::ldexp(uni() - 0.5, -(14 + pick(14)))));
        return y;
    };
    long long mismatches = 0, hits = 0;
    for (long long i = 0; i < n; ++i) {
        const float eps = pick(8) == 0 ? 0.f : pick(2) ? 1e-7f : 1e-6f;
        const double mag = pick(6) == 0 ? std::ldexp(uni() + 0.5, pick(250) - 140) : std::ldexp(uni() + 0.5, pick(40) - 20);
        const float A = pick(2) ? near(mag) : -near(mag);
        const float len = pick(6) == 0 ? near(2.0 * eps) : (float)std::ldexp(uni() + 0.5, pick(40) - 20);
        const double L = (double)len - 2.0 * eps;
        const double ru = pick(3) ? uni() : pick(2) ? 0.0 : 1.0;
        const double rv = pick(3) == 0 ? uni() : (1.0 - ru) * (pick(2) ? 1.0 : 1.0 + std::ldexp(uni() - 0.5, -(14 + pick(40))));
        const double ends[5] = {2.0 * eps, L, 4.0 * eps, -uni() * L, uni() * L * 1.2};
        const float u = near(ru * A), v = near(rv * A), w = pick(20) ? near(ends[pick(5)] * A) : 0.f;
        bool ours = false, ref = false;
        if (!(lyem::ratio_negative(u, A) || lyem::ratio_above_one(u, A) || lyem::ratio_negative(v, A)))
            ours = lyem::numba_tail(A, u, v, w, len, eps);
        const double F = 1.0 / (double)A, U = F * (double)u, V = F * (double)v, t = F * (double)w;
        if (!(U < 0.0 || U > 1.0 || V < 0.0 || U + V > 1.0))
            ref = t > 2.0 * (double)eps && t < (double)len - 2.0 * (double)eps;
        hits += ref;
        if (ours != ref && ++mismatches < 10)
            std::printf("A=%a u=%a v=%a w=%a len=%a eps=%a ours=%d ref=%d\n", A, u, v, w, len, eps, ours, ref);
    }
    std::printf("%lld %lld %lld\n", n, mismatches, hits);
    return mismatches ? 1 : 0;
}
