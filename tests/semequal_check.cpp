// Host check of sem_quick_equal (csrc/cpd_model.h): wherever it answers, it answers as sem_test
// on the sums that h equal hits make, q1 = h q and q2 = h q^2; and it leaves few states open.
// prints: cases <n> disagree <m> open <states left to sem_test>
#include <cmath>
#include <cstdio>
#include <random>

#include "cpd_model.h"

using namespace cpd;

int main()
{
    std::mt19937_64 g(12);
    long n = 0, bad = 0, open = 0;
    const auto check = [&](uint64_t N, uint64_t h, uint64_t q, uint32_t delta, bool count) {
        if (h > N || N < 1 || N > (1u << 22) || q > (1u << 20)) return;
        const int v = sem_quick_equal((uint32_t)N, (uint32_t)h, sem_equal((uint32_t)q, delta));
        n++;
        if (v < 0) open += count;
        else if (v != sem_test(N, h, h * q, h * q * q, delta)) bad++;
    };
    for (int i = 0; i < 400000; i++) {
        const uint64_t N = 1 + (uint64_t)std::exp2(std::uniform_real_distribution<double>(0, 22)(g)) % (1u << 22);
        const uint64_t q = i % 7 == 0 ? g() % 64 : i % 11 == 0 ? (1u << 20) - g() % 3 : g() % ((1u << 20) + 1);
        check(N, g() % (N + 1), q, i & 1 ? 2u : 0u, true);
        // at the test's boundary: 40000 q^2 h (N - h) = N^2 (N - 1) 2^40
        const double c = (double)N * N * (N - 1.0) * 0x1p40 / (40000.0 * ((double)q * q + 1e-9));
        const double disc = (double)N * N - 4.0 * c;
        if (disc >= 0) {
            const double r = 0.5 * ((double)N - std::sqrt(disc));
            for (int k = -2; k <= 2; k++) {
                check(N, (uint64_t)std::max(0.0, r + k), q, 0u, false);
                check(N, (uint64_t)std::max(0.0, (double)N - r + k), q, 2u, false);
            }
        }
    }
    std::printf("cases %ld disagree %ld open %ld\n", n, bad, open);
    return 0;
}
