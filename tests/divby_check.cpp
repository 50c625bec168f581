// Host check of x::div_by (csrc/cpd_model.h): for whole divisors below 2^17 it is the rounded
// quotient, bit for bit, also where the first estimate is an ulp off.
// prints: cases <n> wrong <m> far <first estimates an ulp or more off the rounded quotient>
#include <cmath>
#include <cstdio>
#include <random>

#include "cpd_model.h"

using namespace cpd;

int main()
{
    std::mt19937_64 g(5);
    long n = 0, wrong = 0, far = 0;
    const auto check = [&](double a, uint32_t b) {
        const double d = (double)b, r = 1.0 / d, q = a / d;
        n++;
        far += std::fabs(a * r - q) >= std::nextafter(std::fabs(q), INFINITY) - std::fabs(q) && q != 0.0;
        wrong += x::div_by(a, d, r) != q;
    };
    const auto significand = [&]() { return 1.0 + (double)(g() >> 12) * 0x1p-52; };
    for (uint32_t b = 1; b < (1u << 17); b++) {
        check(0.0, b);
        for (int i = 0; i < 60; i++) {
            // the range of sums of counts and transmittances: 2^-40 to 2^40, both signs
            const double a = std::ldexp(significand(), (int)(g() % 81) - 40);
            check(i & 1 ? -a : a, b);
            // beside a tie between two quotients
            const double q = significand(), half = std::ldexp(1.0, -53);
            const double t = std::fma(q, (double)b, half * (double)b);
            check(t, b);
            check(std::nextafter(t, 0.0), b);
            check(std::nextafter(t, INFINITY), b);
        }
    }
    std::printf("cases %ld wrong %ld far %ld\n", n, wrong, far);
    return 0;
}
