// Operands that are hardest for csrc/ct_fp64.cuh: quotients and square roots next to the middle of two
// doubles, all-ones mantissas, the limits of the fast paths' exponents, and random ones.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <vector>

namespace fp64_cases {

struct Rng {
    uint64_t s = 88172645463325252ull;
    uint64_t operator()() {
        s ^= s << 13;
        s ^= s >> 7;
        s ^= s << 17;
        return s * 2685821657736338717ull;
    }
};
constexpr uint64_t ONE = 1ull << 52;
inline double make(uint64_t mantissa, int exponent, bool negative = false) {
    const uint64_t b = ((uint64_t)(1023 + exponent) << 52) | (mantissa & (ONE - 1)) | ((uint64_t)negative << 63);
    double d;
    memcpy(&d, &b, 8);
    return d;
}

// n / d with 2^(s + 1) N = j modulo D: the quotient is j / (2 D) units from the middle of two doubles
inline void divisions(long count, std::vector<double>& n, std::vector<double>& d) {
    Rng r;
    auto put = [&](uint64_t N, uint64_t D, int en = 0, int ed = 0) {
        n.push_back(make(N, en, r() & 1));
        d.push_back(make(D, ed, r() & 1));
    };
    for (long i = 0; i < count; ++i) {
        uint64_t D = ONE | (r() >> 12);
        if (i % 4 == 1) D = 2 * ONE - 1 - 2 * (r() % 100000);
        if (i % 4 == 2) D = 2 * ONE - 1 - 2 * (r() >> (12 + r() % 40));
        if (i % 4 == 3) D = ONE + 1 + 2 * (r() % 100000);
        D |= 1;
        const uint64_t half = (D + 1) / 2;   // 1/2 modulo D
        unsigned __int128 p = 1;
        for (int k = 0; k < 53; ++k) p = p * half % D;
        for (int s = 0; s < 2; ++s, p = p * half % D)
            for (int j = -3; j <= 3; ++j) {
                if (j == 0) continue;
                uint64_t N = (uint64_t)(j > 0 ? p * (unsigned)j % D : D - p * (unsigned)-j % D);
                while (N < ONE) N += D;
                for (; N < 2 * ONE; N += D) put(N, D);
            }
        put(r() >> 12, r() >> 12);
        put(2 * ONE - 1 - r() % 2000, 2 * ONE - 1 - r() % 2000);
        put(r() >> 12, r() >> 12, (int)(r() % 2040) - 1020, (int)(r() % 2040) - 1020);
        put(r() >> 12, r() >> 12, (int)(r() % 5) - 625, (int)(r() % 5) + 623);   // the middle's limits
    }
    const double special[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 4.9e-324, 2.2250738585072014e-308, 1.7976931348623157e308};
    for (double a : special)
        for (double b : special) {
            n.push_back(a);
            d.push_back(b);
        }
}

// sqrt(x) next to the middle of m and m + 1: x = m (m + 1) + j, a multiple of 2^52 or 2^53
inline void roots(long count, std::vector<double>& x) {
    Rng r;
    for (int mod = 52; mod <= 53; ++mod)
        for (long long j = -12; j <= 12; j += 2) {
            // (2 m + 1)^2 = 1 - 4 j modulo 2^(mod + 2), its square roots bit by bit
            const unsigned __int128 c = (unsigned __int128)(__int128)(1 - 4 * j);
            std::vector<unsigned __int128> q = {1, 3, 5, 7};
            for (int b = 3; b < mod + 2; ++b) {
                std::vector<unsigned __int128> next;
                for (auto v : q)
                    for (int w = 0; w < 4; ++w) {
                        const unsigned __int128 u = (v + ((unsigned __int128)(w & 1) << (b - 1)) + ((unsigned __int128)(w >> 1) << b)) &
                                                    (((unsigned __int128)1 << (b + 1)) - 1);
                        bool seen = ((u * u - c) & (((unsigned __int128)1 << (b + 1)) - 1)) != 0;
                        for (auto o : next) seen |= o == u;
                        if (!seen) next.push_back(u);
                    }
                q = next;
            }
            for (auto v : q)
                for (unsigned __int128 m = (v - 1) / 2 & (((unsigned __int128)1 << mod) - 1); m < 2 * ONE; m += (unsigned __int128)1 << mod) {
                    if (m < ONE) continue;
                    const unsigned __int128 X = m * m + m + (unsigned __int128)(__int128)j;
                    const uint64_t M = (uint64_t)(X >> mod);
                    if ((X & (((unsigned __int128)1 << mod) - 1)) || M < ONE || M >= 2 * ONE) continue;
                    for (int e = -4; e <= 4; ++e) x.push_back(make(M, e));
                }
        }
    for (long i = 0; i < count; ++i) {
        x.push_back(make(r() >> 12, (int)(r() % 2040) - 1020));
        x.push_back(make(2 * ONE - 1 - r() % 64, (int)(r() % 2040) - 1020));
        x.push_back(make(ONE + r() % 64, (int)(r() % 2040) - 1020));
        x.push_back(make(r() >> 12, (int)(r() % 4) - 625));
    }
    for (double v : {0.0, -0.0, 1.0, -1.0, (double)INFINITY, (double)-INFINITY, (double)NAN, 4.9e-324}) x.push_back(v);
}

inline bool same(double a, double b) {
    uint64_t u, v;
    memcpy(&u, &a, 8);
    memcpy(&v, &b, 8);
    return u == v || (a != a && b != b);
}

}  // namespace fp64_cases
