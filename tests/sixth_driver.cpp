// Host build of csrc/kernels/ucb_exact.cuh: ucb_sixth(x) against x / 6, bit for bit wherever it
// reports its argument in range, which it does for zero and for every exponent allowed.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>

#define __device__
#define __forceinline__ inline
static inline int __float_as_int(float v) {
    int b;
    std::memcpy(&b, &v, 4);
    return b;
}
static inline int __double2hiint(double v) {
    long long b;
    std::memcpy(&b, &v, 8);
    return (int)(b >> 32);
}
static inline int __double2loint(double v) {
    long long b;
    std::memcpy(&b, &v, 8);
    return (int)b;
}
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
#include "ucb_exact.cuh"

template <class T, class I>
static bool same(I bits) {
    T x, q, p;
    std::memcpy(&x, &bits, sizeof x);
    unsigned int range = 0;
    q = ucb_sixth(x, range);
    p = x / (T)6;
    const bool allowed = x == 0 || (std::fabs(x) >= std::ldexp((T)1, sizeof(T) == 4 ? -63 : -959) && x - x == 0);
    if ((range <= kSixthRange) != allowed) return false;
    return !allowed || std::memcmp(&q, &p, sizeof q) == 0;
}

int main() {
#ifdef UCB_NUMB_F32
    // every positive float (and zero, infinity, NaN), a sample of the negative ones
    for (unsigned long long b = 0; b < (1ULL << 32); b += b >> 31 ? 16381 : 1)
        if (!same<float>((unsigned int)b)) return std::printf("differs: %08llx\n", b), 1;
#else
    std::mt19937_64 rng(3);
    // every exponent with random, all-zero, all-one and sparse mantissas, both signs; and
    // the neighbours of six times the values half way between two doubles
    for (unsigned long long e = 0; e < 2048; ++e)
        for (int t = 0; t < 60000; ++t) {
            const unsigned long long r = rng() & 0xFFFFFFFFFFFFFULL, k = rng() % 53;
            unsigned long long m = r;
            if (t % 4 == 1) m = (r >> k) << k & 0xFFFFFFFFFFFFFULL;
            if (t % 4 == 2) m = (~0ULL >> 12) - (r >> (k < 52 ? k : 51));
            if (t % 4 == 3) {
                const double q = std::ldexp(1.0 + (double)r * 0x1p-52, 0);
                const double x = 6.0 * q + (double)((long long)(rng() % 9) - 4) * 0x1p-51;
                std::memcpy(&m, &x, 8);
                m &= 0xFFFFFFFFFFFFFULL;
            }
            const unsigned long long b = (rng() & 1) << 63 | e << 52 | m;
            if (!same<double>(b)) return std::printf("differs: %016llx\n", b), 1;
        }
#endif
    std::printf("same\n");
    return 0;
}
