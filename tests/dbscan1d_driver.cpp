// Host build of csrc/kernels/ucb_dbscan1d.cuh (lanes one after the other) against the scan
// form of the same dbscan: argv[1] = seed; prints the number of cases compared.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#define __device__
#define __forceinline__ inline
#ifndef NUMB
#define NUMB double
#endif
typedef NUMB numb;
template <class To, class From>
static To cast(From v) {
    To t;
    std::memcpy(&t, &v, sizeof t);
    return t;
}
static inline int __float_as_int(float v) { return cast<int>(v); }
static inline float __int_as_float(int v) { return cast<float>(v); }
static inline long long __double_as_longlong(double v) { return cast<long long>(v); }
static inline double __longlong_as_double(long long v) { return cast<double>(v); }
static inline int __ffs(int v) { return __builtin_ffs(v); }
static inline int __ffsll(long long v) { return __builtin_ffsll(v); }
#include "ucb_dbscan1d.cuh"

static int scans(const std::vector<numb>& p, numb eps) {
    const int P = (int)p.size();
    if (P < 2) return P;
    std::vector<int> lab(P, 0), stk(P, 0);
    int cluster = 0, nn = 0;
    for (int i = 0; i < P; i++) {
        if (nn >= 1) {
            const int v = stk[nn - 1];
            stk[nn - 1] = 0;
            i = v;
            nn = nn - 1;
        } else if (lab[i] == 0) {
            lab[i] = ++cluster;
        } else {
            continue;
        }
        for (int k = 0; k < P - 1; ++k)
            if (i != k && lab[k] == 0 && std::fabs(p[k] - p[i]) < eps) {
                lab[k] = cluster;
                stk[k] = k;
                ++nn;
            }
    }
    return cluster - 1;
}

static int replay(const std::vector<numb>& p, numb eps) {
    const int P = (int)p.size();
    std::vector<ucbdev::PeakKey> ka(P), kb(P);
    std::vector<unsigned short> ia(P), ib(P), order(P);
    std::vector<unsigned int> range(P), bits(3 * ((P + 31) / 32) * 2 + 1);
    if (P >= 2) {
        for (int e = 0; e < P; ++e) {
            ka[e] = ucbdev::peak_key(p[e]);
            ia[e] = (unsigned short)e;
        }
        for (int run = 1; run < P; run *= 2) {
            for (int lane = 0; lane < 32; ++lane)
                ucbdev::merge_level(ka.data(), ia.data(), kb.data(), ib.data(), P, run, lane);
            ka.swap(kb);
            ia.swap(ib);
        }
        for (int lane = 0; lane < 32; ++lane)
            ucbdev::peak_ranges(ka.data(), ia.data(), P, eps, range.data(), order.data(), lane);
    }
    return ucbdev::dbscan_replay(P, range.data(), order.data(), bits.data(), 2);
}

int main(int, char** argv) {
    std::mt19937_64 rng(std::strtoull(argv[1], nullptr, 10));
    std::uniform_real_distribution<double> u(0, 1);
    const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
    const double special[] = {0.0, -0.0, inf, -inf, nan, -nan, 1e300, -1e300, 5e-324, std::numeric_limits<numb>::max()};
    const int sizes[] = {0, 1, 2, 3, 31, 32, 33, 64, 65, 127, 128, 129, 600, 2047, 2048, 2049, 2499, 2500};
    long long done = 0;
    for (int t = 0; t < 600; ++t) {
        const int P = t % 3 ? (int)(u(rng) * 200) : sizes[(t / 3) % 18];
        const int kind = (int)(u(rng) * 6);
        const int levels = 1 + (int)(u(rng) * 12);
        std::vector<numb> p(P);
        for (int i = 0; i < P; ++i) {
            double v = 40 * u(rng) - 20;                                  // chaotic: spread
            if (kind == 1) v = (int)(levels * u(rng));                    // periodic: exact repeats
            if (kind == 2) v = (int)(levels * u(rng)) + 1e-3 * u(rng);    // periodic with noise
            if (kind == 3) v = (i % levels) * 0.1;                        // at eps exactly, in order
            if (kind == 4) v = 0.05 * i;                                  // a chain
            if (kind == 5 && u(rng) < 0.3) v = special[(int)(u(rng) * 10)];
            p[i] = (numb)v;
        }
        for (double eps : {0.1, 0.5, 0.05, 1e-3, 100.0, 1e-60, inf}) {
            const int a = scans(p, (numb)eps), b = replay(p, (numb)eps);
            if (a != b) {
                std::printf("differs: P=%d kind=%d eps=%g scans=%d replay=%d\n", P, kind, eps, a, b);
                return 1;
            }
            ++done;
        }
    }
    std::printf("%lld\n", done);
    return 0;
}
