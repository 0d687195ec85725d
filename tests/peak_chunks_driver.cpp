// Host build of the chunked peak finder (csrc/kernels/ucb_bif.cuh) against the finder that
// takes one sample at a time; prints the number of series compared.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#define __device__
#define __global__
#define __forceinline__ inline
#define __noinline__
#define UCB_BIF_NO_KERNELS 1
#define UCB_WV 0
#define UCB_NX 1
#define UCB_NV 1
#define UCB_STEP_LOOP
#define UCB_STR_(x) #x
#define UCB_PRAGMA_(x)
#ifndef NUMB
#define NUMB double
#endif
typedef NUMB numb;
constexpr numb pi = (numb)3.14159265358979, euler = (numb)2.718281828;
static inline int __ffs(int v) { return __builtin_ffs(v); }
using std::fabs;
namespace ucbdev {
constexpr int kCheckInterval = 100, kMaxAmountOfPeaks = 2500;
constexpr double kEpsPeakDelta = 1e-14, kPeakThreshold = -1e25;
inline bool diverged(const numb*, numb) { return false; }
inline int fixed_point_flag(const numb*, const numb*) { return 1; }
template <bool Check, class S>
int run_single(const S&, numb*, const numb*, numb, int, numb) {
    return 1;
}
}  // namespace ucbdev
#include "ucb_bif.cuh"

struct List {
    std::vector<double>* out;
    void put(int k, numb value, numb dt) const {
        out->push_back(k);
        out->push_back((double)value);
        out->push_back((double)dt);
    }
};

// The reference's loop (cudaLibrary.cu:1503-1633) over the whole series.
static void whole(const std::vector<numb>& d, std::vector<double>& out) {
    const long long n = (long long)d.size();
    int found = 0;
    numb prev = 0;
    for (long long i = 2; i < n - 2; ++i) {
        if (!(d[i] - d[i - 1] > (numb)1e-14 && d[i] > (numb)-1e25 && d[i] >= d[i + 1])) continue;
        for (long long j = i; j < n - 2; ++j) {
            if (d[j] < d[j + 1]) {
                i = j + 1;
                break;
            }
            if (d[j] - d[j + 1] > (numb)1e-14) {
                const numb denom = d[j - 1] - (numb)2.0 * d[j] + d[j + 1];
                numb delta = 0;
                if (std::fabs(denom) > 1e-12) delta = 0.5 * (d[j - 1] - d[j + 1]) / denom;
                const numb value = d[j] - 0.25 * (d[j - 1] - d[j + 1]) * delta;
                const numb t = (numb)(j - 1) + delta;
                if (found > 0) {
                    out.push_back(found - 1);
                    out.push_back((double)value);
                    out.push_back((double)(t - prev));
                }
                prev = t;
                ++found;
                i = j + 1;
                break;
            }
            if (j == n - 3) i = n;  // a plateau to the end of the series
        }
    }
}

static void chunked(const std::vector<numb>& d, std::vector<double>& out) {
    using namespace ucbdev;
    const long long n = (long long)d.size();
    PeakScan s;
    s.init();
    const List sink{&out};
    std::vector<numb> w(kScanChunk + 2, (numb)0);
    for (long long q0 = 0; q0 < n; q0 += kScanChunk) {
        const int m = (int)std::min<long long>(n - q0, kScanChunk);
        for (int c = 0; c < m; ++c) w[c + 2] = d[q0 + c];
        scan_chunk(s, w.data(), q0, m, n, sink);
        w[0] = w[m];
        w[1] = w[m + 1];
    }
}

int main() {
    std::mt19937_64 rng(11);
    std::uniform_real_distribution<double> u(0, 1);
    const numb inf = std::numeric_limits<numb>::infinity();
    const numb special[] = {inf, -inf, (numb)std::nan(""), std::numeric_limits<numb>::max(), (numb)-2e25, (numb)0};
    long long done = 0;
    for (int n = 1; n <= 130; ++n)
        for (int kind = 0; kind < 8; ++kind)
            for (int rep = 0; rep < 20; ++rep) {
                std::vector<numb> d(n);
                const double f = 0.05 + 1.5 * u(rng), ph = 6.28 * u(rng);
                double walk = 0;
                for (int i = 0; i < n; ++i) {
                    double v = std::sin(f * i + ph);
                    if (kind == 1) v = (int)(u(rng) * 3);              // plateaus of every length
                    if (kind == 2) v = std::round(4 * v);              // flat tops
                    if (kind == 3) v = u(rng) - 0.5;                   // peaks as dense as they come
                    if (kind == 4) v = 1.0 + 1e-15 * (int)(u(rng) * 40);  // steps about the threshold
                    if (kind == 5) v = i % 2;
                    if (kind == 6) v = (walk += (int)(u(rng) * 3) - 1);
                    d[i] = (numb)v;
                    if (kind == 7 && u(rng) < 0.2) d[i] = special[(int)(u(rng) * 6)];
                }
                std::vector<double> a, b;
                whole(d, a);
                chunked(d, b);
                if (a.size() != b.size() || (a.size() && std::memcmp(a.data(), b.data(), a.size() * 8) != 0)) {
                    std::printf("differs: n=%d kind=%d rep=%d: %zu and %zu values\n", n, kind, rep, a.size(), b.size());
                    return 1;
                }
                ++done;
            }
    std::printf("%lld\n", done);
    return 0;
}
