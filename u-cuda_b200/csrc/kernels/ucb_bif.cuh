// ucb_bif.cuh — bifurcation diagrams with fused peak capture (NVRTC header).
//
// One thread per sweep point. The reference (run_bif1d, parametric_engine.cpp:1940-2084)
// writes the whole recorded series of every point to HBM (calculateDiscreteModelCUDA,
// cudaLibrary.cu:944-1077), re-reads it in a second kernel (peakFinderCUDA, :1641-1674)
// and copies points x record_steps values back. Here the recorded value of every step
// is consumed as it is produced by a streaming form of peakFinder (:1503-1633): a
// three-sample window plus the scan state of its outer/inner loops reproduces the same
// peaks (parabolic interpolation, plateau handling, skip of the sample after a peak,
// first peak dropped, intervals = (t_{k+1} - t_k) * step, count capped at 2500), so only
// the first max_out peaks and intervals per point ever reach memory.
#pragma once

struct UcbBifParams {
    int n_pts;                 // sweep points
    int pre_scaller;
    int writable_var;          // -1: x0 + pi x1 + e x2 combination
    int max_out;               // peaks stored per point
    long long skip;            // (int)(transient / h), host double arithmetic
    long long iters;           // ceil(tMax / worstCaseH / preScaller), host double arithmetic
    numb h, maxv, transient, tmax, time_step;
    numb ic[UCB_NX];
    numb vals[UCB_NV];
    const numb* axis0;         // n_pts sweep values
    int* out_counts;           // per point: peaks (>= 0), -1 fixed point, 0 diverged
    double* out_peaks;         // n_pts x max_out
    double* out_intervals;     // n_pts x max_out
    unsigned long long* counter;
    unsigned long long* steps;
};

namespace ucbdev {

// State of the streaming peakFinder between chunks of samples. A position is decided once
// the sample after it is there, as in the reference loop that looks one sample ahead;
// positions >= n-2 are never candidates.
struct PeakScan {
    numb last;                 // the last sample
    long long next_i;          // first index allowed as a new candidate (outer loop i)
    bool plateau;              // inside the inner loop (j) of a candidate
    int found;                 // peaks found so far (before dropping the first)
    numb prev_t;               // raw time of the previous peak
    __device__ __forceinline__ void init() {
        last = 0;
        next_i = 2;
        plateau = false;
        found = 0;
        prev_t = 0;
    }
};

// The recorded variable is a constant of the build (UCB_WV): a select by a run-time index
// waited for every component at the end of each step (Lorenz diagram of 1,024 values, FP64,
// 11,000 steps, kernel: 1.24 -> 1.10 ms).
__device__ __forceinline__ numb recorded_value(const numb* x) {
#if UCB_WV >= 0
    return x[UCB_WV];
#elif UCB_NX >= 3
    return x[0] + pi * x[1] + euler * x[2];
#elif UCB_NX == 2
    return x[0] + pi * x[1];
#else
    return x[0];
#endif
}

// Where the peaks of one point go: the first max_out peaks and intervals of a 1-D
// diagram (Bif1dSink), or every peak the 2-D period count clusters (Bif2dSink).
struct Bif1dSink {
    double* peaks;
    double* intervals;
    int max_out;
    numb time_step;
    __device__ __forceinline__ void put(int k, numb value, numb dt) const {
        if (k < max_out) {
            peaks[k] = (double)value;
            intervals[k] = (double)((numb)dt * time_step);
        }
    }
};

// Emits a peak at position j (samples d0, d1, d2 at j - 1, j, j + 1) with the reference's
// interpolation.
template <class Sink>
__device__ __forceinline__ void emit_peak(PeakScan& s, long long j, numb d0, numb d1, numb d2, const Sink& sink) {
    numb denom = d0 - (numb)2.0 * d1 + d2;
    numb delta = 0.0;
    if (fabs(denom) > 1e-12) delta = 0.5 * (d0 - d2) / denom;
    const numb value = d1 - 0.25 * (d0 - d2) * delta;
    const numb t = (numb)(j - 1) + delta;
    if (s.found > 0) sink.put(s.found - 1, value, t - s.prev_t);
    s.prev_t = t;
    s.found += 1;
}

// Samples are searched for peaks a chunk at a time. Searched one by one inside the step
// loop, every sample waited for the finder's comparisons and branches, and whenever one of
// the warp's 32 lanes had a peak all of them waited for its division (about every second
// sample of a chaotic map). Collected first (one local-memory store a sample), a chunk's
// comparisons are independent of each other and give a bit mask of candidates, and the lanes
// work through their few peaks of the chunk together. A divisor of kCheckInterval.
// B200, native FP64: Lorenz diagram of 1,024 values 6.12 -> 3.60 ms, period map 256^2
// 17.7 -> 14.7 ms; Duffing features 256^2 (FP32) 75.0 -> 73.1 ms. (Chunks of 25 took 2-6 % less
// than chunks of 20.)
constexpr int kScanChunk = 25;
// Samples in flight in the comparison loop. A diagram runs about one warp per scheduler, so it
// takes the whole chunk at once (3.6 against 4.3 ms with 5); the maps keep
// their resident warps (256^2 period map: 64 against 120 registers, 14.7 against 15.1 ms).
#if defined(UCB_BIF2D) || defined(UCB_BIF_NO_KERNELS)
#define UCB_SCAN_UNROLL 5
#else
#define UCB_SCAN_UNROLL 25
#endif

// Decides the positions q0 - 1 .. q0 + m - 2 of a series of n samples, w[2 .. m + 1] holding
// the samples q0 .. q0 + m - 1 and w[0], w[1] the two before them.
template <class Sink>
__device__ __forceinline__ void scan_chunk(PeakScan& s, const numb* w, long long q0, int m, long long n,
                                           const Sink& sink) {
    // bit c: position q0 + c - 1 is above its predecessor and not below its successor (also
    // set beside a NaN); w beyond the chunk's samples is stale and masked out
    unsigned int cand = 0;
    numb prev = w[1];
    bool up = prev > w[0];
    UCB_PRAGMA_(unroll UCB_SCAN_UNROLL)
    for (int c = 0; c < kScanChunk; ++c) {
        const numb v = w[c + 2];
        const bool next_up = v > prev;
        if (up && !next_up) cand |= 1u << c;
        up = next_up;
        prev = v;
    }
    int c = q0 < 3 ? (int)(3 - q0) : 0;                     // positions from 2
    const int end = n - 1 - q0 < m ? (int)(n - 1 - q0) : m;  // to n - 3
    while (c < end) {
        if (s.plateau) {
            const numb d1 = w[c + 1], d2 = w[c + 2];
            if (d1 < d2) {
                s.plateau = false;
                s.next_i = q0 + c + 1;
            } else if (d1 - d2 > (numb)kEpsPeakDelta) {
                emit_peak(s, q0 + c - 1, w[c], d1, d2, sink);
                s.plateau = false;
                s.next_i = q0 + c + 1;
            }
            ++c;
            continue;
        }
        const unsigned int left = cand & (~0u << c);
        if (!left) break;
        c = __ffs((int)left) - 1;
        if (c >= end) break;
        const long long pos = q0 + c - 1;
        const numb d0 = w[c], d1 = w[c + 1], d2 = w[c + 2];
        ++c;
        if (pos < s.next_i) continue;
        if (d1 - d0 > (numb)kEpsPeakDelta && d1 > (numb)kPeakThreshold && d1 >= d2) {
            // inner loop starts at j = i with the same window
            if (d1 - d2 > (numb)kEpsPeakDelta) {
                emit_peak(s, pos, d0, d1, d2, sink);
                s.next_i = pos + 2;
            } else {
                s.plateau = true;
            }
        }
    }
}

// The next m samples of a series to w[2 ..], each with its `pre` steps; with check the
// divergence test after the first sample's steps. 0: diverged there.
template <class S>
__device__ __forceinline__ int sample_chunk(const S& st, numb* x, const numb* a, numb h, numb* w, int m, bool check,
                                            int pre, numb maxv) {
    int c = 0;
    if (check) {
        w[2] = recorded_value(x);
        st.step(x, a, h);
        for (int j = 1; j < pre; ++j) st.step(x, a, h);
        if (diverged(x, maxv)) return 0;
        c = 1;
    }
    if (pre == 1) {
        // by fours, so that the next samples' selects and stores fall into the steps' latencies
        // (Lorenz diagram, kernel: FP64 3.11 -> 2.66 ms, FP32 2.59 -> 2.13 ms; period maps 1-5 %)
#pragma unroll 4
        for (; c < m; ++c) {
            w[c + 2] = recorded_value(x);
            st.step(x, a, h);
        }
        return 1;
    }
    for (; c < m; ++c) {
        w[c + 2] = recorded_value(x);
        for (int j = 0; j < pre; ++j) st.step(x, a, h);
    }
    return 1;
}

#ifdef UCB_SIXTH
__device__ __noinline__ int redo_samples(numb* x, const numb* a, numb h, numb* w, int m, bool check, int pre,
                                         numb maxv) {
    return sample_chunk(VerbatimStepper(), x, a, h, w, m, check, pre, maxv);
}
__device__ __forceinline__ int run_samples(const Stepper& st, numb* x, const numb* a, numb h, numb* w, int m,
                                           bool check, int pre, numb maxv) {
    numb keep[UCB_NX];
    copy_state<UCB_NX>(x, keep);
    int r = st.verbatim ? 0 : sample_chunk(st, x, a, h, w, m, check, pre, maxv);
    if (st.failed()) {
        numb av[UCB_NV];
        copy_values(a, av);
        r = redo_samples(keep, av, h, w, m, check, pre, maxv);
        copy_state<UCB_NX>(keep, x);
    }
    return r;
}
#else
template <class S>
__device__ __forceinline__ int run_samples(const S& st, numb* x, const numb* a, numb h, numb* w, int m, bool check,
                                           int pre, numb maxv) {
    return sample_chunk(st, x, a, h, w, m, check, pre, maxv);
}
#endif

#ifdef UCB_FORCED
// The loops of a build whose warp shares its forcing: every lane takes every step, and a lane
// without a live cell (past the grid, or diverged) only does not count.
template <class Sink>
__device__ __forceinline__ int loop_record(const ForcedStepper& st, numb* x, const numb* a, numb h, long long iters,
                                           int pre, numb maxv, PeakScan& scan, const Sink& sink,
                                           long long& ns, bool live) {
    if (!__any_sync(0xFFFFFFFFu, live)) return 0;
    numb w[kScanChunk + 2];
#pragma unroll
    for (int k = 0; k < kScanChunk + 2; ++k) w[k] = 0;
    for (long long q0 = 0; q0 < iters; q0 += kScanChunk) {
        const int m = (iters - q0 < kScanChunk) ? (int)(iters - q0) : kScanChunk;
        int c = 0;
        if (q0 % kCheckInterval == 0) {
            st.set_phase(x);
            w[2] = recorded_value(x);
            st.steps(x, a, h, pre);
            if (live && diverged(x, maxv)) {
                ns += pre;
                live = false;
            }
            if (!__any_sync(0xFFFFFFFFu, live)) return 0;
            c = 1;
        }
        if (pre == 1 && UCB_WV >= 0 && UCB_WV != UCB_TRIG_PHASE) {
            numb* at = w + c + 2;
            st.steps(x, a, h, m - c, [&](int i) { at[i] = recorded_value(x); });
        } else {
            for (; c < m; ++c) {
                st.set_phase(x);
                w[c + 2] = recorded_value(x);
                st.steps(x, a, h, pre);
            }
        }
        if (live) {
            ns += (long long)pre * m;
            scan_chunk(scan, w, q0, m, iters, sink);
        }
        w[0] = w[m];
        w[1] = w[m + 1];
    }
    scan.last = w[1];
    st.set_phase(x);
    numb xPrev[UCB_NX];
#pragma unroll
    for (int j = 0; j < UCB_NX; ++j) xPrev[j] = x[j];
    st.steps(x, a, h, pre);
    if (!live) return 0;
    ns += pre;
    return fixed_point_flag(x, xPrev);
}

__device__ __forceinline__ int loop_transient(const ForcedStepper& st, numb* x, const numb* a, numb h, long long iters,
                                              int pre, numb maxv, long long& ns, bool live) {
    for (long long i0 = 0; i0 < iters; i0 += kCheckInterval) {
        st.steps(x, a, h, 1);
        if (live) {
            ns += 1;
            if (diverged(x, maxv)) live = false;
        }
        if (!__any_sync(0xFFFFFFFFu, live)) return 0;
        const int n = (iters - i0 < kCheckInterval) ? (int)(iters - i0) : kCheckInterval;
        st.steps(x, a, h, n - 1);
        if (live) ns += n - 1;
    }
    numb xPrev[UCB_NX];
#pragma unroll
    for (int j = 0; j < UCB_NX; ++j) xPrev[j] = x[j];
    st.steps(x, a, h, pre);
    if (!live) return 0;
    ns += pre;
    return fixed_point_flag(x, xPrev);
}
#define UCB_CELL_STEPPER(h, x) \
    __shared__ numb forced_tab[UCB_BLOCK / 32][kForced * kForcedEntry]; \
    const ForcedStepper st(h, forced_tab[threadIdx.x >> 5], (x)[UCB_TRIG_PHASE], threadIdx.x & 31)
#define UCB_RECORDS(flag) true  // the warp together
#else
#define UCB_CELL_STEPPER(h, x) const Stepper st(h)
#define UCB_RECORDS(flag) ((flag) == 1 || (flag) == -1)
template <class S, class Sink>
__device__ __forceinline__ int loop_record(const S& st, numb* x, const numb* a, numb h, long long iters, int pre,
                                           numb maxv, PeakScan& scan, const Sink& sink, long long& ns,
                                           bool /*live*/) {
    numb w[kScanChunk + 2];
#pragma unroll
    for (int k = 0; k < kScanChunk + 2; ++k) w[k] = 0;
    // The divergence test comes after the steps of samples 0, kCheckInterval, ...
    for (long long q0 = 0; q0 < iters; q0 += kScanChunk) {
        const int m = (iters - q0 < kScanChunk) ? (int)(iters - q0) : kScanChunk;
        if (q0 % kCheckInterval == 0) meet(st);
        if (run_samples(st, x, a, h, w, m, q0 % kCheckInterval == 0, pre, maxv) == 0) {
            ns += pre;
            return 0;
        }
        ns += (long long)pre * m;
        scan_chunk(scan, w, q0, m, iters, sink);
        w[0] = w[m];
        w[1] = w[m + 1];
    }
    scan.last = w[1];
    numb xPrev[UCB_NX];
#pragma unroll
    for (int j = 0; j < UCB_NX; ++j) xPrev[j] = x[j];
    run_single<false>(st, x, a, h, pre, maxv);
    ns += pre;
    return fixed_point_flag(x, xPrev);
}

// Transient of calculateDiscreteModelCUDA: one step per iteration, preScaller extra steps.
template <class S>
__device__ __forceinline__ int loop_transient(const S& st, numb* x, const numb* a, numb h, long long iters, int pre,
                                              numb maxv, long long& ns, bool /*live*/) {
    for (long long i0 = 0; i0 < iters; i0 += kCheckInterval) {
        const int n = (iters - i0 < kCheckInterval) ? (int)(iters - i0) : kCheckInterval;
        meet(st);
        if (run_single<true>(st, x, a, h, n, maxv) == 0) {
            ns += 1;
            return 0;
        }
        ns += n;
    }
    numb xPrev[UCB_NX];
#pragma unroll
    for (int j = 0; j < UCB_NX; ++j) xPrev[j] = x[j];
    run_single<false>(st, x, a, h, pre, maxv);
    ns += pre;
    return fixed_point_flag(x, xPrev);
}
#endif

}  // namespace ucbdev

#if defined(UCB_BIF_PAIRED) && !defined(UCB_BIF2D) && !defined(UCB_BIF_NO_KERNELS)
// A diagram with two warps for 32 points: the first integrates and leaves a chunk's samples in
// shared memory, the second searches them for peaks while the first takes the next chunk. One
// warp doing both spent 100 of a sample's 230 cycles on the search, with no other warp on its
// scheduler to use them (B200, Lorenz, 1,024 values, native FP64,
// 25,000 steps, kernel: 2.3 -> 1.79 ms). The two meet at a
// barrier of their own once a chunk; both run the same number of chunks.
namespace ucbdev {

struct BifPair {
    numb samples[2][kScanChunk][32];
    int m[2][32];     // samples of a lane's chunk (0: none, diverged or past its end)
    int live[2];      // any lane goes on
    int found[32];
};

__device__ __forceinline__ void pair_barrier(int pair) {
    __syncwarp();
    asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
}

// Samples of one chunk to `out` (stride 32), with the steps of sample_chunk().
template <class S>
__device__ __forceinline__ int sample_strided(const S& st, numb* x, const numb* a, numb h, numb* out, int m, bool check,
                                              int pre, numb maxv) {
    int c = 0;
    if (check) {
        out[0] = recorded_value(x);
        st.step(x, a, h);
        for (int j = 1; j < pre; ++j) st.step(x, a, h);
        if (diverged(x, maxv)) return 0;
        c = 1;
    }
    if (pre == 1) {
#pragma unroll 4
        for (; c < m; ++c) {
            out[c * 32] = recorded_value(x);
            st.step(x, a, h);
        }
        return 1;
    }
    for (; c < m; ++c) {
        out[c * 32] = recorded_value(x);
        for (int j = 0; j < pre; ++j) st.step(x, a, h);
    }
    return 1;
}
#ifdef UCB_SIXTH
__device__ __noinline__ int redo_strided(numb* x, const numb* a, numb h, numb* out, int m, bool check, int pre,
                                         numb maxv) {
    return sample_strided(VerbatimStepper(), x, a, h, out, m, check, pre, maxv);
}
__device__ __forceinline__ int run_strided(const Stepper& st, numb* x, const numb* a, numb h, numb* out, int m,
                                           bool check, int pre, numb maxv) {
    numb keep[UCB_NX];
    copy_state<UCB_NX>(x, keep);
    int r = st.verbatim ? 0 : sample_strided(st, x, a, h, out, m, check, pre, maxv);
    if (st.failed()) {
        numb av[UCB_NV];
        copy_values(a, av);
        r = redo_strided(keep, av, h, out, m, check, pre, maxv);
        copy_state<UCB_NX>(keep, x);
    }
    return r;
}
#else
template <class S>
__device__ __forceinline__ int run_strided(const S& st, numb* x, const numb* a, numb h, numb* out, int m, bool check,
                                           int pre, numb maxv) {
    return sample_strided(st, x, a, h, out, m, check, pre, maxv);
}
#endif

}  // namespace ucbdev

// A register cap is a number of resident blocks of UCB_BLOCK threads (UCB_LAUNCH_BOUNDS): half as many
// of twice the threads.
#ifdef UCB_MIN_BLOCKS
#define UCB_PAIRED_BOUNDS __launch_bounds__(2 * UCB_BLOCK, (UCB_MIN_BLOCKS + 1) / 2)
#else
#define UCB_PAIRED_BOUNDS __launch_bounds__(2 * UCB_BLOCK)
#endif
extern "C" __global__ void UCB_PAIRED_BOUNDS ucb_bif_kernel(const UcbBifParams p) {
    using namespace ucbdev;
    __shared__ BifPair pairs[UCB_BLOCK / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pair = warp % (UCB_BLOCK / 32);
    const bool integrates = warp < UCB_BLOCK / 32;
    BifPair& s = pairs[pair];
    const long long cell = ((long long)blockIdx.x * (UCB_BLOCK / 32) + pair) * 32 + lane;
    const bool here = cell < p.n_pts;
    const long long at = here ? cell : p.n_pts - 1;
    numb h = p.h;
    long long skip = p.skip, iters = p.iters, most = p.iters;
#if UCB_HAXIS == 0
    h = p.axis0[at];
    if (h > 0) {
        skip = (long long)ceil(p.transient / h);
        const long long il = (long long)ceil(p.tmax / h / (numb)p.pre_scaller);
        iters = il > p.iters ? p.iters : il;
    }
#endif
    if (integrates) {
        numb x[UCB_NX], a[UCB_NV];
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) x[i] = p.ic[i];
#pragma unroll
        for (int i = 0; i < UCB_NV; ++i) a[i] = p.vals[i];
#if UCB_HAXIS != 0
#if UCB_POV == 1
        a[UCB_IDX0] = p.axis0[at];
#else
        x[UCB_IDX0] = p.axis0[at];
#endif
#endif
        long long ns = 0;
        const Stepper st(h);
        int flag = -1;
        bool live = here && h > 0;
        if (live) {
            flag = loop_transient(st, x, a, h, skip, p.pre_scaller, p.maxv, ns, true);
            live = flag != 0;
        }
        int b = 0, since = 0;  // samples since the divergence test
        for (long long q0 = 0; q0 < most; q0 += kScanChunk, b ^= 1) {
            int m = 0;
            if (live && q0 < iters) {
                m = (iters - q0 < kScanChunk) ? (int)(iters - q0) : kScanChunk;
                if (since == 0) meet(st);
                if (run_strided(st, x, a, h, &s.samples[b][0][lane], m, since == 0, p.pre_scaller, p.maxv) == 0) {
                    ns += p.pre_scaller;
                    m = 0;
                    flag = 0;
                    live = false;
                } else {
                    ns += (long long)p.pre_scaller * m;
                }
            }
            since = since + kScanChunk == kCheckInterval ? 0 : since + kScanChunk;
            __syncwarp();
            s.m[b][lane] = m;
            const int go = __any_sync(0xFFFFFFFFu, live);
            if (lane == 0) s.live[b] = go;
            pair_barrier(pair);
            if (!go) break;
        }
        if (live) {
            numb xPrev[UCB_NX];
#pragma unroll
            for (int j = 0; j < UCB_NX; ++j) xPrev[j] = x[j];
            run_single<false>(st, x, a, h, p.pre_scaller, p.maxv);
            ns += p.pre_scaller;
            flag = fixed_point_flag(x, xPrev);
        }
        pair_barrier(pair);  // the second warp's counts
        if (here) {
            int count = flag;
            if (live && flag == 1) {
                int n = (s.found[lane] > 1) ? s.found[lane] - 1 : 0;
                if (n >= kMaxAmountOfPeaks) n = kMaxAmountOfPeaks;
                count = (iters < 5) ? 0 : n;
            }
            p.out_counts[cell] = count;
        }
        warp_add_steps(p.steps, ns, lane);
    } else {
        PeakScan scan;
        scan.init();
        const Bif1dSink sink{p.out_peaks + at * p.max_out, p.out_intervals + at * p.max_out, p.max_out, p.time_step};
        numb w[kScanChunk + 2];
#pragma unroll
        for (int k = 0; k < kScanChunk + 2; ++k) w[k] = 0;
        int b = 0;
        for (long long q0 = 0; q0 < most; q0 += kScanChunk, b ^= 1) {
            pair_barrier(pair);
            const int m = s.m[b][lane];
            if (m > 0) {
#pragma unroll
                for (int c = 0; c < kScanChunk; ++c) w[c + 2] = s.samples[b][c][lane];
                scan_chunk(scan, w, q0, m, iters, sink);
                w[0] = w[m];
                w[1] = w[m + 1];
            }
            if (!s.live[b]) break;
        }
        s.found[lane] = scan.found;
        pair_barrier(pair);
    }
}
#endif  // UCB_BIF_PAIRED

#if !defined(UCB_BIF_PAIRED) && !defined(UCB_BIF2D) && !defined(UCB_BIF_NO_KERNELS)
extern "C" __global__ void UCB_LAUNCH_BOUNDS ucb_bif_kernel(const UcbBifParams p) {
    long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    long long ns = 0;
    const bool live = cell < p.n_pts;
#ifdef UCB_FORCED
    if (!live) cell = p.n_pts - 1;  // its lane steps with the warp
    {
#else
    if (live) {
#endif
        numb x[UCB_NX], a[UCB_NV];
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) x[i] = p.ic[i];
#pragma unroll
        for (int i = 0; i < UCB_NV; ++i) a[i] = p.vals[i];
        numb h = p.h;
        long long skip = p.skip, iters = p.iters;
#if UCB_HAXIS == 0
        h = p.axis0[cell];
        skip = (long long)ceil(p.transient / h);
        long long il = (long long)ceil(p.tmax / h / (numb)p.pre_scaller);
        iters = il > p.iters ? p.iters : il;
#elif UCB_POV == 1
        a[UCB_IDX0] = p.axis0[cell];
#else
        x[UCB_IDX0] = p.axis0[cell];
#endif
        int count;
        if (!(h > 0)) {
            count = -1;
        } else {
            using namespace ucbdev;
            UCB_CELL_STEPPER(h, x);
            int flag = ucbdev::loop_transient(st, x, a, h, skip, p.pre_scaller, p.maxv, ns, live);
            if (UCB_RECORDS(flag)) {
                ucbdev::PeakScan scan;
                scan.init();
                const ucbdev::Bif1dSink sink{p.out_peaks + cell * p.max_out, p.out_intervals + cell * p.max_out,
                                             p.max_out, p.time_step};
                flag = ucbdev::loop_record(st, x, a, h, iters, p.pre_scaller, p.maxv, scan, sink,
                                           ns, flag != 0);
                if (flag == 1) {
                    int n = (scan.found > 1) ? scan.found - 1 : 0;
                    if (n >= ucbdev::kMaxAmountOfPeaks) n = ucbdev::kMaxAmountOfPeaks;
                    count = (iters < 5) ? 0 : n;
                } else {
                    count = flag;
                }
            } else {
                count = flag;
            }
        }
        if (live) p.out_counts[cell] = count;
    }
    ucbdev::warp_add_steps(p.steps, ns, lane);
}
#endif  // 1-D kernel

#if defined(UCB_BIF2D) && !defined(UCB_BIF_NO_KERNELS)
// ---------------------------------------------------------------------------------------
// 2-D bifurcation (period) maps: run_bif2d (parametric_engine.cpp:5487-5910) = per cell the
// 1-D trajectory + peakFinder above, then dbscan of the peaks (cudaLibrary.cu:2088-2166,
// dbscanCUDA :2321) whose cluster count is the "period". The reference keeps the whole
// recorded series, the peaks, the intervals and a helper array per cell in HBM and runs
// three kernels. Here a warp integrates its 32 cells (one per lane) with the peaks
// streaming into the warp's own scratch slot (one contiguous row of `cap` peaks per
// lane), then finds their periods (ucb_dbscan1d.cuh). Scratch is per resident warp, not per
// cell.
struct UcbBif2dParams {
    long long total;           // cells
    int n_pts;
    int swap_xy;               // 1: write transposed (user X = kernel axis 1)
    int pre_scaller;
    int writable_var;
    int cap;                   // peaks kept per cell (>= the largest possible count)
    int pad0;
    long long skip;            // (int)(transient / h), host double arithmetic
    long long iters;           // ceil(tMax / worstCaseH / preScaller), host double arithmetic
    numb h, maxv, transient, tmax, eps;
    numb ic[UCB_NX];
    numb vals[UCB_NV];
    const numb* axis0;
    const numb* axis1;
    char* rows;                // per warp slot: 32 rows of cap 8-byte entries
    char* work;                // per warp slot: bif2d_work_bytes(cap)
    double* out_values;        // period (-1 where the dbscan result is negative)
    int* out_flags;            // -1 / 1
    unsigned long long* counter;
    unsigned long long* steps;
};

namespace ucbdev {

struct Bif2dSink {
    numb* peaks;
    int cap;
    __device__ __forceinline__ void put(int k, numb value, numb) const {
        if (k < cap) peaks[k] = value;
    }
};

// Scratch of one warp besides its 32 peak rows (the host sizes it by the same rule): the
// sort's two key and two index buffers of one cell, then the bit sets of the 32 replays,
// interleaved by lane.
__device__ __forceinline__ long long bif2d_sort_bytes(int cap) { return ((long long)cap * 20 + 127) & ~127LL; }
__device__ __forceinline__ long long bif2d_work_bytes(int cap) {
    return bif2d_sort_bytes(cap) + (long long)((cap + 31) / 32) * 3 * 32 * 4;
}

// Periods of a warp's 32 cells from their peak rows: the rows are sorted one after the other
// by the whole warp, each giving way to its cell's ranges and order (6 bytes a peak in rows
// of 8), then every lane replays its own cell's dbscan.
__device__ __noinline__ int bif2d_periods(char* rows, char* work, int cap, int count, numb eps, int lane) {
    PeakKey* keys = reinterpret_cast<PeakKey*>(work);
    unsigned short* idx = reinterpret_cast<unsigned short*>(work + (long long)cap * 16);
    for (int c = 0; c < 32; ++c) {
        const int P = __shfl_sync(0xFFFFFFFFu, count, c);
        if (P < 2) continue;
        char* row = rows + (long long)c * cap * 8;
        PeakKey *ka = keys, *kb = keys + cap;
        unsigned short *ia = idx, *ib = idx + cap;
        for (int e = lane; e < P; e += 32) {
            ka[e] = peak_key(reinterpret_cast<const numb*>(row)[e]);
            ia[e] = (unsigned short)e;
        }
        __syncwarp();
        for (int run = 1; run < P; run *= 2) {
            merge_level(ka, ia, kb, ib, P, run, lane);
            __syncwarp();
            PeakKey* tk = ka;
            ka = kb;
            kb = tk;
            unsigned short* ti = ia;
            ia = ib;
            ib = ti;
        }
        peak_ranges(ka, ia, P, eps, reinterpret_cast<unsigned int*>(row),
                    reinterpret_cast<unsigned short*>(row + (long long)cap * 4), lane);
        __syncwarp();
    }
    const char* row = rows + (long long)lane * cap * 8;
    return dbscan_replay(count, reinterpret_cast<const unsigned int*>(row),
                         reinterpret_cast<const unsigned short*>(row + (long long)cap * 4),
                         reinterpret_cast<unsigned int*>(work + bif2d_sort_bytes(cap)) + lane, 32);
}

// Trajectory and peaks of one cell of a 2-D period map: the peak count (or the -1 / 0
// trajectory flag), peaks in row[0, min(count, cap)).
__device__ __forceinline__ int bif2d_peaks(const UcbBif2dParams& p, long long kidx, numb* row, long long& ns,
                                           bool live) {
    const ucbdev::CellAxes c = ucbdev::cell_axes(kidx, p.n_pts);
    numb x[UCB_NX], a[UCB_NV];
#pragma unroll
    for (int k = 0; k < UCB_NX; ++k) x[k] = p.ic[k];
#pragma unroll
    for (int k = 0; k < UCB_NV; ++k) a[k] = p.vals[k];
    ucbdev::apply_sweep(c, p.axis0, p.axis1, x, a);
    numb h = p.h;
    long long skip = p.skip, iters = p.iters;
#if UCB_HAXIS == 0 || UCB_HAXIS == 1
#if UCB_HAXIS == 0
    h = p.axis0[c.i0];
#else
    h = p.axis1[c.i1];
#endif
    skip = (long long)ceil(p.transient / h);
    const long long il = (long long)ceil(p.tmax / h / (numb)p.pre_scaller);
    iters = il > p.iters ? p.iters : il;
#endif
    int count;
    if (!(h > 0)) {
        count = -1;
    } else {
        UCB_CELL_STEPPER(h, x);
        int flag = ucbdev::loop_transient(st, x, a, h, skip, p.pre_scaller, p.maxv, ns, live);
        if (UCB_RECORDS(flag)) {
            ucbdev::PeakScan scan;
            scan.init();
            const ucbdev::Bif2dSink sink{row, p.cap};
            flag = ucbdev::loop_record(st, x, a, h, iters, p.pre_scaller, p.maxv, scan, sink,
                                       ns, flag != 0);
            if (flag == 1) {
                int n = (scan.found > 1) ? scan.found - 1 : 0;
                if (n >= ucbdev::kMaxAmountOfPeaks) n = ucbdev::kMaxAmountOfPeaks;
                count = (iters < 5) ? 0 : n;
            } else {
                count = flag;
            }
        } else {
            count = flag;
        }
    }
    return count > p.cap ? p.cap : count;  // cannot clip: cap covers the largest count
}

}  // namespace ucbdev

extern "C" __global__ void UCB_LAUNCH_BOUNDS ucb_bif2d_kernel(const UcbBif2dParams p) {
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    char* rows = p.rows + warp * 32 * (long long)p.cap * 8;
    char* work = p.work + warp * ucbdev::bif2d_work_bytes(p.cap);
    long long ns = 0;
    for (;;) {
        const long long base = ucbdev::warp_fetch(p.counter, lane);
        if (base >= p.total) break;
        const long long i = base + lane;
        numb* row = reinterpret_cast<numb*>(rows + (long long)lane * p.cap * 8);
#ifdef UCB_FORCED
        int count = ucbdev::bif2d_peaks(p, i < p.total ? i : p.total - 1, row, ns, i < p.total);
        if (i >= p.total) count = 0;
#else
        const int count = i < p.total ? ucbdev::bif2d_peaks(p, i, row, ns, true) : 0;
#endif
        __syncwarp();
        const int mine = ucbdev::bif2d_periods(rows, work, p.cap, count, p.eps, lane);
        if (i < p.total) {
            long long out = i;
            if (p.swap_xy) out = (i % p.n_pts) * p.n_pts + i / p.n_pts;
            p.out_values[out] = mine < 0 ? -1.0 : (double)mine;
            p.out_flags[out] = mine < 0 ? -1 : 1;
        }
        __syncwarp();
    }
    ucbdev::warp_add_steps(p.steps, ns, lane);
}
#endif  // UCB_BIF2D

