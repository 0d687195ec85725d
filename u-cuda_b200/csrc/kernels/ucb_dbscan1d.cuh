// ucb_dbscan1d.cuh — the period count of one cell's peaks (NVRTC header, after ucb_device.cuh).
//
// The reference's dbscan (cudaLibrary.cu:2088-2166) labels, for every point it visits, all
// unlabelled points within eps by a scan over the whole list: P visits x P distances. Its
// result depends on the order of its visits (a stack slot is written at the point's own
// index and popped at NumNeibor - 1; the loop goes on from the popped index), so that order
// is kept and only the scans are replaced. In one dimension the points within eps of a
// point are neighbours in sorted order (the rounded difference p - x grows with p), so
//   1. a warp sorts a cell's peaks (merge by rank: every lane places its elements by binary
//      search in the sibling run) and finds for every peak the sorted range [lo, hi) within
//      eps of it — about 10 P log2(P) / 32 warp instructions instead of P^2 / 32 loads;
//   2. a lane per cell replays the visits on bit sets (unlabelled by sorted position,
//      unlabelled by index, filled stack slots): a visit reads its range and takes the set
//      bits in it, so every peak is touched once over the whole run.
// The scans were bound by the latency of their dependent loads, one visit after the other.
// B200, Lorenz period map 256^2 (native FP64, 25,000 steps, several hundred peaks a cell),
// whole call: 76.0 ms with the scans (one warp per cell's visits), 17.7 ms sorted.
#pragma once

namespace ucbdev {

#ifdef UCB_NUMB_F32
typedef int PeakKey;
constexpr PeakKey kKeyFlip = 0x7FFFFFFF;
__device__ __forceinline__ PeakKey key_bits(float v) { return __float_as_int(v); }
__device__ __forceinline__ float bits_value(PeakKey b) { return __int_as_float(b); }
#else
typedef long long PeakKey;
constexpr PeakKey kKeyFlip = 0x7FFFFFFFFFFFFFFFLL;
__device__ __forceinline__ PeakKey key_bits(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ double bits_value(PeakKey b) { return __longlong_as_double(b); }
#endif

// Integer keys in the order of the values, every NaN last (a NaN is within eps of nothing).
__device__ __forceinline__ PeakKey peak_key(numb v) {
    if (v != v) return kKeyFlip;
    const PeakKey b = key_bits(v);
    return b >= 0 ? b : (b ^ kKeyFlip);
}
__device__ __forceinline__ numb peak_value(PeakKey k) { return bits_value(k >= 0 ? k : (k ^ kKeyFlip)); }

// Elements a lane places at once: their binary searches are independent, so their loads
// overlap (one search alone waits an L1 round trip per halving).
constexpr int kMergeIlp = 4;

// One merge level, lane's share: sorted runs of `run` (a power of two) keys in (ka, ia) are
// merged pairwise into (kb, ib), equal keys in the order of the input.
__device__ __forceinline__ void merge_level(const PeakKey* ka, const unsigned short* ia, PeakKey* kb,
                                            unsigned short* ib, int P, int run, int lane) {
    for (int e0 = lane; e0 < P; e0 += 32 * kMergeIlp) {
        PeakKey key[kMergeIlp];
        int first[kMergeIlp], n[kMergeIlp], at[kMergeIlp];
        bool right[kMergeIlp];
#pragma unroll
        for (int q = 0; q < kMergeIlp; ++q) {
            const int e = e0 + 32 * q;
            const int base = e & ~(2 * run - 1);
            right[q] = (e & run) != 0;
            first[q] = right[q] ? base : base + run;  // the sibling run
            const int left = P - first[q];
            n[q] = e < P ? (left < run ? left : run) : 0;
            key[q] = e < P ? ka[e] : 0;
            at[q] = 0;
        }
        for (int s = run; s > 0; s >>= 1) {
#pragma unroll
            for (int q = 0; q < kMergeIlp; ++q) {
                if (at[q] + s <= n[q]) {
                    const PeakKey k = ka[first[q] + at[q] + s - 1];
                    if (k < key[q] || (right[q] && k == key[q])) at[q] += s;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < kMergeIlp; ++q) {
            const int e = e0 + 32 * q;
            if (e < P) {
                const int dst = (right[q] ? e - run : e) + at[q];
                kb[dst] = key[q];
                ib[dst] = ia[e];
            }
        }
    }
}

// Sorted positions [lo, hi) within eps of every peak, lane's share: lo | hi << 16 at the
// peak's index, and the peak at every sorted position.
__device__ __forceinline__ void peak_ranges(const PeakKey* ka, const unsigned short* ia, int P, numb eps,
                                            unsigned int* range, unsigned short* order, int lane) {
    int top = 1;
    while (2 * top <= P) top *= 2;
    for (int e0 = lane; e0 < P; e0 += 32 * kMergeIlp) {
        numb x[kMergeIlp];
        int lo[kMergeIlp], hi[kMergeIlp];
#pragma unroll
        for (int q = 0; q < kMergeIlp; ++q) {
            const int e = e0 + 32 * q;
            x[q] = peak_value(ka[e < P ? e : P - 1]);
            lo[q] = hi[q] = 0;
        }
        for (int s = top; s > 0; s >>= 1) {
#pragma unroll
            for (int q = 0; q < kMergeIlp; ++q) {
                if (lo[q] + s <= P && peak_value(ka[lo[q] + s - 1]) - x[q] <= -eps) lo[q] += s;
                if (hi[q] + s <= P && peak_value(ka[hi[q] + s - 1]) - x[q] < eps) hi[q] += s;
            }
        }
#pragma unroll
        for (int q = 0; q < kMergeIlp; ++q) {
            const int e = e0 + 32 * q;
            if (e < P) {
                const unsigned short k = ia[e];
                range[k] = (unsigned int)lo[q] | ((unsigned int)hi[q] << 16);
                order[e] = k;
            }
        }
    }
}

// Which of up to 96 words of a bit set are not empty.
struct WordSet {
    unsigned long long a;
    unsigned int b;
    __device__ __forceinline__ explicit WordSet(int words)
        : a(words >= 64 ? ~0ULL : (1ULL << words) - 1), b(words > 64 ? (1u << (words - 64)) - 1 : 0) {}
    __device__ __forceinline__ int next(int w) const {  // first non-empty word >= w, 96 if none
        if (w < 64) {
            const unsigned long long m = a >> w;
            if (m) return w + __ffsll((long long)m) - 1;
            w = 64;
        }
        const unsigned int m = w < 96 ? b >> (w - 64) : 0;
        return m ? w + __ffs((int)m) - 1 : 96;
    }
    __device__ __forceinline__ void clear(int w) {
        if (w < 64) a &= ~(1ULL << w);
        else b &= ~(1u << (w - 64));
    }
};

// The reference's dbscan of one cell's P peaks (P <= 2,500) from their ranges: clusters - 1,
// or P itself where it returns early (-1, 0, 1). `bits`: three sets of (P + 31) / 32 words,
// word w of set s at bits[(s * words + w) * stride].
__device__ __forceinline__ int dbscan_replay(int P, const unsigned int* range, const unsigned short* order,
                                             unsigned int* bits, int stride) {
    if (P < 2) return P;
    const int words = (P + 31) >> 5;
    unsigned int* un_pos = bits;                       // unlabelled, by sorted position
    unsigned int* un_idx = bits + words * stride;      // unlabelled, by index
    unsigned int* slots = bits + 2 * words * stride;   // stack slots written and not yet popped
    for (int w = 0; w < words; ++w) {
        const unsigned int all = (w == words - 1 && (P & 31)) ? (1u << (P & 31)) - 1 : ~0u;
        un_pos[w * stride] = all;
        un_idx[w * stride] = all;
        slots[w * stride] = 0;
    }
    WordSet pos_words(words), idx_words(words);
    int cluster = 0, nn = 0;
    for (int i = 0; i < P; ++i) {
        if (nn >= 1) {
            // the slot holds its own index, or 0 once popped
            const int s = --nn;
            const unsigned int w = slots[(s >> 5) * stride], bit = 1u << (s & 31);
            i = (w & bit) ? s : 0;
            if (w & bit) slots[(s >> 5) * stride] = w & ~bit;
        } else {
            // the next unlabelled index opens a cluster
            int w = i >> 5;
            unsigned int m = (idx_words.next(w) == w) ? un_idx[w * stride] & (~0u << (i & 31)) : 0;
            if (!m) {
                w = idx_words.next(w + 1);
                if (w >= words) break;
                m = un_idx[w * stride];
            }
            i = w * 32 + __ffs((int)m) - 1;
            ++cluster;
            const unsigned int left = un_idx[w * stride] & ~(1u << (i & 31));
            un_idx[w * stride] = left;
            if (!left) idx_words.clear(w);
        }
        const unsigned int r = range[i];
        const int lo = (int)(r & 0xFFFFu), hi = (int)(r >> 16);
        for (int w = pos_words.next(lo >> 5); w * 32 < hi; w = pos_words.next(w + 1)) {
            const unsigned int word = un_pos[w * stride];
            unsigned int m = word;
            if (w == (lo >> 5)) m &= ~0u << (lo & 31);
            if (hi - w * 32 < 32) m &= (1u << (hi & 31)) - 1;
            if (!m) continue;
            un_pos[w * stride] = word ^ m;
            if (word == m) pos_words.clear(w);
            for (; m; m &= m - 1) {
                const int k = order[w * 32 + __ffs((int)m) - 1];
                // the last peak is never a neighbour (inner bound P - 1), and a seed not its own
                if (k == P - 1 || k == i) continue;
                const unsigned int bit = 1u << (k & 31);
                const unsigned int left = un_idx[(k >> 5) * stride] & ~bit;
                un_idx[(k >> 5) * stride] = left;
                if (!left) idx_words.clear(k >> 5);
                slots[(k >> 5) * stride] |= bit;
                ++nn;
            }
        }
    }
    return cluster - 1;
}

}  // namespace ucbdev
