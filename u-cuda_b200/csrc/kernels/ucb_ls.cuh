// ucb_ls.cuh — full Lyapunov spectrum maps (NVRTC header, after ucb_device.cuh).
//
// Two methods, one thread per cell, everything in registers, persistent grid:
//
//  * UCB_LS_FIXED (the reference's method, LSKernelCUDA cudaLibrary.cu:2878-3073):
//    fixed-step trajectory + N shadow probes at distance eps, random unit directions
//    (RNG subsequence = cell index) orthonormalised once, then every NT block: advance
//    x and the probes, subtract x, classical Gram-Schmidt (gramSchmidtProcess :2848-2874,
//    projections against the unnormalised b_j), sum log(|b_k| / eps), re-seat the probes.
//
//  * UCB_LS_DP5: tangent-linear spectrum with the adaptive Dormand-Prince 5(4) pair
//    (Dormand & Prince 1980, FSAL) integrating x' = f(x) and V' = J(x) V for N tangent
//    vectors, with the mixed absolute/relative RMS error norm taken over the whole
//    augmented state (x and V: controlling x alone lets the step grow past what the
//    contracting tangent directions need, and the most negative exponents then follow the
//    method's stability function instead of the flow), step factor 0.9 err^-1/5 clamped
//    to [0.2, 5] (2 after a rejection), with
//    modified Gram-Schmidt every `gs_every` accepted steps — or earlier, when the time
//    since the last pass times the running estimate of lambda_1 - lambda_N exceeds the
//    precision's budget (UCB_GS_BUDGET nats: 20 for FP64, 8 for FP32), because beyond it
//    the most contracted direction sinks below the rounding of the stored tangent vectors;
//    the norms, log sums, time and the error norm are FP64 whatever numb is.
#pragma once

struct UcbLsParams {
    long long total;
    long long cell_offset;
    int n_pts;
    int swap_xy;
    int n_blocks;          // (int)(tMax / NT)   [fixed]
    int gs_every;          // accepted steps between MGS   [dp5]
    long long skip;        // (int)(transient / h)        [fixed]
    long long nt_steps;    // (size_t)(NT / h) in numb     [fixed]
    long long max_steps;   // step attempt cap per cell   [dp5]
    numb h, NT, tmax, eps, maxv, transient;
    double rtol, atol, t_end, h0;   // [dp5]
    numb ic[UCB_NX];
    numb vals[UCB_NV];
    const numb* axis0;
    const numb* axis1;
    double* out_values;    // plane-major: values[k * cells + cell] (cells = n^2, or n for one axis)
    int* out_flags;
    unsigned long long* counter;
    unsigned long long* steps;
    long long* out_cell_steps;  // per cell: steps (fixed) / step attempts (DP5); may be null
    int groups;                 // cells a warp at a time (UCB_LS_GROUP)
};

namespace ucbdev {

__device__ __forceinline__ long long ls_out_cell(const UcbLsParams& p, long long kidx) {
    if (!p.swap_xy) return kidx;
    const long long kix = kidx % p.n_pts, kiy = kidx / p.n_pts;
    return kix * p.n_pts + kiy;
}

__device__ __forceinline__ void ls_store(const UcbLsParams& p, long long kidx, const double* v) {
    const long long cell = ls_out_cell(p, kidx);
#if UCB_DIM == 2
    const long long plane = (long long)p.n_pts * p.n_pts;
#else
    const long long plane = p.n_pts;  // one swept axis: n_pts cells per exponent plane
#endif
    bool bad = false;
#pragma unroll
    for (int k = 0; k < UCB_NX; ++k) {
        p.out_values[k * plane + cell] = v[k];
        if (v[k] == 999.0 || v[k] == -999.0) bad = true;
    }
    p.out_flags[cell] = bad ? -1 : 1;
}

#if defined(UCB_LS_FIXED)
// gramSchmidtProcess(a -> b, dens): classical GS, rows are vectors.
__device__ __forceinline__ void gram_schmidt_classical(const numb (*a)[UCB_NX], numb (*b)[UCB_NX], numb* dens) {
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) {
#pragma unroll
        for (int j = 0; j < UCB_NX; ++j) b[i][j] = a[i][j];
#pragma unroll
        for (int j = 0; j < i; ++j) {
            numb num = 0, den = 0;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) {
                num += a[i][l] * b[j][l];
                den += b[j][l] * b[j][l];
            }
            const numb frac = den == 0 ? 0 : num / den;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) b[i][l] -= frac * b[j][l];
        }
    }
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) {
        numb den = 0;
#pragma unroll
        for (int j = 0; j < UCB_NX; ++j) den += b[i][j] * b[i][j];
        den = sqrt(den);
#pragma unroll
        for (int j = 0; j < UCB_NX; ++j) b[i][j] = den == 0 ? 0 : b[i][j] / den;
        if (dens) dens[i] = den;
    }
}

// `n` steps of x and the N probes in lock step (the reference advances them one after the
// other; they never interact inside a block); with Check the divergence test after the first
// of them. 0 if any diverged there.
template <bool Check, class S>
__device__ __forceinline__ int block_probes(const S& s, numb* x, numb (*y)[UCB_NX], const numb* a, numb h, int n,
                                            numb maxValue) {
    s.step(x, a, h);
#pragma unroll
    for (int j = 0; j < UCB_NX; ++j) s.step(y[j], a, h);
    if (Check) {
        bool bad = diverged(x, maxValue);
#pragma unroll
        for (int j = 0; j < UCB_NX; ++j) bad = bad || diverged(y[j], maxValue);
        if (bad) return 0;
    }
    for (int i = 1; i < n; ++i) {
        s.step(x, a, h);
#pragma unroll
        for (int j = 0; j < UCB_NX; ++j) s.step(y[j], a, h);
    }
    return 1;
}

#ifdef UCB_SIXTH
// One trajectory of a block with the division, on a copy in registers. The cell's trajectories go one
// after the other (the body's time is its divisions', in lock step too): all of them in registers
// at once took the kernel of 4 variables, FP64, from 126 to 166 registers, three blocks an SM
// instead of four; in memory at once, 256^2 FP32 cells that settle took 37.8 instead of 36.2 ms.
__device__ __noinline__ int redo_probe(numb* x, const numb* a, numb h, int n, numb maxValue, bool check) {
    numb xr[UCB_NX], ar[UCB_NV];
    copy_state<UCB_NX>(x, xr);
    copy_values(a, ar);
    calculateDiscreteModel(xr, ar, h);
    const int r = check && diverged(xr, maxValue) ? 0 : 1;
#pragma unroll 1
    for (int i = 1; i < (r ? n : 1); ++i) calculateDiscreteModel(xr, ar, h);
    copy_state<UCB_NX>(xr, x);
    return r;
}
template <bool Check>
__device__ __forceinline__ int run_probes(const Stepper& s, numb* x, numb (*y)[UCB_NX], const numb* a, numb h, int n,
                                          numb maxValue) {
    numb keep[UCB_NX + UCB_NX * UCB_NX];
    copy_state<UCB_NX>(x, keep);
#pragma unroll
    for (int j = 0; j < UCB_NX; ++j) copy_state<UCB_NX>(y[j], keep + UCB_NX + j * UCB_NX);
    int r = s.verbatim ? 0 : block_probes<Check>(s, x, y, a, h, n, maxValue);
    if (s.failed()) {
        numb av[UCB_NV];
        copy_values(a, av);
        r = 1;
        for (int j = 0; j <= UCB_NX && r; ++j) r = redo_probe(keep + j * UCB_NX, av, h, n, maxValue, Check);
        copy_state<UCB_NX>(keep, x);
#pragma unroll
        for (int j = 0; j < UCB_NX; ++j) copy_state<UCB_NX>(keep + UCB_NX + j * UCB_NX, y[j]);
    }
    return r;
}
#else
template <bool Check, class S>
__device__ __forceinline__ int run_probes(const S& s, numb* x, numb (*y)[UCB_NX], const numb* a, numb h, int n,
                                          numb maxValue) {
    return block_probes<Check>(s, x, y, a, h, n, maxValue);
}
#endif

// A whole loop call of x and the probes. 0 if any diverged.
template <class S>
__device__ __forceinline__ int loop_probes(const S& s, numb* x, numb (*y)[UCB_NX], const numb* a, numb h,
                                           long long iters, numb maxValue, long long& ns) {
    for (long long i0 = 0; i0 < iters; i0 += kCheckInterval) {
        const int n = (iters - i0 < kCheckInterval) ? (int)(iters - i0) : kCheckInterval;
        if (i0 > 0) meet(s);
        if (run_probes<true>(s, x, y, a, h, n, maxValue) == 0) {
            ns += UCB_NX + 1;
            return 0;
        }
        ns += (long long)(UCB_NX + 1) * n;
    }
#if UCB_EXTRA_STEP
    run_probes<false>(s, x, y, a, h, 1, maxValue);
    ns += UCB_NX + 1;
#endif
    return 1;
}

#if defined(UCB_LS_TANGENT) && defined(UCB_HAS_JVP) && !defined(UCB_EXACT)
// Tangent-vector form of the fixed method (native FP32 builds): instead of N shadow
// trajectories x + eps z, whose differences from x fall below FP32 resolution for small eps,
// the N tangent vectors v' = J(x) v are advanced with x in one RK4 sweep (the stage sums
// accumulated stage by stage), and the block's Gram-Schmidt, norms and log sums are FP64.
template <int M>
__device__ __forceinline__ void ls_tangent_step(numb* x, numb (*V)[UCB_NX], const numb* a, numb h) {
    const numb hh = h * (numb)0.5, h6 = h * (numb)(1.0 / 6.0), two = (numb)2;
    numb k[UCB_NX], l[UCB_NX], xt[UCB_NX], sx[UCB_NX];
    numb vt[M][UCB_NX], sv[M][UCB_NX];
    ucb_rhs(x, a, k);
#pragma unroll
    for (int j = 0; j < M; ++j) {
        ucb_jvp(x, a, V[j], l);
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) {
            sv[j][i] = l[i];
            vt[j][i] = fma(hh, l[i], V[j][i]);
        }
    }
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) {
        sx[i] = k[i];
        xt[i] = fma(hh, k[i], x[i]);
    }
#pragma unroll
    for (int stage = 2; stage <= 3; ++stage) {
        const numb c = stage == 2 ? hh : h;
        ucb_rhs(xt, a, k);
#pragma unroll
        for (int j = 0; j < M; ++j) {
            ucb_jvp(xt, a, vt[j], l);
#pragma unroll
            for (int i = 0; i < UCB_NX; ++i) {
                sv[j][i] = fma(two, l[i], sv[j][i]);
                vt[j][i] = fma(c, l[i], V[j][i]);
            }
        }
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) {
            sx[i] = fma(two, k[i], sx[i]);
            xt[i] = fma(c, k[i], x[i]);
        }
    }
    ucb_rhs(xt, a, k);
#pragma unroll
    for (int j = 0; j < M; ++j) {
        ucb_jvp(xt, a, vt[j], l);
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) V[j][i] = fma(h6, sv[j][i] + l[i], V[j][i]);
    }
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) x[i] = fma(h6, sx[i] + k[i], x[i]);
}

// Classical Gram-Schmidt of the rows of V in FP64 (the reference's gramSchmidtProcess
// order): V becomes orthonormal (rounded to numb), dens[i] the norm of row i after
// removing its projections on the earlier rows.
__device__ __forceinline__ void gs_classical_f64(numb (*V)[UCB_NX], double* dens) {
    double b[UCB_NX][UCB_NX];
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) {
#pragma unroll
        for (int l = 0; l < UCB_NX; ++l) b[i][l] = (double)V[i][l];
#pragma unroll
        for (int j = 0; j < i; ++j) {
            double num = 0, den = 0;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) {
                num = fma((double)V[i][l], b[j][l], num);
                den = fma(b[j][l], b[j][l], den);
            }
            const double frac = den == 0 ? 0 : num / den;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) b[i][l] = fma(-frac, b[j][l], b[i][l]);
        }
    }
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) {
        double den = 0;
#pragma unroll
        for (int l = 0; l < UCB_NX; ++l) den = fma(b[i][l], b[i][l], den);
        den = sqrt(den);
        const double inv = den == 0 ? 0 : 1.0 / den;
#pragma unroll
        for (int l = 0; l < UCB_NX; ++l) V[i][l] = (numb)(b[i][l] * inv);
        dens[i] = den;
    }
}

// NT-step block of x and the tangent vectors with the divergence test of loop_probes
// (tangent vectors: non-finite only). 0 if anything diverged.
template <int M>
__device__ __forceinline__ int loop_tangents(numb* x, numb (*V)[UCB_NX], const numb* a, numb h, long long iters,
                                             numb maxValue, long long& ns) {
    for (long long i0 = 0; i0 < iters; i0 += kCheckInterval) {
        ls_tangent_step<M>(x, V, a, h);
        ns += UCB_NX + 1;
        bool bad = diverged(x, maxValue);
#pragma unroll
        for (int j = 0; j < M; ++j) bad = bad || diverged(V[j], (numb)0);
        if (bad) return 0;
        const long long n = (iters - i0 < kCheckInterval) ? iters - i0 : kCheckInterval;
        for (long long i = 1; i < n; ++i) ls_tangent_step<M>(x, V, a, h);
        ns += (long long)(UCB_NX + 1) * (n - 1);
    }
#if UCB_EXTRA_STEP
    ls_tangent_step<M>(x, V, a, h);
    ns += UCB_NX + 1;
#endif
    return 1;
}
#define UCB_LS_FIXED_TANGENT 1
#endif

__device__ __forceinline__ void ls_cell_fixed(const UcbLsParams& p, long long kidx, long long& ns) {
    double outv[UCB_NX];
    const CellAxes c = cell_axes(kidx, p.n_pts);
    numb h = p.h;
    long long nt = p.nt_steps, skip = p.skip;
#if UCB_HAXIS == 0
    h = p.axis0[c.i0];
#elif UCB_HAXIS == 1
    h = p.axis1[c.i1];
#endif
#if UCB_HAXIS != -1
    nt = (long long)ceil(p.NT / h);
    skip = (long long)ceil(p.transient / h);
#endif
    if (!(h > 0)) {
#pragma unroll
        for (int m = 0; m < UCB_NX; ++m) outv[m] = (double)nan("");
        ls_store(p, kidx, outv);
        return;
    }
    numb x[UCB_NX], a[UCB_NV];
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) x[i] = p.ic[i];
#pragma unroll
    for (int i = 0; i < UCB_NV; ++i) a[i] = p.vals[i];
    apply_sweep(c, p.axis0, p.axis1, x, a);
    numb y[UCB_NX][UCB_NX], z[UCB_NX][UCB_NX], dens[UCB_NX];
    double result[UCB_NX];
    {
        Rng st;
        rng_init(1234567891ULL, (unsigned long long)kidx, 0ULL, &st);
#pragma unroll
        for (int j = 0; j < UCB_NX; ++j) {
            numb zPower = 0;
#pragma unroll
            for (int i = 0; i < UCB_NX; ++i) {
                z[j][i] = rng_uniform(&st) - 0.5;
                zPower += z[j][i] * z[j][i];
            }
            zPower = sqrt(zPower);
#pragma unroll
            for (int i = 0; i < UCB_NX; ++i) z[j][i] /= zPower;
        }
    }
    const Stepper st(h);
    if (loop_single(st, x, a, h, skip, p.maxv, ns) == 0) {
#pragma unroll
        for (int m = 0; m < UCB_NX; ++m) outv[m] = 999.0;
        ls_store(p, kidx, outv);
        return;
    }
#if defined(UCB_LS_FIXED_TANGENT)
    {
        double d[UCB_NX], sum[UCB_NX];
        gs_classical_f64(z, d);  // the same random start, orthonormal
#pragma unroll
        for (int k = 0; k < UCB_NX; ++k) sum[k] = 0.0;
        for (int b = 0; b < p.n_blocks; ++b) {
            if (loop_tangents<UCB_NX>(x, z, a, h, nt, p.maxv, ns) == 0) {
#pragma unroll
                for (int m = 0; m < UCB_NX; ++m) outv[m] = 999.0;
                ls_store(p, kidx, outv);
                return;
            }
            gs_classical_f64(z, d);
#pragma unroll
            for (int k = 0; k < UCB_NX; ++k) sum[k] += log(d[k]);
        }
        (void)y;
        (void)dens;
#pragma unroll
        for (int k = 0; k < UCB_NX; ++k) result[k] = sum[k] / (double)p.tmax;
        ls_store(p, kidx, result);
        return;
    }
#endif
    gram_schmidt_classical(z, y, nullptr);
#pragma unroll
    for (int j = 0; j < UCB_NX; ++j)
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) y[j][i] = y[j][i] * p.eps + x[i];
    numb res_n[UCB_NX];
#pragma unroll
    for (int k = 0; k < UCB_NX; ++k) res_n[k] = 0;
    for (int b = 0; b < p.n_blocks; ++b) {
        if ((b & 7) == 0) meet(st);
        if (loop_probes(st, x, y, a, h, nt, p.maxv, ns) == 0) {
#pragma unroll
            for (int m = 0; m < UCB_NX; ++m) outv[m] = 999.0;
            ls_store(p, kidx, outv);
            return;
        }
#pragma unroll
        for (int k = 0; k < UCB_NX; ++k)
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) y[k][l] = y[k][l] - x[l];
        gram_schmidt_classical(y, z, dens);
#pragma unroll
        for (int k = 0; k < UCB_NX; ++k) {
            res_n[k] += log(dens[k] / p.eps);
#pragma unroll
            for (int j = 0; j < UCB_NX; ++j) y[k][j] = (numb)(x[j] + z[k][j] * p.eps);
        }
    }
#pragma unroll
    for (int k = 0; k < UCB_NX; ++k) result[k] = (double)(res_n[k] / p.tmax);
    ls_store(p, kidx, result);
}

#if defined(UCB_LS_GROUP) && UCB_HAXIS == -1
// ls_cell_fixed with a cell on several lanes, the same values and order of operations: a
// trajectory a lane (x on the group's first lane and the N shadows after it) or, in the tangent
// form, x and one tangent vector a lane. Every lane takes the transient; the rows of the
// Gram-Schmidt pass are exchanged by shuffles, so all lanes of the warp stay in the loop until
// all its cells are done. Where each form runs and its times: ls_groups of ucb_ls.cpp.
#ifdef UCB_LS_FIXED_TANGENT
constexpr int kLanes = UCB_NX, kFirstRow = 0;
#else
constexpr int kLanes = UCB_NX + 1, kFirstRow = 1;
#endif

// gram_schmidt_classical() over the group's rows: lane kFirstRow + i holds row i (row < 0: none).
template <class T>
__device__ __forceinline__ void group_gs(const T* a, T* b, T& dens, int row, int base) {
#pragma unroll
    for (int l = 0; l < UCB_NX; ++l) b[l] = a[l];
#pragma unroll
    for (int j = 0; j + 1 < UCB_NX; ++j) {
        T w[UCB_NX];
#pragma unroll
        for (int l = 0; l < UCB_NX; ++l) w[l] = __shfl_sync(0xFFFFFFFFu, b[l], base + kFirstRow + j);
        if (row > j) {
            T num = 0, den = 0;
#ifdef UCB_LS_FIXED_TANGENT
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) {
                num = fma(a[l], w[l], num);
                den = fma(w[l], w[l], den);
            }
            const T frac = den == 0 ? 0 : num / den;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) b[l] = fma(-frac, w[l], b[l]);
#else
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) {
                num += a[l] * w[l];
                den += w[l] * w[l];
            }
            const T frac = den == 0 ? 0 : num / den;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) b[l] -= frac * w[l];
#endif
        }
        __syncwarp();
    }
    T den = 0;
#ifdef UCB_LS_FIXED_TANGENT
#pragma unroll
    for (int l = 0; l < UCB_NX; ++l) den = fma(b[l], b[l], den);
    den = sqrt(den);
    const T inv = den == 0 ? 0 : 1.0 / den;
#pragma unroll
    for (int l = 0; l < UCB_NX; ++l) b[l] *= inv;
#else
#pragma unroll
    for (int l = 0; l < UCB_NX; ++l) den += b[l] * b[l];
    den = sqrt(den);
#pragma unroll
    for (int l = 0; l < UCB_NX; ++l) b[l] = den == 0 ? 0 : b[l] / den;
#endif
    dens = den;
}

__device__ __forceinline__ void ls_groups_fixed(const UcbLsParams& p, long long& ns) {
    const unsigned int full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const bool member = lane < p.groups * kLanes;
    const int k = member ? lane % kLanes : 0, base = lane - k, row = member ? k - kFirstRow : -1;
    const unsigned int group = member ? ((1u << kLanes) - 1u) << base : 0u;
    const numb h = p.h;
    for (;;) {
        const long long first = warp_fetch(p.counter, lane, (unsigned long long)p.groups);
        if (first >= p.total) return;
        const long long at = first + lane / kLanes;
        bool live = member && at < p.total;
        const bool mine = live;
        const long long kidx = p.cell_offset + (at < p.total ? at : p.total - 1);
        numb x[UCB_NX], a[UCB_NV];  // x: this lane's trajectory
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) x[i] = p.ic[i];
#pragma unroll
        for (int i = 0; i < UCB_NV; ++i) a[i] = p.vals[i];
        apply_sweep(cell_axes(kidx, p.n_pts), p.axis0, p.axis1, x, a);
        numb z[UCB_NX];  // this lane's row
        {
            Rng st;
            rng_init(1234567891ULL, (unsigned long long)kidx, 0ULL, &st);
#pragma unroll
            for (int j = 0; j < UCB_NX; ++j) {
                numb r[UCB_NX];
                numb zPower = 0;
#pragma unroll
                for (int i = 0; i < UCB_NX; ++i) {
                    r[i] = rng_uniform(&st) - 0.5;
                    zPower += r[i] * r[i];
                }
                zPower = sqrt(zPower);
#pragma unroll
                for (int i = 0; i < UCB_NX; ++i)
                    if (j == row || (j == 0 && row < 0)) z[i] = r[i] / zPower;
            }
        }
        const Stepper st(h);
        long long steps = 0;  // of the cell, counted by all its lanes
        if (loop_single<false>(st, x, a, h, p.skip, p.maxv, steps) == 0) live = false;
#ifdef UCB_LS_FIXED_TANGENT
        double za[UCB_NX], zb[UCB_NX], dens, sum = 0;
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) za[i] = (double)z[i];
        group_gs(za, zb, dens, row, base);
        numb v[1][UCB_NX];
#pragma unroll
        for (int i = 0; i < UCB_NX; ++i) v[0][i] = (numb)zb[i];
        for (int b = 0; b < p.n_blocks; ++b) {
            if (!__any_sync(full, live)) break;
            long long own = 0;
            const int r = loop_tangents<1>(x, v, a, h, p.nt_steps, p.maxv, own);
            const unsigned int bad = __ballot_sync(full, r == 0);
            if (bad) {  // the count of the lane that stopped first
                long long least = own;
#pragma unroll
                for (int j = 0; j < kLanes; ++j) {
                    const long long o = __shfl_sync(full, own, base + j);
                    least = o < least ? o : least;
                }
                own = least;
            }
            if (live) steps += own;
            if (bad & group) live = false;
#pragma unroll
            for (int i = 0; i < UCB_NX; ++i) za[i] = (double)v[0][i];
            group_gs(za, zb, dens, row, base);
#pragma unroll
            for (int i = 0; i < UCB_NX; ++i) v[0][i] = (numb)zb[i];
            if (live) sum += log(dens);
        }
        const double out = live ? sum / (double)p.tmax : 999.0;
#else
        numb zb[UCB_NX], dens, sum = 0;
        group_gs(z, zb, dens, row, base);
        if (row >= 0) {
#pragma unroll
            for (int i = 0; i < UCB_NX; ++i) x[i] = zb[i] * p.eps + x[i];
        }
        for (int b = 0; b < p.n_blocks; ++b) {
            if (!__any_sync(full, live)) break;
#ifdef UCB_NT
            {
                const int r = run_nt(st, x, a, h, p.maxv);
                const unsigned int bad = __ballot_sync(full, r == 0);
                const bool stop = (bad & group) != 0;
                if (live) steps += (UCB_NX + 1) * (stop ? 1 : UCB_NT + UCB_EXTRA_STEP);
                if (stop) live = false;
            }
#else
            for (long long i0 = 0; i0 < p.nt_steps; i0 += kCheckInterval) {
                const int n = (p.nt_steps - i0 < kCheckInterval) ? (int)(p.nt_steps - i0) : kCheckInterval;
                const int r = run_single<true>(st, x, a, h, n, p.maxv);
                const unsigned int bad = __ballot_sync(full, r == 0);
                const bool stop = (bad & group) != 0;
                if (live) steps += (UCB_NX + 1) * (stop ? 1 : n);
                if (stop) live = false;
            }
#if UCB_EXTRA_STEP
            run_single<false>(st, x, a, h, 1, p.maxv);
            if (live) steps += UCB_NX + 1;
#endif
#endif
            numb xs[UCB_NX], d[UCB_NX];
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) {
                xs[l] = __shfl_sync(full, x[l], base);
                d[l] = x[l] - xs[l];
            }
            group_gs(d, zb, dens, row, base);
            if (row >= 0) {
                sum += log(dens / p.eps);
#pragma unroll
                for (int l = 0; l < UCB_NX; ++l) x[l] = (numb)(xs[l] + zb[l] * p.eps);
            }
        }
        const double out = live ? (double)(sum / p.tmax) : 999.0;
#endif
        const unsigned int bad = __ballot_sync(full, mine && row >= 0 && (out == 999.0 || out == -999.0));
        if (mine) {
            const long long cell = ls_out_cell(p, kidx);
#if UCB_DIM == 2
            const long long plane = (long long)p.n_pts * p.n_pts;
#else
            const long long plane = p.n_pts;
#endif
            if (row >= 0) p.out_values[row * plane + cell] = out;
            if (k == 0) {
                p.out_flags[cell] = (bad & group) ? -1 : 1;
                if (p.out_cell_steps) p.out_cell_steps[cell] = steps;
                ns += steps;
            }
        }
    }
}
#endif  // UCB_LS_GROUP
#endif  // UCB_LS_FIXED

#if defined(UCB_LS_DP5)
#ifndef UCB_GS_BUDGET
#define UCB_GS_BUDGET 20.0
#endif
// Dormand-Prince 5(4) coefficients (Dormand & Prince, J. Comp. Appl. Math. 6, 1980).
#define DP_A21 (1.0 / 5.0)
#define DP_A31 (3.0 / 40.0)
#define DP_A32 (9.0 / 40.0)
#define DP_A41 (44.0 / 45.0)
#define DP_A42 (-56.0 / 15.0)
#define DP_A43 (32.0 / 9.0)
#define DP_A51 (19372.0 / 6561.0)
#define DP_A52 (-25360.0 / 2187.0)
#define DP_A53 (64448.0 / 6561.0)
#define DP_A54 (-212.0 / 729.0)
#define DP_A61 (9017.0 / 3168.0)
#define DP_A62 (-355.0 / 33.0)
#define DP_A63 (46732.0 / 5247.0)
#define DP_A64 (49.0 / 176.0)
#define DP_A65 (-5103.0 / 18656.0)
#define DP_B1 (35.0 / 384.0)
#define DP_B3 (500.0 / 1113.0)
#define DP_B4 (125.0 / 192.0)
#define DP_B5 (-2187.0 / 6784.0)
#define DP_B6 (11.0 / 84.0)
#define DP_E1 (71.0 / 57600.0)
#define DP_E3 (-71.0 / 16695.0)
#define DP_E4 (71.0 / 1920.0)
#define DP_E5 (-17253.0 / 339200.0)
#define DP_E6 (22.0 / 525.0)
#define DP_E7 (-1.0 / 40.0)

// Modified Gram-Schmidt on the rows of V; log of the norms added to acc (FP64).
__device__ __forceinline__ bool mgs(numb (*V)[UCB_NX], double* acc) {
#pragma unroll
    for (int k = 0; k < UCB_NX; ++k) {
#pragma unroll
        for (int j = 0; j < k; ++j) {
            double d = 0;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) d = fma((double)V[k][l], (double)V[j][l], d);
            const numb dn = (numb)d;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) V[k][l] = fma(-dn, V[j][l], V[k][l]);
        }
        double n2 = 0;
#pragma unroll
        for (int l = 0; l < UCB_NX; ++l) n2 = fma((double)V[k][l], (double)V[k][l], n2);
        const double nrm = sqrt(n2);
        if (!(nrm > 0) || !isfinite(nrm)) return false;
        acc[k] += log(nrm);
        const numb inv = (numb)(1.0 / nrm);
#pragma unroll
        for (int l = 0; l < UCB_NX; ++l) V[k][l] *= inv;
    }
    return true;
}

// The Butcher rows scaled by the step once per attempt, so that every stage point is a
// chain of fused multiply-adds from the base point: x + sum_j (h a_ij) k_j.
struct Dp5Coef {
    numb c21, c31, c32, c41, c42, c43, c51, c52, c53, c54, c61, c62, c63, c64, c65, b1, b3, b4, b5, b6;
    double e1, e3, e4, e5, e6, e7;  // h times the error weights (FP64: the error norm is FP64)
};

__device__ __forceinline__ Dp5Coef dp5_coef(numb hn, double h) {
    Dp5Coef c;
    c.c21 = hn * (numb)DP_A21;
    c.c31 = hn * (numb)DP_A31; c.c32 = hn * (numb)DP_A32;
    c.c41 = hn * (numb)DP_A41; c.c42 = hn * (numb)DP_A42; c.c43 = hn * (numb)DP_A43;
    c.c51 = hn * (numb)DP_A51; c.c52 = hn * (numb)DP_A52; c.c53 = hn * (numb)DP_A53; c.c54 = hn * (numb)DP_A54;
    c.c61 = hn * (numb)DP_A61; c.c62 = hn * (numb)DP_A62; c.c63 = hn * (numb)DP_A63; c.c64 = hn * (numb)DP_A64;
    c.c65 = hn * (numb)DP_A65;
    c.b1 = hn * (numb)DP_B1; c.b3 = hn * (numb)DP_B3; c.b4 = hn * (numb)DP_B4; c.b5 = hn * (numb)DP_B5;
    c.b6 = hn * (numb)DP_B6;
    c.e1 = h * DP_E1; c.e3 = h * DP_E3; c.e4 = h * DP_E4; c.e5 = h * DP_E5; c.e6 = h * DP_E6; c.e7 = h * DP_E7;
    return c;
}

// sum_i (e_i / s_i)^2 for s_i > 0, one division per group of four: 1 / (s0 s1 s2 s3) times
// the other three scales gives each 1 / s_i. A group whose product leaves the normal range
// (scales below 1e-75 or above 1e75) divides component by component.
template <int N>
__device__ __forceinline__ double scaled_sum_sq(const double* e, const double* s) {
    double acc = 0.0;
#pragma unroll
    for (int g = 0; g < N; g += 4) {
        const int m = (N - g) < 4 ? (N - g) : 4;
        if (m == 1) {
            const double q = e[g] / s[g];
            acc = fma(q, q, acc);
            continue;
        }
        double pre[4], suf[4];  // products of the scales before / after position i
        pre[0] = 1.0;
#pragma unroll
        for (int i = 1; i < m; ++i) pre[i] = pre[i - 1] * s[g + i - 1];
        suf[m - 1] = 1.0;
#pragma unroll
        for (int i = m - 2; i >= 0; --i) suf[i] = suf[i + 1] * s[g + i + 1];
        const double prod = pre[m - 1] * s[g + m - 1];
        if (prod > 1e-300 && prod < 1e300) {
            const double r = 1.0 / prod;
#pragma unroll
            for (int i = 0; i < m; ++i) {
                const double q = e[g + i] * (r * (pre[i] * suf[i]));
                acc = fma(q, q, acc);
            }
        } else {
#pragma unroll
            for (int i = 0; i < m; ++i) {
                const double q = e[g + i] / s[g + i];
                acc = fma(q, q, acc);
            }
        }
    }
    return acc;
}

// Step-size factor 0.9 err^(-1/5) of the controller, from err^2. A heuristic factor (it is
// clamped to [0.2, facmax] next), so the power is taken in FP32 (relative error ~1e-6),
// off the FP64 pipe; err^2 below the FP32 range gives +inf (clamped to facmax) and above it
// 0 (clamped to 0.2), as the FP64 power would after clamping.
__device__ __forceinline__ double dp5_factor(double err2) {
    return 0.9 * (double)__powf((float)err2, -0.1f);
}

// One DP5 step of the state: stage points X2..X6, the 5th-order solution xn and its
// derivative k7 (FSAL), and the sum of squared scaled errors of the embedded 4th-order
// difference.
struct Dp5State {
    numb X[6][UCB_NX];  // stage points X1 (= x) .. X6
    numb k1[UCB_NX], k7[UCB_NX], xn[UCB_NX];
};

__device__ __forceinline__ double dp5_state_step(Dp5State& S, const numb* a, const Dp5Coef& c, double rtol,
                                                 double atol) {
    numb k2[UCB_NX], k3[UCB_NX], k4[UCB_NX], k5[UCB_NX], k6[UCB_NX];
    const numb* x = S.X[0];
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) S.X[1][i] = fma(c.c21, S.k1[i], x[i]);
    ucb_rhs(S.X[1], a, k2);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) S.X[2][i] = fma(c.c32, k2[i], fma(c.c31, S.k1[i], x[i]));
    ucb_rhs(S.X[2], a, k3);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) S.X[3][i] = fma(c.c43, k3[i], fma(c.c42, k2[i], fma(c.c41, S.k1[i], x[i])));
    ucb_rhs(S.X[3], a, k4);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i)
        S.X[4][i] = fma(c.c54, k4[i], fma(c.c53, k3[i], fma(c.c52, k2[i], fma(c.c51, S.k1[i], x[i]))));
    ucb_rhs(S.X[4], a, k5);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i)
        S.X[5][i] = fma(c.c65, k5[i], fma(c.c64, k4[i], fma(c.c63, k3[i], fma(c.c62, k2[i], fma(c.c61, S.k1[i], x[i])))));
    ucb_rhs(S.X[5], a, k6);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i)
        S.xn[i] = fma(c.b6, k6[i], fma(c.b5, k5[i], fma(c.b4, k4[i], fma(c.b3, k3[i], fma(c.b1, S.k1[i], x[i])))));
    ucb_rhs(S.xn, a, S.k7);
    double e[UCB_NX], sc[UCB_NX];
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) {
        e[i] = fma(c.e7, (double)S.k7[i], fma(c.e6, (double)k6[i], fma(c.e5, (double)k5[i],
               fma(c.e4, (double)k4[i], fma(c.e3, (double)k3[i], c.e1 * (double)S.k1[i])))));
        sc[i] = fma(rtol, fmax(fabs((double)x[i]), fabs((double)S.xn[i])), atol);
    }
    return scaled_sum_sq<UCB_NX>(e, sc);
}

// One tangent vector through the same DP5 stages (v' = J(x) v with J at the stored stage
// points): writes the 5th-order vn and returns its sum of squared scaled errors.
__device__ __forceinline__ double dp5_tangent_step(const Dp5State& S, const numb* a, const Dp5Coef& c, double rtol,
                                                   double atol, const numb* v, numb* vn) {
    numb L1[UCB_NX], L2[UCB_NX], L3[UCB_NX], L4[UCB_NX], L5[UCB_NX], L6[UCB_NX], vt[UCB_NX];
    ucb_jvp(S.X[0], a, v, L1);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) vt[i] = fma(c.c21, L1[i], v[i]);
    ucb_jvp(S.X[1], a, vt, L2);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) vt[i] = fma(c.c32, L2[i], fma(c.c31, L1[i], v[i]));
    ucb_jvp(S.X[2], a, vt, L3);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) vt[i] = fma(c.c43, L3[i], fma(c.c42, L2[i], fma(c.c41, L1[i], v[i])));
    ucb_jvp(S.X[3], a, vt, L4);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i)
        vt[i] = fma(c.c54, L4[i], fma(c.c53, L3[i], fma(c.c52, L2[i], fma(c.c51, L1[i], v[i]))));
    ucb_jvp(S.X[4], a, vt, L5);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i)
        vt[i] = fma(c.c65, L5[i], fma(c.c64, L4[i], fma(c.c63, L3[i], fma(c.c62, L2[i], fma(c.c61, L1[i], v[i])))));
    ucb_jvp(S.X[5], a, vt, L6);
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i)
        vn[i] = fma(c.b6, L6[i], fma(c.b5, L5[i], fma(c.b4, L4[i], fma(c.b3, L3[i], fma(c.b1, L1[i], v[i])))));
    ucb_jvp(S.xn, a, vn, L2);  // L7, reusing L2's registers
    double e[UCB_NX], sc[UCB_NX];
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) {
        e[i] = fma(c.e7, (double)L2[i], fma(c.e6, (double)L6[i], fma(c.e5, (double)L5[i],
               fma(c.e4, (double)L4[i], fma(c.e3, (double)L3[i], c.e1 * (double)L1[i])))));
        sc[i] = fma(rtol, fmax(fabs((double)v[i]), fabs((double)vn[i])), atol);
    }
    return scaled_sum_sq<UCB_NX>(e, sc);
}

// An adaptive cell whose remaining horizon needs more than this many times its remaining
// step attempts (at the current step size) is given up as escaping.
constexpr double kEscapeFactor = 8.0;

__device__ __forceinline__ void ls_cell_dp5(const UcbLsParams& p, long long kidx, long long& ns) {
    double outv[UCB_NX];
    const CellAxes c = cell_axes(kidx, p.n_pts);
    Dp5State S;
    numb a[UCB_NV];
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) S.X[0][i] = p.ic[i];
#pragma unroll
    for (int i = 0; i < UCB_NV; ++i) a[i] = p.vals[i];
    apply_sweep(c, p.axis0, p.axis1, S.X[0], a);
#ifdef UCB_KAHAN_CLOCK
    // the clock of an FP32 build is set from the FP64 time after every accepted step
    const double clock0 = (double)S.X[0][UCB_CLOCK_VAR];
#endif
    numb V[UCB_NX][UCB_NX];
    {
        Rng st;
        rng_init(1234567891ULL, (unsigned long long)kidx, 0ULL, &st);
#pragma unroll
        for (int j = 0; j < UCB_NX; ++j)
#pragma unroll
            for (int i = 0; i < UCB_NX; ++i) V[j][i] = rng_uniform(&st) - 0.5;
    }
    double acc[UCB_NX], junk[UCB_NX];
#pragma unroll
    for (int k = 0; k < UCB_NX; ++k) acc[k] = junk[k] = 0;
    bool ok = mgs(V, junk);
    // The transient [0, transient) moves the state only; tangents are measured over
    // [transient, transient + t_end] with MGS every gs_every accepted steps and at the end.
    double t = 0.0;
    const double t_stop = (double)p.transient + p.t_end;
    double h = p.h0, facmax = 5.0;
    int since_gs = 0;
    double t_gs = 0.0, t_meas = 0.0, spread = 1e300;  // spread: running lambda_1 - lambda_N
    bool measuring = !((double)p.transient > 0);
    long long attempts = 0, accepted = 0;
    ucb_rhs(S.X[0], a, S.k1);
    while (ok && t < t_stop) {
        if (++attempts > p.max_steps) { ok = false; break; }
        // a cell can take millions of attempts: a cancelled run abandons it
        if ((attempts & 4095) == 0 && run_cancelled()) { ok = false; break; }
        const double t_target = measuring ? t_stop : (double)p.transient;
        bool last = false;
        if (t + h >= t_target) { h = t_target - t; last = true; }
        const Dp5Coef cf = dp5_coef((numb)h, h);
        const double ex2 = dp5_state_step(S, a, cf, p.rtol, p.atol);
        ns += 1;
        // err^2: the mean of the squared scaled errors (the RMS norm, squared)
        double err2 = ex2 * (1.0 / UCB_NX);
        numb Vn[UCB_NX][UCB_NX];
        if (err2 <= 1.0 && measuring) {
            double ev2 = 0;
#pragma unroll
            for (int k = 0; k < UCB_NX; ++k) ev2 += dp5_tangent_step(S, a, cf, p.rtol, p.atol, V[k], Vn[k]);
            err2 = (ex2 + ev2) * (1.0 / (UCB_NX + UCB_NX * UCB_NX));
        }
        if (!isfinite(err2)) { ok = false; break; }
        if (err2 <= 1.0) {
            if (measuring) {
#pragma unroll
                for (int k = 0; k < UCB_NX; ++k)
#pragma unroll
                    for (int i = 0; i < UCB_NX; ++i) V[k][i] = Vn[k][i];
            }
            const double t_new = last ? t_target : t + h;
            if (measuring) t_gs += t_new - t;
            t = t_new;
#pragma unroll
            for (int i = 0; i < UCB_NX; ++i) { S.X[0][i] = S.xn[i]; S.k1[i] = S.k7[i]; }
#ifdef UCB_KAHAN_CLOCK
            S.X[0][UCB_CLOCK_VAR] = (numb)fma((double)UCB_CLOCK_RATE, t, clock0);
#endif
            if (diverged(S.X[0], p.maxv)) { ok = false; break; }
            // Escape test, every 16 accepted steps: at the step size just taken the rest of the
            // horizon would need more than kEscapeFactor times the attempts left. Such a cell
            // (in practice one escaping towards max_value through ever stiffer, ever smaller
            // steps) would end at the attempt cap with the same flag; it ends here instead.
            if ((++accepted & 15) == 0 && t_stop - t > kEscapeFactor * h * (double)(p.max_steps - attempts)) {
                ok = false;
                break;
            }
            if (measuring && (++since_gs >= p.gs_every || last || t_gs * spread > UCB_GS_BUDGET)) {
                ok = mgs(V, acc);
                since_gs = 0;
                t_meas += t_gs;
                t_gs = 0.0;
                spread = fmax(0.0, (acc[0] - acc[UCB_NX - 1]) / t_meas);
            }
            if (last && !measuring) measuring = true;
            const double fac = (err2 > 0) ? dp5_factor(err2) : facmax;
            h *= fmin(facmax, fmax(0.2, fac));
            facmax = 5.0;
        } else {
            h *= fmax(0.2, dp5_factor(err2));
            facmax = 2.0;
            if (!(h > 1e-14)) { ok = false; break; }
        }
    }
#pragma unroll
    for (int k = 0; k < UCB_NX; ++k) outv[k] = ok ? acc[k] / p.t_end : 999.0;
    ls_store(p, kidx, outv);
}

#if defined(UCB_LS_GROUP)
// mgs() over the group's rows (lane k holds row k), for groups with `act`; the log of the
// norms added to acc. False if the group's rows are not independent and finite.
__device__ __forceinline__ bool group_mgs(numb* v, double& acc, bool act, int k, int base, unsigned int group) {
    double norm = 1.0;
    bool good = true;
#pragma unroll
    for (int j = 0; j < UCB_NX; ++j) {
        if (act && k == j) {
            double n2 = 0;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) n2 = fma((double)v[l], (double)v[l], n2);
            norm = sqrt(n2);
            good = norm > 0 && isfinite(norm);
            const numb inv = (numb)(1.0 / norm);
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) v[l] *= inv;
        }
        __syncwarp();
        numb w[UCB_NX];
#pragma unroll
        for (int l = 0; l < UCB_NX; ++l) w[l] = __shfl_sync(0xFFFFFFFFu, v[l], base + j);
        if (act && k > j) {
            double d = 0;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) d = fma((double)v[l], (double)w[l], d);
            const numb dn = (numb)d;
#pragma unroll
            for (int l = 0; l < UCB_NX; ++l) v[l] = fma(-dn, w[l], v[l]);
        }
    }
    const unsigned int ok = __ballot_sync(0xFFFFFFFFu, good);
    if (act) acc += log(norm);
    return (ok & group) == group;
}

// ls_cell_dp5 with a cell on UCB_NX lanes, one tangent vector each (the same values and order of
// operations): every lane of a group takes the state's step and its own vector's, the error
// sums and Gram-Schmidt rows are exchanged by shuffles. An attempt is then two chains of
// stages instead of N + 1 and its registers fall from 254 to 204 (FP64), so a map of few cells,
// which lasts as long as its slowest ones, ends sooner; a group takes its next cell as soon as
// it is done. The exchanges are taken by the whole warp; what a group does between them
// depends on values that all its lanes hold. (The tangent's stages beside the state's, before
// its step is accepted, gave the same times.) B200, 96^2 hyper-chaotic Rossler, t_end 50, FP64:
// 68 -> 46 ms; where each form runs and its times: ls_groups of ucb_ls.cpp.
__device__ __forceinline__ void ls_groups_dp5(const UcbLsParams& p, long long& ns) {
    const unsigned int full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const bool member = lane < p.groups * UCB_NX;
    const int k = member ? lane % UCB_NX : 0, base = lane - k;
    const unsigned int group = member ? ((1u << UCB_NX) - 1u) << base : 0u;
    // the group's cell, the same in all its lanes but for the vector and its log sum
    Dp5State S;
    numb a[UCB_NV], v[UCB_NX];
    double acc = 0, t = 0, h = 0, facmax = 5.0, t_gs = 0, t_meas = 0, spread = 0, clock0 = 0;
    long long kidx = 0, attempts = 0, accepted = 0, cell_ns = 0;
    int since_gs = 0;
    bool busy = false, drained = !member, measuring = false, ok = true;
    const double t_stop = (double)p.transient + p.t_end;
#pragma unroll
    for (int i = 0; i < UCB_NX; ++i) v[i] = 0;
    for (;;) {
        const bool need = !busy && !drained;
        const unsigned int asking = __ballot_sync(full, need && k == 0);
        if (asking) {
            unsigned long long first = 0;
            if (lane == 0) {
                const bool stop = run_cancelled();
                first = atomicAdd(p.counter, (unsigned long long)__popc(asking));
                if (stop) first = 0x7fffffffffffffffULL;
            }
            first = __shfl_sync(full, first, 0);
            const unsigned long long i = first + __popc(asking & ((1u << base) - 1u));
            bool fresh = false;
            if (need) {
                if (i >= (unsigned long long)p.total) {
                    drained = true;
                } else {
                    fresh = busy = true;
                    kidx = p.cell_offset + (long long)i;
                    const CellAxes c = cell_axes(kidx, p.n_pts);
#pragma unroll
                    for (int j = 0; j < UCB_NX; ++j) S.X[0][j] = p.ic[j];
#pragma unroll
                    for (int j = 0; j < UCB_NV; ++j) a[j] = p.vals[j];
                    apply_sweep(c, p.axis0, p.axis1, S.X[0], a);
#ifdef UCB_KAHAN_CLOCK
                    clock0 = (double)S.X[0][UCB_CLOCK_VAR];
#endif
                    Rng st;
                    rng_init(1234567891ULL, (unsigned long long)kidx, 0ULL, &st);
#pragma unroll
                    for (int j = 0; j < UCB_NX; ++j)
#pragma unroll
                        for (int l = 0; l < UCB_NX; ++l) {
                            const numb u = rng_uniform(&st) - 0.5;
                            if (j == k) v[l] = u;
                        }
                    acc = t = t_gs = t_meas = 0.0;
                    spread = 1e300;
                    h = p.h0;
                    facmax = 5.0;
                    attempts = accepted = cell_ns = 0;
                    since_gs = 0;
                    measuring = !((double)p.transient > 0);
                    ucb_rhs(S.X[0], a, S.k1);
                }
            }
            double junk = 0;
            const bool good = group_mgs(v, junk, fresh, k, base, group);
            if (fresh) ok = good;
        }
        if (!__any_sync(full, busy)) break;
        // a cell can take millions of attempts: a cancelled run abandons it
        if (__any_sync(full, busy && (attempts & 4095) == 4095)) {
            const int stop = __shfl_sync(full, (int)run_cancelled(), 0);
            if (stop && (attempts & 4095) == 4095) ok = false;
        }
        // one attempt of every group that goes on
        bool tried = false, tangent = false, last = false;
        double ex2 = 0, err2 = 0, e_own = 0, t_target = 0;
        numb vn[UCB_NX];
        if (busy && ok && t < t_stop) {
            if (++attempts > p.max_steps) {
                ok = false;
            } else {
                tried = true;
                t_target = measuring ? t_stop : (double)p.transient;
                if (t + h >= t_target) { h = t_target - t; last = true; }
                const Dp5Coef cf = dp5_coef((numb)h, h);
                ex2 = dp5_state_step(S, a, cf, p.rtol, p.atol);
                cell_ns += 1;
                // err^2: the mean of the squared scaled errors (the RMS norm, squared)
                err2 = ex2 * (1.0 / UCB_NX);
                tangent = err2 <= 1.0 && measuring;
                if (tangent) e_own = dp5_tangent_step(S, a, cf, p.rtol, p.atol, v, vn);
            }
        }
        if (__any_sync(full, tangent)) {
            double ev2 = 0;
#pragma unroll
            for (int j = 0; j < UCB_NX; ++j) ev2 += __shfl_sync(full, e_own, base + j);
            if (tangent) err2 = (ex2 + ev2) * (1.0 / (UCB_NX + UCB_NX * UCB_NX));
        }
        bool gs = false;
        if (tried) {
            if (!isfinite(err2)) {
                ok = false;
            } else if (err2 <= 1.0) {
                if (measuring) {
#pragma unroll
                    for (int i = 0; i < UCB_NX; ++i) v[i] = vn[i];
                }
                const double t_new = last ? t_target : t + h;
                if (measuring) t_gs += t_new - t;
                t = t_new;
#pragma unroll
                for (int i = 0; i < UCB_NX; ++i) { S.X[0][i] = S.xn[i]; S.k1[i] = S.k7[i]; }
#ifdef UCB_KAHAN_CLOCK
                S.X[0][UCB_CLOCK_VAR] = (numb)fma((double)UCB_CLOCK_RATE, t, clock0);
#endif
                if (diverged(S.X[0], p.maxv)) {
                    ok = false;
                } else if ((++accepted & 15) == 0 &&
                           t_stop - t > kEscapeFactor * h * (double)(p.max_steps - attempts)) {
                    ok = false;  // the escape test of ls_cell_dp5
                } else {
                    gs = measuring && (++since_gs >= p.gs_every || last || t_gs * spread > UCB_GS_BUDGET);
                    if (last && !measuring) measuring = true;
                    const double fac = (err2 > 0) ? dp5_factor(err2) : facmax;
                    h *= fmin(facmax, fmax(0.2, fac));
                    facmax = 5.0;
                }
            } else {
                h *= fmax(0.2, dp5_factor(err2));
                facmax = 2.0;
                if (!(h > 1e-14)) ok = false;
            }
        }
        if (__any_sync(full, gs)) {
            const bool good = group_mgs(v, acc, gs, k, base, group);
            const double a0 = __shfl_sync(full, acc, base), an = __shfl_sync(full, acc, base + UCB_NX - 1);
            if (gs) {
                ok = good;
                since_gs = 0;
                t_meas += t_gs;
                t_gs = 0.0;
                spread = fmax(0.0, (a0 - an) / t_meas);
            }
        }
        const bool done = busy && (!ok || !(t < t_stop));
        if (__any_sync(full, done)) {
            const double out = ok ? acc / p.t_end : 999.0;
            const unsigned int bad = __ballot_sync(full, done && (out == 999.0 || out == -999.0));
            if (done) {
                const long long cell = ls_out_cell(p, kidx);
#if UCB_DIM == 2
                const long long plane = (long long)p.n_pts * p.n_pts;
#else
                const long long plane = p.n_pts;
#endif
                p.out_values[k * plane + cell] = out;
                if (k == 0) {
                    p.out_flags[cell] = (bad & group) ? -1 : 1;
                    if (p.out_cell_steps) p.out_cell_steps[cell] = cell_ns;
                    ns += cell_ns;
                }
                busy = false;
            }
        }
    }
}
#endif  // UCB_LS_GROUP
#endif  // UCB_LS_DP5

}  // namespace ucbdev

extern "C" __global__ void UCB_LAUNCH_BOUNDS ucb_ls_kernel(const UcbLsParams p) {
    const int lane = threadIdx.x & 31;
    long long ns = 0;
#if defined(UCB_LS_GROUP)
#if defined(UCB_LS_DP5)
    ucbdev::ls_groups_dp5(p, ns);
#else
    ucbdev::ls_groups_fixed(p, ns);
#endif
    ucbdev::warp_add_steps(p.steps, ns, lane);
    return;
#endif
    for (;;) {
        const long long base = ucbdev::warp_fetch(p.counter, lane);
        if (base >= p.total) break;
        const long long i = base + lane;
        if (i < p.total) {
            const long long ns0 = ns;
#if defined(UCB_LS_DP5)
            ucbdev::ls_cell_dp5(p, p.cell_offset + i, ns);
#else
            ucbdev::ls_cell_fixed(p, p.cell_offset + i, ns);
#endif
            if (p.out_cell_steps) p.out_cell_steps[ucbdev::ls_out_cell(p, p.cell_offset + i)] = ns - ns0;
        }
    }
    ucbdev::warp_add_steps(p.steps, ns, lane);
}
