// tridiag.cuh -- device helpers for the small symmetric tridiagonal
// eigenproblems of the Krylov solvers (Sturm multisection, last eigenvector
// component, pivoted tridiagonal solve for inverse iteration).
#pragma once
#include <cuda_runtime.h>

namespace tnb {
namespace {

// Number of eigenvalues of the symmetric tridiagonal (a, b) below x: the sign
// changes of p_0 = 1, p_k = (a_{k-1} - x) p_{k-1} - b_{k-2}^2 p_{k-2}, the
// leading principal minors of T - x.  The three-term recurrence needs no
// division (the ratio form q_k = p_k / p_{k-1} spends an FP64 division, a long
// serial latency, on every step); the pair is rescaled to stay in range.  A
// zero minor takes its predecessor's sign, as the ratio form's +pivmin does.
__device__ int sturm_count(int n, const double* a, const double* b, double x) {
    double pm = 1.0, p = a[0] - x;
    bool neg = p < 0;
    int cnt = neg;
    for (int i = 1; i < n; ++i) {
        const double pn = fma(a[i] - x, p, -(b[i - 1] * b[i - 1]) * pm);
        pm = p;
        p = pn;
        const bool ng = p < 0 ? true : (p > 0 ? false : neg);
        cnt += (ng != neg);
        neg = ng;
        const double mx = fmax(fabs(p), fabs(pm));
        if (mx > 1e150) {
            p *= 1e-150;
            pm *= 1e-150;
        } else if (mx < 1e-150 && mx > 0) {
            p *= 1e150;
            pm *= 1e150;
        }
    }
    return cnt;
}

// k-th smallest eigenvalue by block-wide multisection: every round each
// thread evaluates one Sturm count, shrinking the bracket by blockDim+1.
__device__ double block_eig_k(int n, const double* a, const double* b, int k) {
    __shared__ double s_lo, s_hi;
    double lo = a[0], hi = a[0];
    for (int i = 0; i < n; ++i) {
        double r = (i > 0 ? fabs(b[i - 1]) : 0.0) + (i < n - 1 ? fabs(b[i]) : 0.0);
        lo = fmin(lo, a[i] - r);
        hi = fmax(hi, a[i] + r);
    }
    double scale = fmax(fabs(lo), fabs(hi));
    lo -= 1e-14 * scale + 1e-300;
    hi += 1e-14 * scale + 1e-300;
    const int T = blockDim.x;
    // the trial points' fractions of the bracket, divided once rather than every round
    const double inv = 1.0 / (double)(T + 1), frac = (double)(threadIdx.x + 1) * inv;
    for (int round = 0; round < 12; ++round) {
        double x = lo + (hi - lo) * frac;
        int ok = sturm_count(n, a, b, x) <= k;
        int cnt = __syncthreads_count(ok);
        if (threadIdx.x == 0) {
            double nlo = cnt > 0 ? lo + (hi - lo) * ((double)cnt * inv) : lo;
            double nhi = cnt < T ? lo + (hi - lo) * ((double)(cnt + 1) * inv) : hi;
            s_lo = nlo;
            s_hi = nhi;
        }
        __syncthreads();
        lo = s_lo;
        hi = s_hi;
        __syncthreads();
        if (hi - lo <= 2.2e-16 * fmax(fabs(lo), fabs(hi)) + 1e-300) break;
    }
    return 0.5 * (lo + hi);
}

// |last component| of the normalised eigenvector of T for eigenvalue th:
// y_n^2 = p_{n-1}(th) / p_n'(th) with the monic characteristic polynomials of
// the leading blocks (scaled recurrences; the ratio is scale-free).
__device__ double last_component(int n, const double* a, const double* b, double th) {
    if (n == 1) return 1.0;
    double pm2 = 1.0, pm1 = th - a[0];  // p0, p1
    double dm2 = 0.0, dm1 = 1.0;        // p0', p1'
    for (int k = 2; k <= n; ++k) {
        double bb = b[k - 2] * b[k - 2];
        double p = (th - a[k - 1]) * pm1 - bb * pm2;
        double dp = pm1 + (th - a[k - 1]) * dm1 - bb * dm2;
        pm2 = pm1; pm1 = p;
        dm2 = dm1; dm1 = dp;
        double mx = fmax(fmax(fabs(pm1), fabs(pm2)), fmax(fabs(dm1), fabs(dm2)));
        if (mx > 1e150) { pm1 *= 1e-150; pm2 *= 1e-150; dm1 *= 1e-150; dm2 *= 1e-150; }
        else if (mx < 1e-150 && mx > 0) { pm1 *= 1e150; pm2 *= 1e150; dm1 *= 1e150; dm2 *= 1e150; }
    }
    // after the loop: pm2 = p_{n-1}, dm1 = p_n'
    double r = (dm1 != 0.0) ? pm2 / dm1 : 1.0;
    return sqrt(fabs(r));
}

// Tridiagonal (T - shift) y = rhs with partial pivoting (dlagtf/dlagts style).
__device__ void tri_solve(int n, const double* a, const double* b, double shift, double pivmin, double* rhs,
                          double* dl, double* dd, double* du, double* du2, int* piv) {
    for (int i = 0; i < n; ++i) dd[i] = a[i] - shift;
    for (int i = 0; i < n - 1; ++i) { dl[i] = b[i]; du[i] = b[i]; }
    for (int i = 0; i < n - 1; ++i) {
        du2[i] = 0;
        if (fabs(dd[i]) >= fabs(dl[i])) {
            piv[i] = 0;
            if (fabs(dd[i]) < pivmin) dd[i] = (dd[i] < 0 ? -pivmin : pivmin);
            double f = dl[i] / dd[i];
            dl[i] = f;
            dd[i + 1] -= f * du[i];
        } else {
            piv[i] = 1;
            double f = dd[i] / dl[i];
            dd[i] = dl[i];
            dl[i] = f;
            double t = du[i];
            du[i] = dd[i + 1];
            dd[i + 1] = t - f * du[i];
            if (i < n - 2) { du2[i] = du[i + 1]; du[i + 1] = -f * du[i + 1]; }
        }
    }
    if (fabs(dd[n - 1]) < pivmin) dd[n - 1] = (dd[n - 1] < 0 ? -pivmin : pivmin);
    for (int i = 0; i < n - 1; ++i) {
        if (piv[i] == 0) rhs[i + 1] -= dl[i] * rhs[i];
        else { double t = rhs[i]; rhs[i] = rhs[i + 1]; rhs[i + 1] = t - dl[i] * rhs[i]; }
    }
    rhs[n - 1] /= dd[n - 1];
    if (n > 1) rhs[n - 2] = (rhs[n - 2] - du[n - 2] * rhs[n - 1]) / dd[n - 2];
    for (int i = n - 3; i >= 0; --i) rhs[i] = (rhs[i] - du[i] * rhs[i + 1] - du2[i] * rhs[i + 2]) / dd[i];
}

// ---- the same values as sturm_count, last_component and tri_solve, bit for bit, in fewer cycles ----

// sturm_count on rows (a_i, b_{i-1}^2) in shared memory: the same recurrence with four rows'
// loads in flight, signs and ranges read off the high words as integers.  *odd is set
// where a minor is zero or sturm_count would have rescaled (both minors under 1e-150,
// or one over 1e150): the count is then sturm_count's to make.
__device__ __forceinline__ int sturm_count_rows(int n, const double2* rows, double x, bool* odd) {
    constexpr int LOW = 0x20D00000, HIGH = 0x5F100000;  // high words: 2^-498 > 1e-150, 2^498 < 1e150
    double pm = 1.0, p = rows[0].x - x;
    int hs = __double2hiint(p), hp = hs & 0x7fffffff, cnt = (unsigned)hs >> 31;
    int mn1 = hp, mn = 0x7fffffff, mx = 0;
    auto row = [&](double2 r) {
        const double t = r.y * pm;
        pm = p;
        p = fma(r.x - x, p, -t);
        const int h = __double2hiint(p), ha = h & 0x7fffffff, m = max(ha, hp);
        cnt += (unsigned)(h ^ hs) >> 31;
        hs = h;
        hp = ha;
        mn1 = min(mn1, ha);
        mn = min(mn, m);
        mx = max(mx, m);
    };
    int i = 1;
    for (; i + 4 <= n; i += 4) {
        double2 r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) r[q] = rows[i + q];
#pragma unroll
        for (int q = 0; q < 4; ++q) row(r[q]);
    }
    for (; i < n; ++i) row(rows[i]);
    *odd = mn1 == 0 || (n > 1 && (mn < LOW || mx > HIGH));
    return cnt;
}

// last_component on those rows, with the range test afterwards.
__device__ __forceinline__ double last_component_rows(int n, const double2* rows, const double* a, const double* b,
                                                      double th) {
    constexpr int LOW = 0x20D00000, HIGH = 0x5F100000;
    if (n == 1) return 1.0;
    double pm2 = 1.0, pm1 = th - rows[0].x;
    double dm2 = 0.0, dm1 = 1.0;
    int mn = 0x7fffffff, mx = 0;
    auto row = [&](double2 r) {
        const double bb = r.y, ak = r.x;
        double p = (th - ak) * pm1 - bb * pm2;
        double dp = pm1 + (th - ak) * dm1 - bb * dm2;
        const int h = max(max(__double2hiint(p) & 0x7fffffff, __double2hiint(pm1) & 0x7fffffff),
                          max(__double2hiint(dp) & 0x7fffffff, __double2hiint(dm1) & 0x7fffffff));
        pm2 = pm1; pm1 = p;
        dm2 = dm1; dm1 = dp;
        mn = min(mn, h);
        mx = max(mx, h);
    };
    int k = 1;
    for (; k + 4 <= n; k += 4) {
        double2 r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) r[q] = rows[k + q];
#pragma unroll
        for (int q = 0; q < 4; ++q) row(r[q]);
    }
    for (; k < n; ++k) row(rows[k]);
    if (mn < LOW || mx > HIGH) return last_component(n, a, b, th);
    double r = (dm1 != 0.0) ? pm2 / dm1 : 1.0;
    return sqrt(fabs(r));
}

// k-th smallest eigenvalue by multisection in one warp (every lane must call it; a, b in shared memory): 32 of
// those counts per round shrink the bracket 33-fold, so ~11 rounds reach rounding level from the Gershgorin
// interval.  The block version spends 16 warps of one SM on its counts; one warp costs a sixteenth of the issue
// slots for one more round.  rows: scratch of n pairs in shared memory; midway() is called once on the way.
template <class F>
__device__ __forceinline__ double warp_eig_exact(int n, const double* a, const double* b, double2* rows, int k,
                                                 F midway) {
    const int lane = threadIdx.x & 31;
    double lo = a[0], hi = a[0];
    for (int i = lane; i < n; i += 32) {
        const double bp = i > 0 ? b[i - 1] : 0.0;
        const double r = (i > 0 ? fabs(bp) : 0.0) + (i < n - 1 ? fabs(b[i]) : 0.0);
        lo = fmin(lo, a[i] - r);
        hi = fmax(hi, a[i] + r);
        rows[i] = make_double2(a[i], bp * bp);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __syncwarp();
    const double scale = fmax(fabs(lo), fabs(hi));
    lo -= 1e-14 * scale + 1e-300;
    hi += 1e-14 * scale + 1e-300;
    const double inv = 1.0 / 33.0, frac = (double)(lane + 1) * inv;
    bool called = false;
    for (int round = 0; round < 24; ++round) {
        if (round == 6) {
            midway();
            called = true;
        }
        const double x = lo + (hi - lo) * frac;
        bool odd;
        int c = sturm_count_rows(n, rows, x, &odd);
        if (__any_sync(0xffffffffu, odd)) c = sturm_count(n, a, b, x);
        const int ok = c <= k;
        const int cnt = __popc(__ballot_sync(0xffffffffu, ok));  // trial points with at most k eigenvalues below
        const double nlo = cnt > 0 ? lo + (hi - lo) * ((double)cnt * inv) : lo;
        const double nhi = cnt < 32 ? lo + (hi - lo) * ((double)(cnt + 1) * inv) : hi;
        lo = nlo;
        hi = nhi;
        if (hi - lo <= 2.2e-16 * fmax(fabs(lo), fabs(hi)) + 1e-300) break;
    }
    if (!called) midway();
    __syncwarp();
    return 0.5 * (lo + hi);
}

// tri_solve's factorisation and solve as separate steps, in arrays that do not alias (the next
// rows' loads need not wait for this row's stores).
__device__ __forceinline__ void tri_factor(int n, const double* a, const double* b, double shift, double pivmin,
                                           double* __restrict__ dl, double* __restrict__ dd, double* __restrict__ du,
                                           double* __restrict__ du2, int* __restrict__ piv) {
    double d = a[0] - shift, u = n > 1 ? b[0] : 0.0;  // row i as it stands
    for (int i = 0; i < n - 1; ++i) {
        const double l = b[i], dn = a[i + 1] - shift, un = i < n - 2 ? b[i + 1] : 0.0;
        if (fabs(d) >= fabs(l)) {
            piv[i] = 0;
            if (fabs(d) < pivmin) d = (d < 0 ? -pivmin : pivmin);
            const double f = l / d;
            dd[i] = d;
            dl[i] = f;
            du[i] = u;
            du2[i] = 0;
            d = fma(-f, u, dn);
            u = un;
        } else {
            piv[i] = 1;
            const double f = d / l;
            dd[i] = l;
            dl[i] = f;
            du[i] = dn;
            du2[i] = un;
            d = fma(-f, dn, u);
            u = -f * un;
        }
    }
    if (fabs(d) < pivmin) d = (d < 0 ? -pivmin : pivmin);
    dd[n - 1] = d;
}
// a / b, correctly rounded, from r = 1 / b correctly rounded: Markstein's correction (IBM J.
// Res. Dev. 34, 1990) of a r by its remainder, exact away from the ends of the range
// (|a|, |b| within 2^+-900 here), three dependent operations instead of a division.
__device__ __forceinline__ double div_by_reciprocal(double a, double b, double r) {
    const double q = a * r;
    return fma(fma(-q, b, a), r, q);
}

// The Ritz coefficients of lz_ritz_coeffs_kernel for the eigenvalue th, by one warp: the
// factorisation, the same in every iteration, made once; the divisions of the back
// substitution by reciprocals that the lanes form together.  work: 6 n doubles.
__device__ void tri_ritz_exact(int n, const double* a, const double* b, double th, double* y, double* work,
                               int* piv) {
    const int lane = threadIdx.x & 31;
    double* __restrict__ dl = work;
    double* __restrict__ dd = work + n;
    double* __restrict__ du = work + 2 * n;
    double* __restrict__ du2 = work + 3 * n;
    double* __restrict__ z = work + 4 * n;
    double* __restrict__ rd = work + 5 * n;
    double scale = 0;
    for (int i = lane; i < n; i += 32) {
        scale = fmax(scale, fabs(a[i]) + (i < n - 1 ? fabs(b[i]) : 0.0));
        y[i] = 1.0 + 0.1 * ((i * 7919) % 97) / 97.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) scale = fmax(scale, __shfl_xor_sync(0xffffffffu, scale, o));
    scale = fmax(scale, 1e-300);
    if (lane == 0) tri_factor(n, a, b, th + 4e-15 * scale, 2.2e-16 * scale, dl, dd, du, du2, piv);
    __syncwarp();
    bool fits = true;  // for div_by_reciprocal
    for (int i = lane; i < n; i += 32) {
        rd[i] = 1.0 / dd[i];
        const int e = (__double2hiint(dd[i]) >> 20) & 0x7ff;
        fits = fits && e > 123 && e < 1923;
    }
    fits = __all_sync(0xffffffffu, fits);
    __syncwarp();
    for (int it = 0; it < 3; ++it) {
        // every lane runs the substitutions (the same values), lane 0 stores
        double r = y[0];
#pragma unroll 4
        for (int i = 0; i < n - 1; ++i) {
            const double q = y[i + 1], f = dl[i];
            const bool s = piv[i] != 0;
            const double u = s ? q : r, v = s ? r : q;
            if (lane == 0) z[i] = u;
            r = fma(-f, u, v);
        }
        if (lane == 0) z[n - 1] = r;
        __syncwarp();
        double x1 = 0, x2 = 0, mx = 0;
#pragma unroll 4
        for (int i = n - 1; i >= 0; --i) {
            double t = z[i];
            if (i < n - 1) t = fma(-du[i], x1, t);
            if (i < n - 2) t = fma(-du2[i], x2, t);
            double x = div_by_reciprocal(t, dd[i], rd[i]);
            const int e = (__double2hiint(t) >> 20) & 0x7ff;
            if (!fits || (t != 0.0 && (e <= 123 || e >= 1923))) x = t / dd[i];
            if (lane == 0) y[i] = x;
            mx = fmax(mx, fabs(x));
            x2 = x1;
            x1 = x;
        }
        __syncwarp();
        if (mx > 0)
            for (int i = lane; i < n; i += 32) y[i] /= mx;
        __syncwarp();
    }
    double nr = 0;
    int im = 0;
    double best = 0;
#pragma unroll 4
    for (int i = 0; i < n; ++i) {
        const double v = y[i];
        nr += v * v;
        if (fabs(v) > best) {
            best = fabs(v);
            im = i;
        }
    }
    nr = sqrt(nr);
    const double sg = (y[im] < 0) ? -1.0 : 1.0;
    __syncwarp();
    for (int i = lane; i < n; i += 32) y[i] = sg * y[i] / nr;
    __syncwarp();
}

}  // namespace
}  // namespace tnb
