// lzsite.cu -- restarted Lanczos for the lowest eigenpair of one site's Heff, the
// whole solve in one launch.
//
// The solve is lanczos_solve's, bit for bit: full reorthogonalisation by
// classical Gram-Schmidt applied twice, FP64 throughout, the same stopping
// rules, and every sum in the order in which the chain of launches forms it
// (vector elements in blocks of 512, warp butterflies, blocks in groups of 32;
// products in k order; MPO terms in list order).  The order matters to a
// caller: with targets below the root of the rounding error the stopping
// decisions hang on rounding, and a sweep from a random state moves by 1e-8
// when one sum is formed differently.
// As a chain a Krylov step is seven kernels of 2-20 us each, most of it launch
// latency, the reductions' tails and the one-warp tridiagonal decision; here
// the CTAs stay and meet at barriers (a cluster barrier of ~360 cycles for up to
// eight CTAs, a counter in L2 of ~2300 above):
//   A  P[w1, n] = F_w1 v_n           32 x 32 DMMA tiles, four warps each
//   B  Y[w2, m] = Q G_w2^T           the MPO combination Q = sum c P formed while
//                                    the tile is loaded
//   C  w = sum_w2 Y on the CTA's own 512 elements; its share of V^T w
//   D  w -= V h; its share of V^T w and |w|^2
//   E  v_next = (w - V h2) / beta
// A CTA that owns elements keeps its rows of the whole Krylov basis in shared
// memory (in rows of 33 per 32 elements: a lane sums a group of 32 in the
// butterfly's order without bank conflicts), so C, D and E read no basis vector
// from memory; only v (the next products' operand), P, Y and the partial dots go
// through L2.  The stopping decision of a step is made by a ninth warp of every
// CTA, redundantly, while the others already run A, B and C of the next one;
// these are dropped when it says stop.
// Bound: the five barriers, the L2 round trips between the phases and, for the
// smallest sites, the decision.  Per Krylov step (20 in the basis, d = 2, Dw = 5)
// against the chain of launches: D = 8 12.9 us (49.0), 32 14.5 (52.1), 64 18.7
// (56.1), 128 25.2 (61.4); d = 3, D = 90 22.8 (60.1).
#include "lzsite.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "dgemm.cuh"
#include "qr.h"
#include "tridiag.cuh"

namespace cg = cooperative_groups;

namespace tnb {

namespace {

constexpr int LS_THREADS = 288;    // eight warps of products, one of decisions
constexpr int LS_GW = 8;           // product warps: two groups of four
constexpr int LS_WARPS = LS_THREADS / 32;
constexpr int LS_TILE = 32;
constexpr int LS_STAGES = 4;
constexpr int LS_MAXTERMS = 192, LS_MAXOUT = 64;
constexpr int LS_STAGE = 32 * (DG_BK + 4) + 16 * (LS_TILE + 4);  // doubles of one stage, both operands (at most)
constexpr int LS_BLK = 512;                    // vector elements per CTA: a block of the chain's reductions
constexpr int LS_ROW = LS_BLK / 32 * 33;       // their place in shared memory
__device__ __forceinline__ int ls_at(int e) { return e + (e >> 5); }

struct LsArgs {
    int d, Dw1, Dw2, D1, D2, nterms;
    long long N;
    const double *F, *G;
    const WTermDev* terms;
    double *x, *xc, *P, *Y;            // xc, P, Y: blocks of D2 columns with the even leading dimension ldp
    double *partA, *partB, *partN;     // [k][CTA] partial sums
    unsigned* bar;
    int* derr;
    LzSummary* sum;
    int ldp, nblk, mm, maxR, clustered;  // nblk: CTAs that own vector elements
    double tol, tol_rel;
    int polls;                         // of a grid barrier
};

struct LsSm {
    double alpha[LZ_MAXK], beta[LZ_MAXK], rhist[LZ_MAXK], y[LZ_MAXK], hs[LZ_MAXK + 8];
    double2 rows[LZ_MAXK];                 // (a_i, b_{i-1}^2) of the decision's matrix
    double work[6 * LZ_MAXK];
    int piv[LZ_MAXK];
    double theta, theta2, resid;
    int done, conv, nb, err;
    unsigned long long used;
    int nblist, blist[64];
    int ms[LS_MAXOUT + 1];                 // first term of each output (m, w2)
    int tin[LS_MAXTERMS];
    double tc[LS_MAXTERMS];
};
// dynamic shared memory beside the static LsSm, of the 227 KB a CTA may have
constexpr int LS_DYN_MAX = 227 * 1024 - (int)((sizeof(LsSm) + 1023) / 1024 * 1024);

__device__ __forceinline__ double ls_wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void ls_named(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void ls_cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void ls_cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// All CTAs have met.  gemm: only the eight product warps of each CTA take part
// (the clustered form needs every thread: the decision warp arrives for itself).
// False once a wait has run out of polls (sm.err, the context's error word).
constexpr int LS_POLLS = 1 << 23;  // unless the context says otherwise
__device__ bool ls_barrier(const LsArgs& a, LsSm& sm, unsigned& target, bool gemm) {
    if (a.clustered) {
        ls_cluster_arrive();
        ls_cluster_wait();
        return true;
    }
    if (gemm) ls_named(1, 32 * LS_GW);
    else __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        unsigned v = 0;
        int left = a.polls;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
        } while (v < target && --left > 0);
        if (v < target) {
            atomicExch(a.derr, 1);
            sm.err = 1;
        }
    }
    if (gemm) ls_named(1, 32 * LS_GW);
    else __syncthreads();
    return sm.err == 0;
}

// acc = A(m0.., :) B(:, n0..) for a 32 x 32 tile by the four warps of a group:
// A(m, k) at k lda + m, B(k, n) at n ldb + k (BK) or k ldb + n; VA, VB doubles per copy.
template <int VA, bool BK, int VB>
__device__ __forceinline__ void ls_tile(double (&acc)[2][2][2], const double* A, long long lda, const double* B,
                                        long long ldb, int M, int N, int K, int m0, int n0, double* st, int group,
                                        int gtid) {
    using OpA = DgOperand<LS_TILE, true, VA, 128>;
    using OpB = DgOperand<LS_TILE, !BK, VB, 128>;
    static_assert(OpA::STAGE + OpB::STAGE <= LS_STAGE, "stage");
    const int lane = gtid & 31, warp = gtid >> 5, gid = lane >> 2, tig = lane & 3;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
    OpA oa;
    OpB ob;
    oa.init(gtid, A, 1, lda, m0, M);
    ob.init(gtid, B, BK ? ldb : 1, BK ? 1 : ldb, n0, N);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int nt = (K + DG_BK - 1) / DG_BK;
#pragma unroll
    for (int s = 0; s < LS_STAGES - 1; ++s) {
        if (s < nt) {
            oa.load(st + s * LS_STAGE, A, K - s * DG_BK);
            ob.load(st + s * LS_STAGE + OpA::STAGE, B, K - s * DG_BK);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    int rd = 0, wr = LS_STAGES - 1;
    for (int kt = 0; kt < nt; ++kt) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(LS_STAGES - 2) : "memory");
        ls_named(2 + group, 128);
        if (kt + LS_STAGES - 1 < nt) {
            oa.load(st + wr * LS_STAGE, A, K - (kt + LS_STAGES - 1) * DG_BK);
            ob.load(st + wr * LS_STAGE + OpA::STAGE, B, K - (kt + LS_STAGES - 1) * DG_BK);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const double* a = st + rd * LS_STAGE;
        const double* b = a + OpA::STAGE;
#pragma unroll
        for (int ks = 0; ks < DG_BK; ks += 4) {
            double af[2], bf[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                af[i] = OpA::get(a, wm + 8 * i + gid, ks + tig);
                bf[i] = OpB::get(b, wn + 8 * i + gid, ks + tig);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) dmma(acc[i][j], af[i], bf[j]);
        }
        rd = rd + 1 == LS_STAGES ? 0 : rd + 1;
        wr = wr + 1 == LS_STAGES ? 0 : wr + 1;
    }
    ls_named(2 + group, 128);  // the stages may be refilled
}

// acc = Q(m0.., :) G(n0.., :)^T for a 32 x 32 tile, Q = sum_t c_t P[in_t] over the terms
// [t0, t1) formed on the way into shared memory (in list order from zero), one k-tile
// ahead in registers; G by asynchronous copies as in ls_tile.
template <int VB>
__device__ __forceinline__ void ls_tile_combined(double (&acc)[2][2][2], const LsSm& sm, int t0, int t1,
                                                 const double* P, size_t blkp, int ldp, const double* G, int M, int K,
                                                 int m0, int n0, double* st, int group, int gtid) {
    using OpA = DgOperand<LS_TILE, true, 2, 128>;
    using OpB = DgOperand<LS_TILE, true, VB, 128>;
    static_assert(2 * OpA::STAGE + LS_STAGES * OpB::STAGE <= LS_STAGES * LS_STAGE, "stages");
    const int lane = gtid & 31, warp = gtid >> 5, gid = lane >> 2, tig = lane & 3;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
    double* Bs = st + 2 * OpA::STAGE;
    OpB ob;
    ob.init(gtid, G, 1, K, n0, K);
    const int x = gtid % 16 * 2, k0 = gtid / 16;  // this thread's pairs of rows, at k0 and k0 + 8
    const bool in = m0 + x < M;
    const double* Px = P + m0 + x;
    double2 raw[2][4];  // the first four terms' values of the next k-tile
    auto value = [&](int i, int kt, int t) {
        const int k = kt * DG_BK + k0 + 8 * i;
        return in && k < K && t < t1
                   ? __ldcg(reinterpret_cast<const double2*>(Px + (size_t)k * ldp + sm.tin[t] * blkp))
                   : make_double2(0.0, 0.0);
    };
    auto fetch = [&](int kt) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int u = 0; u < 4; ++u) raw[i][u] = value(i, kt, t0 + u);
    };
    auto combined = [&](int i, int kt) {
        double2 v = make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (t0 + u < t1) {
                v.x = fma(sm.tc[t0 + u], raw[i][u].x, v.x);
                v.y = fma(sm.tc[t0 + u], raw[i][u].y, v.y);
            }
        for (int t = t0 + 4; t < t1; ++t) {  // (no Heisenberg MPO has more than four)
            const double2 q = value(i, kt, t);
            v.x = fma(sm.tc[t], q.x, v.x);
            v.y = fma(sm.tc[t], q.y, v.y);
        }
        return v;
    };
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int nt = (K + DG_BK - 1) / DG_BK;
#pragma unroll
    for (int s = 0; s < LS_STAGES - 1; ++s) {
        if (s < nt) ob.load(Bs + s * OpB::STAGE, G, K - s * DG_BK);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    fetch(0);
    int rd = 0, wr = LS_STAGES - 1;
    for (int kt = 0; kt < nt; ++kt) {
        double* a = st + (kt & 1) * OpA::STAGE;
#pragma unroll
        for (int i = 0; i < 2; ++i) *reinterpret_cast<double2*>(a + (k0 + 8 * i) * OpA::LD + x) = combined(i, kt);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(LS_STAGES - 2) : "memory");
        ls_named(2 + group, 128);
        if (kt + 1 < nt) fetch(kt + 1);
        if (kt + LS_STAGES - 1 < nt) ob.load(Bs + wr * OpB::STAGE, G, K - (kt + LS_STAGES - 1) * DG_BK);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const double* b = Bs + rd * OpB::STAGE;
#pragma unroll
        for (int ks = 0; ks < DG_BK; ks += 4) {
            double af[2], bf[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                af[i] = OpA::get(a, wm + 8 * i + gid, ks + tig);
                bf[i] = OpB::get(b, wn + 8 * i + gid, ks + tig);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) dmma(acc[i][j], af[i], bf[j]);
        }
        rd = rd + 1 == LS_STAGES ? 0 : rd + 1;
        wr = wr + 1 == LS_STAGES ? 0 : wr + 1;
    }
    ls_named(2 + group, 128);  // the stages may be refilled
}

__device__ __forceinline__ void ls_store(const double (&acc)[2][2][2], double* C, int ldc, int M, int N,
                                         int m0, int n0, int gtid) {
    const int lane = gtid & 31, warp = gtid >> 5, gid = lane >> 2, tig = lane & 3;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int gm = m0 + wm + 8 * i + gid;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int gn = n0 + wn + 8 * j + 2 * tig + q;
                if (gm < M && gn < N) C[(size_t)gn * ldc + gm] = acc[i][j][q];
            }
    }
}

// The decision of step j by one warp: lz_decide_step of the launch chain.  midway() is called
// once, after some rounds of the eigenvalue search.
template <class F>
__device__ __forceinline__ void ls_decide(const LsArgs& a, LsSm& sm, int j, F midway) {
    const int lane = threadIdx.x & 31, nk = j + 1;
    const double th = warp_eig_exact(nk, sm.alpha, sm.beta, sm.rows, 0, midway);
    if (lane == 0) {
        const double yl = last_component_rows(nk, sm.rows, sm.alpha, sm.beta, th);
        const double bj = sm.beta[j];
        const double resid = bj * yl;
        double tolEff = fmax(a.tol, 1e-13 * fmax(1.0, fabs(th)));
        if (a.tol_rel > 0) {
            double tn = 0;
            for (int i = 0; i < nk; ++i)
                tn = fmax(tn, fabs(sm.alpha[i]) + fabs(sm.beta[i]) + (i > 0 ? fabs(sm.beta[i - 1]) : 0.0));
            tolEff = fmax(tolEff, a.tol_rel * tn);
        }
        sm.theta = th;
        sm.resid = resid;
        sm.nb = nk;
        sm.rhist[j] = resid;
        int done = 0;
        const bool conv = (resid <= tolEff) || (bj <= 1e-14 * fmax(1.0, fabs(th)));
        if (conv) {
            done = 1;
            sm.conv = 1;
        }
        if (a.tol_rel > 0 && j >= 2 && resid > 0.5 * sm.rhist[j - 2]) done = 1;
        if (nk >= a.mm || nk >= LZ_MAXK - 1) done = 1;  // basis exhausted for this restart
        sm.done = done;
    }
    __syncwarp();
}

template <int VC>  // doubles per copy of the environments (2: even D1 and D2, 16-byte bases)
__global__ void __launch_bounds__(LS_THREADS, 1) lz_site_kernel(const LsArgs a) {
    extern __shared__ __align__(16) double ls_dyn[];
    __shared__ LsSm sm;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int G = (int)gridDim.x, cta = (int)blockIdx.x;
    const int group = wid >> 2, gtid = tid & 127;
    double* st = ls_dyn + (size_t)group * LS_STAGES * LS_STAGE;  // this group's stages
    double* V = ls_dyn + (size_t)2 * LS_STAGES * LS_STAGE;       // [k][LS_ROW]
    double* ws = V + (size_t)a.mm * LS_ROW;
    int* off = reinterpret_cast<int*>(ws + LS_ROW);              // element -> place in xc (blocks of blkp)
    const long long c0 = (long long)cta * LS_BLK;
    const int cnt = (int)max(0LL, min((long long)LS_BLK, a.N - c0));
    const bool owner = cta < a.nblk;
    const int blk = a.D1 * a.D2, blkp = a.D2 * a.ldp;
    const int mt = (a.D1 + LS_TILE - 1) / LS_TILE, nt = (a.D2 + LS_TILE - 1) / LS_TILE, mn = mt * nt;
    const int nout = a.d * a.Dw2;
    unsigned target = 0;
    if (tid == 0) {
        sm.err = 0;
        sm.used = 0;
    }
    __syncthreads();
    for (int t = tid; t < a.nterms; t += LS_THREADS) {
        const WTermDev tm = a.terms[t];
        sm.tin[t] = tm.in;
        sm.tc[t] = tm.c;
        atomicOr(&sm.used, 1ULL << tm.in);
        if (t == 0 || a.terms[t - 1].out != tm.out) sm.ms[tm.out] = t;
    }
    if (tid == 0) sm.ms[nout] = a.nterms;
    // elements past the vector's end are zeros for the sums
    for (int e = tid; e < a.mm * LS_ROW; e += LS_THREADS) V[e] = 0.0;
    for (int e = tid; e < LS_BLK; e += LS_THREADS) {
        double v = 0.0;
        if (e < cnt) {
            const long long i = c0 + e;
            const int r = (int)(i % blk);
            off[e] = (int)(i / blk) * blkp + (r / a.D1) * a.ldp + r % a.D1;
            v = a.x[i];
        }
        ws[ls_at(e)] = v;
    }
    __syncthreads();
    if (tid == 0) {
        int n = 0;
        for (int b = 0; b < a.Dw1 * a.d; ++b)
            if (sm.used >> b & 1) sm.blist[n++] = b;
        sm.nblist = n;
    }
    // The sum of v . w over the CTA's 512 elements in the order of a block of 512 threads: a
    // butterfly over each 32 elements, then one over the 16 groups.  Half a warp per sum: the
    // lane of a group forms its butterfly tree from shared memory.
    auto block_dot = [&](const double* v, const double* w) {
        const int g = lane & 15;
        const double *vg = v + 33 * g, *wg = w + 33 * g;
        double t[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) t[i] = fma(vg[i], wg[i], 0.0) + fma(vg[i + 16], wg[i + 16], 0.0);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < o; ++i) t[i] += t[i + o];
        double s = t[0];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    };
    // this CTA's share of V_k . w for k < nk, and of |w|^2 as k = nk when asked
    auto dots = [&](double* part, int nk, bool norm, int warps) {
        const int n = nk + (norm ? 1 : 0);
        for (int k2 = 2 * wid; k2 < n; k2 += 2 * warps) {
            const int k = k2 + (lane >> 4);
            const double s = block_dot(k < nk ? V + (size_t)k * LS_ROW : ws, ws);
            if ((lane & 15) == 0 && k < n) part[(size_t)k * a.nblk + cta] = s;
        }
    };
    // sums over the owning CTAs of part[k * nblk + .], k < nk, into sm.hs in the order of a block
    // of 512 threads with one partial each: butterflies over 32, then over the groups of 32
    auto gather = [&](const double* part, int nk) {
        for (int k = wid; k < nk; k += LS_WARPS) {
            double g[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                const int c = lane + 32 * q;
                g[q] = c < a.nblk ? __ldcg(part + (size_t)k * a.nblk + c) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 5; ++q)
                if (32 * q < a.nblk) g[q] = ls_wsum(g[q]);
            if (lane == 0) sm.hs[k] = ((g[0] + g[4]) + g[2]) + (g[1] + g[3]);
        }
        __syncthreads();
    };
    // to = f (ws - V hs) element by element in k order, also into xc when asked; two elements a
    // thread (256 of them), four basis rows' loads in flight
    auto project = [&](int nk, double f, double* to, bool pub) {
        if (tid >= LS_BLK / 2) return;
        const int e0 = tid, e1 = tid + LS_BLK / 2, i0 = ls_at(e0), i1 = ls_at(e1);
        double w0 = ws[i0], w1 = ws[i1];
        int k = 0;
        for (; k + 4 <= nk; k += 4) {
            double v0[4], v1[4], h[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                h[q] = sm.hs[k + q];
                v0[q] = V[(k + q) * LS_ROW + i0];
                v1[q] = V[(k + q) * LS_ROW + i1];
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                w0 = fma(-h[q], v0[q], w0);
                w1 = fma(-h[q], v1[q], w1);
            }
        }
        for (; k < nk; ++k) {
            w0 = fma(-sm.hs[k], V[k * LS_ROW + i0], w0);
            w1 = fma(-sm.hs[k], V[k * LS_ROW + i1], w1);
        }
        w0 *= f;
        w1 *= f;
        if (e0 < cnt) {
            to[i0] = w0;
            if (pub) a.xc[off[e0]] = w0;
        }
        if (e1 < cnt) {
            to[i1] = w1;
            if (pub) a.xc[off[e1]] = w1;
        }
    };
    int restarts = 0, steps = 0, conv = 0;
    double prev_resid = 1e300;
    for (;;) {
        // v_0 = x / |x|
        __syncthreads();
        if (owner && wid == 0) {
            const double s = block_dot(ws, ws);
            if (lane == 0) a.partN[cta] = s;
        }
        if (tid == 0) {
            sm.done = 0;
            sm.conv = 0;
            sm.nb = 0;
        }
        if (!ls_barrier(a, sm, target, false)) return;
        gather(a.partN, 1);
        const double nr = sqrt(sm.hs[0]);
        for (int e = tid; e < cnt; e += LS_THREADS) {
            double v;
            if (nr > 0) v = ws[ls_at(e)] / nr;
            else {
                // deterministic start vector when x = 0
                unsigned long long h = (unsigned long long)(c0 + e) * 0x9E3779B97F4A7C15ULL;
                h ^= h >> 29;
                v = ((double)((h >> 11) & 0xFFFFF) / 1048576.0 - 0.5) / sqrt((double)a.N / 12.0);
            }
            V[ls_at(e)] = v;
            a.xc[off[e]] = v;
        }
        if (!ls_barrier(a, sm, target, false)) return;
        for (int j = 0;; ++j) {
            const int nk = j + 1;
            if (wid < LS_GW) {
                // A: P[b] = F_w1 v_n for the (w1, n) that an MPO term uses
                const int tiles = sm.nblist * mn;
                for (int t = 2 * cta + group; t < tiles; t += 2 * G) {
                    const int b = sm.blist[t / mn], r = t % mn;
                    const int m0 = r % mt * LS_TILE, n0 = r / mt * LS_TILE;
                    double acc[2][2][2];
                    ls_tile<VC, true, 2>(acc, a.F + (size_t)(b / a.d) * a.D1 * a.D1, a.D1,
                                         a.xc + (size_t)(b % a.d) * blkp, a.ldp, a.D1, a.D2, a.D1, m0, n0, st, group,
                                         gtid);
                    ls_store(acc, a.P + (size_t)b * blkp, a.ldp, a.D1, a.D2, m0, n0, gtid);
                }
                if (!ls_barrier(a, sm, target, true)) return;
                // B: Y[w2, m] = (sum c P) G_w2^T
                const int tiles2 = nout * mn;
                for (int t = 2 * cta + group; t < tiles2; t += 2 * G) {
                    const int q = t / mn, r = t % mn, w2 = q % a.Dw2, m = q / a.Dw2;
                    const int m0 = r % mt * LS_TILE, n0 = r / mt * LS_TILE;
                    double acc[2][2][2];
                    ls_tile_combined<VC>(acc, sm, sm.ms[q], sm.ms[q + 1], a.P, blkp, a.ldp,
                                         a.G + (size_t)w2 * a.D2 * a.D2, a.D1, a.D2, m0, n0, st, group, gtid);
                    ls_store(acc, a.Y + (size_t)(w2 * a.d + m) * blkp, a.ldp, a.D1, a.D2, m0, n0, gtid);
                }
                if (!ls_barrier(a, sm, target, true)) return;
                // C: the partial products of w2 = 0, 1, .. added in that order
                const size_t slab = (size_t)a.d * blkp;
                for (int e = tid; e < cnt; e += 32 * LS_GW) {
                    const double* y = a.Y + off[e];
                    double s = 0;
                    for (int w0 = 0; w0 < a.Dw2; w0 += 8) {  // eight slabs' loads in flight
                        double v[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) v[q] = w0 + q < a.Dw2 ? __ldcg(y + (w0 + q) * slab) : 0.0;
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            if (w0 + q < a.Dw2) s += v[q];
                    }
                    ws[ls_at(e)] = s;
                }
                ls_named(1, 32 * LS_GW);
                if (owner) dots(a.partA, nk, false, LS_GW);
            } else {
                // the cluster barriers of A and B want every thread: this warp arrives early for
                // each and waits when it gets there
                if (a.clustered) ls_cluster_arrive();
                auto between = [&] {
                    if (a.clustered) {
                        ls_cluster_wait();
                        ls_cluster_arrive();
                    }
                };
                if (j > 0) ls_decide(a, sm, j - 1, between);
                else between();
                if (a.clustered) ls_cluster_wait();
            }
            if (!ls_barrier(a, sm, target, false)) return;
            if (j > 0 && sm.done) break;  // the step before was the last
            // D
            gather(a.partA, nk);
            const double hj = sm.hs[j];
            project(nk, 1.0, ws, false);
            __syncthreads();
            if (owner) dots(a.partB, nk, true, LS_WARPS);
            if (!ls_barrier(a, sm, target, false)) return;
            // E
            gather(a.partB, nk + 1);
            double ss = 0;
            for (int k = 0; k < nk; ++k) ss = fma(sm.hs[k], sm.hs[k], ss);
            const double beta = sqrt(fmax(sm.hs[nk] - ss, 0.0));
            const double inv = beta > 0 ? 1.0 / beta : 0.0;
            if (tid == 0) {
                sm.alpha[j] = hj + sm.hs[j];
                sm.beta[j] = beta;
            }
            if (nk >= a.mm) {  // the basis is full: decide now
                __syncthreads();
                if (wid == LS_GW) ls_decide(a, sm, j, [] {});
                __syncthreads();
                break;
            }
            project(nk, inv, V + (size_t)nk * LS_ROW, true);
            if (!ls_barrier(a, sm, target, false)) return;
        }
        // the Ritz vector replaces the start vector
        if (wid == LS_GW) tri_ritz_exact(sm.nb, sm.alpha, sm.beta, sm.theta, sm.y, sm.work, sm.piv);
        if (wid == 0) {  // the next eigenvalue, for the gap
            const double t2 = sm.nb > 1 ? warp_eig_exact(sm.nb, sm.alpha, sm.beta, sm.rows, 1, [] {}) : sm.theta;
            if (lane == 0) sm.theta2 = t2;
        }
        __syncthreads();
        const int nb = sm.nb;
        for (int e = tid; e < cnt; e += LS_THREADS) {
            const int i = ls_at(e);
            double s = 0;
            for (int k = 0; k < nb; ++k) s = fma(sm.y[k], V[k * LS_ROW + i], s);
            ws[i] = s;
        }
        // another restart? (the rule of lz_decide_kernel; the same in every thread)
        const int r = restarts++;
        steps += nb;
        bool stop = false;
        if (sm.conv) {
            conv = 1;
            stop = true;
        } else if ((long long)a.mm >= a.N) {
            conv = 1;
            stop = true;
        } else if (a.tol_rel > 0) {
            if (r > 0 && sm.resid > 0.5 * prev_resid) stop = true;
            else prev_resid = sm.resid;
        }
        if (r + 1 >= a.maxR) stop = true;
        if (stop) break;
    }
    for (int e = tid; e < cnt; e += LS_THREADS) a.x[c0 + e] = ws[ls_at(e)];
    if (cta == 0 && tid == 0) {
        a.sum->theta = sm.theta;
        a.sum->theta2 = sm.theta2;
        a.sum->resid = sm.resid;
        a.sum->matvecs = steps;
        a.sum->restarts = restarts;
        a.sum->converged = conv;
        a.sum->steps = steps;
        a.sum->launches = 0;  // counted where it was launched
    }
}

struct LsPlan {
    int ctas = 0;  // 0: not served
    bool clustered = false;
};

size_t ls_smem(int mm) {
    return sizeof(double) * ((size_t)2 * LS_STAGES * LS_STAGE + (size_t)(mm + 1) * LS_ROW) + sizeof(int) * LS_BLK;
}

// One tile of each group of warps at a time where the SMs allow it, and a CTA for every
// 512 vector elements; up to eight CTAs as one cluster, whose barrier is a fifth of
// the grid's (D = 32: 14.5 us a step on a cluster of 8, 16.2 on a grid of 16; D = 64, 40
// tiles: 22.6 on 16 CTAs, 19.5 on 37, 18.7 on 74).
LsPlan ls_plan(const ContractShape& s, long long N, int sms) {
    const int mn = ((s.D1 + LS_TILE - 1) / LS_TILE) * ((s.D2 + LS_TILE - 1) / LS_TILE);
    const long long tiles = (long long)std::max(s.Dw1, s.Dw2) * s.d * mn;
    const int nblk = (int)((N + LS_BLK - 1) / LS_BLK);
    int want = (int)std::min<long long>((tiles + 1) / 2, sms);  // two tiles at a time per CTA
    want = std::max(want, nblk);
    LsPlan p;
    p.clustered = want <= 8;
    p.ctas = want;
    if (p.clustered)
        for (p.ctas = 1; p.ctas < want;) p.ctas *= 2;
    return p;
}

int ls_enqueue(Ctx& c, const LsPlan& p, const ContractShape& s, const WTermDev* terms, int nterms, const double* F,
               const double* G, double* x, long long N, int mm, int maxRestarts, double tol, double tol_rel) {
    cudaStream_t st = c.stream;
    LsArgs a{};
    a.d = s.d; a.Dw1 = s.Dw1; a.Dw2 = s.Dw2; a.D1 = s.D1; a.D2 = s.D2; a.nterms = nterms;
    a.N = N; a.F = F; a.G = G; a.terms = terms; a.x = x;
    a.ldp = (s.D1 + 1) & ~1;
    const size_t blkp = (size_t)a.ldp * s.D2;
    const size_t nP = (size_t)s.Dw1 * s.d * blkp, nY = (size_t)s.Dw2 * s.d * blkp, nX = (size_t)s.d * blkp;
    const int nblk = (int)((N + LS_BLK - 1) / LS_BLK);
    const size_t nPart = (size_t)(LZ_MAXK + 1) * nblk;
    TN_CHECK(c.lz.ensure(sizeof(double) * (nP + nY + nX + 3 * nPart + 64)));
    TN_CHECK(ensure_summary(c));
    TN_CHECK(c.lzbar.ensure(sizeof(unsigned)));
    TN_CHECK(ensure_device_error_word(c));
    a.P = c.lz.as<double>();
    a.Y = a.P + nP;
    a.xc = a.Y + nY;
    a.partA = a.xc + nX;
    a.partB = a.partA + nPart;
    a.partN = a.partB + nPart;
    a.bar = c.lzbar.as<unsigned>();
    a.derr = c.derr.as<int>();
    a.sum = c.lzsum.as<LzSummary>();
    a.nblk = nblk; a.mm = mm; a.maxR = maxRestarts > 0 ? maxRestarts : 1; a.clustered = p.clustered;
    a.tol = tol; a.tol_rel = tol_rel;
    a.polls = c.wait_polls < 0 ? LS_POLLS : c.wait_polls;
    const bool wide = s.D1 % 2 == 0 && s.D2 % 2 == 0 && ((reinterpret_cast<uintptr_t>(F) | reinterpret_cast<uintptr_t>(G)) & 15) == 0;
    auto kern = wide ? lz_site_kernel<2> : lz_site_kernel<1>;
    TN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LS_DYN_MAX));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.ctas);
    cfg.blockDim = dim3(LS_THREADS);
    cfg.dynamicSmemBytes = ls_smem(mm);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (p.clustered) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)p.ctas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        TN_CUDA_CHECK(cudaMemsetAsync(a.bar, 0, sizeof(unsigned), st));
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return LZ_SITE_UNAVAILABLE;
    }
    TN_CUDA_CHECK(e);
    count_launch();
    return TN_OK;
}

}  // namespace

int lanczos_site(Ctx& c, const ContractShape& s, const WTermDev* terms, int nterms, const double* F, const double* G,
                 double* x, int m, int maxRestarts, double tol, double tol_rel, LzSummary* host_out) {
    const long long N = (long long)s.d * s.D1 * s.D2;
    // one element per thread of the chain's reductions (at most one block of 512 per SM), which
    // the sums' order follows
    if (!c.use_site_solve || N <= 0 || N > (long long)LS_BLK * c.sm_count || c.sm_count > 160 || s.d * s.Dw2 > LS_MAXOUT ||
        nterms > LS_MAXTERMS || s.Dw1 * s.d > 64)
        return LZ_SITE_UNAVAILABLE;
    int mm = std::min(m, LZ_MAXK - 1);
    if ((long long)mm > N) mm = (int)N;
    if (mm < 1) mm = 1;
    if (ls_smem(mm) > (size_t)LS_DYN_MAX) return LZ_SITE_UNAVAILABLE;
    const LsPlan p = ls_plan(s, N, c.sm_count);
    const int rc = ls_enqueue(c, p, s, terms, nterms, F, G, x, N, mm, maxRestarts, tol, tol_rel);
    if (rc != TN_OK) return rc;
    TN_CUDA_CHECK(cudaMemcpyAsync(host_out, c.lzsum.p, sizeof(LzSummary), cudaMemcpyDeviceToHost, c.stream));
    return TN_OK;
}

}  // namespace tnb
