// qrc.cu -- Householder QR by thread-block clusters, one launch (FP64).
//
// Cluster q of C CTAs owns columns 32q .. 32q + 31 for the whole factorisation,
// their rows dealt to the CTAs in groups of 8W (W warps) and kept in shared
// memory.  It applies the block reflectors of panels 0 .. q - 1 as their owners
// publish them, factors its own panel and publishes it; clusters past the last
// panel only apply.  Further clusters, if all fit on the device, hold 32 rows of
// Q each, that is columns of Q^T = H_{K-1} .. H_0 I, and apply every panel as
// it appears; otherwise cluster q forms its columns of Q afterwards
// (H_0 .. H_q e_c).  No column leaves its CTAs before it is final.
//
// Panel: a lane holds 2 RL rows x 4 columns in registers.  Step j takes the
// reflector u_j (column j below the diagonal, unscaled) to the other columns by
// shuffles; the 32 dots u_j . p_c of a warp come out of a transposed butterfly,
// one column per lane, and go with row j to every CTA of the cluster (st.async,
// counted by an mbarrier).  Every warp adds the same partial sums in the same
// order and so has the step's scalars: one exchange per column, no barrier.
// The dots with finished columns are the Gram entries v_c^T v_j, from which each
// warp continues its rows of T while the next step's sums travel.
//
// Block reflector on a cluster's columns: Z = V^T C by DMMA on the CTA's rows, the
// partial Z summed and multiplied by T^T (or T) a slice of columns per CTA, then
// C -= V Z2 by DMMA; V and T come in one bulk copy.
//
// What bounds it: the chain of k column steps, ~0.85 us each (u by shuffles 0.1,
// dots and butterfly 0.15, exchange 0.2, sums of 4C warps 0.12, two reciprocal square
// roots 0.13, update 0.06, the divisions of tau and 1 / (alpha - beta) 0.1), and per panel ~9 us of publication (3) and application (6: DMMA
// at the FP64 rate on C SMs).  A call of tn_qr takes 325 us at 512 x 256 against 492 with
// the kernels of qr.cu (one CTA per panel, one task queue), 90 (113) at 64 x 64,
// 819 (1827) at 1024 x 512, 1127 (2428) at 1536 x 512, 634 (1843) at 512 x 1536.
//
// Rounding: 512 x 256, graded over five decades, |Q^T Q - I|_F 9.0e-15 and |QR - A| / |A| 5.0e-16 in extended
// precision (persistent kernel 1.3e-14, 6.1e-16).  Without the divisions (tau and 1 / (alpha - beta)
// from the chain's kap: 8 % less time) and with the products accumulated onto C the factors
// were a quarter further from the exact ones.
#include <cooperative_groups.h>

#include <algorithm>
#include <utility>

#include "dgemm.cuh"
#include "qr.h"

namespace cg = cooperative_groups;

namespace tnb {

namespace {

constexpr int QC_TLD = 37;        // leading dimension of T: odd, so that rows are conflict-free
constexpr int QC_ZLD = 36;        // of Z2: 4 mod 16, as the column blocks
constexpr int QC_POLLS = 1 << 20;  // of an mbarrier (a poll waits some microseconds by itself), unless the context says otherwise

struct QcArgs {
    int m, n, k, K;               // K panels
    int nb;                       // column blocks of A; clusters past them take blocks of Q's rows
    const double* A;
    long long ars, acs;           // row and column strides
    const int* colmap;            // columns of A in the matrix's order, or null
    double* Q;                    // m x k
    long long qrs, qcs;
    double* R;                    // k x n
    long long rrs, rcs;
    double* pub;                  // per panel and rank: V part, T
    long long pub_stride;         // doubles per (panel, rank)
    int* ready;                   // [panel][rank]
    int* err;                     // this launch's error word
    int* derr;                    // the context's, and its range word
    long long spin_limit;
    int polls;                    // of the exchanges' mbarriers
};

__device__ __forceinline__ unsigned qc_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned qc_remote(unsigned a, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void qc_st_async(unsigned dst, double a, double b, unsigned mbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "d"(a), "d"(b), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void qc_mbar_init(unsigned long long* b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(qc_smem(b)) : "memory");
}
__device__ __forceinline__ void qc_mbar_expect(unsigned long long* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(qc_smem(b)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ int qc_ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Bounded.  Returns false when the polls ran out, or, with an error word, when
// another wait of the launch has already failed.
__device__ __forceinline__ bool qc_mbar_wait(unsigned long long* b, unsigned phase, int polls, const int* err) {
    for (int i = 1; i <= polls; ++i) {
        unsigned done;
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(qc_smem(b)), "r"(phase)
            : "memory");
        if (done) return true;
        if (err && (i & 15) == 0 && qc_ld_acquire(err)) return false;
    }
    return false;
}
__device__ __forceinline__ int qc_ld_relaxed(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void qc_st_release(int* p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void qc_st_async(unsigned dst, double a, unsigned mbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
                 "l"(__double_as_longlong(a)), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ double qc_shfl(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// Shared memory of a CTA (doubles): C CTAs per cluster, W warps, RL rows per lane.
template <int RL, int C, int W>
struct QcLayout {
    static constexpr int rows = 8 * W * RL, ldr = rows + (rows % 16 ? 12 : 4);  // 4 mod 16
    static constexpr int NS = W * C;                                          // senders of a step's sums
    static constexpr int msg = 32 * ldr + 32 * QC_TLD;                        // what a panel publishes per CTA
    static constexpr int c = 0, v = 32 * ldr, t = v + 32 * ldr;               // T follows V
    static constexpr int x = v + msg;  // exchange: sums and row j by parity, or partial Z and Z2
    static constexpr int row = x + 2 * NS * 32, end_panel = row + 2 * 32;
    static constexpr int zp = x, z2 = x + 32 * 32, end_apply = z2 + 32 * QC_ZLD;
    static constexpr int end = end_panel > end_apply ? end_panel : end_apply;
    static_assert(ldr % 16 == 4 && msg % 2 == 0 && x % 2 == 0, "alignment");
};

// den and kap of a column below 2^-511 or above 2^511 are not finite (or have lost their digits).  Its scale 1 /
// (alpha - beta) tells (1 for a column without a reflector), looked at once, at the kernel's end, by one warp, in a
// function of its own: in the panel the test cost 2 % of a 512 x 1536 QR.
__device__ __noinline__ void qc_check_range(const double* scal, int* word) {
    const double x = fabs(scal[threadIdx.x & 31]);
    if (!(x <= 0x1p500 && x >= 0x1p-500)) atomicExch(word, 1);
}

template <int RL, int C, int W>
__global__ void __launch_bounds__(32 * W) qr_cluster_kernel(const QcArgs a) {
    using L = QcLayout<RL, C, W>;
    constexpr int NT = 32 * W, ldr = L::ldr, NS = L::NS, SC = 32 / C, SL = 8 * W;  // SL: rows of a slot in a CTA
    extern __shared__ __align__(16) double qc_dyn[];
    __shared__ unsigned long long pbar[2], zbar, wbar, vbar;
    __shared__ __align__(16) double fs[W][2][32];
    __shared__ __align__(16) double gcol[W][32];
    __shared__ double sc_s[32], be_s[32];
    __shared__ int flag_ok, bad;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), q = (int)blockIdx.x / C;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int gid = lane >> 2, tig = lane & 3;
    double* Cs = qc_dyn + L::c;
    double* Vs = qc_dyn + L::v;
    double* Ts = qc_dyn + L::t;           // [row][column]
    double* recv = qc_dyn + L::x;         // [parity][sender][column]: partial dots
    double* rowj = qc_dyn + L::row;       // [parity][column]: row j
    double* zp = qc_dyn + L::zp;          // [source CTA][32][SC]: partial Z of this CTA's slice of columns
    double* z2 = qc_dyn + L::z2;          // -Z2, [row][column]
    const bool qrows = q >= a.nb;         // a block of Q's rows: columns of Q^T = H_{K-1} .. H_0 I
    const int c0 = 32 * (qrows ? q - a.nb : q), ncol = min(32, (qrows ? a.m : a.n) - c0);
    const int nap = qrows ? a.K : min(q, a.K);
    constexpr unsigned vbytes = sizeof(double) * L::msg;
    if (tid == 0) {
        bad = 0;
        qc_mbar_init(&pbar[0]);
        qc_mbar_init(&pbar[1]);
        qc_mbar_init(&zbar);
        qc_mbar_init(&wbar);
        qc_mbar_init(&vbar);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    auto row_of = [&](int lr) { return ((lr / SL) * C + rank) * SL + lr % SL; };  // global row of a local one
    // the CTA's elements with rows < rows_end, along the index whose stride is 1
    auto each = [&](int rows_end, bool by_rows, auto f) {
        const int nr = min(L::rows, (rows_end + SL * C - 1) / (SL * C) * SL);
        for (int e = tid; e < 32 * nr; e += NT) {
            const int c = by_rows ? e / nr : e % 32, lr = by_rows ? e % nr : e / 32;
            f(c, lr, row_of(lr));
        }
    };
    if (qrows)
        each(L::rows * C, true, [&](int c, int lr, int i) { Cs[c * ldr + lr] = i == c0 + c ? 1.0 : 0.0; });
    else
        each(L::rows * C, a.ars == 1, [&](int c, int lr, int i) {
            double v = 0.0;
            if (i < a.m && c < ncol)
                v = a.A[(long long)i * a.ars + (long long)(a.colmap ? a.colmap[c0 + c] : c0 + c) * a.acs];
            Cs[c * ldr + lr] = v;
        });
    cl.sync();  // barriers are initialised before the first remote arrival
    // A wait that ran out raises the error words and marks the CTA; its threads go on
    // (on whatever is in shared memory) to the next point where the CTA leaves together.
    auto fail = [&]() {
        *reinterpret_cast<volatile int*>(&bad) = 1;
        atomicExch(a.err, 1);
        atomicExch(a.derr, 1);
    };
    bool ok = true;
    unsigned aphase = 0;  // applications so far: phase of zbar, wbar and vbar
    // C <- (I - V T^T V^T) C (trans) or (I - V T V^T) C of panel kk on the columns in Cs
    auto apply = [&](int kk, bool trans) -> bool {
        __syncthreads();  // Cs and Vs are settled
        if (tid == 0) {
            int f = 0;
            if (*reinterpret_cast<volatile int*>(&bad) == 0) {
                const int* rd = a.ready + kk * C + rank;
                for (long long it = 1; it <= a.spin_limit; ++it) {
                    if (qc_ld_relaxed(rd)) {
                        f = qc_ld_acquire(rd);
                        break;
                    }
                    if ((it & 15) == 0 && qc_ld_relaxed(a.err)) break;
                    if (it > 256) __nanosleep(32);
                }
                if (!f) {
                    atomicExch(a.err, 1);
                    atomicExch(a.derr, 1);
                }
            }
            if (f) {
                asm volatile("fence.proxy.async;" ::: "memory");
                qc_mbar_expect(&vbar, vbytes);
                const double* src = a.pub + ((long long)kk * C + rank) * L::msg;
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        qc_smem(Vs)),
                    "l"(src), "r"(vbytes), "r"(qc_smem(&vbar))
                    : "memory");
                qc_mbar_expect(&zbar, 32 * 32 * 8);
                qc_mbar_expect(&wbar, 32 * 32 * 8);
            }
            flag_ok = f;
        }
        __syncthreads();
        if (!flag_ok) return false;
        const unsigned ph = aphase & 1;
        ++aphase;
        if (!qc_mbar_wait(&vbar, ph, QC_POLLS, nullptr)) fail();  // this CTA's own copy
        const int lr0 = 32 * kk / (SL * C) * SL;        // local rows above are zero in V
        // Z = V^T C over the CTA's rows: 16 tiles of 8 x 8 dealt to the warps
        {
            constexpr int JN = 16 / W;
            const int rt = w & 3, j0 = (w >> 2) * JN;
            double acc[JN][2], ac2[JN][2];  // two halves of the rows' chain: less rounding, more in flight
#pragma unroll
            for (int j = 0; j < JN; ++j) acc[j][0] = acc[j][1] = ac2[j][0] = ac2[j][1] = 0.0;
            const double* vp = Vs + (8 * rt + gid) * ldr + tig;
            const double* cp = Cs + (8 * j0 + gid) * ldr + tig;
#pragma unroll 2
            for (int r = lr0; r < L::rows; r += 8) {
                const double av = vp[r], aw = vp[r + 4];
#pragma unroll
                for (int j = 0; j < JN; ++j) dmma(acc[j], av, cp[8 * j * ldr + r]);
#pragma unroll
                for (int j = 0; j < JN; ++j) dmma(ac2[j], aw, cp[8 * j * ldr + r + 4]);
            }
            // to the CTA that owns the columns: [source][row][column in slice]
#pragma unroll
            for (int j = 0; j < JN; ++j) {
                const int col = 8 * (j0 + j) + 2 * tig, dst = col / SC;
                const int at = rank * 32 * SC + (8 * rt + gid) * SC + col % SC;
                qc_st_async(qc_remote(qc_smem(zp + at), dst), acc[j][0] + ac2[j][0], acc[j][1] + ac2[j][1],
                            qc_remote(qc_smem(&zbar), dst));
            }
        }
        if (!qc_mbar_wait(&zbar, ph, a.polls, a.err)) fail();
        // Z2 = T^T Z or T Z on the slice, -Z2 to every CTA
        for (int ct = w >> 2; 8 * ct < SC; ct += W / 4) {
            const int rt = w & 3;
            const bool in = 8 * ct + gid < SC;  // C = 8: slices of 4 columns
            double acc[2] = {0.0, 0.0};
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const int kr = 4 * ks + tig;
                double z = 0.0;
#pragma unroll
                for (int src = 0; src < C; ++src) z += in ? zp[src * 32 * SC + kr * SC + 8 * ct + gid] : 0.0;
                dmma(acc, trans ? Ts[kr * QC_TLD + 8 * rt + gid] : Ts[(8 * rt + gid) * QC_TLD + kr], z);
            }
            if (8 * ct + 2 * tig < SC) {
                const unsigned at = qc_smem(z2 + (8 * rt + gid) * QC_ZLD + rank * SC + 8 * ct + 2 * tig);
#pragma unroll
                for (int d = 0; d < C; ++d)
                    qc_st_async(qc_remote(at, d), -acc[0], -acc[1], qc_remote(qc_smem(&wbar), d));
            }
        }
        if (!qc_mbar_wait(&wbar, ph, a.polls, a.err)) fail();
        // C += V (-Z2), row tiles of 8 dealt to the warps
        double bz[4][8];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) bz[j][ks] = z2[(4 * ks + tig) * QC_ZLD + 8 * j + gid];
#pragma unroll 2
        for (int r = lr0 + 8 * w; r < L::rows; r += 8 * W) {
            // the product by itself, then one addition to C: one rounding of C's size instead of eight
            double av[8], acc[4][2];
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) av[ks] = Vs[(4 * ks + tig) * ldr + r + gid];
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc[j], av[ks], bz[j][ks]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                Cs[(8 * j + 2 * tig) * ldr + r + gid] += acc[j][0];
                Cs[(8 * j + 2 * tig + 1) * ldr + r + gid] += acc[j][1];
            }
        }
        return true;
    };
    for (int kk = 0; ok && kk < nap; ++kk) ok = apply(kk, true);
    // the panel's messages land where Z2 was read
    cl.sync();
    if (bad) ok = false;
    if (ok && q < a.K && !qrows) {
        // ---- the panel.  Lane (gid, tig): rows 4i + tig of the warp's 8 in a slot, columns gid + 8c; rows of slot rp
        // (the pivots') first, finished slots left out.  `lc` is the column whose sums this lane has.
        const int b = min(32, a.k - c0), rp = c0 / (SL * C), prow0 = c0 - rp * SL * C;  // pivots: slot rp, from prow0 on
        const int gw = rank * W + w, lc = gid + 8 * tig;
        constexpr int PR = 2 * RL;
        double p[PR][4];
#pragma unroll
        for (int r = 0; r < PR; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int sl = rp + (r >> 1);
                p[r][c] = sl < RL ? Cs[(gid + 8 * c) * ldr + sl * SL + w * 8 + 4 * (r & 1) + tig] : 0.0;
            }
        const int pr0 = gw * 8 + tig;  // this lane's rows of the pivots' slot: pr0 and pr0 + 4
        if (tid < 32) {
            sc_s[tid] = 1.0;
            be_s[tid] = 0.0;
        }
        unsigned dsum[C], dbar[C];  // this lane's place in the receivers' buffers, their barriers
#pragma unroll
        for (int d = 0; d < C; ++d) {
            dsum[d] = qc_remote(qc_smem(recv + gw * 32 + lane), d);
            dbar[d] = qc_remote(qc_smem(&pbar[0]), d);
        }
        const unsigned drow = qc_smem(rowj + 4 * gid) - qc_smem(recv + gw * 32 + lane);
        __syncthreads();
        constexpr unsigned step_bytes = NS * 32 * 8 + 32 * 8;
        bool live = true;  // after a failed wait: no more waiting
        // T by rows: 32 / W rows per warp, four lanes to a row, each with eight columns (W = 8: the upper half of
        // the lanes repeats the lower).  Column jt is formed while the sums of the next step travel:
        // T(i, jt) = -tau sum_k T(i, k) v_k^T v_jt.
        constexpr int TR = 32 / W;
        const int ti = TR * w + gid % TR;
        double myscal = 1.0, gl = 0.0, tl = 0.0;  // scal of column lc; Gram entry and tau of the last step
        double tr[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) tr[c] = 0.0;
        auto t_column = [&](int jt) {
            gcol[w][lc] = lc < jt ? gl : 0.0;
            __syncwarp();
            double s0 = 0.0, s1 = 0.0;
#pragma unroll
            for (int c = 0; c < 8; c += 2) {
                const double2 g = *reinterpret_cast<const double2*>(&gcol[w][8 * tig + c]);
                s0 = fma(tr[c], g.x, s0);
                s1 = fma(tr[c + 1], g.y, s1);
            }
            double t = s0 + s1;
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            t = ti < jt ? -tl * t : ti == jt ? tl : 0.0;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (8 * tig + c == jt) tr[c] = t;
        };
#pragma unroll
        for (int jc = 0; jc < 4; ++jc) {
#pragma unroll 2
            for (int jj = 0; jj < 8; ++jj) {
                const int j = 8 * jc + jj, par = jj & 1;
                if (j < b) {
                    const int pj = prow0 + j;  // the pivot's row within its slot
                    double u[PR], s[4];
#pragma unroll
                    for (int r = 0; r < PR; ++r) u[r] = qc_shfl(p[r][jc], 4 * jj + tig);
                    // row j, from the eight lanes that hold it
                    if (gw == pj >> 3 && tig == (pj & 3)) {
                        const bool hi = pj & 4;
#pragma unroll
                        for (int d = 0; d < C; ++d) {
                            const unsigned at = dsum[d] + drow + par * 256, mb = dbar[d] + 8 * par;
                            qc_st_async(at, hi ? p[1][0] : p[0][0], hi ? p[1][1] : p[0][1], mb);
                            qc_st_async(at + 16, hi ? p[1][2] : p[0][2], hi ? p[1][3] : p[0][3], mb);
                        }
                    }
                    if (pr0 <= pj) u[0] = 0.0;
                    if (pr0 + 4 <= pj) u[1] = 0.0;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        double x = 0, y = 0;
#pragma unroll
                        for (int r = 0; r < PR; r += 2) {
                            x = fma(u[r], p[r][c], x);
                            y = fma(u[r + 1], p[r + 1][c], y);
                        }
                        s[c] = x + y;
                    }
                    // transposed butterfly over tig: lane ends with column lc
                    const bool b1 = tig & 2, b0 = tig & 1;
                    double t2[2];
#pragma unroll
                    for (int c = 0; c < 2; ++c)
                        t2[c] = (b1 ? s[c + 2] : s[c]) + __shfl_xor_sync(0xffffffffu, b1 ? s[c] : s[c + 2], 2);
                    const double part = (b0 ? t2[1] : t2[0]) + __shfl_xor_sync(0xffffffffu, b0 ? t2[0] : t2[1], 1);
#pragma unroll
                    for (int d = 0; d < C; ++d) qc_st_async(dsum[d] + par * NS * 256, part, dbar[d] + 8 * par);
                    if (tid == 0 && live) qc_mbar_expect(&pbar[par], step_bytes);  // one arrival per phase
                    if (j > 0) t_column(j - 1);
                    if (live && !qc_mbar_wait(&pbar[par], (j >> 1) & 1, a.polls, a.err)) {
                        live = false;
                        fail();
                    }
                    const double ar = rowj[par * 32 + lane];
                    double S;
                    {
                        const double* rv = recv + par * NS * 32 + lane;
                        double s4[4] = {0, 0, 0, 0};
#pragma unroll
                        for (int x = 0; x < NS; x += 4)
#pragma unroll
                            for (int y = 0; y < 4; ++y) s4[y] += rv[(x + y) * 32];
                        S = (s4[0] + s4[1]) + (s4[2] + s4[3]);
                    }
                    fs[w][0][lc] = S;
                    fs[w][1][lc] = ar;
                    __syncwarp();
                    const double xn2 = fs[w][0][j], alpha = fs[w][1][j];
                    double cu[4], ca[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        cu[c] = fs[w][0][gid + 8 * c];
                        ca[c] = fs[w][1][gid + 8 * c];
                    }
                    // w_j = u_j + (alpha - beta) e_j, beta = -sign(alpha) |(alpha, u)|, H = I - kap w w^T with
                    // kap = 1 / (|beta| |alpha - beta|): two reciprocal square roots, each with one Newton
                    // correction, on the chain; dlarfg's tau and 1 / (alpha - beta) by division beside it.
                    double kap = 0, beta = alpha, amb = 0;
                    if (xn2 > 0.0) {
                        const double n2 = fma(alpha, alpha, xn2), rn = rsqrt(n2);
                        double nrm = n2 * rn;
                        nrm = fma(0.5 * rn, fma(-nrm, nrm, n2), nrm);
                        const double den = fma(fabs(alpha), nrm, n2), rd = rsqrt(den);
                        kap = rd * rd;
                        kap = fma(kap, fma(-den, kap, 1.0), kap);
                        beta = alpha >= 0 ? -nrm : nrm;
                        amb = alpha - beta;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) cu[c] = gid + 8 * c > j ? kap * fma(amb, ca[c], cu[c]) : 0.0;
                    if (pr0 == pj) u[0] = amb;
                    if (pr0 + 4 == pj) u[1] = amb;
#pragma unroll
                    for (int r = 0; r < PR; ++r)
#pragma unroll
                        for (int c = 0; c < 4; ++c) p[r][c] = fma(-cu[c], u[r], p[r][c]);
                    const bool trivial = !(amb != 0.0);
                    const double scal = trivial ? 1.0 : 1.0 / amb;
                    gl = myscal * fma(scal, S, ar);  // v_lc^T v_j (lc < j)
                    tl = trivial ? 0.0 : -amb / beta;
                    if (lc == j) {
                        myscal = scal;
                        if (w == 0) {
                            sc_s[j] = scal;
                            be_s[j] = beta;
                        }
                    }
                }
            }
        }
        t_column(b - 1);
#pragma unroll
        for (int c = 0; c < 8; ++c) Ts[ti * QC_TLD + 8 * tig + c] = tr[c];
        __syncthreads();
        // V (unit diagonal, zeros above) into Vs, R's entries into Cs
        for (int sl = 0; sl < rp; ++sl)
#pragma unroll
            for (int c = 0; c < 8; ++c) Vs[(gid + 8 * (c >> 1)) * ldr + sl * SL + w * 8 + 4 * (c & 1) + tig] = 0.0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int col = gid + 8 * c, piv = prow0 + col;
            const double sc = sc_s[col], be = be_s[col];
#pragma unroll
            for (int r = 0; r < PR; ++r) {
                if (rp + (r >> 1) < RL) {
                    const int at = col * ldr + (rp + (r >> 1)) * SL + w * 8 + 4 * (r & 1) + tig;
                    const int row = r < 2 ? pr0 + 4 * r : piv + 1;
                    Vs[at] = (row < piv || col >= b) ? 0.0 : row == piv ? 1.0 : sc * p[r][c];
                    if (r < 2 || col >= b)  // (k < n within the block: columns past the panel)
                        Cs[at] = row == piv && col < b ? be : p[r][c];
                }
            }
        }
        asm volatile("fence.proxy.async;" ::: "memory");  // read by a bulk copy
        __syncthreads();
        if (tid == 0 && bad == 0) {
            double* out = a.pub + ((long long)q * C + rank) * L::msg;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out), "r"(qc_smem(Vs)),
                         "r"(vbytes)
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;\ncp.async.bulk.wait_group 0;" ::: "memory");
            qc_st_release(a.ready + q * C + rank, 1);
        }
        ok = bad == 0;
    }
    cl.sync();  // nor may a mate's partial Z land where the last step's sums are read
    if (ok && a.R && !qrows)  // this block's columns of R
        each(a.k, a.rrs == 1, [&](int c, int lr, int i) {
            if (i < a.k && c < ncol)
                a.R[(long long)i * a.rrs + (long long)(c0 + c) * a.rcs] = i <= c0 + c ? Cs[c * ldr + lr] : 0.0;
        });
    if (qrows) {
        __syncthreads();
        if (ok && bad == 0)  // column c of Q^T is row c0 + c of Q
            each(a.k, a.qcs == 1, [&](int c, int lr, int i) {
                if (i < a.k && c < ncol) a.Q[(long long)(c0 + c) * a.qrs + (long long)i * a.qcs] = Cs[c * ldr + lr];
            });
    } else if (ok && a.Q && a.nb * C == (int)gridDim.x && q < a.K) {
        // no clusters for Q's rows: Q(:, block) = H_0 .. H_q [e_c]
        const int b = min(32, a.k - c0);
        __syncthreads();
        each(L::rows * C, true, [&](int c, int lr, int i) { Cs[c * ldr + lr] = i == c0 + c ? 1.0 : 0.0; });
        for (int kk = q; ok && kk >= 0; --kk) ok = apply(kk, false);
        __syncthreads();
        if (ok && bad == 0)
            each(a.m, a.qrs == 1, [&](int c, int lr, int i) {
                if (i < a.m && c < b) a.Q[(long long)i * a.qrs + (long long)(c0 + c) * a.qcs] = Cs[c * ldr + lr];
            });
    }
    if (q < a.K && !qrows && w == 1) qc_check_range(sc_s, a.derr + 1);
    cl.sync();  // no CTA leaves while its shared memory may still be addressed
    // after a failure messages that nobody waits for may still be on their way
    if (qc_ld_acquire(a.err)) __nanosleep(200000);
    cl.sync();
}

// Enqueues with clusters for Q's rows if all clusters can be resident, else without them; *served stays
// false when neither fits.
template <int RL, int C, int W>
int qc_launch(Ctx& c, QcArgs a, bool* served) {
    using L = QcLayout<RL, C, W>;
    static_assert(sizeof(double) * L::end + 18 * 256 <= 227 * 1024, "shared memory");
    constexpr size_t smem = sizeof(double) * L::end;
    auto kern = qr_cluster_kernel<RL, C, W>;
    TN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(32 * W);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeCooperative;
    at[1].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const int with_q = a.Q ? a.nb + (a.m + 31) / 32 : a.nb;
    int clusters = with_q, fit = 0;
    // clusters wait for the ones before them: all of them have to be resident
    cfg.gridDim = dim3((unsigned)(C * clusters));
    if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return TN_OK;
    }
    if (fit < clusters) clusters = a.nb;
    if (fit < clusters) return TN_OK;
    TN_CHECK(c.qrw.ensure(sizeof(double) * (size_t)L::msg * a.K * C));
    TN_CHECK(c.qrsync.ensure(sizeof(int) * ((size_t)a.K * C + 1)));
    TN_CHECK(ensure_device_error_word(c));
    a.pub = c.qrw.as<double>();
    a.err = c.qrsync.as<int>();
    a.ready = a.err + 1;
    a.derr = c.derr.as<int>();
    a.spin_limit = c.qr_spin_limit;
    a.polls = c.wait_polls < 0 ? QC_POLLS : c.wait_polls;
    TN_CUDA_CHECK(cudaMemsetAsync(c.qrsync.p, 0, sizeof(int) * ((size_t)a.K * C + 1), c.stream));
    cfg.gridDim = dim3((unsigned)(C * clusters));
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return TN_OK;
    }
    TN_CUDA_CHECK(e);
    count_launch();
    *served = true;
    return TN_OK;
}

}  // namespace

int qr_cluster(Ctx& c, int m, int n, const double* A, long long ars, long long acs, double* Q, long long qrs,
               long long qcs, double* R, long long rrs, long long rcs, const int* colmap) {
    if (!c.use_cluster_qr || !c.use_persistent_qr || !c.qr_forward_q || m < 1 || n < 1 || m > 1536) return QR_UNAVAILABLE;
    const int k = std::min(m, n);
    // a block of A is read when its cluster starts: outputs in A's memory take the path with a copy
    auto span = [](const double* p, int r, int cl, long long rs, long long cs) {
        const long long x = (r - 1) * rs, y = (cl - 1) * cs;
        return std::make_pair(p + std::min(0LL, x) + std::min(0LL, y), p + std::max(0LL, x) + std::max(0LL, y));
    };
    const auto sa = span(A, m, n, ars, acs);
    auto meets = [&](const std::pair<const double*, const double*>& o) {
        return o.first <= sa.second && sa.first <= o.second;
    };
    if ((Q && meets(span(Q, m, k, qrs, qcs))) || (R && meets(span(R, k, n, rrs, rcs)))) return QR_UNAVAILABLE;
    QcArgs a{};
    a.m = m; a.n = n; a.k = k;
    a.K = (k + 31) / 32;
    a.nb = (n + 31) / 32;
    a.A = A; a.ars = ars; a.acs = acs; a.colmap = colmap;
    a.Q = Q; a.qrs = qrs; a.qcs = qcs;
    a.R = R; a.rrs = rrs; a.rcs = rcs;
    bool served = false;
    int st = TN_OK;
    // Rows per CTA: as few as keep the exchange small.  A call of tn_qr with half the CTAs a cluster: 128 x 128 165 us
    // (151 here), 256 x 256 300 (278); with twice as many (RL = 2): 512 x 256 351 (324), 512 x 1536 735 (634);
    // with 8 warps a CTA instead of 8 CTAs: 1024 x 512 1020 (819) -- above 512 rows that is left for when the
    // clusters of 8 do not all fit (1536 x 512: 15 of 16).
    if (m <= 32) st = qc_launch<1, 1, 4>(c, a, &served);
    else if (m <= 64) st = qc_launch<2, 1, 4>(c, a, &served);
    else if (m <= 128) st = qc_launch<2, 2, 4>(c, a, &served);
    else if (m <= 256) st = qc_launch<2, 4, 4>(c, a, &served);
    else if (m <= 384) st = qc_launch<3, 4, 4>(c, a, &served);
    else if (m <= 512) st = qc_launch<4, 4, 4>(c, a, &served);
    else if (m <= 1024) {
        st = qc_launch<4, 8, 4>(c, a, &served);
        if (!st && !served) st = qc_launch<4, 4, 8>(c, a, &served);
    } else {
        st = qc_launch<6, 8, 4>(c, a, &served);
        if (!st && !served) st = qc_launch<6, 4, 8>(c, a, &served);
    }
    return st ? st : served ? TN_OK : QR_UNAVAILABLE;
}

}  // namespace tnb
