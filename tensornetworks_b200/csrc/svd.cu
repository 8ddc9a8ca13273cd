// svd.cu -- one-sided (Hestenes) Jacobi SVD in FP64: a thread-block cluster per
// matrix with the columns in registers, or one CTA per matrix past its limits.
//
// Replaces LapackSVDSolver<T>::Solve (zgesvd, LapackSVDSolver.C:42-90).  The
// columns of the tall working matrix are orthogonalised pairwise; pairs follow
// the round-robin (circle) ordering so that all n/2 pairs of a round are
// independent and run on different warps; rotation angles, dot products and
// convergence tests are FP64.  Small problems run entirely in shared memory.
// Singular values come out descending; zero singular values get orthonormal
// completion columns in U (as zgesvd provides), which the zero-padded bond
// growth of the sweep relies on.  A batch of matrices runs as one launch.
#include <cooperative_groups.h>

#include <algorithm>

#include "qr.h"

namespace cg = cooperative_groups;

namespace tnb {

namespace {

constexpr int SVD_THREADS = 512;
constexpr int SVD_MAX_SWEEPS = 60;

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The power of two that the rows to be orthogonalised are multiplied by, from their largest entry: 1 between
// 2^-400 and 2^400 (and for zero, an infinity or NaN), else what brings it near 1.  Squared norms and dots then
// neither underflow nor overflow for the columns that count.
__device__ __forceinline__ double jc_matrix_scale(double amax) {
    const int e = (__double2hiint(amax) >> 20) & 0x7ff;
    if (amax == 0.0 || e == 0x7ff || (e >= 0x3ff - 400 && e <= 0x3ff + 400)) return 1.0;
    return __hiloint2double(max(1, 0x7fe - e) << 20, 0);
}

// Descending order of values with their indices, NaN first: a total order, so that every column gets its own place.
__device__ __forceinline__ bool ranks_before(double si, int i, double sj, int j) {
    const bool ni = si != si, nj = sj != sj;
    return ni || nj ? (ni && (!nj || i < j)) : si > sj || (si == sj && i < j);
}

__device__ __forceinline__ double nan_value() { return __longlong_as_double(0x7ff8000000000000LL); }

// A column of U is that of the matrix, not one of its completion.  (NaN: the values of a matrix with a NaN in it
// are all NaN, and nothing is completed.)
__device__ __forceinline__ bool keeps_column(double s, double cut) { return !(s <= cut) && s != 0.0; }

__device__ __forceinline__ int rr_pos(int q, int r, int ne) {
    return q == 0 ? 0 : ((q - 1 + r) % (ne - 1)) + 1;
}

// Orthonormal completion of the U columns whose singular value is at most the
// cut, by one whole block: unit vectors e_0, e_1, ... projected off every
// accepted column (classical Gram-Schmidt applied twice: all dots of a pass are
// independent, a warp each, and one barrier separates them from the update; the
// column-after-column form takes three barriers per column), kept when more
// than half of the unit vector is left.  Once the unit vectors are used up (the
// rest of the space may be spread evenly over them), the one with the largest
// remainder 1 - sum_p U(e, p)^2 is taken, which is never zero while columns are
// missing.  U is read by L2 loads: other CTAs may have written it in this
// launch.  U(i, c), i < m, at U[i rs + c cs].  dots: n doubles of shared memory, red and at: 32 each.
__device__ void complete_u(const SvdJob& jb, double* U, long long rs, long long cs, int m, double cut, double* red,
                           double* dots, int* at) {
    const int n = jb.n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    int next_e = 0;
    for (int c = 0; c < n; ++c) {
        const double sc = __ldcg(jb.s + c);
        if (keeps_column(sc, cut)) continue;
        double* uc = U + c * cs;
        auto accepted = [&](int p) {
            const double sp = __ldcg(jb.s + p);
            return p != c && (keeps_column(sp, cut) || p < c);
        };
        for (bool placed = false; !placed;) {
            int e = next_e++;
            const bool last = e >= m;
            if (last) {
                double best = -1.0;
                int bi = 0;
                for (int i = tid; i < m; i += blockDim.x) {
                    double r = 1.0;
                    for (int p = 0; p < n; ++p)
                        if (accepted(p)) {
                            const double u = __ldcg(U + p * cs + i * rs);
                            r = fma(-u, u, r);
                        }
                    if (r > best) { best = r; bi = i; }
                }
                for (int o = 16; o > 0; o >>= 1) {
                    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
                }
                if (lane == 0) {
                    red[wid] = best;
                    at[wid] = bi;
                }
                __syncthreads();
                if (tid == 0) {
                    int w0 = 0;
                    for (int w = 1; w < nw; ++w)
                        if (red[w] > red[w0]) w0 = w;
                    at[0] = at[w0];
                }
                __syncthreads();
                e = at[0];
            }
            for (int i = tid; i < m; i += blockDim.x) uc[i * rs] = (i == e) ? 1.0 : 0.0;
            __syncthreads();
            for (int pass = 0; pass < 2; ++pass) {
                for (int p = wid; p < n; p += nw) {
                    double part = 0;
                    if (accepted(p)) {
                        const double* up = U + p * cs;
                        for (int i = lane; i < m; i += 32) part = fma(__ldcg(up + i * rs), __ldcg(uc + i * rs), part);
                    }
                    part = wsum(part);
                    if (lane == 0) dots[p] = part;
                }
                __syncthreads();
                for (int i = tid; i < m; i += blockDim.x) {
                    double v = __ldcg(uc + i * rs);
                    for (int p = 0; p < n; ++p)
                        if (dots[p] != 0.0) v = fma(-dots[p], __ldcg(U + p * cs + i * rs), v);
                    uc[i * rs] = v;
                }
                __syncthreads();
            }
            double part = 0;
            for (int i = tid; i < m; i += blockDim.x) part = fma(__ldcg(uc + i * rs), __ldcg(uc + i * rs), part);
            part = wsum(part);
            if (lane == 0) red[wid] = part;
            __syncthreads();
            double nr2 = 0;
            for (int w = 0; w < nw; ++w) nr2 += red[w];
            __syncthreads();
            const double nr = sqrt(nr2);
            if (nr > 0.5 || last) {
                for (int i = tid; i < m; i += blockDim.x) uc[i * rs] = nr > 0.0 ? __ldcg(uc + i * rs) / nr : 0.0;
                placed = true;
            }
            __syncthreads();
        }
    }
}

__global__ void __launch_bounds__(SVD_THREADS) jacobi_svd_kernel(const SvdJob* __restrict__ jobs, int vectors,
                                                                   size_t smem_cap) {
    extern __shared__ double smem[];
    const SvdJob jb = jobs[blockIdx.x];
    const int m = jb.m, n = jb.n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    __shared__ int s_rot;
    __shared__ int s_sweeps;
    __shared__ double red[32];
    __shared__ int at[32];

    // shared memory: norms (n), ranks (n ints), then A (m x n) and V (n x n) when they fit
    double* norms = smem;
    int* rank = reinterpret_cast<int*>(smem + n);
    double* tail = smem + n + (n + 1) / 2 + 1;
    size_t fixed = (size_t)n + (n + 1) / 2 + 1;
    size_t need = fixed + (size_t)m * n + (vectors ? (size_t)n * n : 0);
    bool in_smem = need * sizeof(double) <= smem_cap;
    double* A = in_smem ? tail : jb.W;
    double* V = vectors ? (in_smem ? tail + (size_t)m * n : jb.V) : nullptr;
    double amax = 0.0;
    for (size_t e = tid; e < (size_t)m * n; e += blockDim.x) amax = fmax(amax, fabs(jb.W[e]));
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) red[wid] = amax;
    __syncthreads();
    for (int w = 0; w < nw; ++w) amax = fmax(amax, red[w]);
    const double scale = jc_matrix_scale(amax);
    if (in_smem || scale != 1.0)
        for (size_t e = tid; e < (size_t)m * n; e += blockDim.x) A[e] = scale * jb.W[e];
    if (vectors)
        for (size_t e = tid; e < (size_t)n * n; e += blockDim.x) V[e] = ((e % n) == (e / n)) ? 1.0 : 0.0;
    __syncthreads();

    const int ne = n + (n & 1);
    const double tol = 1e-15 * fmax(1.0, sqrt((double)m) / 4.0);
    int sweep = 0;
    for (sweep = 0; sweep < SVD_MAX_SWEEPS && n > 1; ++sweep) {
        if (tid == 0) s_rot = 0;
        __syncthreads();
        for (int r = 0; r < ne - 1; ++r) {
            for (int p = wid; p < ne / 2; p += nw) {
                int a = rr_pos(p, r, ne), b = rr_pos(ne - 1 - p, r, ne);
                if (a >= n || b >= n) continue;
                double* ca = A + (size_t)a * m;
                double* cb = A + (size_t)b * m;
                double al = 0, be = 0, ga = 0;
                for (int i = lane; i < m; i += 32) {
                    double x = ca[i], y = cb[i];
                    al = fma(x, x, al);
                    be = fma(y, y, be);
                    ga = fma(x, y, ga);
                }
                al = wsum(al);
                be = wsum(be);
                ga = wsum(ga);
                if (ga == 0.0 || fabs(ga) <= tol * sqrt(al * be)) continue;
                double zeta = (be - al) / (2.0 * ga);
                double t = (zeta >= 0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
                double c = 1.0 / sqrt(1.0 + t * t), s = c * t;
                for (int i = lane; i < m; i += 32) {
                    double x = ca[i], y = cb[i];
                    ca[i] = c * x - s * y;
                    cb[i] = s * x + c * y;
                }
                if (vectors) {
                    double* va = V + (size_t)a * n;
                    double* vb = V + (size_t)b * n;
                    for (int i = lane; i < n; i += 32) {
                        double x = va[i], y = vb[i];
                        va[i] = c * x - s * y;
                        vb[i] = s * x + c * y;
                    }
                }
                if (lane == 0) s_rot = 1;
            }
            __syncthreads();
        }
        int rot = s_rot;
        __syncthreads();
        if (!rot) break;
    }
    if (tid == 0) s_sweeps = sweep;

    // column norms = singular values (unsorted)
    for (int j = wid; j < n; j += nw) {
        const double* cj = A + (size_t)j * m;
        double s = 0;
        for (int i = lane; i < m; i += 32) s = fma(cj[i], cj[i], s);
        s = wsum(s);
        if (lane == 0) norms[j] = sqrt(s);
    }
    __syncthreads();
    // descending rank, ties broken by column index; a NaN anywhere makes every value NaN
    bool nan = false;
    for (int j = 0; j < n; ++j) nan = nan || norms[j] != norms[j];
    const double unscale = nan ? nan_value() : 1.0 / scale;
    for (int j = tid; j < n; j += blockDim.x) {
        const double sj = norms[j];
        int rk = 0;
        for (int i = 0; i < n; ++i) rk += ranks_before(norms[i], i, sj, j);
        rank[j] = rk;
        jb.s[rk] = sj * unscale;
    }
    __syncthreads();
    double smax = 0;
    for (int j = 0; j < n; ++j) smax = fmax(smax, norms[j]);
    const double cut = smax * 1e-13 * fmax(1.0, (double)m) * unscale;
    if (vectors) {
        for (int j = wid; j < n; j += nw) {
            const int rk = rank[j];
            const double sj = norms[j];
            const double* cj = A + (size_t)j * m;
            double* uo = jb.U + (size_t)rk * jb.ldu;
            const bool good = keeps_column(sj * unscale, cut);
            for (int i = lane; i < m; i += 32) uo[i] = good ? cj[i] / sj : 0.0;
            const double* vj = V + (size_t)j * n;
            for (int i = lane; i < n; i += 32) jb.Vt[(size_t)i * jb.ldvt + rk] = vj[i];
        }
        __syncthreads();
        complete_u(jb, jb.U, 1, jb.ldu, m, cut, red, norms, at);
    }
    if (tid == 0 && jb.sweeps) *jb.sweeps = s_sweeps;
}

// ---------------------------------------------------------------------------
// Cluster kernel: one matrix per thread-block cluster, its columns in registers.
//
// Warp w of the cluster holds four columns, two blocks of two ("top" and
// "bottom"); lane l holds rows l + 32 q of each, the matrix's rows in the first
// ET slots and, with vectors, the accumulated rotations' rows after them, so a
// rotation is one pass over the registers.  A round rotates the four
// top x bottom pairs as two steps of two independent pairs: the two dots of a
// step share one butterfly (pair 0 ends in lanes 0-15, pair 1 in 16-31), each
// half warp computes its own pair's angle at the same time, and one exchange
// hands it to the other half.  The columns' squared norms travel with them and
// follow the rotations, (al, be) -> (al - t ga, be + t ga); they are summed
// afresh at the start of every sweep, whose last one (no rotation left) is the
// convergence test.  Between rounds the blocks move one warp on (circle
// method, block 0 fixed): written straight into the receiving warp's inbox,
// in this CTA or by st.async in the neighbouring one, whose mbarrier counts the
// arrivals and bytes: a warp waits for its two neighbours only, and nothing
// needs a release at cluster scope (measured at over 1000 cycles).  Inboxes alternate by round parity; what a warp
// received in round r + 1 tells that the neighbours have emptied theirs of
// round r.  Where two parities do not fit, a cluster barrier per round frees
// the one.
//
// What bounds it: the serial chain of a round -- inbox read, two times (dot,
// butterfly, angle, update: 650-1000 cycles), write -- 1.3-1.9 us, times
// n / 2 - 1 rounds, times the sweeps (9-11 after a QR factorisation, 14-19 without).  One CTA per matrix spends that latency per pair of each
// warp's share and reads every column from shared memory (or L2) three times
// per round.
constexpr int SVD_PRE_MIN = 25;   // columns from which a single matrix is factored first
constexpr int JC_SLOTS_MAX = 16;  // row slots per column: four columns x 16 doubles = 128 registers

__device__ __forceinline__ double jc_pick(bool hi, double a, double b) { return hi ? b : a; }

// pow2 scale bringing x (>= 0) near 1 (1 for x = 0 or not finite)
__device__ __forceinline__ double jc_scale(double x) {
    const int e = (__double2hiint(x) >> 20) & 0x7ff;
    return (e == 0 || e >= 0x7fe) ? 1.0 : __hiloint2double((0x7fe - e) << 20, 0);
}

// The rotations of the pairs (x0, y0) and (x1, y1); norms updated in place.
// With d = be - al, g2 = 2 ga and h = sqrt(d^2 + g2^2) the angle that
// orthogonalises a pair has cos(2 theta) = |d| / h, so c^2 = (1 + |d| / h) / 2
// (in [1/2, 1]: no cancellation) and s = g2 / (2 h c) with d's sign: two
// reciprocal square roots in a row (about 75 cycles each) where the tangent
// form takes two square roots and two divisions (400).
template <int E>
__device__ __forceinline__ bool jc_rotate2(double (&x0)[E], double (&y0)[E], double (&x1)[E], double (&y1)[E],
                                           double& nx0, double& ny0, double& nx1, double& ny1, int ET, double tol2) {
    const bool hi = threadIdx.x & 16;
    const double al = jc_pick(hi, nx0, nx1), be = jc_pick(hi, ny0, ny1);
    const bool real = al >= 0.0 && be >= 0.0;  // a padding column (norm -1) is never rotated
    const double sc = jc_scale(fmax(al, be));
    const double d = (be - al) * sc;
    // at least 2^-800: a smaller rotation changes nothing, and where the norms that followed the rotations have come
    // out zero (columns that were equal), the squares below would be denormal and the rotation no longer orthogonal
    const double thr = fma(tol2, (al * sc) * (be * sc), 0x1p-800);
    double a0 = 0, b0 = 0, a1 = 0, b1 = 0;
#pragma unroll
    for (int q = 0; q < E; q += 2) {
        if (q < ET) {
            a0 = fma(x0[q], y0[q], a0);
            a1 = fma(x1[q], y1[q], a1);
        }
        if (q + 1 < E && q + 1 < ET) {
            b0 = fma(x0[q + 1], y0[q + 1], b0);
            b1 = fma(x1[q + 1], y1[q + 1], b1);
        }
    }
    a0 += b0;
    a1 += b1;
    double g = jc_pick(hi, a0, a1) + __shfl_xor_sync(0xffffffffu, jc_pick(hi, a1, a0), 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    const double gs = g * sc, g2 = gs + gs;
    const bool rot = real && gs * gs > thr;
    if (!__any_sync(0xffffffffu, rot)) return false;
    const double rh = rsqrt(fma(d, d, g2 * g2));
    const double c2 = fma(0.5 * fabs(d), rh, 0.5);
    const double rc = rsqrt(c2);
    const double sn = 0.5 * g2 * rh * rc;
    const double c = rot ? c2 * rc : 1.0;
    const double s = rot ? (d >= 0 ? sn : -sn) : 0.0;
    const double co = __shfl_xor_sync(0xffffffffu, c, 16), so = __shfl_xor_sync(0xffffffffu, s, 16);
    const double c0 = jc_pick(hi, c, co), s0 = jc_pick(hi, s, so), c1 = jc_pick(hi, co, c), s1 = jc_pick(hi, so, s);
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const double u0 = x0[q], v0 = y0[q], u1 = x1[q], v1 = y1[q];
        x0[q] = fma(c0, u0, -s0 * v0);
        y0[q] = fma(s0, u0, c0 * v0);
        x1[q] = fma(c1, u1, -s1 * v1);
        y1[q] = fma(s1, u1, c1 * v1);
    }
    const double tg = s * rc * g;  // tan(theta) ga
    const double na = rot ? fmax(al - tg, 0.0) : al, nb = rot ? fmax(be + tg, 0.0) : be;
    const double nao = __shfl_xor_sync(0xffffffffu, na, 16), nbo = __shfl_xor_sync(0xffffffffu, nb, 16);
    nx0 = jc_pick(hi, na, nao);
    ny0 = jc_pick(hi, nb, nbo);
    nx1 = jc_pick(hi, nao, na);
    ny1 = jc_pick(hi, nbo, nb);
    return true;
}

template <int E>
__device__ __forceinline__ double jc_norm2(const double (&x)[E], int ET) {
    double a = 0, b = 0;
#pragma unroll
    for (int q = 0; q < E; q += 2) {
        if (q < ET) a = fma(x[q], x[q], a);
        if (q + 1 < E && q + 1 < ET) b = fma(x[q + 1], x[q + 1], b);
    }
    return wsum(a + b);
}

// Doubles of one inbox slot: a block's two columns interleaved by lane (16-byte
// accesses, no bank conflicts) and its two norms.
template <int E> __host__ __device__ constexpr int jc_slot() { return 64 * E + 2; }

template <int E>
size_t jc_smem_bytes(int warps, int parities, int nmax) {
    return sizeof(double) * ((size_t)jc_slot<E>() * 2 * warps * parities + (size_t)nmax + 2) + sizeof(int) * nmax;
}

__device__ __forceinline__ unsigned jc_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void jc_mbar_init(unsigned long long* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(jc_smem(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void jc_mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(jc_smem(b)) : "memory");
}
__device__ __forceinline__ void jc_mbar_expect(unsigned long long* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(jc_smem(b)), "r"(bytes)
                 : "memory");
}
// the shared::cluster address, in CTA `rank`, of this CTA's shared memory address p
__device__ __forceinline__ unsigned jc_remote(const void* p, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(jc_smem(p)), "r"(rank));
    return r;
}
// 16 bytes into another CTA's shared memory, counted by the mbarrier there
__device__ __forceinline__ void jc_st_async(unsigned dst, double a, double b, unsigned mbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "d"(a), "d"(b), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ bool jc_mbar_try(unsigned long long* b, unsigned phase) {
    unsigned done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(jc_smem(b)), "r"(phase)
        : "memory");
    return done;
}
// The polls after a warp's first: true in every lane once the phase has completed; false after `limit` polls,
// or when the error word says that another wait has run out.
__device__ __noinline__ bool jc_mbar_poll(unsigned long long* b, unsigned phase, int limit, const int* err) {
    for (int i = 1; i < limit; ++i) {
        if (__all_sync(0xffffffffu, jc_mbar_try(b, phase))) return true;
        if ((i & 15) == 0) {
            int e;
            asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(e) : "l"(err) : "memory");
            if (__any_sync(0xffffffffu, e)) return false;
        }
    }
    return false;
}
__device__ __forceinline__ bool jc_mbar_wait(unsigned long long* b, unsigned phase, int limit, const int* err) {
    if (limit > 0 && __all_sync(0xffffffffu, jc_mbar_try(b, phase))) return true;
    return jc_mbar_poll(b, phase, limit, err);
}
constexpr int JC_WAIT_POLLS = 1 << 20;  // a round takes about a microsecond; the waits end long before

template <int E>
__global__ void __launch_bounds__(256, 1) jacobi_cluster_kernel(const SvdJob* __restrict__ jobs, SvdJob one,
                                                                 int vectors, int parities, int nmax, int polls, int* __restrict__ derr) {
    extern __shared__ __align__(16) double smem[];
    cg::cluster_group cl = cg::this_cluster();
    const int ncta = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const SvdJob jb = jobs ? jobs[blockIdx.x / ncta] : one;
    const int m = jb.m, n = jb.n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    const int gw = rank * nw + wid;          // warp of the cluster
    const int NW = max(1, (n + 3) / 4);      // warps that hold columns
    const bool pre = jb.perm != nullptr;     // on R^T (n x n) with Q's rows below, see svd_batched
    const int mt = pre ? n : m, mb = pre ? m : n;  // rows that are orthogonalised, rows that follow
    const int ET = (mt + 31) / 32;
    const bool on = gw < NW;
    __shared__ int flags[3];                 // rank 0's are used: "something rotated", by sweep modulo 3
    __shared__ int failed;                   // rank 0's is used: a wait has run out
    __shared__ double red[32];
    __shared__ double scale_sh;              // for the singular values (not a register through the sweeps)
    __shared__ double wmax[8];               // largest entry of each warp's columns
    __shared__ int at[32];
    constexpr int SLOT = jc_slot<E>();
    double* inbox = smem;                    // [parity][warp][top, bottom][SLOT]
    double* sig = smem + (size_t)SLOT * 2 * nw * parities;  // nmax
    int* rk = reinterpret_cast<int*>(sig + nmax + 2);
    __shared__ unsigned long long mbar[2][8];  // [parity][warp]: the blocks of this round are in the inbox
    if (tid < 3) flags[tid] = 0;
    if (tid == 0) failed = 0;
    // mbarrier of a warp's inbox: one arrival from each neighbour in this CTA, and the
    // warp's own, which also announces the bytes of those in other CTAs
    const bool from_left = on && gw > 0, from_right = on && gw < NW - 1;
    const bool left_here = wid > 0, right_here = wid + 1 < nw;  // where the neighbours are
    constexpr unsigned BLOCK_BYTES = 512 * E + 16;
    const unsigned remote_bytes =
        (from_left && !left_here ? BLOCK_BYTES : 0) + (from_right && !right_here ? BLOCK_BYTES : 0);
    if (lane == 0 && on && NW > 1) {
        const unsigned local = (from_left && left_here) + (from_right && right_here);
        jc_mbar_init(&mbar[0][wid], local + 1);
        jc_mbar_init(&mbar[1][wid], local + 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    auto slot = [&](int w, int which, int par) {  // inbox slot of warp w of this CTA
        return inbox + (size_t)SLOT * (((parities > 1 ? par * nw : 0) + w) * 2 + which);
    };
    double x0[E], x1[E], y0[E], y1[E];       // top block, bottom block
    double nx0, nx1, ny0, ny1;
    auto load = [&](double(&v)[E], int col) -> double {
#pragma unroll
        for (int q = 0; q < E; ++q) {
            double e = 0.0;
            if (on && col < n) {
                const int row = lane + 32 * q;
                const int low = row - 32 * ET;
                if (q < ET) e = row < mt ? jb.W[(size_t)col * mt + row] : 0.0;
                else if (!vectors) e = 0.0;
                else if (pre) e = low < mb ? jb.V[(size_t)col * mb + low] : 0.0;
                else e = low == col ? 1.0 : 0.0;
            }
            v[q] = e;
        }
        return (on && col < n) ? 0.0 : -1.0;
    };
    nx0 = load(x0, 2 * gw);
    nx1 = load(x1, 2 * gw + 1);
    ny0 = load(y0, 2 * (NW + gw));
    ny1 = load(y1, 2 * (NW + gw) + 1);
    // a block into the inbox of the neighbour on the left (side -1) or right (+1)
    auto put = [&](int side, int which, int par, const double(&a)[E], const double(&b)[E], double na, double nb) {
        if (side < 0 ? left_here : right_here) {
            double* p = slot(wid + side, which, par);
#pragma unroll
            for (int q = 0; q < E; ++q) reinterpret_cast<double2*>(p)[32 * q + lane] = make_double2(a[q], b[q]);
            if (lane == 0) reinterpret_cast<double2*>(p)[32 * E] = make_double2(na, nb);
            __syncwarp();
            if (lane == 0) jc_mbar_arrive(&mbar[par][wid + side]);
        } else {
            const int w = side < 0 ? nw - 1 : 0;
            const unsigned p = jc_remote(slot(w, which, par), rank + side);
            const unsigned mb = jc_remote(&mbar[par][w], rank + side);
#pragma unroll
            for (int q = 0; q < E; ++q) jc_st_async(p + 16 * (32 * q + lane), a[q], b[q], mb);
            if (lane == 0) jc_st_async(p + 16 * 32 * E, na, nb, mb);
        }
    };
    auto get = [&](const double* p, double(&a)[E], double(&b)[E], double& na, double& nb) {
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const double2 v = reinterpret_cast<const double2*>(p)[32 * q + lane];
            a[q] = v.x;
            b[q] = v.y;
        }
        const double2 v = reinterpret_cast<const double2*>(p)[32 * E];
        na = v.x;
        nb = v.y;
    };
    // the largest entry of this warp's columns; every warp gets the whole matrix's
    double amax = 0.0;
#pragma unroll
    for (int q = 0; q < E; ++q)
        if (q < ET) amax = fmax(amax, fmax(fmax(fabs(x0[q]), fabs(x1[q])), fmax(fabs(y0[q]), fabs(y1[q]))));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) wmax[wid] = amax;
    cl.sync();  // every CTA of the cluster runs before the first remote write; flags are zero
    amax = 0.0;
    for (int w = lane; w < ncta * nw; w += 32) amax = fmax(amax, cl.map_shared_rank(wmax, w / nw)[w % nw]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const double scale = jc_matrix_scale(amax);
    if (tid == 0) scale_sh = scale;
    if (scale != 1.0) {
#pragma unroll
        for (int q = 0; q < E; ++q)
            if (q < ET) {
                x0[q] *= scale;
                x1[q] *= scale;
                y0[q] *= scale;
                y1[q] *= scale;
            }
    }

    const double tol = 1e-15 * fmax(1.0, sqrt((double)m) / 4.0), tol2 = tol * tol;
    int sweep = 0;
    unsigned round = 0;  // over all sweeps: inbox parity and mbarrier phase
    // A warp whose wait ran out sends and waits no more; its neighbours' waits run out or see the error word, and the
    // cluster leaves together at the end of the sweep.  (Reported in front of the next barrier: by the wait
    // itself 256 x 256 took 3.78 instead of 3.54 ms.)
    bool live = on;
    auto report = [&]() {
        if (on && !live && lane == 0) {
            atomicExch(derr, 1);
            *cl.map_shared_rank(&failed, 0) = 1;
        }
    };
    for (sweep = 0; sweep < SVD_MAX_SWEEPS && n > 1; ++sweep) {
        bool rot = false;
        if (on) {
            if (nx0 >= 0) nx0 = jc_norm2(x0, ET);
            if (nx1 >= 0) nx1 = jc_norm2(x1, ET);
            if (ny0 >= 0) ny0 = jc_norm2(y0, ET);
            if (ny1 >= 0) ny1 = jc_norm2(y1, ET);
            rot |= jc_rotate2(x0, x1, y0, y1, nx0, nx1, ny0, ny1, ET, tol2);  // inside the blocks
        }
        const int rounds = 2 * NW - 1;
        for (int r = 0; r < rounds; ++r, ++round) {
            if (on) {
                rot |= jc_rotate2(x0, y0, x1, y1, nx0, ny0, nx1, ny1, ET, tol2);
                rot |= jc_rotate2(x0, y1, x1, y0, nx0, ny1, nx1, ny0, ET, tol2);
            }
            if (NW == 1) continue;
            const int par = round & 1;
            if (parities == 1 && round > 0) {
                report();
                cl.sync();  // the inboxes have been read
            }
            if (!live) continue;
            if (lane == 0) jc_mbar_expect(&mbar[par][wid], remote_bytes);
            if (gw == 0) put(1, 0, par, y0, y1, ny0, ny1);
            else put(-1, 1, par, y0, y1, ny0, ny1);
            if (gw == NW - 1) {
#pragma unroll
                for (int q = 0; q < E; ++q) {
                    y0[q] = x0[q];
                    y1[q] = x1[q];
                }
                ny0 = nx0;
                ny1 = nx1;
            } else if (gw > 0) {
                put(1, 0, par, x0, x1, nx0, nx1);
            }
            live = jc_mbar_wait(&mbar[par][wid], (round >> 1) & 1, polls, derr);
            if (!live) continue;
            if (from_left) get(slot(wid, 0, par), x0, x1, nx0, nx1);
            if (from_right) get(slot(wid, 1, par), y0, y1, ny0, ny1);
        }
        report();
        // flags: [sweep % 3] collects, [(sweep + 2) % 3] was read by all before the previous barrier
        if (rot && lane == 0) *cl.map_shared_rank(&flags[sweep % 3], 0) = 1;
        if (rank == 0 && tid == 0) flags[(sweep + 1) % 3] = 0;
        cl.sync();
        // the same values in every thread of the cluster
        const int f = *cl.map_shared_rank(&failed, 0), rotated = *cl.map_shared_rank(&flags[sweep % 3], 0);
        if (f) {
            __nanosleep(200000);  // messages that were given up may still be on their way
            cl.sync();
            return;
        }
        if (!rotated) break;
    }

    // singular values: every CTA gets all of them (slots 4 gw .. 4 gw + 3; padding columns -1)
    if (on) {
        const double s0 = nx0 < 0 ? -1.0 : sqrt(jc_norm2(x0, ET)), s1 = nx1 < 0 ? -1.0 : sqrt(jc_norm2(x1, ET));
        const double s2 = ny0 < 0 ? -1.0 : sqrt(jc_norm2(y0, ET)), s3 = ny1 < 0 ? -1.0 : sqrt(jc_norm2(y1, ET));
        if (lane < ncta) {
            double* p = cl.map_shared_rank(sig, lane) + 4 * gw;
            p[0] = s0;
            p[1] = s1;
            p[2] = s2;
            p[3] = s3;
        }
    }
    cl.sync();
    // descending rank, ties broken by position; a NaN anywhere makes every value NaN
    const int np = 4 * NW;
    bool nan = false;
    for (int j = 0; j < np; ++j) nan = nan || sig[j] != sig[j];
    const double unscale = nan ? nan_value() : 1.0 / scale_sh;
    for (int j = tid; j < np; j += blockDim.x) {
        const double sj = sig[j];
        int k = 0;
        for (int i = 0; i < np; ++i) k += ranks_before(sig[i], i, sj, j);
        rk[j] = sj < 0 ? -1 : k;
        if (rank == 0 && !(sj < 0)) jb.s[min(k, n - 1)] = sj * unscale;
    }
    __syncthreads();
    if (vectors) {
        double smax = 0;
        for (int j = 0; j < np; ++j) smax = fmax(smax, sig[j]);
        const double cut = smax * 1e-13 * fmax(1.0, (double)m) * unscale;
        auto emit = [&](const double(&v)[E], int j) {
            const int k = rk[j];
            if (k < 0) return;
            const double sj = sig[j];
            const bool good = keeps_column(sj * unscale, cut);
            const int kc = min(k, n - 1);
#pragma unroll
            for (int q = 0; q < E; ++q) {
                const int row = lane + 32 * q, low = row - 32 * ET;
                if (q < ET) {
                    const double e = good ? v[q] / sj : 0.0;
                    if (row < mt) {
                        if (pre) jb.Vt[(size_t)jb.perm[row] * jb.ldvt + kc] = e;
                        else jb.U[(size_t)kc * jb.ldu + row] = e;
                    }
                } else if (low < mb) {
                    if (pre) jb.U[(size_t)kc * jb.ldu + low] = v[q];
                    else jb.Vt[(size_t)low * jb.ldvt + kc] = v[q];
                }
            }
        };
        if (on) {
            emit(x0, 4 * gw);
            emit(x1, 4 * gw + 1);
            emit(y0, 4 * gw + 2);
            emit(y1, 4 * gw + 3);
        }
        __threadfence();
        cl.sync();
        if (rank == 0) {
            if (pre) complete_u(jb, jb.Vt, jb.ldvt, 1, n, cut, red, sig, at);
            else complete_u(jb, jb.U, 1, jb.ldu, m, cut, red, sig, at);
        }
    }
    if (rank == 0 && tid == 0 && jb.sweeps) *jb.sweeps = sweep;
    cl.sync();  // no CTA leaves while its shared memory may still be addressed
}

// perm: the columns of W (m x n) by descending norm, ties by index (a norm that is not a number counts as infinite).
// *range is raised for a matrix that the Jacobi kernel scales: its factorisation would not.
__global__ void __launch_bounds__(1024) svd_order_kernel(const double* __restrict__ W, int m, int n, int* __restrict__ perm,
                                                         int* range) {
    extern __shared__ double nrm2[];
    __shared__ double wmax[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double amax = 0.0;
    for (int c = wid; c < n; c += 32) {
        const double* w = W + (size_t)c * m;
        double s = 0, x = 0;
#pragma unroll 4
        for (int i = lane; i < m; i += 32) {
            s = fma(w[i], w[i], s);
            x = fmax(x, fabs(w[i]));
        }
        s = wsum(s);
        for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
        amax = fmax(amax, x);
        if (lane == 0) nrm2[c] = s >= 0 ? s : __longlong_as_double(0x7ff0000000000000LL);
    }
    if (lane == 0) wmax[wid] = amax;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 32; ++w) amax = fmax(amax, wmax[w]);
        if (jc_matrix_scale(amax) != 1.0) *range = 1;
    }
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const double sj = nrm2[j];
        int k = 0;
        for (int i = 0; i < n; ++i) {
            const double si = nrm2[i];
            k += (si > sj) || (si == sj && i < j);
        }
        perm[k] = j;
    }
}

// Cluster shapes for the largest n and row-slot count of a batch, best first;
// none: not served.  Four warps per CTA (one per scheduler) up to n = 128, eight
// above, so that eight CTAs hold n = 256; with 16 row slots eight warps'
// inboxes fit one parity only, and 16 CTAs of four warps are tried first
// (256 x 256 with vectors, graded over three decades: 3.5 against 5.8 ms, 5.2 against 8.9 without the factorisation).
struct JcShape {
    int ncta = 0, warps = 0;
};
std::vector<JcShape> jc_shapes(int n, int slots) {
    std::vector<JcShape> v;
    if (slots > JC_SLOTS_MAX || n > 512) return v;
    const int NW = std::max(1, (n + 3) / 4);
    if (NW > 32 && NW <= 64 && slots > 12) v.push_back({16, 4});
    JcShape s;
    s.warps = NW <= 32 ? 4 : 8;
    s.ncta = 1;
    while (s.ncta * s.warps < NW) s.ncta *= 2;
    v.push_back(s);
    return v;
}

template <int E>
int jc_launch(Ctx& c, const SvdJob* dev_jobs, const SvdJob& one, int njobs, JcShape sh, int nmax, bool vectors,
              bool* served) {
    *served = false;
    const size_t cap = 220 * 1024;
    const int np = 4 * sh.ncta * sh.warps;
    int parities = 2;
    size_t smem = jc_smem_bytes<E>(sh.warps, 2, std::max(np, nmax));
    if (smem > cap) {
        parities = 1;
        smem = jc_smem_bytes<E>(sh.warps, 1, std::max(np, nmax));
    }
    if (smem > cap) return TN_OK;
    auto kern = jacobi_cluster_kernel<E>;
    TN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    if (sh.ncta > 8) TN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(njobs * sh.ncta));
    cfg.blockDim = dim3((unsigned)(32 * sh.warps));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)sh.ncta;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (sh.ncta > 8) {
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) != cudaSuccess || nc < 1) {
            cudaGetLastError();
            return TN_OK;
        }
    }
    TN_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, dev_jobs, one, vectors ? 1 : 0, parities, std::max(np, nmax),
                                     c.wait_polls < 0 ? JC_WAIT_POLLS : c.wait_polls, c.derr.as<int>()));
    TN_LAUNCH_CHECK();
    *served = true;
    return TN_OK;
}

}  // namespace

int svd_batched(Ctx& c, const std::vector<SvdJob>& jobs, bool vectors) {
    if (jobs.empty()) return TN_OK;
    for (const auto& j : jobs) {
        if (j.m < j.n || j.n < 1) {
            set_error("svd: job needs m >= n >= 1 (got %d x %d)", j.m, j.n);
            return TN_BAD_SHAPE;
        }
        if ((size_t)j.n * 12 + 64 > 200 * 1024) {
            set_error("svd: n too large for the single-CTA Jacobi kernel (%d)", j.n);
            return TN_BAD_SHAPE;
        }
    }
    const SvdJob* dev = nullptr;  // a single job travels as a kernel argument
    if (jobs.size() > 1) {
        TN_CHECK(c.svdw.ensure(sizeof(SvdJob) * jobs.size()));
        TN_CUDA_CHECK(cudaMemcpyAsync(c.svdw.p, jobs.data(), sizeof(SvdJob) * jobs.size(), cudaMemcpyHostToDevice,
                                      c.stream));
        dev = c.svdw.as<SvdJob>();
    }
    int nmax = 1, slots = 1;
    for (const auto& j : jobs) {
        nmax = std::max(nmax, j.n);
        slots = std::max(slots, (j.m + 31) / 32 + (vectors ? (j.n + 31) / 32 : 0));
    }
    // Every job of the batch fits the cluster kernel (n <= 512 and at most 16
    // slots of 32 rows per column, rows of U and V together): there it is the
    // faster one at every size (25 x 25 0.22 against 0.44 ms, 150 x 128 1.87 against
    // 26.7, both without the factorisation below); otherwise one CTA per matrix with its columns in shared
    // memory or L2.
    TN_CHECK(ensure_device_error_word(c));
    bool served = false;
    const int nj = (int)jobs.size();
    const auto shapes = jc_shapes(nmax, slots);
    auto run = [&](const SvdJob& one) -> int {
        for (const JcShape& sh : shapes) {
            if (served) break;
            if (slots <= 2) TN_CHECK(jc_launch<2>(c, dev, one, nj, sh, nmax, vectors, &served));
            else if (slots <= 4) TN_CHECK(jc_launch<4>(c, dev, one, nj, sh, nmax, vectors, &served));
            else if (slots <= 6) TN_CHECK(jc_launch<6>(c, dev, one, nj, sh, nmax, vectors, &served));
            else if (slots <= 8) TN_CHECK(jc_launch<8>(c, dev, one, nj, sh, nmax, vectors, &served));
            else if (slots <= 12) TN_CHECK(jc_launch<12>(c, dev, one, nj, sh, nmax, vectors, &served));
            else TN_CHECK(jc_launch<16>(c, dev, one, nj, sh, nmax, vectors, &served));
        }
        return TN_OK;
    };
    // A single matrix of some size is factored first, its columns by descending norm: A P = Q R, and the rotations
    // that orthogonalise the columns of R^T (Drmac and Veselic, SIAM J. Matrix Anal. Appl. 29, 2008: R^T is closer to
    // diagonal than A) turn Q into U: R^T J = V' S gives A = (Q J) S (P V')^T.  The same kernel with R^T
    // above and Q's rows below, 9-11 sweeps instead of 14-19.  Factored and not (a call of tn_svd, graded over three
    // decades): 16 x 16 135 and 122 us, 20 x 20 159 and 146, 25 x 25 204 and 226, 64 x 64 479 and 605,
    // 150 x 128 1431 and 1881, 160 x 160 2154 and 3211; 150 x 128 26.7 ms with one CTA per matrix.
    const SvdJob& j0 = jobs[0];
    if (nj == 1 && j0.n >= SVD_PRE_MIN && !shapes.empty()) {
        const size_t nq = vectors ? (size_t)j0.m * j0.n : 0, nr = (size_t)j0.n * j0.n;
        TN_CHECK(c.svdpre.ensure(sizeof(double) * (nq + nr) + sizeof(int) * (size_t)j0.n));
        double* Q = c.svdpre.as<double>();
        double* X = Q + nq;
        int* perm = reinterpret_cast<int*>(X + nr);
        svd_order_kernel<<<1, 1024, sizeof(double) * j0.n, c.stream>>>(j0.W, j0.m, j0.n, perm,
                                                                                 c.derr.as<int>() + 1);
        TN_LAUNCH_CHECK();
        const int st = qr_cluster(c, j0.m, j0.n, j0.W, 1, j0.m, vectors ? Q : nullptr, 1, j0.m, X, j0.n, 1, perm);
        if (st != QR_UNAVAILABLE) {
            TN_CHECK(st);
            SvdJob p = j0;
            p.W = X;
            p.V = Q;
            p.perm = perm;
            TN_CHECK(run(p));
            if (served) {
                const int rc = qr_cluster_status(c);
                if (rc != QR_UNAVAILABLE) return rc;
                served = false;  // out of its range: the matrix itself, which only the QR has read
            }
        }
        TN_CUDA_CHECK(cudaMemsetAsync(c.derr.as<int>() + 1, 0, sizeof(int), c.stream));
    }
    if (!served) TN_CHECK(run(j0));
    if (!served) {
        if (!dev) {
            TN_CHECK(c.svdw.ensure(sizeof(SvdJob)));
            TN_CUDA_CHECK(cudaMemcpyAsync(c.svdw.p, jobs.data(), sizeof(SvdJob), cudaMemcpyHostToDevice, c.stream));
            dev = c.svdw.as<SvdJob>();
        }
        const size_t cap = 200 * 1024;
        TN_CUDA_CHECK(cudaFuncSetAttribute(jacobi_svd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
        jacobi_svd_kernel<<<(unsigned)jobs.size(), SVD_THREADS, cap, c.stream>>>(dev, vectors ? 1 : 0, cap);
        TN_LAUNCH_CHECK();
    }
    // the job array must stay valid until the kernel has read it
    if (served) return check_device_error_on_stream(c);
    TN_CUDA_CHECK(cudaStreamSynchronize(c.stream));
    return TN_OK;
}

}  // namespace tnb
