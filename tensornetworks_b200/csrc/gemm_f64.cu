// gemm_f64.cu -- FP64 batched GEMM with split-index addressing (tensor-core DMMA, SIMT for
// split indices).
//
// Used by the plain FP64 sweep for the three contraction stages of the
// effective-Hamiltonian matvec and of the environment updates
// (MPSSite::GetHeff / IterateLeft_F / IterateRightF in the reference,
// MPSSite_Contractions.C:155-400), and for small gauge products.
// Plain strided operands take the FP64 tensor-core (DMMA) kernel below;
// split-index operands the SIMT kernel: tile 64x64x16, 256 threads, 4x4
// outputs per thread, register-staged double buffering of the next k-tile.
#include "dgemm.cuh"
#include "pdl.cuh"
#include "tn_internal.h"

namespace tnb {

namespace {

constexpr int BM = 64, BN = 64, BK = 16, NT = 256;

template <bool A_MCONTIG, bool B_KCONTIG>
__global__ void __launch_bounds__(NT) gemm_f64_kernel(GemmArgs g) {
    if (g.skip && *g.skip) return;
    __shared__ double As[BK][BM + 1];
    __shared__ double Bs[BK][BN + 1];
    const int t = threadIdx.x;
    const int tx = t & 15, ty = t >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int b = blockIdx.z;
    const int b0 = b / g.nb1, b1 = b - (b / g.nb1) * g.nb1;
    const double* Ab = g.A.ptr + b0 * g.A.sb0 + b1 * g.A.sb1;
    const double* Bb = g.B.ptr + b0 * g.B.sb0 + b1 * g.B.sb1;

    // Per-slot fixed coordinates for the tile loads.
    int am[4], ak[4], bk[4], bn[4];
    long long aoff[4], boff[4];
    bool aok[4], bok[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        int e = t + NT * r;
        if (A_MCONTIG) { am[r] = e % BM; ak[r] = e / BM; }
        else           { ak[r] = e % BK; am[r] = e / BK; }
        if (B_KCONTIG) { bk[r] = e % BK; bn[r] = e / BK; }
        else           { bn[r] = e % BN; bk[r] = e / BN; }
        int gm = m0 + am[r], gn = n0 + bn[r];
        aok[r] = gm < g.M;
        bok[r] = gn < g.N;
        aoff[r] = aok[r] ? g.A.mn.at(gm) : 0;
        boff[r] = bok[r] ? g.B.mn.at(gn) : 0;
    }

    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;

    double ra[4], rb[4];
    auto load = [&](int k0) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            int gk = k0 + ak[r];
            ra[r] = (aok[r] && gk < g.K) ? __ldg(Ab + aoff[r] + g.A.k.at(gk)) : 0.0;
            int hk = k0 + bk[r];
            rb[r] = (bok[r] && hk < g.K) ? __ldg(Bb + boff[r] + g.B.k.at(hk)) : 0.0;
        }
    };
    auto store = [&]() {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            As[ak[r]][am[r]] = ra[r];
            Bs[bk[r]][bn[r]] = rb[r];
        }
    };

    load(0);
    for (int k0 = 0; k0 < g.K; k0 += BK) {
        store();
        __syncthreads();
        if (k0 + BK < g.K) load(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            double a[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) bv[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }

    double* Cb = g.C.ptr + b0 * g.C.sb0 + b1 * g.C.sb1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int gm = m0 + ty + 16 * i;
        if (gm >= g.M) continue;
        long long mo = g.C.m.at(gm);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int gn = n0 + tx + 16 * j;
            if (gn >= g.N) continue;
            double* c = Cb + mo + g.C.n.at(gn);
            double v = g.alpha * acc[i][j];
            if (g.beta != 0.0) v += g.beta * *c;
            *c = v;
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 tensor-core path: mma.sync m8n8k4 (DMMA), for operands whose index maps
// are plain strides over the ranges used (no split indices).  CTA tile
// BM x BN, four warps in a 2 x 2 grid, k-tiles of 16 in a ring of DG_STAGES
// shared-memory stages filled by asynchronous copies (one barrier per k-tile;
// the copies of the next two tiles are in flight behind the products).  An
// operand keeps its contiguous index contiguous in shared memory, [k][m] or
// [m][k], with rows of 4 mod 16 doubles: the fragment loads of a half warp
// then hit 16 distinct bank pairs in both forms, and copies are 16 bytes
// where base, strides and batch strides allow it (V = 2), 8 otherwise.
// Bound: the FP64 pipe (37 TFLOP/s); what keeps smaller products off it is
// the number of tiles per SM and the pipeline's fill.
constexpr int DG_STAGES = 3, DG_NT = 128;

struct LinGemm {
    int M, N, K, nb1;
    long long sAm, sAk, sBk, sBn, sCm, sCn;
    long long sA0, sA1, sB0, sB1, sC0, sC1;
    const double *A, *B;
    double* C;
    double alpha, beta;
    const int* skip;
};

template <int BM, int BN, bool A_MC, bool B_KC, int V>
constexpr int dg_smem_bytes() {
    return (int)sizeof(double) * DG_STAGES * (DgOperand<BM, A_MC, V, DG_NT>::STAGE + DgOperand<BN, !B_KC, V, DG_NT>::STAGE);
}

template <int BM, int BN, bool A_MC, bool B_KC, int V>
__global__ void __launch_bounds__(DG_NT) gemm_f64_dmma_kernel(LinGemm g) {
    constexpr int WM = BM / 2, WN = BN / 2, MI = WM / 8, NI = WN / 8;
    using OpA = DgOperand<BM, A_MC, V, DG_NT>;
    using OpB = DgOperand<BN, !B_KC, V, DG_NT>;
    extern __shared__ __align__(16) double dg_smem[];
    double* As = dg_smem;
    double* Bs = dg_smem + DG_STAGES * OpA::STAGE;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int gid = lane >> 2, tig = lane & 3;
    const int wm = (warp >> 1) * WM, wn = (warp & 1) * WN;
    const int mt = (g.M + BM - 1) / BM;  // tiles of one column of C in a row
    const int m0 = blockIdx.x % mt * BM, n0 = blockIdx.x / mt * BN;
    const int b = blockIdx.z;
    const int b0 = b / g.nb1, b1 = b - b0 * g.nb1;
    const double* Ab = g.A + b0 * g.sA0 + b1 * g.sA1;
    const double* Bb = g.B + b0 * g.sB0 + b1 * g.sB1;
    OpA oa;
    OpB ob;
    oa.init(t, Ab, g.sAm, g.sAk, m0, g.M);
    ob.init(t, Bb, g.sBn, g.sBk, n0, g.N);
    // nothing above reads memory: launch and prologue run beside the predecessor's tail
    pdl_wait();
    if (g.skip && *g.skip) return;
    double acc[MI][NI][2];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int ntile = (g.K + DG_BK - 1) / DG_BK;
#pragma unroll
    for (int s = 0; s < DG_STAGES - 1; ++s) {
        if (s < ntile) {
            oa.load(As + s * OpA::STAGE, Ab, g.K - s * DG_BK);
            ob.load(Bs + s * OpB::STAGE, Bb, g.K - s * DG_BK);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    int rd = 0, wr = DG_STAGES - 1;
    for (int kt = 0; kt < ntile; ++kt) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(DG_STAGES - 2) : "memory");
        __syncthreads();  // tile kt has arrived for all threads, and stage wr has been read by all
        if (kt + DG_STAGES - 1 < ntile) {
            const int kleft = g.K - (kt + DG_STAGES - 1) * DG_BK;
            oa.load(As + wr * OpA::STAGE, Ab, kleft);
            ob.load(Bs + wr * OpB::STAGE, Bb, kleft);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const double* a = As + rd * OpA::STAGE;
        const double* bb = Bs + rd * OpB::STAGE;
#pragma unroll
        for (int ks = 0; ks < DG_BK; ks += 4) {
            double af[MI], bf[NI];
#pragma unroll
            for (int i = 0; i < MI; ++i) af[i] = OpA::get(a, wm + i * 8 + gid, ks + tig);  // A(row gid, col tig)
#pragma unroll
            for (int j = 0; j < NI; ++j) bf[j] = OpB::get(bb, wn + j * 8 + gid, ks + tig);  // B(row tig, col gid)
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NI; ++j) dmma(acc[i][j], af[i], bf[j]);
        }
        rd = rd + 1 == DG_STAGES ? 0 : rd + 1;
        wr = wr + 1 == DG_STAGES ? 0 : wr + 1;
    }
    double* Cb = g.C + b0 * g.sC0 + b1 * g.sC1;
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int gm = m0 + wm + i * 8 + gid;
        if (gm >= g.M) continue;
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int gn = n0 + wn + j * 8 + tig * 2 + q;
                if (gn >= g.N) continue;
                double* c = Cb + gm * g.sCm + gn * g.sCn;
                double v = g.alpha * acc[i][j][q];
                if (g.beta != 0.0) v += g.beta * *c;
                *c = v;
            }
    }
}

template <int BM, int BN, bool A_MC, bool B_KC, int V>
int dg_launch(const LinGemm& l, int batches, cudaStream_t st) {
    constexpr int bytes = dg_smem_bytes<BM, BN, A_MC, B_KC, V>();
    auto kern = gemm_f64_dmma_kernel<BM, BN, A_MC, B_KC, V>;
    if (bytes > 48 * 1024) {
        static thread_local int dev_set = -1;
        int dev = 0;
        TN_CUDA_CHECK(cudaGetDevice(&dev));
        if (dev_set != dev) {
            TN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
            dev_set = dev;
        }
    }
    const long long tiles = (long long)((l.N + BN - 1) / BN) * ((l.M + BM - 1) / BM);
    if (tiles > 0x7fffffffLL) {
        set_error("gemm_f64: grid too large");
        return TN_BAD_SHAPE;
    }
    const dim3 grid((unsigned)tiles, 1, batches);
    return launch_pdl(kern, grid, DG_NT, bytes, st, l);
}

template <int BM, int BN>
int dg_dispatch(const LinGemm& l, int batches, bool amc, bool bkc, bool wide, cudaStream_t st) {
    if (wide) {
        if (amc && bkc) return dg_launch<BM, BN, true, true, 2>(l, batches, st);
        if (amc) return dg_launch<BM, BN, true, false, 2>(l, batches, st);
        if (bkc) return dg_launch<BM, BN, false, true, 2>(l, batches, st);
        return dg_launch<BM, BN, false, false, 2>(l, batches, st);
    }
    if (amc && bkc) return dg_launch<BM, BN, true, true, 1>(l, batches, st);
    if (amc) return dg_launch<BM, BN, true, false, 1>(l, batches, st);
    if (bkc) return dg_launch<BM, BN, false, true, 1>(l, batches, st);
    return dg_launch<BM, BN, false, false, 1>(l, batches, st);
}

// 16-byte copies: the contiguous index has stride 1, and the base and every
// other stride keep 16-byte alignment.
inline bool wide_operand(const double* p, long long contiguous, long long other, long long s0, long long s1) {
    return contiguous == 1 && (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ((other | s0 | s1) & 1) == 0;
}

// An index map that is a plain stride over [0, n).
inline bool plain(const IdxMap& m, int n) { return m.div >= n; }

}  // namespace

int gemm_f64(const GemmArgs& g, cudaStream_t st) {
    if (g.M <= 0 || g.N <= 0) return TN_OK;
    if (g.K <= 0) {
        // C = beta*C: express as a K=1 product with a zero operand is wasteful;
        // callers never ask for it.
        set_error("gemm_f64: K must be positive");
        return TN_BAD_ARG;
    }
    dim3 grid((g.N + BN - 1) / BN, (g.M + BM - 1) / BM, g.nb0 * g.nb1);
    if (grid.y > 65535 || grid.z > 65535) {
        set_error("gemm_f64: grid too large");
        return TN_BAD_SHAPE;
    }
    bool amc = (g.A.mn.s == 1);
    bool bkc = (g.B.k.s == 1);
    if (plain(g.A.mn, g.M) && plain(g.A.k, g.K) && plain(g.B.k, g.K) && plain(g.B.mn, g.N) && plain(g.C.m, g.M) &&
        plain(g.C.n, g.N)) {
        LinGemm l;
        l.M = g.M; l.N = g.N; l.K = g.K; l.nb1 = g.nb1;
        l.sAm = g.A.mn.s; l.sAk = g.A.k.s; l.sBk = g.B.k.s; l.sBn = g.B.mn.s; l.sCm = g.C.m.s; l.sCn = g.C.n.s;
        l.sA0 = g.A.sb0; l.sA1 = g.A.sb1; l.sB0 = g.B.sb0; l.sB1 = g.B.sb1; l.sC0 = g.C.sb0; l.sC1 = g.C.sb1;
        l.A = g.A.ptr; l.B = g.B.ptr; l.C = g.C.ptr; l.alpha = g.alpha; l.beta = g.beta; l.skip = g.skip;
        const bool wide = wide_operand(l.A, amc ? l.sAm : l.sAk, amc ? l.sAk : l.sAm, l.sA0, l.sA1) &&
                          wide_operand(l.B, bkc ? l.sBk : l.sBn, bkc ? l.sBn : l.sBk, l.sB0, l.sB1);
        static int sms = 0;
        if (sms == 0) {
            int dev = 0;
            cudaGetDevice(&dev);
            if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
        }
        // 32 x 32 tiles until 32 x 64 ones give every SM eight: below that the
        // finer split wins by what the last round of tiles leaves idle (10 x 256^3:
        // 18.5 us against 20.5 with 32 x 64 and 24.6 with 64 x 64; 10 x 250 x 203 x 250:
        // 16.4, 22.6, 24.6; 15 x 90^3: 6.2, 8.3, 10.3), above it the wider one by its
        // operand reuse (15 x 512^3: 133 us against 137).
        const int nb = g.nb0 * g.nb1;
        const long long tiles = (long long)((g.N + 63) / 64) * ((g.M + 31) / 32) * nb;
        if (tiles >= 8LL * sms) return dg_dispatch<32, 64>(l, nb, amc, bkc, wide, st);
        return dg_dispatch<32, 32>(l, nb, amc, bkc, wide, st);
    }
    if (amc && bkc) gemm_f64_kernel<true, true><<<grid, NT, 0, st>>>(g);
    else if (amc && !bkc) gemm_f64_kernel<true, false><<<grid, NT, 0, st>>>(g);
    else if (!amc && bkc) gemm_f64_kernel<false, true><<<grid, NT, 0, st>>>(g);
    else gemm_f64_kernel<false, false><<<grid, NT, 0, st>>>(g);
    TN_LAUNCH_CHECK();
    return TN_OK;
}

}  // namespace tnb
