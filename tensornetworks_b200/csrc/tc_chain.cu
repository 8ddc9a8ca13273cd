// tc_chain.cu -- segmented split-K BF16xN GEMM on the 5th-generation tensor
// cores, the building block of the fused split-precision Heff matvec.
//
//   C[ob](m, n) = sum_{s in segments(ob)} sum_k A[s.a](m, k) B[s.b](n, k)
//
// An output batch is a list of K segments (operand batch pairs); all chunks of
// all segments of one 128 x 64 output tile are dealt out to `splitk` CTAs that
// form one thread-block cluster.  Each CTA runs the usual tcgen05 pipeline on
// its chunk range (warp 0: TMA loads into a 128-byte-swizzled ring; warp 1:
// one elected thread issues the BF16 piece products into a TMEM accumulator;
// warps 2-5: tcgen05.ld of the accumulator).  With splitk > 1 CTA r sums rows
// [r*128/splitk, (r+1)*128/splitk) of the tile: warps 2-5 send every row of their CTA's
// partial to the CTA that sums it (st.async, counted by an mbarrier there) and each
// CTA adds the partials in rank order (deterministic).  The results are written either as
// BF16 pieces (row-major: the A operand of the next GEMM) or as FP64
// (column-major: the site-tensor layout); with splitk = 1 straight from the
// accumulator.  No partial ever goes to HBM.
//
// What bounds it at the sizes of a sweep (2 to 6 chunks per CTA) is a chain of latencies:
// first TMA ~0.9 us, ~0.6 us per chunk (48 KB), the accumulator 0.5, then the exchange.  Staging the
// partial, a cluster barrier, reading the peers' staging and a second barrier took 4.4 of
// 7.6 us; with the partials sent the d = 2, D = 256 matvec (two of these kernels and the splitting of x)
// went from 26.7 to 22.8 us.
//
// Every mbarrier wait is bounded; on expiry the CTA records an error code, still
// sends its partial and takes the cluster barriers, so no CTA of a cluster waits for a peer
// that has left.
#include <cuda_bf16.h>

#include "pdl.cuh"
#include "tc_chain.h"
#include "tc_ptx.cuh"

namespace tnb {

namespace {

using namespace tcp;

constexpr int CBN = 64;  // output tile columns

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
    uint32_t out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
    return out;
}

__device__ __forceinline__ void st_async_v4(uint32_t addr, float a, float b, float c, float d, uint32_t mbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "f"(a), "f"(b), "f"(c), "f"(d), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <int NS>
struct ChainSmem {
    static constexpr int A_BYTES = BM * BK * 2;   // 16 KB per piece
    static constexpr int B_BYTES = CBN * BK * 2;  // 8 KB per piece
    static constexpr int STAGE_BYTES = NS * (A_BYTES + B_BYTES);
    static constexpr int NSTAGE = (4 * STAGE_BYTES + 1024 <= 220 * 1024) ? 4 : ((3 * STAGE_BYTES + 1024 <= 220 * 1024) ? 3 : 2);
    static constexpr int RING = NSTAGE * STAGE_BYTES;
    // landing place of the partials: behind the ring where both fit, else over it (once no CTA's MMA reads it)
    static constexpr int LAND_BYTES = BM * CBN * 4;
    static constexpr bool OWN_LAND = RING + LAND_BYTES + 2048 <= 227 * 1024;
    static constexpr int LAND = OWN_LAND ? RING : 0;
    static constexpr int TOTAL = (OWN_LAND ? RING + LAND_BYTES : RING) + 1024;
};

// Four columns of a row as BF16 pieces (`left` of them exist): one 8-byte store per piece (row pitch and first
// column are multiples of 4).
template <int NS>
__device__ __forceinline__ void store_pieces(uint16_t* dst, long long piece, const float* v, int left) {
    float rem[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
    for (int pc = 0; pc < NS; ++pc) {
        uint16_t h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat16 b = __float2bfloat16_rn(rem[i]);
            h[i] = __bfloat16_as_ushort(b);
            rem[i] -= __bfloat162float(b);
        }
        uint16_t* d = dst + (long long)pc * piece;
        if (left >= 4) {
            *reinterpret_cast<uint2*>(d) =
                make_uint2((uint32_t)h[0] | ((uint32_t)h[1] << 16), (uint32_t)h[2] | ((uint32_t)h[3] << 16));
        } else {
#pragma unroll
            for (int i = 0; i < 3; ++i)
                if (i < left) d[i] = h[i];
        }
    }
}

template <int NS, int OUT, int SK>
__global__ void __launch_bounds__(THREADS, 1)
    tc_chain_kernel(const __grid_constant__ TcMaps maps, TcChainArgs p) {
    using SL = ChainSmem<NS>;
    constexpr int STAGES = SL::NSTAGE;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[4], empty_bar[4], accum_bar, land_bar;
    __shared__ uint32_t tmem_base_sh;
    __shared__ int s_fail;

    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * CBN;
    const int split = SK > 1 ? (int)cluster_ctarank() : 0;
    const int ob = blockIdx.z / SK;
    const int nkseg = (p.K + BK - 1) / BK;
    const int sbeg = p.seg_start[ob], send = p.seg_start[ob + 1];
    const int nchunk = (send - sbeg) * nkseg;
    const int q0 = (int)((long long)split * nchunk / SK);
    const int q1 = (int)((long long)(split + 1) * nchunk / SK);
    const bool has_work = q1 > q0;

    if (threadIdx.x == 32) {
        // descriptor prefetch overlaps the predecessor's tail
#pragma unroll
        for (int pc = 0; pc < NS; ++pc) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.a[pc])) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.b[pc])) : "memory");
        }
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&accum_bar, 1);
        mbar_init(&land_bar, 1);
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (SK > 1) mbar_expect_tx(&land_bar, SL::LAND_BYTES);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                     "r"((uint32_t)CBN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base_sh;
    if (SK > 1) cluster_arrive();  // land_bar is ready for the peers' messages
    TcSeg sg = {};                 // the segment tables are the plan's, not the predecessor's
    if (threadIdx.x == 0 && has_work) sg = p.segs[sbeg + q0 / nkseg];
    // the prologue above touched nothing the predecessor writes
    pdl_launch_dependents();
    pdl_wait();
    if (SK > 1) cluster_wait();
    // the flag is read by every CTA of a cluster alike, so a skipped launch leaves no peer waiting
    if (p.skip && *p.skip) {
        if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)CBN));
        return;
    }

    if (warp == 0) {
        if (lane == 0 && has_work) {
            for (int q = q0; q < q1; ++q) {
                const int it = q - q0;
                const int s = it % STAGES;
                const uint32_t ph = (it / STAGES) & 1;
                if (!mbar_wait(&empty_bar[s], ph ^ 1)) { s_fail = 1; break; }
                const int kc = q % nkseg;
                if (q > q0 && kc == 0) sg = p.segs[sbeg + q / nkseg];
                uint8_t* st = smem + s * SL::STAGE_BYTES;
                mbar_expect_tx(&full_bar[s], SL::STAGE_BYTES);
#pragma unroll
                for (int pc = 0; pc < NS; ++pc) {
                    tma_load_3d(st + pc * SL::A_BYTES, &maps.a[pc], &full_bar[s], kc * BK, m0, sg.a_batch);
                    tma_load_3d(st + NS * SL::A_BYTES + pc * SL::B_BYTES, &maps.b[pc], &full_bar[s], kc * BK, n0,
                                sg.b_batch);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && has_work) {
            constexpr uint32_t idesc = idesc_bf16(BM, CBN);
            for (int q = q0; q < q1; ++q) {
                const int it = q - q0;
                const int s = it % STAGES;
                const uint32_t ph = (it / STAGES) & 1;
                if (!mbar_wait(&full_bar[s], ph)) { s_fail = 1; break; }
                fence_after();
                const uint32_t st = smem_u32(smem + s * SL::STAGE_BYTES);
                const uint32_t a0 = st, b0 = st + NS * SL::A_BYTES;
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk) {
                    const uint32_t off = kk * 32;
                    mma_bf16(tmem, sdesc_sw128(a0 + off), sdesc_sw128(b0 + off), idesc, (it > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
                    for (int t = 1; t < NS; ++t)
#pragma unroll
                        for (int i = 0; i <= t; ++i)
                            mma_bf16(tmem, sdesc_sw128(a0 + i * SL::A_BYTES + off),
                                     sdesc_sw128(b0 + (t - i) * SL::B_BYTES + off), idesc, 1u);
                }
                mma_commit(&empty_bar[s]);
            }
            mma_commit(&accum_bar);
        }
    } else {
        // warps 2..5: TMEM lane quarter (warp % 4) = tile rows 32 q .. 32 q + 31
        const int qd = warp & 3;
        const int r = qd * 32 + lane;
        bool ok = true;
        if (has_work) ok = __all_sync(0xffffffffu, mbar_wait(&accum_bar, 0) ? 1 : 0) != 0;
        fence_after();
        if (!ok) s_fail = 1;
        if (SK > 1 && !SL::OWN_LAND) {
            cluster_arrive();  // this CTA's MMA has read the ring (warps 0 and 1 below)
            cluster_wait();
        }
        constexpr int RB = BM / SK;
        const uint32_t tbase = tmem + ((uint32_t)(qd * 32) << 16);
        const int row = m0 + r;
        uint32_t dst = 0, bar = 0;
        if (SK > 1) {
            dst = mapa_shared(smem_u32(smem + SL::LAND), r / RB) + (split * RB + r % RB) * (CBN * 4);
            bar = mapa_shared(smem_u32(&land_bar), r / RB);
        }
#pragma unroll 1
        for (int c0 = 0; c0 < CBN; c0 += 16) {
            float v[16];
            if (has_work && ok)
                tmem_ld16(tbase + (uint32_t)c0, v);
            else
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = 0.f;
            if (SK > 1) {  // granules of 16 bytes, swizzled by the row so that neither side has bank conflicts
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    st_async_v4(dst + (((c0 + i) / 4) ^ (r % RB & 15)) * 16, v[i], v[i + 1], v[i + 2], v[i + 3], bar);
            } else if (row < p.M) {
                if (OUT == TCC_OUT_F64_COLMAJOR) {
                    double* d64 = p.c64 + (long long)ob * p.c64_batch + (long long)(n0 + c0) * p.ldc64 + row;
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (n0 + c0 + i < p.N) d64[(long long)i * p.ldc64] = (double)v[i];
                } else {
                    uint16_t* d16 = p.c16 + (long long)ob * p.c16_batch + (long long)row * p.ldc16 + n0 + c0;
#pragma unroll
                    for (int i = 0; i < 16; i += 4) store_pieces<NS>(d16 + i, p.c16_piece, v + i, p.N - (n0 + c0 + i));
                }
            }
        }
    }
    if (SK > 1 && !SL::OWN_LAND && warp < 2) {
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)CBN));
    }
    if (SK > 1) {
        cluster_arrive();  // this CTA's messages are on their way
        if (!mbar_wait(&land_bar, 0)) s_fail = 2;
        // this CTA's rows: work item = one row and four consecutive columns
        constexpr int RB = BM / SK, CG = CBN / 4;
        const uint8_t* land = smem + SL::LAND;
#pragma unroll 1
        for (int e = threadIdx.x; e < RB * CG; e += THREADS) {
            // FP64: consecutive threads consecutive rows (coalesced column writes); BF16: column groups of a row
            const int lr = OUT == TCC_OUT_F64_COLMAJOR ? e % RB : e / CG, cg = OUT == TCC_OUT_F64_COLMAJOR ? e / RB : e % CG;
            float4 part[SK];
#pragma unroll
            for (int pr = 0; pr < SK; ++pr)
                part[pr] = *reinterpret_cast<const float4*>(land + (pr * RB + lr) * (CBN * 4) + (cg ^ (lr & 15)) * 16);
            const int row = m0 + split * RB + lr, col0 = n0 + 4 * cg;
            if (row >= p.M) continue;
            if (OUT == TCC_OUT_F64_COLMAJOR) {
                double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int pr = 0; pr < SK; ++pr) {
                    acc[0] += (double)part[pr].x;
                    acc[1] += (double)part[pr].y;
                    acc[2] += (double)part[pr].z;
                    acc[3] += (double)part[pr].w;
                }
                double* dst = p.c64 + (long long)ob * p.c64_batch + (long long)col0 * p.ldc64 + row;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (col0 + i < p.N) dst[(long long)i * p.ldc64] = acc[i];
            } else {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int pr = 0; pr < SK; ++pr) {
                    acc[0] += part[pr].x;
                    acc[1] += part[pr].y;
                    acc[2] += part[pr].z;
                    acc[3] += part[pr].w;
                }
                store_pieces<NS>(p.c16 + (long long)ob * p.c16_batch + (long long)row * p.ldc16 + col0, p.c16_piece, acc,
                                 p.N - col0);
            }
        }
        if (s_fail == 2) __nanosleep(200000);  // messages that were given up may still be on their way
        __syncwarp();
        cluster_wait();                        // no CTA leaves before its peers have sent
    }
    if (threadIdx.x == 0 && s_fail && p.err) atomicExch(p.err, 1);
}

template <int NS, int OUT, int SK>
int launch_chain(const TcChainPlan& pl, cudaStream_t st) {
    const TcChainArgs& p = pl.args;
    const int smem = ChainSmem<NS>::TOTAL;
    auto kern = tc_chain_kernel<NS, OUT, SK>;
    TN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + CBN - 1) / CBN, (p.M + BM - 1) / BM, p.nbatch * SK);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int na = 0;
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
    if (SK > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = 1;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = SK;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    TN_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, pl.maps, p));
    count_launch();
    return TN_OK;
}

template <int NS, int OUT>
int launch_chain(const TcChainPlan& pl, cudaStream_t st) {
    switch (pl.args.splitk) {
        case 1: return launch_chain<NS, OUT, 1>(pl, st);
        case 2: return launch_chain<NS, OUT, 2>(pl, st);
        case 4: return launch_chain<NS, OUT, 4>(pl, st);
        default: return launch_chain<NS, OUT, 8>(pl, st);
    }
}

}  // namespace

int tc_chain_splitk(int tiles, int chunks, int sm_count) {
    int sk = 1;
    while (sk < 8 && sk * 2 <= chunks && (long long)tiles * sk * 2 <= sm_count) sk *= 2;
    return sk;
}

int tc_chain_plan(const TcChainArgs& p, TcChainPlan* plan) {
    if (p.K % 8 != 0 || p.lda % 8 != 0 || p.ldb % 8 != 0) {
        set_error("tc_chain: K and operand pitches must be multiples of 8 (K=%d)", p.K);
        return TN_BAD_SHAPE;
    }
    if (p.nsplit != 2 && p.nsplit != 3) {
        set_error("tc_chain: nsplit must be 2 or 3");
        return TN_BAD_ARG;
    }
    if (p.splitk != 1 && p.splitk != 2 && p.splitk != 4 && p.splitk != 8) {
        set_error("tc_chain: splitk must be 1, 2, 4 or 8");
        return TN_BAD_ARG;
    }
    if (!p.seg_start || !p.segs || p.nbatch < 1) {
        set_error("tc_chain: no segment table");
        return TN_BAD_ARG;
    }
    if (p.out_mode == TCC_OUT_BF16_ROWMAJOR ? !p.c16 : !p.c64) {
        set_error("tc_chain: no output buffer");
        return TN_BAD_ARG;
    }
    plan->args = p;
    for (int q = 0; q < p.nsplit; ++q) {
        TN_CHECK(tc_make_map(&plan->maps.a[q], p.a[q], p.K, p.M, p.a_nbatch, p.lda, p.a_batch, BM));
        TN_CHECK(tc_make_map(&plan->maps.b[q], p.b[q], p.K, p.N, p.b_nbatch, p.ldb, p.b_batch, CBN));
    }
    return TN_OK;
}

int tc_chain_run(const TcChainPlan& pl, cudaStream_t st) {
    const TcChainArgs& p = pl.args;
    if (p.M <= 0 || p.N <= 0 || p.K <= 0 || p.nbatch <= 0) return TN_OK;
    if (p.out_mode == TCC_OUT_BF16_ROWMAJOR)
        return p.nsplit == 3 ? launch_chain<3, TCC_OUT_BF16_ROWMAJOR>(pl, st) : launch_chain<2, TCC_OUT_BF16_ROWMAJOR>(pl, st);
    return p.nsplit == 3 ? launch_chain<3, TCC_OUT_F64_COLMAJOR>(pl, st) : launch_chain<2, TCC_OUT_F64_COLMAJOR>(pl, st);
}

unsigned long long tc_chain_hash(const TcChainPlan& pl, unsigned long long h) {
    const TcChainArgs& p = pl.args;
    for (int q = 0; q < p.nsplit; ++q) {
        h = hash_val(h, pl.maps.a[q]);
        h = hash_val(h, pl.maps.b[q]);
    }
    for (long long v : {(long long)p.M, (long long)p.N, (long long)p.K, (long long)p.nbatch, (long long)p.splitk,
                        (long long)p.nsplit, p.lda, p.a_batch, p.ldb, p.b_batch, (long long)p.a_nbatch,
                        (long long)p.b_nbatch, (long long)p.out_mode, p.c16_piece, p.ldc16, p.c16_batch, p.ldc64,
                        p.c64_batch})
        h = hash_val(h, v);
    for (const void* v : {(const void*)p.seg_start, (const void*)p.segs, (const void*)p.c16, (const void*)p.err})
        h = hash_val(h, v);
    return h;
}

}  // namespace tnb
