// dgemm.cuh -- device pieces of the FP64 tensor-core products: the DMMA, the
// asynchronous copies and an operand's staging in shared memory.
#pragma once
#include <cuda_runtime.h>

namespace tnb {
namespace {

constexpr int DG_BK = 16;  // k-tile

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// V doubles to shared memory, the first `valid` of them read, zeros for the rest
template <int V>
__device__ __forceinline__ void dg_copy(double* dst, const double* src, int valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (V == 2)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(8 * valid) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(8 * valid) : "memory");
}

// One operand's share of a pipeline run by NT threads.  X x DG_BK elements per
// stage, x the row index of A or the column index of B; XC: x is the contiguous one.
template <int X, bool XC, int V, int NT>
struct DgOperand {
    static constexpr int LD = XC ? X + 4 : DG_BK + 4;
    static constexpr int STAGE = XC ? DG_BK * LD : X * LD;
    static constexpr int N = X * DG_BK / V / NT;  // copies per thread
    const double* src[N];
    int xleft[N];  // valid elements along x at the copy's place
    int dst[N], kk[N];
    long long step;
    __device__ __forceinline__ void init(int tid, const double* base, long long sx, long long sk, int x0, int nx) {
        step = DG_BK * sk;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int e = tid + NT * i;
            int x, k;
            if (XC) {
                x = e % (X / V) * V;
                k = e / (X / V);
                dst[i] = k * LD + x;
            } else {
                k = e % (DG_BK / V) * V;
                x = e / (DG_BK / V);
                dst[i] = x * LD + k;
            }
            xleft[i] = nx - x0 - x;
            kk[i] = k;
            src[i] = base + (xleft[i] > 0 ? (long long)(x0 + x) * sx : 0) + (long long)k * sk;
        }
    }
    // the stage of k-tile k0 (kleft = K - k0), then on to the next
    __device__ __forceinline__ void load(double* stage, const double* safe, int kleft) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int along = XC ? xleft[i] : kleft - kk[i];
            const bool in = xleft[i] > 0 && kk[i] < kleft;
            const int valid = in ? (along < V ? along : V) : 0;
            dg_copy<V>(stage + dst[i], valid > 0 ? src[i] : safe, valid);
            src[i] += step;
        }
    }
    __device__ static __forceinline__ double get(const double* stage, int x, int k) {
        return XC ? stage[k * LD + x] : stage[x * LD + k];
    }
};

}  // namespace
}  // namespace tnb
