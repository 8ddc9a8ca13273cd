// mlp.cu -- hand-written inference, gradient and Adam kernels of the learned
// Davidson correction (no reference counterpart).  The network maps the
// features of one element (f0 = (diag - theta)/sigma, f1 = r/rms(r),
// f2 = u sqrt(N), f3 = bond position) to the error of the diagonal correction
// in units of rms(r)/sigma; it is trained by mean squared error on pairs the
// plain FP64 Davidson solver records in its own sweeps (target: the exact
// correction x/(u.x) - u towards the converged eigenvector x, minus the
// diagonal correction r/(theta - diag)).
//
// Inference reads BF16 weights, with the hidden layer on the tensor cores
// (mlp_tiles); training keeps an FP32 master copy: a block runs forward and
// backward for chunks of pairs as register-tiled FP32 products, writes one
// partial gradient, and the Adam kernel sums the partials in a fixed order
// (deterministic).
#include "mlp.h"

#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

namespace tnb {

namespace {

__global__ void mlp_forward_kernel(const __nv_bfloat16* __restrict__ w16, const float* __restrict__ F, long long n,
                                   float* __restrict__ Y) {
    __shared__ MlpInferSmem s;
    mlp_stage(w16, s);
    __syncthreads();
    mlp_tiles(
        s, n,
        [&](long long e, float(&f)[MLP_IN]) {
#pragma unroll
            for (int q = 0; q < MLP_IN; ++q) f[q] = e < n ? F[e * MLP_IN + q] : 0.f;
        },
        [&](long long e, float y) { Y[e] = y; });
}

// Gradient of L = inv_n * sum (y - t)^2 over pairs [first, first + count) of
// the (optionally permuted) set; one partial gradient per block.
//
// A block of 256 threads takes chunks of PAIRS pairs; the four 64-wide
// products of a chunk -- H1 W2, D2 W2^T and H1^T D2, with H1 itself -- are
// register-tiled FP32 products on operands in shared memory.  Thread (ty, tx)
// owns PAIRS / 16 pairs x 4 hidden units in the first two (the pairs' outputs
// are summed over the 16 lanes tx) and the 4 x 4 entries (ty, tx) of dW2 in the
// third, which stay in registers over all chunks.  H1 and D2 are kept by hidden
// unit with the pairs contiguous and four words of padding, so every access is
// a conflict-free 16-byte one.
// Bound: FP32 issue (24.6 kflop a pair: 43 us for 131 072 pairs at the
// peak).  One thread per pair with its activations in shared memory at a
// stride of 64 words made every access a 32-way bank conflict.
constexpr int GR_THREADS = 256;

template <int PAIRS>
struct GradSmem {
    static constexpr int LD = PAIRS + 4;
    // w2 and w2t also hold, at the end, the 16 thread rows' sums of the vectors' gradients
    float w2[MLP_H][MLP_H];        // [j][k]
    float w2t[MLP_H][MLP_H + 4];   // [k][j]
    float h1[MLP_H][LD];           // [j][pair]
    float d2[MLP_H][LD];           // [k][pair]
    float f[MLP_IN][PAIRS], tgt[PAIRS];
    float w1[MLP_IN][MLP_H], b1[MLP_H], b2[MLP_H], w3[MLP_H], b3;
    double loss[GR_THREADS / 32];
    float db3[16];
};

template <int PAIRS>
__global__ void __launch_bounds__(GR_THREADS) mlp_grad_kernel(const float* __restrict__ w32,
                                                              const float* __restrict__ F, const float* __restrict__ T,
                                                              const int* __restrict__ perm, long long first,
                                                              long long count, double inv_n, float* __restrict__ part,
                                                              double* __restrict__ loss_part) {
    constexpr int PT = PAIRS / 16;  // pairs of a thread
    extern __shared__ __align__(16) unsigned char grad_dyn[];
    GradSmem<PAIRS>& s = *reinterpret_cast<GradSmem<PAIRS>*>(grad_dyn);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    for (int e = tid; e < MLP_H * MLP_H; e += GR_THREADS) {
        const float v = w32[MLP_W2 + e];
        s.w2[e / MLP_H][e % MLP_H] = v;
        s.w2t[e % MLP_H][e / MLP_H] = v;
    }
    for (int e = tid; e < MLP_IN * MLP_H; e += GR_THREADS) s.w1[e / MLP_H][e % MLP_H] = w32[MLP_W1 + e];
    if (tid < MLP_H) {
        s.b1[tid] = w32[MLP_B1 + tid];
        s.b2[tid] = w32[MLP_B2 + tid];
        s.w3[tid] = w32[MLP_W3 + tid];
    }
    if (tid == 0) s.b3 = w32[MLP_B3];
    float gW2[4][4], gW1[MLP_IN][4], gB1[4], gB2[4], gW3[4], gB3 = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        gB1[c] = gB2[c] = gW3[c] = 0.f;
#pragma unroll
        for (int r = 0; r < 4; ++r) gW2[r][c] = gW1[r][c] = 0.f;
    }
    double lacc = 0;
    const long long nchunks = (count + PAIRS - 1) / PAIRS;
    for (long long ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        __syncthreads();  // the previous chunk's operands have been read
        for (int e = tid; e < PAIRS; e += GR_THREADS) {
            const long long idx = ch * PAIRS + e;
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            float t = 0.f;
            if (idx < count) {
                const long long q = perm ? (long long)perm[first + idx] : first + idx;
                f = make_float4(F[4 * q], F[4 * q + 1], F[4 * q + 2], F[4 * q + 3]);
                t = T[q];
            }
            s.f[0][e] = f.x;
            s.f[1][e] = f.y;
            s.f[2][e] = f.z;
            s.f[3][e] = f.w;
            s.tgt[e] = t;
        }
        __syncthreads();
        for (int e = tid; e < MLP_H * PAIRS; e += GR_THREADS) {  // a warp: one hidden unit, 32 pairs
            const int j = e / PAIRS, q = e % PAIRS;
            float a = s.b1[j];
#pragma unroll
            for (int i = 0; i < MLP_IN; ++i) a = fmaf(s.f[i][q], s.w1[i][j], a);
            s.h1[j][q] = tanhf(a);
        }
        __syncthreads();
        float acc[PT][4];
        // the thread's PT x 4 tile of sum_j a[j][pairs] b[j][units]
        auto product = [&](const float(*a)[GradSmem<PAIRS>::LD], const float* b, int ldb) {
#pragma unroll
            for (int p = 0; p < PT; ++p)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[p][c] = 0.f;
#pragma unroll 4
            for (int j = 0; j < MLP_H; ++j) {
                float av[PT];
                if constexpr (PT % 4 == 0) {
#pragma unroll
                    for (int p = 0; p < PT; p += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(&a[j][PT * ty + p]);
                        av[p] = v.x; av[p + 1] = v.y; av[p + 2] = v.z; av[p + 3] = v.w;
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < PT; p += 2) {
                        const float2 v = *reinterpret_cast<const float2*>(&a[j][PT * ty + p]);
                        av[p] = v.x; av[p + 1] = v.y;
                    }
                }
                const float4 bv = *reinterpret_cast<const float4*>(b + j * ldb + 4 * tx);
#pragma unroll
                for (int p = 0; p < PT; ++p) {
                    acc[p][0] = fmaf(av[p], bv.x, acc[p][0]);
                    acc[p][1] = fmaf(av[p], bv.y, acc[p][1]);
                    acc[p][2] = fmaf(av[p], bv.z, acc[p][2]);
                    acc[p][3] = fmaf(av[p], bv.w, acc[p][3]);
                }
            }
        };
        product(s.h1, &s.w2[0][0], MLP_H);
        float dy[PT];
#pragma unroll
        for (int p = 0; p < PT; ++p) {
            float y = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                acc[p][c] = tanhf(acc[p][c] + s.b2[4 * tx + c]);
                y = fmaf(acc[p][c], s.w3[4 * tx + c], y);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
            const int q = PT * ty + p;
            const float err = ch * PAIRS + q < count ? (y + s.b3) - s.tgt[q] : 0.f;
            dy[p] = (float)(2.0 * inv_n) * err;
            if (tx == 0) {
                lacc += (double)err * err;
                gB3 += dy[p];
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float d[PT];
#pragma unroll
            for (int p = 0; p < PT; ++p) {
                const float h = acc[p][c];
                d[p] = dy[p] * s.w3[4 * tx + c] * (1.f - h * h);
                gW3[c] = fmaf(h, dy[p], gW3[c]);
                gB2[c] += d[p];
                s.d2[4 * tx + c][PT * ty + p] = d[p];
            }
        }
        __syncthreads();
        product(s.d2, &s.w2t[0][0], MLP_H + 4);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int p = 0; p < PT; ++p) {
                const int q = PT * ty + p;
                const float h = s.h1[4 * tx + c][q];
                const float d = acc[p][c] * (1.f - h * h);
                gB1[c] += d;
#pragma unroll
                for (int i = 0; i < MLP_IN; ++i) gW1[i][c] = fmaf(s.f[i][q], d, gW1[i][c]);
            }
        // dW2[j][k] over the chunk's pairs, four at a time: rows j = ty + 16 r, columns k = tx + 16 c
        // (neighbouring rows are 4 words apart modulo the banks, so the 16-byte reads of a phase do not collide)
        float w[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) w[r][c] = 0.f;
#pragma unroll 2
        for (int q = 0; q < PAIRS; q += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float4*>(&s.h1[ty + 16 * r][q]);
#pragma unroll
            for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(&s.d2[tx + 16 * c][q]);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    w[r][c] = fmaf(a[r].x, b[c].x, w[r][c]);
                    w[r][c] = fmaf(a[r].y, b[c].y, w[r][c]);
                    w[r][c] = fmaf(a[r].z, b[c].z, w[r][c]);
                    w[r][c] = fmaf(a[r].w, b[c].w, w[r][c]);
                }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) gW2[r][c] += w[r][c];
    }
    float* out = part + (size_t)blockIdx.x * MLP_NP;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) out[MLP_W2 + (ty + 16 * r) * MLP_H + tx + 16 * c] = gW2[r][c];
    // the sums over the 16 thread rows, in order
    float(*red)[16][MLP_H] = reinterpret_cast<float(*)[16][MLP_H]>(&s.w2[0][0]);  // dW1 rows, db1, db2, dW3
    static_assert(7 * 16 * MLP_H * sizeof(float) <= sizeof(s.w2) + sizeof(s.w2t), "the sums fit the weights' place");
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int i = 0; i < MLP_IN; ++i) red[i][ty][4 * tx + c] = gW1[i][c];
        red[4][ty][4 * tx + c] = gB1[c];
        red[5][ty][4 * tx + c] = gB2[c];
        red[6][ty][4 * tx + c] = gW3[c];
    }
    if (tx == 0) s.db3[ty] = gB3;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lacc += __shfl_xor_sync(0xffffffffu, lacc, o);
    if ((tid & 31) == 0) s.loss[tid >> 5] = lacc;
    __syncthreads();
    for (int e = tid; e < 7 * MLP_H; e += GR_THREADS) {
        const int v = e / MLP_H, j = e % MLP_H;
        float g = 0.f;
#pragma unroll
        for (int r = 0; r < 16; ++r) g += red[v][r][j];
        const int at = v < 4 ? MLP_W1 + v * MLP_H : v == 4 ? MLP_B1 : v == 5 ? MLP_B2 : MLP_W3;
        out[at + j] = g;
    }
    if (tid == 0) {
        float g = 0.f;
        for (int r = 0; r < 16; ++r) g += s.db3[r];
        out[MLP_B3] = g;
        double l = 0;
        for (int q = 0; q < GR_THREADS / 32; ++q) l += s.loss[q];
        loss_part[blockIdx.x] = l * inv_n;
    }
}

// Sum the block partials in a fixed order (ADAM_SLICES interleaved sums, then
// those in order); Adam update of the FP32 master and BF16 copy when lr > 0; the
// summed gradient goes to g when given.
constexpr int ADAM_SLICES = 8, ADAM_COLS = 32;
__global__ void __launch_bounds__(ADAM_SLICES * ADAM_COLS)
    mlp_adam_kernel(const float* __restrict__ part, int nblocks, float* __restrict__ w32,
                    __nv_bfloat16* __restrict__ w16, float* __restrict__ m, float* __restrict__ v, double lr, double b1t,
                    double b2t, float* __restrict__ g) {
    __shared__ double sums[ADAM_SLICES][ADAM_COLS];
    const int col = threadIdx.x % ADAM_COLS, slice = threadIdx.x / ADAM_COLS;
    const int p = blockIdx.x * ADAM_COLS + col;
    double gs = 0;
    if (p < MLP_NP)
        for (int b = slice; b < nblocks; b += ADAM_SLICES) gs += part[(size_t)b * MLP_NP + p];
    sums[slice][col] = gs;
    __syncthreads();
    if (slice != 0 || p >= MLP_NP) return;
#pragma unroll
    for (int q = 1; q < ADAM_SLICES; ++q) gs += sums[q][col];
    if (g) g[p] = (float)gs;
    if (lr <= 0) return;
    const double beta1 = 0.9, beta2 = 0.999, eps = 1e-8;
    const double mm = beta1 * m[p] + (1 - beta1) * gs;
    const double vv = beta2 * v[p] + (1 - beta2) * gs * gs;
    m[p] = (float)mm;
    v[p] = (float)vv;
    const double mh = mm / (1 - b1t), vh = vv / (1 - b2t);
    const float nw = (float)(w32[p] - lr * mh / (sqrt(vh) + eps));
    w32[p] = nw;
    w16[p] = __float2bfloat16(nw);
}
constexpr int ADAM_BLOCKS = (MLP_NP + ADAM_COLS - 1) / ADAM_COLS;

__global__ void mlp_to_bf16_kernel(const float* __restrict__ w32, __nv_bfloat16* __restrict__ w16) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < MLP_NP) w16[p] = __float2bfloat16(w32[p]);
}

// Chunks of 32 pairs while those still find an SM each to themselves (a training
// batch: 4096 pairs on 128 blocks), 128 above, where the products reuse
// their operands most.
constexpr int GR_SMALL = 32, GR_LARGE = 128;
bool grad_small(long long count, int sm) { return count <= (long long)GR_SMALL * sm; }

int grad_blocks(long long count, int sm) {
    const long long chunk = grad_small(count, sm) ? GR_SMALL : GR_LARGE;
    return (int)std::max<long long>(1, std::min<long long>((count + chunk - 1) / chunk, 2LL * sm));  // two fit an SM
}

template <int PAIRS>
int launch_grad_pairs(cudaStream_t st, int nb, const MlpModel& m, const float* F, const float* T, const int* perm,
                      long long first, long long count, double inv_n) {
    static thread_local int dev_set = -1;
    int dev = 0;
    TN_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev_set != dev) {
        TN_CUDA_CHECK(cudaFuncSetAttribute(mlp_grad_kernel<PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sizeof(GradSmem<PAIRS>)));
        dev_set = dev;
    }
    mlp_grad_kernel<PAIRS><<<nb, GR_THREADS, sizeof(GradSmem<PAIRS>), st>>>(m.w32.as<float>(), F, T, perm, first, count,
                                                                          inv_n, m.part.as<float>(),
                                                                          m.loss.as<double>());
    TN_LAUNCH_CHECK();
    return TN_OK;
}

// m.part and m.loss hold grad_blocks(count) partials.
int launch_grad(const Ctx& c, const MlpModel& m, const float* F, const float* T, const int* perm, long long first,
                long long count) {
    const int nb = grad_blocks(count, c.sm_count);
    if (grad_small(count, c.sm_count))
        return launch_grad_pairs<GR_SMALL>(c.stream, nb, m, F, T, perm, first, count, 1.0 / count);
    return launch_grad_pairs<GR_LARGE>(c.stream, nb, m, F, T, perm, first, count, 1.0 / count);
}

}  // namespace

int mlp_init(MlpModel& m, Ctx& c, unsigned long long seed) {
    m.ctx = &c;
    TN_CHECK(m.w32.ensure(sizeof(float) * MLP_NP));
    TN_CHECK(m.w16.ensure(sizeof(__nv_bfloat16) * MLP_NP));
    TN_CHECK(m.m.ensure(sizeof(float) * MLP_NP));
    TN_CHECK(m.v.ensure(sizeof(float) * MLP_NP));
    // Glorot-uniform weights from a seeded generator, zero biases
    std::vector<float> h(MLP_NP, 0.f);
    std::mt19937_64 g(seed);
    auto fill = [&](int off, int fan_in, int fan_out, int cnt) {
        const double a = std::sqrt(6.0 / (fan_in + fan_out));
        for (int i = 0; i < cnt; ++i) h[off + i] = (float)(((g() >> 11) * (1.0 / 9007199254740992.0) * 2 - 1) * a);
    };
    fill(MLP_W1, MLP_IN, MLP_H, MLP_IN * MLP_H);
    fill(MLP_W2, MLP_H, MLP_H, MLP_H * MLP_H);
    fill(MLP_W3, MLP_H, 1, MLP_H);
    return mlp_set_params(m, h.data());
}

int mlp_set_params(MlpModel& m, const float* host) {
    cudaStream_t st = m.ctx->stream;
    TN_CUDA_CHECK(cudaMemcpyAsync(m.w32.p, host, sizeof(float) * MLP_NP, cudaMemcpyHostToDevice, st));
    TN_CUDA_CHECK(cudaMemsetAsync(m.m.p, 0, sizeof(float) * MLP_NP, st));
    TN_CUDA_CHECK(cudaMemsetAsync(m.v.p, 0, sizeof(float) * MLP_NP, st));
    mlp_to_bf16_kernel<<<(MLP_NP + 255) / 256, 256, 0, st>>>(m.w32.as<float>(), m.w16.as<__nv_bfloat16>());
    TN_LAUNCH_CHECK();
    TN_CUDA_CHECK(cudaStreamSynchronize(st));
    m.adam_t = 0;
    return TN_OK;
}

int mlp_get_params(const MlpModel& m, float* host) {
    cudaStream_t st = m.ctx->stream;
    TN_CUDA_CHECK(cudaMemcpyAsync(host, m.w32.p, sizeof(float) * MLP_NP, cudaMemcpyDeviceToHost, st));
    TN_CUDA_CHECK(cudaStreamSynchronize(st));
    return TN_OK;
}

int mlp_forward(const MlpModel& m, const float* F, long long n, float* Y, cudaStream_t st) {
    if (n <= 0) return TN_OK;
    const long long b = (n + 127) / 128;  // 8 warps of 16-element tiles per block
    const int grid = (int)std::min<long long>(b, (long long)m.ctx->sm_count * 4);
    mlp_forward_kernel<<<grid, 256, 0, st>>>(m.w16.as<__nv_bfloat16>(), F, n, Y);
    TN_LAUNCH_CHECK();
    return TN_OK;
}

int mlp_gradient(MlpModel& m, const float* F, const float* T, long long n, float* grad_host, double* loss) {
    Ctx& c = *m.ctx;
    cudaStream_t st = c.stream;
    if (n <= 0) return TN_BAD_ARG;
    const int nb = grad_blocks(n, c.sm_count);
    TN_CHECK(m.part.ensure(sizeof(float) * ((size_t)nb * MLP_NP + MLP_NP)));
    TN_CHECK(m.loss.ensure(sizeof(double) * nb));
    TN_CHECK(launch_grad(c, m, F, T, nullptr, 0, n));
    float* g = m.part.as<float>() + (size_t)nb * MLP_NP;
    mlp_adam_kernel<<<ADAM_BLOCKS, ADAM_SLICES * ADAM_COLS, 0, st>>>(m.part.as<float>(), nb, m.w32.as<float>(),
                                                          m.w16.as<__nv_bfloat16>(), m.m.as<float>(), m.v.as<float>(),
                                                          0.0, 0.0, 0.0, g);
    TN_LAUNCH_CHECK();
    std::vector<double> lp(nb);
    TN_CUDA_CHECK(cudaMemcpyAsync(grad_host, g, sizeof(float) * MLP_NP, cudaMemcpyDeviceToHost, st));
    TN_CUDA_CHECK(cudaMemcpyAsync(lp.data(), m.loss.p, sizeof(double) * nb, cudaMemcpyDeviceToHost, st));
    TN_CUDA_CHECK(cudaStreamSynchronize(st));
    double l = 0;
    for (double x : lp) l += x;
    if (loss) *loss = l;
    return TN_OK;
}

int mlp_train(MlpModel& m, const float* F, const float* T, long long n, int steps, int batch, double lr,
              unsigned long long seed, double* final_loss) {
    Ctx& c = *m.ctx;
    cudaStream_t st = c.stream;
    if (n <= 0 || steps <= 0) return TN_BAD_ARG;
    if (batch <= 0 || batch > n) batch = (int)std::min<long long>(n, 4096);
    // seeded permutation of the pairs (host Fisher-Yates, uploaded once)
    std::vector<int> perm(n);
    for (long long i = 0; i < n; ++i) perm[i] = (int)i;
    std::mt19937_64 g(seed);
    for (long long i = n - 1; i > 0; --i) {
        const long long j = (long long)(g() % (unsigned long long)(i + 1));
        std::swap(perm[i], perm[j]);
    }
    DevBuf dperm;
    TN_CHECK(dperm.ensure(sizeof(int) * n));
    TN_CUDA_CHECK(cudaMemcpyAsync(dperm.p, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
    const int nb = grad_blocks(batch, c.sm_count);
    TN_CHECK(m.part.ensure(sizeof(float) * ((size_t)nb * MLP_NP + MLP_NP)));
    TN_CHECK(m.loss.ensure(sizeof(double) * nb));
    const long long nbatches = std::max<long long>(1, n / batch);
    for (int s = 0; s < steps; ++s) {
        const long long first = (s % nbatches) * batch;
        TN_CHECK(launch_grad(c, m, F, T, dperm.as<int>(), first, batch));
        ++m.adam_t;
        const double b1t = std::pow(0.9, (double)m.adam_t), b2t = std::pow(0.999, (double)m.adam_t);
        mlp_adam_kernel<<<ADAM_BLOCKS, ADAM_SLICES * ADAM_COLS, 0, st>>>(m.part.as<float>(), nb, m.w32.as<float>(),
                                                              m.w16.as<__nv_bfloat16>(), m.m.as<float>(),
                                                              m.v.as<float>(), lr, b1t, b2t, nullptr);
        TN_LAUNCH_CHECK();
    }
    std::vector<double> lp(nb);
    TN_CUDA_CHECK(cudaMemcpyAsync(lp.data(), m.loss.p, sizeof(double) * nb, cudaMemcpyDeviceToHost, st));
    TN_CUDA_CHECK(cudaStreamSynchronize(st));
    double l = 0;
    for (double x : lp) l += x;
    if (final_loss) *final_loss = l;
    return TN_OK;
}

int recorder_init(DvRecorder& r, Ctx& c, long long capacity) {
    r.ctx = &c;
    r.capacity = capacity;
    r.size = 0;
    TN_CHECK(r.feats.ensure(sizeof(float) * MLP_IN * (size_t)capacity));
    TN_CHECK(r.targets.ensure(sizeof(float) * (size_t)capacity));
    return TN_OK;
}

}  // namespace tnb
