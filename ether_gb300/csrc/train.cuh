// train.cuh -- one training step of the learned proposals' networks (IN -> 128 -> 128 -> OUT,
// ReLU, BF16-rounded weights and activations, FP32 arithmetic, Adam), shared by the Ising
// (k_learn.cu) and the Heisenberg (k_learn_xyz.cu) learner.
//
// Two launches per step.  A minibatch of 1024 rows is 0.34 GFLOP, about 5 us of the FP32
// pipes; as 20 launches of general 64 x 64 GEMM tiles, whose gradients ran on four to ten
// blocks, and of bias sums that ran on one block, a step took 580 us.
//   train_rows    8 rows per block (128 blocks for 1024 rows): the rows' gather, the three
//                 layers, the loss and the backward pass to both hidden layers, activations in
//                 shared memory; the weights, packed as BF16 pairs along the summed index,
//                 stream from the L2 coalesced over the outputs.
//   train_wgrad   the three weight gradients and the bias sums, 16 x 32 tiles (136 blocks for
//                 the XYZ network: the outputs, not the batch, are what is divided), and Adam,
//                 the rounded and the packed weights of the tile.
// Every sum is one chain in increasing order of its index, so the result does not depend on
// the tiles: Adam divides by the gradient's size, so after a few steps another order of the
// batch sums moves the weights by 1e-3, through the BF16 roundings.  That rules a split of
// the batch out (measured 12x against the 20 launches, with other weights).  As it stands a
// step of 1024 rows of the XYZ network takes 53 us (580 before; train_rows 37-39 us and
// train_wgrad 21-22 us with cold caches).  train_rows waits for its weights: of 12 warp cycles per
// issue 7.7 are loads from the L2, each layer's begun when the layer before has ended (the chain of
// 784 fmaf itself is about 2 us); train_wgrad has one warp a scheduler, short of parallel work.
#pragma once
#include <cuda_bf16.h>

#include "learn_common.cuh"
#include "rng_math.cuh"

namespace ether {
namespace learn {

constexpr int kTrainRows = 8;      // rows per block of train_rows

// Parameter offsets (W1, b1, W2, b2, W3, b3; row = output unit) and the packed weights' offsets
// in 32-bit words: F1, F2, F3 for the forward sums (pairs along the inputs), B3, B2 for the
// backward ones (pairs along the outputs).
template <int IN, int OUT>
struct TrainNet {
    static constexpr int W1 = 0, b1 = W1 + NH * IN, W2 = b1 + NH, b2 = W2 + NH * NH, W3 = b2 + NH,
                         b3 = W3 + OUT * NH, N = b3 + OUT;
    static constexpr int F1 = 0, F2 = F1 + IN / 2 * NH, F3 = F2 + NH / 2 * NH, B3 = F3 + NH / 2 * OUT,
                         B2 = B3 + OUT / 2 * NH, WORDS = B2 + NH / 2 * NH;
};

__device__ __forceinline__ float bf16_round(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// acc[r] = sum over k < K, in order, of x[(r0 + r) * K + k] * W(k, c): one column c of a layer
// for RPT rows of shared memory.
template <int K, int C, int RPT>
__device__ __forceinline__ void train_column(const float *x, const uint32_t *__restrict__ W, int c, int r0,
                                             float (&acc)[RPT]) {
#pragma unroll
    for (int r = 0; r < RPT; ++r) acc[r] = 0.f;
#pragma unroll 8
    for (int k = 0; k < K; k += 4) {
        const uint32_t w0 = __ldg(W + (k >> 1) * C + c), w1 = __ldg(W + (k >> 1) * C + C + c);
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const float4 v = *reinterpret_cast<const float4 *>(x + (r0 + r) * K + k);
            acc[r] = fmaf(v.x, bf_lo(w0), acc[r]);
            acc[r] = fmaf(v.y, bf_hi(w0), acc[r]);
            acc[r] = fmaf(v.z, bf_lo(w1), acc[r]);
            acc[r] = fmaf(v.w, bf_hi(w1), acc[r]);
        }
    }
}

struct TrainIo {
    const __nv_bfloat16 *X;  // data set (rows of IN); null: Xb and Yb hold the batch already
    const void *Y;           // targets: XYZ float[OUT] per row, Ising one word of bits
    long long n;             // samples in the data set
    int B;
    uint32_t seed, step, stream;  // Philox address of the minibatch
    float *Xb, *Yb, *H1, *H2, *dZ, *dH1, *dH2;
    double *loss_part;       // one sum per block
};

// Loss and its gradient of output pair (row, site k): XYZ, the von Mises-Fisher negative log
// density -(log C(kappa) + m . y), C(kappa) = kappa / (4 pi sinh kappa), m = z + b3, and
// -(y + A(kappa) m) / B, A = (1/kappa - coth kappa) / kappa (series below 1e-2); Ising, the
// cross entropy softplus(z) - y z of output k and (sigmoid - y) / B.
template <int OUT>
__device__ __forceinline__ double train_loss(const float *z, const float *b3, const float *y, float *g, int k, int B) {
    if constexpr (OUT == 96) {
        constexpr float kLog4Pi = 2.53102425f, kLog2Pi = 1.83787707f;
        const float mx = z[3 * k] + b3[3 * k], my = z[3 * k + 1] + b3[3 * k + 1], mz = z[3 * k + 2] + b3[3 * k + 2];
        const float *t = y + 3 * k;
        const float kap = sqrtf(mx * mx + my * my + mz * mz);
        float logc, A;
        if (kap < 1e-2f) {
            const float k2 = kap * kap;
            logc = -kLog4Pi - k2 * (1.0f / 6.0f) + k2 * k2 * (1.0f / 180.0f);
            A = -1.0f / 3.0f + k2 * (1.0f / 45.0f);
        } else {
            logc = logf(kap) - kap - logf(-expm1f(-2.0f * kap)) - kLog2Pi;
            A = (1.0f / kap - 1.0f / tanhf(kap)) / kap;
        }
        const float dot = mx * t[0] + my * t[1] + mz * t[2];
        g[3 * k] = -(t[0] + A * mx) / (float)B;
        g[3 * k + 1] = -(t[1] + A * my) / (float)B;
        g[3 * k + 2] = -(t[2] + A * mz) / (float)B;
        return -(double)(logc + dot);
    } else {
        const float zz = z[k] + b3[k];
        const float p = 1.0f / (1.0f + expf(-zz));
        g[k] = (p - y[k]) / (float)B;
        const float sp = zz > 0.0f ? zz + log1pf(expf(-zz)) : log1pf(expf(zz));
        return (double)(sp - y[k] * zz);
    }
}

// See the head of the file.  pq: parameters with rounded weights (its biases are used).
template <int IN, int OUT>
__global__ void __launch_bounds__(256) train_rows(TrainIo T, const float *__restrict__ pq,
                                                  const uint32_t *__restrict__ wp) {
    using Net = TrainNet<IN, OUT>;
    constexpr int R = kTrainRows;
    __shared__ __align__(16) float xs[R * IN];
    __shared__ __align__(16) float h1[R * NH], h2[R * NH], d2[R * NH];
    __shared__ __align__(16) float zs[R * OUT], ys[R * OUT], dz[R * OUT];
    __shared__ long long row[R];
    __shared__ double red[8];
    const int tid = threadIdx.x;
    const int b0 = blockIdx.x * R, nr = min(R, T.B - b0);
    if (T.X) {
        if (tid < nr) {
            const U4 d = draw((uint32_t)(b0 + tid), T.step, T.stream, kLearn | (0xFDu << 8), T.seed);
            row[tid] = (long long)((((unsigned long long)d.y << 32) | d.x) % (unsigned long long)T.n);
        }
        __syncthreads();
    }
    for (int e = tid; e < R * (IN / 2); e += 256) {
        const int r = e / (IN / 2), i = 2 * (e - r * (IN / 2));
        float2 v = make_float2(0.f, 0.f);
        if (r < nr) {
            float2 *xb = reinterpret_cast<float2 *>(T.Xb + (size_t)(b0 + r) * IN + i);
            if (T.X) {
                v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(T.X + (size_t)row[r] * IN + i));
                *xb = v;
            } else {
                v = *xb;
            }
        }
        *reinterpret_cast<float2 *>(xs + r * IN + i) = v;
    }
    for (int e = tid; e < R * OUT; e += 256) {
        const int r = e / OUT, o = e - r * OUT;
        float v = 0.f;
        if (r < nr) {
            if (!T.X) v = T.Yb[(size_t)(b0 + r) * OUT + o];
            else if constexpr (OUT == 96) v = static_cast<const float *>(T.Y)[(size_t)row[r] * OUT + o];
            else v = (float)((static_cast<const uint32_t *>(T.Y)[row[r]] >> o) & 1u);
        }
        ys[e] = v;
    }
    __syncthreads();
    const int c = tid & (NH - 1), r0 = (tid >> 7) * 4;
    float acc[4];
    train_column<IN, NH, 4>(xs, wp + Net::F1, c, r0, acc);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float v = bf16_round(fmaxf(acc[r] + pq[Net::b1 + c], 0.0f));
        h1[(r0 + r) * NH + c] = v;
        if (r0 + r < nr) T.H1[(size_t)(b0 + r0 + r) * NH + c] = v;
    }
    __syncthreads();
    train_column<NH, NH, 4>(h1, wp + Net::F2, c, r0, acc);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float v = bf16_round(fmaxf(acc[r] + pq[Net::b2 + c], 0.0f));
        h2[(r0 + r) * NH + c] = v;
        if (r0 + r < nr) T.H2[(size_t)(b0 + r0 + r) * NH + c] = v;
    }
    __syncthreads();
    {
        constexpr int G = OUT == 96 ? 2 : 256 / OUT, RPT = R / G;  // row groups, rows per thread
        const int g = tid / OUT, o = tid - g * OUT;
        if (g < G) {
            float az[RPT];
            train_column<NH, OUT, RPT>(h2, wp + Net::F3, o, g * RPT, az);
#pragma unroll
            for (int r = 0; r < RPT; ++r) zs[(g * RPT + r) * OUT + o] = az[r];
        }
    }
    __syncthreads();
    double s = 0.0;
    {
        const int r = tid >> 5, k = tid & 31;  // 8 rows x 32 sites
        if (r < nr) {
            s = train_loss<OUT>(zs + r * OUT, pq + Net::b3, ys + r * OUT, dz + r * OUT, k, T.B);
        } else {
            for (int j = 0; j < OUT / 32; ++j) dz[r * OUT + k + 32 * j] = 0.f;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((tid & 31) == 0) red[tid >> 5] = s;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w];
        T.loss_part[blockIdx.x] = t;
    }
    for (int e = tid; e < nr * OUT; e += 256) T.dZ[(size_t)b0 * OUT + e] = dz[e];
    train_column<OUT, NH, 4>(dz, wp + Net::B3, c, r0, acc);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float v = h2[(r0 + r) * NH + c] > 0.0f ? acc[r] : 0.0f;
        d2[(r0 + r) * NH + c] = v;
        if (r0 + r < nr) T.dH2[(size_t)(b0 + r0 + r) * NH + c] = v;
    }
    __syncthreads();
    train_column<NH, NH, 4>(d2, wp + Net::B2, c, r0, acc);
#pragma unroll
    for (int r = 0; r < 4; ++r)
        if (r0 + r < nr) T.dH1[(size_t)(b0 + r0 + r) * NH + c] = h1[(r0 + r) * NH + c] > 0.0f ? acc[r] : 0.0f;
}

struct TrainParams {
    float *p, *g, *m, *v, *pq;
    uint32_t *wp;  // TrainNet::WORDS
    double *loss;
};
// Adam's step (lr = 0: none, the gradient alone is kept) with bias corrections c1, c2.
struct AdamStep {
    float lr, c1, c2;
};

// Parameter i (of row o, column k of its matrix; biases: k < 0): its rounded value into pq and
// into the packed weights.
template <int IN, int OUT>
__device__ __forceinline__ void train_put(const TrainParams &P, int i, int layer, int o, int k, float x) {
    using Net = TrainNet<IN, OUT>;
    if (k < 0) {
        P.pq[i] = x;
        return;
    }
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    P.pq[i] = __bfloat162float(h);
    __nv_bfloat16 *w = reinterpret_cast<__nv_bfloat16 *>(P.wp);
    if (layer == 0) {
        w[2 * (Net::F1 + (k >> 1) * NH + o) + (k & 1)] = h;
    } else if (layer == 1) {
        w[2 * (Net::F2 + (k >> 1) * NH + o) + (k & 1)] = h;
        w[2 * (Net::B2 + (o >> 1) * NH + k) + (o & 1)] = h;
    } else {
        w[2 * (Net::F3 + (k >> 1) * OUT + o) + (k & 1)] = h;
        w[2 * (Net::B3 + (o >> 1) * NH + k) + (o & 1)] = h;
    }
}

// Parameter i's gradient is known: keep it, and with lr > 0 Adam's update.
template <int IN, int OUT>
__device__ __forceinline__ void train_update(const TrainParams &P, const AdamStep &S, int i, int layer, int o, int k,
                                             float gi) {
    P.g[i] = gi;
    if (!(S.lr > 0.f)) return;
    const float mi = 0.9f * P.m[i] + 0.1f * gi;
    const float vi = 0.999f * P.v[i] + 0.001f * gi * gi;
    P.m[i] = mi;
    P.v[i] = vi;
    const float x = P.p[i] - S.lr * (mi / S.c1) / (sqrtf(vi / S.c2) + 1e-8f);
    P.p[i] = x;
    train_put<IN, OUT>(P, i, layer, o, k, x);
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// One 16 x 32 tile of a weight gradient G(m, n) = sum over the batch rows of A(b, m) D(b, n),
// and (first column of tiles) the bias gradient sum of A(b, m); then the tile's parameters.
// 128 threads of 2 x 2 outputs; 64 batch rows per stage, three stages of cp.async (a tile is
// one chain of B dependent fmaf, so what bounds the kernel is keeping that chain fed).
template <int IN, int OUT>
__global__ void __launch_bounds__(128) train_wgrad(TrainIo T, TrainParams P, AdamStep S) {
    using Net = TrainNet<IN, OUT>;
    constexpr int TM = 16, TN = 32, KB = 64, ST = 3, NT1 = (IN + TN - 1) / TN, NT = NH / TN, MT = NH / TM;
    __shared__ __align__(16) float As[ST][KB][TM], Ds[ST][KB][TN];
    const int tid = threadIdx.x;
    int tile = blockIdx.x;
    const float *A, *D;
    int M, N, offW, offb, mt, nt, layer;
    if (tile < MT * NT1) {
        A = T.dH1; D = T.Xb; M = NH; N = IN; offW = Net::W1; offb = Net::b1; layer = 0;
        mt = tile / NT1; nt = tile - mt * NT1;
    } else if ((tile -= MT * NT1) < MT * NT) {
        A = T.dH2; D = T.H1; M = NH; N = NH; offW = Net::W2; offb = Net::b2; layer = 1;
        mt = tile / NT; nt = tile - mt * NT;
    } else {
        tile -= MT * NT;
        A = T.dZ; D = T.H2; M = OUT; N = NH; offW = Net::W3; offb = Net::b3; layer = 2;
        mt = tile / NT; nt = tile - mt * NT;
    }
    const int m0 = mt * TM, n0 = nt * TN, B = T.B;
    const int tx = tid & 15, ty = tid >> 4;
    auto load = [&](int kb, int st) {
#pragma unroll
        for (int u = 0; u < KB * TM / 4 / 128; ++u) {
            const int e = tid + 128 * u, kk = e >> 2, q = (e & 3) * 4;
            const bool in = kb + kk < B;
            cp_async16(&As[st][kk][q], A + (size_t)(in ? kb + kk : 0) * M + m0 + q, in);
        }
#pragma unroll
        for (int u = 0; u < KB * TN / 4 / 128; ++u) {
            const int e = tid + 128 * u, kk = e >> 3, q = (e & 7) * 4;
            const bool in = kb + kk < B && n0 + q < N;
            cp_async16(&Ds[st][kk][q], D + (in ? (size_t)(kb + kk) * N + n0 + q : 0), in);
        }
    };
    float acc[2][2] = {};
    float bias[2] = {0.f, 0.f};
    const bool want_bias = nt == 0;
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        load(s * KB, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int st = 0;
    for (int kb = 0; kb < B; kb += KB) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();
        load(kb + (ST - 1) * KB, st == 0 ? ST - 1 : st - 1);  // the stage read in the last turn
        asm volatile("cp.async.commit_group;" ::: "memory");
        // rows past the batch were zero-filled: adding 0 * 0 keeps a sum, and its zero's sign is
        // that of +0, which every chain starts with
#pragma unroll 16
        for (int kk = 0; kk < KB; ++kk) {
            const float2 a = *reinterpret_cast<const float2 *>(&As[st][kk][2 * ty]);
            const float2 d = *reinterpret_cast<const float2 *>(&Ds[st][kk][2 * tx]);
            acc[0][0] = fmaf(a.x, d.x, acc[0][0]);
            acc[0][1] = fmaf(a.x, d.y, acc[0][1]);
            acc[1][0] = fmaf(a.y, d.x, acc[1][0]);
            acc[1][1] = fmaf(a.y, d.y, acc[1][1]);
        }
        if (want_bias && tx == 0)
#pragma unroll 16
            for (int kk = 0; kk < KB; ++kk) {
                bias[0] += As[st][kk][2 * ty];
                bias[1] += As[st][kk][2 * ty + 1];
            }
        st = st == ST - 1 ? 0 : st + 1;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int m = m0 + 2 * ty + i;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int n = n0 + 2 * tx + j;
            if (n < N) train_update<IN, OUT>(P, S, offW + m * N + n, layer, m, n, acc[i][j]);
        }
        if (want_bias && tx == 0) train_update<IN, OUT>(P, S, offb + m, layer, m, -1, bias[i]);
    }
}

template <int IN, int OUT>
constexpr int train_tiles() { return NH / 16 * ((IN + 31) / 32) + NH / 16 * (NH / 32) + OUT / 16 * (NH / 32); }

// The rounded and packed weights of p.
template <int IN, int OUT>
__global__ void train_pack_kernel(TrainParams P) {
    using Net = TrainNet<IN, OUT>;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Net::N) return;
    const int layer = i < Net::W2 ? 0 : i < Net::W3 ? 1 : 2;
    const int off = layer == 0 ? Net::W1 : layer == 1 ? Net::W2 : Net::W3, cols = layer == 0 ? IN : NH;
    const int bias = layer == 0 ? Net::b1 : layer == 1 ? Net::b2 : Net::b3;
    const int o = i >= bias ? i - bias : (i - off) / cols, k = i >= bias ? -1 : (i - off) - o * cols;
    train_put<IN, OUT>(P, i, layer, o, k, P.p[i]);
}

// loss = the blocks' sums, in a fixed order, / B (one warp).
static __global__ void train_loss_sum(const double *__restrict__ part, int n, int B, double *__restrict__ loss) {
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += 32) s += part[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *loss = s / B;
}

// The device buffers of a learner's training: batch rows up to maxB.
struct TrainBuffers {
    int maxB = 0;
    float *Xb = nullptr, *Yb = nullptr, *H1 = nullptr, *H2 = nullptr, *dZ = nullptr, *dH1 = nullptr, *dH2 = nullptr;
    double *loss_part = nullptr;  // one per block of train_rows
    void release() {
        void *ptrs[] = {Xb, Yb, H1, H2, dZ, dH1, dH2, loss_part};
        for (void *q : ptrs)
            if (q) cudaFree(q);
        *this = TrainBuffers{};
    }
    template <int IN, int OUT>
    cudaError_t ensure(int B) {
        if (B <= maxB) return cudaSuccess;
        release();
        struct {
            float **p;
            size_t n;
        } bufs[] = {{&Xb, (size_t)B * IN}, {&Yb, (size_t)B * OUT}, {&H1, (size_t)B * NH}, {&H2, (size_t)B * NH},
                    {&dZ, (size_t)B * OUT}, {&dH1, (size_t)B * NH}, {&dH2, (size_t)B * NH}};
        for (auto &b : bufs) {
            const cudaError_t e = cudaMalloc((void **)b.p, b.n * sizeof(float));
            if (e != cudaSuccess) return e;
        }
        const cudaError_t e = cudaMalloc((void **)&loss_part, (size_t)((B + kTrainRows - 1) / kTrainRows) * sizeof(double));
        if (e != cudaSuccess) return e;
        maxB = B;
        return cudaSuccess;
    }
};

template <int IN, int OUT>
cudaError_t train_pack(const TrainParams &P, cudaStream_t st) {
    train_pack_kernel<IN, OUT><<<(TrainNet<IN, OUT>::N + 255) / 256, 256, 0, st>>>(P);
    return cudaGetLastError();
}

// One step on a batch: gradients into P.g, with S.lr > 0 the update; with want_loss the mean
// loss into P.loss.  Adds its launches to *launches.
template <int IN, int OUT>
cudaError_t train_step(const TrainParams &P, TrainIo T, TrainBuffers &b, const AdamStep &S, bool want_loss,
                       cudaStream_t st, uint64_t *launches) {
    T.Xb = b.Xb; T.Yb = b.Yb; T.H1 = b.H1; T.H2 = b.H2; T.dZ = b.dZ; T.dH1 = b.dH1; T.dH2 = b.dH2;
    T.loss_part = b.loss_part;
    const int blocks = (T.B + kTrainRows - 1) / kTrainRows;
    train_rows<IN, OUT><<<blocks, 256, 0, st>>>(T, P.pq, P.wp);
    train_wgrad<IN, OUT><<<train_tiles<IN, OUT>(), 128, 0, st>>>(T, P, S);
    *launches += 2;
    if (want_loss) {
        train_loss_sum<<<1, 32, 0, st>>>(b.loss_part, blocks, T.B, P.loss);
        *launches += 1;
    }
    return cudaGetLastError();
}

}  // namespace learn
}  // namespace ether
