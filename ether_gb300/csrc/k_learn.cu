// k_learn.cu -- learned patch proposal for the simple-cubic Ising model (ether_learn_* in the
// C-ABI).  The reference has no learned move; what it fixes is the target distribution,
// exp(-beta E) with E = sum over bonds of J s_i s_j (src/Hamiltonian.f90:57-105,
// src/Metropolis.f90:50-56), and every learned move below is accepted or rejected by exact
// Metropolis-Hastings against that energy, so the stationary distribution is unchanged.
//
// Move (one "learned sweep" = patch class 0, then class 1; patches of a class share no bond):
//   * per replica and sweep a Philox offset (ox, oy, oz) in [0,4)^3 tiles the lattice with 4^3
//     patches; canonical frame reflected in x when ox+oy+oz is odd, so the 32 network-proposed
//     A-sites are always colour 0 and the 32 B-sites colour 1;
//   * network: input = the 96 boundary spins and 4 beta J; 128 -> 128 -> 128 -> 32 MLP, BF16
//     weights and activations, FP32 accumulation, on the tensor cores (tcgen05, accumulators in
//     TMEM): a group of 128 threads takes 128 patches, thread p owns patch p = TMEM lane p through all three
//     layers;
//   * proposal: A-site k up with probability T_k / 2^32 from the logit; every B-site then from
//     its exact heat-bath conditional given the new A-sites and the boundary;
//   * acceptance: log alpha = log q(old) - log q(new) - beta J (bond change), FP32 in a fixed
//     order with an own exp (the same operations as oracle/learn_oracle.c, which replays a
//     sweep bit for bit given the logits).
// A class is three launches (gather_kernel, patch_kernel, mh_kernel): only the network needs the
// weights' shared memory, which leaves few warps on an SM, so the gather and the
// Metropolis-Hastings step, most of the instructions, run on their own with many (a class of
// 64^3 x 256: one kernel 510 us, the three 173 us).
// Training: maximum likelihood of the A-sites given the boundary on configurations the plain
// sweep produced (any temperature of the context's ladder), Adam, straight-through BF16
// rounding (train.cuh).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "internal.h"
#include "learn_common.cuh"
#include "rng_math.cuh"
#include "tc_util.cuh"
#include "train.cuh"

namespace ether {
namespace learn {

constexpr int NI = 128, NO = 32;  // network input and output widths (hidden: NH)
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NH * NI, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH,
              OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NO * NH, NPARAM = OFF_B3 + NO;

// Packed inference image (global memory, copied to shared memory by every CTA):
// W1 (2 tiles x 128 rows x 128 B), W2 (same), W3 (2 tiles x 32 rows x 128 B), b1, b2, b3 (FP32).
constexpr int IMG_W1 = 0, IMG_W2 = 32768, IMG_W3 = 65536, IMG_B1 = 73728, IMG_B2 = IMG_B1 + 512,
              IMG_B3 = IMG_B2 + 512, IMG_BYTES = IMG_B3 + 128;
// Shared memory of the patch kernel (from a 1024-byte aligned base).
constexpr int kGroups = 4, SM_A = 73728, SM_BIAS = SM_A + kGroups * 32768, SM_BAR = SM_BIAS + 1152,
              SM_BYTES = SM_BAR + 8 * kGroups + 16;
// Patches of one pass: bounds the logits' memory (128 MB).  Smaller passes, whose logits would
// stay in L2, lose more at their ends: 2^18 and 2^17 made a 64^3 x 256 sweep 8 and 19% slower.
constexpr long long kPassPatches = 1LL << 20;
constexpr int kThreads = 128;  // rows of a tile = threads of a group

// ------------------------------------------------------------------ patch geometry ----
// Local sites 0..31 = A-sites, 32..63 = B-sites, packed (a | b << 2 | c << 4); boundary
// sites packed ((a+1) | (b+1) << 4 | (c+1) << 8).  The neighbour tables below (B-site
// neighbours: >= 0 A-site index, < 0 boundary -(1 + index); A-site boundary neighbours) are
// built once on the host and must agree with the closed forms the kernels use.
__constant__ uint8_t c_site[64];
__constant__ uint16_t c_bnd[96];

struct Geometry {
    uint8_t site[64];
    uint16_t bnd[96];
    int8_t Bn[32][6];
    int8_t Ab[32][3];
};

static int face_index(int a, int b, int c) {
    if (a == -1) return b + 4 * c;
    if (a == 4) return 16 + b + 4 * c;
    if (b == -1) return 32 + a + 4 * c;
    if (b == 4) return 48 + a + 4 * c;
    if (c == -1) return 64 + a + 4 * b;
    return 80 + a + 4 * b;
}

static bool closed_forms_agree(const Geometry &g);

static Geometry make_geometry() {
    Geometry g;
    int A[32][3], B[32][3], na = 0, nb = 0, idx_of[64];
    for (int lin = 0; lin < 64; ++lin) {
        const int a = lin & 3, b = (lin >> 2) & 3, c = lin >> 4;
        if (((a + b + c) & 1) == 0) {
            A[na][0] = a; A[na][1] = b; A[na][2] = c;
            idx_of[lin] = na++;
        } else {
            B[nb][0] = a; B[nb][1] = b; B[nb][2] = c;
            idx_of[lin] = nb++;
        }
    }
    for (int k = 0; k < 32; ++k) {
        g.site[k] = (uint8_t)(A[k][0] | (A[k][1] << 2) | (A[k][2] << 4));
        g.site[32 + k] = (uint8_t)(B[k][0] | (B[k][1] << 2) | (B[k][2] << 4));
    }
    for (int f = 0; f < 6; ++f)
        for (int u = 0; u < 4; ++u)
            for (int v = 0; v < 4; ++v) {
                const int e = (f & 1) ? 4 : -1;
                int a, b, c;
                if (f < 2) { a = e; b = u; c = v; }
                else if (f < 4) { a = u; b = e; c = v; }
                else { a = u; b = v; c = e; }
                g.bnd[face_index(a, b, c)] = (uint16_t)((a + 1) | ((b + 1) << 4) | ((c + 1) << 8));
            }
    static const int d[6][3] = {{-1, 0, 0}, {1, 0, 0}, {0, -1, 0}, {0, 1, 0}, {0, 0, -1}, {0, 0, 1}};
    for (int m = 0; m < 32; ++m)
        for (int q = 0; q < 6; ++q) {
            const int a = B[m][0] + d[q][0], b = B[m][1] + d[q][1], c = B[m][2] + d[q][2];
            if (a < 0 || a > 3 || b < 0 || b > 3 || c < 0 || c > 3) g.Bn[m][q] = (int8_t)(-(1 + face_index(a, b, c)));
            else g.Bn[m][q] = (int8_t)idx_of[a + 4 * b + 16 * c];
        }
    for (int k = 0; k < 32; ++k) {
        int n = 0;
        for (int q = 0; q < 3; ++q) g.Ab[k][q] = -1;
        for (int q = 0; q < 6; ++q) {
            const int a = A[k][0] + d[q][0], b = A[k][1] + d[q][1], c = A[k][2] + d[q][2];
            if (a < 0 || a > 3 || b < 0 || b > 3 || c < 0 || c > 3) g.Ab[k][n++] = (int8_t)face_index(a, b, c);
        }
    }
    return g;
}

// Closed forms of the same geometry (geo_*) are in learn_common.cuh.

// ------------------------------------------------------------- own FP32 functions ----
// Same operation sequence as oracle/learn_oracle.c (compiled with --fmad=false: explicit
// fmaf only).
// sigmoid(z) = r or e r with e = exp(-|z|), r = 1 / (1 + e) correctly rounded.
__device__ __forceinline__ float sigmoid_own(float z) {
    const float e = expf_neg(-fabsf(z));
    const float r = __frcp_rn(1.0f + e);
    return z >= 0.0f ? r : e * r;
}
__device__ __forceinline__ uint32_t thr_of_logit(float z) {
    float t = sigmoid_own(z) * 4294967296.0f;
    t = fmaxf(t, 1.0f);
    t = fminf(t, 4294967040.0f);
    return (uint32_t)t;
}

// ------------------------------------------------------------------- the patch kernel ----
struct PatchParams {
    const uint8_t *img;           // packed weights + biases (IMG_BYTES)
    int *err;
    // lattice mode: patches of class cls of replicas r0 .. (n of them, replica-major)
    uint8_t *spins;
    int L1, L2, L3, H;
    long long half;               // sites per colour per replica
    int P1, P2, P3, cls, r0, n;
    FastDiv fPc, fhalf1, fP2;     // patches of a class per replica, P1 / 2, P2
    const uint32_t *stream_id, *lstep;
    const int32_t *slot_of_rep;
    const float *k4, *betaJf;     // per slot
    const uint4 *HB;              // per slot x 7: heat-bath threshold, log probabilities up, down
    RoundKeys K;                  // of the context's seed
    unsigned long long *acc;      // per replica: accepted patches
    uint32_t *bits;               // [5][n]: boundary (3 words), A-sites, B-sites of a patch
    float *dump;                  // optional [n][32]: the pass's logits, kept
    // forward mode
    const __nv_bfloat16 *X;       // [n][128]
    float *Z;                     // logits: [n][32] (forward mode), [8][n] of four (lattice mode)
};

__device__ __forceinline__ int wrap(int x, int L) { return x >= L ? x - L : (x < 0 ? x + L : x); }

// storage byte of canonical (a, b, c) in [-1, 4] of the patch at origin o with reflection par
__device__ __forceinline__ long long site_addr(const PatchParams &P, int o0, int o1, int o2, int par,
                                               int a, int b, int c) {
    const int x = wrap(o0 + (par ? 3 - a : a), P.L1);
    const int y = wrap(o1 + b, P.L2);
    const int z = wrap(o2 + c, P.L3);
    return (long long)((x + y + z) & 1) * P.half + ((long long)z * P.L2 + y) * P.H + (x >> 1);
}

// Patch w of a pass: replica, number, sweep counter, origin and reflection.
struct Patch {
    int r, o0, o1, o2, par;
    uint32_t pidx, t, stream;
};
__device__ __forceinline__ Patch decode(const PatchParams &P, int w) {
    Patch D;
    const int rr = (int)fdiv((uint32_t)w, P.fPc);
    const int q = w - rr * (int)P.fPc.d;
    D.r = P.r0 + rr;
    const int row = (int)fdiv((uint32_t)q, P.fhalf1);
    const int tt = q - row * (int)P.fhalf1.d;
    const int pk = (int)fdiv((uint32_t)row, P.fP2), pj = row - pk * P.P2;
    const int pi = 2 * tt + ((P.cls + pj + pk) & 1);
    D.pidx = (uint32_t)(pi + P.P1 * (pj + P.P2 * pk));
    D.t = P.lstep[D.r];
    D.stream = P.stream_id[D.r];
    const U4 ow = draw_rk(0xFFFFFFFFu, D.t, D.stream, kLearn | (0xFFu << 8), P.K);
    const int ox = (int)(ow.x & 3u), oy = (int)((ow.x >> 2) & 3u), oz = (int)((ow.x >> 4) & 3u);
    D.par = (ox + oy + oz) & 1;
    D.o0 = 4 * pi + ox;
    D.o1 = 4 * pj + oy;
    D.o2 = 4 * pk + oz;
    return D;
}

// The spins of every patch of a pass as bits, one thread per patch.  The sites a = -1, 1, 3 (the
// odd ones) of a patch row are three neighbouring bytes of one colour's array, and so are a = 0,
// 2, 4: one or two aligned words and a byte permute (which also undoes the reflection) bring them,
// and shifted additions collect the same a of eight rows in a byte.  Lanes are neighbouring
// patches of a lattice row, four bytes apart.  (64^3 x 256, per class: a warp gathering its
// patches one after another, five sites per lane, 240 us; a byte load per site 45 us; this
// 34 us.)
struct RowWords {
    int w0, w1;     // byte offsets of the words in a row
    uint32_t sel;   // the three bytes, in order of a
    bool two;       // they reach into the second word
};
__device__ __forceinline__ RowWords row_words(int x, int H, bool reversed) {
    RowWords W;
    const int h = x >> 1, s = h & 3;
    W.w0 = h & ~3;
    W.w1 = W.w0 + 4 < H ? W.w0 + 4 : 0;
    W.two = s > 1;
    W.sel = reversed ? (uint32_t)((s + 2) | ((s + 1) << 4) | (s << 8)) : (uint32_t)(s | ((s + 1) << 4) | ((s + 2) << 8));
    return W;
}
__device__ __forceinline__ uint32_t row_bytes(const uint8_t *row, const RowWords &W) {
    const uint32_t lo = *reinterpret_cast<const uint32_t *>(row + W.w0);
    uint32_t hi = 0;
    if (W.two) hi = *reinterpret_cast<const uint32_t *>(row + W.w1);
    return __byte_perm(lo, hi, W.sel) & 0x00FFFFFFu;
}
// 16 bits to the even positions.
__host__ __device__ __forceinline__ uint32_t spread(uint32_t x) {
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}
// Byte i of eight faces' rows (rows 0-3 of the low face, 4-7 of the high one): to bits 4 u.
__host__ __device__ __forceinline__ uint32_t face_bits(uint32_t acc, int i) {
    uint32_t x = (acc >> (8 * i)) & 0xFFu;
    x = (x & 15u) | ((x & 0xF0u) << 12);
    return (x | (x << 3) | (x << 6) | (x << 9)) & 0x11111111u;
}
// Bits of a 16-row class word from the a = 0, 2 (even) and a = 1, 3 (odd) columns over the rows;
// the class has the even columns in the rows of `even_rows`.
__host__ __device__ __forceinline__ uint32_t class_bits(uint32_t a0, uint32_t a2, uint32_t a1, uint32_t a3,
                                                        uint32_t even_rows) {
    const uint32_t odd_rows = ~even_rows & 0xFFFFu;
    return spread((a0 & even_rows) | (a1 & odd_rows)) | (spread((a2 & even_rows) | (a3 & odd_rows)) << 1);
}
constexpr uint32_t kEvenRows = 0xA5A5u;  // bit b + 4 c set where b + c is even

__global__ void __launch_bounds__(256) gather_kernel(const PatchParams P) {
    const int w = blockIdx.x * 256 + threadIdx.x;
    if (w >= P.n) return;
    after_wait();
    after_release();  // not before the wait: patch_kernel reads the weights before its own
    const Patch D = decode(P, w);
    const uint8_t *sp = P.spins + (long long)D.r * 2 * P.half;
    const bool rev = D.par != 0;
    const int x0 = wrap(D.o0 - 1, P.L1), x1 = wrap(D.o0, P.L1);
    const RowWords odd = row_words(rev ? x1 : x0, P.H, rev), even = row_words(rev ? x0 : x1, P.H, rev);
    int yo[6];
    long long zo[6];
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        yo[a] = wrap(D.o1 + a - 1, P.L2) * P.H;
        zo[a] = (long long)wrap(D.o2 + a - 1, P.L3) * P.L2 * P.H;
    }
    uint32_t io[2] = {0, 0}, ie[2] = {0, 0};        // inner rows 0-7, 8-15: odd and even a
    uint32_t fo[2] = {0, 0}, fe[2] = {0, 0};        // y and z faces' rows
#pragma unroll
    for (int c = -1; c <= 4; ++c) {
#pragma unroll
        for (int b = -1; b <= 4; ++b) {
            const bool yin = b >= 0 && b < 4, zin = c >= 0 && c < 4;
            if (!yin && !zin) continue;
            const uint8_t *row = sp + zo[c + 1] + yo[b + 1];
            const uint32_t vo = row_bytes(row + (((1 + b + c) & 1) ? P.half : 0), odd);
            const uint32_t ve = row_bytes(row + (((b + c) & 1) ? P.half : 0), even);
            if (yin && zin) {
                const int k = b + 4 * c;
                io[k >> 3] += vo << (k & 7);
                ie[k >> 3] += ve << (k & 7);
            } else {
                const int f = yin ? 1 : 0, k = yin ? b + (c < 0 ? 0 : 4) : c + (b < 0 ? 0 : 4);
                fo[f] += vo << k;
                fe[f] += ve << k;
            }
        }
    }
    // odd bytes: a = -1, 1, 3; even bytes: a = 0, 2, 4
    const uint32_t am = __byte_perm(io[0], io[1], 0x40) & 0xFFFFu, a1 = __byte_perm(io[0], io[1], 0x51) & 0xFFFFu,
                   a3 = __byte_perm(io[0], io[1], 0x62) & 0xFFFFu, a0 = __byte_perm(ie[0], ie[1], 0x40) & 0xFFFFu,
                   a2 = __byte_perm(ie[0], ie[1], 0x51) & 0xFFFFu, a4 = __byte_perm(ie[0], ie[1], 0x62) & 0xFFFFu;
    uint32_t word[5];
    word[0] = am | (a4 << 16);
#pragma unroll
    for (int f = 0; f < 2; ++f)
        word[1 + f] = face_bits(fe[f], 0) | (face_bits(fo[f], 1) << 1) | (face_bits(fe[f], 1) << 2) |
                      (face_bits(fo[f], 2) << 3);
    word[3] = class_bits(a0, a2, a1, a3, kEvenRows);
    word[4] = class_bits(a0, a2, a1, a3, ~kEvenRows & 0xFFFFu);
#pragma unroll
    for (int k = 0; k < 5; ++k) P.bits[(size_t)k * P.n + w] = word[k];
}

// All threads of group g agree (barrier 1 + g; 0 is __syncthreads).
__device__ __forceinline__ void group_sync(int g) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(kThreads) : "memory");
}
__device__ __forceinline__ bool group_and(int g, bool v) {
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\t"
                 "selp.s32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((int)v), "r"(1 + g), "n"(kThreads) : "memory");
    return r != 0;
}

// The network on tiles of 128 rows: thread p of a group writes its input row (lattice mode:
// boundary spins from the gathered bits, 4 beta J) into the group's A tile, then three tcgen05
// layers, TMEM lane p = row p; logits to Z.  A layer is a chain (tile in shared memory, MMA,
// TMEM to registers and back), so the time is latency: four groups share one copy of the weights
// and keep 16 warps on the SM (two CTAs with a copy each keep 8; 524288 patches: 90 -> 71 us),
// and a group loads its next 32 columns from TMEM while it works on these (-> 65 us).
template <int MODE>  // 0: lattice patches, 1: network forward on X
__global__ void __launch_bounds__(kGroups * kThreads, 1) patch_kernel(const PatchParams P) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float *bias = reinterpret_cast<float *>(base + SM_BIAS);  // b1[128], b2[128], b3[32]
    uint64_t *bar = reinterpret_cast<uint64_t *>(base + SM_BAR);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(base + SM_BAR + 8 * kGroups);
    const int group = threadIdx.x >> 7, tid = threadIdx.x & 127, warp = tid >> 5;
    bar += group;
    after_release();

    // weights and biases into shared memory (plain 16-byte copies; the image is pre-swizzled)
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(P.img);
        uint4 *dw = reinterpret_cast<uint4 *>(base);
        constexpr int nw = IMG_B1 / 16, nt = kGroups * kThreads;  // 4608 = 9 x 512
        uint4 v[nw / nt];
#pragma unroll
        for (int u = 0; u < nw / nt; ++u) v[u] = __ldg(src + u * nt + threadIdx.x);
#pragma unroll
        for (int u = 0; u < nw / nt; ++u) dw[u * nt + threadIdx.x] = v[u];
        uint4 *db = reinterpret_cast<uint4 *>(base + SM_BIAS);
        for (int i = threadIdx.x; i < (IMG_BYTES - IMG_B1) / 16; i += nt) db[i] = src[nw + i];
    }
    if (tid == 0) {  // a barrier per group
        tc::mbar_init(tc::smem_u32(bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc::smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tmem_slot + 128u * (uint32_t)group;
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    const uint32_t sA = tc::smem_u32(base + SM_A + group * 32768);
    const uint32_t sW1 = tc::smem_u32(base + IMG_W1), sW2 = tc::smem_u32(base + IMG_W2),
                   sW3 = tc::smem_u32(base + IMG_W3);
    uint8_t *arow = base + SM_A + group * 32768;
    uint32_t phase = 0;
    bool ok = true;

    after_wait();  // the gathered bits
    const int ntiles = (P.n + kThreads - 1) / kThreads;
    for (int tile = blockIdx.x + group * gridDim.x; tile < ntiles && ok; tile += kGroups * gridDim.x) {
        const int w = tile * kThreads + tid;
        const bool valid = w < P.n;
        // ------------------------------------------------------------- input row ---------
        uint32_t bw[4] = {0u, 0u, 0u, 0u};  // boundary bits; the last word stays zero
        float k4 = 0.f;
        if (MODE == 0 && valid) {
#pragma unroll
            for (int k = 0; k < 3; ++k) bw[k] = P.bits[(size_t)k * P.n + w];
            k4 = P.k4[P.slot_of_rep[P.r0 + (int)fdiv((uint32_t)w, P.fPc)]];
        }
#pragma unroll
        for (int ch = 0; ch < 16; ++ch) {
            uint32_t pk4[4] = {0u, 0u, 0u, 0u};
            if (MODE == 1) {
                if (valid) {
                    const uint4 v = reinterpret_cast<const uint4 *>(P.X + (size_t)w * NI)[ch];
                    pk4[0] = v.x; pk4[1] = v.y; pk4[2] = v.z; pk4[3] = v.w;
                }
            } else if (valid) {
                if (ch < 12) {  // BF16 1.0 or -1.0 (sign bit from the complement of the spin)
                    const uint32_t nb = ~(bw[ch >> 2] >> (8 * (ch & 3)));
#pragma unroll
                    for (int h = 0; h < 4; ++h)
                        pk4[h] = 0x3F803F80u | ((nb << (15 - 2 * h)) & 0x8000u) | ((nb << (30 - 2 * h)) & 0x80000000u);
                } else if (ch == 12) {
                    const __nv_bfloat162 bv = __floats2bfloat162_rn(k4, 0.f);
                    pk4[0] = *reinterpret_cast<const uint32_t *>(&bv);
                }
            }
            const int k = ch * 8;
            uint8_t *dst = arow + (k >> 6) * 16384 + tc::swz(tid, k & 63);
            *reinterpret_cast<uint4 *>(dst) = make_uint4(pk4[0], pk4[1], pk4[2], pk4[3]);
        }
        // ---------------------------------------------------------------- layers -------
        float z[32];
#pragma unroll 1
        for (int layer = 0; layer < 3 && ok; ++layer) {
            tc::fence_proxy_async();
            tc::fence_before();
            group_sync(group);
            if (tid == 0) {
                tc::fence_after();
                const int n = layer == 2 ? NO : NH;
                const uint32_t idesc = tc::make_idesc(128, n);
                const uint32_t sw = layer == 0 ? sW1 : (layer == 1 ? sW2 : sW3);
                const uint32_t wtile = (uint32_t)n * 128u;  // bytes of one 64-column tile of W
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    const uint32_t ao_ = (uint32_t)(kk >> 2) * 16384u + (uint32_t)(kk & 3) * 32u;
                    const uint32_t bo_ = (uint32_t)(kk >> 2) * wtile + (uint32_t)(kk & 3) * 32u;
                    tc::umma(tmem, tc::make_desc(sA + ao_), tc::make_desc(sw + bo_), idesc, kk > 0 ? 1u : 0u);
                }
                tc::umma_commit(tc::smem_u32(bar));
            }
            const bool got = tc::mbar_wait(tc::smem_u32(bar), phase, P.err, 1);
            phase ^= 1u;
            ok = group_and(group, got);
            if (!ok) break;
            tc::fence_after();
            if (layer < 2) {
                // bias, ReLU, BF16, back into the A tile as the next layer's input
                const float *bl = bias + layer * 128;
                uint32_t v2[2][32];  // the next 32 columns come while these are worked on
                tc::tmem_ld32(lane_base, v2[0]);
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    uint32_t(&v)[32] = v2[cc & 1];
                    tc::tmem_wait_ld(v);
                    if (cc < 3) tc::tmem_ld32(lane_base + 32u * (cc + 1), v2[(cc + 1) & 1]);
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        uint32_t pk4[4];
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            const int c0 = 8 * g + 2 * h;
                            const float a0 = fmaxf(__uint_as_float(v[c0]) + bl[32 * cc + c0], 0.0f);
                            const float a1 = fmaxf(__uint_as_float(v[c0 + 1]) + bl[32 * cc + c0 + 1], 0.0f);
                            const __nv_bfloat162 bv = __floats2bfloat162_rn(a0, a1);
                            pk4[h] = *reinterpret_cast<const uint32_t *>(&bv);
                        }
                        const int k = 32 * cc + 8 * g;
                        uint8_t *dst = arow + (k >> 6) * 16384 + tc::swz(tid, k & 63);
                        *reinterpret_cast<uint4 *>(dst) = make_uint4(pk4[0], pk4[1], pk4[2], pk4[3]);
                    }
                }
            } else {
                uint32_t v[32];
                tc::tmem_ld32(lane_base, v);
                tc::tmem_wait_ld();
#pragma unroll
                for (int k = 0; k < 32; ++k) z[k] = __uint_as_float(v[k]) + bias[256 + k];
            }
        }
        if (!ok) break;
        tc::fence_before();  // TMEM reads done before the next tile's MMAs (barrier at its layer 0)
        if (!valid) continue;
        float4 *zo = reinterpret_cast<float4 *>(P.Z) + (MODE == 0 ? (size_t)w : (size_t)w * 8);
        const size_t zs = MODE == 0 ? (size_t)P.n : 1;
#pragma unroll
        for (int k = 0; k < 8; ++k) zo[k * zs] = make_float4(z[4 * k], z[4 * k + 1], z[4 * k + 2], z[4 * k + 3]);
        if (MODE == 0 && P.dump) {
            float4 *dp = reinterpret_cast<float4 *>(P.dump + (size_t)w * NO);
#pragma unroll
            for (int k = 0; k < 8; ++k) dp[k] = make_float4(z[4 * k], z[4 * k + 1], z[4 * k + 2], z[4 * k + 3]);
        }
    }
    tc::fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc::fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

// ------------------------------------------------------ Metropolis-Hastings by bit masks ----
// The sites of a parity class of a patch are the bits 2 (b + 4 c) + (a >> 1) of a word, and with
// p = (b + c) & 1 a row holds the A-sites a = p, p + 2 and the B-sites a = 1 - p, 3 - p.  So the
// neighbours of all 32 sites of a class in one direction are a word: in x the other class's word
// (rows of one parity) or that word moved by one bit (the others), in y moved by a row (2 bits),
// in z by a plane (8 bits), with the boundary's faces where the patch ends.
constexpr uint32_t rows_with(int parity) {  // bits of the rows with (b + c) & 1 == parity
    uint32_t m = 0;
    for (int row = 0; row < 16; ++row)
        if ((((row & 3) + (row >> 2)) & 1) == parity) m |= 3u << (2 * row);
    return m;
}
constexpr uint32_t kOdd = rows_with(1), kEven = rows_with(0), kBit0 = 0x55555555u, kBit1 = 0xAAAAAAAAu;
constexpr uint32_t kY0 = 0x03030303u, kY3 = 0xC0C0C0C0u, kZ0 = 0x000000FFu, kZ3 = 0xFF000000u;

// A y or z face (bits a + 4 u, u = c or b) to the sites of class cl (0 A, 1 B): of the four bits
// of row u the two with a & 1 == (u + edge + cl) & 1 (edge: the face's b or c, 0 or 3), at bits
// 2 u + (a >> 1) of the result.
__device__ __forceinline__ uint32_t pick(uint32_t face, int odd_first) {
    // bits a = 0, 2 (even) or 1, 3 (odd) of each nibble, alternating over the nibbles
    const uint32_t even = face & 0x5555u, odd = (face >> 1) & 0x5555u;
    uint32_t x = odd_first ? (odd & 0x0F0Fu) | (even & 0xF0F0u) : (even & 0x0F0Fu) | (odd & 0xF0F0u);
    // x: nibble u holds the two bits at 0 and 2; bring them to 0 and 1, nibbles to pairs
    x = (x | (x >> 1)) & 0x3333u;
    x = (x | (x >> 2)) & 0x0F0Fu;
    return (x | (x >> 4)) & 0x00FFu;
}
// The eight pairs of bits of `pairs` (2 bits per row u) to the y faces: rows b = 0 (at = 0) or 3.
__device__ __forceinline__ uint32_t to_y(uint32_t pairs, int at) {
    const uint32_t x = (pairs | (pairs << 12)) & 0x000F000Fu;   // u = 0, 1 | u = 2, 3
    return ((x | (x << 6)) & 0x03030303u) << at;                // one pair per plane
}

// Boundary neighbours of one class's sites per direction, where there are any (mask m).
struct Faces {
    uint32_t w[6];
};
template <int CL>
__device__ __forceinline__ Faces class_faces(uint32_t f0, uint32_t f1, uint32_t f2) {
    // x: bnd bits 0-15 face a = -1 (row order), 16-31 face a = 4; the site next to a = -1 is bit
    // 0 of its row where the class has a = 0 there (A: even rows, B: odd rows), the one next to
    // a = 4 bit 1 where it has a = 3 (A: odd rows, B: even rows)
    Faces F;
    F.w[0] = spread(f0 & 0xFFFFu) & (CL ? kOdd : kEven);
    F.w[1] = (spread(f0 >> 16) << 1) & (CL ? kEven : kOdd);
    // y faces b = 0, 3: plane c, bits a + 4 c; class CL has a & 1 == (b + c + CL) & 1
    F.w[2] = to_y(pick(f1 & 0xFFFFu, CL), 0);
    F.w[3] = to_y(pick(f1 >> 16, CL ^ 1), 6);
    // z faces c = 0, 3: row b, bits a + 4 b
    F.w[4] = pick(f2 & 0xFFFFu, CL);
    F.w[5] = pick(f2 >> 16, CL ^ 1) << 24;
    return F;
}
__host__ __device__ constexpr uint32_t face_mask(int cl, int q) {
    return q == 0 ? kBit0 & (cl ? kOdd : kEven) : q == 1 ? kBit1 & (cl ? kEven : kOdd)
         : q == 2 ? kY0 : q == 3 ? kY3 : q == 4 ? kZ0 : kZ3;
}
// Up neighbours of the 32 B-sites as three bit planes, from the A-sites and the faces.
struct Planes {
    uint32_t n0, n1, n2;
};
__device__ __forceinline__ Planes b_neighbours(uint32_t A, const Faces &F) {
    const uint32_t q0 = (A & kEven) | ((A << 1) & kBit1 & kOdd) | F.w[0];
    const uint32_t q1 = (A & kOdd) | ((A >> 1) & kBit0 & kEven) | F.w[1];
    const uint32_t q2 = ((A << 2) & ~kY0) | F.w[2], q3 = ((A >> 2) & ~kY3) | F.w[3];
    const uint32_t q4 = (A << 8) | F.w[4], q5 = (A >> 8) | F.w[5];
    const uint32_t s0 = q0 ^ q1 ^ q2, c0 = (q0 & q1) | (q2 & (q0 ^ q1));
    const uint32_t s1 = q3 ^ q4 ^ q5, c1 = (q3 & q4) | (q5 & (q3 ^ q4));
    const uint32_t k = s0 & s1;
    return Planes{s0 ^ s1, c0 ^ c1 ^ k, (c0 & c1) | (k & (c0 ^ c1))};
}
// Sum over the B-sites of s (2 n - 6), s = +-1 from the bits of S.
__device__ __forceinline__ int bond_sum(uint32_t S, const Planes &n) {
    const int up = __popc(n.n0 & S) + 2 * __popc(n.n1 & S) + 4 * __popc(n.n2 & S);
    const int all = __popc(n.n0) + 2 * __popc(n.n1) + 4 * __popc(n.n2);
    return 2 * (2 * up - all) - 6 * (2 * __popc(S) - 32);
}
// Sum over the A-sites' boundary bonds of s_i s_j.
__device__ __forceinline__ int edge_sum(uint32_t A, const Faces &F) {
    int same = 0;
#pragma unroll
    for (int q = 0; q < 6; ++q) same += __popc(~(A ^ F.w[q]) & face_mask(0, q));
    return 2 * same - 48;  // 48 boundary bonds
}

// 17 Philox blocks, 32 sigmoids and 64 table rows per patch: instruction issue bounds it (524288
// patches 73 us; with a loop over six neighbours per site, the loops unrolled and each thread
// writing its own accepted patch 115 us).
// One thread per patch: proposal from the logits, heat bath of the B-sites, acceptance.
// d = log q(new) - log q(old): A-sites that changed add +-z_k (log-odds), then the B-sites'
// heat-bath log probabilities (tables); log alpha = (0 - d) - beta J dB.
__global__ void __launch_bounds__(128, 8) mh_kernel(const PatchParams P) {
    after_release();
    after_wait();
    if (*P.err) return;  // a network pass that gave up leaves the state as it was
    const bool valid = blockIdx.x * 128 + threadIdx.x < P.n;
    const int w = valid ? blockIdx.x * 128 + threadIdx.x : P.n - 1;
    const Patch D = decode(P, w);
    const uint32_t f0 = P.bits[w], f1 = P.bits[(size_t)P.n + w], f2 = P.bits[2 * (size_t)P.n + w];
    const uint32_t ao = P.bits[3 * (size_t)P.n + w], bo = P.bits[4 * (size_t)P.n + w];
    const int slot = P.slot_of_rep[D.r];
    const uint4 *HB = P.HB + 7 * slot;
    const float4 *z4 = reinterpret_cast<const float4 *>(P.Z) + w;
    uint32_t an = 0, bn = 0;
    float d = 0.0f;
    // loops of four sites stay rolled: unrolled, the kernel waits on its own instructions
    float4 z = z4[0];
#pragma unroll 1
    for (int k4 = 0; k4 < 8; ++k4) {
        const float4 zn = k4 < 7 ? z4[(size_t)(k4 + 1) * P.n] : z;
        const U4 rw = draw_rk(D.pidx, D.t, D.stream, kLearn | ((uint32_t)k4 << 16), P.K);
        const float zs[4] = {z.x, z.y, z.z, z.w};
        const uint32_t us[4] = {rw.x, rw.y, rw.z, rw.w};
        const uint32_t old = ao >> (4 * k4);
        uint32_t nib = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool up = us[j] < thr_of_logit(zs[j]);
            nib |= (up ? 1u : 0u) << j;
            if (up != (((old >> j) & 1u) != 0)) d += up ? zs[j] : -zs[j];
        }
        an |= nib << (4 * k4);
        z = zn;
    }
    const Faces FB = class_faces<1>(f0, f1, f2);
    const Planes nn = b_neighbours(an, FB), no = b_neighbours(ao, FB);
    Planes sn = nn, so = no;
#pragma unroll 1
    for (int m4 = 0; m4 < 8; ++m4) {
        const U4 rw = draw_rk(D.pidx, D.t, D.stream, kLearn | ((uint32_t)(8 + m4) << 16), P.K);
        const uint32_t us[4] = {rw.x, rw.y, rw.z, rw.w};
        const uint32_t old = bo >> (4 * m4);
        uint32_t nib = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t qn = ((sn.n0 >> j) & 1u) | (((sn.n1 >> j) & 1u) << 1) | (((sn.n2 >> j) & 1u) << 2);
            const uint32_t qo = ((so.n0 >> j) & 1u) | (((so.n1 >> j) & 1u) << 1) | (((so.n2 >> j) & 1u) << 2);
            const uint4 hn = HB[qn], ho = HB[qo];
            const bool up = us[j] < hn.x;
            nib |= (up ? 1u : 0u) << j;
            d += __uint_as_float(up ? hn.y : hn.z) - __uint_as_float(((old >> j) & 1u) ? ho.y : ho.z);
        }
        bn |= nib << (4 * m4);
        sn.n0 >>= 4; sn.n1 >>= 4; sn.n2 >>= 4;
        so.n0 >>= 4; so.n1 >>= 4; so.n2 >>= 4;
    }
    const Faces FA = class_faces<0>(f0, f1, f2);
    const int bond_n = bond_sum(bn, nn) + edge_sum(an, FA), bond_o = bond_sum(bo, no) + edge_sum(ao, FA);
    const U4 ra = draw_rk(D.pidx, D.t, D.stream, kLearn | (16u << 16), P.K);
    const float la = (0.0f - d) - P.betaJf[slot] * (float)(bond_n - bond_o);
    bool acc = la >= 0.0f;
    if (!acc) acc = u01(ra.x) < expf_neg(la);
    acc = acc && valid;
    if (acc) atomicAdd(P.acc + D.r, 1ull);
    // An accepted patch is written by its warp, two sites per lane (by its own thread it costs
    // the warp the longest lane's number of changed sites).
    const int lane = threadIdx.x & 31;
    const uint32_t e0 = c_site[lane], e1 = c_site[32 + lane];
    for (uint32_t m = __ballot_sync(0xffffffffu, acc); m; m &= m - 1) {
        const int src = __ffs((int)m) - 1;
        const uint32_t ca = __shfl_sync(0xffffffffu, an ^ ao, src), cb = __shfl_sync(0xffffffffu, bn ^ bo, src);
        const uint32_t va = __shfl_sync(0xffffffffu, an, src), vb = __shfl_sync(0xffffffffu, bn, src);
        const int o0 = __shfl_sync(0xffffffffu, D.o0, src), o1 = __shfl_sync(0xffffffffu, D.o1, src);
        const int o2 = __shfl_sync(0xffffffffu, D.o2, src);
        uint8_t *sp = P.spins + (long long)__shfl_sync(0xffffffffu, D.r, src) * 2 * P.half;
        const int par = (o0 + o1 + o2) & 1;
        if ((ca >> lane) & 1u)
            sp[site_addr(P, o0, o1, o2, par, e0 & 3, (e0 >> 2) & 3, e0 >> 4)] = (uint8_t)((va >> lane) & 1u);
        if ((cb >> lane) & 1u)
            sp[site_addr(P, o0, o1, o2, par, e1 & 3, (e1 >> 2) & 3, e1 >> 4)] = (uint8_t)((vb >> lane) & 1u);
    }
}

// ------------------------------------------------------------------ training data ----
// n samples per replica: a random offset and patch, its network input (BF16) and A-site bits.
__global__ void collect_kernel(const uint8_t *__restrict__ spins, int L1, int L2, int L3, int H,
                               long long half, int R, int per_rep, const uint32_t *__restrict__ stream_id,
                               const int32_t *__restrict__ slot_of_rep, const float *__restrict__ k4,
                               uint32_t seed, uint32_t call, __nv_bfloat16 *__restrict__ X,
                               uint32_t *__restrict__ Y, long long write0, long long cap) {
    const long long total = (long long)R * per_rep;
    for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < total;
         w += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(w / per_rep), s = (int)(w - (long long)r * per_rep);
        const U4 d = draw((uint32_t)s, call, stream_id[r], kLearn | (0xFEu << 8), seed);
        const int ox = (int)(d.x & 3u), oy = (int)((d.x >> 2) & 3u), oz = (int)((d.x >> 4) & 3u);
        const int par = (ox + oy + oz) & 1;
        const int o0 = 4 * (int)(d.y % (uint32_t)(L1 / 4)) + ox;
        const int o1 = 4 * (int)(d.z % (uint32_t)(L2 / 4)) + oy;
        const int o2 = 4 * (int)(d.w % (uint32_t)(L3 / 4)) + oz;
        const uint8_t *sp = spins + (long long)r * 2 * half;
        PatchParams P;
        P.L1 = L1; P.L2 = L2; P.L3 = L3; P.H = H; P.half = half;
        const long long row = (write0 + w) % cap;
        __nv_bfloat16 *xr = X + (size_t)row * NI;
        for (int i = 0; i < 96; ++i) {
            const uint16_t e = c_bnd[i];
            const int a = (int)(e & 15u) - 1, b = (int)((e >> 4) & 15u) - 1, c = (int)(e >> 8) - 1;
            xr[i] = __float2bfloat16_rn(sp[site_addr(P, o0, o1, o2, par, a, b, c)] ? 1.0f : -1.0f);
        }
        xr[96] = __float2bfloat16_rn(k4[slot_of_rep[r]]);
        for (int i = 97; i < NI; ++i) xr[i] = __float2bfloat16_rn(0.0f);
        uint32_t ab = 0;
        for (int k = 0; k < 32; ++k) {
            const uint8_t e = c_site[k];
            ab |= (uint32_t)sp[site_addr(P, o0, o1, o2, par, e & 3, (e >> 2) & 3, e >> 4)] << k;
        }
        Y[row] = ab;
    }
}

// inference image: quantised weights as BF16 in the swizzled K-major tiles, biases FP32
__global__ void pack_kernel(const float *__restrict__ q, uint8_t *__restrict__ img) {
    const int total = NH * NI + NH * NH + NO * NH;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        int base, rows, off, idx = e;
        if (idx < NH * NI) { base = IMG_W1; rows = NH; off = OFF_W1; }
        else if ((idx -= NH * NI) < NH * NH) { base = IMG_W2; rows = NH; off = OFF_W2; }
        else { idx -= NH * NH; base = IMG_W3; rows = NO; off = OFF_W3; }
        const int n = idx / NI, k = idx % NI;
        const uint32_t o = (uint32_t)base + (uint32_t)(k >> 6) * (uint32_t)(rows * 128) + tc::swz(n, k & 63);
        *reinterpret_cast<__nv_bfloat16 *>(img + o) = __float2bfloat16_rn(q[off + idx]);
    }
    float *bf = reinterpret_cast<float *>(img + IMG_B1);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NH + NH + NO; i += gridDim.x * blockDim.x)
        bf[i] = i < NH ? q[OFF_B1 + i] : (i < 2 * NH ? q[OFF_B2 + i - NH] : q[OFF_B3 + i - 2 * NH]);
}

__global__ void advance_lstep_kernel(uint32_t *c, int R) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < R) c[r] += 1u;
}

static bool closed_forms_agree(const Geometry &g) {
    for (int m = 0; m < 32; ++m) {
        for (int q = 0; q < 6; ++q)
            if (geo_bn(m, q) != g.Bn[m][q]) return false;
        int n = 0;
        for (int q = 0; q < 6; ++q) {
            const int bi = geo_ab(m, q);
            if (bi >= 0 && (n >= 3 || g.Ab[m][n++] != bi)) return false;
        }
        if (n < 3 && g.Ab[m][n] != -1) return false;
        if ((g.site[m] & 3) != geo_a_a(m) || (g.site[32 + m] & 3) != geo_b_a(m)) return false;
    }
    return true;
}

}  // namespace learn
}  // namespace ether

using namespace ether;
using namespace ether::learn;

struct ether_learn {
    ether_ctx *ctx = nullptr;
    learn::XyzLearn *xyz = nullptr;  // an XYZ context's learner (k_learn_xyz.cu); the rest unused
    uint32_t seed = 0;
    int R = 0, L[3] = {0, 0, 0}, P[3] = {0, 0, 0};
    long long Pc = 0, half = 0;
    double J = 0.0;
    // parameters (device): master, quantised, gradient, Adam moments; inference image
    float *p = nullptr, *pq = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    uint8_t *img = nullptr;
    int adam_t = 0;
    // data set
    __nv_bfloat16 *X = nullptr;
    uint32_t *Y = nullptr;
    long long cap = 0, n = 0, write = 0;
    uint32_t collect_calls = 0;
    TrainBuffers tb;               // training scratch
    uint32_t *wp = nullptr;        // packed weights of the training kernels
    double *loss = nullptr;
    // sweeps: a pass of up to `rows` patches
    long long rows = 0;
    uint32_t *bits = nullptr;
    float *Zp = nullptr;
    uint32_t *lstep = nullptr;
    float *k4 = nullptr, *betaJf = nullptr;
    uint4 *HB = nullptr;
    unsigned long long *acc = nullptr;
    float *dump = nullptr;
    bool dump_on = false;
    std::vector<double> tables_for;  // beta slots the tables were built for
    int *err = nullptr;
    int sm_count = 0;
    uint64_t launches = 0, proposed = 0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    float sweep_ms = 0.f, train_ms = 0.f;
    int timed = 0;  // 1: sweep, 2: train pending in e0/e1
    int timed_n = 0;
};

namespace {

int lfail(int code, const std::string &msg) {
    set_error(msg);
    return code;
}

#define LCUDA(expr)                                                                          \
    do {                                                                                     \
        cudaError_t _e = (expr);                                                             \
        if (_e != cudaSuccess)                                                               \
            return lfail(_e == cudaErrorMemoryAllocation ? ETHER_ERR_NOMEM : ETHER_ERR_CUDA,  \
                         std::string(#expr) + ": " + cudaGetErrorString(_e));                \
    } while (0)

bool g_geometry_uploaded = false;

int upload_geometry() {
    if (g_geometry_uploaded) return ETHER_OK;
    const Geometry g = make_geometry();
    if (!closed_forms_agree(g)) return lfail(ETHER_ERR_CUDA, "learned proposal: inconsistent patch geometry");
    LCUDA(cudaMemcpyToSymbol(c_site, g.site, sizeof g.site));
    LCUDA(cudaMemcpyToSymbol(c_bnd, g.bnd, sizeof g.bnd));
    g_geometry_uploaded = true;
    return ETHER_OK;
}

float bf16_host(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    u += 0x7FFFu + ((u >> 16) & 1u);
    u &= 0xFFFF0000u;
    std::memcpy(&f, &u, 4);
    return f;
}

// Per temperature slot: 4 beta J (BF16-exact), beta J (FP32), heat-bath thresholds and logs.
int refresh_tables(ether_learn &l) {
    const Ctx &c = l.ctx->c;
    if (l.tables_for == c.beta_slots) return ETHER_OK;
    const int S = c.n_slots;
    std::vector<float> k4(S), bj(S);
    std::vector<uint4> hb(7 * S);
    for (int s = 0; s < S; ++s) {
        const double betaJ = c.beta_slots[s] * l.J;
        k4[s] = bf16_host((float)(4.0 * betaJ));
        bj[s] = (float)betaJ;
        for (int qi = 0; qi < 7; ++qi) {
            const int nsum = 2 * qi - 6;
            const double pu = 1.0 / (1.0 + std::exp(2.0 * betaJ * nsum));
            double t = std::floor(pu * 4294967296.0 + 0.5);
            t = std::min(std::max(t, 1.0), 4294967295.0);
            const float up = (float)std::log(t / 4294967296.0);
            const float dn = (float)std::log((4294967296.0 - t) / 4294967296.0);
            uint4 &h = hb[7 * s + qi];
            h = make_uint4((uint32_t)t, 0u, 0u, 0u);
            std::memcpy(&h.y, &up, 4);
            std::memcpy(&h.z, &dn, 4);
        }
    }
    cudaFree(l.k4); cudaFree(l.betaJf); cudaFree(l.HB);
    l.k4 = l.betaJf = nullptr;
    l.HB = nullptr;
    LCUDA(cudaMalloc((void **)&l.k4, S * sizeof(float)));
    LCUDA(cudaMalloc((void **)&l.betaJf, S * sizeof(float)));
    LCUDA(cudaMalloc((void **)&l.HB, 7 * S * sizeof(uint4)));
    LCUDA(cudaMemcpy(l.k4, k4.data(), S * sizeof(float), cudaMemcpyHostToDevice));
    LCUDA(cudaMemcpy(l.betaJf, bj.data(), S * sizeof(float), cudaMemcpyHostToDevice));
    LCUDA(cudaMemcpy(l.HB, hb.data(), 7 * S * sizeof(uint4), cudaMemcpyHostToDevice));
    l.tables_for = c.beta_slots;
    return ETHER_OK;
}

using Net = TrainNet<NI, NO>;
static_assert(Net::N == NPARAM && Net::W2 == OFF_W2 && Net::W3 == OFF_W3, "parameter layout");

TrainParams train_params(ether_learn &l) { return TrainParams{l.p, l.g, l.m, l.v, l.pq, l.wp, l.loss}; }

// The inference image of the rounded parameters.
int pack_image(ether_learn &l, cudaStream_t st) {
    pack_kernel<<<64, 256, 0, st>>>(l.pq, l.img);
    l.launches++;
    LCUDA(cudaGetLastError());
    return ETHER_OK;
}

int quantise_and_pack(ether_learn &l, cudaStream_t st) {
    LCUDA((train_pack<NI, NO>(train_params(l), st)));
    l.launches++;
    return pack_image(l, st);
}

int read_err(ether_learn &l) {
    int e = 0;
    LCUDA(cudaMemcpy(&e, l.err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) {
        cudaMemset(l.err, 0, sizeof(int));
        return lfail(ETHER_ERR_TIMEOUT, "learned-proposal kernel: a bounded tensor-core wait ran out (code " +
                                            std::to_string(e) + ")");
    }
    return ETHER_OK;
}

// One class of a learned sweep, in passes of whole replicas.
int launch_patches(ether_learn &l, int cls, float *dump) {
    Ctx &c = l.ctx->c;
    PatchParams P;
    std::memset(&P, 0, sizeof(P));
    P.img = l.img;
    P.err = l.err;
    P.spins = c.spins;
    P.L1 = l.L[0]; P.L2 = l.L[1]; P.L3 = l.L[2]; P.H = l.L[0] / 2;
    P.half = l.half;
    P.P1 = l.P[0]; P.P2 = l.P[1]; P.P3 = l.P[2];
    P.cls = cls;
    P.fPc = make_fastdiv((uint32_t)l.Pc);
    P.fhalf1 = make_fastdiv((uint32_t)(l.P[0] / 2));
    P.fP2 = make_fastdiv((uint32_t)l.P[1]);
    P.stream_id = c.stream_id;
    P.lstep = l.lstep;
    P.slot_of_rep = c.slot_of_rep;
    P.k4 = l.k4; P.betaJf = l.betaJf; P.HB = l.HB;
    P.K = round_keys(c.seed);
    P.acc = l.acc;
    P.bits = l.bits;
    P.Z = l.Zp;
    const int per = (int)std::max<long long>(1, std::min<long long>(l.R, l.rows / l.Pc));
    for (int r0 = 0; r0 < l.R; r0 += per) {
        P.r0 = r0;
        P.n = std::min(per, l.R - r0) * (int)l.Pc;
        P.dump = dump ? dump + (size_t)r0 * l.Pc * NO : nullptr;
        const int tiles = (P.n + kThreads - 1) / kThreads;
        LCUDA(launch_after(gather_kernel, (P.n + 255) / 256, 256, 0, c.stream, true, P));
        LCUDA(launch_after(patch_kernel<0>, std::min(tiles, l.sm_count), kGroups * kThreads, SM_BYTES + 1024, c.stream, true, P));
        // mh_kernel follows closely only where an SM is free for each of its blocks: the network's
        // blocks fill an SM's registers, so blocks that start beside them crowd on the few SMs left
        // and stay there (a class of 32^3 x 64, 128 tiles: 37 us closely, 25 so; x 100 38 and 27;
        // 64^3 x 32 45 and 36; 16^3 x 16, four tiles, 21 and 23)
        LCUDA(launch_after(mh_kernel, (P.n + 127) / 128, 128, 0, c.stream, 2 * tiles <= l.sm_count, P));
        l.launches += 3;
    }
    LCUDA(cudaGetLastError());
    return ETHER_OK;
}

}  // namespace

extern "C" int ether_learn_create(ether_ctx *h, const ether_learn_desc *d, ether_learn **out) {
    if (!out) return lfail(ETHER_ERR_ARG, "null output handle");
    *out = nullptr;
    if (!h || !d) return lfail(ETHER_ERR_ARG, "null context or descriptor");
    Ctx &c = h->c;
    if (d->patch != 4 || d->hidden != 128)
        return lfail(ETHER_ERR_UNSUPPORTED, "learned proposal: patch 4 and hidden width 128 only");
    if (c.model == ETHER_MODEL_XYZ) {
        learn::XyzLearn *x = nullptr;
        const int rc = learn::xyz_create(h, d, &x);
        if (rc) return rc;
        ether_learn *l = new ether_learn();
        l->ctx = h;
        l->xyz = x;
        *out = l;
        return ETHER_OK;
    }
    // c.L is set once the lattice is verified to be the periodic simple-cubic one (whose
    // storage is the checkerboard split the kernels address arithmetically)
    if (c.model != ETHER_MODEL_ISING || c.L[0] <= 0 || c.nsp != 1 || c.nsh != 1 || c.zeeman)
        return lfail(ETHER_ERR_UNSUPPORTED, "learned proposal: simple-cubic Ising, one species, one shell, no Zeeman term");
    if (c.L[0] % 8 || c.L[1] % 8 || c.L[2] % 8 || c.L[0] > 1016 || c.L[1] > 1016 || c.L[2] > 1016)
        return lfail(ETHER_ERR_UNSUPPORTED, "learned proposal: every extent a multiple of 8, at most 1016");
    if (d->capacity < 1024) return lfail(ETHER_ERR_ARG, "training capacity below 1024 samples");
    int rc = upload_geometry();
    if (rc) return rc;
    ether_learn *l = new ether_learn();
    l->ctx = h;
    l->seed = d->seed;
    l->R = c.R;
    for (int a = 0; a < 3; ++a) {
        l->L[a] = c.L[a];
        l->P[a] = c.L[a] / 4;
    }
    l->Pc = (long long)l->P[0] * l->P[1] * l->P[2] / 2;
    l->half = (long long)(c.L[0] / 2) * c.L[1] * c.L[2];
    l->J = c.h_Jd[2];
    l->cap = d->capacity;
    auto fail_free = [&](cudaError_t e) {
        ether_learn_destroy(l);
        return lfail(e == cudaErrorMemoryAllocation ? ETHER_ERR_NOMEM : ETHER_ERR_CUDA,
                     std::string("learned proposal set-up: ") + cudaGetErrorString(e));
    };
    cudaError_t e = cudaSuccess;
    int dev = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&l->sm_count, cudaDevAttrMultiProcessorCount, dev);
    float **pb[] = {&l->p, &l->pq, &l->g, &l->m, &l->v};
    for (float **b : pb)
        if (e == cudaSuccess) e = cudaMalloc((void **)b, NPARAM * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->img, IMG_BYTES);
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->wp, Net::WORDS * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->X, (size_t)l->cap * NI * sizeof(__nv_bfloat16));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->Y, (size_t)l->cap * sizeof(uint32_t));
    l->rows = std::max<long long>(l->Pc, std::min<long long>((long long)l->R * l->Pc, kPassPatches));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->bits, 5 * (size_t)l->rows * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->Zp, (size_t)l->rows * NO * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->loss, sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->lstep, l->R * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->acc, l->R * sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMalloc((void **)&l->err, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(l->lstep, 0, l->R * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(l->acc, 0, l->R * sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(l->err, 0, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(l->m, 0, NPARAM * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(l->v, 0, NPARAM * sizeof(float));
    if (e == cudaSuccess) e = cudaEventCreate(&l->e0);
    if (e == cudaSuccess) e = cudaEventCreate(&l->e1);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(patch_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_BYTES + 1024);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(patch_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_BYTES + 1024);
    if (e != cudaSuccess) return fail_free(e);
    // He initialisation (last layer small): the untrained network proposes nearly uniform spins
    std::vector<float> p(NPARAM, 0.f);
    std::mt19937 gen(d->seed ^ 0x9E3779B9u);
    std::normal_distribution<float> nd(0.f, 1.f);
    for (int i = 0; i < NH * NI; ++i) p[OFF_W1 + i] = nd(gen) * std::sqrt(2.0f / NI);
    for (int i = 0; i < NH * NH; ++i) p[OFF_W2 + i] = nd(gen) * std::sqrt(2.0f / NH);
    for (int i = 0; i < NO * NH; ++i) p[OFF_W3 + i] = nd(gen) * 0.01f;
    e = cudaMemcpy(l->p, p.data(), NPARAM * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return fail_free(e);
    rc = quantise_and_pack(*l, c.stream);
    if (rc) {
        ether_learn_destroy(l);
        return rc;
    }
    *out = l;
    return ETHER_OK;
}

extern "C" int ether_learn_destroy(ether_learn *l) {
    if (!l) return ETHER_OK;
    if (l->xyz) {
        learn::xyz_destroy(l->xyz);
        delete l;
        return ETHER_OK;
    }
    if (l->ctx) cudaStreamSynchronize(l->ctx->c.stream);
    l->tb.release();
    void *ptrs[] = {l->p, l->pq, l->g, l->m, l->v, l->img, l->X, l->Y, l->wp, l->loss, l->bits, l->Zp, l->lstep, l->k4, l->betaJf, l->HB,
                    l->acc, l->dump, l->err};
    for (void *q : ptrs)
        if (q) cudaFree(q);
    if (l->e0) cudaEventDestroy(l->e0);
    if (l->e1) cudaEventDestroy(l->e1);
    delete l;
    return ETHER_OK;
}

extern "C" int ether_learn_collect(ether_learn *l, int32_t per_replica) {
    if (!l) return lfail(ETHER_ERR_ARG, "null handle");
    if (per_replica < 1) return lfail(ETHER_ERR_ARG, "samples per replica must be positive");
    Ctx &c = l->ctx->c;
    if (!c.beta_set) return lfail(ETHER_ERR_STATE, "beta not set");
    if (l->xyz) return learn::xyz_collect(l->xyz, per_replica);
    int rc = refresh_tables(*l);
    if (rc) return rc;
    const long long total = (long long)l->R * per_replica;
    const int grid = (int)std::min<long long>((total + 255) / 256, 4LL * l->sm_count);
    collect_kernel<<<grid, 256, 0, c.stream>>>(c.spins, l->L[0], l->L[1], l->L[2], l->L[0] / 2, l->half,
                                               l->R, per_replica, c.stream_id, c.slot_of_rep, l->k4,
                                               c.seed, l->collect_calls, l->X, l->Y, l->write, l->cap);
    LCUDA(cudaGetLastError());
    l->launches++;
    l->collect_calls++;
    l->write = (l->write + total) % l->cap;
    l->n = std::min(l->cap, l->n + total);
    return ETHER_OK;
}

extern "C" int ether_learn_train(ether_learn *l, int32_t steps, int32_t batch, float lr, double *loss_out) {
    if (!l) return lfail(ETHER_ERR_ARG, "null handle");
    if (steps < 0 || batch < 1 || batch > 65536 || !(lr > 0.f)) return lfail(ETHER_ERR_ARG, "bad training arguments");
    if (l->xyz) return learn::xyz_train(l->xyz, steps, batch, lr, loss_out);
    if (l->n == 0) return lfail(ETHER_ERR_STATE, "no training samples (ether_learn_collect)");
    LCUDA((l->tb.ensure<NI, NO>(batch)));
    cudaStream_t st = l->ctx->c.stream;
    LCUDA(cudaEventRecord(l->e0, st));
    for (int s = 0; s < steps; ++s) {
        TrainIo T{l->X, l->Y, l->n, batch, l->seed, (uint32_t)(l->adam_t + 1), 0x4C524E00u};
        ++l->adam_t;
        const float c1 = 1.0f - std::pow(0.9f, (float)l->adam_t), c2 = 1.0f - std::pow(0.999f, (float)l->adam_t);
        LCUDA((train_step<NI, NO>(train_params(*l), T, l->tb, AdamStep{lr, c1, c2}, s == steps - 1, st, &l->launches)));
    }
    const int rc = pack_image(*l, st);
    if (rc) return rc;
    LCUDA(cudaEventRecord(l->e1, st));
    if (loss_out) {
        LCUDA(cudaMemcpyAsync(loss_out, l->loss, sizeof(double), cudaMemcpyDeviceToHost, st));
        LCUDA(cudaStreamSynchronize(st));
    }
    l->timed = 2;
    return ETHER_OK;
}

extern "C" int ether_learn_sweep(ether_learn *l, int32_t nsweeps) {
    if (!l) return lfail(ETHER_ERR_ARG, "null handle");
    if (nsweeps < 0) return lfail(ETHER_ERR_ARG, "negative sweep count");
    Ctx &c = l->ctx->c;
    if (!c.beta_set) return lfail(ETHER_ERR_STATE, "beta not set");
    if (l->xyz) return learn::xyz_sweep(l->xyz, nsweeps);
    int rc = refresh_tables(*l);
    if (rc) return rc;
    if (l->dump_on && !l->dump)
        LCUDA(cudaMalloc((void **)&l->dump, 2 * (size_t)l->R * l->Pc * NO * sizeof(float)));
    LCUDA(cudaEventRecord(l->e0, c.stream));
    for (int s = 0; s < nsweeps; ++s) {
        for (int cls = 0; cls < 2; ++cls) {
            float *dump = (l->dump_on && s == nsweeps - 1) ? l->dump + (size_t)cls * l->R * l->Pc * NO : nullptr;
            rc = launch_patches(*l, cls, dump);
            if (rc) return rc;
        }
        advance_lstep_kernel<<<(l->R + 255) / 256, 256, 0, c.stream>>>(l->lstep, l->R);
        l->launches++;
        l->proposed += 2ull * (uint64_t)l->R * (uint64_t)l->Pc;
    }
    LCUDA(cudaEventRecord(l->e1, c.stream));
    LCUDA(cudaGetLastError());
    l->timed = 1;
    l->timed_n = nsweeps;
    return ETHER_OK;
}

extern "C" int ether_learn_batch_sweep(ether_learn *const *learns, int32_t n, int32_t nsweeps,
                                       int32_t plain_per_sweep) {
    if (!learns || n <= 0 || nsweeps < 0 || plain_per_sweep < 0) return lfail(ETHER_ERR_ARG, "invalid argument");
    for (int k = 0; k < n; ++k) {
        if (!learns[k]) return lfail(ETHER_ERR_ARG, "null learner");
        if (!learns[k]->ctx->c.beta_set) return lfail(ETHER_ERR_STATE, "beta not set");
        for (int j = 0; j < k; ++j)
            if (learns[j]->ctx == learns[k]->ctx) return lfail(ETHER_ERR_ARG, "two learners of one context");
    }
    // step s of every context before step s + 1 of any: each context's stream gets its own
    // work in order, the contexts run side by side
    for (int s = 0; s < nsweeps; ++s)
        for (int k = 0; k < n; ++k) {
            int rc = plain_sweeps(learns[k]->ctx->c, plain_per_sweep);
            if (rc) return rc;
            rc = ether_learn_sweep(learns[k], 1);
            if (rc) return rc;
        }
    return ETHER_OK;
}

extern "C" int ether_learn_record_series(ether_learn *l, int32_t nsteps, int32_t plain_per_step,
                                         int32_t learned_per_step, int32_t stride, double *absM) {
    if (!l || !absM) return lfail(ETHER_ERR_ARG, "null argument");
    if (nsteps < 1 || plain_per_step < 0 || learned_per_step < 0 || plain_per_step + learned_per_step < 1 ||
        stride < 1 || nsteps / stride < 1)
        return lfail(ETHER_ERR_ARG, "need nsteps >= stride >= 1 and at least one sweep per step");
    Ctx &c = l->ctx->c;
    if (!c.beta_set) return lfail(ETHER_ERR_STATE, "beta not set");
    if (l->xyz) return learn::xyz_record_series(l->xyz, nsteps, plain_per_step, learned_per_step, stride, absM);
    int rc = refresh_tables(*l);
    if (rc) return rc;
    const int nrec = nsteps / stride;
    const size_t bytes = sizeof(double) * (size_t)nrec * l->R;
    double *mser = nullptr;
    LCUDA(cudaMalloc((void **)&mser, bytes));
    for (int t = 0; t < nsteps && rc == ETHER_OK; ++t) {
        rc = plain_sweeps(c, plain_per_step);
        for (int k = 0; k < learned_per_step && rc == ETHER_OK; ++k) {
            for (int cls = 0; cls < 2 && rc == ETHER_OK; ++cls) rc = launch_patches(*l, cls, nullptr);
            if (rc == ETHER_OK) {
                advance_lstep_kernel<<<(l->R + 255) / 256, 256, 0, c.stream>>>(l->lstep, l->R);
                l->launches++;
                l->proposed += 2ull * (uint64_t)l->R * (uint64_t)l->Pc;
            }
        }
        if (rc == ETHER_OK && (t + 1) % stride == 0 && (t + 1) / stride <= nrec) {
            const cudaError_t e = launch_record(c, (t + 1) / stride - 1, false, mser, nullptr);
            if (e != cudaSuccess) rc = lfail(ETHER_ERR_CUDA, std::string("record: ") + cudaGetErrorString(e));
        }
    }
    if (rc == ETHER_OK) {
        cudaError_t e = cudaMemcpyAsync(absM, mser, bytes, cudaMemcpyDeviceToHost, c.stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c.stream);
        if (e != cudaSuccess) rc = lfail(ETHER_ERR_CUDA, std::string("series copy: ") + cudaGetErrorString(e));
    }
    cudaFree(mser);
    if (rc) return rc;
    return read_err(*l);
}

extern "C" int ether_learn_get_accepts(ether_learn *l, uint64_t *accepted) {
    if (!l || !accepted) return lfail(ETHER_ERR_ARG, "null argument");
    if (l->xyz) return learn::xyz_get_accepts(l->xyz, accepted);
    LCUDA(cudaMemcpyAsync(accepted, l->acc, l->R * sizeof(uint64_t), cudaMemcpyDeviceToHost, l->ctx->c.stream));
    LCUDA(cudaStreamSynchronize(l->ctx->c.stream));
    return read_err(*l);
}

extern "C" int ether_learn_set_dump(ether_learn *l, int32_t on) {
    if (!l) return lfail(ETHER_ERR_ARG, "null handle");
    if (l->xyz) learn::xyz_set_dump(l->xyz, on != 0);
    l->dump_on = on != 0;
    return ETHER_OK;
}

extern "C" int ether_learn_get_dump(ether_learn *l, float *logits) {
    if (!l || !logits) return lfail(ETHER_ERR_ARG, "null argument");
    if (l->xyz) return learn::xyz_get_dump(l->xyz, logits);
    if (!l->dump) return lfail(ETHER_ERR_STATE, "no logits recorded (ether_learn_set_dump, then a sweep)");
    LCUDA(cudaMemcpyAsync(logits, l->dump, 2 * (size_t)l->R * l->Pc * NO * sizeof(float),
                          cudaMemcpyDeviceToHost, l->ctx->c.stream));
    LCUDA(cudaStreamSynchronize(l->ctx->c.stream));
    return read_err(*l);
}

extern "C" int ether_learn_get_params(ether_learn *l, float *params) {
    if (!l || !params) return lfail(ETHER_ERR_ARG, "null argument");
    if (l->xyz) return learn::xyz_get_params(l->xyz, params);
    LCUDA(cudaMemcpyAsync(params, l->p, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, l->ctx->c.stream));
    LCUDA(cudaStreamSynchronize(l->ctx->c.stream));
    return ETHER_OK;
}

extern "C" int ether_learn_set_params(ether_learn *l, const float *params) {
    if (!l || !params) return lfail(ETHER_ERR_ARG, "null argument");
    if (l->xyz) return learn::xyz_set_params(l->xyz, params);
    for (int i = 0; i < NPARAM; ++i)
        if (!std::isfinite(params[i])) return lfail(ETHER_ERR_ARG, "non-finite parameter " + std::to_string(i));
    cudaStream_t st = l->ctx->c.stream;
    LCUDA(cudaMemcpyAsync(l->p, params, NPARAM * sizeof(float), cudaMemcpyHostToDevice, st));
    LCUDA(cudaMemsetAsync(l->m, 0, NPARAM * sizeof(float), st));
    LCUDA(cudaMemsetAsync(l->v, 0, NPARAM * sizeof(float), st));
    l->adam_t = 0;
    int rc = quantise_and_pack(*l, st);
    if (rc) return rc;
    LCUDA(cudaStreamSynchronize(st));
    return ETHER_OK;
}

extern "C" int ether_learn_loss_grad(ether_learn *l, const float *x, const uint32_t *y, int32_t B,
                                     double *loss, float *grad) {
    if (!l || !x || !y || !grad) return lfail(ETHER_ERR_ARG, "null argument");
    if (B < 1 || B > 65536) return lfail(ETHER_ERR_ARG, "batch out of range");
    if (l->xyz) return lfail(ETHER_ERR_UNSUPPORTED, "XYZ learner: targets are spin components (ether_learn_loss_grad_f)");
    LCUDA((l->tb.ensure<NI, NO>(B)));
    cudaStream_t st = l->ctx->c.stream;
    std::vector<float> yf((size_t)B * NO);
    for (int b = 0; b < B; ++b)
        for (int o = 0; o < NO; ++o) yf[(size_t)b * NO + o] = (float)((y[b] >> o) & 1u);
    LCUDA(cudaMemcpyAsync(l->tb.Xb, x, (size_t)B * NI * sizeof(float), cudaMemcpyHostToDevice, st));
    LCUDA(cudaMemcpyAsync(l->tb.Yb, yf.data(), (size_t)B * NO * sizeof(float), cudaMemcpyHostToDevice, st));
    TrainIo T{};
    T.B = B;
    LCUDA((train_step<NI, NO>(train_params(*l), T, l->tb, AdamStep{0.f, 1.f, 1.f}, true, st, &l->launches)));
    double lv = 0.0;
    LCUDA(cudaMemcpyAsync(&lv, l->loss, sizeof(double), cudaMemcpyDeviceToHost, st));
    LCUDA(cudaMemcpyAsync(grad, l->g, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, st));
    LCUDA(cudaStreamSynchronize(st));
    if (loss) *loss = lv;
    return ETHER_OK;
}

extern "C" int ether_learn_forward(ether_learn *l, const float *x, int32_t B, float *logits) {
    if (!l || !x || !logits) return lfail(ETHER_ERR_ARG, "null argument");
    if (B < 1 || B > (1 << 22)) return lfail(ETHER_ERR_ARG, "batch out of range");
    if (l->xyz) return learn::xyz_forward(l->xyz, x, B, logits);
    cudaStream_t st = l->ctx->c.stream;
    std::vector<__nv_bfloat16> xb((size_t)B * NI);
    for (size_t i = 0; i < xb.size(); ++i) xb[i] = __float2bfloat16_rn(x[i]);
    __nv_bfloat16 *dX = nullptr;
    float *dZ = nullptr;
    LCUDA(cudaMalloc((void **)&dX, xb.size() * sizeof(__nv_bfloat16)));
    cudaError_t e = cudaMalloc((void **)&dZ, (size_t)B * NO * sizeof(float));
    if (e == cudaSuccess) e = cudaMemcpyAsync(dX, xb.data(), xb.size() * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        PatchParams P;
        std::memset(&P, 0, sizeof(P));
        P.img = l->img;
        P.err = l->err;
        P.X = dX;
        P.n = B;
        P.Z = dZ;
        const int tiles = (B + kThreads - 1) / kThreads;
        patch_kernel<1><<<std::min(tiles, l->sm_count), kGroups * kThreads, SM_BYTES + 1024, st>>>(P);
        l->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(logits, dZ, (size_t)B * NO * sizeof(float), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(dX);
    cudaFree(dZ);
    if (e != cudaSuccess) return lfail(ETHER_ERR_CUDA, std::string("learned forward: ") + cudaGetErrorString(e));
    return read_err(*l);
}

extern "C" int ether_learn_get_info(ether_learn *l, ether_learn_info *info) {
    if (!l || !info) return lfail(ETHER_ERR_ARG, "null argument");
    if (l->xyz) return learn::xyz_info(l->xyz, info);
    if (l->timed) {
        float ms = 0.f;
        LCUDA(cudaEventSynchronize(l->e1));
        LCUDA(cudaEventElapsedTime(&ms, l->e0, l->e1));
        if (l->timed == 1) l->sweep_ms = l->timed_n > 0 ? ms / l->timed_n : 0.f;
        else l->train_ms = ms;
        l->timed = 0;
    }
    int rc = read_err(*l);
    if (rc) return rc;
    info->n_params = NPARAM;
    info->patches_per_class = l->Pc;
    info->n_samples = l->n;
    info->capacity = l->cap;
    info->train_steps = l->adam_t;
    info->proposed = l->proposed;
    info->kernel_launches = l->launches;
    info->last_sweep_ms = l->sweep_ms;
    info->last_train_ms = l->train_ms;
    return ETHER_OK;
}

extern "C" int ether_learn_loss_grad_f(ether_learn *l, const float *x, const float *y, int32_t B, double *loss,
                                       float *grad) {
    if (!l || !x || !y || !grad) return lfail(ETHER_ERR_ARG, "null argument");
    if (B < 1 || B > 65536) return lfail(ETHER_ERR_ARG, "batch out of range");
    if (l->xyz) return learn::xyz_loss_grad(l->xyz, x, y, B, loss, grad);
    // Ising: targets 0 / 1 per output, packed as the A-site bits
    std::vector<uint32_t> bits((size_t)B, 0u);
    for (int b = 0; b < B; ++b)
        for (int o = 0; o < NO; ++o)
            if (y[(size_t)b * NO + o] > 0.5f) bits[b] |= 1u << o;
    return ether_learn_loss_grad(l, x, bits.data(), B, loss, grad);
}

extern "C" int ether_learn_get_shape(ether_learn *l, int32_t *n_inputs, int32_t *n_outputs, int32_t *n_params) {
    if (!l || !n_inputs || !n_outputs || !n_params) return lfail(ETHER_ERR_ARG, "null argument");
    int ni = NI, no = NO, np = NPARAM;
    if (l->xyz) learn::xyz_shape(&ni, &no, &np);
    *n_inputs = ni;
    *n_outputs = no;
    *n_params = np;
    return ETHER_OK;
}
