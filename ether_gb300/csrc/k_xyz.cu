// k_xyz.cu -- per-context launches of the Heisenberg (XYZ) colour phases (Metropolis bodies
// in sweep_xyz.cuh); overrelaxation (src/overrelaxation.f90:30-61 with
// get_ovrr_vec.f90:41-85); fresh_spins (src/fresh_spins.f90:31-38).
#include <algorithm>

#include "sweep_xyz.cuh"

namespace ether {

// ------------------------------------------------------------------ general lattice ----
// One thread per rank of the colour class (xyz_ell_site); W: the class's ELL width at compile
// time (0: at run time).  Bound: latency of the neighbour loads.  With the counter from a read-only
// load the compiler keeps all of a site's loads in flight (exchange only: 60 registers; 44 with a
// plain load, and they wait in turns).  A sweep, plain and read-only: pyrochlore 12^3 x 1 38.0 and
// 30.5 us, x 64 89.5 and 82.7; 20^3 fcc cells, 18 neighbours, x 1 73.8 and 59.0; bcc, 8, x 1 7.9 and
// 6.3; 31 x 33 x 35 cubic x 64 37.8 both.  The run-time width loses by it (26 neighbours 127 and 132).
template <int OPT, int W>
__global__ void __launch_bounds__(256)
xyz_ell_kernel(float4 *__restrict__ spins4, int N, int col_off, int n_c, uint32_t colour,
               const int32_t *__restrict__ ell, const uint16_t *__restrict__ ej,
               const uint16_t *__restrict__ deg, int width, const float4 *__restrict__ J4, XyzParams P,
               const float *__restrict__ beta_slot_f, const int32_t *__restrict__ slot_of_rep,
               const uint32_t *__restrict__ stream_id, const uint32_t *__restrict__ step, uint32_t ahead,
               const RoundKeys K, unsigned long long *__restrict__ acc_count) {
    const int r = blockIdx.y;
    float4 *sp = spins4 + (size_t)r * N;
    const float beta_f = beta_slot_f[slot_of_rep[r]];
    const uint32_t k1 = stream_id[r], t = (W > 0 ? __ldg(step + r) : step[r]) + ahead;
    const uint32_t c3 = kMetro | (colour << 8);
    unsigned acc = 0;
    for (int rho = blockIdx.x * blockDim.x + threadIdx.x; rho < n_c; rho += gridDim.x * blockDim.x) {
        acc += xyz_ell_site<OPT, W>(P, sp, col_off, n_c, rho, ell, ej, deg, width, J4, beta_f, t, c3, K, k1) ? 1u : 0u;
    }
    warp_add_count_x(acc_count + r, acc);
}

// Simple cubic, a thread per column and chunk of ZC planes.  POOL > 0: Marsaglia proposals whose
// second blocks a warp draws together (xyz_sc_columns); 0: each site's draws in place (angle
// proposals, which need one block only, single planes, and arrays of 4 GB and more).  Bound: issue
// (65%; IMAD.WIDE occupies the dispatch port longer) and the neighbour loads behind it: 275
// instructions per update, 1.3 Philox blocks among them (292 and 2.3 in place; 400 when every site
// looked up its six neighbours and its indices itself).  Updates/ns at T_c, every site on its own,
// by columns, and pooled: 64^3 x 64 66, 83.8 and 92.7 (0.66 of the measured copy rate at 48 bytes
// per update), 32^3 x 290 58, 74.8 and 82.9.
// Measured and not kept: 256 threads (four blocks: 87.1 and 77.5); nine and ten blocks (90.7 and
// 87.0: less L1 for the neighbours); 8 planes a pool in 24 KB a block (81.9); the next site's
// loads one site ahead, in registers (83.6) or as prefetches (91.2).
constexpr int kColThreads = 128, kColBlocks = 8;
template <int OPT, bool NEAR, int POOL>
__global__ void __launch_bounds__(kColThreads, kColBlocks)
xyz_col_kernel(float4 *__restrict__ spins4, int L1, int L2, int L3, FastDiv fH, FastDiv fP, int ZC, int items,
               uint32_t colour, float jx, float jy, float jz, XyzParams P, const float *__restrict__ beta_slot_f,
               const int32_t *__restrict__ slot_of_rep, const uint32_t *__restrict__ stream_id,
               const uint32_t *__restrict__ step, uint32_t ahead, const RoundKeys K,
               unsigned long long *__restrict__ acc_count) {
    const int r = blockIdx.y;
    const int H = L1 >> 1;
    const int half = H * L2 * L3;
    float4 *base = spins4 + (size_t)r * 2 * half;
    const XyzSc A{base + (size_t)colour * half, base + (size_t)(colour ^ 1u) * half, L1, L2, L3, H,
                  fH, fP, colour, jx, jy, jz};
    const float beta_f = beta_slot_f[slot_of_rep[r]];
    const uint32_t k1 = stream_id[r], t = step[r] + ahead;
    unsigned acc = 0;
    const int i = blockIdx.x * kColThreads + threadIdx.x;
    if constexpr (POOL > 0) {
        __shared__ ScPool<POOL> pool[kColThreads / 32];
        const int u = min(i, items - 1), chunk = (int)fdiv((uint32_t)u, fP), col = u - chunk * (int)fP.d;
        const int nz = i < items ? min(ZC, L3 - chunk * ZC) : 0;
        acc = xyz_sc_columns<OPT, NEAR, POOL>(A, P, col, chunk * ZC, nz, ZC, beta_f, t, kMetro | (colour << 8), K, k1,
                                        pool[threadIdx.x >> 5]);
    } else if (i < items) {
        const int chunk = (int)fdiv((uint32_t)i, fP), col = i - chunk * (int)fP.d;
        acc = xyz_sc_column<OPT>(A, P, col, chunk * ZC, min(chunk * ZC + ZC, L3), beta_f, t, kMetro | (colour << 8), K,
                                 k1);
    }
    warp_add_count_x(acc_count + r, acc);
}

// ------------------------------------------------------------------ overrelaxation ----
// Reflection of overrelaxation.f90:44-47 about the exchange field A (get_ovrr_vec),
// then normalisation.  A site with A = 0 is left unchanged (the reference would divide
// by zero).  Pass `pass` < floor(ovrr_para) reflects every site; the last pass reflects a
// site iff its uniform < part.  Neighbours from the colour class's ELL block.
__device__ __forceinline__ void ovrr_reflect(float4 *site, float hx, float hy, float hz) {
    const float4 S = *site;
    float d = hx * S.x;
    d = fmaf(hy, S.y, d);
    d = fmaf(hz, S.z, d);
    float a2 = hx * hx;
    a2 = fmaf(hy, hy, a2);
    a2 = fmaf(hz, hz, a2);
    if (!(a2 > 0.0f)) return;
    const float f = 2.0f * (d / a2);
    const float nx = f * hx - S.x, ny = f * hy - S.y, nz = f * hz - S.z;
    const float inv = 1.0f / sqrtf(nx * nx + ny * ny + nz * nz);
    *site = make_float4(nx * inv, ny * inv, nz * inv, S.w);
}

__global__ void __launch_bounds__(256)
ovrr_ell_kernel(float4 *__restrict__ spins4, int N, int col_off, int n_c, uint32_t colour,
                int pass, float part, const int32_t *__restrict__ ell, const uint16_t *__restrict__ ej,
                const uint16_t *__restrict__ deg, int width, const float4 *__restrict__ J4,
                const uint32_t *__restrict__ stream_id, const uint32_t *__restrict__ ovrr_step,
                uint32_t seed) {
    const int r = blockIdx.y;
    float4 *sp = spins4 + (size_t)r * N;
    const uint32_t k1 = stream_id[r], t = ovrr_step[r];
    const uint32_t c3 = kOvrr | (colour << 8);
    for (int rho = blockIdx.x * blockDim.x + threadIdx.x; rho < n_c; rho += gridDim.x * blockDim.x) {
        const int s = col_off + rho;
        if (part < 1.0f) {
            U4 o = draw((uint32_t)rho, t, k1, c3 | ((uint32_t)pass << 16), seed);
            if (!(u01(o.x) < part)) continue;
        }
        const Acc3 h = ell_field(sp, ell, ej, J4, n_c, width, rho, deg[s]);
        ovrr_reflect(sp + s, h.x, h.y, h.z);
    }
}

// The same on a simple-cubic lattice: neighbours from the other colour's array in closed
// form (sc_field sums them in the order of the ELL block, so the results are the same).
__global__ void __launch_bounds__(256)
ovrr_sc_kernel(float4 *__restrict__ spins4, int L1, int L2, int L3, FastDiv fH, FastDiv fL2, uint32_t colour,
               int pass, float part, float jx, float jy, float jz, const uint32_t *__restrict__ stream_id,
               const uint32_t *__restrict__ ovrr_step, uint32_t seed) {
    const int r = blockIdx.y;
    const int H = L1 >> 1;
    const int half = H * L2 * L3;
    float4 *base = spins4 + (size_t)r * 2 * half;
    float4 *own = base + (size_t)colour * half;
    const float4 *opp = base + (size_t)(colour ^ 1u) * half;
    const uint32_t k1 = stream_id[r], t = ovrr_step[r];
    const uint32_t c3 = kOvrr | (colour << 8);
    for (int rho = blockIdx.x * blockDim.x + threadIdx.x; rho < half; rho += gridDim.x * blockDim.x) {
        if (part < 1.0f) {
            U4 o = draw((uint32_t)rho, t, k1, c3 | ((uint32_t)pass << 16), seed);
            if (!(u01(o.x) < part)) continue;
        }
        const int row = (int)fdiv((uint32_t)rho, fH);
        const int xh = rho - row * H;
        const int z = (int)fdiv((uint32_t)row, fL2), y = row - z * L2;
        const int p = (y + z + (int)colour) & 1;
        const Acc3 h = sc_field(opp + rho, L2, L3, H, xh, y, z, p, jx, jy, jz);
        ovrr_reflect(own + rho, h.x, h.y, h.z);
    }
}

// ------------------------------------------------------------------ fresh spins -------
// key (seed, stream), counter (site number, call, block, kFresh).  Marsaglia pairs:
// p -> block p/2, words 2(p&1), 2(p&1)+1.  ANGLE: z from word 0, phi step from word 1.
__global__ void fresh_kernel(uint8_t *__restrict__ spins, float4 *__restrict__ spins4, int N,
                             int model, int angle, float dphi,
                             const int32_t *__restrict__ site_of_storage,
                             const uint32_t *__restrict__ stream_id,
                             const uint32_t *__restrict__ fresh_call, uint32_t seed) {
    const int r = blockIdx.y;
    const uint32_t k1 = stream_id[r], call = fresh_call[r];
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < N; s += gridDim.x * blockDim.x) {
        if (model == 0) {
            spins[(size_t)r * N + s] ^= 1u;
            continue;
        }
        const uint32_t i = (uint32_t)site_of_storage[s];
        float4 S = spins4[(size_t)r * N + s];
        U4 o = draw(i, call, k1, kFresh, seed);
        float nx, ny, nz, nphi;
        if (!angle) {
            float v1 = 0.f, v2 = 0.f, q = 0.f;
            bool ok = false;
            U4 w = o;
            for (int p = 0; p < kMarsagliaMaxPairs; ++p) {
                if (p >= 2 && (p & 1) == 0) w = draw(i, call, k1, kFresh | ((uint32_t)(p / 2) << 16), seed);
                uint32_t a = (p & 1) ? w.z : w.x;
                uint32_t b = (p & 1) ? w.w : w.y;
                v1 = upm1(a);
                v2 = upm1(b);
                q = v1 * v1 + v2 * v2;
                if (q < 1.0f) { ok = true; break; }
            }
            if (!ok) continue;
            float tq = sqrtf(1.0f - q);
            nx = (2.0f * v1) * tq;
            ny = (2.0f * v2) * tq;
            nz = 1.0f - 2.0f * q;
            nphi = 0.0f;
        } else {
            nz = upm1(o.x);
            nphi = S.w + dphi * upm1(o.y);
            if (nphi >= kPiF) nphi = nphi - kTwoPiF;
            else if (nphi < -kPiF) nphi = nphi + kTwoPiF;
            float rr = sqrtf(1.0f - nz * nz);
            float sn, cs;
            sincos_own(nphi, &sn, &cs);
            nx = rr * cs;
            ny = rr * sn;
        }
        float inv = 1.0f / sqrtf(nx * nx + ny * ny + nz * nz);
        spins4[(size_t)r * N + s] = make_float4(nx * inv, ny * inv, nz * inv, nphi);
    }
}

__global__ void advance_kernel(uint32_t *__restrict__ counter, int R, uint32_t by) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < R) counter[r] += by;
}

static int blocks_for_x(const Ctx &c, long work, int bs) {
    long need = (work + bs - 1) / bs;
    long cap = (long)c.sm_count * 8 / (c.R > 0 ? c.R : 1);
    if (cap < 1) cap = 1;
    if (need > cap) need = cap;
    if (need < 1) need = 1;
    return (int)need;
}

XyzParams xyz_params(const Ctx &c) {
    XyzParams P;
    P.zeeman = c.zeeman;
    P.sia = c.sia;
    P.angle = c.angle;
    P.dphi = (float)c.dphi;
    P.species = c.t.species;
    P.zee = c.t.zee;
    P.D = c.t.D;
    P.nsp = c.nsp;
    P.sia_local = c.sia_local;
    P.sia_cls = c.t.sia_cls;
    P.sia_ax = c.t.sia_ax;
    return P;
}

// Planes per thread: the most of 8, 4, 2 that still gives six blocks of 256 per SM (64^3 x 64: 92.7
// updates/ns with 8, 90.0 with 4, 91.1 with 16; 48^3 x 32, where 8 leaves 864 blocks: 68.3, 71.8
// with 4, 61.6 with 2; 16^3 x 512: 56.7 with 2, 52.1 with 1).  Variants 12 and 13 halve and double it.
static int xyz_planes(const Ctx &c) {
    const long plane = (long)(c.L[0] / 2) * c.L[1];
    int zc = 1;
    for (int v = 8; v > 1 && zc == 1; v /= 2)
        if (c.R * ((plane * ((c.L[2] + v - 1) / v) + 255) / 256) >= 6L * c.sm_count) zc = v;
    if (c.xyz_variant == 12) zc = std::max(1, zc / 2);
    if (c.xyz_variant == 13) zc *= 2;
    return zc;
}

template <int OPT>
static void launch_xyz_col(Ctx &c, int colour, const XyzParams &P, const RoundKeys &K) {
    const int half = c.N / 2, plane = c.L[0] / 2 * c.L[1], ZC = xyz_planes(c);
    const int items = plane * ((c.L[2] + ZC - 1) / ZC);
    dim3 grid((items + kColThreads - 1) / kColThreads, c.R);
    XyzParams Pc = P;  // the kernel indexes sites by rank in the colour array
    if (Pc.sia_cls) Pc.sia_cls += (size_t)colour * half;
    // single shell, single species: J(1,1,1,:)
    auto k = xyz_col_kernel<OPT, false, 0>;  // rejected pairs in place
    if (!P.angle && half < (1 << 28))
        k = ZC >= 4 ? xyz_col_kernel<OPT, true, 4> : ZC >= 2 ? xyz_col_kernel<OPT, true, 2> : k;
    k<<<grid, kColThreads, 0, c.stream>>>(
        c.spins4, c.L[0], c.L[1], c.L[2], make_fastdiv((uint32_t)(c.L[0] / 2)), make_fastdiv((uint32_t)plane), ZC, items,
        (uint32_t)colour, c.h_Jf[0], c.h_Jf[1], c.h_Jf[2], Pc, c.beta_slot_f, c.slot_of_rep, c.stream_id, c.step, c.ahead, K,
        c.acc_count);
}

// The general-lattice kernel for a class's ELL width: common widths at compile time.
template <int OPT>
static auto ell_kernel_for(int width) {
    switch (width) {
        case 4: return xyz_ell_kernel<OPT, 4>;
        case 6: return xyz_ell_kernel<OPT, 6>;
        case 8: return xyz_ell_kernel<OPT, 8>;
        case 12: return xyz_ell_kernel<OPT, 12>;
        case 14: return xyz_ell_kernel<OPT, 14>;
        case 18: return xyz_ell_kernel<OPT, 18>;
        case 24: return xyz_ell_kernel<OPT, 24>;
        default: return xyz_ell_kernel<OPT, 0>;
    }
}

bool xyz_variant_valid(int v) { return (v >= 11 && v <= 15) || v == 21 || v == 22; }

cudaError_t launch_xyz_sweep(Ctx &c, int colour) {
    const int bs = 256;
    XyzParams P = xyz_params(c);
    const RoundKeys K = round_keys(c.seed);
    const bool exchange_only = !P.zeeman && !P.sia && !P.angle && !P.sia_local;
    if (c.fast) {
        if (exchange_only) launch_xyz_col<kXyzExchange>(c, colour, P, K);
        else launch_xyz_col<kXyzGeneral>(c, colour, P, K);
    } else {
        const int n_c = c.col_off[colour + 1] - c.col_off[colour];
        if (n_c == 0) return cudaSuccess;
        const int r0 = c.rw0, nr = c.rwn ? c.rwn : c.R;  // replica window (the grid keeps the full R's width)
        dim3 grid(blocks_for_x(c, n_c, bs), nr);
        const int32_t *ell = c.t.ell_nbr + c.ell_off[colour];
        const uint16_t *ej = c.t.ell_j + c.ell_off[colour];
        auto k = exchange_only ? ell_kernel_for<kXyzExchange>(c.ell_width[colour])
                               : ell_kernel_for<kXyzGeneral>(c.ell_width[colour]);
        k<<<grid, bs, 0, c.stream>>>(c.spins4 + (size_t)r0 * c.N, c.N, c.col_off[colour], n_c, (uint32_t)colour, ell,
                                     ej, c.t.ell_deg, c.ell_width[colour], c.t.J4, P, c.beta_slot_f,
                                     c.slot_of_rep + r0, c.stream_id + r0, c.step + r0, c.ahead, K, c.acc_count + r0);
    }
    c.launches++;
    return cudaGetLastError();
}

cudaError_t launch_overrelax(Ctx &c, int colour, int pass, float part) {
    const int bs = 256;
    const int n_c = c.col_off[colour + 1] - c.col_off[colour];
    if (n_c == 0) return cudaSuccess;
    dim3 grid(blocks_for_x(c, n_c, bs), c.R);
    if (c.fast) {
        ovrr_sc_kernel<<<grid, bs, 0, c.stream>>>(c.spins4, c.L[0], c.L[1], c.L[2], make_fastdiv((uint32_t)(c.L[0] / 2)),
                                                  make_fastdiv((uint32_t)c.L[1]), (uint32_t)colour, pass, part,
                                                  c.h_Jf[0], c.h_Jf[1], c.h_Jf[2], c.stream_id, c.ovrr_step, c.seed);
        c.launches++;
        return cudaGetLastError();
    }
    ovrr_ell_kernel<<<grid, bs, 0, c.stream>>>(c.spins4, c.N, c.col_off[colour], n_c, (uint32_t)colour, pass,
                                               part, c.t.ell_nbr + c.ell_off[colour],
                                               c.t.ell_j + c.ell_off[colour], c.t.ell_deg,
                                               c.ell_width[colour], c.t.J4, c.stream_id, c.ovrr_step,
                                               c.seed);
    c.launches++;
    return cudaGetLastError();
}

cudaError_t launch_fresh(Ctx &c) {
    const int bs = 256;
    dim3 grid(blocks_for_x(c, c.N, bs), c.R);
    fresh_kernel<<<grid, bs, 0, c.stream>>>(c.spins, c.spins4, c.N, c.model, c.angle,
                                            (float)c.dphi, c.t.site_of_storage, c.stream_id,
                                            c.fresh_call, c.seed);
    c.launches++;
    return cudaGetLastError();
}

// Replica 0's bytes copied into replicas 1 .. R-1 (16-byte words when the size allows).
__global__ void broadcast_kernel(uint8_t *__restrict__ base, long long bytes, int R) {
    const long long total = bytes * (R - 1);
    const long long stride = (long long)gridDim.x * blockDim.x;
    if ((bytes & 15) == 0) {
        const uint4 *src = reinterpret_cast<const uint4 *>(base);
        uint4 *dst = reinterpret_cast<uint4 *>(base + bytes);
        const long long w = bytes >> 4;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (total >> 4); i += stride)
            dst[i] = src[i % w];
    } else {
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += stride)
            base[bytes + i] = base[i % bytes];
    }
}

cudaError_t launch_broadcast(Ctx &c, void *base, size_t bytes_per_replica) {
    if (c.R < 2) return cudaSuccess;
    const long long work = (long long)bytes_per_replica * (c.R - 1) / 16 + 1;
    const int grid = (int)std::min<long long>((work + 255) / 256, (long long)c.sm_count * 8);
    broadcast_kernel<<<grid, 256, 0, c.stream>>>(reinterpret_cast<uint8_t *>(base), (long long)bytes_per_replica, c.R);
    c.launches++;
    return cudaGetLastError();
}

// Acceptance ratios of the sweeps since the snapshot: out[r] = (acc[r] - before[r]) / N.
__global__ void accept_ratio_kernel(const unsigned long long *__restrict__ acc,
                                    const unsigned long long *__restrict__ before, int R, double invN,
                                    double *__restrict__ out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < R) out[r] = (double)(acc[r] - before[r]) * invN;
}

cudaError_t launch_accept_ratio(Ctx &c, double *out) {
    accept_ratio_kernel<<<(c.R + 255) / 256, 256, 0, c.stream>>>(c.acc_count, c.acc_before, c.R,
                                                                  1.0 / (double)c.N, out);
    c.launches++;
    return cudaGetLastError();
}

cudaError_t launch_advance(Ctx &c, uint32_t *counter, int by) {
    const int r0 = c.rw0, nr = c.rwn ? c.rwn : c.R;
    advance_kernel<<<(nr + 255) / 256, 256, 0, c.stream>>>(counter + r0, nr, (uint32_t)by);
    c.launches++;
    return cudaGetLastError();
}

}  // namespace ether
