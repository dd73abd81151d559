// sweep_xyz.cuh -- device bodies of the Heisenberg (XYZ) Metropolis colour phase
// (src/Metropolis.f90:39-62 with update_spin_details.f90:30-51 and Hamiltonian.f90:34-143),
// shared by the per-context kernels (k_xyz.cu) and the persistent batch kernel (k_batch.cu).
//
// FP32 throughout, compiled with --fmad=false; the local exchange field is one fmaf chain
// per component over the neighbours in the reference's nn order (shells in order,
// neighbours by increasing site number), so every kernel variant and the oracle's FP32
// mirror round identically.
#pragma once
#include "internal.h"
#include "rng_math.cuh"

namespace ether {

__device__ __forceinline__ void warp_add_count_x(unsigned long long *dst, unsigned v) {
    unsigned s = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(dst, (unsigned long long)s);
}

struct XyzParams {
    int zeeman, sia, angle;
    float dphi;
    const uint8_t *species;
    const float *zee;
    const float *D;
    int nsp;  // species count: with one, the per-site species is not read
    int sia_local;            // per-site local-axis anisotropy D (a . S)^2
    const uint8_t *sia_cls;   // site -> class, indexed like the spin array the kernel updates:
                              // by storage index (general lattices) or, for the simple-cubic
                              // colour arrays, by rank (the table offset to the colour at launch)
    const float4 *sia_ax;     // class -> (a_x, a_y, a_z, D)
};

XyzParams xyz_params(const Ctx &c);  // k_xyz.cu

// Option sets of the XYZ kernels: kXyzExchange folds the Zeeman, SIA and ANGLE branches away
// at compile time (exchange only, Marsaglia proposals); kXyzGeneral reads them from P.
enum : int { kXyzExchange = 0, kXyzGeneral = 1 };

// ΔE of src/Hamiltonian.f90 for S -> n given the exchange field h.
template <int OPT>
__device__ __forceinline__ float delta_e(const XyzParams &P, int s, const float4 &S,
                                         const Spin4 &n, float hx, float hy, float hz) {
    float dx = n.x - S.x, dy = n.y - S.y, dz = n.z - S.z;
    float e = dx * hx;
    e = fmaf(dy, hy, e);
    e = fmaf(dz, hz, e);
    if (OPT != kXyzExchange && (P.zeeman || P.sia || P.sia_local)) {
        const int si = P.nsp == 1 ? 0 : P.species[s] - 1;
        if (P.zeeman) {
            const float *z = P.zee + 3 * si;
            e = fmaf(dx, z[0], e);
            e = fmaf(dy, z[1], e);
            e = fmaf(dz, z[2], e);
        }
        if (P.sia) {
            const float *D = P.D + 3 * si;
            float qx = n.x * n.x - S.x * S.x;
            float qy = n.y * n.y - S.y * S.y;
            float qz = n.z * n.z - S.z * S.z;
            e = fmaf(D[0], qx, e);
            e = fmaf(D[1], qy, e);
            e = fmaf(D[2], qz, e);
        }
        if (P.sia_local) {
            const float4 a = P.sia_ax[P.sia_cls[s]];
            float pn = a.x * n.x;
            pn = fmaf(a.y, n.y, pn);
            pn = fmaf(a.z, n.z, pn);
            float ps = a.x * S.x;
            ps = fmaf(a.y, S.y, ps);
            ps = fmaf(a.z, S.z, ps);
            e = fmaf(a.w, pn * pn - ps * ps, e);
        }
    }
    return e;
}

// Is the proposal n for a site in state S accepted?
template <int OPT>
__device__ __forceinline__ bool metro_accept(const XyzParams &P, int s, const float4 &S, const Spin4 &n, float eta,
                                             float hx, float hy, float hz, float beta_f, float4 &out) {
    const float e = delta_e<OPT>(P, s, S, n, hx, hy, hz);
    // exp evaluated on every lane (no divergent short-circuit); e <= 0 accepts regardless
    const float p = expf_neg(-(beta_f * fmaxf(e, 0.0f)));
    out = make_float4(n.x, n.y, n.z, n.w);
    return (e <= 0.0f) || (eta < p);
}

// The Metropolis decision of one site from its state S, the exchange field h and blocks 0
// and 1 of its draw (block 1 only for Marsaglia proposals): returns whether the proposal is
// accepted and, if so, the new state in out.
template <int OPT>
__device__ __forceinline__ bool metro_decide(const XyzParams &P, int s, const float4 &S, const U4 &b0,
                                             const U4 &b1, float hx, float hy, float hz, float beta_f,
                                             uint32_t rho, uint32_t t, uint32_t c3, const RoundKeys &K,
                                             uint32_t stream, float4 &out) {
    const bool angle = OPT != kXyzExchange && P.angle != 0;
    const float eta = u01(b0.x);
    Spin4 n;
    const Spin4 So{S.x, S.y, S.z, S.w};
    if (!propose(angle, P.dphi, So, rho, t, stream, c3, K, b0, b1, &n)) return false;
    return metro_accept<OPT>(P, s, S, n, eta, hx, hy, hz, beta_f, out);
}

template <int OPT>
__device__ __forceinline__ void site_draws(const XyzParams &P, uint32_t rho, uint32_t t, uint32_t c3,
                                           const RoundKeys &K, uint32_t stream, U4 &b0, U4 &b1) {
    b0 = draw_rk(rho, t, stream, c3, K);
    b1 = U4{0u, 0u, 0u, 0u};
    if (!(OPT != kXyzExchange && P.angle != 0)) b1 = draw_rk(rho, t, stream, c3 | (1u << 16), K);
}

template <int OPT>
__device__ __forceinline__ bool metro_site(const XyzParams &P, float4 *sp, int s, uint32_t rho,
                                           float hx, float hy, float hz, float beta_f,
                                           uint32_t t, uint32_t c3, const RoundKeys &K, uint32_t stream) {
    const float4 S = sp[s];
    U4 b0, b1;
    site_draws<OPT>(P, rho, t, c3, K, stream, b0, b1);
    float4 n;
    const bool acc = metro_decide<OPT>(P, s, S, b0, b1, hx, hy, hz, beta_f, rho, t, c3, K, stream, n);
    if (acc) sp[s] = n;
    return acc;
}

// ------------------------------------------------------- simple cubic, colour-split ----
// Neighbours are summed in increasing site-number order, which is the reference's nn order.
struct Acc3 {
    float x, y, z;
};
__device__ __forceinline__ void fma3(Acc3 &h, float jx, float jy, float jz, const float4 &S) {
    h.x = fmaf(jx, S.x, h.x);
    h.y = fmaf(jy, S.y, h.y);
    h.z = fmaf(jz, S.z, h.z);
}

// The six neighbours of rank rho of a colour array; o points at that rank in the other
// colour's array, where they sit at six offsets (one of the x pair at 0), and increasing site
// number is increasing offset.  Away from the y and z faces that is z, y, x, x, y, z; at a face
// a pair's offsets have one sign.  Loads and sum are separate steps, so that the sweep draws
// its random numbers while the loads are in flight.
struct ScNbr {
    float4 za, zb, ya, yb, xa, xb;  // a: the lower site number of the pair
    int nz, ny;                     // neighbours of the pair below the site (1 inside)
};
__device__ __forceinline__ ScNbr sc_neighbours(const float4 *__restrict__ o, int L2, int L3, int H, int xh, int y,
                                               int z, int p) {
    ScNbr n;
    const int plane = L2 * H;
    const int d = p == 0 ? (xh == 0 ? H - 1 : -1) : (xh == H - 1 ? 1 - H : 1);
    const bool y0 = y == 0, y1 = y == L2 - 1, z0 = z == 0, z1 = z == L3 - 1;
    const int far = (L3 - 1) * plane;
    n.za = o[z0 ? plane : z1 ? -far : -plane];
    n.ya = o[y0 ? H : y1 ? H - plane : -H];
    n.xa = o[min(d, 0)];
    n.xb = o[max(d, 0)];
    n.yb = o[y0 ? plane - H : y1 ? -H : H];
    n.zb = o[z0 ? far : z1 ? -plane : plane];
    n.ny = y0 ? 0 : y1 ? 2 : 1;
    n.nz = z0 ? 0 : z1 ? 2 : 1;
    return n;
}
__device__ __forceinline__ Acc3 sc_sum(const ScNbr &n, float jx, float jy, float jz) {
    Acc3 h{0.f, 0.f, 0.f};
    if ((n.ny & n.nz) == 1) {  // whole rows take this path: 94% of a 64^3 lattice's
        fma3(h, jx, jy, jz, n.za);
        fma3(h, jx, jy, jz, n.ya);
        fma3(h, jx, jy, jz, n.xa);
        fma3(h, jx, jy, jz, n.xb);
        fma3(h, jx, jy, jz, n.yb);
        fma3(h, jx, jy, jz, n.zb);
        return h;
    }
    if (n.nz > 0) fma3(h, jx, jy, jz, n.za);
    if (n.nz > 1) fma3(h, jx, jy, jz, n.zb);
    if (n.ny > 0) fma3(h, jx, jy, jz, n.ya);
    if (n.ny > 1) fma3(h, jx, jy, jz, n.yb);
    fma3(h, jx, jy, jz, n.xa);
    fma3(h, jx, jy, jz, n.xb);
    if (n.ny == 0) fma3(h, jx, jy, jz, n.ya);
    if (n.ny < 2) fma3(h, jx, jy, jz, n.yb);
    if (n.nz == 0) fma3(h, jx, jy, jz, n.za);
    if (n.nz < 2) fma3(h, jx, jy, jz, n.zb);
    return h;
}
__device__ __forceinline__ Acc3 sc_field(const float4 *__restrict__ o, int L2, int L3, int H, int xh, int y, int z,
                                         int p, float jx, float jy, float jz) {
    return sc_sum(sc_neighbours(o, L2, L3, H, xh, y, z, p), jx, jy, jz);
}

// Exchange field of rank rho of a colour class from its ELL block (ell: entries k * n_c + rho,
// coalesced across a warp), in the CSR's order -- the reference's nn order -- so the fmaf
// chain rounds as the oracle's.
// W > 0: the class's ELL width, known at compile time (every load of the site issued at
// once); W = 0: width at run time.
template <int W = 0>
__device__ __forceinline__ Acc3 ell_field(const float4 *__restrict__ sp, const int32_t *__restrict__ ell,
                                          const uint16_t *__restrict__ ej, const float4 *__restrict__ J4,
                                          int n_c, int width, int rho, int deg) {
    // The padding entries point at valid memory (the site itself, coupling 0), so the loads
    // are unconditional and can all be in flight at once; only the fmaf is predicated.
    Acc3 h{0.f, 0.f, 0.f};
    if constexpr (W > 0) {
        // the neighbours' storage indices, then all their spins, then the field
        int nb[W];
#pragma unroll
        for (int k = 0; k < W; ++k) nb[k] = ell[k * n_c + rho];  // ELL blocks hold < 2^31 entries
        float4 Sj[W];
#pragma unroll
        for (int k = 0; k < W; ++k) Sj[k] = sp[nb[k]];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const float4 Jv = J4[ej[k * n_c + rho]];
            if (k < deg) {
                h.x = fmaf(Jv.x, Sj[k].x, h.x);
                h.y = fmaf(Jv.y, Sj[k].y, h.y);
                h.z = fmaf(Jv.z, Sj[k].z, h.z);
            }
        }
    } else {
#pragma unroll 6
        for (int k = 0; k < width; ++k) {
            const int e = k * n_c + rho;
            const float4 Jv = J4[ej[e]];
            const float4 Sj = sp[ell[e]];
            if (k < deg) {
                h.x = fmaf(Jv.x, Sj.x, h.x);
                h.y = fmaf(Jv.y, Sj.y, h.y);
                h.z = fmaf(Jv.z, Sj.z, h.z);
            }
        }
    }
    return h;
}

// One Metropolis update of rank rho of a colour class of a general lattice (ELL block of the
// class: ell, ej; deg per storage index; W as ell_field's).
template <int OPT, int W = 0>
__device__ __forceinline__ bool xyz_ell_site(const XyzParams &P, float4 *sp, int col_off, int n_c, int rho,
                                             const int32_t *__restrict__ ell, const uint16_t *__restrict__ ej,
                                             const uint16_t *__restrict__ deg, int width,
                                             const float4 *__restrict__ J4, float beta_f, uint32_t t,
                                             uint32_t c3, const RoundKeys &K, uint32_t stream) {
    const int s = col_off + rho;
    const Acc3 h = ell_field<W>(sp, ell, ej, J4, n_c, width, rho, deg[s]);
    return metro_site<OPT>(P, sp, s, (uint32_t)rho, h.x, h.y, h.z, beta_f, t, c3, K, stream);
}

// A replica's simple-cubic colour arrays: the updated colour's (own) and the other's (opp).
struct XyzSc {
    float4 *own;
    const float4 *opp;
    int L1, L2, L3, H;
    FastDiv fH, fL2;
    uint32_t colour;
    float jx, jy, jz;
};
// One column (col = y H + xh) of a simple-cubic replica, its sites taken up the z axis.  Of a
// site's neighbours two are known from the site below it -- its z - 1 neighbour was that site's x
// neighbour at offset 0, and its own one at offset 0 was that site's z + 1 neighbour -- and
// the column fixes all indices but z: four neighbour loads a site instead of six, and a fifth
// fewer instructions.  NEAR: arrays below 4 GB, byte offsets of 32 bits beside their addresses.
template <bool NEAR>
struct ScColumn {
    const XyzSc &A;
    const int H, L2, L3, plane, y, xh, d0, d1, dym, dyp;
    const bool y0, y1;
    int z, rho, p;
    float4 zm, x0;            // carried up
    float4 ym, yp, xd, zp, S;  // loaded for the present site

    __device__ __forceinline__ const float4 *at(const float4 *base, int i) const {
        if constexpr (NEAR) return reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(base) + (uint32_t)i * 16u);
        else return base + i;
    }
    __device__ __forceinline__ ScColumn(const XyzSc &A_, int col, int z0)
        : A(A_), H(A_.H), L2(A_.L2), L3(A_.L3), plane(A_.L2 * A_.H), y((int)fdiv((uint32_t)col, A_.fH)),
          xh(col - y * A_.H), d0(xh == 0 ? H - 1 : -1), d1(xh == H - 1 ? 1 - H : 1),
          dym(y == 0 ? plane - H : -H), dyp(y == L2 - 1 ? H - plane : H), y0(y == 0), y1(y == L2 - 1), z(z0),
          rho(z0 * plane + col), p((y + z0 + (int)A_.colour) & 1) {
        zm = *at(A.opp, rho + (z0 == 0 ? (L3 - 1) * plane : -plane));
        x0 = *at(A.opp, rho);
    }
    __device__ __forceinline__ void load() {
        ym = *at(A.opp, rho + dym);
        yp = *at(A.opp, rho + dyp);
        xd = *at(A.opp, rho + (p ? d1 : d0));
        zp = *at(A.opp, rho + (z == L3 - 1 ? plane - L3 * plane : plane));
        S = *at(A.own, rho);
    }
    // increasing site number; at a face the wrapped neighbour changes side
    __device__ __forceinline__ Acc3 field() const {
        Acc3 h{0.f, 0.f, 0.f};
        const int d = p ? d1 : d0;
        const float4 xa = d < 0 ? xd : x0, xb = d < 0 ? x0 : xd;
        if (!y0 && !y1 && z != 0 && z != L3 - 1) {
            fma3(h, A.jx, A.jy, A.jz, zm);
            fma3(h, A.jx, A.jy, A.jz, ym);
            fma3(h, A.jx, A.jy, A.jz, xa);
            fma3(h, A.jx, A.jy, A.jz, xb);
            fma3(h, A.jx, A.jy, A.jz, yp);
            fma3(h, A.jx, A.jy, A.jz, zp);
        } else {
            if (z == L3 - 1) fma3(h, A.jx, A.jy, A.jz, zp);
            if (z != 0) fma3(h, A.jx, A.jy, A.jz, zm);
            if (y1) fma3(h, A.jx, A.jy, A.jz, yp);
            if (!y0) fma3(h, A.jx, A.jy, A.jz, ym);
            fma3(h, A.jx, A.jy, A.jz, xa);
            fma3(h, A.jx, A.jy, A.jz, xb);
            if (!y1) fma3(h, A.jx, A.jy, A.jz, yp);
            if (y0) fma3(h, A.jx, A.jy, A.jz, ym);
            if (z != L3 - 1) fma3(h, A.jx, A.jy, A.jz, zp);
            if (z == 0) fma3(h, A.jx, A.jy, A.jz, zm);
        }
        return h;
    }
    __device__ __forceinline__ float4 *site() const { return const_cast<float4 *>(at(A.own, rho)); }
    __device__ __forceinline__ void up() {
        zm = x0;
        x0 = zp;
        rho += plane;
        ++z;
        p ^= 1;
    }
};

// The sites z0 <= z < z1 of a column, each with its own draws, made while its loads are in flight.
template <int OPT>
__device__ __forceinline__ unsigned xyz_sc_column(const XyzSc &A, const XyzParams &P, int col, int z0, int z1,
                                                  float beta_f, uint32_t t, uint32_t c3, const RoundKeys &K,
                                                  uint32_t stream) {
    ScColumn<false> C(A, col, z0);
    unsigned acc = 0;
#pragma unroll 1
    while (C.z < z1) {
        C.load();
        U4 b0, b1;
        site_draws<OPT>(P, (uint32_t)C.rho, t, c3, K, stream, b0, b1);
        const Acc3 h = C.field();
        float4 nv;
        if (metro_decide<OPT>(P, C.rho, C.S, b0, b1, h.x, h.y, h.z, beta_f, (uint32_t)C.rho, t, c3, K, stream, nv)) {
            *C.site() = nv;
            ++acc;
        }
        C.up();
    }
    return acc;
}

// The same for a warp's 32 columns of one replica, nz <= planes sites each (lanes without work:
// nz = 0), Marsaglia proposals only.  21% of the sites need pairs beyond their first block, so
// almost every warp would draw a second block for all its sites; here the sites of POOL planes
// that need one are queued and drawn for 32 at a time (1.3 blocks a site instead of 2.3).
template <int POOL>
struct ScPool {                     // of a warp, in shared memory
    float4 prop[POOL][32];          // v1 (of a rejected pair: the rank), v2, s, eta
    uint8_t queue[POOL * 32];       // places in prop
};
template <int OPT, bool NEAR, int POOL>
__device__ __forceinline__ unsigned xyz_sc_columns(const XyzSc &A, const XyzParams &P, int col, int z0, int nz, int planes,
                                                   float beta_f, uint32_t t, uint32_t c3, const RoundKeys &K,
                                                   uint32_t stream, ScPool<POOL> &pool) {
    const int lane = threadIdx.x & 31;
    ScColumn<NEAR> C(A, col, z0);
    unsigned acc = 0;
#pragma unroll 1
    for (int zb = 0; zb < planes; zb += POOL) {
        int queued = 0;
#pragma unroll 1
        for (int j = 0; j < POOL; ++j) {
            const uint32_t rho = (uint32_t)(C.rho + j * C.plane);
            const U4 b = draw_rk(rho, t, stream, c3, K);
            const float v1 = upm1(b.y), v2 = upm1(b.z), s = v1 * v1 + v2 * v2;
            const bool more = !(s < 1.0f) && zb + j < nz;
            pool.prop[j][lane] = make_float4(more ? __uint_as_float(rho) : v1, v2, s, u01(b.x));
            const uint32_t m = __ballot_sync(0xffffffffu, more);
            if (more) pool.queue[queued + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(j * 32 + lane);
            queued += __popc(m);
        }
        __syncwarp();
        for (int q = lane; q < queued; q += 32) {
            float4 *const w = &pool.prop[0][0] + pool.queue[q];
            const uint32_t rho = __float_as_uint(w->x);
            const U4 b = draw_rk(rho, t, stream, c3 | (1u << 16), K);
            float v1 = upm1(b.x), v2 = upm1(b.y), s = v1 * v1 + v2 * v2;
            if (!(s < 1.0f)) {
                v1 = upm1(b.z);
                v2 = upm1(b.w);
                s = v1 * v1 + v2 * v2;
                // with no pair accepted this one stays, and there is no proposal
                if (!(s < 1.0f)) marsaglia_tail(rho, t, stream, c3, K, &v1, &v2, &s);
            }
            w->x = v1;
            w->y = v2;
            w->z = s;
        }
        __syncwarp();
#pragma unroll 1
        for (int j = 0; j < POOL && zb + j < nz; ++j) {
            C.load();
            const float4 v = pool.prop[j][lane];
            const Acc3 h = C.field();
            float4 nv;
            if (v.z < 1.0f && metro_accept<OPT>(P, C.rho, C.S, marsaglia_spin(v.x, v.y, v.z), v.w, h.x, h.y, h.z, beta_f, nv)) {
                *C.site() = nv;
                ++acc;
            }
            C.up();
        }
        __syncwarp();
    }
    return acc;
}

}  // namespace ether
