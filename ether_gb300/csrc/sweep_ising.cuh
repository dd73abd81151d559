// sweep_ising.cuh -- device bodies of the Ising Metropolis colour phase
// (src/Metropolis.f90:39-62 with the Ising branch of update_spin_details.f90:34-35 and
// Hamiltonian.f90:34-52), shared by the per-context kernels (k_ising.cu) and the persistent
// batch kernel (k_batch.cu).
//
// Decision: a site flips iff its uniform u32 u <= T, T = max(ceil(2^32 p), 1) - 1 with
// p = exp(-β ΔE) -- the reference's -βΔE > log(η) for η = u 2^-32, η = 0 included.  T comes
// from a per-temperature table indexed by (site type, own spin, up-neighbour counts per
// (shell, neighbour species) group), built in FP64 on the host.
//
// Random numbers: the sites of a colour class are taken in groups of eight (rank >> 3).
// Site k of a group owns halfword k of two Philox blocks: block 0 gives the high 16 bits
// of its u, block 1 the low 16 bits.  Since u <= T  <=>  uh < Th  or  (uh == Th and
// ul <= Tl), block 1 is only evaluated when a high half ties (probability 2^-16): one
// Philox call serves eight site updates, and the decision is still the exact 32-bit one.
#pragma once
#include "internal.h"
#include "rng_math.cuh"

namespace ether {

__device__ __forceinline__ void warp_add_count(unsigned long long *dst, unsigned v) {
    unsigned s = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(dst, (unsigned long long)s);
}

__device__ __forceinline__ uint32_t half_of(const U4 &b, int k) {  // halfword k = 0..7
    const uint32_t w = (k >> 1) == 0 ? b.x : (k >> 1) == 1 ? b.y : (k >> 1) == 2 ? b.z : b.w;
    return (k & 1) ? (w >> 16) : (w & 0xFFFFu);
}

// ------------------------------------------------------------------ general lattice ----
// Neighbours of a colour class in ELL form: entry k of rank rho at k * n_c + rho (coalesced
// across a warp), in the CSR's order, padded to the class's widest site with entries that
// point at the site itself, so the loads are unconditional and only the sum is predicated.
struct IsingEll {
    uint8_t *sp;  // this replica's spins
    int col_off, n_c, width;
    const int32_t *ell, *ews;  // this class's block: neighbour storage index, table stride
    const uint16_t *deg;       // neighbours per storage index
    const uint16_t *itype;
    const int32_t *type_base, *type_half;
    const uint32_t *tb;  // this replica's temperature slot's thresholds
};

// One site: rank rho.  Threshold-table index = sum of stride * up-spin over the neighbours;
// the draw is halfword rho & 7 of the Philox block of group rho >> 3, and on a tie the
// same halfword of the group's second block.  W > 0: the class's ELL width, known at compile
// time (every load of the site issued at once); W = 0: A.width at run time.
template <int W = 0>
__device__ __forceinline__ bool ising_ell_site(const IsingEll &A, int rho, uint32_t t, uint32_t stream,
                                               uint32_t c3, uint32_t seed) {
    const int s = A.col_off + rho;
    const int dg = A.deg[s];
    int idx = 0;
    if constexpr (W > 0) {
        // the neighbours' storage indices, then all their spins, then the index sum
        int nb[W];
#pragma unroll
        for (int k = 0; k < W; ++k) nb[k] = A.ell[k * A.n_c + rho];  // ELL blocks hold < 2^31 entries
        int up[W];
#pragma unroll
        for (int k = 0; k < W; ++k) up[k] = A.sp[nb[k]];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int w = A.ews[k * A.n_c + rho];
            if (k < dg) idx += w * up[k];
        }
    } else {
#pragma unroll 6
        for (int k = 0; k < A.width; ++k) {
            const int e = k * A.n_c + rho;
            const int up = A.sp[A.ell[e]];
            const int w = A.ews[e];
            if (k < dg) idx += w * up;
        }
    }
    const int own = A.sp[s];
    const int ty = A.itype[s];
    const uint32_t T = A.tb[A.type_base[ty] + own * A.type_half[ty] + idx];
    const uint32_t g = (uint32_t)rho >> 3;
    const int j = rho & 7;
    const U4 hi = draw(g, t, stream, c3, seed);
    const uint32_t uh = half_of(hi, j), th = T >> 16;
    bool flip = uh < th;
    if (uh == th) {
        const U4 lo = draw(g, t, stream, c3 | (1u << 16), seed);
        flip = half_of(lo, j) <= (T & 0xFFFFu);
    }
    if (flip) A.sp[s] = (uint8_t)(own ^ 1);
    return flip;
}

// ------------------------------------------------------- simple cubic, colour-split ----
// Colour c array: rho = (z*L2 + y)*H + xh, H = L1/2, site x = 2*xh + ((y+z+c)&1).
// All six neighbours live in the other colour's array: same xh in rows (y±1,z), (y,z±1),
// and xh, xh∓1 in row (y,z).  A thread takes W (4, 8 or 16) consecutive bytes of one row
// (W | H): half of a random-number group, one or two.  Byte sums of 0/1 spins never carry
// (max 6); the table indices e = n + 7 s (<= 13) are formed for four sites at once.
template <int W>
struct Vec {
    uint32_t w[W / 4];
};

template <int W>
__device__ __forceinline__ Vec<W> ldv(const uint8_t *p) {
    Vec<W> v;
    if constexpr (W == 4) {
        v.w[0] = *reinterpret_cast<const uint32_t *>(p);
    } else if constexpr (W == 8) {
        uint2 q = *reinterpret_cast<const uint2 *>(p);
        v.w[0] = q.x; v.w[1] = q.y;
    } else {
        uint4 q = *reinterpret_cast<const uint4 *>(p);
        v.w[0] = q.x; v.w[1] = q.y; v.w[2] = q.z; v.w[3] = q.w;
    }
    return v;
}
template <int W>
__device__ __forceinline__ void stv(uint8_t *p, const Vec<W> &v) {
    if constexpr (W == 4) {
        *reinterpret_cast<uint32_t *>(p) = v.w[0];
    } else if constexpr (W == 8) {
        *reinterpret_cast<uint2 *>(p) = make_uint2(v.w[0], v.w[1]);
    } else {
        *reinterpret_cast<uint4 *>(p) = make_uint4(v.w[0], v.w[1], v.w[2], v.w[3]);
    }
}

// Thresholds of a replica, in shared memory.  The decision is taken for two sites at once: one
// 32-bit load, indexed by the two sites' e = n + 7 s (n up neighbours, s the own spin;
// e <= 13), gives both thresholds' high halves, packed as the random halves are:
// pair[14 e0 + e1] = (T[e1] >> 16) << 16 | T[e0] >> 16 (e0: the site in the low halfword);
// thr[e] = the whole T (for the rare ties).  At T_c the 32 lanes' loads take 2.5 wavefronts on
// average with the row length 14, 3.4 with 16 (bank = index mod 32; counted on a 64^3
// configuration).
struct ScTab {
    const uint32_t *pair;  // kPairEntries words
    const uint32_t *thr;   // 14 words
};
constexpr int kPairEntries = 14 * 14;
constexpr int kScTabWords = kPairEntries + 14;

// Fills a replica's table (kScTabWords words at tab) from its 14 thresholds in global memory;
// the caller synchronises the n threads.
__device__ __forceinline__ void fill_sc_table(const uint32_t *__restrict__ thr, uint32_t *tab, int tid, int n) {
    for (int i = tid; i < kScTabWords; i += n) {
        const int e0 = i / 14, e1 = i - 14 * e0;
        tab[i] = e0 < 14 ? (thr[e0] >> 16) | (thr[e1] & 0xFFFF0000u) : thr[e1];
    }
}
__device__ __forceinline__ ScTab sc_tab(const uint32_t *tab) { return ScTab{tab, tab + kPairEntries}; }

// The eight sites of a random-number group whose high random halves tie with their
// threshold's high half: decided by the low halves (block 1 of the group).  E0, E1: bytewise
// table indices of the group's two words.  Returns the XOR masks of the extra flips (word 0 in
// the low half of the result).  Kept out of line: it runs for about one vector in 2000 and
// must not cost the hot loop registers.
__device__ __noinline__ inline uint64_t resolve_ties(uint32_t grp, uint32_t t, uint32_t stream, uint32_t c3,
                                                     uint32_t seed, uint32_t E0, uint32_t E1, const uint32_t *thr) {
    const U4 rh = draw(grp, t, stream, c3, seed);
    uint32_t tie = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t T = thr[((k < 4 ? E0 : E1) >> (8 * (k & 3))) & 15u];
        if (half_of(rh, k) == T >> 16) tie |= 1u << k;
    }
    if (!tie) return 0;
    const U4 rl = draw(grp, t, stream, c3 | (1u << 16), seed);
    uint64_t m = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t T = thr[((k < 4 ? E0 : E1) >> (8 * (k & 3))) & 15u];
        if (((tie >> k) & 1u) && half_of(rl, k) <= (T & 0xFFFFu)) m |= 1ull << (8 * k);
    }
    return m;
}

struct IsingSc {
    uint8_t *own_a;       // this replica's array of the updated colour
    const uint8_t *opp;   // ... and of the other colour
    int L1, L2, L3, H;
    FastDiv fH, fL2;
    uint32_t colour;
};

// Halfword-wise floor((t + ~u) / 2): (t & ~u) + ((t ^ ~u) >> 1), no carry crosses the halves.
// The logic operations are explicit: the compiler complements u on its own otherwise (five
// instructions instead of three).
__device__ __forceinline__ uint32_t havg2_not(uint32_t t, uint32_t u) {
    uint32_t a, b;
    asm("lop3.b32 %0, %1, %2, 0, 0x30;" : "=r"(a) : "r"(t), "r"(u));
    asm("lop3.b32 %0, %1, %2, %3, 0x82;" : "=r"(b) : "r"(t), "r"(u), "r"(0xFFFEFFFEu));
    return a + (b >> 1);
}
// prmt with sign replication: byte i of the result is 0xFF if bit 7 of the selected byte is set.
__device__ __forceinline__ uint32_t sign_bytes(uint32_t a, uint32_t b) {
    uint32_t r;  // bytes 1, 3 of a, then 1, 3 of b
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(0xFDB9u));
    return r;
}

// The decisions of one W-byte vector (sites rho0 .. rho0+W-1 of the updated colour) from its
// own spins `me` and the bytewise up-neighbour counts n; returns the new spins and adds the
// flips to cnt as -1 per flip and byte lane (flip_bytes turns the sum into bytewise counts).
// Two sites per step: with t their thresholds' high halves and u their random halves, bit 15
// of each half of d = floor((t + ~u) / 2) is u < t, and t == u gives d = 0x7FFF (so does
// t == u - 1): the minimum over the vector of d + 0x8001 mod 2^16 is zero iff some site may
// tie (probability 2^-15 each), and only then the words are looked at again by resolve_ties.
// Bound: ALU and FMA-heavy pipes.  Against one site at a time (a threshold load, an extracted
// half, two compares and a predicated OR per site: 22.7 instructions per update) this takes
// about half the instructions; 64^3 x 1024 replicas: see ising_sc_kernel.
// block(g) is the draw of the vector's group g (first block); ising_sc_decide makes it in place.
template <int W, class Block>
__device__ __forceinline__ Vec<W> ising_sc_decide_by(const Vec<W> &me, const Vec<W> &n, int rho0, const ScTab &tab,
                                                     uint32_t t, uint32_t stream, uint32_t c3, uint32_t seed,
                                                     const Block &block, uint32_t &cnt) {
    constexpr int NW = W / 4;
    Vec<W> out;
    uint32_t E[NW];
    const char *pair = reinterpret_cast<const char *>(tab.pair);
    uint32_t near = 0xFFFFFFFFu;
    U4 rh{0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < NW; ++q) {
        // word q's half of its group's block: q & 1, or for W = 4 the vector's own half
        const int odd = W == 4 ? (rho0 >> 2) & 1 : q & 1;
        if (W == 4 || (q & 1) == 0) rh = block(q >> 1);
        // byte offsets 56 e0 + 4 e1 of the pairs (0, 1) and (2, 3) by one byte dot product each
        E[q] = me.w[q] * 7u + n.w[q];
        const uint32_t t01 = *reinterpret_cast<const uint32_t *>(pair + __dp4a(E[q], 0x00000438u, 0u));
        const uint32_t t23 = *reinterpret_cast<const uint32_t *>(pair + __dp4a(E[q], 0x04380000u, 0u));
        const uint32_t d01 = havg2_not(t01, odd ? rh.z : rh.x), d23 = havg2_not(t23, odd ? rh.w : rh.y);
        near = __viaddmin_u16x2(d01, 0x80018001u, near);
        near = __viaddmin_u16x2(d23, 0x80018001u, near);
        const uint32_t m = sign_bytes(d01, d23);
        out.w[q] = me.w[q] ^ (m & 0x01010101u);
        cnt += m;
    }
    if ((near & 0xFFFFu) == 0 || near < 0x10000u) {
        if constexpr (W == 4) {  // the vector is one half of its group; the other is not ours
            const int odd = (rho0 >> 2) & 1;
            const uint64_t m2 = resolve_ties((uint32_t)(rho0 >> 3), t, stream, c3, seed, E[0], E[0], tab.thr);
            const uint32_t m = odd ? (uint32_t)(m2 >> 32) : (uint32_t)m2;
            out.w[0] ^= m;
            cnt += 255u * m;
        } else {
#pragma unroll
            for (int q = 0; q < NW; q += 2) {
                const uint64_t m2 = resolve_ties((uint32_t)((rho0 >> 3) + (q >> 1)), t, stream, c3, seed, E[q],
                                                 E[q + 1], tab.thr);
                out.w[q] ^= (uint32_t)m2;
                out.w[q + 1] ^= (uint32_t)(m2 >> 32);
                cnt += 255u * ((uint32_t)m2 + (uint32_t)(m2 >> 32));
            }
        }
    }
    return out;
}
template <int W>
__device__ __forceinline__ Vec<W> ising_sc_decide(const Vec<W> &me, const Vec<W> &n, int rho0, const ScTab &tab,
                                                  uint32_t t, uint32_t stream, uint32_t c3, uint32_t seed,
                                                  const RoundKeys &K, uint32_t &cnt) {
    return ising_sc_decide_by<W>(
        me, n, rho0, tab, t, stream, c3, seed,
        [&](int g) { return draw_rk((uint32_t)((rho0 >> 3) + g), t, stream, c3, K); }, cnt);
}

// Bytewise flip counts from ising_sc_decide's sum: that sum is 255 times the counts' word
// modulo 2^32, and 255 * 0x01010101 = -1 there.
__device__ __forceinline__ uint32_t flip_bytes(uint32_t cnt) { return 0u - cnt * 0x01010101u; }

// Window of the x neighbours of a vector of the other colour's same row: parity 0 takes the
// byte before each site (x-1 -> xh-1), parity 1 the byte after it.
template <int W>
__device__ __forceinline__ uint32_t sc_side(const Vec<W> &o, uint32_t edge, int par, int q) {
    constexpr int NW = W / 4;
    if (par == 0) {
        const uint32_t lo = (q == 0) ? (edge << 24) : o.w[q > 0 ? q - 1 : 0];
        return __funnelshift_l(lo, o.w[q], 8);
    }
    const uint32_t hi = (q == NW - 1) ? edge : o.w[q < NW - 1 ? q + 1 : q];
    return __funnelshift_r(o.w[q], hi, 8);
}

// The update of one W-byte vector from the six neighbour words of the other colour.
template <int W>
__device__ __forceinline__ Vec<W> ising_sc_update(const Vec<W> &me, const Vec<W> &o0, const Vec<W> &a,
                                                  const Vec<W> &b, const Vec<W> &c, const Vec<W> &d,
                                                  uint32_t edge, int par, int rho0, const ScTab &tab,
                                                  uint32_t t, uint32_t stream, uint32_t c3, uint32_t seed,
                                                  const RoundKeys &K, uint32_t &cnt) {
    Vec<W> n;
#pragma unroll
    for (int q = 0; q < W / 4; ++q)
        n.w[q] = o0.w[q] + sc_side<W>(o0, edge, par, q) + a.w[q] + b.w[q] + c.w[q] + d.w[q];
    return ising_sc_decide<W>(me, n, rho0, tab, t, stream, c3, seed, K, cnt);
}

// VPT vectors of W bytes per thread, vector indices vfirst + j*vstride (j < VPT, < nvec),
// one after another, loaded from global memory.  Returns the flips as bytewise counts (each
// byte <= NW VPT).
template <int W, int VPT>
__device__ __forceinline__ uint32_t ising_sc_vectors(const IsingSc &A, int vfirst, int vstride,
                                                     int nvec, const ScTab &tab, uint32_t t,
                                                     uint32_t stream, uint32_t c3, uint32_t seed,
                                                     const RoundKeys &K) {
    static_assert(W == 4 || W == 8 || W == 16, "vector of half, one or two random-number groups");
    const int H = A.H, L2 = A.L2, L3 = A.L3;
    uint32_t cnt = 0;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
        const int v = vfirst + j * vstride;
        if (v >= nvec) break;
        const int rho0 = v * W;
        const int row = (int)fdiv((uint32_t)rho0, A.fH);
        const int xh0 = rho0 - row * H;
        const int z = (int)fdiv((uint32_t)row, A.fL2);
        const int y = row - z * L2;
        const int par = (y + z + (int)A.colour) & 1;
        const int ym = (y == 0 ? L2 - 1 : y - 1), yp = (y == L2 - 1 ? 0 : y + 1);
        const int zm = (z == 0 ? L3 - 1 : z - 1), zp = (z == L3 - 1 ? 0 : z + 1);
        const Vec<W> me = ldv<W>(A.own_a + rho0);
        const Vec<W> o0 = ldv<W>(A.opp + rho0);
        const Vec<W> a = ldv<W>(A.opp + (z * L2 + ym) * H + xh0);
        const Vec<W> b = ldv<W>(A.opp + (z * L2 + yp) * H + xh0);
        const Vec<W> c = ldv<W>(A.opp + (zm * L2 + y) * H + xh0);
        const Vec<W> d = ldv<W>(A.opp + (zp * L2 + y) * H + xh0);
        const uint32_t edge = par == 0 ? A.opp[row * H + (xh0 == 0 ? H - 1 : xh0 - 1)]
                                       : A.opp[row * H + (xh0 + W == H ? 0 : xh0 + W)];
        const Vec<W> out = ising_sc_update<W>(me, o0, a, b, c, d, edge, par, rho0, tab, t, stream,
                                              c3, seed, K, cnt);
        stv<W>(A.own_a + rho0, out);
    }
    return flip_bytes(cnt);
}

// A pair of vectors: the same (y, xh) in the planes z0 and z0 + 1 (z0 even; every extent of
// these lattices is even).  Of the two vectors the one whose sites have their x neighbours at
// xh-1 (parity y + z + colour even) comes first on every lane, so the window shift is the
// same for the whole warp, each of the two serves the other as one z neighbour (ten vector
// loads for two vectors instead of twelve), and the index arithmetic is done once for 2 W
// sites.  Offsets are unsigned, so that the loads take them beside the replica's uniform base
// address.  The loads are a step of their own, so that a kernel can issue them before it has
// its thresholds.
template <int W>
struct ScPair {
    Vec<W> meA, meB, o0A, o0B, aA, aB, bA, bB, uA, uB;
    uint32_t eA, eB, oA, oB;
};
template <int W>
__device__ __forceinline__ ScPair<W> sc_pair_load(const IsingSc &A, int p) {
    const uint32_t H = A.H, L2 = A.L2, L3 = A.L3;
    const uint32_t plane = L2 * H;
    const uint8_t *const own = A.own_a;
    const uint8_t *const opp = A.opp;
    const uint32_t pos = (uint32_t)p * W;
    const uint32_t row = fdiv(pos, A.fH);
    const uint32_t xh0 = pos - row * H;
    const uint32_t zp = fdiv(row, A.fL2);
    const uint32_t y = row - zp * L2;
    const bool pz = (y + A.colour) & 1u;  // parity of plane z0 = 2 zp: the first vector lies in z0 + pz
    const uint32_t base = pos + zp * plane;  // (2 zp L2 + y) H + xh0
    const uint32_t oA = base + (pz ? plane : 0u), oB = base + (pz ? 0u : plane);
    const uint32_t below = base + (zp == 0 ? (L3 - 1) * plane : 0u - plane);
    const uint32_t above = base + (2 * zp + 2 == L3 ? (2 - L3) * plane : 2 * plane);
    const uint32_t dym = y == 0 ? plane - H : 0u - H, dyp = y == L2 - 1 ? H - plane : H;
    ScPair<W> I;
    I.oA = oA;
    I.oB = oB;
    I.o0A = ldv<W>(opp + oA);
    I.o0B = ldv<W>(opp + oB);
    I.aA = ldv<W>(opp + (oA + dym));
    I.aB = ldv<W>(opp + (oB + dym));
    I.bA = ldv<W>(opp + (oA + dyp));
    I.bB = ldv<W>(opp + (oB + dyp));
    I.uA = ldv<W>(opp + (pz ? above : below));
    I.uB = ldv<W>(opp + (pz ? below : above));
    I.eA = opp[oA + (xh0 == 0 ? H - 1 : ~0u)];
    I.eB = opp[oB + (xh0 + W == H ? W - H : (uint32_t)W)];
    I.meA = ldv<W>(own + oA);
    I.meB = ldv<W>(own + oB);
    return I;
}
// Decides and stores both vectors; adds the flips to cnt as ising_sc_decide does.
template <int W>
__device__ __forceinline__ void sc_pair_update(const IsingSc &A, const ScPair<W> &I, const ScTab &tab, uint32_t t,
                                               uint32_t stream, uint32_t c3, uint32_t seed, const RoundKeys &K,
                                               uint32_t &cnt) {
    Vec<W> nA, nB;
#pragma unroll
    for (int q = 0; q < W / 4; ++q) {
        const uint32_t both = I.o0A.w[q] + I.o0B.w[q];
        nA.w[q] = both + sc_side<W>(I.o0A, I.eA, 0, q) + I.aA.w[q] + I.bA.w[q] + I.uA.w[q];
        nB.w[q] = both + sc_side<W>(I.o0B, I.eB, 1, q) + I.aB.w[q] + I.bB.w[q] + I.uB.w[q];
    }
    stv<W>(A.own_a + I.oA, ising_sc_decide<W>(I.meA, nA, (int)I.oA, tab, t, stream, c3, seed, K, cnt));
    stv<W>(A.own_a + I.oB, ising_sc_decide<W>(I.meB, nB, (int)I.oB, tab, t, stream, c3, seed, K, cnt));
}

// Sum of the four byte lanes (each <= 255).
__device__ __forceinline__ unsigned byte_sum(uint32_t cnt) {
    const uint32_t x = (cnt & 0x00FF00FFu) + ((cnt >> 8) & 0x00FF00FFu);
    return (x & 0xFFFFu) + (x >> 16);
}

}  // namespace ether
