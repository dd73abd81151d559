// k_ising.cu -- per-context launches of the Ising colour phase (bodies in sweep_ising.cuh).
#include <algorithm>

#include "measure.cuh"
#include "shared_limit.h"
#include "sweep_ising.cuh"

namespace ether {

// General lattice.  One thread = one group of eight consecutive ranks of the colour class
// (one random-number group).  Neighbours come from the class's ELL block, entry k of rank rho
// at k * n_c + rho: the eight ranks' entries are adjacent and a warp's are contiguous.  The
// neighbour loads are unconditional (padding entries point at valid memory); the threshold
// index idx = sum of stride * up-spin over the site's own entries.  The decision is
// ising_ell_site's: same draws, same thresholds.
__global__ void __launch_bounds__(256)
ising_ell_kernel(uint8_t *__restrict__ spins, int N, int col_off, int n_c, uint32_t colour,
                 const int32_t *__restrict__ ell, const int32_t *__restrict__ ews,
                 const uint16_t *__restrict__ deg, int width, const uint16_t *__restrict__ itype,
                 const int32_t *__restrict__ type_base, const int32_t *__restrict__ type_half,
                 const uint32_t *__restrict__ thr, int table_entries,
                 const int32_t *__restrict__ slot_of_rep, const uint32_t *__restrict__ stream_id,
                 const uint32_t *__restrict__ step, uint32_t ahead, uint32_t seed,
                 unsigned long long *__restrict__ acc_count) {
    const int r = blockIdx.y;
    uint8_t *sp = spins + (size_t)r * N;
    const uint32_t *tb = thr + (size_t)slot_of_rep[r] * table_entries;
    const uint32_t stream = stream_id[r], t = step[r] + ahead;
    const uint32_t c3 = kMetro | (colour << 8);
    const int ng = (n_c + 7) >> 3;
    unsigned acc = 0;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x) {
        const int rho0 = 8 * g;
        int idx[8], dg[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            idx[j] = 0;
            dg[j] = rho0 + j < n_c ? (int)deg[col_off + rho0 + j] : 0;
        }
#pragma unroll 2
        for (int k = 0; k < width; ++k) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int rho = min(rho0 + j, n_c - 1);
                const int e = k * n_c + rho;  // ELL blocks hold < 2^31 entries (checked at creation)
                const int up = sp[ell[e]];
                const int w = ews[e];
                if (k < dg[j]) idx[j] += w * up;
            }
        }
        const U4 hi = draw((uint32_t)g, t, stream, c3, seed);
        bool have_lo = false;
        U4 lo{0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int rho = rho0 + j;
            if (rho >= n_c) break;
            const int s = col_off + rho;
            const int own = sp[s];
            const int ty = itype[s];
            const uint32_t T = tb[type_base[ty] + own * type_half[ty] + idx[j]];
            const uint32_t uh = half_of(hi, j), th = T >> 16;
            bool flip = uh < th;
            if (uh == th) {
                if (!have_lo) {
                    lo = draw((uint32_t)g, t, stream, c3 | (1u << 16), seed);
                    have_lo = true;
                }
                flip = half_of(lo, j) <= (T & 0xFFFFu);
            }
            if (flip) {
                sp[s] = (uint8_t)(own ^ 1);
                ++acc;
            }
        }
    }
    warp_add_count(acc_count + r, acc);
}

// The same update with one site per thread, for colour classes too small to fill the GPU
// with groups of eight: every lane draws its group's Philox block itself (the draws, and so
// the decisions, are those of ising_ell_kernel).  W: the class's ELL width at compile time
// (0: at run time).
template <int W>
__global__ void __launch_bounds__(256)
ising_ell_site_kernel(uint8_t *__restrict__ spins, int N, int col_off, int n_c, uint32_t colour,
                      const int32_t *__restrict__ ell, const int32_t *__restrict__ ews,
                      const uint16_t *__restrict__ deg, int width, const uint16_t *__restrict__ itype,
                      const int32_t *__restrict__ type_base, const int32_t *__restrict__ type_half,
                      const uint32_t *__restrict__ thr, int table_entries,
                      const int32_t *__restrict__ slot_of_rep, const uint32_t *__restrict__ stream_id,
                      const uint32_t *__restrict__ step, uint32_t ahead, uint32_t seed,
                      unsigned long long *__restrict__ acc_count) {
    const int r = blockIdx.y;
    uint8_t *sp = spins + (size_t)r * N;
    const uint32_t *tb = thr + (size_t)slot_of_rep[r] * table_entries;
    const uint32_t stream = stream_id[r], t = step[r] + ahead;
    const uint32_t c3 = kMetro | (colour << 8);
    unsigned acc = 0;
    const IsingEll A{sp, col_off, n_c, width, ell, ews, deg, itype, type_base, type_half, tb};
    for (int rho = blockIdx.x * blockDim.x + threadIdx.x; rho < n_c; rho += gridDim.x * blockDim.x)
        acc += ising_ell_site<W>(A, rho, t, stream, c3, seed) ? 1u : 0u;
    warp_add_count(acc_count + r, acc);
}

// One colour phase.  VPT = 1: one vector per thread; VPT = 2, 4, 8: that many / 2 pairs of
// vectors (sc_pair_update).  MINB = 4 caps the registers at 64, four blocks per SM.
// 64^3 x 1024 replicas at T_c, VPT = 8: 91 us per phase, 1471 updates/ns = 0.65 of the measured
// copy rate at 3 bytes per update (115 us, 1120 updates/ns before two sites shared a decision
// and two planes a thread); 16.1 instructions per update instead of 22.7, FMA-heavy pipe 62%,
// ALU 58%, shared/L1 pipe 58%, so what is left is latency between them.  Measured and not
// kept: register prefetch of the next pair (1186-1300: spills or too few warps), L2 bulk
// prefetch of a later block's planes (+2%), marching up z with x neighbours from lane shuffles
// (1311: fewer L1 wavefronts, more instructions).
template <int W, int VPT, int MINB>
__global__ void __launch_bounds__(256, MINB)
ising_sc_kernel(uint8_t *__restrict__ spins, int L1, int L2, int L3, FastDiv fH, FastDiv fL2,
                uint32_t colour, const uint32_t *__restrict__ thr, int table_entries,
                const int32_t *__restrict__ slot_of_rep, const uint32_t *__restrict__ stream_id,
                const uint32_t *__restrict__ step, uint32_t ahead, uint32_t seed, const RoundKeys K,
                unsigned long long *__restrict__ acc_count) {
    const int r = blockIdx.y;
    const int H = L1 >> 1;
    const int half = H * L2 * L3;
    __shared__ uint32_t s_tab[kScTabWords];
    const IsingSc A{spins + (size_t)r * 2 * half + (size_t)colour * half,
                    spins + (size_t)r * 2 * half + (size_t)(colour ^ 1u) * half,
                    L1, L2, L3, H, fH, fL2, colour};
    const uint32_t c3 = kMetro | (colour << 8);
    const uint32_t t = step[r] + ahead, stream = stream_id[r];
    uint32_t cnt = 0;
    if constexpr (VPT == 1) {
        fill_sc_table(thr + (size_t)slot_of_rep[r] * table_entries, s_tab, threadIdx.x, 256);
        __syncthreads();
        cnt = ising_sc_vectors<W, 1>(A, blockIdx.x * 256 + threadIdx.x, 256, half / W, sc_tab(s_tab), t, stream, c3,
                                     seed, K);
    } else {
        constexpr int NP = VPT / 2;
        const int npair = half / (2 * W);
        int p = blockIdx.x * NP * 256 + threadIdx.x;
        // the first pair's loads are in flight while the block fills its table
        ScPair<W> I = sc_pair_load<W>(A, min(p, npair - 1));
        fill_sc_table(thr + (size_t)slot_of_rep[r] * table_entries, s_tab, threadIdx.x, 256);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NP; ++j, p += 256) {
            if (p >= npair) break;
            if (j) I = sc_pair_load<W>(A, p);
            sc_pair_update<W>(A, I, sc_tab(s_tab), t, stream, c3, seed, K, cnt);
        }
        cnt = flip_bytes(cnt);
    }
    warp_add_count(acc_count + r, byte_sum(cnt));
}

// The variants 401x .. 404x name a form whose neighbour planes are staged in shared memory: it
// was 30% slower than the phase kernel and runs as one now; the lattices it took stay the same
// (H = L1 / 2 a power of two >= 16, a 4096 vs byte step dividing the colour array, a ring of at
// most 160 KB).
bool ising_staged_shape(const Ctx &c, int vs) {
    const int H = c.L[0] / 2;
    if (!c.fast || c.model != ETHER_MODEL_ISING || H < 16 || H > 4096 || (H & (H - 1))) return false;
    const int S = vs * 4096 / H, rows = c.L[1] * c.L[2];
    if (S < 1 || rows % S || (256 % (H / 16) && H < 4096)) return false;
    const int h = (2 * c.L[1] + S - 1) / S;
    int P = 4;
    while (P < h + 3) P *= 2;
    return (long)P * S * H <= 160 * 1024;
}

template <int W, int VPT, int MINB>
static void launch_sc(Ctx &c, int colour) {
    const int bs = 256;
    const int nvec = (c.N / 2) / W;  // even: every extent is
    dim3 grid((nvec + bs * VPT - 1) / (bs * VPT), c.R);
    ising_sc_kernel<W, VPT, MINB><<<grid, bs, 0, c.stream>>>(
        c.spins, c.L[0], c.L[1], c.L[2], make_fastdiv((uint32_t)(c.L[0] / 2)),
        make_fastdiv((uint32_t)c.L[1]), (uint32_t)colour, c.thr, c.table_entries, c.slot_of_rep,
        c.stream_id, c.step, c.ahead, c.seed, round_keys(c.seed), c.acc_count);
}

static int blocks_for(const Ctx &c, long work, int bs) {
    long need = (work + bs - 1) / bs;
    long cap = (long)c.sm_count * 8 / (c.R > 0 ? c.R : 1);
    if (cap < 1) cap = 1;
    if (need > cap) need = cap;
    if (need < 1) need = 1;
    return (int)need;
}

// Resident forms for small simple-cubic lattices: one block per replica holds both colour
// arrays in shared memory and runs nsweeps whole sweeps (colour 0, colour 1, counter + 1)
// between two visits to global memory.  The draws, thresholds and vector update are the
// phase kernels', so every decision is the same; the sweep counter is advanced here instead of
// by advance_kernel.
struct ResidentIsing {
    uint8_t *spins;
    int L1, L2, L3;
    FastDiv fH, fL2;
    const uint32_t *thr;
    int table_entries;
    const int32_t *slot_of_rep;
    const uint32_t *stream_id;
    uint32_t *step;
    uint32_t seed;
    RoundKeys K;
    int nsweeps;
    unsigned long long *acc_count;
    double invN;
    ResidentEvents ev;
    // measurements
    int N, R, nblk, n_slots, zeeman;
    double juni, mw_abs;
    const double *zeed;
    double *E, *M, *sums;
};
constexpr int kMeasureBlocks = 32;  // partial sums a measuring launch can keep

__device__ __forceinline__ void resident_load(const ResidentIsing &P, uint8_t *s_sp, uint32_t *s_tab, unsigned *s_acc) {
    const int r = blockIdx.x, n16 = (P.L1 * P.L2 * P.L3) >> 4;  // W | H and the even extents: whole
    const uint4 *g = reinterpret_cast<const uint4 *>(P.spins) + (size_t)r * n16;
    for (int i = threadIdx.x; i < n16; i += blockDim.x) reinterpret_cast<uint4 *>(s_sp)[i] = g[i];
    fill_sc_table(P.thr + (size_t)P.slot_of_rep[r] * P.table_entries, s_tab, threadIdx.x, blockDim.x);
    if (threadIdx.x == 0) *s_acc = 0;
    __syncthreads();
}
__device__ __forceinline__ void resident_store(const ResidentIsing &P, const uint8_t *s_sp, unsigned *s_acc,
                                               unsigned flips, uint32_t t0) {
    const int r = blockIdx.x, n16 = (P.L1 * P.L2 * P.L3) >> 4;
    uint4 *g = reinterpret_cast<uint4 *>(P.spins) + (size_t)r * n16;
    for (int i = threadIdx.x; i < n16; i += blockDim.x) g[i] = reinterpret_cast<const uint4 *>(s_sp)[i];
    flips = __reduce_add_sync(0xffffffffu, flips);
    if ((threadIdx.x & 31) == 0) atomicAdd(s_acc, flips);
    __syncthreads();
    if (threadIdx.x == 0) {
        P.step[r] = t0 + (uint32_t)P.nsweeps;
        P.acc_count[r] += *s_acc;
        if (P.ev.ratio) P.ev.ratio[r] = (double)*s_acc * P.invN;
    }
}

// The energy and the magnetisation of the replica from the counts of its energy blocks, in the
// division and the order of energy_mag_kernel and its finish (whose tree over 128 slots is this
// one over the first 32: the others hold zeros), by the first warp; measure: into the sums too.
__device__ __forceinline__ void resident_measure(const ResidentIsing &P, int (*cnt)[2], bool measure) {
    const int r = blockIdx.x, lane = threadIdx.x;
    double q[3] = {0.0, 0.0, 0.0};  // total energy, exchange energy, M_z
    if (lane < P.nblk) {
        const int t0 = cnt[lane][0], t1 = cnt[lane][1];
        cnt[lane][0] = cnt[lane][1] = 0;
        const double e_ex = P.juni * (double)t0;
        q[0] = P.zeeman ? e_ex + P.zeed[2] * (double)t1 : e_ex;
        q[1] = e_ex;
        q[2] = P.mw_abs * (double)t1;
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1)
#pragma unroll
        for (int j = 0; j < 3; ++j) q[j] += __shfl_down_sync(0xffffffffu, q[j], w);
    if (lane == 0) {
        P.E[r] = q[0];
        P.E[P.R + r] = q[1];
        P.M[3 * r] = P.M[3 * r + 1] = 0.0;
        P.M[3 * r + 2] = q[2];
        if (measure) measure_one(P.E, P.M, P.N, P.n_slots, P.slot_of_rep, P.sums, r);
    }
}

// NV vectors of each colour per thread, kept in registers; shared memory serves the neighbours.
// A half-sweep is a chain: barrier, neighbour loads, table, decision, store, barrier.  The
// addresses are worked out once, the vector opposite is the thread's own of the other colour,
// and the next half-sweep's random numbers are drawn before the barrier that ends this one.
// Measurements (counts of colour 0's bonds, as sc_ising_counts) stay in the launch too, so a run
// ends only where replicas meet.
// (16^3, 190 replicas, per sweep: 1.8 us with the addresses and draws inside the
// chain, 0.90 so; by launches per colour 11.4.  One replica: 0.59 and 11.4.)
template <int W, int NV, bool MEASURE>
__global__ void __launch_bounds__(1024) ising_sc_resident(const ResidentIsing P) {
    extern __shared__ __align__(16) uint8_t s_sp[];  // colour 0 array, then colour 1
    __shared__ uint32_t s_tab[kScTabWords];
    __shared__ unsigned s_acc;
    __shared__ int s_cnt[kMeasureBlocks][2];
    for (int i = threadIdx.x; i < 2 * kMeasureBlocks; i += blockDim.x) (&s_cnt[0][0])[i] = 0;
    constexpr int G = W == 16 ? 2 : 1;  // random-number groups of a vector
    const int H = P.L1 >> 1, L2 = P.L2, L3 = P.L3, half = H * L2 * L3, nvec = half / W;
    const uint32_t stream = P.stream_id[blockIdx.x], t0 = P.step[blockIdx.x];
    int rho[NV], oa[NV], ob[NV], oc[NV], od[NV], e0[NV], e1[NV];
    bool odd[NV], live[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int v = threadIdx.x + j * blockDim.x;
        live[j] = v < nvec;
        rho[j] = live[j] ? v * W : 0;
        const int row = (int)fdiv((uint32_t)rho[j], P.fH), xh = rho[j] - row * H;
        const int z = (int)fdiv((uint32_t)row, P.fL2), y = row - z * L2;
        odd[j] = (y + z) & 1;
        oa[j] = (z * L2 + (y == 0 ? L2 - 1 : y - 1)) * H + xh;
        ob[j] = (z * L2 + (y == L2 - 1 ? 0 : y + 1)) * H + xh;
        oc[j] = ((z == 0 ? L3 - 1 : z - 1) * L2 + y) * H + xh;
        od[j] = ((z == L3 - 1 ? 0 : z + 1) * L2 + y) * H + xh;
        const int before = row * H + (xh == 0 ? H - 1 : xh - 1), after = row * H + (xh + W == H ? 0 : xh + W);
        e0[j] = odd[j] ? after : before;  // colour 0: parity y + z
        e1[j] = odd[j] ? before : after;
    }
    U4 rnd[NV][G];
    auto draws = [&](uint32_t t, uint32_t c3) {
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int g = 0; g < G; ++g) rnd[j][g] = draw_rk((uint32_t)((rho[j] >> 3) + g), t, stream, c3, P.K);
    };
    draws(t0, kMetro);
    resident_load(P, s_sp, s_tab, &s_acc);
    Vec<W> me[2][NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        me[0][j] = ldv<W>(s_sp + rho[j]);
        me[1][j] = ldv<W>(s_sp + half + rho[j]);
    }
    const ScTab tab = sc_tab(s_tab);
    unsigned flips = 0;
    uint32_t cnt = 0;
    for (int k = 0; k < P.nsweeps; ++k) {
        const uint32_t t = t0 + (uint32_t)k;
#pragma unroll
        for (int colour = 0; colour < 2; ++colour) {
            uint8_t *own = s_sp + colour * half;
            const uint8_t *opp = s_sp + (colour ^ 1) * half;
            const uint32_t c3 = kMetro | ((uint32_t)colour << 8);
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                if (!live[j]) continue;
                const Vec<W> &o0 = me[colour ^ 1][j];
                const Vec<W> a = ldv<W>(opp + oa[j]), b = ldv<W>(opp + ob[j]), c = ldv<W>(opp + oc[j]),
                             d = ldv<W>(opp + od[j]);
                const uint32_t edge = opp[colour ? e1[j] : e0[j]];
                const int par = (odd[j] ? 1 : 0) ^ colour;
                Vec<W> n;
#pragma unroll
                for (int q = 0; q < W / 4; ++q)
                    n.w[q] = o0.w[q] + sc_side<W>(o0, edge, par, q) + a.w[q] + b.w[q] + c.w[q] + d.w[q];
                me[colour][j] = ising_sc_decide_by<W>(me[colour][j], n, rho[j], tab, t, stream, c3, P.seed,
                                                      [&](int g) { return rnd[j][g]; }, cnt);
                stv<W>(own + rho[j], me[colour][j]);
            }
            draws(colour ? t + 1u : t, colour ? kMetro : kMetro | (1u << 8));
            __syncthreads();
        }
        // a byte counts at most NV W / 4 <= 8 flips per half-sweep
        if ((k & 7) == 7 || k + 1 == P.nsweeps) {
            flips += byte_sum(flip_bytes(cnt));
            cnt = 0;
        }
        const bool measure = (P.ev.measure[(k >> 5) & 7] >> (k & 31)) & 1u;
        if (MEASURE && (measure || (P.ev.energy && k + 1 == P.nsweeps))) {
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                int sn = 0, ssn = 0, ss = 0, so = 0;
                if (live[j]) {
                    const uint8_t *opp = s_sp + half;
                    const Vec<W> &o0 = me[1][j];
                    const Vec<W> a = ldv<W>(opp + oa[j]), b = ldv<W>(opp + ob[j]), c = ldv<W>(opp + oc[j]),
                                 d = ldv<W>(opp + od[j]);
                    const uint32_t edge = opp[e0[j]];
#pragma unroll
                    for (int q = 0; q < W / 4; ++q) {
                        const uint32_t n = o0.w[q] + sc_side<W>(o0, edge, odd[j] ? 1 : 0, q) + a.w[q] + b.w[q] + c.w[q] + d.w[q];
                        sn = (int)__dp4a(n, 0x01010101u, (uint32_t)sn);
                        ssn = (int)__dp4a(n, me[0][j].w[q], (uint32_t)ssn);
                        ss = (int)__dp4a(me[0][j].w[q], 0x01010101u, (uint32_t)ss);
                        so = (int)__dp4a(o0.w[q], 0x01010101u, (uint32_t)so);
                    }
                }
                const int same = live[j] ? 6 * W - sn + 2 * ssn - 6 * ss : 3 * W;
                const int bonds = __reduce_add_sync(0xffffffffu, 2 * (2 * same - 6 * W));
                const int spins = __reduce_add_sync(0xffffffffu, live[j] ? 2 * (ss + so) - 2 * W : 0);
                if ((threadIdx.x & 31) == 0) {
                    const int blk = ((threadIdx.x + j * blockDim.x) >> 8) % P.nblk;
                    atomicAdd(&s_cnt[blk][0], bonds);
                    atomicAdd(&s_cnt[blk][1], spins);
                }
            }
            __syncthreads();  // the next counts come two barriers later
            if (threadIdx.x < 32) resident_measure(P, s_cnt, measure);
        }
    }
    resident_store(P, s_sp, &s_acc, flips, t0);
}

// More vectors than a block's threads can keep: a loop over them.
template <int W>
__global__ void __launch_bounds__(256) ising_sc_resident_loop(const ResidentIsing P) {
    extern __shared__ __align__(16) uint8_t s_sp[];
    __shared__ uint32_t s_tab[kScTabWords];
    __shared__ unsigned s_acc;
    const int H = P.L1 >> 1, half = H * P.L2 * P.L3, nvec = half / W;
    const uint32_t stream = P.stream_id[blockIdx.x], t0 = P.step[blockIdx.x];
    resident_load(P, s_sp, s_tab, &s_acc);
    unsigned flips = 0;
    for (int k = 0; k < P.nsweeps; ++k) {
        const uint32_t t = t0 + (uint32_t)k;
        for (int colour = 0; colour < 2; ++colour) {
            const IsingSc A{s_sp + (size_t)colour * half, s_sp + (size_t)(colour ^ 1) * half,
                            P.L1, P.L2, P.L3, H, P.fH, P.fL2, (uint32_t)colour};
            uint32_t cnt = 0;
            for (int v = threadIdx.x; v < nvec; v += blockDim.x)
                cnt += ising_sc_vectors<W, 1>(A, v, 0, nvec, sc_tab(s_tab), t, stream, kMetro | ((uint32_t)colour << 8),
                                              P.seed, P.K);
            flips += byte_sum(cnt);  // each byte <= (W / 4) * ceil(nvec / blockDim) per colour
            __syncthreads();
        }
    }
    resident_store(P, s_sp, &s_acc, flips, t0);
}

static long resident_vectors(const Ctx &c, int W) { return (long)c.L[0] * c.L[1] * c.L[2] / 2 / W; }

bool ising_resident_possible(const Ctx &c, size_t smem_max) {
    if (!c.fast || c.model != ETHER_MODEL_ISING || c.vec_bytes == 0) return false;
    const size_t bytes = (size_t)c.L[0] * c.L[1] * c.L[2];  // both colours
    // (W/4) ceil(nvec/256) flips per byte of a vector count must stay below 256
    return bytes <= smem_max && (c.vec_bytes / 4) * ((resident_vectors(c, c.vec_bytes) + 255) / 256) < 256;
}
// Replicas of so few vectors that a phase kernel's blocks mostly fill their table: n sweeps are better
// off in shared memory (a sweep and |M|, shared memory and phases, us: 8^3 x 9000 54.7 and 69.7, x
// 30000 151 and 197, 16 x 8 x 12 x 10000 66 and 87; 16^3 x 4000, 256 vectors, 50 and 50, two sweeps 58
// and 76; 24 x 16 x 16 x 2500, 768, 75 and 51).
bool ising_resident_tiny(const Ctx &c, int n) { return resident_vectors(c, c.vec_bytes) <= (n > 1 ? 256 : 128); }
bool ising_resident_in_registers(const Ctx &c) { return resident_vectors(c, c.vec_bytes) <= 2048; }

// Vectors in registers up to two per thread of the largest block.
using ResidentKernel = void (*)(ResidentIsing);
template <int W, bool MEASURE>
static ResidentKernel resident_kernel(long nvec) {
    return nvec <= 1024 ? ising_sc_resident<W, 1, MEASURE> : nvec <= 2048 ? ising_sc_resident<W, 2, MEASURE> : ising_sc_resident_loop<W>;
}
template <bool MEASURE>
static ResidentKernel resident_kernel(const Ctx &c, int W) {
    const long n = resident_vectors(c, W);
    return W == 16 ? resident_kernel<16, MEASURE>(n) : W == 8 ? resident_kernel<8, MEASURE>(n) : resident_kernel<4, MEASURE>(n);
}

// Opts the kernels of every vector width into shared memory (once, at creation: not during a
// stream capture).
cudaError_t prepare_ising_resident(const Ctx &c) {
    for (int k = 0; k < 6; ++k) {
        const ResidentKernel kern = k & 1 ? resident_kernel<true>(c, 4 << (k >> 1)) : resident_kernel<false>(c, 4 << (k >> 1));
        const cudaError_t e = allow_shared((const void *)kern);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

bool ising_resident_measures(const Ctx &c) {
    return ising_resident_in_registers(c) && ising_counts(c) && c.mw_pos && c.partial_blocks <= kMeasureBlocks;
}

cudaError_t launch_ising_resident(Ctx &c, int nsweeps, const ResidentEvents &ev) {
    const long nvec = resident_vectors(c, c.vec_bytes);
    const int nv = nvec <= 1024 ? 1 : 2;
    const int bs = nvec > 2048 ? 256 : (int)(((nvec + nv - 1) / nv + 31) / 32 * 32);
    const ResidentIsing P{c.spins, c.L[0], c.L[1], c.L[2], make_fastdiv((uint32_t)(c.L[0] / 2)),
                          make_fastdiv((uint32_t)c.L[1]), c.thr, c.table_entries, c.slot_of_rep, c.stream_id, c.step,
                          c.seed, round_keys(c.seed), nsweeps, c.acc_count, 1.0 / (double)c.N, ev,
                          c.N, c.R, c.partial_blocks, c.n_slots, c.zeeman ? 1 : 0, c.ising_juni, c.mw_abs, c.t.zeed,
                          c.E, c.M, c.sums};
    bool measures = ev.energy != 0;
    for (uint32_t m : ev.measure) measures = measures || m != 0;
    const ResidentKernel kern = measures ? resident_kernel<true>(c, c.vec_bytes) : resident_kernel<false>(c, c.vec_bytes);
    kern<<<c.R, bs, c.L[0] * c.L[1] * c.L[2], c.stream>>>(P);
    c.launches++;
    return cudaGetLastError();
}

// Vectors per thread of a simple-cubic context whose variant nobody chose: the most of 8, 4, 2
// that still gives full blocks and six of them per SM (64^3 x 1024: 1471 updates/ns with 8,
// 1433 with 4, 1310 with 2, 917 with 1; 64^3 x 128, where 8 leaves 512 blocks: 935 with 8, 970
// with 4; 16^3 x 1024, where 2 leaves half a block: 230 with 2, 268 with 1).
int ising_default_vpt(const Ctx &c) {
    const long nvec = (long)c.N / 2 / c.vec_bytes;
    for (int v = 8; v > 1; v /= 2)
        if (nvec >= 256L * v && c.R * ((nvec + 256 * v - 1) / (256 * v)) >= 6L * c.sm_count) return v;
    return 1;
}

cudaError_t launch_ising_sweep(Ctx &c, int colour) {
    const int bs = 256;
    if (c.fast) {
        switch (c.vec_bytes * 10 + c.ising_vpt) {
            case 161: launch_sc<16, 1, 1>(c, colour); break;
            case 162: launch_sc<16, 2, 4>(c, colour); break;
            case 164: launch_sc<16, 4, 4>(c, colour); break;
            case 168: launch_sc<16, 8, 4>(c, colour); break;
            case 81: launch_sc<8, 1, 1>(c, colour); break;
            case 82: launch_sc<8, 2, 1>(c, colour); break;
            case 84: launch_sc<8, 4, 1>(c, colour); break;
            case 88: launch_sc<8, 8, 1>(c, colour); break;
            case 41: launch_sc<4, 1, 1>(c, colour); break;
            case 42: launch_sc<4, 2, 1>(c, colour); break;
            case 44: launch_sc<4, 4, 1>(c, colour); break;
            default: launch_sc<4, 8, 1>(c, colour); break;
        }
    } else {
        const int n_c = c.col_off[colour + 1] - c.col_off[colour];
        if (n_c == 0) return cudaSuccess;
        const int32_t *ell = c.t.ell_nbr + c.ell_off[colour];
        const int32_t *ews = c.t.ell_ws + c.ell_off[colour];
        const int r0 = c.rw0, nr = c.rwn ? c.rwn : c.R;  // replica window (the kernel form follows the full R)
        uint8_t *spins = c.spins + (size_t)r0 * c.N;
        const long groups = (long)c.R * ((n_c + 7) / 8);
        if (groups < 2L * c.sm_count * bs) {  // too few groups of eight to fill the GPU
            dim3 grid(blocks_for(c, n_c, bs), nr);
            auto k = ising_ell_site_kernel<0>;
            switch (c.ell_width[colour]) {  // common widths at compile time
                case 4: k = ising_ell_site_kernel<4>; break;
                case 6: k = ising_ell_site_kernel<6>; break;
                case 8: k = ising_ell_site_kernel<8>; break;
                case 12: k = ising_ell_site_kernel<12>; break;
                case 14: k = ising_ell_site_kernel<14>; break;
                case 18: k = ising_ell_site_kernel<18>; break;
                case 24: k = ising_ell_site_kernel<24>; break;
                default: break;
            }
            k<<<grid, bs, 0, c.stream>>>(
                spins, c.N, c.col_off[colour], n_c, (uint32_t)colour, ell, ews, c.t.ell_deg,
                c.ell_width[colour], c.t.itype, c.t.type_base, c.t.type_half, c.thr, c.table_entries,
                c.slot_of_rep + r0, c.stream_id + r0, c.step + r0, c.ahead, c.seed, c.acc_count + r0);
        } else {
            dim3 grid(blocks_for(c, (n_c + 7) / 8, bs), nr);
            ising_ell_kernel<<<grid, bs, 0, c.stream>>>(
                spins, c.N, c.col_off[colour], n_c, (uint32_t)colour, ell, ews, c.t.ell_deg,
                c.ell_width[colour], c.t.itype, c.t.type_base, c.t.type_half, c.thr, c.table_entries,
                c.slot_of_rep + r0, c.stream_id + r0, c.step + r0, c.ahead, c.seed, c.acc_count + r0);
        }
    }
    c.launches++;
    return cudaGetLastError();
}

}  // namespace ether
