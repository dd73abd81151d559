// k_resident.cu -- general lattices whose replicas fit in shared memory: whole runs of Metropolis
// sweeps (src/Metropolis.f90:34-68) without a launch per colour phase.
//
// A cluster of 1, 2 or 4 thread blocks (Ising: 1 or 2, which both hold all spins) holds a replica's spins in shared
// memory and runs nsweeps sweeps with a cluster (block) barrier between colour phases; the spins
// are read from and written to global memory once per run.  Each site's arithmetic, draws and
// neighbour order are the phase kernels' (sweep_ising.cuh, sweep_xyz.cuh), so the results are
// the same bits.
//
// Why: a colour phase of a general lattice is a small dependent launch that waits on scattered
// neighbour reads through the L2 (pyrochlore 12^3 cells x 64 replicas: 8 colours, 221 000 sites
// and 14 us a phase, a tenth of the issue rate, even with four chains of launches side by side).
// In shared memory a neighbour costs a load of some tens of cycles, and a phase ends with a
// barrier.  What does not depend on the spins -- a site's neighbour entries and its random
// numbers -- is fetched and drawn for the thread's next site before the barrier.
//
// Neighbour entries are 16-bit indices, eight to a 16-byte load, coalesced, shared by all
// replicas (L2): slots of shell 0, then of shell 1, ...; a site with fewer neighbours in a
// shell has its free slots point at a spin of zeros, which adds nothing.  The order of a
// site's real neighbours stays the reference's, so one species is required (the coupling then
// depends on the shell alone).
//
// A warp reads the same slot of 32 sites at once; the 16-byte spins of eight lanes cost one
// wavefront where they lie side by side.  On a lattice with a basis the sites of a rank range mix
// the basis, and their neighbours lie scattered; so a block takes and keeps the sites of a colour
// basis by basis (res_arrange: pyrochlore 12^3, 18 slots, 153 -> 100 wavefronts a warp, a third
// fewer warps with a neighbour in the other block; a sweep of 64 replicas 80 -> 64 us).
//
// A cluster divides every colour class evenly by rank; ranks follow the site numbers, so a
// block's share is a slab of the lattice and only the slab's faces read the other blocks'
// shared memory.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <utility>

#include "shared_limit.h"
#include "sweep_ising.cuh"
#include "sweep_xyz.cuh"

namespace ether {

constexpr int kResThreads = 1024;
constexpr int kResMaxQ = 4;      // 16-byte words of entries per site: at most 32 slots
constexpr int kResIdxBits = 14;  // clusters: index in the owning block's array, block above it

struct ResShape {
    int ncol, slots;             // slots: of all shells together
    int off[kMaxColours + 1];    // first storage index of a colour
    int stride[8 * kResMaxQ];    // Ising: stride of a slot's shell in the threshold table
};
// XYZ: the coupling of each slot, a kernel parameter so that every fmaf takes it as a constant.
struct ResCouplings {
    float x[8 * kResMaxQ], y[8 * kResMaxQ], z[8 * kResMaxQ];
};

// ------------------------------------------------------------------------ Ising ----
// One block per replica; a thread takes two neighbouring ranks (one Philox block serves both).
// s_sp[N] is the zero spin.  Threshold-table index = sum over shells of stride * up-spins.
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();  // .aligned: the warp arrives as one
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The block's accepted moves into the replica's counter and, where ratio is given, the whole
// replica's share of its sites into *ratio (the cluster's first block adds up).
template <int CS>
__device__ __forceinline__ void res_accepts(unsigned long long *count, unsigned acc, double invN, double *ratio, int blk) {
    __shared__ unsigned s_acc[32], s_part[4];
    acc = __reduce_add_sync(0xffffffffu, acc);
    if ((threadIdx.x & 31) == 0) s_acc[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) acc += s_acc[w];
        atomicAdd(count, (unsigned long long)acc);
    }
    if (!ratio) return;
    if constexpr (CS > 1) {
        if (threadIdx.x == 0) {
            uint32_t to;
            asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"((uint32_t)__cvta_generic_to_shared(s_part + blk)));
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to), "r"(acc) : "memory");
        }
        cluster_barrier();
        if (blk == 0 && threadIdx.x == 0)
            for (int k = 1; k < CS; ++k) acc += *(volatile unsigned *)(s_part + k);
    }
    if (blk == 0 && threadIdx.x == 0) *ratio = (double)acc * invN;
}

template <int NQ, int CS>
__global__ void __launch_bounds__(kResThreads, 1)
ising_resident_general(uint8_t *__restrict__ spins, int N, const __grid_constant__ ResShape C,
                       const uint4 *__restrict__ ent, const uint16_t *__restrict__ itype,
                       const int32_t *__restrict__ type_base, const int32_t *__restrict__ type_half, int n_types,
                       const uint32_t *__restrict__ thr, int table_entries, const int32_t *__restrict__ slot_of_rep,
                       const uint32_t *__restrict__ stream_id, uint32_t *__restrict__ step, const RoundKeys K,
                       int nsweeps, unsigned long long *__restrict__ acc_count, double invN, double *ratio) {
    extern __shared__ __align__(16) uint8_t s_raw[];
    uint32_t *s_tb = reinterpret_cast<uint32_t *>(s_raw);         // table_entries thresholds
    int2 *s_ty = reinterpret_cast<int2 *>(s_tb + ((table_entries + 1) & ~1));  // per type: base, half
    uint8_t *s_sp = reinterpret_cast<uint8_t *>(s_ty + n_types);
    const int r = blockIdx.x / CS;
    const int blk = CS > 1 ? (int)(blockIdx.x % CS) : 0;
    // the other block's spins, in the cluster window
    uint32_t other = 0;
    if constexpr (CS == 2)
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(other) : "r"((uint32_t)__cvta_generic_to_shared(s_sp)), "r"(blk ^ 1));
    auto barrier = [] {
        if constexpr (CS > 1) cluster_barrier();
        else __syncthreads();
    };
    // this block's pairs of a colour of n sites
    auto share = [&](int n, int &a, int &b) {
        const int pairs = (n + 1) / 2;
        a = pairs * blk / CS;
        b = pairs * (blk + 1) / CS;
    };
    uint8_t *g = spins + (size_t)r * N;
    const uint32_t *tb = thr + (size_t)slot_of_rep[r] * table_entries;
    const uint32_t stream = stream_id[r], t0 = step[r];
    for (int i = threadIdx.x; i < table_entries; i += blockDim.x) s_tb[i] = tb[i];
    for (int i = threadIdx.x; i < n_types; i += blockDim.x) s_ty[i] = make_int2(type_base[i], type_half[i]);
    for (int i = threadIdx.x; i <= N; i += blockDim.x) s_sp[i] = i < N ? g[i] : (uint8_t)0;
    barrier();
    unsigned acc = 0;
    struct Next {  // a pair of sites: what does not depend on the spins
        uint4 e[2][NQ];
        int2 ty[2];
        U4 hi;
    } nx;
    auto fetch = [&](int col, int pair, uint32_t t) {
        const int off = C.off[col], n = C.off[col + 1] - off, rho = 2 * pair;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int s = off + min(rho + j, n - 1);
#pragma unroll
            for (int q = 0; q < NQ; ++q) nx.e[j][q] = ent[(size_t)q * N + s];
            nx.ty[j] = s_ty[itype[s]];
        }
        nx.hi = draw_rk((uint32_t)rho >> 3, t, stream, kMetro | ((uint32_t)col << 8), K);
    };
    int a, b;
    share(C.off[1], a, b);
    if (a + (int)threadIdx.x < b) fetch(0, a + (int)threadIdx.x, t0);
    for (int k = 0; k < nsweeps; ++k) {
        const uint32_t t = t0 + (uint32_t)k;
        for (int col = 0; col < C.ncol; ++col) {
            const int off = C.off[col], n = C.off[col + 1] - off;
            share(n, a, b);
            for (int p = a + (int)threadIdx.x; p < b; p += blockDim.x) {
                if (p != a + (int)threadIdx.x) fetch(col, p, t);
                const int rho = 2 * p;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int s = off + rho + j;
                    if (rho + j >= n) break;
                    // table index: every up spin adds its shell's stride, a constant operand per slot
                    // (a sum per shell with its ends tested took ten instructions a slot: pyrochlore
                    // 6^3 cells, Ising, 17.6 us a sweep; 10.6 so; 21 x 18 x 15 8.0 and 6.5)
                    int idx = 0;
#pragma unroll
                    for (int e = 0; e < NQ; ++e) {
                        if (8 * e >= C.slots) break;  // uniform; also keeps the loads of a word together
                        const uint4 &q = nx.e[j][e];
#pragma unroll
                        for (int m = 0; m < 8; ++m) {
                            const uint32_t w = (m & 6) == 0 ? q.x : (m & 6) == 2 ? q.y : (m & 6) == 4 ? q.z : q.w;
                            idx += (int)s_sp[(m & 1) ? w >> 16 : w & 0xFFFFu] * C.stride[8 * e + m];
                        }
                    }
                    const int own = s_sp[s];
                    const uint32_t T = s_tb[nx.ty[j].x + own * nx.ty[j].y + idx];
                    const uint32_t uh = half_of(nx.hi, (rho + j) & 7), th = T >> 16;
                    bool flip = uh < th;
                    if (uh == th) {
                        const U4 lo = draw_rk((uint32_t)rho >> 3, t, stream,
                                              kMetro | ((uint32_t)col << 8) | (1u << 16), K);
                        flip = half_of(lo, (rho + j) & 7) <= (T & 0xFFFFu);
                    }
                    if (flip) {
                        s_sp[s] = (uint8_t)(own ^ 1);
                        if constexpr (CS == 2)
                            asm volatile("st.shared::cluster.u8 [%0], %1;" ::"r"(other + (uint32_t)s), "r"(own ^ 1) : "memory");
                        ++acc;
                    }
                }
            }
            // the first pair of the next phase
            const int nc = col + 1 < C.ncol ? col + 1 : 0;
            share(C.off[nc + 1] - C.off[nc], a, b);
            if ((nc || k + 1 < nsweeps) && a + (int)threadIdx.x < b) fetch(nc, a + (int)threadIdx.x, nc ? t : t + 1);
            barrier();
        }
    }
    for (int i = blk * (int)blockDim.x + (int)threadIdx.x; i < N; i += CS * blockDim.x) g[i] = s_sp[i];
    if (blk == 0 && threadIdx.x == 0) step[r] = t0 + (uint32_t)nsweeps;
    res_accepts<CS>(acc_count + r, acc, invN, ratio ? ratio + r : nullptr, (int)blk);
}

// -------------------------------------------------------------------------- XYZ ----
// The spin of a 16-bit entry: index i in block blk of the cluster.  base: this block's array in
// the shared window; first, delta: the first block's in the cluster window, the distance to the
// second's.
__device__ __forceinline__ float4 ld_own(uint32_t base, uint32_t i) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(base + i * 16u) : "memory");
    return v;
}
template <int CS>
__device__ __forceinline__ float4 ld_cluster(uint32_t base, uint32_t first, uint32_t delta, uint32_t i, uint32_t blk) {
    float4 v;
    uint32_t a;
    if constexpr (CS == 2) a = first + i * 16u + blk * delta;
    else asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(base + i * 16u), "r"(blk));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}

// Exchange field of a site from its entries: six neighbours in flight; unused slots hold the
// zero spin.  LOCAL: every neighbour is in this block.
template <int CS, int NQ, bool LOCAL>
__device__ __forceinline__ Acc3 res_field(const uint4 (&e)[NQ], int slots, const ResCouplings &J, uint32_t base,
                                          uint32_t first, uint32_t delta) {
    Acc3 h{0.f, 0.f, 0.f};
    constexpr int CH = 6;
#pragma unroll
    for (int m0 = 0; m0 < 8 * NQ; m0 += CH) {
        if (m0 >= slots) break;
        float4 S[CH];
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int m = m0 + j;
            if (m < 8 * NQ) {
                const uint4 &q = e[m >> 3];
                const uint32_t w = (m & 6) == 0 ? q.x : (m & 6) == 2 ? q.y : (m & 6) == 4 ? q.z : q.w;
                const uint32_t v = (m & 1) ? w >> 16 : w & 0xFFFFu;
                if constexpr (CS == 1) S[j] = ld_own(base, v);
                else if constexpr (LOCAL) S[j] = ld_own(base, v & ((1u << kResIdxBits) - 1));
                else S[j] = ld_cluster<CS>(base, first, delta, v & ((1u << kResIdxBits) - 1), v >> kResIdxBits);
            }
        }
#pragma unroll
        for (int j = 0; j < CH; ++j)
            if (m0 + j < 8 * NQ) fma3(h, J.x[m0 + j], J.y[m0 + j], J.z[m0 + j], S[j]);
    }
    return h;
}

// A cluster of CS blocks per replica.  Shared memory: the zero spin, then this block's spins (the
// entries index from the zero spin).  Bound: the shared-memory pipe; a load through the cluster
// window takes twice the wavefronts of one from the block's own window even where it is the same
// block (15 against 8 on the pyrochlore), so sites without remote neighbours take their own path.
template <int OPT, int CS, int NQ>
__global__ void __launch_bounds__(kResThreads, 1)
xyz_resident_general(float4 *__restrict__ spins4, int N, const __grid_constant__ ResShape C,
                     const uint4 *__restrict__ ent, const int32_t *__restrict__ order,
                     const __grid_constant__ ResCouplings J, XyzParams P,
                     const float *__restrict__ beta_slot_f, const int32_t *__restrict__ slot_of_rep,
                     const uint32_t *__restrict__ stream_id, uint32_t *__restrict__ step, const RoundKeys K,
                     int nsweeps, unsigned long long *__restrict__ acc_count, double invN, double *ratio) {
    extern __shared__ __align__(16) float4 s_sp[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_sp);
    const int r = blockIdx.x / CS;
    const uint32_t blk = blockIdx.x % CS;  // the block's rank in its cluster (clusters of CS along x)
    uint32_t first = base, delta = 0;
    if constexpr (CS == 2) {
        uint32_t second;
        asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(first) : "r"(base));
        asm("mapa.shared::cluster.u32 %0, %1, 1;" : "=r"(second) : "r"(base));
        delta = second - first;
    }
    float4 *g = spins4 + (size_t)r * N;
    const float beta_f = beta_slot_f[slot_of_rep[r]];
    const uint32_t stream = stream_id[r], t0 = step[r];
    auto share = [&](int col, int &a, int &b) {
        const long n_c = C.off[col + 1] - C.off[col];
        a = (int)(n_c * blk / CS);
        b = (int)(n_c * (blk + 1) / CS);
    };
    if (threadIdx.x == 0) s_sp[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int col = 0, loc = 1; col < C.ncol; ++col) {
        int a, b;
        share(col, a, b);
        for (int i = a + (int)threadIdx.x; i < b; i += blockDim.x) s_sp[loc + i - a] = g[order[C.off[col] + i]];
        loc += b - a;
    }
    // the next site's entries and rank come while this one is decided, and the first of the next
    // phase, with its draws, before the barrier
    uint4 e[NQ];
    U4 b0, b1;
    int rho = 0;
    auto fetch = [&](int col, int i) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) e[q] = ent[(size_t)q * N + C.off[col] + i];
        rho = order[C.off[col] + i] - C.off[col];
    };
    auto draws = [&](int col, uint32_t t) {
        site_draws<OPT>(P, (uint32_t)rho, t, kMetro | ((uint32_t)col << 8), K, stream, b0, b1);
    };
    {
        int a, b;
        share(0, a, b);
        if (a + (int)threadIdx.x < b) {
            fetch(0, a + (int)threadIdx.x);
            draws(0, t0);
        }
    }
    if constexpr (CS > 1) cluster_barrier();
    else __syncthreads();
    unsigned acc = 0;
    for (int k = 0; k < nsweeps; ++k) {
        const uint32_t t = t0 + (uint32_t)k;
        for (int col = 0, loc = 1; col < C.ncol; ++col) {
            int a, b;
            share(col, a, b);
            for (int i = a + (int)threadIdx.x; i < b; i += blockDim.x) {
                if (i != a + (int)threadIdx.x) draws(col, t);
                bool local = true;
                if constexpr (CS > 1) {  // own block's number in the block bits of every entry
                    const uint32_t mine2 = (blk << kResIdxBits) | (blk << (16 + kResIdxBits));
                    uint32_t differ = 0;
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
                        differ |= (e[q].x ^ mine2) | (e[q].y ^ mine2) | (e[q].z ^ mine2) | (e[q].w ^ mine2);
                    constexpr uint32_t top = (0xFFFFu >> kResIdxBits) << kResIdxBits;
                    local = (differ & (top | top << 16)) == 0;
                }
                const Acc3 h = local ? res_field<CS, NQ, true>(e, C.slots, J, base, first, delta)
                                     : res_field<CS, NQ, false>(e, C.slots, J, base, first, delta);
                const int site = rho;
                if (i + (int)blockDim.x < b) fetch(col, i + (int)blockDim.x);
                float4 *mine = s_sp + loc + i - a;
                const float4 S = *mine;
                float4 nv;
                if (metro_decide<OPT>(P, C.off[col] + site, S, b0, b1, h.x, h.y, h.z, beta_f, (uint32_t)site, t,
                                      kMetro | ((uint32_t)col << 8), K, stream, nv)) {
                    *mine = nv;
                    ++acc;
                }
            }
            loc += b - a;
            // the first site of the next phase
            const int nc = col + 1 < C.ncol ? col + 1 : 0;
            if (nc || k + 1 < nsweeps) {
                share(nc, a, b);
                if (a + (int)threadIdx.x < b) {
                    fetch(nc, a + (int)threadIdx.x);
                    draws(nc, nc ? t : t + 1);
                }
            }
            if constexpr (CS > 1) cluster_barrier();
            else __syncthreads();
        }
    }
    for (int col = 0, loc = 1; col < C.ncol; ++col) {
        int a, b;
        share(col, a, b);
        for (int i = a + (int)threadIdx.x; i < b; i += blockDim.x) g[order[C.off[col] + i]] = s_sp[loc + i - a];
        loc += b - a;
    }
    if (blk == 0 && threadIdx.x == 0) step[r] = t0 + (uint32_t)nsweeps;
    res_accepts<CS>(acc_count + r, acc, invN, ratio ? ratio + r : nullptr, (int)blk);
}

// ------------------------------------------------------------------------ host side ----
static bool xyz_exchange_only(const Ctx &c) { return !c.zeeman && !c.sia && !c.angle && !c.sia_local; }

static void res_range(const Ctx &c, int cs, int col, int k, int &a, int &b) {
    const long n_c = c.col_off[col + 1] - c.col_off[col];
    a = (int)(n_c * k / cs);
    b = (int)(n_c * (k + 1) / cs);
}

// Sites of the largest block share of all colours (phase < 0) or of the largest colour.
static int res_share(const Ctx &c, int cs, bool one_colour) {
    int most = 0;
    for (int k = 0; k < cs; ++k) {
        int n = 0;
        for (int col = 0; col < c.ncol; ++col) {
            int a, b;
            res_range(c, cs, col, k, a, b);
            n = one_colour ? std::max(n, b - a) : n + b - a;
        }
        most = std::max(most, n);
    }
    return most;
}

static size_t res_smem(const Ctx &c, int cs) {
    if (c.model == ETHER_MODEL_ISING)
        return ((size_t)(c.table_entries + 1) / 2 * 2) * 4 + (size_t)c.n_types * 8 + ((size_t)c.N + 16) / 16 * 16;
    return (size_t)(1 + res_share(c, cs, false)) * sizeof(float4);
}

// Kernel of a context (its res_q and cluster size).
static const void *res_kernel(const Ctx &c, int cs) {
    const int q = c.res_q;
    if (c.model == ETHER_MODEL_ISING)
        return cs == 1 ? (q == 1 ? (const void *)ising_resident_general<1, 1> : q == 2 ? (const void *)ising_resident_general<2, 1>
                          : q == 3 ? (const void *)ising_resident_general<3, 1> : (const void *)ising_resident_general<4, 1>)
                       : (q == 1 ? (const void *)ising_resident_general<1, 2> : q == 2 ? (const void *)ising_resident_general<2, 2>
                          : q == 3 ? (const void *)ising_resident_general<3, 2> : (const void *)ising_resident_general<4, 2>);
    auto pick = [&](auto opt) -> const void * {
        constexpr int O = decltype(opt)::value;
        auto qs = [&](auto csv) -> const void * {
            constexpr int S = decltype(csv)::value;
            return q == 1 ? (const void *)xyz_resident_general<O, S, 1> : q == 2 ? (const void *)xyz_resident_general<O, S, 2>
                 : q == 3 ? (const void *)xyz_resident_general<O, S, 3> : (const void *)xyz_resident_general<O, S, 4>;
        };
        return cs == 1 ? qs(std::integral_constant<int, 1>{}) : cs == 2 ? qs(std::integral_constant<int, 2>{})
                                                                        : qs(std::integral_constant<int, 4>{});
    };
    return xyz_exchange_only(c) ? pick(std::integral_constant<int, kXyzExchange>{})
                                : pick(std::integral_constant<int, kXyzGeneral>{});
}

// Orders every block's share of every colour by (site number modulo period, site number) into
// `order` (entry col_off + i: the storage index in place i) and returns the shared-memory wavefronts
// of a sample of its neighbour loads: eight lanes read 16-byte spins from eight banks' width.  The
// period is a constant, as a division by a variable is most of the work (creating a pyrochlore 12^3
// context: 17.9 ms with a variable, 16.9 so; 14.3 without a resident sweep).
template <int period>
static long res_arrange(const Ctx &c, int cs, const std::vector<int32_t> &row_ptr, const std::vector<int32_t> &nbr,
                        std::vector<int32_t> &order, std::vector<int32_t> &pos) {
    std::vector<int> used(cs, 1);
    int start[period];
    for (int col = 0; col < c.ncol; ++col)
        for (int k = 0; k < cs; ++k) {
            int a, b;
            res_range(c, cs, col, k, a, b);
            int32_t *o = order.data() + c.col_off[col];
            // ranks follow the site numbers: one bucket per remainder
            std::fill(start, start + period, 0);
            const int32_t *site = c.site_of_storage.data() + c.col_off[col];
            for (int i = a; i < b; ++i) ++start[(uint32_t)site[i] % period];
            for (int m = 0, n = a; m < period; ++m) n += std::exchange(start[m], n);
            for (int i = a; i < b; ++i) {
                const int to = start[(uint32_t)site[i] % period]++, at = c.col_off[col] + i;
                o[to] = at;
                pos[at] = used[k] + to - a;
            }
            used[k] += b - a;
        }
    const int step = 8 * std::max(1, c.N / 1024);  // about 128 groups of eight lanes
    long cost = 0;
    for (int i = 0; i + 8 <= c.N; i += step)
        for (int m = 0; m < c.res_slots; ++m) {
            int hits[8] = {0, 0, 0, 0, 0, 0, 0, 0}, most = 0, p[8];
            for (int j = 0; j < 8; ++j) {
                const int s = order[i + j];
                p[j] = row_ptr[s] + m < row_ptr[s + 1] ? pos[nbr[row_ptr[s] + m]] : 0;
                bool seen = false;
                for (int q = 0; q < j; ++q) seen = seen || p[q] == p[j];
                if (!seen) most = std::max(most, ++hits[p[j] & 7]);
            }
            cost += most;
        }
    return cost;
}

template <int... P, class F>
static void for_each_period(std::integer_sequence<int, P...>, F &&f) {
    (f(std::integral_constant<int, P>{}), ...);
}

// Sets up a context's resident sweep from its neighbour lists (CSR in storage order; shell of an
// entry = its coupling index, one species): cluster size, slots and packed entries.  smem_max:
// the opt-in shared memory of a block.  Leaves c.gen_resident 0 where it does not apply.
void plan_general_resident(Ctx &c, size_t smem_max, const std::vector<int32_t> &row_ptr, const std::vector<int32_t> &nbr,
                           const std::vector<uint16_t> &jidx, const std::vector<int32_t> &wstride,
                           std::vector<uint4> &ent, std::vector<int32_t> &order) {
    c.gen_resident = 0;
    const bool ising = c.model == ETHER_MODEL_ISING;
    if (c.N >= 65535) return;  // 16-bit entries; four blocks' shared memory holds fewer XYZ spins still
    if ((c.fast && ising) || c.nsp != 1 || c.nsh < 1 || c.nsh > (ising ? 4 : 8)) return;
    if (!ising)  // a free slot adds its coupling times zero
        for (float j : c.h_Jf)
            if (!std::isfinite(j)) return;
    std::vector<int> slots(c.nsh, 0), count(c.nsh);
    std::vector<int> stride(c.nsh, 0);
    for (int s = 0; s < c.N; ++s) {
        std::fill(count.begin(), count.end(), 0);
        for (int k = row_ptr[s]; k < row_ptr[s + 1]; ++k) {
            const int sh = jidx[k];
            if (sh >= c.nsh || (k > row_ptr[s] && sh < jidx[k - 1])) return;  // not in shell order
            ++count[sh];
            if (ising) {
                // the stride of a shell's group depends on the site's type only through the shells
                // before it; the kernel wants one per shell
                if (stride[sh] && stride[sh] != wstride[k]) return;
                stride[sh] = wstride[k];
            }
        }
        for (int sh = 0; sh < c.nsh; ++sh) slots[sh] = std::max(slots[sh], count[sh]);
    }
    int total = 0;
    for (int sh = 0; sh < c.nsh; ++sh) {
        if (slots[sh] == 0) return;
        total += slots[sh];
        c.res_shell_end[sh] = total;
        c.res_stride[sh] = stride[sh];
    }
    if (total < 1 || total > 8 * kResMaxQ) return;
    c.res_q = (total + 7) / 8;
    c.res_slots = total;
    int cs = 0;
    if (ising) {
        if (c.N < 65535 && res_smem(c, 1) <= smem_max) cs = 1;
        // two blocks, which both hold all spins, while all replicas still run at once and a colour is
        // more than a round of pairs (per sweep, before the slots' constant strides: 30 x 34 x 38 x 60
        // 31 us with one block, 18 with two; 23 x 21 x 19 16.6 and 9.0; 21 x 18 x 15 8.4 and 8.0; 14^3
        // 3.4 and 3.8; with them pyrochlore 12^3 39.8 and 27.7, 33 x 31 x 45 27.1 and 15.8, 29 x 27 x 25
        // 13.4 and 10.7, 21 x 18 x 15 6.0 and 6.5)
        if (cs && 2L * c.R * 10 <= 9L * c.sm_count && res_share(c, 1, true) >= 2048) cs = 2;
    } else {
        // the smallest cluster that holds a replica; then larger ones while all replicas still run
        // at once (nine tenths of the SMs: clusters need neighbouring ones) and a block keeps 512
        // sites of a colour (per sweep: pyrochlore 9^3 cells x 64 48.9 us with 1 block, 44.8 with
        // 2; 7^3, 343 sites a block, 26.9 and 32.0; 21 x 18 x 15 open cubic 14.1 and 10.3)
        for (int v : {1, 2, 4}) {
            if (res_smem(c, v) > smem_max || (v == 1 ? c.N >= 65535 : res_share(c, v, false) + 1 >= (1 << kResIdxBits)))
                continue;
            if (!cs || ((long)c.R * v * 10 <= 9L * c.sm_count && res_share(c, v, true) >= 512)) cs = v;
        }
    }
    // Against the phase kernels: a replica's sweep here takes its sites' time in turn, theirs the
    // whole context's work over the GPU but at least a launch's latency per colour.  Measured per
    // site: here 0.3 ns + 0.07 per slot, and 1 us a colour (Ising), 1.0 + 0.1425 per slot (XYZ; 1.3 times that in a cluster); there,
    // over all replicas, 0.037 ns (Ising), 0.004 per slot - 0.008 (XYZ), and 3 us (4 us) a colour.
    // The Ising terms are those of the kernel before its slots' constant strides; it takes 0.22 ns +
    // 0.055 per slot and 0.9 us a colour now (152 replicas: 13^3 3.7 us, 29 x 27 x 25 13.4,
    // pyrochlore 12^3 39.8), its phases 4.1 us a colour, so the line lies on the phases' side: a single
    // pyrochlore 12^3 replica stays with them at 45 us where two blocks would take 28.
    if (cs) {
        const double waves = std::ceil((double)c.R * cs / c.sm_count), share = (double)c.N / cs, all = (double)c.N * c.R;
        const double here = ising ? 1.0 * c.ncol + waves * share * (0.3e-3 + 0.07e-3 * total)
                                  : waves * share * (1.0e-3 + 0.1425e-3 * total) * (cs > 1 ? 1.3 : 1.0);
        const double there = std::max(c.ncol * (ising ? 3.0 : 4.0), all * (ising ? 0.037e-3 : std::max(0.008e-3, 0.004e-3 * total - 0.008e-3)));
        if (here > there) cs = 0;
    }
    if (!cs) return;
    // the order in which a block takes a colour's sites and keeps them: sites that are equal modulo
    // a period (a basis of the unit cell) side by side, with the period whose sampled loads have the
    // fewest bank conflicts (none: sites in rank order)
    order.resize(c.N);
    for (int s = 0; s < c.N; ++s) order[s] = s;
    if (!ising) {
        long best = -1;
        std::vector<int32_t> trial(c.N), pos(c.N);
        auto attempt = [&](auto period) {
            const long cost = res_arrange<decltype(period)::value>(c, cs, row_ptr, nbr, trial, pos);
            if (best < 0 || cost < best) {
                best = cost;
                order.swap(trial);
            }
        };
        for_each_period(std::integer_sequence<int, 1, 2, 3, 4, 6, 8, 12, 16, 24, 32>{}, attempt);
    }
    // where a storage index lives: XYZ, 1 + its place in the owning block's array | block << 14
    std::vector<uint16_t> where(c.N);
    std::vector<int> used(cs, ising ? 0 : 1);
    for (int col = 0; col < c.ncol; ++col)
        for (int k = 0; k < cs; ++k) {
            int a, b;
            res_range(c, cs, col, k, a, b);
            for (int i = a; i < b; ++i)
                where[order[c.col_off[col] + i]] =
                    ising ? (uint16_t)(c.col_off[col] + i) : (uint16_t)((used[k] + i - a) | (cs > 1 ? k << kResIdxBits : 0));
            used[k] += b - a;
        }
    std::vector<uint16_t> e16((size_t)c.res_q * c.N * 8, ising ? (uint16_t)c.N : (uint16_t)0);
    for (int col = 0; col < c.ncol; ++col)
        for (int blk = 0; blk < cs; ++blk) {
            int a, b;
            res_range(c, cs, col, blk, a, b);
            for (int i = a; i < b; ++i) {
                const int s = order[c.col_off[col] + i], e = c.col_off[col] + i;
                // the zero spin of the block that updates the site
                const uint16_t zero = ising ? (uint16_t)c.N : (uint16_t)(cs > 1 ? blk << kResIdxBits : 0);
                for (int m = 0; m < 8 * c.res_q; ++m) e16[((size_t)(m >> 3) * c.N + e) * 8 + (m & 7)] = zero;
                int sh = -1, m = 0;
                for (int k = row_ptr[s]; k < row_ptr[s + 1]; ++k) {
                    if (jidx[k] != sh) {
                        sh = jidx[k];
                        m = sh ? c.res_shell_end[sh - 1] : 0;
                    }
                    e16[((size_t)(m >> 3) * c.N + e) * 8 + (m & 7)] = where[nbr[k]];
                    ++m;
                }
            }
        }
    ent.resize((size_t)c.res_q * c.N);
    static_assert(sizeof(uint4) == 8 * sizeof(uint16_t), "eight entries to a word");
    std::memcpy(ent.data(), e16.data(), e16.size() * sizeof(uint16_t));
    c.gen_resident = cs;
}

// A graph replays launches 2.1 us apart and more (the calls that launch directly, 4.1), so there a short run
// of a few large replicas is better off by phases: no load and store of all spins, no cluster
// barriers.  Fitted to the rows of series (a sweep and |M|), shared memory and phases, us: Ising
// 29 x 27 x 25 x 1 27.6 and 19.6 (four sweeps a row 58.3 and 46.9), 21 x 18 x 15 x 1 19.4 and 17.7 (two
// sweeps 25.6 and 26.1), 9^3 x 1 13.1 and 15.6; XYZ 16^3 x 16 19.5 and 17.5 (four 31.3 and 32.2), 16^3 x
// 64 21.6 and 19.7 (three 33.3 and 36.3), 20^3 x 1 19.4 and 15.4 (four 37.9 and 30.0), 8^3 x 1 11.3
// and 12.2; pyrochlore 8^3 Ising x 8, 18 neighbours, 32.1 and 39.1.
bool general_resident_pays(const Ctx &c, int n) {
    const bool ising = c.model == ETHER_MODEL_ISING;
    const int cs = c.gen_resident, slots = c.res_slots;
    const double share = (double)c.N / cs, waves = std::ceil((double)c.R * cs / c.sm_count);
    const double barrier = (ising ? 0.6 : 0.6 * 0.95) * (cs > 1 ? 2.0 : 1.0);
    const double site = (ising ? 0.22e-3 + 0.055e-3 * slots : 0.35e-3 + 0.15e-3 * slots) * (!ising && cs > 1 ? 1.5 : 1.0);
    const double once = ising ? 2.3 + 0.25e-3 * c.N : 0.5 + 1.2e-3 * share + (cs > 1 ? 1.0 : 0.0);
    const double here = once + n * (barrier * c.ncol + waves * share * site);
    const double launch = ising ? 1.6 + 0.083 * slots : c.fast ? 2.1 : 2.0 + 0.1 * slots, size = ising ? 0.04e-3 : c.fast ? 0.03e-3 : 0.26e-3;
    const double rate = ising ? 0.011e-3 : c.fast ? 0.016e-3 : 0.026e-3;
    return here <= n * (launch * c.ncol + size * c.N + rate * c.N * c.R);
}

// Opts the context's kernel into its shared memory (once, at creation: not during a capture).
cudaError_t prepare_general_resident(const Ctx &c) { return allow_shared(res_kernel(c, c.gen_resident)); }

cudaError_t launch_general_resident(Ctx &c, int nsweeps, double *ratio) {
    if (nsweeps < 1) return cudaSuccess;
    const int cs = c.gen_resident;
    const bool ising = c.model == ETHER_MODEL_ISING;
    ResShape C;
    C.ncol = c.ncol;
    C.slots = c.res_slots;
    for (int col = 0; col <= c.ncol; ++col) C.off[col] = col < c.ncol ? c.col_off[col] : c.N;
    for (int m = 0, sh = 0; m < 8 * kResMaxQ; ++m) {
        if (m < c.res_slots && m >= c.res_shell_end[sh]) ++sh;
        C.stride[m] = m < c.res_slots ? c.res_stride[sh] : 0;
    }
    RoundKeys K = round_keys(c.seed);
    // full rounds of at most 1024 threads over the largest class (Ising: pairs of sites)
    const int work = ising ? ((res_share(c, 1, true) + 1) / 2 + cs - 1) / cs : res_share(c, cs, true);
    const int rounds = std::max(1, (work + kResThreads - 1) / kResThreads);
    const int threads = std::max(64, ((work + rounds - 1) / rounds + 31) / 32 * 32);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c.R * cs);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = res_smem(c, cs);
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cs > 1 ? 1 : 0;
    c.launches++;
    double invN = 1.0 / (double)c.N;
    if (ising) {
        void *args[] = {&c.spins, &c.N, &C, &c.t.res_ent, &c.t.itype, &c.t.type_base, &c.t.type_half,
                        &c.n_types, &c.thr, &c.table_entries, &c.slot_of_rep, &c.stream_id, &c.step, &K, &nsweeps,
                        &c.acc_count, &invN, &ratio};
        return cudaLaunchKernelExC(&cfg, res_kernel(c, cs), args);
    }
    XyzParams P = xyz_params(c);
    ResCouplings J = {};
    for (int m = 0, sh = 0; m < c.res_slots; ++m) {
        if (m >= c.res_shell_end[sh]) ++sh;
        J.x[m] = c.h_Jf[3 * sh];
        J.y[m] = c.h_Jf[3 * sh + 1];
        J.z[m] = c.h_Jf[3 * sh + 2];
    }
    void *args[] = {&c.spins4, &c.N, &C, &c.t.res_ent, &c.t.res_order, &J, &P, &c.beta_slot_f, &c.slot_of_rep, &c.stream_id,
                    &c.step, &K, &nsweeps, &c.acc_count, &invN, &ratio};
    return cudaLaunchKernelExC(&cfg, res_kernel(c, cs), args);
}

}  // namespace ether
