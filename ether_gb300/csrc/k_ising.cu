// k_ising.cu -- per-context launches of the Ising colour phase (bodies in sweep_ising.cuh).
#include <algorithm>

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
                 const uint32_t *__restrict__ step, uint32_t seed,
                 unsigned long long *__restrict__ acc_count) {
    const int r = blockIdx.y;
    uint8_t *sp = spins + (size_t)r * N;
    const uint32_t *tb = thr + (size_t)slot_of_rep[r] * table_entries;
    const uint32_t stream = stream_id[r], t = step[r];
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
                      const uint32_t *__restrict__ step, uint32_t seed,
                      unsigned long long *__restrict__ acc_count) {
    const int r = blockIdx.y;
    uint8_t *sp = spins + (size_t)r * N;
    const uint32_t *tb = thr + (size_t)slot_of_rep[r] * table_entries;
    const uint32_t stream = stream_id[r], t = step[r];
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
                const uint32_t *__restrict__ step, uint32_t seed, const RoundKeys K,
                unsigned long long *__restrict__ acc_count) {
    const int r = blockIdx.y;
    const int H = L1 >> 1;
    const int half = H * L2 * L3;
    __shared__ uint32_t s_tab[kScTabWords];
    const IsingSc A{spins + (size_t)r * 2 * half + (size_t)colour * half,
                    spins + (size_t)r * 2 * half + (size_t)(colour ^ 1u) * half,
                    L1, L2, L3, H, fH, fL2, colour};
    const uint32_t c3 = kMetro | (colour << 8);
    const uint32_t t = step[r], stream = stream_id[r];
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
        c.stream_id, c.step, c.seed, round_keys(c.seed), c.acc_count);
}

static int blocks_for(const Ctx &c, long work, int bs) {
    long need = (work + bs - 1) / bs;
    long cap = (long)c.sm_count * 8 / (c.R > 0 ? c.R : 1);
    if (cap < 1) cap = 1;
    if (need > cap) need = cap;
    if (need < 1) need = 1;
    return (int)need;
}

// Resident form for small simple-cubic lattices: one block per replica holds both colour
// arrays in shared memory and runs nsweeps whole sweeps (colour 0, colour 1, counter + 1)
// between two visits to global memory.  The draws, thresholds and vector update are the
// phase kernels' (ising_sc_vectors), so every decision is the same; the sweep counter is
// advanced here instead of by advance_kernel.
template <int W>
__global__ void __launch_bounds__(256)
ising_sc_resident(uint8_t *__restrict__ spins, int L1, int L2, int L3, FastDiv fH, FastDiv fL2,
                  const uint32_t *__restrict__ thr, int table_entries,
                  const int32_t *__restrict__ slot_of_rep, const uint32_t *__restrict__ stream_id,
                  uint32_t *__restrict__ step, uint32_t seed, const RoundKeys K, int nsweeps,
                  unsigned long long *__restrict__ acc_count) {
    extern __shared__ __align__(16) uint8_t s_sp[];  // colour 0 array, then colour 1
    __shared__ uint32_t s_tab[kScTabWords];
    const int r = blockIdx.x;
    const int H = L1 >> 1;
    const int half = H * L2 * L3;
    const int nvec = half / W;
    uint4 *g = reinterpret_cast<uint4 *>(spins + (size_t)r * 2 * half);
    uint4 *sv = reinterpret_cast<uint4 *>(s_sp);
    const int n16 = (2 * half) >> 4;  // 2 half is a multiple of 16 (W | H)
    for (int i = threadIdx.x; i < n16; i += blockDim.x) sv[i] = g[i];
    fill_sc_table(thr + (size_t)slot_of_rep[r] * table_entries, s_tab, threadIdx.x, blockDim.x);
    const uint32_t stream = stream_id[r];
    const uint32_t t0 = step[r];
    __syncthreads();
    unsigned flips = 0;
    for (int k = 0; k < nsweeps; ++k) {
        const uint32_t t = t0 + (uint32_t)k;
        for (int colour = 0; colour < 2; ++colour) {
            const IsingSc A{s_sp + (size_t)colour * half, s_sp + (size_t)(colour ^ 1) * half,
                            L1, L2, L3, H, fH, fL2, (uint32_t)colour};
            uint32_t cnt = 0;
            for (int v = threadIdx.x; v < nvec; v += blockDim.x)
                cnt += ising_sc_vectors<W, 1>(A, v, 0, nvec, sc_tab(s_tab), t, stream, kMetro | ((uint32_t)colour << 8),
                                              seed, K);
            flips += byte_sum(cnt);  // each byte <= (W / 4) * ceil(nvec / blockDim) per colour
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < n16; i += blockDim.x) g[i] = sv[i];
    if (threadIdx.x == 0) step[r] = t0 + (uint32_t)nsweeps;
    warp_add_count(acc_count + r, flips);
}

bool ising_resident_possible(const Ctx &c, size_t smem_max) {
    if (!c.fast || c.model != ETHER_MODEL_ISING || c.vec_bytes == 0) return false;
    const size_t bytes = (size_t)c.L[0] * c.L[1] * c.L[2];  // both colours
    // (W/4) ceil(nvec/256) flips per byte of a vector count must stay below 256
    const size_t nvec = bytes / 2 / (size_t)c.vec_bytes;
    return bytes <= smem_max && (c.vec_bytes / 4) * ((nvec + 255) / 256) < 256;
}

// Opts the resident kernel into the shared memory a replica needs (once, at creation: not
// during a stream capture).
cudaError_t prepare_ising_resident(const Ctx &c) {
    const int smem = c.L[0] * c.L[1] * c.L[2];
    return c.vec_bytes == 16  ? cudaFuncSetAttribute(ising_sc_resident<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)
           : c.vec_bytes == 8 ? cudaFuncSetAttribute(ising_sc_resident<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)
                              : cudaFuncSetAttribute(ising_sc_resident<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

cudaError_t launch_ising_resident(Ctx &c, int nsweeps) {
    const int smem = c.L[0] * c.L[1] * c.L[2];
    const int bs = 256;
    if (c.vec_bytes == 16) {
        ising_sc_resident<16><<<c.R, bs, smem, c.stream>>>(
            c.spins, c.L[0], c.L[1], c.L[2], make_fastdiv((uint32_t)(c.L[0] / 2)), make_fastdiv((uint32_t)c.L[1]),
            c.thr, c.table_entries, c.slot_of_rep, c.stream_id, c.step, c.seed, round_keys(c.seed), nsweeps,
            c.acc_count);
    } else if (c.vec_bytes == 8) {
        ising_sc_resident<8><<<c.R, bs, smem, c.stream>>>(
            c.spins, c.L[0], c.L[1], c.L[2], make_fastdiv((uint32_t)(c.L[0] / 2)), make_fastdiv((uint32_t)c.L[1]),
            c.thr, c.table_entries, c.slot_of_rep, c.stream_id, c.step, c.seed, round_keys(c.seed), nsweeps,
            c.acc_count);
    } else {
        ising_sc_resident<4><<<c.R, bs, smem, c.stream>>>(
            c.spins, c.L[0], c.L[1], c.L[2], make_fastdiv((uint32_t)(c.L[0] / 2)), make_fastdiv((uint32_t)c.L[1]),
            c.thr, c.table_entries, c.slot_of_rep, c.stream_id, c.step, c.seed, round_keys(c.seed), nsweeps,
            c.acc_count);
    }
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
                c.slot_of_rep + r0, c.stream_id + r0, c.step + r0, c.seed, c.acc_count + r0);
        } else {
            dim3 grid(blocks_for(c, (n_c + 7) / 8, bs), nr);
            ising_ell_kernel<<<grid, bs, 0, c.stream>>>(
                spins, c.N, c.col_off[colour], n_c, (uint32_t)colour, ell, ews, c.t.ell_deg,
                c.ell_width[colour], c.t.itype, c.t.type_base, c.t.type_half, c.thr, c.table_entries,
                c.slot_of_rep + r0, c.stream_id + r0, c.step + r0, c.seed, c.acc_count + r0);
        }
    }
    c.launches++;
    return cudaGetLastError();
}

}  // namespace ether
