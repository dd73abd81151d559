// measure.cuh -- the observable accumulation of one replica, shared by the reductions (k_obs.cu)
// and the resident Ising sweep, which measures without leaving its launch (k_ising.cu).
#pragma once
#include <cstdint>

namespace ether {

// get_eng('eng') / get_mag('mag') of replica r, into its (group, slot) accumulator.
__device__ __forceinline__ void measure_one(const double *E, const double *M, int N, int n_slots,
                                            const int32_t *__restrict__ slot_of_rep, double *__restrict__ sums, int r) {
    const int idx = (r / n_slots) * n_slots + slot_of_rep[r];
    const double e = E[r] / (2.0 * N);
    const double mx = M[3 * r], my = M[3 * r + 1], mz = M[3 * r + 2];
    const double m = sqrt(mx * mx + my * my + mz * mz) / N;
    double *a = sums + (size_t)idx * 7;
    a[0] += 1.0;
    a[1] += e;
    a[2] += e * e;
    a[3] += (e * e) * (e * e);
    a[4] += m;
    a[5] += m * m;
    a[6] += (m * m) * (m * m);
}

}  // namespace ether
