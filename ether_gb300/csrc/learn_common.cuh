// learn_common.cuh -- what the two learned patch proposals share: the 4^3 patch geometry in
// closed form, the sweep counter's kernel (k_learn.cu), and the entry points of
// the Heisenberg learner (k_learn_xyz.cu) that the ether_learn_* functions hand an XYZ
// context over to.
#pragma once
#include <cstdint>

#include <cuda_bf16.h>

#include "internal.h"

namespace ether {
namespace learn {

constexpr uint32_t kLearn = 4;  // Philox purpose
constexpr int NH = 128;         // hidden width of both networks

// ------------------------------------------------------------------ patch geometry ----
// Canonical frame of a patch: local (a, b, c) in [0, 4)^3; A-sites ((a + b + c) even) and
// B-sites numbered 0..31 each in order of a + 4b + 16c.  Row = b + 4c; the two A-sites
// (B-sites) of a row sit at a = p, p + 2 (a = 1 - p, 3 - p), p = (b + c) & 1, and have
// indices 2 row + (a >> 1).  Boundary sites (faces a = -1, 4, b = -1, 4, c = -1, 4) are
// numbered face * 16 + (the two other coordinates u + 4 v).
__host__ __device__ constexpr int geo_b_a(int m) { return (1 - ((((m >> 1) & 3) + ((m >> 1) >> 2)) & 1)) + 2 * (m & 1); }
__host__ __device__ constexpr int geo_a_a(int k) { return ((((k >> 1) & 3) + ((k >> 1) >> 2)) & 1) + 2 * (k & 1); }
// Neighbour q (-x, +x, -y, +y, -z, +z) of B-site m: A-site index (>= 0) or -(1 + boundary index).
__host__ __device__ constexpr int geo_bn(int m, int q) {
    const int row = m >> 1, b = row & 3, c = row >> 2, a = geo_b_a(m);
    return q == 0 ? (a == 0 ? -(1 + b + 4 * c) : 2 * row + ((a - 1) >> 1))
         : q == 1 ? (a == 3 ? -(1 + 16 + b + 4 * c) : 2 * row + ((a + 1) >> 1))
         : q == 2 ? (b == 0 ? -(1 + 32 + a + 4 * c) : 2 * (row - 1) + (a >> 1))
         : q == 3 ? (b == 3 ? -(1 + 48 + a + 4 * c) : 2 * (row + 1) + (a >> 1))
         : q == 4 ? (c == 0 ? -(1 + 64 + a + 4 * b) : 2 * (row - 4) + (a >> 1))
                  : (c == 3 ? -(1 + 80 + a + 4 * b) : 2 * (row + 4) + (a >> 1));
}
// Boundary neighbour q of A-site k (-1 if that neighbour is inside the patch).
__host__ __device__ constexpr int geo_ab(int k, int q) {
    const int row = k >> 1, b = row & 3, c = row >> 2, a = geo_a_a(k);
    return q == 0 ? (a == 0 ? b + 4 * c : -1)
         : q == 1 ? (a == 3 ? 16 + b + 4 * c : -1)
         : q == 2 ? (b == 0 ? 32 + a + 4 * c : -1)
         : q == 3 ? (b == 3 ? 48 + a + 4 * c : -1)
         : q == 4 ? (c == 0 ? 64 + a + 4 * b : -1)
                  : (c == 3 ? 80 + a + 4 * b : -1);
}

__global__ void advance_lstep_kernel(uint32_t *c, int R);

// The kernels of a class follow one another closely: each lets the next one start while it runs
// (after_release), and reads what the one before it wrote only when that has ended
// (after_wait).  What lies before the wait -- a network's weights, a patch's position -- overlaps,
// and so does the launch.  Only the wait makes an earlier kernel's writes visible, so a class's
// first kernel, which may follow the one that packed the weights, releases the network's kernel
// after its own wait.  close = false: an ordinary launch.
__device__ __forceinline__ void after_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool close, A &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = close ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// ------------------------------------------------ the Heisenberg learner (k_learn_xyz.cu) ----
struct XyzLearn;
int xyz_create(ether_ctx *h, const ether_learn_desc *d, XyzLearn **out);
void xyz_destroy(XyzLearn *x);
int xyz_collect(XyzLearn *x, int per_replica);
int xyz_train(XyzLearn *x, int steps, int batch, float lr, double *loss);
int xyz_sweep(XyzLearn *x, int nsweeps);
int xyz_record_series(XyzLearn *x, int nsteps, int plain_per_step, int learned_per_step, int stride,
                      double *absM);
int xyz_get_accepts(XyzLearn *x, uint64_t *accepted);
void xyz_set_dump(XyzLearn *x, bool on);
int xyz_get_dump(XyzLearn *x, float *out);
int xyz_get_params(XyzLearn *x, float *params);
int xyz_set_params(XyzLearn *x, const float *params);
int xyz_loss_grad(XyzLearn *x, const float *xin, const float *y, int B, double *loss, float *grad);
int xyz_forward(XyzLearn *x, const float *xin, int B, float *out);
int xyz_info(XyzLearn *x, ether_learn_info *info);
void xyz_shape(int *n_inputs, int *n_outputs, int *n_params);

}  // namespace learn
}  // namespace ether
