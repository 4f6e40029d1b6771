// k_relax.cu -- the voxel-wise steps of the unrolled relaxed MLEM
// (mlem_b200/torch_ext.py): x_next = x * r ** omega with r = calcUpdate's factor,
// and its gradient.
//
// Each step is one pass over vectors of one float per voxel, bound by HBM (or L2)
// and, on small images, by its launch: as tensor expressions the forward step was
// eight launches with as many temporaries and the gradient step about fifteen
// (a gradient step of five iterations over 1,048,576 rows and voxels 6.58 -> 5.79
// ms, over 50,001 rows 2,228 -> 684 us, of four over 900 rows 1,823 -> 737 us).
// Compiled without flush-to-zero: a subnormal factor r is positive here, as it is
// to the tensor expressions these kernels replace.
#include <algorithm>

#include "kernels.h"

namespace mlem {

namespace {

constexpr int kRelaxThreads = 256;
constexpr float kRatioFloor = 1e-38f;

__device__ __forceinline__ float over_norm(float v, float n) { return n != 0.0f ? v / n : v; }

__global__ void __launch_bounds__(kRelaxThreads) k_relax_step(const float* x, const float* u,
                                                              const float* norm, const float* omega,
                                                              uint32_t C, float* r, float* x_next) {
    const float w = *omega;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < C;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const float q = over_norm(u[i], norm[i]);
        r[i] = q;
        x_next[i] = x[i] * (q > 0.0f ? powf(fmaxf(q, kRatioFloor), w) : 0.0f);
    }
}

// g (+ g2) -> gx = the direct path, du = the gradient of the update's numerator,
// and the block's part of omega's gradient (double, fixed order).
__global__ void __launch_bounds__(kRelaxThreads) k_relax_grad(const float* g, const float* g2,
                                                              const float* x, const float* r,
                                                              const float* norm, const float* omega,
                                                              uint32_t C, float* gx, float* du,
                                                              double* partial) {
    __shared__ double part[kRelaxThreads / 32];
    const float w = *omega;
    double s = 0.0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < C;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const float gi = g2 ? g[i] + g2[i] : g[i], xi = x[i], ri = r[i];
        const bool pos = ri > 0.0f;
        const float rs = pos ? ri : 1.0f;
        const float p = pos ? powf(rs, w) : 0.0f;
        s += (double)(gi * (xi * p) * (pos ? logf(rs) : 0.0f));  // not finite where g or x is not
        gx[i] = gi * p;
        du[i] = over_norm(pos ? gi * xi * w * powf(rs, w - 1.0f) : 0.0f, norm[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < kRelaxThreads / 32; ++k) t += part[k];
        partial[blockIdx.x] = t;
    }
}

}  // namespace

cudaError_t relax_step(const float* x, const float* u, const float* norm, const float* omega,
                       uint32_t C, float* r, float* x_next, cudaStream_t st) {
    if (C == 0) return cudaSuccess;
    const unsigned grid = (unsigned)std::min<uint64_t>(((uint64_t)C + kRelaxThreads - 1) / kRelaxThreads, 148 * 8);
    k_relax_step<<<grid, kRelaxThreads, 0, st>>>(x, u, norm, omega, C, r, x_next);
    return cudaGetLastError();
}

cudaError_t relax_grad(const float* g, const float* g2, const float* x, const float* r,
                       const float* norm, const float* omega, uint32_t C, float* gx, float* du,
                       double* partial, cudaStream_t st) {
    k_relax_grad<<<kRelaxPartials, kRelaxThreads, 0, st>>>(g, g2, x, r, norm, omega, C, gx, du, partial);
    return cudaGetLastError();
}

}  // namespace mlem
