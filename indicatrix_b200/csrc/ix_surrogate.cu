// ix_surrogate.cu -- the learned surrogate's elementwise kernels: the MSE loss gradient,
// bias gradients, the Adam update and f32 -> bf16 conversion, all on device pointers and
// the caller's stream (include/ix_surrogate.h).  The GEMMs, with their bias / SiLU
// epilogues, are the tcgen05 kernels of ix_umma.cu.  The network maps stone design
// parameters to tilt-resolved brilliance / fire / scintillation measured on the tracer's
// renders (ix_design.h) and screens candidate designs before the tracer re-renders the
// survivors.  No reference counterpart: the reference has no tracer-trained surrogate.
#include <cstdint>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace ix {
namespace mlp {
namespace {

// Mean squared error over the m x n outputs: dy = 2 (y - t) / (m n) (f32 and bf16), and
// the loss summed into *loss (one atomic per warp).
__global__ void mse_grad_kernel(int m, int n, const float* __restrict__ y, const float* __restrict__ t,
                                float* __restrict__ dy, __nv_bfloat16* __restrict__ dyb, float* __restrict__ loss) {
    const int64_t total = (int64_t)m * n;
    const float inv = 1.0f / (float)total;
    float part = 0.0f;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const float d = y[i] - t[i];
        const float g = 2.0f * d * inv;
        dy[i] = g;
        dyb[i] = __float2bfloat16_rn(g);
        part += d * d * inv;
    }
    for (int off = 16; off > 0; off >>= 1) part += __shfl_down_sync(0xFFFFFFFFu, part, off);
    if ((threadIdx.x & 31) == 0 && loss) atomicAdd(loss, part);
}

// db[col] = sum over rows of dz.  Reading the rows bounds it (4 MB at 4096 x 256), so a
// cluster of CTAs takes 32 columns: a warp reads 32 neighbouring columns of one row, each
// thread sums every (32 ranks)-th row, and the partial sums fold in a fixed tree -- the 32 of
// a CTA, then the CTAs in rank order -- whatever the scheduling.  4096 x 256: 235 us with a
// thread per column walking the rows, 7.5 us so.
constexpr int BIAS_ROWS = 32;     // rows of a CTA pass
constexpr int BIAS_CLUSTER = 8;
__global__ void __launch_bounds__(32 * BIAS_ROWS) bias_grad_kernel(int m, int n, const float* __restrict__ dz,
                                                                  float* __restrict__ db) {
    namespace cg = cooperative_groups;
    __shared__ float s_part[BIAS_ROWS][33];
    __shared__ float s_sum[32];
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
    const int c = threadIdx.x & 31, ry = threadIdx.x >> 5;
    const int col = (blockIdx.x / ranks) * 32 + c;
    float s = 0.0f;
    if (col < n)
        for (int64_t r = rank * BIAS_ROWS + ry; r < m; r += (int64_t)ranks * BIAS_ROWS) s += dz[r * n + col];
    s_part[ry][c] = s;
    __syncthreads();
    // Warp ry folds column ry: lane i holds partial i.
    float v = s_part[c][ry];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, off);
    if (c == 0) s_sum[ry] = v;
    cluster.sync();
    if (rank == 0 && ry == 0 && col < n) {
        float total = 0.0f;
        for (int k = 0; k < ranks; ++k) total += *cluster.map_shared_rank(&s_sum[c], k);
        db[col] = total;
    }
    cluster.sync();  // the ranks' shared memory outlives the read
}

// Adam on f32 master weights, with their bf16 copy refreshed (Kingma & Ba 2015).
__global__ void adam_kernel(int64_t count, float* __restrict__ w, __nv_bfloat16* __restrict__ wb,
                            const float* __restrict__ g, float* __restrict__ mom, float* __restrict__ vel, float lr,
                            float beta1, float beta2, float eps, float bias1, float bias2) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = beta1 * mom[i] + (1.0f - beta1) * gi;
        const float vi = beta2 * vel[i] + (1.0f - beta2) * gi * gi;
        mom[i] = mi;
        vel[i] = vi;
        const float wi = w[i] - lr * (mi / bias1) / (sqrtf(vi / bias2) + eps);
        w[i] = wi;
        if (wb) wb[i] = __float2bfloat16_rn(wi);
    }
}

__global__ void to_bf16_kernel(int64_t count, const float* __restrict__ x, __nv_bfloat16* __restrict__ xb) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
        xb[i] = __float2bfloat16_rn(x[i]);
}

unsigned int grid_for(int64_t n) {
    const int64_t b = (n + 255) / 256;
    return (unsigned int)(b < 1 ? 1 : (b > 148 * 16 ? 148 * 16 : b));
}

}  // namespace

cudaError_t mse_grad(int m, int n, const float* y, const float* t, float* dy, void* dyb, float* loss,
                     cudaStream_t s) {
    mse_grad_kernel<<<grid_for((int64_t)m * n), 256, 0, s>>>(m, n, y, t, dy, (__nv_bfloat16*)dyb, loss);
    return cudaGetLastError();
}
cudaError_t bias_grad(int m, int n, const float* dz, float* db, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    // One CTA does while the rows are one pass of it.
    int ranks = 1;
    while (ranks < BIAS_CLUSTER && (int64_t)ranks * BIAS_ROWS < m) ranks *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((n + 31) / 32) * (unsigned)ranks);
    cfg.blockDim = dim3(32 * BIAS_ROWS);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, bias_grad_kernel, m, n, dz, db);
}
cudaError_t adam(int64_t count, float* w, void* wb, const float* g, float* mom, float* vel, float lr, float beta1,
                 float beta2, float eps, float bias1, float bias2, cudaStream_t s) {
    adam_kernel<<<grid_for(count), 256, 0, s>>>(count, w, (__nv_bfloat16*)wb, g, mom, vel, lr, beta1, beta2, eps,
                                               bias1, bias2);
    return cudaGetLastError();
}
cudaError_t to_bf16(int64_t count, const float* x, void* xb, cudaStream_t s) {
    to_bf16_kernel<<<grid_for(count), 256, 0, s>>>(count, x, (__nv_bfloat16*)xb);
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace ix

#include "../../include/ix_surrogate.h"

#include <cmath>

namespace {
int rc(cudaError_t e) { return e == cudaSuccess ? 0 : 1; }
cudaStream_t st(void* s) { return (cudaStream_t)s; }
}  // namespace

extern "C" {

int ix_mlp_mse_grad(uint32_t m, uint32_t n, const float* y, const float* t, float* dy, void* dyb, float* loss,
                    void* stream) {
    if (!y || !t || !dy || !dyb) return 1;
    return rc(ix::mlp::mse_grad((int)m, (int)n, y, t, dy, dyb, loss, st(stream)));
}
int ix_mlp_bias_grad(uint32_t m, uint32_t n, const float* dz, float* db, void* stream) {
    if (!dz || !db) return 1;
    return rc(ix::mlp::bias_grad((int)m, (int)n, dz, db, st(stream)));
}
int ix_mlp_adam(uint64_t count, float* w, void* wb, const float* g, float* m, float* v, float lr, float beta1,
                float beta2, float eps, uint32_t t, void* stream) {
    if (!w || !g || !m || !v || t == 0) return 1;
    const float b1 = 1.0f - std::pow(beta1, (float)t), b2 = 1.0f - std::pow(beta2, (float)t);
    return rc(ix::mlp::adam((int64_t)count, w, wb, g, m, v, lr, beta1, beta2, eps, b1, b2, st(stream)));
}
int ix_mlp_to_bf16(uint64_t count, const float* x, void* xb, void* stream) {
    if (!x || !xb) return 1;
    return rc(ix::mlp::to_bf16((int64_t)count, x, xb, st(stream)));
}

}  // extern "C"
