// ix_surrogate.cu -- the learned surrogate's elementwise kernels: the MSE loss gradient,
// bias gradients, the Adam update and f32 -> bf16 conversion, all on device pointers and
// the caller's stream (include/ix_surrogate.h).  The GEMMs, with their bias / SiLU
// epilogues, are the tcgen05 kernels of ix_umma.cu.  The network maps stone design
// parameters to tilt-resolved brilliance / fire / scintillation measured on the tracer's
// renders (ix_design.h) and screens candidate designs before the tracer re-renders the
// survivors.  No reference counterpart: the reference has no tracer-trained surrogate.
#include <cmath>
#include <cstdint>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/ix_surrogate.h"

namespace ix {
namespace mlp {
namespace {

// Mean squared error over the m x n outputs: dy = 2 (y - t) / (m n) (f32 and bf16), and
// the loss summed into *loss: a block's share in f64, then one f32 atomic.  The order of the
// atomics is the scheduler's, so their number is what the loss's last bits depend on: 432 at
// 4096 x 27, where one per warp made it 3456, all on one address (6.8 us; 2.5 us so).
constexpr int MSE_THREADS = 256;
__global__ void __launch_bounds__(MSE_THREADS) mse_grad_kernel(int m, int n, const float* __restrict__ y, const float* __restrict__ t,
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
    if (!loss) return;
    __shared__ double s_part[MSE_THREADS / 32];
    double sum = (double)part;
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xFFFFFFFFu, sum, off);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double total_part = 0.0;
        for (int i = 0; i < MSE_THREADS / 32; ++i) total_part += s_part[i];
        atomicAdd(loss, (float)total_part);
    }
}

// db[col] = sum over rows of dz.  Reading the rows bounds it (4 MB at 4096 x 256), so a
// cluster of CTAs takes 32 columns: a warp reads 32 neighbouring columns of one row, each
// thread sums every (32 ranks)-th row, and the partial sums fold in a fixed tree -- the 32 of
// a CTA, then the CTAs in rank order -- whatever the scheduling.  4096 x 256: 235 us with a
// thread per column walking the rows, 7.5 us so.
constexpr int BIAS_ROWS = 32;     // rows of a CTA pass
constexpr int BIAS_CLUSTER = 8;
constexpr int BIAS_WARPS = 4;     // of the wide kernel's CTA
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

// The same sums, in the same order, by one CTA of 4 warps for 32 columns: warp y takes rows y,
// y + 4, ... of a pass, whose partial sums fold in the thread that holds them, and the ranks
// follow one another.  For few rows, where a cluster's barriers are most of its time, and for
// columns enough to fill the GPU without splitting their rows, where 1024-thread CTAs cost
// a wave each (us, clusters / so / a thread per column): 64 x 256 4.8 / 3.9 / 4.0, 33 x 100000
// 68 / 8.3 / 4.3, 1000 x 20000 73 / 14 / 27.  With 2 and 8 warps 64 x 256 takes 8.3 and 4.1,
// 1024 x 16384 74 and 14.4 against 12.4.
__global__ void __launch_bounds__(32 * BIAS_WARPS) bias_grad_wide_kernel(int m, int n, int ranks,
                                                                        const float* __restrict__ dz,
                                                                        float* __restrict__ db) {
    constexpr int WARPS = BIAS_WARPS, ROWS = BIAS_ROWS / WARPS;  // rows of a pass in one thread
    __shared__ float s_part[BIAS_CLUSTER][WARPS][32];
    const int c = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int64_t col = blockIdx.x * (int64_t)32 + c, row = (int64_t)WARPS * n, step = (int64_t)ranks * BIAS_ROWS;
    for (int rank = 0; rank < ranks; ++rank) {
        float v[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) v[i] = 0.0f;
        if (col < n) {
            int64_t r = (int64_t)rank * BIAS_ROWS + y;
            const float* p = dz + r * n + col;
            for (; r + (ROWS - 1) * WARPS < m; r += step, p += step * n) {
#pragma unroll
                for (int i = 0; i < ROWS; ++i) v[i] += p[i * row];
            }
#pragma unroll
            for (int i = 0; i < ROWS - 1; ++i)
                if (r + i * WARPS < m) v[i] += p[i * row];
        }
#pragma unroll
        for (int off = ROWS / 2; off > 0; off >>= 1)
#pragma unroll
            for (int i = 0; i < off; ++i) v[i] += v[i + off];
        s_part[rank][y][c] = v[0];
    }
    __syncthreads();
    if (y == 0 && col < n) {
        float total = 0.0f;
        for (int k = 0; k < ranks; ++k) {
            float v[WARPS];
#pragma unroll
            for (int i = 0; i < WARPS; ++i) v[i] = s_part[k][i][c];
#pragma unroll
            for (int off = WARPS / 2; off > 0; off >>= 1)
#pragma unroll
                for (int i = 0; i < off; ++i) v[i] += v[i + off];
            total += v[0];
        }
        db[col] = total;
    }
}

// Adam on f32 master weights, with their bf16 copy refreshed (Kingma & Ba 2015), of up to
// ADAM_TENSORS tensors: blockIdx.y is the tensor.  A network's tensors are small (at most
// 256 x 256: 1.6 MB of traffic, 2 us), so launches bound the step, and one launch updates
// them all: 8 tensors 42 -> 16 us on the host's clock.
constexpr int ADAM_TENSORS = 16;
struct AdamLaunch {
    ix_mlp_adam_tensor t[ADAM_TENSORS];
    float lr, beta1, beta2, eps, bias1, bias2;
};
__global__ void __launch_bounds__(256) adam_kernel(const __grid_constant__ AdamLaunch L) {
    const ix_mlp_adam_tensor& T = L.t[blockIdx.y];
    __nv_bfloat16* const wb = (__nv_bfloat16*)T.wb;
    const int64_t count = (int64_t)T.count;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = T.g[i];
        const float mi = L.beta1 * T.m[i] + (1.0f - L.beta1) * gi;
        const float vi = L.beta2 * T.v[i] + (1.0f - L.beta2) * gi * gi;
        T.m[i] = mi;
        T.v[i] = vi;
        const float wi = T.w[i] - L.lr * (mi / L.bias1) / (sqrtf(vi / L.bias2) + L.eps);
        T.w[i] = wi;
        if (wb) wb[i] = __float2bfloat16_rn(wi);
    }
}

// The network's standardised outputs as metrics.
__global__ void scale_shift_kernel(int64_t count, uint32_t n, const float* __restrict__ y,
                                   const float* __restrict__ scale, const float* __restrict__ shift,
                                   float* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t c = (uint32_t)(i % n);
        out[i] = __fadd_rn(__fmul_rn(y[i], scale[c]), shift[c]);
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
    mse_grad_kernel<<<grid_for((int64_t)m * n), MSE_THREADS, 0, s>>>(m, n, y, t, dy, (__nv_bfloat16*)dyb, loss);
    return cudaGetLastError();
}
cudaError_t bias_grad(int m, int n, const float* dz, float* db, cudaStream_t s) {
    if (n <= 0) return cudaErrorInvalidValue;  // no columns, or more than an int counts
    // One CTA does while the rows are one pass of it.
    int ranks = 1;
    while (ranks < BIAS_CLUSTER && (int64_t)ranks * BIAS_ROWS < m) ranks *= 2;
    // Clusters pay up to a wave of their CTAs (two an SM: 5 us, 12 ns for each CTA past it); the
    // wide kernel pays 3 us and 7 ns a row.  Either gives the same bits.
    const int64_t groups = ((int64_t)n + 31) / 32, ctas = groups * ranks, wave = 2 * 148;
    if (m <= 128 + 2 * (ctas > wave ? ctas - wave : 0)) {
        bias_grad_wide_kernel<<<(unsigned)groups, 32 * BIAS_WARPS, 0, s>>>(m, n, ranks, dz, db);
        return cudaGetLastError();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(32 * BIAS_ROWS);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, bias_grad_kernel, m, n, dz, db);
    return cudaGetLastError();  // and leaves none for the next call to find
}
cudaError_t adam(uint32_t n, const ix_mlp_adam_tensor* t, float lr, float beta1, float beta2, float eps, float bias1,
                 float bias2, cudaStream_t s) {
    for (uint32_t begin = 0; begin < n; begin += ADAM_TENSORS) {
        const uint32_t k = n - begin < ADAM_TENSORS ? n - begin : ADAM_TENSORS;
        AdamLaunch L{};
        uint64_t most = 0;
        for (uint32_t i = 0; i < k; ++i) {
            L.t[i] = t[begin + i];
            if (L.t[i].count > most) most = L.t[i].count;
        }
        L.lr = lr, L.beta1 = beta1, L.beta2 = beta2, L.eps = eps, L.bias1 = bias1, L.bias2 = bias2;
        adam_kernel<<<dim3(grid_for((int64_t)most), k), 256, 0, s>>>(L);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
cudaError_t scale_shift(int64_t count, uint32_t n, const float* y, const float* scale, const float* shift, float* out,
                        cudaStream_t s) {
    scale_shift_kernel<<<grid_for(count), 256, 0, s>>>(count, n, y, scale, shift, out);
    return cudaGetLastError();
}
cudaError_t to_bf16(int64_t count, const float* x, void* xb, cudaStream_t s) {
    to_bf16_kernel<<<grid_for(count), 256, 0, s>>>(count, x, (__nv_bfloat16*)xb);
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace ix

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
    const ix_mlp_adam_tensor one{count, w, wb, g, m, v};
    return ix_mlp_adam_multi(1, &one, lr, beta1, beta2, eps, t, stream);
}
int ix_mlp_adam_multi(uint32_t n, const ix_mlp_adam_tensor* tensors, float lr, float beta1, float beta2, float eps,
                      uint32_t t, void* stream) {
    if (!tensors || t == 0) return 1;
    for (uint32_t i = 0; i < n; ++i)
        if (!tensors[i].w || !tensors[i].g || !tensors[i].m || !tensors[i].v) return 1;
    const float b1 = 1.0f - std::pow(beta1, (float)t), b2 = 1.0f - std::pow(beta2, (float)t);
    return rc(ix::mlp::adam(n, tensors, lr, beta1, beta2, eps, b1, b2, st(stream)));
}
int ix_mlp_scale_shift(uint32_t m, uint32_t n, const float* y, const float* scale, const float* shift, float* out,
                       void* stream) {
    if (m == 0 || n == 0) return 0;
    if (!y || !scale || !shift || !out) return 1;
    return rc(ix::mlp::scale_shift((int64_t)m * n, n, y, scale, shift, out, st(stream)));
}
int ix_mlp_to_bf16(uint64_t count, const float* x, void* xb, void* stream) {
    if (!x || !xb) return 1;
    return rc(ix::mlp::to_bf16((int64_t)count, x, xb, st(stream)));
}

}  // extern "C"
