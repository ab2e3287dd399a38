// arc_norm.cu - one step of VecNormalize's running normalisation on the
// device (vec_env.py: Stable-Baselines3's algorithm, FP64 statistics).
//
// Bound by memory and launches: the batch is read for its moments, and read
// and written once to normalise it. As tensor operations the same step took
// 55 launches (six FP64 copies of the batch among them) and 207 us of GPU
// time at 10,007 x 195; here three launches and 25 us (4.5, 4.8 and 16; the
// 40 MB read and written take 6 us at the copy rate, the rest is the FP64
// arithmetic per element and launch latency):
//   k_norm_moments  per block of rows and 256 columns: sums of (x - x0) and
//                   (x - x0)^2 in FP64, x0 the column's first row, so that a
//                   constant column has no variance at all; the last column
//                   of blocks does the same for the discounted returns.
//   k_norm_merge    a warp per column adds the blocks' sums and merges them
//                   into the running statistics (Chan, Golub, LeVeque 1979).
//   k_norm_apply    observations, terminal observations, rewards; the ended
//                   worlds' returns to zero.
// Sums are added in one order, so a step gives the same bits every time.
#include "arc_kernels.cuh"
#include "../../include/arc_sim.h"

namespace arc {

namespace {

constexpr int kNormThreads = 256;
constexpr int kNormMaxCols = 2048;   // mean and scale of every column in shared memory
constexpr int kNormBlocks = 256;     // blocks of rows at most

int norm_row_blocks(long long rows)
{
    const long long blocks = (rows + 31) / 32;  // at least 32 rows each
    return (int)(blocks < kNormBlocks ? blocks : kNormBlocks);
}

// The new discounted return of row i (two roundings, as the tensor form).
__device__ __forceinline__ double next_return(const arc_norm_step_args& a, long long i)
{
    return a.training ? __dadd_rn(__dmul_rn(a.returns[i], a.gamma), (double)a.rewards[i]) : a.returns[i];
}

// The value a column's sums are taken around: its first row's, if finite.
__device__ __forceinline__ double origin_of(double first) { return isfinite(first) ? first : 0.0; }

// blockIdx.y: a tile of 256 columns, or (the last, when training) the
// returns. work: [2][row blocks][cols + 1] sums.
__global__ void __launch_bounds__(kNormThreads) k_norm_moments(const __grid_constant__ arc_norm_step_args a)
{
    const int tid = threadIdx.x, col = blockIdx.y * kNormThreads + tid, blocks = gridDim.x;
    const long long per = (a.rows + blocks - 1) / blocks, r0 = blockIdx.x * per;
    const long long r1 = r0 + per < a.rows ? r0 + per : a.rows;
    double* first = a.work + (size_t)blockIdx.x * (a.cols + 1);
    double* second = first + (size_t)blocks * (a.cols + 1);
    double s = 0.0, q = 0.0;
    if (blockIdx.y + 1 < gridDim.y) {
        if (col >= a.cols || !a.norm_obs)
            return;
        const double x0 = origin_of((double)a.obs[col]);
        const float* x = a.obs + (size_t)r0 * a.cols + col;
        long long r = r0;
        for (; r + 8 <= r1; r += 8, x += (size_t)8 * a.cols) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                v[u] = x[(size_t)u * a.cols];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const double d = (double)v[u] - x0;
                s += d;
                q = __fma_rn(d, d, q);
            }
        }
        for (; r < r1; ++r, x += a.cols) {
            const double d = (double)*x - x0;
            s += d;
            q = __fma_rn(d, d, q);
        }
        first[col] = s;
        second[col] = q;
        return;
    }
    __shared__ double sum[2][kNormThreads / 32];
    const double x0 = origin_of(next_return(a, 0));
    for (long long r = r0 + tid; r < r1; r += kNormThreads) {
        const double d = next_return(a, r) - x0;
        s += d;
        q = __fma_rn(d, d, q);
    }
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, off);
        q += __shfl_xor_sync(0xffffffffu, q, off);
    }
    if ((tid & 31) == 0) {
        sum[0][tid / 32] = s;
        sum[1][tid / 32] = q;
    }
    __syncthreads();
    if (tid == 0) {
        s = q = 0.0;
        for (int w = 0; w < kNormThreads / 32; ++w) {
            s += sum[0][w];
            q += sum[1][w];
        }
        first[a.cols] = s;
        second[a.cols] = q;
    }
}

// A warp per column (the last: the returns).
__global__ void __launch_bounds__(kNormThreads) k_norm_merge(const __grid_constant__ arc_norm_step_args a, int blocks)
{
    const int col = blockIdx.x * (kNormThreads / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (col > a.cols || (col < a.cols && !a.norm_obs))
        return;
    const double* first = a.work + col;
    const double* second = first + (size_t)blocks * (a.cols + 1);
    double s = 0.0, q = 0.0;
    for (int b = lane; b < blocks; b += 32) {
        s += first[(size_t)b * (a.cols + 1)];
        q += second[(size_t)b * (a.cols + 1)];
    }
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, off);
        q += __shfl_xor_sync(0xffffffffu, q, off);
    }
    if (lane != 0)
        return;
    const bool ret = col == a.cols;
    const double n = (double)a.rows, shift = s / n;
    const double batch_mean = origin_of(ret ? next_return(a, 0) : (double)a.obs[col]) + shift;
    double batch_var = q / n - shift * shift;
    batch_var = batch_var < 0.0 ? 0.0 : batch_var;  // NaN stays
    const double mean = ret ? *a.ret_mean : a.obs_mean[col], var = ret ? *a.ret_var : a.obs_var[col];
    const double count = ret ? a.ret_count : a.obs_count, total = count + n;
    const double delta = batch_mean - mean;
    const double m2 = var * count + batch_var * n + delta * delta * (count * n / total);
    (ret ? a.ret_mean_out : a.obs_mean_out + col)[0] = mean + delta * (n / total);
    (ret ? a.ret_var_out : a.obs_var_out + col)[0] = m2 / total;
}

__device__ __forceinline__ double clip_to(double v, double c) { return v < -c ? -c : (v > c ? c : v); }

// blockIdx.y: 0 the observations (and, in the first blocks, rewards and
// returns), 1 the terminal observations.
__global__ void __launch_bounds__(kNormThreads) k_norm_apply(const __grid_constant__ arc_norm_step_args a)
{
    extern __shared__ double stats[];
    const int tid = threadIdx.x;
    const float* src = blockIdx.y ? a.terminal_obs : a.obs;
    float* dst = blockIdx.y ? a.terminal_out : a.obs_out;
    const bool updated = a.training && a.norm_obs;
    if (src && dst) {
        double* mean = stats;
        double* scale = stats + a.cols;
        for (int c = tid; c < a.cols; c += kNormThreads) {
            mean[c] = updated ? a.obs_mean_out[c] : a.obs_mean[c];
            scale[c] = 1.0 / sqrt((updated ? a.obs_var_out[c] : a.obs_var[c]) + a.epsilon);
        }
        __syncthreads();
        const size_t total = (size_t)a.rows * a.cols;
        const size_t step = (size_t)gridDim.x * kNormThreads;
        size_t e = (size_t)blockIdx.x * kNormThreads + tid;
        int c = (int)(e % a.cols);
        const int dc = (int)(step % a.cols);
        for (; e < total; e += step) {
            dst[e] = (float)clip_to(((double)src[e] - mean[c]) * scale[c], a.clip_obs);
            c += dc;
            c -= c >= a.cols ? a.cols : 0;
        }
    }
    if (blockIdx.y)
        return;
    const double rs = a.norm_reward ? sqrt((a.training ? *a.ret_var_out : *a.ret_var) + a.epsilon) : 1.0;
    for (long long i = (long long)blockIdx.x * kNormThreads + tid; i < a.rows;
         i += (long long)gridDim.x * kNormThreads) {
        if (a.norm_reward)
            a.rewards_out[i] = (float)clip_to((double)a.rewards[i] / rs, a.clip_reward);
        a.returns_out[i] = a.dones[i] ? 0.0 : next_return(a, i);
    }
}

}  // namespace

}  // namespace arc

extern "C" {

long long arc_norm_work_size(long long rows, int cols)
{
    return rows > 0 && cols > 0 ? 2ll * arc::norm_row_blocks(rows) * (cols + 1) : 0;
}

int arc_norm_step(const arc_norm_step_args* a, void* stream)
{
    using namespace arc;
    if (!a || a->rows <= 0 || a->cols <= 0 || a->cols > kNormMaxCols || !a->obs || !a->rewards || !a->dones ||
        !a->returns || !a->returns_out || !a->work || (a->norm_reward && !a->rewards_out))
        return ARC_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const int blocks = norm_row_blocks(a->rows);
    if (a->training) {
        const dim3 grid(blocks, (a->cols + kNormThreads - 1) / kNormThreads + 1);
        k_norm_moments<<<grid, kNormThreads, 0, st>>>(*a);
        k_norm_merge<<<(a->cols + 1 + kNormThreads / 32 - 1) / (kNormThreads / 32), kNormThreads, 0, st>>>(*a, blocks);
    }
    const size_t each = (size_t)a->rows * a->cols, per_block = (size_t)kNormThreads * 8;
    const size_t want = (each + per_block - 1) / per_block;
    k_norm_apply<<<dim3((unsigned)(want < 1024 ? want : 1024), a->terminal_obs && a->terminal_out ? 2 : 1), kNormThreads,
                   2 * sizeof(double) * a->cols, st>>>(*a);
    return cudaGetLastError() == cudaSuccess ? ARC_OK : ARC_ERR_CUDA;
}

}  // extern "C"
