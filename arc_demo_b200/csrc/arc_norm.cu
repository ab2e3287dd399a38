// arc_norm.cu - one step of VecNormalize's running normalisation on the
// device (vec_env.py: Stable-Baselines3's algorithm, FP64 statistics).
//
// Bound by memory and launches: the batch is read for its moments, and read
// and written once to normalise it. As tensor operations the same step took
// 55 launches (six FP64 copies of the batch among them) and 207 us of GPU
// time at 10,007 x 195; here three launches and 30 us within a training step
// (5.3, 7.1 and 17.9; with nothing else running 25; the 40 MB read and written take 6 us at the copy rate, the
// rest is the FP64 arithmetic per element and launch latency):
//   k_norm_moments  per block of rows and 256 columns: the column's mean and
//                   sum of squared deviations from it, in FP64 and two passes
//                   (the second reads from L1 and L2) with the deviations'
//                   own sum as the correction (Chan, Golub, LeVeque 1983); the
//                   last column of blocks does the same for the discounted
//                   returns.
//   k_norm_merge    a warp per column merges the blocks' moments in the same
//                   two passes, and the result into the running statistics
//                   (Chan, Golub, LeVeque 1979). A constant column has no
//                   variance at all, and no row is a reference for the others:
//                   in one pass around the first row's values (3.8 and 4.4
//                   us) a first row 1,000 deviations out cost the variance
//                   three digits.
//   k_norm_apply    observations, terminal observations, rewards; the ended
//                   worlds' returns to zero. Divides by the deviation: with a
//                   product by its reciprocal it took 11.2 us, and rounded
//                   once more than a division.
// Sums are added in one order, so a step gives the same bits every time.
#include "arc_kernels.cuh"
#include "../../include/arc_sim.h"

namespace arc {

namespace {

constexpr int kNormThreads = 256;
constexpr int kNormMaxCols = 2048;   // mean, deviation and its reciprocal of every column in shared memory
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

// The rows of block b of `blocks`: first, and how many.
__device__ __forceinline__ void rows_of(long long rows, int blocks, int b, long long& first, int& count)
{
    const long long per = (rows + blocks - 1) / blocks;
    first = b * per;
    const long long left = rows - first;
    count = (int)(left < per ? (left > 0 ? left : 0) : per);
}

// Of n values whose deviations from the rounded mean `hi` sum to s and their
// squares to q: the mean's rest, and the squared deviations' sum from hi + rest.
struct Moments {
    double rest, m2;
};
__device__ __forceinline__ Moments corrected(double hi, double s, double q, double n)
{
    const double m2 = q - s * (s / n);
    return Moments{isfinite(hi) ? s / n : 0.0, m2 < 0.0 ? 0.0 : m2};  // NaN stays
}

// The sums of s and q over the block, to every thread.
__device__ __forceinline__ void block_sums(double& s, double& q)
{
    __shared__ double sum[2][kNormThreads / 32];
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, off);
        q += __shfl_xor_sync(0xffffffffu, q, off);
    }
    __syncthreads();  // an earlier call's sums are read
    if ((threadIdx.x & 31) == 0) {
        sum[0][threadIdx.x / 32] = s;
        sum[1][threadIdx.x / 32] = q;
    }
    __syncthreads();
    s = q = 0.0;
    for (int w = 0; w < kNormThreads / 32; ++w) {
        s += sum[0][w];
        q += sum[1][w];
    }
}

// f(x[0]), f(x[cols]), ..., `count` of them, eight loads in flight.
template <class Fn> __device__ __forceinline__ void each_row(const float* x, int count, int cols, Fn&& f)
{
    int r = 0;
    for (; r + 8 <= count; r += 8, x += (size_t)8 * cols) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            v[u] = x[(size_t)u * cols];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            f((double)v[u]);
    }
    for (; r < count; ++r, x += cols)
        f((double)*x);
}

// blockIdx.y: a tile of 256 columns, or (the last, when training) the
// returns. work: [3][row blocks][cols + 1] means, their rests (a block's mean
// rounded to FP64 is too far off where the deviations are small beside it),
// sums of squares.
__global__ void __launch_bounds__(kNormThreads) k_norm_moments(const __grid_constant__ arc_norm_step_args a)
{
    const int tid = threadIdx.x, col = blockIdx.y * kNormThreads + tid, blocks = gridDim.x;
    long long r0;
    int count;
    rows_of(a.rows, blocks, blockIdx.x, r0, count);
    if (count == 0)
        return;  // k_norm_merge does not read its moments
    const size_t plane = (size_t)blocks * (a.cols + 1);
    double* out = a.work + (size_t)blockIdx.x * (a.cols + 1);
    double s = 0.0, q = 0.0;
    if (blockIdx.y + 1 < gridDim.y) {
        if (col >= a.cols || !a.norm_obs)
            return;
        const float* x = a.obs + (size_t)r0 * a.cols + col;
        each_row(x, count, a.cols, [&](double v) { s += v; });
        const double mean = s / count;
        s = 0.0;
        each_row(x, count, a.cols, [&](double v) {
            const double d = v - mean;
            s += d;
            q = __fma_rn(d, d, q);
        });
        const Moments m = corrected(mean, s, q, count);
        out[col] = mean;
        out[plane + col] = m.rest;
        out[2 * plane + col] = m.m2;
        return;
    }
    for (int r = tid; r < count; r += kNormThreads)
        s += next_return(a, r0 + r);
    block_sums(s, q);
    const double mean = s / count;
    s = q = 0.0;
    for (int r = tid; r < count; r += kNormThreads) {
        const double d = next_return(a, r0 + r) - mean;
        s += d;
        q = __fma_rn(d, d, q);
    }
    block_sums(s, q);
    if (tid == 0) {
        const Moments m = corrected(mean, s, q, count);
        out[a.cols] = mean;
        out[plane + a.cols] = m.rest;
        out[2 * plane + a.cols] = m.m2;
    }
}

// A warp per column (the last: the returns).
__global__ void __launch_bounds__(kNormThreads) k_norm_merge(const __grid_constant__ arc_norm_step_args a, int blocks)
{
    const int col = blockIdx.x * (kNormThreads / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (col > a.cols || (col < a.cols && !a.norm_obs))
        return;
    constexpr int kEach = kNormBlocks / 32;
    const size_t plane = (size_t)blocks * (a.cols + 1);
    double mean_of[kEach], rest_of[kEach], m2_of[kEach], n_of[kEach];
    double s = 0.0, q = 0.0;
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
        const int b = lane + 32 * u;
        long long first = 0;
        int count = 0;
        if (b < blocks)
            rows_of(a.rows, blocks, b, first, count);
        const double* at = a.work + (size_t)b * (a.cols + 1) + col;
        n_of[u] = count;
        mean_of[u] = count ? at[0] : 0.0;
        rest_of[u] = count ? at[plane] : 0.0;
        m2_of[u] = count ? at[2 * plane] : 0.0;
        s += n_of[u] * (mean_of[u] + rest_of[u]);
    }
    for (int off = 16; off > 0; off >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, off);
    const double n = (double)a.rows, hi = s / n;
    s = 0.0;
#pragma unroll
    for (int u = 0; u < kEach; ++u)
        if (n_of[u] != 0.0) {
            const double d = mean_of[u] - hi + rest_of[u];
            s += n_of[u] * d;
            q += m2_of[u] + n_of[u] * d * d;
        }
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, off);
        q += __shfl_xor_sync(0xffffffffu, q, off);
    }
    if (lane != 0)
        return;
    const Moments m = corrected(hi, s, q, n);
    const double batch_mean = hi + m.rest;
    const bool ret = col == a.cols;
    const double batch_var = m.m2 / n;
    const double mean = ret ? *a.ret_mean : a.obs_mean[col], var = ret ? *a.ret_var : a.obs_var[col];
    const double count = ret ? a.ret_count : a.obs_count, total = count + n;
    const double delta = batch_mean - mean;
    const double m2 = var * count + batch_var * n + delta * delta * (count * n / total);
    (ret ? a.ret_mean_out : a.obs_mean_out + col)[0] = mean + delta * (n / total);
    (ret ? a.ret_var_out : a.obs_var_out + col)[0] = m2 / total;
}

// a / b where y = 1 / b, infinities and NaN as a division gives them
__device__ __forceinline__ double quotient(double a, double b, double y)
{
    const double q = divide(a, b, y);
    return isfinite(q) ? q : a * y;
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
        double* dev = stats + a.cols;
        double* scale = dev + a.cols;
        for (int c = tid; c < a.cols; c += kNormThreads) {
            mean[c] = updated ? a.obs_mean_out[c] : a.obs_mean[c];
            dev[c] = sqrt((updated ? a.obs_var_out[c] : a.obs_var[c]) + a.epsilon);
            scale[c] = 1.0 / dev[c];
        }
        __syncthreads();
        const size_t total = (size_t)a.rows * a.cols;
        const size_t step = (size_t)gridDim.x * kNormThreads;
        size_t e = (size_t)blockIdx.x * kNormThreads + tid;
        int c = (int)(e % a.cols);
        const int dc = (int)(step % a.cols);
        for (; e < total; e += step) {
            dst[e] = (float)clip_to(quotient((double)src[e] - mean[c], dev[c], scale[c]), a.clip_obs);
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
    return rows > 0 && cols > 0 ? 3ll * arc::norm_row_blocks(rows) * (cols + 1) : 0;
}

int arc_norm_step(const arc_norm_step_args* a, void* stream)
{
    using namespace arc;
    if (!a || a->rows <= 0 || a->cols <= 0 || a->cols > kNormMaxCols || !a->obs || !a->rewards || !a->dones ||
        !a->returns || !a->returns_out || !a->work || (a->norm_reward && !a->rewards_out))
        return ARC_ERR_ARG;
    // the statistics that the step reads and writes
    const bool reads_obs = (a->training && a->norm_obs) || a->obs_out || (a->terminal_obs && a->terminal_out);
    if ((reads_obs && (!a->obs_mean || !a->obs_var)) ||
        (a->training && a->norm_obs && (!a->obs_mean_out || !a->obs_var_out)) ||
        (a->training && (!a->ret_mean || !a->ret_mean_out || !a->ret_var_out)) ||
        ((a->training || a->norm_reward) && !a->ret_var))
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
                   3 * sizeof(double) * a->cols, st>>>(*a);
    return cudaGetLastError() == cudaSuccess ? ARC_OK : ARC_ERR_CUDA;
}

}  // extern "C"
