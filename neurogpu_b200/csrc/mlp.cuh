// The surrogate network's work beside its GEMMs (gemm_tc.cuh): operand
// preparation, the loss and its gradient, bias gradients, and the Adam step.
//
// As elementwise torch operations these were ~90 launches of a training step
// whose GEMMs take a tenth of a millisecond; each kernel here makes all that
// its point of the step needs in one pass.  What bounds them is their launch:
// a minibatch of 4,096 x 512 is a few megabytes.  So each kernel of a step is
// launched while the one before it runs and waits for its end in
// dependent_wait() (programmatic dependent launch), its first statement that
// touches memory; a kernel ends only after its own wait, so waiting for the
// one before is waiting for all.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ngpu {

// What the step's kernels add into, zeroed by its first kernel: one pass
// instead of five memsets (1.4 us each and a gap).
struct MlpZero {
    float* p[4];
    int64_t n[4];
    unsigned* done;
};

// xb[Mp][k_in] = bf16((X - mu) / sd), zero past M rows and n_in columns; xbt
// its transpose (or nullptr).  mu, sd nullptr: X as it is.  One CTA per 32
// rows, through shared memory so that both are written in rows.  zero: see
// MlpZero.
__global__ void __launch_bounds__(256) k_mlp_input(const float* X, int M, int n_in, const float* mu, const float* sd,
                                                   int Mp, int k_in, __nv_bfloat16* xb, __nv_bfloat16* xbt,
                                                   const MlpZero zero) {
    dependent_launch();
    const int64_t threads = (int64_t)gridDim.x * gridDim.y * 256;
    const int64_t id = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * 256 + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        for (int64_t t = id; t < zero.n[k]; t += threads) zero.p[k][t] = 0.f;
    if (zero.done && id == 0) *zero.done = 0;
    __shared__ __nv_bfloat16 tile[32][33];
    const int m0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int r = threadIdx.x >> 5; r < 32; r += 8) {
        const int m = m0 + r, c = c0 + (threadIdx.x & 31);
        float x = 0.f;
        if (m < M && c < n_in) {
            x = X[(size_t)m * n_in + c];
            if (mu) x = __fdiv_rn(__fsub_rn(x, mu[c]), sd[c]);
        }
        const __nv_bfloat16 h = __float2bfloat16_rn(x);
        tile[r][threadIdx.x & 31] = h;
        if (m < Mp) xb[(size_t)m * k_in + c] = h;
    }
    if (!xbt) return;
    __syncthreads();
    for (int r = threadIdx.x >> 5; r < 32; r += 8) {
        const int c = c0 + r, m = m0 + (threadIdx.x & 31);
        if (m < Mp) xbt[(size_t)c * Mp + m] = tile[threadIdx.x & 31][r];
    }
}

// out[M][n_out] = y[.][n_out_p] * sd + mu (nullptr: y as it is)
__global__ void __launch_bounds__(256) k_mlp_output(const float* y, int M, int n_out, int n_out_p, const float* mu,
                                                    const float* sd, float* out) {
    dependent_wait();
    const size_t total = (size_t)M * n_out;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t m = t / n_out;
        const int c = (int)(t % n_out);
        float v = y[m * n_out_p + c];
        if (mu) v = __fadd_rn(__fmul_rn(v, sd[c]), mu[c]);
        out[t] = v;
    }
}

// Loss and its gradient at the output: diff = (y - target) * weight, target
// standardised; dy = 2 diff / count as bf16, row-major [Mp][64] (zero past
// n_out columns and M rows) and transposed [n_out_p][Mp].  A CTA per 32 rows
// leaves its sum of diff^2 and its column sums of dy in part[block][1 +
// n_out_p]; the last CTA to finish adds them up in block order.
struct MlpLossArgs {
    const float* y;          // [Mp][n_out_p]
    const float* Y;          // [M][n_out] targets
    const float* mu;         // target statistics, or nullptr
    const float* sd;
    const float* weight;     // [M], or nullptr
    int M, Mp, n_out, n_out_p;
    __nv_bfloat16* dyb;
    __nv_bfloat16* dybt;
    float* part;
    unsigned* done;          // zeroed before
    float* loss;
    float* gb;               // [n_out_p]
};
constexpr int kMlpLossRows = 32;
__global__ void __launch_bounds__(256) k_mlp_loss(const MlpLossArgs a) {
    __shared__ float d_s[kMlpLossRows][65];
    __shared__ float sq_s[8];
    __shared__ bool last;
    const int m0 = blockIdx.x * kMlpLossRows;
    const float count = (float)((int64_t)a.M * a.n_out);
    // a thread has eight rows of a column; their loads go out together (where
    // each row's waited for the row before, the kernel took 14 us)
    constexpr int kRows = kMlpLossRows / 4;
    const int c = threadIdx.x & 63, r0 = threadIdx.x >> 6;
    const bool col = c < a.n_out;
    float target[kRows], y[kRows], weight[kRows], sq = 0.f;
    dependent_launch();
    dependent_wait();
    const float mu = col && a.mu ? a.mu[c] : 0.f, sd = col && a.mu ? a.sd[c] : 1.f;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
        const int m = m0 + r0 + 4 * k;
        const bool in = col && m < a.M;
        target[k] = in ? a.Y[(size_t)m * a.n_out + c] : 0.f;
        weight[k] = in && a.weight ? a.weight[m] : 1.f;
        y[k] = in ? a.y[(size_t)m * a.n_out_p + c] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
        const int r = r0 + 4 * k, m = m0 + r;
        float dy = 0.f;
        if (col && m < a.M) {
            float t = target[k];
            if (a.mu) t = __fdiv_rn(__fsub_rn(t, mu), sd);
            float diff = __fsub_rn(y[k], t);
            if (a.weight) diff = __fmul_rn(diff, weight[k]);
            sq += diff * diff;
            dy = __fdiv_rn(2.0f * diff, count);
        }
        d_s[r][c] = dy;
        if (m < a.Mp) a.dyb[(size_t)m * 64 + c] = __float2bfloat16_rn(dy);
    }
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
    if ((threadIdx.x & 31) == 0) sq_s[threadIdx.x >> 5] = sq;
    __syncthreads();
    for (int t = threadIdx.x; t < a.n_out_p * kMlpLossRows; t += 256) {
        const int tc = t / kMlpLossRows, r = t % kMlpLossRows;
        if (m0 + r < a.Mp) a.dybt[(size_t)tc * a.Mp + m0 + r] = __float2bfloat16_rn(d_s[r][tc]);
    }
    const int np = 1 + a.n_out_p;
    if (threadIdx.x < np) {
        float s = 0.f;
        if (threadIdx.x == 0) {
            for (int t = 0; t < 8; ++t) s += sq_s[t];
        } else {
#pragma unroll
            for (int r = 0; r < kMlpLossRows; ++r) s += d_s[r][threadIdx.x - 1];
        }
        a.part[(size_t)blockIdx.x * np + threadIdx.x] = s;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(a.done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    // four threads per sum, each every fourth block (np <= 65)
    __shared__ double sum_s[4][65];
    for (int t = threadIdx.x; t < 4 * np; t += 256) {
        const int k = t % np, q = t / np;
        double s = 0.0;
#pragma unroll 16
        for (unsigned b = q; b < gridDim.x; b += 4) s += (double)__ldcg(a.part + (size_t)b * np + k);
        sum_s[q][k] = s;
    }
    __syncthreads();
    if (threadIdx.x < np) {
        const int k = threadIdx.x;
        const double s = (sum_s[0][k] + sum_s[1][k]) + (sum_s[2][k] + sum_s[3][k]);
        if (k == 0) *a.loss = __fdiv_rn((float)s, count);
        else a.gb[k - 1] = (float)s;
    }
}

// Bias gradients of the hidden layers: gb[l][n] = the sum of row n of the
// layer's dZ^T [width][Mp].  A CTA per row.
struct MlpBiasArgs {
    const __nv_bfloat16* dzt[3];
    float* gb[3];
    int Mp;                  // a multiple of 128
};
__global__ void __launch_bounds__(128) k_mlp_bias_grads(const MlpBiasArgs a) {
    const __nv_bfloat162* row =
        reinterpret_cast<const __nv_bfloat162*>(a.dzt[blockIdx.y] + (size_t)blockIdx.x * a.Mp);
    float s = 0.f;
    dependent_wait();
    for (int t = threadIdx.x; t < a.Mp / 2; t += 128) {
        const float2 f = __bfloat1622float2(row[t]);
        s += f.x + f.y;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    __shared__ float part[4];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) a.gb[blockIdx.y][blockIdx.x] = (part[0] + part[1]) + (part[2] + part[3]);
}

// out[c][r] = in[r][c], float
__global__ void __launch_bounds__(256) k_mlp_transpose(const float* in, int rows, int cols, float* out) {
    __shared__ float tile[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32, x = threadIdx.x & 31;
    dependent_launch();
    dependent_wait();
    for (int k = threadIdx.x >> 5; k < 32; k += 8)
        if (r0 + k < rows && c0 + x < cols) tile[k][x] = in[(size_t)(r0 + k) * cols + c0 + x];
    __syncthreads();
    for (int k = threadIdx.x >> 5; k < 32; k += 8)
        if (c0 + k < cols && r0 + x < rows) out[(size_t)(c0 + k) * rows + r0 + x] = tile[x][k];
}

// One Adam step of every weight and bias, with the bf16 copies of the new
// weights (row-major, and transposed; the output layer's transpose padded to
// 64 columns with zeros).  Weight columns / rows past the network's own
// inputs and outputs stay zero.  A CTA per 32 x 32 tile of a weight matrix,
// and per 1,024 entries of a bias.
struct MlpAdamArgs {
    float* p[8];             // W 0..3, b 0..3
    const float* g[8];
    float* m[8];
    float* v[8];
    __nv_bfloat16* wb[4];
    __nv_bfloat16* wtb[4];
    int rows[8], cols[8];    // a bias: rows 1
    int ldt[4];              // columns of the transposed copy
    int tile0[9];            // first CTA of each tensor
    int n_in, n_out;
    float lr, b1, b2, d1, d2, eps, c1, c2;  // d1 = 1 - b1, d2 = 1 - b2 (rounded once each)
};
__device__ __forceinline__ float mlp_adam(const MlpAdamArgs& a, int k, size_t o, bool keep) {
    const float g = a.g[k][o];
    const float m = fmaf(a.d1, g, a.m[k][o] * a.b1);
    const float v = fmaf(a.d2 * g, g, a.v[k][o] * a.b2);
    a.m[k][o] = m;
    a.v[k][o] = v;
    float p = a.p[k][o] - a.lr * __fdiv_rn(__fdiv_rn(m, a.c1), __fadd_rn(__fsqrt_rn(__fdiv_rn(v, a.c2)), a.eps));
    if (!keep) p = 0.f;
    a.p[k][o] = p;
    return p;
}
__global__ void __launch_bounds__(256) k_mlp_adam(const MlpAdamArgs a) {
    __shared__ __nv_bfloat16 tile[32][33];
    int k = 0;
    while (k < 7 && (int)blockIdx.x >= a.tile0[k + 1]) ++k;
    const int t = blockIdx.x - a.tile0[k], x = threadIdx.x & 31;
    const int rows = a.rows[k], cols = a.cols[k];
    if (k >= 4) {
        for (int c = t * 1024 + threadIdx.x; c < min(cols, (t + 1) * 1024); c += 256)
            mlp_adam(a, k, c, k < 7 || c < a.n_out);
        return;
    }
    const int tc = (cols + 31) / 32, r0 = (t / tc) * 32, c0 = (t % tc) * 32;
    for (int r = threadIdx.x >> 5; r < 32; r += 8) {
        const int i = r0 + r, c = c0 + x;
        if (i < rows && c < cols) {
            const size_t o = (size_t)i * cols + c;
            const __nv_bfloat16 h =
                __float2bfloat16_rn(mlp_adam(a, k, o, (k != 0 || c < a.n_in) && (k != 3 || i < a.n_out)));
            a.wb[k][o] = h;
            tile[r][x] = h;
        }
    }
    __syncthreads();
    const int ldt = a.ldt[k];
    for (int r = threadIdx.x >> 5; r < 32; r += 8) {
        const int c = c0 + r, i = r0 + x;
        if (c < cols && i < rows && i < ldt) a.wtb[k][(size_t)c * ldt + i] = tile[x][r];
        // the padding columns of the transpose, by the tiles of the last rows
        if (c < cols && r0 + 32 >= rows)
            for (int q = rows + x; q < ldt; q += 32) a.wtb[k][(size_t)c * ldt + q] = __float2bfloat16_rn(0.f);
    }
}

}  // namespace ngpu
