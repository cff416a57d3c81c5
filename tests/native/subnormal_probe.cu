// Test-only kernels: the channel headers' functions in FP32 over a range of
// every float's bits, in the form that the product compiles (namespace
// product) and with the general exponential and quotient throughout
// (namespace general).  Compiled by tests/test_subnormals.py against two
// copies of the headers.
#include <cuda_runtime.h>
#include <stdint.h>

#define ngpu product
#include "product/channels_ttpc.cuh"
#undef ngpu
#define ngpu general
#undef NGPU_HD
#include "general/channels_ttpc.cuh"
#undef ngpu

#define FUNCTIONS(N)                                                                            \
    {                                                                                           \
        using M = N::Math<float>;                                                               \
        using Q = N::TTPCRates<float>;                                                          \
        int k = 0;                                                                              \
        float a, b, c, d;                                                                       \
        out[k++] = N::efun(x);                                                                  \
        N::efun_pair(x, a, b);                                                                  \
        out[k++] = a; out[k++] = b;                                                             \
        out[k++] = N::sigm(x);                                                                  \
        out[k++] = M::one_minus_exp_neg(x);                                                     \
        out[k++] = M::em1(x);                                                                   \
        Q::ca_hva(x, a, b, c, d); out[k++] = a; out[k++] = b; out[k++] = c; out[k++] = d;       \
        Q::ca_lva(x, a, b, c, d); out[k++] = a; out[k++] = b; out[k++] = c; out[k++] = d;       \
        Q::ih(x, a, b); out[k++] = a; out[k++] = b;                                             \
        Q::im(x, a, b); out[k++] = a; out[k++] = b;                                             \
        Q::k_pst(x, a, b, c, d); out[k++] = a; out[k++] = b; out[k++] = c; out[k++] = d;        \
        Q::k_tst(x, a, b, c, d); out[k++] = a; out[k++] = b; out[k++] = c; out[k++] = d;        \
        Q::nap(x, a, b, c, d); out[k++] = a; out[k++] = b; out[k++] = c; out[k++] = d;          \
        Q::nat(x, -38.f, -66.f, a, b, c, d); out[k++] = a; out[k++] = b; out[k++] = c; out[k++] = d; \
        out[k++] = Q::sk_zinf(x);                                                               \
        Q::skv3(x, a, b); out[k++] = a; out[k++] = b;                                           \
    }
constexpr int kOut = 37;

// differ[k]: inputs for which output k differs between the two
__global__ void k_compare(unsigned long long* differ, unsigned* at) {
    __shared__ unsigned long long s[kOut];
    if (threadIdx.x < kOut) s[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < (1ull << 32); t += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((unsigned)t);
        float p[kOut], g[kOut];
        {
            float* out = p;
            FUNCTIONS(product)
        }
        {
            float* out = g;
            FUNCTIONS(general)
        }
#pragma unroll
        for (int k = 0; k < kOut; ++k)
            if (__float_as_uint(p[k]) != __float_as_uint(g[k]) && !(p[k] != p[k] && g[k] != g[k])) {
                atomicAdd(&s[k], 1ull);
                at[k] = (unsigned)t;
            }
    }
    __syncthreads();
    if (threadIdx.x < kOut && s[threadIdx.x]) atomicAdd(differ + threadIdx.x, s[threadIdx.x]);
}

extern "C" int probe_outputs() { return kOut; }
extern "C" int probe_compare(unsigned long long* differ, unsigned* at) {
    k_compare<<<148 * 8, 256>>>(differ, at);
    return (int)cudaDeviceSynchronize();
}
