// Parameter-exploration score of many voltage traces, a warp per 32 traces and
// stretch of time:
// the number of peaks of dV/dt that scipy.signal.find_peaks(dvdt, height,
// distance) returns (scipy 1.x; not vendored in the reference).  This is the
// score of the reference's exploration run (GUI/plot_param_explor.py:77-107:
// dvdt = numpy.diff(v) / dt, find_peaks(dvdt, 15, distance=5), the count),
// computed where the traces lie instead of on the host after a 554 MB
// VHotP0.dat readback.
//
// The steps are scipy's published ones:
//   1. local maxima of x = dvdt: x[i-1] < x[i] followed by a run of samples
//      equal to x[i] and then a smaller sample; the peak is the middle of the
//      run ((first + last) // 2); first and last samples never peak;
//   2. heights: keep peaks with x >= height;
//   3. distance: visit peaks by decreasing height and remove every peak
//      closer than `distance` samples to a kept one (equal heights: the later
//      peak first, which is the order of a stable sort; scipy leaves the order
//      of ties to numpy's unstable argsort).
// Step 3 is done per cluster (a maximal run of peaks whose neighbours are
// closer than `distance`): peaks of different clusters never remove each
// other.
//
// dvdt is computed as here in double from the float32 trace: ((double)v[j+1]
// - (double)v[j]) / dt, the value numpy computes from the same samples read
// as float64 (the difference of two float32 values in this range is exact
// in double and the quotient is correctly rounded), so every comparison
// matches.
//
// Scratch: the candidate peaks' sample positions, [cap][n_traces] int32 with
// cap = n_samples / 2 + 1 (peaks are at least two samples apart); threads of a
// warp touch one row at a time, consecutive traces.
//
// A trace is scanned in stretches side by side (k_dvdt_peaks): whether a rise
// at sample j starts a peak depends on x[j-1], x[j] and the first later
// sample that differs from x[j], so the stretch that holds j decides alone.
// The scan compares differences instead of quotients, which order alike
// unless two different differences round to one quotient; that takes
// differences within 2^-51 of each other, which samples with 2^-17 <= |v| <
// 2^8 cannot have (their differences are exact multiples of 2^-40 below
// 2^9).  Around any other sample (0, NaN, infinities, beyond 256 mV) the
// quotients themselves are compared.  Differences are compared as float32
// first: rounding keeps their order, so where two round apart they are apart
// that way, and where every |difference| is below every |v| they are exact
// (the samples of a pair then lie within a factor of two).  Only a batch with
// two equal rounded differences that may not be exact compares in float64.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace ngpu {

struct PeakArgs {
    const float* v;
    int64_t stride_trace, stride_sample;
    int n_traces, n_samples;
    double dt, height;
    int distance;
    int32_t* pos;      // scratch [cap][n_traces]
    int cap;
    int32_t* out;      // [n_traces] peak counts
};

__host__ __device__ inline int peak_scratch_cap(int n_samples) { return n_samples / 2 + 1; }

__host__ __device__ __forceinline__ double dvdt_at(const PeakArgs& a, const float* v, int j) {
    return ((double)v[(int64_t)(j + 1) * a.stride_sample] - (double)v[(int64_t)j * a.stride_sample]) / a.dt;
}

// Removed peaks carry kPeakGone in their position word, kept ones kPeakKept.
constexpr int32_t kPeakGone = 1 << 30, kPeakKept = 1 << 29;

// Step 3, distance, cluster by cluster, over the m candidates of a trace (in
// position order, ps elements apart): the peaks kept.
__host__ __device__ inline int peaks_keep(const PeakArgs& a, const float* v, int32_t* pos, int64_t ps, int m) {
    const int d = a.distance;
    int kept = 0;
    int c0 = 0;
    while (c0 < m) {
        int c1 = c0 + 1;
        while (c1 < m && pos[(int64_t)c1 * ps] - pos[(int64_t)(c1 - 1) * ps] < d) ++c1;
        if (c1 - c0 == 1) {
            ++kept;
        } else {
            // greedy by height over the cluster [c0, c1): the open peak of
            // largest (height, position) is kept and its close neighbours go
            for (;;) {
                int best = -1;
                double hb = 0.0;
                for (int k = c0; k < c1; ++k) {
                    const int32_t p = pos[(int64_t)k * ps];
                    if (p & (kPeakGone | kPeakKept)) continue;
                    const double h = dvdt_at(a, v, p);
                    if (best < 0 || h >= hb) {  // equal heights: the later peak
                        best = k;
                        hb = h;
                    }
                }
                if (best < 0) break;
                const int32_t pb = pos[(int64_t)best * ps];
                pos[(int64_t)best * ps] = pb | kPeakKept;
                ++kept;
                for (int k = best - 1; k >= c0; --k) {
                    const int32_t p = pos[(int64_t)k * ps];
                    if (pb - (p & (kPeakKept - 1)) >= d) break;
                    pos[(int64_t)k * ps] = p | kPeakGone;
                }
                for (int k = best + 1; k < c1; ++k) {
                    const int32_t p = pos[(int64_t)k * ps];
                    if ((p & (kPeakKept - 1)) - pb >= d) break;
                    pos[(int64_t)k * ps] = p | kPeakGone;
                }
            }
        }
        c0 = c1;
    }
    return kept;
}

// Samples s0 .. s0 + 7 of a trace; row: samples lie side by side and 16-byte
// aligned (s0 a multiple of 8), two vector loads.
constexpr int kTraceBatch = 8;
__host__ __device__ __forceinline__ void load_batch(const float* v, int64_t st, bool row, int s0,
                                                    float (&x)[kTraceBatch]) {
#ifdef __CUDA_ARCH__
    if (row) {
        const float4 p = *reinterpret_cast<const float4*>(v + s0), q = *reinterpret_cast<const float4*>(v + s0 + 4);
        x[0] = p.x, x[1] = p.y, x[2] = p.z, x[3] = p.w, x[4] = q.x, x[5] = q.y, x[6] = q.z, x[7] = q.w;
        return;
    }
#endif
#pragma unroll
    for (int u = 0; u < kTraceBatch; ++u) x[u] = v[(int64_t)(s0 + u) * st];
}

// Samples whose differences order as their quotients do: 2^-17 <= |v| < 2^8.
// The smallest and the largest |v|; a NaN fails the test.
struct PlainRange {
    float lo = INFINITY, hi = 0;
    __host__ __device__ __forceinline__ void add(float a, float b) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000  // (the tests' host build compiles for another)
        asm("min.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(lo) : "f"(a), "f"(b));
        asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(hi) : "f"(a), "f"(b));
#else
        lo = a != a || b != b ? 0 : fminf(lo, fminf(fabsf(a), fabsf(b)));
        hi = fmaxf(hi, fmaxf(fabsf(a), fabsf(b)));
#endif
    }
    __host__ __device__ __forceinline__ bool ok() const { return lo >= 0x1p-17f && hi < 0x1p8f; }
};

// The largest float32 that is not above x (a NaN stays one).
__host__ __device__ __forceinline__ float float_below(double x) {
#ifdef __CUDA_ARCH__
    return __double2float_rd(x);
#else
    const float f = (float)x;
    return (double)f > x ? nextafterf(f, -INFINITY) : f;
#endif
}

// Steps 1 and 2 for the rises of trace t in [lo, hi) (lo a multiple of 8):
// their peaks' positions go to rows lo / 2, lo / 2 + 1, ... of the scratch
// (rises are two samples apart, so stretches do not meet); their number.
// h_lo: differences below it are below the height whatever the rounding.
// quotients: compare quotients throughout.
//
// Between two changes of x all its values are equal, so a rise that the next
// change undoes is a peak: `up` says that the last change was a rise, at i0.
// A NaN undoes nothing and ends the run.
__host__ __device__ inline int peaks_scan(const PeakArgs& a, int t, int lo, int hi, double h_lo, bool quotients,
                                          bool row) {
    const float* v = a.v + (int64_t)t * a.stride_trace;
    const int64_t st = a.stride_sample, ps = a.n_traces;
    int32_t* pos = a.pos + (int64_t)(lo / 2) * ps + t;
    const int nx = a.n_samples - 1;
    const int j0 = lo > 1 ? lo : 1, j1 = hi < nx - 1 ? hi : nx - 1;  // rises in [j0, j1)
    int m = 0, i0 = 0;
    if (j0 >= j1) return 0;
    bool up = false;
    float xa = v[(int64_t)(j0 - 1) * st], xb = v[(int64_t)j0 * st];  // the two samples before the next
    const float h_f = float_below(h_lo);
    // sample j + 1 closes difference j; a fall from difference j - 1 = x1 - x0 ends a peak there
    auto peak = [&](float x0, float x1, int j) {
        if (((double)x1 - (double)x0) / a.dt >= a.height) pos[(int64_t)m++ * ps] = (i0 + j - 1) / 2;
    };
    auto step_exact = [&](float x, int j, bool quotient, bool may_rise) {
        double d = (double)x - (double)xb, dp = (double)xb - (double)xa;
        if (quotient) {
            d /= a.dt;
            dp /= a.dt;
        }
        const bool lt = dp < d;
        if (up && d < dp) peak(xa, xb, j);
        up = lt ? may_rise : (up && d == dp);
        if (lt) i0 = j;
        xa = xb;
        xb = x;
    };
    // samples j0 + 1 .. j1, in whole batches of 8 where they fit
    int s = j0 + 1;
    for (; s <= j1 && (s & (kTraceBatch - 1)); ++s) step_exact(v[(int64_t)s * st], s - 1, true, true);
    if (s + kTraceBatch - 1 <= j1) {
        float nx8[kTraceBatch];
        load_batch(v, st, row, s, nx8);
        for (; s + kTraceBatch - 1 <= j1; s += kTraceBatch) {
            float x[kTraceBatch + 2] = {xa, xb};
#pragma unroll
            for (int u = 0; u < kTraceBatch; ++u) x[u + 2] = nx8[u];
            if (s + 2 * kTraceBatch - 1 <= j1) load_batch(v, st, row, s + kTraceBatch, nx8);
            PlainRange value, rise;
            bool equal = false;
            float d[kTraceBatch + 1];
#pragma unroll
            for (int u = 0; u <= kTraceBatch; ++u) {
                d[u] = x[u + 1] - x[u];
                if (u) equal = equal | (d[u] == d[u - 1]);
            }
#pragma unroll
            for (int u = 0; u <= kTraceBatch; u += 2) {
                value.add(x[u], x[u + 1]);
                rise.add(d[u], d[u + 1 <= kTraceBatch ? u + 1 : u]);
            }
            const bool plain = value.ok() && !quotients;
            if (plain && !(equal && !(rise.hi < value.lo))) {
#pragma unroll
                for (int u = 0; u < kTraceBatch; ++u) {
                    const bool lt = d[u] < d[u + 1], gt = d[u + 1] < d[u];
                    if (up & gt & (d[u] >= h_f)) peak(x[u], x[u + 1], s + u - 1);  // one predicate: a warp rarely goes in
                    up = lt | (up & !gt);
                    i0 = lt ? s + u - 1 : i0;
                }
                xa = x[kTraceBatch];
                xb = x[kTraceBatch + 1];
            } else {
                for (int u = 0; u < kTraceBatch; ++u) step_exact(v[(int64_t)(s + u) * st], s + u - 1, !plain, true);
            }
        }
    }
    for (; s <= j1; ++s) step_exact(v[(int64_t)s * st], s - 1, true, true);
    for (; up && s <= nx; ++s) step_exact(v[(int64_t)s * st], s - 1, true, false);  // only an open run goes on
    return m;
}

// Heights below this difference fail whatever the rounding of the quotient.
__host__ __device__ inline double peak_h_lo(const PeakArgs& a) {
    const double hd = a.height * a.dt;
    return hd - fabs(hd) * 1e-9;
}
// Quotients that overflow or vanish (steps no trace has) compare as quotients throughout.
__host__ __device__ inline bool peak_odd_step(const PeakArgs& a) { return !(a.dt > 1e-100 && a.dt < 1e100); }

// The score of trace t in one stretch (host-callable; the tests' host build).
__host__ __device__ inline int dvdt_peaks_trace(const PeakArgs& a, int t) {
    const int m = peaks_scan(a, t, 0, a.n_samples, peak_h_lo(a), peak_odd_step(a), false);
    return peaks_keep(a, a.v + (int64_t)t * a.stride_trace, a.pos + t, a.n_traces, m);
}

// Blocks of 32 traces (lane = trace) and blockDim.y stretches of `stretch`
// samples (even).  What bounds it: reading the traces once.  10,000 traces
// of 3,168 samples (127 MB): 89 us, 78 us where a trace's samples lie side by
// side; comparing every difference in FP64 instead took 124 us (52 warp
// instructions per 32 samples), one thread per trace 0.79 ms (two
// warps per SM, each walking 3,168 FP64 quotients one after another).  Left:
// 313 blocks of eight warps are two to three per SM, with 8 rows in flight.
constexpr int kPeakList = 256;
__global__ void __launch_bounds__(1024) k_dvdt_peaks(const PeakArgs a, int stretch, int row) {
    __shared__ int cnt[32][33];
    extern __shared__ int32_t peak_list[];  // [blockDim.y][kPeakList]
    const int lane = threadIdx.x, w = threadIdx.y, nw = blockDim.y, t = blockIdx.x * 32 + lane;
    if (t < a.n_traces)
        cnt[w][lane] = peaks_scan(a, t, w * stretch, (w + 1) * stretch, peak_h_lo(a), peak_odd_step(a), row);
    __syncthreads();
    // the distance rule, a warp per trace: its peaks in order into shared
    // memory; where no two are close that is their count
    int32_t* const list = peak_list + w * kPeakList;
    for (int i = w; i < 32; i += nw) {
        const int tr = blockIdx.x * 32 + i;
        if (tr >= a.n_traces) break;
        int mine = lane < nw ? cnt[lane][i] : 0, upto = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xFFFFFFFFu, upto, o);
            if (lane >= o) upto += x;
        }
        const int m = __shfl_sync(0xFFFFFFFFu, upto, 31);
        int32_t* pos = a.pos + tr;
        const int64_t ps = a.n_traces;
        const float* v = a.v + (int64_t)tr * a.stride_trace;
        if (m > kPeakList) {  // too many for the list: closed up in the scratch
            if (lane == 0) {
                int n = cnt[0][i];
                for (int c = 1; c < nw; ++c)
                    for (int k = 0; k < cnt[c][i]; ++k)
                        pos[(int64_t)n++ * ps] = pos[(int64_t)(c * (stretch / 2) + k) * ps];
                a.out[tr] = peaks_keep(a, v, pos, ps, n);
            }
            continue;
        }
        for (int c = 0; c < nw; ++c) {
            const int n = cnt[c][i], first = __shfl_sync(0xFFFFFFFFu, upto - mine, c);
            for (int k = lane; k < n; k += 32) list[first + k] = pos[(int64_t)(c * (stretch / 2) + k) * ps];
        }
        __syncwarp();
        bool close = false;
        for (int k = lane; k + 1 < m; k += 32) close = close || list[k + 1] - list[k] < a.distance;
        if (!__any_sync(0xFFFFFFFFu, close)) {
            if (lane == 0) a.out[tr] = m;
        } else if (lane == 0) {
            a.out[tr] = peaks_keep(a, v, list, 1, m);
        }
        __syncwarp();
    }
}

}  // namespace ngpu
