// Spike / ISI / amplitude / AHP / voltage features of many voltage traces, a
// warp per 32 traces and stretch of time.
//
// The reference extracts features trace by trace on a CPU pool (eFEL through
// P/efel_ext.py:23-96, GUI/score_functions.py); here a trace never leaves the
// GPU: the kernel reads the simulator's trace buffer where it lies.  Traces
// are addressed with two strides, element (trace t, sample s) at
// v[t * stride_trace + s * stride_sample]: the simulator's buffer is
// sample-major ([sample][site][instance], stride_trace 1), so at each sample
// the threads of a warp read 32 consecutive instances, one coalesced row, and
// every thread walks its own trace's stretch forward in time.  Pass 1 finds the upward
// threshold crossings inside the stimulus window and accumulates ISIs, the
// maximum and minimum of each inter-crossing segment (AP peaks, AHP troughs)
// and the window statistics; pass 2 counts the samples at or above the
// half-amplitude level, which needs pass 1's mean peak and trough.
//
// The definitions are those of neurogpu_b200/features.py (the batched torch
// statement the surrogate network is trained on), feature for feature:
// crossing times (index + 1) * dt in float32 as there, sums in FP64.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "explore.cuh"  // load_batch

namespace ngpu {

constexpr int kNFeatures = 20;

struct FeatureArgs {
    const float* v;
    int64_t stride_trace, stride_sample;
    int n_traces, n_samples;
    float dt, threshold;
    float dur;               // (i_off - i_on) dt
    int i_on, i_off;         // stimulus window [i_on, i_off) in samples
    int vb_lo, vb_hi;        // voltage_base window
    int ss_lo, ss_hi;        // steady-state window
    int af_lo, af_hi;        // after-stimulus window (af_lo < 0: the last sample)
    float* out;              // [n_traces][20]
};

// A trace is walked in stretches of time side by side: blocks of 32 traces
// (lane = trace) and blockDim.y stretches.  Each stretch keeps what the whole
// needs of it (the kF* rows in shared memory: extremes, sums, its first and last crossing, the
// sums over the segments that start and end inside it, and the extremes of
// the open pieces at its two ends); one warp joins the stretches in time
// order, then every stretch counts its samples above half amplitude.
//
// What bounds it: reading the traces, and the window a second time.  10,000
// traces of 3,168 samples (127 MB): 135 us, traces side by side (103 us where a
// trace's samples lie side by side).  One thread per trace (the
// form this replaces) took 0.49 ms: two warps per SM.
constexpr int kFeatDoubles = 10, kFeatFloats = 9, kFeatInts = 3;
// a stretch's fields in shared memory, [field][stretch][32]
enum { kFWsum, kFWsq, kFPk, kFPk2, kFTr, kFIsi, kFIsi2, kFVb, kFSs, kFAf };
enum { kFVmax, kFWmin, kFWmax, kFHeadMax, kFHeadMin, kFTailMax, kFTailMin, kFIsiFirst, kFIsiLast };
enum { kFN, kFFirst, kFLast };  // crossings; samples of the first and the last, from the window's start

// shared memory per thread of the block
constexpr int kFeatEvents = 8;  // crossings held back (sample, extremes of the segment before), see k_trace_features
constexpr int kFeatBytes = kFeatDoubles * 8 + (kFeatFloats + kFeatInts + 3 * kFeatEvents) * 4;

__global__ void __launch_bounds__(1024) k_trace_features(const FeatureArgs a, int stretch, int rowv) {
    extern __shared__ __align__(16) char feat_smem[];
    __shared__ float half_s[32];
    __shared__ int first_s[32], above_s[32];
    const int lane = threadIdx.x, w = threadIdx.y, nw = blockDim.y;
    const int t = blockIdx.x * 32 + lane;
    const bool in = t < a.n_traces;
    const float* v = a.v + (int64_t)(in ? t : 0) * a.stride_trace;
    const int64_t st = a.stride_sample;
    const float TH = a.threshold, dt = a.dt;
    const int W = a.i_off - a.i_on;
    const int lo = min(w * stretch, a.n_samples), hi = min(lo + stretch, a.n_samples);
    const int row = nw * 32, at = w * 32 + lane;
    double* sd = (double*)feat_smem;
    float* sf = (float*)(sd + kFeatDoubles * row);
    int* si = (int*)(sf + kFeatFloats * row);
    for (int k = 0; k < kFeatDoubles; ++k) sd[k * row + at] = 0.0;
    for (int k = 0; k < kFeatInts; ++k) si[k * row + at] = 0;
    // pass 1.  Some lane of a warp crosses at nearly every other sample of a
    // spiking batch, so a crossing only notes its sample and its segment's
    // extremes; the sums take the notes when half the list may be full.
    float* ev_max = (float*)(si + kFeatInts * row);
    float* ev_min = ev_max + kFeatEvents * row;
    int* ev_at = (int*)(ev_min + kFeatEvents * row);
    int held = 0;
    double wsum = 0, wsq = 0;
    float vmax = -INFINITY, wmin = INFINITY, wmax = -INFINITY, seg_max = -INFINITY, seg_min = INFINITY;
    float prev = lo > a.i_on && lo < a.i_off ? v[(int64_t)(lo - 1) * st] : INFINITY;  // no crossing into the first sample
    auto take = [&]() {
        for (int e = 0; e < held; ++e) {
            const int j = ev_at[e * row + at];  // a crossing between samples j - 1 and j: t = j dt
            const float mx = ev_max[e * row + at], mn = ev_min[e * row + at];
            const int n = si[kFN * row + at];
            if (n > 0) {  // a segment that began in this stretch ends
                sd[kFPk * row + at] += mx;
                sd[kFPk2 * row + at] += (double)mx * mx;
                sd[kFTr * row + at] += mn;
                const float isi = __fsub_rn(__fmul_rn((float)j, dt), __fmul_rn((float)si[kFLast * row + at], dt));
                sd[kFIsi * row + at] += isi;
                sd[kFIsi2 * row + at] += (double)isi * isi;
                if (n == 1) sf[kFIsiFirst * row + at] = isi;
                sf[kFIsiLast * row + at] = isi;
            } else {
                si[kFFirst * row + at] = j;
                sf[kFHeadMax * row + at] = mx;
                sf[kFHeadMin * row + at] = mn;
            }
            si[kFLast * row + at] = j;
            si[kFN * row + at] = n + 1;
        }
        held = 0;
    };
    auto window = [&](float y, int s) {
        wsq += (double)y * y;
        wmin = fminf(wmin, y);
        wmax = fmaxf(wmax, y);
        if ((prev < TH) & (y >= TH)) {
            ev_at[held * row + at] = s - a.i_on;
            ev_max[held * row + at] = seg_max;
            ev_min[held * row + at] = seg_min;
            ++held;
            seg_max = -INFINITY;
            seg_min = INFINITY;
        }
        seg_max = fmaxf(seg_max, y);
        seg_min = fminf(seg_min, y);
        prev = y;
    };
    auto inside = [](int s, int l, int h) { return s >= l && s < h; };
    const int cuts[8] = {a.i_on, a.i_off, a.vb_lo, a.vb_hi, a.ss_lo, a.ss_hi, a.af_lo, a.af_hi};
    float nx[kTraceBatch];
    if (lo + kTraceBatch <= hi) load_batch(v, st, rowv, lo, nx);
    int cut = lo;  // the next window's edge (or the stretch's end)
    for (int s0 = lo; s0 < hi; s0 += kTraceBatch) {
        const int s1 = s0 + kTraceBatch;
        if (cut <= s0) {
            cut = hi;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (cuts[c] > s0 && cuts[c] < cut) cut = cuts[c];
        }
        float x[kTraceBatch];
#pragma unroll
        for (int u = 0; u < kTraceBatch; ++u) x[u] = nx[u];
        if (s1 + kTraceBatch <= hi) load_batch(v, st, rowv, s1, nx);
        if (held > kFeatEvents - kTraceBatch / 2) take();  // two samples at least between crossings
        if (s1 <= cut) {  // no window's edge inside

            const bool win = inside(s0, a.i_on, a.i_off);
            double sum = 0;
#pragma unroll
            for (int u = 0; u < kTraceBatch; ++u) {
                vmax = fmaxf(vmax, x[u]);
                sum += (double)x[u];
                if (win) window(x[u], s0 + u);
            }
            if (win) wsum += sum;
            if (inside(s0, a.vb_lo, a.vb_hi)) sd[kFVb * row + at] += sum;
            if (inside(s0, a.ss_lo, a.ss_hi)) sd[kFSs * row + at] += sum;
            if (inside(s0, a.af_lo, a.af_hi)) sd[kFAf * row + at] += sum;
        } else {
            for (int s = s0; s < min(s1, hi); ++s) {
                const float y = v[(int64_t)s * st];
                vmax = fmaxf(vmax, y);
                if (inside(s, a.i_on, a.i_off)) {
                    wsum += (double)y;
                    window(y, s);
                }
                if (inside(s, a.vb_lo, a.vb_hi)) sd[kFVb * row + at] += (double)y;
                if (inside(s, a.ss_lo, a.ss_hi)) sd[kFSs * row + at] += (double)y;
                if (inside(s, a.af_lo, a.af_hi)) sd[kFAf * row + at] += (double)y;
            }
        }
    }
    take();
    sd[kFWsum * row + at] = wsum;
    sd[kFWsq * row + at] = wsq;
    sf[kFVmax * row + at] = vmax;
    sf[kFWmin * row + at] = wmin;
    sf[kFWmax * row + at] = wmax;
    // without a crossing the whole stretch belongs to the segment before it
    const int first_seg = si[kFN * row + at] > 0 ? kFTailMax : kFHeadMax;
    sf[first_seg * row + at] = seg_max;
    sf[(first_seg + 1) * row + at] = seg_min;
    if (w == 0) above_s[lane] = 0;
    __syncthreads();
    vmax = wmax = -INFINITY;
    wmin = INFINITY;
    wsum = wsq = 0;
    double vb = 0, ss = 0, af = 0;
    int n = 0, first_idx = 0;
    float first_t = 0, last_t = 0, first_isi = 0, last_isi = 0;
    double isi_sum = 0, isi_sq = 0, pk_sum = 0, pk_sq = 0, tr_sum = 0;
    double pk_mean = 0, pk_std = 0, ahp = 0;
    if (w == 0) {
        seg_max = -INFINITY;
        seg_min = INFINITY;
        auto close = [&]() {
            pk_sum += seg_max;
            pk_sq += (double)seg_max * seg_max;
            tr_sum += seg_min;
        };
        for (int c = 0; c < nw; ++c) {
            const double* d = sd + c * 32 + lane;
            const float* f = sf + c * 32 + lane;
            const int* q = si + c * 32 + lane;
            wsum += d[kFWsum * row];
            wsq += d[kFWsq * row];
            vb += d[kFVb * row];
            ss += d[kFSs * row];
            af += d[kFAf * row];
            vmax = fmaxf(vmax, f[kFVmax * row]);
            wmin = fminf(wmin, f[kFWmin * row]);
            wmax = fmaxf(wmax, f[kFWmax * row]);
            if (n > 0) {
                seg_max = fmaxf(seg_max, f[kFHeadMax * row]);
                seg_min = fminf(seg_min, f[kFHeadMin * row]);
            }
            const int k = q[kFN * row];
            if (k == 0) continue;
            const float tc = __fmul_rn((float)q[kFFirst * row], dt);
            if (n > 0) {
                close();
                const float isi = __fsub_rn(tc, last_t);
                isi_sum += isi;
                isi_sq += (double)isi * isi;
                if (n == 1) first_isi = isi;
                last_isi = isi;
            } else {
                first_t = tc;
                first_idx = q[kFFirst * row];
            }
            pk_sum += d[kFPk * row];
            pk_sq += d[kFPk2 * row];
            tr_sum += d[kFTr * row];
            isi_sum += d[kFIsi * row];
            isi_sq += d[kFIsi2 * row];
            if (k > 1) {
                if (n == 0) first_isi = f[kFIsiFirst * row];
                last_isi = f[kFIsiLast * row];
            }
            n += k;
            last_t = __fmul_rn((float)q[kFLast * row], dt);
            seg_max = f[kFTailMax * row];
            seg_min = f[kFTailMin * row];
        }
        if (n > 0) close();
        const double nd = (double)n;
        pk_mean = n >= 1 ? pk_sum / nd : (double)wmax;
        pk_std = n >= 1 ? sqrt(fmax(0.0, pk_sq / nd - pk_mean * pk_mean)) : 0.0;
        ahp = n >= 1 ? tr_sum / nd : (double)wmin;
        half_s[lane] = (float)(0.5 * (pk_mean + ahp));
        first_s[lane] = n >= 1 ? a.i_on + first_idx : a.n_samples;
    }
    __syncthreads();
    // pass 2: samples at or above half amplitude after the first crossing
    {
        const float half = half_s[lane];
        const int from = max(lo, first_s[lane]), to = min(hi, a.i_off);
        int above = 0, s = lo;
        if (__any_sync(0xFFFFFFFFu, from < to)) {
#pragma unroll 2
            for (; s + kTraceBatch <= to; s += kTraceBatch) {
                float x[kTraceBatch];
                load_batch(v, st, rowv, s, x);
#pragma unroll
                for (int u = 0; u < kTraceBatch; ++u) above += s + u >= from && x[u] >= half ? 1 : 0;
            }
            for (; s < to; ++s) above += s >= from && v[(int64_t)s * st] >= half ? 1 : 0;
        }
        if (above) atomicAdd(&above_s[lane], above);
    }
    __syncthreads();
    if (w != 0 || !in) return;
    const bool has1 = n >= 1, has2 = n >= 2;
    const float dur = a.dur;
    const double n_isi = (double)(n - 1);
    const double mean_isi = has2 ? isi_sum / n_isi : (double)dur;
    double isi_cv = 0;
    if (has2) {
        const double var = fmax(0.0, isi_sq / n_isi - mean_isi * mean_isi);
        isi_cv = sqrt(var) / fmax(mean_isi, 1e-6);
    }
    const double wmean = W > 0 ? wsum / W : 0.0;
    const double wstd = W > 1 ? sqrt(fmax(0.0, (wsq - (double)W * wmean * wmean) / (double)(W - 1))) : 0.0;
    auto mean = [](double s, int l, int h) { return h > l ? s / (double)(h - l) : 0.0; };
    float* o = a.out + (int64_t)t * kNFeatures;
    o[0] = (float)n;
    o[1] = has1 ? first_t : dur;
    o[2] = (float)mean_isi;
    o[3] = (float)isi_cv;
    o[4] = has2 ? first_isi : dur;
    o[5] = has2 ? last_isi : dur;
    o[6] = has2 ? last_isi / fmaxf(first_isi, 1e-6f) : 1.0f;
    o[7] = (float)pk_mean;
    o[8] = (float)pk_std;
    o[9] = (float)ahp;
    o[10] = (float)(pk_mean - ahp);
    o[11] = has1 ? (float)above_s[lane] * dt / (float)n : 0.0f;
    o[12] = (float)mean(vb, a.vb_lo, a.vb_hi);
    o[13] = (float)mean(ss, a.ss_lo, a.ss_hi);
    o[14] = a.af_lo < 0 ? v[(int64_t)(a.n_samples - 1) * st] : (float)mean(af, a.af_lo, a.af_hi);
    o[15] = vmax;
    o[16] = wmin;
    o[17] = (float)wmean;
    o[18] = (float)wstd;
    o[19] = has1 ? last_t : dur;
}

}  // namespace ngpu
