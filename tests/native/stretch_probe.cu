// Test-only host build of the exploration score's stretch-wise scan
// (neurogpu_b200/csrc/explore.cuh): the steps of k_dvdt_peaks on one trace,
// cut into stretches of the given length (a multiple of 8).
#include <stdint.h>

#include <vector>

#include "../../neurogpu_b200/csrc/explore.cuh"

extern "C" int probe_stretches(const float* v, int n_samples, int64_t stride, double dt, double height, int distance,
                               int stretch) {
    ngpu::PeakArgs a;
    a.v = v;
    a.stride_trace = 0;
    a.stride_sample = stride;
    a.n_traces = 1;
    a.n_samples = n_samples;
    a.dt = dt;
    a.height = height;
    a.distance = distance;
    a.cap = ngpu::peak_scratch_cap(n_samples);
    std::vector<int32_t> pos((size_t)a.cap);
    a.pos = pos.data();
    a.out = nullptr;
    int m = 0;
    for (int lo = 0; lo < n_samples; lo += stretch) {
        const int n = ngpu::peaks_scan(a, 0, lo, lo + stretch, ngpu::peak_h_lo(a), ngpu::peak_odd_step(a), false);
        for (int k = 0; k < n; ++k) pos[(size_t)m++] = pos[(size_t)(lo / 2 + k)];
    }
    return ngpu::peaks_keep(a, v, pos.data(), 1, m);
}
