// Genetic-algorithm variation and selection on the GPU, so that a generation
// (offspring -> simulation -> features -> scores -> survivors) never leaves
// the device.
//
// The reference runs these steps on the host between simulator calls:
// DEAP's varOr / eaMuPlusLambda (GUI/DEAP_helper.py:126-271) and bluepyopt's
// DEAPOptimisation with a multi-objective selector
// (Figures/Figure4_DEAP/optimize_parameters_genetic_alg.py:49).  Restated
// here from the published operators:
//   * binary tournament on (front rank ascending, crowding descending);
//   * bounded simulated binary crossover (Deb & Agrawal 1995, in the bounded
//     form of Deb's NSGA-II code) and bounded polynomial mutation (Deb &
//     Goyal 1996), genes in [low, up];
//   * (mu + lambda) truncation on a scalar score, or NSGA-II's
//     non-dominated sorting with crowding distance (Deb, Pratap, Agarwal &
//     Meyarivan 2002) on a vector of objectives, all minimised.
//
// Random numbers are counter based: draw d of child c in generation g is
// SplitMix64 (Steele, Lea & Flood 2014) of a key made from the seed, g, c and
// d, so any child is reproducible on its own and the host restatement
// replays the same stream bit for bit.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

namespace ngpu {

namespace cg = cooperative_groups;

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// the generation's stream key
__host__ __device__ __forceinline__ uint64_t ga_key(uint64_t seed, uint64_t generation) {
    return splitmix64(seed ^ splitmix64(generation));
}

// draw d (< 2^20) of child c: 64 random bits
__device__ __forceinline__ uint64_t ga_bits(uint64_t key, uint64_t child, uint32_t d) {
    return splitmix64(key ^ splitmix64((child << 20) | d));
}

// uniform in [0, 1) with 53 random bits
__device__ __forceinline__ double ga_uniform(uint64_t key, uint64_t child, uint32_t d) {
    return (double)(ga_bits(key, child, d) >> 11) * 0x1.0p-53;
}

// uniform integer in [0, n): the high 32 bits scaled by n (multiply-shift)
__device__ __forceinline__ int ga_index(uint64_t key, uint64_t child, uint32_t d, int n) {
    return (int)(((ga_bits(key, child, d) >> 32) * (uint64_t)n) >> 32);
}

// draw layout of one child: 4 tournament picks, mate, which child of the
// pair; then 5 per gene (crossover?, crossover spread, swap?, mutate?,
// mutation spread)
constexpr uint32_t kGaDrawsFixed = 6;
constexpr uint32_t kGaDrawsPerGene = 5;

struct GaVariation {
    const double* pop;       // [mu][n_genes]
    const int32_t* rank;     // [mu] front rank (lower is better)
    const double* crowd;     // [mu] crowding (higher is better among equal ranks)
    int mu, n_genes, n_kids;
    double low, up, eta_c, eta_m, cx_prob, p_mut;
    uint64_t key;
    double* kids;            // [n_kids][n_genes]
};

__device__ __forceinline__ int ga_tournament(const GaVariation& a, int i, int j) {
    if (a.rank[j] < a.rank[i]) return j;
    if (a.rank[j] == a.rank[i] && a.crowd[j] > a.crowd[i]) return j;
    return i;   // ties: the first pick
}

// spread factor of bounded SBX for one side: beta is 1 + 2 (distance from
// the nearer parent to the bound) / (parent distance)
__device__ __forceinline__ double sbx_beta_q(double beta, double u, double eta) {
    const double alpha = 2.0 - pow(beta, -(eta + 1.0));
    if (u <= 1.0 / alpha) return pow(u * alpha, 1.0 / (eta + 1.0));
    return pow(1.0 / (2.0 - u * alpha), 1.0 / (eta + 1.0));
}

// One thread per gene (its draws depend on nothing but the child and the
// gene; the threads of a child repeat its tournaments).  Bound by the
// latency of the FP64 powers: a thread per child, 12 genes one after another
// on 40 CTAs, took 70 us for 5,000 children.
__global__ void __launch_bounds__(128) k_ga_offspring(const GaVariation a) {
    const int64_t at = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (at >= (int64_t)a.n_kids * a.n_genes) return;
    const int c = (int)(at / a.n_genes), g = (int)(at % a.n_genes);
    const uint64_t key = a.key, ch = (uint64_t)c;
    const int p1 = ga_tournament(a, ga_index(key, ch, 0, a.mu), ga_index(key, ch, 1, a.mu));
    const int p2 = ga_tournament(a, ga_index(key, ch, 2, a.mu), ga_index(key, ch, 3, a.mu));
    const bool mate = ga_uniform(key, ch, 4) < a.cx_prob;
    const bool first = ga_uniform(key, ch, 5) < 0.5;
    const double* x = a.pop + (size_t)p1 * a.n_genes;
    const double* y = a.pop + (size_t)p2 * a.n_genes;
    const double lo = a.low, hi = a.up, span = hi - lo;
    const uint32_t d = kGaDrawsFixed + kGaDrawsPerGene * (uint32_t)g;
    double v = x[g];
    if (mate) {
        // bounded SBX of the pair (x[g], y[g]); the child keeps x[g] where no crossover happens
        const double u_do = ga_uniform(key, ch, d), u = ga_uniform(key, ch, d + 1);
        const double u_sw = ga_uniform(key, ch, d + 2);
        const double a1 = x[g], b1 = y[g];
        if (u_do < 0.5 && fabs(a1 - b1) > 1e-14) {
            const double x1 = fmin(a1, b1), x2 = fmax(a1, b1), dx = x2 - x1;
            const double y1 = fmin(fmax(0.5 * (x1 + x2 - sbx_beta_q(1.0 + 2.0 * (x1 - lo) / dx, u, a.eta_c) * dx), lo), hi);
            const double y2 = fmin(fmax(0.5 * (x1 + x2 + sbx_beta_q(1.0 + 2.0 * (hi - x2) / dx, u, a.eta_c) * dx), lo), hi);
            const bool swap = u_sw < 0.5;
            // the pair's children are (y1, y2), or (y2, y1) when swapped; this child is the first or the second
            v = (first != swap) ? y1 : y2;
        } else if (!first) {
            v = b1;
        }
    }
    // bounded polynomial mutation
    if (ga_uniform(key, ch, d + 3) < a.p_mut) {
        const double r = ga_uniform(key, ch, d + 4);
        const double d1 = (v - lo) / span, d2 = (hi - v) / span, mp = 1.0 / (a.eta_m + 1.0);
        double dq;
        if (r < 0.5) {
            const double val = 2.0 * r + (1.0 - 2.0 * r) * pow(1.0 - d1, a.eta_m + 1.0);
            dq = pow(val, mp) - 1.0;
        } else {
            const double val = 2.0 * (1.0 - r) + 2.0 * (r - 0.5) * pow(1.0 - d2, a.eta_m + 1.0);
            dq = 1.0 - pow(val, mp);
        }
        v = fmin(fmax(v + dq * span, lo), hi);
    }
    a.kids[at] = v;
}

// --------------------------------------------------------------- sorting
// Total order of doubles as unsigned keys (NaN after +inf).
__host__ __device__ __forceinline__ uint64_t ga_order_key(double x) {
    if (x != x) return 0xFFFFFFFFFFFFFFFEull;
    uint64_t b;
    memcpy(&b, &x, 8);
    if (x == 0.0) b = 0;                       // -0 and +0 alike
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

struct GaSortSlice {
    uint64_t* k1;
    uint64_t* k2;
    uint32_t* idx;
};

// Segmented bitonic sort: `count` independent segments of n2 entries (a
// power of two) each, ascending by (k1, k2, idx).  Strides below the tile
// (kGaSortTile entries, one CTA) run in shared memory -- the whole network
// up to the tile size at first, then the tail of every later merge; strides
// of a tile or more run as grid-wide stages, one launch each, every thread
// one compare-exchange.  The direction of a pair follows its position in its
// segment, so segments never mix.
constexpr uint32_t kGaSortTile = 2048;
constexpr int kGaSortThreads = 1024;

__device__ __forceinline__ void ga_cmpswap(uint64_t* k1, uint64_t* k2, uint32_t* ix, size_t i, size_t l, bool asc) {
    const bool less_li = k1[l] != k1[i] ? k1[l] < k1[i] : (k2[l] != k2[i] ? k2[l] < k2[i] : ix[l] < ix[i]);
    if (less_li == asc) {
        const uint64_t a1 = k1[i], a2 = k2[i];
        const uint32_t ai = ix[i];
        k1[i] = k1[l];
        k2[i] = k2[l];
        ix[i] = ix[l];
        k1[l] = a1;
        k2[l] = a2;
        ix[l] = ai;
    }
}

// one tile per CTA: k_merge == 0 sorts the tile (every k up to the tile
// size); otherwise the strides below the tile of merge step k_merge
__global__ void __launch_bounds__(kGaSortThreads) k_ga_sort_tile(GaSortSlice s, uint32_t n2, uint32_t tile,
                                                                 uint32_t k_merge) {
    __shared__ uint64_t k1[kGaSortTile], k2[kGaSortTile];
    __shared__ uint32_t ix[kGaSortTile];
    const size_t base = (size_t)blockIdx.x * tile;
    for (uint32_t t = threadIdx.x; t < tile; t += blockDim.x) {
        k1[t] = s.k1[base + t];
        k2[t] = s.k2[base + t];
        ix[t] = s.idx[base + t];
    }
    __syncthreads();
    const uint32_t pos0 = (uint32_t)(base & (n2 - 1));   // position of the tile in its segment
    const uint32_t k_lo = k_merge ? k_merge : 2, k_hi = k_merge ? k_merge : tile;
    for (uint32_t k = k_lo; k <= k_hi; k <<= 1) {
        for (uint32_t j = (k_merge ? tile : k) >> 1; j > 0; j >>= 1) {
            for (uint32_t t = threadIdx.x; t < tile; t += blockDim.x) {
                const uint32_t l = t ^ j;
                if (l > t) ga_cmpswap(k1, k2, ix, t, l, ((pos0 + t) & k) == 0);
            }
            __syncthreads();
        }
    }
    for (uint32_t t = threadIdx.x; t < tile; t += blockDim.x) {
        s.k1[base + t] = k1[t];
        s.k2[base + t] = k2[t];
        s.idx[base + t] = ix[t];
    }
}

// one grid-wide stage (k, j) with j >= the tile: pair p -> (i, i + j), bit j of i clear
__global__ void k_ga_sort_stage(GaSortSlice s, size_t total, uint32_t n2, uint32_t k, uint32_t j) {
    const size_t pairs = total >> 1;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < pairs; p += (size_t)gridDim.x * blockDim.x) {
        const size_t i = (p / j) * (2 * (size_t)j) + (p % j);
        ga_cmpswap(s.k1, s.k2, s.idx, i, i + j, ((uint32_t)(i & (n2 - 1)) & k) == 0);
    }
}

// host side: sort `count` segments of n2 entries on a stream; returns the launches issued
inline int ga_sort(const GaSortSlice& s, uint32_t n2, int count, cudaStream_t st) {
    const uint32_t tile = n2 < kGaSortTile ? n2 : kGaSortTile;
    const size_t total = (size_t)n2 * count;
    const unsigned tiles = (unsigned)(total / tile);
    const unsigned grid = (unsigned)std::min<size_t>((total / 2 + 255) / 256, 148 * 16);
    int launches = 1;
    k_ga_sort_tile<<<tiles, kGaSortThreads, 0, st>>>(s, n2, tile, 0);
    for (uint32_t k = 2 * tile; k <= n2; k <<= 1) {
        for (uint32_t j = k >> 1; j >= tile; j >>= 1) {
            k_ga_sort_stage<<<grid, 256, 0, st>>>(s, total, n2, k, j);
            ++launches;
        }
        k_ga_sort_tile<<<tiles, kGaSortThreads, 0, st>>>(s, n2, tile, k);
        ++launches;
    }
    return launches;
}

// keys of (mu + lambda) truncation: the score, then the index
__global__ void k_ga_truncation_keys(const double* score, int n, uint32_t n2, GaSortSlice s) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += gridDim.x * blockDim.x) {
        const bool in = i < (uint32_t)n;
        s.k1[i] = in ? ga_order_key(score[i]) : ~0ull;
        s.k2[i] = 0;
        s.idx[i] = i;
    }
}

__global__ void k_ga_take(const uint32_t* sorted_idx, int mu, int32_t* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < mu; i += gridDim.x * blockDim.x) out[i] = (int32_t)sorted_idx[i];
}

// ------------------------------------------------- NSGA-II up to 16,384
// Objectives are replaced by their ranks (a value's position in its
// objective's sorted order, equal values alike; 14 bits, two to a word), so
// that a comparison of two individuals is a packed add and maximum per two
// objectives, and individuals are renumbered by the sum of their ranks: one
// can only be dominated by one of smaller sum, which halves the dominance
// matrix.  Every result is that of the FP64 comparisons.  Against the
// kernels for larger sets further below, 10,000 individuals, B200: 60
// objectives (few fronts) 0.49 ms against 2.05; 2 objectives (198 fronts) 1.2 ms
// against 10.4.
constexpr int kGaSmallMax = 16384;
constexpr int kGaDomThreads = 256;

// Sorts a CTA's (key, index) pairs, ascending by key, then index: eight per
// thread in registers (n2 = 8 x threads, a power of two >= 256), entry e at
// thread e / 8.  A bitonic network, whose stages of distance 1 to 4 are
// within a thread, 8 to 128 within a warp (shuffles), and only those of 256
// and more go through shared memory: 6 of the 66 stages of 2,048 entries.
// With every stage there (a thread a pair), it was bound by its wavefronts:
// 60 x 5 tiles of 2,048 took 61 us, now 43 (compares, of 64-bit keys).
constexpr int kGaPer = 8;
__device__ __forceinline__ bool ga_less(uint64_t x, uint32_t xi, uint64_t y, uint32_t yi) {
    return (x < y) | ((x == y) & (xi < yi));
}
template <int J>
__device__ __forceinline__ void ga_stage_thread(uint64_t (&x)[kGaPer], uint32_t (&id)[kGaPer], uint32_t k) {
#pragma unroll
    for (int u = 0; u < kGaPer; ++u) {
        if (u & J) continue;
        const bool up = ((threadIdx.x * kGaPer + u) & k) == 0;
        if (ga_less(x[u | J], id[u | J], x[u], id[u]) == up) {
            const uint64_t t = x[u];
            x[u] = x[u | J];
            x[u | J] = t;
            const uint32_t ti = id[u];
            id[u] = id[u | J];
            id[u | J] = ti;
        }
    }
}
__device__ __forceinline__ void ga_bitonic(uint64_t (&x)[kGaPer], uint32_t (&id)[kGaPer], uint64_t* key_s,
                                           uint16_t* idx_s, uint32_t n2) {
    const uint32_t T = n2 / kGaPer, tid = threadIdx.x;
    for (uint32_t k = 2; k <= n2; k <<= 1) {
        for (uint32_t j = k >> 1; j >= kGaPer; j >>= 1) {
            const uint32_t d = j / kGaPer;  // the partner thread's distance
            const bool least = ((tid & d) == 0) == ((tid * kGaPer & k) == 0);
            if (d >= 32) {
                __syncthreads();
#pragma unroll
                for (int u = 0; u < kGaPer; ++u) {
                    key_s[u * T + tid] = x[u];
                    idx_s[u * T + tid] = (uint16_t)id[u];
                }
                __syncthreads();
            }
#pragma unroll
            for (int u = 0; u < kGaPer; ++u) {
                uint64_t y;
                uint32_t yi;
                if (d >= 32) {
                    y = key_s[u * T + (tid ^ d)];
                    yi = idx_s[u * T + (tid ^ d)];
                } else {
                    y = __shfl_xor_sync(0xFFFFFFFFu, x[u], d);
                    yi = __shfl_xor_sync(0xFFFFFFFFu, id[u], d);
                }
                if (ga_less(y, yi, x[u], id[u]) == least) {
                    x[u] = y;
                    id[u] = yi;
                }
            }
        }
        if (k >= 8) ga_stage_thread<4>(x, id, k);
        if (k >= 4) ga_stage_thread<2>(x, id, k);
        ga_stage_thread<1>(x, id, k);
    }
}

// An objective's value as a key (NaN as +inf, the worst).
__device__ __forceinline__ uint64_t ga_obj_key(double x) { return ga_order_key(x != x ? INFINITY : x); }

// Every objective's order, in two steps: tiles of up to 2,048 individuals
// sorted in shared memory, one CTA each (k_ga_tiles), then each entry's place
// counted by a binary search in every tile (k_ga_places).  Keys: the
// objective's value (FRONTS false), or the front and the place in the
// objective's order, which makes the order within each front.  One CTA per
// objective sorting all of it took 271 us for 60 x 10,000; the two steps take 43 + 36.
constexpr int kGaTile = 2048;
struct GaOrderArgs {
    const double* obj;       // [n][m]
    const int32_t* rank;     // [n] fronts (FRONTS)
    const int32_t* n_fronts; // (FRONTS)
    int n, m;
    uint32_t tile;           // entries per tile, a power of two >= 256
    uint64_t* key;           // [m][tiles * tile] sorted tiles
    uint16_t* idx;
    uint16_t* order;         // [m][n] individuals in the objective's order
    uint16_t* rank2;         // [ceil(m / 2)][n][2] a value's first place, an odd last half zero
    uint16_t* in_fronts;     // [m][n] individuals by front, then in the objective's order (FRONTS)
};
template <bool FRONTS>
__global__ void __launch_bounds__(kGaTile / kGaPer) k_ga_tiles(const GaOrderArgs a) {
    __shared__ uint64_t key[kGaTile];
    __shared__ uint16_t idx[kGaTile];
    const int k = blockIdx.y;
    const uint32_t T = a.tile / kGaPer;
    uint64_t x[kGaPer];
    uint32_t id[kGaPer];
#pragma unroll
    for (int u = 0; u < kGaPer; ++u) {
        const int p = blockIdx.x * (int)a.tile + (int)(u * T + threadIdx.x);
        x[u] = ~0ull;
        id[u] = p;
        if (p < a.n) {
            if constexpr (FRONTS) {
                id[u] = a.order[(size_t)k * a.n + p];
                x[u] = ((uint64_t)a.rank[id[u]] << 14) | (uint32_t)p;
            } else {
                x[u] = ga_obj_key(a.obj[(size_t)p * a.m + k]);
            }
        }
    }
    const bool sort = !FRONTS || *a.n_fronts > 1;  // (a single front is in order already)
    if (sort) ga_bitonic(x, id, key, idx, a.tile);
    const size_t base = ((size_t)k * gridDim.x + blockIdx.x) * a.tile;
#pragma unroll
    for (int u = 0; u < kGaPer; ++u) {
        const uint32_t t = sort ? threadIdx.x * kGaPer + u : u * T + threadIdx.x;
        a.key[base + t] = x[u];
        a.idx[base + t] = (uint16_t)id[u];
    }
}

// entries of the ascending tile below x (OR_EQUAL: or equal to it)
template <bool OR_EQUAL>
__device__ __forceinline__ uint32_t ga_below(const uint64_t* key, uint32_t tile, uint64_t x) {
    uint32_t lo = 0;
    for (uint32_t step = tile >> 1; step > 0; step >>= 1)
        if (OR_EQUAL ? key[lo + step - 1] <= x : key[lo + step - 1] < x) lo += step;
    return lo + ((OR_EQUAL ? key[lo] <= x : key[lo] < x) ? 1 : 0);
}

template <bool FRONTS>
__global__ void __launch_bounds__(kGaTile / 2) k_ga_places(const GaOrderArgs a) {
    __shared__ uint64_t other[kGaTile];
    const int k = blockIdx.y, tiles = gridDim.x, mine = blockIdx.x;
    const uint64_t* keys = a.key + (size_t)k * tiles * a.tile;
    uint64_t x[2];
    uint32_t place[2], first[2] = {0, 0};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const uint32_t t = threadIdx.x + e * blockDim.x;
        x[e] = keys[(size_t)mine * a.tile + t];
        place[e] = t;
    }
    for (int c = 0; c < tiles; ++c) {
        if (FRONTS && c == mine) continue;
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < a.tile; t += blockDim.x) other[t] = keys[(size_t)c * a.tile + t];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t below = ga_below<false>(other, a.tile, x[e]);
            first[e] += below;
            // equal values: an earlier tile's individuals come first
            if (c < mine) place[e] += FRONTS || other[below < a.tile ? below : 0] != x[e] ? below : ga_below<true>(other, a.tile, x[e]);
            if (c > mine) place[e] += below;
        }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const uint32_t t = threadIdx.x + e * blockDim.x;
        if (x[e] == ~0ull) continue;  // padding
        const uint16_t i = a.idx[((size_t)k * tiles + mine) * a.tile + t];
        if constexpr (FRONTS) {
            a.in_fronts[(size_t)k * a.n + place[e]] = i;
        } else {
            a.order[(size_t)k * a.n + place[e]] = i;
            a.rank2[((size_t)(k >> 1) * a.n + i) * 2 + (k & 1)] = (uint16_t)first[e];
            if (k == a.m - 1 && (a.m & 1)) a.rank2[((size_t)(k >> 1) * a.n + i) * 2 + 1] = 0;
        }
    }
}

// sum[i]: the sum of individual i's ranks; seat[i] and cnt[i] cleared
__global__ void k_ga_rank_sums(const uint32_t* rank2, int n, int q, uint32_t* sum, int32_t* seat) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t s = 0;
    for (int k = 0; k < q; ++k) {
        const uint32_t r = rank2[(size_t)k * n + i];
        s += (r & 0xFFFFu) + (r >> 16);
    }
    sum[i] = s;
    seat[i] = 0;
}

// Places by counting: seat[i] += the entries of a block of kGaCount that come
// before i.  Grid (blocks, blocks); a launch compares every pair, n^2 of
// them, which at 10,000 entries costs less than a sort's dozen launches.  In
// a block before i's own, equal entries come first; in one after, i does.
constexpr int kGaCount = 256;
template <typename Before, typename After>
__device__ __forceinline__ int ga_count(int nj, int j0, int i, Before&& not_after, After&& before) {
    int c = 0;
    if (blockIdx.y < blockIdx.x) {
#pragma unroll 16
        for (int t = 0; t < kGaCount; ++t) c += not_after(t);
    } else if (blockIdx.y > blockIdx.x) {
#pragma unroll 16
        for (int t = 0; t < nj; ++t) c += before(t);
    } else {
        for (int t = 0; t < nj; ++t) c += j0 + t < i ? not_after(t) : before(t);
    }
    return c;
}
__global__ void __launch_bounds__(kGaCount) k_ga_seats_sum(const uint32_t* sum, int n, int32_t* seat) {
    __shared__ uint32_t other[kGaCount];
    const int i = blockIdx.x * kGaCount + threadIdx.x, j0 = blockIdx.y * kGaCount, nj = min(kGaCount, n - j0);
    if ((int)threadIdx.x < nj) other[threadIdx.x] = sum[j0 + threadIdx.x];
    __syncthreads();
    if (i >= n) return;
    const uint32_t mine = sum[i];
    const int c = ga_count(nj, j0, i, [&](int t) { return other[t] <= mine; }, [&](int t) { return other[t] < mine; });
    if (c) atomicAdd(seat + i, c);
}

// The ranks in seat order, and who sits where.
__global__ void k_ga_seat_ranks(const uint32_t* rank2, const uint32_t* sum, const int32_t* seat, int n, int q,
                                uint32_t* sorted2, uint32_t* sorted_sum, int32_t* who) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int p = seat[i];
    who[p] = i;
    sorted_sum[p] = sum[i];
    for (int k = 0; k < q; ++k) sorted2[(size_t)k * n + p] = rank2[(size_t)k * n + i];
}

// dom[w][i] bit b: seat j = 32 w + b dominates seat i: every rank no larger
// and the sum smaller.  A block: 256 seats i against the 128 (64 where 128 do
// not fit) of its words, whose ranks are staged in shared memory; words above i's own stay unread.
// Q: words of two ranks (zero-padded).
__host__ __device__ constexpr int ga_dom_j(int q) { return q > 64 ? 64 : 128; }
template <int Q>
__global__ void __launch_bounds__(256) k_ga_dominance_ranks(const uint32_t* sorted2, const uint32_t* sorted_sum, int n,
                                                            int q, uint32_t* dom) {
    constexpr int kGaDomJ = ga_dom_j(Q);
    __shared__ __align__(16) uint32_t rj[kGaDomJ][Q];
    __shared__ uint32_t sj[kGaDomJ];
    const int i0 = blockIdx.x * 256, j0 = blockIdx.y * kGaDomJ;
    if (j0 > i0 + 255) return;
    for (int t = threadIdx.x; t < kGaDomJ * Q; t += 256) {
        const int k = t / kGaDomJ, j = t % kGaDomJ;
        rj[j][k] = k < q && j0 + j < n ? sorted2[(size_t)k * n + j0 + j] : 0;
    }
    for (int t = threadIdx.x; t < kGaDomJ; t += 256) sj[t] = j0 + t < n ? sorted_sum[j0 + t] : 0xFFFFFFFFu;
    __syncthreads();
    const int i = i0 + threadIdx.x, ic = min(i, n - 1);
    uint32_t neg[Q];  // minus i's ranks, halves apart
#pragma unroll
    for (int k = 0; k < Q; ++k) neg[k] = k < q ? __vneg2(sorted2[(size_t)k * n + ic]) : 0;
    const uint32_t si = sorted_sum[ic];
    for (int w = 0; w < kGaDomJ / 32; ++w) {
        uint32_t word = 0;
        for (int b = 0; b < 32; ++b) {
            const uint32_t* r = rj[w * 32 + b];
            const bool maybe = sj[w * 32 + b] < si;
            if (!__any_sync(0xFFFFFFFFu, maybe)) continue;
            uint32_t acc = 0x80008000u;
            bool open = maybe;
#pragma unroll
            for (int k = 0; k < Q; k += 8) {
#pragma unroll
                for (int u = k; u < k + 8 && u < Q; ++u) acc = __viaddmax_s16x2(r[u], neg[u], acc);
                open = maybe && (int)acc < 0x10000 && (int)(acc << 16) <= 0;  // no rank larger so far
                if (k + 8 < Q && !__any_sync(0xFFFFFFFFu, open)) break;
            }
            word |= (uint32_t)open << b;
        }
        if (i < n && j0 + w * 32 <= i) dom[(size_t)(j0 / 32 + w) * n + i] = word;
    }
}

// Front ranks by counting: cnt = a seat's dominators not yet in a front.  A
// cooperative grid, four threads per seat (a round is the latency of its
// loads and one grid barrier), one barrier per front: round f
// takes front f (mask f % 3) off the counts, puts the seats that reach zero
// into front f + 1 and clears the third mask.  Then the fronts' sizes and
// starts.
struct GaFrontCountArgs {
    const uint32_t* dom;     // [W][n]
    const int32_t* who;      // [n] individual of each seat
    int n, W;
    int32_t* rank;           // [n], by individual
    uint32_t* mask;          // [3][W]
    int32_t* start;          // [n + 1] individuals in fronts before each
    int32_t* n_fronts;
};
__global__ void __launch_bounds__(kGaDomThreads) k_ga_fronts_count(const GaFrontCountArgs a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ uint32_t words[kGaSmallMax / 32];
    __shared__ uint16_t at[kGaSmallMax / 32];
    __shared__ int n_words, part[kGaDomThreads];
    const int at0 = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
    for (int t = at0; t < 3 * a.W; t += gs) a.mask[t] = 0;
    for (int t = at0; t <= a.n; t += gs) a.start[t] = 0;
    const int i = at0 >> 2, sub = at0 & 3;
    const bool in = i < a.n;
    auto seat_sum = [](int x) {
        x += __shfl_xor_sync(0xFFFFFFFFu, x, 1);
        return x + __shfl_xor_sync(0xFFFFFFFFu, x, 2);
    };
    int cnt = 0;
    if (in) {
#pragma unroll 8
        for (int w = sub; w <= i / 32; w += 4) cnt += __popc(a.dom[(size_t)w * a.n + i]);
    }
    cnt = seat_sum(cnt);
    grid.sync();
    int mine = -1;
    if (in && cnt == 0) {
        mine = 0;
        if (sub == 0) atomicOr(a.mask + i / 32, 1u << (i & 31));
    }
    grid.sync();
    int f = 0;
    for (; f < a.n; ++f) {
        const uint32_t* cur = a.mask + (f % 3) * a.W;
        uint32_t* nxt = a.mask + ((f + 1) % 3) * a.W;
        if (threadIdx.x == 0) n_words = 0;
        __syncthreads();
        for (int w = threadIdx.x; w < a.W; w += blockDim.x) {
            const uint32_t x = __ldcg(cur + w);
            if (x) {
                const int p = atomicAdd(&n_words, 1);
                words[p] = x;
                at[p] = (uint16_t)w;
            }
        }
        for (int t = at0; t < a.W; t += gs) a.mask[((f + 2) % 3) * a.W + t] = 0;
        __syncthreads();
        const int nw = n_words;
        if (nw == 0) break;  // the same in every block
        const bool open = in && mine < 0;
        int gone = 0;
        if (open) {
#pragma unroll 8
            for (int p = sub; p < nw; p += 4)
                if (at[p] <= i / 32) gone += __popc(a.dom[(size_t)at[p] * a.n + i] & words[p]);
        }
        cnt -= seat_sum(gone);
        if (open && cnt == 0) {
            mine = f + 1;
            if (sub == 0) atomicOr(nxt + i / 32, 1u << (i & 31));
        }
        grid.sync();
    }
    if (in && sub == 0) {
        a.rank[a.who[i]] = mine;
        atomicAdd(a.start + mine + 1, 1);
    }
    grid.sync();
    if (blockIdx.x != 0) return;
    if (threadIdx.x == 0) *a.n_fronts = f;
    // prefix sums of the fronts' sizes
    const int per = (f + 1 + blockDim.x - 1) / blockDim.x, lo = threadIdx.x * per, hi = min(lo + per, f + 1);
    int s = 0;
    for (int t = lo; t < hi; ++t) s += __ldcg(a.start + t);
    part[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int t = 0; t < (int)blockDim.x; ++t) {
            const int x = part[t];
            part[t] = run;
            run += x;
        }
    }
    __syncthreads();
    int run = part[threadIdx.x];
    for (int t = lo; t < hi; ++t) {
        run += __ldcg(a.start + t);
        a.start[t] = run;
    }
}

// Crowding distance contributions, as k_ga_crowd_contrib: a thread per
// objective and place.
struct GaCrowdSmallArgs {
    const double* obj;       // [n][m]
    const uint16_t* in_fronts;  // [m][n]
    const int32_t* rank;     // [n]
    const int32_t* start;    // [n + 1]
    int n, m;
    double* contrib;         // [m][n]
};
__global__ void __launch_bounds__(256) k_ga_crowd_small(const GaCrowdSmallArgs a) {
    const int k = blockIdx.y, p = blockIdx.x * 256 + threadIdx.x;
    if (p >= a.n) return;
    const uint16_t* in = a.in_fronts + (size_t)k * a.n;
    auto f = [&](int q) {
        const double x = a.obj[(size_t)in[q] * a.m + k];
        return x != x ? INFINITY : x;
    };
    const int i = in[p], r = a.rank[i], p0 = a.start[r], p1 = a.start[r + 1] - 1;
    double c;
    if (p == p0 || p == p1) {
        c = INFINITY;
    } else {
        const double lo = f(p0), hi = f(p1);
        c = hi == lo ? 0.0 : (f(p + 1) - f(p - 1)) / (hi - lo);
    }
    a.contrib[(size_t)k * a.n + i] = c;
}

// crowd[i] = sum over objectives in order; its key (larger first), and the
// seat of i's front's first survivor
__global__ void k_ga_crowd_seats(const double* contrib, const int32_t* rank, const int32_t* start, int n, int m,
                                 double* crowd, uint64_t* key, int32_t* seat) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double c = 0.0;
#pragma unroll 8
    for (int k = 0; k < m; ++k) c += contrib[(size_t)k * n + i];
    crowd[i] = c;
    key[i] = ga_order_key(-c);
    seat[i] = start[rank[i]];
}

// seat[i] += the entries of a block of kGaCount with i's rank that come
// before i by (key, index)  (rank: nullptr, one rank for all)
__global__ void __launch_bounds__(kGaCount) k_ga_seats_key(const uint64_t* key, const int32_t* rank, int n,
                                                           int32_t* seat) {
    __shared__ uint64_t other[kGaCount];
    __shared__ int32_t other_rank[kGaCount];
    const int i = blockIdx.x * kGaCount + threadIdx.x, j0 = blockIdx.y * kGaCount, nj = min(kGaCount, n - j0);
    int32_t r0 = 0;
    if ((int)threadIdx.x < nj) {
        other[threadIdx.x] = key[j0 + threadIdx.x];
        r0 = rank ? rank[j0 + threadIdx.x] : 0;
        other_rank[threadIdx.x] = r0;
    }
    __syncthreads();
    const int32_t r = rank && i < n ? rank[i] : 0;
    // where one rank fills both blocks it need not be compared
    const int32_t all = other_rank[0];
    const bool same = __syncthreads_and((i >= n || r == all) && ((int)threadIdx.x >= nj || r0 == all));
    if (i >= n) return;
    const uint64_t mine = key[i];
    int c;
    if (same)
        c = ga_count(nj, j0, i, [&](int t) { return other[t] <= mine; }, [&](int t) { return other[t] < mine; });
    else
        c = ga_count(nj, j0, i, [&](int t) { return other_rank[t] == r & other[t] <= mine; },
                     [&](int t) { return other_rank[t] == r & other[t] < mine; });
    if (c) atomicAdd(seat + i, c);
}

__global__ void k_ga_take_seats(const int32_t* seat, int n, int mu, int32_t* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && seat[i] < mu) out[seat[i]] = i;
}

// truncation keys for places by counting
__global__ void k_ga_score_keys(const double* score, int n, uint64_t* key, int32_t* seat) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    key[i] = ga_order_key(score[i]);
    seat[i] = 0;
}

// ------------------------------------------- NSGA-II above 16,384
// objectives [n][m] -> [m][n], NaN as +inf (worst)
__global__ void k_ga_transpose(const double* obj, int n, int m, double* fT) {
    const size_t total = (size_t)n * m;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t i = t / m, k = t % m;
        const double x = obj[t];
        fT[k * n + i] = x != x ? INFINITY : x;
    }
}

// dom[i][w] bit b: individual j = 32 w + b dominates i (no worse in every
// objective, better in one).  Block: 256 individuals i against the 32 of
// word w, whose objectives are staged in shared memory.
__global__ void __launch_bounds__(kGaDomThreads) k_ga_dominance(const double* fT, int n, int m, int W, uint32_t* dom) {
    extern __shared__ double fj[];   // [m][32]
    const int w = blockIdx.y, j0 = 32 * w;
    for (int t = threadIdx.x; t < m * 32; t += blockDim.x) {
        const int k = t >> 5, jj = t & 31;
        fj[t] = j0 + jj < n ? fT[(size_t)k * n + j0 + jj] : INFINITY;
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int valid = n - j0;
    uint32_t le = valid >= 32 ? 0xFFFFFFFFu : ((1u << valid) - 1u), lt = 0;
    for (int k = 0; k < m && le; ++k) {
        const double fi = fT[(size_t)k * n + i];
        const double* row = fj + k * 32;
        uint32_t lem = 0, ltm = 0;
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) {
            lem |= (uint32_t)(row[jj] <= fi) << jj;
            ltm |= (uint32_t)(row[jj] < fi) << jj;
        }
        le &= lem;
        lt |= ltm;
    }
    dom[(size_t)i * W + w] = le & lt;
}

// Front ranks by peeling: front r holds the individuals no remaining one
// dominates.  A cooperative grid: each round, every CTA stages the remaining
// set R in shared memory and tests its share of individuals against it
// (dominance rows are read until a remaining dominator turns up, so a
// round's traffic is spread over the grid); new front members are or-ed
// into NF; after a grid barrier R loses NF.  Every front is non-empty
// (dominance is a strict partial order), so at most n rounds.  R, NF and
// the count are written by other CTAs: they are read through L2 (__ldcg).
constexpr int kGaMaxWords = 1024;   // n <= 32768
constexpr int kGaFrontThreads = 256;

struct GaFrontArgs {
    const uint32_t* dom;     // [n][W]
    int n, W;
    int32_t* rank;           // [n]
    uint32_t* R;             // [W] remaining
    uint32_t* NF;            // [W] this round's front
    int* remaining;
    int32_t* n_fronts;
};

__global__ void __launch_bounds__(kGaFrontThreads) k_ga_fronts(const GaFrontArgs a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ uint32_t Rs[kGaMaxWords];
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gstride = gridDim.x * blockDim.x;
    for (int w = gtid; w < a.W; w += gstride) {
        const int valid = a.n - 32 * w;
        a.R[w] = valid >= 32 ? 0xFFFFFFFFu : ((1u << valid) - 1u);
        a.NF[w] = 0;
    }
    if (gtid == 0) *a.remaining = a.n;
    grid.sync();
    int front = 0;
    for (; front < a.n; ++front) {
        if (__ldcg(a.remaining) == 0) break;    // the same value in every thread: read after the barrier
        for (int w = threadIdx.x; w < a.W; w += blockDim.x) Rs[w] = __ldcg(a.R + w);
        __syncthreads();
        for (int i = gtid; i < a.n; i += gstride) {
            if (!((Rs[i >> 5] >> (i & 31)) & 1u)) continue;
            const uint32_t* row = a.dom + (size_t)i * a.W;
            bool dominated = false;
            for (int w = 0; w < a.W; ++w) {
                if (row[w] & Rs[w]) {
                    dominated = true;
                    break;
                }
            }
            if (!dominated) {
                atomicOr(a.NF + (i >> 5), 1u << (i & 31));
                a.rank[i] = front;
            }
        }
        grid.sync();
        for (int w = gtid; w < a.W; w += gstride) {
            const uint32_t nf = __ldcg(a.NF + w);
            if (nf) {
                a.R[w] = __ldcg(a.R + w) & ~nf;
                a.NF[w] = 0;
                atomicSub(a.remaining, __popc(nf));
            }
        }
        grid.sync();
    }
    // unreachable with every front non-empty; kept so that a rank is always a valid index
    for (int i = gtid; i < a.n; i += gstride)
        if ((__ldcg(a.R + (i >> 5)) >> (i & 31)) & 1u) a.rank[i] = min(front, a.n - 1);
    if (gtid == 0) *a.n_fronts = __ldcg(a.remaining) == 0 ? front : -1;
}

// Crowding distance per objective k (one sorted segment each): sort by
// (rank, f_k, index); the first and last of each front get +inf, the others
// (f_next - f_prev) / (f_last - f_first) of their front (0 where the front is
// flat in f_k).
struct GaCrowdArgs {
    const double* fT;        // [m][n]
    const int32_t* rank;     // [n]
    int n, m;
    uint32_t n2;
    GaSortSlice s;           // [m][n2]
    int32_t* start;          // [m][n] first sorted position of each rank
    int32_t* end;
    double* contrib;         // [m][n]
};

__global__ void k_ga_crowd_keys(const GaCrowdArgs a) {
    const size_t total = (size_t)a.m * a.n2;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t k = t / a.n2;
        const uint32_t i = (uint32_t)(t % a.n2);
        const bool in = i < (uint32_t)a.n;
        a.s.k1[t] = in ? (uint64_t)a.rank[i] : ~0ull;
        a.s.k2[t] = in ? ga_order_key(a.fT[k * a.n + i]) : ~0ull;
        a.s.idx[t] = i;
    }
}

__global__ void k_ga_crowd_bounds(const GaCrowdArgs a) {
    const size_t total = (size_t)a.m * a.n;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t k = t / a.n;
        const int p = (int)(t % a.n);
        const uint64_t* k1 = a.s.k1 + k * a.n2;
        const uint64_t r = k1[p];
        if (p == 0 || k1[p - 1] != r) a.start[k * a.n + r] = p;
        if (p == a.n - 1 || k1[p + 1] != r) a.end[k * a.n + r] = p;
    }
}

__global__ void k_ga_crowd_contrib(const GaCrowdArgs a) {
    const size_t total = (size_t)a.m * a.n;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t k = t / a.n;
        const int p = (int)(t % a.n);
        const uint64_t* k1 = a.s.k1 + k * a.n2;
        const uint32_t* ix = a.s.idx + k * a.n2;
        const double* f = a.fT + k * a.n;
        const uint64_t r = k1[p];
        const int p0 = a.start[k * a.n + r], p1 = a.end[k * a.n + r];
        double c;
        if (p == p0 || p == p1) {
            c = INFINITY;
        } else {
            const double lo = f[ix[p0]], hi = f[ix[p1]];
            c = hi == lo ? 0.0 : (f[ix[p + 1]] - f[ix[p - 1]]) / (hi - lo);
        }
        a.contrib[k * a.n + ix[p]] = c;
    }
}

// crowd[i] = sum over objectives in order; then the survivor keys (rank,
// -crowd, index)
__global__ void k_ga_crowd_sum(const double* contrib, const int32_t* rank, int n, int m, uint32_t n2, double* crowd,
                               GaSortSlice s) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += gridDim.x * blockDim.x) {
        if (i < (uint32_t)n) {
            double c = 0.0;
            for (int k = 0; k < m; ++k) c += contrib[(size_t)k * n + i];
            crowd[i] = c;
            s.k1[i] = (uint64_t)rank[i];
            s.k2[i] = ga_order_key(-c);
        } else {
            s.k1[i] = ~0ull;
            s.k2[i] = ~0ull;
        }
        s.idx[i] = i;
    }
}

}  // namespace ngpu
