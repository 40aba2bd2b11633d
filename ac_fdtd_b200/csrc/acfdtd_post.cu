// acfdtd_post.cu -- impulse-response post-processing in FP64.
//
// The steps after the time loop (ac-fdtd src/ac_fdtd/metrics.py:57-111 and the spectral division of
// src/ac_fdtd/sources.py:80-108), on the receiver signals where the recordings already are; every
// sum in FP64.
//
// A channel is one CTA, or for long signals a cluster of up to eight, each with its part; what crosses CTAs
// (a sum, a smallest index) goes through distributed shared memory in a fixed order, so results do
// not depend on timing and no scratch memory is needed. Before, a channel was one CTA that read the signal up to
// three times with a stride and spent some 130 operations in double precision on every level. 48 signals of
// 96,000 samples, with the signal or curve in L2: the curve 111 to 33 us (74 MB of traffic, 11 us at the measured
// copy rate; bound now by double-precision issue and its phases' barriers in two waves of CTAs), a fit 24 to
// 16, a clarity 10 to 8; one signal 109 to 12, 24 to 10 and 9.9 to 4.7. Signals of 600 samples are bound by the
// launch: a curve 2.8 to 2.4, a fit 5.0 to 4.1, a clarity 2.5 to 2.3. From cold caches the spectrum's
// peak takes 29 to 4 us.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "acfdtd_b200.h"
#include "acfdtd_host.cuh"

namespace cg = cooperative_groups;
using namespace acf;

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kCluster = 8;
constexpr int64_t kClusterCtas = 148, kClusterSamples = 160000;   // cluster_size
constexpr int kTile = 4 * kThreads;              // samples per pass of the scan
constexpr int kRun = 24;                         // consecutive samples a thread of the scan holds

// One double per thread: the sum over the CTA, in a fixed order, to every thread.
__device__ __forceinline__ double block_sum(double v, double *shared) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = v;
    __syncthreads();
    double level[kWarps];                        // pairwise: fewer roundings than one after the other
#pragma unroll
    for (int w = 0; w < kWarps; w++) level[w] = shared[w];
#pragma unroll
    for (int width = kWarps / 2; width > 0; width /= 2)
#pragma unroll
        for (int w = 0; w < width; w++) level[w] += level[w + width];
    __syncthreads();
    return level[0];
}

struct Two {
    double a, b;
};

// block_sum of two values, in one pass.
__device__ __forceinline__ Two block_sums(double a, double b, Two *shared) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, d);
        b += __shfl_xor_sync(0xffffffffu, b, d);
    }
    if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = {a, b};
    __syncthreads();
    Two level[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; w++) level[w] = shared[w];
#pragma unroll
    for (int width = kWarps / 2; width > 0; width /= 2)
#pragma unroll
        for (int w = 0; w < width; w++) {
            level[w].a += level[w + width].a;
            level[w].b += level[w + width].b;
        }
    __syncthreads();
    return level[0];
}

__device__ __forceinline__ longlong2 block_mins(int64_t a, int64_t b, longlong2 *shared) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        a = min(a, (int64_t)__shfl_xor_sync(0xffffffffu, a, d));
        b = min(b, (int64_t)__shfl_xor_sync(0xffffffffu, b, d));
    }
    if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = make_longlong2(a, b);
    __syncthreads();
    longlong2 least = shared[0];
#pragma unroll
    for (int w = 1; w < kWarps; w++) {
        least.x = min(least.x, shared[w].x);
        least.y = min(least.y, shared[w].y);
    }
    __syncthreads();
    return least;
}

// Sum of the values of the threads after this one; *total gets the CTA's sum.
__device__ __forceinline__ double block_exclusive_scan_down(double v, double *shared, double *total) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double inclusive = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double down = __shfl_down_sync(0xffffffffu, inclusive, d);
        if (lane + d < 32) inclusive += down;
    }
    double within = __shfl_down_sync(0xffffffffu, inclusive, 1);
    if (lane == 31) within = 0.0;
    if (lane == 0) shared[warp] = inclusive;
    __syncthreads();
    double after = 0.0, all = 0.0;
#pragma unroll
    for (int w = kWarps - 1; w >= 0; w--) {
        if (w == (int)warp) after = all;
        all += shared[w];
    }
    __syncthreads();
    *total = all;
    return after + within;
}

// The part [begin, begin + count) of a channel's n samples that this CTA holds. MANY: the channel is a cluster
// of CTAs; else it is this CTA alone, launched without a cluster (whose launch and barriers cost 1.5 us).
struct Part {
    int64_t begin, count, channel;
    int rank, size;
};

template <bool MANY>
__device__ __forceinline__ Part part_of(int64_t n) {
    if (!MANY) return {0, n, (int64_t)blockIdx.x, 0, 1};
    const cg::cluster_group cluster = cg::this_cluster();
    Part p;
    p.rank = (int)cluster.block_rank();
    p.size = (int)cluster.num_blocks();
    p.channel = blockIdx.x / p.size;
    const int64_t each = (n + p.size - 1) / p.size;
    p.begin = min((int64_t)p.rank * each, n);
    p.count = min(each, n - p.begin);
    return p;
}

// f(first + q, from[q]) for this thread's q below `count`, ascending; sixteen loads in flight at a time while
// there are so many (a CTA alone on its SM is bound by those), then eight.
template <typename Index, typename F>
__device__ __forceinline__ void each_sample(const double *from, int64_t count, Index first, F f) {
    const double *at = from + threadIdx.x;
    Index q = first + (Index)threadIdx.x;
    int64_t left = count - threadIdx.x;
    for (; left > 15 * kThreads; left -= 16 * kThreads, at += 16 * kThreads, q += (Index)(16 * kThreads)) {
        double x[16];
#pragma unroll
        for (int e = 0; e < 16; e++) x[e] = at[e * kThreads];
#pragma unroll
        for (int e = 0; e < 16; e++) f(q + (Index)(e * kThreads), x[e]);
    }
    for (; left > 0; left -= 8 * kThreads, at += 8 * kThreads, q += (Index)(8 * kThreads)) {
        double x[8];
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (left > e * kThreads) x[e] = at[e * kThreads];
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (left > e * kThreads) f(q + (Index)(e * kThreads), x[e]);
    }
}

// log10 by table and series: x = 2^e m with m in [0.75, 1.5), c the nearest multiple of 1/128 to m,
// r = m / c - 1, and log10 x = e log10 2 + log10 c + log10(1 + r) with |r| <= 1/190 summed as
// its Taylor series to r^8 (the next term is below 2^-69). About 15 operations in double precision
// where the library's function takes some 100: the curve of 48 x 96,000 samples spent 58 us on it.
// c = 1 around x = 1, so values there keep their relative accuracy.
constexpr int kLogEntries = 97;                  // c = 0.75, ..., 1.5

struct LogTable {
    double inverse[kLogEntries], log[kLogEntries];
};

__device__ __forceinline__ void fill(LogTable &table) {
    for (int n = threadIdx.x; n < kLogEntries; n += kThreads) {
        const double inverse = 1.0 / (0.75 + n / 128.0);
        table.inverse[n] = inverse;
        table.log[n] = -log10(inverse);          // of the reciprocal as rounded
    }
}

// x positive, finite and normal.
__device__ __forceinline__ double log10_of(const LogTable &table, double x) {
    const int high = __double2hiint(x);
    // the exponent that puts the significand in [0.75, 1.5)
    const int e = (high - 0x3fe80000) >> 20;
    const double m = __hiloint2double(high - (e << 20), __double2loint(x));
    const int n = __double2int_rn(fma(m, 128.0, -96.0));
    const double r = fma(m, table.inverse[n], -1.0);
    double series = -1.0 / 8.0;
    series = fma(series, r, 1.0 / 7.0);
    series = fma(series, r, -1.0 / 6.0);
    series = fma(series, r, 1.0 / 5.0);
    series = fma(series, r, -1.0 / 4.0);
    series = fma(series, r, 1.0 / 3.0);
    series = fma(series, r, -1.0 / 2.0);
    series = fma(series * r, r, r);              // ln(1 + r)
    return fma((double)e, 0.30102999566398119521, fma(series, 0.43429448190325182765, table.log[n]));
}

// Every CTA's value of `mine` (a shared variable written by thread 0 before) into `all`, by rank: one
// thread per rank reads, since a read of another SM's shared memory takes as long as 40 of
// its own. `mine` must not change afterwards, and a CTA may exit only after a later
// cluster barrier.
template <typename V>
__device__ __forceinline__ void gather(V *mine, V *all) {
    const cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (threadIdx.x < cluster.num_blocks()) all[threadIdx.x] = *cluster.map_shared_rank(mine, threadIdx.x);
    __syncthreads();
}

// The channel's sums of two values per thread, in a fixed order.
template <bool MANY>
__device__ __forceinline__ Two channel_sums(const Part &part, double a, double b, Two *shared, Two *mine, Two *all) {
    const Two own = block_sums(a, b, shared);
    if (!MANY) return own;
    if (threadIdx.x == 0) *mine = own;
    gather(mine, all);
    // from the last part on: a response decays, so its small sums come together before the large one
    Two total = {0.0, 0.0};
    for (int r = part.size - 1; r >= 0; r--) {
        total.a += all[r].a;
        total.b += all[r].b;
    }
    return total;
}

// Schroeder's backward integral I(k) = sum_{m >= k} h(m)^2, as 10 log10 max(I(k) / I(0),
// 1e-300) floored at `floor_db` (metrics.py:57-69). The curve is normalised by I(0) as the scan
// forms it, as the reference divides by its first entry, so the first level is exactly 0 dB.

// What the levels of a curve are divided by: its whole energy, scaled by a power of two (exactly, of energies
// that count) to where the reciprocal and the remainder of a division are normal numbers.
struct Whole {
    double scale, scaled, inverse;
    __device__ __forceinline__ explicit Whole(double whole) {
        scale = whole < 1e-250 ? 0x1p600 : whole > 1e250 ? 0x1p-600 : 1.0;
        scaled = whole * scale;
        inverse = 1.0 / scaled;
    }
};

// The level of one sample. The quotient by the reciprocal gets one Newton step on its remainder
// (Markstein's), so that it is rounded as a division is: 48 curves of 96,000 samples are within 1.8e-14 dB
// of the exact ones, and take 35 us. No energy at all and sums that are not finite give NaN here, and
// 1e-300. TABLE: the logarithm by log10_of, else by the library's function (short signals, where filling
// the table takes longer than what it saves).
template <bool TABLE>
__device__ __forceinline__ double level_of(const LogTable &table, double integral, const Whole &whole, double floor_db) {
    integral *= whole.scale;
    double ratio = integral * whole.inverse;
    ratio = fmax(fma(fma(-ratio, whole.scaled, integral), whole.inverse, ratio), 1e-300);
    return fmax(10.0 * (TABLE ? log10_of(table, ratio) : log10(ratio)), floor_db);
}

// Parts of at most kThreads x RUN samples: a thread holds RUN consecutive ones in registers, so the CTA
// scans once. The longest runs come and go through shared memory, with a row of RUN + 1 per thread so
// that neither side has bank conflicts. 48 signals of 96,000 samples: 2 waves of 2 CTAs per SM, by
// the shared memory.
template <int RUN, bool TABLE, bool MANY>
__global__ void __launch_bounds__(kThreads, MANY ? 2 : 1) schroeder_decay_kernel(const double *response, int64_t n,
                                                                                 int64_t each, double floor_db,
                                                                                 double *decay) {
    constexpr bool STAGED = RUN == kRun;
    extern __shared__ double staged[];
    __shared__ double shared[kWarps], sums[kCluster];
    __shared__ double sum, first, whole_sum;
    __shared__ LogTable table;
    const int rank = MANY ? (int)cg::this_cluster().block_rank() : 0;
    const int size = MANY ? (int)cg::this_cluster().num_blocks() : 1;
    const int64_t channel = blockIdx.x / size, begin = min(rank * each, n);
    const int count = (int)min(each, n - begin);
    const double *h = response + channel * n + begin;
    double *out = decay + channel * n + begin;
    if (TABLE) fill(table);
    const int first_sample = (int)threadIdx.x * RUN;
    double *row = staged + threadIdx.x * (RUN + 1);
    double x[RUN], mine = 0.0;
    if (STAGED) {
        each_sample(h, count, 0, [&](int q, double v) { staged[q + q / RUN] = v * v; });
        __syncthreads();
#pragma unroll
        for (int e = 0; e < RUN; e++) x[e] = first_sample + e < count ? row[e] : 0.0;
    } else {
#pragma unroll
        for (int e = 0; e < RUN; e++) x[e] = first_sample + e < count ? h[first_sample + e] : 0.0;
#pragma unroll
        for (int e = 0; e < RUN; e++) x[e] *= x[e];
    }
#pragma unroll
    for (int e = RUN - 1; e >= 0; e--) {         // from the latest sample on: I within the run
        mine += x[e];
        x[e] = mine;
    }
    // the runs later in time: threads in reverse order
    double total;
    const double later = block_exclusive_scan_down(mine, shared, &total);
    double carry = 0.0;                          // the parts later in time, last first
    if (MANY) {
        if (threadIdx.x == 0) sum = total;
        gather(&sum, sums);
        for (int r = size - 1; r > rank; r--) carry += sums[r];
    }
    const double before = carry + later;
    if (rank == 0 && threadIdx.x == 0) first = before + x[0];
    if (MANY) {
        cg::this_cluster().sync();
        if (threadIdx.x == 0) whole_sum = *cg::this_cluster().map_shared_rank(&first, 0);
    }
    __syncthreads();
    const Whole whole(MANY ? whole_sum : first);
#pragma unroll
    for (int e = 0; e < RUN; e++)
        if (first_sample + e < count) {
            const double level = level_of<TABLE>(table, before + x[e], whole, floor_db);
            if (STAGED) row[e] = level;
            else out[first_sample + e] = level;
        }
    if (MANY) cg::this_cluster().sync();         // also: rank 0 stays until every CTA has read it
    else if (STAGED) __syncthreads();
    if (STAGED)
        for (int q = threadIdx.x; q < count; q += kThreads) out[q] = staged[q + q / RUN];
}

// Longer signals: the part's I in the output, scanned tile by tile from its end.
__global__ void __launch_bounds__(kThreads) schroeder_decay_tiles_kernel(const double *response, int64_t n,
                                                                        double floor_db, double *decay) {
    __shared__ double shared[kWarps], sums[kCluster];
    __shared__ double sum, first, whole_sum;
    __shared__ LogTable table;
    const cg::cluster_group cluster = cg::this_cluster();
    const Part part = part_of<true>(n);
    const double *h = response + part.channel * n + part.begin;
    double *out = decay + part.channel * n + part.begin;
    fill(table);
    double mine = 0.0;
    each_sample(h, part.count, (int64_t)0, [&](int64_t q, double x) {
        mine += x * x;
        out[q] = x * x;
    });
    mine = block_sum(mine, shared);
    if (threadIdx.x == 0) sum = mine;
    gather(&sum, sums);
    double carry = 0.0;                          // the parts later in time, last first
    for (int r = part.size - 1; r > part.rank; r--) carry += sums[r];
    for (int64_t low = (part.count - 1) / kTile * kTile; low >= 0; low -= kTile) {
        const int64_t at = low + 4 * (int64_t)threadIdx.x;            // this thread's earliest sample
        double x[4], local = 0.0, total;
#pragma unroll
        for (int e = 3; e >= 0; e--) {
            local += at + e < part.count ? out[at + e] : 0.0;
            x[e] = local;
        }
        const double before = carry + block_exclusive_scan_down(local, shared, &total);
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (at + e < part.count) out[at + e] = before + x[e];
        carry += total;
    }
    __syncthreads();
    if (part.rank == 0 && threadIdx.x == 0) first = out[0];
    cluster.sync();
    if (threadIdx.x == 0) whole_sum = *cluster.map_shared_rank(&first, 0);
    cluster.sync();                              // rank 0 stays until every CTA has read it
    const Whole whole(whole_sum);
    each_sample(out, part.count, (int64_t)0,
                [&](int64_t q, double i) { out[q] = level_of<true>(table, i, whole, floor_db); });
}

// Seconds per 60 dB from a least-squares line through the decay curve between the first sample
// at or below `upper` dB and the first at or below `lower` dB (metrics.py:72-84); NaN and
// `failed[c] = 1` when the curve does not reach `lower` after `upper`, where the reference
// raises.
template <bool MANY>
__global__ void __launch_bounds__(kThreads) decay_fit_kernel(const double *decay, int64_t n, double sample_rate,
                                                             double upper, double lower, double *seconds,
                                                             int32_t *failed) {
    __shared__ Two shared[kWarps];
    __shared__ longlong2 ishared[kWarps];
    __shared__ longlong2 at, every_at[kCluster];
    __shared__ Two sums, products, all[kCluster];
    const Part part = part_of<MANY>(n);
    const double *d = decay + part.channel * n + part.begin;
    int64_t first_upper = n, first_lower = n;
    each_sample(d, part.count, part.begin, [&](int64_t q, double v) {
        if (v <= upper) first_upper = min(first_upper, q);
        if (v <= lower) first_lower = min(first_lower, q);
    });
    const longlong2 own = block_mins(first_upper, first_lower, ishared);
    int64_t start = own.x, end = own.y;
    if (MANY) {
        if (threadIdx.x == 0) at = own;
        gather(&at, every_at);
        for (int r = 0; r < part.size; r++) {
            start = min(start, (int64_t)every_at[r].x);
            end = min(end, (int64_t)every_at[r].y);
        }
    }
    if (start == n) start = 0;   // numpy.argmax of an all-false mask
    if (end == n) end = 0;
    if (end <= start) {          // the same in every CTA of the channel
        if (part.rank == 0 && threadIdx.x == 0) {
            seconds[part.channel] = __longlong_as_double(0x7ff8000000000000ll);
            failed[part.channel] = 1;
        }
        if (MANY) cg::this_cluster().sync();
        return;
    }
    const int64_t q0 = max(start - part.begin, (int64_t)0), q1 = min(end - part.begin, part.count);
    const double m = (double)(end - start);
    // over sample numbers, which are exact (as doubles, by exact sums instead of conversions); the rate
    // scales the slope
    auto each_fitted = [&](auto f) { each_sample(d + q0, q1 - q0, (double)(part.begin + q0), f); };
    double sx = 0.0, sy = 0.0;
    each_fitted([&](double x, double y) {
        sx += x;
        sy += y;
    });
    const Two sum = channel_sums<MANY>(part, sx, sy, shared, &sums, all);
    const double mean_x = sum.a / m, mean_y = sum.b / m;
    double sxy = 0.0, sxx = 0.0;
    each_fitted([&](double x, double y) {
        x -= mean_x;
        sxy = fma(x, y - mean_y, sxy);
        sxx = fma(x, x, sxx);
    });
    const Two product = channel_sums<MANY>(part, sxy, sxx, shared, &products, all);
    const double slope = product.a / product.b;
    if (part.rank == 0 && threadIdx.x == 0) {
        seconds[part.channel] = -60.0 / (slope * sample_rate);
        failed[part.channel] = 0;
    }
    if (MANY) cg::this_cluster().sync();         // every CTA's sums are read
}

// Early-to-late energy ratio in dB with the split at sample `boundary` (metrics.py:104-110).
template <bool MANY>
__global__ void __launch_bounds__(kThreads) clarity_kernel(const double *response, int64_t n, int64_t boundary,
                                                           double *db) {
    __shared__ Two shared[kWarps];
    __shared__ Two sums, all[kCluster];
    const Part part = part_of<MANY>(n);
    const double *h = response + part.channel * n + part.begin;
    double early = 0.0, late = 0.0;
    each_sample(h, part.count, part.begin, [&](int64_t q, double x) {
        const double e = x * x;
        if (q < boundary) early += e;
        else late += e;
    });
    const Two sum = channel_sums<MANY>(part, early, late, shared, &sums, all);
    if (part.rank == 0 && threadIdx.x == 0) db[part.channel] = 10.0 * log10(sum.a / sum.b);
    if (MANY) cg::this_cluster().sync();         // every CTA's sums are read
}

// Largest |S(f)|^2 of the excitation's spectrum (the regularisation's scale). `peak` starts at 0;
// values are not negative, so their order is that of their bits.
__global__ void __launch_bounds__(256) spectrum_peak_power(const double2 *source, int64_t bins, double *peak) {
    double best = 0.0;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < bins; k += (int64_t)gridDim.x * blockDim.x) {
        const double a = hypot(source[k].x, source[k].y);
        best = fmax(best, a * a);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) best = fmax(best, __shfl_xor_sync(0xffffffffu, best, d));
    if ((threadIdx.x & 31) == 0)
        atomicMax(reinterpret_cast<unsigned long long *>(peak), (unsigned long long)__double_as_longlong(best));
}

// R(f) = X(f) conj(S(f)) / (|S(f)|^2 + reg * max |S|^2), zero above max_frequency, for every
// channel's spectrum X (sources.py:103-107). Bin k is at k * bin_hz, as numpy.fft.rfftfreq.
__global__ void spectral_divide_kernel(const double2 *spectra, const double2 *source, int64_t channels,
                                       int64_t bins, double bin_hz, double max_frequency,
                                       double regularisation, const double *peak, double2 *out) {
    const int64_t at = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= channels * bins) return;
    const int64_t k = at % bins;
    double2 r = make_double2(0.0, 0.0);
    if (!((double)k * bin_hz > max_frequency)) {
        const double2 x = spectra[at], src = source[k];
        const double a = hypot(src.x, src.y);
        const double denominator = a * a + regularisation * *peak;
        // x * conj(src): (x.x src.x - x.y (-src.y)) + (x.x (-src.y) + x.y src.x) i
        const double re = x.x * src.x - x.y * -src.y;
        const double im = x.x * -src.y + x.y * src.x;
        r = make_double2(re / denominator, im / denominator);
    }
    out[at] = r;
}

int check_post_args(const void *a, const void *b, int64_t channels, int64_t n) {
    if (!a || !b) return fail(ACF_ERR_ARGUMENT, "null device array");
    if (channels < 1 || channels > 65535 || n < 1) return fail(ACF_ERR_ARGUMENT, "need 1..65535 channels of at least one sample");
    return ACF_OK;
}

// Launches `kernel` with `size` CTAs per channel, a cluster if more than one.
template <typename... Args>
cudaError_t launch(void (*kernel)(Args...), int64_t channels, int size, size_t smem, cudaStream_t st,
                   typename std::common_type<Args>::type... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)channels * (unsigned)size);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = size > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int RUN, bool TABLE, bool MANY>
cudaError_t launch_decay(const double *response, int64_t channels, int64_t n, double floor_db, double *decay,
                         cudaStream_t st) {
    const auto kernel = schroeder_decay_kernel<RUN, TABLE, MANY>;
    constexpr size_t smem = RUN == kRun ? (size_t)kThreads * (RUN + 1) * sizeof(double) : 0;
    const cudaError_t err = smem <= 48 * 1024 ? cudaSuccess
                                              : cudaFuncSetAttribute((const void *)kernel,
                                                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                                     (int)smem);
    if (err != cudaSuccess) return err;
    const int size = (int)((n + kThreads * RUN - 1) / (kThreads * RUN));
    return launch(kernel, channels, size, smem, st, response, n, (n + size - 1) / size, floor_db, decay);
}

// The curve with the shortest runs that hold the signal, of those that pay: one signal of 2500 samples takes 3.5
// us in runs of six, 4.4 of twelve, 7.0 of 24; of 600 2.3, 2.6 (four), 6.5. Runs of one take the library's
// logarithm: filling the table would take longer (100 samples 1.6 us, in runs of two with the table 2.0).
cudaError_t decay_curve(const double *response, int64_t channels, int64_t n, double floor_db, double *decay,
                        cudaStream_t st) {
    if (n <= kThreads) return launch_decay<1, false, false>(response, channels, n, floor_db, decay, st);
    if (n <= 2 * kThreads) return launch_decay<2, true, false>(response, channels, n, floor_db, decay, st);
    if (n <= 4 * kThreads) return launch_decay<4, true, false>(response, channels, n, floor_db, decay, st);
    if (n <= 6 * kThreads) return launch_decay<6, true, false>(response, channels, n, floor_db, decay, st);
    if (n <= 8 * kThreads) return launch_decay<8, true, false>(response, channels, n, floor_db, decay, st);
    if (n <= 12 * kThreads) return launch_decay<12, true, false>(response, channels, n, floor_db, decay, st);
    if (n <= kRun * kThreads) return launch_decay<kRun, true, false>(response, channels, n, floor_db, decay, st);
    if (n <= kCluster * kRun * kThreads) return launch_decay<kRun, true, true>(response, channels, n, floor_db, decay, st);
    return launch(schroeder_decay_tiles_kernel, channels, kCluster, 0, st, response, n, floor_db, decay);
}

// CTAs per channel of a fit and a clarity. A cluster pays for its launch and barriers with 2 to 3 us, and more
// where the clusters do not all fit the device at once, so the most CTAs with which they do (one per SM), and
// only for long signals. us of a fit with 1, 2, 4 and 8 CTAs per signal: one signal of 16,000 samples 6.2, 8.3,
// 7.6, 7.7, of 32,000 8.7, 10.4, 9.0, 8.0, of 96,000 16.1, 15.3, 12.3, 10.3; 24 of 32,000 8.9, 10.7, 9.4, 10.8,
// of 48,000 10.6, 11.7, 10.1, 12.8; 48 of 64,000 13.0, 13.6, 15.9, 21.5, of 96,000 16.5, 15.7, 17.8, 23.4;
// 200 of 96,000 36, 52, 59, 87.
int cluster_size(int64_t n, int64_t channels) {
    int size = kCluster;
    while (size > 1 && (channels * size > kClusterCtas || n * size < kClusterSamples)) size /= 2;
    return size;
}

}  // namespace

extern "C" {

int acf_schroeder_decay(const double *response, int64_t channels, int64_t n, double floor_db,
                        double *decay, acf_stream stream) {
    int rc = check_post_args(response, decay, channels, n);
    if (rc) return rc;
    ACF_CUDA(decay_curve(response, channels, n, floor_db, decay, (cudaStream_t)stream));
    return ACF_OK;
}

int acf_decay_fit(const double *decay, int64_t channels, int64_t n, double sample_rate, double upper_db,
                  double lower_db, double *seconds, int32_t *failed, acf_stream stream) {
    int rc = check_post_args(decay, seconds, channels, n);
    if (rc) return rc;
    if (!failed) return fail(ACF_ERR_ARGUMENT, "null device array");
    if (!(sample_rate > 0.0)) return fail(ACF_ERR_ARGUMENT, "sample rate must be positive");
    const int size = cluster_size(n, channels);
    ACF_CUDA(launch(size > 1 ? decay_fit_kernel<true> : decay_fit_kernel<false>, channels, size, 0, (cudaStream_t)stream,
                    decay, n, sample_rate, upper_db, lower_db, seconds, failed));
    return ACF_OK;
}

int acf_clarity(const double *response, int64_t channels, int64_t n, int64_t boundary, double *db,
                acf_stream stream) {
    int rc = check_post_args(response, db, channels, n);
    if (rc) return rc;
    const int size = cluster_size(n, channels);
    ACF_CUDA(launch(size > 1 ? clarity_kernel<true> : clarity_kernel<false>, channels, size, 0, (cudaStream_t)stream,
                    response, n, boundary, db));
    return ACF_OK;
}

int acf_spectral_divide(const void *spectra, const void *source, int64_t channels, int64_t bins,
                        double bin_hz, double max_frequency, double regularisation, double *scratch,
                        void *out, acf_stream stream) {
    int rc = check_post_args(spectra, source, channels, bins);
    if (rc) return rc;
    if (!scratch || !out) return fail(ACF_ERR_ARGUMENT, "null device array");
    cudaStream_t st = (cudaStream_t)stream;
    ACF_CUDA(cudaMemsetAsync(scratch, 0, sizeof(double), st));
    spectrum_peak_power<<<(unsigned)std::min<int64_t>((bins + 255) / 256, 296), 256, 0, st>>>((const double2 *)source,
                                                                                             bins, scratch);
    const int64_t total = channels * bins;
    spectral_divide_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
        (const double2 *)spectra, (const double2 *)source, channels, bins, bin_hz, max_frequency,
        regularisation, scratch, (double2 *)out);
    ACF_CUDA(cudaGetLastError());
    return ACF_OK;
}

}  // extern "C"
