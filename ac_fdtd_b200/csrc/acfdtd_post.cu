// acfdtd_post.cu -- impulse-response post-processing in FP64.
//
// The steps after the time loop (ac-fdtd src/ac_fdtd/metrics.py:57-111 and the spectral division of
// src/ac_fdtd/sources.py:80-108), on the receiver signals where the recordings already are; every
// sum in FP64.
//
// A channel is a cluster of up to eight CTAs, each with its part of the signal; what crosses them
// (a sum, a smallest index) goes through distributed shared memory in a fixed order, so results do
// not depend on timing and no scratch memory is needed. One CTA per channel left two thirds of the
// SMs idle, read the signal up to three times with a stride and spent some 130 operations in double
// precision on every level. 48 signals of 96,000 samples,
// with the signal or curve in L2: the curve 113 to 37 us (74 MB of traffic, 11 us at the measured copy
// rate; bound now by double-precision issue and its phases' barriers in two waves of CTAs), a fit 27 to
// 23, a clarity 12 to 10; one signal 112 to 14, 26 to 13 and 12 to 7. From cold caches the spectrum's
// peak takes 29 to 4 us. Signals of 600 samples pay for the cluster: a curve 4.3 to 6.2 us, a fit 6.2 to
// 7.2.

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

__device__ __forceinline__ int64_t block_min(int64_t v, int64_t *shared) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = min(v, (int64_t)__shfl_xor_sync(0xffffffffu, v, d));
    if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = v;
    __syncthreads();
    int64_t least = shared[0];
#pragma unroll
    for (int w = 1; w < kWarps; w++) least = min(least, shared[w]);
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

// The part [begin, begin + count) of a channel's n samples that this CTA of its cluster holds.
struct Part {
    int64_t begin, count, channel;
    int rank, size;
};

__device__ __forceinline__ Part part_of(const cg::cluster_group &cluster, int64_t n) {
    Part p;
    p.rank = (int)cluster.block_rank();
    p.size = (int)cluster.num_blocks();
    p.channel = blockIdx.x / p.size;
    const int64_t each = (n + p.size - 1) / p.size;
    p.begin = min((int64_t)p.rank * each, n);
    p.count = min(each, n - p.begin);
    return p;
}

// f(q, from[q]) for this thread's samples of a part, eight loads in flight at a time.
template <typename F>
__device__ __forceinline__ void each_sample(const double *from, int64_t count, F f) {
    for (int64_t q0 = threadIdx.x; q0 < count; q0 += 8 * kThreads) {
        double x[8];
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (q0 + e * kThreads < count) x[e] = from[q0 + e * kThreads];
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (q0 + e * kThreads < count) f(q0 + e * kThreads, x[e]);
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
__device__ __forceinline__ void gather(const cg::cluster_group &cluster, V *mine, V *all) {
    if (cluster.num_blocks() == 1) {
        if (threadIdx.x == 0) all[0] = *mine;    // that thread wrote it
    } else {
        cluster.sync();
        if (threadIdx.x < cluster.num_blocks()) all[threadIdx.x] = *cluster.map_shared_rank(mine, threadIdx.x);
    }
    __syncthreads();
}

struct Two {
    double a, b;
};

// The cluster's sums of two values per thread, in a fixed order.
__device__ __forceinline__ Two cluster_sums(const cg::cluster_group &cluster, double a, double b, double *shared,
                                            Two *mine, Two *all) {
    a = block_sum(a, shared);
    b = block_sum(b, shared);
    if (threadIdx.x == 0) *mine = {a, b};
    gather(cluster, mine, all);
    // from the last part on: a response decays, so its small sums come together before the large one
    Two total = {0.0, 0.0};
    for (int r = (int)cluster.num_blocks() - 1; r >= 0; r--) {
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

// Parts of at most kThreads x kRun samples: a thread holds kRun consecutive ones in registers, so
// the CTA scans once. They come and go through shared memory, with a row of kRun + 1 per thread so
// that neither side has bank conflicts. 48 signals of 96,000 samples: 2 waves of 2 CTAs per SM, by
// the shared memory.
__global__ void __launch_bounds__(kThreads, 2) schroeder_decay_kernel(const double *response, int64_t n, int64_t each,
                                                                      double floor_db, double *decay) {
    extern __shared__ double staged[];
    __shared__ double shared[kWarps], sums[kCluster];
    __shared__ double sum, first, whole_sum;
    __shared__ LogTable table;
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), size = (int)cluster.num_blocks();
    const int64_t channel = blockIdx.x / size, begin = min(rank * each, n);
    const int count = (int)min(each, n - begin);
    const double *h = response + channel * n + begin;
    double *out = decay + channel * n + begin;
    fill(table);
    each_sample(h, count, [&](int64_t q, double x) { staged[q + (int)q / kRun] = x * x; });
    __syncthreads();
    double x[kRun], mine = 0.0;
    const int first_sample = (int)threadIdx.x * kRun;
    double *row = staged + threadIdx.x * (kRun + 1);
#pragma unroll
    for (int e = kRun - 1; e >= 0; e--) {        // from the latest sample on: I within the run
        mine += first_sample + e < count ? row[e] : 0.0;
        x[e] = mine;
    }
    // the runs later in time: threads in reverse order
    double total;
    const double later = block_exclusive_scan_down(mine, shared, &total);
    if (threadIdx.x == 0) sum = total;
    gather(cluster, &sum, sums);
    double carry = 0.0;                          // the parts later in time, last first
    for (int r = size - 1; r > rank; r--) carry += sums[r];
    const double before = carry + later;
    if (rank == 0 && threadIdx.x == 0) first = before + x[0];
    cluster.sync();
    if (threadIdx.x == 0) whole_sum = *cluster.map_shared_rank(&first, 0);
    __syncthreads();
    const Whole whole(whole_sum);
#pragma unroll
    for (int e = 0; e < kRun; e++)
        if (first_sample + e < count) row[e] = level_of<true>(table, before + x[e], whole, floor_db);
    cluster.sync();                              // also: rank 0 stays until every CTA has read it
    for (int q = threadIdx.x; q < count; q += kThreads) out[q] = staged[q + q / kRun];
}

// Other signals: the part's I in the output, scanned tile by tile from its end.
template <bool TABLE>
__global__ void __launch_bounds__(kThreads) schroeder_decay_tiles_kernel(const double *response, int64_t n,
                                                                        double floor_db, double *decay) {
    __shared__ double shared[kWarps], sums[kCluster];
    __shared__ double sum, first, whole_sum;
    __shared__ LogTable table;
    const cg::cluster_group cluster = cg::this_cluster();
    const Part part = part_of(cluster, n);
    const double *h = response + part.channel * n + part.begin;
    double *out = decay + part.channel * n + part.begin;
    if (TABLE) fill(table);
    double mine = 0.0;
    each_sample(h, part.count, [&](int64_t q, double x) {
        mine += x * x;
        out[q] = x * x;
    });
    mine = block_sum(mine, shared);
    if (threadIdx.x == 0) sum = mine;
    gather(cluster, &sum, sums);
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
    each_sample(out, part.count,
                [&](int64_t q, double i) { out[q] = level_of<TABLE>(table, i, whole, floor_db); });
}

// Seconds per 60 dB from a least-squares line through the decay curve between the first sample
// at or below `upper` dB and the first at or below `lower` dB (metrics.py:72-84); NaN and
// `failed[c] = 1` when the curve does not reach `lower` after `upper`, where the reference
// raises.
__global__ void __launch_bounds__(kThreads) decay_fit_kernel(const double *decay, int64_t n, double sample_rate,
                                                             double upper, double lower, double *seconds,
                                                             int32_t *failed) {
    __shared__ double shared[kWarps];
    __shared__ int64_t ishared[kWarps];
    __shared__ longlong2 at, every_at[kCluster];
    __shared__ Two sums, products, all[kCluster];
    const cg::cluster_group cluster = cg::this_cluster();
    const Part part = part_of(cluster, n);
    const double *d = decay + part.channel * n + part.begin;
    int64_t first_upper = n, first_lower = n;
    each_sample(d, part.count, [&](int64_t q, double v) {
        if (v <= upper) first_upper = min(first_upper, part.begin + q);
        if (v <= lower) first_lower = min(first_lower, part.begin + q);
    });
    first_upper = block_min(first_upper, ishared);
    first_lower = block_min(first_lower, ishared);
    if (threadIdx.x == 0) at = make_longlong2(first_upper, first_lower);
    gather(cluster, &at, every_at);
    int64_t start = n, end = n;
    for (int r = 0; r < part.size; r++) {
        start = min(start, (int64_t)every_at[r].x);
        end = min(end, (int64_t)every_at[r].y);
    }
    if (start == n) start = 0;   // numpy.argmax of an all-false mask
    if (end == n) end = 0;
    if (end <= start) {          // the same in every CTA of the cluster
        if (part.rank == 0 && threadIdx.x == 0) {
            seconds[part.channel] = __longlong_as_double(0x7ff8000000000000ll);
            failed[part.channel] = 1;
        }
        cluster.sync();
        return;
    }
    const int64_t q0 = max(start - part.begin, (int64_t)0), q1 = min(end - part.begin, part.count);
    const double m = (double)(end - start);
    // over sample numbers, which are exact (as doubles, by exact sums instead of conversions); the rate
    // scales the slope
    auto each_fitted = [&](auto f) {
        for (int64_t q = q0 + threadIdx.x; q < q1; q += 8 * kThreads) {
            const double k = (double)(part.begin + q);
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (q + e * kThreads < q1) f(k + (double)(e * kThreads), d[q + e * kThreads]);
        }
    };
    double sx = 0.0, sy = 0.0;
    each_fitted([&](double x, double y) {
        sx += x;
        sy += y;
    });
    const Two sum = cluster_sums(cluster, sx, sy, shared, &sums, all);
    const double mean_x = sum.a / m, mean_y = sum.b / m;
    double sxy = 0.0, sxx = 0.0;
    each_fitted([&](double x, double y) {
        x -= mean_x;
        sxy = fma(x, y - mean_y, sxy);
        sxx = fma(x, x, sxx);
    });
    const Two product = cluster_sums(cluster, sxy, sxx, shared, &products, all);
    const double slope = product.a / product.b;
    if (part.rank == 0 && threadIdx.x == 0) {
        seconds[part.channel] = -60.0 / (slope * sample_rate);
        failed[part.channel] = 0;
    }
    cluster.sync();              // every CTA's sums are read
}

// Early-to-late energy ratio in dB with the split at sample `boundary` (metrics.py:104-110).
__global__ void __launch_bounds__(kThreads) clarity_kernel(const double *response, int64_t n, int64_t boundary,
                                                           double *db) {
    __shared__ double shared[kWarps];
    __shared__ Two sums, all[kCluster];
    const cg::cluster_group cluster = cg::this_cluster();
    const Part part = part_of(cluster, n);
    const double *h = response + part.channel * n + part.begin;
    double early = 0.0, late = 0.0;
    each_sample(h, part.count, [&](int64_t q, double x) {
        const double e = x * x;
        if (part.begin + q < boundary) early += e;
        else late += e;
    });
    const Two sum = cluster_sums(cluster, early, late, shared, &sums, all);
    if (part.rank == 0 && threadIdx.x == 0) db[part.channel] = 10.0 * log10(sum.a / sum.b);
    cluster.sync();              // every CTA's sums are read
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

// Launches `kernel` with a cluster of `size` CTAs per channel.
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
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// CTAs per channel of the sums: one below 4096 samples, where a pass is shorter than the
// cluster's barriers.
int cluster_size(int64_t n) { return n <= 4096 ? 1 : kCluster; }

}  // namespace

extern "C" {

int acf_schroeder_decay(const double *response, int64_t channels, int64_t n, double floor_db,
                        double *decay, acf_stream stream) {
    int rc = check_post_args(response, decay, channels, n);
    if (rc) return rc;
    constexpr int64_t held = (int64_t)kThreads * kRun;
    cudaStream_t st = (cudaStream_t)stream;
    if (n <= kTile || n > kCluster * held) {
        ACF_CUDA(n <= kTile ? launch(schroeder_decay_tiles_kernel<false>, channels, 1, 0, st, response, n, floor_db, decay)
                            : launch(schroeder_decay_tiles_kernel<true>, channels, kCluster, 0, st, response, n,
                                     floor_db, decay));
        return ACF_OK;
    }
    constexpr size_t smem = (size_t)kThreads * (kRun + 1) * sizeof(double);
    ACF_CUDA(cudaFuncSetAttribute((const void *)schroeder_decay_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
    const int size = (int)((n + held - 1) / held);
    ACF_CUDA(launch(schroeder_decay_kernel, channels, size, smem, st, response, n, (n + size - 1) / size, floor_db,
                    decay));
    return ACF_OK;
}

int acf_decay_fit(const double *decay, int64_t channels, int64_t n, double sample_rate, double upper_db,
                  double lower_db, double *seconds, int32_t *failed, acf_stream stream) {
    int rc = check_post_args(decay, seconds, channels, n);
    if (rc) return rc;
    if (!failed) return fail(ACF_ERR_ARGUMENT, "null device array");
    if (!(sample_rate > 0.0)) return fail(ACF_ERR_ARGUMENT, "sample rate must be positive");
    ACF_CUDA(launch(decay_fit_kernel, channels, cluster_size(n), 0, (cudaStream_t)stream, decay, n, sample_rate, upper_db,
                    lower_db, seconds, failed));
    return ACF_OK;
}

int acf_clarity(const double *response, int64_t channels, int64_t n, int64_t boundary, double *db,
                acf_stream stream) {
    int rc = check_post_args(response, db, channels, n);
    if (rc) return rc;
    ACF_CUDA(launch(clarity_kernel, channels, cluster_size(n), 0, (cudaStream_t)stream, response, n, boundary, db));
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
