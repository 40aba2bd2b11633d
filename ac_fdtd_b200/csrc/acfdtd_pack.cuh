// acfdtd_pack.cuh -- 16-byte chunks of z elements in either precision: loads, stores and the
// arithmetic of the leapfrog, every element rounded as the scalar operation.

#ifndef ACFDTD_PACK_CUH
#define ACFDTD_PACK_CUH

#include "acfdtd_device.cuh"

namespace acf {

// A chunk: 16 bytes of consecutive z elements, four floats or two doubles.
template <typename T>
struct Pack;

template <>
struct Pack<float> {
    static constexpr int W = 4;
    float2 a, b;
};

template <>
struct Pack<double> {
    static constexpr int W = 2;
    double2 a;
};

__device__ __forceinline__ Pack<float> pload(const float *x) {
    const float4 v = *reinterpret_cast<const float4 *>(x);
    return {lo2(v), hi2(v)};
}
__device__ __forceinline__ Pack<double> pload(const double *x) { return {*reinterpret_cast<const double2 *>(x)}; }
__device__ __forceinline__ void pstore(float *x, const Pack<float> &v) {
    *reinterpret_cast<float4 *>(x) = make_float4(v.a.x, v.a.y, v.b.x, v.b.y);
}
__device__ __forceinline__ void pstore(double *x, const Pack<double> &v) { *reinterpret_cast<double2 *>(x) = v.a; }

__device__ __forceinline__ void pstore_streaming(float *x, const Pack<float> &v) {
    __stcs(reinterpret_cast<float4 *>(x), make_float4(v.a.x, v.a.y, v.b.x, v.b.y));
}
__device__ __forceinline__ void pstore_streaming(double *x, const Pack<double> &v) {
    __stcs(reinterpret_cast<double2 *>(x), v.a);
}

// Sums: in padd y is never a product (see add2); "plus a product" is psub of the product by the
// negated coefficient.
__device__ __forceinline__ Pack<float> psub(const Pack<float> &x, const Pack<float> &y) {
    return {sub2(x.a, y.a), sub2(x.b, y.b)};
}
__device__ __forceinline__ Pack<double> psub(const Pack<double> &x, const Pack<double> &y) {
    return {make_double2(x.a.x - y.a.x, x.a.y - y.a.y)};
}
__device__ __forceinline__ Pack<float> padd(const Pack<float> &x, const Pack<float> &y) {
    return {add2(x.a, y.a), add2(x.b, y.b)};
}
__device__ __forceinline__ Pack<double> padd(const Pack<double> &x, const Pack<double> &y) {
    return {make_double2(x.a.x + y.a.x, x.a.y + y.a.y)};
}
__device__ __forceinline__ Pack<float> pmul(const Pack<float> &x, float c) {
    return {mul2(x.a, dup2(c)), mul2(x.b, dup2(c))};
}
__device__ __forceinline__ Pack<double> pmul(const Pack<double> &x, double c) {
    return {make_double2(x.a.x * c, x.a.y * c)};
}
__device__ __forceinline__ Pack<float> ptimes(const Pack<float> &x, const Pack<float> &y) {
    return {mul2(x.a, y.a), mul2(x.b, y.b)};
}
__device__ __forceinline__ Pack<double> ptimes(const Pack<double> &x, const Pack<double> &y) {
    return {make_double2(x.a.x * y.a.x, x.a.y * y.a.y)};
}
template <typename T>
__device__ __forceinline__ Pack<T> zero_first(Pack<T> x) {
    x.a.x = T(0);
    return x;
}
template <typename T>
__device__ __forceinline__ Pack<T> pzero() {
    if constexpr (sizeof(T) == 4) return {dup2(0.f), dup2(0.f)};
    else return {make_double2(0.0, 0.0)};
}

__device__ __forceinline__ void unpack(const Pack<float> &x, float (&v)[4]) {
    v[0] = x.a.x; v[1] = x.a.y; v[2] = x.b.x; v[3] = x.b.y;
}
__device__ __forceinline__ void unpack(const Pack<double> &x, double (&v)[2]) {
    v[0] = x.a.x; v[1] = x.a.y;
}
__device__ __forceinline__ Pack<float> repack(const float (&v)[4]) {
    return {make_float2(v[0], v[1]), make_float2(v[2], v[3])};
}
__device__ __forceinline__ Pack<double> repack(const double (&v)[2]) { return {make_double2(v[0], v[1])}; }

// The elements one place lower and one place higher in z.
__device__ __forceinline__ Pack<float> below_of(const Pack<float> &x, float below) {
    return {make_float2(below, x.a.x), make_float2(x.a.y, x.b.x)};
}
__device__ __forceinline__ Pack<double> below_of(const Pack<double> &x, double below) {
    return {make_double2(below, x.a.x)};
}
__device__ __forceinline__ Pack<float> above_of(const Pack<float> &x, float above) {
    return {make_float2(x.a.y, x.b.x), make_float2(x.b.y, above)};
}
__device__ __forceinline__ Pack<double> above_of(const Pack<double> &x, double above) {
    return {make_double2(x.a.y, above)};
}
template <typename T>
__device__ __forceinline__ T first_of(const Pack<T> &x) { return x.a.x; }
__device__ __forceinline__ float last_of(const Pack<float> &x) { return x.b.y; }
__device__ __forceinline__ double last_of(const Pack<double> &x) { return x.a.y; }

// `x` with the elements from `from` on replaced by those of `old`.
__device__ __forceinline__ Pack<float> keep_from(Pack<float> x, const Pack<float> &old, int from) {
    if (from <= 1) x.a.y = old.a.y;
    if (from <= 2) x.b.x = old.b.x;
    if (from <= 3) x.b.y = old.b.y;
    return x;
}
__device__ __forceinline__ Pack<double> keep_from(Pack<double> x, const Pack<double> &old, int from) {
    if (from <= 1) x.a.y = old.a.y;
    return x;
}
// `x` with the elements from `from` on replaced by the one before them.
__device__ __forceinline__ Pack<float> mirrored(Pack<float> x, int from) {
    if (from <= 1) x.a.y = x.a.x;
    if (from <= 2) x.b.x = x.a.y;
    if (from <= 3) x.b.y = x.b.x;
    return x;
}
__device__ __forceinline__ Pack<double> mirrored(Pack<double> x, int from) {
    if (from <= 1) x.a.y = x.a.x;
    return x;
}

// finite_acc over the elements: two accumulators for floats, one for doubles.
__device__ __forceinline__ float2 pfinite(float2 acc, const Pack<float> &x) {
    return __ffma2_rn(x.b, dup2(0.f), __ffma2_rn(x.a, dup2(0.f), acc));
}
__device__ __forceinline__ double pfinite(double acc, const Pack<double> &x) {
    return finite_acc(finite_acc(acc, x.a.x), x.a.y);
}
__device__ __forceinline__ bool is_bad(float2 acc) { return acc.x != acc.x || acc.y != acc.y; }
__device__ __forceinline__ bool is_bad(double acc) { return acc != acc; }
__device__ __forceinline__ float2 finite_start(float) { return dup2(0.f); }
__device__ __forceinline__ double finite_start(double) { return 0.0; }

// Blocks over a room's (row, chunk) columns, groups of `planes` x planes along z of the grid: up to 32 chunks of
// a row, and rows, in at most `threads` threads. Rooms of so many rows that their blocks would exceed the
// grid's 65535 take fewer chunks and more rows per block.
struct ChunkShape {
    dim3 grid, block;
};

template <typename T>
ChunkShape chunk_shape(const Room<T> &room, int planes, int threads) {
    const int chunks = (room.nz + Pack<T>::W - 1) / Pack<T>::W;
    int bx = 1;
    while (bx < chunks && bx < 32) bx <<= 1;
    auto rows = [&]() { return threads / bx < 1 ? 1 : threads / bx < room.ny ? threads / bx : room.ny; };
    while (bx > 1 && ((int64_t)room.ny + rows() - 1) / rows() > 65535) bx >>= 1;
    const int by = rows();
    return {dim3((chunks + bx - 1) / bx, (room.ny + by - 1) / by, (room.nx + planes - 1) / planes), dim3(bx, by, 1)};
}

}  // namespace acf

#endif
