// Row products shared by the single-problem and the batched matvec launches and the persistent
// LOBPCG kernel: the diagonal of one X group on a row, and the tiled cached products.
#pragma once

#include "rq_common.cuh"

namespace rq {
namespace {

// sum_k c_k (-1)^popcount(s & z_k) over group g, stopping at the first zero coefficient
template <typename R>
__device__ __forceinline__ cx<R> group_diag(const rq_terms_t &T, int g, uint64_t s) {
    CAcc<R> d;
    const int k1 = __ldg(T.toff + g + 1);
    for (int k = __ldg(T.toff + g); k < k1; ++k) {
        const R re = (R)__ldg(T.coef + 2 * k), im = (R)__ldg(T.coef + 2 * k + 1);
        if (re == (R)0 && im == (R)0) break;
        if (__popcll(s & __ldg(T.zmask + k)) & 1) d.add({-re, -im});
        else d.add({re, im});
    }
    return d.get();
}

// The real part alone, for real vectors (their operators have real coefficients): half of the
// additions, and FP64 additions are what a cached product is made of on GB300 (FP64 runs at 1/64 of
// the FP32 rate).  The same additions in the same order as group_diag's real part.
template <typename R>
__device__ __forceinline__ R group_diag_re(const rq_terms_t &T, int g, uint64_t s) {
    Acc<R> d;
    const int k1 = __ldg(T.toff + g + 1);
    for (int k = __ldg(T.toff + g); k < k1; ++k) {
        const R re = (R)__ldg(T.coef + 2 * k);
        if (re == (R)0 && (R)__ldg(T.coef + 2 * k + 1) == (R)0) break;
        d.add((__popcll(s & __ldg(T.zmask + k)) & 1) ? -re : re);
    }
    return d.get();
}

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// One element's contribution to its row and the row's accumulator: a complex value for complex
// vectors, a real one for real vectors (the product rounded on its own, as cmul's is).  scaled is
// the diagonal's part; inlined into the first addition, the compiler's fused multiply-add keeps
// its rounding error in the 32-bit accumulator's compensation, here as in the matrix-free kernel.
template <typename V, bool CPLX = VT<V>::kComplex>
struct RowTerm;

template <typename V>
struct RowTerm<V, true> {
    using R = typename VT<V>::R;
    using P = cx<R>;
    using A = CAcc<R>;
    static __device__ __forceinline__ P product(const rq_terms_t &T, int g, uint64_t s, const V *x, int64_t m) {
        return cmul(group_diag<R>(T, g, s), VT<V>::ld(x, m));
    }
    static __device__ __forceinline__ P scaled(R d, const V *x, int64_t i) {
        const cx<R> v = VT<V>::ld(x, i);
        return {d * v.re, d * v.im};
    }
    static __device__ __forceinline__ P times(cx<R> v, const V *x, int64_t m) { return cmul(v, VT<V>::ld(x, m)); }
    static __device__ __forceinline__ void store(V *y, int64_t i, const A &a) { VT<V>::st(y, i, a.get()); }
};

template <typename V>
struct RowTerm<V, false> {
    using R = typename VT<V>::R;
    using P = R;
    using A = Acc<R>;
    static __device__ __forceinline__ P product(const rq_terms_t &T, int g, uint64_t s, const V *x, int64_t m) {
        return mul_rn(group_diag_re<R>(T, g, s), x[m]);
    }
    static __device__ __forceinline__ P scaled(R d, const V *x, int64_t i) { return d * x[i]; }
    static __device__ __forceinline__ P times(cx<R> v, const V *x, int64_t m) { return mul_rn(v.re, x[m]); }
    static __device__ __forceinline__ void store(V *y, int64_t i, const A &a) { y[i] = a.get(); }
};

// ------------------------------------------------------------------------------------------
// cached products by tiles: elements in parallel, rows in order
// ------------------------------------------------------------------------------------------
// A thread per row walks its list through three dependent loads per element (list entry -> group
// offsets and source row -> coefficients and x), so the longest list of a warp sets its time:
// 82 us for 2^18 rows of 2.6 elements on average (Hubbard 4x4, float64), 22.6 us with tiles.
// Here a block owns a tile of consecutive rows, whose elements are consecutive in the list: all
// threads form the products of the tile's elements (list reads coalesced, every gather in flight
// at once) into shared memory, then one thread per row adds its row's products from there in list
// order -- the same additions in the same order, so the results keep their bits.
constexpr int kTileBytes = 16 * 1024;  // products of one pass over a tile
constexpr int kTileRows = 256;         // most rows of a tile (one per thread)

template <typename V>
__host__ __device__ constexpr int tile_elems() {
    return kTileBytes / (int)sizeof(typename RowTerm<V>::P);
}

// Rows of a tile: as many as fill the product buffer with average rows, fewer when D is so small
// that blocks would be idle (half of them while the tiles are fewer than two per SM).
template <typename V>
inline int tile_rows(int64_t D, int64_t nnz, int sms) {
    int r = kTileRows;
    const double avg = (double)nnz / (double)D;
    while (r > 16 && (r * avg > tile_elems<V>() || (D + r - 1) / r < 2 * sms)) r >>= 1;
    return r;
}

// Rows [r0, r0 + nr), nr <= kTileRows: elem(e) is element e's product, first(i, acc) adds what
// precedes the elements of row i, done(i, acc) stores.  All threads of the block call it.
template <typename V, typename E, typename F, typename S>
__device__ __forceinline__ void tile_product(const int64_t *rowptr, int64_t r0, int nr, E &&elem, F &&first,
                                             S &&done) {
    using RT = RowTerm<V>;
    constexpr int kT = tile_elems<V>();
    __shared__ int rp[kTileRows + 1];
    __shared__ __align__(16) unsigned char buf[kTileBytes];
    typename RT::P *prod = reinterpret_cast<typename RT::P *>(buf);
    const int64_t base = __ldg(rowptr + r0);
    for (int k = threadIdx.x; k <= nr; k += blockDim.x) rp[k] = (int)(__ldg(rowptr + r0 + k) - base);
    typename RT::A acc;
    const bool own = (int)threadIdx.x < nr;
    if (own) first(r0 + threadIdx.x, acc);
    __syncthreads();
    const int n = rp[nr];
    const int a = own ? rp[threadIdx.x] : 0, b = own ? rp[threadIdx.x + 1] : 0;
    for (int t0 = 0; t0 < n; t0 += kT) {
        const int m = min(kT, n - t0);
        for (int k = threadIdx.x; k < m; k += blockDim.x) prod[k] = elem(base + t0 + k);
        __syncthreads();
        for (int k = max(a - t0, 0); k < min(b - t0, m); ++k) acc.add(prod[k]);
        __syncthreads();
    }
    if (own) done(r0 + threadIdx.x, acc);
    __syncthreads();  // rp is read by every thread of the tile before the next one overwrites it
}

}  // namespace
}  // namespace rq
