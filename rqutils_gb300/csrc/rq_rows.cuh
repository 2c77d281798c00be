// Row products shared by the single-problem and the batched matvec launches and the persistent
// LOBPCG kernel: the diagonal of one X group on a row, and the tiled cached products.
#pragma once

#include <type_traits>

#include "rq_common.cuh"

namespace rq {
namespace {

// 64-bit coefficients enter as bit patterns: on GB300 a warp's FP64 instruction (a comparison too)
// holds its SM quarter for 64 cycles, and integer ones do not.
__device__ __forceinline__ bool is_zero(uint64_t bits) { return (bits << 1) == 0ULL; }
__device__ __forceinline__ bool is_zero(float v) { return v == 0.f; }
__device__ __forceinline__ uint64_t coef_bits(const double *p) {
    return (uint64_t)__ldg(reinterpret_cast<const unsigned long long *>(p));
}
// the value of a coefficient in the arithmetic type, as (R)c
template <typename R>
struct CoefOf;
template <>
struct CoefOf<double> {
    using B = uint64_t;
    static __device__ __forceinline__ B load(const double *p) { return coef_bits(p); }
    static __device__ __forceinline__ double signed_value(B b, bool neg) {
        return __longlong_as_double((long long)(b ^ (neg ? 0x8000000000000000ULL : 0ULL)));
    }
};
template <>
struct CoefOf<float> {
    using B = float;
    static __device__ __forceinline__ B load(const double *p) { return (float)__ldg(p); }
    static __device__ __forceinline__ float signed_value(B v, bool neg) { return neg ? -v : v; }
};

// sum_k c_k (-1)^popcount(s & z_k) over group g, stopping at the first zero coefficient.  A part that
// is zero adds nothing (the sums start at +0, so they never become -0).
template <typename R>
__device__ __forceinline__ cx<R> group_diag(const rq_terms_t &T, int g, uint64_t s) {
    using C = CoefOf<R>;
    CAcc<R> d;
    const int k1 = __ldg(T.toff + g + 1);
    for (int k = __ldg(T.toff + g); k < k1; ++k) {
        const auto re = C::load(T.coef + 2 * k), im = C::load(T.coef + 2 * k + 1);
        const bool zr = is_zero(re), zi = is_zero(im);
        if (zr && zi) break;
        const bool neg = __popcll(s & __ldg(T.zmask + k)) & 1;
        if (!zr) d.re.add(C::signed_value(re, neg));
        if (!zi) d.im.add(C::signed_value(im, neg));
    }
    return d.get();
}

// The real part alone, for real vectors (their operators have real coefficients): the same additions
// in the same order as group_diag's real part.
template <typename R>
__device__ __forceinline__ R group_diag_re(const rq_terms_t &T, int g, uint64_t s) {
    using C = CoefOf<R>;
    Acc<R> d;
    const int k1 = __ldg(T.toff + g + 1);
    for (int k = __ldg(T.toff + g); k < k1; ++k) {
        const auto re = C::load(T.coef + 2 * k);
        if (is_zero(re)) {
            if (is_zero(C::load(T.coef + 2 * k + 1))) break;
            continue;
        }
        d.add(C::signed_value(re, __popcll(s & __ldg(T.zmask + k)) & 1));
    }
    return d.get();
}

__device__ __forceinline__ int group_terms(const rq_terms_t &T, int g) { return __ldg(T.toff + g + 1) - __ldg(T.toff + g); }
// sums with long groups: more than three terms a group on average
__device__ __forceinline__ bool long_groups(const rq_terms_t &T) { return T.K > 3 * (int64_t)T.J; }

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

__device__ __forceinline__ bool zero_bits(float v) { return v == 0.f; }
__device__ __forceinline__ bool zero_bits(double v) { return is_zero((uint64_t)__double_as_longlong(v)); }
__device__ __forceinline__ bool finite_bits(float v) { return (__float_as_uint(v) & 0x7F800000u) != 0x7F800000u; }
__device__ __forceinline__ bool finite_bits(double v) {
    return ((uint32_t)(__double_as_longlong(v) >> 32) & 0x7FF00000u) != 0x7FF00000u;
}

// One element's contribution to its row (P) and the row's accumulator (A).  scaled is the diagonal's
// part; inlined into the first addition, the compiler's fused multiply-add keeps its rounding error in
// the 32-bit accumulator's compensation.
template <typename V, bool CPLX = VT<V>::kComplex>
struct RowTerm;

template <typename V>
struct RowTerm<V, true> {  // the complex product
    using R = typename VT<V>::R;
    using P = cx<R>;
    using A = CAcc<R>;
    // products of one pass over a tile (below): 8 KB of complex64, whose tiles would else be as high as
    // float32's were (CONN, low-energy rows of a 28-qubit molecule, 40,000 of 32 elements: 279 against 161 us;
    // 12 Hubbard sites, 426,000 rows of 13: 73 against 70)
    static constexpr int kTileBytes = (sizeof(V) == 8 ? 8 : 16) * 1024;
    static constexpr bool kPair = false;          // a product takes two values
    static constexpr int kEvenElems = 0;          // with kPair: elements of a tile of even rows
    static __device__ __forceinline__ P product(const rq_terms_t &T, int g, uint64_t s, const V *x, int64_t m) {
        const cx<R> d = group_diag<R>(T, g, s), v = VT<V>::ld(x, m);
        // a real diagonal times a finite value: the products with zero change nothing
        if (zero_bits(d.im) && finite_bits(v.re) && finite_bits(v.im)) return {mul_rn(d.re, v.re), mul_rn(d.re, v.im)};
        return cmul(d, v);
    }
    static __device__ __forceinline__ P scaled(R d, const V *x, int64_t i) {
        const cx<R> v = VT<V>::ld(x, i);
        return {d * v.re, d * v.im};
    }
    static __device__ __forceinline__ P times(cx<R> v, const V *x, int64_t m) { return cmul(v, VT<V>::ld(x, m)); }
    static __device__ __forceinline__ void add(A &a, P p) { a.add(p); }
    static __device__ __forceinline__ void store(V *y, int64_t i, const A &a) { VT<V>::st(y, i, a.get()); }
};

template <>
struct RowTerm<float, false> {  // the product, rounded on its own
    using P = float;
    using A = Acc<float>;
    // (16 KB would hold twice the elements of the other types: tiles twice as high, whose dense rows keep
    // their blocks longest.  CONN, 670,000 uniform rows of 23: 273 against 131 us; 150,000 low-energy rows of
    // a 28-qubit molecule, 40 each: 525 against 188; 200,000 Hubbard rows of 2: 9.5 against 8.5)
    static constexpr int kTileBytes = 8 * 1024;
    static constexpr bool kPair = false;
    static constexpr int kEvenElems = 0;
    static __device__ __forceinline__ P product(const rq_terms_t &T, int g, uint64_t s, const float *x, int64_t m) {
        return mul_rn(group_diag_re<float>(T, g, s), x[m]);
    }
    static __device__ __forceinline__ P scaled(float d, const float *x, int64_t i) { return d * x[i]; }
    static __device__ __forceinline__ void add(A &a, P p) { a.add(p); }
    static __device__ __forceinline__ void store(float *y, int64_t i, const A &a) { y[i] = a.get(); }
};

template <>
struct RowTerm<double, false> {  // both factors: the row's owner adds their exact product (one FP64 instruction, not two)
    struct P {
        double d, x;
    };
    using A = Acc<double>;
    static constexpr int kTileBytes = 16 * 1024;
    static constexpr bool kPair = true;
    static constexpr int kEvenElems = 2048;
    static __device__ __forceinline__ P product(const rq_terms_t &T, int g, uint64_t s, const double *x, int64_t m) {
        return {group_diag_re<double>(T, g, s), x[m]};
    }
    static __device__ __forceinline__ P scaled(double d, const double *x, int64_t i) { return {d, x[i]}; }
    static __device__ __forceinline__ P times(cx<double> v, const double *x, int64_t m) { return {v.re, x[m]}; }
    static __device__ __forceinline__ void add(A &a, P p) { a.s = fma(p.d, p.x, a.s); }
    static __device__ __forceinline__ void store(double *y, int64_t i, const A &a) { y[i] = a.get(); }
};

// The same for cached elements.  In 32 bits a real product comes with its rounding error, which goes into
// the accumulator's compensation.
template <typename V>
struct CsrTerm : RowTerm<V> {};
template <>
struct CsrTerm<float2> : RowTerm<float2> {
    static constexpr int kTileBytes = 16 * 1024;  // (352,000 even rows of 39: 93 us against 121 with 8 KB)
};
template <>
struct CsrTerm<double> : RowTerm<double> {
    static constexpr int kTileBytes = 32 * 1024;  // tiles serve at most 2^15 rows here, which leave room
};
template <>
struct CsrTerm<float> {
    struct P {
        float p, low;
    };
    using A = Acc<float>;
    static constexpr int kTileBytes = 16 * 1024;
    static constexpr bool kPair = true;
    static constexpr int kEvenElems = 4096;
    static __device__ __forceinline__ P of(float d, float x) {
        const float p = mul_rn(d, x);
        return {p, fmaf(d, x, -p)};
    }
    static __device__ __forceinline__ P scaled(float d, const float *x, int64_t i) { return of(d, x[i]); }
    static __device__ __forceinline__ P times(cx<float> v, const float *x, int64_t m) { return of(v.re, x[m]); }
    static __device__ __forceinline__ void add(A &a, P p) {
        a.add(p.p);
        a.c += p.low;
    }
    static __device__ __forceinline__ void store(float *y, int64_t i, const A &a) { y[i] = a.get(); }
};

// ------------------------------------------------------------------------------------------
// cached products by tiles: elements in parallel, rows in order
// ------------------------------------------------------------------------------------------
// A thread per row walks its list through three dependent loads per element (list entry -> group
// offsets and source row -> coefficients and x), so the longest list of a warp sets its time:
// 82 us for 2^18 rows of 2.6 elements on average (Hubbard 4x4, float64), 16.6 us with tiles.
// Here a block owns a tile of consecutive rows, whose elements are consecutive in the list: all
// threads form the products of the tile's elements (list reads coalesced, every gather in flight
// at once) into shared memory, then one thread per row adds its row's products from there in list
// order -- the same additions in the same order, so the results keep their bits.
constexpr int kTileRows = 256;  // most rows of a tile (one per thread)
template <typename RT>
__host__ __device__ constexpr int tile_elems() {
    return RT::kTileBytes / (int)sizeof(typename RT::P);
}

// Rows of a tile: as many as fill the product buffer with average rows, fewer when D is so small
// that blocks would be idle (half of them while the tiles are fewer than two per SM).  Real products that
// take two values fill the buffer sooner, and where their rows are long (kLongRow elements on average)
// the dense rows of a sample, which stand together, would keep a few blocks busy with many passes after
// the others: such tiles fill four fifths and are at least eight per SM (low-energy samples of a
// 28-qubit molecule, 40,000 rows of 32 elements, float64 CONN 306 us with 64 rows a tile and 122 with 16,
// float32 CSR 38 and 22 with 32).  `even` rows (large dense subspaces) take two passes instead, for full warps of
// row owners (23 qubits, 676,000 rows of 56, float64 CONN: 759 us with 8 rows a tile, 533 with 32).
constexpr double kLongRow = 12.;
template <typename RT>
inline int tile_rows(int64_t D, int64_t nnz, int sms, bool even = false) {
    const double avg = (double)nnz / (double)D;
    const bool cut = RT::kPair && avg > kLongRow && !even;
    const double fill = RT::kPair && even ? RT::kEvenElems : (cut ? 0.8 : 1.) * tile_elems<RT>();
    int r = kTileRows;
    while (r > (cut ? 8 : 16) && (r * avg > fill || (D + r - 1) / r < (cut ? 8 : 2) * sms)) r >>= 1;
    return r;
}

// Rows [r0, r0 + nr), nr <= kTileRows: elem(e) is element e's product, first(i, acc) adds what
// precedes the elements of row i, done(i, acc) stores.  All threads of the block call it.  With
// `split` elements of more than kShortTerms terms (terms(e) of them) wait for a second round, where
// they stand together: a warp's additions cost what its longest group costs (molecules: 2 to 24
// terms, most of them 2 or 4; 36 qubits, 150,001 rows, float64: 941 -> 738 us).  RT: RowTerm<V>, or
// CsrTerm<V> for elements without groups.
constexpr int kShortTerms = 4;
template <typename V, typename RT, typename E, typename N, typename F, typename S>
__device__ __forceinline__ void tile_product(const int64_t *rowptr, int64_t r0, int nr, bool split, E &&elem,
                                             N &&terms, F &&first, S &&done) {
    constexpr int kT = tile_elems<RT>();
    constexpr bool kGroups = std::is_same<RT, RowTerm<V>>::value;
    __shared__ int rp[kTileRows + 1];
    __shared__ __align__(16) unsigned char buf[RT::kTileBytes];
    __shared__ uint16_t late[kGroups ? kT : 1];
    __shared__ int nlate;
    if (!kGroups) split = false;
    if (threadIdx.x == 0) nlate = 0;
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
        for (int k = threadIdx.x; k < m; k += blockDim.x) {
            if (split && terms(base + t0 + k) > kShortTerms) late[atomicAdd(&nlate, 1)] = (uint16_t)k;
            else prod[k] = elem(base + t0 + k);
        }
        __syncthreads();
        if (split) {
            const int nl = nlate;
            for (int q = threadIdx.x; q < nl; q += blockDim.x) prod[late[q]] = elem(base + t0 + late[q]);
            __syncthreads();
            if (threadIdx.x == 0) nlate = 0;  // (two barriers before the next pass adds to it)
        }
        for (int k = max(a - t0, 0); k < min(b - t0, m); ++k) RT::add(acc, prod[k]);
        __syncthreads();
    }
    if (own) done(r0 + threadIdx.x, acc);
    __syncthreads();  // rp is read by every thread of the tile before the next one overwrites it
}

}  // namespace
}  // namespace rq
