// Persistent LOBPCG: the iterations of a phase inside one cooperative launch (one problem), or of
// many problems on a group of blocks each (batches).  Included by rq_lobpcg.cu, inside its
// namespaces, after the solver state, the dot accumulators and the 3x3 eigenproblem.
//
// What bounds an iteration: its grid reductions (about 3 us each: block sums, one barrier, every
// block adding all partial sums), FP64 arithmetic (a warp's FP64 instruction occupies its SM
// quarter for 64 cycles on GB300, whichever lanes are active) and the gathers of the products.
// So:
// * a block owns a contiguous range of rows, cut so that rows and list elements are balanced, and
//   keeps its part of the connectivity in shared memory with the element values computed once per
//   launch (group diagonals have up to hundreds of terms), as far as it fits;
// * passes are merged until a reduction or a product forces a barrier: FAST has three barriers an
//   iteration (before its product, and two reductions), REFERENCE eight.  The norms of the
//   update follow from the Gram pass (which adds <x,p>, <y,p>, <p,p>), the projection's inner
//   products are formed while the residual is in registers, and in the projection rounds the
//   inner products of an unscaled vector are scaled afterwards with its norm;
// * a row's list is walked by 1 to 32 lanes (chosen per block from its rows and list length);
// * scalar steps run on one warp with independent square roots on different lanes.
// Measured per iteration (whole solve over its iterations, against one reduction per pass and lists
// walked by one thread per row): Hubbard 4x4, 2^18 rows of 2.6 elements, float64, FAST 180 -> 57 us,
// REFERENCE 477 -> 109 us; 2500 rows of 33 elements, REFERENCE 4,850 -> 109 us, FAST 1,386 -> 75 us.

constexpr long long kBarrierCycles = 4000000000LL;  // ~2 s at 2 GHz: a barrier that waits longer aborts
constexpr int kPersistThreads = 512;                // one block per SM
constexpr int kPersistBatchThreads = 256;           // two blocks per SM: problems need blocks of their own
constexpr int kMaxComps = 18;                       // real components of one reduction
constexpr int kPartStride = kMaxComps / 2;          // float4 of partial sums per block

// Grid barrier on a counter that only grows: each block adds 1 without waiting for the old value
// (the adds pipeline in L2 instead of queueing for their results) and waits until the counter
// reaches (barriers passed) x (blocks); `passed` is the block's own count, kept in shared
// memory.  Every wait is bounded; a block that gives up raises `abort`, which releases every
// other waiter at once.  Returns false after an abort.
__device__ bool group_sync(GridBar *b, unsigned int *passed, unsigned int nblocks) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned int target = (*passed + 1u) * nblocks;
        *passed += 1u;
        volatile unsigned int *count = &b->count;
        volatile int *abort = &b->abort;
        __threadfence();
        atomicAdd(&b->count, 1u);
        const long long t0 = clock64();
        while ((int)(*count - target) < 0) {
            if (*abort) {
                ok = 0;
                break;
            }
            if (clock64() - t0 > kBarrierCycles) {
                atomicExch(&b->abort, 1);
                ok = 0;
                break;
            }
        }
        __threadfence();
        if (*abort) ok = 0;
        ok_s = ok;
    }
    __syncthreads();
    return ok_s != 0;
}

// ------------------------------------------------------------------------------------------
// scalar and accumulator helpers
// ------------------------------------------------------------------------------------------
// 1 / sqrt(a): an FP32 estimate refined by one step of Householder's third-order iteration,
// y (1 + r / 2 + 3 r^2 / 8) with r = 1 - a y^2; seven FP64 instructions where the square root and
// the division take eighteen (64 cycles each here).  Outside FP32's comfortable range, and for
// zero, negative and non-finite values, the plain quotient.
__device__ __forceinline__ double inv_sqrt(double a) {
    if (!(a > 1e-30 && a < 1e30)) return 1. / sqrt(a);
    const double y = (double)rsqrtf((float)a);
    const double r = fma(-a * y, y, 1.);
    return fma(y * r, fma(0.375, r, 0.5), y);
}

// x as a pair of floats (hi + lo, 48 bits) with integer arithmetic: the two conversions and the
// subtraction of df_of are FP64 instructions
__device__ __forceinline__ df df_split(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const uint64_t u = b & 0x7FFFFFFFFFFFFFFFULL;
    const int e = (int)(u >> 52);
    if (u == 0) return {0.f, 0.f};
    if (e < 1023 - 70 || e > 1023 + 126) return df_of(x);  // includes infinities and NaN
    const uint32_t sign = (uint32_t)(b >> 32) & 0x80000000u;
    const uint64_t q = (u + (1ULL << 28)) >> 29;  // exponent and 23 bits, rounded to nearest
    const float hi = __uint_as_float(((uint32_t)q - (896u << 23)) | sign);
    const int rest = (int)((int64_t)u - (int64_t)(q << 29));  // in [-2^28, 2^28), units of 2^(e - 1075)
    const float unit = __uint_as_float((uint32_t)(e - 1075 + 127) << 23 | sign);
    return {hi, (float)rest * unit};
}

__device__ __forceinline__ df dot_df(const DotAcc<float> &a) { return a.get_df(); }
__device__ __forceinline__ df dot_df(const DotAcc<double> &a) { return df_split(a.s); }

// component lists of a reduction: complex values take one component for real vectors, two for
// complex ones; squares one
template <typename V>
constexpr int comps(int values, int squares) { return (VT<V>::kComplex ? 2 : 1) * values + squares; }

template <typename V, typename R>
__device__ __forceinline__ void put(df *c, int &n, const CDot<R> &d) {
    c[n++] = dot_df(d.re);
    if (VT<V>::kComplex) c[n++] = dot_df(d.im);
}

template <typename S>
struct Reader {  // the reduced components in the same order
    const double *p;
    int n = 0;
    __device__ __forceinline__ double real() { return p[n++]; }
    __device__ __forceinline__ S value();
};
template <>
__device__ __forceinline__ double Reader<double>::value() { return p[n++]; }
template <>
__device__ __forceinline__ double2 Reader<double2>::value() {
    n += 2;
    return make_double2(p[n - 2], p[n - 1]);
}

// |v|^2 accumulator
template <typename V>
__device__ __forceinline__ void add_square(DotAcc<typename VT<V>::R> &a, cx<typename VT<V>::R> v) {
    a.prod(v.re, v.re);
    if (VT<V>::kComplex) a.prod(v.im, v.im);
}

// a c + b for complex vectors, the real parts alone for real ones
template <typename V, typename R>
__device__ __forceinline__ cx<R> madd(cx<R> a, cx<R> c, cx<R> b) {
    if (VT<V>::kComplex) return axpy(a, c, b);
    return {a.re * c.re + b.re, (R)0};
}
template <typename V, typename R>
__device__ __forceinline__ cx<R> mulv(cx<R> a, cx<R> c) {
    if (VT<V>::kComplex) return cmul(a, c);
    return {a.re * c.re, (R)0};
}

// ------------------------------------------------------------------------------------------
// the block's rows and lists
// ------------------------------------------------------------------------------------------
struct PersistShared {
    State st;
    double out[kMaxComps];   // the last reduction
    double xx, yy;
    double2 xy;
    double coef[20];         // coefficients of the next pass (R values widened exactly)
    int64_t r0, r1;
    int flip;
    unsigned int passed;
    cdf red[(kPersistThreads / 32) * kPartStride];
    cdf tot[kPartStride];
};

// One problem's lists: states[i] & smask is row i's state, elements [rowptr[i], rowptr[i + 1]).
struct ListOp {
    const int64_t *rowptr;
    const int32_t *col, *grp;
    const void *val;         // cached elements of the vectors' own type (CSR), or null
    const uint64_t *states;
    uint64_t smask;
    const double *diag0;
    rq_terms_t terms;
};

template <typename V, bool CPLX = VT<V>::kComplex>
struct ListVal {
    using T = cx<typename VT<V>::R>;
};
template <typename V>
struct ListVal<V, false> {
    using T = typename VT<V>::R;
};

template <typename V>
__device__ __forceinline__ typename ListVal<V>::T element_value(const ListOp &L, int64_t e, uint64_t s) {
    using R = typename VT<V>::R;
    if (L.val) {
        if constexpr (VT<V>::kComplex) return VT<V>::ld(reinterpret_cast<const V *>(L.val), e);
        else return reinterpret_cast<const V *>(L.val)[e];
    }
    const int g = __ldg(L.grp + e);
    if constexpr (VT<V>::kComplex) return group_diag<R>(L.terms, g, s);
    else return group_diag_re<R>(L.terms, g, s);
}

template <typename V>
struct Lists {
    int *rp;                       // row starts relative to base, or null
    int *col;
    typename ListVal<V>::T *val;
    int64_t base;                  // first element of the block's rows
    int nres;                      // elements [0, nres) are in shared memory
    int lanes;                     // lanes per row
};

extern __shared__ __align__(16) unsigned char persist_dyn[];

// First row of part `lb` of `nb` of rows [p0, p1): parts of equal weight, a row counting for 8 list
// elements (its share of the vector passes).
__device__ inline int64_t part_row(const int64_t *rowptr, int64_t p0, int64_t p1, int lb, int nb) {
    if (lb <= 0) return p0;
    if (lb >= nb) return p1;
    const int64_t e0 = rowptr[p0];
    const int64_t total = rowptr[p1] - e0 + 8 * (p1 - p0);
    const int64_t want = total / nb * lb + total % nb * lb / nb;
    int64_t a = p0, b = p1;
    while (a < b) {
        const int64_t m = (a + b) >> 1;
        if (rowptr[m] - e0 + 8 * (m - p0) < want) a = m + 1;
        else b = m;
    }
    return a;
}

// The block's lists into shared memory, as far as `cap` bytes reach: the row starts (at most a
// half of it), then columns and values.  Rows are found from the source: element e of group g
// with source m belongs to the row of state S[m] ^ x_g.
template <typename V>
__device__ __forceinline__ Lists<V> load_lists(const ListOp &L, int64_t r0, int64_t r1, int cap) {
    using T = typename ListVal<V>::T;
    Lists<V> S;
    const int64_t nrow = r1 - r0;
    S.base = L.rowptr[r0];
    const int64_t ne = L.rowptr[r1] - S.base;
    int used = 0;
    S.rp = nullptr;
    if (4 * (nrow + 1) <= cap / 2 && ne < (int64_t(1) << 31)) {
        S.rp = reinterpret_cast<int *>(persist_dyn);
        used = (int)((4 * (nrow + 1) + 15) & ~int64_t(15));
        for (int64_t k = threadIdx.x; k <= nrow; k += blockDim.x) S.rp[k] = (int)(L.rowptr[r0 + k] - S.base);
    }
    const int64_t fit = (cap - used) / (int)(sizeof(int) + sizeof(T)) & ~3;
    S.nres = (int)(ne < fit ? ne : fit);
    S.val = reinterpret_cast<T *>(persist_dyn + used);
    S.col = reinterpret_cast<int *>(persist_dyn + used + sizeof(T) * ((S.nres + 3) & ~3));
    for (int k = threadIdx.x; k < S.nres; k += blockDim.x) {
        const int64_t e = S.base + k;
        const int m = __ldg(L.col + e);
        S.col[k] = m;
        S.val[k] = element_value<V>(L, e, L.val ? 0ULL : (__ldg(L.states + m) ^ __ldg(L.terms.xmask + __ldg(L.grp + e))) & L.smask);
    }
    // lanes per row: enough that every thread has a row's share, more for long lists
    int lanes = 1;
    while (lanes < 32 && (nrow * lanes < blockDim.x || ne > 16 * nrow * lanes)) lanes <<= 1;
    S.lanes = lanes;
    __syncthreads();
    return S;
}

// accumulator of a product row: FP64 plain, FP32 compensated
template <typename R, bool CPLX>
struct MvAccT {
    Acc<R> re, im;
    __device__ __forceinline__ void mad(R v, cx<R> x) { re.add(v * x.re); }
    __device__ __forceinline__ void mad(cx<R> v, cx<R> x) {
        const cx<R> p = cmul(v, x);
        re.add(p.re);
        im.add(p.im);
    }
};
__device__ __forceinline__ void acc_merge(Acc<double> &a, int o) { a.s += __shfl_xor_sync(0xffffffffu, a.s, o); }
__device__ __forceinline__ void acc_merge(Acc<float> &a, int o) {
    const float s = __shfl_xor_sync(0xffffffffu, a.s, o), c = __shfl_xor_sync(0xffffffffu, a.c, o);
    float t, e;
    two_sum(a.s, s, t, e);
    a.s = t;
    a.c += c + e;
}

// out[k] = H in[k] on the block's rows for NX vectors that share the walk over the lists.  The
// vectors are written by other blocks between barriers, so they are read with plain loads.  All
// threads call it; the caller synchronises the block before other threads read the rows.
template <typename V, int NX>
__device__ __forceinline__ void list_product(const ListOp &L, const Lists<V> &S, int64_t r0, int64_t r1,
                                             const V *const (&in)[NX], V *const (&out)[NX]) {
    using R = typename VT<V>::R;
    using T = typename ListVal<V>::T;
    const int w = S.lanes, lane = threadIdx.x & (w - 1);
    const int64_t step = blockDim.x / w;
    for (int64_t rb = r0; rb < r1; rb += step) {
        const int64_t row = rb + threadIdx.x / w;
        const bool ok = row < r1;
        MvAccT<R, VT<V>::kComplex> acc[NX];
        int64_t e = 0, e1 = 0;
        if (ok) {
            if (S.rp) {
                e = S.rp[row - r0];
                e1 = S.rp[row - r0 + 1];
            } else {
                e = L.rowptr[row] - S.base;
                e1 = L.rowptr[row + 1] - S.base;
            }
        }
        const int nr = (int)min(e1, (int64_t)S.nres);
        int k = (int)min(e, (int64_t)S.nres) + lane;
        for (; k + 3 * w < nr; k += 4 * w) {  // four gathers in flight per vector
            int m[4];
            T v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                m[u] = S.col[k + u * w];
                v[u] = S.val[k + u * w];
            }
#pragma unroll
            for (int q = 0; q < NX; ++q) {
                cx<R> xv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) xv[u] = VT<V>::ld(in[q], m[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[q].mad(v[u], xv[u]);
            }
        }
        for (; k < nr; k += w) {
            const int m = S.col[k];
            const T v = S.val[k];
#pragma unroll
            for (int q = 0; q < NX; ++q) acc[q].mad(v, VT<V>::ld(in[q], m));
        }
        if (e1 > S.nres) {  // the part of the lists that does not fit in shared memory
            const uint64_t s = L.val ? 0ULL : __ldg(L.states + row) & L.smask;
            for (int64_t j = max(e, (int64_t)S.nres) + lane; j < e1; j += w) {
                const int m = __ldg(L.col + S.base + j);
                const T v = element_value<V>(L, S.base + j, s);
#pragma unroll
                for (int q = 0; q < NX; ++q) acc[q].mad(v, VT<V>::ld(in[q], m));
            }
        }
        for (int o = w >> 1; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < NX; ++q) {
                acc_merge(acc[q].re, o);
                if (VT<V>::kComplex) acc_merge(acc[q].im, o);
            }
        if (ok && lane == 0) {
            cx<R> d = {(R)0, (R)0};
            bool with = true;
            if (L.diag0) d.re = (R)L.diag0[row];
            else if (!L.val && L.terms.diag_group >= 0) d = group_diag<R>(L.terms, L.terms.diag_group, __ldg(L.states + row) & L.smask);
            else with = false;
#pragma unroll
            for (int q = 0; q < NX; ++q) {
                if (with) {
                    const cx<R> xi = VT<V>::ld(in[q], row);
                    if (L.diag0 || !VT<V>::kComplex) {
                        acc[q].re.add(d.re * xi.re);
                        if (VT<V>::kComplex) acc[q].im.add(d.re * xi.im);
                    } else {
                        acc[q].mad(d, xi);
                    }
                }
                VT<V>::st(out[q], row, {acc[q].re.get(), VT<V>::kComplex ? acc[q].im.get() : (R)0});
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// the segment of one problem: this block is number lb of nb
// ------------------------------------------------------------------------------------------
struct PSeg {
    PersistShared *sh;
    int64_t r0, r1;
    int lb, nb;
    float4 *part;  // [2][nb * kPartStride]; alternate reductions alternate halves (a block may
                   // write the next sums while another still reads these)
    GridBar *bar;

    __device__ __forceinline__ bool sync() const {
        if (group_sync(bar, &sh->passed, (unsigned int)nb)) return true;
        if (threadIdx.x == 0) sh->st.active = 0;  // aborted: every block stops
        __syncthreads();
        return false;
    }
    // sums of N components over the problem, in sh->out for every thread: the block's partial
    // sums, one barrier, then every block adds all partials itself in the same order, so the
    // blocks' copies of the solver state stay identical without a second barrier
    template <int N>
    __device__ __forceinline__ bool sum(const df (&c)[N]) const {
        constexpr int NV = (N + 1) / 2;
        static_assert(N <= kMaxComps, "too many components");
        cdf w[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) w[k] = {c[2 * k], 2 * k + 1 < N ? c[2 * k + 1 < N ? 2 * k + 1 : 0] : df{0.f, 0.f}};
        block_sum_all<NV>(w, sh->tot, reinterpret_cast<cdf(*)[NV]>(sh->red));
        float4 *pb = part + (size_t)sh->flip * nb * kPartStride;
        if (threadIdx.x < NV) {
            pb[(size_t)lb * kPartStride + threadIdx.x] = cdf_pack(sh->tot[threadIdx.x]);
            __threadfence();
        }
        if (!sync()) return false;
        partials_sum<NV>(pb, nb, kPartStride, sh->tot);
        if (threadIdx.x < N) {
            const cdf t = sh->tot[threadIdx.x >> 1];
            sh->out[threadIdx.x] = df_val((threadIdx.x & 1) ? t.im : t.re);
        }
        if (threadIdx.x == 0) sh->flip ^= 1;
        __syncthreads();
        return true;
    }
};

#define PSEG_LOOP(i) for (int64_t i = seg.r0 + threadIdx.x; i < seg.r1; i += blockDim.x)

// Inner products of the residual pass: <x,r> <y,r> <x,y> |x|^2 |y|^2 |r|^2 |Ax|^2.
template <typename V>
struct ResidDots {
    using R = typename VT<V>::R;
    CDot<R> xr, yr, xy;
    DotAcc<R> xx, yy, rr, aa;
    static constexpr int N = comps<V>(3, 4);
    __device__ __forceinline__ void add(cx<R> x, cx<R> y, cx<R> r, cx<R> ax) {
        constexpr bool c = VT<V>::kComplex;
        xr.add(x, r, c);
        yr.add(y, r, c);
        xy.add(x, y, c);
        add_square<V>(xx, x);
        add_square<V>(yy, y);
        add_square<V>(rr, r);
        add_square<V>(aa, ax);
    }
    __device__ __forceinline__ bool sum(const PSeg &seg) const {
        df c[N];
        int n = 0;
        put<V>(c, n, xr);
        put<V>(c, n, yr);
        put<V>(c, n, xy);
        c[n++] = dot_df(xx);
        c[n++] = dot_df(yy);
        c[n++] = dot_df(rr);
        c[n++] = dot_df(aa);
        return seg.template sum<N>(c);
    }
};

// Scalars after the residual pass, on warps 0 and 1: the convergence test (only with `check`) and,
// FAST, the projection's coefficients (d_proj_coef): p = m r + a0 x + a1 y.
template <typename V, bool FAST>
__device__ __forceinline__ void after_resid(PersistShared *sh, bool check) {
    using R = typename VT<V>::R;
    using S = typename std::conditional<VT<V>::kComplex, double2, double>::type;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0 && check) {
        Reader<S> rd{sh->out};
        rd.value(), rd.value(), rd.value(), rd.real(), rd.real();
        const double rr = rd.real(), aa = rd.real();
        const double q = sqrt(lane == 0 ? rr : aa);  // both roots in one instruction sequence
        const double an = __shfl_sync(0xffffffffu, q, 1);
        if (lane == 0) check_state(&sh->st, q, an, nullptr);
    }
    if (warp == 1) {
        Reader<S> rd{sh->out};
        const S xr = rd.value(), yr = rd.value(), xy = rd.value();
        const double xx = rd.real(), yy = rd.real(), rr = rd.real();
        if (FAST) {
            const S d0 = s_add(s_scale(2., xr), s_scale(-1., s_add(s_scale(xx, xr), s_mul(xy, yr))));
            const S d1 = s_add(s_scale(2., yr), s_scale(-1., s_add(s_mul(s_conj(xy), xr), s_scale(yy, yr))));
            const double n2 = rr - 2. * (s_rdot(d0, xr) + s_rdot(d1, yr)) + s_abs2(d0) * xx + s_abs2(d1) * yy +
                              2. * s_re(s_mul(s_mul(s_conj(d0), d1), xy));
            const double thr = sizeof(R) == 4 ? 1e-5 : 1e-7;
            const double m = (n2 > 0. && n2 > thr * thr * rr) ? inv_sqrt(n2) : 0.;
            if (lane == 0) {
                const double2 a0 = s_pair(s_scale(-m, d0)), a1 = s_pair(s_scale(-m, d1));
                sh->coef[0] = (double)(R)m;
                sh->coef[1] = (double)(R)a0.x;
                sh->coef[2] = (double)(R)a0.y;
                sh->coef[3] = (double)(R)a1.x;
                sh->coef[4] = (double)(R)a1.y;
            }
        }
        if (lane == 0) {
            sh->xx = xx;
            sh->yy = yy;
            sh->xy = s_pair(xy);
        }
    }
    __syncthreads();
}

template <typename V>
struct Coef {
    using R = typename VT<V>::R;
    const double *p;
    __device__ __forceinline__ R r(int k) const { return (R)p[k]; }
    __device__ __forceinline__ cx<R> c(int k) const { return {(R)p[k], VT<V>::kComplex ? (R)p[k + 1] : (R)0}; }
};

// Gram pass and Rayleigh-Ritz: <y,Ax> <p,Ax> <p,Ay> <x,Ax> <y,Ay> <p,Ap> <x,p> <y,p> |p|^2, then the
// coefficients of x' = riu (k0 x + s) and y' = rit (s k0 / |s| - x |s|), s = k1 y + k2 p, as two
// combinations of (x, y, p); their norms follow from the products at hand.  Nothing cancels in them: x, y
// and p are orthonormal to rounding (a zero y or p carries no weight: then ss = 0, and 1 / 0 as with sums
// of squares), so |s|^2 = ss is a sum of squares and |t|^2, |u|^2 are |k0|^2 + ss to rounding, and |k| = 1.
template <typename V, bool FAST>
__device__ __forceinline__ bool gram_step(const PSeg &seg, const Vecs<V> &v) {
    using R = typename VT<V>::R;
    using S = typename std::conditional<VT<V>::kComplex, double2, double>::type;
    constexpr bool c = VT<V>::kComplex;
    PersistShared *sh = seg.sh;
    constexpr int N = comps<V>(8, 1);
    {
        CDot<R> g[8];
        DotAcc<R> pp;
        PSEG_LOOP(i) {
            const cx<R> x = VT<V>::ld(v.x, i), y = VT<V>::ld(v.y, i), p = VT<V>::ld(v.p, i);
            const cx<R> ax = VT<V>::ld(v.ax, i), ay = VT<V>::ld(v.ay, i), ap = VT<V>::ld(v.ap, i);
            g[0].add(y, ax, c);
            g[1].add(p, ax, c);
            g[2].add(p, ay, c);
            g[3].add(x, ax, c);
            g[4].add(y, ay, c);
            g[5].add(p, ap, c);
            g[6].add(x, p, c);
            g[7].add(y, p, c);
            add_square<V>(pp, p);
        }
        df d[N];
        int n = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) put<V>(d, n, g[k]);
        d[n++] = dot_df(pp);
        if (!seg.template sum<N>(d)) return false;
    }
    if (threadIdx.x < 32) {
        State *st = &sh->st;
        Reader<S> rd{sh->out};
        S g[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) g[k] = rd.value();
        const S xp = rd.value(), yp = rd.value();
        const double pp = rd.real();
        double lam;
        S kap[3];
        eig3(g[0], g[1], g[2], g[3], g[4], g[5], lam, kap, st->guard != 0, FAST);
        // the pass combines with the coefficients rounded to its precision: their norms too
        const S k0 = s_round<R>(kap[0]), k1 = s_round<R>(kap[1]), k2 = s_round<R>(kap[2]);
        const double xx = sh->xx, yy = sh->yy;
        S xy;
        if constexpr (c) xy = sh->xy;
        else xy = sh->xy.x;
        double ss = s_abs2(k1) * yy + s_abs2(k2) * pp + 2. * s_re(s_mul(s_mul(s_conj(k1), k2), yp));
        if (ss < 0.) ss = 0.;
        const S xs = s_add(s_mul(k1, xy), s_mul(k2, xp));
        const bool keep_y = st->guard && ss == 0.;  // s = 0: y' = y instead of 0 * inf
        const double tn = keep_y ? yy : s_abs2(k0) + ss * xx - 2. * s_re(s_mul(k0, xs));
        const double un = s_abs2(k0) * xx + ss + 2. * s_rdot(k0, xs);
        const int lane = threadIdx.x;
        const double q = inv_sqrt(lane == 0 ? ss : lane == 1 ? tn : un);
        const double rs = __shfl_sync(0xffffffffu, q, 0), rt = __shfl_sync(0xffffffffu, q, 1),
                     ru = __shfl_sync(0xffffffffu, q, 2);
        const S cs = s_scale(rs * rt, k0);
        // lanes 0..2: the coefficients of x, y, p in x'; lanes 3..5: in y'
        S f = s_scale(ru, lane == 0 ? k0 : lane == 1 ? k1 : k2);
        if (lane >= 3) {
            if (keep_y) f = s_of<S>(lane == 4 ? rt : 0.);
            else f = lane == 3 ? s_of<S>(-(ss * rs) * rt) : s_mul(cs, lane == 4 ? k1 : k2);
        }
        if (lane < 6) {
            const double2 t = s_pair(f);
            sh->coef[2 * lane] = (double)(R)t.x;
            sh->coef[2 * lane + 1] = (double)(R)t.y;
        }
        if (lane == 0) {
            st->theta = lam;
            for (int k = 0; k < 3; ++k) st->kappa[k] = s_pair(kap[k]);
            sh->coef[12] = (double)(R)(-lam);
        }
    }
    __syncthreads();
    return true;
}

template <typename V>
struct Update {  // the two combinations of (a, b, c)
    using R = typename VT<V>::R;
    cx<R> u[3], t[3];
    __device__ __forceinline__ Update(const PersistShared *sh) {
        const Coef<V> cf{sh->coef};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            u[k] = cf.c(2 * k);
            t[k] = cf.c(6 + 2 * k);
        }
    }
    __device__ __forceinline__ void apply(cx<R> a, cx<R> b, cx<R> c, cx<R> &uo, cx<R> &to) const {
        uo = madd<V>(u[0], a, madd<V>(u[1], b, mulv<V>(u[2], c)));
        to = madd<V>(t[0], a, madd<V>(t[1], b, mulv<V>(t[2], c)));
    }
};

// r = Ax - theta x with its inner products (rewrites v.r), then the scalars that follow
template <typename V, bool FAST>
__device__ __forceinline__ bool resid_step(const PSeg &seg, const Vecs<V> &v) {
    using R = typename VT<V>::R;
    const cx<R> mth = {(R)seg.sh->coef[12], (R)0};
    ResidDots<V> d;
    PSEG_LOOP(i) {
        const cx<R> x = VT<V>::ld(v.x, i), ax = VT<V>::ld(v.ax, i);
        const cx<R> r = {mth.re * x.re + ax.re, VT<V>::kComplex ? mth.re * x.im + ax.im : (R)0};
        VT<V>::st(v.r, i, r);
        d.add(x, VT<V>::ld(v.y, i), r, ax);
    }
    if (!d.sum(seg)) return false;
    after_resid<V, FAST>(seg.sh, true);
    return true;
}

// One projection round of REFERENCE: w = f v - x a0 - y a1 (f the scale of the previous round's
// unscaled vector), <x,w> <y,w> |w|^2
template <typename V>
__device__ __forceinline__ bool project_round(const PSeg &seg, const Vecs<V> &v, typename VT<V>::R f,
                                              cx<typename VT<V>::R> a0, cx<typename VT<V>::R> a1, bool dots) {
    using R = typename VT<V>::R;
    CDot<R> xw, yw;
    DotAcc<R> ww;
    const cx<R> m0 = {-a0.re, -a0.im}, m1 = {-a1.re, -a1.im};
    PSEG_LOOP(i) {
        const cx<R> x = VT<V>::ld(v.x, i), y = VT<V>::ld(v.y, i), r = VT<V>::ld(v.r, i);
        const cx<R> w = madd<V>(m1, y, madd<V>(m0, x, {r.re * f, r.im * f}));
        VT<V>::st(v.r, i, w);
        if (dots) {
            xw.add(x, w, VT<V>::kComplex);
            yw.add(y, w, VT<V>::kComplex);
        }
        add_square<V>(ww, w);
    }
    df c[comps<V>(2, 1)];
    int n = 0;
    put<V>(c, n, xw);
    put<V>(c, n, yw);
    c[n++] = dot_df(ww);
    return seg.template sum<comps<V>(2, 1)>(c);
}

// the next round's scale and inner products, from the sums of the last one
template <typename V>
__device__ __forceinline__ void project_coef(PersistShared *sh, bool scale) {
    using R = typename VT<V>::R;
    using S = typename std::conditional<VT<V>::kComplex, double2, double>::type;
    if (threadIdx.x < 32) {
        Reader<S> rd{sh->out};
        const S xw = rd.value(), yw = rd.value();
        const double ww = rd.real();
        const double f = (!scale || ww == 0.) ? 1. : inv_sqrt(ww);
        const double2 a0 = s_pair(s_scale(f, xw)), a1 = s_pair(s_scale(f, yw));
        if (threadIdx.x == 0) {
            sh->coef[0] = (double)(R)f;
            sh->coef[1] = (double)(R)a0.x;
            sh->coef[2] = (double)(R)a0.y;
            sh->coef[3] = (double)(R)a1.x;
            sh->coef[4] = (double)(R)a1.y;
        }
    }
    __syncthreads();
}

// The iterations of one phase (ground_locg.py:288-341) until the problem stops, an abort, or
// iteration `stop`.  On entry v.r = A x - theta x and (REFERENCE) v.ax = A x, as Phase::start and
// every iteration leave them.  Element i is always handled by the same block, so passes over the
// block's own rows need no grid barrier; barriers stand before the products (which gather rows of
// other blocks) and inside every reduction.
template <typename V, bool FAST>
__device__ __forceinline__ void persist_loop(const PSeg &seg, const Vecs<V> &v, const ListOp &L, const Lists<V> &S,
                                             int stop) {
    using R = typename VT<V>::R;
    PersistShared *sh = seg.sh;
    State *st = &sh->st;
    if (!st->active || st->iter >= stop) return;
    {
        ResidDots<V> d;  // the first iteration's inner products
        PSEG_LOOP(i) d.add(VT<V>::ld(v.x, i), VT<V>::ld(v.y, i), VT<V>::ld(v.r, i), {(R)0, (R)0});
        if (!d.sum(seg)) return;
        after_resid<V, FAST>(sh, false);
    }
    const Coef<V> cf{sh->coef};
    while (st->active && st->iter < stop) {
        // project_out((x, y), r) -> p (ground_locg.py:380-421)
        if (FAST) {
            const R m = cf.r(0);
            const cx<R> a0 = cf.c(1), a1 = cf.c(3);
            PSEG_LOOP(i) {
                const cx<R> r = VT<V>::ld(v.r, i);
                VT<V>::st(v.p, i, madd<V>(a1, VT<V>::ld(v.y, i), madd<V>(a0, VT<V>::ld(v.x, i), {r.re * m, r.im * m})));
            }
        } else {
            project_coef<V>(sh, false);  // <x,r>, <y,r> lead the residual's sums
            for (int round = 0; round < 4; ++round) {
                if (!project_round<V>(seg, v, cf.r(0), cf.c(1), cf.c(3), round < 3)) return;
                if (round < 3) project_coef<V>(sh, round < 2);
            }
            if (threadIdx.x == 0) sh->coef[0] = sqrt(sh->out[comps<V>(2, 0)]) >= 0.99 ? 1. : 0.;
            __syncthreads();
            const R m = cf.r(0);
            PSEG_LOOP(i) {
                const cx<R> w = VT<V>::ld(v.r, i);
                VT<V>::st(v.p, i, {w.re * m, w.im * m});
            }
        }
        if (!seg.sync()) return;  // the products gather p (and y) from every block's rows
        if (FAST) {
            const V *const in[1] = {v.p};
            V *const out[1] = {v.ap};
            list_product<V, 1>(L, S, seg.r0, seg.r1, in, out);
        } else {  // A x is still the product of the last iteration's x
            const V *const in[2] = {v.y, v.p};
            V *const out[2] = {v.ay, v.ap};
            list_product<V, 2>(L, S, seg.r0, seg.r1, in, out);
        }
        __syncthreads();  // rows of the product are read by other threads below
        if (!gram_step<V, FAST>(seg, v)) return;
        const Update<V> up(sh);
        if (FAST && !st->want_refresh) {
            const cx<R> mth = {cf.r(12), (R)0};
            ResidDots<V> d;
            PSEG_LOOP(i) {
                cx<R> x, y, ax, ay;
                up.apply(VT<V>::ld(v.x, i), VT<V>::ld(v.y, i), VT<V>::ld(v.p, i), x, y);
                up.apply(VT<V>::ld(v.ax, i), VT<V>::ld(v.ay, i), VT<V>::ld(v.ap, i), ax, ay);
                VT<V>::st(v.x, i, x);
                VT<V>::st(v.y, i, y);
                VT<V>::st(v.ax, i, ax);
                VT<V>::st(v.ay, i, ay);
                const cx<R> r = {mth.re * x.re + ax.re, VT<V>::kComplex ? mth.re * x.im + ax.im : (R)0};
                VT<V>::st(v.r, i, r);
                d.add(x, y, r, ax);
            }
            if (!d.sum(seg)) return;
            after_resid<V, FAST>(sh, true);
            continue;
        }
        PSEG_LOOP(i) {
            cx<R> x, y;
            up.apply(VT<V>::ld(v.x, i), VT<V>::ld(v.y, i), VT<V>::ld(v.p, i), x, y);
            VT<V>::st(v.x, i, x);
            VT<V>::st(v.y, i, y);
        }
        if (!seg.sync()) return;
        if (FAST) {  // refresh: fresh A x and A y instead of the carried ones
            const V *const in[2] = {v.x, v.y};
            V *const out[2] = {v.ax, v.ay};
            list_product<V, 2>(L, S, seg.r0, seg.r1, in, out);
            if (threadIdx.x == 0) {
                st->since_refresh = 0;
                st->matvecs += 2;
            }
        } else {
            const V *const in[1] = {v.x};
            V *const out[1] = {v.ax};
            list_product<V, 1>(L, S, seg.r0, seg.r1, in, out);
        }
        __syncthreads();
        if (!resid_step<V, FAST>(seg, v)) return;
    }
}

// ------------------------------------------------------------------------------------------
// kernels
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void copy_state(State *dst, const State *src) {
    const int n = (int)(sizeof(State) / sizeof(int));
    for (int k = threadIdx.x; k < n; k += blockDim.x)
        reinterpret_cast<int *>(dst)[k] = reinterpret_cast<const int *>(src)[k];
}

template <typename V>
struct PersistArgs {
    State *st;      // global state (read at start, written back by block 0 at the end)
    int64_t D;
    float4 *part;
    ListOp op;
    Vecs<V> v;
    GridBar *bar;
    int cap;        // bytes of dynamic shared memory
};

template <typename V, bool FAST>
__device__ __forceinline__ void persist_problem(PersistShared &sh, State *gst, int64_t p0, int64_t p1, int lb, int nb,
                                                float4 *part, GridBar *bar, const ListOp &op, const Vecs<V> &v,
                                                int cap, int iters) {
    if (threadIdx.x == 0) {
        sh.flip = 0;
        sh.passed = 0u;
    }
    if (threadIdx.x < 2) (threadIdx.x == 0 ? sh.r0 : sh.r1) = part_row(op.rowptr, p0, p1, lb + (int)threadIdx.x, nb);
    copy_state(&sh.st, gst);
    __syncthreads();
    const PSeg seg{&sh, sh.r0, sh.r1, lb, nb, part, bar};
    const Lists<V> lists = load_lists<V>(op, seg.r0, seg.r1, cap);
    const int stop = iters == INT_MAX ? INT_MAX : sh.st.iter + iters;
    persist_loop<V, FAST>(seg, v, op, lists, stop);
    __syncthreads();
    if (lb == 0) copy_state(gst, &sh.st);  // the copies are identical; the first block publishes its own
}

template <typename V, bool FAST>
__global__ void __launch_bounds__(kPersistThreads, 1) k_persist(const PersistArgs<V> a) {
    __shared__ PersistShared sh;
    persist_problem<V, FAST>(sh, a.st, 0, a.D, blockIdx.x, gridDim.x, a.part, a.bar, a.op, a.v, a.cap, INT_MAX);
}

template <typename V>
struct PersistBatchArgs {
    State *states;          // [P], read at start, written back by each problem's first block
    const int64_t *prow;
    ListOp op;
    Vecs<V> v;
    int iter_cap;           // iterations per problem in this launch
    const int32_t *bprob;   // [grid] problem of each block
    const int32_t *bfirst;  // [P] first block of each problem
    const int32_t *nblk;    // [P] blocks of each problem
    const int64_t *poff;    // [P] first float4 of each problem's partial sums
    float4 *part;
    GridBar *bars;          // [P]
    int cap;
};

// Many problems in one cooperative launch: each problem owns a group of blocks and runs
// persist_loop on its own rows with its own reductions and barrier (blocks of different problems
// never wait for each other), at most iter_cap iterations, after which the host re-plans the
// block groups over the problems still active.
template <typename V, bool FAST>
__global__ void __launch_bounds__(kPersistBatchThreads, 2) k_persist_batch(const PersistBatchArgs<V> a) {
    __shared__ PersistShared sh;
    const int q = a.bprob[blockIdx.x];
    persist_problem<V, FAST>(sh, a.states + q, a.prow[q], a.prow[q + 1], blockIdx.x - a.bfirst[q], a.nblk[q],
                             a.part + a.poff[q], a.bars + q, a.op, a.v, a.cap, a.iter_cap);
}
