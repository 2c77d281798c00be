// Pauli-sum matvec restricted to a sorted subspace (rqutils/sqd.py:578-684) and the full-space
// form (rqutils/paulis/symplectic.py:131-150).
//
// Row-side formula: (H x)[i] = sum_j d_j(S[i]) x[m_j(i)],  d_j(s) = sum_k c_jk (-1)^popcount(s & z_jk),
// S[m_j(i)] = S[i] ^ x_j (term dropped when absent).  One thread owns one row; the X masks,
// offsets, Z masks and coefficients of a tile of groups sit in shared memory and every thread of
// the block walks the same group sequence (broadcast reads).  Lookups of four groups are issued
// together (four independent 32-byte bucket loads in flight per thread).  d_j is only evaluated
// on a hit; the x = 0 group's diagonal is either read from a cached FP64 array or computed.
//
// Modes: FREE (lookups every call, cache_level (0, *)), CONN (cached (row -> source, group)
// lists, diagonals recomputed, cache_level (1, 0)), CSR (cached element values, (*, 2)).
#include <algorithm>
#include <cmath>

#include "rq_common.cuh"
#include "rq_rows.cuh"
#include "rq_host.h"
#include "rq_line.cuh"

namespace rq {

// rq_conn.cu: row counts (col null: rows[i] = elements of row i) or the lists at rows[i]
int conn_line(const rq_operator_t &op, int64_t *rows, int32_t *col, int32_t *grp, void *val, int32_t vtype, int *err,
              cudaStream_t st);

namespace {

constexpr int kGT = 512;      // max groups per shared-memory tile
constexpr int kKT = 2048;     // max terms per shared-memory tile
constexpr int kSample = 2048; // shared-memory sample of the binary-search lookup
constexpr int kFilterBytes = 544;

template <typename R>
struct Tile {
    uint64_t *xm;
    uint32_t *hx;  // linear hash of each X mask (hash-lookup kernel only)
    uint2 *gs;     // (low 32 bits of the X mask, its hash): one 8-byte read per group
    int32_t *off;
    uint64_t *zm;
    cx<R> *cf;
};

__host__ __device__ inline size_t align16(size_t b) { return (b + 15) & ~size_t(15); }

template <typename R>
__host__ __device__ inline size_t tile_bytes(int gt, int kt) {
    return align16((size_t)gt * 8) + align16((size_t)gt * 4) + align16((size_t)gt * 8) +
           align16((size_t)(gt + 1) * 4) + align16((size_t)kt * 8) + (size_t)kt * sizeof(cx<R>);
}

template <typename R>
__device__ inline Tile<R> carve(unsigned char *p, int gt, int kt) {
    Tile<R> t;
    t.xm = reinterpret_cast<uint64_t *>(p);
    p += align16((size_t)gt * 8);
    t.hx = reinterpret_cast<uint32_t *>(p);
    p += align16((size_t)gt * 4);
    t.gs = reinterpret_cast<uint2 *>(p);
    p += align16((size_t)gt * 8);
    t.off = reinterpret_cast<int32_t *>(p);
    p += align16((size_t)(gt + 1) * 4);
    t.zm = reinterpret_cast<uint64_t *>(p);
    p += align16((size_t)kt * 8);
    t.cf = reinterpret_cast<cx<R> *>(p);
    return t;
}

// Stage groups [g0, g1) into shared memory, g1 as large as the tile allows.  Returns g1, or -1
// when group g0 alone exceeds the tile.  Every thread of the block must call it.  With a hash
// table T the linear hash of each X mask is stored too.
template <typename R>
__device__ int load_tile(const rq_terms_t &T, int g0, int gt, int kt, const Tile<R> &tl,
                         int *s_g1, const uint32_t *htab = nullptr, int nbytes = 8) {
    __syncthreads();  // previous tile no longer in use; tables written before are visible
    if (threadIdx.x == 0) *s_g1 = g0;
    __syncthreads();
    const int base = T.toff[g0];
    const int gmax = min(T.J, g0 + gt);
    for (int g = g0 + 1 + threadIdx.x; g <= gmax; g += blockDim.x)
        if (T.toff[g] - base <= kt) atomicMax(s_g1, g);
    __syncthreads();
    const int g1 = *s_g1;
    if (g1 == g0) return -1;
    const int ng = g1 - g0;
    const int nk = T.toff[g1] - base;
    for (int g = threadIdx.x; g < ng; g += blockDim.x) {
        const uint64_t xv = T.xmask[g0 + g];
        tl.xm[g] = xv;
        if (htab) {
            const uint32_t h = lin_hash(htab, xv, nbytes);
            tl.hx[g] = h;
            tl.gs[g] = make_uint2((uint32_t)xv, h);
        }
    }
    for (int g = threadIdx.x; g <= ng; g += blockDim.x) tl.off[g] = T.toff[g0 + g] - base;
    for (int k = threadIdx.x; k < nk; k += blockDim.x) {
        tl.zm[k] = T.zmask[base + k];
        tl.cf[k] = {(R)T.coef[2 * (base + k)], (R)T.coef[2 * (base + k) + 1]};
    }
    __syncthreads();
    return g1;
}

// d_j(s) * xv accumulated into acc; the group's terms end at the first zero coefficient when
// stop_at_zero (subspace form) and run to the end otherwise (full-space form).
template <typename R>
__device__ __forceinline__ void add_group(const cx<R> *cf, const uint64_t *zm, int k0, int k1,
                                          uint64_t s, cx<R> xv, bool stop_at_zero, CAcc<R> &acc) {
    CAcc<R> d;
    for (int k = k0; k < k1; ++k) {
        const cx<R> c = cf[k];
        if (stop_at_zero && c.re == (R)0 && c.im == (R)0) break;
        if (__popcll(s & zm[k]) & 1) d.add({-c.re, -c.im});
        else d.add(c);
    }
    acc.add(cmul(d.get(), xv));
}

// Visit the hits of row state s over groups [g0, g1) (xm indexed by g - g0), skipping `skip`,
// calling on_hit(g, m) in ascending g.  Hash lookups hash each target in full (T: tables).
template <int LK, int KB, typename F>
__device__ __forceinline__ void for_hits(const rq_subspace_t &S, const uint32_t *fb,
                                         const uint64_t *samp, int ns, const uint32_t *T,
                                         const uint64_t *xm, int g0, int g1, int skip, uint64_t s,
                                         int *err, F &&on_hit) {
    for (int g = g0; g < g1; ++g) {
        if (g == skip) continue;
        const uint64_t t = s ^ xm[g - g0];
        int64_t m;
        if (LK == RQ_LOOKUP_IDENTITY) {
            m = (t < (uint64_t)S.D) ? (int64_t)t : -1;
        } else {
            if (!sector_ok(fb, S.fmask_a, S.fmask_b, t)) continue;
            if (LK == RQ_LOOKUP_HASH) {
                if (KB == 32 && (t >> 32) != 0) continue;
                const uint32_t h = lin_hash(T, t, KeyWidth<KB>::kNbytes);
                if (S.pbits > 0 && S.pmap && !present(S.pmap, h, S.pbits)) continue;
                m = lookup_hash_at<KB>(S, t, bucket_from_hash(h, S.hbits), err);
            } else {
                m = lookup_bsearch(S, samp, ns, t);
            }
        }
        if (m >= 0) on_hit(g, m);
    }
}

template <int LK>
__device__ inline void load_lookup_smem(const rq_subspace_t &S, uint32_t *fb, uint64_t *samp,
                                        int ns) {
    if (LK != RQ_LOOKUP_IDENTITY)
        for (int w = threadIdx.x; w < RQ_FILTER_WORDS; w += blockDim.x) fb[w] = S.fbits[w];
    if (LK == RQ_LOOKUP_BSEARCH)
        for (int k = threadIdx.x; k < ns; k += blockDim.x)
            samp[k] = S.states[((int64_t)k * S.D) / ns];
}

// ------------------------------------------------------------------------------------------
// FREE mode with the hash table: the hot kernels
// ------------------------------------------------------------------------------------------
// h(s) once per row; per X group t = s ^ x_j, bucket (h(s) ^ h(x_j)) >> shift.  A probe asks whether t
// can be a state; the few groups that can ("hot") are resolved in the table afterwards, so that the
// rare divergent work is not interleaved with the probes.
//
// k_matvec_line (a line filter is present, rq_line.cuh): the probe is a two-bit test in a line chosen by the
// target's prefix t >> lshift.  The rows of a warp are consecutive sorted states that share their
// high bits, so for one X group their targets share them too and the warp's probes fall in a few
// lines.
// k_matvec_hash (no line filter): the probe is the key bucket itself, behind the sector filter and
// the presence bitmap.

template <typename V>
struct UseProduct {  // y = H x
    using RT = RowTerm<V>;
    using R = typename VT<V>::R;
    const rq_operator_t &op;
    const V *x;
    V *y;
    typename RT::A acc;
    __device__ __forceinline__ void start(int64_t i, uint64_t s, bool own) {
        acc = typename RT::A();
        if (!own) return;
        const int skip = op.terms.diag_group;
        if (op.diag0 && skip >= 0) RT::add(acc, RT::scaled((R)op.diag0[i], x, i));
        else if (skip >= 0) RT::add(acc, RT::product(op.terms, skip, s, x, i));
    }
    __device__ __forceinline__ void hit(int g, uint64_t s, int m) { RT::add(acc, RT::product(op.terms, g, s, x, m)); }
    __device__ __forceinline__ bool resolve(WarpWork<V> &W, int q, int g, uint64_t s, int m) {
        if (group_terms(op.terms, g) > kShortTerms) return true;
        W.prod[q] = RT::product(op.terms, g, s, x, m);
        return false;
    }
    __device__ __forceinline__ void late(WarpWork<V> &W, int q, int g, uint64_t s) {
        W.prod[q] = RT::product(op.terms, g, s, x, W.src[q]);
    }
    __device__ __forceinline__ void take(const WarpWork<V> &W, int q, int) { RT::add(acc, W.prod[q]); }
    __device__ __forceinline__ void finish(int64_t i) { RT::store(y, i, acc); }
};

template <typename V, int KB, int FM, int BLOCK, bool QUEUE>
__global__ void __launch_bounds__(BLOCK, BLOCK == 1024 ? 1 : QUEUE ? 4 : 6)
k_matvec_line(const rq_operator_t op, const V *__restrict__ x, V *__restrict__ y, int *err, int lw, int kt,
              int spread, const int *gate, const int *gate2) {
    if (gate && (*gate == 0 || (gate2 && *gate2 == 0))) return;
    UseProduct<V> use{op, x, y, {}};
    line_subspace<V, KB, FM, BLOCK, QUEUE>(op, err, lw, kt, spread, use);
}

// ---- probes of the key buckets ----------------------------------------------------------------
// Group keys live in shared memory for the whole launch: (x_j, h(x_j)) packed as uint2 for 32-bit
// keys or as uint64 + uint32 arrays for 64-bit keys (8 or 12 B per group), without the x = 0 group.
// Large J runs one 1024-thread block per SM so that up to max_resident_groups fit; above that the
// keys are streamed through in tiles.
template <int KB>
__host__ __device__ constexpr int max_resident_groups() {
    return KB == 32 ? 24576 : 16384;  // 192 KB of shared memory either way
}

template <int KB>
__host__ __device__ inline size_t group_key_bytes(int J) {
    return align16((size_t)J * 8) + (KB == 32 ? 0 : align16((size_t)J * 4));
}

// Group keys of resident indices [c0, c0 + cn) into shared-memory slots [0, cn); the layout holds
// kt slots.  All threads of the block call it.
template <int KB>
__device__ __forceinline__ void load_group_keys(const rq_terms_t &T, int c0, int cn, int kt) {
    constexpr int NB = KeyWidth<KB>::kNbytes;
    const int skip = T.diag_group;
    for (int c = threadIdx.x; c < cn; c += blockDim.x) {
        const int j = c0 + c + (skip >= 0 && c0 + c >= skip);
        const uint64_t xv = T.xmask[j];
        const uint32_t h = T.xhash ? T.xhash[j] : lin_hash(hk_htab, xv, NB);
        if (KB == 32) {
            reinterpret_cast<uint2 *>(hk_dyn)[c] = make_uint2((uint32_t)xv, h);
        } else {
            reinterpret_cast<uint64_t *>(hk_dyn)[c] = xv;
            reinterpret_cast<uint32_t *>(hk_dyn + align16((size_t)kt * 8))[c] = h;
        }
    }
}

// TL: the group keys may need streaming in tiles (1024-thread kernels only; with 256-thread blocks
// they always fit and the tile loop is one pass known at compile time).  FM: the sector filter's
// form, chosen on the host from rq_subspace_t.fpoint.
template <typename V, int KB, int FM, int BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK == 1024 ? 1 : (sizeof(V) <= 8 ? 6 : 4))
k_matvec_hash(const rq_operator_t op, const V *__restrict__ x, V *__restrict__ y, int *err,
              const int *gate, const int *gate2) {
    using R = typename VT<V>::R;
    using RT = RowTerm<V>;
    using K = typename KeyWidth<KB>::K;
    constexpr bool TL = BLOCK == 1024;
    constexpr int NB = KeyWidth<KB>::kNbytes;
    constexpr int kBucketBytes = KeyWidth<KB>::kBucketBytes;
    constexpr int U = 4;  // buckets in flight: 16 or 32 bytes each fill the registers of six blocks
    if (gate && (*gate == 0 || (gate2 && *gate2 == 0))) return;
    const rq_subspace_t &S = op.sub;
    const rq_terms_t &T = op.terms;
    const int64_t D = S.D;
    const int skip = T.diag_group;  // the x = 0 group is applied outside the probe loop
    const int nres = T.J - (skip >= 0 ? 1 : 0);  // groups of the probe loop
    copy_hash_tables(hk_htab, NB);
    if (FM == kFiltSet)
        for (int w = threadIdx.x; w < RQ_FILTER_WORDS; w += blockDim.x) hk_fb[w] = S.fbits[w];
    __syncthreads();
    constexpr int kMaxRes = max_resident_groups<KB>();
    const int kt = (!TL || nres <= kMaxRes) ? nres : kMaxRes;
    const bool tiled = TL && nres > kt;
    if (!tiled) load_group_keys<KB>(T, 0, nres, nres);
    __syncthreads();
    const uint2 *gk32 = reinterpret_cast<const uint2 *>(hk_dyn);
    const uint64_t *gx64 = reinterpret_cast<const uint64_t *>(hk_dyn);
    const uint32_t *gh64 = reinterpret_cast<const uint32_t *>(hk_dyn + align16((size_t)kt * 8));
    const int pa0 = S.fpoint / 65, pb0 = S.fpoint % 65;
    const K fa = (K)S.fmask_a, fbm = (K)S.fmask_b, empty = (K)S.empty_key;
    const int shift = 32 - S.hbits;
    const uint32_t *pmap = S.pbits > 0 ? S.pmap : nullptr;
    const int pshift = 32 - S.pbits;
    const unsigned char *keys = static_cast<const unsigned char *>(S.hkeys);
    // Every lane runs the same row batches and super-chunks, so that the warp can be
    // re-converged after each super-chunk's hot-group resolution; without the explicit
    // __syncwarp the lanes that took the rare path stay split from the rest for the remainder of
    // the row.  Lanes past D probe the last row again and store nothing.
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < D;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = base + threadIdx.x;
        const bool active = i < D;
        const int64_t ir = active ? i : D - 1;
        const uint64_t s64 = __ldg(S.states + ir);
        const K s = (K)s64;
        const uint32_t hs = lin_hash(hk_htab, s64, NB);
        typename RT::A acc;
        if (op.diag0 && skip >= 0) RT::add(acc, RT::scaled((R)op.diag0[ir], x, ir));
        else if (skip >= 0) RT::add(acc, RT::product(T, skip, s64, x, ir));
        for (int t0 = 0; TL ? t0 < nres : t0 < 1; t0 += TL ? kt : 1) {
            const int tn = TL ? min(kt, nres - t0) : nres;
            if (tiled) {
                __syncthreads();  // the previous tile is no longer read
                load_group_keys<KB>(T, t0, tn, kt);
                __syncthreads();
            }
            for (int gs0 = 0; gs0 < tn; gs0 += 64) {
                const int gs1 = min(tn, gs0 + 64);
                uint64_t hot = 0ULL;
                int g = gs0;
                for (; g + U <= gs1; g += U) {
                    K t[U];
                    uint32_t b[U];
                    bool q[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        uint32_t hxg;
                        if (KB == 32) {
                            const uint2 e = gk32[g + u];
                            t[u] = s ^ (K)e.x;
                            hxg = e.y;
                        } else {
                            t[u] = s ^ (K)gx64[g + u];
                            hxg = gh64[g + u];
                        }
                        q[u] = sector_pass<K, FM>(t[u], fa, fbm, pa0, pb0);
                        b[u] = hs ^ hxg;
                    }
                    if (pmap) {  // presence bitmap (L2-resident) in front of a table that is not
                        uint32_t pw[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const uint32_t idx = b[u] >> pshift;
                            pw[u] = q[u] ? __ldg(pmap + (idx >> 5)) : 0u;
                        }
#pragma unroll
                        for (int u = 0; u < U; ++u) q[u] = q[u] && ((pw[u] >> ((b[u] >> pshift) & 31)) & 1u);
                    }
                    uint32_t hb = 0u;  // hot bits of this batch, constant shifts
                    typename KeyWidth<KB>::Bucket w[U];
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        w[u] = KeyWidth<KB>::load(keys + (size_t)(b[u] >> shift) * kBucketBytes,
                                                  q[u], S.empty_key);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        bool any, open;
                        test_bucket(w[u], t[u], empty, any, open);
                        if (q[u] && (any || !open)) hb |= 1u << u;
                    }
                    hot |= (uint64_t)hb << (g - gs0);
                }
                for (; g < gs1; ++g) {  // tail: mark and resolve below
                    const K t = s ^ (KB == 32 ? (K)gk32[g].x : (K)gx64[g]);
                    if (sector_pass<K, FM>(t, fa, fbm, pa0, pb0)) hot |= 1ULL << (g - gs0);
                }
                while (hot) {
                    const int gc = gs0 + __ffsll((long long)hot) - 1;  // slot in shared memory
                    hot &= hot - 1ULL;
                    const int gr = t0 + gc;                             // index among the groups
                    const int gg = gr + (skip >= 0 && gr >= skip);
                    const uint64_t xv = __ldg(T.xmask + gg);
                    const uint32_t hxg = KB == 32 ? gk32[gc].y : gh64[gc];
                    const int m = lookup_hash_at<KB>(S, s64 ^ xv, (hs ^ hxg) >> shift, err);
                    if (m >= 0) RT::add(acc, RT::product(T, gg, s64, x, m));
                }
                __syncwarp();
            }
        }
        if (active) RT::store(y, i, acc);
    }
}

// xhash[j] = h(xmask[j])
template <int KB>
__global__ void k_terms_hash(const uint64_t *__restrict__ xmask, int J, uint32_t *__restrict__ out) {
    __shared__ __align__(16) uint32_t htab[KeyWidth<KB>::kNbytes * 256];
    copy_hash_tables(htab, KeyWidth<KB>::kNbytes);
    __syncthreads();
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < J; j += gridDim.x * blockDim.x)
        out[j] = lin_hash(htab, xmask[j], KeyWidth<KB>::kNbytes);
}

// ------------------------------------------------------------------------------------------
// FREE mode, generic lookups (sampled binary search; identity for the full space)
// ------------------------------------------------------------------------------------------
template <typename V, int LK>
__global__ void __launch_bounds__(kThreads)
k_matvec_free(const rq_operator_t op, const V *__restrict__ x, V *__restrict__ y, int gt, int kt,
              int stop_at_zero, int *err, const int *gate, const int *gate2) {
    using R = typename VT<V>::R;
    if (gate && (*gate == 0 || (gate2 && *gate2 == 0))) return;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_g1;
    const rq_subspace_t &S = op.sub;
    const rq_terms_t &T = op.terms;
    uint32_t *fb = reinterpret_cast<uint32_t *>(smem);
    uint64_t *samp = reinterpret_cast<uint64_t *>(smem + kFilterBytes);
    const int ns = (LK == RQ_LOOKUP_BSEARCH) ? (int)(S.D < kSample ? S.D : kSample) : 0;
    const Tile<R> tl =
        carve<R>(smem + kFilterBytes + (LK == RQ_LOOKUP_BSEARCH ? kSample * 8 : 0), gt, kt);
    load_lookup_smem<LK>(S, fb, samp, ns);

    const int64_t D = S.D;
    const bool d0 = (op.diag0 != nullptr) && (T.diag_group >= 0);
    const int gstart = (d0 && T.diag_group == 0) ? 1 : 0;
    const int skip = T.diag_group;  // handled outside the hit loop
    int g1_first = (gstart < T.J) ? load_tile<R>(T, gstart, gt, kt, tl, &s_g1) : T.J;
    if (g1_first < 0) {
        if (err && threadIdx.x == 0) atomicExch(err, RQ_E_RANGE);
        return;
    }
    __syncthreads();
    const bool resident = (g1_first >= T.J);
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < D;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = base + threadIdx.x;
        const bool active = i < D;
        const uint64_t s =
            active ? (LK == RQ_LOOKUP_IDENTITY ? (uint64_t)i : __ldg(S.states + i)) : 0ULL;
        CAcc<R> acc;
        if (active && d0) {
            const R dv = (R)op.diag0[i];
            const cx<R> xv = VT<V>::ld(x, i);
            acc.add({dv * xv.re, dv * xv.im});
        }
        if (!resident && base != (int64_t)blockIdx.x * blockDim.x)
            g1_first = load_tile<R>(T, gstart, gt, kt, tl, &s_g1);
        int g0 = gstart, g1 = g1_first;
        while (g0 < T.J) {
            if (g1 < 0) {
                if (err && threadIdx.x == 0) atomicExch(err, RQ_E_RANGE);
                return;  // uniform across the block
            }
            if (active) {
                if (!d0 && skip >= g0 && skip < g1)
                    add_group<R>(tl.cf, tl.zm, tl.off[skip - g0], tl.off[skip - g0 + 1], s,
                                 VT<V>::ld(x, i), stop_at_zero, acc);
                for_hits<LK, 64>(S, fb, samp, ns, nullptr, tl.xm, g0, g1, skip, s, err,
                                 [&](int g, int64_t m) {
                                     add_group<R>(tl.cf, tl.zm, tl.off[g - g0], tl.off[g - g0 + 1],
                                                  s, VT<V>::ld(x, m), stop_at_zero, acc);
                                 });
            }
            if (g1 >= T.J) break;
            g0 = g1;
            g1 = load_tile<R>(T, g0, gt, kt, tl, &s_g1);
        }
        if (active) VT<V>::st(y, i, acc.get());
    }
}

// ------------------------------------------------------------------------------------------
// connectivity cache
// ------------------------------------------------------------------------------------------
template <int LK, int KB>
__global__ void __launch_bounds__(kThreads)
k_conn_count(const rq_operator_t op, int64_t *__restrict__ rowcnt, int *err) {
    __shared__ uint32_t fb[RQ_FILTER_WORDS];
    __shared__ uint64_t samp[LK == RQ_LOOKUP_BSEARCH ? kSample : 1];
    __shared__ __align__(16) uint32_t T[LK == RQ_LOOKUP_HASH ? kHashTableWords : 4];
    const rq_subspace_t &S = op.sub;
    const int ns = (LK == RQ_LOOKUP_BSEARCH) ? (int)(S.D < kSample ? S.D : kSample) : 0;
    load_lookup_smem<LK>(S, fb, samp, ns);
    if (LK == RQ_LOOKUP_HASH) copy_hash_tables(T, KeyWidth<KB>::kNbytes);
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < S.D;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t c = 0;
        for_hits<LK, KB>(S, fb, samp, ns, T, op.terms.xmask, 0, op.terms.J, op.terms.diag_group,
                         __ldg(S.states + i), err, [&](int, int64_t) { ++c; });
        rowcnt[i] = c;
    }
}

template <typename V, int LK, int KB>
__global__ void __launch_bounds__(kThreads)
k_conn_fill(const rq_operator_t op, const int64_t *__restrict__ rowptr, int32_t *__restrict__ col,
            int32_t *__restrict__ grp, V *__restrict__ val, int *err) {
    using R = typename VT<V>::R;
    __shared__ uint32_t fb[RQ_FILTER_WORDS];
    __shared__ uint64_t samp[LK == RQ_LOOKUP_BSEARCH ? kSample : 1];
    __shared__ __align__(16) uint32_t T[LK == RQ_LOOKUP_HASH ? kHashTableWords : 4];
    const rq_subspace_t &S = op.sub;
    const int ns = (LK == RQ_LOOKUP_BSEARCH) ? (int)(S.D < kSample ? S.D : kSample) : 0;
    load_lookup_smem<LK>(S, fb, samp, ns);
    if (LK == RQ_LOOKUP_HASH) copy_hash_tables(T, KeyWidth<KB>::kNbytes);
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < S.D;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t p = rowptr[i];
        const uint64_t s = __ldg(S.states + i);
        for_hits<LK, KB>(S, fb, samp, ns, T, op.terms.xmask, 0, op.terms.J, op.terms.diag_group, s, err,
                     [&](int g, int64_t m) {
                         col[p] = (int32_t)m;
                         if (grp) grp[p] = g;
                         if (val) VT<V>::st(val, p, group_diag<R>(op.terms, g, s));
                         ++p;
                     });
    }
}

// Inclusive scan of rowptr[1..D] in place (three phases: block scans, scan of block totals,
// add block offsets).  Block b covers rows [b * 1024, (b + 1) * 1024).
__global__ void __launch_bounds__(kThreads) k_scan_blocks(int64_t *v, int64_t n, int64_t *bsum) {
    __shared__ int64_t ws[kThreads / 32];
    const int64_t base = (int64_t)blockIdx.x * 1024;
    int64_t loc[4];
    int64_t t = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int64_t idx = base + threadIdx.x * 4 + k;
        loc[k] = (idx < n) ? v[idx] : 0;
        t += loc[k];
    }
    // exclusive scan of per-thread totals across the block
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int64_t w = (lane < kThreads / 32) ? ws[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        if (lane < kThreads / 32) ws[lane] = w;
    }
    __syncthreads();
    int64_t run = inc - t + (warp > 0 ? ws[warp - 1] : 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int64_t idx = base + threadIdx.x * 4 + k;
        run += loc[k];
        if (idx < n) v[idx] = run;
    }
    if (threadIdx.x == kThreads - 1) bsum[blockIdx.x] = run;
}

__global__ void k_scan_totals(int64_t *bsum, int64_t nb) {
    // one block: sequential chunks per thread, then a block scan of chunk totals
    __shared__ int64_t tot[kThreads];
    const int64_t per = (nb + blockDim.x - 1) / blockDim.x;
    const int64_t a = threadIdx.x * per, b = min(nb, a + per);
    int64_t s = 0;
    for (int64_t k = a; k < b; ++k) s += bsum[k];
    tot[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t r = 0;
        for (int k = 0; k < (int)blockDim.x; ++k) {
            const int64_t u = tot[k];
            tot[k] = r;
            r += u;
        }
    }
    __syncthreads();
    int64_t r = tot[threadIdx.x];
    for (int64_t k = a; k < b; ++k) {  // exclusive offsets of blocks
        const int64_t u = bsum[k];
        bsum[k] = r;
        r += u;
    }
}

__global__ void k_scan_add(int64_t *v, int64_t n, const int64_t *boff) {
    const int64_t base = (int64_t)blockIdx.x * 1024;
    const int64_t off = boff[blockIdx.x];
    for (int k = threadIdx.x; k < 1024; k += blockDim.x) {
        const int64_t idx = base + k;
        if (idx < n) v[idx] += off;
    }
}

int grid_rows(int64_t n) {
    int64_t g = (n + kThreads - 1) / kThreads;
    const int64_t cap = (int64_t)sm_count() * 8;
    return (int)(g > cap ? cap : (g < 1 ? 1 : g));
}

// Blocks of the tiled cached products: one per tile, so that a block that ends makes room for the next
// (with as many as are resident, each walking several tiles, the chip waited for the longest walk:
// 36 qubits, 150,001 rows, CONN 731 against 570 us in float64, 1616 against 1297 in complex128).
int grid_tiles(int64_t D, int rows) { return (int)std::min<int64_t>((D + rows - 1) / rows, 0x7FFFFFFF); }

// ------------------------------------------------------------------------------------------
// CONN and CSR modes
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float shfl_product(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ CsrTerm<float>::P shfl_product(CsrTerm<float>::P v, int src) {
    return {__shfl_sync(0xffffffffu, v.p, src), __shfl_sync(0xffffffffu, v.low, src)};
}
__device__ __forceinline__ RowTerm<double>::P shfl_product(RowTerm<double>::P v, int src) {
    return {__shfl_sync(0xffffffffu, v.d, src), __shfl_sync(0xffffffffu, v.x, src)};
}
template <typename R>
__device__ __forceinline__ cx<R> shfl_product(cx<R> v, int src) {
    return {__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
}

// Rows shorter than one element on average: a warp takes 32 kShortRows rows, whose elements are
// consecutive in the list, forms up to 32 products at once (the FP64 pipe takes 64 cycles for a
// warp's instruction, however few lanes have an element) and hands them to the rows by shuffles, in
// list order.  No barriers, and twice the loads in flight.  2^20 rows of 0.2 (Hubbard 4x4), CSR, against
// a thread per row: float64 10.4 us against 14.4, complex64 8.3 against 10.4, complex128 18.5 against
// 32.8 (one row a lane: 11.5, 8.9, 22.6; four: 10.8, 8.4, 19.7); CONN, against tiles: float64 14.5
// against 16.7, complex64 13.7 against 16.7, but complex128 28.7 against 26.9: that one keeps them.
// elem, first and done as of tile_product.
constexpr int kShortRows = 2;
template <typename RT, typename E, typename F, typename S>
__device__ __forceinline__ void short_rows(const int64_t *rowptr, int64_t D, E &&elem, F &&first, S &&done) {
    constexpr int kR = kShortRows;
    const int lane = threadIdx.x & 31;
    const int64_t b = (blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 * kR);
    if (b >= D) return;
    int64_t e[kR], e1[kR];
    typename RT::A acc[kR];
#pragma unroll
    for (int k = 0; k < kR; ++k) {
        const int64_t i = b + 32 * k + lane;
        e[k] = rowptr[i < D ? i : D];
        e1[k] = rowptr[i < D ? i + 1 : D];
        if (i < D) first(i, acc[k]);
    }
    const int64_t w0 = __shfl_sync(0xffffffffu, e[0], 0), w1 = __shfl_sync(0xffffffffu, e1[kR - 1], 31);
    for (int64_t c = w0; c < w1; c += 32) {
        typename RT::P p{};
        if (c + lane < w1) p = elem(c + lane);
#pragma unroll
        for (int k = 0; k < kR; ++k) {
            const int64_t stop = e1[k] < c + 32 ? e1[k] : c + 32;
            while (__any_sync(0xffffffffu, e[k] < stop)) {
                const typename RT::P q = shfl_product(p, (int)(e[k] - c) & 31);
                if (e[k] < stop) {
                    RT::add(acc[k], q);
                    ++e[k];
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kR; ++k) {
        const int64_t i = b + 32 * k + lane;
        if (i < D) done(i, acc[k]);
    }
}
inline bool rows_short(int64_t D, int64_t nnz) { return nnz < D; }
inline unsigned grid_short(int64_t D) {
    constexpr int kRows = kThreads * kShortRows;
    return (unsigned)((D + kRows - 1) / kRows);
}

// Element e of group g with source row m belongs to the row of state S[m] ^ x_g, so an element
// needs no search for its row.  SHORT: rows shorter than one element.
template <typename V, bool SHORT>
__global__ void __launch_bounds__(kThreads)
k_matvec_conn(const rq_operator_t op, const V *__restrict__ x, V *__restrict__ y, int rows, const int *gate,
              const int *gate2) {
    using RT = RowTerm<V>;
    using R = typename VT<V>::R;
    if (gate && (*gate == 0 || (gate2 && *gate2 == 0))) return;
    const rq_terms_t &T = op.terms;
    const int64_t D = op.sub.D;
    auto elem = [&](int64_t e) {
        const int m = __ldg(op.col + e), g = __ldg(op.grp + e);
        return RT::product(T, g, __ldg(op.sub.states + m) ^ __ldg(T.xmask + g), x, m);
    };
    auto first = [&](int64_t i, typename RT::A &acc) {
        if (op.diag0) RT::add(acc, RT::scaled((R)op.diag0[i], x, i));
        else if (T.diag_group >= 0) RT::add(acc, RT::product(T, T.diag_group, __ldg(op.sub.states + i), x, i));
    };
    auto done = [&](int64_t i, const typename RT::A &acc) { RT::store(y, i, acc); };
    if constexpr (SHORT)
        short_rows<RT>(op.rowptr, D, elem, first, done);
    else
        for (int64_t r0 = (int64_t)blockIdx.x * rows; r0 < D; r0 += (int64_t)gridDim.x * rows)
            tile_product<V, RT>(
                op.rowptr, r0, (int)min((int64_t)rows, D - r0), long_groups(T), elem,
                [&](int64_t e) { return group_terms(T, __ldg(op.grp + e)); }, first, done);
}

// VV: storage type of the element values (converted to the vector's precision on load)
template <typename V, typename VV, bool SHORT>
__global__ void __launch_bounds__(kThreads)
k_matvec_csr(const rq_operator_t op, const V *__restrict__ x, V *__restrict__ y, int rows, const int *gate,
             const int *gate2) {
    using RT = CsrTerm<V>;
    using R = typename VT<V>::R;
    if (gate && (*gate == 0 || (gate2 && *gate2 == 0))) return;
    const VV *val = reinterpret_cast<const VV *>(op.val);
    const int64_t D = op.sub.D;
    auto elem = [&](int64_t e) {
        const auto v = VT<VV>::ld(val, e);
        return RT::times(cx<R>{(R)v.re, (R)v.im}, x, __ldg(op.col + e));
    };
    auto first = [&](int64_t i, typename RT::A &acc) {
        if (op.diag0) RT::add(acc, RT::scaled((R)op.diag0[i], x, i));
    };
    auto done = [&](int64_t i, const typename RT::A &acc) { RT::store(y, i, acc); };
    if constexpr (SHORT)
        short_rows<RT>(op.rowptr, D, elem, first, done);
    else
        for (int64_t r0 = (int64_t)blockIdx.x * rows; r0 < D; r0 += (int64_t)gridDim.x * rows)
            tile_product<V, RT>(op.rowptr, r0, (int)min((int64_t)rows, D - r0), false, elem, [](int64_t) { return 0; }, first,
                            done);
}

// A thread per row, for 64-bit rows that are many: a row's owner adds them one by one either way, and with
// full warps of owners the FP64 pipe does more a cycle than in tiles.  float64: 400,000 rows of 4 elements
// 15.2 us against 18.2 with tiles (28.6 with each product rounded before its addition), 700,000 rows of 7
// 40 against 42; 20,000 rows of 34 44 against 26.  complex128, long rows only, whose tiles are low:
// 150,001 of 83 750 us against 805 with tiles, 352,000 of 39 in a dense subspace 236 against 274 (150,000 of
// 40 that differ 282 against 213).
constexpr int64_t kCsrRowsD = int64_t(1) << 15;
template <typename V, typename VV>
__global__ void __launch_bounds__(kThreads)
k_matvec_csr_rows(const rq_operator_t op, const V *__restrict__ x, V *__restrict__ y, const int *gate,
                  const int *gate2) {
    using RT = CsrTerm<V>;
    using R = typename VT<V>::R;
    if (gate && (*gate == 0 || (gate2 && *gate2 == 0))) return;
    const VV *val = reinterpret_cast<const VV *>(op.val);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < op.sub.D;
         i += (int64_t)gridDim.x * blockDim.x) {
        typename RT::A acc;
        if (op.diag0) RT::add(acc, RT::scaled((R)op.diag0[i], x, i));
        const int64_t e1 = op.rowptr[i + 1];
        for (int64_t e = op.rowptr[i]; e < e1; ++e) {
            const auto v = VT<VV>::ld(val, e);
            RT::add(acc, RT::times(cx<R>{(R)v.re, (R)v.im}, x, __ldg(op.col + e)));
        }
        RT::store(y, i, acc);
    }
}

template <typename V, typename VV>
void run_csr(const rq_operator_t &op, const V *x, V *y, cudaStream_t st, const int *gate, const int *gate2) {
    const int64_t D = op.sub.D;
    const double avg = (double)op.nnz / (double)D;
    const bool many = std::is_same<V, double>::value && D >= kCsrRowsD;
    if (rows_short(D, op.nnz) && !many) {
        k_matvec_csr<V, VV, true><<<grid_short(D), kThreads, 0, st>>>(op, x, y, 0, gate, gate2);
    } else if (many || (sizeof(V) == 16 && D > 65536 && avg > (dense(op.sub) ? 32. : 48.))) {
        k_matvec_csr_rows<V, VV><<<grid_rows(D), kThreads, 0, st>>>(op, x, y, gate, gate2);
    } else {
        const int rows = tile_rows<CsrTerm<V>>(D, op.nnz, sm_count(), even_rows(op.sub, sm_count()));
        k_matvec_csr<V, VV, false><<<grid_tiles(D, rows), kThreads, 0, st>>>(op, x, y, rows, gate, gate2);
    }
}

template <typename V>
int launch_csr(const rq_operator_t &op, const void *x, void *y, cudaStream_t st, const int *gate, const int *gate2) {
    const V *xx = static_cast<const V *>(x);
    V *yy = static_cast<V *>(y);
    switch (op.val_vtype) {
        case RQ_F32: run_csr<V, float>(op, xx, yy, st, gate, gate2); break;
        case RQ_F64: run_csr<V, double>(op, xx, yy, st, gate, gate2); break;
        case RQ_C64:
            if (!VT<V>::kComplex) return fail(RQ_E_ARG, "rq_matvec: complex CSR values need complex vectors");
            run_csr<V, float2>(op, xx, yy, st, gate, gate2);
            break;
        case RQ_C128:
            if (!VT<V>::kComplex) return fail(RQ_E_ARG, "rq_matvec: complex CSR values need complex vectors");
            run_csr<V, double2>(op, xx, yy, st, gate, gate2);
            break;
        default: return fail(RQ_E_ARG, "rq_matvec: bad val_vtype");
    }
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

// ------------------------------------------------------------------------------------------
// host dispatch
// ------------------------------------------------------------------------------------------
template <typename V, int KB, int FM, int BLOCK>
int launch_hash_block(const rq_operator_t &op, const void *x, void *y, int *err, cudaStream_t st,
                      const int *gate, const int *gate2) {
    auto kern = k_matvec_hash<V, KB, FM, BLOCK>;
    const int nres = op.terms.J - (op.terms.diag_group >= 0 ? 1 : 0);
    constexpr int kMaxRes = max_resident_groups<KB>();
    const size_t smem = group_key_bytes<KB>(nres < kMaxRes ? nres : kMaxRes);
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    KernelLaunchCache *c = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &c));
    RQ_TRY(configure_kernel(kern, *c, smem, BLOCK, &per_sm));
    int64_t g = (op.sub.D + BLOCK - 1) / BLOCK;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    if (g > cap) g = cap;
    kern<<<(int)(g < 1 ? 1 : g), BLOCK, smem, st>>>(op, static_cast<const V *>(x),
                                                   static_cast<V *>(y), err, gate, gate2);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

template <typename V, int KB, int FM, int BLOCK, bool QUEUE>
int launch_line_block(const rq_operator_t &op, int lw, const void *x, void *y, int *err, cudaStream_t st,
                      const int *gate, const int *gate2) {
    auto kern = k_matvec_line<V, KB, FM, BLOCK, QUEUE>;
    const int nres = op.terms.J - (op.terms.diag_group >= 0 ? 1 : 0);
    constexpr int kMaxTile = line_tile_groups<V, FM, BLOCK>();
    static_assert(kMaxTile <= 65536, "a queue entry holds 16 bits of group");
    const int kt = nres < kMaxTile ? std::max(nres, 1) : kMaxTile;
    const size_t smem = line_work_bytes<V, BLOCK, QUEUE>() + (size_t)(kt + kPart) * line_key_bytes<FM>();
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    KernelLaunchCache *c = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &c));
    RQ_TRY(configure_kernel(kern, *c, smem, BLOCK, &per_sm));
    const int64_t rows = BLOCK >> lw;
    int64_t g = (op.sub.D + rows - 1) / rows;
    // As many blocks as are resident, each walking several tiles; four times as many where each still has
    // a tile: one that ends early makes room (Hubbard 4x4, 2^20 rows, complex64: 75.7 against 71.8 us;
    // with fewer tiles the group keys of the extra blocks cost more: 2^18 low-energy rows, float64, 44.3
    // against 47.2 us, 2760 groups and 150,001 rows 1.95 against 2.85 ms)
    const int64_t cap = (int64_t)sm_count() * per_sm;
    if (g > cap) g = g >= 4 * cap ? 4 * cap : cap;
    kern<<<(int)g, BLOCK, smem, st>>>(op, static_cast<const V *>(x), static_cast<V *>(y), err, lw, kt,
                                      clustered(op.sub, op.terms.J) ? 1 : 0, gate, gate2);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

template <typename V, int KB, int FM>
int launch_hash(const rq_operator_t &op, const void *x, void *y, int *err, cudaStream_t st,
                const int *gate, const int *gate2) {
    // small group sets: several 256-thread blocks per SM; large ones (streamed in tiles above what
    // fits): one 1024-thread block
    if (op.sub.lmap) {
        const int lw = line_lanes_log2(op.sub, op.terms.J, sm_count());
        if constexpr (KB == 32 && FM == kFiltNone && sizeof(typename VT<V>::R) == 4)
            if (lw == 0 && own_hits(op.sub, op.terms.J, sm_count()))
                return launch_line_block<V, KB, FM, 256, false>(op, lw, x, y, err, st, gate, gate2);
        return line_small<FM>(op.terms.J)
                   ? launch_line_block<V, KB, FM, 256, true>(op, lw, x, y, err, st, gate, gate2)
                   : launch_line_block<V, KB, FM, 1024, true>(op, lw, x, y, err, st, gate, gate2);
    }
    const bool small = op.terms.J <= max_resident_groups<KB>() &&
                       group_key_bytes<KB>(op.terms.J) <= 16 * 1024;
    return small ? launch_hash_block<V, KB, FM, 256>(op, x, y, err, st, gate, gate2)
                 : launch_hash_block<V, KB, FM, 1024>(op, x, y, err, st, gate, gate2);
}

template <typename V, int LK>
int launch_free(const rq_operator_t &op, const void *x, void *y, int stop_at_zero, int *err,
                cudaStream_t st, const int *gate = nullptr, const int *gate2 = nullptr) {
    using R = typename VT<V>::R;
    const rq_terms_t &T = op.terms;
    const int gt = T.J < kGT ? (T.J > 0 ? T.J : 1) : kGT;
    const int kt = T.K < kKT ? (T.K > 0 ? T.K : 1) : kKT;
    const size_t smem = kFilterBytes + (LK == RQ_LOOKUP_BSEARCH ? kSample * 8 : 0) +
                        tile_bytes<R>(gt, kt);
    auto kern = k_matvec_free<V, LK>;
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    KernelLaunchCache *c = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &c));
    RQ_TRY(configure_kernel(kern, *c, smem, kThreads, &per_sm));
    int64_t g = (op.sub.D + kThreads - 1) / kThreads;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    if (g > cap) g = cap;
    kern<<<(int)g, kThreads, smem, st>>>(op, static_cast<const V *>(x), static_cast<V *>(y), gt, kt,
                                         stop_at_zero, err, gate, gate2);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

template <typename V>
int matvec_typed(const rq_operator_t &op, const void *x, void *y, void *scratch, cudaStream_t st,
                 const int *gate, const int *gate2) {
    int *err = scratch ? scratch_err(scratch) : nullptr;
    switch (op.mode) {
        case RQ_MODE_FREE:
            if (op.sub.lookup == RQ_LOOKUP_HASH) {
                // the sector filter is off when both masks are zero; a subspace in one sector
                // (fpoint >= 0) tests two popcounts instead of the bitset.  Behind a small line
                // filter the sector test costs more than it saves: a target it would reject
                // costs one L2-resident word of the line filter instead; a larger line filter
                // keeps it, since its words then compete for L2 or come from DRAM.
                const int fm = ((op.sub.fmask_a | op.sub.fmask_b) == 0 || (line_in_l2(op.sub) && !clustered(op.sub, op.terms.J))) ? kFiltNone
                               : op.sub.fpoint >= 0                                     ? kFiltPoint
                                                                                        : kFiltSet;
                if (op.sub.key_bits == 32) {
                    if (fm == kFiltPoint) return launch_hash<V, 32, kFiltPoint>(op, x, y, err, st, gate, gate2);
                    if (fm == kFiltSet) return launch_hash<V, 32, kFiltSet>(op, x, y, err, st, gate, gate2);
                    return launch_hash<V, 32, kFiltNone>(op, x, y, err, st, gate, gate2);
                }
                if (fm == kFiltPoint) return launch_hash<V, 64, kFiltPoint>(op, x, y, err, st, gate, gate2);
                if (fm == kFiltSet) return launch_hash<V, 64, kFiltSet>(op, x, y, err, st, gate, gate2);
                return launch_hash<V, 64, kFiltNone>(op, x, y, err, st, gate, gate2);
            }
            if (op.sub.lookup == RQ_LOOKUP_BSEARCH)
                return launch_free<V, RQ_LOOKUP_BSEARCH>(op, x, y, 1, err, st, gate, gate2);
            return fail(RQ_E_ARG, "rq_matvec: unsupported lookup for a subspace");
        case RQ_MODE_CONN:
            if (!op.rowptr || (op.nnz > 0 && (!op.col || !op.grp)))
                return fail(RQ_E_ARG, "rq_matvec: RQ_MODE_CONN needs rowptr, col and grp");
            if (sizeof(V) < 16 && rows_short(op.sub.D, op.nnz)) {
                k_matvec_conn<V, true><<<grid_short(op.sub.D), kThreads, 0, st>>>(
                    op, static_cast<const V *>(x), static_cast<V *>(y), 0, gate, gate2);
            } else {
                const int rows = tile_rows<RowTerm<V>>(op.sub.D, op.nnz, sm_count(), even_rows(op.sub, sm_count()));
                k_matvec_conn<V, false><<<grid_tiles(op.sub.D, rows), kThreads, 0, st>>>(
                    op, static_cast<const V *>(x), static_cast<V *>(y), rows, gate, gate2);
            }
            RQ_CUDA(cudaGetLastError());
            return RQ_OK;
        case RQ_MODE_CSR:
            if (!op.rowptr || (op.nnz > 0 && (!op.col || !op.val)))
                return fail(RQ_E_ARG, "rq_matvec: RQ_MODE_CSR needs rowptr, col and val");
            if (op.terms.diag_group >= 0 && !op.diag0)
                return fail(RQ_E_ARG, "rq_matvec: RQ_MODE_CSR needs diag0 when a diagonal group exists");
            return launch_csr<V>(op, x, y, st, gate, gate2);
        default:
            return fail(RQ_E_ARG, "rq_matvec: unknown mode");
    }
}

int check_operator(const rq_operator_t *op, int32_t vtype) {
    if (!op) return fail(RQ_E_ARG, "null operator");
    const rq_terms_t &T = op->terms;
    if (T.J < 0 || T.K < 0 || (T.J > 0 && (!T.xmask || !T.toff)) || (T.K > 0 && (!T.zmask || !T.coef)))
        return fail(RQ_E_ARG, "terms: bad sizes or null arrays");
    if (T.diag_group >= T.J) return fail(RQ_E_ARG, "terms: diag_group out of range");
    if ((vtype == RQ_F32 || vtype == RQ_F64) && !T.is_real)
        return fail(RQ_E_ARG, "real vectors need real coefficients (terms.is_real)");
    if (vtype_size(vtype) == 0) return fail(RQ_E_ARG, "unknown value type");
    if (op->sub.D < 1 || op->sub.D >= (int64_t(1) << 31))
        return fail(RQ_E_RANGE, "subspace dimension must be in [1, 2^31)");
    return RQ_OK;
}

}  // namespace

// Inclusive scan of D row counts in place (block scans, scan of block totals, offsets).
int scan_row_counts(int64_t *v, int64_t D, int64_t *bsum, cudaStream_t st) {
    const int64_t nb = (D + 1023) / 1024;
    k_scan_blocks<<<(int)nb, kThreads, 0, st>>>(v, D, bsum);
    k_scan_totals<<<1, kThreads, 0, st>>>(bsum, nb);
    k_scan_add<<<(int)nb, kThreads, 0, st>>>(v, D, bsum);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

// entry used by the LOBPCG driver (same translation-unit-independent dispatch)
int matvec_dispatch(const rq_operator_t &op, int32_t vtype, const void *x, void *y, void *scratch,
                    cudaStream_t st, const int *gate, const int *gate2) {
    switch (vtype) {
        case RQ_F32: return matvec_typed<float>(op, x, y, scratch, st, gate, gate2);
        case RQ_F64: return matvec_typed<double>(op, x, y, scratch, st, gate, gate2);
        case RQ_C64: return matvec_typed<float2>(op, x, y, scratch, st, gate, gate2);
        case RQ_C128: return matvec_typed<double2>(op, x, y, scratch, st, gate, gate2);
        default: return fail(RQ_E_ARG, "unknown value type");
    }
}

}  // namespace rq

using namespace rq;

RQ_API int rq_matvec(const rq_operator_t *op, int32_t vtype, const void *x, void *y, void *scratch,
                     void *stream) {
    RQ_TRY(check_operator(op, vtype));
    if (!x || !y || x == y) return fail(RQ_E_ARG, "rq_matvec: x and y must be distinct non-null");
    if (op->mode == RQ_MODE_FREE && !scratch)
        return fail(RQ_E_ARG, "rq_matvec: RQ_MODE_FREE needs scratch (error flag)");
    return matvec_dispatch(*op, vtype, x, y, scratch, as_stream(stream), nullptr, nullptr);
}

RQ_API int rq_fullspace_matvec(const rq_terms_t *terms, int32_t n, int32_t vtype, const void *x,
                               void *y, void *stream) {
    if (!terms || !x || !y || x == y || n < 0 || n > 31)
        return fail(RQ_E_ARG, "rq_fullspace_matvec: bad arguments (n must be <= 31)");
    rq_operator_t op = {};
    op.terms = *terms;
    op.terms.diag_group = -1;  // the x = 0 group is handled like any other (source = row)
    op.sub.D = int64_t(1) << n;
    op.sub.lookup = RQ_LOOKUP_IDENTITY;
    op.mode = RQ_MODE_FREE;
    RQ_TRY(check_operator(&op, vtype));
    cudaStream_t st = as_stream(stream);
    // PauliSumXZ.matmul sums every stored coefficient (no stop at a zero), symplectic.py:142-147
    switch (vtype) {
        case RQ_F32: return launch_free<float, RQ_LOOKUP_IDENTITY>(op, x, y, 0, nullptr, st);
        case RQ_F64: return launch_free<double, RQ_LOOKUP_IDENTITY>(op, x, y, 0, nullptr, st);
        case RQ_C64: return launch_free<float2, RQ_LOOKUP_IDENTITY>(op, x, y, 0, nullptr, st);
        case RQ_C128: return launch_free<double2, RQ_LOOKUP_IDENTITY>(op, x, y, 0, nullptr, st);
        default: return fail(RQ_E_ARG, "unknown value type");
    }
}

RQ_API int rq_terms_hash(const rq_terms_t *terms, uint32_t *xhash, void *stream) {
    if (!terms || !xhash || terms->J < 0 || (terms->J > 0 && !terms->xmask))
        return fail(RQ_E_ARG, "rq_terms_hash: bad arguments");
    if (terms->J == 0) return RQ_OK;
    // the hash is GF(2)-linear over the key bytes; masks below 2^32 hash the same with the
    // 4-byte and the 8-byte tables, so the 8-byte tables serve both key widths
    const int grid = (terms->J + kThreads - 1) / kThreads;
    k_terms_hash<64><<<grid, kThreads, 0, as_stream(stream)>>>(terms->xmask, terms->J, xhash);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

RQ_API int rq_terms_upload(int32_t J, int32_t K, const uint64_t *xmask, const int32_t *toff,
                           const uint64_t *zmask, const double *coef, uint64_t *d_xmask,
                           int32_t *d_toff, uint64_t *d_zmask, double *d_coef, uint32_t *d_xhash,
                           rq_terms_t *t, void *stream) {
    if (!t || J < 0 || K < 0 || !toff || !d_toff || (J > 0 && (!xmask || !d_xmask || !d_xhash)) ||
        (K > 0 && (!zmask || !coef || !d_zmask || !d_coef)))
        return fail(RQ_E_ARG, "rq_terms_upload: bad arguments");
    if (toff[0] != 0 || toff[J] != K) return fail(RQ_E_ARG, "rq_terms_upload: toff must span [0, K]");
    for (int32_t j = 0; j < J; ++j) {
        if (toff[j + 1] < toff[j]) return fail(RQ_E_ARG, "rq_terms_upload: toff decreases");
        if (j > 0 && xmask[j] <= xmask[j - 1])
            return fail(RQ_E_ARG, "rq_terms_upload: X masks must be strictly increasing");
    }
    int32_t real = 1;
    for (int64_t k = 0; k < K; ++k)
        if (coef[2 * k + 1] != 0.) real = 0;
    cudaStream_t st = as_stream(stream);
    if (J > 0) RQ_CUDA(cudaMemcpyAsync(d_xmask, xmask, sizeof(uint64_t) * J, cudaMemcpyHostToDevice, st));
    RQ_CUDA(cudaMemcpyAsync(d_toff, toff, sizeof(int32_t) * (J + 1), cudaMemcpyHostToDevice, st));
    if (K > 0) {
        RQ_CUDA(cudaMemcpyAsync(d_zmask, zmask, sizeof(uint64_t) * K, cudaMemcpyHostToDevice, st));
        RQ_CUDA(cudaMemcpyAsync(d_coef, coef, sizeof(double) * 2 * K, cudaMemcpyHostToDevice, st));
    }
    rq_terms_t T{};
    T.J = J;
    T.K = K;
    T.diag_group = (J > 0 && xmask[0] == 0) ? 0 : -1;
    T.is_real = real;
    T.xmask = d_xmask;
    T.toff = d_toff;
    T.zmask = d_zmask;
    T.coef = d_coef;
    T.xhash = nullptr;
    RQ_TRY(rq_terms_hash(&T, d_xhash, stream));
    T.xhash = J > 0 ? d_xhash : nullptr;
    RQ_CUDA(cudaStreamSynchronize(st));
    *t = T;
    return RQ_OK;
}

RQ_API int rq_conn_build(const rq_operator_t *op, int64_t *rowptr, int32_t *col, int32_t *grp,
                         void *val, int32_t vtype, int64_t *nnz, void *scratch, void *stream) {
    RQ_TRY(check_operator(op, val ? vtype : RQ_C128));
    if (!rowptr || !scratch || !nnz) return fail(RQ_E_ARG, "rq_conn_build: null argument");
    const rq_subspace_t &S = op->sub;
    if (S.lookup != RQ_LOOKUP_HASH && S.lookup != RQ_LOOKUP_BSEARCH)
        return fail(RQ_E_ARG, "rq_conn_build: needs a hash or binary-search subspace");
    cudaStream_t st = as_stream(stream);
    int *err = scratch_err(scratch);
    const int64_t D = S.D;
    if (!col) {
        RQ_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
        RQ_CUDA(cudaMemsetAsync(rowptr, 0, sizeof(int64_t), st));
        if (line_in_l2(S))
            RQ_TRY(conn_line(*op, rowptr + 1, nullptr, nullptr, nullptr, RQ_C128, err, st));
        else if (S.lookup == RQ_LOOKUP_HASH && S.key_bits == 32)
            k_conn_count<RQ_LOOKUP_HASH, 32><<<grid_rows(D), kThreads, 0, st>>>(*op, rowptr + 1, err);
        else if (S.lookup == RQ_LOOKUP_HASH)
            k_conn_count<RQ_LOOKUP_HASH, 64><<<grid_rows(D), kThreads, 0, st>>>(*op, rowptr + 1, err);
        else
            k_conn_count<RQ_LOOKUP_BSEARCH, 64><<<grid_rows(D), kThreads, 0, st>>>(*op, rowptr + 1, err);
        RQ_CUDA(cudaGetLastError());
        RQ_TRY(scan_row_counts(rowptr + 1, D, scratch_scan(scratch), st));
        int h_err = 0;
        RQ_CUDA(cudaMemcpyAsync(nnz, rowptr + D, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        RQ_CUDA(cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, st));
        RQ_CUDA(cudaStreamSynchronize(st));
        if (h_err) return fail(h_err, "rq_conn_build: lookup failed");
        return RQ_OK;
    }
    if (line_in_l2(S)) return conn_line(*op, rowptr, col, grp, val, val ? vtype : RQ_C128, err, st);
    const int g = grid_rows(D);
#define RQ_FILL(V)                                                                                  \
    do {                                                                                            \
        if (S.lookup == RQ_LOOKUP_HASH && S.key_bits == 32)                                         \
            k_conn_fill<V, RQ_LOOKUP_HASH, 32><<<g, kThreads, 0, st>>>(*op, rowptr, col, grp,       \
                                                                       static_cast<V *>(val), err); \
        else if (S.lookup == RQ_LOOKUP_HASH)                                                        \
            k_conn_fill<V, RQ_LOOKUP_HASH, 64><<<g, kThreads, 0, st>>>(*op, rowptr, col, grp,       \
                                                                       static_cast<V *>(val), err); \
        else                                                                                        \
            k_conn_fill<V, RQ_LOOKUP_BSEARCH, 64><<<g, kThreads, 0, st>>>(*op, rowptr, col, grp,    \
                                                                          static_cast<V *>(val), err); \
    } while (0)
    switch (val ? vtype : RQ_C128) {
        case RQ_F32: RQ_FILL(float); break;
        case RQ_F64: RQ_FILL(double); break;
        case RQ_C64: RQ_FILL(float2); break;
        case RQ_C128: RQ_FILL(double2); break;
        default: return fail(RQ_E_ARG, "rq_conn_build: unknown value type");
    }
#undef RQ_FILL
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}
