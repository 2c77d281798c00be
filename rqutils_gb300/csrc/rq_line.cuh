// Rows against X groups through the line filter: the shared part of the matrix-free matvec
// (rq_matvec.cu) and of the connectivity build (rq_conn.cu).
#pragma once

#include <algorithm>

#include "rq_common.cuh"
#include "rq_host.h"
#include "rq_rows.cuh"

namespace rq {
namespace {

// Sector filter of the hash kernels: none, the general (popcount a, popcount b) bitset, or the
// common case of a subspace in one sector (a single bit set: two popcount compares, no table).
enum { kFiltNone = 0, kFiltSet = 1, kFiltPoint = 2 };
// line filters of at most 2^25 bytes (32 MB, a quarter of GB300's L2) skip the sector test:
// measured faster without it at 16 MB (Hubbard D = 2^20: 0.089 against 0.107 ms) and slower at
// 64 MB (chemistry, 2^22 rows: 80.2 against 65.6 ms); clustered subspaces keep it at any size, since
// their probes are bound by the lines a warp touches (36 qubits, 150,001 rows: 2.03 against 2.29 ms)
constexpr int kLineFilterL2Log2Bytes = 25;

// shared memory of the hash kernels: the sector bitset, the hash byte tables (64-bit keys use
// all eight) and, in dynamic shared memory, the resident group keys
__shared__ uint32_t hk_fb[RQ_FILTER_WORDS];
__shared__ __align__(16) uint32_t hk_htab[kHashTableWords];
extern __shared__ __align__(16) unsigned char hk_dyn[];

// The sector test of a target for the filter form FM (pa0, pb0: the popcounts of the one sector).
template <typename K, int FM>
__device__ __forceinline__ bool sector_pass(K t, K fa, K fbm, int pa0, int pb0) {
    if (FM == kFiltPoint) {
        int pa, pb;
        if (sizeof(K) == 8) {
            pa = __popcll((unsigned long long)(t & fa));
            pb = __popcll((unsigned long long)(t & fbm));
        } else {
            pa = __popc((unsigned)(t & fa));
            pb = __popc((unsigned)(t & fbm));
        }
        return (pa == pa0) & (pb == pb0);
    }
    if (FM == kFiltSet) return sector_ok_k<K>(hk_fb, fa, fbm, t);
    return true;
}

// ---- probes of the line filter ---------------------------------------------------------------
// What bounds it: instruction issue and L2 latency when hits are rare (Hubbard 4x4, 2^20 rows: 0.24
// hits a row of 64 groups), the resolution of hits when they are not (a molecule's low-energy
// samples: 84 of 2760 groups).  So
// * a row is probed by w = 1 to 32 lanes: small subspaces would leave most of the chip idle, and the
//   rows of a sample with the most hits stand together and would keep one warp busy long after the
//   others (for such samples the tiles of a block are spread over the array, too; otherwise they
//   stand together, because neighbouring tiles share filter lines);
// * the hits of all lanes are gathered, in row and group order, into a queue that the whole warp
//   resolves in full rounds (bucket, row index, terms, x): no lane waits for another's longer list,
//   and FP64 instructions, which cost a warp the same however few lanes are active, run full;
//   groups of more than kShortTerms terms go to a second queue, so that short ones do not wait;
// * the owner lane of a row adds its products from the queue in group order, as the cached products do.
// Hubbard 4x4, complex64, against a loop of each lane over its own hits: 2^20 rows 75 us against 78, 2^18
// low-energy rows 47 against 59.
// QUEUE = false: that loop (own_hits).  It needs fewer registers (48 warps per SM instead of 32), and where
// every lane has about as many hits as its neighbours no lane waits for another.
constexpr int kQueueSlots = 128;  // hits resolved together

template <typename V>
struct WarpWork {
    uint32_t hit[kQueueSlots];                   // lane << 16 | resident group, or kMissed
    int src[kQueueSlots];                        // source row
    typename RowTerm<V>::P prod[kQueueSlots];
    uint8_t late[kQueueSlots];                   // queue slots of long groups
};
constexpr uint32_t kMissed = 0xFFFFFFFFu;

// Group keys in shared memory: (h(x), line word) and, for the sector test, x.  The x = 0 group is
// left out (its diagonal is applied before the probes); resident index c is group
// c + (c >= diag_group).  More groups than fit stream through in tiles.  Entries past the last group
// are probed and masked out: they hold a valid word.
template <int FM>
__host__ __device__ constexpr size_t line_key_bytes() { return FM != kFiltNone ? 16 : 8; }
// groups a lane probes between two resolutions (256 measured slower: 2.6 against 2.3 ms on the
// molecule above), and the entries past the last group
constexpr int kPart = 64;

template <typename V, int BLOCK, bool QUEUE = true>
__host__ __device__ constexpr size_t line_work_bytes() { return QUEUE ? (BLOCK / 32) * sizeof(WarpWork<V>) : 0; }

constexpr size_t kLineSmem = 216 * 1024;  // shared memory of a block with many groups (one per SM)
template <typename V, int FM, int BLOCK>
__host__ __device__ constexpr int line_tile_groups() {  // groups of a tile, at most 2^16
    return ((int)((kLineSmem - 16 * 1024 - (BLOCK / 32) * sizeof(WarpWork<V>)) / line_key_bytes<FM>()) & ~63) - kPart;
}

// Line-filter word of a key (a state or an X mask): the word index line << (lwbits - 5) | word
// within the line, line = h(k >> lshift) >> (32 - lbits), word = (h(k) mod 2^lwbits) >> 5.  Every
// step is linear over XOR, so the word of a target s ^ x is word(s) ^ word(x) (lbits + lwbits - 5
// <= 32 bits, rq_line_filter_bits).
__device__ __forceinline__ uint32_t line_word(uint32_t h, uint32_t hpre, const rq_subspace_t &S) {
    return ((hpre >> (32 - S.lbits)) << (S.lwbits - 5)) | ((h & ((1u << S.lwbits) - 1u)) >> 5);
}

// The rows of the operator over its X groups (without the x = 0 group).  The consumer C, one per lane,
// sees for each row: start(i, s, own) -- own: the lane that sums the row -- then for each hit
// resolve(W, q, g, s, m) on some lane of the warp (queue slot q, group g, row state s, source m;
// true: call late() for it in the second round), take(W, q, g) on the owner in list order, and
// finish(i).  Without a queue: hit(g, s, m) on the owner.  A warp takes the 32 >> lw rows from
// `first` + a multiple of `stride` while some row of the block's turn lies below `end`; the caller
// has filled hk_htab (and hk_fb), and every thread of the block calls.
template <typename V, int KB, int FM, int BLOCK, bool QUEUE = true, typename C>
__device__ __forceinline__ void line_rows(const rq_subspace_t &S, const rq_terms_t &T, int *err, int lw, int kt,
                                          int64_t first, int64_t turn, int64_t stride, int64_t end, C &use) {
    using K = typename KeyWidth<KB>::K;
    constexpr int NB = KeyWidth<KB>::kNbytes;
    // probes in flight per lane: what 64 (QUEUE) and 40 registers hold
    constexpr int U = FM != kFiltNone ? 8 : QUEUE ? 16 : KB == 32 ? 32 : 8;
    const int skip = T.diag_group;
    const int nres = T.J - (skip >= 0 ? 1 : 0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    WarpWork<V> &W = reinterpret_cast<WarpWork<V> *>(hk_dyn)[QUEUE ? warp : 0];
    uint2 *gk = reinterpret_cast<uint2 *>(hk_dyn + line_work_bytes<V, BLOCK, QUEUE>());  // [kt + kPart]
    uint64_t *gx = reinterpret_cast<uint64_t *>(gk + kt + kPart);                       // the same, FM only
    auto load_keys = [&](int c0, int n) {
        for (int c = threadIdx.x; c < n + kPart; c += blockDim.x) {
            const int j = c0 + c + (skip >= 0 && c0 + c >= skip);
            const uint64_t xv = c < n ? T.xmask[j] : 0ULL;
            const uint32_t h = c >= n ? 0u : T.xhash ? T.xhash[j] : lin_hash(hk_htab, xv, NB);
            gk[c] = make_uint2(h, line_word(h, lin_hash(hk_htab, S.lshift < 64 ? xv >> S.lshift : 0ULL, NB), S));
            if (FM != kFiltNone) gx[c] = xv;
        }
    };
    __syncthreads();
    const bool tiled = nres > kt;
    if (!tiled) {
        load_keys(0, nres);
        __syncthreads();
    }
    const int pa0 = S.fpoint / 65, pb0 = S.fpoint % 65;
    const K fa = (K)S.fmask_a, fbm = (K)S.fmask_b;
    const int shift = 32 - S.hbits;
    const uint32_t *lmap = S.lmap;
    const unsigned lt = (1u << lane) - 1u;
    const int w = 1 << lw, sub = lane & (w - 1);
    for (int64_t base = 0; turn + base < end; base += stride) {  // the same trips for every warp of a block
        const int64_t i = first + base + (lane >> lw);
        const bool active = i < end;
        if (!tiled && first + base >= end) break;
        const int64_t ir = active ? i : end - 1;
        const uint64_t s64 = __ldg(S.states + ir);
        const K s = (K)s64;
        const uint32_t hs = lin_hash(hk_htab, s64, NB);
        // the row's line-filter word: a target's word is wrow ^ word(x), its bits those of hs ^ h(x)
        const uint32_t wrow = line_word(hs, lin_hash(hk_htab, S.lshift < 64 ? s64 >> S.lshift : 0ULL, NB), S);
        use.start(ir, s64, sub == 0);
        for (int t0 = 0; t0 < nres; t0 += kt) {
            const int tn = min(kt, nres - t0);
            if (tiled) {
                __syncthreads();  // the previous tile is no longer read
                load_keys(t0, tn);
                __syncthreads();
            }
            // lane `sub` of a row takes the sub-th part of the next up to kPart w groups
            int part = 0;
            for (int g0 = 0; g0 < tn; g0 += part << lw) {
                part = min(kPart, (tn - g0 + w - 1) >> lw);
                const int e0 = min(g0 + sub * part, tn), en = active ? min(part, tn - e0) : 0;
                uint64_t hot = 0ULL;
                for (int k0 = 0; k0 < part; k0 += U) {
                    const uint2 *key = gk + e0 + k0;
                    uint32_t v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const uint32_t *p = lmap + (wrow ^ key[u].y);
                        v[u] = FM == kFiltNone ? __ldg(p)
                                               : load_word(p, sector_pass<K, FM>(s ^ (K)gx[e0 + k0 + u], fa, fbm, pa0, pb0));
                    }
                    uint32_t hb = 0u;
#pragma unroll
                    for (int u = 0; u < U; ++u) {  // (the funnel shift takes its count mod 32)
                        const uint32_t b = hs ^ key[u].x;
                        hb += (__funnelshift_r(v[u], 0u, b) & (v[u] >> (b >> 27)) & 1u) << u;
                    }
                    hot |= (uint64_t)hb << k0;
                }
                hot &= en >= 64 ? ~0ULL : (1ULL << en) - 1ULL;
                if constexpr (!QUEUE) {
                    while (hot) {
                        const int e = e0 + __ffsll((long long)hot) - 1, c = t0 + e, gg = c + (skip >= 0 && c >= skip);
                        hot &= hot - 1ULL;
                        const int m = lookup_hash_at<KB>(S, s64 ^ __ldg(T.xmask + gg), (hs ^ gk[e].x) >> shift, err);
                        if (m >= 0) use.hit(gg, s64, m);
                    }
                    __syncwarp();  // re-converge before the next probes
                    continue;
                }
                // resolve the hits of the warp, kQueueSlots at a time
                const int cnt = __popcll(hot);
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                if (total == 0) continue;
                int off = incl - cnt;
                // the row's range of the queue
                const int ra = __shfl_sync(0xffffffffu, off, lane & ~(w - 1));
                const int rb = __shfl_sync(0xffffffffu, incl, lane | (w - 1));
                for (int q0 = 0; q0 < total; q0 += kQueueSlots) {
                    const int n = min(kQueueSlots, total - q0);
                    while (hot && off < q0 + n) {
                        W.hit[off - q0] = (uint32_t)lane << 16 | (uint32_t)(e0 + __ffsll((long long)hot) - 1);
                        hot &= hot - 1ULL;
                        ++off;
                    }
                    __syncwarp();
                    int late = 0;
                    for (int q = lane; q - lane < n; q += 32) {
                        const bool ok = q < n;
                        const uint32_t hit = ok ? W.hit[q] : 0u;
                        const uint64_t rs = __shfl_sync(0xffffffffu, s64, hit >> 16);
                        const uint32_t rh = __shfl_sync(0xffffffffu, hs, hit >> 16);
                        bool defer = false;
                        if (ok) {
                            const int e = (int)(hit & 0xFFFFu), c = t0 + e, gg = c + (skip >= 0 && c >= skip);
                            const uint64_t xv = __ldg(T.xmask + gg);
                            const int m = lookup_hash_at<KB>(S, rs ^ xv, (rh ^ gk[e].x) >> shift, err);
                            W.src[q] = m;
                            if (m < 0) W.hit[q] = kMissed;
                            else defer = use.resolve(W, q, gg, rs, m);
                        }
                        const unsigned dm = __ballot_sync(0xffffffffu, defer);
                        if (defer) W.late[late + __popc(dm & lt)] = (uint8_t)q;
                        late += __popc(dm);
                    }
                    __syncwarp();
                    for (int k = lane; k - lane < late; k += 32) {
                        const bool ok = k < late;
                        const int q = ok ? W.late[k] : 0;
                        const uint32_t hit = ok ? W.hit[q] : 0u;
                        const uint64_t rs = __shfl_sync(0xffffffffu, s64, hit >> 16);
                        if (ok) {
                            const int c = t0 + (int)(hit & 0xFFFFu), gg = c + (skip >= 0 && c >= skip);
                            use.late(W, q, gg, rs);
                        }
                    }
                    __syncwarp();
                    if (sub == 0)
                        for (int k = max(ra, q0) - q0; k < min(rb - q0, n); ++k)
                            if (W.hit[k] != kMissed) {
                                const int c = t0 + (int)(W.hit[k] & 0xFFFFu);
                                use.take(W, k, c + (skip >= 0 && c >= skip));
                            }
                    __syncwarp();
                }
            }
        }
        if (active && sub == 0) use.finish(i);
    }
}

// The tables and the calling warp's place for a kernel that walks the whole subspace: neighbouring
// tiles of 32 >> lw rows to the same block, or (spread) to different SMs.
template <typename V, int KB, int FM, int BLOCK, bool QUEUE = true, typename C>
__device__ __forceinline__ void line_subspace(const rq_operator_t &op, int *err, int lw, int kt, int spread, C &use) {
    copy_hash_tables(hk_htab, KeyWidth<KB>::kNbytes);
    if (FM == kFiltSet)
        for (int w = threadIdx.x; w < RQ_FILTER_WORDS; w += blockDim.x) hk_fb[w] = op.sub.fbits[w];
    const int warp = threadIdx.x >> 5;
    const int64_t rows = 32 >> lw, stride = (int64_t)gridDim.x * (BLOCK / 32) * rows;
    const int64_t first =
        (spread ? (int64_t)warp * gridDim.x + blockIdx.x : (int64_t)blockIdx.x * (BLOCK / 32) + warp) * rows;
    line_rows<V, KB, FM, BLOCK, QUEUE>(op.sub, op.terms, err, lw, kt, first, 0, stride, op.sub.D, use);
}

// ---- launch rules -----------------------------------------------------------------------------
// Clustered subspaces (low-energy samples of a molecule) with many groups: their hits crowd on some
// rows, which stand together, and their line prefix is short, so that a warp's probes fall in many
// lines.  The prefix shift tells them: states spread over n bits get about n - log2 D + 3, less the
// few bits that a sector takes (measured 1 to 3; molecules 4 to 11).
constexpr int kClusterBits = 4;
constexpr int kClusterGroups = 256;
inline bool clustered(const rq_subspace_t &S, int J) {
    const uint64_t used = S.fmask_a | S.fmask_b;
    const int n = used ? 64 - __builtin_clzll(used) : 0, d = 63 - __builtin_clzll((uint64_t)S.D);
    return J >= kClusterGroups && n - d + 3 - S.lshift >= kClusterBits;
}

// Lanes per row (log2): the most with which all rows are still resident at once, kLineThreads
// threads per SM.  One lane is best for large subspaces (the rows of a warp share filter lines, and
// every lane sums a row); at 16,384 rows one lane leaves 9 of 10 warp slots of the chip empty.
// Clustered subspaces take as many lanes as make kLineWaves passes over the chip: 36 qubits, 150,001
// rows, float64: 2.3 against 3.8 ms with one lane, 2.6 with eight passes; spread states want one lane
// (40 qubits, 100,000 rows: 84 us against 121 with four).
constexpr int kLineThreads = 1024;
constexpr int kLineWaves = 4;
inline int line_lanes_log2(const rq_subspace_t &S, int J, int sms) {
    const int waves = clustered(S, J) ? kLineWaves : 1;
    int lw = 0;
    while (lw < 5 && ((S.D << (lw + 1)) <= (int64_t)sms * kLineThreads ||
                      (J >= 64 << (lw + 1) && (S.D << (lw + 1)) <= (int64_t)sms * kLineThreads * waves)))
        ++lw;
    return lw;
}

// threads per block: several 256-thread blocks per SM for small group sets; for large ones (streamed
// in tiles above what fits) one 1024-thread block
template <int FM>
inline bool line_small(int J) { return J * line_key_bytes<FM>() <= 16 * 1024; }

// Dense subspaces, whose rows have many hits each and about as many as their neighbours.  The prefix shift
// tells them, as above: shift b is about 2^(lwbits - 5) states among 2^b neighbours.
constexpr int kDenseShift = 7;  // for lines of 2^8 bits
inline bool dense(const rq_subspace_t &S) {
    return S.lookup == RQ_LOOKUP_HASH && S.lmap && S.lshift <= kDenseShift + S.lwbits - 8;
}

// more of them than are resident with the queue
inline bool even_rows(const rq_subspace_t &S, int sms) { return S.D > (int64_t)sms * kLineThreads && dense(S); }

// Whether the lanes resolve their own hits, in 32-bit arithmetic.  complex64,
// queue against own hits: 20 qubits, 157,000 rows (shift 5) 131 us against 86; 23 qubits, 676,000 rows
// (6) 514 against 435; 24 qubits, 500,000 rows (7) 126 against 121, 250,000 (8) 50 against 54; 32 qubits,
// 400,000 low-energy rows (13) 69 against 92; 21 qubits, 120,000 rows, all resident, 51 against 53.
inline bool own_hits(const rq_subspace_t &S, int J, int sms) {
    return even_rows(S, sms) && line_small<kFiltNone>(J);
}

// whether there is a line filter (rq_subspace_build fills it for hash lookups only, whatever lmap holds
// otherwise) and it stays in L2 beside the other tables
inline bool line_in_l2(const rq_subspace_t &S) {
    return S.lookup == RQ_LOOKUP_HASH && S.lmap && S.lbits + S.lwbits - 3 <= kLineFilterL2Log2Bytes;
}

}  // namespace
}  // namespace rq
