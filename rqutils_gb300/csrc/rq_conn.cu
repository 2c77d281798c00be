// Connectivity build through the line filter: the probes, the hit queue and the lanes per row of the
// matrix-free matvec (rq_line.cuh) with other consumers.  The count and the fill pass each resolved
// every target in the hash table, one dependent load after the other on one thread per row: 0.38 ms
// for 500,009 rows of 64 groups and 4.2 ms for 125,000 rows of 2760, both passes; now 0.20 and 2.0 ms.
#include "rq_line.cuh"

namespace rq {
namespace {

struct UseCount {  // elements per row
    int64_t *out;
    int64_t n;
    __device__ __forceinline__ void start(int64_t, uint64_t, bool) { n = 0; }
    __device__ __forceinline__ bool resolve(WarpWork<float> &, int, int, uint64_t, int) { return false; }
    __device__ __forceinline__ void late(WarpWork<float> &, int, int, uint64_t) {}
    __device__ __forceinline__ void take(const WarpWork<float> &, int, int) { ++n; }
    __device__ __forceinline__ void finish(int64_t i) { out[i] = n; }
};

template <typename V>
struct UseFill {  // (source, group) lists and, CSR, the elements
    const rq_terms_t &T;
    const int64_t *rowptr;
    int32_t *col, *grp;
    V *val;
    int64_t p;
    __device__ __forceinline__ void value(WarpWork<V> &W, int q, int g, uint64_t s) const {
        if constexpr (VT<V>::kComplex) W.prod[q] = group_diag<typename VT<V>::R>(T, g, s);
        else reinterpret_cast<V &>(W.prod[q]) = group_diag_re<V>(T, g, s);
    }
    __device__ __forceinline__ void start(int64_t i, uint64_t, bool own) { p = own ? rowptr[i] : 0; }
    __device__ __forceinline__ bool resolve(WarpWork<V> &W, int q, int g, uint64_t s, int) {
        if (!val) return false;
        if (group_terms(T, g) > kShortTerms) return true;
        value(W, q, g, s);
        return false;
    }
    __device__ __forceinline__ void late(WarpWork<V> &W, int q, int g, uint64_t s) { value(W, q, g, s); }
    __device__ __forceinline__ void take(const WarpWork<V> &W, int q, int g) {
        col[p] = W.src[q];
        if (grp) grp[p] = g;
        if (val) {
            if constexpr (VT<V>::kComplex) VT<V>::st(val, p, W.prod[q]);
            else val[p] = reinterpret_cast<const V &>(W.prod[q]);
        }
        ++p;
    }
    __device__ __forceinline__ void finish(int64_t) {}
};

template <int KB, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK)
k_conn_count_line(const rq_operator_t op, int64_t *__restrict__ rows, int *err, int lw, int kt, int spread) {
    UseCount use{rows, 0};
    line_subspace<float, KB, kFiltNone, BLOCK>(op, err, lw, kt, spread, use);
}

template <typename V, int KB, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK)
k_conn_fill_line(const rq_operator_t op, const int64_t *__restrict__ rowptr, int32_t *__restrict__ col,
                 int32_t *__restrict__ grp, V *__restrict__ val, int *err, int lw, int kt, int spread) {
    UseFill<V> use{op.terms, rowptr, col, grp, val, 0};
    line_subspace<V, KB, kFiltNone, BLOCK>(op, err, lw, kt, spread, use);
}

// grid and shared memory of a kernel over the rows; launches through go(grid, smem, lw, kt, spread)
template <typename V, int BLOCK, typename K, typename F>
int launch(K kern, KernelLaunchCache (&table)[kMaxCachedDevices], const rq_operator_t &op, F &&go) {
    const int nres = op.terms.J - (op.terms.diag_group >= 0 ? 1 : 0);
    constexpr int kMaxTile = line_tile_groups<V, kFiltNone, BLOCK>();
    static_assert(kMaxTile <= 65536, "a queue entry holds 16 bits of group");
    const int kt = nres < kMaxTile ? std::max(nres, 1) : kMaxTile;
    const size_t smem = line_work_bytes<V, BLOCK>() + (size_t)(kt + kPart) * line_key_bytes<kFiltNone>();
    KernelLaunchCache *c = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &c));
    RQ_TRY(configure_kernel(kern, *c, smem, BLOCK, &per_sm));
    const int lw = line_lanes_log2(op.sub, op.terms.J, sm_count());
    const int64_t rows = BLOCK >> lw;
    const int64_t g = std::min<int64_t>((op.sub.D + rows - 1) / rows, (int64_t)sm_count() * per_sm);
    go((int)g, smem, lw, kt, clustered(op.sub, op.terms.J) ? 1 : 0);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

template <int KB, int BLOCK>
int count_rows(const rq_operator_t &op, int64_t *rows, int *err, cudaStream_t st) {
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    auto kern = k_conn_count_line<KB, BLOCK>;
    return launch<float, BLOCK>(kern, table, op, [&](int g, size_t smem, int lw, int kt, int spread) {
        kern<<<g, BLOCK, smem, st>>>(op, rows, err, lw, kt, spread);
    });
}

template <typename V, int KB, int BLOCK>
int fill_rows(const rq_operator_t &op, const int64_t *rows, int32_t *col, int32_t *grp, void *val, int *err,
              cudaStream_t st) {
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    auto kern = k_conn_fill_line<V, KB, BLOCK>;
    return launch<V, BLOCK>(kern, table, op, [&](int g, size_t smem, int lw, int kt, int spread) {
        kern<<<g, BLOCK, smem, st>>>(op, rows, col, grp, static_cast<V *>(val), err, lw, kt, spread);
    });
}

template <int KB, int BLOCK>
int dispatch(const rq_operator_t &op, int64_t *rows, int32_t *col, int32_t *grp, void *val, int32_t vtype, int *err,
             cudaStream_t st) {
    if (!col) return count_rows<KB, BLOCK>(op, rows, err, st);
    switch (vtype) {
        case RQ_F32: return fill_rows<float, KB, BLOCK>(op, rows, col, grp, val, err, st);
        case RQ_F64: return fill_rows<double, KB, BLOCK>(op, rows, col, grp, val, err, st);
        case RQ_C64: return fill_rows<float2, KB, BLOCK>(op, rows, col, grp, val, err, st);
        case RQ_C128: return fill_rows<double2, KB, BLOCK>(op, rows, col, grp, val, err, st);
        default: return fail(RQ_E_ARG, "rq_conn_build: unknown value type");
    }
}

}  // namespace

int conn_line(const rq_operator_t &op, int64_t *rows, int32_t *col, int32_t *grp, void *val, int32_t vtype, int *err,
              cudaStream_t st) {
    const bool small = line_small<kFiltNone>(op.terms.J);
    if (op.sub.key_bits == 32)
        return small ? dispatch<32, 256>(op, rows, col, grp, val, vtype, err, st)
                     : dispatch<32, 1024>(op, rows, col, grp, val, vtype, err, st);
    return small ? dispatch<64, 256>(op, rows, col, grp, val, vtype, err, st)
                 : dispatch<64, 1024>(op, rows, col, grp, val, vtype, err, st);
}

}  // namespace rq
