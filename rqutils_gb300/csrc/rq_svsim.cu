// State-vector simulation of Pauli-rotation circuits (the reference's svsim, svsim.py:88-122).
//
// A gate is (x, z, c, s): out[i] = i s (-1)^popcount(i & z) state[i ^ x] + c state[i] (the c term
// is dropped when c == 0, as the reference does).  Products and sums are rounded one at a time (no
// fused multiply-add) in the order of the reference's complex arithmetic, so results equal the
// reference arithmetic bit for bit (up to the sign of zero results).
//
// What bounds it on GB300 is FP64 arithmetic: six operations per amplitude and gate at 1/64 of the
// FP32 rate (n = 20: 10 us a gate, when a pass over the 16 MB state in L2 takes 5).  One pass per gate
// adds its launch, its ramp and its memory time to that.  So the circuit is cut into segments of
// consecutive gates whose X masks stay within m index bits: a block loads a tile (the 2^m amplitudes
// that differ in those bits) into shared memory and takes it through all gates of the segment.  The
// three lowest bits always belong to the tile (128 contiguous bytes).  n = 20, 120 gates (rx, rz, rzz,
// ry, x): 2.64 -> 1.72 ms.
#include <algorithm>
#include <cmath>
#include <vector>

#include "rq_common.cuh"
#include "rq_host.h"

namespace rq {
namespace {

struct Gate {
    uint64_t x, z;  // x: in tile coordinates inside a segment
    double c, s;
};

constexpr int kLowBits = 3;          // index bits that every tile holds
constexpr int kMaxTileBits = 11;     // 32 KB of amplitudes
constexpr int kSegmentGates = 256;   // most gates of a segment (8 KB of shared memory)

__device__ __forceinline__ double flip_if(double v, bool f) {
    return __longlong_as_double(__double_as_longlong(v) ^ (f ? (long long)0x8000000000000000ULL : 0LL));
}

// out = i s sigma v_src + c v_self   (sigma = +-1).  (0 + i a)(re + i im) = (0 re - a im) +
// i (0 im + a re); the 0 x terms only decide the sign of a zero result and are left out, as is the
// product s sigma (exact).  unit: |s| = 1, whose product is a sign.
__device__ __forceinline__ double2 rot(double c, double s, bool neg, double2 self, double2 src, bool with_c,
                                       bool unit) {
    double re, im;
    if (unit) {
        const bool f = neg != ((__double_as_longlong(s) >> 63) != 0);
        re = flip_if(src.y, !f);
        im = flip_if(src.x, f);
    } else {
        // (the minus of -(a src.y) goes into the sign of a: on its own it is an FP64 instruction)
        re = __dmul_rn(flip_if(s, !neg), src.y);
        im = __dmul_rn(flip_if(s, neg), src.x);
    }
    if (with_c) {
        re = __dadd_rn(re, __dmul_rn(c, self.x));
        im = __dadd_rn(im, __dmul_rn(c, self.y));
    }
    return make_double2(re, im);
}

__device__ __forceinline__ bool parity_odd(uint64_t i, uint64_t z) { return __popcll(i & z) & 1; }
__device__ __forceinline__ bool is_zero(double c) { return (__double_as_longlong(c) << 1) == 0; }
__device__ __forceinline__ bool is_unit(double s) {
    return ((uint64_t)__double_as_longlong(s) & 0x7FFFFFFFFFFFFFFFULL) == 0x3FF0000000000000ULL;
}

struct Tile {
    int32_t m, low;               // index bits of a tile; the lowest `low` of them are 0 .. low - 1
    uint8_t bit[kMaxTileBits];    // the tile's index bits, ascending
};

// The gates [g0, g1) (at most kSegmentGates) on every tile.
__global__ void __launch_bounds__(kThreads)
k_segment(double2 *__restrict__ psi, uint64_t tiles, const Gate *__restrict__ gates, int g0, int g1, const Tile T) {
    extern __shared__ __align__(16) unsigned char dyn[];
    double2 *amp = reinterpret_cast<double2 *>(dyn);                              // [2^m]
    uint64_t *off = reinterpret_cast<uint64_t *>(amp + (size_t(1) << T.m));       // [2^(m - low)]
    __shared__ Gate gs[kSegmentGates];
    const int n = 1 << T.m, lowmask = (1 << T.low) - 1, ng = g1 - g0;
    for (int k = threadIdx.x; k < ng; k += blockDim.x) gs[k] = gates[g0 + k];
    for (int h = threadIdx.x; h < n >> T.low; h += blockDim.x) {
        uint64_t v = 0;
        for (int b = T.low; b < T.m; ++b) v |= (uint64_t)((h >> (b - T.low)) & 1) << T.bit[b];
        off[h] = v;
    }
    __syncthreads();
    auto place = [&](int l) { return off[l >> T.low] | (uint64_t)(l & lowmask); };
    for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint64_t base = t;  // the tile's number with zeros at its own bits
        for (int b = 0; b < T.m; ++b)
            base = (base >> T.bit[b] << (T.bit[b] + 1)) | (base & ((1ULL << T.bit[b]) - 1ULL));
        for (int l = threadIdx.x; l < n; l += blockDim.x) amp[l] = psi[base | place(l)];
        __syncthreads();
        int g = 0;
        while (g < ng) {
            if (gs[g].x == 0) {  // a run of diagonal gates: each amplitude through all of them
                int e = g + 1;
                while (e < ng && gs[e].x == 0) ++e;
                for (int l = threadIdx.x; l < n; l += blockDim.x) {
                    const uint64_t i = base | place(l);
                    double2 v = amp[l];
                    for (int k = g; k < e; ++k)
                        v = rot(gs[k].c, gs[k].s, parity_odd(i, gs[k].z), v, v, !is_zero(gs[k].c), is_unit(gs[k].s));
                    amp[l] = v;
                }
                g = e;
            } else {  // pairs (l, l ^ x)
                const Gate G = gs[g];
                const int x = (int)G.x, low = (x & -x) - 1;
                const bool wc = !is_zero(G.c), unit = is_unit(G.s);
                for (int p = threadIdx.x; p < n >> 1; p += blockDim.x) {
                    const int l = ((p & ~low) << 1) | (p & low), r = l ^ x;
                    const double2 a = amp[l], b = amp[r];
                    amp[l] = rot(G.c, G.s, parity_odd(base | place(l), G.z), a, b, wc, unit);
                    amp[r] = rot(G.c, G.s, parity_odd(base | place(r), G.z), b, a, wc, unit);
                }
                ++g;
            }
            __syncthreads();
        }
        for (int l = threadIdx.x; l < n; l += blockDim.x) psi[base | place(l)] = amp[l];
        __syncthreads();
    }
}

// one gate whose X mask does not fit a tile, in place over pairs (i, i ^ x); lb = lowest set bit of x
__global__ void k_pair(double2 *__restrict__ psi, uint64_t N, const Gate *__restrict__ gates, int g, int lb) {
    const Gate G = gates[g];
    const uint64_t half = N >> 1;
    const uint64_t low = (1ULL << lb) - 1ULL;
    const bool wc = !is_zero(G.c), unit = is_unit(G.s);
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < half; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = ((t & ~low) << 1) | (t & low);  // bit lb of i is 0
        const uint64_t j = i ^ G.x;
        const double2 a = psi[i], b = psi[j];
        psi[i] = rot(G.c, G.s, parity_odd(i, G.z), a, b, wc, unit);
        psi[j] = rot(G.c, G.s, parity_odd(j, G.z), b, a, wc, unit);
    }
}

int grid_for(uint64_t n) {
    uint64_t g = (n + kThreads - 1) / kThreads;
    const uint64_t cap = (uint64_t)sm_count() * 8;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

struct Segment {
    int g0, g1;
    uint64_t bits;  // the tile's index bits; 0: one gate by k_pair
};

// Greedy cut for tiles of m bits: a segment takes gates while their X masks fit.
std::vector<Segment> cut(const std::vector<Gate> &gates, int n, int m) {
    std::vector<Segment> out;
    const int low = std::min(kLowBits, m);
    const uint64_t lowbits = (1ULL << low) - 1ULL;
    const int ng = (int)gates.size();
    int g = 0;
    while (g < ng) {
        uint64_t bits = lowbits;
        int e = g;
        while (e < ng && e - g < kSegmentGates && __builtin_popcountll(bits | gates[e].x) <= m) bits |= gates[e++].x;
        if (e == g) {
            out.push_back({g, g + 1, 0});
            ++g;
            continue;
        }
        for (int b = 0; b < n && __builtin_popcountll(bits) < m; ++b) bits |= 1ULL << b;
        out.push_back({g, e, bits});
        g = e;
    }
    return out;
}

// Estimated microseconds of a cut: a launch and a pass over the state per segment (3 us; 32 bytes an
// amplitude at 6 TB/s, or the latency of a tile), and the FP64 time of its gates, whole warps of
// 12 x 64 cycles a pair on the quarters of the SM that takes the most tiles (at 2 GHz).
double cut_cost(const std::vector<Segment> &segs, int n, int m, int sms) {
    const double N = (double)(1ULL << n);
    const double tiles = (double)(1ULL << (n - m)), per_sm = std::max(1., std::ceil(tiles / sms));
    const double warps = std::max(1., (double)(1ULL << (m > 0 ? m - 1 : 0)) / 32.);
    double us = 0.;
    for (const Segment &s : segs) {
        us += 3. + std::max(2., 32. * N / 6e6);
        const double gate = s.bits ? std::ceil(per_sm * warps / 4.) * 768. / 2000. : N / 2. / 32. / (4. * sms) * 768. / 2000.;
        us += (s.g1 - s.g0) * std::max(gate, 0.1 + 768. / 2000.);
    }
    return us;
}

// x with only its bits at the positions of `bits`, packed
uint64_t extract(uint64_t x, uint64_t bits) {
    uint64_t out = 0;
    for (int k = 0; bits; ++k, bits &= bits - 1ULL)
        if (x & (bits & -bits)) out |= 1ULL << k;
    return out;
}

}  // namespace
}  // namespace rq

using namespace rq;

RQ_API int rq_svsim(const uint64_t *x, const uint64_t *z, const double *cosv, const double *sinv, int32_t ngates,
                    int32_t n, void *state, void *gates_scratch, void *stream) {
    if (!x || !z || !cosv || !sinv || !state || ngates < 0 || n < 1 || n > 40 || (ngates > 0 && !gates_scratch))
        return fail(RQ_E_ARG, "rq_svsim: bad arguments (1 <= n <= 40)");
    const uint64_t N = 1ULL << n;
    std::vector<Gate> h(ngates);
    for (int g = 0; g < ngates; ++g) {
        if ((x[g] >> n) != 0 || (z[g] >> n) != 0) return fail(RQ_E_ARG, "rq_svsim: a gate acts beyond n qubits");
        h[g] = Gate{x[g], z[g], cosv[g], sinv[g]};
    }
    if (ngates == 0) return RQ_OK;
    cudaStream_t st = as_stream(stream);
    Gate *dg = static_cast<Gate *>(gates_scratch);
    double2 *psi = static_cast<double2 *>(state);
    // the tile size with the lowest estimate: larger tiles take more gates per pass, smaller ones
    // spread a small state over more SMs
    std::vector<Segment> segs;
    int m = 0;
    double best = 0.;
    for (int k = std::min(n, 4); k <= std::min(n, kMaxTileBits); ++k) {
        std::vector<Segment> c = cut(h, n, k);
        const double us = cut_cost(c, n, k, sm_count());
        if (m == 0 || us < best) {
            best = us;
            m = k;
            segs.swap(c);
        }
    }
    for (const Segment &s : segs)
        if (s.bits)
            for (int g = s.g0; g < s.g1; ++g) h[g].x = extract(h[g].x, s.bits);
    RQ_CUDA(cudaMemcpyAsync(dg, h.data(), sizeof(Gate) * ngates, cudaMemcpyHostToDevice, st));
    const size_t smem = (sizeof(double2) << m) + (sizeof(uint64_t) << (m - std::min(kLowBits, m)));
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    KernelLaunchCache *cache = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &cache));
    RQ_TRY(configure_kernel(k_segment, *cache, smem, kThreads, &per_sm));
    const uint64_t tiles = N >> m;
    const int threads = std::max(32, std::min(kThreads, 1 << (m > 0 ? m - 1 : 0)));
    const int grid = (int)std::min<uint64_t>(tiles, (uint64_t)sm_count() * 32);
    for (const Segment &s : segs) {
        if (!s.bits) {
            k_pair<<<grid_for(N >> 1), kThreads, 0, st>>>(psi, N, dg, s.g0, __builtin_ctzll(h[s.g0].x));
            continue;
        }
        Tile T{};
        T.m = m;
        T.low = std::min(kLowBits, m);
        int k = 0;
        for (uint64_t b = s.bits; b; b &= b - 1ULL) T.bit[k++] = (uint8_t)__builtin_ctzll(b);
        k_segment<<<grid, threads, smem, st>>>(psi, tiles, dg, s.g0, s.g1, T);
    }
    RQ_CUDA(cudaGetLastError());
    RQ_CUDA(cudaStreamSynchronize(st));  // the host gate list is freed on return
    return RQ_OK;
}
