// Learned warm start: a BF16 MLP (64 -> 256 -> 256 -> 2, GELU) mapping (state, U) to the ground
// state's log-amplitude and sign, trained and evaluated with tcgen05 tensor-core GEMMs.
//
// GEMM (k_gemm: the layers of the separate forward and backward passes): C[M][N] = A[M][K] B[N][K]^T,
// both operands K-major BF16, FP32 accumulators in TMEM.  A persistent CTA takes 128-row tiles with all
// N <= 256 columns; warp 0 fills shared memory by TMA in the 128-byte swizzled layout, one thread of
// warp 1 issues the tcgen05.mma, and eight warps read the accumulator rows back (tcgen05.ld, one row
// per thread, two accumulators in turn) and fuse bias, GELU, the 256 -> 2 output layer, GELU' and the
// bias-gradient column sums.
// Inference (k_infer) and a training step (k_train, k_wgrad: rq_mlp_train.cuh) have fused kernels.
//
// Every mbarrier wait is bounded (about one second of clock cycles); on expiry the kernel records
// RQ_E_CUDA in the error flags, skips the remaining work, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>

#include "rq_common.cuh"
#include "rq_host.h"

namespace rq {
namespace {

typedef __nv_bfloat16 bf16;

constexpr int kIn = RQ_MLP_IN, kHid = RQ_MLP_HIDDEN, kOut = RQ_MLP_OUT;
constexpr int kTileM = 128, kChunkK = 64;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kHid * kIn, kOffW2 = kOffB1 + kHid,
              kOffB2 = kOffW2 + kHid * kHid, kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kOut * kHid,
              kNParams = kOffB3 + kOut;
static_assert(kNParams == RQ_MLP_NPARAMS, "parameter layout");
constexpr int kHeadPart = kHid + kOut * kHid + kOut;  // db2 | dW3 | db3 partial sums per tile
constexpr long long kWaitCycles = 2000000000LL;

enum Epi { EPI_F32 = 0, EPI_HIDDEN = 1, EPI_HEAD = 2, EPI_DGELU = 3 };

// ---------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
// bounded wait for the phase of the given parity; false when the limit expired (the abort flag is
// then set) or when another role has set the abort flag (abort may be null: no early exit)
__device__ __forceinline__ bool wait_bar(uint64_t *bar, uint32_t parity, volatile int *abort) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (abort && *abort) return false;
        if (clock64() - t0 > kWaitCycles) {
            if (abort) *abort = 1;
            return false;
        }
    }
    return true;
}

// the same for a whole warp, with one answer for its lanes: one that gave up alone would miss the
// others' next __syncwarp or tcgen05.ld, which wait for all 32
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort) {
    return __all_sync(0xffffffffu, wait_bar(bar, parity, abort)) != 0;
}

// the workspace's two flags (rqsqd.h): of this call, and of all calls
__device__ __forceinline__ void report_error(int *err) {
    atomicExch(err, RQ_E_CUDA);
    atomicExch(err + 1, RQ_E_CUDA);
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}

// 2-D TMA load of one box (x = column, y = row of the tensor map) into shared memory, completing
// on bar
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];\n" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(nthreads) : "memory");
}
// arrives without waiting (the waiting threads use named_bar_sync with the same count)
__device__ __forceinline__ void named_bar_arrive(int id, int nthreads) {
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(nthreads) : "memory");
}
// barrier over nthreads threads returning the OR of their predicates (the same in every thread)
__device__ __forceinline__ bool named_bar_or(int id, int nthreads, bool p) {
    uint32_t r;
    asm volatile(
        "{\n.reg .pred pi, po;\nsetp.ne.b32 pi, %1, 0;\nbar.red.or.pred po, %2, %3, pi;\nselp.b32 %0, 1, 0, po;\n}\n"
        : "=r"(r)
        : "r"((uint32_t)p), "r"(id), "r"(nthreads)
        : "memory");
    return r != 0;
}

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}

// instruction descriptor of kind::f16: BF16 x BF16 -> FP32, M x N, both K-major (kIdescTransA,
// kIdescTransB: the operand is MN-major)
constexpr uint32_t kIdescTransA = 1u << 15, kIdescTransB = 1u << 16;
__host__ __device__ constexpr uint32_t make_idesc(int M, int N) {
    return (1u << 4)                          // D: FP32
           | (1u << 7)                        // A: BF16
           | (1u << 10)                       // B: BF16
           | ((uint32_t)(N >> 3) << 17)       // N / 8
           | ((uint32_t)(M >> 4) << 24);      // M / 16
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// 32 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        "tcgen05.wait::ld.sync.aligned;\n"  // in the same statement: the outputs exist after the wait
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int q = 0; q < 32; ++q) v[q] = __uint_as_float(r[q]);
}

// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
}

// ---------------------------------------------------------------------------------------------
// activations
// ---------------------------------------------------------------------------------------------
// GELU in its tanh form (Hendrycks and Gimpel): 0.5 z (1 + tanh(k0 (z + k1 z^3))), k0 = sqrt(2 / pi),
// k1 = 0.044715, with the hardware tanh (tanh.approx.f32, relative error about 2^-11, below the BF16
// rounding of the activations): one special-function operation per element for the activation and
// its derivative together
__device__ __forceinline__ float tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
constexpr float kGeluK0 = 0.7978845608028654f;           // sqrt(2 / pi)
constexpr float kGeluK01 = 0.7978845608028654f * 0.044715f;
__device__ __forceinline__ float gelu(float z) {
    return z * fmaf(0.5f, tanh_approx(z * fmaf(kGeluK01, z * z, kGeluK0)), 0.5f);
}
// activation a and derivative d of one pre-activation
__device__ __forceinline__ void gelu_both(float z, float &a, float &d) {
    const float z2 = z * z;
    const float t = tanh_approx(z * fmaf(kGeluK01, z2, kGeluK0));
    const float h = fmaf(0.5f, t, 0.5f);
    a = z * h;
    d = fmaf(0.5f * z * (1.f - t * t), fmaf(3.f * kGeluK01, z2, kGeluK0), h);
}
__device__ __forceinline__ float dgelu(float z) {
    float a, d;
    gelu_both(z, a, d);
    return d;
}

// Two columns at a time: the packed FP32 instructions of sm_100 and later round each half as the scalar
// ones do (the same bits) and take one issue slot for both, which bounds the fused kernels.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 pack2(uint32_t lo, uint32_t hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 x, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(x));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 tanh2(f32x2 x) {
    float a, b;
    unpack2(x, a, b);
    return pack2(tanh_approx(a), tanh_approx(b));
}
__device__ __forceinline__ f32x2 both(float x) { return pack2(x, x); }
__device__ __forceinline__ f32x2 gelu2(f32x2 z) {
    const f32x2 t = tanh2(mul2(z, fma2(both(kGeluK01), mul2(z, z), both(kGeluK0))));
    return mul2(z, fma2(both(0.5f), t, both(0.5f)));
}
__device__ __forceinline__ void gelu_both2(f32x2 z, f32x2 &a, f32x2 &d) {
    const f32x2 z2 = mul2(z, z);
    const f32x2 t = tanh2(mul2(z, fma2(both(kGeluK01), z2, both(kGeluK0))));
    const f32x2 h = fma2(both(0.5f), t, both(0.5f));
    a = mul2(z, h);
    // (-z / 2) (t^2 - 1): the packed forms take no negated operand
    d = fma2(mul2(mul2(both(-0.5f), z), fma2(t, t, both(-1.f))), fma2(both(3.f * kGeluK01), z2, both(kGeluK0)), h);
}
__device__ __forceinline__ uint32_t bf16x2(f32x2 x) {  // both halves rounded to nearest
    float lo, hi;
    unpack2(x, lo, hi);
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// ---------------------------------------------------------------------------------------------
// the GEMM
// ---------------------------------------------------------------------------------------------
constexpr int kGemmThreads = 320;  // warp 0: TMA producer, warp 1: MMA issuer, warps 2..9: epilogue
constexpr int kEpiThreads = 256;
constexpr int kEpiBar = 1;         // named barrier of the epilogue warps (0 is __syncthreads)
constexpr uint32_t kTileABytes = kTileM * kChunkK * 2;

struct GemmArgs {
    int64_t M;        // rows of A; rows >= M are read as zeros (TMA fill) and not stored
    int64_t mtiles;   // ceil(M / 128)
    int64_t nchunks;  // K / 64
    const float *bias;
    bf16 *z_rm;       // pre-activations, row-major [M][N] (HIDDEN, HEAD; optional)
    bf16 *h_rm;       // activations, row-major [M][N] (HIDDEN)
    const bf16 *zin_rm;  // pre-activations read by DGELU, row-major [M][N]
    float *out;          // F32: [M][N]; HEAD: [M][2] (optional)
    const float *w3;     // HEAD: [2][N]
    const float *b3;     // HEAD: [2]
    bf16 *dz_rm;         // DGELU: dZ1, row-major [M][N]
    float *colpart;      // DGELU: [gridDim.x][N] (one row per CTA)
    int *err;
};

template <int N, bool BRES>
struct GemmCfg {
    static constexpr uint32_t kBChunk = (uint32_t)N * kChunkK * 2;  // one 64-wide K chunk of B
    static constexpr int kStages = BRES ? 4 : (N == 256 ? 4 : 8);
    static constexpr uint32_t kStageBytes = kTileABytes + (BRES ? 0u : kBChunk);
};

// epilogue constants in shared memory: bias | W3 row 0 | W3 row 1
template <int N, int EPI>
__host__ __device__ constexpr int const_floats() {
    return EPI == EPI_HIDDEN ? N : (EPI == EPI_HEAD ? 3 * N : 4);
}
// lane l returns sum over the 32 lanes of v[l] (v is consumed): each of the five exchange rounds
// halves the columns a lane keeps, 31 shuffles for 32 column sums, in a fixed order
__device__ __forceinline__ float col_sum32(float (&v)[32], int lane) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float send = up ? v[i] : v[i + o];
            const float keep = up ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

__device__ __forceinline__ void store_bf16x32(bf16 *dst, const float (&v)[32]) {
    __align__(16) bf16 b[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) b[i] = __float2bfloat16_rn(v[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i) reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(b)[i];
}

// 32 consecutive floats of shared memory (16-byte aligned; the same address in every lane)
__device__ __forceinline__ void lds32(const float *p, float (&v)[32]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float4 t = reinterpret_cast<const float4 *>(p)[i];
        v[4 * i] = t.x;
        v[4 * i + 1] = t.y;
        v[4 * i + 2] = t.z;
        v[4 * i + 3] = t.w;
    }
}

// one epilogue thread: row `row` of the tile (its TMEM lane), columns [h N/2, (h + 1) N/2); DGELU: col =
// the running column sums of this thread's row quarter over the CTA's tiles (each slot has one thread)
template <int N, int EPI>
__device__ __forceinline__ void epilogue(const GemmArgs &g, uint32_t taddr, int h, int lane, int row, int64_t m,
                                         bool valid, int par, float (*xch)[kTileM][2],
                                         const float *cst, float *col) {
    constexpr int kHalf = N / 2;
    const int col0 = h * kHalf;
    if constexpr (EPI == EPI_F32) {
#pragma unroll 1
        for (int g0 = 0; g0 < kHalf; g0 += 32) {
            float v[32];
            tmem_ld32(taddr + (uint32_t)(col0 + g0), v);
            if (valid) {
                float4 *dst = reinterpret_cast<float4 *>(g.out + m * N + col0 + g0);
#pragma unroll
                for (int i = 0; i < 8; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        }
    } else if constexpr (EPI == EPI_HIDDEN) {
#pragma unroll 1
        for (int g0 = 0; g0 < kHalf; g0 += 32) {
            const int c0 = col0 + g0;
            float z[32], b[32];
            tmem_ld32(taddr + (uint32_t)c0, z);
            lds32(cst + c0, b);
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                z[i] += b[i];
                b[i] = gelu(z[i]);
            }
            if (valid) {
                if (g.z_rm) store_bf16x32(g.z_rm + m * N + c0, z);
                store_bf16x32(g.h_rm + m * N + c0, b);
            }
        }
    } else if constexpr (EPI == EPI_HEAD) {
        // Z2 = acc + b2, H2 = GELU(Z2), the output layer's dot products over this half
        float o0 = 0.f, o1 = 0.f;
#pragma unroll 1
        for (int g0 = 0; g0 < kHalf; g0 += 32) {
            const int c0 = col0 + g0;
            float z[32], w[32];
            tmem_ld32(taddr + (uint32_t)c0, z);
            lds32(cst + c0, w);
#pragma unroll
            for (int i = 0; i < 32; ++i) z[i] += w[i];
            if (valid && g.z_rm) store_bf16x32(g.z_rm + m * N + c0, z);
#pragma unroll
            for (int i = 0; i < 32; ++i) z[i] = gelu(z[i]);
            lds32(cst + N + c0, w);
#pragma unroll
            for (int i = 0; i < 32; ++i) o0 += z[i] * w[i];
            lds32(cst + 2 * N + c0, w);
#pragma unroll
            for (int i = 0; i < 32; ++i) o1 += z[i] * w[i];
        }
        if (h == 1) {
            xch[par][row][0] = o0;
            xch[par][row][1] = o1;
        }
        named_bar_sync(kEpiBar, kEpiThreads);
        if (h == 0) {
            o0 += xch[par][row][0] + __ldg(g.b3);
            o1 += xch[par][row][1] + __ldg(g.b3 + 1);
            if (valid && g.out) {
                g.out[m * 2] = o0;
                g.out[m * 2 + 1] = o1;
            }
        }
    } else {  // EPI_DGELU: dZ1 = acc * GELU'(Z1) with the column sums of db1
#pragma unroll 1
        for (int g0 = 0; g0 < kHalf; g0 += 32) {
            const int c0 = col0 + g0;
            float v[32];
            tmem_ld32(taddr + (uint32_t)c0, v);
            __align__(16) bf16 zin[32];
            if (valid) {
                const uint4 *src = reinterpret_cast<const uint4 *>(g.zin_rm + m * N + c0);
#pragma unroll
                for (int i = 0; i < 4; ++i) reinterpret_cast<uint4 *>(zin)[i] = src[i];
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = valid ? v[i] * dgelu(__bfloat162float(zin[i])) : 0.f;
            if (valid) store_bf16x32(g.dz_rm + m * N + c0, v);
            col[c0 + lane] += col_sum32(v, lane);
        }
    }
}

// shared-memory matrix descriptor of a K-major operand in the 128-byte swizzled layout that a TMA
// load with CU_TENSOR_MAP_SWIZZLE_128B writes to a 1 KB-aligned tile (rows of 128 B = 64 BF16 of K,
// 8-row atoms of 1 KB in which row r's 16-byte chunks are permuted by r mod 8): stride byte offset
// 1024 between 8-row groups, leading byte offset unused (one MMA's 16-wide K slice lies within a
// row), and the K slice kk of a 64-wide chunk starts 32 kk bytes into the tile (the hardware
// applies the permutation to the address)
__device__ __forceinline__ uint64_t make_sdesc_sw128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;               // leading byte offset, unused
    d |= (uint64_t)(1024u >> 4) << 32;    // stride byte offset
    d |= (uint64_t)1 << 46;               // descriptor version of tcgen05
    d |= (uint64_t)2 << 61;               // swizzle mode: 128 B
    return d;
}

// the same of an MN-major operand: rows of 128 B = 64 consecutive M (or N) at one K, eight K to an atom
// of 1 KB; stride byte offset 1024 to the next eight K, leading byte offset `lead` to the next 64 of
// M (N); one MMA's 16 K are 2048 B
__device__ __forceinline__ uint64_t make_sdesc_mn(uint32_t addr, uint32_t lead) {
    return (make_sdesc_sw128(addr) & ~((uint64_t)0x3FFFu << 16)) | (uint64_t)(lead >> 4) << 16;
}

// C = A B^T over the row tiles of the grid-stride loop.  BRES: B (N x K, K <= 256)
// is loaded once and stays in shared memory; otherwise each stage of the ring holds a 64-wide K
// chunk of A and of B.  Every operand tile is one TMA box of 64 columns (128 B) x its rows.
template <int N, int EPI, bool BRES>
__global__ void __launch_bounds__(kGemmThreads, 1)
k_gemm(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmArgs g) {
    static_assert(N == 64 || N == 256, "N is 64 or 256");
    using C = GemmCfg<N, BRES>;
    constexpr int S = C::kStages;
    constexpr bool kCols = EPI == EPI_DGELU;
    constexpr uint32_t kIdesc = make_idesc(kTileM, N);
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[S], empty[S], tfull[2], tempty[2], bfull, fin;
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s, bwait_s;
    __shared__ long long issued_s, consumed_s;
    __shared__ __align__(16) float cst[const_floats<N, EPI>()];
    __shared__ float xch[EPI == EPI_HEAD ? 2 : 1][kTileM][2];
    __shared__ float csum[4][kCols ? N : 1];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t units = g.mtiles;
    const uint32_t sbase = (smem_u32(smem) + 1023u) & ~1023u;  // the launch adds 1 KB for this
    const uint32_t ring = BRES ? (uint32_t)g.nchunks * C::kBChunk : 0u;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], kEpiThreads / 32);
        }
        mbar_init(&bfull, 1);
        mbar_init(&fin, 1);
        fence_mbar_init();
        abort_s = 0;
        bwait_s = 0;
        issued_s = 0;
        consumed_s = 0;
    }
    if (warp == 1) tmem_alloc(&tmem_s, 2u * N);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s;
    volatile int *abort_p = &abort_s;

    if (warp == 0) {  // ---- TMA producer
        if (BRES && lane == 0) {
            mbar_expect_tx(&bfull, (uint32_t)g.nchunks * C::kBChunk);
            for (int c = 0; c < (int)g.nchunks; ++c)
                tma_load_2d(sbase + (uint32_t)c * C::kBChunk, &tma_b, c * kChunkK, 0, &bfull);
        }
        long long it = 0;
        bool bad = false;
        for (int64_t u = blockIdx.x; u < units && !bad; u += gridDim.x) {
            for (int64_t c = 0; c < g.nchunks; ++c, ++it) {
                const int s = (int)(it % S);
                if (it >= S && !warp_wait(&empty[s], (uint32_t)((it / S - 1) & 1), abort_p)) {
                    bad = true;
                    break;
                }
                if (lane == 0) {
                    const uint32_t st = sbase + ring + (uint32_t)s * C::kStageBytes;
                    mbar_expect_tx(&full[s], C::kStageBytes);
                    tma_load_2d(st, &tma_a, (int)(c * kChunkK), (int)(u * kTileM), &full[s]);
                    if (!BRES) tma_load_2d(st + kTileABytes, &tma_b, (int)(c * kChunkK), 0, &full[s]);
                    issued_s = it + 1;
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {  // ---- MMA issuer
        bool bad = BRES && !warp_wait(&bfull, 0u, abort_p);
        if (BRES && !bad && lane == 0) bwait_s = 1;
        long long it = 0, t = 0;
        for (int64_t u = blockIdx.x; u < units && !bad; u += gridDim.x, ++t) {
            const int b = (int)(t & 1);
            if (t >= 2 && !warp_wait(&tempty[b], (uint32_t)((t / 2 - 1) & 1), abort_p)) break;
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)(b * N);
            for (int64_t c = 0; c < g.nchunks; ++c, ++it) {
                const int s = (int)(it % S);
                if (!warp_wait(&full[s], (uint32_t)((it / S) & 1), abort_p)) {
                    bad = true;
                    break;
                }
                tc_fence_after();
                if (lane == 0) {
                    const uint32_t sa = sbase + ring + (uint32_t)s * C::kStageBytes;
                    const uint32_t sb = BRES ? sbase + (uint32_t)c * C::kBChunk : sa + kTileABytes;
#pragma unroll
                    for (int kk = 0; kk < kChunkK / 16; ++kk)
                        mma_bf16(acc, make_sdesc_sw128(sa + (uint32_t)kk * 32u), make_sdesc_sw128(sb + (uint32_t)kk * 32u),
                                 kIdesc, (c > 0 || kk > 0) ? 1u : 0u);
                    mma_commit(&empty[s]);
                    consumed_s = it + 1;
                }
                __syncwarp();
            }
            if (bad) break;
            if (lane == 0) mma_commit(&tfull[b]);
            __syncwarp();
        }
    } else {  // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 and half (w - 2) / 4 of the columns
        const int q = warp & 3, h = (warp - 2) >> 2, row = 32 * q + lane, e = threadIdx.x - 64;
        if constexpr (const_floats<N, EPI>() > 4) {
            for (int i = e; i < N; i += kEpiThreads) {
                cst[i] = g.bias[i];
                if (EPI != EPI_HIDDEN) {
                    cst[N + i] = g.w3[i];
                    cst[2 * N + i] = g.w3[N + i];
                }
            }
            named_bar_sync(kEpiBar, kEpiThreads);
        }
        if constexpr (kCols)
            for (int k = 0; k < N / 64; ++k) csum[q][h * (N / 2) + 32 * k + lane] = 0.f;
        bool broke = false;
        long long t = 0;
        for (int64_t u = blockIdx.x; u < units; u += gridDim.x, ++t) {
            const int b = (int)(t & 1);
            const bool ok = warp_wait(&tfull[b], (uint32_t)((t >> 1) & 1), abort_p);
            if (named_bar_or(kEpiBar, kEpiThreads, !ok || *abort_p != 0)) {  // the same answer in every epilogue thread
                broke = true;
                break;
            }
            tc_fence_after();
            const int64_t m = u * kTileM + row;
            epilogue<N, EPI>(g, tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(b * N), h, lane, row, m, m < g.M,
                             b, xch, cst, csum[q]);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[b]);
        }
        if (kCols && !broke) {
            // this CTA's column sums: the four row quarters added in order, one row of partials
            named_bar_sync(kEpiBar, kEpiThreads);
            for (int c = e; c < (kCols ? N : 0); c += kEpiThreads)
                g.colpart[(int64_t)blockIdx.x * N + c] = ((csum[0][c] + csum[1][c]) + csum[2][c]) + csum[3][c];
        }
    }
    __syncthreads();
    const bool aborted = abort_s != 0;
    if (aborted) {
        // let the copies and MMAs already issued land before the memory is released
        if (threadIdx.x == 0) {
            for (long long it = consumed_s; it < issued_s; ++it) {
                const int s = (int)(it % S);
                wait_bar(&full[s], (uint32_t)((it / S) & 1), nullptr);
            }
            if (BRES && !bwait_s) wait_bar(&bfull, 0u, nullptr);
            if (g.err) report_error(g.err);
        }
        if (warp == 1) {
            if (lane == 0) mma_commit(&fin);
            __syncwarp();
            wait_bar(&fin, 0u, nullptr);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 2u * N);
    }
}

// cuTensorMapEncodeTiled, from the driver through the runtime (no link against the driver library)
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_fn(EncodeTiledFn *out) {
    static std::atomic<void *> cached{nullptr};
    void *p = cached.load();
    if (!p) {
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        RQ_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !p) return fail(RQ_E_CUDA, "cuTensorMapEncodeTiled not available");
        cached.store(p);
    }
    *out = reinterpret_cast<EncodeTiledFn>(p);
    return RQ_OK;
}

// BF16 matrix of `rows` rows x `cols` columns (row stride ld elements, cols a multiple of 64) read
// in boxes of 64 columns x box_rows rows with the 128-byte swizzle; rows past the end read as zeros
int make_tma(CUtensorMap *map, const bf16 *base, int64_t cols, int64_t rows, int64_t ld, int box_rows) {
    if (reinterpret_cast<uintptr_t>(base) % 16 != 0 || ld % 8 != 0 || cols % kChunkK != 0)
        return fail(RQ_E_ARG, "bf16 GEMM: operands need 16-byte aligned rows");
    EncodeTiledFn enc = nullptr;
    RQ_TRY(encode_fn(&enc));
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kChunkK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1u, 1u};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16 *>(base), dims, strides, box,
                           estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(RQ_E_CUDA, "cuTensorMapEncodeTiled failed");
    return RQ_OK;
}

// A [M][K] (lda), B [N][K] (ldb), K a multiple of 64; g.M and the epilogue fields set by
// the caller; *grid_out (optional) = the CTAs launched (rows of the per-CTA partial sums)
template <int N, int EPI, bool BRES>
int launch_gemm_t(const bf16 *A, int64_t lda, const bf16 *B, int64_t ldb, int64_t K, GemmArgs g, cudaStream_t st,
                  int64_t *grid_out) {
    using C = GemmCfg<N, BRES>;
    if (g.M < 1 || K < kChunkK || K % kChunkK != 0 || (BRES && K > 256))
        return fail(RQ_E_ARG, "bf16 GEMM: bad shape");
    g.mtiles = (g.M + kTileM - 1) / kTileM;
    g.nchunks = K / kChunkK;
    CUtensorMap ta, tb;
    RQ_TRY(make_tma(&ta, A, K, g.M, lda, kTileM));
    RQ_TRY(make_tma(&tb, B, K, N, ldb, N));
    uint32_t smem = BRES ? (uint32_t)g.nchunks * C::kBChunk + C::kStages * kTileABytes : C::kStages * C::kStageBytes;
    smem += 1024;  // alignment of the operand tiles to 1 KB
    if (N == 256 && smem < 116u * 1024u) smem = 116u * 1024u;  // one CTA per SM: its 512 TMEM columns are all of them
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    KernelLaunchCache *c = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &c));
    RQ_TRY(configure_kernel(k_gemm<N, EPI, BRES>, *c, smem, kGemmThreads, &per_sm));
    const int64_t units = g.mtiles;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    const int64_t grid = units < cap ? units : cap;
    if (grid > 0x7FFFFFFF) return fail(RQ_E_RANGE, "bf16 GEMM: grid out of range");
    k_gemm<N, EPI, BRES><<<(unsigned)grid, kGemmThreads, smem, st>>>(ta, tb, g);
    RQ_CUDA(cudaGetLastError());
    if (grid_out) *grid_out = grid;
    return RQ_OK;
}

template <int N, int EPI>
int launch_gemm(const bf16 *A, int64_t lda, const bf16 *B, int64_t ldb, int64_t K, const GemmArgs &g,
                cudaStream_t st, int64_t *grid_out = nullptr) {
    if constexpr (EPI == EPI_F32) {  // K <= 256: B stays in shared memory; else B streams with A
        if (K <= 256) return launch_gemm_t<N, EPI, true>(A, lda, B, ldb, K, g, st, grid_out);
        return launch_gemm_t<N, EPI, false>(A, lda, B, ldb, K, g, st, grid_out);
    } else {  // the layer GEMMs: K = 64 or 256
        return launch_gemm_t<N, EPI, true>(A, lda, B, ldb, K, g, st, grid_out);
    }
}

// ---------------------------------------------------------------------------------------------
// fused inference
// ---------------------------------------------------------------------------------------------
// Both layers and the output layer of a 128-row tile in one persistent kernel: the hidden activations
// H1 go from the epilogue warps to shared memory (the 128-byte swizzled layout that the MMA reads) and
// never to HBM; as two GEMMs they were written and read back, 134 MB each way for 2^18 rows.  W1 and
// W2 (160 KB) stay in shared memory, which leaves one tile of X (16 KB) and two of H1's four 64-column
// quarters (32 KB).  TMEM holds both accumulators (2 x 256 columns).  Bound by the epilogue warps,
// about 8 instructions per hidden unit of each layer: sixteen of them (eight left three of four issue
// slots empty).  2^18 rows: 113 us as two GEMMs, 100 with eight epilogue warps, 80 with sixteen, 75 with
// the packed instructions.
constexpr uint32_t kInfW2 = 0, kInfW1 = 4 * 32768, kInfA = kInfW1 + 32768, kInfH = kInfA + kTileABytes,
                   kInfEnd = kInfH + 2 * kTileABytes;  // 208 KB
constexpr int kInfWarps = 16;                  // epilogue warps
constexpr int kInfThreads = 64 + 32 * kInfWarps;

struct InferArgs {
    int64_t M, tiles;
    const float *params;
    float *out;  // [M][2]
    int *err;
};

struct InferShared {
    uint64_t wfull, afull, aempty, d1full, d1empty, d2full, d2empty, hfull[2], hempty[2], fin;
    uint32_t tmem;
    int abort, wwait;
    int64_t issued, consumed;  // X tiles
    __align__(16) float cst[4 * kHid];     // b1 | b2 | W3 row 0 | W3 row 1
    float xch[2][3][kTileM][2];            // output sums: quarters 0 and 2, then 2 and 3 together
};

__global__ void __launch_bounds__(kInfThreads, 1)
k_infer(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w1,
        const __grid_constant__ CUtensorMap tma_w2, const InferArgs g) {
    // all of it dynamic, so that the operand tiles start at the beginning of the block's memory,
    // which is 1 KB aligned (checked: there is no room for slack)
    extern __shared__ __align__(1024) unsigned char smem[];
    InferShared &sh = *reinterpret_cast<InferShared *>(smem + kInfEnd);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sbase = smem_u32(smem);
    constexpr uint32_t kIdesc = make_idesc(kTileM, kHid);
    if ((sbase & 1023u) != 0u) {
        if (threadIdx.x == 0) report_error(g.err);
        return;
    }
    if (threadIdx.x == 0) {
        mbar_init(&sh.wfull, 1);
        mbar_init(&sh.afull, 1);
        mbar_init(&sh.aempty, 1);
        mbar_init(&sh.d1full, 1);
        mbar_init(&sh.d1empty, kInfWarps);
        mbar_init(&sh.d2full, 1);
        mbar_init(&sh.d2empty, kInfWarps);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&sh.hfull[s], kInfWarps);
            mbar_init(&sh.hempty[s], 1);
        }
        mbar_init(&sh.fin, 1);
        fence_mbar_init();
        sh.abort = sh.wwait = 0;
        sh.issued = sh.consumed = 0;
    }
    if (warp == 1) tmem_alloc(&sh.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    volatile int *abort_p = &sh.abort;

    if (warp == 0) {  // ---- TMA producer
        if (lane == 0) {
            mbar_expect_tx(&sh.wfull, 5 * 32768);
            tma_load_2d(sbase + kInfW1, &tma_w1, 0, 0, &sh.wfull);
            for (int c = 0; c < 4; ++c) tma_load_2d(sbase + kInfW2 + 32768u * (uint32_t)c, &tma_w2, c * kChunkK, 0, &sh.wfull);
        }
        int64_t it = 0;
        for (int64_t u = blockIdx.x; u < g.tiles; u += gridDim.x, ++it) {
            if (it >= 1 && !warp_wait(&sh.aempty, (uint32_t)((it - 1) & 1), abort_p)) break;
            if (lane == 0) {
                mbar_expect_tx(&sh.afull, kTileABytes);
                tma_load_2d(sbase + kInfA, &tma_x, 0, (int)(u * kTileM), &sh.afull);
                sh.issued = it + 1;
            }
            __syncwarp();
        }
    } else if (warp == 1) {  // ---- MMA issuer
        bool ok = warp_wait(&sh.wfull, 0u, abort_p);
        if (ok && lane == 0) sh.wwait = 1;
        int64_t it = 0, hq = 0;
        for (int64_t u = blockIdx.x; u < g.tiles && ok; u += gridDim.x, ++it) {
            ok = warp_wait(&sh.afull, (uint32_t)(it & 1), abort_p) &&
                 (it < 1 || warp_wait(&sh.d1empty, (uint32_t)((it - 1) & 1), abort_p));
            if (!ok) break;
            tc_fence_after();
            if (lane == 0) {
#pragma unroll
                for (int kk = 0; kk < kChunkK / 16; ++kk)
                    mma_bf16(tmem, make_sdesc_sw128(sbase + kInfA + (uint32_t)kk * 32u),
                             make_sdesc_sw128(sbase + kInfW1 + (uint32_t)kk * 32u), kIdesc, kk > 0 ? 1u : 0u);
                mma_commit(&sh.aempty);
                mma_commit(&sh.d1full);
                sh.consumed = it + 1;
            }
            __syncwarp();
            if (it >= 1 && !warp_wait(&sh.d2empty, (uint32_t)((it - 1) & 1), abort_p)) break;
            for (int q = 0; q < 4; ++q, ++hq) {
                const int s = (int)(hq & 1);
                ok = warp_wait(&sh.hfull[s], (uint32_t)((hq >> 1) & 1), abort_p);
                if (!ok) break;
                tc_fence_after();
                if (lane == 0) {
                    const uint32_t a = sbase + kInfH + kTileABytes * (uint32_t)s, b = sbase + kInfW2 + 32768u * (uint32_t)q;
#pragma unroll
                    for (int kk = 0; kk < kChunkK / 16; ++kk)
                        mma_bf16(tmem + kHid, make_sdesc_sw128(a + (uint32_t)kk * 32u), make_sdesc_sw128(b + (uint32_t)kk * 32u),
                                 kIdesc, (q > 0 || kk > 0) ? 1u : 0u);
                    mma_commit(&sh.hempty[s]);
                    if (q == 3) mma_commit(&sh.d2full);
                }
                __syncwarp();
            }
        }
    } else {  // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31; quarter (w - 2) / 4 of the columns
        const int q4 = warp & 3, cq = (warp - 2) >> 2, row = 32 * q4 + lane, e = threadIdx.x - 64;
        constexpr int kThreadsE = 32 * kInfWarps;
        const uint32_t lanes = tmem + ((uint32_t)(32 * q4) << 16);
        for (int i = e; i < kHid; i += kThreadsE) {
            sh.cst[i] = g.params[kOffB1 + i];
            sh.cst[kHid + i] = g.params[kOffB2 + i];
            sh.cst[2 * kHid + i] = g.params[kOffW3 + i];
            sh.cst[3 * kHid + i] = g.params[kOffW3 + kHid + i];
        }
        named_bar_sync(kEpiBar, kThreadsE);
        int64_t it = 0, hq = 0;
        for (int64_t u = blockIdx.x; u < g.tiles; u += gridDim.x, ++it) {
            // a wait that gives up changes nothing until the vote below, when the tile is dropped: lanes that
            // left the path alone would miss what waits for all 32 of them
            bool ok = wait_bar(&sh.d1full, (uint32_t)(it & 1), abort_p);
            tc_fence_after();
            for (int q = 0; q < 4; ++q, ++hq) {  // H1 quarter by quarter; this warp's 16 columns of it
                const int s = (int)(hq & 1);
                const int c0 = 64 * q + 16 * cq;
                float z[16];
                tmem_ld16(lanes + (uint32_t)c0, z);
                if (q == 3) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.d1empty);
                }
                __align__(16) uint32_t o[8];
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(sh.cst + c0 + i);
                    o[i / 2] = bf16x2(gelu2(add2(pack2(z[i], z[i + 1]), b.x)));
                    o[i / 2 + 1] = bf16x2(gelu2(add2(pack2(z[i + 2], z[i + 3]), b.y)));
                }
                // 16-byte chunk c of row r sits at chunk c ^ (r mod 8) of the row's 128 bytes
                unsigned char *dst = smem + kInfH + kTileABytes * (uint32_t)s + row * 128;
                if (hq >= 2 && !wait_bar(&sh.hempty[s], (uint32_t)(((hq >> 1) - 1) & 1), abort_p)) ok = false;
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    *reinterpret_cast<uint4 *>(dst + (((2 * cq + j) ^ (row & 7)) << 4)) = reinterpret_cast<const uint4 *>(o)[j];
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the MMA reads through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.hfull[s]);
            }
            ok = ok && wait_bar(&sh.d2full, (uint32_t)(it & 1), abort_p);
            if (named_bar_or(kEpiBar, kThreadsE, !ok || *abort_p != 0)) break;  // the same answer in every epilogue thread
            tc_fence_after();
            // Z2 = acc + b2, H2 = GELU(Z2) of this quarter, and the output layer's dot products in the
            // order of the forward pass: over each half's 128 columns, then the halves.  An odd
            // quarter holds its activations and goes on from the sums of the even one before it,
            // which has gone to the next tile by then.
            float z[2][32];
            const int c0 = cq * (kHid / 4);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                tmem_ld32(lanes + (uint32_t)(kHid + c0 + 32 * k), z[k]);
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(sh.cst + kHid + c0 + 32 * k + i);
                    unpack2(gelu2(add2(pack2(z[k][i], z[k][i + 1]), b.x)), z[k][i], z[k][i + 1]);
                    unpack2(gelu2(add2(pack2(z[k][i + 2], z[k][i + 3]), b.y)), z[k][i + 2], z[k][i + 3]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.d2empty);
            float o0 = 0.f, o1 = 0.f;
            float (*x)[kTileM][2] = sh.xch[it & 1];
            if (cq & 1) {
                named_bar_sync(kEpiBar + 1, kThreadsE);
                o0 = x[cq >> 1][row][0];
                o1 = x[cq >> 1][row][1];
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 a = *reinterpret_cast<const float4 *>(sh.cst + 2 * kHid + c0 + 32 * k + i);
                    const float4 b = *reinterpret_cast<const float4 *>(sh.cst + 3 * kHid + c0 + 32 * k + i);
                    o0 += z[k][i] * a.x;
                    o1 += z[k][i] * b.x;
                    o0 += z[k][i + 1] * a.y;
                    o1 += z[k][i + 1] * b.y;
                    o0 += z[k][i + 2] * a.z;
                    o1 += z[k][i + 2] * b.z;
                    o0 += z[k][i + 3] * a.w;
                    o1 += z[k][i + 3] * b.w;
                }
            if (!(cq & 1)) {
                x[cq >> 1][row][0] = o0;
                x[cq >> 1][row][1] = o1;
                named_bar_arrive(kEpiBar + 1, kThreadsE);
            } else if (cq == 3) {
                x[2][row][0] = o0;
                x[2][row][1] = o1;
                named_bar_arrive(kEpiBar + 2, kThreadsE / 2);
            } else {
                named_bar_sync(kEpiBar + 2, kThreadsE / 2);
                const int64_t m = u * kTileM + row;
                o0 += x[2][row][0] + __ldg(g.params + kOffB3);
                o1 += x[2][row][1] + __ldg(g.params + kOffB3 + 1);
                if (m < g.M) {
                    g.out[2 * m] = o0;
                    g.out[2 * m + 1] = o1;
                }
            }
        }
    }
    __syncthreads();
    if (sh.abort != 0) {
        // let the copies and MMAs already issued land before the memory is released
        if (threadIdx.x == 0) {
            if (sh.consumed < sh.issued) wait_bar(&sh.afull, (uint32_t)((sh.issued - 1) & 1), nullptr);
            if (!sh.wwait) wait_bar(&sh.wfull, 0u, nullptr);
            report_error(g.err);
        }
        if (warp == 1) {
            if (lane == 0) mma_commit(&sh.fin);
            __syncwarp();
            wait_bar(&sh.fin, 0u, nullptr);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

int launch_infer(const rq_mlp_t *m, int64_t rows, const bf16 *x, float *out, int *err, cudaStream_t st) {
    CUtensorMap tx, t1, t2;
    RQ_TRY(make_tma(&tx, x, kIn, rows, kIn, kTileM));
    RQ_TRY(make_tma(&t1, reinterpret_cast<const bf16 *>(m->w1b), kIn, kHid, kIn, kHid));
    RQ_TRY(make_tma(&t2, reinterpret_cast<const bf16 *>(m->w2b), kHid, kHid, kHid, kHid));
    constexpr size_t smem = kInfEnd + sizeof(InferShared);
    static_assert(smem <= 227 * 1024, "one block's shared memory");
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    KernelLaunchCache *c = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &c));
    RQ_TRY(configure_kernel(k_infer, *c, smem, kInfThreads, &per_sm));
    const InferArgs g{rows, (rows + kTileM - 1) / kTileM, m->params, out, err};
    k_infer<<<(unsigned)std::min<int64_t>(g.tiles, sm_count()), kInfThreads, smem, st>>>(tx, t1, t2, g);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

#include "rq_mlp_train.cuh"

// ---------------------------------------------------------------------------------------------
// elementwise kernels
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {  // SplitMix64 finaliser
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

__device__ __forceinline__ float feature(uint64_t s, double u, int f) {
    if (f < 32) return ((s >> f) & 1ULL) ? 1.f : -1.f;
    if (f == 32) return (float)u;
    if (f == 33) return (float)(u * u);
    if (f == 34) return (float)(u * u * u);
    return 0.f;
}

__device__ __forceinline__ void write_features(bf16 *row, uint64_t s, double u) {
#pragma unroll
    for (int f0 = 0; f0 < kIn; f0 += 8) {
        __align__(16) bf16 b[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) b[q] = __float2bfloat16_rn(feature(s, u, f0 + q));
        *reinterpret_cast<uint4 *>(row + f0) = *reinterpret_cast<const uint4 *>(b);
    }
}

// A thread per 16-byte piece of a row, so that a warp writes 512 contiguous bytes; the features of U
// are computed once, on the host (FP64 arithmetic per row took half of the kernel: 14.5 -> 8.4 us for
// 2^18 rows).
struct UFeatures {
    float u[3];
};
__global__ void k_features(const uint64_t *__restrict__ S, int64_t D, const UFeatures f, bf16 *__restrict__ x) {
    constexpr int kPieces = kIn / 8;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < D * kPieces; k += (int64_t)gridDim.x * blockDim.x) {
        const int p = (int)(k % kPieces);
        __align__(16) bf16 b[8];
        if (p < 4) {
            const uint32_t s = (uint32_t)(__ldg(S + k / kPieces) >> (8 * p));
#pragma unroll
            for (int q = 0; q < 8; ++q) b[q] = __float2bfloat16_rn((s >> q) & 1u ? 1.f : -1.f);
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) b[q] = __float2bfloat16_rn(p == 4 && q < 3 ? f.u[q < 3 ? q : 0] : 0.f);
        }
        *reinterpret_cast<uint4 *>(x + k * 8) = *reinterpret_cast<const uint4 *>(b);
    }
}

__global__ void k_sample(const uint64_t *__restrict__ S, int64_t D, const double *__restrict__ U,
                         const float *__restrict__ psi, int P, uint64_t seed, int64_t step, int64_t rows,
                         bf16 *__restrict__ x, bf16 *__restrict__ xt, float *__restrict__ tgt) {
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < rows; m += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t r = mix64(seed ^ mix64((uint64_t)step * 0x100000001B3ULL + (uint64_t)m));
        const int i = (int)((r >> 32) % (uint64_t)P);
        const int64_t k = (int64_t)((r & 0xFFFFFFFFULL) % (uint64_t)D);
        const uint64_t s = S[k];
        const double u = (U[i] - 5.0) / 3.0;
        write_features(x + m * kIn, s, u);
        for (int f = 0; f < kIn; ++f) xt[(int64_t)f * rows + m] = __float2bfloat16_rn(feature(s, u, f));
        const float p = psi[(int64_t)i * D + k];
        const float ap = fabsf(p);
        const float a = logf(fmaxf(ap, 1e-30f)) + 0.5f * logf((float)D);
        const float w = fminf(fmaxf((float)D * p * p, 0.05f), 20.f);
        tgt[m * 3] = fmaxf(a, -30.f);
        tgt[m * 3 + 1] = p < 0.f ? -1.f : 1.f;
        tgt[m * 3 + 2] = w;
    }
}

// loss and its gradient; one partial sum per block (summed in block order by k_loss_sum)
__global__ void k_loss(int64_t rows, const float *__restrict__ out, const float *__restrict__ tgt,
                       float *__restrict__ dout, double *__restrict__ part) {
    __shared__ double red[kThreads / 32];
    const float inv = 1.f / (float)rows;
    double acc = 0.;
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < rows; m += (int64_t)gridDim.x * blockDim.x) {
        const float o0 = out[m * 2], o1 = out[m * 2 + 1];
        const float a = tgt[m * 3], sg = tgt[m * 3 + 1], w = tgt[m * 3 + 2];
        const float e = o0 - a;
        const float t = -sg * o1;
        const float sp = t > 20.f ? t : log1pf(expf(t));  // softplus(-s o1)
        const float sig = 1.f / (1.f + expf(-t));         // sigmoid(-s o1)
        acc += (double)(w * (e * e + sp));
        dout[m * 2] = w * inv * 2.f * e;
        dout[m * 2 + 1] = -w * inv * sg * sig;
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        part[blockIdx.x] = s;
    }
}

// loss = sum of the n partial sums / rows: thread t adds part[t], part[t + 256], ... in order, then
// a fixed tree over the threads (the same sum on every run)
struct LossSum {
    const double *part;
    int n;
    int64_t rows;
    double *loss;  // null: no sum
};
__device__ __forceinline__ void loss_sum(const LossSum &L) {
    __shared__ double red[kThreads];
    double s = 0.;
    for (int i = threadIdx.x; i < L.n; i += kThreads) s += L.part[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *L.loss = red[0] / (double)L.rows;
}
__global__ void __launch_bounds__(kThreads) k_loss_sum(const LossSum L) { loss_sum(L); }

// backward through the output layer: thread j = hidden unit j, 128 rows per block
__global__ void __launch_bounds__(kHid) k_head_bwd(const bf16 *__restrict__ z2, const float *__restrict__ dout,
                                                   const float *__restrict__ params,
                                                   bf16 *__restrict__ dz2_rm, float *__restrict__ part) {
    __shared__ float d_s[kTileM][2];
    const int64_t m0 = (int64_t)blockIdx.x * kTileM;
    for (int i = threadIdx.x; i < kTileM * 2; i += blockDim.x) d_s[i >> 1][i & 1] = dout[m0 * 2 + i];
    __syncthreads();
    const int j = threadIdx.x;
    const float w30 = params[kOffW3 + j], w31 = params[kOffW3 + kHid + j];
    float aw0 = 0.f, aw1 = 0.f, ab = 0.f;
    for (int r0 = 0; r0 < kTileM; r0 += 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int64_t m = m0 + r0 + q;
            const float z = __bfloat162float(z2[m * kHid + j]);
            const float h = gelu(z);
            const float d0 = d_s[r0 + q][0], d1 = d_s[r0 + q][1];
            const float dz = (d0 * w30 + d1 * w31) * dgelu(z);
            dz2_rm[m * kHid + j] = __float2bfloat16_rn(dz);
            aw0 += d0 * h;
            aw1 += d1 * h;
            ab += dz;
        }
    }
    float *p = part + (int64_t)blockIdx.x * kHeadPart;
    p[j] = ab;
    p[kHid + j] = aw0;
    p[2 * kHid + j] = aw1;
    if (j < kOut) {
        float s = 0.f;
        for (int r = 0; r < kTileM; ++r) s += d_s[r][j];
        p[3 * kHid + j] = s;
    }
}

// Bound by the latency of its reads (31 MB of partials for 65,536 rows): kColsumRows rows are in flight
// per lane (two: 11.2 us; eight, with the loss sum that was a launch of 4.6 us: 9.9 us).
// dst[c] = sum_t part[t * ncols + c] for up to four sets of partial sums in one launch: a block
// of kColsumWarps warps per 32 VW columns of one set (lane = VW consecutive columns, so every row
// of partials is read in 32 VW-wide coalesced pieces); warp w adds the rows t in its contiguous
// range with two interleaved accumulators, then the warp sums are added in warp order.  The
// order of every addition is fixed, so the sums are the same on every run.  VW = 4 needs ncols a
// multiple of 4 and 16-byte aligned rows.
constexpr int kColsumWarps = 8;
constexpr int kColsumRows = 8;  // even
struct ColsumSet {
    const float *part;
    int64_t nt, ncols;
    float *dst;
    int vw;      // 4 or 1
    int blocks;  // blocks of the launch that serve this set
};
struct ColsumSets {
    ColsumSet s[4];
    int n;
};

template <int VW>
__device__ __forceinline__ void colsum_block(const ColsumSet &g, int64_t blk, float (*ws)[32 * 4 + 1]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t nt = g.nt, ncols = g.ncols;
    const float *part = g.part;
    const int64_t c = (blk * 32 + lane) * VW;
    const int64_t t0 = w * nt / kColsumWarps, t1 = (w + 1) * nt / kColsumWarps;
    float a[2][VW] = {};
    if (c < ncols) {
        int64_t t = t0;
        for (; t + kColsumRows <= t1; t += kColsumRows) {  // rows in flight together
            float v[kColsumRows][VW];
#pragma unroll
            for (int k = 0; k < kColsumRows; ++k) {
                if constexpr (VW == 4) {
                    const float4 f = __ldg(reinterpret_cast<const float4 *>(part + (t + k) * ncols + c));
                    v[k][0] = f.x;
                    v[k][1] = f.y;
                    v[k][2] = f.z;
                    v[k][3] = f.w;
                } else {
                    v[k][0] = __ldg(part + (t + k) * ncols + c);
                }
            }
#pragma unroll
            for (int k = 0; k < kColsumRows; ++k)
#pragma unroll
                for (int j = 0; j < VW; ++j) a[k & 1][j] += v[k][j];
        }
        for (; t + 2 <= t1; t += 2) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if constexpr (VW == 4) {
                    const float4 v = __ldg(reinterpret_cast<const float4 *>(part + (t + k) * ncols + c));
                    a[k][0] += v.x;
                    a[k][1] += v.y;
                    a[k][2] += v.z;
                    a[k][3] += v.w;
                } else {
                    a[k][0] += __ldg(part + (t + k) * ncols + c);
                }
            }
        }
        if (t < t1) {
            if constexpr (VW == 4) {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(part + t * ncols + c));
                a[0][0] += v.x;
                a[0][1] += v.y;
                a[0][2] += v.z;
                a[0][3] += v.w;
            } else {
                a[0][0] += __ldg(part + t * ncols + c);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < VW; ++j) ws[w][lane * VW + j] = a[0][j] + a[1][j];
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * VW; i += blockDim.x) {
        const int64_t ci = blk * 32 * VW + i;
        if (ci < ncols) {
            float s = 0.f;
            for (int k = 0; k < kColsumWarps; ++k) s += ws[k][i];
            g.dst[ci] = s;
        }
    }
}

__global__ void __launch_bounds__(kColsumWarps * 32) k_colsum(const ColsumSets S, const LossSum L) {
    static_assert(kColsumWarps * 32 == kThreads, "the blocks of loss_sum");
    __shared__ float ws[kColsumWarps][32 * 4 + 1];
    int64_t b = blockIdx.x;
    int k = 0;
    while (k < S.n && b >= S.s[k].blocks) b -= S.s[k++].blocks;
    if (k == S.n)  // the block after the last set's
        loss_sum(L);
    else if (S.s[k].vw == 4)
        colsum_block<4>(S.s[k], b, ws);
    else
        colsum_block<1>(S.s[k], b, ws);
}

// the column sums of n (<= 4) sets of partials and, where wanted, the loss, one launch
int launch_colsums(const ColsumSet *sets, int n, const LossSum &loss, cudaStream_t st) {
    ColsumSets S{};
    S.n = n;
    int64_t total = 0;
    for (int k = 0; k < n; ++k) {
        S.s[k] = sets[k];
        S.s[k].vw = (sets[k].ncols % 4 == 0 && reinterpret_cast<uintptr_t>(sets[k].part) % 16 == 0) ? 4 : 1;
        S.s[k].blocks = (int)((sets[k].ncols + 32 * S.s[k].vw - 1) / (32 * S.s[k].vw));
        total += S.s[k].blocks;
    }
    if (n < 1 || n > 4 || total < 1 || total >= 0x7FFFFFFF) return fail(RQ_E_RANGE, "column sums: bad sets");
    k_colsum<<<(unsigned)(total + (loss.loss ? 1 : 0)), kColsumWarps * 32, 0, st>>>(S, loss);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

__device__ __forceinline__ void write_bf16_copies(const rq_mlp_t &M, int i, float p) {
    if (i >= kOffW1 && i < kOffB1) {
        M.w1b[i - kOffW1] = __bfloat16_as_ushort(__float2bfloat16_rn(p));
    } else if (i >= kOffW2 && i < kOffB2) {
        const int e = i - kOffW2, n = e / kHid, k = e % kHid;
        const unsigned short b = __bfloat16_as_ushort(__float2bfloat16_rn(p));
        M.w2b[e] = b;
        M.w2tb[k * kHid + n] = b;
    }
}

__global__ void k_sync(const rq_mlp_t M) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNParams; i += gridDim.x * blockDim.x)
        write_bf16_copies(M, i, M.params[i]);
}

__global__ void k_adam(const rq_mlp_t M, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNParams; i += gridDim.x * blockDim.x) {
        const float g = M.grads[i];
        const float m = b1 * M.adam_m[i] + (1.f - b1) * g;
        const float v = b2 * M.adam_v[i] + (1.f - b2) * g * g;
        M.adam_m[i] = m;
        M.adam_v[i] = v;
        const float p = M.params[i] - lr * (m / c1) / (sqrtf(v / c2) + eps);
        M.params[i] = p;
        write_bf16_copies(M, i, p);
    }
}

template <typename V>
__global__ void k_warm_start(int64_t D, const float *__restrict__ out, V *__restrict__ x0) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < D; k += (int64_t)gridDim.x * blockDim.x) {
        const float a = fminf(out[k * 2], 30.f);
        const double v = (out[k * 2 + 1] < 0.f ? -1.0 : 1.0) * exp((double)a);
        VT<V>::st(x0, k, cx<typename VT<V>::R>{(typename VT<V>::R)v, (typename VT<V>::R)0});
    }
}

// ---------------------------------------------------------------------------------------------
// workspace layout for `rows` rows (Mp = rows rounded up to 128)
// ---------------------------------------------------------------------------------------------
struct MlpLayout {
    int64_t Mp, tiles, nsplit, nsplit1;
    size_t err, z1, h1, z2, dz2, dz1, colpart1, part2, split2, split1, lossp, total;
};


MlpLayout mlp_layout(int64_t rows) {
    MlpLayout L{};
    L.Mp = (rows + kTileM - 1) / kTileM * kTileM;
    L.tiles = L.Mp / kTileM;
    L.nsplit = std::min<int64_t>(kSplitK, L.Mp / kChunkK);       // dW2: 2 row tiles x nsplit units
    L.nsplit1 = std::min<int64_t>(2 * kSplitK, L.Mp / kChunkK);  // dW1: 1 row tile x nsplit1 units
    size_t off = 0;
    auto take = [&](size_t n) {
        const size_t o = off;
        off += (n + 255) & ~size_t(255);
        return o;
    };
    const size_t act = (size_t)L.Mp * kHid * sizeof(bf16);
    L.err = take(16);
    L.z1 = take(act);
    L.h1 = take(act);
    L.z2 = take(act);
    L.dz2 = take(act);
    L.dz1 = take(act);
    L.colpart1 = take((size_t)L.tiles * kHid * sizeof(float));  // one row per tile (k_head_bwd) or CTA
    L.part2 = take((size_t)L.tiles * kHeadPart * sizeof(float));
    L.split2 = take((size_t)L.nsplit * kHid * kHid * sizeof(float));
    L.split1 = take((size_t)L.nsplit1 * kHid * kIn * sizeof(float));
    L.lossp = take((size_t)std::max<int64_t>(4096, L.tiles) * sizeof(double));
    L.total = off;
    return L;
}

int check_mlp(const rq_mlp_t *m) {
    if (!m || !m->params || !m->w1b || !m->w2b || !m->w2tb) return fail(RQ_E_ARG, "rq_mlp: null parameter arrays");
    return RQ_OK;
}

int grid_for(int64_t n, int threads = kThreads) {
    int64_t g = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * 16;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace
}  // namespace rq

using namespace rq;

RQ_API int rq_mlp_workspace_size(int64_t rows, size_t *bytes) {
    if (rows < 1 || !bytes) return fail(RQ_E_ARG, "rq_mlp_workspace_size: bad arguments");
    *bytes = mlp_layout(rows).total;
    return RQ_OK;
}

RQ_API int rq_mlp_sync(const rq_mlp_t *m, void *stream) {
    RQ_TRY(check_mlp(m));
    k_sync<<<grid_for(kNParams), kThreads, 0, as_stream(stream)>>>(*m);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

RQ_API int rq_mlp_features(const uint64_t *states, int64_t D, double U, uint16_t *x, void *stream) {
    if (!states || !x || D < 1) return fail(RQ_E_ARG, "rq_mlp_features: bad arguments");
    const double u = (U - 5.0) / 3.0;
    const UFeatures f{{(float)u, (float)(u * u), (float)(u * u * u)}};
    k_features<<<grid_for(D * (kIn / 8)), kThreads, 0, as_stream(stream)>>>(states, D, f, reinterpret_cast<bf16 *>(x));
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

RQ_API int rq_mlp_sample(const uint64_t *states, int64_t D, const double *U, const float *psi, int32_t P,
                         uint64_t seed, int64_t step, int64_t rows, uint16_t *x, uint16_t *xt, float *tgt,
                         void *stream) {
    if (!states || !U || !psi || !x || !xt || !tgt || D < 1 || P < 1 || rows < 1)
        return fail(RQ_E_ARG, "rq_mlp_sample: bad arguments");
    k_sample<<<grid_for(rows), kThreads, 0, as_stream(stream)>>>(states, D, U, psi, P, seed, step, rows,
                                                                 reinterpret_cast<bf16 *>(x),
                                                                 reinterpret_cast<bf16 *>(xt), tgt);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

namespace rq {
namespace {

// layer 1: Z1 = X W1^T + b1 and H1 = GELU(Z1)
int layer1(const rq_mlp_t *m, int64_t rows, const uint16_t *x, const MlpLayout &L, char *w, int *err,
           cudaStream_t st) {
    GemmArgs g{};
    g.M = rows;
    g.bias = m->params + kOffB1;
    g.z_rm = reinterpret_cast<bf16 *>(w + L.z1);
    g.h_rm = reinterpret_cast<bf16 *>(w + L.h1);
    g.err = err;
    return launch_gemm<kHid, EPI_HIDDEN>(reinterpret_cast<const bf16 *>(x), kIn,
                                         reinterpret_cast<const bf16 *>(m->w1b), kIn, kIn, g, st);
}

// dW2 = dZ2^T H1 and dW1 = dZ1^T X split over the rows, and the sums of every set of partials (b1's of
// np1, the head's of np2 rows) into m->grads; with loss, the sum of its np2 partials there
int weight_grads(const rq_mlp_t *m, int64_t rows, const uint16_t *xt, const MlpLayout &L, char *w, int *err,
                 int64_t np1, int64_t np2, double *loss, cudaStream_t st) {
    RQ_TRY(launch_wgrad(reinterpret_cast<const bf16 *>(w + L.h1), reinterpret_cast<const bf16 *>(w + L.dz2),
                        reinterpret_cast<const bf16 *>(xt), reinterpret_cast<const bf16 *>(w + L.dz1), L.Mp, L.nsplit,
                        L.nsplit1, reinterpret_cast<float *>(w + L.split2), reinterpret_cast<float *>(w + L.split1), err,
                        st));
    const ColsumSet sets[4] = {
        {reinterpret_cast<const float *>(w + L.split1), L.nsplit1, kHid * kIn, m->grads + kOffW1, 0, 0},
        {reinterpret_cast<const float *>(w + L.colpart1), np1, kHid, m->grads + kOffB1, 0, 0},
        {reinterpret_cast<const float *>(w + L.split2), L.nsplit, kHid * kHid, m->grads + kOffW2, 0, 0},
        {reinterpret_cast<const float *>(w + L.part2), np2, kHeadPart, m->grads + kOffB2, 0, 0}};
    return launch_colsums(sets, 4, LossSum{reinterpret_cast<const double *>(w + L.lossp), (int)np2, rows, loss}, st);
}

}  // namespace
}  // namespace rq

RQ_API int rq_mlp_fwd(const rq_mlp_t *m, int64_t rows, const uint16_t *x, float *out, void *ws, void *stream) {
    RQ_TRY(check_mlp(m));
    if (rows < 1 || !x || !out || !ws) return fail(RQ_E_ARG, "rq_mlp_fwd: bad arguments");
    const MlpLayout L = mlp_layout(rows);
    char *w = static_cast<char *>(ws);
    cudaStream_t st = as_stream(stream);
    int *err = reinterpret_cast<int *>(w + L.err);
    RQ_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    RQ_TRY(layer1(m, rows, x, L, w, err, st));
    GemmArgs h{};
    h.M = rows;
    h.bias = m->params + kOffB2;
    h.z_rm = reinterpret_cast<bf16 *>(w + L.z2);
    h.out = out;
    h.w3 = m->params + kOffW3;
    h.b3 = m->params + kOffB3;
    h.err = err;
    return launch_gemm<kHid, EPI_HEAD>(reinterpret_cast<const bf16 *>(w + L.h1), kHid,
                                       reinterpret_cast<const bf16 *>(m->w2b), kHid, kHid, h, st);
}

RQ_API int rq_mlp_infer(const rq_mlp_t *m, int64_t rows, const uint16_t *x, float *out, void *ws, void *stream) {
    RQ_TRY(check_mlp(m));
    if (rows < 1 || !x || !out || !ws) return fail(RQ_E_ARG, "rq_mlp_infer: bad arguments");
    const MlpLayout L = mlp_layout(rows);
    char *w = static_cast<char *>(ws);
    cudaStream_t st = as_stream(stream);
    int *err = reinterpret_cast<int *>(w + L.err);
    RQ_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    return launch_infer(m, rows, reinterpret_cast<const bf16 *>(x), out, err, st);
}

RQ_API int rq_mlp_loss(int64_t rows, const float *out, const float *tgt, float *dout, double *loss, void *ws,
                       void *stream) {
    if (rows < 1 || !out || !tgt || !dout || !ws) return fail(RQ_E_ARG, "rq_mlp_loss: bad arguments");
    const MlpLayout L = mlp_layout(rows);
    double *part = reinterpret_cast<double *>(static_cast<char *>(ws) + L.lossp);
    const int grid = std::min(grid_for(rows), 4096);
    cudaStream_t st = as_stream(stream);
    k_loss<<<grid, kThreads, 0, st>>>(rows, out, tgt, dout, part);
    if (loss) k_loss_sum<<<1, kThreads, 0, st>>>(LossSum{part, grid, rows, loss});
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

RQ_API int rq_mlp_bwd(const rq_mlp_t *m, int64_t rows, const uint16_t *xt, const float *dout, void *ws,
                      void *stream) {
    RQ_TRY(check_mlp(m));
    if (!m->grads || !xt || !dout || !ws) return fail(RQ_E_ARG, "rq_mlp_bwd: null argument");
    if (rows < kTileM || rows % kTileM != 0) return fail(RQ_E_ARG, "rq_mlp_bwd: rows must be a multiple of 128");
    const MlpLayout L = mlp_layout(rows);
    char *w = static_cast<char *>(ws);
    cudaStream_t st = as_stream(stream);
    int *err = reinterpret_cast<int *>(w + L.err);
    float *part2 = reinterpret_cast<float *>(w + L.part2);
    k_head_bwd<<<(unsigned)L.tiles, kHid, 0, st>>>(reinterpret_cast<const bf16 *>(w + L.z2), dout, m->params,
                                                   reinterpret_cast<bf16 *>(w + L.dz2), part2);
    RQ_CUDA(cudaGetLastError());
    // dZ1 = (dZ2 W2) * GELU'(Z1) with the b1 partial sums
    GemmArgs g{};
    g.M = rows;
    g.zin_rm = reinterpret_cast<const bf16 *>(w + L.z1);
    g.dz_rm = reinterpret_cast<bf16 *>(w + L.dz1);
    g.colpart = reinterpret_cast<float *>(w + L.colpart1);
    g.err = err;
    int64_t grid1 = 0;
    RQ_TRY((launch_gemm<kHid, EPI_DGELU>(reinterpret_cast<const bf16 *>(w + L.dz2), kHid,
                                         reinterpret_cast<const bf16 *>(m->w2tb), kHid, kHid, g, st, &grid1)));
    return weight_grads(m, rows, xt, L, w, err, grid1, L.tiles, nullptr, st);
}

RQ_API int rq_mlp_train(const rq_mlp_t *m, int64_t rows, const uint16_t *x, const uint16_t *xt, const float *tgt,
                        float *out, double *loss, void *ws, void *stream) {
    RQ_TRY(check_mlp(m));
    if (!m->grads || !x || !xt || !tgt || !ws) return fail(RQ_E_ARG, "rq_mlp_train: null argument");
    if (rows < kTileM || rows % kTileM != 0) return fail(RQ_E_ARG, "rq_mlp_train: rows must be a multiple of 128");
    const MlpLayout L = mlp_layout(rows);
    char *w = static_cast<char *>(ws);
    cudaStream_t st = as_stream(stream);
    int *err = reinterpret_cast<int *>(w + L.err);
    RQ_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    int64_t grid = 0;
    RQ_TRY(launch_train(m, rows, reinterpret_cast<const bf16 *>(x), tgt, out, reinterpret_cast<bf16 *>(w + L.h1),
                        reinterpret_cast<bf16 *>(w + L.dz2), reinterpret_cast<bf16 *>(w + L.dz1),
                        reinterpret_cast<float *>(w + L.colpart1), reinterpret_cast<float *>(w + L.part2),
                        reinterpret_cast<double *>(w + L.lossp), err, st, &grid));
    return weight_grads(m, rows, xt, L, w, err, grid, grid, loss, st);
}

RQ_API int rq_mlp_step(const rq_mlp_t *m, int32_t t, float lr, float beta1, float beta2, float eps,
                       void *stream) {
    RQ_TRY(check_mlp(m));
    if (!m->grads || !m->adam_m || !m->adam_v || t < 1) return fail(RQ_E_ARG, "rq_mlp_step: bad arguments");
    const float c1 = 1.f - powf(beta1, (float)t), c2 = 1.f - powf(beta2, (float)t);
    k_adam<<<grid_for(kNParams), kThreads, 0, as_stream(stream)>>>(*m, lr, beta1, beta2, eps, c1, c2);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

RQ_API int rq_mlp_warm_start(int64_t D, const float *out, int32_t vtype, void *x0, void *stream) {
    if (D < 1 || !out || !x0) return fail(RQ_E_ARG, "rq_mlp_warm_start: bad arguments");
    cudaStream_t st = as_stream(stream);
    const int grid = grid_for(D);
    switch (vtype) {
        case RQ_F32: k_warm_start<float><<<grid, kThreads, 0, st>>>(D, out, static_cast<float *>(x0)); break;
        case RQ_F64: k_warm_start<double><<<grid, kThreads, 0, st>>>(D, out, static_cast<double *>(x0)); break;
        case RQ_C64: k_warm_start<float2><<<grid, kThreads, 0, st>>>(D, out, static_cast<float2 *>(x0)); break;
        case RQ_C128: k_warm_start<double2><<<grid, kThreads, 0, st>>>(D, out, static_cast<double2 *>(x0)); break;
        default: return fail(RQ_E_ARG, "rq_mlp_warm_start: bad vtype");
    }
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

RQ_API int rq_bf16_gemm(const uint16_t *A, int64_t lda, const uint16_t *B, int64_t ldb, int64_t M, int32_t N,
                        int64_t K, float *C, void *ws, void *stream) {
    if (!A || !B || !C || !ws || M < 1 || K < kChunkK || K % kChunkK != 0 || lda % 8 != 0 || ldb % 8 != 0 ||
        lda < K || ldb < K)
        return fail(RQ_E_ARG, "rq_bf16_gemm: bad arguments");
    if (N != 64 && N != 256) return fail(RQ_E_ARG, "rq_bf16_gemm: N must be 64 or 256");
    cudaStream_t st = as_stream(stream);
    int *err = static_cast<int *>(ws);
    RQ_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    GemmArgs g{};
    g.M = M;
    g.out = C;
    g.err = err;
    const bf16 *a = reinterpret_cast<const bf16 *>(A), *b = reinterpret_cast<const bf16 *>(B);
    if (N == 64) return launch_gemm<64, EPI_F32>(a, lda, b, ldb, K, g, st);
    return launch_gemm<256, EPI_F32>(a, lda, b, ldb, K, g, st);
}
