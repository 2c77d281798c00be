// Forward, loss and the gradients down to dZ1 of a training step in one kernel (included by
// rq_mlp.cu, inside its namespace).
//
// A persistent CTA takes 128-row tiles and keeps a tile on chip from X to dZ1:
//   Z1 = X W1^T + b1, H1 = GELU(Z1), Z2 = H1 W2^T + b2, out = GELU(Z2) W3^T + b3, loss, dout,
//   dZ2 = (dout W3) GELU'(Z2), dZ1 = (dZ2 W2) GELU'(Z1).
// What bounds it: the epilogue warps, four GELU or GELU' (8 cycles of a warp's special-function unit
// each) and four column sums (16 shuffles for 16 columns) per element; 65,536 rows take 74 us.  As three
// GEMMs (layer 1, layer 2 with the loss, dZ1) with eight epilogue warps each they took 148 us: Z1 was
// written and read back, and H1, dZ2 and dZ1 were stored feature by feature for the weight gradients.
// * W2 (128 KB) stays in shared memory; the dZ1 product reads the same copy as the forward one, as an
//   MN-major operand.  One 64 KB buffer of four 64-column chunks holds H1, dZ2 and dZ1 in turn; each is
//   the next product's A operand and leaves by TMA stores, row-major, from the layout in which the MMA
//   reads it.  X comes to chunk 0, and the first half of W1 to chunk 1 with it (the second half stays):
//   that leaves room for the layer constants (read through L1 they cost another 15 us).
// * TMEM: Z1 in columns 0 to 255, until dZ1 needs it; Z2, then dZ2 W2, in columns 256 to 511.
// * Sixteen epilogue warps: warp w has the TMEM lanes (rows) 32 (w % 4) .. + 31 and a quarter of the
//   columns.  H1 is handed to the tensor core chunk by chunk; dZ2 W2 comes back in two halves.
// * The column sums (db1, db2, dW3) stay in registers over the CTA's tiles, two columns of each per lane.
constexpr uint32_t kTrW2 = 0, kTrW1 = 4 * 32768, kTrH = kTrW1 + kTileABytes,
                   kTrEnd = kTrH + 4 * kTileABytes;  // 208 KB
constexpr int kTrWarps = 16;  // epilogue warps
constexpr int kTrEpi = 32 * kTrWarps, kTrThreads = 64 + kTrEpi;

struct TrainArgs {
    int64_t tiles;
    const float *params;
    const float *tgt;           // [M][3] = log-amplitude target, sign, weight
    float inv_rows;             // the loss is a mean over the rows
    float *out;                 // [M][2] (optional)
    float *part1, *part2;       // [gridDim.x][kHid]: db1; [gridDim.x][kHeadPart]: db2 | dW3 | db3
    double *losspart;           // [gridDim.x]
    int *err;
};

struct TrainShared {
    uint64_t wfull, xfull, d1full, hfull[4], hfree, d2full, zfull, zfree, d3full[2], gfull[2], gfree, dfree, fin;
    uint32_t tmem;
    int abort, wwait;
    int64_t issued, consumed;   // X tiles
    __align__(16) float b1[kHid], b2[kHid], w3[kOut * kHid];
    float xch[2][kTileM][2];    // output sums of a half's columns, then dout in xch[0]
    float dsum[4][2];
    double lsum[4];
};

__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, int x, int y, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];\n" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(src)
                 : "memory");
}
// ends the group of this thread's stores; returns when they have read their shared memory
__device__ __forceinline__ void tma_store_read() {
    asm volatile("cp.async.bulk.commit_group;\ncp.async.bulk.wait_group.read 0;\n" ::: "memory");
}

// s[k] += x with s in registers
__device__ __forceinline__ void add_at(float (&s)[2], int k, float x) {
    if (k == 0) s[0] += x;
    else s[1] += x;
}

// 16 consecutive floats of shared memory (16-byte aligned; the same address in every lane)
__device__ __forceinline__ void lds16(const float *p, f32x2 (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const ulonglong2 t = reinterpret_cast<const ulonglong2 *>(p)[i];
        v[2 * i] = t.x;
        v[2 * i + 1] = t.y;
    }
}

// The chunk buffer holds rows of 128 B (64 BF16 columns); 16-byte piece c of row r sits at piece
// c ^ (r mod 8).  16 columns (from a multiple of 16) of a row as BF16 pairs:
__device__ __forceinline__ void sts_bf16x16(unsigned char *buf, int row, int c0, const uint32_t (&o)[8]) {
    unsigned char *dst = buf + kTileABytes * (uint32_t)(c0 >> 6) + row * 128;
    const int c = (c0 & 63) >> 3;
#pragma unroll
    for (int j = 0; j < 2; ++j)
        *reinterpret_cast<uint4 *>(dst + (((c + j) ^ (row & 7)) << 4)) =
            make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
}

// lanes 2 l and 2 l + 1 return the sum over the 32 lanes of column l of 16, added in the order of
// col_sum32: 16 shuffles, each round halving the columns a lane keeps.  (Through shared memory, 4
// 16-byte stores and 8 reads a lane, the sums took longer: 12.8 against 11.2 thousand cycles for the
// three of dZ2.)
__device__ __forceinline__ float col_sum16(const f32x2 (&x)[8], int lane) {
    f32x2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = x[i];
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o / 4; ++i) {
            const f32x2 send = up ? v[i] : v[i + o / 4];
            const f32x2 keep = up ? v[i + o / 4] : v[i];
            v[i] = add2(keep, __shfl_xor_sync(0xffffffffu, send, o));
        }
    }
    float a, b;
    unpack2(v[0], a, b);
    const bool up = (lane & 2) != 0;
    const float s = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// the same 16 TMEM columns without the wait: the values exist after tmem_wait16 of them
__device__ __forceinline__ void tmem_issue16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait16(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

// the warp's shared-memory writes are complete for the async proxy (MMA, TMA)
__device__ __forceinline__ void warp_arrive_async(uint64_t *bar, int lane) {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

__global__ void __launch_bounds__(kTrThreads, 1)
k_train(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w1,
        const __grid_constant__ CUtensorMap tma_w2, const __grid_constant__ CUtensorMap tma_h1,
        const __grid_constant__ CUtensorMap tma_dz2, const __grid_constant__ CUtensorMap tma_dz1, const TrainArgs g) {
    // all of it dynamic, so that the operand tiles start at the beginning of the block's memory,
    // which is 1 KB aligned (checked: there is no room for slack)
    extern __shared__ __align__(1024) unsigned char smem[];
    TrainShared &sh = *reinterpret_cast<TrainShared *>(smem + kTrEnd);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0u) {
        if (threadIdx.x == 0) report_error(g.err);
        return;
    }
    if (threadIdx.x == 0) {
        uint64_t *one[] = {&sh.wfull,     &sh.xfull,     &sh.d1full, &sh.hfree, &sh.d2full, &sh.zfree,
                           &sh.d3full[0], &sh.d3full[1], &sh.gfree,  &sh.fin};
        uint64_t *all[] = {&sh.hfull[0], &sh.hfull[1], &sh.hfull[2], &sh.hfull[3],
                           &sh.zfull,    &sh.gfull[0], &sh.gfull[1], &sh.dfree};
        for (uint64_t *b : one) mbar_init(b, 1);
        for (uint64_t *b : all) mbar_init(b, kTrWarps);
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
    auto wait = [&](uint64_t *bar, uint32_t parity) { return warp_wait(bar, parity, abort_p); };
    // every barrier completes once per tile: phase it & 1 of the CTA's tile `it`

    if (warp == 0) {  // ---- TMA: X in, H1, dZ2 and dZ1 out
        if (lane == 0) {
            mbar_expect_tx(&sh.wfull, 4 * 32768 + kTileABytes);
            tma_load_2d(sbase + kTrW1, &tma_w1, 0, kHid / 2, &sh.wfull);
            for (int c = 0; c < 4; ++c) tma_load_2d(sbase + kTrW2 + 32768u * (uint32_t)c, &tma_w2, c * kChunkK, 0, &sh.wfull);
        }
        auto load_x = [&](int64_t u) {
            if (lane == 0) {
                mbar_expect_tx(&sh.xfull, 2 * kTileABytes);
                tma_load_2d(sbase + kTrH, &tma_x, 0, (int)(u * kTileM), &sh.xfull);
                tma_load_2d(sbase + kTrH + kTileABytes, &tma_w1, 0, 0, &sh.xfull);
                sh.issued = sh.issued + 1;
            }
        };
        auto store = [&](const CUtensorMap *map, int c, int y) {
            if (lane == 0) tma_store_2d(map, c * kChunkK, y, sbase + kTrH + kTileABytes * (uint32_t)c);
        };
        auto release = [&](uint64_t *bar) {  // the chunks stored last may be written again
            if (lane == 0) {
                tma_store_read();
                if (bar) mbar_arrive(bar);
            }
            __syncwarp();
        };
        if (blockIdx.x < g.tiles) load_x(blockIdx.x);
        bool ok = true;
        uint32_t p = 0;
        for (int64_t u = blockIdx.x; u < g.tiles && ok; u += gridDim.x, p ^= 1u) {
            const int y = (int)(u * kTileM);
            for (int c = 0; c < 4 && ok; ++c) {
                ok = wait(&sh.hfull[c], p);
                if (ok) store(&tma_h1, c, y);
            }
            release(&sh.hfree);
            ok = ok && wait(&sh.zfull, p);
            if (ok)
                for (int c = 0; c < 4; ++c) store(&tma_dz2, c, y);
            release(&sh.zfree);
            for (int h = 0; h < 2 && ok; ++h) {
                ok = wait(&sh.gfull[h], p);
                if (!ok) break;
                store(&tma_dz1, 2 * h, y);
                store(&tma_dz1, 2 * h + 1, y);
                release(h ? &sh.gfree : nullptr);
                if (h == 0 && u + gridDim.x < g.tiles) load_x(u + gridDim.x);
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
        __syncwarp();
    } else if (warp == 1) {  // ---- MMA issuer
        constexpr uint32_t kFull = make_idesc(kTileM, kHid), kHalf = make_idesc(kTileM, kHid / 2);
        const uint32_t hb = sbase + kTrH;
        bool ok = wait(&sh.wfull, 0u);
        if (ok && lane == 0) sh.wwait = 1;
        int64_t it = 0;
        for (int64_t u = blockIdx.x; u < g.tiles && ok; u += gridDim.x, ++it) {
            const uint32_t p = (uint32_t)(it & 1);
            ok = wait(&sh.xfull, p) && (it < 1 || wait(&sh.dfree, p ^ 1u));
            if (!ok) break;
            tc_fence_after();
            if (lane == 0) {
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int kk = 0; kk < kChunkK / 16; ++kk)
                        mma_bf16(tmem + (uint32_t)h * (kHid / 2), make_sdesc_sw128(hb + (uint32_t)kk * 32u),
                                 make_sdesc_sw128((h ? sbase + kTrW1 : hb + kTileABytes) + (uint32_t)kk * 32u), kHalf,
                                 kk > 0 ? 1u : 0u);
                mma_commit(&sh.d1full);
                sh.consumed = it + 1;
            }
            __syncwarp();
            for (int c = 0; c < 4; ++c) {
                ok = wait(&sh.hfull[c], p);
                if (!ok) break;
                tc_fence_after();
                if (lane == 0) {
                    const uint32_t a = hb + kTileABytes * (uint32_t)c, b = sbase + kTrW2 + 32768u * (uint32_t)c;
#pragma unroll
                    for (int kk = 0; kk < kChunkK / 16; ++kk)
                        mma_bf16(tmem + kHid, make_sdesc_sw128(a + (uint32_t)kk * 32u),
                                 make_sdesc_sw128(b + (uint32_t)kk * 32u), kFull, (c > 0 || kk > 0) ? 1u : 0u);
                    if (c == 3) mma_commit(&sh.d2full);
                }
                __syncwarp();
            }
            ok = ok && wait(&sh.zfull, p);
            if (!ok) break;
            tc_fence_after();
            if (lane == 0) {
                // dZ2 W2, half of its columns at a time: B is W2 with the columns contiguous, 16 rows a step
                for (int h = 0; h < 2; ++h) {
                    for (int kk = 0; kk < kHid / 16; ++kk)
                        mma_bf16(tmem + kHid + (uint32_t)h * (kHid / 2),
                                 make_sdesc_sw128(hb + kTileABytes * (uint32_t)(kk >> 2) + (uint32_t)(kk & 3) * 32u),
                                 make_sdesc_mn(sbase + kTrW2 + 65536u * (uint32_t)h + (uint32_t)kk * 2048u, 32768u),
                                 kHalf | kIdescTransB, kk > 0 ? 1u : 0u);
                    mma_commit(&sh.d3full[h]);
                }
            }
            __syncwarp();
        }
    } else {  // ---- epilogue
        const int q4 = warp & 3, cq = (warp - 2) >> 2, row = 32 * q4 + lane, e = threadIdx.x - 64;
        const uint32_t lanes = tmem + ((uint32_t)(32 * q4) << 16);
        unsigned char *buf = smem + kTrH;
        float sb1[2] = {}, sb2[2] = {}, sw30[2] = {}, sw31[2] = {};  // column sums
        float sd0 = 0.f, sd1 = 0.f;
        double loss = 0.;
        for (int i = e; i < kHid; i += kTrEpi) {
            sh.b1[i] = g.params[kOffB1 + i];
            sh.b2[i] = g.params[kOffB2 + i];
            sh.w3[i] = g.params[kOffW3 + i];
            sh.w3[kHid + i] = g.params[kOffW3 + kHid + i];
        }
        named_bar_sync(kEpiBar, kTrEpi);
        bool broke = false;
        int64_t it = 0;
        for (int64_t u = blockIdx.x; u < g.tiles; u += gridDim.x, ++it) {
            const uint32_t p = (uint32_t)(it & 1);
            bool ok = wait(&sh.d1full, p);
            tc_fence_after();
            float t0 = 0.f, t1 = 0.f, t2 = 0.f;  // the row's target, wanted after Z2
            if (cq == 1) {
                const float *t = g.tgt + (u * kTileM + row) * 3;
                t0 = t[0];
                t1 = t[1];
                t2 = t[2];
            }
            // H1 chunk by chunk, 16 columns of it per warp; the next chunk's loads are in flight meanwhile
            uint32_t zn[16];
            tmem_issue16(lanes + (uint32_t)(16 * cq), zn);
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                if (c == 2 && it >= 1) ok = ok && wait(&sh.gfree, p ^ 1u);
                const int c0 = 64 * c + 16 * cq;
                f32x2 b[8];
                uint32_t o[8];
                lds16(sh.b1 + c0, b);
                tmem_wait16(zn);
#pragma unroll
                for (int i = 0; i < 8; ++i) b[i] = add2(pack2(zn[2 * i], zn[2 * i + 1]), b[i]);
                if (c < 3) tmem_issue16(lanes + (uint32_t)(c0 + 64), zn);
                if (!ok) continue;
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = bf16x2(gelu2(b[i]));
                sts_bf16x16(buf, row, c0, o);
                warp_arrive_async(&sh.hfull[c], lane);
            }
            ok = ok && wait(&sh.d2full, p);
            if (named_bar_or(kEpiBar, kTrEpi, !ok || *abort_p != 0)) {  // the same answer in every epilogue thread
                broke = true;
                break;
            }
            tc_fence_after();
            // the output sums in the order of the forward pass: along the columns of each half, then
            // the halves; an odd quarter goes on from the sums of the even one before it
            float o0 = 0.f, o1 = 0.f;
            {
                const int c0 = cq * (kHid / 4);
                uint32_t zr[4][16];
                float z[4][16];
#pragma unroll
                for (int k = 0; k < 4; ++k) tmem_issue16(lanes + (uint32_t)(kHid + c0 + 16 * k), zr[k]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    f32x2 b[8];
                    lds16(sh.b2 + c0 + 16 * k, b);
                    tmem_wait16(zr[k]);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        unpack2(gelu2(add2(pack2(zr[k][2 * i], zr[k][2 * i + 1]), b[i])), z[k][2 * i], z[k][2 * i + 1]);
                }
                if (cq & 1) {
                    named_bar_sync(kEpiBar + 1, kTrEpi);
                    o0 = sh.xch[cq >> 1][row][0];
                    o1 = sh.xch[cq >> 1][row][1];
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 w0 = *reinterpret_cast<const float4 *>(sh.w3 + c0 + 16 * k + i);
                        const float4 w1 = *reinterpret_cast<const float4 *>(sh.w3 + kHid + c0 + 16 * k + i);
                        o0 += z[k][i] * w0.x;
                        o1 += z[k][i] * w1.x;
                        o0 += z[k][i + 1] * w0.y;
                        o1 += z[k][i + 1] * w1.y;
                        o0 += z[k][i + 2] * w0.z;
                        o1 += z[k][i + 2] * w1.z;
                        o0 += z[k][i + 3] * w0.w;
                        o1 += z[k][i + 3] * w1.w;
                    }
                }
            }
            if (cq != 1) {
                sh.xch[cq >> 1][row][0] = o0;
                sh.xch[cq >> 1][row][1] = o1;
                if (cq == 3) named_bar_arrive(kEpiBar + 2, kTrEpi / 2);
                else named_bar_arrive(kEpiBar + 1, kTrEpi);
            } else {
                named_bar_sync(kEpiBar + 2, kTrEpi / 2);
                o0 += sh.xch[1][row][0] + __ldg(g.params + kOffB3);
                o1 += sh.xch[1][row][1] + __ldg(g.params + kOffB3 + 1);
                const int64_t m = u * kTileM + row;
                if (g.out) {
                    g.out[m * 2] = o0;
                    g.out[m * 2 + 1] = o1;
                }
                // the loss of the row and its gradient
                const float sg = t1, w = t2;
                const float d = o0 - t0;
                const float tt = -sg * o1;
                const float sp = tt > 20.f ? tt : log1pf(expf(tt));  // softplus(-s o1)
                const float sig = 1.f / (1.f + expf(-tt));           // sigmoid(-s o1)
                loss += (double)(w * (d * d + sp));
                const float d0 = w * g.inv_rows * 2.f * d, d1 = -w * g.inv_rows * sg * sig;
                sd0 += d0;
                sd1 += d1;
                sh.xch[0][row][0] = d0;
                sh.xch[0][row][1] = d1;
            }
            named_bar_sync(kEpiBar, kTrEpi);
            // dZ2 of this warp's 64 columns, and the column sums of db2 and dW3
            ok = wait(&sh.hfree, p);
            const f32x2 d0 = both(sh.xch[0][row][0]), d1 = both(sh.xch[0][row][1]);
            tmem_issue16(lanes + (uint32_t)(kHid + 64 * cq), zn);
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                const int c0 = 64 * cq + 16 * k;
                f32x2 dz[8], a[8], t[8];
                uint32_t o[8];
                lds16(sh.b2 + c0, t);
                tmem_wait16(zn);
#pragma unroll
                for (int i = 0; i < 8; ++i) gelu_both2(add2(pack2(zn[2 * i], zn[2 * i + 1]), t[i]), a[i], dz[i]);
                if (k < 3) tmem_issue16(lanes + (uint32_t)(kHid + c0 + 16), zn);
                lds16(sh.w3 + c0, t);
#pragma unroll
                for (int i = 0; i < 8; ++i) t[i] = mul2(t[i], d0);
                {
                    f32x2 w1[8];
                    lds16(sh.w3 + kHid + c0, w1);
#pragma unroll
                    for (int i = 0; i < 8; ++i) dz[i] = mul2(dz[i], fma2(d1, w1[i], t[i]));
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = bf16x2(dz[i]);
                if (ok) sts_bf16x16(buf, row, c0, o);
                const float s0 = col_sum16(dz, lane);
#pragma unroll
                for (int i = 0; i < 8; ++i) t[i] = mul2(d0, a[i]);
                const float s1 = col_sum16(t, lane);
#pragma unroll
                for (int i = 0; i < 8; ++i) t[i] = mul2(d1, a[i]);
                const float s2 = col_sum16(t, lane);
                if ((lane & 1) == (k & 1)) {  // this lane keeps the column's sums
                    add_at(sb2, k >> 1, s0);
                    add_at(sw30, k >> 1, s1);
                    add_at(sw31, k >> 1, s2);
                }
            }
            tc_fence_before();
            if (ok) warp_arrive_async(&sh.zfull, lane);
            // dZ1: half by half, 32 columns per warp, and the column sums of db1
            uint32_t vn[16];
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                const int h = k >> 1, c0 = 128 * h + 32 * cq + 16 * (k & 1);
                f32x2 v[8], b[8];
                uint32_t o[8];
                if ((k & 1) == 0) {
                    ok = ok && wait(&sh.d3full[h], p);
                    tc_fence_after();
                }
                tmem_issue16(lanes + (uint32_t)(kHid + c0), vn);
                tmem_issue16(lanes + (uint32_t)c0, zn);
                lds16(sh.b1 + c0, b);
                tmem_wait16(vn);
                tmem_wait16(zn);
                if (k == 3) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0 && ok) mbar_arrive(&sh.dfree);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {  // Z1 as the separate passes keep it, in BF16
                    const uint32_t z = bf16x2(add2(pack2(zn[2 * i], zn[2 * i + 1]), b[i]));
                    f32x2 a, d;
                    gelu_both2(pack2(z << 16, z & 0xFFFF0000u), a, d);
                    v[i] = mul2(pack2(vn[2 * i], vn[2 * i + 1]), d);
                    o[i] = bf16x2(v[i]);
                }
                // dZ2 has been read by the second half's product and by its store
                if (k == 0) ok = ok && wait(&sh.d3full[1], p) && wait(&sh.zfree, p);
                if (ok) sts_bf16x16(buf, row, c0, o);
                const float s = col_sum16(v, lane);
                if ((lane & 1) == (k & 1)) add_at(sb1, h, s);
                if ((k & 1) && ok) warp_arrive_async(&sh.gfull[h], lane);
            }
        }
        if (!broke) {
            // this CTA's column sums: the four row quarters added in order, one row of partials
            if (cq == 1) {
                const float s0 = warp_sum(sd0), s1 = warp_sum(sd1);
                const double sl = warp_sum(loss);
                if (lane == 0) {
                    sh.dsum[q4][0] = s0;
                    sh.dsum[q4][1] = s1;
                    sh.lsum[q4] = sl;
                }
            }
            // in the chunk buffer, once the last tile's dZ1 has been read
            const bool ok = it < 1 || wait(&sh.gfree, (uint32_t)((it - 1) & 1));
            if (!named_bar_or(kEpiBar, kTrEpi, !ok || *abort_p != 0)) {
                float (*red)[4][kHid] = reinterpret_cast<float (*)[4][kHid]>(buf);  // [db2, dW3, dW3, db1][q4]
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int k = 2 * j + (lane & 1), c0 = 64 * cq + 16 * k + (lane >> 1);
                    red[0][q4][c0] = sb2[j];
                    red[1][q4][c0] = sw30[j];
                    red[2][q4][c0] = sw31[j];
                    red[3][q4][128 * j + 32 * cq + 16 * (lane & 1) + (lane >> 1)] = sb1[j];
                }
                named_bar_sync(kEpiBar, kTrEpi);
                float *part = g.part2 + (int64_t)blockIdx.x * kHeadPart, *part1 = g.part1 + (int64_t)blockIdx.x * kHid;
                for (int i = e; i < 4 * kHid; i += kTrEpi) {
                    const int j = i / kHid, c = i % kHid;
                    const float s = ((red[j][0][c] + red[j][1][c]) + red[j][2][c]) + red[j][3][c];
                    if (j < 3) part[i] = s;
                    else part1[c] = s;
                }
                if (e < 2) part[3 * kHid + e] = ((sh.dsum[0][e] + sh.dsum[1][e]) + sh.dsum[2][e]) + sh.dsum[3][e];
                if (e == 0) g.losspart[blockIdx.x] = ((sh.lsum[0] + sh.lsum[1]) + sh.lsum[2]) + sh.lsum[3];
            }
        }
    }
    __syncthreads();
    if (sh.abort != 0) {
        // let the copies and MMAs already issued land before the memory is released
        if (threadIdx.x == 0) {
            if (sh.consumed < sh.issued) wait_bar(&sh.xfull, (uint32_t)((sh.issued - 1) & 1), nullptr);
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

// *grid_out = the CTAs launched (rows of the per-CTA partial sums); rows a multiple of 128
int launch_train(const rq_mlp_t *m, int64_t rows, const bf16 *x, const float *tgt, float *out, bf16 *h1, bf16 *dz2,
                 bf16 *dz1, float *part1, float *part2, double *losspart, int *err, cudaStream_t st,
                 int64_t *grid_out) {
    CUtensorMap tx, t1, t2, th, tz2, tz1;
    RQ_TRY(make_tma(&tx, x, kIn, rows, kIn, kTileM));
    RQ_TRY(make_tma(&t1, reinterpret_cast<const bf16 *>(m->w1b), kIn, kHid, kIn, kHid / 2));
    RQ_TRY(make_tma(&t2, reinterpret_cast<const bf16 *>(m->w2b), kHid, kHid, kHid, kHid));
    RQ_TRY(make_tma(&th, h1, kHid, rows, kHid, kTileM));
    RQ_TRY(make_tma(&tz2, dz2, kHid, rows, kHid, kTileM));
    RQ_TRY(make_tma(&tz1, dz1, kHid, rows, kHid, kTileM));
    constexpr size_t smem = kTrEnd + sizeof(TrainShared);
    static_assert(smem <= 227 * 1024, "one block's shared memory");
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    KernelLaunchCache *c = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &c));
    RQ_TRY(configure_kernel(k_train, *c, smem, kTrThreads, &per_sm));
    const int64_t tiles = rows / kTileM, grid = std::min<int64_t>(tiles, sm_count());
    const TrainArgs g{tiles, m->params, tgt, 1.f / (float)rows, out, part1, part2, losspart, err};
    k_train<<<(unsigned)grid, kTrThreads, smem, st>>>(tx, t1, t2, th, tz2, tz1, g);
    RQ_CUDA(cudaGetLastError());
    *grid_out = grid;
    return RQ_OK;
}

// ---- weight gradients -------------------------------------------------------------------------
// dW2^T = H1^T dZ2 [256][256] and dW1^T = X^T dZ1 [64][256], split over the rows (their K): unit u of
// the first 2 nsplit2 is a 128-row half of dW2 over one of nsplit2 ranges of 64-row chunks, the other
// nsplit1 are dW1 (64 rows; the tile's other 64 read as zeros) over one of nsplit1 ranges.  H1, dZ2 and
// dZ1 are row-major, so their tiles are MN-major operands: boxes of 64 columns x 64 rows, 8 KB each,
// and no transposed copy is written for this product (three copies of 33 MB at 65,536 rows).  X^T is
// K-major.  The partial products are stored column-major ([column][row]: dW in its row-major
// layout).  Both products in one launch, a CTA per SM: the store of a unit runs under the next one's
// MMAs.  Bound by the reads: 109 MB at 65,536 rows, 22.5 us (two launches: 31 us).
constexpr int kWgStages = 4;
constexpr uint32_t kWgBox = 64 * kChunkK * 2, kWgStage = 6 * kWgBox;

struct WgradArgs {
    int64_t chunks, nsplit2, nsplit1;
    float *out2, *out1;  // [nsplit2][256][256], [nsplit1][256][64]
    int *err;
};

__global__ void __launch_bounds__(kGemmThreads, 1)
k_wgrad(const __grid_constant__ CUtensorMap tma_h1, const __grid_constant__ CUtensorMap tma_dz2,
        const __grid_constant__ CUtensorMap tma_xt, const __grid_constant__ CUtensorMap tma_dz1, const WgradArgs g) {
    constexpr int S = kWgStages;
    constexpr uint32_t kIdesc2 = make_idesc(kTileM, kHid) | kIdescTransA | kIdescTransB,
                       kIdesc1 = make_idesc(kTileM, kHid) | kIdescTransB;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[S], empty[S], tfull[2], tempty[2], fin;
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s;
    __shared__ long long issued_s, consumed_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sbase = (smem_u32(smem) + 1023u) & ~1023u;  // the launch adds 1 KB for this
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], kEpiThreads / 32);
        }
        mbar_init(&fin, 1);
        fence_mbar_init();
        abort_s = 0;
        issued_s = consumed_s = 0;
    }
    if (warp == 1) tmem_alloc(&tmem_s, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s;
    volatile int *abort_p = &abort_s;
    const int64_t units2 = 2 * g.nsplit2, units = units2 + g.nsplit1;
    auto range = [&](int64_t u, int64_t &c0, int64_t &c1) {  // the chunks of unit u
        const int64_t n = u < units2 ? g.nsplit2 : g.nsplit1, sp = u < units2 ? u >> 1 : u - units2;
        c0 = sp * g.chunks / n;
        c1 = (sp + 1) * g.chunks / n;
    };
    auto wait = [&](uint64_t *bar, uint32_t parity) { return warp_wait(bar, parity, abort_p); };

    if (warp == 0) {  // ---- TMA producer
        long long it = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
            int64_t c0, c1;
            range(u, c0, c1);
            for (int64_t c = c0; c < c1; ++c, ++it) {
                const int s = (int)(it % S), k = (int)(c * kChunkK);
                ok = it < S || wait(&empty[s], (uint32_t)((it / S - 1) & 1));
                if (!ok) break;
                if (lane == 0) {
                    const uint32_t st = sbase + (uint32_t)s * kWgStage;
                    mbar_expect_tx(&full[s], kWgStage);
                    if (u < units2) {
                        for (int j = 0; j < 2; ++j)
                            tma_load_2d(st + (uint32_t)j * kWgBox, &tma_h1, (int)(u & 1) * kTileM + 64 * j, k, &full[s]);
                    } else {
                        tma_load_2d(st, &tma_xt, k, 0, &full[s]);
                    }
                    for (int j = 0; j < kHid / 64; ++j)
                        tma_load_2d(st + kTileABytes + (uint32_t)j * kWgBox, u < units2 ? &tma_dz2 : &tma_dz1, 64 * j, k,
                                    &full[s]);
                    issued_s = it + 1;
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {  // ---- MMA issuer
        long long it = 0, t = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x, ++t) {
            const int b = (int)(t & 1);
            if (t >= 2 && !wait(&tempty[b], (uint32_t)((t / 2 - 1) & 1))) break;
            tc_fence_after();
            int64_t c0, c1;
            range(u, c0, c1);
            for (int64_t c = c0; c < c1; ++c, ++it) {
                const int s = (int)(it % S);
                ok = wait(&full[s], (uint32_t)((it / S) & 1));
                if (!ok) break;
                tc_fence_after();
                if (lane == 0) {
                    const uint32_t sa = sbase + (uint32_t)s * kWgStage, sb = sa + kTileABytes;
#pragma unroll
                    for (int kk = 0; kk < kChunkK / 16; ++kk)
                        mma_bf16(tmem + (uint32_t)(b * kHid),
                                 u < units2 ? make_sdesc_mn(sa + (uint32_t)kk * 2048u, kWgBox)
                                            : make_sdesc_sw128(sa + (uint32_t)kk * 32u),
                                 make_sdesc_mn(sb + (uint32_t)kk * 2048u, kWgBox), u < units2 ? kIdesc2 : kIdesc1,
                                 (c > c0 || kk > 0) ? 1u : 0u);
                    mma_commit(&empty[s]);
                    consumed_s = it + 1;
                }
                __syncwarp();
            }
            if (!ok) break;
            if (lane == 0) mma_commit(&tfull[b]);
            __syncwarp();
        }
    } else {  // ---- epilogue: warp w stores TMEM lanes 32 (w % 4) .. + 31 of half (w - 2) / 4 of the columns
        const int q = warp & 3, h = (warp - 2) >> 2, row = 32 * q + lane;
        long long t = 0;
        for (int64_t u = blockIdx.x; u < units; u += gridDim.x, ++t) {
            const int b = (int)(t & 1);
            if (!wait(&tfull[b], (uint32_t)((t >> 1) & 1))) break;
            tc_fence_after();
            const bool two = u < units2;
            if (two || q < kIn / 32) {
                const int64_t ld = two ? kHid : kIn;
                float *dst = two ? g.out2 + (u >> 1) * kHid * kHid + (u & 1) * kTileM : g.out1 + (u - units2) * kHid * kIn;
                dst += (int64_t)(h * (kHid / 2)) * ld + row;
#pragma unroll 1
                for (int g0 = 0; g0 < kHid / 2; g0 += 32) {
                    float v[32];
                    tmem_ld32(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(b * kHid + h * (kHid / 2) + g0), v);
#pragma unroll
                    for (int i = 0; i < 32; ++i) dst[(g0 + i) * ld] = v[i];
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[b]);
        }
    }
    __syncthreads();
    if (abort_s != 0) {
        // let the copies and MMAs already issued land before the memory is released
        if (threadIdx.x == 0) {
            for (long long it = consumed_s; it < issued_s; ++it) wait_bar(&full[it % S], (uint32_t)((it / S) & 1), nullptr);
            report_error(g.err);
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
        tmem_dealloc(tmem, 512);
    }
}

// splits of dW2 (two row tiles each) and of dW1: a unit of each per SM
constexpr int kSplitK = 76;

int launch_wgrad(const bf16 *h1, const bf16 *dz2, const bf16 *xt, const bf16 *dz1, int64_t rows, int64_t nsplit2,
                 int64_t nsplit1, float *out2, float *out1, int *err, cudaStream_t st) {
    CUtensorMap th, tz2, tx, tz1;
    RQ_TRY(make_tma(&th, h1, kHid, rows, kHid, kChunkK));
    RQ_TRY(make_tma(&tz2, dz2, kHid, rows, kHid, kChunkK));
    RQ_TRY(make_tma(&tx, xt, rows, kIn, rows, kTileM));
    RQ_TRY(make_tma(&tz1, dz1, kHid, rows, kHid, kChunkK));
    constexpr size_t smem = kWgStages * kWgStage + 1024;
    thread_local KernelLaunchCache table[kMaxCachedDevices];
    KernelLaunchCache *c = nullptr;
    int per_sm = 1;
    RQ_TRY(cache_slot(table, &c));
    RQ_TRY(configure_kernel(k_wgrad, *c, smem, kGemmThreads, &per_sm));
    const int64_t units = 2 * nsplit2 + nsplit1, grid = std::min<int64_t>(units, sm_count());
    const WgradArgs g{rows / kChunkK, nsplit2, nsplit1, out2, out1, err};
    k_wgrad<<<(unsigned)grid, kGemmThreads, smem, st>>>(th, tz2, tx, tz1, g);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}
