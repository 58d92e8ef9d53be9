// The surrogate's backward pass in fused tcgen05 kernels (64 channels), the
// counterparts of fno_layer.cu:
//
//   k_proj_bwd   one grid row: gradient through both projections and GELU,
//                the last layer's BF16 gradient and its transform along W;
//   k_row_bwd    one grid row of a layer: dv = dz w + FW^T dXw (two TMEM
//                accumulators), times GELU'(z) of the layer before, that
//                layer's BF16 gradient out and its transform along W;
//   k_inv_h_bwd, k_modes_bwd, k_fwd_h_bwd   the adjoints of the transforms
//                along H and of the mode mixing, with the mode weights'
//                gradient in the epilogue;
//   k_wgrad      out = dz^T x over all points, both operands MN-major
//                straight from the channels-last rows, one partial product
//                per chunk of points.
//
// The layer-by-layer path spent its time in transposes of the activations,
// FP32 gradients written and read back, and skinny products; here each
// gradient is written once in BF16 for the products and once in FP32 for the
// bias gradient's column sums.  Products, their order, every BF16 rounding
// and those sums are that path's, so the gradients are the same bits (summing
// the bias gradients inside the row kernels, in another order, would save a
// fifth, but one FP32 ulp of a bias moves the next step's BF16 activations,
// and its gradients by 4e-4).  Bound: memory (the FP32 pre-activations and
// gradients) and GELU' (erff and expf), about equally.
// 24 epilogue warps take half of the channels each, with one copy of GELU' in
// the instruction cache.
// Measured at 64 samples of 128 x 384 points (ncu): k_proj_bwd 1133 us (12 warps,
// unrolled code, gradients stored by rows: 1309), k_row_bwd 390 (452), k_wgrad
// 110 (64 x 64) and 153 (128 wide), k_modes_bwd 40, k_fwd_h_bwd 36, k_inv_h_bwd
// 22; the training step 8.6 -> 7.7 ms with k_sum_batches_staged (by GEMMs layer
// by layer 44).

#include "fno_tc.cuh"

namespace {

// ---------------------------------------------------------------- rows
// The FP32 gradients are written in blocks of 32 points x 8 channels (a warp
// stores one block, 1 KB, at a time; by rows its 32-byte pieces lay in 32
// different lines); gf_fno_colsum_blocked reads them.
__device__ __forceinline__ long long blocked(long long m, int c, int C) {
    return ((m >> 5) * (C / 8) + (c >> 3)) * 256 + (m & 31) * 8 + (c & 7);
}
struct RowBwdArgs {
    int rows, K2;
    const float *z;     // pre-activations of the layer before (FP32), or null: no GELU
    __nv_bfloat16 *dZ;  // [rows][K2][64]: transform of the new gradient along W, or null
    float *df;          // the new gradient in FP32 (its column sums are the bias gradient)
};
// as RowSmem (fno_layer.cu): IWT first (its MMA reads 128 rows per block), FW, w, dXw, gradients
template <int NT> struct BwdSmem {
    __host__ __device__ static uint32_t fw(int K2) { return (uint32_t)(2 * NT * K2 * 128); }
    __host__ __device__ static uint32_t wl(int K2) { return 2 * fw(K2); }
    __host__ __device__ static uint32_t xx(int K2) { return wl(K2) + 8192; }
    __host__ __device__ static uint32_t vv(int K2) { return xx(K2) + 2 * 8192; }
    __host__ __device__ static uint32_t bars(int K2) { return vv(K2) + 2 * NT * 16384; }
    __host__ __device__ static uint32_t total(int K2) { return bars(K2) + 128 + 1024; }
};

// warps as in k_row; the phases of its barriers too (see there)
template <int NT>
__global__ void __launch_bounds__(NT * 256 + 128, 1)
    k_row_bwd(const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmX,
              const __grid_constant__ CUtensorMap tmFW, const __grid_constant__ CUtensorMap tmW,
              const __grid_constant__ CUtensorMap tmIWT, const __grid_constant__ CUtensorMap tmO, RowBwdArgs a) {
    extern __shared__ uint8_t dsmem[];
    typedef BwdSmem<NT> L;
    constexpr int W = NT * 128, EW = NT * 8;
    constexpr uint32_t TCOLS = NT == 1 ? 256 : 512;
    uint8_t *base = align1k(dsmem);
    uint8_t *sI = base, *sF = base + L::fw(a.K2), *sW = base + L::wl(a.K2), *sX = base + L::xx(a.K2),
            *sV = base + L::vv(a.K2);
    uint64_t *full = reinterpret_cast<uint64_t *>(base + L::bars(a.K2));
    uint64_t *wfull = full + 2, *dready = full + 3, *dfree = full + 4, *vready = full + 5, *fready = full + 6,
             *ffree = full + 7;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool has_tr = a.dZ != nullptr;
    if (threadIdx.x == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_init(wfull, 1);
        mbar_init(dready, 1);
        mbar_init(dfree, EW);
        mbar_init(vready, EW + 2);
        mbar_init(fready, 1);
        mbar_init(ffree, 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, TCOLS, warp);
    const int r0 = blockIdx.x, step = gridDim.x, n = (a.rows - r0 + step - 1) / step;
    bool ok = true;

    if (warp == EW + 2) {
        if (lane == 0) { // TMA
            auto load = [&](int it) {
                const int s = it & 1, r = r0 + it * step;
                mbar_expect_tx(&full[s], NT * 16384 + a.K2 * 128);
                for (int t = 0; t < NT; ++t)
                    tma_load_2d(sV + (s * NT + t) * 16384, &tmD, 0, r * W + t * 128, &full[s]);
                tma_load_2d(sX + s * 8192, &tmX, 0, r * a.K2, &full[s]);
            };
            mbar_expect_tx(wfull, 8192 + (has_tr ? 2 : 1) * 2 * NT * a.K2 * 128);
            tma_load_2d(sW, &tmW, 0, 0, wfull);
            for (int k = 0; k < 2 * NT; ++k) {
                tma_load_2d(sF + k * a.K2 * 128, &tmFW, k * 64, 0, wfull);
                if (has_tr) tma_load_2d(sI + k * a.K2 * 128, &tmIWT, k * 64, 0, wfull);
            }
            int loaded = 0;
            for (; loaded < 2 && loaded < n; ++loaded) load(loaded);
            mbar_arrive(vready);
            for (int it = 0; ok && it < n; ++it) {
                ok = mbar_wait(vready, it & 1);
                if (!ok) break;
                for (int t = 0; t < NT; ++t)
                    tma_store_2d(&tmO, 0, (r0 + it * step) * W + t * 128, sV + ((it & 1) * NT + t) * 16384);
                bulk_commit();
                if (it + 2 < n) {
                    if (has_tr) ok = mbar_wait(fready, it & 1);
                    bulk_wait_read();
                    if (ok) load(loaded++);
                }
                mbar_arrive(vready);
            }
            bulk_wait();
            mbar_wait(wfull, 0);
            for (int q = loaded > 2 ? loaded - 2 : 0; q < loaded; ++q) mbar_wait(&full[q & 1], (q >> 1) & 1);
        }
        __syncwarp();
    } else if (warp == EW + 3) {
        if (lane == 0) { // MMA
            // dz [w][o] times w [o][i]; FW [kp][w] as an MN-major A against dXw [kp][c]
            const uint32_t idw = idesc_of(64, 0, 1), idf = idesc_of(64, 1, 1), idt = idesc_of(64, 0, 1);
            ok = mbar_wait(wfull, 0);
            auto mix = [&](int it) {
                const int s = it & 1;
                ok = ok && mbar_wait(&full[s], (it >> 1) & 1);
                if (!ok) return;
                fence_after();
                const uint64_t dw = sdesc_mn(smem_u32(sW), 1024), dx = sdesc_mn(smem_u32(sX + s * 8192), 1024);
                for (int t = 0; t < NT; ++t) {
                    const uint64_t dv = sdesc(smem_u32(sV + (s * NT + t) * 16384)),
                                   df = sdesc_mn(smem_u32(sF + 2 * t * a.K2 * 128), a.K2 * 128);
                    for (int k = 0; k < 4; ++k) mma(tmem + t * 64, dv + K_STEP * k, dw + MN_STEP * k, idw, k > 0);
                    for (int k = 0; k < a.K2 / 16; ++k)
                        mma(tmem + (NT + t) * 64, df + MN_STEP * k, dx + MN_STEP * k, idf, k > 0);
                }
                mma_commit(dready);
            };
            if (n > 0) mix(0);
            mbar_arrive(vready);
            for (int it = 0; ok && it < n; ++it) {
                if (it + 1 < n) {
                    ok = mbar_wait(dfree, it & 1);
                    if (ok) mix(it + 1);
                }
                ok = ok && mbar_wait(vready, it & 1);
                mbar_arrive(vready);
                if (has_tr && ok) {
                    ok = it == 0 || mbar_wait(ffree, (it - 1) & 1);
                    if (!ok) break;
                    fence_after();
                    for (int kb = 0; kb < 2 * NT; ++kb) {
                        const uint64_t di = sdesc(smem_u32(sI + kb * a.K2 * 128)),
                                       dv = sdesc_mn(smem_u32(sV + (it & 1) * NT * 16384 + kb * 8192), 1024);
                        for (int k = 0; k < 4; ++k)
                            mma(tmem + 2 * NT * 64, di + K_STEP * k, dv + MN_STEP * k, idt, (kb | k) > 0);
                    }
                    mma_commit(fready);
                }
            }
        }
        __syncwarp();
    } else if (warp >= EW) {
        if (has_tr) {
            const int kp = (warp - EW) * 32 + lane;
            const uint32_t tf = tmem + 2 * NT * 64 + ((uint32_t)((warp - EW) * 32) << 16);
            for (int it = 0; it < n; ++it) {
                ok = mbar_wait(fready, it & 1);
                if (!ok) break;
                fence_after();
                float v[64];
                tmem_ld<32>(tf, v);
                tmem_ld<32>(tf + 32, v + 32);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(ffree);
                if (kp < a.K2) {
                    uint4 *o = reinterpret_cast<uint4 *>(a.dZ + ((long long)(r0 + it * step) * a.K2 + kp) * CH);
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] = pack8(v + 8 * j);
                }
            }
        }
    } else {
        const int t = (warp >> 2) % NT, q = warp & 3, w = t * 128 + q * 32 + lane, ch = warp / (4 * NT) * 32;
        const uint32_t td = tmem + t * 64 + ((uint32_t)(q * 32) << 16);
        for (int it = 0; it < n; ++it) {
            const long long m = (long long)(r0 + it * step) * W + w;
            float *frow = a.df + blocked(m, ch, CH);
            const float *zrow = a.z ? a.z + m * CH : nullptr;
            float zn[16]; // the next 16 pre-activations, in flight while this chunk is worked on
            if (zrow) {
                ld_global8(zrow + ch, zn);
                ld_global8(zrow + ch + 8, zn + 8);
            }
            ok = mbar_wait(dready, it & 1);
            if (!ok) break;
            fence_after();
            uint8_t *tile = sV + (it & 1) * NT * 16384;
#pragma unroll 1
            for (int c0 = ch; c0 < ch + 32; c0 += 16, frow += 512) { // (one copy of GELU' in the instruction cache)
                float v[16], s[16];
                tmem_ld<16>(td + c0, v);
                tmem_ld<16>(td + NT * 64 + c0, s);
                if (c0 == ch + 16) {
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(dfree);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = v[i] + s[i];
                if (zrow) {
                    float z[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) z[i] = zn[i];
                    if (c0 == ch) {
                        ld_global8(zrow + c0 + 16, zn);
                        ld_global8(zrow + c0 + 24, zn + 8);
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = v[i] * gelu_d(z[i]);
                }
                st_global8(frow, v);
                st_global8(frow + 256, v + 8);
                *swz(tile, w, c0 / 8) = pack8(v);
                *swz(tile, w, c0 / 8 + 1) = pack8(v + 8);
            }
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(vready);
        }
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    tmem_free(tmem, TCOLS, warp);
}

// ---------------------------------------------------------------- projection
struct ProjBwdArgs {
    int rows, K2;
    const float *zp;
    __nv_bfloat16 *dZ;
    float *df1, *df; // both gradients in FP32 ([M][128], [M][64]; their column sums are the bias gradients)
};
template <int NT> struct ProjBwdSmem {
    __host__ __device__ static uint32_t hh(int K2) { return (uint32_t)(2 * NT * K2 * 128); }
    __host__ __device__ static uint32_t vv(int K2) { return hh(K2) + NT * 32768; }
    __host__ __device__ static uint32_t p1(int K2) { return vv(K2) + NT * 16384; }
    __host__ __device__ static uint32_t p2(int K2) { return p1(K2) + 16384; }
    __host__ __device__ static uint32_t dd(int K2) { return p2(K2) + 4096; }
    __host__ __device__ static uint32_t bars(int K2) { return dd(K2) + NT * 4096; }
    __host__ __device__ static uint32_t total(int K2) { return bars(K2) + 128 + 1024; }
};
// Row by row: dh = dout P2 -> times GELU'(zp) -> dzp (BF16 to shared memory and
// memory) -> dv = dzp P1 (in dh's TMEM columns) -> BF16 -> transform along W.
template <int NT>
__global__ void __launch_bounds__(NT * 256 + 128, 1)
    k_proj_bwd(const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmP1,
               const __grid_constant__ CUtensorMap tmP2, const __grid_constant__ CUtensorMap tmIWT,
               const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmO, ProjBwdArgs a) {
    extern __shared__ uint8_t dsmem[];
    typedef ProjBwdSmem<NT> L;
    constexpr int W = NT * 128, EW = NT * 8, P = 128;
    constexpr uint32_t TCOLS = NT == 1 ? 256 : 512;
    uint8_t *base = align1k(dsmem);
    uint8_t *sI = base, *sH = base + L::hh(a.K2), *sV = base + L::vv(a.K2), *sP1 = base + L::p1(a.K2),
            *sP2 = base + L::p2(a.K2), *sD = base + L::dd(a.K2);
    uint64_t *full = reinterpret_cast<uint64_t *>(base + L::bars(a.K2));
    uint64_t *wfull = full + 1, *dready = full + 2, *hready = full + 3, *oready = full + 4, *ofree = full + 5,
             *vready = full + 6, *fready = full + 7, *ffree = full + 8, *bfree = full + 9;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 10);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(wfull, 1);
        mbar_init(dready, 1);
        mbar_init(hready, EW);
        mbar_init(oready, 1);
        mbar_init(ofree, EW);
        mbar_init(vready, EW);
        mbar_init(fready, 1);
        mbar_init(ffree, 2);
        mbar_init(bfree, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, TCOLS, warp);
    const int r0 = blockIdx.x, step = gridDim.x, n = (a.rows - r0 + step - 1) / step;
    bool ok = true;

    if (warp == EW + 2) {
        if (lane == 0) { // TMA
            auto load = [&](int it) {
                mbar_expect_tx(full, NT * 4096);
                for (int t = 0; t < NT; ++t)
                    tma_load_2d(sD + t * 4096, &tmD, 0, (r0 + it * step) * W + t * 128, full);
            };
            mbar_expect_tx(wfull, 16384 + 4096 + 2 * NT * a.K2 * 128);
            tma_load_2d(sP1, &tmP1, 0, 0, wfull);
            for (int k = 0; k < 2; ++k) tma_load_2d(sP2 + k * 2048, &tmP2, k * 64, 0, wfull);
            for (int k = 0; k < 2 * NT; ++k) tma_load_2d(sI + k * a.K2 * 128, &tmIWT, k * 64, 0, wfull);
            int loads = 0;
            if (n > 0) load(loads++);
            for (int it = 0; ok && it < n; ++it) {
                const int m = (r0 + it * step) * W;
                ok = mbar_wait(dready, it & 1); // dout's tile has been read
                if (ok && it + 1 < n) load(loads++);
                ok = ok && mbar_wait(hready, it & 1);
                if (!ok) break;
                for (int t = 0; t < NT; ++t)
                    for (int k = 0; k < 2; ++k)
                        tma_store_2d(&tmH, k * 64, m + t * 128, sH + t * 32768 + k * 16384);
                bulk_commit();
                ok = mbar_wait(vready, it & 1);
                if (!ok) break;
                for (int t = 0; t < NT; ++t) tma_store_2d(&tmO, 0, m + t * 128, sV + t * 16384);
                bulk_commit();
                ok = mbar_wait(fready, it & 1);
                bulk_wait_read();
                mbar_arrive(bfree); // both tiles may be written again
            }
            bulk_wait();
            mbar_wait(wfull, 0);
            if (loads) mbar_wait(full, (loads - 1) & 1);
        }
        __syncwarp();
    } else if (warp == EW + 3) {
        if (lane == 0) { // MMA
            const uint32_t id1 = idesc_of(P, 0, 1), id2 = idesc_of(64, 0, 1);
            ok = mbar_wait(wfull, 0);
            auto first = [&](int it) { // dout [w][16] times P2 [16][128]
                ok = ok && mbar_wait(full, it & 1);
                if (!ok) return;
                fence_after();
                for (int t = 0; t < NT; ++t)
                    mma(tmem + t * P, sdesc_k16(smem_u32(sD + t * 4096)), sdesc_mn(smem_u32(sP2), 2048), id1, 0);
                mma_commit(dready);
            };
            if (n > 0) first(0);
            for (int it = 0; ok && it < n; ++it) {
                ok = mbar_wait(hready, it & 1);
                if (!ok) break;
                fence_after();
                for (int t = 0; t < NT; ++t) // dzp [w][128] times P1 [128][64]
                    for (int k = 0; k < 8; ++k)
                        mma(tmem + t * P, sdesc(smem_u32(sH + t * 32768 + (k >> 2) * 16384)) + K_STEP * (k & 3),
                            sdesc_mn(smem_u32(sP1), 1024) + MN_STEP * k, id2, k > 0);
                mma_commit(oready);
                ok = mbar_wait(ofree, it & 1);
                if (ok && it + 1 < n) first(it + 1);
                ok = ok && mbar_wait(vready, it & 1) && (it == 0 || mbar_wait(ffree, (it - 1) & 1));
                if (!ok) break;
                fence_after();
                for (int kb = 0; kb < 2 * NT; ++kb) {
                    const uint64_t di = sdesc(smem_u32(sI + kb * a.K2 * 128)),
                                   dv = sdesc_mn(smem_u32(sV + kb * 8192), 1024);
                    for (int k = 0; k < 4; ++k)
                        mma(tmem + NT * P, di + K_STEP * k, dv + MN_STEP * k, id2, (kb | k) > 0);
                }
                mma_commit(fready);
            }
        }
        __syncwarp();
    } else if (warp >= EW) {
        const int kp = (warp - EW) * 32 + lane;
        const uint32_t tf = tmem + NT * P + ((uint32_t)((warp - EW) * 32) << 16);
        for (int it = 0; it < n; ++it) {
            ok = mbar_wait(fready, it & 1);
            if (!ok) break;
            fence_after();
            float v[64];
            tmem_ld<32>(tf, v);
            tmem_ld<32>(tf + 32, v + 32);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ffree);
            if (kp < a.K2) {
                uint4 *o = reinterpret_cast<uint4 *>(a.dZ + ((long long)(r0 + it * step) * a.K2 + kp) * CH);
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = pack8(v + 8 * j);
            }
        }
    } else {
        const int t = (warp >> 2) % NT, q = warp & 3, rt = q * 32 + lane, w = t * 128 + rt, half = warp / (4 * NT);
        const uint32_t td = tmem + t * P + ((uint32_t)(q * 32) << 16);
        uint8_t *th = sH + t * 32768 + half * 16384, *tv = sV + t * 16384;
        for (int it = 0; it < n; ++it) {
            const long long m = (long long)(r0 + it * step) * W + w;
            const float *zrow = a.zp + m * P + half * 64;
            float *frow = a.df1 + blocked(m, half * 64, P);
            float zn[16];
            ld_global8(zrow, zn);
            ld_global8(zrow + 8, zn + 8);
            ok = mbar_wait(dready, it & 1) && (it == 0 || mbar_wait(bfree, (it - 1) & 1));
            if (!ok) break;
            fence_after();
#pragma unroll 1
            for (int c = 0; c < 64; c += 16, frow += 512) { // (one copy of GELU', as in k_row_bwd)
                float v[16], z[16];
                tmem_ld<16>(td + half * 64 + c, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) z[i] = zn[i];
                if (c < 48) {
                    ld_global8(zrow + c + 16, zn);
                    ld_global8(zrow + c + 24, zn + 8);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = v[i] * gelu_d(z[i]);
                st_global8(frow, v);
                st_global8(frow + 256, v + 8);
                *swz(th, rt, c / 8) = pack8(v);
                *swz(th, rt, c / 8 + 1) = pack8(v + 8);
            }
            fence_before();
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(hready);
            ok = mbar_wait(oready, it & 1);
            if (!ok) break;
            fence_after();
            frow = a.df + blocked(m, half * 32, CH);
#pragma unroll
            for (int c0 = 0; c0 < 32; c0 += 16, frow += 512) {
                float v[16];
                tmem_ld<16>(td + half * 32 + c0, v);
                if (c0 == 16) {
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(ofree);
                }
                st_global8(frow, v);
                st_global8(frow + 256, v + 8);
                *swz(tv, rt, half * 4 + c0 / 8) = pack8(v);
                *swz(tv, rt, half * 4 + c0 / 8 + 1) = pack8(v + 8);
            }
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(vready);
        }
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    tmem_free(tmem, TCOLS, warp);
}

// ---------------------------------------------------------------- along H
struct BwdHArgs {
    int B, H, m2, Q, pairs;
    __nv_bfloat16 *out;
};
// dV[(k2, q)][b][(c, re|im)] from dZ[b][h][(k2, re|im)][c]: the adjoint of k_inv_h
__global__ void __launch_bounds__(128) k_inv_h_bwd(const __grid_constant__ CUtensorMap tmZ,
                                                   const __grid_constant__ CUtensorMap tmI, BwdHArgs a) {
    extern __shared__ uint8_t dsmem[];
    uint8_t *base = align1k(dsmem);
    const int kb_n = 2 * a.H / 64, tile = 2 * a.H * 128, ib = 2 * a.Q * 128;
    uint8_t *sZ = base, *sI = base + 2 * tile;
    uint64_t *full = reinterpret_cast<uint64_t *>(sI + kb_n * ib), *done = full + 1;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k2 = blockIdx.x;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, 128, warp);
    int loads = 0;
    auto load = [&](int p) { // rows (h, part) x 64 channels of samples 2p and 2p + 1
        mbar_expect_tx(full, 2 * tile + (loads == 0 ? kb_n * ib : 0));
        if (loads++ == 0)
            for (int k = 0; k < kb_n; ++k) tma_load_2d(sI + k * ib, &tmI, k * 64, 0, full);
        for (int k = 0; k < 2; ++k) tma_load_5d(sZ + k * tile, &tmZ, 0, 0, k2, 0, 2 * p + k, full);
    };
    bool ok = true;
    int it = 0;
    if (threadIdx.x == 0) load(blockIdx.y);
    for (int p = blockIdx.y; p < a.pairs; p += gridDim.y, ++it) {
        if (threadIdx.x == 0 && (ok = mbar_wait(full, it & 1))) {
            fence_after();
            const uint32_t id = idesc_of(2 * a.Q, 1, 0);
            const uint64_t dz = sdesc_mn(smem_u32(sZ), tile);
            for (int k = 0; k < 2 * a.H / 16; ++k)
                mma(tmem, dz + MN_STEP * k, sdesc(smem_u32(sI + (k >> 2) * ib)) + K_STEP * (k & 3), id, k > 0);
            mma_commit(done);
        }
        const bool good = mbar_wait(done, it & 1);
        ok = ok && good;
        if (!good) break;
        fence_after();
        if (threadIdx.x == 0 && p + (int)gridDim.y < a.pairs) load(p + gridDim.y);
        const int b = 2 * p + (warp >> 1), c = (warp & 1) * 32 + lane;
        const uint32_t tr = tmem + ((uint32_t)(warp * 32) << 16);
        for (int q0 = 0; q0 < a.Q; q0 += 16) {
            float v[32]; // (q, part)
            tmem_ld<32>(tr + 2 * q0, v);
            if (b < a.B) {
                __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(a.out) +
                                    ((long long)(k2 * a.Q + q0) * a.B + b) * CH + c;
#pragma unroll
                for (int i = 0; i < 16; ++i) o[(long long)i * a.B * CH] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            }
        }
        fence_before();
        __syncthreads();
        fence_after();
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    if (threadIdx.x == 0) mbar_wait(full, (loads - 1) & 1);
    tmem_free(tmem, 128, warp);
}

// dXw[b][h][kp][c] from dU[(k2, q)][b][re|im][c]: the adjoint of k_fwd_h.  With
// g = dU: the real row of mode k2 is sum_q g_re cos - g_im sin, the imaginary
// row sum_q g_im cos + g_re sin.
__global__ void __launch_bounds__(128) k_fwd_h_bwd(const __grid_constant__ CUtensorMap tmU,
                                                   const __grid_constant__ CUtensorMap tmF, BwdHArgs a) {
    extern __shared__ uint8_t dsmem[];
    uint8_t *base = align1k(dsmem);
    const int kb_n = (2 * a.Q + 63) / 64, tile = a.Q * 128, fb = a.H * 128;
    // FHT first: its MMA reads 128 rows from each block (H = 64: into what follows, ignored)
    uint8_t *sF = base, *sU = base + kb_n * fb;
    uint64_t *full = reinterpret_cast<uint64_t *>(sU + 4 * tile + (a.H == 64 ? 8192 : 0)), *done = full + 1;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k2 = blockIdx.x;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, 256, warp);
    int loads = 0;
    auto load = [&](int p) { // tiles (re, b), (re, b + 1), (im, b), (im, b + 1): rows q x 64 channels
        mbar_expect_tx(full, 4 * tile + (loads == 0 ? kb_n * fb : 0));
        if (loads++ == 0)
            for (int k = 0; k < kb_n; ++k) tma_load_2d(sF + k * fb, &tmF, k * 64, 0, full);
        for (int k = 0; k < 4; ++k) tma_load_5d(sU + k * tile, &tmU, 0, k >> 1, 2 * p + (k & 1), 0, k2, full);
    };
    bool ok = true;
    int it = 0;
    if (threadIdx.x == 0) load(blockIdx.y);
    for (int p = blockIdx.y; p < a.pairs; p += gridDim.y, ++it) {
        if (threadIdx.x == 0 && (ok = mbar_wait(full, it & 1))) {
            fence_after();
            const uint32_t id = idesc_of(128, 0, 1), idn = idesc_of(128, 0, 1, 1);
            const uint64_t gre = sdesc_mn(smem_u32(sU), tile), gim = sdesc_mn(smem_u32(sU + 2 * tile), tile);
            const int ks = a.Q / 16;
            for (int part = 0; part < 2; ++part)
                for (int k = 0; k < 2 * ks; ++k) {
                    const uint64_t df = sdesc(smem_u32(sF + (k >> 2) * fb)) + K_STEP * (k & 3);
                    const uint64_t g = (k < ks) == (part == 0) ? gre : gim;
                    mma(tmem + part * 128, df, g + MN_STEP * (k < ks ? k : k - ks), part == 0 && k >= ks ? idn : id,
                        k > 0);
                }
            mma_commit(done);
        }
        const bool good = mbar_wait(done, it & 1);
        ok = ok && good;
        if (!good) break;
        fence_after();
        if (threadIdx.x == 0 && p + (int)gridDim.y < a.pairs) load(p + gridDim.y);
        const int h = warp * 32 + lane;
        if (warp * 32 < a.H)
            for (int part = 0; part < 2; ++part)
                for (int s = 0; s < 2; ++s) {
                    float v[64];
                    const uint32_t tr = tmem + part * 128 + s * 64 + ((uint32_t)(warp * 32) << 16);
                    tmem_ld<32>(tr, v);
                    tmem_ld<32>(tr + 32, v + 32);
                    const int b = 2 * p + s;
                    if (b >= a.B) continue;
                    uint4 *o = reinterpret_cast<uint4 *>(
                        a.out + (((long long)b * a.H + h) * 2 * a.m2 + k2 + part * a.m2) * CH);
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] = pack8(v + 8 * j);
                }
        fence_before();
        __syncthreads();
        fence_after();
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    if (threadIdx.x == 0) mbar_wait(full, (loads - 1) & 1);
    tmem_free(tmem, 256, warp);
}

// ---------------------------------------------------------------- per mode
// dU[mode][b][(part, i)] = dV[mode][b] times the transposed real block, and
// the weights' gradient dR[mode][i][o][re, im] from the block gradient
// M = dV^T U (over all samples): re = M[2o][2i] + M[2o+1][2i+1],
// im = M[2o+1][2i] - M[2o][2i+1].  C2: R's complex values, FP32 or as k_modes kept them.
__device__ __forceinline__ __nv_bfloat162 bf2(float2 c) { return __floats2bfloat162_rn(c.x, c.y); }
__device__ __forceinline__ __nv_bfloat162 bf2(__nv_bfloat162 c) { return c; }
template <class C2>
__global__ void __launch_bounds__(128) k_modes_bwd(const __grid_constant__ CUtensorMap tmV,
                                                   const __grid_constant__ CUtensorMap tmU,
                                                   const C2 *__restrict__ R, __nv_bfloat16 *__restrict__ dU,
                                                   float *__restrict__ dR, int B) {
    extern __shared__ uint8_t dsmem[];
    uint8_t *base = align1k(dsmem);
    uint8_t *sV = base, *sU = base + 32768, *sR = base + 65536;
    uint64_t *full = reinterpret_cast<uint64_t *>(sR + 32768), *done = full + 1;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mode = blockIdx.x;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, 256, warp);
    int loads = 0;
    auto load = [&](int m0) {
        ++loads;
        mbar_expect_tx(full, 65536);
        for (int k = 0; k < 2; ++k) {
            tma_load_3d(sV + k * 16384, &tmV, k * 64, m0, mode, full);
            tma_load_3d(sU + k * 16384, &tmU, k * 64, m0, mode, full);
        }
    };
    if (threadIdx.x == 0) load(0);
    // rows (part, i), columns (o, part')
    const C2 *w = R + (long long)mode * CH * CH;
#pragma unroll 4
    for (int k = threadIdx.x; k < CH * CH; k += 128) {
        const int o = k % CH, i = k / CH;
        const __nv_bfloat162 c = bf2(w[k]);
        const int col = (2 * o) % 64, off = (((col >> 3) ^ (i & 7)) << 4) + (col & 7) * 2;
        uint8_t *r0 = sR + (o / 32) * 16384 + i * 128 + off;
        *reinterpret_cast<__nv_bfloat162 *>(r0) = c;
        *reinterpret_cast<__nv_bfloat162 *>(r0 + CH * 128) = __halves2bfloat162(__hneg(c.y), c.x);
    }
    fence_async();
    __syncthreads();
    bool ok = true;
    int it = 0;
    const uint32_t tl = (uint32_t)(warp * 32) << 16;
    for (int m0 = 0; m0 < B; m0 += 128, ++it) {
        if (threadIdx.x == 0 && (ok = mbar_wait(full, it & 1))) {
            fence_after();
            const uint32_t id = idesc_of(128, 0, 0), idm = idesc_of(128, 1, 1);
            for (int k = 0; k < 8; ++k)
                mma(tmem, sdesc(smem_u32(sV + (k >> 2) * 16384)) + K_STEP * (k & 3),
                    sdesc(smem_u32(sR + (k >> 2) * 16384)) + K_STEP * (k & 3), id, k > 0);
            const int ks = (min(B - m0, 128) + 15) / 16; // samples past B are zero rows
            for (int k = 0; k < ks; ++k)
                mma(tmem + 128, sdesc_mn(smem_u32(sV), 16384) + MN_STEP * k, sdesc_mn(smem_u32(sU), 16384) + MN_STEP * k,
                    idm, it > 0 || k > 0);
            mma_commit(done);
        }
        const bool good = mbar_wait(done, it & 1);
        ok = ok && good;
        if (!good) break;
        fence_after();
        if (threadIdx.x == 0 && m0 + 128 < B) load(m0 + 128);
        const int b = m0 + warp * 32 + lane;
        if (m0 + warp * 32 < B) {
#pragma unroll
            for (int c0 = 0; c0 < 128; c0 += 32) {
                float v[32];
                tmem_ld<32>(tmem + tl + c0, v);
                if (b < B) {
                    uint4 *o = reinterpret_cast<uint4 *>(dU + ((long long)mode * B + b) * 128 + c0);
#pragma unroll
                    for (int j = 0; j < 4; ++j) o[j] = pack8(v + 8 * j);
                }
            }
        }
        fence_before();
        __syncthreads();
        fence_after();
    }
    if (ok) {
        const int row = warp * 32 + lane; // (o, part)
        float *g = dR + (long long)mode * CH * CH * 2 + row;
        for (int c0 = 0; c0 < 128; c0 += 32) { // columns (i, part')
            float v[32];
            tmem_ld<32>(tmem + 128 + tl + c0, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float y = __shfl_xor_sync(0xffffffffu, v[2 * i + 1], 1);
                g[(long long)(c0 / 2 + i) * CH * 2] = (lane & 1) ? v[2 * i] - y : v[2 * i] + y;
            }
        }
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    if (threadIdx.x == 0) mbar_wait(full, (loads - 1) & 1);
    tmem_free(tmem, 256, warp);
}

// ---------------------------------------------------------------- weights
// part[s][j][n] (or, tr, part[s][n][j]) = sum over the s-th chunk of points of
// A[m][j] B[m][n]: A of NA groups of 64 columns, B of nb <= 64, both read as
// they lie (MN-major).  Chunks are strided over the CTAs; two accumulators
// let a chunk's products start while the one before is written out.
struct WgradArgs {
    int chunks, tiles; // chunks of `tiles` x 128 points
    int rows_a, nb, tr;
    float *part;
};
template <int NA, int ST>
__global__ void __launch_bounds__(256) k_wgrad(const __grid_constant__ CUtensorMap tmA,
                                               const __grid_constant__ CUtensorMap tmB, WgradArgs a) {
    extern __shared__ uint8_t dsmem[];
    uint8_t *base = align1k(dsmem);
    constexpr uint32_t SB = (NA + 1) * 16384;
    uint64_t *full = reinterpret_cast<uint64_t *>(base + ST * SB), *empty = full + ST, *dready = empty + ST,
             *dfree = dready + 2;
    uint32_t *slot = reinterpret_cast<uint32_t *>(dfree + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int k = 0; k < 2; ++k) {
            mbar_init(&dready[k], 1);
            mbar_init(&dfree[k], 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, 128, warp);
    const int n = (a.chunks - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            int g = 0;
            for (int it = 0; ok && it < n; ++it)
                for (int k = 0; k < a.tiles; ++k, ++g) {
                    const int s = g % ST, m = ((blockIdx.x + it * gridDim.x) * a.tiles + k) * 128;
                    if (g >= ST) ok = mbar_wait(&empty[s], (g / ST - 1) & 1);
                    if (!ok) break;
                    mbar_expect_tx(&full[s], SB);
                    for (int j = 0; j < NA; ++j) tma_load_2d(base + s * SB + j * 16384, &tmA, j * 64, m, &full[s]);
                    tma_load_2d(base + s * SB + NA * 16384, &tmB, 0, m, &full[s]);
                }
            for (int q = g > ST ? g - ST : 0; q < g; ++q) mbar_wait(&full[q % ST], (q / ST) & 1);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t id = idesc_of(a.nb, 1, 1);
            int g = 0;
            for (int it = 0; ok && it < n; ++it) {
                if (it >= 2) ok = mbar_wait(&dfree[it & 1], ((it >> 1) - 1) & 1);
                for (int k = 0; ok && k < a.tiles; ++k, ++g) {
                    const int s = g % ST;
                    ok = mbar_wait(&full[s], (g / ST) & 1);
                    if (!ok) break;
                    fence_after();
                    // one group of A columns: the second half of the 128 rows is B's tile, ignored
                    const uint64_t da = sdesc_mn(smem_u32(base + s * SB), 16384),
                                   db = sdesc_mn(smem_u32(base + s * SB + NA * 16384), 1024);
                    for (int q = 0; q < 8; ++q)
                        mma(tmem + (it & 1) * 64, da + MN_STEP * q, db + MN_STEP * q, id, (k | q) > 0);
                    mma_commit(&empty[s]);
                }
                if (ok) mma_commit(&dready[it & 1]);
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        const int q = warp - 4, j = q * 32 + lane;
        for (int it = 0; it < n; ++it) {
            ok = mbar_wait(&dready[it & 1], (it >> 1) & 1);
            if (!ok) break;
            fence_after();
            float v[64];
            const uint32_t td = tmem + (it & 1) * 64 + ((uint32_t)(q * 32) << 16);
            tmem_ld<32>(td, v);
            tmem_ld<32>(td + 32, v + 32);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&dfree[it & 1]);
            float *p = a.part + (long long)(blockIdx.x + it * gridDim.x) * a.rows_a * a.nb;
            if (j < a.rows_a) {
                if (a.tr) {
#pragma unroll
                    for (int c = 0; c < 16; ++c) p[c * a.rows_a + j] = v[c]; // nb = 16
                } else {
#pragma unroll
                    for (int c = 0; c < 64; c += 8)
                        if (c < a.nb) st_global8(p + j * a.nb + c, v + c);
                }
            }
        }
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    tmem_free(tmem, 128, warp);
}

// ---------------------------------------------------------------- host
template <int NT> int run_row_bwd(const CUtensorMap *m, const RowBwdArgs &a, int grid, cudaStream_t s) {
    const uint32_t smem = BwdSmem<NT>::total(a.K2);
    if (!allow_smem(k_row_bwd<NT>, smem)) return GF_FNO_ERR_CUDA;
    k_row_bwd<NT><<<grid, NT * 256 + 128, smem, s>>>(m[0], m[1], m[2], m[3], m[4], m[5], a);
    return launched();
}
template <int NT> int run_proj_bwd(const CUtensorMap *m, const ProjBwdArgs &a, int grid, cudaStream_t s) {
    const uint32_t smem = ProjBwdSmem<NT>::total(a.K2);
    if (!allow_smem(k_proj_bwd<NT>, smem)) return GF_FNO_ERR_CUDA;
    k_proj_bwd<NT><<<grid, NT * 256 + 128, smem, s>>>(m[0], m[1], m[2], m[3], m[4], m[5], a);
    return launched();
}
template <int NA, int ST> int run_wgrad(const CUtensorMap &ma, const CUtensorMap &mb, const WgradArgs &a,
                                        cudaStream_t s) {
    const uint32_t smem = ST * (NA + 1) * 16384 + 256 + 1024;
    if (!allow_smem(k_wgrad<NA, ST>, smem)) return GF_FNO_ERR_CUDA;
    const int cap = 2 * sm_count();
    k_wgrad<NA, ST><<<a.chunks < cap ? a.chunks : cap, 256, smem, s>>>(ma, mb, a);
    return launched();
}
template <class C2>
int run_modes_bwd(const void *dV, const void *U, const C2 *R, void *dU, float *dR, int B, int modes, void *stream) {
    if (!dV || !U || !R || !dU || !dR || B < 1 || modes < 1) return GF_FNO_ERR_ARG;
    if (unaligned(dV) || unaligned(U) || unaligned(R, sizeof(C2)) || unaligned(dU)) return GF_FNO_ERR_ALIGN;
    CUtensorMap mv, mu;
    const long long d[3] = {128, B, modes}, st[2] = {128, 128LL * B};
    const int box[3] = {64, 128, 1};
    if (!map_of(&mv, dV, 3, d, st, box) || !map_of(&mu, U, 3, d, st, box)) return GF_FNO_ERR_CUDA;
    const uint32_t smem = 98304 + 64 + 1024;
    if (!allow_smem(k_modes_bwd<C2>, smem)) return GF_FNO_ERR_CUDA;
    k_modes_bwd<C2><<<modes, 128, smem, (cudaStream_t)stream>>>(mv, mu, R, (__nv_bfloat16 *)dU, dR, B);
    return launched();
}
bool bad_w(int W) { return W != 128 && W != 256 && W != 384; }
bool bad_modes(int B, int H, int m2, int Q) {
    return B < 1 || (H != 64 && H != 128) || m2 < 1 || m2 > 32 || Q % 16 || Q < 16 || Q > 64;
}

} // namespace

int gf_fno_back_error() { return take_tc_error(); }

extern "C" {

int gf_fno_row_bwd(const void *dz, const void *dXw, const void *FW, const void *Wl, const float *z, const void *IWT,
                   void *dzo, float *df, void *dZ, int rows, int W, int K2, void *stream) {
    if (!dz || !dXw || !FW || !Wl || !dzo || !df || rows < 1 || bad_w(W) || K2 < 16 || K2 > 64 || K2 % 16 ||
        (dZ && !IWT) || (long long)rows * W > 0x7fffffffLL)
        return GF_FNO_ERR_ARG;
    if (unaligned(dz) || unaligned(dXw) || unaligned(FW) || unaligned(Wl) || unaligned(z, 32) || unaligned(IWT) ||
        unaligned(dzo) || unaligned(dZ) || unaligned(df, 32))
        return GF_FNO_ERR_ALIGN;
    CUtensorMap m[6];
    const long long M = (long long)rows * W;
    if (!map2(&m[0], dz, CH, M, 128) || !map2(&m[1], dXw, CH, (long long)rows * K2, K2) || !map2(&m[2], FW, W, K2, K2) ||
        !map2(&m[3], Wl, CH, CH, 64) || !map2(&m[4], IWT ? IWT : FW, W, K2, K2) || !map2(&m[5], dzo, CH, M, 128))
        return GF_FNO_ERR_CUDA;
    RowBwdArgs a{rows, K2, z, (__nv_bfloat16 *)dZ, df};
    cudaStream_t s = (cudaStream_t)stream;
    const int sms = sm_count(), grid = rows < sms ? rows : sms;
    return W == 128 ? run_row_bwd<1>(m, a, grid, s) : W == 256 ? run_row_bwd<2>(m, a, grid, s)
                                                               : run_row_bwd<3>(m, a, grid, s);
}

int gf_fno_proj_bwd(const void *dout, const float *zp, const void *P1, const void *P2, const void *IWT, void *dzp,
                    float *df1, void *dzo, float *df, void *dZ, int rows, int W, int K2, void *stream) {
    if (!dout || !zp || !P1 || !P2 || !IWT || !dzp || !dzo || !dZ || !df1 || !df || rows < 1 || bad_w(W) ||
        K2 < 16 || K2 > 64 || K2 % 16 || (long long)rows * W > 0x7fffffffLL)
        return GF_FNO_ERR_ARG;
    if (unaligned(dout) || unaligned(zp, 32) || unaligned(P1) || unaligned(P2) || unaligned(IWT) || unaligned(dzp) ||
        unaligned(dzo) || unaligned(dZ) || unaligned(df1, 32) || unaligned(df, 32))
        return GF_FNO_ERR_ALIGN;
    CUtensorMap m[6];
    const long long M = (long long)rows * W;
    if (!map2(&m[0], dout, 16, M, 128, 16) || !map2(&m[1], P1, CH, 128, 128) || !map2(&m[2], P2, 128, 16, 16) ||
        !map2(&m[3], IWT, W, K2, K2) || !map2(&m[4], dzp, 128, M, 128) || !map2(&m[5], dzo, CH, M, 128))
        return GF_FNO_ERR_CUDA;
    ProjBwdArgs a{rows, K2, zp, (__nv_bfloat16 *)dZ, df1, df};
    cudaStream_t s = (cudaStream_t)stream;
    const int sms = sm_count(), grid = rows < sms ? rows : sms;
    return W == 128 ? run_proj_bwd<1>(m, a, grid, s) : W == 256 ? run_proj_bwd<2>(m, a, grid, s)
                                                                : run_proj_bwd<3>(m, a, grid, s);
}

int gf_fno_inv_h_bwd(const void *dZ, const void *IHT, void *dV, int B, int H, int m2, int Q, void *stream) {
    if (!dZ || !IHT || !dV || bad_modes(B, H, m2, Q)) return GF_FNO_ERR_ARG;
    if (unaligned(dZ) || unaligned(IHT) || unaligned(dV)) return GF_FNO_ERR_ALIGN;
    CUtensorMap mz, mi;
    const long long d[5] = {CH, 2, m2, H, B}, st[4] = {CH, 2 * CH, 2LL * m2 * CH, 2LL * m2 * CH * H};
    const int box[5] = {CH, 2, 1, H, 1};
    if (!map_of(&mz, dZ, 5, d, st, box) || !map2(&mi, IHT, 2 * H, 2 * Q, 2 * Q)) return GF_FNO_ERR_CUDA;
    const uint32_t smem = 2 * 2 * H * 128 + (2 * H / 64) * 2 * Q * 128 + 64 + 1024;
    if (!allow_smem(k_inv_h_bwd, smem)) return GF_FNO_ERR_CUDA;
    BwdHArgs a{B, H, m2, Q, (B + 1) / 2, (__nv_bfloat16 *)dV};
    const int per = (2 * sm_count() + m2 - 1) / m2, gy = a.pairs < per ? a.pairs : per;
    k_inv_h_bwd<<<dim3(m2, gy), 128, smem, (cudaStream_t)stream>>>(mz, mi, a);
    return launched();
}

int gf_fno_fwd_h_bwd(const void *dU, const void *FHT, void *dXw, int B, int H, int m2, int Q, void *stream) {
    if (!dU || !FHT || !dXw || bad_modes(B, H, m2, Q)) return GF_FNO_ERR_ARG;
    if (unaligned(dU) || unaligned(FHT) || unaligned(dXw)) return GF_FNO_ERR_ALIGN;
    CUtensorMap mu, mf;
    const long long d[5] = {CH, 2, B, Q, m2}, st[4] = {CH, 2 * CH, 2LL * CH * B, 2LL * CH * B * Q};
    const int box[5] = {CH, 1, 1, Q, 1};
    if (!map_of(&mu, dU, 5, d, st, box) || !map2(&mf, FHT, 2 * Q, H, H)) return GF_FNO_ERR_CUDA;
    const uint32_t smem = ((2 * Q + 63) / 64) * H * 128 + 4 * Q * 128 + (H == 64 ? 8192 : 0) + 64 + 1024;
    if (!allow_smem(k_fwd_h_bwd, smem)) return GF_FNO_ERR_CUDA;
    BwdHArgs a{B, H, m2, Q, (B + 1) / 2, (__nv_bfloat16 *)dXw};
    const int per = (2 * sm_count() + m2 - 1) / m2, gy = a.pairs < per ? a.pairs : per;
    k_fwd_h_bwd<<<dim3(m2, gy), 128, smem, (cudaStream_t)stream>>>(mu, mf, a);
    return launched();
}

int gf_fno_modes_bwd(const void *dV, const void *U, const float *R, void *dU, float *dR, int B, int modes,
                     void *stream) {
    return run_modes_bwd(dV, U, (const float2 *)R, dU, dR, B, modes, stream);
}
int gf_fno_modes_bwd_kept(const void *dV, const void *U, const void *Rb, void *dU, float *dR, int B, int modes,
                          void *stream) {
    return run_modes_bwd(dV, U, (const __nv_bfloat162 *)Rb, dU, dR, B, modes, stream);
}

int gf_fno_wgrad(const void *A, int na, const void *B, int nb, int transposed, float *part, long long M, int chunks,
                 void *stream) {
    if (!A || !B || !part || (na != 64 && na != 128) || (nb != 16 && nb != 32 && nb != 48 && nb != 64) || chunks < 1 ||
        M < 1 || M > 0x7fffffffLL || M % chunks || (M / chunks) % 128 || (transposed && nb != 16))
        return GF_FNO_ERR_ARG;
    if (unaligned(A) || unaligned(B) || unaligned(part, 32)) return GF_FNO_ERR_ALIGN;
    CUtensorMap ma, mb;
    if (!map2(&ma, A, na, M, 128) || !map2(&mb, B, nb, M, 128)) return GF_FNO_ERR_CUDA;
    WgradArgs a{chunks, (int)(M / chunks / 128), na, nb, transposed, part};
    cudaStream_t s = (cudaStream_t)stream;
    return na == 128 ? run_wgrad<2, 2>(ma, mb, a, s) : run_wgrad<1, 3>(ma, mb, a, s);
}

} // extern "C"
