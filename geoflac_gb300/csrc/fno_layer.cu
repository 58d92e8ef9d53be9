// The surrogate's forward pass as five fused tcgen05 kernels (64 channels):
//
//   k_row    one grid row (b, h) of W points x 64 channels per CTA pass:
//            z = v Wl^T + bias + IW Z (1x1 mixing and the inverse DFT along
//            W, two TMEM accumulators), GELU, the row's new activations into
//            shared memory and out by TMA, and from there its forward DFT
//            along W for the next layer (the lift is the same kernel without
//            the spectral term);
//   k_fwd_h  forward DFT along H of one W-mode for two samples and the complex
//            bookkeeping -> the per-mode spectra U;
//   k_modes  per-mode complex mixing, the real 2C x 2C block built from the
//            FP32 weights in shared memory;
//   k_inv_h  inverse DFT along H of one W-mode for two samples -> Z;
//   k_proj   64 -> 128, GELU, 128 -> 16 of one grid row.
//
// What bounds them and why this split: the layer-by-layer GEMMs moved the
// activations five times per layer (transposes into the DFT's K-major layout,
// the spectral term in FP32, the product's read-modify-write).  tcgen05 takes
// a channels-last row as an MN-major operand, so no transposed copy exists
// here; the FP32 spectral term stays in TMEM; an activation is read once and
// written once per layer.  Sums, their order and every BF16 rounding are those
// of the GEMM path, so the results are the same bits.  A row CTA is then bound
// by the GELU's erff (about 30 instructions per value, half of them on the
// half-rate ALU pipe), for which 24 epilogue warps, half of the channels each,
// share the SM with one TMA and one MMA warp.
// The new activations have a tile of their own, so that the next row's load
// starts when the products have read v, not when the row is stored.
// Measured at 64 samples of 128 x 384 points (ncu): k_row 160 us for the lift
// and 286 us per layer (12 warps writing in place: 302), k_proj 422 us (12
// warps that wait for the row's second product: 453), k_fwd_h 17, k_modes 27
// and k_inv_h 30 us; the forecast of 64 members 2.27 -> 2.17 ms (by GEMMs layer
// by layer 11.9).
//
// Every mbarrier wait is bounded; a wait that gives up raises the error flag
// that gf_gemm_error() reads.

#include "fno_tc.cuh"

namespace {

// ---------------------------------------------------------------- rows
struct RowArgs {
    int rows, K2, kin, act;
    const float *bias;
    float *z;              // FP32 pre-activations (training), or null
    __nv_bfloat16 *Xw;     // [rows][K2][64]: the new activations' DFT along W, or null
    int has_spec, store_v; // spectral term present; activations written
};
// shared memory of k_row: the DFT matrix of the forward transform first (its
// MMA reads 128 rows from every 64-column block and ignores all but K2, so
// 16 KB past the last block must stay inside), then IW, Wl, Z, v and the new v
template <int NT> struct RowSmem {
    __host__ __device__ static uint32_t iw(int K2) { return (uint32_t)(2 * NT * K2 * 128); }
    __host__ __device__ static uint32_t wl(int K2) { return iw(K2) + NT * 16384; }
    __host__ __device__ static uint32_t zz(int K2) { return wl(K2) + 8192; }
    __host__ __device__ static uint32_t vv(int K2) { return zz(K2) + 8192; }
    __host__ __device__ static uint32_t oo(int K2) { return vv(K2) + NT * 16384; }
    __host__ __device__ static uint32_t bars(int K2) { return oo(K2) + NT * 16384; }
    __host__ __device__ static uint32_t total(int K2) { return bars(K2) + 512 + 1024; }
};

// warps 0 .. 8 NT - 1: epilogue of point tile (warp / 4) % NT, half of the
// channels each; then two warps for the DFT's accumulator, the TMA warp and the
// MMA warp
template <int NT>
__global__ void __launch_bounds__(NT * 256 + 128, 1)
    k_row(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmZ,
          const __grid_constant__ CUtensorMap tmIW, const __grid_constant__ CUtensorMap tmW,
          const __grid_constant__ CUtensorMap tmFW, const __grid_constant__ CUtensorMap tmO, RowArgs a) {
    extern __shared__ uint8_t dsmem[];
    typedef RowSmem<NT> L;
    constexpr int W = NT * 128, EW = NT * 8;
    constexpr uint32_t TCOLS = NT == 1 ? 256 : 512;
    uint8_t *base = align1k(dsmem);
    uint8_t *sFW = base, *sIW = base + L::iw(a.K2), *sW = base + L::wl(a.K2), *sZ = base + L::zz(a.K2),
            *sV = base + L::vv(a.K2), *sO = base + L::oo(a.K2);
    uint64_t *full = reinterpret_cast<uint64_t *>(base + L::bars(a.K2));
    uint64_t *ofree = full + 1, *wfull = full + 2, *dready = full + 3, *dfree = full + 4, *vready = full + 5,
             *fready = full + 6, *ffree = full + 7;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 8);
    float *sbias = reinterpret_cast<float *>(full + 10);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool has_fw = a.Xw != nullptr;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(ofree, 1);
        mbar_init(wfull, 1);
        mbar_init(dready, 1);
        mbar_init(dfree, EW);
        mbar_init(vready, EW);
        mbar_init(fready, 1);
        mbar_init(ffree, 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < CH) sbias[threadIdx.x] = a.bias[threadIdx.x];
    const uint32_t tmem = tmem_alloc(slot, TCOLS, warp);
    const int r0 = blockIdx.x, n = (a.rows - r0 + (int)gridDim.x - 1) / (int)gridDim.x; // rows r0 + it * gridDim.x
    bool ok = true;

    if (warp == EW + 2) {
        if (lane == 0) { // TMA
            const uint32_t bytes = NT * 16384 + (a.has_spec ? a.K2 * 128 : 0);
            int loaded = 0;
            auto load = [&]() {
                const int r = r0 + loaded++ * (int)gridDim.x;
                mbar_expect_tx(full, bytes);
                for (int t = 0; t < NT; ++t) tma_load_2d(sV + t * 16384, &tmV, 0, r * W + t * 128, full);
                if (a.has_spec) tma_load_2d(sZ, &tmZ, 0, r * a.K2, full);
            };
            mbar_expect_tx(wfull, 8192 + (a.has_spec ? NT * 16384 : 0) + (has_fw ? 2 * NT * a.K2 * 128 : 0));
            tma_load_2d(sW, &tmW, 0, 0, wfull);
            if (a.has_spec)
                for (int t = 0; t < NT; ++t) tma_load_2d(sIW + t * 16384, &tmIW, 0, t * 128, wfull);
            if (has_fw)
                for (int k = 0; k < 2 * NT; ++k) tma_load_2d(sFW + k * a.K2 * 128, &tmFW, k * 64, 0, wfull);
            if (n > 0) load();
            if (n > 1) {
                ok = mbar_wait(dready, 0); // row 0's products have read v and Z
                if (ok) load();
            }
            for (int it = 0; ok && it < n; ++it) {
                ok = mbar_wait(vready, it & 1);
                if (!ok) break;
                if (a.store_v) {
                    for (int t = 0; t < NT; ++t)
                        tma_store_2d(&tmO, 0, (r0 + it * (int)gridDim.x) * W + t * 128, sO + t * 16384);
                    bulk_commit();
                }
                if (it + 2 < n) { // before the store's and the DFT's reads are waited for
                    ok = mbar_wait(dready, (it + 1) & 1);
                    if (!ok) break;
                    load();
                }
                if (has_fw) ok = mbar_wait(fready, it & 1);
                bulk_wait_read();
                mbar_arrive(ofree);
            }
            bulk_wait();
            // no copy of this CTA is in flight when it ends, on any path
            mbar_wait(wfull, 0);
            if (loaded > 0) mbar_wait(full, (loaded - 1) & 1);
        }
        __syncwarp();
    } else if (warp == EW + 3) {
        if (lane == 0) { // MMA
            const uint32_t id = idesc_of(64, 0, 0), ids = idesc_of(64, 0, 1);
            ok = mbar_wait(wfull, 0);
            auto mix = [&](int it) {
                ok = ok && mbar_wait(full, it & 1);
                if (!ok) return;
                fence_after();
                const uint64_t dw = sdesc(smem_u32(sW)), dz = sdesc_mn(smem_u32(sZ), 1024);
                for (int t = 0; t < NT; ++t) {
                    const uint64_t dv = sdesc(smem_u32(sV + t * 16384));
                    for (int k = 0; k < a.kin / 16; ++k)
                        mma(tmem + t * 64, dv + K_STEP * k, dw + K_STEP * k, id, k > 0);
                    if (a.has_spec) {
                        const uint64_t di = sdesc(smem_u32(sIW + t * 16384));
                        for (int k = 0; k < a.K2 / 16; ++k)
                            mma(tmem + (NT + t) * 64, di + K_STEP * k, dz + MN_STEP * k, ids, k > 0);
                    }
                }
                mma_commit(dready);
            };
            if (n > 0) mix(0);
            for (int it = 0; ok && it < n; ++it) {
                if (it + 1 < n) {
                    ok = mbar_wait(dfree, it & 1);
                    if (ok) mix(it + 1);
                }
                if (has_fw && ok) {
                    ok = mbar_wait(vready, it & 1) && (it == 0 || mbar_wait(ffree, (it - 1) & 1));
                    if (!ok) break;
                    fence_after();
                    for (int kb = 0; kb < 2 * NT; ++kb) {
                        const uint64_t df = sdesc(smem_u32(sFW + kb * a.K2 * 128)),
                                       dv = sdesc_mn(smem_u32(sO + kb * 8192), 1024);
                        for (int k = 0; k < 4; ++k)
                            mma(tmem + 2 * NT * 64, df + K_STEP * k, dv + MN_STEP * k, ids, (kb | k) > 0);
                    }
                    mma_commit(fready);
                }
            }
        }
        __syncwarp();
    } else if (warp >= EW) {
        if (has_fw) { // the DFT's rows: lanes 0 .. K2 - 1
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
                    uint4 *o = reinterpret_cast<uint4 *>(
                        a.Xw + ((long long)(r0 + it * (int)gridDim.x) * a.K2 + kp) * CH);
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] = pack8(v + 8 * j);
                }
            }
        }
    } else {
        const int t = (warp >> 2) % NT, q = warp & 3, w = t * 128 + q * 32 + lane, ch = warp / (4 * NT) * 32;
        const uint32_t td = tmem + t * 64 + ((uint32_t)(q * 32) << 16);
        for (int it = 0; it < n; ++it) {
            ok = mbar_wait(dready, it & 1);
            if (!ok) break;
            fence_after();
            float *zrow = a.z ? a.z + ((long long)(r0 + it * (int)gridDim.x) * W + w) * CH : nullptr;
#pragma unroll 1
            for (int c0 = ch; c0 < ch + 32; c0 += 16) { // (one copy of the GELU's code)
                float v[16];
                tmem_ld<16>(td + c0, v);
                if (a.has_spec) {
                    float s[16];
                    tmem_ld<16>(td + NT * 64 + c0, s);
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = (v[i] + sbias[c0 + i]) + s[i];
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = v[i] + sbias[c0 + i];
                }
                if (c0 == ch + 16) { // this warp's part of both accumulators is in registers
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(dfree);
                }
                if (zrow) {
#pragma unroll
                    for (int i = 0; i < 16; i += 8) st_global8(zrow + c0 + i, v + i);
                }
                if (a.act) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = act_gelu(v[i]);
                }
                if (c0 == ch && it > 0) { // row it - 1's new activations are stored and transformed
                    ok = mbar_wait(ofree, (it - 1) & 1);
                    if (!ok) break;
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) *swz(sO, w, c0 / 8 + j) = pack8(v + 8 * j);
            }
            if (!ok) break;
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(vready);
        }
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    tmem_free(tmem, TCOLS, warp);
}

// ---------------------------------------------------------------- projection
struct ProjArgs {
    int rows;
    const float *b1, *b2;
    float *zp;   // FP32 pre-activations [M][128] (training), or null
    int store_h; // BF16 activations [M][128] written
    float *out;  // [M][16]
};
template <int NT>
__global__ void __launch_bounds__(NT * 256 + 64, 1)
    k_proj(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmP1,
           const __grid_constant__ CUtensorMap tmP2, const __grid_constant__ CUtensorMap tmH, ProjArgs a) {
    extern __shared__ uint8_t dsmem[];
    constexpr int W = NT * 128, EW = NT * 8, P = 128, CO = 16;
    constexpr uint32_t TCOLS = NT == 1 ? 256 : 512;
    uint8_t *base = align1k(dsmem);
    uint8_t *sV = base, *sH = sV + 2 * NT * 16384, *sP1 = sH + NT * 32768, *sP2 = sP1 + 16384;
    uint64_t *full = reinterpret_cast<uint64_t *>(sP2 + 4096);
    uint64_t *wfull = full + 2, *dready = full + 3, *dfree = full + 4, *hready = full + 5, *oready = full + 6,
             *hfree = full + 7;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 8);
    float *sb1 = reinterpret_cast<float *>(full + 10), *sb2 = sb1 + P;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_init(wfull, 1);
        mbar_init(dready, 1);
        mbar_init(dfree, EW);
        mbar_init(hready, EW);
        mbar_init(oready, 1);
        mbar_init(hfree, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < P) sb1[threadIdx.x] = a.b1[threadIdx.x];
    if (threadIdx.x < CO) sb2[threadIdx.x] = a.b2[threadIdx.x];
    const uint32_t tmem = tmem_alloc(slot, TCOLS, warp);
    const int r0 = blockIdx.x, n = (a.rows - r0 + (int)gridDim.x - 1) / (int)gridDim.x;
    bool ok = true;

    if (warp == EW) {
        if (lane == 0) { // TMA
            auto load = [&](int it) {
                const int s = it & 1, r = r0 + it * (int)gridDim.x;
                mbar_expect_tx(&full[s], NT * 16384);
                for (int t = 0; t < NT; ++t)
                    tma_load_2d(sV + (s * NT + t) * 16384, &tmV, 0, r * W + t * 128, &full[s]);
            };
            mbar_expect_tx(wfull, 16384 + 4096);
            tma_load_2d(sP1, &tmP1, 0, 0, wfull);
            for (int k = 0; k < 2; ++k) tma_load_2d(sP2 + k * 2048, &tmP2, k * 64, 0, wfull);
            int loaded = 0;
            for (; loaded < 2 && loaded < n; ++loaded) load(loaded);
            for (int it = 0; ok && it < n; ++it) {
                ok = mbar_wait(hready, it & 1); // the row's first product has read v
                if (!ok) break;
                if (it + 2 < n) load(loaded++);
                if (a.store_h) {
                    for (int t = 0; t < NT; ++t)
                        for (int k = 0; k < 2; ++k)
                            tma_store_2d(&tmH, k * 64, (r0 + it * (int)gridDim.x) * W + t * 128,
                                         sH + t * 32768 + k * 16384);
                    bulk_commit();
                    bulk_wait_read();
                }
                mbar_arrive(hfree);
            }
            bulk_wait();
            mbar_wait(wfull, 0);
            for (int q = loaded > 2 ? loaded - 2 : 0; q < loaded; ++q) mbar_wait(&full[q & 1], (q >> 1) & 1);
        }
        __syncwarp();
    } else if (warp == EW + 1) {
        if (lane == 0) { // MMA
            const uint32_t id1 = idesc_of(P, 0, 0), id2 = idesc_of(CO, 0, 0);
            ok = mbar_wait(wfull, 0);
            auto first = [&](int it) {
                const int s = it & 1;
                ok = ok && mbar_wait(&full[s], (it >> 1) & 1);
                if (!ok) return;
                fence_after();
                const uint64_t dp = sdesc(smem_u32(sP1));
                for (int t = 0; t < NT; ++t) {
                    const uint64_t dv = sdesc(smem_u32(sV + (s * NT + t) * 16384));
                    for (int k = 0; k < 4; ++k) mma(tmem + t * P, dv + K_STEP * k, dp + K_STEP * k, id1, k > 0);
                }
                mma_commit(dready);
            };
            if (n > 0) first(0);
            for (int it = 0; ok && it < n; ++it) {
                if (it + 1 < n) {
                    ok = mbar_wait(dfree, it & 1);
                    if (ok) first(it + 1);
                }
                ok = ok && mbar_wait(hready, it & 1);
                if (!ok) break;
                fence_after();
                for (int t = 0; t < NT; ++t)
                    for (int kb = 0; kb < 2; ++kb) {
                        const uint64_t dh = sdesc(smem_u32(sH + t * 32768 + kb * 16384)),
                                       dp = sdesc(smem_u32(sP2 + kb * 2048));
                        for (int k = 0; k < 4; ++k)
                            mma(tmem + NT * P + t * CO, dh + K_STEP * k, dp + K_STEP * k, id2, (kb | k) > 0);
                    }
                mma_commit(oready);
            }
        }
        __syncwarp();
    } else {
        const int t = (warp >> 2) % NT, q = warp & 3, rt = q * 32 + lane, w = t * 128 + rt, half = warp / (4 * NT);
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const uint32_t td = tmem + t * P + lanes, to = tmem + NT * P + t * CO + lanes;
        uint8_t *tile = sH + t * 32768 + half * 16384;
        // the second product of row it - 1 is read and stored after the first
        // chunk of row it is computed, which hides it
        auto finish = [&](int it) {
            if (!mbar_wait(oready, it & 1)) return false;
            if (half) return true;
            fence_after();
            float o[16];
            tmem_ld<16>(to, o);
            fence_before();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = o[i] + sb2[i];
            float *out = a.out + ((long long)(r0 + it * (int)gridDim.x) * W + w) * CO;
            st_global8(out, o);
            st_global8(out + 8, o + 8);
            return true;
        };
        for (int it = 0; ok && it < n; ++it) {
            ok = mbar_wait(dready, it & 1);
            if (!ok) break;
            fence_after();
            const long long m = (long long)(r0 + it * (int)gridDim.x) * W + w;
#pragma unroll 1
            for (int c = 0; c < 64; c += 16) { // (one copy of the GELU's code, as in k_row)
                const int c0 = half * 64 + c;
                float v[16];
                tmem_ld<16>(td + c0, v);
                if (c == 48) {
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(dfree);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = v[i] + sb1[c0 + i];
                if (a.zp) {
#pragma unroll
                    for (int i = 0; i < 16; i += 8) st_global8(a.zp + m * P + c0 + i, v + i);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = act_gelu(v[i]);
                if (c == 0 && it > 0) { // row it - 1: its product has read the tile, its copy out too
                    ok = finish(it - 1) && mbar_wait(hfree, (it - 1) & 1);
                    if (!ok) break;
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) *swz(tile, rt, c / 8 + j) = pack8(v + 8 * j);
            }
            if (!ok) break;
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(hready);
        }
        if (ok && n > 0) ok = finish(n - 1);
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    tmem_free(tmem, TCOLS, warp);
}
template <int NT> constexpr uint32_t proj_smem() {
    return NT * (32768 + 32768) + 16384 + 4096 + 1024 + 1024;
}

// ---------------------------------------------------------------- along H
// U[(k2, q)][b][(c, re|im)] of W-mode k2 = blockIdx.x, for pairs of samples
struct FwdHArgs {
    int B, H, m2, Q, pairs;
    __nv_bfloat16 *U;
};
__global__ void __launch_bounds__(128) k_fwd_h(const __grid_constant__ CUtensorMap tmX,
                                               const __grid_constant__ CUtensorMap tmF, FwdHArgs a) {
    extern __shared__ uint8_t dsmem[];
    uint8_t *base = align1k(dsmem);
    const int kb_n = (a.H + 63) / 64, tile = a.H * 128, fb = 2 * a.Q * 128;
    uint8_t *sX = base, *sF = base + 4 * tile;
    uint64_t *full = reinterpret_cast<uint64_t *>(sF + kb_n * fb), *done = full + 1;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k2 = blockIdx.x;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, 256, warp);
    int loads = 0;
    auto load = [&](int p) { // tiles (b, re), (b + 1, re), (b, im), (b + 1, im): rows h x 64 channels
        ++loads;
        mbar_expect_tx(full, 4 * tile + (p == (int)blockIdx.y ? kb_n * fb : 0));
        if (p == (int)blockIdx.y)
            for (int k = 0; k < kb_n; ++k) tma_load_2d(sF + k * fb, &tmF, k * 64, 0, full);
        for (int k = 0; k < 4; ++k) tma_load_4d(sX + k * tile, &tmX, 0, k2 + (k >> 1) * a.m2, 0, 2 * p + (k & 1), full);
    };
    bool ok = true;
    int it = 0;
    if (threadIdx.x == 0) load(blockIdx.y);
    for (int p = blockIdx.y; p < a.pairs; p += gridDim.y, ++it) {
        if (threadIdx.x == 0 && (ok = mbar_wait(full, it & 1))) {
            fence_after();
            const uint32_t id = idesc_of(2 * a.Q, 1, 0);
            for (int part = 0; part < 2; ++part) {
                const uint64_t dx = sdesc_mn(smem_u32(sX + 2 * part * tile), tile);
                for (int k = 0; k < a.H / 16; ++k)
                    mma(tmem + part * 128, dx + MN_STEP * k, sdesc(smem_u32(sF + (k >> 2) * fb)) + K_STEP * (k & 3), id,
                        k > 0);
            }
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
            float rc[16], rs[16], ic[16], is[16]; // cosine and sine sums of the real and imaginary parts
            tmem_ld<16>(tr + q0, rc);
            tmem_ld<16>(tr + a.Q + q0, rs);
            tmem_ld<16>(tr + 128 + q0, ic);
            tmem_ld<16>(tr + 128 + a.Q + q0, is);
            if (b < a.B) {
                __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(a.U) +
                                    ((long long)(k2 * a.Q + q0) * a.B + b) * CH + c;
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    o[(long long)i * a.B * CH] = __floats2bfloat162_rn(rc[i] + is[i], ic[i] - rs[i]);
            }
        }
        fence_before();
        __syncthreads();
        fence_after();
    }
    if (!ok) atomicExch(&g_tc_err, 1);
    if (threadIdx.x == 0) mbar_wait(full, (loads - 1) & 1); // the last load has landed
    tmem_free(tmem, 256, warp);
}

// Z[b][h][k2][re|im][c] of W-mode k2 = blockIdx.x from V[(k2, q)][b][re|im][c]
struct InvHArgs {
    int B, H, m2, Q, pairs;
    __nv_bfloat16 *Z;
};
__global__ void __launch_bounds__(128) k_inv_h(const __grid_constant__ CUtensorMap tmV,
                                               const __grid_constant__ CUtensorMap tmI, InvHArgs a) {
    extern __shared__ uint8_t dsmem[];
    uint8_t *base = align1k(dsmem);
    const int kb_n = (2 * a.Q + 63) / 64, tile = 2 * a.Q * 128, ib = 2 * a.H * 128, mt = 2 * a.H / 128;
    uint8_t *sI = base, *sX = base + kb_n * ib;
    uint64_t *full = reinterpret_cast<uint64_t *>(sX + 2 * tile), *done = full + 1;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k2 = blockIdx.x;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, 256, warp);
    int loads = 0;
    auto load = [&](int p) { // rows (q, part) x 64 channels of samples 2p and 2p + 1
        ++loads;
        mbar_expect_tx(full, 2 * tile + (p == (int)blockIdx.y ? kb_n * ib : 0));
        if (p == (int)blockIdx.y)
            for (int k = 0; k < kb_n; ++k) tma_load_2d(sI + k * ib, &tmI, k * 64, 0, full);
        for (int k = 0; k < 2; ++k) tma_load_5d(sX + k * tile, &tmV, 0, 0, 2 * p + k, 0, k2, full);
    };
    bool ok = true;
    int it = 0;
    if (threadIdx.x == 0) load(blockIdx.y);
    for (int p = blockIdx.y; p < a.pairs; p += gridDim.y, ++it) {
        if (threadIdx.x == 0 && (ok = mbar_wait(full, it & 1))) {
            fence_after();
            const uint32_t id = idesc_of(128, 0, 1);
            const uint64_t dx = sdesc_mn(smem_u32(sX), tile);
            for (int t = 0; t < mt; ++t)
                for (int k = 0; k < 2 * a.Q / 16; ++k)
                    mma(tmem + t * 128, sdesc(smem_u32(sI + (k >> 2) * ib + t * 16384)) + K_STEP * (k & 3),
                        dx + MN_STEP * k, id, k > 0);
            mma_commit(done);
        }
        const bool good = mbar_wait(done, it & 1);
        ok = ok && good;
        if (!good) break;
        fence_after();
        if (threadIdx.x == 0 && p + (int)gridDim.y < a.pairs) load(p + gridDim.y);
        for (int t = 0; t < mt; ++t) {
            const int hr = t * 128 + warp * 32 + lane, h = hr >> 1, part = hr & 1;
            for (int s = 0; s < 2; ++s) {
                float v[64];
                const uint32_t tr = tmem + t * 128 + s * 64 + ((uint32_t)(warp * 32) << 16);
                tmem_ld<32>(tr, v);
                tmem_ld<32>(tr + 32, v + 32);
                const int b = 2 * p + s;
                if (b >= a.B) continue;
                uint4 *o = reinterpret_cast<uint4 *>(
                    a.Z + ((((long long)b * a.H + h) * a.m2 + k2) * 2 + part) * CH);
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = pack8(v + 8 * j);
            }
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
// V[mode][b][(part, o)] = sum over (i, part') of U[mode][b][(i, part')] times
// the mode's real block, built from R[mode][i][o][re, im]:
//   out_re = sum_i u_re re - u_im im ; out_im = sum_i u_re im + u_im re
// Rb: R as it was multiplied by, in BF16, for the backward pass (null: not kept).
__global__ void __launch_bounds__(128) k_modes(const __grid_constant__ CUtensorMap tmU, const float *__restrict__ R,
                                               __nv_bfloat16 *__restrict__ V, __nv_bfloat162 *__restrict__ Rb, int B) {
    extern __shared__ uint8_t dsmem[];
    uint8_t *base = align1k(dsmem);
    uint8_t *sU = base, *sR = base + 32768;
    uint64_t *full = reinterpret_cast<uint64_t *>(sR + 32768), *done = full + 1;
    uint32_t *slot = reinterpret_cast<uint32_t *>(full + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mode = blockIdx.x;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_alloc(slot, 128, warp);
    int loads = 0;
    auto load = [&](int m0) {
        ++loads;
        mbar_expect_tx(full, 32768);
        for (int k = 0; k < 2; ++k) tma_load_3d(sU + k * 16384, &tmU, k * 64, m0, mode, full);
    };
    if (threadIdx.x == 0) load(0);
    // rows (part, o), columns (i, part'): two input channels at a time
    const float2 *w = reinterpret_cast<const float2 *>(R) + (long long)mode * CH * CH;
#pragma unroll 4
    for (int k = threadIdx.x; k < CH * CH; k += 128) {
        const int o = k % CH, i = k / CH;
        const float2 c = w[k];
        const int col = (2 * i) % 64, off = (((col >> 3) ^ (o & 7)) << 4) + (col & 7) * 2;
        uint8_t *r0 = sR + (i / 32) * 16384 + o * 128 + off; // (CH + o) & 7 == o & 7
        *reinterpret_cast<__nv_bfloat162 *>(r0) = __floats2bfloat162_rn(c.x, -c.y);
        *reinterpret_cast<__nv_bfloat162 *>(r0 + CH * 128) = __floats2bfloat162_rn(c.y, c.x);
        if (Rb) Rb[(long long)mode * CH * CH + k] = __floats2bfloat162_rn(c.x, c.y);
    }
    fence_async();
    __syncthreads();
    bool ok = true;
    int it = 0;
    for (int m0 = 0; m0 < B; m0 += 128, ++it) {
        if (threadIdx.x == 0 && (ok = mbar_wait(full, it & 1))) {
            fence_after();
            const uint32_t id = idesc_of(128, 0, 0);
            for (int k = 0; k < 8; ++k)
                mma(tmem, sdesc(smem_u32(sU + (k >> 2) * 16384)) + K_STEP * (k & 3),
                    sdesc(smem_u32(sR + (k >> 2) * 16384)) + K_STEP * (k & 3), id, k > 0);
            mma_commit(done);
        }
        const bool good = mbar_wait(done, it & 1);
        ok = ok && good;
        if (!good) break;
        fence_after();
        if (threadIdx.x == 0 && m0 + 128 < B) load(m0 + 128);
        const int b = m0 + warp * 32 + lane;
        const uint32_t tr = tmem + ((uint32_t)(warp * 32) << 16);
        if (m0 + warp * 32 < B) {
#pragma unroll
            for (int c0 = 0; c0 < 128; c0 += 32) {
                float v[32];
                tmem_ld<32>(tr + c0, v);
                if (b < B) {
                    uint4 *o = reinterpret_cast<uint4 *>(V + ((long long)mode * B + b) * 128 + c0);
#pragma unroll
                    for (int j = 0; j < 4; ++j) o[j] = pack8(v + 8 * j);
                }
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

// ---------------------------------------------------------------- host
template <int NT> int run_row(const CUtensorMap *m, const RowArgs &a, cudaStream_t s) {
    const uint32_t smem = RowSmem<NT>::total(a.K2);
    if (!allow_smem(k_row<NT>, smem)) return GF_FNO_ERR_CUDA;
    const int sms = sm_count(), grid = a.rows < sms ? a.rows : sms;
    k_row<NT><<<grid, NT * 256 + 128, smem, s>>>(m[0], m[1], m[2], m[3], m[4], m[5], a);
    return launched();
}
template <int NT> int run_proj(const CUtensorMap *m, const ProjArgs &a, cudaStream_t s) {
    if (!allow_smem(k_proj<NT>, proj_smem<NT>())) return GF_FNO_ERR_CUDA;
    const int sms = sm_count(), grid = a.rows < sms ? a.rows : sms;
    k_proj<NT><<<grid, NT * 256 + 64, proj_smem<NT>(), s>>>(m[0], m[1], m[2], m[3], a);
    return launched();
}

} // namespace

int gf_fno_layer_error() { return take_tc_error(); }

extern "C" {

int gf_fno_layer_ok(int H, int W, int C, int m2, int Q, int cin, int P, int cout) {
    return C == CH && (W == 128 || W == 256 || W == 384) && (H == 64 || H == 128) && (2 * m2) % 16 == 0 &&
           2 * m2 <= 64 && Q % 16 == 0 && Q <= 64 && cin % 16 == 0 && cin <= 64 && P == 128 && cout == 16;
}

int gf_fno_row(const void *v, int kin, const void *Z, const void *IW, const void *Wl, const float *bias, int act,
               const void *FW, float *z, void *vout, void *Xw, int rows, int W, int K2, void *stream) {
    if (!v || !Wl || !bias || rows < 1 || (W != 128 && W != 256 && W != 384) || K2 < 16 || K2 > 64 || K2 % 16 ||
        kin < 16 || kin > CH || kin % 16 || (Z && !IW) || (Xw && !FW) || (!vout && !Xw) ||
        (long long)rows * W > 0x7fffffffLL)
        return GF_FNO_ERR_ARG;
    if (unaligned(v) || unaligned(Z) || unaligned(IW) || unaligned(Wl) || unaligned(FW) || unaligned(vout) ||
        unaligned(Xw) || unaligned(z, 32))
        return GF_FNO_ERR_ALIGN;
    CUtensorMap m[6];
    const long long M = (long long)rows * W;
    if (!map2(&m[0], v, kin, M, 128) || !map2(&m[1], Z ? Z : v, Z ? CH : kin, Z ? (long long)rows * K2 : M, K2) ||
        !map2(&m[2], IW ? IW : Wl, IW ? K2 : kin, IW ? W : CH, IW ? 128 : 64) || !map2(&m[3], Wl, kin, CH, 64) ||
        !map2(&m[4], FW ? FW : Wl, FW ? W : kin, FW ? K2 : CH, FW ? K2 : 64) ||
        !map2(&m[5], vout ? vout : v, vout ? CH : kin, M, 128))
        return GF_FNO_ERR_CUDA;
    RowArgs a{rows, K2, kin, act, bias, z, (__nv_bfloat16 *)Xw, Z ? 1 : 0, vout ? 1 : 0};
    cudaStream_t s = (cudaStream_t)stream;
    return W == 128 ? run_row<1>(m, a, s) : W == 256 ? run_row<2>(m, a, s) : run_row<3>(m, a, s);
}

int gf_fno_fwd_h(const void *Xw, const void *FH, void *U, int B, int H, int m2, int Q, void *stream) {
    if (!Xw || !FH || !U || B < 1 || (H != 64 && H != 128) || m2 < 1 || Q % 16 || Q < 16 || Q > 64 || m2 > 32)
        return GF_FNO_ERR_ARG;
    if (unaligned(Xw) || unaligned(FH) || unaligned(U)) return GF_FNO_ERR_ALIGN;
    CUtensorMap mx, mf;
    const long long d[4] = {CH, 2 * m2, H, B}, st[3] = {CH, 2LL * m2 * CH, 2LL * m2 * CH * H};
    const int box[4] = {CH, 1, H, 1};
    if (!map_of(&mx, Xw, 4, d, st, box) || !map2(&mf, FH, H, 2 * Q, 2 * Q)) return GF_FNO_ERR_CUDA;
    const uint32_t smem = 4 * H * 128 + (H / 64) * 2 * Q * 128 + 64 + 1024;
    if (!allow_smem(k_fwd_h, smem)) return GF_FNO_ERR_CUDA;
    FwdHArgs a{B, H, m2, Q, (B + 1) / 2, (__nv_bfloat16 *)U};
    // two CTAs per SM in all (their shared memory and TMEM), each over a share of the pairs
    const int per = (2 * sm_count() + m2 - 1) / m2, gy = a.pairs < per ? a.pairs : per;
    k_fwd_h<<<dim3(m2, gy), 128, smem, (cudaStream_t)stream>>>(mx, mf, a);
    return launched();
}

int gf_fno_modes_keep(const void *U, const float *R, void *V, void *Rb, int B, int modes, void *stream) {
    if (!U || !R || !V || B < 1 || modes < 1) return GF_FNO_ERR_ARG;
    if (unaligned(U) || unaligned(R, 8) || unaligned(V) || unaligned(Rb, 4)) return GF_FNO_ERR_ALIGN;
    CUtensorMap mu;
    const long long d[3] = {128, B, modes}, st[2] = {128, 128LL * B};
    const int box[3] = {64, 128, 1};
    if (!map_of(&mu, U, 3, d, st, box)) return GF_FNO_ERR_CUDA;
    const uint32_t smem = 65536 + 64 + 1024;
    if (!allow_smem(k_modes, smem)) return GF_FNO_ERR_CUDA;
    k_modes<<<modes, 128, smem, (cudaStream_t)stream>>>(mu, R, (__nv_bfloat16 *)V, (__nv_bfloat162 *)Rb, B);
    return launched();
}
int gf_fno_modes(const void *U, const float *R, void *V, int B, int modes, void *stream) {
    return gf_fno_modes_keep(U, R, V, nullptr, B, modes, stream);
}

int gf_fno_inv_h(const void *V, const void *IH, void *Z, int B, int H, int m2, int Q, void *stream) {
    if (!V || !IH || !Z || B < 1 || (H != 64 && H != 128) || m2 < 1 || m2 > 32 || Q % 16 || Q < 16 || Q > 64)
        return GF_FNO_ERR_ARG;
    if (unaligned(V) || unaligned(IH) || unaligned(Z)) return GF_FNO_ERR_ALIGN;
    CUtensorMap mv, mi;
    const long long d[5] = {CH, 2, B, Q, m2}, st[4] = {CH, 2 * CH, 2LL * CH * B, 2LL * CH * B * Q};
    const int box[5] = {CH, 2, 1, Q, 1};
    if (!map_of(&mv, V, 5, d, st, box) || !map2(&mi, IH, 2 * Q, 2 * H, 2 * H)) return GF_FNO_ERR_CUDA;
    const uint32_t smem = ((2 * Q + 63) / 64) * 2 * H * 128 + 2 * 2 * Q * 128 + 64 + 1024;
    if (!allow_smem(k_inv_h, smem)) return GF_FNO_ERR_CUDA;
    InvHArgs a{B, H, m2, Q, (B + 1) / 2, (__nv_bfloat16 *)Z};
    const int per = (2 * sm_count() + m2 - 1) / m2, gy = a.pairs < per ? a.pairs : per;
    k_inv_h<<<dim3(m2, gy), 128, smem, (cudaStream_t)stream>>>(mv, mi, a);
    return launched();
}

int gf_fno_proj(const void *v, const void *P1, const float *b1, const void *P2, const float *b2, float *zp, void *h,
                float *out, int rows, int W, void *stream) {
    if (!v || !P1 || !b1 || !P2 || !b2 || !out || rows < 1 || (W != 128 && W != 256 && W != 384) ||
        (long long)rows * W > 0x7fffffffLL)
        return GF_FNO_ERR_ARG;
    if (unaligned(v) || unaligned(P1) || unaligned(P2) || unaligned(h) || unaligned(zp, 32) || unaligned(out, 32))
        return GF_FNO_ERR_ALIGN;
    CUtensorMap m[4];
    const long long M = (long long)rows * W;
    if (!map2(&m[0], v, CH, M, 128) || !map2(&m[1], P1, CH, 128, 128) || !map2(&m[2], P2, 128, 16, 16) ||
        !map2(&m[3], h ? h : v, h ? 128 : CH, M, 128))
        return GF_FNO_ERR_CUDA;
    ProjArgs a{rows, b1, b2, zp, h ? 1 : 0, out};
    cudaStream_t s = (cudaStream_t)stream;
    return W == 128 ? run_proj<1>(m, a, s) : W == 256 ? run_proj<2>(m, a, s) : run_proj<3>(m, a, s);
}

} // extern "C"
