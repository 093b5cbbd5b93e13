// ps_nn_conv.cu -- 3x3 convolutions of the warm-start network as implicit GEMMs on the tensor cores
// (tcgen05): y[p][n] = act(sum over taps and channels of x[p + tap][c] * W[n][tap][c] + bias[n]), bf16
// operands, FP32 accumulation in tensor memory, bf16 result. No column matrix is formed: a tap's 128
// input pixels by KC channels are one 4-D TMA box of the NHWC activations, shifted by the tap, and the
// pixels outside the image arrive as the zero fill that "same" padding wants.
//
// A tile is 128 output pixels -- a box of bw x bh x bb pixels of x, y and image, powers of two chosen on
// the host so that the fewest tiles cover the layer -- by BN output channels. Persistent and
// warp-specialised like the GEMM (ps_nn_gemm.cu): warp 0 feeds a ring of A (pixels) and B (weights)
// blocks, warp 1 issues the MMAs into one of two accumulators, warps 2-5 add the bias, apply ReLU and
// store while the next tile's MMAs run; every wait is bounded, and a wait that gives up raises
// DEV_ERR_TMA_TIMEOUT, drains the copies in flight and frees the tensor memory. Two CTAs share an SM (the
// rings are sized for that; 2 BN accumulator columns each leave tensor memory for both).
//
// KC = 64 channels (128-byte swizzle rows) where cin is a multiple of 64, else 32 (64-byte rows).
// BN: 32 columns for narrow layers; 128 where the layer has tiles enough to fill the GPU, smaller where
// splitting the channels over more CTAs is what fills it.
//
// Bound: L2 -> shared memory (each input value is loaded once per tap). @@
#include <cuda_bf16.h>

#include <algorithm>

#include "ps_common.cuh"
#include "ps_nn.cuh"
#include "ps_nn_tc.cuh"

namespace ps {

constexpr int kConvM = 128;
template <int BN, int KC>
struct ConvCfg {
    static constexpr int ABYTES = kConvM * KC * 2, BBYTES = BN * KC * 2, STAGE = ABYTES + BBYTES;
    static constexpr int S = (100 * 1024) / STAGE;  // ring stages: 76 to 113 KB, so that two CTAs fit an SM, not three
    static constexpr int SMEM = S * STAGE + 1024 + 256;
    static_assert(S >= 3 && SMEM > 77 * 1024 && SMEM < 113 * 1024, "two CTAs per SM");
    static constexpr uint32_t TMEM = 2 * BN;  // two accumulators; two CTAs' columns fit the SM's 512
};

// The pixel box of a tile (log2 extents) and the layer.
struct ConvGeom {
    int B, H, W, cin, cout;
    int lw, lh, lb;            // bw = 1 << lw, ...
    int tx, ty, tn, ntiles;    // tiles along x, y, channels; all tiles
};

template <int BN, int KC>
__global__ void __launch_bounds__(192, 2)
    nn_conv3_k(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB, ConvGeom g,
               const float* __restrict__ bias, int relu, __nv_bfloat16* __restrict__ y, int* __restrict__ err) {
    using C = ConvCfg<BN, KC>;
    constexpr int S = C::S;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * C::STAGE);
    uint64_t* empty = full + S;
    uint64_t* tfull = empty + S;    // [2] accumulator ready (MMA -> epilogue)
    uint64_t* tempty = tfull + 2;   // [2] accumulator drained (epilogue warps -> MMA)
    uint64_t* done = tempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    int* counts = reinterpret_cast<int*>(tmem_slot + 1);  // [0] stages filled, [1] stages consumed
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cblk = g.cin / KC, KB = 9 * cblk;  // K blocks of a tile: taps, channel blocks fastest

    if (threadIdx.x == 0) {
        prefetch_tensormap(&mA);
        prefetch_tensormap(&mB);
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], 4);  // one arrival per epilogue warp
        }
        mbar_init(done, 1);
        counts[0] = counts[1] = 0;
        fence_mbar_init();
    }
    if (warp == 0) tc_alloc(tmem_slot, C::TMEM);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // the previous layer's activations
    grid_dependency_wait();
    grid_dependents_may_launch();

    if (threadIdx.x == 0) {  // TMA producer
        int it = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < g.ntiles && ok; t += gridDim.x) {
            const int n0 = (t % g.tn) * BN, m = t / g.tn;
            const int x0 = (m % g.tx) << g.lw, y0 = ((m / g.tx) % g.ty) << g.lh, b0 = (m / (g.tx * g.ty)) << g.lb;
            for (int tap = 0; tap < 9 && ok; tap++)
                for (int cb = 0; cb < cblk; cb++, it++) {
                    const int s = it % S;
                    // stage s was last read by the MMAs of ring step it - S
                    if (it >= S && !mbar_wait_bounded(&empty[s], ((it / S) - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    unsigned char* st = smem + s * C::STAGE;
                    mbar_arrive_expect_tx(&full[s], C::STAGE);
                    tma_load_4d(st, &mA, &full[s], cb * KC, x0 + tap % 3 - 1, y0 + tap / 3 - 1, b0);
                    tma_load_2d(st + C::ABYTES, &mB, &full[s], tap * g.cin + cb * KC, n0);
                }
        }
        counts[0] = it;
        if (!ok) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
    } else if (threadIdx.x == 32) {  // MMA issuer
        constexpr uint32_t idesc = umma_idesc_bf16(kConvM, BN);
        int it = 0, j = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < g.ntiles && ok; t += gridDim.x, j++) {
            const int acc = j & 1, use = j >> 1;
            // the epilogue must have drained this accumulator's previous tile (its (use-1)th phase)
            if (use >= 1 && !mbar_wait_bounded(&tempty[acc], (use - 1) & 1)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)(acc * BN);
            for (int i = 0; i < KB; i++, it++) {
                const int s = it % S;
                if (!mbar_wait_bounded(&full[s], (it / S) & 1)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sa = smem_u32(smem + s * C::STAGE);
                const uint64_t da = KC == 64 ? umma_desc_sw128(sa) : umma_desc_sw64(sa);
                const uint64_t db = KC == 64 ? umma_desc_sw128(sa + C::ABYTES) : umma_desc_sw64(sa + C::ABYTES);
#pragma unroll
                for (int k = 0; k < KC / 16; k++)  // K = 16 per MMA: +32 bytes along the swizzled row
                    tc_mma(d, da + 2 * k, db + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                tc_commit(&empty[s]);
            }
            if (!ok) break;
            tc_commit(&tfull[acc]);  // arrives when this tile's MMAs have completed
        }
        counts[1] = it;
        if (!ok) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
        tc_commit(done);  // arrives when every MMA issued above has completed
    } else if (warp >= 2) {  // epilogue: warp w reads TMEM lanes (tile rows) 32 (w % 4) .. + 31
        const int q = warp & 3, row = q * 32 + lane;
        const int rx = row & ((1 << g.lw) - 1), ry = (row >> g.lw) & ((1 << g.lh) - 1), rb = row >> (g.lw + g.lh);
        int j = 0;
        for (int t = blockIdx.x; t < g.ntiles; t += gridDim.x, j++) {
            const int n0 = (t % g.tn) * BN, m = t / g.tn;
            const int px = ((m % g.tx) << g.lw) + rx, py = (((m / g.tx) % g.ty) << g.lh) + ry,
                      pb = ((m / (g.tx * g.ty)) << g.lb) + rb;
            const int acc = j & 1, use = j >> 1;
            // warp-uniform: tcgen05.ld below is a warp-collective instruction
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&tfull[acc], use & 1))) {
                if (lane == 0) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
                break;
            }
            tc_fence_after();
            const bool ok = px < g.W && py < g.H && pb < g.B;
            __nv_bfloat16* o = y + (((int64_t)pb * g.H + py) * g.W + px) * g.cout + n0;
            const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN);
#pragma unroll 2
            for (int c = 0; c < BN; c += 16) {
                float v[16];
                tc_ld16(tl + (uint32_t)c, v);  // whole warp, no divergence
                uint4 w[2];
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(w);
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 bv = __ldg(reinterpret_cast<const float4*>(bias + n0 + c + i));
                    const float lo = relu ? 0.0f : -INFINITY;
                    h[i / 2] = __floats2bfloat162_rn(fmaxf(v[i] + bv.x, lo), fmaxf(v[i + 1] + bv.y, lo));
                    h[i / 2 + 1] = __floats2bfloat162_rn(fmaxf(v[i + 2] + bv.z, lo), fmaxf(v[i + 3] + bv.w, lo));
                }
                if (ok) {
                    reinterpret_cast<uint4*>(o + c)[0] = w[0];
                    reinterpret_cast<uint4*>(o + c)[1] = w[1];
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive1(&tempty[acc]);
        }
    }
    __syncwarp();
    if (!mbar_wait_bounded(done, 0) && threadIdx.x == 0) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
    tc_fence_after();
    __syncthreads();  // counts[] visible
    if (threadIdx.x == 0 && counts[1] < counts[0])  // a wait gave up: drain the copies still in flight
        for (int i = counts[1]; i < counts[0]; i++) mbar_wait_bounded(&full[i % S], (i / S) & 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tc_dealloc(tmem, C::TMEM);
}

template <int BN, int KC>
static int conv3_launch(ConvGeom g, const void* x, const void* wgt, const float* bias, int relu, void* y, int sms,
                        cudaStream_t s, int* d_err) {
    using C = ConvCfg<BN, KC>;
    g.tn = g.cout / BN;
    const int bw = 1 << g.lw, bh = 1 << g.lh, bb = 1 << g.lb;
    const int64_t nt = (int64_t)g.tx * g.ty * ((g.B + bb - 1) / bb) * g.tn;
    if (nt > 0x7FFFFFFF - 65536) return fail(PS_ERR_SHAPE, "nn_conv3: layer too large");
    g.ntiles = (int)nt;
    CUtensorMap mA, mB;
    const uint64_t da[4] = {(uint64_t)g.cin, (uint64_t)g.W, (uint64_t)g.H, (uint64_t)g.B};
    const uint32_t ba[4] = {KC, (uint32_t)bw, (uint32_t)bh, (uint32_t)bb};
    const uint64_t db[2] = {(uint64_t)g.cin * 9, (uint64_t)g.cout};
    const uint32_t b2[2] = {KC, BN};
    PS_TRY(encode_bf16_box(&mA, x, 4, da, ba));
    PS_TRY(encode_bf16_box(&mB, wgt, 2, db, b2));
    // every launch sets it: the attribute belongs to the device's current context
    PS_CUDA_TRY(cudaFuncSetAttribute(nn_conv3_k<BN, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    const int grid = (int)std::min<int64_t>(nt, 2 * (int64_t)std::max(1, sms));
    PS_CUDA_TRY(launch_dependent(nn_conv3_k<BN, KC>, dim3((unsigned)grid), dim3(192), (size_t)C::SMEM, s, mA, mB, g, bias,
                                 relu, static_cast<__nv_bfloat16*>(y), d_err));
    return PS_OK;
}

int nn_conv3_tc(const void* x, int B, int H, int W, int cin, const void* wgt, int cout, const float* bias, int relu,
                void* y, cudaStream_t s, int* d_err) {
    if (cin % 32 || cout % 32 || B < 1 || H < 1 || W < 1) return fail(PS_ERR_SHAPE, "nn_conv3: layer %d -> %d", cin, cout);
    ConvGeom g{};
    g.B = B;
    g.H = H;
    g.W = W;
    g.cin = cin;
    g.cout = cout;
    // the box of 128 pixels that covers the layer in the fewest tiles; wide boxes first (longer contiguous runs)
    int64_t best = INT64_MAX;
    for (int lw = 7; lw >= 0; lw--)
        for (int lh = 7 - lw; lh >= 0; lh--) {
            const int lb = 7 - lw - lh;
            const int64_t tx = (W + (1 << lw) - 1) >> lw, ty = (H + (1 << lh) - 1) >> lh, tb = (B + (1 << lb) - 1) >> lb;
            if (tx * ty * tb < best) {
                best = tx * ty * tb;
                g.lw = lw;
                g.lh = lh;
                g.lb = lb;
                g.tx = (int)tx;
                g.ty = (int)ty;
            }
        }
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    // 128 channels per tile where that still gives every SM a tile, else 64, else 32
    const int bn = cout % 128 == 0 && best * (cout / 128) >= st->num_sms  ? 128
                   : cout % 64 == 0 && best * (cout / 64) >= st->num_sms ? 64
                                                                         : 32;
    auto run = [&](auto k) {
        constexpr int KC = decltype(k)::value;
        return bn == 128  ? conv3_launch<128, KC>(g, x, wgt, bias, relu, y, st->num_sms, s, d_err)
               : bn == 64 ? conv3_launch<64, KC>(g, x, wgt, bias, relu, y, st->num_sms, s, d_err)
                          : conv3_launch<32, KC>(g, x, wgt, bias, relu, y, st->num_sms, s, d_err);
    };
    return cin % 64 == 0 ? run(std::integral_constant<int, 64>{}) : run(std::integral_constant<int, 32>{});
}

}  // namespace ps
