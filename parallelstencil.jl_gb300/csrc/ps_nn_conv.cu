// ps_nn_conv.cu -- 3x3 convolutions of the warm-start network as implicit GEMMs on the tensor cores
// (tcgen05): y[p][n] = act(sum over taps and channels of x[p + tap][c] * W[n][tap][c] + bias[n]), bf16
// operands, FP32 accumulation in tensor memory, bf16 result. No column matrix is formed: a tap's 128
// input pixels by KC channels are one 4-D TMA box of the NHWC activations, shifted by the tap, and the
// pixels outside the image arrive as the zero fill that "same" padding wants. In layers whose rows fill
// tiles of 128 pixels the three taps of a kernel row share one load (ROW below).
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
// BN: 64 channels where the layer then still has a tile for every SM, else 32: splitting the channels over more
// CTAs is what fills the GPU.
//
// Bound: L2 -> shared memory. 8 images of 256^2, GPU time of a layer: 32 -> 32 channels 31 us, 96 -> 32 75 us
// (41 and 118 with every tap's pixels loaded by themselves); the 64-channel layers at a quarter of the
// size 10 to 16 us, the 128- and 256-channel ones 7 to 19 us. The whole forward pass: 7.52 ms through
// column matrices, 0.38 ms now.
#include <cuda_bf16.h>

#include <algorithm>

#include "ps_common.cuh"
#include "ps_nn.cuh"
#include "ps_nn_tc.cuh"

namespace ps {

constexpr int kConvM = 128;
// ROW: a tile is 128 pixels of one image row, and a ring stage holds the 130 pixels that the three taps of
// one kernel row need, loaded once: a tap's A operand is the same block read from one pixel further on
// (swizzling goes by the address, so a descriptor may start at any row of it), with the weights of the
// three taps beside it. DEEP: one CTA per SM with twice the stages, for layers with fewer tiles than SMs.
template <int BN, int KC, bool ROW, bool DEEP>
struct ConvCfg {
    static constexpr int TAPS = ROW ? 3 : 1;  // taps per stage
    static constexpr int ABOX = (ROW ? kConvM + 2 : kConvM) * KC * 2, ABYTES = (ABOX + 1023) / 1024 * 1024;
    static constexpr int BBYTES = BN * KC * 2, STAGE = ABYTES + TAPS * BBYTES;
    // 76 to 113 KB of stages, so that two CTAs fit an SM, not three; DEEP: one
    static constexpr int S = (DEEP ? 200 * 1024 : 105 * 1024) / STAGE;
    static constexpr int SMEM = S * STAGE + 1024 + 512;
    static_assert(S >= 2 && (DEEP ? SMEM > 115 * 1024 && SMEM < 226 * 1024 : SMEM > 77 * 1024 && SMEM < 113 * 1024),
                  "CTAs per SM");
    static constexpr uint32_t TMEM = 2 * BN;  // two accumulators; two CTAs' columns fit the SM's 512
};

// The pixel box of a tile (log2 extents) and the layer.
struct ConvGeom {
    int B, H, W, cin, cout;
    int lw, lh, lb;            // bw = 1 << lw, ...
    int tx, ty, tn, ntiles;    // tiles along x, y, channels; all tiles
};

template <int BN, int KC, bool ROW, bool DEEP>
__global__ void __launch_bounds__(192, 2)
    nn_conv3_k(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB, ConvGeom g,
               const float* __restrict__ bias, int relu, __nv_bfloat16* __restrict__ y, int* __restrict__ err) {
    using C = ConvCfg<BN, KC, ROW, DEEP>;
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
    const int cblk = g.cin / KC, KB = 9 / C::TAPS * cblk;  // ring steps of a tile: taps, channel blocks fastest

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
            for (int tap = 0; tap < 9 && ok; tap += C::TAPS)
                for (int cb = 0; cb < cblk; cb++, it++) {
                    const int s = it % S;
                    // stage s was last read by the MMAs of ring step it - S
                    if (it >= S && !mbar_wait_bounded(&empty[s], ((it / S) - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    unsigned char* st = smem + s * C::STAGE;
                    mbar_arrive_expect_tx(&full[s], C::ABOX + C::TAPS * C::BBYTES);
                    tma_load_4d(st, &mA, &full[s], cb * KC, x0 + tap % 3 - 1, y0 + tap / 3 - 1, b0);
#pragma unroll
                    for (int d = 0; d < C::TAPS; d++)
                        tma_load_2d(st + C::ABYTES + d * C::BBYTES, &mB, &full[s], (tap + d) * g.cin + cb * KC, n0);
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
#pragma unroll
                for (int e = 0; e < C::TAPS; e++) {
                    const uint32_t pa = sa + e * KC * 2, pb = sa + C::ABYTES + e * C::BBYTES;
                    const uint64_t da = KC == 64 ? umma_desc_sw128(pa) : umma_desc_sw64(pa);
                    const uint64_t db = KC == 64 ? umma_desc_sw128(pb) : umma_desc_sw64(pb);
#pragma unroll
                    for (int k = 0; k < KC / 16; k++)  // K = 16 per MMA: +32 bytes along the swizzled row
                        tc_mma(d, da + 2 * k, db + 2 * k, idesc, (i > 0 || e > 0 || k > 0) ? 1u : 0u);
                }
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

template <int BN, int KC, bool ROW, bool DEEP>
static int conv3_launch(const ConvGeom& g, const void* x, const void* wgt, const float* bias, int relu, void* y, int sms,
                        cudaStream_t s, int* d_err) {
    using C = ConvCfg<BN, KC, ROW, DEEP>;
    CUtensorMap mA, mB;
    const uint64_t da[4] = {(uint64_t)g.cin, (uint64_t)g.W, (uint64_t)g.H, (uint64_t)g.B};
    const uint32_t ba[4] = {KC, ROW ? kConvM + 2u : 1u << g.lw, 1u << g.lh, 1u << g.lb};
    const uint64_t db[2] = {(uint64_t)g.cin * 9, (uint64_t)g.cout};
    const uint32_t b2[2] = {KC, BN};
    PS_TRY(encode_bf16_box(&mA, x, 4, da, ba));
    PS_TRY(encode_bf16_box(&mB, wgt, 2, db, b2));
    const auto kernel = nn_conv3_k<BN, KC, ROW, DEEP>;
    // every launch sets it: the attribute belongs to the device's current context
    PS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    const int grid = std::min(g.ntiles, (DEEP ? 1 : 2) * sms);
    PS_CUDA_TRY(launch_dependent(kernel, dim3((unsigned)grid), dim3(192), (size_t)C::SMEM, s, mA, mB, g, bias, relu,
                                 static_cast<__nv_bfloat16*>(y), d_err));
    return PS_OK;
}

int nn_conv3_tc(const void* x, int B, int H, int W, int cin, const void* wgt, int cout, const float* bias, int relu,
                void* y, cudaStream_t s, int* d_err) {
    if (cin % 32 || cout % 32 || B < 1 || H < 1 || W < 1) return fail(PS_ERR_SHAPE, "nn_conv3: layer %d -> %d", cin, cout);
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    ConvGeom g{};
    g.B = B;
    g.H = H;
    g.W = W;
    g.cin = cin;
    g.cout = cout;
    // Whole rows of 128 pixels where at least three quarters of them are in the image: the input is read three
    // times instead of nine. Else the box of 128 pixels that covers the layer in the fewest tiles, wide
    // boxes first (longer contiguous runs).
    const bool row = W % kConvM == 0 || W % kConvM >= 3 * kConvM / 4 || (W > kConvM && W % kConvM >= kConvM / 2);
    int64_t best = INT64_MAX;
    for (int lw = 7; lw >= (row ? 7 : 0); lw--)
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
    // 64 channels per tile where that still gives every SM a tile, else 32
    const int bn = cout % 64 == 0 && best * (cout / 64) >= st->num_sms ? 64 : 32;
    g.tn = cout / bn;
    if (best * g.tn > 0x7FFFFFFF - 65536) return fail(PS_ERR_SHAPE, "nn_conv3: layer too large");
    g.ntiles = (int)(best * g.tn);
    const bool deep = g.ntiles < st->num_sms;
    auto run = [&](auto k, auto r, auto d) {
        constexpr int KC = decltype(k)::value;
        constexpr bool R = decltype(r)::value, D = decltype(d)::value;
        if constexpr (!D)  // (64 channels are taken only where there are tiles for every SM)
            if (bn == 64) return conv3_launch<64, KC, R, D>(g, x, wgt, bias, relu, y, st->num_sms, s, d_err);
        return conv3_launch<32, KC, R, D>(g, x, wgt, bias, relu, y, st->num_sms, s, d_err);
    };
    auto kc = [&](auto r, auto d) {
        return cin % 64 == 0 ? run(std::integral_constant<int, 64>{}, r, d) : run(std::integral_constant<int, 32>{}, r, d);
    };
    if (deep) return row ? kc(std::true_type{}, std::true_type{}) : kc(std::false_type{}, std::true_type{});
    return row ? kc(std::true_type{}, std::false_type{}) : kc(std::false_type{}, std::false_type{});
}

}  // namespace ps
