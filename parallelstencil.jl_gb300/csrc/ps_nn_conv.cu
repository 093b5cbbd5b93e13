// ps_nn_conv.cu -- 3x3 convolutions of the warm-start network as implicit GEMMs on the tensor cores
// (tcgen05): y[p][n] = relu(sum over taps and channels of x[p + tap][c] * W[n][tap][c] + bias[n]), bf16
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
// Layers with 32 outputs on whole rows, and the first layer, have kernels of their own below.
//
// Bound: L2 -> shared memory, and for the small layers the chain of launch, loads and MMAs. 8 images of 256^2, GPU
// time of a layer: the 64-channel layers at a quarter of the size 10 to 16 us, the 128- and 256-channel
// ones 7 to 19 us. The whole forward pass: 7.52 ms through column matrices, 0.26 ms now.
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
               const float* __restrict__ bias, __nv_bfloat16* __restrict__ y, int* __restrict__ err) {
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
                    h[i / 2] = __floats2bfloat162_rn(fmaxf(v[i] + bv.x, 0.0f), fmaxf(v[i + 1] + bv.y, 0.0f));
                    h[i / 2 + 1] = __floats2bfloat162_rn(fmaxf(v[i + 2] + bv.z, 0.0f), fmaxf(v[i + 3] + bv.w, 0.0f));
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
static int conv3_launch(const ConvGeom& g, const void* x, const void* wgt, const float* bias, void* y, int sms,
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
    PS_CUDA_TRY(launch_dependent(kernel, dim3((unsigned)grid), dim3(192), (size_t)C::SMEM, s, mA, mB, g, bias,
                                 static_cast<__nv_bfloat16*>(y), d_err));
    return PS_OK;
}

// ---- layers with 32 output channels on many rows ------------------------------------------------------
// A CTA walks down a strip of 128 pixels: every input row is loaded once and serves the three output rows that
// its kernel rows reach, whose accumulators lie beside each other in tensor memory. The weights stay in
// shared memory, ordered [kernel column][channel block][kernel row 2, 1, 0][output] so that one MMA of
// N = 96 columns adds a kernel column of all three (its 32-column form would leave two thirds of the tensor
// pipe idle: the A operand is read from shared memory once per MMA whatever N is). The accumulators are a ring of
// eight; a row's newest output starts with an MMA of its own that does not accumulate.
// With `last` the 1x1 output layer is computed from the row's rounded activations in the same epilogue.
// 8 images of 256^2: 32 -> 32 channels 21 us (31 in tiles of nn_conv3_k), 96 -> 32 43 us (75), 32 -> 32 with the
// output layer 25 us (39, and 15 by itself). Bound with 96 channels by the MMAs' operand reads (7 KB of shared
// memory per 128 x 96 x 16, about 110 cycles), with 32 by the per-row chain of load, MMAs and epilogue.
constexpr int kAccs = 8;  // accumulators of 32 columns: two CTAs fill the SM's 512
//
// UB > 0: the first UB blocks of 32 channels are a quarter-size layer's, upsampled to the nearest, which nobody
// has written out: four more warps copy its row once for every four input rows into two buffers in turn, each
// pixel to its four (the layout is the one TMA would store); RB blocks come by TMA. The layer over the
// largest concatenation (64 + 32 channels) so takes 45 us by itself, instead of 28 to write its input and 43.
template <int RB, int UB>
struct RowsCfg {
    static constexpr int CB = RB + UB, THREADS = UB ? 320 : 192;
    static constexpr int ABOX = (kConvM + 2) * 64, ABYTES = (ABOX + 1023) / 1024 * 1024;
    static constexpr int WBYTES = 3 * CB * 3 * 32 * 64;  // [kx][cb][ky][32 outputs] rows of 64 bytes
    static constexpr int S = UB ? 2 : 8;
    static constexpr int UBYTES = 2 * UB * ABYTES;
    static constexpr int SMEM = WBYTES + S * ABYTES + UBYTES + 1024 + 1024;
    static_assert(SMEM > 77 * 1024 && SMEM < 113 * 1024, "two CTAs per SM");
};
struct RowsGeom {
    int B, H, W;
    int tx, chunks, rows, jobs;  // strips per image, chunks of `rows` output rows per strip, all jobs
};
struct LastLayer {  // y[p][0..2] = W a[p] + b over the 32 channels; y NULL: none
    const __nv_bfloat16* w;
    int kpad;
    const float* b;
    float* y;
};

template <int RB, int UB>
__global__ void __launch_bounds__(RowsCfg<RB, UB>::THREADS, 2)
    nn_conv3_rows_k(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB, RowsGeom g,
                    const uint4* __restrict__ low, const float* __restrict__ bias, __nv_bfloat16* __restrict__ y,
                    LastLayer last, int* __restrict__ err) {
    using C = RowsCfg<RB, UB>;
    constexpr int S = C::S, CB = C::CB, CIN = 32 * CB;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* ring = smem + C::WBYTES;
    unsigned char* ups = ring + S * C::ABYTES;  // [2][UB] blocks of upsampled pixels
    uint64_t* full = reinterpret_cast<uint64_t*>(ups + C::UBYTES);
    uint64_t* empty = full + S;
    uint64_t* ufull = empty + S;        // [2] a row of upsampled pixels has been written
    uint64_t* uempty = ufull + 2;       // [2] and read by its last MMAs
    uint64_t* wfull = uempty + 2;       // the weights have arrived
    uint64_t* afull = wfull + 1;        // [kAccs] an output row's MMAs have completed
    uint64_t* aempty = afull + kAccs;   // [kAccs] its accumulator has been read
    uint64_t* done = aempty + kAccs;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    int* counts = reinterpret_cast<int*>(tmem_slot + 1);  // [0] stages filled, [1] stages consumed
    float* sw = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(counts + 2) + 15) & ~(uintptr_t)15);  // [3][32]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        prefetch_tensormap(&mA);
        prefetch_tensormap(&mB);
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int u = 0; u < 2; u++) {
            mbar_init(&ufull[u], 128);
            mbar_init(&uempty[u], 1);
        }
        mbar_init(wfull, 1);
        for (int a = 0; a < kAccs; a++) {
            mbar_init(&afull[a], 1);
            mbar_init(&aempty[a], 4);  // one arrival per epilogue warp
        }
        mbar_init(done, 1);
        counts[0] = counts[1] = 0;
        fence_mbar_init();
    }
    if (warp == 0) tc_alloc(tmem_slot, kAccs * 32);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // the previous layer's activations
    grid_dependency_wait();
    if (last.y) {
        for (int i = threadIdx.x; i < 96; i += blockDim.x) sw[i] = __bfloat162float(last.w[(i / 32) * last.kpad + i % 32]);
        __syncthreads();
    }

    auto job = [&](int t, int* x0, int* b, int* o0, int* o1) {
        const int c = t % g.chunks, m = t / g.chunks;
        *x0 = (m % g.tx) * kConvM;
        *b = m / g.tx;
        *o0 = c * g.rows;
        *o1 = min(g.H, *o0 + g.rows);
    };
    int x0, b, o0, o1;
    if (threadIdx.x == 0) {  // TMA producer
        mbar_arrive_expect_tx(wfull, C::WBYTES);
        for (int kx = 0; kx < 3; kx++)
            for (int cb = 0; cb < CB; cb++)
                for (int j = 0; j < 3; j++)  // kernel row 2 - j
                    tma_load_2d(smem + ((kx * CB + cb) * 3 + j) * 2048, &mB, wfull, ((2 - j) * 3 + kx) * CIN + cb * 32, 0);
        int it = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < g.jobs && ok; t += gridDim.x) {
            job(t, &x0, &b, &o0, &o1);
            for (int r = o0 - 1; r <= o1 && ok; r++)  // (rows outside the image arrive as zeros)
                for (int cb = 0; cb < RB; cb++, it++) {
                    const int s = it % S;
                    if (it >= S && !mbar_wait_bounded(&empty[s], ((it / S) - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&full[s], C::ABOX);
                    tma_load_4d(ring + s * C::ABYTES, &mA, &full[s], cb * 32, x0 - 1, r, b);
                }
        }
        counts[0] = it;
        if (!ok) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
    } else if (threadIdx.x == 32) {  // MMA issuer
        int it = 0, n = 0;           // n: sequence number of the CTA's output row o0
        int ug = 0;                  // upsampled rows taken
        bool ok = mbar_wait_bounded(wfull, 0);
        const uint64_t wdesc = umma_desc_sw64(smem_u32(smem));
        for (int t = blockIdx.x; t < g.jobs && ok; t += gridDim.x) {
            job(t, &x0, &b, &o0, &o1);
            int row4 = -1;  // the upsampled row in use
            for (int r = o0 - 1; r <= o1 && ok; r++) {
                const int lo = max(r - 1, o0), hi = min(r + 1, o1 - 1);
                const bool fresh = hi == r + 1;  // this row starts the accumulator of output row r + 1
                if (fresh) {
                    const int q = n + (r + 1 - o0);
                    if (q >= kAccs && !mbar_wait_bounded(&aempty[q % kAccs], (q / kAccs - 1) & 1)) {
                        ok = false;
                        break;
                    }
                }
                // the accumulators of output rows lo .. hi, in at most two pieces (the ring may wrap between them),
                // and each piece's first weight row: worked out once per row, since one thread issues all
                const int slot = (n + lo - o0) % kAccs, len = hi - lo + 1, len0 = min(len, kAccs - slot);
                const uint32_t d0 = tmem + slot * 32, d1 = tmem;
                const uint64_t b0 = wdesc + (uint64_t)(((lo - r + 1) * 2048) >> 4), b1 = b0 + (uint64_t)((len0 * 2048) >> 4);
                const uint32_t i0 = umma_idesc_bf16(kConvM, 32 * len0), i1 = umma_idesc_bf16(kConvM, 32 * (len - len0));
                const bool image = r >= 0 && r < g.H;
                if (UB && image && r / 4 != row4) {
                    if (row4 >= 0) tc_commit(&uempty[(ug - 1) & 1]);  // arrives when the MMAs on it have completed
                    row4 = r / 4;
                    ok = mbar_wait_bounded(&ufull[ug & 1], (ug >> 1) & 1);
                    ug++;
                }
                for (int cb = 0; cb < RB && ok; cb++) ok = mbar_wait_bounded(&full[(it + cb) % S], ((it + cb) / S) & 1);
                if (!ok) break;
                tc_fence_after();
                const int cb0 = UB && !image ? UB : 0;  // zeros above and below the image: the ring's block alone
                // (kernel column, channel block, 16 channels): each output's sum runs over taps, then channels
#pragma unroll
                for (int kx = 0; kx < 3; kx++)
                    for (int cb = cb0; cb < CB; cb++) {
                        const int s = (it + cb - UB) % S;
                        const uint64_t a0 =
                            umma_desc_sw64(smem_u32(cb < UB ? ups + ((ug - 1 & 1) * UB + cb) * C::ABYTES : ring + s * C::ABYTES)) +
                            kx * 4;
                        const uint64_t w = (uint64_t)(((kx * CB + cb) * 3 * 2048) >> 4);
#pragma unroll
                        for (int k = 0; k < 2; k++) {  // K = 16 per MMA
                            const uint64_t da = a0 + 2 * k, wk = w + 2 * k;
                            if (fresh && cb == cb0 && kx == 0 && k == 0) {
                                // the new row's accumulator is set, the others (one or two, maybe wrapping) added to
                                const uint32_t one = umma_idesc_bf16(kConvM, 32);
                                for (int a = lo; a <= r; a++)
                                    tc_mma(tmem + (n + a - o0) % kAccs * 32, da, wdesc + wk + (((a - r + 1) * 2048) >> 4), one, 1u);
                                tc_mma(tmem + (n + r + 1 - o0) % kAccs * 32, da, wdesc + wk + ((2 * 2048) >> 4), one, 0u);
                            } else {
                                tc_mma(d0, da, b0 + wk, i0, 1u);
                                if (len > len0) tc_mma(d1, da, b1 + wk, i1, 1u);
                            }
                        }
                        if (kx == 2 && cb >= UB) tc_commit(&empty[s]);  // this block has been read by its last MMAs
                    }
                it += RB;
                if (ok && r - 1 >= o0) tc_commit(&afull[(n + r - 1 - o0) % kAccs]);  // output row r - 1 is complete
            }
            if (UB && row4 >= 0) tc_commit(&uempty[(ug - 1) & 1]);
            n += o1 - o0;
        }
        counts[1] = it;
        if (!ok) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
        tc_commit(done);  // arrives when every MMA issued above has completed
    } else if (UB && warp >= 6) {  // upsampled pixels: 34 of a low row, 16 bytes of one at a time
        const int u0 = threadIdx.x - 192, lw = g.W / 4;
        int n = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < g.jobs && ok; t += gridDim.x) {
            job(t, &x0, &b, &o0, &o1);
            const int last4 = min(g.H - 1, o1) / 4;
            for (int r4 = max(0, o0 - 1) / 4; r4 <= last4; r4++, n++) {
                if (n >= 2 && !mbar_wait_bounded(&uempty[n & 1], ((n >> 1) - 1) & 1)) {
                    ok = false;
                    break;
                }
                unsigned char* buf = ups + (n & 1) * UB * C::ABYTES;
                const uint4* src = low + ((int64_t)b * (g.H / 4) + r4) * lw * (UB * 4);
                for (int i = u0; i < 34 * UB * 4; i += 128) {
                    const int j = i / (UB * 4), c = i % (UB * 4), lx = x0 / 4 - 1 + j;
                    uint4 v = make_uint4(0, 0, 0, 0);
                    if (lx >= 0 && lx < lw) v = src[lx * (UB * 4) + c];
                    const int p0 = j == 0 ? 0 : 4 * j - 3, p1 = j == 0 || j == 33 ? p0 : p0 + 3;
                    for (int p = p0; p <= p1; p++)
                        *reinterpret_cast<uint4*>(buf + (c >> 2) * C::ABYTES + p * 64 + (((c ^ (p >> 1)) & 3) << 4)) = v;
                }
                fence_proxy_async_smem();  // the MMAs read what these threads wrote
                mbar_arrive1(&ufull[n & 1]);
            }
        }
        if (!ok && lane == 0) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
    } else if (warp >= 2) {  // epilogue: warp w reads TMEM lanes (pixels of the row) 32 (w % 4) .. + 31
        const int q = warp & 3;
        int n = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < g.jobs && ok; t += gridDim.x) {
            job(t, &x0, &b, &o0, &o1);
            const int px = x0 + q * 32 + lane;
            for (int o = o0; o < o1; o++, n++) {
                const int slot = n % kAccs;
                // warp-uniform: tcgen05.ld below is a warp-collective instruction
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(&afull[slot], (n / kAccs) & 1))) {
                    if (lane == 0) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
                    ok = false;
                    break;
                }
                tc_fence_after();
                float v[32];
                const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(slot * 32);
                tc_ld16(tl, v);
                tc_ld16(tl + 16, v + 16);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive1(&aempty[slot]);
                uint4 w[4];
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(w);
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 bv = __ldg(reinterpret_cast<const float4*>(bias + i));
                    h[i / 2] = __floats2bfloat162_rn(fmaxf(v[i] + bv.x, 0.0f), fmaxf(v[i + 1] + bv.y, 0.0f));
                    h[i / 2 + 1] = __floats2bfloat162_rn(fmaxf(v[i + 2] + bv.z, 0.0f), fmaxf(v[i + 3] + bv.w, 0.0f));
                }
                if (px >= g.W) continue;
                const int64_t p = ((int64_t)b * g.H + o) * g.W + px;
#pragma unroll
                for (int i = 0; i < 4; i++) reinterpret_cast<uint4*>(y + p * 32)[i] = w[i];
                if (last.y) {
                    float a[3] = {};
#pragma unroll
                    for (int c = 0; c < 32; c += 4) {
                        const float2 t0 = __bfloat1622float2(h[c / 2]), t1 = __bfloat1622float2(h[c / 2 + 1]);
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            const float4 u = *reinterpret_cast<const float4*>(sw + 32 * d + c);
                            a[d] = fmaf(t0.y, u.y, fmaf(t0.x, u.x, a[d]));
                            a[d] = fmaf(t1.y, u.w, fmaf(t1.x, u.z, a[d]));
                        }
                    }
#pragma unroll
                    for (int d = 0; d < 3; d++) last.y[3 * p + d] = a[d] + __ldg(last.b + d);
                }
            }
        }
    }
    __syncwarp();
    if (!mbar_wait_bounded(done, 0) && threadIdx.x == 0) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
    tc_fence_after();
    __syncthreads();  // counts[] visible
    if (threadIdx.x == 0) {  // where a wait gave up: drain the copies still in flight
        mbar_wait_bounded(wfull, 0);
        for (int i = counts[1]; i < counts[0]; i++) mbar_wait_bounded(&full[i % S], (i / S) & 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tc_dealloc(tmem, kAccs * 32);
}

template <int RB, int UB>
static int conv3_rows_launch(const RowsGeom& g, const void* x, const void* low, const void* wgt, const float* bias,
                             void* y, const LastLayer& last, int sms, cudaStream_t s, int* d_err) {
    using C = RowsCfg<RB, UB>;
    CUtensorMap mA, mB;
    const uint64_t da[4] = {32 * RB, (uint64_t)g.W, (uint64_t)g.H, (uint64_t)g.B};
    const uint32_t ba[4] = {32, kConvM + 2, 1, 1};
    const uint64_t db[2] = {32 * C::CB * 9, 32};
    const uint32_t b2[2] = {32, 32};
    PS_TRY(encode_bf16_box(&mA, x, 4, da, ba));
    PS_TRY(encode_bf16_box(&mB, wgt, 2, db, b2));
    const auto kernel = nn_conv3_rows_k<RB, UB>;
    // every launch sets it: the attribute belongs to the device's current context
    PS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    PS_CUDA_TRY(launch_dependent(kernel, dim3((unsigned)std::min(g.jobs, 2 * sms)), dim3(C::THREADS), (size_t)C::SMEM, s, mA, mB,
                                 g, static_cast<const uint4*>(low), bias, static_cast<__nv_bfloat16*>(y), last, d_err));
    return PS_OK;
}

// ---- the first layer: 2 -> 32 channels, bias and ReLU -------------------------------------------------
// K = 18 (9 taps of 2 channels), padded to 32: each thread gathers its pixel's taps into one 64-byte row of A
// (swizzled as TMA would store it), two MMAs of 128 pixels by 32 outputs follow, and each thread stores its
// pixel. Several CTAs per SM hide one another's gathers and waits; a CTA takes the tiles blockIdx.x,
// + gridDim.x, ... 8 images of 256^2: 18 us (30 us as 576 FMAs per pixel on the ordinary pipes, 4 pixels by 16
// outputs per thread).
constexpr int kFirstCtas = 8;  // per SM: 32 accumulator columns each
__global__ void __launch_bounds__(128, kFirstCtas)
    nn_conv3_first_k(const __nv_bfloat162* __restrict__ x, int64_t P, int H, int W, const __nv_bfloat16* __restrict__ wgt,
                     int kpad, const float* __restrict__ bias, __nv_bfloat16* __restrict__ y, int* __restrict__ err) {
    __shared__ __align__(1024) unsigned char sA[128 * 64];
    __shared__ __align__(1024) unsigned char sB[32 * 64];
    __shared__ uint64_t bar;
    __shared__ uint32_t slot;
    __shared__ __align__(16) float sbias[32];
    const int t = threadIdx.x, warp = t >> 5;
    if (t == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    if (warp == 0) tc_alloc(&slot, 32);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = slot;
    grid_dependency_wait();
    if (t < 32) sbias[t] = bias[t];
    for (int i = t; i < 32 * 32; i += 128) {  // weights [output][k], zero beyond 18
        const int n = i >> 5, k = i & 31;
        *reinterpret_cast<__nv_bfloat16*>(sB + n * 64 + ((((k >> 3) ^ (n >> 1)) & 3) << 4) + (k & 7) * 2) =
            k < 18 ? wgt[(int64_t)n * kpad + k] : __float2bfloat16(0.0f);
    }
    const uint64_t da = umma_desc_sw64(smem_u32(sA)), db = umma_desc_sw64(smem_u32(sB));
    uint32_t phase = 0;
    bool ok = true;  // of a warp: every wait so far ended (a block stops where one of a warp's gave up)
    for (int64_t p0 = blockIdx.x * (int64_t)128; p0 < P; p0 += gridDim.x * (int64_t)128) {
        const int64_t p = p0 + t, q = p / W;
        const int xx = (int)(p - q * W), yy = (int)(q % H);
        uint32_t v[12] = {};
        if (p < P) {
#pragma unroll
            for (int tap = 0; tap < 9; tap++) {
                const int ty = tap / 3 - 1, tx = tap % 3 - 1;
                if ((unsigned)(xx + tx) < (unsigned)W && (unsigned)(yy + ty) < (unsigned)H)
                    v[tap] = *reinterpret_cast<const uint32_t*>(x + p + ty * W + tx);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; c++)
            *reinterpret_cast<uint4*>(sA + t * 64 + (((c ^ (t >> 1)) & 3) << 4)) =
                c < 3 ? make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]) : make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();  // the MMAs read what these threads wrote
        tc_fence_before();         // and overwrite the accumulator they have read
        if (!__syncthreads_and(ok)) break;
        if (t == 0) {
            tc_fence_after();
            constexpr uint32_t idesc = umma_idesc_bf16(128, 32);
            tc_mma(tmem, da, db, idesc, 0u);
            tc_mma(tmem, da + 2, db + 2, idesc, 1u);
            tc_commit(&bar);
        }
        __syncwarp();
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bar, phase));
        phase ^= 1;
        if (!ok) {
            if ((t & 31) == 0) atomicOr(err, DEV_ERR_TMA_TIMEOUT);
            continue;
        }
        tc_fence_after();
        float a[32];
        const uint32_t tl = tmem + ((uint32_t)(warp * 32) << 16);
        tc_ld16(tl, a);
        tc_ld16(tl + 16, a + 16);
        if (p < P) {
            uint4 w[4];
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(w);
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 bv = *reinterpret_cast<const float4*>(sbias + i);
                h[i / 2] = __floats2bfloat162_rn(fmaxf(a[i] + bv.x, 0.0f), fmaxf(a[i + 1] + bv.y, 0.0f));
                h[i / 2 + 1] = __floats2bfloat162_rn(fmaxf(a[i + 2] + bv.z, 0.0f), fmaxf(a[i + 3] + bv.w, 0.0f));
            }
#pragma unroll
            for (int i = 0; i < 4; i++) reinterpret_cast<uint4*>(y + p * 32)[i] = w[i];
        }
    }
    if (!ok) mbar_wait_bounded(&bar, phase ^ 1);  // the MMAs in flight, before their accumulator is freed
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tc_dealloc(tmem, 32);
}

int nn_conv3_first(const void* x, int64_t P, int H, int W, const void* wgt, int kpad, const float* bias, void* y,
                   cudaStream_t s, int* d_err) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    const int64_t tiles = (P + 127) / 128;
    PS_CUDA_TRY(launch_dependent(nn_conv3_first_k, dim3((unsigned)std::min<int64_t>(tiles, kFirstCtas * st->num_sms)), dim3(128),
                                 (size_t)0, s, static_cast<const __nv_bfloat162*>(x), P, H, W,
                                 static_cast<const __nv_bfloat16*>(wgt), kpad, bias, static_cast<__nv_bfloat16*>(y), d_err));
    return PS_OK;
}

// Whether a tile of 128 pixels of one row is at least three quarters inside the image.
static bool whole_rows(int W) {
    return W % kConvM == 0 || W % kConvM >= 3 * kConvM / 4 || (W > kConvM && W % kConvM >= kConvM / 2);
}

// The layer by rows (see above), with the 1x1 output layer after it; *taken = false (and nothing launched) where
// it does not apply: other channel counts, narrow images, or too few rows for the walk (with 4 per CTA the
// input is read 1.5 times; below that the tiles of nn_conv3_k read no more). low (or NULL): 64 channels of a
// quarter-size layer that come upsampled before x's 32.
int nn_conv3_rows(const void* x, const void* low, int B, int H, int W, int cin, const void* wgt, int cout, const float* bias,
                  void* y, const void* wlast, int kpad_last, const float* blast, float* ylast, bool* taken,
                  cudaStream_t s, int* d_err) {
    *taken = false;
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    if (cout != 32 || cin != (low ? 96 : 32) || !whole_rows(W) || (low && (H % 4 || W % 4))) return PS_OK;
    const int64_t tx = (W + kConvM - 1) / kConvM, strips = tx * B, ctas = 2 * (int64_t)st->num_sms;
    if (strips * H < 4 * ctas || strips * H > 0x7FFFFFFF - 65536) return PS_OK;
    RowsGeom g{};
    g.B = B;
    g.H = H;
    g.W = W;
    g.tx = (int)tx;
    // one job per CTA where the image's rows allow it, else chunks of 64 rows
    g.rows = (int)std::min<int64_t>(64, (strips * H + ctas - 1) / ctas);
    g.chunks = (H + g.rows - 1) / g.rows;
    g.jobs = (int)(strips * g.chunks);
    const LastLayer last{static_cast<const __nv_bfloat16*>(wlast), kpad_last, blast, ylast};
    *taken = true;
    return low ? conv3_rows_launch<1, 2>(g, x, low, wgt, bias, y, last, st->num_sms, s, d_err)
               : conv3_rows_launch<1, 0>(g, x, nullptr, wgt, bias, y, last, st->num_sms, s, d_err);
}

int nn_conv3_tc(const void* x, int B, int H, int W, int cin, const void* wgt, int cout, const float* bias,
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
    // Whole rows of 128 pixels where at least three quarters of them are in the image and one block holds the
    // channels (the sum of an output runs over taps, then channels, in every path): the input is read three
    // times instead of nine. Else the box of 128 pixels that covers the layer in the fewest tiles, wide
    // boxes first (longer contiguous runs).
    const bool row = whole_rows(W) && (cin == 32 || cin == 64);
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
            if (bn == 64) return conv3_launch<64, KC, R, D>(g, x, wgt, bias, y, st->num_sms, s, d_err);
        return conv3_launch<32, KC, R, D>(g, x, wgt, bias, y, st->num_sms, s, d_err);
    };
    auto kc = [&](auto r, auto d) {
        return cin % 64 == 0 ? run(std::integral_constant<int, 64>{}, r, d) : run(std::integral_constant<int, 32>{}, r, d);
    };
    if (deep) return row ? kc(std::true_type{}, std::true_type{}) : kc(std::false_type{}, std::true_type{});
    return row ? kc(std::true_type{}, std::false_type{}) : kc(std::false_type{}, std::false_type{});
}

}  // namespace ps
