// ps_diffusion_split.cu -- FP64 diffusion step with split-FP32 arithmetic (fp64_mode = PS_FP64_SPLIT).
//
// GB300 executes FP64 arithmetic, and f64<->f32 conversions, at 2 instructions / clk / SM, but
// FP32 and integer instructions at 128 / clk / SM. An IEEE-FP64 z-sweep of the diffusion step
// therefore runs at ~6 % of HBM bandwidth. This kernel keeps the arrays in FP64 but evaluates the
// stencil on pairs of FP32 numbers (h + l, a 47-bit significand):
//   - doubles are split into (h, l) with integer bit operations, never with conversions;
//   - sums use the exact two-sum of the high parts plus an FP32 sum of the low parts;
//   - products use FMA to recover the rounding error of h*h;
//   - the update is applied in FP64 as T2 = (T + δh) + δl (two FP64 additions per cell), so T
//     itself is never truncated.
// The result differs from the IEEE evaluation of the reference's statements by <= ~1e-14 of
// max|T| per step (the fixed tolerance is 1e-12 relative max-norm). Magnitudes >= 2^128 raise a
// device flag (PS_ERR_UNSUPPORTED at the next synchronisation); magnitudes < 2^-80 keep 24 bits
// (absolute error < 2^-104), so the bound holds for fields with max|T| >= 2^-60.
//
// Staging is the same TMA z-sweep as diff3d_zsweep_tma: planes of T (and lam) with an x-y halo
// and of Ci land in a shared-memory ring; each plane is converted in place once (every value is
// split exactly once per step), face fluxes are shared between the two cells of a face (x faces
// inside a thread, y faces through shared memory, z faces through registers).
#include <stdlib.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "ps_common.cuh"
#include "ps_dd.cuh"

namespace ps {

struct SplitParams {
    dd c[3];  // per-dimension coefficients (unused when ISO)
    dd g;     // δ = (Ci * g) * Σ_d c_d (F_d+ - F_d-)
};

constexpr int SP_TX = 64;  // cells per row (32 lanes x 2)

template <bool LAM, int TY, int S>
struct SplitCfg {
    static constexpr int PW = SP_TX + 4;  // staged plane: x in [X0-2, X0+66) keeps TMA x 16-byte aligned
    static constexpr int PH = TY + 2;
    static constexpr int PLANE = ((PW * PH * 8 + 127) / 128) * 128;
    static constexpr int CIB = SP_TX * TY * 8;
    static constexpr int STAGE = PLANE * (LAM ? 2 : 1) + CIB;
    static constexpr uint32_t TX_BYTES = (uint32_t)(PW * PH * 8 * (LAM ? 2 : 1) + SP_TX * TY * 8);
    static constexpr int FACE = (TY + 1) * SP_TX * 8;  // y-face fluxes, one float2 per cell (x2 buffers)
    static constexpr int HALO = 2 * PH + 2 * SP_TX;    // halo values per staged array
    static constexpr int SMEM = S * STAGE + 2 * FACE + 8 * S;
};

// dd normalisation (fast two-sum; |a.l| is small against |a.h|)
__device__ __forceinline__ dd dd_norm(dd a) {
    const float s = a.h + a.l;
    return {s, a.l - (s - a.h)};
}

// Face flux between cells a (lower) and b (upper): K*D (LAM) or D, D = T_b - T_a, K = l_a + l_b.
template <bool LAM>
__device__ __forceinline__ dd face(dd Ta, dd Tb, dd la, dd lb) {
    dd D = dd_sub(Tb, Ta);
    if constexpr (LAM) return dd_mul(dd_add(la, lb), D);
    return D;
}

// PRE:   lam and Ci arrays already hold split pairs (float2 per cell, 8 bytes like a double).
// STATE: T and T2 hold split pairs too (the state of a multi-step run); otherwise IEEE doubles.
template <bool LAM, bool ISO, int TY, int S, int MINB, bool PRE, bool STATE>
__global__ void __launch_bounds__(32 * TY, MINB) diff3d_split_tma(const __grid_constant__ CUtensorMap mT,
                                                                  const __grid_constant__ CUtensorMap mL,
                                                                  const __grid_constant__ CUtensorMap mC,
                                                                  double* __restrict__ T2, SplitParams p, int64_t nx,
                                                                  int64_t ny, Box cb, int L, int* __restrict__ err,
                                                                  const int* __restrict__ pred, TileOrder ord) {
    // pred (may be NULL): the launch runs only if *pred is set -- the device-side fallback of a
    // fixed-grid run whose values left the grid
    if (pred) {  // (first: a launch that does not run costs no set-up)
        grid_dependency_wait();
        if (!*reinterpret_cast<const volatile int*>(pred)) return;
    }
    using C = SplitCfg<LAM, TY, S>;
    // staged arrays converted in place each step: T (unless STATE) and lam (unless PRE)
    constexpr int NCONV = (STATE ? 0 : 1) + ((LAM && !PRE) ? 1 : 0);
    constexpr int NHALO = C::HALO * NCONV;
    constexpr int HPT = NHALO > 0 ? (NHALO + 32 * TY - 1) / (32 * TY) : 1;
    extern __shared__ __align__(128) unsigned char smem[];
    float2* faceY0 = reinterpret_cast<float2*>(smem + S * C::STAGE);  // 2 x [TY+1][SP_TX]
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + S * C::STAGE + 2 * C::FACE);

    const int lx = threadIdx.x, ly = threadIdx.y, tid = ly * 32 + lx;
    const uint3 tile = ordered_tile(ord);
    const int X0 = (int)(cb.lo[0] & ~(int64_t)1) + (int)tile.x * SP_TX;
    const int Y0 = (int)cb.lo[1] + (int)tile.y * TY;
    const int Z0 = (int)cb.lo[2] + (int)tile.z * L;
    const int nk = min(L, (int)cb.hi[2] - Z0);
    const int nq = nk + 2;

    auto slot = [&](int q) { return smem + (q % S) * C::STAGE; };
    if (tid == 0) {
        prefetch_tensormap(&mT);
        if constexpr (LAM) prefetch_tensormap(&mL);
        prefetch_tensormap(&mC);
        for (int s = 0; s < S; s++) mbar_init(&bar[s], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (!pred) grid_dependency_wait();  // the kernel before has completed
    int next_q = 0;
    auto issue = [&](int q) {
        unsigned char* b = slot(q);
        int s = q % S, z = Z0 - 1 + q;
        mbar_arrive_expect_tx(&bar[s], C::TX_BYTES);
        tma_load_3d(b, &mT, &bar[s], X0 - 2, Y0 - 1, z);
        if constexpr (LAM) tma_load_3d(b + C::PLANE, &mL, &bar[s], X0 - 2, Y0 - 1, z);
        tma_load_3d(b + C::PLANE * (LAM ? 2 : 1), &mC, &bar[s], X0, Y0, z);
    };
    if (tid == 0)
        for (; next_q < min(S, nq); ++next_q) issue(next_q);

    const int own = (1 + ly) * C::PW + 2 + 2 * lx;  // staged-plane index of this thread's first cell
    const int64_t gx = X0 + 2 * lx, gy = Y0 + ly;
    const bool row_in = gy >= cb.lo[1] && gy < cb.hi[1];
    const bool in0 = row_in && gx >= cb.lo[0] && gx < cb.hi[0];
    const bool in1 = row_in && gx + 1 >= cb.lo[0] && gx + 1 < cb.hi[0];
    // this thread's halo values (byte offsets inside a stage; -1 = none): columns 1 and PW-2 of
    // every row, then rows 0 and PH-1 of the interior columns; T first, then lam
    int hoff[HPT];
#pragma unroll
    for (int r = 0; r < HPT; r++) {
        const int h = tid + r * 32 * TY;
        const int a = h % C::HALO;
        const int idx = a < 2 * C::PH ? (a % C::PH) * C::PW + (a < C::PH ? 1 : C::PW - 2)
                                      : ((a - 2 * C::PH) < SP_TX ? 0 : (C::PH - 1)) * C::PW + 2 + ((a - 2 * C::PH) % SP_TX);
        const int base = (h < C::HALO && !STATE) ? 0 : C::PLANE;  // T plane first unless T is already split
        hoff[r] = h < NHALO ? base + idx * 8 : -1;
    }

    bool big = false, timed_out = false;
    // Converts plane q in place (own cells, returned; raw T kept) and this thread's halo values.
    auto convert = [&](int q, dd* Tn, dd* ln, double2& rawT) {
        unsigned char* b = slot(q);
        double* tp = reinterpret_cast<double*>(b);
        if constexpr (STATE) {
            float4 v = *reinterpret_cast<const float4*>(tp + own);
            Tn[0] = dd{v.x, v.y};
            Tn[1] = dd{v.z, v.w};
        } else {
            rawT = *reinterpret_cast<const double2*>(tp + own);
            Tn[0] = dd_split(rawT.x, big);
            Tn[1] = dd_split(rawT.y, big);
            *reinterpret_cast<float4*>(tp + own) = make_float4(Tn[0].h, Tn[0].l, Tn[1].h, Tn[1].l);
        }
        if constexpr (LAM) {
            double* lp = reinterpret_cast<double*>(b + C::PLANE);
            if constexpr (PRE) {
                float4 v = *reinterpret_cast<const float4*>(lp + own);
                ln[0] = dd{v.x, v.y};
                ln[1] = dd{v.z, v.w};
            } else {
                double2 r = *reinterpret_cast<const double2*>(lp + own);
                ln[0] = dd_split(r.x, big);
                ln[1] = dd_split(r.y, big);
                *reinterpret_cast<float4*>(lp + own) = make_float4(ln[0].h, ln[0].l, ln[1].h, ln[1].l);
            }
        }
        if constexpr (NHALO > 0) {
#pragma unroll
            for (int r = 0; r < HPT; r++) {
                if (hoff[r] >= 0) {
                    double* v = reinterpret_cast<double*>(b + hoff[r]);
                    dd d = dd_split(*v, big);
                    *reinterpret_cast<float2*>(v) = make_float2(d.h, d.l);
                }
            }
        }
        if constexpr (NCONV > 0) fence_proxy_async_smem();  // the slot is refilled by TMA after a later barrier
    };
    auto ld2 = [&](const double* plane, int off) {
        float2 v = *reinterpret_cast<const float2*>(plane + off);
        return dd{v.x, v.y};
    };

    dd Tc[2], lc[2], Tz[2], lz[2], Fzm[2];
    double2 rawTc, rawTz;
    timed_out |= !mbar_wait_bounded(&bar[0], 0);
    timed_out |= !mbar_wait_bounded(&bar[1], 0);
    {
        dd T0[2], l0[2];
        double2 r0;
        convert(0, T0, l0, r0);
        convert(1, Tc, lc, rawTc);
#pragma unroll
        for (int j = 0; j < 2; j++) Fzm[j] = face<LAM>(T0[j], Tc[j], l0[j], lc[j]);
    }

    for (int k = 0; k < nk; ++k) {
        const int q = k + 2;
        timed_out |= !mbar_wait_bounded(&bar[q % S], (q / S) & 1);
        if (!timed_out) convert(q, Tz, lz, rawTz);
        if constexpr (NCONV > 0) __syncthreads();  // A: plane q converted in place
        float2* faceY = faceY0 + (k & 1) * (TY + 1) * SP_TX;
        const unsigned char* b1 = slot(k + 1);
        const double* tp = reinterpret_cast<const double*>(b1);
        const double* lp = reinterpret_cast<const double*>(b1 + C::PLANE);
        dd Fx[3], Fym[2], Fzp[2], ci[2];
        if (!timed_out) {
            const double* cp = reinterpret_cast<const double*>(b1 + C::PLANE * (LAM ? 2 : 1)) + ly * SP_TX + 2 * lx;
            if constexpr (PRE) {
                float4 v = *reinterpret_cast<const float4*>(cp);
                ci[0] = dd{v.x, v.y};
                ci[1] = dd{v.z, v.w};
            } else {
                double2 rc = *reinterpret_cast<const double2*>(cp);
                ci[0] = dd_split(rc.x, big);
                ci[1] = dd_split(rc.y, big);
            }
            // x faces: left of cell 0, between the cells, right of cell 1
            dd Txm = ld2(tp, own - 1), Txp = ld2(tp, own + 2);
            dd lxm{0.f, 0.f}, lxp{0.f, 0.f};
            if constexpr (LAM) {
                lxm = ld2(lp, own - 1);
                lxp = ld2(lp, own + 2);
            }
            Fx[0] = face<LAM>(Txm, Tc[0], lxm, lc[0]);
            Fx[1] = face<LAM>(Tc[0], Tc[1], lc[0], lc[1]);
            Fx[2] = face<LAM>(Tc[1], Txp, lc[1], lxp);
            // y faces below this row (and above, for the top row) go through shared memory
            {
                float4 tb = *reinterpret_cast<const float4*>(tp + own - C::PW);
                float4 lb = LAM ? *reinterpret_cast<const float4*>(lp + own - C::PW) : make_float4(0, 0, 0, 0);
                Fym[0] = face<LAM>(dd{tb.x, tb.y}, Tc[0], dd{lb.x, lb.y}, lc[0]);
                Fym[1] = face<LAM>(dd{tb.z, tb.w}, Tc[1], dd{lb.z, lb.w}, lc[1]);
                *reinterpret_cast<float4*>(faceY + ly * SP_TX + 2 * lx) =
                    make_float4(Fym[0].h, Fym[0].l, Fym[1].h, Fym[1].l);
            }
            if (ly == TY - 1) {
                float4 ta = *reinterpret_cast<const float4*>(tp + own + C::PW);
                float4 la = LAM ? *reinterpret_cast<const float4*>(lp + own + C::PW) : make_float4(0, 0, 0, 0);
                dd f0 = face<LAM>(Tc[0], dd{ta.x, ta.y}, lc[0], dd{la.x, la.y});
                dd f1 = face<LAM>(Tc[1], dd{ta.z, ta.w}, lc[1], dd{la.z, la.w});
                *reinterpret_cast<float4*>(faceY + TY * SP_TX + 2 * lx) = make_float4(f0.h, f0.l, f1.h, f1.l);
            }
#pragma unroll
            for (int j = 0; j < 2; j++) Fzp[j] = face<LAM>(Tc[j], Tz[j], lc[j], lz[j]);
        }
        // B: y faces published; planes <= k+1 are no longer read
        if (__syncthreads_or(timed_out)) {
            if (tid == 0) {
                atomicOr(err, DEV_ERR_TMA_TIMEOUT);
                for (int r = q + 1; r < next_q; ++r) mbar_wait_bounded(&bar[r % S], (r / S) & 1);
            }
            return;
        }
        if (tid == 0)
            for (; next_q < min(nq, k + 2 + S); ++next_q) issue(next_q);
        float4 fa = *reinterpret_cast<const float4*>(faceY + (ly + 1) * SP_TX + 2 * lx);
        dd Fyp[2] = {dd{fa.x, fa.y}, dd{fa.z, fa.w}};
        double out[2];
        const double rawc[2] = {rawTc.x, rawTc.y};
#pragma unroll
        for (int j = 0; j < 2; j++) {
            dd Sm;
            if constexpr (ISO) {
                Sm = dd_sub(Fx[j + 1], Fx[j]);
                Sm = dd_add(Sm, Fyp[j]);
                Sm = dd_sub(Sm, Fym[j]);
                Sm = dd_add(Sm, Fzp[j]);
                Sm = dd_sub(Sm, Fzm[j]);
            } else {
                Sm = dd_mul(p.c[0], dd_sub(Fx[j + 1], Fx[j]));
                Sm = dd_add(Sm, dd_mul(p.c[1], dd_sub(Fyp[j], Fym[j])));
                Sm = dd_add(Sm, dd_mul(p.c[2], dd_sub(Fzp[j], Fzm[j])));
            }
            dd delta = dd_mul(dd_mul(ci[j], p.g), Sm);
            if constexpr (STATE) {
                dd r = dd_norm(dd_add(Tc[j], delta));
                out[j] = __hiloint2double(__float_as_int(r.l), __float_as_int(r.h));  // (h, l) bit pair
            } else {
                out[j] = (rawc[j] + f32_to_f64(delta.h)) + f32_to_f64(delta.l);
            }
        }
        const int64_t gz = Z0 + k;
        double* dst = T2 + gx + nx * (gy + ny * gz);
        if (in0 && in1)
            *reinterpret_cast<double2*>(dst) = make_double2(out[0], out[1]);
        else {
            if (in0) dst[0] = out[0];
            if (in1) dst[1] = out[1];
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            Tc[j] = Tz[j];
            lc[j] = lz[j];
            Fzm[j] = Fzp[j];
        }
        rawTc = rawTz;
    }
    if (__syncthreads_or(big) && tid == 0) atomicOr(err, DEV_ERR_RANGE);
    ordered_tile_done(ord);
}

static void split_const(dd& d, double v) {
    float h = (float)v;
    d.h = h;
    d.l = (float)(v - (double)h);
}

template <bool LAM, bool ISO, bool PRE, bool STATE>
static int launch_split_variant(const ps_array& Tin, const ps_array& Ci, const ps_array* lam, const ps_array& T2,
                                const SplitParams& p, const Box& cb, int L, cudaStream_t s, int* d_err,
                                const int* pred, HideReq* hr) {
    constexpr int TY = 8, S = 4, MINB = 3;
    using C = SplitCfg<LAM, TY, S>;
    CUtensorMap mT, mL, mC;
    PS_TRY(encode_plane_map(&mT, Tin, C::PW, C::PH));
    if (LAM)
        PS_TRY(encode_plane_map(&mL, *lam, C::PW, C::PH));
    else
        mL = mT;
    PS_TRY(encode_plane_map(&mC, Ci, SP_TX, TY));
    static bool attr = false;
    if (!attr) {
        PS_CUDA_TRY(cudaFuncSetAttribute(diff3d_split_tma<LAM, ISO, TY, S, MINB, PRE, STATE>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        attr = true;
    }
    int64_t x0 = cb.lo[0] & ~(int64_t)1;
    dim3 blk(32, TY, 1);
    const int64_t bx = (cb.hi[0] - x0 + SP_TX - 1) / SP_TX, by = (cb.hi[1] - cb.lo[1] + TY - 1) / TY;
    if (L <= 0) {
        static const int occ = resident_ctas(diff3d_split_tma<LAM, ISO, TY, S, MINB, PRE, STATE>, 32 * TY, C::SMEM);
        DeviceState* st = nullptr;
        PS_TRY(current_state(&st));
        L = auto_loopsize(bx * by, cb.hi[2] - cb.lo[2], (int64_t)occ * st->num_sms);
    }
    const int64_t bz = (cb.hi[2] - cb.lo[2] + L - 1) / L;
    dim3 grd((unsigned)bx, (unsigned)by, (unsigned)bz);
    TileOrder ord{};
    if (hr) {  // boundary tiles first, as one 1-D grid
        const int64_t nt[3] = {bx, by, bz}, lo[3] = {x0, cb.lo[1], cb.lo[2]}, tl[3] = {SP_TX, TY, L};
        const int64_t end[3] = {cb.hi[0], cb.hi[1], cb.hi[2]};
        ord = make_tile_order(nt, lo, tl, end, hr->lo_end, hr->hi_start, hr->counter);
        hr->nb = ord.nb;
        grd = dim3((unsigned)(bx * by * bz), 1, 1);
    }
    const auto kernel = diff3d_split_tma<LAM, ISO, TY, S, MINB, PRE, STATE>;
    if (hr)
        kernel<<<grd, blk, C::SMEM, s>>>(mT, mL, mC, static_cast<double*>(T2.ptr), p, T2.n[0], T2.n[1], cb, L, d_err, pred, ord);
    else
        PS_CUDA_TRY(launch_dependent(kernel, grd, blk, (size_t)C::SMEM, s, mT, mL, mC, static_cast<double*>(T2.ptr), p,
                                     T2.n[0], T2.n[1], cb, L, d_err, pred, ord));
    return PS_OK;
}

template <bool LAM, bool ISO>
static int launch_split_flags(bool pre, bool state, const ps_array& Tin, const ps_array& Ci, const ps_array* lam,
                              const ps_array& T2, const SplitParams& p, const Box& cb, int L, cudaStream_t s,
                              int* d_err, const int* pred, HideReq* hr) {
    if (pre)
        return state ? launch_split_variant<LAM, ISO, true, true>(Tin, Ci, lam, T2, p, cb, L, s, d_err, pred, hr)
                     : launch_split_variant<LAM, ISO, true, false>(Tin, Ci, lam, T2, p, cb, L, s, d_err, pred, hr);
    return state ? launch_split_variant<LAM, ISO, false, true>(Tin, Ci, lam, T2, p, cb, L, s, d_err, pred, hr)
                 : launch_split_variant<LAM, ISO, false, false>(Tin, Ci, lam, T2, p, cb, L, s, d_err, pred, hr);
}

// Per-dimension coefficients of the forms (split into p->c) and the common factor g: the
// increment is g * Ci * sum_d c_d (F_d+ - F_d-); isotropic c is folded into g (returns true).
static bool split_coeffs(int form, double lam_s, double dt, double hx, double hy, double hz, SplitParams* p,
                         double* g) {
    double c[3];
    const double h[3] = {hx, hy, hz};
    for (int d = 0; d < 3; d++) {
        switch (form) {
        case PS_DIFF_DIV: c[d] = 1.0 / (h[d] * h[d]); break;
        case PS_DIFF_FLUX_LAM: c[d] = 0.5 * (h[d] * h[d]); break;
        default: c[d] = h[d] * h[d]; break;
        }
    }
    *g = form == PS_DIFF_FLUX_LAM ? dt : dt * lam_s;
    const bool iso = c[0] == c[1] && c[1] == c[2];
    if (iso) *g *= c[0];
    for (int d = 0; d < 3; d++) split_const(p->c[d], c[d]);
    return iso;
}

// Split-arithmetic z-sweep over the cell box cb. pre: lam / Ci hold split pairs; state: T / T2
// hold split pairs. Returns PS_ERR_UNSUPPORTED when the arrays are not TMA-eligible (the caller
// then uses the IEEE kernels).
static int launch_split(int form, const ps_array& T2, const ps_array& Tin, const ps_array& Ci, const ps_array* lam,
                        double lam_s, double dt, double hx, double hy, double hz, const Box& cb, int L, bool pre,
                        bool state, cudaStream_t s, int* d_err, const int* pred = nullptr, HideReq* hr = nullptr) {
    bool tma = tma_eligible(T2) && tma_eligible(Tin) && tma_eligible(Ci) && (!lam || tma_eligible(*lam));
    if (!tma || T2.dtype != PS_F64) return PS_ERR_UNSUPPORTED;
    SplitParams p{};
    double g;
    const bool iso = split_coeffs(form, lam_s, dt, hx, hy, hz, &p, &g);
    split_const(p.g, g);
    if (form == PS_DIFF_FLUX_LAM)
        return iso ? launch_split_flags<true, true>(pre, state, Tin, Ci, lam, T2, p, cb, L, s, d_err, pred, hr)
                   : launch_split_flags<true, false>(pre, state, Tin, Ci, lam, T2, p, cb, L, s, d_err, pred, hr);
    return iso ? launch_split_flags<false, true>(pre, state, Tin, Ci, lam, T2, p, cb, L, s, d_err, pred, hr)
               : launch_split_flags<false, false>(pre, state, Tin, Ci, lam, T2, p, cb, L, s, d_err, pred, hr);
}

int launch_diffusion_split(int form, const ps_array& T2, const ps_array& Tin, const ps_array& Ci, const ps_array* lam,
                           double lam_s, double dt, double hx, double hy, double hz, const Box& cb, int L,
                           cudaStream_t s, int* d_err, HideReq* hr) {
    return launch_split(form, T2, Tin, Ci, lam, lam_s, dt, hx, hy, hz, cb, L, false, false, s, d_err, nullptr, hr);
}

// =======================================================================================
// Fixed-grid split state (PS_FP64_SPLIT_GRID, multi-step runs).
//
// T and lam are held as float pairs (h, l) on a power-of-two grid fixed for the whole run:
// value = (h + l) * u, u = 2^-sh, where sh is chosen from max|T| (max|lam|) so that the largest
// magnitude is below 2^23 grid units; h is an integer-valued float (|h| <= 2^23), |l| <= 1/2.
// Differences of h parts (|.| <= 2^24) and sums of lam h parts are exact in one FP32 addition,
// where value-relative pairs need a two-sum; the face flux K*D keeps the exact FMA remainder of
// the high product, so a face costs 8 FP32 operations instead of 20. Rounding per value and step:
// <= 1.5 * 2^-25 grid units, i.e. <= 1.5 * 2^-47 of max|T|.
// =======================================================================================

// Run header in library scratch (written by the setup kernels on the device).
struct GridRun {
    unsigned long long maxT, maxL;  // max|T|, max|lam| as (largest high word << 32) | (any low word != 0)
    int shT, shL;                   // grid units = value * 2^sh
    int bad;                        // a value left the grid range: the run is redone with split pairs
    int pad;
    double g;                       // coefficient scale G * 2^-shL folded into the Ci pairs
};

template <bool LAM>
__device__ __forceinline__ dd gface(dd Ta, dd Tb, dd la, dd lb) {
    const float Dh = Tb.h - Ta.h, Dl = Tb.l - Ta.l;  // Dh exact (integers, |.| <= 2^24)
    if constexpr (!LAM) {
        return {Dh, Dl};
    } else {
        const float Kh = la.h + lb.h, Kl = la.l + lb.l;  // Kh exact
        const float pr = Kh * Dh;
        float e = fmaf(Kh, Dh, -pr);  // exact remainder of the high product
        e = fmaf(Kh, Dl, e);
        e = fmaf(Kl, Dh, e);
        return {pr, e};
    }
}

// A double as a grid pair (h, l): v * 2^sh = h + l, h integer-valued, |l| <= 1/2. Non-finite
// values set `bad`.
__device__ __forceinline__ float2 to_grid(double v, int sh, bool& bad) {
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7FF);
    if (e == 0x7FF) {
        bad = true;
        return make_float2(0.f, 0.f);
    }
    if (e == 0 || e + sh <= 0) return make_float2(0.f, 0.f);  // below 2^-1022 grid units
    const double x = __longlong_as_double(b + ((long long)sh << 52));  // v * 2^sh, |x| < 2^23
    bool big = false;
    const dd d = dd_split(x, big);
    const float h = rintf(d.h);
    return make_float2(h, (d.h - h) + d.l);
}

// The run's coefficient scale g as a float pair (Ci pairs are Ci * g).
__device__ __forceinline__ dd g_pair(double g) {
    dd gd;
    gd.h = (float)g;
    gd.l = (float)(g - (double)gd.h);
    return gd;
}

// Ci as the value pair of Ci * g; magnitudes outside FP32's range set `big`.
__device__ __forceinline__ dd ci_pair(double c, dd gd, bool& big) {
    const dd r = dd_norm(dd_mul(dd_split(c, big), gd));
    big |= !(fabsf(r.h) < 0x1p127f);
    return r;
}

// Exact double of the grid value (h + l) * 2^-sh (h, l floats; values below 2^-1022 -> 0).
__device__ __forceinline__ double grid_to_f64(double y, int sh) {
    const long long b = __double_as_longlong(y);
    const int e = (int)((b >> 52) & 0x7FF);
    return (e == 0 || e - sh <= 0) ? 0.0 : __longlong_as_double(b - ((long long)sh << 52));
}

// One step on grid pairs: T, lam as (h, l) grid pairs, Ci as value pairs of Ci * G * u_lam; T2 as
// grid pairs, or (OUT64, the last step of a run) as IEEE doubles. Every launch returns at once when
// an earlier kernel of the run flagged a value outside the grid (the run is then redone).
//
// IN64 (the first step of a run of two or more steps): T, lam and Ci are the caller's FP64 arrays.
// Each staged plane of T and lam is converted to grid pairs in place in shared memory (own cells by
// their thread, the x-y halo by assigned threads), and the step also writes its own cells' lam grid
// pairs and Ci value pairs to Lout / Cout for the later steps, so the run never converts T, lam or
// Ci in separate passes. The conversions are the setup kernels' functions, so the run's results do
// not depend on which step converted a value.
template <bool LAM, bool ISO, int TY, int S, int MINB, bool OUT64, bool IN64>
__global__ void __launch_bounds__(32 * TY, MINB)
    diff3d_grid_tma(const __grid_constant__ CUtensorMap mT, const __grid_constant__ CUtensorMap mL,
                    const __grid_constant__ CUtensorMap mC, void* __restrict__ T2v, SplitParams p, int64_t nx,
                    int64_t ny, Box cb, int L, int* __restrict__ err, GridRun* __restrict__ run,
                    float4* __restrict__ Lout, float4* __restrict__ Cout) {
    static_assert(!(IN64 && OUT64), "a one-step run converts its input first");
    using C = SplitCfg<LAM, TY, S>;
    constexpr int NHALO = IN64 ? C::HALO * (LAM ? 2 : 1) : 0;
    constexpr int HPT = NHALO > 0 ? (NHALO + 32 * TY - 1) / (32 * TY) : 1;
    extern __shared__ __align__(128) unsigned char smem[];
    float2* faceY0 = reinterpret_cast<float2*>(smem + S * C::STAGE);  // 2 x [TY+1][SP_TX]
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + S * C::STAGE + 2 * C::FACE);

    const int lx = threadIdx.x, ly = threadIdx.y, tid = ly * 32 + lx;
    const int X0 = (int)(cb.lo[0] & ~(int64_t)1) + blockIdx.x * SP_TX;
    const int Y0 = (int)cb.lo[1] + blockIdx.y * TY;
    const int Z0 = (int)cb.lo[2] + blockIdx.z * L;
    const int nk = min(L, (int)cb.hi[2] - Z0);
    const int nq = nk + 2;

    auto slot = [&](int q) { return smem + (q % S) * C::STAGE; };
    if (tid == 0) {
        prefetch_tensormap(&mT);
        if constexpr (LAM) prefetch_tensormap(&mL);
        prefetch_tensormap(&mC);
        for (int s = 0; s < S; s++) mbar_init(&bar[s], 1);
        fence_mbar_init();
    }
    grid_dependency_wait();  // the step before has completed
    // One thread reads the flag for the block (and the barriers are set up): blocks of this launch raise it while
    // others start, and a block of which only some threads left would wait for loads that nobody issues.
    if (__syncthreads_or(tid == 0 && *reinterpret_cast<volatile int*>(&run->bad))) return;
    const int sh = run->shT;
    int next_q = 0;
    auto issue = [&](int q) {
        unsigned char* b = slot(q);
        int s = q % S, z = Z0 - 1 + q;
        mbar_arrive_expect_tx(&bar[s], C::TX_BYTES);
        tma_load_3d(b, &mT, &bar[s], X0 - 2, Y0 - 1, z);
        if constexpr (LAM) tma_load_3d(b + C::PLANE, &mL, &bar[s], X0 - 2, Y0 - 1, z);
        tma_load_3d(b + C::PLANE * (LAM ? 2 : 1), &mC, &bar[s], X0, Y0, z);
    };
    if (tid == 0)
        for (; next_q < min(S, nq); ++next_q) issue(next_q);

    const int own = (1 + ly) * C::PW + 2 + 2 * lx;  // staged-plane index of this thread's first cell
    const int64_t gx = X0 + 2 * lx, gy = Y0 + ly;
    const bool row_in = gy >= cb.lo[1] && gy < cb.hi[1];
    const bool in0 = row_in && gx >= cb.lo[0] && gx < cb.hi[0];
    const bool in1 = row_in && gx + 1 >= cb.lo[0] && gx + 1 < cb.hi[0];
    const bool in_array = gx < nx && gy < ny;  // gx even, nx even: the pair (gx, gx+1) is in the array
    auto ld1 = [](const unsigned char* b, int off) {
        const float2 v = reinterpret_cast<const float2*>(b)[off];
        return dd{v.x, v.y};
    };
    auto ld2 = [](const unsigned char* b, int off, dd* v) {  // off even: 16-byte aligned
        const float4 t = *reinterpret_cast<const float4*>(reinterpret_cast<const float2*>(b) + off);
        v[0] = dd{t.x, t.y};
        v[1] = dd{t.z, t.w};
    };

    // IN64: this thread's halo values (byte offsets inside a stage; -1 = none): columns 1 and PW-2
    // of every row, then rows 0 and PH-1 of the interior columns; T first, then lam
    int hoff[HPT];
    int shL = 0;
    dd gd{0.f, 0.f};
    if constexpr (IN64) {
        shL = run->shL;
        gd = g_pair(run->g);
#pragma unroll
        for (int r = 0; r < HPT; r++) {
            const int h = tid + r * 32 * TY;
            const int a = h % C::HALO;
            const int idx = a < 2 * C::PH ? (a % C::PH) * C::PW + (a < C::PH ? 1 : C::PW - 2)
                                          : ((a - 2 * C::PH) < SP_TX ? 0 : (C::PH - 1)) * C::PW + 2 +
                                                ((a - 2 * C::PH) % SP_TX);
            hoff[r] = h < NHALO ? (h < C::HALO ? 0 : C::PLANE) + idx * 8 : -1;
        }
    }
    bool bad = false, timed_out = false;
    // IN64: converts plane q of T (and lam) in place: own cells (returned) and this thread's halo
    auto convert = [&](int q, dd* Tn, dd* ln) {
        unsigned char* b = slot(q);
        double* tp = reinterpret_cast<double*>(b);
        const double2 rt = *reinterpret_cast<const double2*>(tp + own);
        const float2 t0 = to_grid(rt.x, sh, bad), t1 = to_grid(rt.y, sh, bad);
        *reinterpret_cast<float4*>(tp + own) = make_float4(t0.x, t0.y, t1.x, t1.y);
        Tn[0] = dd{t0.x, t0.y};
        Tn[1] = dd{t1.x, t1.y};
        if constexpr (LAM) {
            double* lp = reinterpret_cast<double*>(b + C::PLANE);
            const double2 rl = *reinterpret_cast<const double2*>(lp + own);
            const float2 l0 = to_grid(rl.x, shL, bad), l1 = to_grid(rl.y, shL, bad);
            *reinterpret_cast<float4*>(lp + own) = make_float4(l0.x, l0.y, l1.x, l1.y);
            ln[0] = dd{l0.x, l0.y};
            ln[1] = dd{l1.x, l1.y};
        }
#pragma unroll
        for (int r = 0; r < HPT; r++) {
            if (hoff[r] >= 0) {
                double* v = reinterpret_cast<double*>(b + hoff[r]);
                *reinterpret_cast<float2*>(v) = to_grid(*v, hoff[r] >= C::PLANE ? shL : sh, bad);
            }
        }
        fence_proxy_async_smem();  // the slot is refilled by TMA after a later barrier
    };

    dd Tc[2], lc[2], Tz[2], lz[2], Fzm[2];
    timed_out |= !mbar_wait_bounded(&bar[0], 0);
    timed_out |= !mbar_wait_bounded(&bar[1], 0);
    {
        dd T0[2], l0[2];
        if constexpr (IN64) {
            if (!timed_out) {
                convert(0, T0, l0);
                convert(1, Tc, lc);
            }
            __syncthreads();  // plane 1's halo is read by the neighbours in the first z step
        } else {
            ld2(slot(0), own, T0);
            ld2(slot(1), own, Tc);
            if constexpr (LAM) {
                ld2(slot(0) + C::PLANE, own, l0);
                ld2(slot(1) + C::PLANE, own, lc);
            }
        }
#pragma unroll
        for (int j = 0; j < 2; j++) Fzm[j] = gface<LAM>(T0[j], Tc[j], l0[j], lc[j]);
    }

    for (int k = 0; k < nk; ++k) {
        const int q = k + 2;
        timed_out |= !mbar_wait_bounded(&bar[q % S], (q / S) & 1);
        const unsigned char* bz = slot(q);
        if constexpr (IN64) {
            // plane q is read by the other threads only in the next z step, after barrier B below
            if (!timed_out) convert(q, Tz, lz);
        } else {
            ld2(bz, own, Tz);
            if constexpr (LAM) ld2(bz + C::PLANE, own, lz);
        }
        float2* faceY = faceY0 + (k & 1) * (TY + 1) * SP_TX;
        const unsigned char* tp = slot(k + 1);
        const unsigned char* lp = tp + C::PLANE;
        const int64_t gz = Z0 + k;
        const int64_t o = gx + nx * (gy + ny * gz);
        dd Fx[3], Fym[2], Fzp[2], ci[2];
        if constexpr (IN64) {
            const double2 rc = *reinterpret_cast<const double2*>(
                reinterpret_cast<const double*>(tp + C::PLANE * (LAM ? 2 : 1)) + ly * SP_TX + 2 * lx);
            ci[0] = ci_pair(rc.x, gd, bad);
            ci[1] = ci_pair(rc.y, gd, bad);
            if (in_array) {  // the later steps' lam and Ci pairs of this thread's cells
                Cout[o / 2] = make_float4(ci[0].h, ci[0].l, ci[1].h, ci[1].l);
                if constexpr (LAM) Lout[o / 2] = make_float4(lc[0].h, lc[0].l, lc[1].h, lc[1].l);
            }
        } else {
            ld2(tp + C::PLANE * (LAM ? 2 : 1), ly * SP_TX + 2 * lx, ci);
        }
        {
            const dd Txm = ld1(tp, own - 1), Txp = ld1(tp, own + 2);
            dd lxm{0.f, 0.f}, lxp{0.f, 0.f};
            if constexpr (LAM) {
                lxm = ld1(lp, own - 1);
                lxp = ld1(lp, own + 2);
            }
            Fx[0] = gface<LAM>(Txm, Tc[0], lxm, lc[0]);
            Fx[1] = gface<LAM>(Tc[0], Tc[1], lc[0], lc[1]);
            Fx[2] = gface<LAM>(Tc[1], Txp, lc[1], lxp);
        }
        {
            dd tb[2], lb[2] = {{0.f, 0.f}, {0.f, 0.f}};
            ld2(tp, own - C::PW, tb);
            if constexpr (LAM) ld2(lp, own - C::PW, lb);
            Fym[0] = gface<LAM>(tb[0], Tc[0], lb[0], lc[0]);
            Fym[1] = gface<LAM>(tb[1], Tc[1], lb[1], lc[1]);
            *reinterpret_cast<float4*>(faceY + ly * SP_TX + 2 * lx) = make_float4(Fym[0].h, Fym[0].l, Fym[1].h, Fym[1].l);
        }
        if (ly == TY - 1) {
            dd ta[2], la[2] = {{0.f, 0.f}, {0.f, 0.f}};
            ld2(tp, own + C::PW, ta);
            if constexpr (LAM) ld2(lp, own + C::PW, la);
            const dd f0 = gface<LAM>(Tc[0], ta[0], lc[0], la[0]);
            const dd f1 = gface<LAM>(Tc[1], ta[1], lc[1], la[1]);
            *reinterpret_cast<float4*>(faceY + TY * SP_TX + 2 * lx) = make_float4(f0.h, f0.l, f1.h, f1.l);
        }
#pragma unroll
        for (int j = 0; j < 2; j++) Fzp[j] = gface<LAM>(Tc[j], Tz[j], lc[j], lz[j]);
        // B: y faces published; planes <= k+1 are no longer read
        if (__syncthreads_or(timed_out)) {
            if (tid == 0) {
                atomicOr(err, DEV_ERR_TMA_TIMEOUT);
                for (int r = q + 1; r < next_q; ++r) mbar_wait_bounded(&bar[r % S], (r / S) & 1);
            }
            return;
        }
        if (tid == 0)
            for (; next_q < min(nq, k + 2 + S); ++next_q) issue(next_q);
        const float4 fa = *reinterpret_cast<const float4*>(faceY + (ly + 1) * SP_TX + 2 * lx);
        const dd Fyp[2] = {dd{fa.x, fa.y}, dd{fa.z, fa.w}};
        float2 out[2];
        double out64[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            dd Sm;
            if constexpr (ISO) {
                Sm = dd_sub(Fx[j + 1], Fx[j]);
                Sm = dd_add(Sm, Fyp[j]);
                Sm = dd_sub(Sm, Fym[j]);
                Sm = dd_add(Sm, Fzp[j]);
                Sm = dd_sub(Sm, Fzm[j]);
            } else {
                Sm = dd_mul(p.c[0], dd_sub(Fx[j + 1], Fx[j]));
                Sm = dd_add(Sm, dd_mul(p.c[1], dd_sub(Fyp[j], Fym[j])));
                Sm = dd_add(Sm, dd_mul(p.c[2], dd_sub(Fzp[j], Fzm[j])));
            }
            const dd d = dd_mul(ci[j], Sm);  // increment in grid units
            // T2 = T + d on the grid: move the integer part of d into h, keep |l| <= 1/2
            constexpr float M = 12582912.0f;       // 1.5 * 2^23: (x + M) - M is an integer near x
            const float q0 = (d.h + M) - M;
            float l2 = (d.h - q0) + d.l;           // d.h - q0 exact
            l2 = l2 + Tc[j].l;
            const float q1 = (l2 + M) - M;
            const float h2 = (Tc[j].h + q0) + q1;  // integers: exact while in range
            const bool in_range = fabsf(h2) <= 8388608.0f;
            if constexpr (OUT64) {
                // the last step leaves the grid: a value that grew past it is summed in FP64 instead
                const double y = in_range ? f32_to_f64(h2) + f32_to_f64(l2 - q1)
                                          : ((f32_to_f64(Tc[j].h) + f32_to_f64(Tc[j].l)) + f32_to_f64(d.h)) +
                                                f32_to_f64(d.l);
                out64[j] = grid_to_f64(y, sh);
            } else {
                bad |= !in_range;  // left the grid (or not finite)
                out[j] = make_float2(h2, l2 - q1);
            }
        }
        if constexpr (OUT64) {
            double* dst = static_cast<double*>(T2v) + o;
            if (in0 && in1)
                *reinterpret_cast<double2*>(dst) = make_double2(out64[0], out64[1]);
            else {
                if (in0) dst[0] = out64[0];
                if (in1) dst[1] = out64[1];
            }
        } else {
            float2* dst = static_cast<float2*>(T2v) + o;
            if (in0 && in1)
                *reinterpret_cast<float4*>(dst) = make_float4(out[0].x, out[0].y, out[1].x, out[1].y);
            else {
                if (in0) dst[0] = out[0];
                if (in1) dst[1] = out[1];
            }
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            Tc[j] = Tz[j];
            lc[j] = lz[j];
            Fzm[j] = Fzp[j];
        }
    }
    if (__syncthreads_or(bad) && tid == 0) atomicOr(&run->bad, 1);
}

// Boundary cells (the six faces) of T converted to grid pairs into both run states a and b, and of
// lam (if given) into the lam pairs: the first step of a run (IN64) writes the inner cells of b, of
// lam's pairs and of Ci's pairs, so these faces are the rest of what the later steps read.
__global__ void grid_faces64_kernel(const double* __restrict__ T, float2* __restrict__ a, float2* __restrict__ b,
                                    const double* __restrict__ lam, float2* __restrict__ lg, int64_t nx, int64_t ny,
                                    int64_t nz, GridRun* r) {
    if (r->bad) return;
    const int shT = r->shT, shL = r->shL;
    bool bad = false;
    const int f = blockIdx.y;  // 0,1: z faces; 2,3: y faces; 4,5: x faces
    const int64_t n0 = f < 4 ? nx : ny, n1 = f < 2 ? ny : nz;
    const int64_t fixed = (f & 1) ? (f < 2 ? nz : f < 4 ? ny : nx) - 1 : 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n0 * n1; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t u = i % n0, v = i / n0;
        const int64_t ix = f < 4 ? u : fixed, iy = f < 2 ? v : f < 4 ? fixed : u, iz = f < 2 ? fixed : v;
        const int64_t o = ix + nx * (iy + ny * iz);
        const float2 t = to_grid(T[o], shT, bad);
        a[o] = t;
        b[o] = t;
        if (lam) lg[o] = to_grid(lam[o], shL, bad);
    }
    if (bad) atomicOr(&r->bad, 1);
}

// The setup kernels below run on TMA-eligible arrays (nx even), so they work on pairs of values
// (16-byte accesses); n2 = numel / 2.

// max |a[i]| reduced to what the grid needs: the largest high word (sign cleared: it carries the
// exponent) and whether any low word is nonzero, composed as (max_hi << 32) | any_lo. The result
// has the exponent of max |a[i]| and is zero exactly when every a[i] is zero.
struct AbsmaxBits {
    unsigned hi = 0, lo = 0;
    __device__ __forceinline__ void add(double2 v) {
        hi = max(hi, max((unsigned)__double2hiint(v.x) & 0x7FFFFFFFu, (unsigned)__double2hiint(v.y) & 0x7FFFFFFFu));
        lo |= (unsigned)__double2loint(v.x) | (unsigned)__double2loint(v.y);
    }
    __device__ __forceinline__ void publish(unsigned long long* out) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
            lo |= __shfl_xor_sync(0xFFFFFFFFu, lo, o);
        }
        const unsigned long long m = ((unsigned long long)hi << 32) | (lo ? 1ull : 0ull);
        if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
    }
};

// max |a[i]| and max |b[i]| (b may be NULL) in one pass over both arrays. A persistent grid (4 CTAs
// of 256 threads per SM, all resident) walks the pairs with four 16-byte loads per array in flight
// per thread.
constexpr int kAbsmaxUnroll = 4;
__global__ void __launch_bounds__(256, 4)
    absmax2_bits_kernel(const double2* __restrict__ a, const double2* __restrict__ b, int64_t n2,
                        unsigned long long* out_a, unsigned long long* out_b) {
    AbsmaxBits ma, mb;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (; i + (kAbsmaxUnroll - 1) * stride < n2; i += kAbsmaxUnroll * stride) {
        double2 va[kAbsmaxUnroll], vb[kAbsmaxUnroll];
#pragma unroll
        for (int u = 0; u < kAbsmaxUnroll; u++) va[u] = __ldcs(a + i + u * stride);
        if (b) {
#pragma unroll
            for (int u = 0; u < kAbsmaxUnroll; u++) vb[u] = __ldcs(b + i + u * stride);
#pragma unroll
            for (int u = 0; u < kAbsmaxUnroll; u++) mb.add(vb[u]);
        }
#pragma unroll
        for (int u = 0; u < kAbsmaxUnroll; u++) ma.add(va[u]);
    }
    for (; i < n2; i += stride) {
        ma.add(__ldcs(a + i));
        if (b) mb.add(__ldcs(b + i));
    }
    ma.publish(out_a);
    if (b) mb.publish(out_b);
}

// Grid exponent of a maximum: largest magnitude < 2^23 grid units. Maxima outside
// [2^-823, 2^877) (and non-finite ones) are left to the split-pair path.
__device__ bool grid_shift(unsigned long long m, int* sh) {
    if (m == 0) {
        *sh = 0;
        return true;
    }
    const int e = (int)(m >> 52);  // max in [2^(e-1023), 2^(e-1022))
    if (e < 200 || e > 1900) return false;
    *sh = 1045 - e;
    return true;
}

__global__ void grid_setup_kernel(GridRun* r, double G, int has_lam) {
    bool ok = grid_shift(r->maxT, &r->shT);
    if (has_lam)
        ok = ok && grid_shift(r->maxL, &r->shL);
    else
        r->shL = 0;
    const double g = ok ? ldexp(G, -r->shL) : 0.0;
    const double ag = fabs(g);
    if (!ok || (ag != 0.0 && (ag < 0x1p-100 || ag > 0x1p100))) r->bad = 1;
    r->g = g;
}

// T -> grid pairs (lam_grid = 0) or lam -> grid pairs (lam_grid = 1)
__global__ void to_grid_kernel(const double2* __restrict__ in, float4* __restrict__ a, int64_t n2, GridRun* r,
                               int lam_grid) {
    if (r->bad) return;
    const int sh = lam_grid ? r->shL : r->shT;
    bool bad = false;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n2; i += stride) {
        const double2 v = __ldcs(in + i);
        const float2 g0 = to_grid(v.x, sh, bad), g1 = to_grid(v.y, sh, bad);
        a[i] = make_float4(g0.x, g0.y, g1.x, g1.y);
    }
    if (bad) atomicOr(&r->bad, 1);
}

// Ci -> value pairs of Ci * g
__global__ void ci_grid_kernel(const double2* __restrict__ in, float4* __restrict__ out, int64_t n2, GridRun* r) {
    if (r->bad) return;
    const dd gd = g_pair(r->g);
    bool big = false;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n2; i += stride) {
        const double2 v = __ldcs(in + i);
        const dd c0 = ci_pair(v.x, gd, big), c1 = ci_pair(v.y, gd, big);
        out[i] = make_float4(c0.h, c0.l, c1.h, c1.l);
    }
    if (big) atomicOr(&r->bad, 1);
}

// Rows of a grid step's tile: 8, or 6 for the steps between a run's first and last. With a conductivity array three
// and four CTAs fit an SM, 24 rows both, and the smaller tile's four groups of warps wait less on each other (512^3
// 660 -> 647 us per step, 256^3 98.2 -> 96.0); without one four and five do, 32 rows and 30. Which is faster is a
// matter of the last wave too (without an array 512 x 256 x 128: 70 us with 8 rows, 76 with 6; 300^3 120 and 115), so the
// tile whose fullest SM has no more to do is taken, 6 rows where they are equal. There, over 34 grids of 10^6 to
// 10^8 cells, 6 rows are 1.3 % faster on average, and from 9 % faster (288 x 340 x 150) to 3.6 % slower (512 x 280 x 70;
// 384 x 384 x 128 108 -> 111 us): nothing that the model counts tells those apart.
constexpr int kGridRows = 8, kGridRowsMiddle = 6;

// z-sweep length and relative time of a launch of tiles of `rows` rows: the fullest SM's tiles, their rows and their
// planes (on average; the last z-block may be short).
struct GridPick {
    int L;
    double cost;
};
static GridPick grid_pick(const Box& cb, int rows, int occ, int sms) {
    const int64_t x0 = cb.lo[0] & ~(int64_t)1;
    const int64_t xy = ((cb.hi[0] - x0 + SP_TX - 1) / SP_TX) * ((cb.hi[1] - cb.lo[1] + rows - 1) / rows);
    const int64_t wz = cb.hi[2] - cb.lo[2];
    const int L = auto_loopsize(xy, wz, (int64_t)occ * sms);
    const int64_t chunks = (wz + L - 1) / L, ctas = xy * chunks, slots = (int64_t)occ * sms;
    const int64_t per_sm = ctas < slots ? (ctas + sms - 1) / sms : (ctas + slots - 1) / slots * occ;
    return {L, (double)per_sm * rows * ((double)wz / chunks + 2)};
}

constexpr int kGridStages = 4;
template <bool LAM, bool ISO, bool OUT64, bool IN64, int TY>
constexpr auto grid_kernel() {
    return diff3d_grid_tma<LAM, ISO, TY, kGridStages, TY == kGridRows ? 3 : 4, OUT64, IN64>;
}
template <bool LAM, bool ISO, bool OUT64, bool IN64, int TY>
static int grid_occupancy() {
    constexpr int smem = SplitCfg<LAM, TY, kGridStages>::SMEM;
    cudaFuncSetAttribute(grid_kernel<LAM, ISO, OUT64, IN64, TY>(), cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return resident_ctas(grid_kernel<LAM, ISO, OUT64, IN64, TY>(), 32 * TY, smem);
}

// One step of a grid run. IN64 (first step): Tin, Cs and Ls are the caller's FP64 T, Ci and lam,
// and the step writes the lam / Ci pairs of its cells to Lout / Cout.
template <bool LAM, bool ISO, bool OUT64, bool IN64, int TY>
static int launch_grid_tile(const ps_array& Tin, const ps_array& Cs, const ps_array* Ls, const ps_array& T2,
                            const SplitParams& p, const Box& cb, int L, cudaStream_t s, int* d_err, GridRun* run,
                            void* Lout, void* Cout) {
    using C = SplitCfg<LAM, TY, kGridStages>;
    const auto kernel = grid_kernel<LAM, ISO, OUT64, IN64, TY>();
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    static bool attr = false;
    if (!attr) {
        PS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        attr = true;
    }
    if (L <= 0) {
        static const int occ = resident_ctas(kernel, 32 * TY, C::SMEM);
        const GridPick pick = grid_pick(cb, TY, occ, st->num_sms);
        L = pick.L;
        if constexpr (!OUT64 && !IN64 && TY == kGridRows) {
            static const int occ6 = grid_occupancy<LAM, ISO, OUT64, IN64, kGridRowsMiddle>();
            const GridPick six = grid_pick(cb, kGridRowsMiddle, occ6, st->num_sms);
            if (six.cost <= pick.cost && cb.hi[1] - cb.lo[1] <= 65535 * kGridRowsMiddle)
                return launch_grid_tile<LAM, ISO, OUT64, IN64, kGridRowsMiddle>(Tin, Cs, Ls, T2, p, cb, 0, s, d_err, run, Lout, Cout);
        }
    }
    CUtensorMap mT, mL, mC;
    PS_TRY(encode_plane_map(&mT, Tin, C::PW, C::PH));
    if (LAM)
        PS_TRY(encode_plane_map(&mL, *Ls, C::PW, C::PH));
    else
        mL = mT;
    PS_TRY(encode_plane_map(&mC, Cs, SP_TX, TY));
    const int64_t x0 = cb.lo[0] & ~(int64_t)1;
    const int64_t bx = (cb.hi[0] - x0 + SP_TX - 1) / SP_TX, by = (cb.hi[1] - cb.lo[1] + TY - 1) / TY;
    dim3 grd((unsigned)bx, (unsigned)by, (unsigned)((cb.hi[2] - cb.lo[2] + L - 1) / L));
    PS_CUDA_TRY(launch_dependent(kernel, grd, dim3(32, TY, 1), (size_t)C::SMEM, s, mT, mL, mC, T2.ptr, p, T2.n[0], T2.n[1], cb,
                                 L, d_err, run, static_cast<float4*>(Lout), static_cast<float4*>(Cout)));
    return PS_OK;
}
template <bool LAM, bool ISO, bool OUT64, bool IN64>
static int launch_grid_variant(const ps_array& Tin, const ps_array& Cs, const ps_array* Ls, const ps_array& T2,
                               const SplitParams& p, const Box& cb, int L, cudaStream_t s, int* d_err, GridRun* run,
                               void* Lout, void* Cout) {
    return launch_grid_tile<LAM, ISO, OUT64, IN64, kGridRows>(Tin, Cs, Ls, T2, p, cb, L, s, d_err, run, Lout, Cout);
}

enum GridStep { GRID_FIRST64 = 0, GRID_MIDDLE = 1, GRID_LAST64 = 2 };

template <bool LAM, bool ISO>
static int launch_grid_step(GridStep kind, const ps_array& Tin, const ps_array& Cs, const ps_array* Ls,
                            const ps_array& T2, const SplitParams& p, const Box& cb, int L, cudaStream_t s, int* d_err,
                            GridRun* run, void* Lout = nullptr, void* Cout = nullptr) {
    switch (kind) {
    case GRID_FIRST64:
        return launch_grid_variant<LAM, ISO, false, true>(Tin, Cs, Ls, T2, p, cb, L, s, d_err, run, Lout, Cout);
    case GRID_LAST64:
        return launch_grid_variant<LAM, ISO, true, false>(Tin, Cs, Ls, T2, p, cb, L, s, d_err, run, nullptr, nullptr);
    default:
        return launch_grid_variant<LAM, ISO, false, false>(Tin, Cs, Ls, T2, p, cb, L, s, d_err, run, nullptr, nullptr);
    }
}

// ---- multi-step runs -------------------------------------------------------------------
__global__ void split_pairs_kernel(const double* __restrict__ in, double* __restrict__ out, int64_t n, int* err,
                                   const int* __restrict__ pred = nullptr) {
    if (pred && !*reinterpret_cast<const volatile int*>(pred)) return;
    bool big = false;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        dd d = dd_split(in[i], big);
        out[i] = __hiloint2double(__float_as_int(d.l), __float_as_int(d.h));
    }
    if (big) atomicOr(err, DEV_ERR_RANGE);
}

// Final state of a split-pair run back to doubles, inner cells only: the boundary cells of T keep
// their initial values exactly (a split pair holds only 24 bits of magnitudes below 2^-80).
__global__ void join_pairs_kernel(const double* __restrict__ in, double* __restrict__ out, int64_t nx, int64_t ny,
                                  int64_t nz, const int* __restrict__ pred = nullptr) {
    if (pred && !*reinterpret_cast<const volatile int*>(pred)) return;
    const int64_t n = nx * ny * nz;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t x = i % nx, y = (i / nx) % ny, z = i / (nx * ny);
        if (x == 0 || y == 0 || z == 0 || x == nx - 1 || y == ny - 1 || z == nz - 1) continue;
        const double v = in[i];
        out[i] = f32_to_f64(__int_as_float(__double2loint(v))) + f32_to_f64(__int_as_float(__double2hiint(v)));
    }
}

// out = in (n 8-byte words) when *pred is set
__global__ void copy_words_if_kernel(const double* __restrict__ in, double* __restrict__ out, int64_t n,
                                     const int* __restrict__ pred) {
    if (!*reinterpret_cast<const volatile int*>(pred)) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = in[i];
}

// Grow-only scratch for the split pairs of lam, Ci and the run state, one per device and stream:
// a run is asynchronous, so runs on different streams may execute at the same time (freed by
// ps_finalize).
struct RunScratch {
    void* ptr = nullptr;
    size_t bytes = 0;
};
static std::mutex g_run_mutex;
static std::map<std::pair<int, cudaStream_t>, RunScratch> g_run_scratch;  // (device, stream)

// Grow-only scratch of the fixed-grid misfit gradient (freed by ps_finalize).
static void* g_grad_scratch = nullptr;
static size_t g_grad_bytes = 0;

void diffusion_free_scratch() {
    {
        std::lock_guard<std::mutex> lock(g_run_mutex);
        for (auto& kv : g_run_scratch)
            if (kv.second.ptr) cudaFree(kv.second.ptr);
        g_run_scratch.clear();
    }
    if (g_grad_scratch) cudaFree(g_grad_scratch);
    g_grad_scratch = nullptr;
    g_grad_bytes = 0;
}

static int run_scratch(size_t bytes, char** p, cudaStream_t s) {
    int dev = 0;
    PS_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_run_mutex);
    RunScratch& r = g_run_scratch[{dev, s}];
    if (bytes > r.bytes) {
        if (r.ptr) cudaFree(r.ptr);  // waits for the work that used it
        r.ptr = nullptr;
        r.bytes = 0;
        if (cudaMalloc(&r.ptr, bytes) != cudaSuccess) {
            cudaGetLastError();
            r.ptr = nullptr;
            return fail(PS_ERR_NOMEM, "ps_diffusion3d_run: scratch allocation of %zu bytes failed", bytes);
        }
        r.bytes = bytes;
    }
    *p = static_cast<char*>(r.ptr);
    return PS_OK;
}

// =======================================================================================
// Misfit gradient on the fixed grid (ps_diffusion3d_misfit_gradient with PS_FP64_SPLIT_GRID).
//
// The flux-form step with a conductivity array is T' = T + dt Ci L T with L symmetric, so its
// adjoint is λ = λ' + L μ' with μ = dt Ci λ (zero off the inner cells), and μ itself obeys
// μ = μ' + dt Ci L μ': the same step as the forward one. Each reverse step is one sweep
// (diff3d_grid_adj_tma) that applies that step to μ (its own power-of-two grid, fixed from
// max|μ_nt|; the step is a diffusion, so |μ| does not grow) and accumulates
//   glam[c] += Σ over the faces (a, b = a + e_d) of c of -1/2 hh_d (μ_b - μ_a)(T_b - T_a)
// from μ_{n+1} and the forward state T_n (both grid pairs: the differences of their integer
// parts are exact), summed on FP32 pairs and added to glam in FP64. The forward states and the
// checkpoints are grid pairs of the forward run's grid. If any value leaves its grid, the caller
// redoes the gradient with value-relative split pairs.
// =======================================================================================

// ---- fused reverse step ------------------------------------------------------------------
// One z-sweep that does both halves of a reverse step: μ_out = μ_in + (dt Ci) L μ_in on the inner
// cells (the forward grid step applied to μ, same operations as diff3d_grid_tma) and
// glam += Σ_faces -1/2 hh_d Dμ DT from μ_in and the forward state T_n, for the cells of the rows
// 1 .. ny-2 and planes 1 .. nz-2 (every x); glam_boundary_kernel does rows 0, ny-1 and planes 0,
// nz-1. Planes of μ, lam, T_n (with their x-y halo) and of Ci are staged by TMA; y-face terms go
// through shared memory, z-face terms through registers.
template <int TY, int S>
struct AdjCfg {
    static constexpr int PW = SP_TX + 4;
    static constexpr int PH = TY + 2;
    static constexpr int PLANE = ((PW * PH * 8 + 127) / 128) * 128;
    static constexpr int CIB = SP_TX * TY * 8;
    static constexpr int STAGE = 3 * PLANE + CIB;  // μ, lam, T_n, Ci
    static constexpr uint32_t TX_BYTES = (uint32_t)(3 * PW * PH * 8 + SP_TX * TY * 8);
    static constexpr int FACE = (TY + 1) * SP_TX * 8;
    static constexpr int SMEM = S * STAGE + 4 * FACE + 8 * S;  // K·Dμ and Dμ·DT of the y faces, 2 buffers each
};

// K·D of a face from its difference D (the operations of gface<true>)
__device__ __forceinline__ dd grid_kd(dd D, dd la, dd lb) {
    const float Kh = la.h + lb.h, Kl = la.l + lb.l;
    const float pr = Kh * D.h;
    float e = fmaf(Kh, D.h, -pr);
    e = fmaf(Kh, D.l, e);
    e = fmaf(Kl, D.h, e);
    return {pr, e};
}
__device__ __forceinline__ dd grid_diff(dd a, dd b) { return {b.h - a.h, b.l - a.l}; }  // b - a, high part exact

template <bool ISO, int TY, int S>
__global__ void __launch_bounds__(32 * TY, 2)
    diff3d_grid_adj_tma(const __grid_constant__ CUtensorMap mM, const __grid_constant__ CUtensorMap mL,
                        const __grid_constant__ CUtensorMap mC, const __grid_constant__ CUtensorMap mT,
                        float2* __restrict__ Mout, double* __restrict__ glam, SplitParams p, dd gc0, dd gc1, dd gc2,
                        int64_t nx, int64_t ny, Box cb, int L, int* __restrict__ err, GridRun* __restrict__ run,
                        const GridRun* __restrict__ mrun) {
    using C = AdjCfg<TY, S>;
    extern __shared__ __align__(128) unsigned char smem[];
    float2* faceY0 = reinterpret_cast<float2*>(smem + S * C::STAGE);
    float2* wY0 = reinterpret_cast<float2*>(smem + S * C::STAGE + 2 * C::FACE);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + S * C::STAGE + 4 * C::FACE);

    const int lx = threadIdx.x, ly = threadIdx.y, tid = ly * 32 + lx;
    const int X0 = (int)(cb.lo[0] & ~(int64_t)1) + blockIdx.x * SP_TX;
    const int Y0 = (int)cb.lo[1] + blockIdx.y * TY;
    const int Z0 = (int)cb.lo[2] + blockIdx.z * L;
    const int nk = min(L, (int)cb.hi[2] - Z0);
    const int nq = nk + 2;

    auto slot = [&](int q) { return smem + (q % S) * C::STAGE; };
    if (tid == 0) {
        prefetch_tensormap(&mM);
        prefetch_tensormap(&mL);
        prefetch_tensormap(&mC);
        prefetch_tensormap(&mT);
        for (int s = 0; s < S; s++) mbar_init(&bar[s], 1);
        fence_mbar_init();
    }
    grid_dependency_wait();        // the step before (or the recomputed states) has completed
    grid_dependents_may_launch();  // glam_boundary_kernel of this step runs beside this kernel
    // (one thread reads the flags for the block, see diff3d_grid_tma)
    if (__syncthreads_or(tid == 0 && (*reinterpret_cast<volatile int*>(&run->bad) ||
                                      *reinterpret_cast<const volatile int*>(&mrun->bad))))
        return;
    const int sh = mrun->shT + run->shT;
    int next_q = 0;
    auto issue = [&](int q) {
        unsigned char* b = slot(q);
        int s = q % S, z = Z0 - 1 + q;
        mbar_arrive_expect_tx(&bar[s], C::TX_BYTES);
        tma_load_3d(b, &mM, &bar[s], X0 - 2, Y0 - 1, z);
        tma_load_3d(b + C::PLANE, &mL, &bar[s], X0 - 2, Y0 - 1, z);
        tma_load_3d(b + 2 * C::PLANE, &mT, &bar[s], X0 - 2, Y0 - 1, z);
        tma_load_3d(b + 3 * C::PLANE, &mC, &bar[s], X0, Y0, z);
    };
    if (tid == 0)
        for (; next_q < min(S, nq); ++next_q) issue(next_q);

    const int own = (1 + ly) * C::PW + 2 + 2 * lx;
    const int64_t gx = X0 + 2 * lx, gy = Y0 + ly;
    const bool row_in = gy >= cb.lo[1] && gy < cb.hi[1];
    const bool in0 = row_in && gx >= cb.lo[0] && gx < cb.hi[0];
    const bool in1 = row_in && gx + 1 >= cb.lo[0] && gx + 1 < cb.hi[0];
    const bool glam_row = gx < nx && gy >= 1 && gy < ny - 1;  // rows 0 and ny-1: glam_boundary_kernel
    auto ld1 = [](const unsigned char* b, int off) {
        const float2 v = reinterpret_cast<const float2*>(b)[off];
        return dd{v.x, v.y};
    };
    auto ld2 = [](const unsigned char* b, int off, dd* v) {
        const float4 t = *reinterpret_cast<const float4*>(reinterpret_cast<const float2*>(b) + off);
        v[0] = dd{t.x, t.y};
        v[1] = dd{t.z, t.w};
    };

    bool bad = false, timed_out = false;
    dd Mc[2], lc[2], Nc[2], Mz[2], lz[2], Nz[2], Fzm[2], Wzm[2];
    timed_out |= !mbar_wait_bounded(&bar[0], 0);
    timed_out |= !mbar_wait_bounded(&bar[1], 0);
    {
        dd M0[2], l0[2], N0[2];
        ld2(slot(0), own, M0);
        ld2(slot(1), own, Mc);
        ld2(slot(0) + C::PLANE, own, l0);
        ld2(slot(1) + C::PLANE, own, lc);
        ld2(slot(0) + 2 * C::PLANE, own, N0);
        ld2(slot(1) + 2 * C::PLANE, own, Nc);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const dd D = grid_diff(M0[j], Mc[j]);
            Fzm[j] = grid_kd(D, l0[j], lc[j]);
            Wzm[j] = dd_mul(D, grid_diff(N0[j], Nc[j]));
        }
    }

    for (int k = 0; k < nk; ++k) {
        const int q = k + 2;
        const int64_t gz = Z0 + k;
        const int64_t o = gx + nx * (gy + ny * gz);
        // glam of this plane: loaded first, so its latency hides behind the face arithmetic
        double2 gv = make_double2(0.0, 0.0);
        if (glam_row) gv = *reinterpret_cast<const double2*>(glam + o);
        timed_out |= !mbar_wait_bounded(&bar[q % S], (q / S) & 1);
        const unsigned char* bz = slot(q);
        ld2(bz, own, Mz);
        ld2(bz + C::PLANE, own, lz);
        ld2(bz + 2 * C::PLANE, own, Nz);
        float2* faceY = faceY0 + (k & 1) * (TY + 1) * SP_TX;
        float2* wY = wY0 + (k & 1) * (TY + 1) * SP_TX;
        const unsigned char* mp = slot(k + 1);
        const unsigned char* lp = mp + C::PLANE;
        const unsigned char* np = mp + 2 * C::PLANE;
        dd Fx[3], Wx[3], Fym[2], Wym[2], Fzp[2], Wzp[2], ci[2];
        ld2(mp + 3 * C::PLANE, ly * SP_TX + 2 * lx, ci);
        {
            const dd Mxm = ld1(mp, own - 1), Mxp = ld1(mp, own + 2);
            const dd lxm = ld1(lp, own - 1), lxp = ld1(lp, own + 2);
            const dd Nxm = ld1(np, own - 1), Nxp = ld1(np, own + 2);
            const dd D0 = grid_diff(Mxm, Mc[0]), D1 = grid_diff(Mc[0], Mc[1]), D2 = grid_diff(Mc[1], Mxp);
            Fx[0] = grid_kd(D0, lxm, lc[0]);
            Fx[1] = grid_kd(D1, lc[0], lc[1]);
            Fx[2] = grid_kd(D2, lc[1], lxp);
            Wx[0] = dd_mul(D0, grid_diff(Nxm, Nc[0]));
            Wx[1] = dd_mul(D1, grid_diff(Nc[0], Nc[1]));
            Wx[2] = dd_mul(D2, grid_diff(Nc[1], Nxp));
        }
        {
            dd mb[2], lb[2], nb[2];
            ld2(mp, own - C::PW, mb);
            ld2(lp, own - C::PW, lb);
            ld2(np, own - C::PW, nb);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const dd D = grid_diff(mb[j], Mc[j]);
                Fym[j] = grid_kd(D, lb[j], lc[j]);
                Wym[j] = dd_mul(D, grid_diff(nb[j], Nc[j]));
            }
            *reinterpret_cast<float4*>(faceY + ly * SP_TX + 2 * lx) = make_float4(Fym[0].h, Fym[0].l, Fym[1].h, Fym[1].l);
            *reinterpret_cast<float4*>(wY + ly * SP_TX + 2 * lx) = make_float4(Wym[0].h, Wym[0].l, Wym[1].h, Wym[1].l);
        }
        if (ly == TY - 1) {
            dd ma[2], la[2], na[2];
            ld2(mp, own + C::PW, ma);
            ld2(lp, own + C::PW, la);
            ld2(np, own + C::PW, na);
            dd f[2], w[2];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const dd D = grid_diff(Mc[j], ma[j]);
                f[j] = grid_kd(D, lc[j], la[j]);
                w[j] = dd_mul(D, grid_diff(Nc[j], na[j]));
            }
            *reinterpret_cast<float4*>(faceY + TY * SP_TX + 2 * lx) = make_float4(f[0].h, f[0].l, f[1].h, f[1].l);
            *reinterpret_cast<float4*>(wY + TY * SP_TX + 2 * lx) = make_float4(w[0].h, w[0].l, w[1].h, w[1].l);
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const dd D = grid_diff(Mc[j], Mz[j]);
            Fzp[j] = grid_kd(D, lc[j], lz[j]);
            Wzp[j] = dd_mul(D, grid_diff(Nc[j], Nz[j]));
        }
        if (__syncthreads_or(timed_out)) {
            if (tid == 0) {
                atomicOr(err, DEV_ERR_TMA_TIMEOUT);
                for (int r = q + 1; r < next_q; ++r) mbar_wait_bounded(&bar[r % S], (r / S) & 1);
            }
            return;
        }
        if (tid == 0)
            for (; next_q < min(nq, k + 2 + S); ++next_q) issue(next_q);
        const float4 fa = *reinterpret_cast<const float4*>(faceY + (ly + 1) * SP_TX + 2 * lx);
        const float4 wa = *reinterpret_cast<const float4*>(wY + (ly + 1) * SP_TX + 2 * lx);
        const dd Fyp[2] = {dd{fa.x, fa.y}, dd{fa.z, fa.w}};
        const dd Wyp[2] = {dd{wa.x, wa.y}, dd{wa.z, wa.w}};
        float2 out[2];
        double gout[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            dd Sm;
            if constexpr (ISO) {
                Sm = dd_sub(Fx[j + 1], Fx[j]);
                Sm = dd_add(Sm, Fyp[j]);
                Sm = dd_sub(Sm, Fym[j]);
                Sm = dd_add(Sm, Fzp[j]);
                Sm = dd_sub(Sm, Fzm[j]);
            } else {
                Sm = dd_mul(p.c[0], dd_sub(Fx[j + 1], Fx[j]));
                Sm = dd_add(Sm, dd_mul(p.c[1], dd_sub(Fyp[j], Fym[j])));
                Sm = dd_add(Sm, dd_mul(p.c[2], dd_sub(Fzp[j], Fzm[j])));
            }
            const dd d = dd_mul(ci[j], Sm);
            constexpr float Mg = 12582912.0f;
            const float q0 = (d.h + Mg) - Mg;
            float l2 = (d.h - q0) + d.l;
            l2 = l2 + Mc[j].l;
            const float q1 = (l2 + Mg) - Mg;
            const float h2 = (Mc[j].h + q0) + q1;
            bad |= !(fabsf(h2) <= 8388608.0f);
            out[j] = make_float2(h2, l2 - q1);
            // glam: the six faces of the cell, by dimension
            dd g = dd_mul(gc0, dd_add(Wx[j], Wx[j + 1]));
            g = dd_add(g, dd_mul(gc1, dd_add(Wym[j], Wyp[j])));
            g = dd_add(g, dd_mul(gc2, dd_add(Wzm[j], Wzp[j])));
            gout[j] = grid_to_f64(f32_to_f64(g.h) + f32_to_f64(g.l), sh);
        }
        {
            float2* dst = Mout + o;
            if (in0 && in1)
                *reinterpret_cast<float4*>(dst) = make_float4(out[0].x, out[0].y, out[1].x, out[1].y);
            else {
                if (in0) dst[0] = out[0];
                if (in1) dst[1] = out[1];
            }
        }
        if (glam_row) {
            gv.x = gv.x + gout[0];
            gv.y = gv.y + gout[1];
            *reinterpret_cast<double2*>(glam + o) = gv;
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            Mc[j] = Mz[j];
            lc[j] = lz[j];
            Nc[j] = Nz[j];
            Fzm[j] = Fzp[j];
            Wzm[j] = Wzp[j];
        }
    }
    if (__syncthreads_or(bad) && tid == 0) atomicOr(&run->bad, 1);
}

// glam of the cells in the planes z = 0, nz-1 and the rows y = 0, ny-1 (the rest is done by
// diff3d_grid_adj_tma): the same face sums from global loads, one thread per cell. It does not let the next step's
// blocks in early: they took places beside the running step's blocks, which left SMs with two steps' blocks and others with
// one (gradient per step, with that / without: 16 x 1024 x 64 161 / 135 us, 256 x 256 x 32 92 / 79, 128^3 63.2 / 62.7,
// 64^3 20.9 / 21.3).
__global__ void glam_boundary_kernel(const float2* __restrict__ M, const float2* __restrict__ Tg,
                                     double* __restrict__ glam, dd gc0, dd gc1, dd gc2, int64_t nx, int64_t ny,
                                     int64_t nz, const GridRun* __restrict__ run, const GridRun* __restrict__ mrun) {
    const bool skip = run->bad || mrun->bad;
    const int sh = mrun->shT + run->shT;
    const int f = blockIdx.y;  // 0, 1: planes z = 0, nz-1 (all x, y); 2, 3: rows y = 0, ny-1 (z = 1 .. nz-2)
    const int64_t n0 = nx, n1 = f < 2 ? ny : nz - 2;
    const int64_t sy = nx, sz = nx * ny;
    auto ld = [](const float2* a, int64_t o) {
        const float2 v = a[o];
        return dd{v.x, v.y};
    };
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n0 * n1 && !skip; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t x = t % n0, v = t / n0;
        const int64_t y = f < 2 ? v : (f == 2 ? 0 : ny - 1), z = f < 2 ? (f == 0 ? 0 : nz - 1) : v + 1;
        const int64_t o = x + nx * (y + ny * z);
        const dd mc = ld(M, o), tc = ld(Tg, o);
        dd s3[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
        const int64_t pos[3] = {x, y, z}, ext[3] = {nx, ny, nz}, st[3] = {1, sy, sz};
#pragma unroll
        for (int d = 0; d < 3; d++) {
            if (pos[d] > 0) {
                const int64_t nb = o - st[d];
                s3[d] = dd_add(s3[d], dd_mul(grid_diff(ld(M, nb), mc), grid_diff(ld(Tg, nb), tc)));
            }
            if (pos[d] + 1 < ext[d]) {
                const int64_t nb = o + st[d];
                s3[d] = dd_add(s3[d], dd_mul(grid_diff(mc, ld(M, nb)), grid_diff(tc, ld(Tg, nb))));
            }
        }
        dd g = dd_mul(gc0, s3[0]);
        g = dd_add(g, dd_mul(gc1, s3[1]));
        g = dd_add(g, dd_mul(gc2, s3[2]));
        glam[o] = glam[o] + grid_to_f64(f32_to_f64(g.h) + f32_to_f64(g.l), sh);
    }
    grid_dependency_wait();
}

template <bool ISO>
static int launch_grid_adj(const ps_array& Min, const ps_array& Ls, const ps_array& Cs, const ps_array& Tn,
                           const ps_array& Mout, const ps_array& glam, const SplitParams& p, const dd gc[3],
                           const Box& cb, cudaStream_t s, int* d_err, GridRun* run, const GridRun* mrun) {
    constexpr int TY = 8, S = 4;
    using C = AdjCfg<TY, S>;
    auto kernel = diff3d_grid_adj_tma<ISO, TY, S>;
    CUtensorMap mM, mL, mC, mT;
    PS_TRY(encode_plane_map(&mM, Min, C::PW, C::PH));
    PS_TRY(encode_plane_map(&mL, Ls, C::PW, C::PH));
    PS_TRY(encode_plane_map(&mT, Tn, C::PW, C::PH));
    PS_TRY(encode_plane_map(&mC, Cs, SP_TX, TY));
    static bool attr = false;
    if (!attr) {
        PS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        attr = true;
    }
    const int64_t x0 = cb.lo[0] & ~(int64_t)1;
    const int64_t bx = (cb.hi[0] - x0 + SP_TX - 1) / SP_TX, by = (cb.hi[1] - cb.lo[1] + TY - 1) / TY;
    static const int occ = resident_ctas(kernel, 32 * TY, C::SMEM);
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    const int L = auto_loopsize(bx * by, cb.hi[2] - cb.lo[2], (int64_t)occ * st->num_sms);
    dim3 grd((unsigned)bx, (unsigned)by, (unsigned)((cb.hi[2] - cb.lo[2] + L - 1) / L));
    PS_CUDA_TRY(launch_dependent(kernel, grd, dim3(32, TY, 1), (size_t)C::SMEM, s, mM, mL, mC, mT,
                                 static_cast<float2*>(Mout.ptr), static_cast<double*>(glam.ptr), p, gc[0], gc[1], gc[2],
                                 Mout.n[0], Mout.n[1], cb, L, d_err, run, mrun));
    // The boundary rows and planes of glam run beside the kernel above (programmatic dependent
    // launch; it starts once every block of that kernel has waited for the step before): they read μ and
    // T_n, which the step before completed, and write glam cells the kernel above does not touch. They wait
    // for that kernel at their end, so the next step, which waits for them, waits for both.
    const int64_t nmax = std::max(Mout.n[0] * Mout.n[1], Mout.n[0] * Mout.n[2]);
    const dim3 gb((unsigned)std::min<int64_t>((nmax + 255) / 256, st->num_sms * 4), 4);
    if (launch_dependent(glam_boundary_kernel, gb, dim3(256), 0, s, static_cast<const float2*>(Min.ptr),
                         static_cast<const float2*>(Tn.ptr), static_cast<double*>(glam.ptr), gc[0], gc[1], gc[2],
                         Mout.n[0], Mout.n[1], Mout.n[2], static_cast<const GridRun*>(run), mrun) != cudaSuccess) {
        cudaGetLastError();
        glam_boundary_kernel<<<gb, 256, 0, s>>>(static_cast<const float2*>(Min.ptr), static_cast<const float2*>(Tn.ptr),
                                                static_cast<double*>(glam.ptr), gc[0], gc[1], gc[2], Mout.n[0],
                                                Mout.n[1], Mout.n[2], run, mrun);
    }
    return PS_OK;
}

// FP64 state from grid pairs (every cell): (h + l) 2^-sh
__global__ void grid_state_to_f64_kernel(const float2* __restrict__ S, double* __restrict__ out, int64_t n,
                                         const GridRun* __restrict__ r) {
    if (r->bad) return;
    const int sh = r->shT;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const float2 v = S[c];
        out[c] = grid_to_f64(f32_to_f64(v.x) + f32_to_f64(v.y), sh);
    }
}

// μ_nt = dt Ci (T_nt - T_obs) on inner cells, 0 elsewhere; loss += 1/2 Σ (T_nt - T_obs)^2 (all cells)
__global__ void grid_misfit_kernel(double* mu, const double* Tn,
                                   const double* __restrict__ Tobs, const double* __restrict__ Ci, double dt, int64_t nx,
                                   int64_t ny, int64_t nz, double* __restrict__ loss) {
    double s = 0.0;
    const int64_t n = nx * ny * nz;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = c % nx, j = (c / nx) % ny, k = c / (nx * ny);
        const double r = Tn[c] - Tobs[c];
        s += 0.5 * r * r;
        const bool inner = i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 2 && k >= 1 && k <= nz - 2;
        mu[c] = inner ? dt * Ci[c] * r : 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, s);
}

// The six faces of the state `from` copied into the `count` states that lie `stride` values apart from `to`
// (a step writes inner cells only, so a buffer's faces are set once). blockIdx.z: the buffer.
__global__ void __launch_bounds__(256) grid_faces_copy_kernel(const float2* __restrict__ from, float2* __restrict__ to,
                                                             int64_t stride, int64_t nx, int64_t ny, int64_t nz) {
    float2* out = to + stride * blockIdx.z;
    const int f = blockIdx.y;  // 0,1: z faces; 2,3: y faces; 4,5: x faces
    const int64_t n0 = f < 4 ? nx : ny, n1 = f < 2 ? ny : nz;
    const int64_t fixed = (f & 1) ? (f < 2 ? nz : f < 4 ? ny : nx) - 1 : 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n0 * n1; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = i / n0, u = i - v * n0;
        const int64_t ix = f < 4 ? u : fixed, iy = f < 2 ? v : f < 4 ? fixed : u, iz = f < 2 ? fixed : v;
        const int64_t o = ix + nx * (iy + ny * iz);
        out[o] = from[o];
    }
}

int grid_misfit_gradient(const ps_array& T0, const ps_array& Tobs, const ps_array& Ci, const ps_array& lam, double dt,
                         double hx, double hy, double hz, int64_t nt, int64_t ce, const ps_array& glam,
                         const ps_array& T_final, double* loss, int64_t* recomputed, bool* redo, cudaStream_t s) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    *redo = false;
    *recomputed = 0;
    const int64_t n = numel(T0), n2 = n / 2, nseg = (nt + ce - 1) / ce;
    const size_t bytes = (size_t)n * 8, stride = (bytes + 255) / 256 * 256;
    const int64_t nbuf = 7 + nseg + ce - 1;  // Cs, Ls, μA, μB, μ64, fA, fB, checkpoints, segment states after them
    if (stride * nbuf + 512 > g_grad_bytes) {
        if (g_grad_scratch) cudaFree(g_grad_scratch);
        g_grad_scratch = nullptr;
        g_grad_bytes = 0;
        if (cudaMalloc(&g_grad_scratch, stride * nbuf + 512) != cudaSuccess) {
            cudaGetLastError();
            return fail(PS_ERR_NOMEM, "ps_diffusion3d_misfit_gradient: grid scratch of %zu bytes failed",
                        stride * nbuf + 512);
        }
        g_grad_bytes = stride * nbuf + 512;
    }
    char* scr = static_cast<char*>(g_grad_scratch);
    GridRun* r = reinterpret_cast<GridRun*>(scr);         // the forward's grid (T, lam)
    GridRun* rm = reinterpret_cast<GridRun*>(scr + 256);  // the adjoint's grid (μ)
    double* d_loss = reinterpret_cast<double*>(scr + 128);
    auto arr = [&](int64_t b) {
        ps_array a = T0;
        a.ptr = scr + 512 + stride * b;
        return a;
    };
    ps_array Cs = arr(0), Ls = arr(1), mA = arr(2), mB = arr(3), mu64 = arr(4), fA = arr(5), fB = arr(6);
    auto ckpt = [&](int64_t i) { return arr(7 + i); };
    auto seg = [&](int64_t j) { return arr(7 + nseg + j - 1); };  // j = 1 .. ce - 1
    SplitParams p{};
    double G;
    const bool iso = split_coeffs(PS_DIFF_FLUX_LAM, 0.0, dt, hx, hy, hz, &p, &G);
    const Box cells = {{1, 1, 1}, {T0.n[0] - 1, T0.n[1] - 1, T0.n[2] - 1}};
    const int g = st->num_sms * 8;
    auto copy = [&](const ps_array& dst, const ps_array& src) {
        return cudaMemcpyAsync(dst.ptr, src.ptr, bytes, cudaMemcpyDeviceToDevice, s) == cudaSuccess
                   ? PS_OK
                   : fail(PS_ERR_CUDA, "device copy failed");
    };
    auto step = [&](const ps_array& in, const ps_array& out) {
        return iso ? launch_grid_step<true, true>(GRID_MIDDLE, in, Cs, &Ls, out, p, cells, 0, s, st->d_err, r)
                   : launch_grid_step<true, false>(GRID_MIDDLE, in, Cs, &Ls, out, p, cells, 0, s, st->d_err, r);
    };
    // setup: grids of T and lam, pairs of lam and Ci, the first state
    PS_CUDA_TRY(cudaMemsetAsync(scr, 0, 512, s));
    absmax2_bits_kernel<<<st->num_sms * 4, 256, 0, s>>>(static_cast<const double2*>(T0.ptr),
                                                        static_cast<const double2*>(lam.ptr), n2, &r->maxT, &r->maxL);
    grid_setup_kernel<<<1, 1, 0, s>>>(r, G, 1);
    to_grid_kernel<<<g, 256, 0, s>>>(static_cast<const double2*>(T0.ptr), static_cast<float4*>(fB.ptr), n2, r, 0);
    to_grid_kernel<<<g, 256, 0, s>>>(static_cast<const double2*>(lam.ptr), static_cast<float4*>(Ls.ptr), n2, r, 1);
    ci_grid_kernel<<<g, 256, 0, s>>>(static_cast<const double2*>(Ci.ptr), static_cast<float4*>(Cs.ptr), n2, r);
    // every state buffer holds T0's boundary values (the steps write inner cells only): fA, and the checkpoints and
    // segment states behind fB, where T0 itself is
    PS_TRY(copy(ckpt(0), fB));
    const int64_t nmax = std::max(T0.n[0] * T0.n[1], std::max(T0.n[0] * T0.n[2], T0.n[1] * T0.n[2]));
    const unsigned gf = (unsigned)std::min<int64_t>((nmax + 255) / 256, 64);
    auto faces = [&](const ps_array& first, int64_t count) {  // grid.z <= 65535 per launch
        for (int64_t i = 0; i < count; i += 32768)
            grid_faces_copy_kernel<<<dim3(gf, 6, (unsigned)std::min<int64_t>(32768, count - i)), 256, 0, s>>>(
                static_cast<const float2*>(fB.ptr), reinterpret_cast<float2*>(static_cast<char*>(first.ptr) + stride * i),
                (int64_t)(stride / 8), T0.n[0], T0.n[1], T0.n[2]);
    };
    faces(fA, 1);
    if (nseg > 1) faces(ckpt(1), nseg - 1);
    if (std::min(ce, nt) > 1) faces(seg(1), std::min(ce, nt) - 1);
    // forward; a step that reaches a checkpoint writes its state there
    ps_array cur = ckpt(0);
    for (int64_t it = 0; it < nt; it++) {
        const bool at_ckpt = (it + 1) % ce == 0 && it + 1 < nt;
        const ps_array next = at_ckpt ? ckpt((it + 1) / ce) : cur.ptr == fA.ptr ? fB : fA;
        PS_TRY(step(cur, next));
        cur = next;
    }
    // T_nt in FP64, the misfit, μ_nt on its own grid
    grid_state_to_f64_kernel<<<g, 256, 0, s>>>(static_cast<const float2*>(cur.ptr), static_cast<double*>(mu64.ptr), n, r);
    if (T_final.ptr) PS_TRY(copy(T_final, mu64));
    grid_misfit_kernel<<<g, 256, 0, s>>>(static_cast<double*>(mu64.ptr), static_cast<const double*>(mu64.ptr),
                                         static_cast<const double*>(Tobs.ptr), static_cast<const double*>(Ci.ptr), dt,
                                         T0.n[0], T0.n[1], T0.n[2], d_loss);
    absmax2_bits_kernel<<<st->num_sms * 4, 256, 0, s>>>(static_cast<const double2*>(mu64.ptr), nullptr, n2, &rm->maxT,
                                                        nullptr);
    grid_setup_kernel<<<1, 1, 0, s>>>(rm, 1.0, 0);
    to_grid_kernel<<<g, 256, 0, s>>>(static_cast<const double2*>(mu64.ptr), static_cast<float4*>(mA.ptr), n2, rm, 0);
    PS_CUDA_TRY(cudaMemsetAsync(mB.ptr, 0, bytes, s));  // μ is zero on the boundary cells
    PS_CUDA_TRY(cudaMemsetAsync(glam.ptr, 0, bytes, s));
    // glam coefficients: -1/2 hh_d; the grid scales 2^-(shμ + shT) are applied in FP64 per cell
    dd c[3];
    const double h[3] = {hx, hy, hz};
    for (int d = 0; d < 3; d++) split_const(c[d], -0.5 * (h[d] * h[d]));
    // reverse sweep over the segments
    for (int64_t sidx = nseg - 1; sidx >= 0; sidx--) {
        const int64_t n0 = sidx * ce, n1 = std::min(nt, n0 + ce);
        auto state = [&](int64_t j) { return j == 0 ? ckpt(sidx) : seg(j); };
        for (int64_t j = 1; j < n1 - n0; j++) {
            PS_TRY(step(state(j - 1), state(j)));
            (*recomputed)++;
        }
        for (int64_t nn = n1 - 1; nn >= n0; nn--) {
            // glam from μ_{nn+1} and T_nn, and μ_nn, in one sweep
            PS_TRY(iso ? launch_grid_adj<true>(mA, Ls, Cs, state(nn - n0), mB, glam, p, c, cells, s, st->d_err, r, rm)
                       : launch_grid_adj<false>(mA, Ls, Cs, state(nn - n0), mB, glam, p, c, cells, s, st->d_err, r,
                                                rm));
            std::swap(mA, mB);
        }
    }
    PS_CUDA_TRY(cudaGetLastError());
    GridRun hr[2];
    double hl;
    PS_TRY(read_device_words(hr, scr, sizeof(GridRun), s));
    PS_TRY(read_device_words(hr + 1, rm, sizeof(GridRun), s));
    PS_TRY(read_device_words(&hl, d_loss, sizeof(double), s));
    *loss = hl;
    *redo = (hr[0].bad | hr[1].bad) != 0;
    return PS_OK;
}

}  // namespace ps

using namespace ps;

namespace ps {
int diffusion_box(int32_t form, const ps_array& T2, const ps_array& Tin, const ps_array& Ci, const ps_array& lam,
                  double lam_s, double dt, double hx, double hy, double hz, const Box& thread_box, int memopt,
                  int loopsize, int fp64_mode, cudaStream_t s, int* d_err, HideReq* hr = nullptr);
int diffusion_args(int32_t form, const ps_array& T2, const ps_array& Tin, const ps_array& Ci, const ps_array& lam);
}

extern "C" int ps_diffusion3d_run(int32_t form, ps_array T, ps_array T2, ps_array Ci, ps_array lam_arr, double lam,
                                  double dt, double hx, double hy, double hz, int64_t nt, const ps_launch* cfg,
                                  void* stream) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    PS_TRY(diffusion_args(form, T2, T, Ci, lam_arr));
    if (nt < 0) return fail(PS_ERR_ARG, "ps_diffusion3d_run: nt must be >= 0");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int memopt = cfg ? cfg->memopt : 1, loopsize = cfg ? cfg->loopsize : 0;
    int mode = cfg ? cfg->fp64_mode : PS_FP64_IEEE;
    if (mode < PS_FP64_IEEE || mode > PS_FP64_SPLIT_GRID) return fail(PS_ERR_ARG, "unknown fp64_mode %d", mode);
    const int64_t n = numel(T);
    const size_t bytes = (size_t)n * 8;
    const bool has_lam = form == PS_DIFF_FLUX_LAM;
    const Box full = {{0, 0, 0}, {T.n[0], T.n[1], T.n[2]}};
    const Box cells = {{1, 1, 1}, {T.n[0] - 1, T.n[1] - 1, T.n[2] - 1}};
    const int L = loopsize;  // 0: chosen per launch from the wave count
    bool split = T.dtype == PS_F64 && mode != PS_FP64_IEEE && tma_eligible(T) && tma_eligible(T2) &&
                 tma_eligible(Ci) && (!has_lam || tma_eligible(lam_arr)) && cells.hi[0] > cells.lo[0] &&
                 cells.hi[1] > cells.lo[1] && cells.hi[2] > cells.lo[2];
    ps_array A = T, B = T2;
    if (split && mode == PS_FP64_SPLIT_GRID && nt > 0) {
        // state, lam and Ci as grid / value pairs in scratch; T is written only by the final
        // conversion, which the device skips when a value left the grid range. The fallback (the
        // same run on value-relative split pairs) is enqueued behind the grid run with every
        // kernel predicated on the run's flag, so the call stays asynchronous; its pairs live in
        // four more scratch arrays.
        char* scr = nullptr;
        const size_t head = 256;
        PS_TRY(run_scratch(head + bytes * ((has_lam ? 1 : 0) + 3 + 4), &scr, s));
        GridRun* r = reinterpret_cast<GridRun*>(scr);
        ps_array Cs = Ci, Ls = lam_arr, Sa = T, Sb = T;
        Cs.ptr = scr + head;
        Sa.ptr = scr + head + bytes;
        Sb.ptr = scr + head + 2 * bytes;
        if (has_lam) Ls.ptr = scr + head + 3 * bytes;
        SplitParams p{};
        double G;
        const bool iso = split_coeffs(form, lam, dt, hx, hy, hz, &p, &G);
        const int g = st->num_sms * 8;
        PS_CUDA_TRY(cudaMemsetAsync(r, 0, sizeof(GridRun), s));
        const int64_t n2 = n / 2;  // nx is even (TMA eligibility)
        absmax2_bits_kernel<<<st->num_sms * 4, 256, 0, s>>>(static_cast<const double2*>(T.ptr),
                                              has_lam ? static_cast<const double2*>(lam_arr.ptr) : nullptr, n2,
                                              &r->maxT, &r->maxL);
        grid_setup_kernel<<<1, 1, 0, s>>>(r, G, has_lam ? 1 : 0);
        auto step = [&](GridStep kind, const ps_array& Tin, const ps_array& Cin, const ps_array* Lin,
                        const ps_array& out) {
            const ps_array* lin = has_lam ? Lin : nullptr;
            void* lout = has_lam ? Ls.ptr : nullptr;
            if (form == PS_DIFF_FLUX_LAM)
                return iso ? launch_grid_step<true, true>(kind, Tin, Cin, lin, out, p, cells, L, s, st->d_err, r, lout,
                                                          Cs.ptr)
                           : launch_grid_step<true, false>(kind, Tin, Cin, lin, out, p, cells, L, s, st->d_err, r,
                                                           lout, Cs.ptr);
            return iso ? launch_grid_step<false, true>(kind, Tin, Cin, nullptr, out, p, cells, L, s, st->d_err, r,
                                                       nullptr, Cs.ptr)
                       : launch_grid_step<false, false>(kind, Tin, Cin, nullptr, out, p, cells, L, s, st->d_err, r,
                                                        nullptr, Cs.ptr);
        };
        if (nt >= 2) {
            // the first step reads the caller's FP64 T, lam and Ci and converts them as it stages
            // them (writing the lam / Ci pairs of its cells); the boundary faces are converted here
            grid_faces64_kernel<<<dim3(st->num_sms, 6), 256, 0, s>>>(
                static_cast<const double*>(T.ptr), static_cast<float2*>(Sa.ptr), static_cast<float2*>(Sb.ptr),
                has_lam ? static_cast<const double*>(lam_arr.ptr) : nullptr, static_cast<float2*>(Ls.ptr), T.n[0],
                T.n[1], T.n[2], r);
            PS_TRY(step(GRID_FIRST64, T, Ci, &lam_arr, Sb));
            A = Sb;
            B = Sa;
        } else {
            // one step: convert first (the step writes T itself)
            to_grid_kernel<<<g, 256, 0, s>>>(static_cast<const double2*>(T.ptr), static_cast<float4*>(Sa.ptr), n2, r,
                                             0);
            if (has_lam)
                to_grid_kernel<<<g, 256, 0, s>>>(static_cast<const double2*>(lam_arr.ptr),
                                                 static_cast<float4*>(Ls.ptr), n2, r, 1);
            ci_grid_kernel<<<g, 256, 0, s>>>(static_cast<const double2*>(Ci.ptr), static_cast<float4*>(Cs.ptr), n2,
                                             r);
            A = Sa;
            B = Sb;
        }
        for (int64_t it = nt >= 2 ? 1 : 0; it < nt; ++it) {
            const bool last = it == nt - 1;  // the last step writes T as IEEE doubles
            PS_TRY(step(last ? GRID_LAST64 : GRID_MIDDLE, A, Cs, &Ls, last ? T : B));
            std::swap(A, B);
        }
        // the fallback: a PS_FP64_SPLIT_STATE run from T (left untouched by a flagged grid run),
        // each launch returning at once unless the flag is set
        const int* pred = &r->bad;
        char* fb = scr + head + bytes * ((has_lam ? 1 : 0) + 3);
        ps_array C2 = Ci, L2 = lam_arr, Fa = T, Fb = T;
        C2.ptr = fb;
        L2.ptr = fb + bytes;
        Fa.ptr = fb + 2 * bytes;
        Fb.ptr = fb + 3 * bytes;
        // small grids (one CTA per SM for the elementwise kernels, whole-z sweeps for the steps:
        // results do not depend on the sweep length), so the launches cost little when skipped
        const int gp = st->num_sms;
        const int Lz = (int)(cells.hi[2] - cells.lo[2]);
        split_pairs_kernel<<<gp, 256, 0, s>>>(static_cast<const double*>(Ci.ptr), static_cast<double*>(C2.ptr), n,
                                              st->d_err, pred);
        if (has_lam)
            split_pairs_kernel<<<gp, 256, 0, s>>>(static_cast<const double*>(lam_arr.ptr),
                                                  static_cast<double*>(L2.ptr), n, st->d_err, pred);
        split_pairs_kernel<<<gp, 256, 0, s>>>(static_cast<const double*>(T.ptr), static_cast<double*>(Fa.ptr), n,
                                              st->d_err, pred);
        copy_words_if_kernel<<<gp, 256, 0, s>>>(static_cast<const double*>(Fa.ptr), static_cast<double*>(Fb.ptr), n,
                                                pred);
        for (int64_t it = 0; it < nt; ++it) {
            PS_TRY(launch_split(form, Fb, Fa, C2, has_lam ? &L2 : nullptr, lam, dt, hx, hy, hz, cells, Lz, true, true,
                                s, st->d_err, pred));
            std::swap(Fa, Fb);
        }
        join_pairs_kernel<<<gp, 256, 0, s>>>(static_cast<const double*>(Fa.ptr), static_cast<double*>(T.ptr), T.n[0],
                                             T.n[1], T.n[2], pred);
        return finish_launch(s, 0, "ps_diffusion3d_run");
    }
    if (!split) {
        for (int64_t it = 0; it < nt; ++it) {
            PS_TRY(diffusion_box(form, B, A, Ci, lam_arr, lam, dt, hx, hy, hz, full, memopt, loopsize, PS_FP64_IEEE, s,
                                 st->d_err));
            std::swap(A, B);
        }
    } else {
        const bool state = mode == PS_FP64_SPLIT_STATE;
        char* scr = nullptr;
        const size_t need = bytes * ((has_lam ? 2 : 1) + (state ? 2 : 0));
        PS_TRY(run_scratch(need, &scr, s));
        ps_array Cs = Ci, Ls = lam_arr, Sa = T, Sb = T;
        Cs.ptr = scr;
        if (has_lam) Ls.ptr = scr + bytes;
        const int g = st->num_sms * 8;
        split_pairs_kernel<<<g, 256, 0, s>>>(static_cast<const double*>(Ci.ptr), static_cast<double*>(Cs.ptr), n,
                                             st->d_err);
        if (has_lam)
            split_pairs_kernel<<<g, 256, 0, s>>>(static_cast<const double*>(lam_arr.ptr),
                                                 static_cast<double*>(Ls.ptr), n, st->d_err);
        if (state) {
            Sa.ptr = scr + bytes * (has_lam ? 2 : 1);
            Sb.ptr = static_cast<char*>(Sa.ptr) + bytes;
            split_pairs_kernel<<<g, 256, 0, s>>>(static_cast<const double*>(T.ptr), static_cast<double*>(Sa.ptr), n,
                                                 st->d_err);
            PS_CUDA_TRY(cudaMemcpyAsync(Sb.ptr, Sa.ptr, bytes, cudaMemcpyDeviceToDevice, s));
            A = Sa;
            B = Sb;
        }
        for (int64_t it = 0; it < nt; ++it) {
            PS_TRY(launch_split(form, B, A, Cs, has_lam ? &Ls : nullptr, lam, dt, hx, hy, hz, cells, L, true, state, s,
                                st->d_err));
            std::swap(A, B);
        }
        if (state) {
            join_pairs_kernel<<<g, 256, 0, s>>>(static_cast<const double*>(A.ptr), static_cast<double*>(T.ptr), T.n[0],
                                                T.n[1], T.n[2]);
            A = T;
        }
    }
    if (A.ptr != T.ptr)  // odd nt: the last state is in T2
        PS_CUDA_TRY(cudaMemcpyAsync(T.ptr, A.ptr, (size_t)n * elsize(T.dtype), cudaMemcpyDeviceToDevice, s));
    return finish_launch(s, 0, "ps_diffusion3d_run");
}
