// ps_common.cuh -- shared host/device helpers of libps_b200.so.
#pragma once

#include <cuda.h>  // CUtensorMap and its enums only; the driver is reached through cudart
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <limits>
#include <utility>

#include "ps_gb300.h"

namespace ps {

// ---------------------------------------------------------------------------------------
// Error state (thread-local message, status codes of ps_gb300.h).
// ---------------------------------------------------------------------------------------
int fail(int status, const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
void clear_error();

#define PS_CUDA_TRY(call)                                       \
    do {                                                        \
        cudaError_t _ps_e = (call);                             \
        if (_ps_e != cudaSuccess) return ps::cuda_fail(_ps_e, #call); \
    } while (0)

#define PS_TRY(expr)                      \
    do {                                  \
        int _ps_rc = (expr);              \
        if (_ps_rc != PS_OK) return _ps_rc; \
    } while (0)

// Device-side error word bits (kernels OR them in; the host reads and clears the word).
enum : int { DEV_ERR_NONE = 0, DEV_ERR_TMA_TIMEOUT = 1, DEV_ERR_GRID_TIMEOUT = 2, DEV_ERR_RANGE = 4 };

// Per-device library state.
struct DeviceState {
    bool ready = false;
    int* d_err = nullptr;        // device error word (DEV_ERR_*)
    double* d_scratch = nullptr;  // small reduction scratch (library-owned)
    size_t scratch_bytes = 0;
    int num_sms = 0;
};

// Returns PS_ERR_NOT_INIT unless ps_init succeeded for the current device.
int current_state(DeviceState** st);
// Frees library-owned solver scratch (ps_finalize).
void stokes2d_free_scratch();
void diffusion_free_scratch();
void adjoint_free_scratch();
void acoustic_free_scratch();
void stokes3d_free_scratch();

// Copies `bytes` (<= 256 through pinned staging) from device memory on stream s and synchronises s.
int read_device_words(void* dst, const void* src, size_t bytes, cudaStream_t s);
// Reads (and clears) the device error word after a synchronisation.
int check_device_error(DeviceState* st, cudaStream_t s);

// After a launch: report launch errors; if sync, synchronise and report execution errors.
int finish_launch(cudaStream_t s, int sync, const char* what);

// ---------------------------------------------------------------------------------------
// Array validation.
// ---------------------------------------------------------------------------------------
inline int64_t numel(const ps_array& a) { return a.n[0] * a.n[1] * a.n[2]; }
inline size_t elsize(int32_t dtype) { return dtype == PS_F64 ? 8 : dtype == PS_F32 ? 4 : 2; }
int check_array(const ps_array& a, const char* name);
int check_same_dtype(const ps_array& a, const ps_array& b, const char* na, const char* nb);
int check_shape(const ps_array& a, int64_t nx, int64_t ny, int64_t nz, const char* name);

// Thread-index box of one call: full grid unless cfg gives a non-empty range.
struct Box {
    int64_t lo[3];
    int64_t hi[3];
};
Box launch_box(const ps_launch* cfg, const int64_t grid[3]);

// ---------------------------------------------------------------------------------------
// TMA tensor maps (cuTensorMapEncodeTiled through cudaGetDriverEntryPointByVersion).
// ---------------------------------------------------------------------------------------
// Encodes a 3-D tiled map over a dense column-major array with box (bx, by, 1), zero OOB
// fill. Returns PS_ERR_ALIGN if the array does not meet TMA's 16-byte rules.
int encode_plane_map(CUtensorMap* map, const ps_array& a, uint32_t bx, uint32_t by);
bool tma_eligible(const ps_array& a);
// 2-D map of a row-major bf16 matrix [rows][cols] with 128-byte swizzle; box = box_rows x 64
// columns (one 128-byte swizzle row). Reads past the matrix are zero-filled.
int encode_bf16_rows_sw128(CUtensorMap* map, const void* ptr, uint64_t cols, uint64_t rows, uint32_t box_cols,
                           uint32_t box_rows);
// Dense bf16 array of `rank` (2..4) dimensions, dims[0] fastest; the box's first extent is one swizzle row of
// 64 bytes (32 elements) or 128 bytes (64). Reads outside the array are zero-filled.
int encode_bf16_box(CUtensorMap* map, const void* ptr, int rank, const uint64_t* dims, const uint32_t* box);

// z-sweep length for loopsize = 0: a launch of cta_xy CTAs per z-block over wz planes with
// `slots` CTAs resident at once (occupancy x SMs) loses the idle part of its last wave and
// re-reads two halo planes per z-block; the candidate with the best product wins (ties: longer).
// Lengths below 16 are for grids whose launch would not fill the GPU at 16 (a step of the grid run
// at 128^3: 23.7 us with 16 planes per CTA on 256 of 456 places, 21.5 with 9 on 448; 64^3: 21.0
// with 16, 10.5 with 4). Results do not depend on the choice (every cell is computed the same way).
inline int auto_loopsize(int64_t cta_xy, int64_t wz, int64_t slots) {
    static const int cand[] = {64, 56, 48, 40, 32, 28, 24, 20, 16, 14, 12, 11, 10, 9, 8, 7, 6, 5, 4};
    int best = 64;
    double best_score = -1.0;
    for (int L : cand) {
        if (L < 16 && cta_xy * ((wz + 15) / 16) >= slots) break;
        const int64_t ctas = cta_xy * ((wz + L - 1) / L);
        const int64_t waves = (ctas + slots - 1) / slots;
        const double score = (double)ctas / (double)(waves * slots) * (double)L / (L + 2.0);
        if (score > best_score + 1e-9) {
            best_score = score;
            best = L;
        }
    }
    return best;
}

// Row blocks that one launch dimension holds. Kernels with blocks of few rows run taller grids in their
// 64-bit variants, whose blocks have 8.
constexpr int64_t kGridY = 65535;

// CTAs of `kernel` resident per SM (queried once per kernel by the caller's static cache).
template <typename K>
inline int resident_ctas(K kernel, int threads, int smem) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = 1;
    }
    return n;
}

// ---------------------------------------------------------------------------------------
// Boundary-first tile order (`@hide_communication` in one launch).
// ---------------------------------------------------------------------------------------
// A z-sweep launch over TX x TY x TZ tiles (x tile columns, y tile rows, z chunks) can run as a
// 1-D grid whose first `nb` CTAs take the tiles holding boundary cells -- bx0 / bx1 tile columns
// at the low / high x end, by0 / by1 rows, bz0 / bz1 chunks -- and the rest the inner block. Each
// boundary CTA, once its stores are done, increments `counter` (host-mapped memory); the host
// calls the communication when the counter reaches nb, while the inner tiles still run. The
// kernel never waits on the host. counter == NULL: an ordinary launch (blockIdx is the tile).
struct TileOrder {
    unsigned* counter;
    int TX, TY, TZ;
    int bx0, bx1, by0, by1, bz0, bz1;
    int nb;
};
// Host: the order of a TX x TY x TZ tile launch whose tiles start at cell lo + t * tile (per
// axis) over the cells [lo, end); boundary cells are c < lo_end or c >= hi_start.
TileOrder make_tile_order(const int64_t ntiles[3], const int64_t lo[3], const int64_t tile[3], const int64_t end[3],
                          const int64_t lo_end[3], const int64_t hi_start[3], unsigned* counter);
// What a caller asks of a boundary-first launch (the launcher fills nb).
struct HideReq {
    int64_t lo_end[3], hi_start[3];
    unsigned* counter;
    int nb;
};
// Host: the thread's host-mapped progress word (allocated on first use; NULL pointers if the
// device cannot map host memory).
int progress_word(volatile unsigned** host, unsigned** dev);

__device__ __forceinline__ uint3 ordered_tile(const TileOrder& o) {
    if (!o.counter) return make_uint3(blockIdx.x, blockIdx.y, blockIdx.z);
    int i = (int)blockIdx.x;
    const int IX = o.TX - o.bx0 - o.bx1, IY = o.TY - o.by0 - o.by1;
    if (i >= o.nb) {  // the inner block, x fastest
        i -= o.nb;
        return make_uint3(o.bx0 + i % IX, o.by0 + (i / IX) % IY, o.bz0 + i / (IX * IY));
    }
    const int layer = o.TX * o.TY;
    const int nzfull = (o.bz0 + o.bz1) * layer;
    if (i < nzfull) {  // whole layers at both z ends
        const int l = i / layer, r = i % layer;
        return make_uint3(r % o.TX, r / o.TX, l < o.bz0 ? l : o.TZ - o.bz1 + (l - o.bz0));
    }
    i -= nzfull;  // the frames of the middle layers: whole rows at both y ends, then column ends
    const int frame = layer - IX * IY;
    const int z = o.bz0 + i / frame;
    int r = i % frame;
    const int nyfull = (o.by0 + o.by1) * o.TX;
    if (r < nyfull) {
        const int row = r / o.TX;
        return make_uint3(r % o.TX, row < o.by0 ? row : o.TY - o.by1 + (row - o.by0), z);
    }
    r -= nyfull;
    const int ex = o.bx0 + o.bx1, c = r % ex;
    return make_uint3(c < o.bx0 ? c : o.TX - o.bx1 + (c - o.bx0), o.by0 + r / ex, z);
}

// Called by every thread of a CTA after its last global store (plain stores only).
__device__ __forceinline__ void ordered_tile_done(const TileOrder& o) {
    if (!o.counter || (int)blockIdx.x >= o.nb) return;  // uniform over the CTA
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0 && threadIdx.z == 0) {
        __threadfence_system();
        atomicAdd_system(o.counter, 1u);
    }
}

// ---------------------------------------------------------------------------------------
// Division by a number known on the host, correctly rounded.
// ---------------------------------------------------------------------------------------
// Method of N. Brisebarre, J.-M. Muller and S. K. Raina ("Accelerating correctly rounded floating-point
// division when the divisor is known in advance", IEEE Trans. Computers 53 (2004) 1069-1072): with
// 1/b held as yh + yl, RN(a yh + RN(a yl)) -- one multiply and one FMA -- equals RN(a/b) unless a/b
// lies within about 2^-2p of a midpoint between neighbouring p-bit numbers. Such dividends are few
// and computable: with integer significands A, B in [2^(p-1), 2^p) and a midpoint M/2^p (A >= B) or
// M/2^(p+1) (A < B), the distance is |k| / (2^p B) or |k| / (2^(p+1) B), k = 2^p A - M B (2^(p+1) A - M B)
// != 0, so they solve a linear congruence for each small k. make_div solves it, tries the scheme on
// each solution against the IEEE division and moves yl by an ulp until all agree (significands
// enter only, so that covers every exponent). yh is 1/b rounded towards zero, so yl has its sign
// and a zero dividend keeps the quotient's sign; yl is never 0, so infinities pass too.
//
// Dividends below `lo` in magnitude, where a yl or the quotient could be subnormal (zeros
// excepted), take div_slow; so do all dividends of divisors outside [2^-20, 2^20] (FP32) or
// [2^-60, 2^60] (FP64), and of the 3 % of divisors for which no yl within an ulp passes (a wider search
// finds no more of them). Large dividends, infinities and NaN need no test: the quotient overflows
// where a/b does. The test is on integer keys (zero has the largest) and costs no FP64 instruction;
// the FP64 division is 2 FP64 instructions instead of 7 (GB300 issues 2 FP64 per clock per SM).
//
// A launch with a divisor without a pair runs a variant of its kernel that tests every dividend at once (PAIR =
// false, DivG). Quotients taken untested first, for nothing, and then the tested ones: acoustic FP32 255^3 214 us per step
// instead of 142 (110 where all have pairs), FP64 1744 instead of 1355 (870); Stokes3D 127^3 FP32 91 instead of
// 75 (61) per iteration, FP64 1306 instead of 752 (449).
//
// div_slow, for a divisor without a pair: Markstein's method (P. W. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Develop. 34 (1990)
// 111-119): with y = RN(1/b) and a quotient q within one ulp of a/b, the remainder r = a - b q is
// exact in one FMA and RN(q + r y) = RN(a/b). The first quotient RN(a y) can be 1.5 ulps off, so one
// correction brings it within an ulp and a second rounds it correctly: 1 multiply + 4 FMAs, for
// dividends that keep a y and the quotient normal and the remainder, a multiple of 2^(e(a) - 2p + 1),
// representable. Everything else there is the IEEE division. Results equal a / b bit for bit (checked
// against the IEEE division by ps_check_division).
template <typename T>
struct DivC {
    T b, yh, yl;
    uint32_t lo;   // div_key of the smallest dividend of the pair; kNoPair: no pair (zeros only)
    uint32_t fix;  // no pair, Markstein's method: yh = RN(1/b), yl a zero of its sign (exact for zeros), and the
                   // number of keys from kMarkstein on that it takes
};
constexpr uint32_t kNoPair = 0xFFFFFFFFu;
// Keys of Markstein's method: 2^-100 <= |a| <= 2^70 (FP32), 2^-960 <= |a| <= 2^900 (FP64).
template <typename T>
constexpr uint32_t kMarkstein = sizeof(T) == 4 ? 0x1AFFFFFFu : 0x07DFFFFFu;
template <typename T>
constexpr uint32_t kMarksteinEnd = sizeof(T) == 4 ? 0xC5000000u : 0xF0600000u;

// Key of a dividend: grows with |a|, largest for zeros.
__host__ __device__ __forceinline__ uint32_t div_key_bits(uint32_t hi, uint32_t rest) {
    return (hi << 1) + (rest ? 0u : 0xFFFFFFFFu);
}
__device__ __forceinline__ uint32_t div_key(float a) { return div_key_bits(__float_as_uint(a), 0u); }
__device__ __forceinline__ uint32_t div_key(double a) {
    return div_key_bits((uint32_t)__double2hiint(a), (uint32_t)__double2loint(a));
}

// Whether RN(a yh + RN(a yl)) = RN(a/b) for every dividend that can fail: b = B in [2^(p-1), 2^p).
template <typename T>
inline bool div_pair_exact(T b, T yh, T yl) {
    constexpr int p = sizeof(T) == 4 ? 24 : 53;
    const uint64_t B = (uint64_t)b;
    int t = 0;
    while (!((B >> t) & 1)) t++;
    const uint64_t Bo = B >> t;
    uint64_t inv = Bo;  // Bo^-1 mod 2^64 (Newton)
    for (int i = 0; i < 6; i++) inv *= 2 - Bo * inv;
    // relative error of the pair: at most 3/2 ulp(yl) (yl rounded, then moved by one ulp), half an ulp of
    // a yl and 2^-2p / 4 from its underflow, together 8.25 2^-2p at most (|yl| <= 2^(1-p) yh): |k| < 17 for
    // A < B, half of that for A >= B
    for (int side = 0; side < 2; side++) {
        const int m = p + side;  // midpoints M / 2^m, M odd in (2^p, 2^(p+1))
        for (int k = -20; k <= 20; k++) {
            if (k == 0 || t > 4 || (k & ((1 << t) - 1))) continue;  // k is a multiple of 2^t
            // M Bo = -k / 2^t (mod 2^(m - t)): 2^t or 2^(t+1) values of M below 2^(p+1)
            const uint64_t mod = 1ull << (m - t);
            const uint64_t M0 = ((uint64_t)(-(int64_t)(k >> t)) * inv) & (mod - 1);
            for (uint64_t M = M0; M < (2ull << p); M += mod) {
                if (M <= (1ull << p) || !(M & 1)) continue;
                const __int128 v = (__int128)M * B + k;
                const uint64_t A = (uint64_t)(v >> m);
                if (((__int128)A << m) != v || A < (1ull << (p - 1)) || A >= (1ull << p)) continue;
                if (side == 0 ? A < B : A >= B) continue;
                const T a = (T)A;
                if (std::fma(a, yh, a * yl) != a / b) return false;
            }
        }
    }
    return true;
}
template <typename T>
inline DivC<T> div_without_pair(DivC<T> d) {
    d.yh = (T)1 / d.b;
    d.yl = std::copysign((T)0, d.b);  // (of yh's sign, for a zero quotient's)
    d.lo = kNoPair;
    d.fix = kMarksteinEnd<T> - kMarkstein<T>;
    return d;
}
template <typename T>
inline DivC<T> make_div(T b) {
    const T lim = sizeof(T) == 4 ? (T)0x1p20 : (T)0x1p60;
    const T ab = std::fabs(b);
    DivC<T> d;
    d.b = b;
    d.lo = kNoPair;  // zeros only: their quotient is a zero, or NaN for a zero or NaN divisor
    d.yh = ab > 0 ? std::copysign((T)1, b) : std::numeric_limits<T>::quiet_NaN();
    d.yl = d.yh;
    d.fix = 0;
    if (!(ab >= 1 / lim && ab <= lim)) return d;
    constexpr int p = sizeof(T) == 4 ? 24 : 53;
    const int e = std::ilogb(ab);
    const T B = std::ldexp(ab, p - 1 - e);  // the integer significand
    T yh = (T)1 / B;
    T r = std::fma(-B, yh, (T)1);  // exact
    if (r < 0) {
        yh = std::nextafter(yh, (T)0);
        r = std::fma(-B, yh, (T)1);
    }
    // a power of two has r = 0: any yl far below the last place of yh leaves the exact quotient
    const T y0 = r == 0 ? std::ldexp(yh, -2 * p) : r / B;
    for (int j = 0; j < 3; j++) {
        const T yl = j == 0 ? y0 : std::nextafter(y0, j == 1 ? (T)1 : (T)0);
        if (!(yl > 0) || !div_pair_exact(B, yh, yl)) continue;
        d.yh = std::copysign(std::ldexp(yh, p - 1 - e), b);
        d.yl = std::copysign(std::ldexp(yl, p - 1 - e), b);
        // quotients of 2^-100 (2^-960) and above: a yl is rounded to 2^-50 (2^-113) of the quotient or better
        const T lo = std::ldexp((T)1, e + 1 - (sizeof(T) == 4 ? 100 : 960));
        if (sizeof(T) == 4) {
            uint32_t u;
            memcpy(&u, &lo, 4);
            d.lo = div_key_bits(u, 0u);
        } else {
            uint64_t u;
            memcpy(&u, &lo, 8);
            d.lo = div_key_bits((uint32_t)(u >> 32), 0u);
        }
        return d;
    }
    return div_without_pair(d);
}
// The divisors of one kernel; returns the key from which all of them take their pairs. Where one has none, it is kNoPair
// and they all divide by Markstein's method (or IEEE).
template <typename T>
inline uint32_t make_div3(const T b[3], DivC<T> d[3]) {
    d[0] = make_div(b[0]);
    d[1] = b[1] == b[0] ? d[0] : make_div(b[1]);
    d[2] = b[2] == b[0] ? d[0] : b[2] == b[1] ? d[1] : make_div(b[2]);
    const uint32_t lo = std::max(d[0].lo, std::max(d[1].lo, d[2].lo));
    if (lo == kNoPair)
        for (int i = 0; i < 3; i++)
            if (d[i].lo != kNoPair) d[i] = div_without_pair(d[i]);
    return lo;
}
__device__ __forceinline__ float div_pair(float a, const DivC<float>& d) { return fmaf(a, d.yh, a * d.yl); }
__device__ __forceinline__ double div_pair(double a, const DivC<double>& d) { return fma(a, d.yh, a * d.yl); }
__device__ __forceinline__ float div_markstein(float a, const DivC<float>& d) {
    float q = a * d.yh;
    float r = fmaf(-q, d.b, a);
    q = fmaf(r, d.yh, q);
    r = fmaf(-q, d.b, a);
    return fmaf(r, d.yh, q);
}
__device__ __forceinline__ double div_markstein(double a, const DivC<double>& d) {
    double q = a * d.yh;
    double r = fma(-q, d.b, a);
    q = fma(r, d.yh, q);
    r = fma(-q, d.b, a);
    return fma(r, d.yh, q);
}
template <typename T>
__device__ __forceinline__ T div_slow(T a, const DivC<T>& d) {
    const uint32_t k = div_key(a);
    if (d.fix && k >= kMarkstein<T> && k < kMarksteinEnd<T>) return div_markstein(a, d);
    return a / d.b;
}
template <typename T>
__device__ __forceinline__ T div_c(T a, const DivC<T>& d) {
    return div_key(a) >= d.lo ? div_pair(a, d) : div_slow(a, d);
}

// A divisor whose quotients are taken without the test: the smallest key of the dividends is kept in
// *key, and the caller computes again with DivC where *key came out below its divisors' lo.
template <typename T>
struct DivF {
    const DivC<T>& d;
    uint32_t* key;
};
// A divisor that has a pair, for kernels that only test (FP32 one-launch Stokes3D iteration at 127^3: 205 us against 209
// with DivC, whose Markstein branch is one more).
template <typename T>
struct DivP {
    const DivC<T>& d;
};
// A divisor of a launch whose divisors have no pairs (make_div3).
template <typename T>
struct DivG {
    const DivC<T>& d;
};
// A divisor of either kind, in a kernel that is compiled once for both: keys lo .. lo + span - 1 take its pair or
// Markstein's method (the README's FP32 diffusion step at 255^3: 102 us with pairs, 113 without; with DivC 112
// and 134).
template <typename T>
struct DivA {
    const DivC<T>& d;
    uint32_t lo, span;
};
template <typename T>
inline void div_keys(const DivC<T>& d, uint32_t* lo, uint32_t* span) {
    *lo = d.fix ? kMarkstein<T> : d.lo == kNoPair ? 0u : d.lo;
    *span = d.fix ? d.fix : 0u - *lo;
}
// What a kernel that tests every dividend once divides by.
template <typename T, bool PAIR>
using DivBy = std::conditional_t<PAIR, const DivC<T>&, DivG<T>>;

// x * 2^k by an integer addition to the exponent (a multiplication is an FP64 instruction). Equal to
// the product, bit for bit, for zeros and wherever x and x 2^k are normal: *key keeps x's key as
// DivF does, so small x make the caller compute again, and becomes 0 for |x| >= 2^900, infinities and
// NaN. lo >= 2^-1019 with the divisors' range, so k >= -2 keeps the result normal.
__device__ __forceinline__ double scale_pow2(double x, int k, uint32_t* key) {
    const int hi = __double2hiint(x);
    const uint32_t kx = div_key(x);
    *key = min(*key, kx < 0xF0600000u || kx == 0xFFFFFFFFu ? kx : 0u);
    return __hiloint2double(kx == 0xFFFFFFFFu ? hi : hi + (k << 20), __double2loint(x));
}

// 2 a b for a finite 2 a, as the product times two: equal to (2 a) b bit for bit where scale_pow2 is, and a product
// that underflowed to zero (whose double may not) makes the caller compute again too.
__device__ __forceinline__ double twice_product(double a, double b, uint32_t* key) {
    const double x = a * b;
    if (div_key(x) == 0xFFFFFFFFu && div_key(a) != 0xFFFFFFFFu && div_key(b) != 0xFFFFFFFFu) *key = 0u;
    if ((__double2hiint(a) & 0x7FFFFFFF) >= 0x78300000) *key = 0u;  // |a| < 2^900: 2 a is finite
    return scale_pow2(x, 1, key);
}

// a / h for statement helpers used with a plain divisor (host or device) or a DivC (device)
template <typename T>
__host__ __device__ __forceinline__ T dvd(T a, T h) {
    return a / h;
}
template <typename T>
__device__ __forceinline__ T dvd(T a, const DivC<T>& h) {
    return div_c(a, h);
}
// A value that the compiler may not compute with before this point: without it the instructions of an IEEE division
// that is hardly ever taken are issued beside the quotient that is (3 of them on the FP64 pipe).
__device__ __forceinline__ float not_ahead(float a) {
    asm volatile("" : "+f"(a));
    return a;
}
__device__ __forceinline__ double not_ahead(double a) {
    asm volatile("" : "+d"(a));
    return a;
}
template <typename T>
__device__ __forceinline__ T dvd(T a, const DivG<T>& h) {
    const uint32_t k = div_key(a);
    if (k - kMarkstein<T> < h.d.fix) return div_markstein(a, h.d);
    if (k == 0xFFFFFFFFu) return a * h.d.yh;
    return not_ahead(a) / h.d.b;
}
template <typename T>
__device__ __forceinline__ T dvd(T a, const DivP<T>& h) {
    if (div_key(a) >= h.d.lo) return div_pair(a, h.d);
    return not_ahead(a) / h.d.b;
}
template <typename T>
__device__ __forceinline__ T dvd(T a, const DivA<T>& h) {
    const uint32_t k = div_key(a);
    if (k - h.lo < h.span) return h.d.fix ? div_markstein(a, h.d) : div_pair(a, h.d);
    return k == 0xFFFFFFFFu ? div_pair(a, h.d) : a / h.d.b;
}
template <typename T>
__device__ __forceinline__ T dvd(T a, const DivF<T>& h) {
    *h.key = min(*h.key, div_key(a));
    return div_pair(a, h.d);
}

// ---------------------------------------------------------------------------------------
// Programmatic dependent launch: a kernel launched with launch_dependent() may start while the
// kernel before it on the stream finishes its last wave; it waits in grid_dependency_wait() (a
// no-op in an ordinary launch) until that kernel has completed and its stores are visible, so
// every read of data the previous kernel wrote must come after the wait.
//
// A kernel that calls grid_dependents_may_launch() lets the next one's blocks in while its own run. That is for
// kernels meant to run beside each other: in a chain the early blocks take the places that come free
// first, and the SMs are loaded unevenly for the rest of the launch (accelerated Stokes2D iteration, FP64
// 350^2: 19.7 us with the call, 14.8 without, 18.4 in ordinary launches; FP32 300 x 411 5.6 and 4.6).
// Without it the next kernel's blocks start as the last of this one's finish.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependents_may_launch() { asm volatile("griddepcontrol.launch_dependents;"); }
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                    Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// ---------------------------------------------------------------------------------------
// Device helpers.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ int64_t idx3(int64_t x, int64_t y, int64_t z, int64_t nx, int64_t ny) {
    return x + nx * (y + ny * z);
}

// Julia's Base.max / Base.min for IEEE floats (NaN-propagating; -0.0 < 0.0).
template <typename T>
__device__ __forceinline__ T jl_max(T x, T y) {
    T diff = x - y;
    T r = signbit(diff) ? y : x;
    return (isnan(x) || isnan(y)) ? diff : r;
}
template <typename T>
__device__ __forceinline__ T jl_min(T x, T y) {
    T diff = x - y;
    T r = signbit(diff) ? x : y;
    return (isnan(x) || isnan(y)) ? diff : r;
}
// The same for doubles without FP64 instructions (GB300 issues FP64 at 2 per clock per SM): the
// bits of a double with the magnitude bits flipped for negative values order as the values do,
// with -0.0 below 0.0, so for non-NaN operands the larger key is the result above, bit for bit
// (equal keys are equal values); a NaN operand is returned itself, as Julia's max and min do (a
// NaN either way: its payload is the operand's instead of the difference's).
__device__ __forceinline__ long long jl_key(long long b) { return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFLL); }
__device__ __forceinline__ bool jl_nan_bits(long long b) { return (b & 0x7FFFFFFFFFFFFFFFLL) > 0x7FF0000000000000LL; }
template <>
__device__ __forceinline__ double jl_max<double>(double x, double y) {
    const long long bx = __double_as_longlong(x), by = __double_as_longlong(y);
    const double r = jl_key(bx) >= jl_key(by) ? x : y;
    return jl_nan_bits(bx) ? x : jl_nan_bits(by) ? y : r;
}
template <>
__device__ __forceinline__ double jl_min<double>(double x, double y) {
    const long long bx = __double_as_longlong(x), by = __double_as_longlong(y);
    const double r = jl_key(bx) < jl_key(by) ? x : y;
    return jl_nan_bits(bx) ? x : jl_nan_bits(by) ? y : r;
}
// Floats: max.NaN / min.NaN order -0.0 below 0.0 and give the canonical NaN when an operand is NaN,
// as the subtraction above does on the GPU (checked over signed zeros, subnormals, infinities and
// NaNs against Julia's rules): one instruction instead of six.
template <>
__device__ __forceinline__ float jl_max<float>(float x, float y) {
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(x), "f"(y));
    return d;
}
template <>
__device__ __forceinline__ float jl_min<float>(float x, float y) {
    float d;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(x), "f"(y));
    return d;
}

// --- mbarrier / TMA inline PTX (sm_90+; used on sm_103a) ---------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Orders this thread's generic-proxy shared-memory writes before later async-proxy (TMA) accesses
// of the same bytes (a staged slot rewritten in place and later refilled by a TMA load).
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after ~2^22 polls (each poll may itself suspend briefly).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < (1 << 22); ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

}  // namespace ps
