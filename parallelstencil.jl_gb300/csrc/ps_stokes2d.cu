// ps_stokes2d.cu -- pseudo-transient (PT) viscous Stokes 2-D kernels and solvers of libps_b200.so.
//
// Reference: miniapps/Stokes2D.jl:11-55 (kernels), :107-125 (PT loop), :117-123 (error check).
//
//   s2_* device functions     the arithmetic of each reference statement, shared by every kernel
//                             below so all paths round identically
//   one-to-one kernels        compute_timesteps!, compute_P!, compute_τ!, compute_dV!, compute_V!,
//                             bc_x!, bc_y! -- the drop-in replacements of the six `@parallel` calls
//   s2_cells, s2_faces        one whole PT iteration in place, one thread per position; results are
//                             identical to the six-kernel sequence. Optional fused FP64 reduction of
//                             Σ|Rx|, Σ|Ry|, Σ|∇V|.
//   s2_residual64             FP64 residuals of the current state (no pseudo-time update) for the
//                             defect-correction outer loop.
//   ps_stokes2d_solve         PT solve to `tol` in FP64 (mode 0) or with FP32 PT sweeps on the
//                             correction and an FP64 residual / update / convergence check (mode 1).
//                             Iterations run as CUDA graphs of `nout` iterations.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <mutex>
#include <vector>

#include "ps_common.cuh"

namespace ps {

// =======================================================================================
// Statement arithmetic (Stokes2D.jl:11-37); literals cast to T like the reference does.
// =======================================================================================
template <typename T>
__host__ __device__ __forceinline__ T s2_dtV(T Vsc, T min_dxy2, T m0, T m1) {
    T av = (m0 + m1) * T(0.5);
    return ((Vsc * min_dxy2) / av) / T(4.1);
}
template <typename T>
__host__ __device__ __forceinline__ T s2_dtPt(T Ptsc, T mus, T max_nxy) {
    return ((Ptsc * T(4.1)) * mus) / max_nxy;
}
// H: the divisor's type -- T, or DivC<T> (the correctly rounded division by a host-known number)
template <typename T, typename H>
__host__ __device__ __forceinline__ T s2_divV(T vx0, T vx1, T vy0, T vy1, H dx, H dy) {
    return dvd(vx1 - vx0, dx) + dvd(vy1 - vy0, dy);
}
template <typename T, typename H>
__host__ __device__ __forceinline__ T s2_tau_nn(T mus, T v0, T v1, T divV, H h) {
    return (T(2.0) * mus) * (dvd(v1 - v0, h) - (T(1.0) / T(3.0)) * divV);
}
// msum: the four corner viscosities summed in the macro's order ((m00 + m10) + m01) + m11
template <typename T, typename H>
__host__ __device__ __forceinline__ T s2_tau_xy_sum(T msum, T dyVx, T dxVy, H dx, H dy) {
    T av = msum * T(0.25);
    return (T(2.0) * av) * (T(0.5) * (dvd(dyVx, dy) + dvd(dxVy, dx)));
}
template <typename T, typename H>
__host__ __device__ __forceinline__ T s2_tau_xy(T m00, T m10, T m01, T m11, T dyVx, T dxVy, H dx, H dy) {
    return s2_tau_xy_sum(((m00 + m10) + m01) + m11, dyVx, dxVy, dx, dy);
}
// The same two statements in FP64 with the factors 2, 0.25 and 0.5 gathered into one power of two applied
// to the product (equal bit for bit while nothing on the way is subnormal or overflows: the keys).
__device__ __forceinline__ double s2_tau_nn(double mus, double v0, double v1, double divV, DivF<double> h) {
    const double e = dvd(v1 - v0, h) - (1.0 / 3.0) * divV;
    return twice_product(mus, e, h.key);
}
__device__ __forceinline__ double s2_tau_xy_sum(double msum, double dyVx, double dxVy, DivF<double> dx, DivF<double> dy) {
    const double e = dvd(dyVx, dy) + dvd(dxVy, dx);
    *dx.key = min(*dx.key, min(div_key(msum), div_key(e)));
    return scale_pow2(msum * e, -2, dx.key);
}
template <typename T, typename H>
__host__ __device__ __forceinline__ T s2_Rx(T txx_l, T txx_r, T txy_b, T txy_t, T p_l, T p_r, H dx, H dy) {
    return (dvd(txx_r - txx_l, dx) + dvd(txy_t - txy_b, dy)) - dvd(p_r - p_l, dx);
}
template <typename T, typename H>
__host__ __device__ __forceinline__ T s2_Ry_core(T tyy_b, T tyy_t, T txy_l, T txy_r, T p_b, T p_t, H dx, H dy) {
    return (dvd(tyy_t - tyy_b, dy) + dvd(txy_r - txy_l, dx)) - dvd(p_t - p_b, dy);
}

template <typename T>
struct S2P {
    DivC<T> dx, dy;
    T dampX, dampY, Vsc, Ptsc, min_dxy2, max_nxy;
    uint32_t lo;  // the smallest dividend key both divisors take without a test
};

template <typename T>
static S2P<T> s2p(const ps_stokes2d_params& p) {
    const T h[3] = {(T)p.dx, (T)p.dy, (T)p.dx};
    DivC<T> d[3];
    const uint32_t lo = make_div3(h, d);
    return S2P<T>{d[0],      d[1],      (T)p.dampX,    (T)p.dampY,    (T)p.Vsc,
                  (T)p.Ptsc, (T)p.min_dxy2, (T)p.max_nxy, lo};
}

#define A2(a, i, j, n0) (a)[(int64_t)(i) + (int64_t)(n0) * (int64_t)(j)]

// =======================================================================================
// One-to-one kernels (grid = max extents of the kernel's array arguments).
// =======================================================================================
template <typename T>
__global__ void s2_timesteps_k(T* dtVx, T* dtVy, T* dtPt, const T* __restrict__ Mus, int64_t nx, int64_t ny, S2P<T> p) {
    int64_t tx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, ty = blockIdx.y * (int64_t)blockDim.y + threadIdx.y;
    if (tx >= nx || ty >= ny) return;
    if (tx < nx - 1 && ty < ny - 2)
        A2(dtVx, tx, ty, nx - 1) = s2_dtV(p.Vsc, p.min_dxy2, A2(Mus, tx, ty + 1, nx), A2(Mus, tx + 1, ty + 1, nx));
    if (tx < nx - 2 && ty < ny - 1)
        A2(dtVy, tx, ty, nx - 2) = s2_dtV(p.Vsc, p.min_dxy2, A2(Mus, tx + 1, ty, nx), A2(Mus, tx + 1, ty + 1, nx));
    A2(dtPt, tx, ty, nx) = s2_dtPt(p.Ptsc, A2(Mus, tx, ty, nx), p.max_nxy);
}

template <typename T>
__global__ void s2_P_k(T* divV, T* Pt, const T* __restrict__ Vx, const T* __restrict__ Vy, const T* __restrict__ dtPt,
                       int64_t nx, int64_t ny, S2P<T> p) {
    int64_t tx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, ty = blockIdx.y * (int64_t)blockDim.y + threadIdx.y;
    if (tx >= nx || ty >= ny) return;
    T d = s2_divV(A2(Vx, tx, ty, nx + 1), A2(Vx, tx + 1, ty, nx + 1), A2(Vy, tx, ty, nx), A2(Vy, tx, ty + 1, nx), p.dx, p.dy);
    A2(divV, tx, ty, nx) = d;
    A2(Pt, tx, ty, nx) = A2(Pt, tx, ty, nx) - A2(dtPt, tx, ty, nx) * d;
}

template <typename T>
__global__ void s2_tau_k(const T* __restrict__ divV, T* txx, T* tyy, T* txy, const T* __restrict__ Vx,
                         const T* __restrict__ Vy, const T* __restrict__ Mus, int64_t nx, int64_t ny, S2P<T> p) {
    int64_t tx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, ty = blockIdx.y * (int64_t)blockDim.y + threadIdx.y;
    if (tx >= nx || ty >= ny) return;
    T m = A2(Mus, tx, ty, nx), d = A2(divV, tx, ty, nx);
    A2(txx, tx, ty, nx) = s2_tau_nn(m, A2(Vx, tx, ty, nx + 1), A2(Vx, tx + 1, ty, nx + 1), d, p.dx);
    A2(tyy, tx, ty, nx) = s2_tau_nn(m, A2(Vy, tx, ty, nx), A2(Vy, tx, ty + 1, nx), d, p.dy);
    if (tx < nx - 1 && ty < ny - 1)
        A2(txy, tx, ty, nx - 1) =
            s2_tau_xy(A2(Mus, tx, ty, nx), A2(Mus, tx + 1, ty, nx), A2(Mus, tx, ty + 1, nx), A2(Mus, tx + 1, ty + 1, nx),
                      A2(Vx, tx + 1, ty + 1, nx + 1) - A2(Vx, tx + 1, ty, nx + 1),
                      A2(Vy, tx + 1, ty + 1, nx) - A2(Vy, tx, ty + 1, nx), p.dx, p.dy);
}

template <typename T>
__global__ void s2_dV_k(T* Rx, T* Ry, T* dVxdt, T* dVydt, const T* __restrict__ Pt, const T* __restrict__ Rog,
                        const T* __restrict__ txx, const T* __restrict__ tyy, const T* __restrict__ txy, int64_t nx,
                        int64_t ny, S2P<T> p) {
    int64_t tx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, ty = blockIdx.y * (int64_t)blockDim.y + threadIdx.y;
    if (tx >= nx || ty >= ny) return;
    if (tx < nx - 1 && ty < ny - 2) {
        T r = s2_Rx(A2(txx, tx, ty + 1, nx), A2(txx, tx + 1, ty + 1, nx), A2(txy, tx, ty, nx - 1),
                    A2(txy, tx, ty + 1, nx - 1), A2(Pt, tx, ty + 1, nx), A2(Pt, tx + 1, ty + 1, nx), p.dx, p.dy);
        A2(Rx, tx, ty, nx - 1) = r;
        A2(dVxdt, tx, ty, nx - 1) = p.dampX * A2(dVxdt, tx, ty, nx - 1) + r;
    }
    if (tx < nx - 2 && ty < ny - 1) {
        T r = s2_Ry_core(A2(tyy, tx + 1, ty, nx), A2(tyy, tx + 1, ty + 1, nx), A2(txy, tx, ty, nx - 1),
                         A2(txy, tx + 1, ty, nx - 1), A2(Pt, tx + 1, ty, nx), A2(Pt, tx + 1, ty + 1, nx), p.dx, p.dy) +
              (A2(Rog, tx + 1, ty, nx) + A2(Rog, tx + 1, ty + 1, nx)) * T(0.5);
        A2(Ry, tx, ty, nx - 2) = r;
        A2(dVydt, tx, ty, nx - 2) = p.dampY * A2(dVydt, tx, ty, nx - 2) + r;
    }
}

template <typename T>
__global__ void s2_V_k(T* Vx, T* Vy, const T* __restrict__ dVxdt, const T* __restrict__ dVydt,
                       const T* __restrict__ dtVx, const T* __restrict__ dtVy, int64_t nx, int64_t ny) {
    int64_t tx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, ty = blockIdx.y * (int64_t)blockDim.y + threadIdx.y;
    if (tx > nx || ty > ny) return;
    if (tx < nx - 1 && ty < ny - 2)
        A2(Vx, tx + 1, ty + 1, nx + 1) = A2(Vx, tx + 1, ty + 1, nx + 1) + A2(dtVx, tx, ty, nx - 1) * A2(dVxdt, tx, ty, nx - 1);
    if (tx < nx - 2 && ty < ny - 1)
        A2(Vy, tx + 1, ty + 1, nx) = A2(Vy, tx + 1, ty + 1, nx) + A2(dtVy, tx, ty, nx - 2) * A2(dVydt, tx, ty, nx - 2);
}

template <typename T>
__global__ void s2_bc_x_k(T* A, int64_t n0, int64_t n1) {
    int64_t iy = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (iy >= n1) return;
    A2(A, 0, iy, n0) = A2(A, 1, iy, n0);
    A2(A, n0 - 1, iy, n0) = A2(A, n0 - 2, iy, n0);
}
template <typename T>
__global__ void s2_bc_y_k(T* A, int64_t n0, int64_t n1) {
    int64_t ix = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (ix >= n0) return;
    A2(A, ix, 0, n0) = A2(A, ix, 1, n0);
    A2(A, ix, n1 - 1, n0) = A2(A, ix, n1 - 2, n0);
}

// =======================================================================================
// Fused PT iteration
// =======================================================================================
template <typename T>
struct S2Fused {
    // the state and the pseudo-velocities, in place
    T* Vx;
    T* Vy;
    T* P;
    T* dVxdt;
    T* dVydt;
    const T* Mus;
    const T* Rog;  // PLAIN: buoyancy (nx, ny); DEFECT: unused
    const T* dtVx;
    const T* dtVy;
    const T* dtPt;
    // DEFECT sources (the FP64 residual of the outer state, rounded to T)
    const T* fp;  // (nx, ny)
    const T* fx;  // (nx-1, ny-2)
    const T* fy;  // (nx-2, ny-1)
    T* txx;
    T* tyy;
    T* txy;
    // temporaries of the reference (written only if STORE_TMP)
    T* divV;
    T* Rx;
    T* Ry;
    double* red;  // Σ|Rx|, Σ|Ry|, Σ|∇V| (NULL: no reduction)
    int64_t nx, ny;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One PT iteration as two kernels in place, one thread per position: s2_cells (∇V, P and the stresses) and
// s2_faces (residuals, pseudo-velocities, velocities and the free-slip copies; a face reads no other
// face's velocity). Nothing is computed twice, every load of a thread is issued before its first store,
// and the constant arrays' loads go out while the kernel before still runs.
//
// Bound: FP64 pipe (FP64: 57 FP64 instructions per cell, 80 % busy), L2 and launches (FP32: 24 words per
// cell). Per iteration, against one kernel on shared-memory tiles that computed a halo twice and tested
// every dividend: FP64 511^2 82 -> 32.8 us, 1023^2 270 -> 118 us; FP32 1023^2 37.8 -> 14.4 us, 511^2 5.7 us,
// 63^2 3.3 us. A march along y with rows in registers and shuffles (one kernel, 15 words per cell) was
// measured at 16.6, 7.8 and 3.5 us in FP32 and 150 us in FP64 at 1023^2: its few long warps wait on loads
// and, in FP64, leave the pipe idle.
//
// RED: a.red is set (the FP64 sums are compiled in only then: the conversions to double run on the FP64
// pipe even when predicated off). I: index type (int where every array has fewer than 2^31 elements).
//
// S2_DIV evaluates a statement without testing each dividend, and again with the tests (and the IEEE
// division where they fail) in the rare case that one of its dividends is too small. PAIR: both divisors have a
// reciprocal pair; without one every dividend is tested from the start (see DivC).
#define S2_DIV(stmt)                                                            \
    do {                                                                        \
        if constexpr (PAIR) {                                                   \
            uint32_t key_ = 0xFFFFFFFFu;                                        \
            stmt(DivF<T>{p.dx, &key_}, DivF<T>{p.dy, &key_});                   \
            if (key_ < p.lo) stmt(p.dx, p.dy);                                  \
        } else {                                                                \
            stmt(DivG<T>{p.dx}, DivG<T>{p.dy});                                 \
        }                                                                       \
    } while (0)

// (a + b) * 0.5, the buoyancy average
template <typename T, typename H>
__device__ __forceinline__ T s2_half_sum(T a, T b, H) {
    return (a + b) * T(0.5);
}
__device__ __forceinline__ double s2_half_sum(double a, double b, DivF<double> h) { return scale_pow2(a + b, -1, h.key); }

// Rows of 32 threads per block. FP32: 8; FP64, bound by the FP64 pipe: 2, which spreads a small grid more
// evenly over the SMs (4 rows -> 2: 255^2 11.4 -> 10.5 us per iteration, 130^2 6.9 -> 6.1, 1023^2 118 both).
// The 64-bit variants, which run grids taller than 65535 such blocks too, have 8 (FP32) and 16 rows: with s2_max_rows
// their faces are 65535 blocks.
template <typename T, typename I>
__host__ __device__ constexpr int s2_block_rows() {
    return sizeof(I) == 8 && sizeof(T) == 8 ? 16 : sizeof(I) == 8 || sizeof(T) == 4 ? 8 : 2;
}
template <typename T>
constexpr int64_t s2_max_rows() {
    return kGridY * s2_block_rows<T, int64_t>() - 1;
}

template <typename T, bool DEFECT, typename I, bool STORE_TMP, bool RED, bool PAIR>
__global__ void __launch_bounds__(32 * s2_block_rows<T, I>()) s2_cells(S2Fused<T> a, S2P<T> p) {
    const I nx = (I)a.nx, ny = (I)a.ny;
    const I i = (I)(blockIdx.x * 32 + threadIdx.x), j = (I)(blockIdx.y * s2_block_rows<T, I>() + threadIdx.y);
    const I c = i + nx * j, cx = c + j;  // Vx rows have nx + 1 faces
    const bool cell = i < nx && j < ny, corner = i < nx - 1 && j < ny - 1;
    // what no iteration writes, while the kernel before this one still runs
    T m00 = T(0), m10 = T(0), m01 = T(0), m11 = T(0), dtp = T(0);
    [[maybe_unused]] T f = T(0);
    if (cell) {
        m00 = __ldg(a.Mus + c);
        dtp = __ldg(a.dtPt + c);
        if constexpr (DEFECT) f = __ldg(a.fp + c);
    }
    if (corner) {
        m10 = __ldg(a.Mus + c + 1);
        m01 = __ldg(a.Mus + c + nx);
        m11 = __ldg(a.Mus + c + nx + 1);
    }
    grid_dependency_wait();  // the state is read with plain loads: __ldg need not see the kernel before
    T vx0 = T(0), vx1 = T(0), vy0 = T(0), vy1 = T(0), pt = T(0), vxu = T(0), vyr = T(0);
    if (cell) {
        vx0 = a.Vx[cx];
        vx1 = a.Vx[cx + 1];
        vy0 = a.Vy[c];
        vy1 = a.Vy[c + nx];
        pt = a.P[c];
    }
    if (corner) {
        vxu = a.Vx[cx + nx + 2];
        vyr = a.Vy[c + nx + 1];
    }
    double acc = 0.0;
    T d, txx, tyy, txy;
    auto stresses = [&](auto hx, auto hy) {
        d = s2_divV(vx0, vx1, vy0, vy1, hx, hy);
        txx = s2_tau_nn(m00, vx0, vx1, d, hx);
        tyy = s2_tau_nn(m00, vy0, vy1, d, hy);
        txy = s2_tau_xy_sum(((m00 + m10) + m01) + m11, vxu - vx1, vyr - vy1, hx, hy);
    };
    S2_DIV(stresses);
    if (cell) {
        T dp = d;
        if constexpr (DEFECT) dp = d + f;
        a.P[c] = pt - dtp * dp;
        a.txx[c] = txx;
        a.tyy[c] = tyy;
        if constexpr (STORE_TMP) a.divV[c] = d;
        if constexpr (RED) acc = fabs((double)dp);
    }
    if (corner) a.txy[c - j] = txy;
    if constexpr (RED) {
        acc = warp_sum(acc);
        if (threadIdx.x == 0) atomicAdd(a.red + 2, acc);
    }
}

template <typename T, bool DEFECT, typename I, bool STORE_TMP, bool RED, bool PAIR>
__global__ void __launch_bounds__(32 * s2_block_rows<T, I>()) s2_faces(S2Fused<T> a, S2P<T> p) {
    const I nx = (I)a.nx, ny = (I)a.ny;
    const I i = (I)(blockIdx.x * 32 + threadIdx.x), j = (I)(blockIdx.y * s2_block_rows<T, I>() + threadIdx.y);
    const I c = i + nx * j, cx = c + j;  // cell and Vy face (i, j), Vx face (i, j)
    const I kx = (i - 1) + (nx - 1) * (j - 1), ky = (i - 1) + (nx - 2) * (j - 1);  // residuals; kx: corner (i-1, j-1) too
    const bool colx = i <= nx && j >= 1 && j <= ny - 2, fx = colx && i >= 1 && i <= nx - 1;  // Vx faces, with a residual
    const bool coly = i >= 1 && i <= nx - 2 && j <= ny, fy = coly && j >= 1 && j <= ny - 1;
    // what no iteration writes, while the kernel before this one still runs
    T xt = T(0), yt = T(0), g0 = T(0), g1 = T(0);
    [[maybe_unused]] T xf = T(0);
    if (fx) {
        xt = __ldg(a.dtVx + kx);
        if constexpr (DEFECT) xf = __ldg(a.fx + kx);
    }
    if (fy) {
        yt = __ldg(a.dtVy + ky);
        if constexpr (DEFECT) {
            g0 = __ldg(a.fy + ky);
        } else {
            g0 = __ldg(a.Rog + c - nx);
            g1 = __ldg(a.Rog + c);
        }
    }
    grid_dependency_wait();
    T xr = T(0), xl = T(0), s00 = T(0), s01 = T(0), s10 = T(0), p0 = T(0), pl = T(0), pd = T(0), yu = T(0), yd = T(0);
    T xg = T(0), yg = T(0), vx = T(0), vy = T(0);
    if (fx || fy) {
        s00 = a.txy[kx];
        p0 = a.P[c];
    }
    if (fx) {
        xr = a.txx[c];
        xl = a.txx[c - 1];
        s01 = a.txy[kx + (nx - 1)];
        pl = a.P[c - 1];
        xg = a.dVxdt[kx];
    }
    if (fy) {
        yu = a.tyy[c];
        yd = a.tyy[c - nx];
        s10 = a.txy[kx + 1];
        pd = a.P[c - nx];
        yg = a.dVydt[ky];
    }
    if (colx) vx = a.Vx[cx];
    if (coly) vy = a.Vy[c];
    double acc_x = 0.0, acc_y = 0.0;
    T rx, ry;
    auto resid = [&](auto hx, auto hy) {
        rx = s2_Rx(xl, xr, s00, s01, pl, p0, hx, hy);
        ry = s2_Ry_core(yd, yu, s00, s10, pd, p0, hx, hy);
        if constexpr (!DEFECT) ry = ry + s2_half_sum(g0, g1, hx);
    };
    S2_DIV(resid);
    if constexpr (DEFECT) {
        rx = rx + xf;
        ry = ry + g0;
    }
    // Vx face (i, j); bc_y!(Vx): rows 0 and ny-1 copy rows 1 and ny-2
    if (fx) {
        const T dv = p.dampX * xg + rx;
        a.dVxdt[kx] = dv;
        if constexpr (STORE_TMP) a.Rx[kx] = rx;
        if constexpr (RED) acc_x = fabs((double)rx);
        vx = vx + xt * dv;
        a.Vx[cx] = vx;
    }
    if (colx && j == 1) a.Vx[i] = vx;
    if (colx && j == ny - 2) a.Vx[cx + nx + 1] = vx;
    // Vy face (i, j); bc_x!(Vy): columns 0 and nx-1 copy columns 1 and nx-2
    if (fy) {
        const T dv = p.dampY * yg + ry;
        a.dVydt[ky] = dv;
        if constexpr (STORE_TMP) a.Ry[ky] = ry;
        if constexpr (RED) acc_y = fabs((double)ry);
        vy = vy + yt * dv;
        a.Vy[c] = vy;
    }
    if (coly && i == 1) a.Vy[c - 1] = vy;
    if (coly && i == nx - 2) a.Vy[c + 1] = vy;
    if constexpr (RED) {
        acc_x = warp_sum(acc_x);
        acc_y = warp_sum(acc_y);
        if (threadIdx.x == 0) {
            atomicAdd(a.red, acc_x);
            atomicAdd(a.red + 1, acc_y);
        }
    }
}

// =======================================================================================
// FP64 residual of the outer state (defect correction): no pseudo-time update.
// Outputs fp = ∇V, fx = Rx, fy = Ry rounded to float, and Σ|.| in FP64.
// =======================================================================================
__global__ void s2_residual64(const double* __restrict__ Vx, const double* __restrict__ Vy,
                              const double* __restrict__ P, const double* __restrict__ Mus,
                              const double* __restrict__ Rog, float* fp, float* fx, float* fy, double* red, int64_t nx,
                              int64_t ny, S2P<double> p) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, j = blockIdx.y * (int64_t)blockDim.y + threadIdx.y;
    auto div_at = [&](int64_t ci, int64_t cj) {
        return s2_divV(A2(Vx, ci, cj, nx + 1), A2(Vx, ci + 1, cj, nx + 1), A2(Vy, ci, cj, nx), A2(Vy, ci, cj + 1, nx), p.dx,
                       p.dy);
    };
    auto txx_at = [&](int64_t ci, int64_t cj) {
        return s2_tau_nn(A2(Mus, ci, cj, nx), A2(Vx, ci, cj, nx + 1), A2(Vx, ci + 1, cj, nx + 1), div_at(ci, cj), p.dx);
    };
    auto tyy_at = [&](int64_t ci, int64_t cj) {
        return s2_tau_nn(A2(Mus, ci, cj, nx), A2(Vy, ci, cj, nx), A2(Vy, ci, cj + 1, nx), div_at(ci, cj), p.dy);
    };
    auto txy_at = [&](int64_t a_, int64_t b_) {
        return s2_tau_xy(A2(Mus, a_, b_, nx), A2(Mus, a_ + 1, b_, nx), A2(Mus, a_, b_ + 1, nx), A2(Mus, a_ + 1, b_ + 1, nx),
                         A2(Vx, a_ + 1, b_ + 1, nx + 1) - A2(Vx, a_ + 1, b_, nx + 1),
                         A2(Vy, a_ + 1, b_ + 1, nx) - A2(Vy, a_, b_ + 1, nx), p.dx, p.dy);
    };
    double ax = 0, ay = 0, ad = 0;
    if (i < nx && j < ny) {
        double d = div_at(i, j);
        fp[i + nx * j] = (float)d;
        ad = fabs(d);
    }
    if (i >= 1 && i <= nx - 1 && j >= 1 && j <= ny - 2) {
        double r = s2_Rx(txx_at(i - 1, j), txx_at(i, j), txy_at(i - 1, j - 1), txy_at(i - 1, j), A2(P, i - 1, j, nx),
                         A2(P, i, j, nx), p.dx, p.dy);
        fx[(i - 1) + (nx - 1) * (j - 1)] = (float)r;
        ax = fabs(r);
    }
    if (i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 1) {
        double r = s2_Ry_core(tyy_at(i, j - 1), tyy_at(i, j), txy_at(i - 1, j - 1), txy_at(i, j - 1), A2(P, i, j - 1, nx),
                              A2(P, i, j, nx), p.dx, p.dy) +
                   (A2(Rog, i, j - 1, nx) + A2(Rog, i, j, nx)) * 0.5;
        fy[(i - 1) + (nx - 2) * (j - 1)] = (float)r;
        ay = fabs(r);
    }
    __shared__ double sred[3][8];
    double s0 = warp_sum(ax), s1 = warp_sum(ay), s2 = warp_sum(ad);
    int tid = threadIdx.y * blockDim.x + threadIdx.x, w = tid >> 5;
    if ((tid & 31) == 0) {
        sred[0][w] = s0;
        sred[1][w] = s1;
        sred[2][w] = s2;
    }
    __syncthreads();
    if (tid < 3) {
        double s = 0;
        for (int k = 0; k < (int)(blockDim.x * blockDim.y) / 32; k++) s += sred[tid][k];
        atomicAdd(red + tid, s);
    }
}

// x64 += (double) d32 over n elements
__global__ void s2_axpy32(double* x, const float* d, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] += (double)d[i];
}

__global__ void s2_to_f32(float* y, const double* x, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = (float)x[i];
}

// =======================================================================================
// Host side
// =======================================================================================
static int check2(const ps_array& a, int64_t n0, int64_t n1, int32_t dt, const char* name) {
    PS_TRY(check_array(a, name));
    if (a.dtype != dt) return fail(PS_ERR_DTYPE, "Stokes2D: array %s has a different dtype", name);
    return check_shape(a, n0, n1, 1, name);
}

static int check_fields(const ps_stokes2d_fields* f, int64_t* nx, int64_t* ny, bool need_dt) {
    if (!f) return fail(PS_ERR_NULL, "Stokes2D: NULL fields");
    PS_TRY(check_array(f->Pt, "Pt"));
    int64_t X = f->Pt.n[0], Y = f->Pt.n[1];
    int32_t dt = f->Pt.dtype;
    if (X < 3 || Y < 3 || f->Pt.n[2] != 1) return fail(PS_ERR_SHAPE, "Stokes2D: Pt must be 2-D with nx, ny >= 3");
    PS_TRY(check2(f->Vx, X + 1, Y, dt, "Vx"));
    PS_TRY(check2(f->Vy, X, Y + 1, dt, "Vy"));
    PS_TRY(check2(f->divV, X, Y, dt, "∇V"));
    PS_TRY(check2(f->txx, X, Y, dt, "τxx"));
    PS_TRY(check2(f->tyy, X, Y, dt, "τyy"));
    PS_TRY(check2(f->txy, X - 1, Y - 1, dt, "τxy"));
    PS_TRY(check2(f->Rx, X - 1, Y - 2, dt, "Rx"));
    PS_TRY(check2(f->Ry, X - 2, Y - 1, dt, "Ry"));
    PS_TRY(check2(f->dVxdtau, X - 1, Y - 2, dt, "dVxdτ"));
    PS_TRY(check2(f->dVydtau, X - 2, Y - 1, dt, "dVydτ"));
    PS_TRY(check2(f->Mus, X, Y, dt, "Mus"));
    PS_TRY(check2(f->Rog, X, Y, dt, "Rog"));
    if (need_dt) {
        PS_TRY(check2(f->dtauPt, X, Y, dt, "dτPt"));
        PS_TRY(check2(f->dtauVx, X - 1, Y - 2, dt, "dτVx"));
        PS_TRY(check2(f->dtauVy, X - 2, Y - 1, dt, "dτVy"));
    }
    *nx = X;
    *ny = Y;
    return PS_OK;
}

template <typename T>
static T* P_(const ps_array& a) {
    return static_cast<T*>(a.ptr);
}

static dim3 g2(int64_t wx, int64_t wy, dim3 b) {
    return dim3((unsigned)((wx + b.x - 1) / b.x), (unsigned)((wy + b.y - 1) / b.y), 1);
}

// Library-owned scratch of the solvers (freed by ps_finalize).
static std::mutex g_scr_mutex;
static std::vector<void*> g_scratch_all;

static int scratch_alloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(PS_ERR_NOMEM, "Stokes2D scratch allocation of %zu bytes failed", bytes);
    }
    std::lock_guard<std::mutex> l(g_scr_mutex);
    g_scratch_all.push_back(*p);
    return PS_OK;
}
static void scratch_free(void* p) {
    if (!p) return;
    cudaFree(p);
    std::lock_guard<std::mutex> l(g_scr_mutex);
    g_scratch_all.erase(std::remove(g_scratch_all.begin(), g_scratch_all.end(), p), g_scratch_all.end());
}

// 32-bit indices while every array's size and the offsets a few rows past it stay below 2^31
static bool s2_index32(int64_t nx, int64_t ny) { return (nx + 32) * (ny + 4) < ((int64_t)1 << 31); }

// Refused before the first launch, so that no iteration stops halfway.
template <typename T>
static int check_rows(int64_t ny, const char* what) {
    if (ny > s2_max_rows<T>())
        return fail(PS_ERR_SHAPE, "%s: %lld rows, at most %lld", what, (long long)ny, (long long)s2_max_rows<T>());
    return PS_OK;
}

// One iteration. dependent: the kernel before it on the stream is the previous iteration's.
template <typename T, bool DEFECT, bool STORE_TMP>
static void launch_cells_faces(const S2Fused<T>& a, const S2P<T>& p, cudaStream_t s, bool dependent) {
    const bool i32 = s2_index32(a.nx, a.ny) && a.ny / s2_block_rows<T, int>() < kGridY;
    const dim3 blk(32, i32 ? s2_block_rows<T, int>() : s2_block_rows<T, int64_t>()), gc = g2(a.nx, a.ny, blk),
               gf = g2(a.nx + 1, a.ny + 1, blk);
    auto launch = [&](auto cells, auto faces) {
        if (dependent) launch_dependent(cells, gc, blk, 0, s, a, p);
        else cells<<<gc, blk, 0, s>>>(a, p);
        launch_dependent(faces, gf, blk, 0, s, a, p);
    };
    auto with = [&](auto index, auto red, auto pair) {
        using I = decltype(index);
        constexpr bool RED = decltype(red)::value, PAIR = decltype(pair)::value;
        launch(s2_cells<T, DEFECT, I, STORE_TMP, RED, PAIR>, s2_faces<T, DEFECT, I, STORE_TMP, RED, PAIR>);
    };
    auto pairs = [&](auto index, auto red) {
        if (p.lo != kNoPair) with(index, red, std::true_type{});
        else with(index, red, std::false_type{});
    };
    auto sums = [&](auto index) {
        if (a.red) pairs(index, std::true_type{});
        else pairs(index, std::false_type{});
    };
    if (i32) sums(int{});
    else sums(int64_t{});
}

template <typename T>
static S2Fused<T> s2_dropin_args(const ps_stokes2d_fields* f) {
    S2Fused<T> a{};
    a.Vx = P_<T>(f->Vx);
    a.Vy = P_<T>(f->Vy);
    a.P = P_<T>(f->Pt);
    a.Mus = P_<T>(f->Mus);
    a.Rog = P_<T>(f->Rog);
    a.dtVx = P_<T>(f->dtauVx);
    a.dtVy = P_<T>(f->dtauVy);
    a.dtPt = P_<T>(f->dtauPt);
    a.dVxdt = P_<T>(f->dVxdtau);
    a.dVydt = P_<T>(f->dVydtau);
    a.divV = P_<T>(f->divV);
    a.txx = P_<T>(f->txx);
    a.tyy = P_<T>(f->tyy);
    a.txy = P_<T>(f->txy);
    a.Rx = P_<T>(f->Rx);
    a.Ry = P_<T>(f->Ry);
    a.nx = f->Pt.n[0];
    a.ny = f->Pt.n[1];
    return a;
}

// n_iter iterations; the temporaries nothing reads between iterations are stored in the last
template <typename T>
static int s2_iterate(const ps_stokes2d_fields* f, const ps_stokes2d_params* pp, int64_t n_iter, cudaStream_t s,
                      const char* what) {
    PS_TRY(check_rows<T>(f->Pt.n[1], what));
    const S2P<T> p = s2p<T>(*pp);
    const S2Fused<T> a = s2_dropin_args<T>(f);
    for (int64_t it = 0; it + 1 < n_iter; ++it) launch_cells_faces<T, false, false>(a, p, s, it > 0);
    if (n_iter > 0) launch_cells_faces<T, false, true>(a, p, s, n_iter > 1);
    return finish_launch(s, 1, what);
}

// ---- solver ---------------------------------------------------------------------------
// Runs `nout` iterations per CUDA graph launch; the last one of each graph accumulates Σ|Rx|, Σ|Ry|,
// Σ|∇V| into `red`.
struct PTRunner {
    cudaGraphExec_t exec = nullptr;
    cudaGraph_t graph = nullptr;

    // iteration(it, red): enqueues iteration `it` (red: null except in the last)
    template <typename F>
    int build(cudaStream_t s, int64_t nout, double* red, F iteration) {
        PS_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        cudaMemsetAsync(red, 0, 3 * sizeof(double), s);
        for (int64_t it = 0; it < nout; ++it) iteration(it, it == nout - 1 ? red : nullptr);
        PS_CUDA_TRY(cudaStreamEndCapture(s, &graph));
        PS_CUDA_TRY(cudaGraphInstantiate(&exec, graph, 0));
        return PS_OK;
    }
    void destroy() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
    }
};

// The pseudo-time steps of a solve, computed once (compute_timesteps!) instead of in every iteration.
template <typename T>
static void s2_solver_timesteps(S2Fused<T>& a, const S2P<T>& p, T* dtVx, T* dtVy, T* dtPt, cudaStream_t s) {
    const dim3 blk(32, s2_block_rows<T, int64_t>());
    s2_timesteps_k<T><<<g2(a.nx, a.ny, blk), blk, 0, s>>>(dtVx, dtVy, dtPt, a.Mus, a.nx, a.ny, p);
    a.dtVx = dtVx;
    a.dtVy = dtVy;
    a.dtPt = dtPt;
}

static double now_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

static int solve_fp64(const ps_stokes2d_fields* f, const ps_stokes2d_params* pp, double tol, int64_t max_iter,
                      int64_t nout, double max_seconds, ps_solve_stats* st, cudaStream_t s) {
    int64_t nx = f->Pt.n[0], ny = f->Pt.n[1];
    const int64_t nRx = (nx - 1) * (ny - 2), nRy = (nx - 2) * (ny - 1), nP = nx * ny;
    void* buf = nullptr;
    // τxx, τyy, τxy, dτVx, dτVy, dτPt and the three sums
    PS_TRY(scratch_alloc(&buf, (3 * nP + (nx - 1) * (ny - 1) + nRx + nRy + 3) * sizeof(double) + 256));
    double* c = static_cast<double*>(buf);
    S2Fused<double> a = s2_dropin_args<double>(f);
    const S2P<double> p = s2p<double>(*pp);
    a.txx = c;
    a.tyy = c + nP;
    a.txy = c + 2 * nP;
    double* dt = a.txy + (nx - 1) * (ny - 1);
    s2_solver_timesteps(a, p, dt, dt + nRx, dt + nRx + nRy, s);
    double* red = dt + nRx + nRy + nP;
    PTRunner r;
    int rc = r.build(s, nout, red, [&](int64_t it, double* rd) {
        S2Fused<double> k = a;
        k.red = rd;
        launch_cells_faces<double, false, false>(k, p, s, it > 0);
    });
    const double nrx = (double)((nx - 1) * (ny - 2)), nry = (double)((nx - 2) * (ny - 1)), nd = (double)(nx * ny);
    double t0 = now_s(), err = INFINITY, h[3];
    int64_t it = 0;
    while (rc == PS_OK && it < max_iter) {
        cudaError_t e = cudaGraphLaunch(r.exec, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(h, red, sizeof(h), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            rc = cuda_fail(e, "ps_stokes2d_solve(fp64)");
            break;
        }
        it += nout;
        err = std::max(std::max(h[0] / nrx, h[1] / nry), h[2] / nd);
        if (!std::isfinite(h[0]) || !std::isfinite(h[1]) || !std::isfinite(h[2])) {  // std::max drops a NaN
            err = NAN;
            rc = fail(PS_ERR_NONFINITE, "ps_stokes2d_solve: non-finite residual after %lld iterations", (long long)it);
            break;
        }
        if (err < tol) break;
        if (max_seconds > 0 && now_s() - t0 > max_seconds) {
            rc = fail(PS_ERR_TIMEOUT, "ps_stokes2d_solve: wall-clock limit reached (err %.3e)", err);
            break;
        }
    }
    r.destroy();
    cudaStreamSynchronize(s);
    scratch_free(buf);
    st->iters = it;
    st->outer = 1;
    st->err = err;
    st->seconds = now_s() - t0;
    st->converged = err < tol;
    if (rc == PS_OK && !(err < tol))
        rc = fail(PS_ERR_NOT_CONVERGED, "ps_stokes2d_solve: err %.3e after %lld iterations", err, (long long)it);
    return rc;
}

// Mixed precision: FP32 PT sweeps on the correction (δP, δV) with the FP64 residual of the
// outer state as source; FP64 residual, update and convergence check.
static int solve_mixed(const ps_stokes2d_fields* f, const ps_stokes2d_params* pp, double tol, int64_t max_iter,
                       int64_t nout, double max_seconds, double inner_rtol, ps_solve_stats* st, cudaStream_t s) {
    int64_t nx = f->Pt.n[0], ny = f->Pt.n[1];
    const int64_t nVx = (nx + 1) * ny, nVy = nx * (ny + 1), nP = nx * ny, nRx = (nx - 1) * (ny - 2),
                  nRy = (nx - 2) * (ny - 1);
    // float buffers: δVx, δVy, δP, dVxdτ, dVydτ, fx, fy, fp, Mus32, dτVx, dτVy, dτPt, τxx, τyy, τxy
    const int64_t counts[15] = {nVx, nVy, nP, nRx, nRy, nRx, nRy, nP, nP, nRx, nRy, nP, nP, nP, (nx - 1) * (ny - 1)};
    size_t off[16];
    off[0] = 0;
    for (int k = 0; k < 15; k++) off[k + 1] = off[k] + ((counts[k] * 4 + 255) / 256) * 256;
    size_t total = off[15] + 2 * 3 * sizeof(double) + 256;
    void* buf = nullptr;
    PS_TRY(scratch_alloc(&buf, total));
    char* c = static_cast<char*>(buf);
    auto F = [&](int k) { return reinterpret_cast<float*>(c + off[k]); };
    double* red_in = reinterpret_cast<double*>(c + off[15]);
    double* red_out = red_in + 3;
    int rc = PS_OK;
    cudaError_t e = cudaMemsetAsync(buf, 0, off[15], s);
    if (e != cudaSuccess) rc = cuda_fail(e, "memset");
    const double* Mus = P_<double>(f->Mus);
    s2_to_f32<<<256, 256, 0, s>>>(F(8), Mus, nP);
    // The corrections keep the free-slip copies (bc_y!(Vx), bc_x!(Vy)) of the state they are added
    // to, so a start state that violates them (an externally supplied guess) would keep its
    // violation: apply the copies once, as the first FP64 PT iteration would.
    s2_bc_y_k<double><<<(unsigned)((nx + 1 + 255) / 256), 256, 0, s>>>(P_<double>(f->Vx), nx + 1, ny);
    s2_bc_x_k<double><<<(unsigned)((ny + 1 + 255) / 256), 256, 0, s>>>(P_<double>(f->Vy), nx, ny + 1);

    S2Fused<float> a{};
    const S2P<float> p32 = s2p<float>(*pp);
    a.Vx = F(0);
    a.Vy = F(1);
    a.P = F(2);
    a.dVxdt = F(3);
    a.dVydt = F(4);
    a.fx = F(5);
    a.fy = F(6);
    a.fp = F(7);
    a.Mus = F(8);
    a.txx = F(12);
    a.tyy = F(13);
    a.txy = F(14);
    a.nx = nx;
    a.ny = ny;
    s2_solver_timesteps(a, p32, F(9), F(10), F(11), s);
    PTRunner r;
    if (rc == PS_OK)
        rc = r.build(s, nout, red_in, [&](int64_t it, double* rd) {
            S2Fused<float> k = a;
            k.red = rd;
            launch_cells_faces<float, true, false>(k, p32, s, it > 0);
        });

    S2P<double> p64 = s2p<double>(*pp);
    const double nrx = (double)nRx, nry = (double)nRy, nd = (double)nP;
    double t0 = now_s(), err = INFINITY, h[3];
    int64_t it = 0, outer = 0;
    dim3 blk(32, 8);
    dim3 grd = g2(nx + 1, ny + 1, blk);
    while (rc == PS_OK) {
        // FP64 residual of the outer state -> fx, fy, fp (float) and err
        cudaMemsetAsync(red_out, 0, 3 * sizeof(double), s);
        s2_residual64<<<grd, blk, 0, s>>>(P_<double>(f->Vx), P_<double>(f->Vy), P_<double>(f->Pt), Mus,
                                          P_<double>(f->Rog), F(7), F(5), F(6), red_out, nx, ny, p64);
        e = cudaMemcpyAsync(h, red_out, sizeof(h), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            rc = cuda_fail(e, "ps_stokes2d_solve(mixed residual)");
            break;
        }
        err = std::max(std::max(h[0] / nrx, h[1] / nry), h[2] / nd);
        if (!std::isfinite(h[0]) || !std::isfinite(h[1]) || !std::isfinite(h[2])) {
            err = NAN;
            rc = fail(PS_ERR_NONFINITE, "ps_stokes2d_solve: non-finite FP64 residual");
            break;
        }
        if (err < tol || it >= max_iter) break;
        if (max_seconds > 0 && now_s() - t0 > max_seconds) {
            rc = fail(PS_ERR_TIMEOUT, "ps_stokes2d_solve: wall-clock limit reached (err %.3e)", err);
            break;
        }
        ++outer;
        // inner FP32 PT on the correction, from zero
        cudaMemsetAsync(c, 0, off[5], s);  // δV, δP, dVxdτ, dVydτ
        double target = std::max(err * inner_rtol, tol * 0.25);
        double ierr = INFINITY;
        while (it < max_iter) {
            e = cudaGraphLaunch(r.exec, s);
            if (e == cudaSuccess) e = cudaMemcpyAsync(h, red_in, sizeof(h), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) {
                rc = cuda_fail(e, "ps_stokes2d_solve(mixed inner)");
                break;
            }
            it += nout;
            double prev = ierr;
            ierr = std::max(std::max(h[0] / nrx, h[1] / nry), h[2] / nd);
            if (!std::isfinite(h[0]) || !std::isfinite(h[1]) || !std::isfinite(h[2])) {
                rc = fail(PS_ERR_NONFINITE, "ps_stokes2d_solve: non-finite FP32 residual");
                break;
            }
            if (ierr < target) break;
            // FP32 floor: stop the sweep once it no longer reduces the residual
            if (ierr > 0.98 * prev && ierr < err * 0.5) break;
        }
        if (rc != PS_OK) break;
        // FP64 update of the outer state with the FP32 correction
        s2_axpy32<<<256, 256, 0, s>>>(P_<double>(f->Vx), F(0), nVx);
        s2_axpy32<<<256, 256, 0, s>>>(P_<double>(f->Vy), F(1), nVy);
        s2_axpy32<<<256, 256, 0, s>>>(P_<double>(f->Pt), F(2), nP);
    }
    r.destroy();
    cudaStreamSynchronize(s);
    scratch_free(buf);
    st->iters = it;
    st->outer = outer;
    st->err = err;
    st->seconds = now_s() - t0;
    st->converged = err < tol;
    if (rc == PS_OK && !(err < tol))
        rc = fail(PS_ERR_NOT_CONVERGED, "ps_stokes2d_solve(mixed): err %.3e after %lld iterations", err, (long long)it);
    return rc;
}

// Σ|a| (FP64 accumulation) -- used by ps_stokes2d_err.
__global__ void ps_sum_abs_f64(const double* a, int64_t n, double* out) {
    double s = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s += fabs(a[i]);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}
__global__ void ps_sum_abs_f32(const float* a, int64_t n, double* out) {
    double s = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s += fabs((double)a[i]);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

void stokes2d_free_scratch() {
    std::lock_guard<std::mutex> l(g_scr_mutex);
    for (void* p : g_scratch_all) cudaFree(p);
    g_scratch_all.clear();
}

}  // namespace ps

using namespace ps;

extern "C" {

int ps_stokes2d_timesteps(const ps_stokes2d_fields* f, const ps_stokes2d_params* p, void* stream, int sync) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, true));
    if (!p) return fail(PS_ERR_NULL, "NULL params");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dim3 blk(32, 8), grd = g2(nx, ny, blk);
    if (f->Pt.dtype == PS_F64)
        s2_timesteps_k<double><<<grd, blk, 0, s>>>(P_<double>(f->dtauVx), P_<double>(f->dtauVy), P_<double>(f->dtauPt),
                                                   P_<double>(f->Mus), nx, ny, s2p<double>(*p));
    else
        s2_timesteps_k<float><<<grd, blk, 0, s>>>(P_<float>(f->dtauVx), P_<float>(f->dtauVy), P_<float>(f->dtauPt),
                                                  P_<float>(f->Mus), nx, ny, s2p<float>(*p));
    return finish_launch(s, sync, "ps_stokes2d_timesteps");
}

int ps_stokes2d_compute_P(const ps_stokes2d_fields* f, const ps_stokes2d_params* p, void* stream, int sync) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, true));
    if (!p) return fail(PS_ERR_NULL, "NULL params");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dim3 blk(32, 8), grd = g2(nx, ny, blk);
    if (f->Pt.dtype == PS_F64)
        s2_P_k<double><<<grd, blk, 0, s>>>(P_<double>(f->divV), P_<double>(f->Pt), P_<double>(f->Vx), P_<double>(f->Vy),
                                           P_<double>(f->dtauPt), nx, ny, s2p<double>(*p));
    else
        s2_P_k<float><<<grd, blk, 0, s>>>(P_<float>(f->divV), P_<float>(f->Pt), P_<float>(f->Vx), P_<float>(f->Vy),
                                          P_<float>(f->dtauPt), nx, ny, s2p<float>(*p));
    return finish_launch(s, sync, "ps_stokes2d_compute_P");
}

int ps_stokes2d_compute_tau(const ps_stokes2d_fields* f, const ps_stokes2d_params* p, void* stream, int sync) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, true));
    if (!p) return fail(PS_ERR_NULL, "NULL params");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dim3 blk(32, 8), grd = g2(nx, ny, blk);
    if (f->Pt.dtype == PS_F64)
        s2_tau_k<double><<<grd, blk, 0, s>>>(P_<double>(f->divV), P_<double>(f->txx), P_<double>(f->tyy),
                                             P_<double>(f->txy), P_<double>(f->Vx), P_<double>(f->Vy),
                                             P_<double>(f->Mus), nx, ny, s2p<double>(*p));
    else
        s2_tau_k<float><<<grd, blk, 0, s>>>(P_<float>(f->divV), P_<float>(f->txx), P_<float>(f->tyy), P_<float>(f->txy),
                                            P_<float>(f->Vx), P_<float>(f->Vy), P_<float>(f->Mus), nx, ny,
                                            s2p<float>(*p));
    return finish_launch(s, sync, "ps_stokes2d_compute_tau");
}

int ps_stokes2d_compute_dV(const ps_stokes2d_fields* f, const ps_stokes2d_params* p, void* stream, int sync) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, true));
    if (!p) return fail(PS_ERR_NULL, "NULL params");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dim3 blk(32, 8), grd = g2(nx, ny, blk);
    if (f->Pt.dtype == PS_F64)
        s2_dV_k<double><<<grd, blk, 0, s>>>(P_<double>(f->Rx), P_<double>(f->Ry), P_<double>(f->dVxdtau),
                                            P_<double>(f->dVydtau), P_<double>(f->Pt), P_<double>(f->Rog),
                                            P_<double>(f->txx), P_<double>(f->tyy), P_<double>(f->txy), nx, ny,
                                            s2p<double>(*p));
    else
        s2_dV_k<float><<<grd, blk, 0, s>>>(P_<float>(f->Rx), P_<float>(f->Ry), P_<float>(f->dVxdtau),
                                           P_<float>(f->dVydtau), P_<float>(f->Pt), P_<float>(f->Rog), P_<float>(f->txx),
                                           P_<float>(f->tyy), P_<float>(f->txy), nx, ny, s2p<float>(*p));
    return finish_launch(s, sync, "ps_stokes2d_compute_dV");
}

int ps_stokes2d_compute_V(const ps_stokes2d_fields* f, const ps_stokes2d_params* p, void* stream, int sync) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, true));
    (void)p;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dim3 blk(32, 8), grd = g2(nx + 1, ny + 1, blk);
    if (f->Pt.dtype == PS_F64)
        s2_V_k<double><<<grd, blk, 0, s>>>(P_<double>(f->Vx), P_<double>(f->Vy), P_<double>(f->dVxdtau),
                                           P_<double>(f->dVydtau), P_<double>(f->dtauVx), P_<double>(f->dtauVy), nx, ny);
    else
        s2_V_k<float><<<grd, blk, 0, s>>>(P_<float>(f->Vx), P_<float>(f->Vy), P_<float>(f->dVxdtau),
                                          P_<float>(f->dVydtau), P_<float>(f->dtauVx), P_<float>(f->dtauVy), nx, ny);
    return finish_launch(s, sync, "ps_stokes2d_compute_V");
}

static int bc2(ps_array A, void* stream, int sync, bool xdir) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    PS_TRY(check_array(A, "A"));
    if (A.n[2] != 1 || A.n[0] < 2 || A.n[1] < 2) return fail(PS_ERR_SHAPE, "bc: A must be 2-D with extents >= 2");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int64_t w = xdir ? A.n[1] : A.n[0];
    unsigned g = (unsigned)((w + 255) / 256);
    if (A.dtype == PS_F64) {
        if (xdir)
            s2_bc_x_k<double><<<g, 256, 0, s>>>(P_<double>(A), A.n[0], A.n[1]);
        else
            s2_bc_y_k<double><<<g, 256, 0, s>>>(P_<double>(A), A.n[0], A.n[1]);
    } else {
        if (xdir)
            s2_bc_x_k<float><<<g, 256, 0, s>>>(P_<float>(A), A.n[0], A.n[1]);
        else
            s2_bc_y_k<float><<<g, 256, 0, s>>>(P_<float>(A), A.n[0], A.n[1]);
    }
    return finish_launch(s, sync, xdir ? "ps_bc_x2d" : "ps_bc_y2d");
}

int ps_bc_x2d(ps_array A, void* stream, int sync) { return bc2(A, stream, sync, true); }
int ps_bc_y2d(ps_array A, void* stream, int sync) { return bc2(A, stream, sync, false); }

int ps_stokes2d_iterate(const ps_stokes2d_fields* f, const ps_stokes2d_params* p, int64_t n_iter, void* stream) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, true));
    if (!p) return fail(PS_ERR_NULL, "NULL params");
    if (n_iter < 0) return fail(PS_ERR_ARG, "n_iter must be >= 0");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return f->Pt.dtype == PS_F64 ? s2_iterate<double>(f, p, n_iter, s, "ps_stokes2d_iterate")
                                 : s2_iterate<float>(f, p, n_iter, s, "ps_stokes2d_iterate");
}

int ps_stokes2d_err(const ps_stokes2d_fields* f, double out_mean_abs[3], void* stream) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, false));
    if (!out_mean_abs) return fail(PS_ERR_NULL, "NULL output");
    // mean(abs.(Rx)), mean(abs.(Ry)), mean(abs.(∇V)) (Stokes2D.jl:119) on the stored arrays
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const ps_array* arrs[3] = {&f->Rx, &f->Ry, &f->divV};
    double* red = st->d_scratch;
    PS_CUDA_TRY(cudaMemsetAsync(red, 0, 3 * sizeof(double), s));
    for (int k = 0; k < 3; k++) {
        int64_t n = numel(*arrs[k]);
        if (f->Pt.dtype == PS_F64)
            ps_sum_abs_f64<<<std::max<int64_t>(1, std::min<int64_t>((n + 1023) / 1024, 1024)), 256, 0, s>>>(
                P_<double>(*arrs[k]), n, red + k);
        else
            ps_sum_abs_f32<<<std::max<int64_t>(1, std::min<int64_t>((n + 1023) / 1024, 1024)), 256, 0, s>>>(
                P_<float>(*arrs[k]), n, red + k);
    }
    double h[3];
    PS_CUDA_TRY(cudaMemcpyAsync(h, red, sizeof(h), cudaMemcpyDeviceToHost, s));
    PS_CUDA_TRY(cudaStreamSynchronize(s));
    for (int k = 0; k < 3; k++) out_mean_abs[k] = h[k] / (double)numel(*arrs[k]);
    return finish_launch(s, 0, "ps_stokes2d_err");
}

int ps_stokes2d_solve(const ps_stokes2d_fields* f, const ps_stokes2d_params* p, int32_t mode, double tol,
                      int64_t max_iter, int64_t nout, double max_seconds, ps_solve_stats* stats, void* stream) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, false));
    if (!p || !stats) return fail(PS_ERR_NULL, "NULL params / stats");
    if (f->Pt.dtype != PS_F64) return fail(PS_ERR_DTYPE, "ps_stokes2d_solve: the state arrays must be FP64");
    if (nout < 2 || nout % 2) return fail(PS_ERR_ARG, "nout must be even and >= 2");
    if (!(tol > 0) || max_iter < 0) return fail(PS_ERR_ARG, "invalid tol / max_iter");
    if (mode != 0 && mode != 1) return fail(PS_ERR_ARG, "mode must be 0 (FP64) or 1 (FP32 + FP64 defect correction)");
    PS_TRY(mode == 0 ? check_rows<double>(ny, "ps_stokes2d_solve") : check_rows<float>(ny, "ps_stokes2d_solve (mixed)"));
    memset(stats, 0, sizeof(*stats));
    // the solver captures CUDA graphs: run on a private stream ordered after `stream`
    cudaStream_t user = static_cast<cudaStream_t>(stream), s;
    PS_CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    cudaEvent_t ev;
    PS_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    cudaEventRecord(ev, user);
    cudaStreamWaitEvent(s, ev, 0);
    int rc = mode == 0 ? solve_fp64(f, p, tol, max_iter, nout, max_seconds, stats, s)
                       : solve_mixed(f, p, tol, max_iter, nout, max_seconds, 1e-3, stats, s);
    cudaStreamSynchronize(s);
    cudaEventDestroy(ev);
    cudaStreamDestroy(s);
    cudaGetLastError();
    return rc;
}

}  // extern "C"


// =======================================================================================
// ps_stokes2d_iterate_static: the PT iteration for callers that cannot let a library allocate device
// memory: an application whose device memory is fully owned by its own pool allocator (CUDA.jl's memory
// pool, a framework caching allocator), where a cudaMalloc behind its back fails or fragments the pool,
// and code that must not call cudaFree, which synchronises the whole device. The iteration works in
// place, so neither entry point allocates; this one keeps the bound on the grid that its callers know.
// =======================================================================================
namespace ps {

constexpr size_t kStaticScratchBytes = size_t(16) << 20;

static size_t round256(size_t b) { return (b + 255) / 256 * 256; }

static int check_static_bound(const ps_stokes2d_fields* f) {
    const int64_t nx = f->Pt.n[0], ny = f->Pt.n[1];
    const size_t es = elsize(f->Pt.dtype);
    const size_t need = round256((nx + 1) * ny * es) + round256(nx * (ny + 1) * es) + round256(nx * ny * es);
    if (need > kStaticScratchBytes)
        return fail(PS_ERR_SHAPE,
                    "ps_stokes2d_iterate_static: the state of a %lld x %lld grid is %zu bytes; the static buffer "
                    "bound is %zu bytes (use ps_stokes2d_iterate)",
                    (long long)nx, (long long)ny, need, kStaticScratchBytes);
    return PS_OK;
}

}  // namespace ps

extern "C" int ps_stokes2d_iterate_static(const ps_stokes2d_fields* f, const ps_stokes2d_params* p, int64_t n_iter,
                                          void* stream) {
    DeviceState* st = nullptr;
    PS_TRY(current_state(&st));
    int64_t nx, ny;
    PS_TRY(check_fields(f, &nx, &ny, true));
    if (!p) return fail(PS_ERR_NULL, "NULL params");
    if (n_iter < 0) return fail(PS_ERR_ARG, "n_iter must be >= 0");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    PS_TRY(check_static_bound(f));
    return f->Pt.dtype == PS_F64 ? s2_iterate<double>(f, p, n_iter, s, "ps_stokes2d_iterate_static")
                                 : s2_iterate<float>(f, p, n_iter, s, "ps_stokes2d_iterate_static");
}
