// FP64 DUGKS step kernels for sm_103a -- the plain drop-in path.
//
// One time step = three launches, in the phase order of
// Ark/Cpp/DUGKS2DSolver.cpp:175-327:
//   k_collide : [deferred P10 MacroSource of the previous step] + P1 + P2
//               (equilibria, force source, f-bar-plus; ghost phi rows)
//   k_faces   : P4 + P6 for every physical face (CD reconstruction, face
//               moments, face equilibrium/source, flux x xi.n dS, wall BB)
//   k_update  : P8 + P9 (finite-volume update, cell macros)
// The pseudopotential models split the face pass in two (face psi, then
// face force) -- the Jacobi semantics of the face psi gradient.
//
// This file is compiled twice (see fp64_exact.cu / fp64_fast.cu):
//  * DUGKS_EXACT = 1 with -fmad=false: every operation of the reference that rounds is
//    rounded here alike, so the step gives the same doubles as the reference solver.
//    The compiler contracts nothing; what is rewritten is what leaves the rounded values
//    as they are: quotients by a shared divisor (qdiv_rn), powers of two taken into a
//    fused multiply-add or a constant, terms that are zero, signs, products formed on the
//    integer pipe (fp64_imul.cuh).  The one exception are subnormal numbers (a phase
//    field below 1e-300 at the tip of its spreading tail): there a factor 1/2 does not
//    commute with the rounding, and results may differ by some units of 2^-1074;
//  * DUGKS_EXACT = 0 with FMA contraction and reciprocal multiplies: the same
//    algorithm with fewer FP64 instructions, equal to the reference to rounding.
#pragma once
#include <cuda_runtime.h>
#include "dugks_device.cuh"
#include "fp64_imul.cuh"
#include "pdl.cuh"

#ifndef DUGKS_EXACT
#error "define DUGKS_EXACT before including fp64_step.cuh"
#endif
#if DUGKS_EXACT
#define DUGKS_KNS exact
// x / d with invd = RN(1/d), the reciprocal of a divisor shared by several quotients:
// correctly rounded (qdiv_rn), so the same double as the reference's division
#define QDIV(x, d, invd) qdiv_rn((x), (d), (invd))
#else
#define DUGKS_KNS fast
#define QDIV(x, d, invd) ((x) * (invd))  // one reciprocal, then multiplies
#endif

// The FP64 pipe bounds every kernel here (one warp instruction per 76 cycles and SM
// quarter, 1.68 lane operations per cycle and SM, measured), so the formulas are arranged
// for few FP64 instructions at unchanged results.  Scaling by a power of two commutes with
// rounding (away from the subnormal range), hence for the exact variant too:
//  * a product with a power of two is folded into the next addition, fma(2^k, a, b) =
//    RN(2^k a + b), or into a constant of the next product;
//  * the D2Q9 models have dt = 1/2, hDt = 1/4 and unit cells whatever the case (CFL 1/2,
//    MinL = 1, max |xi| = sqrt(3 RT) = 1), phi_L = 1, phi_V = 0 and one kinematic
//    viscosity, so the factors they appear in are powers of two, or drop out;
//  * the equilibria of opposite directions share every product whose factors differ in
//    sign only.
// Passes of steps and a read-back, before and after these rewritings alone: 512x2048
// Rayleigh-Taylor box (HCZ, walls) 4.07 -> 3.19 ms a step; 256x256 D2V16 0.453 -> 0.308 ms;
// 128x128 AC drop 74 -> 54 us.  With the launch forms and the integer-pipe products below
// (fp64_imul.cuh) 2.17 ms, 0.275 ms and 43 us.  The FMA
// variant keeps the form its results were published with (another contraction moves the
// velocities of a nearly resting fluid by 1e-9): only what is exact in any contraction, the
// face reconstruction and the split by face direction, is shared: 333x257 HCZ drop 271 ->
// 234 us.  With walls its face kernel is not split, since that changes the contraction.

namespace dugks {
namespace DUGKS_KNS {


// x / d rounded to nearest, from y = RN(1/d): q0 = RN(x y) lies within an ulp of x / d,
// the residual r = x - d q0 is exact in one fused multiply-add, and RN(q0 + r y) is the
// correctly rounded quotient (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Develop. 34 (1990), Theorem 1; operands and
// quotient in the normal range).  Three FP64 operations where a division takes about ten.
// The correction turns the -0 of a zero x into +0, so the sign is taken from q0, by an
// integer operation: a floating-point comparison with 0 occupies the FP64 pipe like an
// addition (76 cycles a warp and SM quarter here).  Checked bit for bit against IEEE
// division on 2e8 random operand pairs (all-ones significands, near powers of two, signed
// zeros included).
__device__ __forceinline__ double qdiv_rn(double x, double d, double y) {
    const double q0 = __dmul_rn(x, y);
    const double r = __fma_rn(-d, q0, x);
    const double q = __fma_rn(r, y, q0);
    return __hiloint2double((__double2hiint(q) & 0x7fffffff) | (__double2hiint(q0) & 0x80000000), __double2loint(q));
}
__device__ __forceinline__ int wrapi(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
// velocity components in units of the model's lattice speed
template <int MODEL>
__host__ __device__ constexpr int vel_u(int q) { return MODEL == PP16 ? d2v16_xu(q) : d2q9_xu(q); }
template <int MODEL>
__host__ __device__ constexpr int vel_v(int q) { return MODEL == PP16 ? d2v16_xv(q) : d2q9_xv(q); }

// Cells and faces of a launch.  Small grids (wide_blocks): one-warp blocks whose threads
// run over the cells in row order without regard to the rows' ends, so only the last warp has
// idle lanes (a warp occupies the FP64 pipe alike however many lanes are active) and the
// warps spread evenly over the SMs (a lone warp issues an FP64 instruction every 64 cycles,
// an SM of four every 19: 256-thread blocks left most SMs of a small grid idle and others
// with eight warps in turn).  Faces: the x-faces, then the y-faces (with walls one row
// more), then (UW) the low-side x and y boundary faces, each group from a multiple of 32 on.
// Larger grids have rounds of blocks enough for any shape, and 32 x 8 blocks (blockIdx.z: the
// face group) read their y neighbours through L1 once: 2 % faster on 512x2048.
// Passes of the benchmark's sizes, 32x8 blocks / one-warp blocks: 32x24 AC 2.67 / 1.86 ms, 128x128
// AC 2.72 / 2.29, 256x256 D2V16 6.16 / 5.49, 333x257 HCZ (FMA) 9.49 / 8.16, 512x2048 HCZ 15.94 /
// 16.27.
__device__ __forceinline__ bool cell_of_thread(const Params &P, int &i, int &j) {
    if (blockDim.y > 1) {
        i = blockIdx.x * 32 + threadIdx.x;
        j = blockIdx.y * blockDim.y + threadIdx.y;
        return i < P.nx && j < P.ny;
    }
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    j = (int)(t / (unsigned)P.nx);
    i = (int)(t - (unsigned)j * (unsigned)P.nx);
    return j < P.ny;
}
__host__ __device__ __forceinline__ unsigned pad32(unsigned n) { return (n + 31u) & ~31u; }
__device__ __forceinline__ bool face_of_thread(const Params &P, bool walls, bool uw, int &i, int &j, bool &xf, bool &lo) {
    const unsigned nx = P.nx, ny = P.ny, yrows = walls ? ny + 1 : ny;
    if (blockDim.y > 1) {
        xf = (blockIdx.z & 1) == 0;
        lo = uw && blockIdx.z >= 2;
        i = blockIdx.x * 32 + threadIdx.x;
        j = blockIdx.y * blockDim.y + threadIdx.y;
        return (unsigned)i < nx && (unsigned)j < (xf ? ny : yrows) && !(lo && (xf ? i != 0 : j != 0));
    }
    unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nX = pad32(nx * ny), nY = pad32(nx * yrows);
    lo = uw && t >= nX + nY;
    if (lo) {
        t -= nX + nY;
        xf = t < pad32(ny);
        if (!xf) t -= pad32(ny);
        i = xf ? 0 : (int)t;
        j = xf ? (int)t : 0;
        return xf ? t < ny : t < nx;
    }
    xf = t < nX;
    if (!xf) t -= nX;
    j = (int)(t / nx);
    i = (int)(t - (unsigned)j * nx);
    return (unsigned)j < (xf ? ny : yrows);
}
// Programmatic launches (pdl.cuh) only while every SM quarter has at most one warp of cells:
// blocks that are placed before the kernel ahead of them ends go to the SMs that finish first,
// and on larger grids that unevenness costs more FP64 pipe time than the launches saved
// (333x257 HCZ, FMA: 7.93 ms plain, 9.33 programmatic; 256x256 D2V16 5.54 / 5.85).
static bool early_launch(const Params &P) { return pad32((unsigned)P.nx * P.ny) <= 32u * 152u * 4u; }
// 32 x 8 blocks: from 486 k cells, or from 230 k where the integer products run with them (us
// per step, one-warp blocks without / 32 x 8 with: 400x400 412 / 429, 460x460 519 / 521, 500x500
// 609 / 589, 600x600 875 / 802; along drops of 1000 steps, with the far tail of far_tail(): HCZ 480x480 564 /
// 496-535, 600x600 876 / 781-828, AC 480x480 349 / 322-345, 600x600 540 / 510-546)
static bool im_model(const Params &P) { return DUGKS_EXACT && (P.model == AC || P.model == HCZ) && !P.uw; }
static bool wide_blocks(const Params &P) {
    const unsigned nx = P.nx;
    if (16 * pad32(nx) > 17 * nx) return false;  // columns that leave many lanes of a row idle
    return pad32(nx) * P.ny >= (im_model(P) ? 230400u : 32u * 152u * 100u);
}
// Products of the collision and the faces by the integer pipe (fp64_imul.cuh): the exact
// variant on grids large enough for 32 x 8 blocks.  A face's 359 FP64 instructions become 277,
// the collision's 373 become 250, and both kernels stay at 70-81 % of the pipe's issue rate (a
// pair's two forms in one body: the HCZ face kernel spills 200 bytes a thread at its 128 registers).
// The code is four times as long, and the one-warp blocks of a smaller grid do not run through
// it together.  us per step, without / with: 256x256 174 / 170, 400x400 412 / 430, 1000x1000
// 2437 / 2059.  (Taken out again: the quotients' and moments' products too, which spilled, and
// the update's, 154 registers: 2289.)
static bool integer_products(const Params &P) { return im_model(P) && wide_blocks(P); }
struct Launch {
    dim3 grid, block;
};
static Launch cell_launch(const Params &P) {
    const unsigned nx = P.nx, ny = P.ny;
    if (wide_blocks(P)) return {dim3((nx + 31) / 32, (ny + 7) / 8), dim3(32, 8)};
    return {dim3(pad32(nx * ny) / 32), dim3(32)};
}
static Launch face_launch(const Params &P, bool walls, bool uw) {
    const unsigned nx = P.nx, ny = P.ny, yrows = walls ? ny + 1 : ny;
    if (wide_blocks(P)) return {dim3((nx + 31) / 32, (yrows + 7) / 8, uw ? 4 : 2), dim3(32, 8)};
    return {dim3((pad32(nx * ny) + pad32(nx * yrows) + (uw ? pad32(ny) + pad32(nx) : 0)) / 32), dim3(32)};
}

// Cell field at logical row j in -1..ny (ghost rows: 2 a0 - a1 with walls,
// wrap otherwise), column i already wrapped.
template <bool WALLS>
__device__ __forceinline__ double cellv(const double *__restrict__ a, int ny, int pitch, int j, int i) {
    if (j < 0) {
        if (WALLS) return 2.0 * a[i] - a[pitch + i];
        j += ny;
    } else if (j >= ny) {
        if (WALLS) return 2.0 * a[(size_t)(ny - 1) * pitch + i] - a[(size_t)(ny - 2) * pitch + i];
        j -= ny;
    }
    return a[(size_t)j * pitch + i];
}

#if DUGKS_EXACT
#include "fp64_exact_math.cuh"
#else
#include "fp64_fma_math.cuh"
#endif

// ---------------------------------------------------------------------------
// UW flux scheme (_FLUX_SCHEME_UW_ARK), periodic grids.
//
// Cell gradients of f-bar-plus, Grad_VS_6points (Ark/Cpp/GradScheme.cpp:205-218,
// Ark/Lib/GradSchemeBasic.h:95-126): apsi = 4 on the axis neighbours, bpsi = 1
// on the diagonals (C0..C3 = E, N, W, S; D0..D3 = NE, NW, SW, SE), divided by
// 6 _2dx, in the reference's operand order.
template <int MODEL>
__global__ void __launch_bounds__(256) k_grad6(Params P, State S) {
    pdl_wait();
    int i, j;
    if (!cell_of_thread(P, i, j)) return;
    const int pitch = P.pitch;
    const int im = wrapi(i - 1, P.nx), ip = wrapi(i + 1, P.nx), jm = wrapi(j - 1, P.ny), jp = wrapi(j + 1, P.ny);
    const size_t c = (size_t)j * pitch + i;
    const size_t cE = (size_t)j * pitch + ip, cW = (size_t)j * pitch + im, cN = (size_t)jp * pitch + i,
                 cS = (size_t)jm * pitch + i, cNE = (size_t)jp * pitch + ip, cNW = (size_t)jp * pitch + im,
                 cSW = (size_t)jm * pitch + im, cSE = (size_t)jm * pitch + ip;
    const double dxd = P._2dx * 6, dyd = P._2dy * 6, rdx = 1.0 / dxd, rdy = 1.0 / dyd;
    (void)rdx;
    (void)rdy;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const double *B = (w ? S.bh : S.bf) + (size_t)q * S.qs;
            const double E = B[cE], W = B[cW], N = B[cN], Sv = B[cS];
            double gx, gy;
            if (P.uw_grad == 1) {
                // Grad_VS_LS (Ark/Lib/GradSchemeBasic.h:127-152): sum over the neighbours
                // E, N, W, S of w_k (B_k - B_c), then the inverse 2x2 matrix.  On this
                // mesh of unit cells the weights of Grad_LSMatrix (:13-75) are exact: the
                // cell centres (two-triangle centroids, Ark/Cpp/Mesh/Cell_2D.cpp:157-179)
                // are i + 1/2, j + 1/2 and the periodic shadows' are offset by exactly
                // Lx / Ly, so wdx = {1, 0, -1, 0}, wdy = {0, 1, 0, -1} and the inverse
                // matrix is {{0.5, -0}, {-0, 0.5}}; every product and sum of the reference
                // is kept (the zero terms included), so the result is the same bits.
                const double C = B[c];
                const double nb[4] = {E, N, W, Sv}, wx[4] = {1.0, 0.0, -1.0, 0.0}, wy[4] = {0.0, 1.0, 0.0, -1.0};
                double sx = 0.0, sy = 0.0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    sx = sx + wx[k] * (nb[k] - C);
                    sy = sy + wy[k] * (nb[k] - C);
                }
                gx = 0.5 * sx + -0.0 * sy;
                gy = -0.0 * sx + 0.5 * sy;
            } else if (P.uw_grad == 2) {
                // Grad_VS_4points (Ark/Lib/GradSchemeBasic.h:76-94): (C0 - C2) / (2 dx)
                gx = QDIV(E - W, P._2dx, 0.5 / P.dx);
                gy = QDIV(N - Sv, P._2dy, 0.5 / P.dy);
            } else {
                const double NE = B[cNE], NW = B[cNW], SW = B[cSW], SE = B[cSE];
                gx = QDIV(4.0 * (E - W) + (((NE - NW) + SE) - SW), dxd, rdx);
                gy = QDIV(4.0 * (N - Sv) + (((NE - SE) + NW) - SW), dyd, rdy);
            }
            (w ? S.ghx : S.gfx)[(size_t)q * S.qs + c] = gx;
            (w ? S.ghy : S.gfy)[(size_t)q * S.qs + c] = gy;
        }
    }
}

// Reconstruction UW_Interior_phi_Bh (Ark/Cpp/DUGKS2DSolver.cpp:558-603, chosen by the
// sign of xi.n dS at :689-706) of velocity (xu, xv) at one face: the upwind
// cell's f-bar-plus + (dx gx + dy gy) with (dx, dy) = x_f - hDt xi - x_c; the
// owner's and the neighbour's values averaged (owner first) along the face.
// The face is at the origin and its two cells at -1/2 ("o", below / left) and
// +1/2 ("n") along the normal: every offset is exact, as the reference's are
// on the unit grid.  The reference computes a periodic boundary face twice, as
// the high-side face (owner o, normal +x / +y: the interior form) and as the
// low-side face (owner n inside the domain, normal -x / -y): lo selects that form.
template <bool XF>
__device__ __forceinline__ double face_uw(const Params &P, const double *__restrict__ B,
                                          const double *__restrict__ GX, const double *__restrict__ GY, size_t co,
                                          size_t cn, double xu, double xv, bool lo) {
    const double xon = XF ? -0.5 : 0.0, yon = XF ? 0.0 : -0.5;  // centre of o
    const double xnn = XF ? 0.5 : 0.0, ynn = XF ? 0.0 : 0.5;    // centre of n
    const double xsh = 0.0 - P.hDt * xu, ysh = 0.0 - P.hDt * xv;
    const double dxo = xsh - xon, dyo = ysh - yon, dxn = xsh - xnn, dyn = ysh - ynn;
    const double Xo = dxo * GX[co] + dyo * GY[co], Xn = dxn * GX[cn] + dyn * GY[cn];
    const double xin = XF ? xu : xv;
    const double s = lo ? -xin : xin;  // xi.n of the reference's face
    if (lo) {                          // owner n, neighbour o
        if (s > 0) return B[cn] + Xn;
        if (s < 0) return B[co] + Xo;
        double t = B[cn] + Xn;
        t = t + B[co];
        t = t + Xo;
        return t / 2;
    }
    if (s > 0) return B[co] + Xo;
    if (s < 0) return B[cn] + Xn;
    double t = B[co] + Xo;
    t = t + B[cn];
    t = t + Xn;
    return t / 2;
}

#if DUGKS_EXACT
#include "fp64_exact_faces.cuh"
#else
#include "fp64_fma_faces.cuh"
#endif

// Wall_3_NEE (Ark/Cpp/Boundary.cpp:140-184) on the wall faces (y-face rows 0 and ny),
// written over what k_faces_ac left there.  The face's U, V keep the initial 0 of
// its MsQh (the routine never sets them); phi and rho are the owner's extrapolated
// with its Phi_x/Phi_y (the phase-field source vector after MacroSource) and
// Rho_x/Rho_y to the face (0.5 below / above the centre), p is the owner's;
// Update_phi_Eqh at those moments (Ark/Lib/D2Q9AC.cpp:106-144,
// Ark/Lib/D2Q9HCZ.cpp:93-131), plus the owner's non-equilibrium part
// (Tilde - Eq + hDt So, Eq and So of this step's collision) times
// 2 tau / (2 tau + dt); then Wall_3_BB.
template <int MODEL>
__global__ void __launch_bounds__(256) k_faces_nee(Params P, State S) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, side = blockIdx.y;
    if (i >= P.nx) return;
    const int ny = P.ny, pitch = P.pitch, jc = side ? ny - 1 : 0;
    const size_t c = (size_t)jc * pitch + i;
    const double dxw = 0.0, dyw = side ? 0.5 : -0.5;
    const double Phi = S.fld[F_PHI][c] + S.fld[F_PHIX][c] * dxw + S.fld[F_PHIY][c] * dyw;
    const double Rho = S.fld[F_RHO][c] + S.fld[F_RHOX][c] * dxw + S.fld[F_RHOY][c] * dyw;
    const double p = S.fld[F_P][c], U = 0.0, V = 0.0;
    const double uu = U * U + V * V;
    const double tau = S.fld[F_TAU][c];
    const double hNEq = 2.0 * P.TauMass / (2.0 * P.TauMass + P.dt);
    const double fNEq = 2.0 * tau / (2.0 * tau + P.dt);
    const size_t ws = (size_t)2 * 9 * pitch;
    double hf[9], hh[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const double xu = d2q9_xu(q), xv = d2q9_xv(q), w = d2q9_w(q);
        const double u1 = (xu * U + xv * V) / P.RT;
        const double G = u1 + 0.5 * u1 * u1 - uu * P.Lambda0;
        const double hEq = w * Phi * (1.0 + u1);
        double fEq;
        if (MODEL == AC) {
            fEq = w * (p / P.RT + Rho * G);
            if (q == 0) fEq = fEq - 1.0 * p / P.RT;
        } else {
            fEq = w * (p + Rho * P.RT * G);
        }
        const size_t wq = ((size_t)side * 9 + q) * pitch + i, o = (size_t)q * S.qs + c;
        hh[q] = hEq + hNEq * (S.h[o] - S.weq[2 * ws + wq] + P.hDt * S.weq[3 * ws + wq]);
        hf[q] = fEq + fNEq * (S.f[o] - S.weq[wq] + P.hDt * S.weq[ws + wq]);
    }
    // bounce-back of the directions entering the fluid (xi.n_out < 0)
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int xv = d2q9_xv(q);
        if (side ? xv < 0 : xv > 0) {
            hh[q] = hh[d2q9_bb(q)];
            hf[q] = hf[d2q9_bb(q)];
        }
    }
    const int jf = side ? ny : 0;
    const size_t cf = (size_t)jf * pitch + i;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int xv = d2q9_xv(q);
        S.yff[(size_t)q * S.qsy + cf] = sx(xv, hf[q]);
        S.yfh[(size_t)q * S.qsy + cf] = sx(xv, hh[q]);
    }
}

// Deferred MacroSource / pseudopotential cell force on its own (used before
// handing the fields to the host).
template <int MODEL, bool WALLS>
__global__ void __launch_bounds__(256) k_finalize(Params P, State S, int gin) {
    pdl_wait();
    int i, j;
    if (!cell_of_thread(P, i, j)) return;
    const size_t c = (size_t)j * P.pitch + i;
    if (MODEL == AC || MODEL == HCZ) {
        const double phi = S.fld[F_PHI][c], U = S.fld[F_U][c], V = S.fld[F_V][c];
        double srcx, srcy, rhox, rhoy, fx, fy;
        macro_source<WALLS>(P, S, i, j, gin, phi, S.fld[F_RHO][c], U, V, S.fld[F_PPU][c], S.fld[F_PPV][c], srcx,
                            srcy, rhox, rhoy, fx, fy);
        // neighbours read phi only, so in-place writes are race-free
        S.fld[F_PHIX][c] = srcx;
        S.fld[F_PHIY][c] = srcy;
        S.fld[F_RHOX][c] = rhox;
        S.fld[F_RHOY][c] = rhoy;
        S.fld[F_FX][c] = fx;
        S.fld[F_FY][c] = fy;
        S.fld[F_PPU][c] = phi * U;
        S.fld[F_PPV][c] = phi * V;
    } else {
        const int nx = P.nx, ny = P.ny, pitch = P.pitch;
        const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx), jm = wrapi(j - 1, ny), jp = wrapi(j + 1, ny);
        const double *__restrict__ PS = S.fld[F_PSI];
        auto at = [&](int jj, int ii) { return PS[(size_t)jj * pitch + ii]; };
        const double gx = iso_gx(at(j, ip), at(j, im), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P.g6x, P.r_g6x);
        const double gy = iso_gy(at(jp, i), at(jm, i), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P.g6y, P.r_g6y);
        const double k = -S.fld[F_SCG][c] * at(j, i);
        S.fld[F_FX][c] = gx * k;
        S.fld[F_FY][c] = gy * k;
    }
}

// ---------------------------------------------------------------------------
// Reductions: per-block partial sums of rho, phi, (rho-rho_last)^2, rho^2,
// fixed-order tree (deterministic), then one block sums the partials.
__global__ void __launch_bounds__(256) k_reduce_partial(Params P, const double *__restrict__ rho,
                                                        const double *__restrict__ phi, double *rho_last,
                                                        double *partial, int has_phi) {
    __shared__ double sh[4][256];
    const int tid = threadIdx.x;
    const long n = (long)P.nx * P.ny;
    double a = 0, b = 0, d = 0, r2 = 0;
    for (long k = (long)blockIdx.x * blockDim.x + tid; k < n; k += (long)gridDim.x * blockDim.x) {
        const int j = (int)(k / P.nx), i = (int)(k % P.nx);
        const size_t c = (size_t)j * P.pitch + i;
        const double r = rho[c];
        a += r;
        if (has_phi) b += phi[c];
        const double dr = r - rho_last[c];
        d += dr * dr;
        r2 += r * r;
        rho_last[c] = r;
    }
    sh[0][tid] = a;
    sh[1][tid] = b;
    sh[2][tid] = d;
    sh[3][tid] = r2;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (tid < s)
            for (int m = 0; m < 4; ++m) sh[m][tid] += sh[m][tid + s];
        __syncthreads();
    }
    if (tid < 4) partial[(size_t)blockIdx.x * 4 + tid] = sh[tid][0];
}

__global__ void k_reduce_final(const double *__restrict__ partial, int nblocks, double *out) {
    __shared__ double sh[4][256];
    const int tid = threadIdx.x;
    double v[4] = {0, 0, 0, 0};
    for (int k = tid; k < nblocks; k += blockDim.x)
        for (int m = 0; m < 4; ++m) v[m] += partial[(size_t)k * 4 + m];
    for (int m = 0; m < 4; ++m) sh[m][tid] = v[m];
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (tid < s)
            for (int m = 0; m < 4; ++m) sh[m][tid] += sh[m][tid + s];
        __syncthreads();
    }
    if (tid < 4) out[tid] = sh[tid][0];
}

__global__ void k_check_finite(const double *__restrict__ a, size_t n, int *flag) {
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
        if (!isfinite(a[k])) {
            atomicOr(flag, 1);
            return;
        }
}

// ---------------------------------------------------------------------------
// Host-side launch helpers (called from capi.cu).

template <int MODEL, bool WALLS>
static void launch_step_t(const Params &P, const State &S, int do_msrc, int gin, int gout, cudaStream_t st,
                          int64_t *launches, cudaEvent_t *ev) {
    const auto [grd, blk] = cell_launch(P);
    const bool early = early_launch(P);
    if (ev) cudaEventRecord(ev[0], st);
    constexpr bool CAN_IM = DUGKS_EXACT && (MODEL == AC || MODEL == HCZ);
    const bool im = CAN_IM && integer_products(P);
    if (im) launch_after(early, k_collide<MODEL, WALLS, CAN_IM>, grd, blk, 0, st, P, S, do_msrc, gin, gout);
    else launch_after(early, k_collide<MODEL, WALLS, false>, grd, blk, 0, st, P, S, do_msrc, gin, gout);
    if (ev) cudaEventRecord(ev[1], st);
    if constexpr (MODEL == AC || MODEL == HCZ) {
        if (!WALLS && P.uw) {  // UW: cell gradients, then the faces with the low-side boundary faces
            launch_after(early, k_grad6<MODEL>, grd, blk, 0, st, P, S);
            const auto [gf, bf] = face_launch(P, false, true);
            launch_after(early, k_faces_ac<MODEL, false, true, false>, gf, bf, 0, st, P, S);
            *launches += 4;
        } else {
            const auto [gf, bf] = face_launch(P, WALLS, false);
            if (im) launch_after(early, k_faces_ac<MODEL, WALLS, false, CAN_IM>, gf, bf, 0, st, P, S);
            else launch_after(early, k_faces_ac<MODEL, WALLS, false, false>, gf, bf, 0, st, P, S);
            *launches += 3;
            if (WALLS && P.nee) {  // NEE wall faces over the bounce-back ones
                launch_after(early, k_faces_nee<MODEL>, dim3((P.nx + 127) / 128, 2), 128, 0, st, P, S);
                *launches += 1;
            }
        }
    } else {
        const auto [gf, bf] = face_launch(P, false, false);
        launch_after(early, k_faces_pp1<MODEL>, gf, bf, 0, st, P, S);
        launch_after(early, k_faces_pp2<MODEL>, gf, bf, 0, st, P, S);
        *launches += 4;
    }
    if (ev) cudaEventRecord(ev[2], st);
    launch_after(early, k_update<MODEL, WALLS>, grd, blk, 0, st, P, S);
    if (ev) cudaEventRecord(ev[3], st);
}

template <int MODEL, bool WALLS>
static void launch_finalize_t(const Params &P, const State &S, int gin, cudaStream_t st) {
    const auto [grd, blk] = cell_launch(P);
    const bool early = early_launch(P);
    launch_after(early, k_finalize<MODEL, WALLS>, grd, blk, 0, st, P, S, gin);
}

void launch_fp64_step(const Params &P, const State &S, int do_msrc, int gin, int gout, cudaStream_t st,
                      int64_t *launches, cudaEvent_t *ev) {
    switch (P.model * 2 + (P.walls ? 1 : 0)) {
        case AC * 2 + 0: launch_step_t<AC, false>(P, S, do_msrc, gin, gout, st, launches, ev); break;
        case AC * 2 + 1: launch_step_t<AC, true>(P, S, do_msrc, gin, gout, st, launches, ev); break;
        case HCZ * 2 + 0: launch_step_t<HCZ, false>(P, S, do_msrc, gin, gout, st, launches, ev); break;
        case HCZ * 2 + 1: launch_step_t<HCZ, true>(P, S, do_msrc, gin, gout, st, launches, ev); break;
        case PP9 * 2 + 0: launch_step_t<PP9, false>(P, S, do_msrc, gin, gout, st, launches, ev); break;
        case PP16 * 2 + 0: launch_step_t<PP16, false>(P, S, do_msrc, gin, gout, st, launches, ev); break;
        default: break;
    }
}

void launch_fp64_finalize(const Params &P, const State &S, int gin, cudaStream_t st, int64_t *launches) {
    switch (P.model * 2 + (P.walls ? 1 : 0)) {
        case AC * 2 + 0: launch_finalize_t<AC, false>(P, S, gin, st); break;
        case AC * 2 + 1: launch_finalize_t<AC, true>(P, S, gin, st); break;
        case HCZ * 2 + 0: launch_finalize_t<HCZ, false>(P, S, gin, st); break;
        case HCZ * 2 + 1: launch_finalize_t<HCZ, true>(P, S, gin, st); break;
        case PP9 * 2 + 0: launch_finalize_t<PP9, false>(P, S, gin, st); break;
        case PP16 * 2 + 0: launch_finalize_t<PP16, false>(P, S, gin, st); break;
        default: return;
    }
    *launches += 1;
}

void launch_reduce(const Params &P, const double *rho, const double *phi, double *rho_last, double *partial,
                   int nblocks, double *out4, int has_phi, cudaStream_t st, int64_t *launches) {
    k_reduce_partial<<<nblocks, 256, 0, st>>>(P, rho, phi, rho_last, partial, has_phi);
    k_reduce_final<<<1, 256, 0, st>>>(partial, nblocks, out4);
    *launches += 2;
}

void launch_check_finite(const double *a, size_t n, int *flag, cudaStream_t st, int64_t *launches) {
    int blocks = (int)((n + 255) / 256);
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    k_check_finite<<<blocks, 256, 0, st>>>(a, n, flag);
    *launches += 1;
}

}  // namespace DUGKS_KNS
}  // namespace dugks
