// FP32 deviation-storage step with the upwind (UW) flux scheme (_FLUX_SCHEME_UW_ARK),
// periodic grids of the Allen-Cahn models (AC, HCZ).
//
// The reference's UW (Ark/Cpp/DUGKS2DSolver.cpp:196-205,540-603,689-706) takes per cell
// the 6-point gradient of f-bar-plus and h-bar-plus (Grad_VS_6points,
// Ark/Lib/GradSchemeBasic.h:95-126) and at each face extrapolates the upwind cell's value
// to x_f - hDt xi (the two cells' extrapolations averaged for the velocities along the
// face).  The gradient needs f-bar-plus of a cell's eight neighbours, so this form runs
// two launches over scratch planes (UW_PLANES, one every qs floats from U):
//   collision  -> f-bar-plus pairs, collision increments, averaged-field inputs;
//   tiles      -> in one block's registers and shared memory: cell gradients of the
//                 f-bar-plus pairs and of the phase field (the 6-point one, or the
//                 least-squares / 4-point ones of DUGKS_FLUX_UW_LS / DUGKS_FLUX_UW_4P),
//                 upwind reconstruction, the same face moments, equilibria and fluxes as
//                 the central scheme (face_state_flux) and the same finite-volume update
//                 (update_cell).
// The per-cell and per-face arithmetic is the central-scheme step's (collide_cell,
// face_state_flux, update_cell in fp32_math.cuh); only the reconstruction differs.
// In the split storage h_q = g_q + w_q phi, so an h extrapolation is the g extrapolation
// plus w_q times the phi extrapolation; the face works relative to w_q times the face's
// phi average, as the central face does:
//   bh_q.y = g_u + d.grad g_u + w_q (phi_u - avg + d.grad phi_u),  d = x_f - hDt xi - x_u,
// with phi_u - avg = -+(phi_n - phi_o)/2 formed from the float-float pairs.
#include <cuda_runtime.h>

#include <cstdint>

#include "fp32_math.cuh"
#include "pdl.cuh"

namespace dugks {
namespace f32 {

namespace {

constexpr int UBX = 32, UBY = 8;

struct Cells {
    int i, j, im, ip, jm, jp;
    size_t c;
};

__device__ __forceinline__ bool cell_of(const P32 &P, Cells &k) {
    k.i = blockIdx.x * UBX + threadIdx.x;
    k.j = blockIdx.y * UBY + threadIdx.y;
    if (k.i >= P.nx || k.j >= P.ny) return false;
    k.im = wrapi(k.i - 1, P.nx);
    k.ip = wrapi(k.i + 1, P.nx);
    k.jm = wrapi(k.j - 1, P.ny);
    k.jp = wrapi(k.j + 1, P.ny);
    k.c = (size_t)k.j * P.pitch + k.i;
    return true;
}

__device__ __forceinline__ size_t at(const P32 &P, int j, int i) { return (size_t)j * P.pitch + i; }

__device__ __forceinline__ float2 phi_at(const S32 &S, size_t c) { return mk2(S.phi[c], S.phi[S.qs + c]); }

// nine pair planes of the scratch, one every qs pairs from plane `first`
__device__ __forceinline__ float2 *pairs(float *U, int first, size_t qs) {
    return reinterpret_cast<float2 *>(U + (size_t)first * qs);
}
__device__ __forceinline__ const float2 *pairs(const float *U, int first, size_t qs) {
    return reinterpret_cast<const float2 *>(U + (size_t)first * qs);
}
// one asynchronous 8-byte global -> shared copy
__device__ __forceinline__ void cp_async_pair(float2 *smem, const float2 *gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// the stored deviations of a cell as (f, g) pairs, g_0 = -sum g; sfz = sum f (AC: without f_0)
template <int MODEL>
__device__ __forceinline__ void load_cell(const S32 &S, size_t c, float2 (&Pq)[9], float &sfz) {
    Pq[0] = mk2(S.df[c], 0.f);
#pragma unroll
    for (int q = 1; q < 9; ++q) Pq[q] = mk2(S.df[(size_t)q * S.qs + c], S.dg[(size_t)(q - 1) * S.qs + c]);
    const float2 za[9] = {mk2(MODEL == AC ? 0.f : Pq[0].x, 0.f), Pq[1], Pq[2], Pq[3], Pq[4],
                          Pq[5], Pq[6], Pq[7], Pq[8]};
    const float2 z = dev_sum9(za);
    sfz = z.x;
    Pq[0].y = -z.y;
}

}  // namespace

// Collision of every cell: f-bar-plus pairs (B), the increments B - T (INC), the
// averaged-field inputs (A) and, HCZ, the MacroSource outputs the next step reads.
template <int MODEL, int MIN_BLOCKS>
__global__ void __launch_bounds__(UBX *UBY, MIN_BLOCKS) k_uw32_collide(P32 P, S32 S, float *U, int first) {
    pdl_wait();
    Cells k;
    if (!cell_of(P, k)) return;
    const size_t qs = S.qs, c = k.c;
    float2 Pq[9];
    float sfz;
    load_cell<MODEL>(S, c, Pq, sfz);
    float a6[A_N];
#pragma unroll
    for (int a = 0; a < A_N; ++a) a6[a] = (MODEL != AC && !first) ? S.aux[(size_t)a * qs + c] : 0.f;
    const float2 ph[8] = {phi_at(S, at(P, k.j, k.ip)),  phi_at(S, at(P, k.j, k.im)),  phi_at(S, at(P, k.jp, k.i)),
                          phi_at(S, at(P, k.jm, k.i)),  phi_at(S, at(P, k.jp, k.ip)), phi_at(S, at(P, k.jp, k.im)),
                          phi_at(S, at(P, k.jm, k.ip)), phi_at(S, at(P, k.jm, k.im))};
    float2 inc[9];
    float src[6], phi, Uu, Vv;
    collide_cell<MODEL, float>(P, S, (long long)c, first, Pq, sfz, a6, phi_at(S, c), ph, inc, src, phi, Uu, Vv);
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        pairs(U, UW_B, qs)[(size_t)q * qs + c] = add2(Pq[q], inc[q]);
        pairs(U, UW_INC, qs)[(size_t)q * qs + c] = inc[q];
    }
#pragma unroll
    for (int a = 0; a < 6; ++a) U[(size_t)(UW_A + a) * qs + c] = src[a];
    if (MODEL != AC) {
        S.oaux[A_FX * qs + c] = src[4];
        S.oaux[A_FY * qs + c] = src[5];
        S.oaux[A_RHOX * qs + c] = src[2];
        S.oaux[A_RHOY * qs + c] = src[3];
        S.oaux[A_PPU * qs + c] = phi * Uu;
        S.oaux[A_PPV * qs + c] = phi * Vv;
    }
}

// Gradients, faces and update of a tile of 30 x (UFY - 2) cells by 32 x UFY threads, one for
// each cell of the tile and of a one-cell ring around it.  Direction by direction: the
// f-bar-plus pairs of the tile and two rings go to shared memory (asynchronously, while the
// direction before is worked on), each thread forms its cell's gradients (axis neighbours 4,
// diagonals 1, over 12 dx; with uw_grad the least-squares or 4-point ones, on unit cells both
// (E - W) / 2 and (N - S) / 2, whose different FP64 roundings are below FP32's) and from them
// its values extrapolated to those of its faces that it is upwind of; the west face takes the
// west cell's value from the lane before, the south face the row below's through shared memory
// one direction later (one barrier a direction).  Every face is formed once per tile, then the
// tile's cells are updated.
// As four launches with the gradients and the fluxes in scratch planes the step moved 1.2 KB a
// cell; now 0.53 KB.  512x512 69.7 -> 40.8 us a step, 2000x2000 1174 -> 588, 64x64 21.6 -> 9.4
// (there the launches).  What bounds it now is the latency of the direction loop and of the
// face arithmetic at 24 to 32 warps an SM; the bytes alone take 20.7 us at 512x512.
// Tiles of 14 rows (16 x 32 threads, two blocks an SM) are as fast on large grids and slower
// on small ones (256x256 18.5 us).
constexpr int UTW = 30, UFX = 32, UPX = UFX + 2;

template <int MODEL, int UFY, int MINB>
__global__ void __launch_bounds__(UFX *UFY, MINB) k_uw32_tile(P32 P, S32 S, const float *U, int ntx) {
    constexpr int UTH = UFY - 2, UPN = UPX * (UFY + 2);  // tile rows; cells of the tile and two rings
    pdl_wait();
    // the fluxes of the south faces take the place of the reconstruction's buffers
    __shared__ __align__(16) union {
        struct {
            float2 B[2][UPN];        // f-bar-plus of one direction, two buffers
            float2 N[2][UFY][UFX];   // values at the north faces
            float2 G[UFY][UFX];      // phi gradients
        } r;
        float2 FS[6][UFY][UFX];
    } sm;
    __shared__ float2 sphi[UPN];         // phi pairs
    __shared__ float sA[6][UFY][UFX];    // averaged-field inputs
    const int e = threadIdx.x, r = threadIdx.y, tid = r * UFX + e;
    const int x0 = (blockIdx.x % ntx) * UTW, y0 = (blockIdx.x / ntx) * UTH;
    const int w = min(UTW, P.nx - x0), hh = min(UTH, P.ny - y0);
    const size_t qs = S.qs;
    const bool act = e <= w + 1 && r <= hh + 1;
    const size_t c = at(P, wrapi(y0 + min(r, hh + 1) - 1, P.ny), wrapi(x0 + min(e, w + 1) - 1, P.nx));
    // this thread's two elements of the staged region
    size_t off[2];
    bool in[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int i = tid + k * UFX * UFY, cy = i / UPX, cx = i - cy * UPX;
        in[k] = i < UPN && cx < w + 4 && cy < hh + 4;
        off[k] = in[k] ? at(P, wrapi(y0 + cy - 2, P.ny), wrapi(x0 + cx - 2, P.nx)) : 0;
    }
    const float2 *B = pairs(U, UW_B, qs);
    auto stage = [&](int q) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (in[k]) cp_async_pair(&sm.r.B[q & 1][tid + k * UFX * UFY], B + (size_t)q * qs + off[k]);
        cp_async_commit();
    };
    stage(0);
#pragma unroll
    for (int k = 0; k < 2; ++k)
        if (in[k]) sphi[tid + k * UFX * UFY] = phi_at(S, off[k]);
#pragma unroll
    for (int a = 0; a < 6; ++a) sA[a][r][e] = U[(size_t)(UW_A + a) * qs + c];
    const int me = (r + 1) * UPX + e + 1;  // this cell in the staged region
    const bool six = P.uw_grad == 0;
    const bool do_x = act && e >= 1 && r >= 1 && r <= hh, do_y = act && r >= 1 && e >= 1 && e <= w;
    float2 bx[9], by[9], gp = mk2(0.f, 0.f), gpw = gp, gps = gp, south = gp;
    float avgx = 0.f, hdx = 0.f, avgy = 0.f, hdy = 0.f;
    // value extrapolated to (dx, dy) from the centre, its phi part relative to the face's average
    auto along = [](float2 b, float2 gx, float2 gy, float dx, float dy) {
        return fma2(mk2(dy, dy), gy, fma2(mk2(dx, dx), gx, b));
    };
    auto with_phi = [](int q, float2 x, float dx, float dy, float phis, float2 g) {
        return mk2(x.x, fmaf((float)d2q9_w(q), fmaf(dy, g.y, fmaf(dx, g.x, phis)), x.y));
    };
    // the south face of direction q, from the row below's value and this cell's (south)
    auto south_face = [&](int q) {
        const float dx = -P.hDt * (float)d2q9_xu(q), sy = -P.hDt * (float)d2q9_xv(q);
        const float2 o = sm.r.N[q & 1][max(r - 1, 0)][e];
        const float2 vo = with_phi(q, o, dx, 0.5f + sy, -hdy, gps), vn = with_phi(q, south, dx, sy - 0.5f, hdy, gp);
        by[q] = d2q9_xv(q) > 0 ? vo : d2q9_xv(q) < 0 ? vn : mul2(mk2(0.5f, 0.5f), add2(vo, vn));
    };
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        cp_async_wait_all();
        __syncthreads();
        if (q < 8) stage(q + 1);
        if (q == 0) {
            const float2 E = sphi[me + 1], W = sphi[me - 1], N = sphi[me + UPX], Sv = sphi[me - UPX];
            if (six) {
                const float2 NE = sphi[me + UPX + 1], NW = sphi[me + UPX - 1], SE = sphi[me - UPX + 1], SW = sphi[me - UPX - 1];
                gp.x = __fmul_rn(fmaf(4.f, pdiff(E, W), pdiff(NE, NW) + pdiff(SE, SW)), P.inv_12dx);
                gp.y = __fmul_rn(fmaf(4.f, pdiff(N, Sv), pdiff(NE, SE) + pdiff(NW, SW)), P.inv_12dy);
            } else {
                gp = mk2(0.5f * pdiff(E, W), 0.5f * pdiff(N, Sv));
            }
            sm.r.G[r][e] = gp;
            gpw = mk2(__shfl_up_sync(0xffffffffu, gp.x, 1), __shfl_up_sync(0xffffffffu, gp.y, 1));
            const float2 pc = sphi[me];
            avgx = 0.5f * (W.x + pc.x);
            hdx = 0.5f * pdiff(pc, W);
            avgy = 0.5f * (Sv.x + pc.x);
            hdy = 0.5f * pdiff(pc, Sv);
        } else {
            if (q == 1) gps = sm.r.G[max(r - 1, 0)][e];
            south_face(q - 1);
        }
        const float2 *b = sm.r.B[q & 1];
        const float2 E = b[me + 1], W = b[me - 1], N = b[me + UPX], Sv = b[me - UPX], C = b[me];
        float2 gx, gy;
        if (six) {
            const float2 NE = b[me + UPX + 1], NW = b[me + UPX - 1], SE = b[me - UPX + 1], SW = b[me - UPX - 1];
            const float2 four = mk2(4.f, 4.f), ix = mk2(P.inv_12dx, P.inv_12dx), iy = mk2(P.inv_12dy, P.inv_12dy);
            gx = mul2(fma2(four, sub2(E, W), add2(sub2(NE, NW), sub2(SE, SW))), ix);
            gy = mul2(fma2(four, sub2(N, Sv), add2(sub2(NE, SE), sub2(NW, SW))), iy);
        } else {
            gx = mul2(mk2(0.5f, 0.5f), sub2(E, W));
            gy = mul2(mk2(0.5f, 0.5f), sub2(N, Sv));
        }
        const int xu = d2q9_xu(q), xv = d2q9_xv(q);
        const float sx = -P.hDt * (float)xu, sy = -P.hDt * (float)xv;
        // west face: the west cell's value at its east face (from the lane before), this cell's at its west
        float2 vo = mk2(0.f, 0.f), vn = vo;
        if (xu >= 0) {
            const float2 x = along(C, gx, gy, 0.5f + sx, sy);
            const float2 o = mk2(__shfl_up_sync(0xffffffffu, x.x, 1), __shfl_up_sync(0xffffffffu, x.y, 1));
            vo = with_phi(q, o, 0.5f + sx, sy, -hdx, gpw);
        }
        if (xu <= 0) vn = with_phi(q, along(C, gx, gy, sx - 0.5f, sy), sx - 0.5f, sy, hdx, gp);
        bx[q] = xu > 0 ? vo : xu < 0 ? vn : mul2(mk2(0.5f, 0.5f), add2(vo, vn));
        if (xv >= 0) sm.r.N[q & 1][r][e] = along(C, gx, gy, sx, 0.5f + sy);
        if (xv <= 0) south = along(C, gx, gy, sx, sy - 0.5f);
    }
    __syncthreads();
    south_face(8);
    float2 FW[6], FS[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) FW[s] = FS[s] = mk2(0.f, 0.f);
    if (do_x) {
        float av[6];
#pragma unroll
        for (int a = 0; a < 6; ++a) av[a] = 0.5f * (sA[a][r][e - 1] + sA[a][r][e]);
        face_state_flux<MODEL, true, float>(P, bx, av, avgx, 0, FW);
    }
    if (do_y) {
        float av[6];
#pragma unroll
        for (int a = 0; a < 6; ++a) av[a] = 0.5f * (sA[a][r - 1][e] + sA[a][r][e]);
        face_state_flux<MODEL, false, float>(P, by, av, avgy, 0, FS);
    }
    __syncthreads();  // the reconstruction's buffers are read: the fluxes take their place
    if (do_y) {
#pragma unroll
        for (int s = 0; s < 6; ++s) sm.FS[s][r][e] = FS[s];
    }
    float2 FE[6];
#pragma unroll
    for (int s = 0; s < 6; ++s)
        FE[s] = mk2(__shfl_down_sync(0xffffffffu, FW[s].x, 1), __shfl_down_sync(0xffffffffu, FW[s].y, 1));
    __syncthreads();
    if (!(do_x && do_y)) return;  // the tile's own cells
    float2 Pq[9], inc[9], FN[6], dn[9];
    float sfz;
    load_cell<MODEL>(S, c, Pq, sfz);
#pragma unroll
    for (int q = 0; q < 9; ++q) inc[q] = pairs(U, UW_INC, qs)[(size_t)q * qs + c];
#pragma unroll
    for (int s = 0; s < 6; ++s) FN[s] = sm.FS[s][r + 1][e];
    const float half_dtv = 0.5f * P.dtV;
    const float px = half_dtv * pdiff(sphi[me - 1], sphi[me + 1]);
    const float py = half_dtv * pdiff(sphi[me - UPX], sphi[me + UPX]);
    float dphi;
    update_cell<float>(P, Pq, inc, FW, FE, FS, FN, px, py, dn, dphi);
    S.odf[c] = dn[0].x;
#pragma unroll
    for (int q = 1; q < 9; ++q) {
        S.odf[(size_t)q * qs + c] = dn[q].x;
        S.odg[(size_t)(q - 1) * qs + c] = dn[q].y;
    }
    const float2 pn = phi_add(sphi[me], dphi);
    S.ophi[c] = pn.x;
    S.ophi[qs + c] = pn.y;
}

template <int MODEL>
static cudaError_t launch_uw32_t(const P32 &P, const S32 &S, float *U, int first, cudaStream_t st) {
    const dim3 blk(UBX, UBY), grd((P.nx + UBX - 1) / UBX, (P.ny + UBY - 1) / UBY);
    // 64 registers (a few of HCZ's spilled) where four blocks an SM make fewer rounds, else the
    // 78 that the compiler takes.  Whole step, us: 256x256 14.4 / 15.5 at 64, 384x384 24.2 / 23.5,
    // 512x512 42.0 / 40.8, 2000x2000 613 / 588.
    launch_pdl(grd.x * grd.y <= 3 * 152 ? k_uw32_collide<MODEL, 3> : k_uw32_collide<MODEL, 4>, grd, blk, 0, st, P, S, U,
               first);
    constexpr int FY = 8;
    const int ntx = (P.nx + UTW - 1) / UTW, tiles = ntx * ((P.ny + FY - 3) / (FY - 2));
    // Four resident blocks an SM at 64 registers (a few spilled) or three at 80: three while
    // that makes at most four rounds of the 152 SMs.  256x256 17.3 / 14.4 us a step, 512x512
    // 42.4 / 41.7, 768x768 100 / 108, 2000x2000 604 / 671.
    launch_pdl(tiles <= 4 * 3 * 152 ? k_uw32_tile<MODEL, FY, 3> : k_uw32_tile<MODEL, FY, 4>, dim3(tiles), dim3(UFX, FY),
               0, st, P, S, U, ntx);
    return cudaGetLastError();
}

// One UW step of a periodic FP32 Allen-Cahn case: reads the copy S.df.., writes S.odf..
// (the caller swaps them); U: UW_PLANES scratch planes of S.qs floats.
cudaError_t launch_uw32(const P32 &P, const S32 &S, float *U, int first, cudaStream_t st, int64_t *launches) {
    if (P.walls || !U) return cudaErrorInvalidValue;
    const cudaError_t e = P.model == AC ? launch_uw32_t<AC>(P, S, U, first, st) : launch_uw32_t<HCZ>(P, S, U, first, st);
    if (e == cudaSuccess) *launches += 2;
    return e;
}

}  // namespace f32
}  // namespace dugks
