// FP32 deviation-storage step of the pseudopotential models (D2Q9PP, D2V16).
//
// The reference's face force reads the face psi of the neighbouring faces of
// the same step (Ark/Cpp/PseudoP.cpp:39-46, Jacobi semantics: all face psi
// first, then the face forces), so face pass 1 (reconstruction, face moments, face
// psi) of every face precedes face pass 2 (face force, equilibrium, He-Shan-Doolen
// source, flux) of any.  Two launches: the collision (with the cell force from the psi of
// the previous update) with face pass 1, and face pass 2 with the update (the fluxes of a
// tile in shared memory; with the cell macros, pressure and psi).
//
// Storage: the density rho in FP64 and f as the FP32 remainders g_q = f_q - e_q rho,
// e_q = eq_q(1, 0, 0) the rest equilibrium per unit density.  At rest f = e rho, so
// the g_q are small (the equilibrium's velocity part and the non-equilibrium part)
// where deviations from one global rest state would span the liquid-vapour density
// difference.  The step carries the e_q rho part in closed form: the collision keeps
// it (sum_q (B - f) = 0), the faces reconstruct it from the FP64 density and work
// relative to e_q times the face average of rho, and the update changes rho by the
// sum of the small face fluxes (the e_q avg(rho) parts cancel: sum_q e_q xi_q = 0)
// and each g_q by small increments.  Moment sums and the equation of state are
// float-float (below).
// (Fusing face pass 2 with the update saved the fluxes' round trip through DRAM, ~0.2 KB
// per cell-update, for 0.8 % of the D2V16 step: the passes are latency- as much as
// bandwidth-bound.  An earlier fusion that recomputed the face reconstruction instead of
// reading it ran slower.)
#include <cuda_runtime.h>

#include <cstdint>

#include "fp32_pp.cuh"
#include "pdl.cuh"

namespace dugks {
namespace f32 {

// 8-neighbour isotropic gradient of a periodic field given as float-float pairs (hi,
// lo planes), from pair differences (Ark/Lib/GradSchemeBasic.h:153-208)
__device__ __forceinline__ void iso_grad(const PPP &P, const float *__restrict__ a, const float *__restrict__ al,
                                         int i, int j, float &gx, float &gy) {
    const int nx = P.nx, ny = P.ny, pitch = P.pitch;
    const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx), jm = wrapi(j - 1, ny), jp = wrapi(j + 1, ny);
    auto at = [&](int jj, int ii) {
        const size_t o = (size_t)jj * pitch + ii;
        return make_float2(a[o], al[o]);
    };
    pp_iso_grad(P, at(j, ip), at(j, im), at(jp, i), at(jm, i), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), gx, gy);
}

// Collision and face pass 1 of a 32x8-cell tile by one or two groups of 256 threads.
// Collision: the cell force F = -G psi grad psi (Ark/Cpp/PseudoP.cpp:31-38, from the previous
// update's psi) when do_msrc, else the stored force; f-bar-plus remainders to shared memory and
// to S.bf for the update.  The first group does the tile's cells, the second (or the first
// again) the ring of one cell around it, which the neighbouring tiles do too, with the same
// results.
// Face pass 1, after a block barrier: half-step reconstruction, face moments with the previous
// face force, face pressure and psi (Ark/Lib/D2Q9PP.cpp:110-136, Ark/Cpp/PseudoP.cpp:23-30),
// stored relative to e_q times the face average of rho; the first group the west faces of the
// tile's cells, the second (or the first then) the south faces.
// As two launches the face pass read the remainders of a face's cells and of their four
// neighbours from L2 and DRAM, the x and the y faces in different blocks.  Bounded by latency at
// 16 to 40 warps an SM and, on small grids, by the launches: 150x150 D2V16 15.6 -> 11.8 us a
// step, D2Q9 15.3 -> 12.0; 1024x1024 214 -> 200 and 148 -> 141.
template <int MODEL, int GROUPS, int MIN_BLOCKS>
__global__ void __launch_bounds__(256 * GROUPS, MIN_BLOCKS) k_pp32_faces1(PPP P, PPS S, int do_msrc) {
    pdl_wait();
    constexpr int Q = PPQ<MODEL>::Q;
    __shared__ float s[Q][10][34];  // f-bar-plus of the tile and its ring
    const int tx = threadIdx.x, r = threadIdx.y & 7, t = r * 32 + tx;
    const bool first = threadIdx.y < 8;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 8;
    const int nx = P.nx, ny = P.ny, pitch = P.pitch;
    const int w = min(32, nx - x0), h = min(8, ny - y0);
    const bool in = tx < w && r < h;
    // collides the cell at (cx, cy) from the tile's corner
    auto collide = [&](int cx, int cy, bool own) {
        const int i = wrapi(x0 + cx, nx), j = wrapi(y0 + cy, ny);
        const size_t c = (size_t)j * pitch + i;
        float g[Q], bf[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) g[q] = S.df[(size_t)q * S.qs + c];
        float fx, fy;
        if (do_msrc) {
            float gx, gy;
            iso_grad(P, S.psi, S.psil, i, j, gx, gy);
            const float k = -S.scg[c] * S.psi[c];
            fx = gx * k;
            fy = gy * k;
            if (own) {
                S.Fx[c] = fx;
                S.Fy[c] = fy;
            }
        } else {
            fx = S.Fx[c];
            fy = S.Fy[c];
        }
        pp_collide<MODEL>(P, g, (float)S.rho[c], (float)S.U[c], (float)S.V[c], fx, fy, bf);
#pragma unroll
        for (int q = 0; q < Q; ++q) s[q][cy + 1][cx + 1] = bf[q];
        if (own) {
#pragma unroll
            for (int q = 0; q < Q; ++q) S.bf[(size_t)q * S.qs + c] = bf[q];
        }
    };
    // the ring: its row below (34 cells), its row above (34), its west and its east column (8 each)
    const int rx = t < 34 ? t - 1 : t < 68 ? t - 35 : t < 76 ? -1 : w;
    const int ry = t < 34 ? -1 : t < 68 ? h : t < 76 ? t - 68 : t - 76;
    const bool ring = t < 84 && rx <= w && (t < 68 || ry < h);
    if (GROUPS == 2) {
        if (first ? in : ring) collide(first ? tx : rx, first ? r : ry, first);
    } else {
#pragma unroll 1
        for (int k = 0; k < 2; ++k)
            if (k == 0 ? in : ring) collide(k == 0 ? tx : rx, k == 0 ? r : ry, k == 0);
    }
    __syncthreads();
    if (!in) return;
    const int i = x0 + tx, j = y0 + r;
    const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx), jm = wrapi(j - 1, ny), jp = wrapi(j + 1, ny);
    const size_t c = (size_t)j * pitch + i;
    auto rh = [&](int jj, int ii) { return S.rho[(size_t)jj * pitch + ii]; };
    float o[Q], n[Q], tn[Q], to[Q], b[Q];
    if (GROUPS == 1 || first) {  // between (i-1, j) and (i, j)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            o[q] = s[q][r + 1][tx];
            n[q] = s[q][r + 1][tx + 1];
            tn[q] = s[q][r + 2][tx + 1] - s[q][r][tx + 1];
            to[q] = s[q][r + 2][tx] - s[q][r][tx];
        }
        const double ro = rh(j, im), rn = rh(j, i);
        const float rt = (float)((rh(jp, i) - rh(jm, i)) + (rh(jp, im) - rh(jm, im)));
        const PPFace f = pp_face1<MODEL, true>(P, o, n, tn, to, ro + rn, (float)(rn - ro), rt, S.xFx[c], S.xFy[c], b);
#pragma unroll
        for (int q = 0; q < Q; ++q)  // what face pass 2 reads
            if (lat_u<MODEL>(q) != 0) S.xb[(size_t)q * S.qs + c] = b[q];
        S.xpsl[c] = f.psil;
        S.xr[c] = f.dr;
        S.xfl[c] = f.R;
        S.xu[c] = f.U;
        S.xv[c] = f.V;
        S.xg[c] = f.scg;
        S.xps[c] = f.psi;
    }
    if (GROUPS == 1 || !first) {  // between (i, j-1) and (i, j)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            o[q] = s[q][r][tx + 1];
            n[q] = s[q][r + 1][tx + 1];
            tn[q] = s[q][r + 1][tx] - s[q][r + 1][tx + 2];
            to[q] = s[q][r][tx] - s[q][r][tx + 2];
        }
        const double ro = rh(jm, i), rn = rh(j, i);
        const float rt = (float)((rh(j, im) - rh(j, ip)) + (rh(jm, im) - rh(jm, ip)));
        const PPFace f = pp_face1<MODEL, false>(P, o, n, tn, to, ro + rn, (float)(rn - ro), rt, S.yFx[c], S.yFy[c], b);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (lat_v<MODEL>(q) != 0) S.yb[(size_t)q * S.qs + c] = b[q];
        S.ypsl[c] = f.psil;
        S.yr[c] = f.dr;
        S.yfl[c] = f.R;
        S.yu[c] = f.U;
        S.yv[c] = f.V;
        S.yg[c] = f.scg;
        S.yps[c] = f.psi;
    }
}

// Face pass 2 of the x face (XF) or y face at (i, j): face force from the face-psi
// stencil (Ark/Cpp/PseudoP.cpp:39-46, Ark/Lib/GradSchemeBasic.h:181-208), stored for the
// next step's face moments when own; equilibrium, source and the fluxes xi.n into out.
template <int MODEL, bool XF>
__device__ __forceinline__ void pp_face2_at(const PPP &P, const PPS &S, int i, int j, bool own,
                                            float (&out)[PPQ<MODEL>::Q]) {
    constexpr int Q = PPQ<MODEL>::Q;
    const size_t c = (size_t)j * P.pitch + i;
    float gx, gy;
    iso_grad(P, XF ? S.xps : S.yps, XF ? S.xpsl : S.ypsl, i, j, gx, gy);
    const float k = -(XF ? S.xg : S.yg)[c] * (XF ? S.xps : S.yps)[c];
    const float Fx = gx * k, Fy = gy * k;
    if (own) {
        (XF ? S.xFx : S.yFx)[c] = Fx;
        (XF ? S.xFy : S.yFy)[c] = Fy;
    }
    PPFace f;
    f.dr = (XF ? S.xr : S.yr)[c];
    f.U = (XF ? S.xu : S.yu)[c];
    f.V = (XF ? S.xv : S.yv)[c];
    f.R = (XF ? S.xfl : S.yfl)[c];
    const float *__restrict__ B = XF ? S.xb : S.yb;
    float b[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
        if ((XF ? lat_u<MODEL>(q) : lat_v<MODEL>(q)) != 0) b[q] = B[(size_t)q * S.qs + c];
    pp_face2<MODEL, XF>(P, b, f, Fx, Fy, out);
}

// Face pass 2 and the update (Ark/Cpp/DUGKS2DSolver.cpp:748-792) with the cell macros
// (Ark/Lib/D2Q9PP.cpp:89-109) in one launch: a block of 32x8 threads owns a 32x8-cell tile;
// each thread computes the fluxes of its cell's west and south faces into shared memory (by two
// groups of 256 threads: the first the west faces, the second the south faces), 40 threads those of the tile's east column and north row (the next tiles' own faces,
// whose forces those tiles store), and after a block barrier each thread updates its cell
// from the four faces' fluxes, which never reach DRAM:
//   rho_new = rho + drho, drho = dt/V sum_q (net face flux of q),
//   g_q,new = g_q + 4/3 (b_q - g_q) + dt/V (net flux of q)
//             + e_q (xi_q,x px + xi_q,y py) - e_q drho,
// px = dt/V (rho_W - rho_E)/2, py = dt/V (rho_S - rho_N)/2 (the e_q avg(rho) flux
// divergence on unit cells, from the FP64 density); U, V, p, psi from float-float
// sums, rho in FP64.
template <int MODEL, int GROUPS, int MIN_BLOCKS>
__global__ void __launch_bounds__(256 * GROUPS, MIN_BLOCKS) k_pp32_faces2u(PPP P, PPS S) {
    pdl_wait();
    constexpr int Q = PPQ<MODEL>::Q;
    __shared__ float xs[Q][8][33];  // x-face fluxes of the tile's rows, columns 0 .. 32
    __shared__ float ys[Q][9][32];  // y-face fluxes of the tile's columns, rows 0 .. 8
    const int tx = threadIdx.x, ty = threadIdx.y & 7, t = ty * 32 + tx;
    const bool first = threadIdx.y < 8, do_x = GROUPS == 1 || first, do_y = GROUPS == 1 || !first;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 8;
    const int w = min(32, P.nx - x0), h = min(8, P.ny - y0);
    const int i = x0 + tx, j = y0 + ty;
    const bool in = tx < w && ty < h;
    float out[Q];
    if (in && do_x) {
        pp_face2_at<MODEL, true>(P, S, i, j, true, out);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (lat_u<MODEL>(q) != 0) xs[q][ty][tx] = out[q];
    }
    if (in && do_y) {
        pp_face2_at<MODEL, false>(P, S, i, j, true, out);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (lat_v<MODEL>(q) != 0) ys[q][ty][tx] = out[q];
    }
    const int ne = GROUPS == 1 ? 32 : 0;  // first thread of the north row's faces
    if (do_x && t < h) {  // x faces east of the tile (column x0 + w, periodic)
        pp_face2_at<MODEL, true>(P, S, wrapi(x0 + w, P.nx), y0 + t, false, out);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (lat_u<MODEL>(q) != 0) xs[q][t][w] = out[q];
    } else if (do_y && t >= ne && t < ne + w) {  // y faces north of the tile (row y0 + h, periodic)
        pp_face2_at<MODEL, false>(P, S, x0 + t - ne, wrapi(y0 + h, P.ny), false, out);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (lat_v<MODEL>(q) != 0) ys[q][h][t - ne] = out[q];
    }
    __syncthreads();
    if (!in || !first) return;
    const int pitch = P.pitch;
    const int ip = wrapi(i + 1, P.nx), im = wrapi(i - 1, P.nx), jn = wrapi(j + 1, P.ny), js = wrapi(j - 1, P.ny);
    const size_t c = (size_t)j * pitch + i;
    const float hdv = 0.5f * P.dtV;
    const float px = hdv * (float)(S.rho[(size_t)j * pitch + im] - S.rho[(size_t)j * pitch + ip]);
    const float py = hdv * (float)(S.rho[(size_t)js * pitch + i] - S.rho[(size_t)jn * pitch + i]);
    float g[Q], bf[Q], fw[Q], fe[Q], fs[Q], fn[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const size_t o = (size_t)q * S.qs;
        g[q] = S.df[o + c];
        bf[q] = S.bf[o + c];
        if (lat_u<MODEL>(q) != 0) {
            fw[q] = xs[q][ty][tx];
            fe[q] = xs[q][ty][tx + 1];
        }
        if (lat_v<MODEL>(q) != 0) {
            fs[q] = ys[q][ty][tx];
            fn[q] = ys[q][ty + 1][tx];
        }
    }
    const PPCell n = pp_update<MODEL>(P, g, bf, fw, fe, fs, fn, S.rho[c], px, py, S.Fx[c], S.Fy[c]);
#pragma unroll
    for (int q = 0; q < Q; ++q) S.df[(size_t)q * S.qs + c] = g[q];
    S.rho_o[c] = n.rho;
    S.psil[c] = n.psil;
    S.U[c] = n.U;
    S.V[c] = n.V;
    S.p[c] = n.p;
    S.scg[c] = n.scg;
    S.psi[c] = n.psi;
}

// One FP64 distribution plane f_q [ny][nx] (dense, as the C ABI passes it) as the
// stored remainder g_q = f_q - e_q rho, rho the FP64 density [ny][pitch]
__global__ void __launch_bounds__(256) k_pp_g_from_f64(float *g, int pitch, const double *__restrict__ f,
                                                       const double *__restrict__ rho, int nx, int ny, double e) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (i >= nx || j >= ny) return;
    const size_t d = (size_t)j * pitch + i;
    g[d] = (float)__dsub_rn(f[(size_t)j * nx + i], __dmul_rn(e, rho[d]));
}

cudaError_t launch_pp_g_from_f64(float *g, int pitch, const double *f, const double *rho, int nx, int ny, double e,
                                 cudaStream_t st, int64_t *launches) {
    const dim3 grd((nx + 255) / 256, ny);
    k_pp_g_from_f64<<<grd, 256, 0, st>>>(g, pitch, f, rho, nx, ny, e);
    *launches += 1;
    return cudaGetLastError();
}

// the cell force of the current psi (the state the reference holds after a step)
__global__ void __launch_bounds__(256) k_pp32_force(PPP P, PPS S) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= P.nx || j >= P.ny) return;
    const size_t c = (size_t)j * P.pitch + i;
    float gx, gy;
    iso_grad(P, S.psi, S.psil, i, j, gx, gy);
    const float k = -S.scg[c] * S.psi[c];
    S.Fx[c] = gx * k;
    S.Fy[c] = gy * k;
}

template <int MODEL>
static cudaError_t launch_pp_t(const PPP &P, const PPS &S, int do_msrc, cudaStream_t st, int64_t *launches,
                               uint32_t step) {
    const dim3 blk(32, 8);
    const dim3 grd((P.nx + 31) / 32, (P.ny + 7) / 8);
    (void)step;
    const unsigned blocks = grd.x * grd.y;
    // Two groups of threads where the blocks are few: each SM's share then takes the latency of
    // one face instead of two.  One group on large grids, at the registers it runs best with
    // (D2V16 three blocks an SM without spills, D2Q9 five).  us per step, two groups / one:
    // D2V16 150x150 11.8 / 15.9, 330x330 (451 blocks) 26.0 / 26.9, 1024x1024 206 / 200;
    // D2Q9 150x150 12.0 / 13.8, 330x330 22.1 / 25.3, 360x360 24.1 / 25.3, 400x400 28.6 / 27.0,
    // 1024x1024 160 / 141 (four blocks 143, three 155).
    if (blocks <= 3 * 152) launch_pdl(k_pp32_faces1<MODEL, 2, 2>, grd, dim3(32, 16), 0, st, P, S, do_msrc);
    else launch_pdl(k_pp32_faces1<MODEL, 1, MODEL == PP16 ? 3 : 5>, grd, blk, 0, st, P, S, do_msrc);
    // face pass 2 compiled for three (D2Q9: four) resident blocks of 256 threads where the grid
    // fills them, with more registers for the few blocks of a small one (D2V16, us per step:
    // when the step had three launches, 1024x1024 212 / 225, 400x400 35.6 / 38.2, 150x150 17.6 /
    // 15.7).
    // Two groups for it too, on D2Q9 grids of one round of such blocks, two an SM (one group /
    // two: 150x150 11.8 / 10.2, 256x256 16.6 / 14.8, 300x300 21.4 / 21.5), and for D2V16, whose
    // threads need the registers of a whole SM then, where every block has one even when placed
    // ahead of the launch before (128x128 12.1 / 11.4, 141x141, 90 blocks, 12.3 / 15.0).
    const dim3 blk2(32, 16);
    if (MODEL == PP16 ? blocks <= 76 : blocks <= 2 * 152)
        launch_pdl(k_pp32_faces2u<MODEL, 2, MODEL == PP16 ? 1 : 2>, grd, blk2, 0, st, P, S);
    else if (MODEL == PP16 && blocks <= 2 * 152) launch_pdl(k_pp32_faces2u<PP16, 1, 2>, grd, blk, 0, st, P, S);
    else launch_pdl(k_pp32_faces2u<MODEL, 1, MODEL == PP16 ? 3 : 4>, grd, blk, 0, st, P, S);
    *launches += 2;
    return cudaGetLastError();
}

cudaError_t launch_pp32_step(const PPP &P, const PPS &S, int do_msrc, cudaStream_t st, int64_t *launches,
                             uint32_t step) {
    return P.model == PP16 ? launch_pp_t<PP16>(P, S, do_msrc, st, launches, step)
                           : launch_pp_t<PP9>(P, S, do_msrc, st, launches, step);
}

cudaError_t launch_pp32_force(const PPP &P, const PPS &S, cudaStream_t st, int64_t *launches) {
    const dim3 blk(32, 8);
    const dim3 grd((P.nx + 31) / 32, (P.ny + 7) / 8);
    k_pp32_force<<<grd, blk, 0, st>>>(P, S);
    *launches += 1;
    return cudaGetLastError();
}

}  // namespace f32
}  // namespace dugks
