// Part of fp64_step.cuh, FMA variant: equilibria, sources, the collision and the face reconstruction.
__device__ __forceinline__ void SetZero(double &d) { if (d < 1.0E-14 && d > -1.0E-14) d = 0.0; }  // Ark/Header/Mesh_2D.h:196-200

// (xu*a + xv*b)/RT for the 9 D2Q9 directions from 4 divisions:
// a/RT, b/RT, (a+b)/RT, (b-a)/RT; the other directions are their negatives
// ((-x)/RT == -(x/RT) and -a + -b == -(a+b) exactly), direction 0 gives 0.
struct Xi4 {
    double a, b, s, d;
    __device__ __forceinline__ double get(int xu, int xv) const {
        if (xu == 0 && xv == 0) return 0.0;
        if (xv == 0) return xu > 0 ? a : -a;
        if (xu == 0) return xv > 0 ? b : -b;
        if (xu == xv) return xu > 0 ? s : -s;
        return xv > 0 ? d : -d;  // (-1,1): b - a;  (1,-1): a - b = -(b - a)
    }
};
__device__ __forceinline__ Xi4 xi4(double a, double b, double RT, double invRT) {
    (void)invRT;
    Xi4 r;
    r.a = QDIV(a, RT, invRT);
    r.b = QDIV(b, RT, invRT);
    r.s = QDIV(a + b, RT, invRT);
    r.d = QDIV(b - a, RT, invRT);
    return r;
}

// ---------------------------------------------------------------------------
// D2V16 equilibrium: Macro16 (Ark/Lib/D2V16.cpp:125-145) at T = T0, p = rho R0 T0,
// then the inverse moment matrix by opposite pairs, without the structural zeros (the handle
// checks the matrix's form when it is made).
__device__ __forceinline__ void d2v16_eq(const Params &P, double rho, double u, double v, double *eq) {
    const double degrees = 3.0, degPlus2 = degrees + 2.0;
    const double T = P.T0, p = rho * P.R0 * T;
    const double u2 = u * u, v2 = v * v, RT = P.R0 * T;
    double M[16];
    M[0] = rho;
    M[1] = rho * u;
    M[2] = rho * v;
    M[3] = rho * (degrees * RT + u2 + v2);
    M[4] = M[1] * v;
    M[5] = rho * u2 + p;
    M[6] = rho * v2 + p;
    M[7] = M[1] * (degPlus2 * RT + u2 + v2);
    M[8] = M[2] * (degPlus2 * RT + u2 + v2);
    M[9] = M[1] * (3.0 * RT + u2);
    M[10] = M[2] * (3.0 * RT + v2);
    M[11] = M[2] * (RT + u2);
    M[12] = M[1] * (RT + v2);
    M[13] = ((degrees + 4.0) * RT + u2 + v2) * M[4];
    M[14] = degPlus2 * rho * RT * RT + p * ((degrees + 5.0) * u2 + v2) + rho * u2 * (u2 + v2);
    M[15] = degPlus2 * rho * RT * RT + p * ((degrees + 5.0) * v2 + u2) + rho * v2 * (u2 + v2);
    // per opposite pair the even and odd partial sums over the matrix entries that are not
    // identically zero (d2v16_entry, d2v16_odd_moment): eq_j = E + O, eq_j' = E - O; 100
    // multiply-adds and loads instead of 256
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int jo = d2v16_opp(j);
        if (jo < j) continue;
        double E = 0, O = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            if (!d2v16_entry(j, k)) continue;
            if (d2v16_odd_moment(k)) O += __ldg(P.iM16 + j * 16 + k) * M[k];
            else E += __ldg(P.iM16 + j * 16 + k) * M[k];
        }
        eq[j] = E + O;
        eq[jo] = E - O;
    }
}

// D2Q9PP equilibrium (Ark/Lib/D2Q9PP.cpp:51-62).
__device__ __forceinline__ void d2q9pp_eq(const Params &P, double rho, double U, double V, double *eq) {
    const double uu = U * U + V * V;
    const double invRT = P.r_RT;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int xu = d2q9_xu(q), xv = d2q9_xv(q);
        double u1 = QDIV(sx(xu, U) + sx(xv, V), P.RT, invRT);
        eq[q] = d2q9_w(q) * rho * (1.0 + u1 + 0.5 * u1 * u1 - uu * P.Lambda0);
    }
}

template <int MODEL>
__device__ __forceinline__ void pp_eq(const Params &P, double rho, double U, double V, double *eq) {
    if (MODEL == PP16) d2v16_eq(P, rho, U, V, eq);
    else d2q9pp_eq(P, rho, U, V, eq);
}

// The He-Shan-Doolen projections (xi_q - u).F by opposite pairs, d - w and -d - w with
// d = xi_q.F, w = u.F (xi_q' = -xi_q); a rest direction has -w.
template <int MODEL>
__device__ __forceinline__ void pp_src_proj(const Params &P, double fx, double fy, double U, double V, double *pr) {
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    const double w = fx * U + fy * V;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int qo = MODEL == PP16 ? d2v16_opp(q) : d2q9_bb(q);
        if (qo < q) continue;
        if (qo == q) {
            pr[q] = -w;
            continue;
        }
        const double d = fx * P.xi_u[q] + fy * P.xi_v[q];
        pr[q] = d - w;
        pr[qo] = -d - w;
    }
}

// Carnahan-Starling, b = 4 (Ark/Lib/nonidealEoS.h:114-118) and calcPsi
// (Ark/Header/Macroscopic.h:64-68).
__device__ __forceinline__ double cs_pressure(const Params &P, double rho) {
    return rho * P.R0 * P.T_CS * (1.0 + rho + rho * rho - rho * rho * rho) /
               ((1.0 - rho) * (1.0 - rho) * (1.0 - rho)) -
           P.aCS * rho * rho;
}
__device__ __forceinline__ void calc_psi(const Params &P, double rho, double p, double &scg, double &psi) {
    double G = (double)((p > rho * P.RT) - (p < rho * P.RT));
    scg = G;
    psi = sqrt(2 * (p - rho * P.RT) / G);
}

// 8-neighbour isotropic gradient (Ark/Lib/GradSchemeBasic.h:153-208).
// r: RN(1/(d2 6)) (Params r_g6x / r_g6y)
__device__ __forceinline__ double iso_gx(double E, double W, double NE, double NW, double SE, double SW, double d2,
                                         double r) {
    return QDIV(4 * (E - W) + 1 * (NE - NW + SE - SW), d2 * 6, r);
}
__device__ __forceinline__ double iso_gy(double N, double S, double NE, double NW, double SE, double SW, double d2,
                                         double r) {
    return QDIV(4 * (N - S) + 1 * (NE - SE + NW - SW), d2 * 6, r);
}

// ---------------------------------------------------------------------------
// MacroSource (Ark/Cpp/SourceM.cpp:35-62) with Grad_Phi_6points
// (Ark/Cpp/GradScheme.cpp:347-376).  Ghost phi rows come from the P2
// extrapolation of the step that produced phi (gphi buffer `gin`).
template <bool WALLS>
__device__ __forceinline__ void macro_source(const Params &P, const State &S, int i, int j, int gin, double phi,
                                             double rho, double U, double V, double ppu_old, double ppv_old,
                                             double &srcx, double &srcy, double &rhox, double &rhoy, double &fx,
                                             double &fy) {
    const int nx = P.nx, ny = P.ny, pitch = P.pitch;
    const double *__restrict__ PH = S.fld[F_PHI];
    const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx);
    auto at = [&](int jj, int ii) -> double {
        if (jj < 0) return WALLS ? S.gphi[(size_t)(gin * 2 + 0) * pitch + ii] : PH[(size_t)(ny - 1) * pitch + ii];
        if (jj >= ny) return WALLS ? S.gphi[(size_t)(gin * 2 + 1) * pitch + ii] : PH[ii];
        return PH[(size_t)jj * pitch + ii];
    };
    const double E = at(j, ip), W = at(j, im), N = at(j + 1, i), Sd = at(j - 1, i);
    const double NE = at(j + 1, ip), NW = at(j + 1, im), SW = at(j - 1, im), SE = at(j - 1, ip);
    double Phi_x = iso_gx(E, W, NE, NW, SE, SW, P._2dx, P.r_g6x);
    double Phi_y = iso_gy(N, Sd, NE, NW, SE, SW, P._2dy, P.r_g6y);
    const double lap = QDIV(4 * (E + N + W + Sd) + (NE + NW + SW + SE) - 20 * phi, 6 * P.MinL * P.MinL, P.r_lap);
    SetZero(Phi_x);
    SetZero(Phi_y);
    const double F = 2 * P.Beta * (phi - P.PhiL) * (phi - P.PhiV) * (2 * phi - P.PhiL - P.PhiV) - P.Kappa * lap;
    rhox = P.aPhi * Phi_x;
    rhoy = P.aPhi * Phi_y;
    fx = F * Phi_x;
    fy = F * Phi_y;
    if (P.gravity) fy -= P.Gy * (rho - P.RhoL);
    const double L = sqrt(Phi_x * Phi_x + Phi_y * Phi_y);
    const double dU = phi * U - ppu_old, dV = phi * V - ppv_old;
    if (L != 0) {
        const double tmp = QDIV(-4 * (phi - P.PhiL) * (phi - P.PhiV), P.wI * (P.PhiL - P.PhiV), P.r_wI);
        const double rL = 1.0 / L;
        srcx = QDIV(Phi_x * tmp, L, rL) + QDIV(dU, P.RT * P.dt, P.r_RTdt);
        srcy = QDIV(Phi_y * tmp, L, rL) + QDIV(dV, P.RT * P.dt, P.r_RTdt);
    } else {
        srcx = QDIV(dU, P.RT * P.dt, P.r_RTdt);
        srcy = QDIV(dV, P.RT * P.dt, P.r_RTdt);
    }
}

// ---------------------------------------------------------------------------
// Collision pre-step.  MODEL AC/HCZ: Update_phi_Eq + Update_DVDF_Source +
// Update_phi_BP (Ark/Lib/D2Q9AC.cpp:69-105,331-344, Ark/Lib/D2Q9HCZ.cpp:54-92,
// Ark/Cpp/DUGKS2DSolver.cpp:379-401); PP: Ark/Lib/D2Q9PP.cpp:51-62,137-145.
// do_msrc: run the previous step's MacroSource / pseudopotential cell force
// (Ark/Cpp/PseudoP.cpp:31-38) first.
template <int MODEL, bool WALLS, bool IM>
__global__ void __launch_bounds__(256) k_collide(Params P, State S, int do_msrc, int gin, int gout) {
    pdl_wait();
    int i, j;
    if (!cell_of_thread(P, i, j)) return;
    const int pitch = P.pitch;
    const size_t c = (size_t)j * pitch + i;
    const double rho = S.fld[F_RHO][c], U = S.fld[F_U][c], V = S.fld[F_V][c], tau = S.fld[F_TAU][c];
    const double aBP = (2.0 * tau - P.hDt) / (2.0 * tau + P.dt), bBP = 1.0 - aBP, cBP = tau * bBP;
    if (MODEL == AC || MODEL == HCZ) {
        const double phi = S.fld[F_PHI][c], p = S.fld[F_P][c];
        double srcx, srcy, rhox, rhoy, fx, fy;
        if (do_msrc) {
            const double ppu = S.fld[F_PPU][c], ppv = S.fld[F_PPV][c];
            macro_source<WALLS>(P, S, i, j, gin, phi, rho, U, V, ppu, ppv, srcx, srcy, rhox, rhoy, fx, fy);
            S.fld[F_PHIX][c] = srcx;
            S.fld[F_PHIY][c] = srcy;
            S.fld[F_RHOX][c] = rhox;
            S.fld[F_RHOY][c] = rhoy;
            S.fld[F_FX][c] = fx;
            S.fld[F_FY][c] = fy;
            S.fld[F_PPU][c] = phi * U;
            S.fld[F_PPV][c] = phi * V;
        } else {
            srcx = S.fld[F_PHIX][c];
            srcy = S.fld[F_PHIY][c];
            rhox = S.fld[F_RHOX][c];
            rhoy = S.fld[F_RHOY][c];
            fx = S.fld[F_FX][c];
            fy = S.fld[F_FY][c];
        }
        if (WALLS) {  // P2: ghost phi for the next MacroSource (Ark/Cpp/Boundary.cpp:38-63)
            if (j == 0) S.gphi[(size_t)(gout * 2 + 0) * pitch + i] = 2.0 * phi - S.fld[F_PHI][c + pitch];
            if (j == P.ny - 1) S.gphi[(size_t)(gout * 2 + 1) * pitch + i] = 2.0 * phi - S.fld[F_PHI][c - pitch];
        }
        const double invRT = P.r_RT;
        const double pRT = QDIV(p, P.RT, invRT);
        const double uu = U * U + V * V;
        // (xi.a)/RT for xi in {0,+-1}^2 takes 4 distinct magnitudes; (-x)/RT == -(x/RT)
        Xi4 ur, fr;
        if (MODEL == AC) fr = xi4(fx, fy, P.RT, invRT);
        else ur = xi4(U, V, P.RT, invRT);
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int xu = d2q9_xu(q), xv = d2q9_xv(q);
            const double w = d2q9_w(q);
            double hEq, fEq, fSo;
            if (MODEL == AC) {  // u = v = 0 (Ark/Lib/D2Q9AC.cpp:197-198): Gamma = 0, u1 = 0
                hEq = w * phi;
                fEq = w * pRT;
                if (q == 0) fEq -= pRT;
                fSo = w * fr.get(xu, xv);
            } else {
                const double u1 = ur.get(xu, xv);
                const double G = u1 + 0.5 * u1 * u1 - uu * P.Lambda0;
                const double cu = xu == 0 ? -U : (double)xu - U, cv = xv == 0 ? -V : (double)xv - V;  // 0 - U as -U
                hEq = w * (1.0 + u1) * phi;
                fEq = w * (p + rho * G * P.RT);
                fSo = w * ((1 + G) * (cu * fx + cv * fy) + G * P.RT * (cu * rhox + cv * rhoy));
            }
            const double hSo = (xu != 0 && xv != 0 ? sx(xu, srcx) + sx(xv, srcy)
                                                : (xu != 0 ? sx(xu, srcx) : sx(xv, srcy))) * w;
            const size_t o = (size_t)q * S.qs + c;
            if (WALLS && P.nee && (j == 0 || j == P.ny - 1)) {  // kept for the NEE wall faces
                const size_t wq = ((size_t)(j == 0 ? 0 : 1) * 9 + q) * pitch + i, ws = (size_t)2 * 9 * pitch;
                S.weq[wq] = fEq;
                S.weq[ws + wq] = fSo;
                S.weq[2 * ws + wq] = hEq;
                S.weq[3 * ws + wq] = hSo;
            }
            S.bh[o] = P.h_aBP * S.h[o] + P.h_bBP * hEq + P.h_cBP * hSo;
            S.bf[o] = aBP * S.f[o] + bBP * fEq + cBP * fSo;
        }
    } else {
        double fx, fy;
        if (do_msrc) {
            const int nx = P.nx, ny = P.ny;
            const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx), jm = wrapi(j - 1, ny), jp = wrapi(j + 1, ny);
            const double *__restrict__ PS = S.fld[F_PSI];
            auto at = [&](int jj, int ii) { return PS[(size_t)jj * pitch + ii]; };
            const double gx = iso_gx(at(j, ip), at(j, im), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P._2dx, P.r_g6x);
            const double gy = iso_gy(at(jp, i), at(jm, i), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P._2dy, P.r_g6y);
            const double k = -S.fld[F_SCG][c] * at(j, i);
            fx = gx * k;
            fy = gy * k;
            S.fld[F_FX][c] = fx;
            S.fld[F_FY][c] = fy;
        } else {
            fx = S.fld[F_FX][c];
            fy = S.fld[F_FY][c];
        }
        constexpr int Q = MODEL == PP16 ? 16 : 9;
        double eq[Q];
        pp_eq<MODEL>(P, rho, U, V, eq);
        const double inv = 1.0 / (rho * P.RT);
        double pr[Q];
        pp_src_proj<MODEL>(P, fx, fy, U, V, pr);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const double So = pr[q] * eq[q] * inv;
            const size_t o = (size_t)q * S.qs + c;
            S.bf[o] = aBP * S.f[o] + bBP * eq[q] + cBP * So;
        }
    }
}

// ---------------------------------------------------------------------------
// Face reconstruction CD_Interior_phi_Bh (Ark/Cpp/DUGKS2DSolver.cpp:604-687)
// for velocity q of one face.  XF: x-face between L=(im,j) and R=(i,j);
// else y-face between B=(i,j-1) and T=(i,j).
template <bool XF, bool WALLS>
__device__ __forceinline__ double face_bh(const Params &P, const double *__restrict__ B, int i, int im, int ip,
                                          int j, double xu, double xv) {
    const int ny = P.ny, pitch = P.pitch;
    // Denominators: the reference divides by _dx = xo - xn = -dx (normal) and by
    // 2(x1 - x0) = +-2d (tangential).  With d = 1
    // the division is the exact multiply by the reciprocal, and
    // 0.5a + 0.5b == 0.5(a + b) exactly (power-of-two scaling commutes with
    // rounding away from the subnormal range), so these forms round alike.
    double o, n, gx, gy;
    if (XF) {
        o = cellv<WALLS>(B, ny, pitch, j, im);
        n = cellv<WALLS>(B, ny, pitch, j, i);
        const double SL = cellv<WALLS>(B, ny, pitch, j - 1, im), SR = cellv<WALLS>(B, ny, pitch, j - 1, i);
        const double NL = cellv<WALLS>(B, ny, pitch, j + 1, im), NR = cellv<WALLS>(B, ny, pitch, j + 1, i);
        gy = (0.5 * ((NR - SR) + (NL - SL))) * P.r_2dy;
        gx = (o - n) * P.r_ndx;
    } else {
        o = cellv<WALLS>(B, ny, pitch, j - 1, i);
        n = cellv<WALLS>(B, ny, pitch, j, i);
        const double WB = cellv<WALLS>(B, ny, pitch, j - 1, im), EB = cellv<WALLS>(B, ny, pitch, j - 1, ip);
        const double WT = cellv<WALLS>(B, ny, pitch, j, im), ET = cellv<WALLS>(B, ny, pitch, j, ip);
        gx = (0.5 * ((WT - ET) + (WB - EB))) * P.r_n2dx;
        gy = (o - n) * P.r_ndy;
    }
    return 0.5 * (o + n) - P.hDt * (gx * xu + gy * xv);
}

// The parts of one face and one velocity: s = o + n, the normal difference d = n - o along
// +x / +y (XF: x-face between (im,j) and (i,j); else y-face between (i,j-1) and (i,j)), and
// t, four times the tangential gradient along +y / +x.
template <bool XF, bool WALLS>
__device__ __forceinline__ void face_on(const Params &P, const double *__restrict__ B, int i, int im, int j, double &o,
                                        double &n) {
    o = XF ? cellv<WALLS>(B, P.ny, P.pitch, j, im) : cellv<WALLS>(B, P.ny, P.pitch, j - 1, i);
    n = cellv<WALLS>(B, P.ny, P.pitch, j, i);
}
template <bool XF, bool WALLS>
__device__ __forceinline__ double face_tan(const Params &P, const double *__restrict__ B, int i, int im, int ip,
                                           int j) {
    const int ny = P.ny, pitch = P.pitch;
    if (XF) {
        const double SL = cellv<WALLS>(B, ny, pitch, j - 1, im), SR = cellv<WALLS>(B, ny, pitch, j - 1, i);
        const double NL = cellv<WALLS>(B, ny, pitch, j + 1, im), NR = cellv<WALLS>(B, ny, pitch, j + 1, i);
        return (NR - SR) + (NL - SL);
    }
    const double WB = cellv<WALLS>(B, ny, pitch, j - 1, im), EB = cellv<WALLS>(B, ny, pitch, j - 1, ip);
    const double WT = cellv<WALLS>(B, ny, pitch, j, im), ET = cellv<WALLS>(B, ny, pitch, j, ip);
    return (ET - WT) + (EB - WB);
}
// Twice the half-step value of a D2Q9 velocity xi = (xu, xv), components in {-1, 0, 1} known
// at compile time after unrolling: 2 (0.5 s - hDt (gx xu + gy xv)) = s - (gx xu + gy xv) / 2
// with hDt = 1/4.  A gradient a zero component multiplies is not formed (the product with 0
// and its sum with the other term only decide the sign of a zero result).  1, 3, 5 and 7
// FP64 operations for the rest, the normal, the tangential and the diagonal directions
// (the value itself, with every factor applied: 2, 6, 9 and 12).
template <bool XF, bool WALLS>
__device__ __forceinline__ double face_bh9(const Params &P, const double *__restrict__ B, int i, int im, int ip,
                                           int j, int xu, int xv) {
    double o, n;
    face_on<XF, WALLS>(P, B, i, im, j, o, n);
    const double s = o + n;
    const int xn = XF ? xu : xv, xt = XF ? xv : xu;
    if (xn == 0 && xt == 0) return s;
    if (xt == 0) return __fma_rn(xn > 0 ? -0.5 : 0.5, n - o, s);
    const double t = face_tan<XF, WALLS>(P, B, i, im, ip, j);
    if (xn == 0) return __fma_rn(xt > 0 ? -0.125 : 0.125, t, s);
    const double g = __fma_rn(xt > 0 ? 0.25 : -0.25, t, xn > 0 ? n - o : o - n);
    return __fma_rn(-0.5, g, s);
}

