// Part of fp64_step.cuh, reference-exact variant: equilibria, sources, the collision and the face reconstruction.
// A product by the FP64 pipe (IM = false) or the integer pipe (fp64_imul.cuh); bad: see there.
template <bool IM>
struct Mul {
    uint32_t bad = 0;
    __device__ __forceinline__ double operator()(double a, double b) { return IM ? mul_int(a, b, bad) : a * b; }
};
// A value whose products leave the integer product's window though it is not zero: the phase field
// beyond an interface is 0 at first and then 1e-80, 1e-100, ... one cell further at every step.  A
// warp that holds one takes the floating-point products at once instead of finding `bad` after the
// integer ones.  us per step of a drop of radius about n / 4 at step 4, then at step 200 finding
// `bad` / so: AC 512x512 372, 431 / 396; HCZ 480x480 496, 572 / 524; HCZ 1024x1024 2045, 2492 / 2264;
// with floating-point products only 417, 575 and 2547.  (Below 2^-235: the distributions of a cell are
// up to 36 times smaller than their sum, and more on a steep front.)
__device__ __forceinline__ bool far_tail(double d) {
    const uint32_t hi = (uint32_t)__double2hiint(d) & 0x7fffffffu;
    return hi < (uint32_t)(1023 - 235) << 20 && (hi | (uint32_t)__double2loint(d)) != 0;
}
template <bool IM>
__device__ __forceinline__ bool warp_any(bool b) {
    return IM && __any_sync(__activemask(), b);
}
// tests of the bits: a floating-point comparison occupies the FP64 pipe like an addition
__device__ __forceinline__ bool is_zero(double d) { return ((__double2hiint(d) & 0x7fffffff) | __double2loint(d)) == 0; }
// d = 0 where |d| < 1e-14 (Ark/Header/Mesh_2D.h:196-200)
__device__ __forceinline__ void SetZero(double &d) {
    if ((__double_as_longlong(d) & 0x7fffffffffffffffLL) < __double_as_longlong(1.0E-14)) d = 0.0;
}

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
// then the inverse moment matrix (Ark/Lib/D2V16.cpp:34-52), row by row.
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
    // The matrix has 23 distinct magnitudes up to powers of two (Params::m16), and the four
    // rows of a ring hold the same ones: each product of a magnitude and a moment is formed
    // once, 44 multiplies for the rows' 100 pairs of entries.
    const D2V16Matrix &A = P.m16;
    const double M0 = M[0], M3 = M[3], M5 = M[5], M6 = M[6];
    // the reference's row sums in its order, less the terms of the matrix's structural zeros
    // (a sum that starts at +0 never becomes -0, so adding 0 * M[k] leaves it unchanged for
    // finite moments; a non-finite moment gives a non-finite sum either way); a factor 2^-k
    // of an entry goes into the addition of its product (fma, exact)
    const double n7 = A.N * M[7], n8 = A.N * M[8], n9 = A.N * M[9], n10 = A.N * M[10], n11 = A.N * M[11],
                 n12 = A.N * M[12];
    {   // ring 1
        const double a3 = A.A * M3, g5 = A.G * M5, h5 = A.H * M5, g6 = A.G * M6, h6 = A.H * M6;
        const double t14 = A.T * M[14], t15 = A.T * M[15];
        const double sx_ = a3 + g5 + h6, sy_ = a3 + h5 + g6;
        eq[0] = sx_ + n7 - n9 - n12 + t14 - t15;
        eq[2] = sx_ - n7 + n9 + n12 + t14 - t15;
        eq[1] = sy_ + n8 - n10 - n11 - t14 + t15;
        eq[3] = sy_ - n8 + n10 + n11 - t14 + t15;
    }
    const double f4 = A.F * M[4], p9 = A.Pc * M[9], p10 = A.Pc * M[10], s13 = A.S * M[13], s14 = A.S * M[14],
                 s15 = A.S * M[15];
    {   // ring 2: xu, xv the signs of the direction
        const double m0 = A.c23 * M0, c1 = A.ic * M[1], c2 = A.ic * M[2], b3 = A.B * M3, i5 = A.I * M5, i6 = A.I * M6;
        auto row = [&](double m01, int xu, int xv) {
            double t = m01 + sx(xv, c2) + b3 + sx(xu * xv, f4) + i5 + i6;
            t = __fma_rn(-0.5 * xu, n7, t);
            t = __fma_rn(-0.5 * xv, n8, t);
            t = t + sx(xu, p9) + sx(xv, p10);
            t = __fma_rn(0.5 * xv, n11, t);
            t = __fma_rn(0.5 * xu, n12, t);
            t = t - sx(xu * xv, s13);
            t = __fma_rn(0.5, s14, t);
            return __fma_rn(0.5, s15, t);
        };
        const double mp = m0 + c1, mm = m0 - c1;
        eq[4] = row(mp, 1, 1);
        eq[5] = row(mm, -1, 1);
        eq[6] = row(mm, -1, -1);
        eq[7] = row(mp, 1, -1);
    }
    const double r11 = A.R * M[11], r12 = A.R * M[12];
    {   // ring 3
        const double d3 = A.D * M3, m03 = __fma_rn(-0.5, M0, d3);
        const double sx_ = m03 + A.J * M5 + A.K * M6, sy_ = m03 + A.K * M5 + A.J * M6;
        const double q9 = A.Qc * M[9], q10 = A.Qc * M[10];
        const double u14 = A.U * M[14], v15 = A.V * M[15], v14 = A.V * M[14], u15 = A.U * M[15];
        eq[8] = __fma_rn(-0.125, n7, sx_) + q9 + r12 + u14 + v15;
        eq[10] = __fma_rn(0.125, n7, sx_) - q9 - r12 + u14 + v15;
        eq[9] = __fma_rn(-0.125, n8, sy_) + q10 + r11 + v14 + u15;
        eq[11] = __fma_rn(0.125, n8, sy_) - q10 - r11 + v14 + u15;
    }
    {   // ring 4
        const double m0 = A.c12 * M0, c1 = A.jc * M[1], c2 = A.jc * M[2], e3 = A.E * M3, l5 = A.L * M5, l6 = A.L * M6;
        auto row = [&](double m01, int xu, int xv) {
            double t = m01 - sx(xv, c2) + e3;
            t = __fma_rn(-0.0625 * (xu * xv), f4, t);
            t = t + l5 + l6;
            t = __fma_rn(0.0625 * xu, n7, t);
            t = __fma_rn(0.0625 * xv, n8, t);
            t = __fma_rn(-0.125 * xu, p9, t);
            t = __fma_rn(-0.125 * xv, p10, t);
            t = __fma_rn(-0.5 * xv, r11, t);
            t = __fma_rn(-0.5 * xu, r12, t);
            t = __fma_rn(0.25 * (xu * xv), s13, t);
            t = __fma_rn(0.25, s14, t);
            return __fma_rn(0.25, s15, t);
        };
        const double mp = m0 + c1, mm = m0 - c1;
        eq[12] = row(mm, 1, 1);
        eq[13] = row(mp, -1, 1);
        eq[14] = row(mp, -1, -1);
        eq[15] = row(mm, 1, -1);
    }
}

// D2Q9PP equilibrium (Ark/Lib/D2Q9PP.cpp:51-62).
__device__ __forceinline__ void d2q9pp_eq(const Params &P, double rho, double U, double V, double *eq) {
    const double uuL = (U * U + V * V) * P.Lambda0;
    const Xi4 ur = xi4(U, V, P.RT, P.r_RT);
    eq[0] = d2q9_w(0) * rho * (1.0 - uuL);
#pragma unroll
    for (int q = 1; q <= 4; ++q) {
        const double u1 = ur.get(d2q9_xu(q), d2q9_xv(q)), w2 = u1 * u1, wr = d2q9_w(q) * rho;
        eq[q] = wr * (__fma_rn(0.5, w2, 1.0 + u1) - uuL);
        eq[d2q9_bb(q)] = wr * (__fma_rn(0.5, w2, 1.0 - u1) - uuL);
    }
}

template <int MODEL>
__device__ __forceinline__ void pp_eq(const Params &P, double rho, double U, double V, double *eq) {
    if (MODEL == PP16) d2v16_eq(P, rho, U, V, eq);
    else d2q9pp_eq(P, rho, U, V, eq);
}

// The He-Shan-Doolen projections (xi_q - u).F: the reference's fx (xi_u - U) + fy (xi_v - V),
// whose products are those of the model's few distinct velocity components (D2Q9: -1, 0, 1;
// D2V16: c times -2 .. 2).
template <int MODEL>
__device__ __forceinline__ void pp_src_proj(const Params &P, double fx, double fy, double U, double V, double *pr) {
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    constexpr int K = MODEL == PP16 ? 2 : 1;
    double pu[2 * K + 1], pv[2 * K + 1];
#pragma unroll
    for (int k = -K; k <= K; ++k) {
        const double c = k == 2 || k == -2 ? P.xi_u[8] : P.c16, x = MODEL == PP16 ? sx(k, c) : (double)k;
        pu[k + K] = fx * (k == 0 ? -U : x - U);  // 0 - U as -U
        pv[k + K] = fy * (k == 0 ? -V : x - V);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) pr[q] = pu[vel_u<MODEL>(q) + K] + pv[vel_v<MODEL>(q) + K];
}

// Carnahan-Starling, b = 4 (Ark/Lib/nonidealEoS.h:114-118) and calcPsi
// (Ark/Header/Macroscopic.h:64-68).
__device__ __forceinline__ double cs_pressure(const Params &P, double rho) {
    const double r2 = rho * rho, m = 1.0 - rho;  // R = 1
    return rho * P.T_CS * (1.0 + rho + r2 - r2 * rho) / (m * m * m) - P.aCS * rho * rho;
}
// G = (p > rho RT) - (p < rho RT), psi = sqrt(2 (p - rho RT) / G): the quotient by +-1 is the
// absolute value, by 0 not a number; the sign is read from the bits, 0 also for a difference that
// is not a number
__device__ __forceinline__ void calc_psi(const Params &P, double rho, double p, double &scg, double &psi) {
    const double d = p - rho * P.RT;
    const int hi = __double2hiint(d);
    const bool zero = is_zero(d), nan = (hi & 0x7fffffff) > 0x7ff00000;  // (a sum's NaN is quiet)
    scg = zero || nan ? 0.0 : (hi < 0 ? -1.0 : 1.0);
    const double r = sqrt(2.0 * fabs(d));
    psi = zero ? __hiloint2double(0x7ff80000, 0) : r;
}

// 8-neighbour isotropic gradient (Ark/Lib/GradSchemeBasic.h:153-208).
// d2: 6 2dx (Params g6x / g6y), r: its reciprocal
__device__ __forceinline__ double iso_gx(double E, double W, double NE, double NW, double SE, double SW, double d2,
                                         double r) {
    return QDIV(__fma_rn(4.0, E - W, NE - NW + SE - SW), d2, r);
}
__device__ __forceinline__ double iso_gy(double N, double S, double NE, double NW, double SE, double SW, double d2,
                                         double r) {
    return QDIV(__fma_rn(4.0, N - S, NE - SE + NW - SW), d2, r);
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
    double Phi_x = iso_gx(E, W, NE, NW, SE, SW, P.g6x, P.r_g6x);
    double Phi_y = iso_gy(N, Sd, NE, NW, SE, SW, P.g6y, P.r_g6y);
    const double lap = QDIV(__fma_rn(4.0, E + N + W + Sd, NE + NW + SW + SE) - 20 * phi, P.lap6, P.r_lap);
    SetZero(Phi_x);
    SetZero(Phi_y);
    // phi_L = 1, phi_V = 0
    const double phi1 = phi - 1.0;
    const double F = P.Beta2 * phi1 * phi * __fma_rn(2.0, phi, -1.0) - P.Kappa * lap;
    rhox = P.aPhi * Phi_x;
    rhoy = P.aPhi * Phi_y;
    fx = F * Phi_x;
    fy = F * Phi_y;
    if (P.gravity) fy -= P.Gy * (rho - P.RhoL);
    const double L = sqrt(Phi_x * Phi_x + Phi_y * Phi_y);
    srcx = QDIV(phi * U - ppu_old, P.RTdt, P.r_RTdt);
    srcy = QDIV(phi * V - ppv_old, P.RTdt, P.r_RTdt);
    if (!is_zero(L)) {  // + Phi_x (-4 (phi - phi_L)(phi - phi_V) / (W (phi_L - phi_V))) / L
        const double tmp = QDIV(phi1 * phi, P.wI, P.r_wI);
        const double rL = 1.0 / L;
        srcx = __fma_rn(-4.0, QDIV(Phi_x * tmp, L, rL), srcx);
        srcy = __fma_rn(-4.0, QDIV(Phi_y * tmp, L, rL), srcy);
    }
}

// ---------------------------------------------------------------------------
// Equilibria and sources of opposite directions (q, q'), xi_q = (xu, xv) = -xi_q'.
// HCZ: Update_phi_Eq / Update_phi_Eqh and the sources, Ark/Lib/D2Q9HCZ.cpp:54-131: with u1 =
// xi.u / RT the quadratic part u1^2 / 2 is the same for both, RN(u1 u1) folded with its 1/2.
struct MomHCZ {
    Xi4 ur;                        // (xi.u)/RT
    double uuL, p, rRT;            // |u|^2 Lambda0, pressure, rho RT
    double cuF[3], cuR[3];         // (xu - U) Fx, (xu - U) rho_x for xu = -1, 0, 1
    double cvF[3], cvR[3];         // (xv - V) Fy, (xv - V) rho_y
};
__device__ __forceinline__ void hcz_products(MomHCZ &m, double U, double V, double Fx, double Fy, double Rx, double Ry) {
    const double a = -1.0 - U, b = 1.0 - U, c = -1.0 - V, d = 1.0 - V;
    m.cuF[0] = a * Fx;
    m.cuF[1] = -U * Fx;  // 0 - U as -U
    m.cuF[2] = b * Fx;
    m.cuR[0] = a * Rx;
    m.cuR[1] = -U * Rx;
    m.cuR[2] = b * Rx;
    m.cvF[0] = c * Fy;
    m.cvF[1] = -V * Fy;
    m.cvF[2] = d * Fy;
    m.cvR[0] = c * Ry;
    m.cvR[1] = -V * Ry;
    m.cvR[2] = d * Ry;
}
// Gamma of both directions; ge: the rest direction's -|u|^2 Lambda0
template <typename M>
__device__ __forceinline__ void hcz_gamma(M &mul, const MomHCZ &m, double u1, double &G, double &Go) {
    const double w2 = mul(u1, u1);
    G = __fma_rn(0.5, w2, u1) - m.uuL;
    Go = __fma_rn(0.5, w2, -u1) - m.uuL;
}
template <typename M>
__device__ __forceinline__ double hcz_source(M &mul, const MomHCZ &m, double RT, double G, int xu, int xv) {
    return mul(1 + G, m.cuF[xu + 1] + m.cvF[xv + 1]) + mul(mul(G, RT), m.cuR[xu + 1] + m.cvR[xv + 1]);
}
// (xi.src) of one direction: sum and difference of the components shared by the diagonals
__device__ __forceinline__ double src_dot(int xu, int xv, double sx_, double sy_, double sum, double dif) {
    if (xu != 0 && xv != 0) return xu == xv ? sx(xu, sum) : sx(xv, dif);  // dif = sy - sx
    return xu != 0 ? sx(xu, sx_) : sx(xv, sy_);
}

// ---------------------------------------------------------------------------
// Collision pre-step.  MODEL AC/HCZ: Update_phi_Eq + Update_DVDF_Source +
// Update_phi_BP (Ark/Lib/D2Q9AC.cpp:69-105,331-344, Ark/Lib/D2Q9HCZ.cpp:54-92,
// Ark/Cpp/DUGKS2DSolver.cpp:379-401); PP: Ark/Lib/D2Q9PP.cpp:51-62,137-145.
// do_msrc: run the previous step's MacroSource / pseudopotential cell force
// (Ark/Cpp/PseudoP.cpp:31-38) first.
template <int MODEL, bool WALLS, bool IM>
__global__ void __launch_bounds__(256, IM ? 2 : 1) k_collide(Params P, State S, int do_msrc, int gin, int gout) {
    pdl_wait();
    int i, j;
    if (!cell_of_thread(P, i, j)) return;
    const int pitch = P.pitch;
    const size_t c = (size_t)j * pitch + i;
    const double rho = S.fld[F_RHO][c], U = S.fld[F_U][c], V = S.fld[F_V][c], tau = S.fld[F_TAU][c];
    // (2 tau - hDt) / (2 tau + dt), both sides halved
    const double aBP = (tau - P.hDt2) / (tau + P.hDt), bBP = 1.0 - aBP, cBP = tau * bBP;
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
        double pRT = 0.0;
        Xi4 fr{};
        MomHCZ m;
        if (MODEL == AC) {
            pRT = QDIV(p, P.RT, P.r_RT);
            fr = xi4(fx, fy, P.RT, P.r_RT);
        } else {
            m.ur = xi4(U, V, P.RT, P.r_RT);
            m.uuL = (U * U + V * V) * P.Lambda0;
            hcz_products(m, U, V, fx, fy, rhox, rhoy);
        }
        const double ssum = srcx + srcy, sdif = srcy - srcx;
        const bool far = warp_any<IM>(far_tail(phi) || (MODEL == HCZ && (far_tail(srcx) || far_tail(srcy))));
        // f-bar-plus and h-bar-plus of direction q from its equilibria and sources; hc: the
        // product h_cBP hSo (opposite directions: the negative)
        auto put = [&](auto &mul, int q, double fEq, double fSo, double hEq, double hSo, double hc) {
            const size_t o = (size_t)q * S.qs + c;
            if (WALLS && P.nee && (j == 0 || j == P.ny - 1)) {  // kept for the NEE wall faces
                const size_t wq = ((size_t)(j == 0 ? 0 : 1) * 9 + q) * pitch + i, ws = (size_t)2 * 9 * pitch;
                S.weq[wq] = fEq;
                S.weq[ws + wq] = fSo;
                S.weq[2 * ws + wq] = hEq;
                S.weq[3 * ws + wq] = hSo;
            }
            const double hb = mul(P.h_aBP, S.h[o]) + mul(P.h_bBP, hEq);
            S.bh[o] = q == 0 ? hb : hb + hc;
            S.bf[o] = mul(aBP, S.f[o]) + mul(bBP, fEq) + mul(cBP, fSo);
        };
        Mul<false> fp;
        {   // rest direction: u1 = 0, no phase source
            const double w = d2q9_w(0);
            if (MODEL == AC) {  // u = v = 0 (Ark/Lib/D2Q9AC.cpp:197-198): Gamma = 0, no force term
                const size_t o = c;
                const double fEq = w * pRT - pRT, hEq = w * phi;
                if (WALLS && P.nee && (j == 0 || j == P.ny - 1)) put(fp, 0, fEq, 0.0, hEq, 0.0, 0.0);
                else {
                    S.bh[o] = P.h_aBP * S.h[o] + P.h_bBP * hEq;
                    S.bf[o] = aBP * S.f[o] + bBP * fEq;
                }
            } else {
                const double G = -m.uuL;
                put(fp, 0, w * (p + rho * G * P.RT), w * hcz_source(fp, m, P.RT, G, 0, 0), w * phi, 0.0, 0.0);
            }
        }
#pragma unroll
        for (int q = 1; q <= 4; ++q) {
            const int xu = d2q9_xu(q), xv = d2q9_xv(q), qo = d2q9_bb(q);
            const double w = d2q9_w(q);
            auto pair = [&](auto &mul) {
                const double hSo = mul(src_dot(xu, xv, srcx, srcy, ssum, sdif), w), hc = mul(P.h_cBP, hSo);
                if (MODEL == AC) {
                    const double hEq = mul(w, phi), fEq = mul(w, pRT), fSo = mul(w, fr.get(xu, xv));
                    put(mul, q, fEq, fSo, hEq, hSo, hc);
                    put(mul, qo, fEq, -fSo, hEq, -hSo, -hc);
                } else {
                    const double u1 = m.ur.get(xu, xv);
                    double G, Go;
                    hcz_gamma(mul, m, u1, G, Go);
                    put(mul, q, mul(w, p + mul(mul(rho, G), P.RT)), mul(w, hcz_source(mul, m, P.RT, G, xu, xv)),
                        mul(mul(w, 1.0 + u1), phi), hSo, hc);
                    put(mul, qo, mul(w, p + mul(mul(rho, Go), P.RT)), mul(w, hcz_source(mul, m, P.RT, Go, -xu, -xv)),
                        mul(mul(w, 1.0 - u1), phi), -hSo, -hc);
                }
            };
            Mul<IM> mul;
            if (far) mul.bad = 1;
            else pair(mul);
            if (IM && mul.bad) pair(fp);  // an operand beyond the integer product's window
        }
    } else {
        double fx, fy;
        if (do_msrc) {
            const int nx = P.nx, ny = P.ny;
            const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx), jm = wrapi(j - 1, ny), jp = wrapi(j + 1, ny);
            const double *__restrict__ PS = S.fld[F_PSI];
            auto at = [&](int jj, int ii) { return PS[(size_t)jj * pitch + ii]; };
            const double gx = iso_gx(at(j, ip), at(j, im), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P.g6x, P.r_g6x);
            const double gy = iso_gy(at(jp, i), at(jm, i), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P.g6y, P.r_g6y);
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
        const double rRT = rho * P.RT, inv = 1.0 / rRT;
        double pr[Q];
        pp_src_proj<MODEL>(P, fx, fy, U, V, pr);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const double So = QDIV(pr[q] * eq[q], rRT, inv);
            const size_t o = (size_t)q * S.qs + c;
            S.bf[o] = aBP * S.f[o] + bBP * eq[q] + cBP * So;
        }
    }
}

// ---------------------------------------------------------------------------
// Face reconstruction CD_Interior_phi_Bh (Ark/Cpp/DUGKS2DSolver.cpp:604-687).  The
// reference divides by _dx = xo - xn = -dx (normal) and by 2(x1 - x0) = +-2d (tangential);
// with d = 1 these are exact multiplies, and 0.5a + 0.5b == 0.5(a + b).
//
// The parts of one face and one velocity: s = o + n, the normal difference d = n - o along
// +x / +y (XF: x-face between (im,j) and (i,j); else y-face between (i,j-1) and (i,j)), and
// t, four times the tangential gradient along +y / +x.
// Cells around a face: offsets of the rows j - 1, j, j + 1 (wrapped); EDGE: a row beyond a wall
// may be read, extrapolated by cellv (its 2 a0 - a1 at every load, predicated, made up a third
// of the FP64 instructions when all rows went that way, so the other rows use offsets only).
struct FaceRows {
    int i, im, ip, j;
    size_t rm, r0, rp;
};
__device__ __forceinline__ FaceRows face_rows(const Params &P, int i, int j) {
    FaceRows r;
    r.i = i;
    r.im = wrapi(i - 1, P.nx);
    r.ip = wrapi(i + 1, P.nx);
    r.j = j;
    r.rm = (size_t)wrapi(j - 1, P.ny) * P.pitch;
    r.r0 = (size_t)wrapi(j, P.ny) * P.pitch;
    r.rp = (size_t)wrapi(j + 1, P.ny) * P.pitch;
    return r;
}
template <bool EDGE>
__device__ __forceinline__ double at_row(const Params &P, const double *__restrict__ B, const FaceRows &r, int dj, int i) {
    if (EDGE) return cellv<true>(B, P.ny, P.pitch, r.j + dj, i);
    return B[(dj < 0 ? r.rm : (dj > 0 ? r.rp : r.r0)) + i];
}
template <bool XF, bool EDGE>
__device__ __forceinline__ void face_on(const Params &P, const double *__restrict__ B, const FaceRows &r, double &o,
                                        double &n) {
    o = XF ? at_row<EDGE>(P, B, r, 0, r.im) : at_row<EDGE>(P, B, r, -1, r.i);
    n = at_row<EDGE>(P, B, r, 0, r.i);
}
template <bool XF, bool EDGE>
__device__ __forceinline__ double face_tan(const Params &P, const double *__restrict__ B, const FaceRows &r) {
    if (XF) {
        const double SL = at_row<EDGE>(P, B, r, -1, r.im), SR = at_row<EDGE>(P, B, r, -1, r.i);
        const double NL = at_row<EDGE>(P, B, r, 1, r.im), NR = at_row<EDGE>(P, B, r, 1, r.i);
        return (NR - SR) + (NL - SL);
    }
    const double WB = at_row<EDGE>(P, B, r, -1, r.im), EB = at_row<EDGE>(P, B, r, -1, r.ip);
    const double WT = at_row<EDGE>(P, B, r, 0, r.im), ET = at_row<EDGE>(P, B, r, 0, r.ip);
    return (ET - WT) + (EB - WB);
}
// Twice the half-step value of a D2Q9 velocity xi = (xu, xv), components in {-1, 0, 1} known
// at compile time after unrolling: 2 (0.5 s - hDt (gx xu + gy xv)) = s - (gx xu + gy xv) / 2
// with hDt = 1/4.  A gradient a zero component multiplies is not formed (the product with 0
// and its sum with the other term only decide the sign of a zero result).  1, 3, 5 and 7
// FP64 operations for the rest, the normal, the tangential and the diagonal directions
// (the value itself, with every factor applied: 2, 6, 9 and 12).
template <bool XF, bool EDGE>
__device__ __forceinline__ double face_bh9(const Params &P, const double *__restrict__ B, const FaceRows &r, int xu,
                                           int xv) {
    double o, n;
    face_on<XF, EDGE>(P, B, r, o, n);
    const double s = o + n;
    const int xn = XF ? xu : xv, xt = XF ? xv : xu;
    if (xn == 0 && xt == 0) return s;
    if (xt == 0) return __fma_rn(xn > 0 ? -0.5 : 0.5, n - o, s);
    const double t = face_tan<XF, EDGE>(P, B, r);
    if (xn == 0) return __fma_rn(xt > 0 ? -0.125 : 0.125, t, s);
    const double g = __fma_rn(xt > 0 ? 0.25 : -0.25, t, xn > 0 ? n - o : o - n);
    return __fma_rn(-0.5, g, s);
}

