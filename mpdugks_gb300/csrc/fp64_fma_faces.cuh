// Part of fp64_step.cuh, FMA variant: the face kernels and the update.
// Allen-Cahn face: Update_MacroVar_h + Update_phi_Eqh + Update_DVDF_Source_h
// + Update_phi_h + Update_phiFlux_h (+ Wall_3_BB) -- Ark/Lib/D2Q9AC.cpp:106-144,
// 232-329,345-358; Ark/Lib/D2Q9HCZ.cpp:93-131,183-271;
// Ark/Cpp/DUGKS2DSolver.cpp:402-441; Ark/Cpp/Boundary.cpp:118-139.
// UW: the threads after the faces do the x and y periodic boundary faces in the
// reference's low-side form (column 0 / row 0 only), written to xlo / ylo.
template <int MODEL, bool WALLS, bool UW, bool XF>
__device__ __forceinline__ void face_ac(const Params &P, const State &S, int i, int j, bool lo, bool xrt) {
    const bool xf = WALLS ? xrt : XF;
    const int nx = P.nx, ny = P.ny, pitch = P.pitch;
    const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx);
    // owner/neighbour cells of this face and the averaged source fields
    int jo, io;
    if (xf) { jo = j; io = im; } else { jo = j - 1; io = i; }
    if (UW && jo < 0) jo += ny;  // periodic y (UW runs without walls)
    double avg[6];
    const int fid[6] = {F_PHIX, F_PHIY, F_RHOX, F_RHOY, F_FX, F_FY};
#pragma unroll
    for (int k = 0; k < 6; ++k)
        avg[k] = 0.5 * (cellv<WALLS>(S.fld[fid[k]], ny, pitch, jo, io) + cellv<WALLS>(S.fld[fid[k]], ny, pitch, j, i));
    const double Phi_x = avg[0], Phi_y = avg[1], Rho_x = avg[2], Rho_y = avg[3], Fx = avg[4], Fy = avg[5];
    double bf[9], bh[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const double xu = d2q9_xu(q), xv = d2q9_xv(q);
        if (UW) {
            const size_t qo = (size_t)q * S.qs;
            const size_t co = (size_t)jo * pitch + io, cn = (size_t)j * pitch + i;
            if (xf) {
                bf[q] = face_uw<true>(P, S.bf + qo, S.gfx + qo, S.gfy + qo, co, cn, xu, xv, lo);
                bh[q] = face_uw<true>(P, S.bh + qo, S.ghx + qo, S.ghy + qo, co, cn, xu, xv, lo);
            } else {
                bf[q] = face_uw<false>(P, S.bf + qo, S.gfx + qo, S.gfy + qo, co, cn, xu, xv, lo);
                bh[q] = face_uw<false>(P, S.bh + qo, S.ghx + qo, S.ghy + qo, co, cn, xu, xv, lo);
            }
        } else if (xf) {
            bf[q] = face_bh9<true, WALLS>(P, S.bf + (size_t)q * S.qs, i, im, ip, j, d2q9_xu(q), d2q9_xv(q));
            bh[q] = face_bh9<true, WALLS>(P, S.bh + (size_t)q * S.qs, i, im, ip, j, d2q9_xu(q), d2q9_xv(q));
        } else {
            bf[q] = face_bh9<false, WALLS>(P, S.bf + (size_t)q * S.qs, i, im, ip, j, d2q9_xu(q), d2q9_xv(q));
            bh[q] = face_bh9<false, WALLS>(P, S.bh + (size_t)q * S.qs, i, im, ip, j, d2q9_xu(q), d2q9_xv(q));
        }
    }
    // the CD reconstruction gives twice the face values: b = SC times the stored number
    constexpr double SC = UW ? 1.0 : 0.5;
    double Phi = bh[0], sumf = bf[0];
#pragma unroll
    for (int q = 1; q < 9; ++q) Phi += bh[q];
#pragma unroll
    for (int q = 1; q < 9; ++q) sumf += bf[q];
    Phi *= SC;
    const double Rho = P.aPhi * Phi + P.bPhi;
    const double invRT = P.r_RT;
    double U, V, p, Mu, tauh;
    if (MODEL == AC) {
        U = 0.0;
        V = 0.0;
        p = (sumf - bf[0]) * (UW ? P.Kp : P.Kp2);  // the u-dependent terms vanish with u = 0
        Mu = Rho * P.RT * P.Tau0;
        tauh = Mu / (Rho * P.RT);
    } else {
        // first moments over the directions with a nonzero component (the others add +-0)
        double su = 0, sv = 0;
#pragma unroll
        for (int q = 0; q < 9; ++q)
            if (d2q9_xu(q) != 0) su += sx(d2q9_xu(q), bf[q]);
#pragma unroll
        for (int q = 0; q < 9; ++q)
            if (d2q9_xv(q) != 0) sv += sx(d2q9_xv(q), bf[q]);
        sumf *= SC;
        su *= SC;
        sv *= SC;
        const double inv = 1.0 / (Rho * P.RT);
        U = QDIV(su, Rho * P.RT, inv);
        V = QDIV(sv, Rho * P.RT, inv);
        U += QDIV(0.5 * P.hDt * Fx, Rho * P.RT, inv);
        V += QDIV(0.5 * P.hDt * Fy, Rho * P.RT, inv);
        p = __fma_rn(0.5 * P.hDt * P.RT, Rho_x * U + Rho_y * V, sumf);
        Mu = P.NuV + (Phi - P.PhiV) * (P.NuL - P.NuV);
        Mu *= Rho;
        tauh = QDIV(Mu, Rho * P.RT, inv);
    }
    const double ah = 2.0 * tauh / (2.0 * tauh + P.hDt), bh_ = 1.0 - ah, ch = tauh * bh_;
    const double ahs = SC * ah, hah = UW ? P.h_ah : P.h_ah2;
    const double uu = U * U + V * V;
    const double pRT = QDIV(p, P.RT, invRT);
    Xi4 ur, fr;
    if (MODEL == AC) fr = xi4(Fx, Fy, P.RT, invRT);
    else ur = xi4(U, V, P.RT, invRT);
    double hf[9], hh[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int xu = d2q9_xu(q), xv = d2q9_xv(q);
        if (!WALLS && (xf ? xu : xv) == 0) continue;  // does not cross the face
        const double w = d2q9_w(q);
        double hEq, fEq, fSo;
        if (MODEL == AC) {
            hEq = w * Phi;
            fEq = w * pRT;
            if (q == 0) fEq -= pRT;
            fSo = w * fr.get(xu, xv);
        } else {
            const double u1 = ur.get(xu, xv);
            const double G = u1 + 0.5 * u1 * u1 - uu * P.Lambda0;
            const double cu = xu == 0 ? -U : (double)xu - U, cv = xv == 0 ? -V : (double)xv - V;  // 0 - U as -U
            hEq = w * Phi * (1.0 + u1);
            fEq = w * (p + Rho * P.RT * G);
            fSo = w * ((1 + G) * (cu * Fx + cv * Fy) + G * P.RT * (cu * Rho_x + cv * Rho_y));
        }
        const double hSo = (xu != 0 && xv != 0 ? sx(xu, Phi_x) + sx(xv, Phi_y)
                                                : (xu != 0 ? sx(xu, Phi_x) : sx(xv, Phi_y))) * w;
        hh[q] = hah * bh[q] + P.h_bh * hEq + P.h_ch * hSo;
        hf[q] = ahs * bf[q] + bh_ * fEq + ch * fSo;
    }
    if (WALLS && !xf && (j == 0 || j == ny)) {
        // bounce-back of the directions entering the fluid (xi.n_out < 0)
        const bool bottom = (j == 0);
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int xv = d2q9_xv(q);
            if (bottom ? xv > 0 : xv < 0) {
                hh[q] = hh[d2q9_bb(q)];
                hf[q] = hf[d2q9_bb(q)];
            }
        }
    }
    double *outf = lo ? (xf ? S.xlo_f : S.ylo_f) : (xf ? S.xff : S.yff);
    double *outh = lo ? (xf ? S.xlo_h : S.ylo_h) : (xf ? S.xfh : S.yfh);
    const size_t qs = lo ? (xf ? (size_t)ny : (size_t)pitch) : (xf ? S.qs : S.qsy);
    const size_t c = lo ? (xf ? (size_t)j : (size_t)i) : (size_t)j * pitch + i;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int s = xf ? d2q9_xu(q) : d2q9_xv(q);
        if (s == 0) continue;  // no flux along the face: the update does not read these slots
        outf[(size_t)q * qs + c] = sx(s, hf[q]);
        outh[(size_t)q * qs + c] = sx(s, hh[q]);
    }
}

template <int MODEL, bool WALLS, bool UW, bool IM>
__global__ void __launch_bounds__(256) k_faces_ac(Params P, State S) {
    pdl_wait();
    int i, j;
    bool xf, lo;
    if (!face_of_thread(P, WALLS, UW, i, j, xf, lo)) return;
    if (WALLS || xf) face_ac<MODEL, WALLS, UW, true>(P, S, i, j, lo, xf);
    else face_ac<MODEL, WALLS, UW, false>(P, S, i, j, lo, xf);
}

// Pseudopotential face pass 1: BhDt, face moments with the previous face
// force, face pressure and psi (Ark/Lib/D2Q9PP.cpp:110-136, Ark/Cpp/PseudoP.cpp:23-30).
template <int MODEL>
__global__ void __launch_bounds__(256) k_faces_pp1(Params P, State S) {
    pdl_wait();
    int i, j;
    bool xf, lo;
    if (!face_of_thread(P, false, false, i, j, xf, lo)) return;
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    const int im = wrapi(i - 1, P.nx), ip = wrapi(i + 1, P.nx);
    const size_t c = (size_t)j * P.pitch + i;
    double R = 0, su = 0, sv = 0, b[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        b[q] = xf ? face_bh<true, false>(P, S.bf + (size_t)q * S.qs, i, im, ip, j, P.xi_u[q], P.xi_v[q])
                  : face_bh<false, false>(P, S.bf + (size_t)q * S.qs, i, im, ip, j, P.xi_u[q], P.xi_v[q]);
        (xf ? S.xbf : S.ybf)[(size_t)q * S.qs + c] = b[q];
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) R += b[q];
#pragma unroll
    for (int q = 0; q < Q; ++q) su += b[q] * P.xi_u[q];
#pragma unroll
    for (int q = 0; q < Q; ++q) sv += b[q] * P.xi_v[q];
    double U = su / R, V = sv / R;
    U += 0.5 * P.hDt * (xf ? S.xfFx : S.yfFx)[c] / R;
    V += 0.5 * P.hDt * (xf ? S.xfFy : S.yfFy)[c] / R;
    const double p = 1.0 * cs_pressure(P, R);
    double scg, psi;
    calc_psi(P, R, p, scg, psi);
    (xf ? S.xrho : S.yrho)[c] = R;
    (xf ? S.xu : S.yu)[c] = U;
    (xf ? S.xv : S.yv)[c] = V;
    (xf ? S.xscg : S.yscg)[c] = scg;
    (xf ? S.xpsi : S.ypsi)[c] = psi;
}

// Pseudopotential face pass 2: face force from the face-psi stencil
// (Ark/Cpp/PseudoP.cpp:39-46 over faceFaces, Ark/Lib/GradSchemeBasic.h:181-208),
// equilibrium, He-Shan-Doolen source and flux (Ark/Lib/D2Q9PP.cpp:97-105).
template <int MODEL>
__global__ void __launch_bounds__(256) k_faces_pp2(Params P, State S) {
    pdl_wait();
    int i, j;
    bool xf, lo;
    if (!face_of_thread(P, false, false, i, j, xf, lo)) return;
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    const int nx = P.nx, ny = P.ny, pitch = P.pitch;
    const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx), jm = wrapi(j - 1, ny), jp = wrapi(j + 1, ny);
    const size_t c = (size_t)j * pitch + i;
    const double *__restrict__ PS = xf ? S.xpsi : S.ypsi;
    auto at = [&](int jj, int ii) { return PS[(size_t)jj * pitch + ii]; };
    const double gx = iso_gx(at(j, ip), at(j, im), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P._2dx, P.r_g6x);
    const double gy = iso_gy(at(jp, i), at(jm, i), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P._2dy, P.r_g6y);
    const double k = -(xf ? S.xscg : S.yscg)[c] * at(j, i);
    const double Fx = gx * k, Fy = gy * k;
    (xf ? S.xfFx : S.yfFx)[c] = Fx;
    (xf ? S.xfFy : S.yfFy)[c] = Fy;
    const double R = (xf ? S.xrho : S.yrho)[c], U = (xf ? S.xu : S.yu)[c], V = (xf ? S.xv : S.yv)[c];
    double eq[Q];
    pp_eq<MODEL>(P, R, U, V, eq);
    const double tauh = P.Tau0;
    const double ah = 2.0 * tauh / (2.0 * tauh + P.hDt), bh = 1.0 - ah, ch = tauh * bh;
    const double inv = 1.0 / (R * P.RT);
    const double *__restrict__ BB = xf ? S.xbf : S.ybf;
    double *out = xf ? S.xff : S.yff;
    const size_t qs = xf ? S.qs : S.qsy;
    double pr[Q];
    pp_src_proj<MODEL>(P, Fx, Fy, U, V, pr);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const double So = pr[q] * eq[q] * inv;
        const double t = ah * BB[(size_t)q * S.qs + c] + bh * eq[q] + ch * So;
        out[(size_t)q * qs + c] = t * (xf ? P.xi_u[q] : P.xi_v[q]);
    }
}

// ---------------------------------------------------------------------------
// Finite-volume update Update_phi_T (Ark/Cpp/DUGKS2DSolver.cpp:748-792) and
// cell macros Update_MacroVar (Ark/Lib/D2Q9AC.cpp:146-231,
// Ark/Lib/D2Q9HCZ.cpp:133-182, Ark/Lib/D2Q9PP.cpp:89-109).
template <int MODEL, bool WALLS>
__global__ void __launch_bounds__(256) k_update(Params P, State S) {
    pdl_wait();
    int i, j;
    if (!cell_of_thread(P, i, j)) return;
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    constexpr bool HASH = (MODEL == AC || MODEL == HCZ);
    const int pitch = P.pitch;
    const int ip = wrapi(i + 1, P.nx);
    const int jn = WALLS ? j + 1 : wrapi(j + 1, P.ny);
    const size_t c = (size_t)j * pitch + i;
    const size_t cE = (size_t)j * pitch + ip, cN = (size_t)jn * pitch + i;
    double sumf = 0, su = 0, sv = 0, Phi = 0, f0 = 0;
#pragma unroll
    // UW: the west face of column 0 and the south face of row 0 are the reference's
    // low-side periodic boundary faces (k_faces_ac, xlo / ylo)
    const bool xlo = P.uw && i == 0, ylo = P.uw && j == 0;
    for (int q = 0; q < Q; ++q) {
        const size_t oq = (size_t)q * S.qs, oy = (size_t)q * S.qsy;
        // net flux E, N, W, S in the reference's order.  D2Q9 Allen-Cahn: the faces
        // a direction runs along carry no flux (xi.n = 0: the reference adds exact zeros,
        // which only decide the sign of a zero sum; k_faces_ac does not store them), so
        // only the crossing faces are added and the rest direction has no flux term
        const bool cx = !HASH || d2q9_xu(q) != 0, cy = !HASH || d2q9_xv(q) != 0;
        double s = 0.0;
        if (cx && cy) {
            s = -S.xff[oq + cE];
            s += -S.yff[oy + cN];
            s += xlo ? S.xlo_f[(size_t)q * P.ny + j] : S.xff[oq + c];
            s += ylo ? S.ylo_f[(size_t)q * pitch + i] : S.yff[oy + c];
        } else if (cx) {
            s = -S.xff[oq + cE];
            s += xlo ? S.xlo_f[(size_t)q * P.ny + j] : S.xff[oq + c];
        } else if (cy) {
            s = -S.yff[oy + cN];
            s += ylo ? S.ylo_f[(size_t)q * pitch + i] : S.yff[oy + c];
        }
        const double fn = (cx || cy) ? P.aTP * S.bf[oq + c] - P.bTP * S.f[oq + c] + P.dtV * s
                                     : P.aTP * S.bf[oq + c] - P.bTP * S.f[oq + c];
        S.f[oq + c] = fn;
        sumf += fn;
        if (q == 0) f0 = fn;
        if (MODEL == PP16) {
            su += fn * P.xi_u[q];
            sv += fn * P.xi_v[q];
        } else {
            if (!HASH || d2q9_xu(q) != 0) su += sx(d2q9_xu(q), fn);
            if (!HASH || d2q9_xv(q) != 0) sv += sx(d2q9_xv(q), fn);
        }
        if (HASH) {
            double t = 0.0;
            if (cx && cy) {
                t = -S.xfh[oq + cE];
                t += -S.yfh[oy + cN];
                t += xlo ? S.xlo_h[(size_t)q * P.ny + j] : S.xfh[oq + c];
                t += ylo ? S.ylo_h[(size_t)q * pitch + i] : S.yfh[oy + c];
            } else if (cx) {
                t = -S.xfh[oq + cE];
                t += xlo ? S.xlo_h[(size_t)q * P.ny + j] : S.xfh[oq + c];
            } else if (cy) {
                t = -S.yfh[oy + cN];
                t += ylo ? S.ylo_h[(size_t)q * pitch + i] : S.yfh[oy + c];
            }
            const double hn = (cx || cy) ? P.aTP * S.bh[oq + c] - P.bTP * S.h[oq + c] + P.dtV * t
                                         : P.aTP * S.bh[oq + c] - P.bTP * S.h[oq + c];
            S.h[oq + c] = hn;
            Phi += hn;
        }
    }
    if (MODEL == AC || MODEL == HCZ) {
        const double Rho = P.aPhi * Phi + P.bPhi;
        double U, V, p, Mu, tau;
        if (MODEL == AC) {
            U = 0.0;
            V = 0.0;
            p = (sumf - f0) * P.Kp;  // (hDt rho_x.u - rho w0 |u|^2 lambda) vanishes with u = 0
            Mu = Rho * P.RT * P.Tau0;
            tau = Mu / (Rho * P.RT);
        } else {
            const double inv = 1.0 / (Rho * P.RT);
            U = QDIV(su, Rho * P.RT, inv);
            V = QDIV(sv, Rho * P.RT, inv);
            U += QDIV(P.hDt * S.fld[F_FX][c], Rho * P.RT, inv);
            V += QDIV(P.hDt * S.fld[F_FY][c], Rho * P.RT, inv);
            p = sumf + P.hDt * (S.fld[F_RHOX][c] * U + S.fld[F_RHOY][c] * V) * P.RT;
            Mu = P.NuV + (Phi - P.PhiV) * (P.NuL - P.NuV);
            Mu *= Rho;
            tau = QDIV(Mu, Rho * P.RT, inv);
        }
        S.fld[F_PHI][c] = Phi;
        S.fld[F_RHO][c] = Rho;
        S.fld[F_U][c] = U;
        S.fld[F_V][c] = V;
        S.fld[F_P][c] = p;
        S.fld[F_TAU][c] = tau;
    } else {
        const double Rho = sumf;
        const double invR = 1.0 / Rho;
        double U = QDIV(su, Rho, invR), V = QDIV(sv, Rho, invR);
        U += QDIV(P.hDt * S.fld[F_FX][c], Rho, invR);
        V += QDIV(P.hDt * S.fld[F_FY][c], Rho, invR);
        const double p = 1.0 * cs_pressure(P, Rho);
        double scg, psi;
        calc_psi(P, Rho, p, scg, psi);
        S.fld[F_RHO][c] = Rho;
        S.fld[F_U][c] = U;
        S.fld[F_V][c] = V;
        S.fld[F_P][c] = p;
        S.fld[F_SCG][c] = scg;
        S.fld[F_PSI][c] = psi;
    }
}

