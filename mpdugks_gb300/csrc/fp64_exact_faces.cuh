// Part of fp64_step.cuh, reference-exact variant: the face kernels and the update.
// Allen-Cahn face: Update_MacroVar_h + Update_phi_Eqh + Update_DVDF_Source_h
// + Update_phi_h + Update_phiFlux_h (+ Wall_3_BB) -- Ark/Lib/D2Q9AC.cpp:106-144,
// 232-329,345-358; Ark/Lib/D2Q9HCZ.cpp:93-131,183-271;
// Ark/Cpp/DUGKS2DSolver.cpp:402-441; Ark/Cpp/Boundary.cpp:118-139.
// UW: the threads after the faces do the x and y periodic boundary faces in the
// reference's low-side form (column 0 / row 0 only), written to xlo / ylo.
// The x and y faces are separate bodies (XF), so each computes the six directions that cross
// its face and no others.  The CD reconstruction gives twice the face values (b = SC times
// the stored number, SC = 1/2); the averaged source fields are kept as sums of the two cells
// (twice the average) and their 1/2 goes into the constants they meet.
// EDGE: a face that reads the rows beyond a wall.
template <int MODEL, bool EDGE, bool UW, bool XF, bool IM>
__device__ __forceinline__ void face_ac(const Params &P, const State &S, int i, int j, bool lo) {
    const int ny = P.ny, pitch = P.pitch;
    constexpr double SC = UW ? 1.0 : 0.5;
    const FaceRows r = face_rows(P, i, j);
    // the source fields summed over the owner and the neighbour cell
    auto both = [&](int k) {
        double o, n;
        face_on<XF, EDGE>(P, S.fld[k], r, o, n);
        return o + n;
    };
    double bf[9], bh[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const size_t qo = (size_t)q * S.qs;
        if (UW) {
            const size_t co = XF ? r.r0 + r.im : r.rm + i, cn = r.r0 + i;
            bf[q] = face_uw<XF>(P, S.bf + qo, S.gfx + qo, S.gfy + qo, co, cn, d2q9_xu(q), d2q9_xv(q), lo);
            bh[q] = face_uw<XF>(P, S.bh + qo, S.ghx + qo, S.ghy + qo, co, cn, d2q9_xu(q), d2q9_xv(q), lo);
        } else {
            bf[q] = face_bh9<XF, EDGE>(P, S.bf + qo, r, d2q9_xu(q), d2q9_xv(q));
            bh[q] = face_bh9<XF, EDGE>(P, S.bh + qo, r, d2q9_xu(q), d2q9_xv(q));
        }
    }
    double Phi = bh[0], sumf = bf[0];
#pragma unroll
    for (int q = 1; q < 9; ++q) Phi += bh[q];
#pragma unroll
    for (int q = 1; q < 9; ++q) sumf += bf[q];
    Phi = SC * Phi;
    const double Rho = P.aPhi * Phi + P.bPhi;
    const double Fx = both(F_FX), Fy = both(F_FY);  // twice the averages
    double pRT = 0.0, tauh;
    Xi4 fr{};
    MomHCZ m;
    if (MODEL == AC) {
        const double p = (sumf - bf[0]) * (UW ? P.Kp : P.Kp2);  // the u-dependent terms vanish with u = 0
        const double rRT = Rho * P.RT;
        tauh = rRT * P.Tau0 / rRT;
        pRT = QDIV(p, P.RT, P.r_RT);
        fr = xi4(Fx, Fy, P.RT, P.r_RT);
    } else {
        // first moments over the directions with a nonzero component (the others add +-0)
        double su = bf[1], sv = bf[2];
#pragma unroll
        for (int q = 2; q < 9; ++q)
            if (d2q9_xu(q) != 0) su += sx(d2q9_xu(q), bf[q]);
#pragma unroll
        for (int q = 3; q < 9; ++q)
            if (d2q9_xv(q) != 0) sv += sx(d2q9_xv(q), bf[q]);
        // quotients of doubled numerators by 2 rho RT; 0.5 hDt = 1/8
        m.rRT = Rho * P.RT;
        const double d = UW ? m.rRT : 2.0 * m.rRT, inv = 1.0 / d, fs = UW ? 0.0625 : 0.125;
        const double U = __fma_rn(fs, QDIV(Fx, d, inv), QDIV(su, d, inv));
        const double V = __fma_rn(fs, QDIV(Fy, d, inv), QDIV(sv, d, inv));
        const double Rx = both(F_RHOX), Ry = both(F_RHOY);
        // 0.5 hDt RT (Rho_x U + Rho_y V): RT / 16 of the doubled averages
        m.p = __fma_rn(SC, sumf, P.RT16 * (Rx * U + Ry * V));
        tauh = QDIV((UW ? P.NuV : P.NuV2) * Rho, d, inv);
        m.uuL = (U * U + V * V) * P.Lambda0;
        m.ur = xi4(U, V, P.RT, P.r_RT);
        hcz_products(m, U, V, Fx, Fy, Rx, Ry);
    }
    // 2 tau / (2 tau + hDt), both sides halved; applied to the reconstruction's scale
    const double ah = tauh / (tauh + P.hDt2), bh_ = 1.0 - ah, ch = tauh * bh_;
    const double ahs = UW ? ah : 0.5 * ah, hah = UW ? P.h_ah : P.h_ah2;
    const double Sx = both(F_PHIX), Sy = both(F_PHIY), ssum = Sx + Sy, sdif = Sy - Sx;
    const bool far = warp_any<IM>(far_tail(Phi) || (MODEL == HCZ && (far_tail(Sx) || far_tail(Sy))));
    double *outf = lo ? (XF ? S.xlo_f : S.ylo_f) : (XF ? S.xff : S.yff);
    double *outh = lo ? (XF ? S.xlo_h : S.ylo_h) : (XF ? S.xfh : S.yfh);
    const size_t qs = lo ? (XF ? (size_t)ny : (size_t)pitch) : (XF ? S.qs : S.qsy);
    const size_t c = lo ? (XF ? (size_t)j : (size_t)i) : (size_t)j * pitch + i;
    // the pairs that cross the face: x (1,5) (2,6) (8,4), y (3,7) (2,6) (4,8)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int q = XF ? (k == 0 ? 1 : (k == 1 ? 2 : 8)) : k + 2, qo = d2q9_bb(q);
        const int xu = d2q9_xu(q), xv = d2q9_xv(q);
        const double w = d2q9_w(q);
        double hf, hfo, hh, hho;
        auto pair = [&](auto &mul) {
            const double hc = mul(P.h_ch, mul(src_dot(xu, xv, Sx, Sy, ssum, sdif), 0.5 * w));
            if (MODEL == AC) {
                const double hE = mul(P.h_bh, mul(w, Phi)), fE = mul(bh_, mul(w, pRT)),
                             fS = mul(ch, mul(0.5 * w, fr.get(xu, xv)));
                hh = mul(hah, bh[q]) + hE + hc;
                hho = mul(hah, bh[qo]) + hE - hc;
                hf = mul(ahs, bf[q]) + fE + fS;
                hfo = mul(ahs, bf[qo]) + fE - fS;
            } else {
                const double u1 = m.ur.get(xu, xv), wPhi = mul(w, Phi);
                double G, Go;
                hcz_gamma(mul, m, u1, G, Go);
                hh = mul(hah, bh[q]) + mul(P.h_bh, mul(wPhi, 1.0 + u1)) + hc;
                hho = mul(hah, bh[qo]) + mul(P.h_bh, mul(wPhi, 1.0 - u1)) - hc;
                hf = mul(ahs, bf[q]) + mul(bh_, mul(w, m.p + mul(m.rRT, G))) +
                     mul(ch, mul(0.5 * w, hcz_source(mul, m, P.RT, G, xu, xv)));
                hfo = mul(ahs, bf[qo]) + mul(bh_, mul(w, m.p + mul(m.rRT, Go))) +
                      mul(ch, mul(0.5 * w, hcz_source(mul, m, P.RT, Go, -xu, -xv)));
            }
        };
        Mul<IM> mul;
        if (far) mul.bad = 1;
        else pair(mul);
        if (IM && mul.bad) {  // an operand beyond the integer product's window
            Mul<false> fp;
            pair(fp);
        }
        if (EDGE && !XF) {  // bounce-back of the directions entering the fluid (xi.n_out < 0): q has xv > 0
            if (j == 0) {
                hh = hho;
                hf = hfo;
            } else if (j == ny) {
                hho = hh;
                hfo = hf;
            }
        }
        outf[(size_t)q * qs + c] = hf;
        outh[(size_t)q * qs + c] = hh;
        outf[(size_t)qo * qs + c] = -hfo;
        outh[(size_t)qo * qs + c] = -hho;
    }
}

// IM: at two resident blocks (unbounded, its 200 registers leave one, and the chains of the
// integer products show: 2.49 ms a step on 1000x1000 against 2.06, without them 2.44)
template <int MODEL, bool WALLS, bool UW, bool IM>
__global__ void __launch_bounds__(256, IM ? 2 : 1) k_faces_ac(Params P, State S) {
    pdl_wait();
    int i, j;
    bool xf, lo;
    if (!face_of_thread(P, WALLS, UW, i, j, xf, lo)) return;
    if (WALLS && (j == 0 || (xf ? j == P.ny - 1 : j == P.ny))) {
        if (xf) face_ac<MODEL, WALLS, UW, true, false>(P, S, i, j, lo);
        else face_ac<MODEL, WALLS, UW, false, false>(P, S, i, j, lo);
        return;
    }
    if (xf) face_ac<MODEL, false, UW, true, IM>(P, S, i, j, lo);
    else face_ac<MODEL, false, UW, false, IM>(P, S, i, j, lo);
}

// Twice the half-step value of a D2V16 velocity xi = c (xu, xv), xu, xv in {-2 .. 2} known at
// compile time: the products of the gradients with c once, the factors 2 and 1/4 exact.
template <bool XF>
__device__ __forceinline__ double face_bh16(const Params &P, const double *__restrict__ B, const FaceRows &r, int xu,
                                            int xv) {
    double o, n;
    face_on<XF, false>(P, B, r, o, n);
    const double s = o + n;
    const int xn = XF ? xu : xv, xt = XF ? xv : xu;
    // g = (n - o) c xn + (t / 4) c xt; 2 hDt g = dt g, the factor of a ring (|xi| = c or 2 c) in dt
    const bool two = xn == 2 || xn == -2 || xt == 2 || xt == -2;
    const double k = two ? P.dt2 : P.dt;
    if (xt == 0) return s - k * sx(xn, (n - o) * P.c16);
    const double t = face_tan<XF, false>(P, B, r) * P.c16;
    if (xn == 0) return s - (two ? P.hDt : P.hDt2) * sx(xt, t);
    return s - k * __fma_rn(xt > 0 ? 0.25 : -0.25, t, sx(xn, (n - o) * P.c16));
}
template <int MODEL, bool XF>
__device__ __forceinline__ double face_bhpp(const Params &P, const double *__restrict__ B, const FaceRows &r, int q) {
    return MODEL == PP16 ? face_bh16<XF>(P, B, r, vel_u<MODEL>(q), vel_v<MODEL>(q))
                         : face_bh9<XF, false>(P, B, r, d2q9_xu(q), d2q9_xv(q));
}

// first moments sum_q xi_q b_q over the directions with a nonzero component, the products
// b_q c once for both components
template <int MODEL>
__device__ __forceinline__ void pp_first_moments(const Params &P, const double *b, double &su, double &sv) {
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    bool fu = true, fv = true;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int xu = vel_u<MODEL>(q), xv = vel_v<MODEL>(q);
        if (xu == 0 && xv == 0) continue;
        const double t = MODEL == PP16 ? b[q] * P.c16 : b[q];
        if (xu != 0) su = fu ? xu * t : ((xu & 1) ? su + sx(xu, t) : __fma_rn((double)xu, t, su));
        if (xv != 0) sv = fv ? xv * t : ((xv & 1) ? sv + sx(xv, t) : __fma_rn((double)xv, t, sv));
        if (xu != 0) fu = false;
        if (xv != 0) fv = false;
    }
}

// Pseudopotential face pass 1: BhDt, face moments with the previous face
// force, face pressure and psi (Ark/Lib/D2Q9PP.cpp:110-136, Ark/Cpp/PseudoP.cpp:23-30).
// xbf / ybf hold twice BhDt.
template <int MODEL, bool XF>
__device__ __forceinline__ void face_pp1(const Params &P, const State &S, int i, int j) {
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    const FaceRows r = face_rows(P, i, j);
    const size_t c = r.r0 + i;
    double R, su, sv, b[Q];
    double *bo = XF ? S.xbf : S.ybf;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        b[q] = face_bhpp<MODEL, XF>(P, S.bf + (size_t)q * S.qs, r, q);
        bo[(size_t)q * S.qs + c] = b[q];
    }
    R = b[0];
#pragma unroll
    for (int q = 1; q < Q; ++q) R += b[q];
    pp_first_moments<MODEL>(P, b, su, sv);
    // su, sv and R are doubled: their quotients are not, the force term's by 2 (0.5 hDt F / R)
    const double inv = 1.0 / R;
    const double U = QDIV(su, R, inv) + QDIV(P.hDt * (XF ? S.xfFx : S.yfFx)[c], R, inv);
    const double V = QDIV(sv, R, inv) + QDIV(P.hDt * (XF ? S.xfFy : S.yfFy)[c], R, inv);
    R = 0.5 * R;
    const double p = cs_pressure(P, R);
    double scg, psi;
    calc_psi(P, R, p, scg, psi);
    (XF ? S.xrho : S.yrho)[c] = R;
    (XF ? S.xu : S.yu)[c] = U;
    (XF ? S.xv : S.yv)[c] = V;
    (XF ? S.xscg : S.yscg)[c] = scg;
    (XF ? S.xpsi : S.ypsi)[c] = psi;
}
template <int MODEL>
__global__ void __launch_bounds__(256) k_faces_pp1(Params P, State S) {
    pdl_wait();
    int i, j;
    bool xf, lo;
    if (!face_of_thread(P, false, false, i, j, xf, lo)) return;
    if (xf) face_pp1<MODEL, true>(P, S, i, j);
    else face_pp1<MODEL, false>(P, S, i, j);
}

// Pseudopotential face pass 2: face force from the face-psi stencil
// (Ark/Cpp/PseudoP.cpp:39-46 over faceFaces, Ark/Lib/GradSchemeBasic.h:181-208),
// equilibrium, He-Shan-Doolen source and flux (Ark/Lib/D2Q9PP.cpp:97-105) of the directions
// that cross the face (the others carry no flux; the update does not read them).
template <int MODEL, bool XF>
__device__ __forceinline__ void face_pp2(const Params &P, const State &S, int i, int j) {
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    const int nx = P.nx, ny = P.ny, pitch = P.pitch;
    const int im = wrapi(i - 1, nx), ip = wrapi(i + 1, nx), jm = wrapi(j - 1, ny), jp = wrapi(j + 1, ny);
    const size_t c = (size_t)j * pitch + i;
    const double *__restrict__ PS = XF ? S.xpsi : S.ypsi;
    auto at = [&](int jj, int ii) { return PS[(size_t)jj * pitch + ii]; };
    const double gx = iso_gx(at(j, ip), at(j, im), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P.g6x, P.r_g6x);
    const double gy = iso_gy(at(jp, i), at(jm, i), at(jp, ip), at(jp, im), at(jm, ip), at(jm, im), P.g6y, P.r_g6y);
    const double k = -(XF ? S.xscg : S.yscg)[c] * at(j, i);
    const double Fx = gx * k, Fy = gy * k;
    (XF ? S.xfFx : S.yfFx)[c] = Fx;
    (XF ? S.xfFy : S.yfFy)[c] = Fy;
    const double R = (XF ? S.xrho : S.yrho)[c], U = (XF ? S.xu : S.yu)[c], V = (XF ? S.xv : S.yv)[c];
    double eq[Q];
    pp_eq<MODEL>(P, R, U, V, eq);
    const double rRT = R * P.RT, inv = 1.0 / rRT;
    const double *__restrict__ BB = XF ? S.xbf : S.ybf;
    double *out = XF ? S.xff : S.yff;
    const size_t qs = XF ? S.qs : S.qsy;
    double pr[Q];
    pp_src_proj<MODEL>(P, Fx, Fy, U, V, pr);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int xn = XF ? vel_u<MODEL>(q) : vel_v<MODEL>(q);
        if (xn == 0) continue;
        const double So = QDIV(pr[q] * eq[q], rRT, inv);
        const double t = P.pp_ah2 * BB[(size_t)q * S.qs + c] + P.pp_bh * eq[q] + P.pp_ch * So;
        out[(size_t)q * qs + c] = MODEL == PP16 ? t * (XF ? P.xi_u[q] : P.xi_v[q]) : sx(xn, t);
    }
}
template <int MODEL>
__global__ void __launch_bounds__(256) k_faces_pp2(Params P, State S) {
    pdl_wait();
    int i, j;
    bool xf, lo;
    if (!face_of_thread(P, false, false, i, j, xf, lo)) return;
    if (xf) face_pp2<MODEL, true>(P, S, i, j);
    else face_pp2<MODEL, false>(P, S, i, j);
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
    double sumf = 0, su = 0, sv = 0, Phi = 0, fq[Q];
    // UW: the west face of column 0 and the south face of row 0 are the reference's
    // low-side periodic boundary faces (k_faces_ac, xlo / ylo)
    const bool xlo = P.uw && i == 0, ylo = P.uw && j == 0;
    // one distribution's new value of direction q: net flux E, N, W, S in the reference's order.
    // The faces a direction runs along carry no flux (xi.n = 0: the reference adds exact
    // zeros, which only decide the sign of a zero sum; the face kernels do not store them),
    // so only the crossing faces are added and the rest direction has no flux term
    auto advance = [&](int q, const double *__restrict__ T, const double *__restrict__ B, const double *__restrict__ X,
                       const double *__restrict__ Y, const double *__restrict__ XL, const double *__restrict__ YL) {
        const size_t oq = (size_t)q * S.qs, oy = (size_t)q * S.qsy;
        const bool cx = vel_u<MODEL>(q) != 0, cy = vel_v<MODEL>(q) != 0;
        const double base = P.aTP * B[oq + c] - P.bTP * T[oq + c];
        if (!cx && !cy) return base;
        double s;
        if (cx) {
            const double W = HASH && xlo ? XL[(size_t)q * P.ny + j] : X[oq + c];
            if (cy) {
                s = -X[oq + cE] - Y[oy + cN];
                s += W;
                s += HASH && ylo ? YL[(size_t)q * pitch + i] : Y[oy + c];
            } else {
                s = W - X[oq + cE];
            }
        } else {
            s = (HASH && ylo ? YL[(size_t)q * pitch + i] : Y[oy + c]) - Y[oy + cN];
        }
        // D2Q9: dt / V = 1/2, an exact product
        return MODEL == PP16 ? base + P.dtV * s : __fma_rn(0.5, s, base);
    };
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const size_t oq = (size_t)q * S.qs;
        fq[q] = advance(q, S.f, S.bf, S.xff, S.yff, S.xlo_f, S.ylo_f);
        S.f[oq + c] = fq[q];
        sumf = q == 0 ? fq[0] : sumf + fq[q];
        if (HASH) {
            const double hn = advance(q, S.h, S.bh, S.xfh, S.yfh, S.xlo_h, S.ylo_h);
            S.h[oq + c] = hn;
            Phi = q == 0 ? hn : Phi + hn;
        }
    }
    if (MODEL != AC) pp_first_moments<MODEL>(P, fq, su, sv);
    if (MODEL == AC || MODEL == HCZ) {
        const double Rho = P.aPhi * Phi + P.bPhi, rRT = Rho * P.RT;
        double U, V, p, tau;
        if (MODEL == AC) {
            U = 0.0;
            V = 0.0;
            p = (sumf - fq[0]) * P.Kp;  // (hDt rho_x.u - rho w0 |u|^2 lambda) vanishes with u = 0
            tau = rRT * P.Tau0 / rRT;
        } else {
            // hDt = 1/4; one kinematic viscosity
            const double inv = 1.0 / rRT;
            U = __fma_rn(0.25, QDIV(S.fld[F_FX][c], rRT, inv), QDIV(su, rRT, inv));
            V = __fma_rn(0.25, QDIV(S.fld[F_FY][c], rRT, inv), QDIV(sv, rRT, inv));
            p = __fma_rn(0.25, (S.fld[F_RHOX][c] * U + S.fld[F_RHOY][c] * V) * P.RT, sumf);
            tau = QDIV(P.NuV * Rho, rRT, inv);
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
        const double p = cs_pressure(P, Rho);
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

