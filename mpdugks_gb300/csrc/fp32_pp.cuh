// Per-cell and per-face arithmetic of the FP32 pseudopotential step (D2Q9PP, D2V16),
// shared by the two tiled kernels (fp32_pp.cu) and the single-pass streaming kernel
// (fp32_pp_stream.cu), so both evaluate the same expressions.  Storage: the density in
// FP64, f as the FP32 remainders g_q = f_q - e_q rho (fp32_pp.cu has the derivation).
#pragma once
#include <cuda_runtime.h>

#include "dugks_device.cuh"
#include "fp32_math.cuh"
#include "fp32_state.cuh"

namespace dugks {
namespace f32 {

template <int MODEL>
struct PPQ {
    static constexpr int Q = MODEL == PP16 ? 16 : 9;
};

// The velocity set as integers times the lattice speed (D2V16: Ark/Lib/D2V16.cpp:53-66,
// D2Q9: Ark/Lib/D2Q9.h:86-88) and each direction's opposite
template <int MODEL>
__host__ __device__ constexpr int lat_u(int q) {
    return MODEL == PP16 ? (q == 0 || q == 4 || q == 7 ? 1 : q == 2 || q == 5 || q == 6 ? -1 : q == 8 || q == 12 || q == 15 ? 2
                                                                                        : q == 10 || q == 13 || q == 14 ? -2 : 0)
                         : d2q9_xu(q);
}
template <int MODEL>
__host__ __device__ constexpr int lat_v(int q) {
    return MODEL == PP16 ? (q == 1 || q == 4 || q == 5 ? 1 : q == 3 || q == 6 || q == 7 ? -1 : q == 9 || q == 12 || q == 13 ? 2
                                                                                        : q == 11 || q == 14 || q == 15 ? -2 : 0)
                         : d2q9_xv(q);
}
template <int MODEL>
__host__ __device__ constexpr int lat_opp(int q) {
    return MODEL == PP16 ? d2v16_opp(q) : d2q9_bb(q);
}

// Equilibrium parts de_q = eq_q(rho, u, v) - e_q rho (zero at rest).
// D2V16: Macro16 (Ark/Lib/D2V16.cpp:125-145) at T = T0, p = rho RT, minus its value at
// (rho, 0, 0) (at rest the moments are linear in rho), times the inverse moment matrix
// (Ark/Lib/D2V16.cpp:34-52).  A ring's four rows are the sums +- of four parts, even or odd in
// u and in v, and each part is rho or rho u times a polynomial of u^2, v^2 whose coefficients
// are combinations of the matrix's entries (PPP::k, formed in FP64 on the host): about 75
// operations and no cancelling moments, where the matrix by opposite pairs took 108 and the
// moments 35 before it.  Every rounding is written out, so that each kernel including this
// evaluates it alike.
template <int MODEL>
__device__ __forceinline__ void pp_deq(const PPP &P, float rho, float u, float v, float *de) {
    if (MODEL == PP16) {
        const float *k = P.k;
        const float a = __fmul_rn(u, u), b = __fmul_rn(v, v), s2 = __fadd_rn(a, b);
        const float M1 = __fmul_rn(rho, u), M2 = __fmul_rn(rho, v), ruv = __fmul_rn(M1, v), rs2 = __fmul_rn(rho, s2);
        auto ring = [&](int q, float ee, float xy, float ox, float oy) {  // diagonals (1,1) (-1,1) (-1,-1) (1,-1)
            const float p = __fadd_rn(ee, xy), m = __fsub_rn(ee, xy), c = __fadd_rn(ox, oy), d = __fsub_rn(ox, oy);
            de[q] = __fadd_rn(p, c);
            de[q + 2] = __fsub_rn(p, c);
            de[q + 1] = __fsub_rn(m, d);
            de[q + 3] = __fadd_rn(m, d);
        };
        auto axis = [&](int q, float e0, float e1, float ox, float oy) {  // (1,0) (0,1) (-1,0) (0,-1)
            de[q] = __fadd_rn(e0, ox);
            de[q + 2] = __fsub_rn(e0, ox);
            de[q + 1] = __fadd_rn(e1, oy);
            de[q + 3] = __fsub_rn(e1, oy);
        };
        {
            const float w = __fmul_rn(__fmul_rn(k[2], __fsub_rn(a, b)), __fadd_rn(k[3], s2));
            const float e0 = __fmul_rn(rho, fmaf(k[0], a, fmaf(k[1], b, w)));
            const float e1 = __fmul_rn(rho, fmaf(k[1], a, fmaf(k[0], b, -w)));
            axis(0, e0, e1, __fmul_rn(k[4], M1), __fmul_rn(k[4], M2));
        }
        ring(4, __fmul_rn(rs2, fmaf(k[6], s2, k[5])), __fmul_rn(ruv, fmaf(k[8], s2, k[7])),
             __fmul_rn(M1, fmaf(k[10], a, k[9])), __fmul_rn(M2, fmaf(k[10], b, k[9])));
        {
            const float U = fmaf(k[12], s2, k[11]), V = fmaf(k[14], s2, k[13]);
            axis(8, __fmul_rn(rho, fmaf(a, U, __fmul_rn(b, V))), __fmul_rn(rho, fmaf(b, U, __fmul_rn(a, V))),
                 __fmul_rn(M1, fmaf(k[16], a, fmaf(k[17], b, k[15]))), __fmul_rn(M2, fmaf(k[16], b, fmaf(k[17], a, k[15]))));
        }
        ring(12, __fmul_rn(rs2, fmaf(k[19], s2, k[18])), __fmul_rn(ruv, fmaf(k[21], s2, k[20])),
             __fmul_rn(M1, fmaf(k[23], a, fmaf(k[24], b, k[22]))), __fmul_rn(M2, fmaf(k[23], b, fmaf(k[24], a, k[22]))));
    } else {
        // D2Q9PP (Ark/Lib/D2Q9PP.cpp:51-62): w rho (1 + u1 + u1^2/2 - |u|^2 lambda) - w rho
        const float uuL = __fmul_rn(fmaf(u, u, __fmul_rn(v, v)), P.Lambda0);
        de[0] = -__fmul_rn(__fmul_rn(P.w9[0], rho), uuL);
#pragma unroll
        for (int q = 1; q <= 4; ++q) {
            const float u1 = __fmul_rn(__fadd_rn(sxf(d2q9_xu(q), u), sxf(d2q9_xv(q), v)), P.invRT);
            const float h = fmaf(__fmul_rn(0.5f, u1), u1, -uuL), wr = __fmul_rn(P.w9[q], rho);
            de[q] = __fmul_rn(wr, __fadd_rn(h, u1));
            de[q + 4] = __fmul_rn(wr, __fsub_rn(h, u1));
        }
    }
}

// ---- float-float arithmetic: a value is the unevaluated sum hi + lo of two
// floats.  TwoSum (Knuth, TAOCP vol. 2, 4.2.2), FastTwoSum (Dekker 1971), the
// product error by fma, the cascaded sum Sum2 (Ogita, Rump and Oishi 2005) and a
// two-step long division as in Bailey's double-double arithmetic: about 44
// significant bits, for the moment sums and the equation of state that the FP64
// path evaluates in double (the FP64 units of this GPU are ~1/60 of its FP32
// rate, and these were most of this path's time).
struct FF {
    float hi, lo;
};
__device__ __forceinline__ FF two_sum(float a, float b) {
    const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ FF fast_two_sum(float a, float b) {  // |a| >= |b|
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ void ff_acc(FF &s, float x) {  // Sum2 step: s += x
    const FF t = two_sum(s.hi, x);
    s.hi = t.hi;
    s.lo = __fadd_rn(s.lo, t.lo);
}
__device__ __forceinline__ FF ff_neg(FF a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ FF ff_add(FF a, FF b) {
    FF t = two_sum(a.hi, b.hi);
    t.lo = __fadd_rn(t.lo, __fadd_rn(a.lo, b.lo));
    return two_sum(t.hi, t.lo);
}
__device__ __forceinline__ FF ff_mul(FF a, FF b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    return fast_two_sum(p, e);
}
__device__ __forceinline__ FF ff_div(FF a, FF b) {
    // quotient digits from one reciprocal (within an ulp; the second digit corrects the first's)
    const float y = rcp(b.hi), q1 = __fmul_rn(a.hi, y);
    const FF r = ff_add(a, ff_neg(ff_mul(b, FF{q1, 0.f})));
    return fast_two_sum(q1, __fmul_rn(__fadd_rn(r.hi, r.lo), y));
}
__device__ __forceinline__ FF ff_norm(FF a) { return two_sum(a.hi, a.lo); }

// Carnahan-Starling pressure (Ark/Lib/nonidealEoS.h:114-118) of the density r:
// r R0 T (1 + r + r^2 - r^3) / (1 - r)^3 - a r^2
__device__ __forceinline__ FF cs_p(const PPP &P, FF r) {
    const FF one{1.f, 0.f};
    const FF r2 = ff_mul(r, r), r3 = ff_mul(r2, r);
    const FF num = ff_add(ff_add(ff_add(one, r), r2), ff_neg(r3));
    const FF om = ff_add(one, ff_neg(r));
    const FF den = ff_mul(ff_mul(om, om), om);
    return ff_add(ff_mul(ff_mul(r, FF{P.rtcs_hi, P.rtcs_lo}), ff_div(num, den)),
                  ff_neg(ff_mul(FF{P.acs_hi, P.acs_lo}, r2)));
}
// calcPsi (Ark/Header/Macroscopic.h:64-68): G = sign(p - rho RT), psi = sqrt(2 (p - rho RT) / G)
// psi as a float-float pair (hi, lo): the square root's head and the correction
// (x - hi^2) / (2 hi) of its residual (hi^2 exactly by fma); the gradient stencil of
// psi then differences pairs, which matters where grad psi is small against psi
__device__ __forceinline__ void cs_psi(const PPP &P, FF rho, FF p, float &scg, float &psi, float &psil) {
    const FF g = ff_add(p, ff_neg(ff_mul(rho, FF{P.rt_hi, P.rt_lo})));
    const float G = (float)((g.hi > 0.f) - (g.hi < 0.f));
    scg = G;
    const float xh = 2.f * g.hi * G, xl = 2.f * g.lo * G;  // G = +-1: exact
    // the root and its residual's correction from one reciprocal root y
    const float y = rsqrtf(xh), hy = __fmul_rn(0.5f, y), r0 = __fmul_rn(xh, y);
    const float r1 = fmaf(fmaf(-r0, r0, xh), hy, r0);
    const bool zero = xh == 0.f;
    psi = zero ? 0.f : r1;
    psil = zero ? 0.f : __fmul_rn(__fadd_rn(fmaf(-r1, r1, xh), xl), hy);
}
__device__ __forceinline__ double ff_to_double(FF a) { return (double)a.hi + (double)a.lo; }

// n b as an exact float for the integer n in {-2, ..., 2}
__device__ __forceinline__ float times_small(int n, float b) { return n == 1 ? b : n == -1 ? -b : n == 2 ? 2.f * b : -2.f * b; }

// First moments sum_q xi_q b_q (x, y) as float-float: over the opposite pairs (q, q') of
// n_q (b_q - b_q'), n_q = xi_q / speed an integer (each term exact scaling of one rounded
// difference, zero components skipped), then times the lattice speed as a pair
template <int MODEL>
__device__ __forceinline__ void pp_first_moments(const PPP &P, const float (&b)[PPQ<MODEL>::Q], FF &su, FF &sv) {
    constexpr int Q = PPQ<MODEL>::Q;
    FF ax{0.f, 0.f}, ay{0.f, 0.f};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int qo = lat_opp<MODEL>(q);
        if (qo <= q) continue;  // each pair once, from its lower index; the rest direction has none
        const float d = __fsub_rn(b[q], b[qo]);
        const int nu = lat_u<MODEL>(q), nv = lat_v<MODEL>(q);
        if (nu != 0) ff_acc(ax, times_small(nu, d));
        if (nv != 0) ff_acc(ay, times_small(nv, d));
    }
    const FF c{P.lat_hi, P.lat_lo};
    su = ff_mul(ff_norm(ax), c);
    sv = ff_mul(ff_norm(ay), c);
}



// 8-neighbour isotropic gradient (Ark/Lib/GradSchemeBasic.h:153-208) from the float-float
// pairs of the eight neighbours, by pair differences
__device__ __forceinline__ void pp_iso_grad(const PPP &P, float2 E, float2 W, float2 N, float2 S, float2 NE,
                                            float2 NW, float2 SE, float2 SW, float &gx, float &gy) {
    gx = (4.f * pdiff(E, W) + (pdiff(NE, NW) + pdiff(SE, SW))) * P.inv_6_2dx;
    gy = (4.f * pdiff(N, S) + (pdiff(NE, SE) + pdiff(NW, SW))) * P.inv_6_2dy;
}

// The He-Shan-Doolen projections (xi_q - u).F of the directions, by opposite pairs: with
// d = xi_q.F and w = u.F, (xi_q - u).F = d - w and (xi_q' - u).F = -d - w (xi_q' = -xi_q);
// a rest direction (D2Q9PP's 0) has -w.
template <int MODEL>
__device__ __forceinline__ void pp_src_proj(const PPP &P, float fx, float fy, float U, float V,
                                            float (&pr)[PPQ<MODEL>::Q]) {
    constexpr int Q = PPQ<MODEL>::Q;
    const float w = fmaf(fx, U, __fmul_rn(fy, V));
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int qo = lat_opp<MODEL>(q);
        if (qo < q) continue;
        if (qo == q) {
            pr[q] = -w;
            continue;
        }
        const float d = fmaf(fx, P.xi_u[q], __fmul_rn(fy, P.xi_v[q]));
        pr[q] = __fsub_rn(d, w);
        pr[qo] = -__fadd_rn(d, w);
    }
}

// Collision pre-step of one cell: f-bar-plus as the remainder
// B_q - e_q rho = g_q + (1 - a)(de_q - g_q) + c S_q, S the He-Shan-Doolen source of the
// cell force (fx, fy).
template <int MODEL>
__device__ __forceinline__ void pp_collide(const PPP &P, const float (&g)[PPQ<MODEL>::Q], float rho, float U, float V,
                                           float fx, float fy, float (&bf)[PPQ<MODEL>::Q]) {
    constexpr int Q = PPQ<MODEL>::Q;
    float de[Q];
    pp_deq<MODEL>(P, rho, U, V, de);
    const float ci = __fmul_rn(P.cBP, rcp(__fmul_rn(rho, P.RT)));
    float pr[Q];
    pp_src_proj<MODEL>(P, fx, fy, U, V, pr);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const float eq = fmaf(P.erest[q], rho, de[q]);
        bf[q] = fmaf(P.bBP, __fsub_rn(de[q], g[q]), fmaf(__fmul_rn(pr[q], eq), ci, g[q]));
    }
}

// Face pass 1 of one face (XF: an x face between o = west and n = east cell, else a y face
// between o = below and n = above): the half-step reconstruction relative to e_q times the
// face average of rho, from the f-bar-plus remainders of the two cells (o, n) and the sums
// tn, to of their tangential differences ((t+) - (t-) of n and of o: x face rows +-1, y face
// columns -1 minus +1).  rsum (FP64), rd, rt: the sum of the two cells' densities, their
// difference n - o and the sum of their tangential differences taken like tn, to; (fxp, fyp):
// the face force of the previous step.  Out: b, the face velocity, the face density (R) and
// it relative to the average (dr), and the face psi pair and sign.
// A direction's reconstruction is s/2 - hDt xi.grad with the lattice speed in the constants
// (PPP::hc = hDt c), the components that are zero left out; the e_q rho part's gradient terms
// are those of four directions, their negatives and doubles.
struct PPFace {
    float U, V, R, dr, psi, psil, scg;
};
template <int MODEL, bool XF>
__device__ __forceinline__ PPFace pp_face1(const PPP &P, const float (&o)[PPQ<MODEL>::Q],
                                           const float (&n)[PPQ<MODEL>::Q], const float (&tn)[PPQ<MODEL>::Q],
                                           const float (&to)[PPQ<MODEL>::Q], double rsum, float rd, float rt,
                                           float fxp, float fyp, float (&b)[PPQ<MODEL>::Q]) {
    constexpr int Q = PPQ<MODEL>::Q;
    constexpr float T = XF ? 0.25f : -0.25f;  // tangential: a quarter of the sum, along +y / +x
    const float rn = __fmul_rn(P.hc, rd), rq = __fmul_rn(P.hc, __fmul_rn(T, rt));
    const float rp = __fadd_rn(rn, rq), rm = __fsub_rn(rn, rq);
    FF sR{0.f, 0.f}, su{0.f, 0.f}, sv{0.f, 0.f};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int nn = XF ? lat_u<MODEL>(q) : lat_v<MODEL>(q), nt = XF ? lat_v<MODEL>(q) : lat_u<MODEL>(q);
        const bool two = nn * nn > 1 || nt * nt > 1;
        const float hc = two ? P.hc2 : P.hc, er = two ? 2.f * P.erest[q] : P.erest[q];
        float bq = __fmul_rn(0.5f, __fadd_rn(o[q], n[q])), r = 0.f;
        if (nn != 0 && nt != 0) {
            const bool same = (nn > 0) == (nt > 0);
            const float g = fmaf(same ? T : -T, __fadd_rn(tn[q], to[q]), __fsub_rn(n[q], o[q]));
            bq = fmaf(nn > 0 ? -hc : hc, g, bq);
            r = same ? rp : rm;
            bq = fmaf(nn > 0 ? -er : er, r, bq);
        } else if (nn != 0) {
            bq = fmaf(nn > 0 ? -hc : hc, __fsub_rn(n[q], o[q]), bq);
            bq = fmaf(nn > 0 ? -er : er, rn, bq);
        } else if (nt != 0) {
            bq = fmaf(nt > 0 ? -T * hc : T * hc, __fadd_rn(tn[q], to[q]), bq);
            bq = fmaf(nt > 0 ? -er : er, rq, bq);
        }
        b[q] = bq;
        ff_acc(sR, bq);
    }
    pp_first_moments<MODEL>(P, b, su, sv);
    sR = ff_norm(sR);
    // the average rsum / 2 as a pair
    const float rah2 = (float)rsum;
    const FF R = ff_add(FF{__fmul_rn(0.5f, rah2), __fmul_rn(0.5f, (float)(rsum - (double)rah2))}, sR);
    const float inv = rcp(R.hi);
    PPFace f;
    f.U = __fmul_rn(fmaf(P.hDt2, fxp, __fadd_rn(su.hi, su.lo)), inv);
    f.V = __fmul_rn(fmaf(P.hDt2, fyp, __fadd_rn(sv.hi, sv.lo)), inv);
    const FF p = cs_p(P, R);
    cs_psi(P, R, p, f.scg, f.psi, f.psil);
    f.R = R.hi;
    f.dr = __fadd_rn(sR.hi, sR.lo);  // face rho - avg(rho)
    return f;
}

// Face pass 2 of one face: equilibrium, source of the face force (fx, fy) and the flux
// xi.n of the face values relative to e_q avg(rho), of the directions that cross the face
// (the others' are not formed).
template <int MODEL, bool XF>
__device__ __forceinline__ void pp_face2(const PPP &P, const float (&b)[PPQ<MODEL>::Q], const PPFace &f, float fx,
                                         float fy, float (&out)[PPQ<MODEL>::Q]) {
    constexpr int Q = PPQ<MODEL>::Q;
    float de[Q];
    pp_deq<MODEL>(P, f.R, f.U, f.V, de);
    const float ci = __fmul_rn(P.ch, rcp(__fmul_rn(f.R, P.RT)));
    float pr[Q];
    pp_src_proj<MODEL>(P, fx, fy, f.U, f.V, pr);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        if ((XF ? lat_u<MODEL>(q) : lat_v<MODEL>(q)) == 0) continue;
        const float eq = fmaf(P.erest[q], f.R, de[q]);
        const float heq = fmaf(P.erest[q], f.dr, de[q]);  // eq - e_q avg(rho)
        const float t = fmaf(__fmul_rn(pr[q], eq), ci, fmaf(P.ah, __fsub_rn(b[q], heq), heq));
        out[q] = __fmul_rn(t, XF ? P.xi_u[q] : P.xi_v[q]);
    }
}

// Update of one cell (Ark/Cpp/DUGKS2DSolver.cpp:748-792) and its macros
// (Ark/Lib/D2Q9PP.cpp:89-109): fw, fe, fs, fn the fluxes of its west, east, south and
// north faces; rho and (px, py) = dt/V (rho_W - rho_E, rho_S - rho_N)/2 in FP64 / FP32;
// (fx, fy) the cell force of this step's collision.
struct PPCell {
    double rho, p;
    float U, V, psi, psil, scg;
};
template <int MODEL>
__device__ __forceinline__ PPCell pp_update(const PPP &P, float (&g)[PPQ<MODEL>::Q],
                                            const float (&bf)[PPQ<MODEL>::Q], const float (&fw)[PPQ<MODEL>::Q],
                                            const float (&fe)[PPQ<MODEL>::Q], const float (&fs)[PPQ<MODEL>::Q],
                                            const float (&fn)[PPQ<MODEL>::Q], double rho, float px, float py,
                                            float fx, float fy) {
    constexpr int Q = PPQ<MODEL>::Q;
    float sq[Q];
    FF sd{0.f, 0.f};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int nu = lat_u<MODEL>(q), nv = lat_v<MODEL>(q);
        float s = 0.f;  // over the faces the direction crosses
        if (nu != 0 && nv != 0) s = __fadd_rn(__fadd_rn(-__fadd_rn(fe[q], fn[q]), fw[q]), fs[q]);
        else if (nu != 0) s = __fsub_rn(fw[q], fe[q]);
        else if (nv != 0) s = __fsub_rn(fs[q], fn[q]);
        sq[q] = s;
        if (nu != 0 || nv != 0) ff_acc(sd, s);
    }
    const double drho = (double)P.dtV * ((double)sd.hi + (double)sd.lo);
    const float drf = (float)drho;
    PPCell c;
    c.rho = rho + drho;
    FF su{0.f, 0.f}, sv{0.f, 0.f};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        float inc = fmaf(P.aTP, __fsub_rn(bf[q], g[q]), __fmul_rn(P.dtV, sq[q]));
        inc = fmaf(P.erest[q], fmaf(P.xi_u[q], px, fmaf(P.xi_v[q], py, -drf)), inc);
        g[q] = __fadd_rn(g[q], inc);
    }
    pp_first_moments<MODEL>(P, g, su, sv);
    const float rh = (float)c.rho;
    const FF R{rh, (float)(c.rho - (double)rh)};
    const float inv = rcp(rh);
    c.U = __fmul_rn(fmaf(P.hDt, fx, __fadd_rn(su.hi, su.lo)), inv);
    c.V = __fmul_rn(fmaf(P.hDt, fy, __fadd_rn(sv.hi, sv.lo)), inv);
    const FF p = cs_p(P, R);
    cs_psi(P, R, p, c.scg, c.psi, c.psil);
    c.p = ff_to_double(p);
    return c;
}

}  // namespace f32
}  // namespace dugks
