// Initial states on the device.
//
// Every initialisation (host_init_plane, host_params.cpp) is one field -- the phase field of the
// Allen-Cahn models, the density of the pseudopotential ones -- and the fluid at rest: all other
// planes follow from it by a few products and sums.  The host evaluates the field (its tanh and
// cos are the reference's, and differ from the device's in the last place) and copies that one
// plane; a kernel per storage form writes the rest, each operation rounded separately (this
// file is compiled without contraction), so the state is the one an upload of the whole host-made
// state gives, bit for bit.  A 512x512 state is 34 or 32 planes of 2 MB: 16 ms (Allen-Cahn) and 22 ms
// (D2V16) to make on one host thread and copy, which set the pace of the serving loop's
// admission; now 0.8 and 0.7 ms (the 24-case serving mix: 172 -> 93 ms).
#include <cuda_runtime.h>

#include <cstdint>

#include "dugks_device.cuh"
#include "fp32_state.cuh"

namespace dugks {

namespace {

__device__ __forceinline__ bool cell_at(const Params &P, size_t &c) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, j = t / (unsigned)P.nx;  // at most 2^31 cells
    c = (size_t)j * P.pitch + (t - j * (unsigned)P.nx);
    return j < (unsigned)P.ny;
}

// Allen-Cahn: rho = aPhi phi + bPhi, p = p0 = 1, tau from the header's viscosity, h_q = w_q phi,
// f_q its rest value (f9)
struct F9 {
    double v[9];
};
__global__ void __launch_bounds__(256) k_init_ac64(Params P, State S, F9 f9) {
    size_t c;
    if (!cell_at(P, c)) return;
    const double phi = S.fld[F_PHI][c], rho = P.aPhi * phi + P.bPhi;
    S.fld[F_RHO][c] = rho;
    S.fld[F_P][c] = 1.0;
    S.fld[F_TAU][c] = P.NuL / (rho * P.RT);
    for (int q = 0; q < 9; ++q) {
        S.h[(size_t)q * S.qs + c] = d2q9_w(q) * phi;
        S.f[(size_t)q * S.qs + c] = f9.v[q];
    }
}

// the same into the deviation storage (fp32_state.cuh); df9: f_q less the rest value it is stored from
template <typename R>
__global__ void __launch_bounds__(256) k_init_dev(Params P, f32::SR<R> S, const double *__restrict__ field, F9 df9) {
    size_t c;
    if (!cell_at(P, c)) return;
    const size_t qs = S.qs;
    const double phi = field[c], rho = P.aPhi * phi + P.bPhi;
    double hq[9], ph = 0.0;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        hq[q] = d2q9_w(q) * phi;
        ph += hq[q];
        S.df[(size_t)q * qs + c] = (R)df9.v[q];
    }
    const R hi = (R)ph;
    S.phi[c] = hi;
    S.phi[qs + c] = (R)(ph - (double)hi);
#pragma unroll
    for (int q = 1; q < 9; ++q) S.dg[(size_t)(q - 1) * qs + c] = (R)(hq[q] - d2q9_w(q) * ph);
#pragma unroll
    for (int k = 0; k < f32::A_N; ++k) S.aux[(size_t)k * qs + c] = R(0);
#pragma unroll
    for (int k = 0; k < f32::I_N; ++k) {
        R v = R(0);
        if (k == f32::I_DPHI) v = (R)(phi - DUGKS_F32_PHI0);
        if (k == f32::I_RHO) v = (R)rho;
        if (k == f32::I_TAU) v = (R)(P.NuL / (rho * P.RT));
        S.init[(size_t)k * qs + c] = v;
    }
}

// Equilibrium at rest of the pseudopotential models: w rho, or the inverse moment matrix times the
// moments at u = 0 (the terms of the vanishing moments add exact zeros)
struct Rest16 {
    double m[16][6];  // the matrix's columns 0, 3, 5, 6, 14, 15
};
template <int MODEL>
__device__ __forceinline__ double rest_eq(const Params &P, const Rest16 &A, double rho, int q) {
    if (MODEL == PP9) return P.omega[q] * rho;
    const double RT = P.RT, p = rho * RT, m3 = rho * (3.0 * RT), m14 = 5.0 * rho * RT * RT;
    return A.m[q][0] * rho + A.m[q][1] * m3 + A.m[q][2] * p + A.m[q][3] * p + A.m[q][4] * m14 + A.m[q][5] * m14;
}
template <int MODEL>
__global__ void __launch_bounds__(256) k_init_pp64(Params P, State S, Rest16 A) {
    size_t c;
    if (!cell_at(P, c)) return;
    const double rho = S.fld[F_RHO][c];
    S.fld[F_P][c] = rho * P.RT;
    S.fld[F_TAU][c] = P.Tau0;
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    for (int q = 0; q < Q; ++q) S.f[(size_t)q * S.qs + c] = rest_eq<MODEL>(P, A, rho, q);
}
template <int MODEL>
__global__ void __launch_bounds__(256) k_init_pp32(Params P, f32::PPP C, f32::PPS S, Rest16 A) {
    size_t c;
    if (!cell_at(P, c)) return;
    const double rho = S.rho[c];
    S.p[c] = rho * P.RT;
    S.U[c] = 0.0;
    S.V[c] = 0.0;
    constexpr int Q = MODEL == PP16 ? 16 : 9;
    for (int q = 0; q < Q; ++q)
        S.df[(size_t)q * S.qs + c] = (float)(rest_eq<MODEL>(P, A, rho, q) - (double)C.erest[q] * rho);
}

Rest16 rest_columns(const double iM[16][16]) {
    Rest16 A;
    const int k[6] = {0, 3, 5, 6, 14, 15};
    for (int q = 0; q < 16; ++q)
        for (int i = 0; i < 6; ++i) A.m[q][i] = iM[q][k[i]];
    return A;
}
dim3 init_grid(const Params &P) { return dim3((unsigned)(((size_t)P.nx * P.ny + 255) / 256)); }

}  // namespace

// The plain FP64 state from its field (phi or rho, in place in S.fld); f9: rest values of f
// (Allen-Cahn), iM: the D2V16 matrix.  The caller has cleared the other fields.
cudaError_t launch_init64(const Params &P, const State &S, const double *f9, const double iM[16][16], cudaStream_t st,
                          int64_t *launches) {
    if (P.model == AC || P.model == HCZ) {
        F9 f;
        for (int q = 0; q < 9; ++q) f.v[q] = f9[q];
        k_init_ac64<<<init_grid(P), 256, 0, st>>>(P, S, f);
    } else if (P.model == PP16) {
        k_init_pp64<PP16><<<init_grid(P), 256, 0, st>>>(P, S, rest_columns(iM));
    } else {
        k_init_pp64<PP9><<<init_grid(P), 256, 0, st>>>(P, S, Rest16{});
    }
    *launches += 1;
    return cudaGetLastError();
}
// the deviation-form state from its phase field [ny][pitch]
template <typename R>
cudaError_t launch_init_dev(const Params &P, const f32::SR<R> &S, const double *field, const double *df9, cudaStream_t st,
                            int64_t *launches) {
    F9 f;
    for (int q = 0; q < 9; ++q) f.v[q] = df9[q];
    k_init_dev<R><<<init_grid(P), 256, 0, st>>>(P, S, field, f);
    *launches += 1;
    return cudaGetLastError();
}
template cudaError_t launch_init_dev<float>(const Params &, const f32::SR<float> &, const double *, const double *,
                                            cudaStream_t, int64_t *);
template cudaError_t launch_init_dev<double>(const Params &, const f32::SR<double> &, const double *, const double *,
                                             cudaStream_t, int64_t *);
// the FP32 pseudopotential state from its density (in place in S.rho)
cudaError_t launch_init_pp32(const Params &P, const f32::PPP &C, const f32::PPS &S, const double iM[16][16],
                             cudaStream_t st, int64_t *launches) {
    if (P.model == PP16) k_init_pp32<PP16><<<init_grid(P), 256, 0, st>>>(P, C, S, rest_columns(iM));
    else k_init_pp32<PP9><<<init_grid(P), 256, 0, st>>>(P, C, S, Rest16{});
    *launches += 1;
    return cudaGetLastError();
}

}  // namespace dugks
