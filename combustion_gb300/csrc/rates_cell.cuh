// One cell of the plain FP64 rates program per thread (reaction.rs:207-391) and of its per-reaction rates
// (reaction.rs:329-354): the form of every temperature and mechanism.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "device_math.cuh"
#include "kernels.h"
#include "rates_core.cuh"
#include "tables.h"

namespace cbg {

template <int KMAX>
struct Cell {
    Temps t;
    double Ctot, C0, rcpC0, rcpC0sq;
    double C[KMAX];              // concentrations, bulk last
    double ex[KMAX], exn[KMAX];  // min(M3, exp(g_k)), min(cbrt(f32::MAX), exp(-g_k))
};

// Prologue of reaction.rs:362-373 and the Gibbs exponentials of reaction.rs:234-263.
template <int KMAX>
__device__ __forceinline__ void cell_setup(const RatesTables& tb, double pressure_R, double T, double V,
                                           const double* const* amounts, size_t i, Cell<KMAX>& c) {
    const RatesHeader& H = *tb.H;
    const int K = H.K, A = H.A;
    const double md = rcp64(V);
    c.t.T = T;
    c.t.rcpT = rcp64(T);
    c.t.lnT = log64(T);
    c.t.T2 = T * T;
    c.t.T3 = T * c.t.T2;
    c.t.T4 = c.t.T2 * c.t.T2;
    c.t.rcpT2 = c.t.rcpT * c.t.rcpT;
    double sum = 0.0;
    for (int k = 0; k < K - 1; k++) {
        c.C[k] = md * max0(amounts[k][i]);
        sum += c.C[k];
    }
    c.Ctot = pressure_R * c.t.rcpT;
    c.C[K - 1] = c.Ctot - sum;
    c.C0 = H.C0 * c.t.rcpT;
    c.rcpC0 = H.rcp_C0 * T;
    c.rcpC0sq = c.rcpC0 * c.rcpC0;
    for (int k = 0; k < A; k++) {
        const Species& s = tb.species[k];
        if (!(s.need_exp | s.need_exp_neg)) continue;
        const double* g = s.g[piece_of(s.split, T)];
        const double x = fma(g[6], c.t.rcpT, fma(g[5], c.t.T4, fma(g[4], c.t.T3, fma(g[3], c.t.T2,
                         fma(g[2], T, fma(g[1], c.t.lnT, g[0]))))));
        if (s.need_exp) c.ex[k] = min_pos(H.M3, exp64(x));
        if (s.need_exp_neg) c.exn[k] = min_pos(H.cbrt_max, exp64(-x));
    }
}

// Reactions without a third body (models 0 and 1), one loop per model; emit(x, cR) takes each rate.
template <int KMAX, int MODEL, class Emit>
__device__ __forceinline__ void plain_group(const RatesTables& tb, const Cell<KMAX>& c, Emit emit) {
    for (int r = MODEL ? tb.H->group_end[MODEL - 1] : 0; r < tb.H->group_end[MODEL]; r++) {
        const Reaction& x = tb.reactions[r];
        emit(x, reaction_rate<MODEL>(tb, x, c, 0.0));
    }
}

// Reactions with a third body (models 2-5: consecutive in the tables, efficiency row e for reaction
// group_end[1] + e). The third-body sums efficiency() (reaction.rs:141-145) of four consecutive rows
// (padded to a multiple of 4) take one pass over the concentrations, one local load of C_k per four
// FMAs, just before their reactions: no array of sums is kept. The model branch is uniform across the
// warp (every lane is at the same reaction).
template <int KMAX, class Emit>
__device__ __forceinline__ void third_body_groups(const RatesTables& tb, const Cell<KMAX>& c, Emit emit) {
    const RatesHeader& H = *tb.H;
    const int K = H.K, r_begin = H.group_end[1], r_end = H.group_end[5];
    for (int r0 = r_begin; r0 < r_end; r0 += 4) {
        const double* E = tb.eff + (size_t)(r0 - r_begin) * K;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        for (int k = 0; k < K; k++) {
            const double ck = c.C[k];
#pragma unroll
            for (int q = 0; q < 4; q++) s[q] = fma(E[q * K + k], ck, s[q]);
        }
        const double M0 = c.Ctot + s[0], M1 = c.Ctot + s[1], M2 = c.Ctot + s[2], M3 = c.Ctot + s[3];
        const int rq = min(r_end - r0, 4);
#pragma unroll 1
        for (int q = 0; q < rq; q++) {
            const int r = r0 + q;
            const double M = q == 0 ? M0 : q == 1 ? M1 : q == 2 ? M2 : M3;  // integer selects
            const Reaction& x = tb.reactions[r];
            double cR;
            if (r < H.group_end[2]) cR = reaction_rate<2>(tb, x, c, M);
            else if (r < H.group_end[3]) cR = reaction_rate<3>(tb, x, c, M);
            else if (r < H.group_end[4]) cR = reaction_rate<4>(tb, x, c, M);
            else cR = reaction_rate<5>(tb, x, c, M);
            emit(x, cR);
        }
    }
}

template <int KMAX>
__device__ void rates_cell(const RatesTables& tb, const RatesArgs<KMAX>& io, size_t i) {
    const RatesHeader& H = *tb.H;
    const int K = H.K, A = H.A;
    const bool uniform = io.flags & kUniformPressure;
    const double pressure_R = uniform ? io.in[0][0] : io.in[0][i];
    const double rcp_pressure_R = uniform ? io.in[1][0] : io.in[1][i];
    const double T = io.in[2][i], V = io.in[3][i];
    Cell<KMAX> c;
    cell_setup<KMAX>(tb, pressure_R, T, V, io.in + 4, i, c);
    double wdot[KMAX];
    for (int k = 0; k < A; k++) wdot[k] = 0.0;
    // species_rates (reaction.rs:312-327), reactions grouped by model
    // read-modify-writes in pairs, the two reads issued together (net species are distinct)
    auto accumulate = [&](const Reaction& x, double cR) {
#pragma unroll 1
        for (int q = 0; q < x.n_net; q += 2) {
            const int k0 = x.net_k[q], k1 = x.net_k[q + 1 < x.n_net ? q + 1 : q];
            const double w0 = wdot[k0], w1 = wdot[k1];
            wdot[k0] = fma(small_int_to_double(x.net_n[q]), cR, w0);
            if (q + 1 < x.n_net) wdot[k1] = fma(small_int_to_double(x.net_n[q + 1]), cR, w1);
        }
    };
    plain_group<KMAX, 0>(tb, c, accumulate);
    plain_group<KMAX, 1>(tb, c, accumulate);
    third_body_groups<KMAX>(tb, c, accumulate);
    // Energy and volume (reaction.rs:375-384).
    double E = 0.0;
    for (int k = 0; k < A; k++) {
        const Species& s = tb.species[k];
        const double* h = s.h[piece_of(s.split, T)];
        const double hk = fma(h[5], c.t.rcpT, fma(h[4], c.t.T4, fma(h[3], c.t.T3, fma(h[2], c.t.T2, fma(h[1], T, h[0])))));
        E = fma(wdot[k], hk, E);
    }
    double Cp = 0.0;
    for (int k = 0; k < K; k++) {
        const Species& s = tb.species[k];
        const double* cp = s.cp[piece_of(s.split, T)];
        const double ck = fma(cp[4], c.t.T4, fma(cp[3], c.t.T3, fma(cp[2], c.t.T2, fma(cp[1], T, cp[0]))));
        Cp = fma(ck, c.C[k], Cp);
    }
    const double dtT_T = div64(-E, Cp);
    double dtE = 0.0;
    for (int k = 0; k < A; k++) dtE = fma(tb.species[k].dtE, wdot[k], dtE);
    io.out[0][i] = T * dtT_T;
    io.out[1][i] = V * fma(rcp_pressure_R * T, dtE, dtT_T);
    for (int k = 0; k < A; k++) io.out[2 + k][i] = wdot[k];
}

template <int KMAX>
__device__ void reaction_rates_cell(const RatesTables& tb, const ReactionRatesArgs<KMAX>& io, size_t i) {
    Cell<KMAX> c;
    cell_setup<KMAX>(tb, io.in[0][i], io.in[1][i], io.in[2][i], io.in + 3, i, c);
    auto store = [&](const Reaction& x, double cR) { io.out[x.orig][i] = cR; };
    plain_group<KMAX, 0>(tb, c, store);
    plain_group<KMAX, 1>(tb, c, store);
    third_body_groups<KMAX>(tb, c, store);
}

}  // namespace cbg
