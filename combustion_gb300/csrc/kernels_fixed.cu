// The plain rates kernels in fixed point (rates_fixed_core.cuh): species production rates
// (reaction.rs:356-391) and per-reaction rates of progress (reaction.rs:329-354), one cell per thread.
//
// The FP64 pipe (64 cycles per warp instruction) bounds the FP64 form of these kernels (kernels.cu): of its
// 15.7 k FP64 instructions per cell at 53 species, 4.9 k are exponentials, 4.0 k third-body sums, 1.4 k
// logarithms and divisions and 0.7 k exponents. Here the exponents, exponentials, logarithms, equilibrium
// constants and third-body sums run on the integer pipe next to it.
// Cells outside the fixed-point range (T, non-finite or non-positive state) take the FP64 form, with its
// tables read from global memory.
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "rates_cell.cuh"
#include "rates_fixed_core.cuh"

namespace cbg {

template <int KMAX>
struct CellX {
    TempsX t;
    double rcpT, Ctot;
    long long ctot;    // Ctot in the third-body sums' unit
    int m_q;           // and the position of its point
    double C[KMAX];    // concentrations, bulk last
    Word2 cw[KMAX];    // the same over S
    long long g[KMAX];  // Gibbs energies over RT, base 2, Qy
};

// Prologue of reaction.rs:362-373; false where the cell needs the FP64 form.
template <int KMAX>
__device__ __forceinline__ bool cell_setup_x(const RatesXTables& tb, double pressure_R, double T, double V,
                                             const double* const* amounts, size_t i, CellX<KMAX>& c) {
    const RatesXHeader& H = *tb.H;
    const int K = H.K, A = H.A;
    if (!(T >= kFixTmin && T < kFixTmax)) return false;
    // both reciprocals and the products rounded as the reference's: the bulk concentration is a difference of
    // totals, whose last bits it magnifies
    const double md = __drcp_rn(V);
    c.rcpT = __drcp_rn(T);
    double sum = 0.0;
    for (int k = 0; k < K - 1; k++) {
        c.C[k] = __dmul_rn(md, max0(amounts[k][i]));
        sum += c.C[k];
    }
    c.Ctot = __dmul_rn(pressure_R, c.rcpT);
    // the larger total must be a positive normal number well inside the exponent range, and the other finite
    const double S = sum > c.Ctot ? sum : c.Ctot;
    if (!(S > 1e-200 && S < 1e200 && c.Ctot > 0.0)) return false;
    c.C[K - 1] = c.Ctot - sum;
    const int ex = ((__double2hiint(S) >> 20) & 0x7ff) - 1022;  // S < 2^ex
    c.m_q = H.eff_shift + 6 - ex;
    c.ctot = dbl_to_fix(c.Ctot, c.m_q);
    if (H.n_eff)
        for (int k = 0; k < K; k++) c.cw[k] = split_word(dbl_to_fix(c.C[k], kCq + kLo - ex));
    c.t = make_temps(H, T, c.rcpT);
    for (int k = 0; k < A; k++) {
        const SpeciesX& s = tb.species[k];
        if (!(s.need_exp | s.need_exp_neg)) continue;
        c.g[k] = gibbs_log2(s, c.t);
    }
    return true;
}

template <int MODEL, bool SUM, int KMAX, class Emit>
__device__ __forceinline__ void plain_group_x(const RatesXTables& tb, const CellX<KMAX>& c, double* w, Emit emit) {
#pragma unroll 1
    for (int r = MODEL ? tb.H->group_end[MODEL - 1] : 0; r < tb.H->group_end[MODEL]; r++)
        reaction_x<MODEL != 1, SUM>(
            tb, r, c, w, [&](const ArrheniusX& k) { return rate_constant(k, c.t); }, emit);
}

// Third-body concentration of a row from its two partial sums (reaction.rs:141-145): Ctot + sum (e - 1) C.
template <class CellT>
__device__ __forceinline__ double third_body(const CellT& c, long long s1, long long s2) {
    return fix_to_dbl(c.ctot + (s1 << 6) + ((s2 + (1ll << (kLo - 7))) >> (kLo - 6)), c.m_q);
}

// Models 2-5: the third-body sums of four consecutive rows in one pass over the concentrations (three
// mad.wide per term), just before their reactions.
template <bool SUM, int KMAX, class Emit>
__device__ __forceinline__ void third_body_groups_x(const RatesXTables& tb, const CellX<KMAX>& c, double* w, Emit emit) {
    const RatesXHeader& H = *tb.H;
    const int K = H.K, r_begin = H.group_end[1], r_end = H.group_end[5];
    for (int r0 = r_begin; r0 < r_end; r0 += 4) {
        const Word2* E = tb.eff + (size_t)(r0 - r_begin) * K;
        long long s1[4] = {0, 0, 0, 0}, s2[4] = {0, 0, 0, 0};
        for (int k = 0; k < K; k++) {
            const Word2 ck = c.cw[k];
#pragma unroll
            for (int q = 0; q < 4; q++) dot_term(E[q * K + k], ck, s1[q], s2[q]);
        }
        const double M0 = third_body(c, s1[0], s2[0]), M1 = third_body(c, s1[1], s2[1]);
        const double M2 = third_body(c, s1[2], s2[2]), M3 = third_body(c, s1[3], s2[3]);
        const int rq = min(r_end - r0, 4);
#pragma unroll 1
        for (int q = 0; q < rq; q++) {
            const int r = r0 + q;
            const double M = q == 0 ? M0 : q == 1 ? M1 : q == 2 ? M2 : M3;
            const FalloffX* f = tb.falloff + (r - r_begin);
            auto forward = [&](const ArrheniusX& k) {
                if (r < H.group_end[2]) return forward_x<2>(H, k, f, c.t, c.rcpT, M);
                if (r < H.group_end[3]) return forward_x<3>(H, k, f, c.t, c.rcpT, M);
                if (r < H.group_end[4]) return forward_x<4>(H, k, f, c.t, c.rcpT, M);
                return forward_x<5>(H, k, f, c.t, c.rcpT, M);
            };
            reaction_x<true, SUM>(tb, r, c, w, forward, emit);
        }
    }
}

template <int KMAX>
__device__ __forceinline__ bool rates_cell_x(const RatesXTables& tb, const RatesArgs<KMAX>& io, size_t i) {
    const RatesXHeader& H = *tb.H;
    const int K = H.K, A = H.A;
    const bool uniform = io.flags & kUniformPressure;
    const double T = io.in[2][i], V = io.in[3][i];
    CellX<KMAX> c;
    if (!cell_setup_x<KMAX>(tb, uniform ? io.in[0][0] : io.in[0][i], T, V, io.in + 4, i, c)) return false;
    double wdot[KMAX];
    for (int k = 0; k < A; k++) wdot[k] = 0.0;
    auto none = [](int, double) {};
    plain_group_x<0, true>(tb, c, wdot, none);
    plain_group_x<1, true>(tb, c, wdot, none);
    third_body_groups_x<true>(tb, c, wdot, none);
    // Energy and volume (reaction.rs:375-384).
    double E = 0.0, Cp = 0.0, dtE = 0.0;
#pragma unroll 1
    for (int k = 0; k < A; k++) {
        const ThermoX& s = tb.thermo[k];
        const int set = piece_x(s.split, T);
        E = fma(wdot[k], enthalpy_x(s, set, c.t), E);
        Cp = fma(heat_capacity_x(s, set, c.t), c.C[k], Cp);
        dtE = fma(s.dtE, wdot[k], dtE);
    }
#pragma unroll 1
    for (int k = A; k < K; k++) Cp = fma(heat_capacity_x(tb.thermo[k], piece_x(tb.thermo[k].split, T), c.t), c.C[k], Cp);
    const double dtT_T = div64(-E, Cp), rcp_pressure_R = uniform ? io.in[1][0] : io.in[1][i];
    io.out[0][i] = T * dtT_T;
    io.out[1][i] = V * fma(rcp_pressure_R * T, dtE, dtT_T);
    for (int k = 0; k < A; k++) io.out[2 + k][i] = wdot[k];
    return true;
}

template <int KMAX>
__device__ __forceinline__ bool reaction_rates_cell_x(const RatesXTables& tb, const ReactionRatesArgs<KMAX>& io,
                                                      size_t i) {
    CellX<KMAX> c;
    if (!cell_setup_x<KMAX>(tb, io.in[0][i], io.in[1][i], io.in[2][i], io.in + 3, i, c)) return false;
    auto store = [&](int orig, double cR) { io.out[orig][i] = cR; };
    plain_group_x<0, false>(tb, c, nullptr, store);
    plain_group_x<1, false>(tb, c, nullptr, store);
    third_body_groups_x<false>(tb, c, nullptr, store);
    return true;
}

// The FP64 form of one cell, out of line: it is rarely taken.
template <int KMAX>
__device__ __noinline__ void rates_cell_f64(const RatesArgs<KMAX>& io, size_t i) {
    rates_cell<KMAX>(RatesTables(io.f64_tab), io, i);
}
template <int KMAX>
__device__ __noinline__ void reaction_rates_cell_f64(const ReactionRatesArgs<KMAX>& io, size_t i) {
    reaction_rates_cell<KMAX>(RatesTables(io.f64_tab), io, i);
}

// The tables into shared memory, or only the functions' tables (the rest is then read through L1).
template <bool SMEM>
__device__ __forceinline__ bool stage_x(const uint8_t* gtab, uint32_t tab_bytes, uint64_t* bar, int* status) {
    if (SMEM) return stage_to_shared(cb_dsmem, gtab, tab_bytes, bar, status);
    const double* src = reinterpret_cast<const double*>(gtab);
    double* dst = reinterpret_cast<double*>(cb_dsmem);
    for (int q = threadIdx.x; q < (kMathBytes + kFixMathBytes) / 8; q += blockDim.x) dst[q] = src[q];
    __syncthreads();
    return true;
}

// The block's warps start each round of cells together: left to drift over tens of rounds they run different
// parts of the program at one time and miss the instruction cache (2^22 cells at 53 species 47.1 -> 37.3 ms).
template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(kRatesXBlock) rates_x_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                                        const __grid_constant__ RatesArgs<KMAX> io, size_t n,
                                                        int* status) {
    __shared__ uint64_t bar;
    if (!stage_x<SMEM>(gtab, tab_bytes, &bar, status)) return;
    const RatesXTables tb(SMEM ? cb_dsmem : gtab);
    for (size_t b = (size_t)blockIdx.x * blockDim.x; b < n; b += (size_t)gridDim.x * blockDim.x) {
        __syncthreads();
        const size_t i = b + threadIdx.x;
        if (i < n && !rates_cell_x<KMAX>(tb, io, i)) rates_cell_f64<KMAX>(io, i);
    }
}

template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(kRatesXBlock) reaction_rates_x_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                                                 const __grid_constant__ ReactionRatesArgs<KMAX> io,
                                                                 size_t n, int* status) {
    __shared__ uint64_t bar;
    if (!stage_x<SMEM>(gtab, tab_bytes, &bar, status)) return;
    const RatesXTables tb(SMEM ? cb_dsmem : gtab);
    for (size_t b = (size_t)blockIdx.x * blockDim.x; b < n; b += (size_t)gridDim.x * blockDim.x) {
        __syncthreads();
        const size_t i = b + threadIdx.x;
        if (i < n && !reaction_rates_cell_x<KMAX>(tb, io, i)) reaction_rates_cell_f64<KMAX>(io, i);
    }
}

CB_DISPATCH(launch_rates_x, rates_x_kernel, RatesArgs, kRatesXBlock, kMathBytes + kFixMathBytes, true)
CB_DISPATCH(launch_reaction_rates_x, reaction_rates_x_kernel, ReactionRatesArgs, kRatesXBlock, kMathBytes + kFixMathBytes, true)
CB_WAVE(wave_rates_x, rates_x_kernel, kRatesXBlock, kMathBytes + kFixMathBytes)
CB_WAVE(wave_reaction_rates_x, reaction_rates_x_kernel, kRatesXBlock, kMathBytes + kFixMathBytes)

cudaError_t set_stage_wait_polls_x(long long polls) { return cudaMemcpyToSymbol(g_stage_wait_polls, &polls, sizeof polls); }

}  // namespace cbg
