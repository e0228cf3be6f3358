// The plain rates kernels in fixed point (rates_fixed_core.cuh): species production rates
// (reaction.rs:356-391) and per-reaction rates of progress (reaction.rs:329-354), one cell per thread.
//
// The FP64 pipe (64 cycles per warp instruction) bounds the FP64 form of these kernels (kernels.cu): of its
// 15.7 k FP64 instructions per cell at 53 species, 4.9 k are exponentials, 4.0 k third-body sums, 1.4 k
// logarithms and divisions and 0.7 k exponents. Here the exponents, exponentials, logarithms, equilibrium
// constants and third-body sums run on the integer pipe next to it.
// Cells outside the fixed-point range (T, non-finite or non-positive state) take the FP64 form, with its
// tables read from global memory: 2^19 cells of 53 species above 8,192 K 17.5 ms (5.5 in range, 16.2 in the FP64 kernel,
// whose tables are in shared memory), in a mixed field up to the sum of both forms; one of them alone 0.94 ms (0.83).
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
    long long ctot;    // Ctot over S, Q60
    int ex;            // S = 2^ex
    double C[KMAX];    // concentrations, bulk last
    Word2 cw[KMAX];    // the same over S, Q60
    long long g[KMAX];  // Gibbs energies over RT, base 2, Qy
};

// e with S < 2^e, S positive and normal.
__device__ __forceinline__ int exponent_above_x(double S) { return ((__double2hiint(S) >> 20) & 0x7ff) - 1022; }

// The larger total S is a positive normal number well inside the exponent range and the other one not negative: every
// concentration is finite and at most S. (False for a NaN sum, of a NaN amount, and for a negative one, of a negative volume.)
__device__ __forceinline__ bool totals_in_range(double sum, double Ctot, double S) {
    return sum >= 0.0 && Ctot > 0.0 && S > 1e-200 && S < 1e200;
}

// Prologue of reaction.rs:362-373; false where the cell needs the FP64 form.
template <int KMAX>
__device__ __forceinline__ bool cell_setup_x(const RatesXTables& tb, double pressure_R, double T, double V,
                                             const double* const* amounts, size_t i, CellX<KMAX>& c) {
    const RatesXHeader& H = *tb.H;
    const int K = H.K, A = H.A;
    if (!(T >= H.Tmin && T < kFixTmax)) return false;
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
    const double S = sum > c.Ctot ? sum : c.Ctot;
    if (!totals_in_range(sum, c.Ctot, S)) return false;
    c.C[K - 1] = c.Ctot - sum;
    c.ex = exponent_above_x(S);
    c.ctot = dbl_to_fix(c.Ctot, 60 - c.ex);
    if (H.n_eff)
        for (int k = 0; k < K; k++) c.cw[k] = split_word<kThirdLo>(dbl_to_fix(c.C[k], 60 - c.ex));
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

// Third-body concentration of a row from its two partial sums (reaction.rs:141-145): Ctot + sum (e - 1) C, in the unit of
// its four rows, 2^-(q + 30) S.
__device__ __forceinline__ long long third_body_total(long long ctot, int q) { return (ctot + (1ll << (29 - q))) >> (30 - q); }
__device__ __forceinline__ double third_body(long long total, int unit, long long s1, long long s2) {
    return fix_to_dbl(total + s1 + ((s2 + (1ll << (kThirdLo - 1))) >> kThirdLo), unit);
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
        const int eq = tb.eff_q[(r0 - r_begin) >> 2], unit = eq + 30 - c.ex;
        const long long total = third_body_total(c.ctot, eq);
        const double M0 = third_body(total, unit, s1[0], s2[0]), M1 = third_body(total, unit, s1[1], s2[1]);
        const double M2 = third_body(total, unit, s1[2], s2[2]), M3 = third_body(total, unit, s1[3], s2[3]);
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
__device__ __noinline__ void rates_cell_f64(const uint8_t* f64_tab, const RatesArgs<KMAX>& io, size_t i) {
    rates_cell<KMAX>(RatesTables(f64_tab), io, i);
}
template <int KMAX>
__device__ __noinline__ void reaction_rates_cell_f64(const uint8_t* f64_tab, const ReactionRatesArgs<KMAX>& io, size_t i) {
    reaction_rates_cell<KMAX>(RatesTables(f64_tab), io, i);
}
// The FP64 tables in place of the others in the block's shared memory, or where they are when they do not fit: one thread
// reads them, one entry after the other (a state of 53 species above 8,192 K 940 us, from global memory 1,330).
__device__ __forceinline__ const uint8_t* stage_f64(const uint8_t* f64_tab) {
    const uint32_t bytes = (uint32_t)reinterpret_cast<const RatesHeader*>(f64_tab + kMathBytes)->total_bytes;
    uint32_t room;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(room));
    if (bytes > room) return f64_tab;
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < bytes / 16; q += blockDim.x)
        reinterpret_cast<uint4*>(cb_dsmem)[q] = reinterpret_cast<const uint4*>(f64_tab)[q];
    __syncthreads();
    return cb_dsmem;
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
    let_next_start();
    __shared__ uint64_t bar;
    if (!stage_x<SMEM>(gtab, tab_bytes, &bar, status)) return;
    const RatesXTables tb(SMEM ? cb_dsmem : gtab);
    for (size_t b = (size_t)blockIdx.x * blockDim.x; b < n; b += (size_t)gridDim.x * blockDim.x) {
        __syncthreads();
        const size_t i = b + threadIdx.x;
        if (i < n && !rates_cell_x<KMAX>(tb, io, i)) rates_cell_f64<KMAX>(io.f64_tab, io, i);
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
        if (i < n && !reaction_rates_cell_x<KMAX>(tb, io, i)) reaction_rates_cell_f64<KMAX>(io.f64_tab, io, i);
    }
}

// ---------------------------------------------------------------------------------------------------
// One cell per warp, for calls too small to fill the GPU with one per thread: lanes share out species, third-body
// rows and reactions; every FP64 sum runs on one lane in the thread form's order (the integer sums are exact), so that
// a cell has the same bits in both forms.
// TEAM warps (a block of its own) share a cell in calls of at most a cell per SM, 1 otherwise.
constexpr int kRatesWarps = 16;  // cells per block at most

template <int KMAX>
struct CellXW {
    TempsX t;
    double rcpT, Ctot;
    long long ctot;
    int ex;
    const double* C;
    const long long* g;
};

// The cell's rates of progress into cR [R] (grouped order); the concentrations stay in sh, followed by two free arrays
// of K doubles and the species rates'. False where the cell needs the FP64 form (the same for all
// its lanes). lane: of all of the cell's.
template <int TEAM, int KMAX>
__device__ __forceinline__ bool cell_progress_warp(const RatesXTables& tb, double pressure_R, double T, double V,
                                                   const double* const* amounts, size_t i, double* sh, int lane,
                                                   CellXW<KMAX>& c) {
    constexpr int kStep = 32 * TEAM;
    const RatesXHeader& H = *tb.H;
    const int K = H.K, A = H.A;
    if (!(T >= H.Tmin && T < kFixTmax)) return false;
    double* C = sh;
    double* cw = sh + K;
    long long* g = reinterpret_cast<long long*>(sh + 2 * K);
    double* M = sh + 4 * K;
    double* cR = M + H.n_eff;
    const double md = __drcp_rn(V);
    c.rcpT = __drcp_rn(T);
    for (int k = lane; k < K - 1; k += kStep) C[k] = __dmul_rn(md, max0(amounts[k][i]));
    team_sync<TEAM>();
    double sum = 0.0;
    if (lane == 0) {
#pragma unroll 4
        for (int k = 0; k < K - 1; k++) sum += C[k];
    }
    sum = team_value<TEAM>(sum, sh + 3 * K, lane);
    c.Ctot = __dmul_rn(pressure_R, c.rcpT);
    const double S = sum > c.Ctot ? sum : c.Ctot;
    if (!totals_in_range(sum, c.Ctot, S)) return false;
    if (lane == 0) C[K - 1] = c.Ctot - sum;
    team_sync<TEAM>();
    c.ex = exponent_above_x(S);
    c.ctot = dbl_to_fix(c.Ctot, 60 - c.ex);
    c.t = make_temps(H, T, c.rcpT);
    c.C = C;
    c.g = g;
    for (int k = lane; k < K; k += kStep) {
        const Word2 w = split_word<kThirdLo>(dbl_to_fix(C[k], 60 - c.ex));
        cw[k] = __hiloint2double(w.hi, w.lo);
        if (k < A && (tb.species[k].need_exp | tb.species[k].need_exp_neg)) g[k] = gibbs_log2(tb.species[k], c.t);
    }
    team_sync<TEAM>();
    for (int e = lane; e < H.n_eff; e += kStep) {
        const Word2* E = tb.eff + (size_t)e * K;
        long long s1 = 0, s2 = 0;
#pragma unroll 4
        for (int k = 0; k < K; k++) dot_term(E[k], Word2{__double2hiint(cw[k]), __double2loint(cw[k])}, s1, s2);
        const int eq = tb.eff_q[e >> 2];
        M[e] = third_body(third_body_total(c.ctot, eq), eq + 30 - c.ex, s1, s2);
    }
    team_sync<TEAM>();
    const int first = H.group_end[1];
    int turn = 0;  // the warp that takes the model's first 32 reactions
#pragma unroll 1
    for (int m = 0; m < 6; m++) {  // one model's program at a time
        const int begin = m ? H.group_end[m - 1] : 0;
        const int mine = TEAM == 1 ? 0 : ((lane >> 5) - turn + TEAM) % TEAM;
        if (TEAM > 1) turn = (turn + (H.group_end[m] - begin + 31) / 32) % TEAM;
#pragma unroll 1
        for (int r = begin + 32 * mine + (lane & 31); r < H.group_end[m]; r += kStep) {
            auto store = [&](int, double v) { cR[r] = v; };
            if (m == 1) {
                reaction_x<false, false>(tb, r, c, nullptr, [&](const ArrheniusX& k) { return rate_constant(k, c.t); }, store);
            } else {
                auto forward = [&](const ArrheniusX& k) {
                    if (m == 0) return rate_constant(k, c.t);
                    const FalloffX* f = tb.falloff + (r - first);
                    if (m == 2) return forward_x<2>(H, k, f, c.t, c.rcpT, M[r - first]);
                    if (m == 3) return forward_x<3>(H, k, f, c.t, c.rcpT, M[r - first]);
                    if (m == 4) return forward_x<4>(H, k, f, c.t, c.rcpT, M[r - first]);
                    return forward_x<5>(H, k, f, c.t, c.rcpT, M[r - first]);
                };
                reaction_x<true, false>(tb, r, c, nullptr, forward, store);
            }
        }
    }
    team_sync<TEAM>();
    return true;
}

template <int TEAM, int KMAX>
__device__ __forceinline__ bool rates_cell_warp(const RatesXTables& tb, const RatesArgs<KMAX>& io, size_t i, double* sh,
                                                int lane) {
    constexpr int kStep = 32 * TEAM;
    const RatesXHeader& H = *tb.H;
    const int K = H.K, A = H.A;
    const bool uniform = io.flags & kUniformPressure;
    const double T = io.in[2][i], V = io.in[3][i], rcp_pressure_R = uniform ? io.in[1][0] : io.in[1][i];
    CellXW<KMAX> c;
    if (!cell_progress_warp<TEAM, KMAX>(tb, uniform ? io.in[0][0] : io.in[0][i], T, V, io.in + 4, i, sh, lane, c)) return false;
    double *C = sh, *h = sh + K, *cp = sh + 2 * K, *w = sh + 3 * K, *cR = sh + 4 * K + H.n_eff;
    for (int k = lane; k < K; k += kStep) {
        if (k < A) {
            double v = 0.0;
            const int end = tb.csr_start[k + 1];
#pragma unroll 4
            for (int q = tb.csr_start[k]; q < end; q++) {
                const int e = tb.csr[q];
                v = fma(small_int_to_double((int)(int8_t)(e & 0xff)), cR[e >> 8], v);
            }
            w[k] = v;
            io.out[2 + k][i] = v;
        }
        const ThermoX& s = tb.thermo[k];
        const int set = piece_x(s.split, T);
        if (k < A) h[k] = enthalpy_x(s, set, c.t);
        cp[k] = heat_capacity_x(s, set, c.t);
    }
    team_sync<TEAM>();
    double acc = 0.0;  // E, Cp and dtE on lanes 0, 1, 2
    if (lane < 3) {
        const int n = lane == 1 ? K : A;
#pragma unroll 4
        for (int k = 0; k < n; k++)
            acc = fma(lane == 0 ? w[k] : lane == 1 ? cp[k] : tb.thermo[k].dtE, lane == 0 ? h[k] : lane == 1 ? C[k] : w[k], acc);
    }
    const double E = __shfl_sync(0xffffffffu, acc, 0), Cp = __shfl_sync(0xffffffffu, acc, 1),
                 dtE = __shfl_sync(0xffffffffu, acc, 2);
    if (lane == 0) {
        const double dtT_T = div64(-E, Cp);
        io.out[0][i] = T * dtT_T;
        io.out[1][i] = V * fma(rcp_pressure_R * T, dtE, dtT_T);
    }
    team_sync<TEAM>();  // the scratch is the warp's next cell's
    return true;
}

template <int TEAM, int KMAX>
__device__ __forceinline__ bool reaction_rates_cell_warp(const RatesXTables& tb, const ReactionRatesArgs<KMAX>& io, size_t i,
                                                         double* sh, int lane) {
    constexpr int kStep = 32 * TEAM;
    CellXW<KMAX> c;
    if (!cell_progress_warp<TEAM, KMAX>(tb, io.in[0][i], io.in[1][i], io.in[2][i], io.in + 3, i, sh, lane, c)) return false;
    const double* cR = sh + 4 * tb.H->K + tb.H->n_eff;
    for (int r = lane; r < tb.H->R; r += kStep) io.out[tb.reactions[r].orig][i] = cR[r];
    team_sync<TEAM>();
    return true;
}

// The warp's cells; those that need the FP64 form are put off until there are 32, one per lane.
template <bool SMEM, int TEAM, class Cell, class F64>
__device__ __forceinline__ void warp_cells(const uint8_t* gtab, uint32_t tab_bytes, const uint8_t* f64_tab, size_t n, int* status,
                                           Cell cell, F64 f64) {
    __shared__ uint64_t bar;
    if (!stage_x<SMEM>(gtab, tab_bytes, &bar, status)) return;
    const RatesXTables tb(SMEM ? cb_dsmem : gtab);
    const uint32_t tables = SMEM ? tab_bytes : (uint32_t)(kMathBytes + kFixMathBytes);
    if (TEAM > 1) {
        // The block's only cell (launch_team_kernel), so that the FP64 tables may take the place of the others. In a loop
        // all the same: without one the compiler takes 80 registers for 128 and spills (250 species 107 -> 110 us).
        for (size_t i = blockIdx.x; i < n; i += gridDim.x) {
            if (!cell(tb, i, reinterpret_cast<double*>(cb_dsmem + tables), (int)threadIdx.x)) {
                const uint8_t* staged = gridDim.x < n ? f64_tab : stage_f64(f64_tab);
                if (threadIdx.x == 0) f64(staged, i);
            }
            __syncthreads();
        }
        return;
    }
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    double* sh = reinterpret_cast<double*>(cb_dsmem + tables) +
                 (size_t)(threadIdx.x >> 5) * (4 * tb.H->K + tb.H->n_eff + tb.H->R);  // rates_warp_bytes
    size_t later = 0;
    int put_off = 0;
    for (size_t i = (size_t)blockIdx.x * warps + (threadIdx.x >> 5); i < n; i += (size_t)gridDim.x * warps) {
        if (cell(tb, i, sh, lane)) continue;
        __syncwarp();
        if (lane == put_off) later = i;
        if (++put_off == 32) {
            f64(f64_tab, later);
            __syncwarp();
            put_off = 0;
        }
    }
    if (lane < put_off) f64(f64_tab, later);
}

template <int KMAX, bool SMEM, int TEAM>
__global__ void __launch_bounds__(32 * (TEAM > 1 ? TEAM : kRatesWarps)) rates_x_warp_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                                                      const __grid_constant__ RatesArgs<KMAX> io, size_t n,
                                                                      int* status) {
    let_next_start();
    warp_cells<SMEM, TEAM>(
        gtab, tab_bytes, io.f64_tab, n, status,
        [&](const RatesXTables& tb, size_t i, double* sh, int lane) { return rates_cell_warp<TEAM, KMAX>(tb, io, i, sh, lane); },
        [&](const uint8_t* tab, size_t i) { rates_cell_f64<KMAX>(tab, io, i); });
}
template <int KMAX, bool SMEM, int TEAM>
__global__ void __launch_bounds__(32 * (TEAM > 1 ? TEAM : kRatesWarps))
    reaction_rates_x_warp_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                 const __grid_constant__ ReactionRatesArgs<KMAX> io, size_t n, int* status) {
    warp_cells<SMEM, TEAM>(
        gtab, tab_bytes, io.f64_tab, n, status,
        [&](const RatesXTables& tb, size_t i, double* sh, int lane) {
            return reaction_rates_cell_warp<TEAM, KMAX>(tb, io, i, sh, lane);
        },
        [&](const uint8_t* tab, size_t i) { reaction_rates_cell_f64<KMAX>(tab, io, i); });
}

namespace {
// Calls of up to a cell per SM go one cell per block of eight warps (one state: 10 species 34 -> 25 us, 53 species 35 ->
// 23, 250 species 391 -> 138: the reactions' eleven (48) rounds become two (six); the FP64 sums stay on one lane).
// Calls of up to this many cells per SM go one cell per warp. A thread's cell takes 60, 500 and 5,000 us however few
// there are (10, 53, 250 species), a warp's 34, 66 and 410 us and then 12, 24 and 360 ns per cell (bound by the FP64
// chains that run on one lane); beyond these lines the thread form is the faster.
template <int KMAX>
constexpr size_t kWarpCellsPerSmR = KMAX == 16 ? 32 : KMAX == 64 ? 150 : 100;

template <int KMAX>
cudaError_t launch_rates_xk(const uint8_t* tab, uint32_t tab_bytes, const RatesArgs<KMAX>& io, size_t n, size_t warp_bytes,
                            cudaStream_t st, int* status) {
    const bool fits = 4 * warp_bytes + 32768 <= (size_t)max_table_smem();
    if (n <= (size_t)sm_count() && fits)
        return launch_team_kernel<kTeamWarps>(rates_x_warp_kernel<KMAX, true, kTeamWarps>, rates_x_warp_kernel<KMAX, false, kTeamWarps>,
                                              tab, tab_bytes, io, n, kMathBytes + kFixMathBytes, warp_bytes, st, status);
    if (n <= (size_t)sm_count() * kWarpCellsPerSmR<KMAX> && fits)
        return launch_warp_kernel<kRatesWarps>(rates_x_warp_kernel<KMAX, true, 1>, rates_x_warp_kernel<KMAX, false, 1>, tab, tab_bytes, io, n,
                                               kMathBytes + kFixMathBytes, warp_bytes, st, status);
    return launch_table_kernel<kRatesXBlock>(rates_x_kernel<KMAX, true>, rates_x_kernel<KMAX, false>, tab, tab_bytes, io, n,
                                             kMathBytes + kFixMathBytes, false, st, status);
}
template <int KMAX>
cudaError_t launch_reaction_rates_xk(const uint8_t* tab, uint32_t tab_bytes, const ReactionRatesArgs<KMAX>& io, size_t n,
                                     size_t warp_bytes, cudaStream_t st, int* status) {
    const bool fits = 4 * warp_bytes + 32768 <= (size_t)max_table_smem();
    if (n <= (size_t)sm_count() && fits)
        return launch_team_kernel<kTeamWarps>(reaction_rates_x_warp_kernel<KMAX, true, kTeamWarps>,
                                              reaction_rates_x_warp_kernel<KMAX, false, kTeamWarps>, tab, tab_bytes, io, n,
                                              kMathBytes + kFixMathBytes, warp_bytes, st, status);
    if (n <= (size_t)sm_count() * kWarpCellsPerSmR<KMAX> && fits)
        return launch_warp_kernel<kRatesWarps>(reaction_rates_x_warp_kernel<KMAX, true, 1>, reaction_rates_x_warp_kernel<KMAX, false, 1>, tab,
                                               tab_bytes, io, n, kMathBytes + kFixMathBytes, warp_bytes, st, status);
    return launch_table_kernel<kRatesXBlock>(reaction_rates_x_kernel<KMAX, true>, reaction_rates_x_kernel<KMAX, false>, tab,
                                             tab_bytes, io, n, kMathBytes + kFixMathBytes, false, st, status);
}
}  // namespace

cudaError_t launch_rates_x(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n, size_t warp_bytes,
                           cudaStream_t st, int* status) {
    switch (kmax) {
    case 16: return launch_rates_xk<16>(tab, tab_bytes, *static_cast<const RatesArgs<16>*>(args), n, warp_bytes, st, status);
    case 64: return launch_rates_xk<64>(tab, tab_bytes, *static_cast<const RatesArgs<64>*>(args), n, warp_bytes, st, status);
    case 256:
        return launch_rates_xk<256>(tab, tab_bytes, *static_cast<const RatesArgs<256>*>(args), n, warp_bytes, st, status);
    default: return cudaErrorInvalidValue;
    }
}
cudaError_t launch_reaction_rates_x(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                                    size_t warp_bytes, cudaStream_t st, int* status) {
    switch (kmax) {
    case 16:
        return launch_reaction_rates_xk<16>(tab, tab_bytes, *static_cast<const ReactionRatesArgs<16>*>(args), n, warp_bytes,
                                            st, status);
    case 64:
        return launch_reaction_rates_xk<64>(tab, tab_bytes, *static_cast<const ReactionRatesArgs<64>*>(args), n, warp_bytes,
                                            st, status);
    case 256:
        return launch_reaction_rates_xk<256>(tab, tab_bytes, *static_cast<const ReactionRatesArgs<256>*>(args), n, warp_bytes,
                                             st, status);
    default: return cudaErrorInvalidValue;
    }
}
CB_WAVE(wave_rates_x, rates_x_kernel, kRatesXBlock, kMathBytes + kFixMathBytes)
CB_WAVE(wave_reaction_rates_x, reaction_rates_x_kernel, kRatesXBlock, kMathBytes + kFixMathBytes)

// Test hook: the fixed-point functions one by one (cb_debug_fixed_math).
__global__ void fixed_math_check_kernel(const uint8_t* tab, int which, const double* x, double* y, size_t n) {
    stage_x<false>(tab, 0, nullptr, nullptr);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double v = x[i];
        y[i] = which == 0   ? exp2_dbl(v)
               : which == 1 ? log2_dbl(v)
               : which == 2 ? rcp_fixed(dbl_to_fix(v, kDq), 1022 + 63 - 56)
                            : fix_to_dbl(dbl_to_fix(v, kYq), kYq);
    }
}
cudaError_t launch_fixed_math_check(const uint8_t* tab, int which, const double* x, double* y, size_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    fixed_math_check_kernel<<<(unsigned)(n < 256 * 4096 ? (n + 255) / 256 : 4096), 256, kMathBytes + kFixMathBytes, st>>>(tab, which, x, y, n);
    return cudaGetLastError();
}

cudaError_t set_stage_wait_polls_x(long long polls) { return cudaMemcpyToSymbol(g_stage_wait_polls, &polls, sizeof polls); }

}  // namespace cbg
