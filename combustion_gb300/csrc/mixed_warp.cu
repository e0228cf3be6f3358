// The mixed-precision kernels, one cell per warp, for calls too small to fill the GPU with one cell per thread
// (kernels_mixed.cu): there a call takes as long as one thread needs for its cell, 520 us at 53 species, where a
// warp needs 67 (10,100 cells: 1,105 -> 315 us; with transport 1,375 -> 394), and a block of eight warps, for calls
// of at most a cell per SM, 51 (250 species, rates and transport: 10,400 -> 748 -> 145).
// The lanes share a cell's species, third-body rows, reactions and rows of the mixture rules; every sum runs in
// the order of the thread's program, so a cell has the same bits in both forms. What is left is latency: the FP64
// sums over the species in that order (a quarter of the FP64 pipe's time on one lane each) and eleven rounds of
// reactions.
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "device_math.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "rates_mixed_core.cuh"
#include "tables_mixed.h"

namespace cbg {

// The warp's cell in shared memory.
struct CellMW {
    const double *C, *ex, *exn;
    double C0, rcpC0, rcpC0sq;
    float Ctotf, Tf, lnTf, rcpTf;
};
// As a thread's cell: the factors' reads issued together, a reaction without net species takes 1.
template <>
constexpr bool kBatchLoads<CellMW> = true;

// turn: the warp that takes the model's first 32 reactions.
template <int TEAM, int MODEL>
__device__ __forceinline__ void progress_group_m(const RatesMixedTables& tb, const CellMW& c, const float* Mf, double* cR,
                                                 int lane, int& turn) {
    const int begin = MODEL ? tb.H->group_end[MODEL - 1] : 0, end = tb.H->group_end[MODEL];
    const int mine = TEAM == 1 ? 0 : ((lane >> 5) - turn + TEAM) % TEAM;
    if (TEAM > 1) turn = (turn + (end - begin + 31) / 32) % TEAM;
    for (int r = begin + 32 * mine + (lane & 31); r < end; r += 32 * TEAM) {
        const ReactionF& x = tb.reactions[r];
        cR[r] = reaction_rate_m<MODEL>(tb, x, c, MODEL >= 2 ? Mf[x.eff_row] : 0.f);
    }
}

// rates_mixed_cell. sh: rates_warp_bytes of scratch. csr: per species its reactions and net coefficients in order.
// TEAM warps (a block of its own) share the cell in calls of at most a cell per SM, 1 otherwise.
template <int TEAM, int KMAX>
__device__ void rates_mixed_cell_warp(const RatesMixedTables& tb, const int* csr_start, const int* csr,
                                      const RatesArgs<KMAX>& io, size_t i, double* sh, int lane) {
    const RatesMixedHeader& H = *tb.H;
    const int K = H.K, A = H.A;
    const bool uniform = io.flags & kUniformPressure;
    const double pressure_R = uniform ? io.in[0][0] : io.in[0][i];
    const double rcp_pressure_R = uniform ? io.in[1][0] : io.in[1][i];
    const double T = io.in[2][i], V = io.in[3][i];
    double *C = sh, *ex = sh + K, *exn = sh + 2 * K, *w = sh + 3 * K, *cR = sh + 4 * K + H.n_eff;
    float* Mf = reinterpret_cast<float*>(sh + 4 * K);
    const double md = rcp64(V), rcpT = rcp64(T), lnT = log64(T);
    const double T2 = T * T, T3 = T * T2, T4 = T2 * T2;
    for (int k = lane; k < K - 1; k += 32 * TEAM) C[k] = __dmul_rn(md, max0(io.in[4 + k][i]));
    team_sync<TEAM>();
    double sum = 0.0;
    if (lane < 32) {
#pragma unroll 4
        for (int k = 0; k < K - 1; k++) sum += C[k];
    }
    const double Ctot = __dmul_rn(pressure_R, rcpT);
    CellMW c;
    c.Ctotf = dbl_to_flt(Ctot);
    c.Tf = dbl_to_flt(T);
    c.lnTf = dbl_to_flt(lnT);
    c.rcpTf = dbl_to_flt(rcpT);
    c.C0 = H.C0 * rcpT;
    c.rcpC0 = H.rcp_C0 * T;
    c.rcpC0sq = c.rcpC0 * c.rcpC0;
    c.C = C;
    c.ex = ex;
    c.exn = exn;
    if (lane == 0) C[K - 1] = Ctot - sum;
    for (int k = lane; k < A; k += 32 * TEAM) {
        const SpeciesF& s = tb.species[k];
        if (!(s.need_exp | s.need_exp_neg)) continue;
        const double* g = s.g[piece_of_m(s.split, T)];
        const double x = fma(g[6], rcpT, fma(g[5], T4, fma(g[4], T3, fma(g[3], T2, fma(g[2], T, fma(g[1], lnT, g[0]))))));
        gibbs_exps(x, s.need_exp, s.need_exp_neg, H.M3, H.cbrt_max, c.C0, c.rcpC0, ex[k], exn[k]);
    }
    team_sync<TEAM>();
    for (int e = lane; e < H.n_eff; e += 32 * TEAM) {
        const float* E = tb.eff + (size_t)e * K;
        float s = 0.f;
#pragma unroll 4
        for (int k = 0; k < K; k++) s = fmaf(E[k], dbl_to_flt(C[k]), s);
        Mf[e] = c.Ctotf + s;
    }
    team_sync<TEAM>();
    int turn = 0;
    progress_group_m<TEAM, 0>(tb, c, Mf, cR, lane, turn);
    progress_group_m<TEAM, 1>(tb, c, Mf, cR, lane, turn);
    progress_group_m<TEAM, 2>(tb, c, Mf, cR, lane, turn);
    progress_group_m<TEAM, 3>(tb, c, Mf, cR, lane, turn);
    progress_group_m<TEAM, 4>(tb, c, Mf, cR, lane, turn);
    progress_group_m<TEAM, 5>(tb, c, Mf, cR, lane, turn);
    team_sync<TEAM>();
    double *hk = ex, *cpk = exn;
    for (int k = lane; k < K; k += 32 * TEAM) {
        const SpeciesF& s = tb.species[k];
        const int p = piece_of_m(s.split, T);
        const float Tf = c.Tf, *cp = s.cp[p], *h = s.h[p];
        const float ck = fmaf(cp[4], Tf, cp[3]);
        cpk[k] = flt_to_dbl(fmaf(fmaf(fmaf(ck, Tf, cp[2]), Tf, cp[1]), Tf, cp[0]));
        if (k >= A) continue;
        hk[k] = flt_to_dbl(fmaf(h[5], c.rcpTf, fmaf(fmaf(fmaf(fmaf(h[4], Tf, h[3]), Tf, h[2]), Tf, h[1]), Tf, h[0])));
        double wk = 0.0;
        for (int q = csr_start[k]; q < csr_start[k + 1]; q++)
            wk = fma(small_int_to_double((int)(int8_t)(csr[q] & 0xff)), cR[csr[q] >> 8], wk);
        w[k] = wk;
        io.out[2 + k][i] = wk;
    }
    team_sync<TEAM>();
    double acc = 0.0;  // E, Cp and dtE on lanes 0, 1, 2
    if (lane < 3) {
        const int n = lane == 1 ? K : A;
#pragma unroll 4
        for (int k = 0; k < n; k++)
            acc = fma(lane == 0 ? w[k] : lane == 1 ? cpk[k] : tb.species[k].dtE, lane == 0 ? hk[k] : lane == 1 ? C[k] : w[k], acc);
    }
    const double E = __shfl_sync(0xffffffffu, acc, 0), Cp = __shfl_sync(0xffffffffu, acc, 1),
                 dtE = __shfl_sync(0xffffffffu, acc, 2);
    if (lane == 0) {
        const double dtT_T = -E * rcp64(Cp);
        io.out[0][i] = T * dtT_T;
        io.out[1][i] = V * fma(rcp_pressure_R * T, dtE, dtT_T);
    }
    team_sync<TEAM>();  // the scratch is the warp's next cell's
}

// The tables into shared memory, or only the functions' (the rest is then read through L1).
template <bool SMEM>
__device__ __forceinline__ bool stage_m(const uint8_t* gtab, uint32_t tab_bytes, uint64_t* bar, int* status) {
    if (SMEM) return stage_to_shared(cb_dsmem, gtab, tab_bytes, bar, status);
    load_math(gtab);
    return true;
}

constexpr int kMixedWarps = 16;  // cells per block at most

template <int KMAX, bool SMEM, int TEAM>
__global__ void __launch_bounds__(32 * (TEAM > 1 ? TEAM : kMixedWarps)) rates_mixed_warp_kernel(const uint8_t* __restrict__ gtab,
                                                                            uint32_t tab_bytes,
                                                                            const __grid_constant__ RatesArgs<KMAX> io,
                                                                            size_t n, int* status) {
    let_next_start();
    __shared__ uint64_t bar;
    if (!stage_m<SMEM>(gtab, tab_bytes, &bar, status)) return;
    const RatesMixedTables tb(SMEM ? cb_dsmem : gtab);
    const int *csr_start = reinterpret_cast<const int*>(gtab + tb.H->total_bytes), *csr = csr_start + tb.H->A + 1;
    // the block's cells: as many as it has warps, or one
    const int lane = TEAM > 1 ? threadIdx.x : threadIdx.x & 31, slot = TEAM > 1 ? 0 : threadIdx.x >> 5;
    const int cells = TEAM > 1 ? 1 : blockDim.x >> 5;
    double* sh = reinterpret_cast<double*>(cb_dsmem + (SMEM ? tab_bytes : (uint32_t)kMathBytes)) +
                 (size_t)slot * (4 * tb.H->K + tb.H->n_eff + tb.H->R);  // rates_warp_bytes
    for (size_t i = (size_t)blockIdx.x * cells + slot; i < n; i += (size_t)gridDim.x * cells)
        rates_mixed_cell_warp<TEAM, KMAX>(tb, csr_start, csr, io, i, sh, lane);
}

// ---------------------------------------------------------------------------------------------------
// transport_mixed_cell, in six arrays of K floats.
template <int TEAM, int KMAX>
__device__ void transport_mixed_cell_warp(const uint8_t* tab, const TransportArgs<KMAX>& io, size_t i, size_t o, float* sh,
                                          int lane) {
    const TransportMixedHeader& H = *reinterpret_cast<const TransportMixedHeader*>(tab + kMathBytes);
    const float* cond = reinterpret_cast<const float*>(tab + H.off_cond);
    const float* visc = reinterpret_cast<const float*>(tab + H.off_visc);
    const float* W = reinterpret_cast<const float*>(tab + H.off_W);
    const float4* diff = reinterpret_cast<const float4*>(tab + H.off_diff);
    const float4* wil = reinterpret_cast<const float4*>(tab + H.off_wilke);
    const int K = H.K;
    float N, Tn;
    const double* const* amounts;
    if (io.flags & kFromRates) {
        const double pressure_R = (io.flags & kUniformPressure) ? io.in[0][0] : io.in[0][i];
        const float T = dbl_to_flt(io.in[2][i]);
        N = __fdividef(dbl_to_flt(pressure_R) * dbl_to_flt(io.in[3][i]), T);
        Tn = T / (float)H.T0;
        amounts = io.in + 4;
    } else {
        N = dbl_to_flt(io.in[0][i]);
        Tn = dbl_to_flt(io.in[1][i]);
        amounts = io.in + 2;
    }
    const float L1 = logf(Tn), L2 = L1 * L1, L3 = L2 * L1, L4 = L3 * L1;
    auto poly = [&](const float* P) { return fmaf(P[4], L4, fmaf(P[3], L3, fmaf(P[2], L2, fmaf(P[1], L1, P[0])))); };
    float *X = sh, *v = sh + K, *Y = sh + 2 * K, *Z = sh + 3 * K, *a = sh + 4 * K, *b = sh + 5 * K;
    for (int k = lane; k < K; k += 32 * TEAM) {
        if (k < K - 1) X[k] = dbl_to_flt(amounts[k][i]);
        const float c = poly(cond + 5 * k);
        a[k] = c;
        b[k] = rcp_f32(c);
        v[k] = poly(visc + 5 * k);
    }
    team_sync<TEAM>();
    float s = 0.f, comp = 0.f;
#pragma unroll 4
    for (int k = 0; k < K - 1; k++) {
        const float y = X[k] - comp, t = s + y;
        comp = (t - s) - y;
        s = t;
    }
    team_sync<TEAM>();
    if (lane == 0) X[K - 1] = (N - s) + comp;
    team_sync<TEAM>();
    for (int k = lane; k < K; k += 32 * TEAM) {
        const float r = rcp_f32(v[k]), y = X[k] * r;
        Y[k] = y;
        Z[k] = y * r;
    }
    const float VT = sqrtf(Tn);
    const float* q = (lane & 31) == 1 ? a : (lane & 31) == 2 ? b : W;  // sums over X: molar mass, conductivities, their reciprocals
    float acc = 0.f;
#pragma unroll 4
    for (int k = 0; k < K; k++) acc = fmaf(X[k], q[k], acc);
    const float MN = __shfl_sync(0xffffffffu, acc, 0), Ac = __shfl_sync(0xffffffffu, acc, 1),
                Bc = __shfl_sync(0xffffffffu, acc, 2);
    const float MVTN = MN * VT;
    team_sync<TEAM>();
    if (lane == 0) io.out[0][o] = flt_to_dbl((__fdividef(Ac, N) + __fdividef(N, Bc)) * VT);
    for (int k = lane; k < K; k += 32 * TEAM) {  // Wilke, a row per lane
        const float4* w = wil + (size_t)k * K;
        float s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 4
        for (int j = 0; j < K; j++) {
            const float4 c = w[j];
            s1 = fmaf(c.x, X[j], s1);
            s2 = fmaf(c.y, Y[j], s2);
            s3 = fmaf(c.z, Z[j], s3);
        }
        a[k] = X[k] * (v[k] * v[k]);
        b[k] = rcp_f32(fmaf(v[k], fmaf(v[k], s3, s2), s1));
    }
    team_sync<TEAM>();
    float mu = 0.f;
#pragma unroll 4
    for (int k = 0; k < K; k++) mu = fmaf(a[k], b[k], mu);
    if (lane == 0) io.out[1][o] = flt_to_dbl(VT * mu);
    // Mixture diffusion, a species k per lane: even and odd j < k apart, then j > k in order. Each pair is evaluated for
    // both of its species (4 FMAs and a reciprocal; the pairs of 250 species would take 124 KB per warp).
    for (int k = lane; k < K; k += 32 * TEAM) {
        const float4* row = diff + (size_t)k * (k - 1);  // pairs (k, 0), two float4 each
        float sa = 0.f, sb = 0.f, S = 0.f;
#pragma unroll 4
        for (int j = 0; j < K; j++) {
            if (j == k) {
                S = sa + sb;
                continue;
            }
            const float4* P = j < k ? row + 2 * j : diff + (size_t)j * (j - 1) + 2 * k;
            const float4 c = P[0];
            const float R = rcp_f32(fmaf(P[1].x, L4, fmaf(c.w, L3, fmaf(c.z, L2, fmaf(c.y, L1, c.x)))));
            if (j > k) S = fmaf(X[j], R, S);
            else if (j & 1) sb = fmaf(X[j], R, sb);
            else sa = fmaf(X[j], R, sa);
        }
        io.out[2 + k][o] = flt_to_dbl(__fdividef(fmaf(-(VT * W[k]), X[k], MVTN), S));
    }
    team_sync<TEAM>();  // the scratch is the warp's next cell's
}

template <int KMAX, bool SMEM, int TEAM>
__global__ void __launch_bounds__(32 * (TEAM > 1 ? TEAM : kMixedWarps))
    transport_mixed_warp_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                const __grid_constant__ TransportArgs<KMAX> io, size_t n, int* status) {
    const EndAfterPrevious last;
    __shared__ uint64_t bar;
    if (!stage_m<SMEM>(gtab, tab_bytes, &bar, status)) return;
    const uint8_t* tab = SMEM ? cb_dsmem : gtab;
    if (io.count) n = min(n, (size_t)*io.count);  // gathered cells: the count is known on the device only
    const int lane = TEAM > 1 ? threadIdx.x : threadIdx.x & 31, slot = TEAM > 1 ? 0 : threadIdx.x >> 5;
    const int cells = TEAM > 1 ? 1 : blockDim.x >> 5;
    float* sh = reinterpret_cast<float*>(cb_dsmem + (SMEM ? tab_bytes : (uint32_t)kMathBytes)) + (size_t)slot * (6 * KMAX);
    for (size_t j = (size_t)blockIdx.x * cells + slot; j < n; j += (size_t)gridDim.x * cells) {
        const size_t i = io.index ? (size_t)(io.index[j] & kIndexMask) : j;
        transport_mixed_cell_warp<TEAM, KMAX>(tab, io, i, (io.flags & kCompactOut) ? j : i, sh, lane);
    }
}

// A cell per block of eight warps up to a cell per SM, a cell per warp beyond.
#define CB_LAUNCH(KERNEL, KM, ARGS, SCRATCH)                                                                             \
    case KM: {                                                                                                           \
        const auto& io = *static_cast<const ARGS<KM>*>(args);                                                            \
        if (n <= (size_t)sm_count())                                                                                     \
            return launch_team_kernel<kTeamWarps>(KERNEL<KM, true, kTeamWarps>, KERNEL<KM, false, kTeamWarps>, tab, tab_bytes, \
                                                  io, n, kMathBytes, SCRATCH, st, status);                               \
        return launch_warp_kernel<kMixedWarps>(KERNEL<KM, true, 1>, KERNEL<KM, false, 1>, tab, tab_bytes, io, n, kMathBytes, \
                                               SCRATCH, st, status);                                                     \
    }
cudaError_t launch_rates_mixed_warp(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                                    size_t warp_bytes, cudaStream_t st, int* status) {
    switch (kmax) {
        CB_LAUNCH(rates_mixed_warp_kernel, 16, RatesArgs, warp_bytes)
        CB_LAUNCH(rates_mixed_warp_kernel, 64, RatesArgs, warp_bytes)
        CB_LAUNCH(rates_mixed_warp_kernel, 256, RatesArgs, warp_bytes)
    default: return cudaErrorInvalidValue;
    }
}
cudaError_t launch_transport_mixed_warp(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                                        cudaStream_t st, int* status) {
    switch (kmax) {
        CB_LAUNCH(transport_mixed_warp_kernel, 16, TransportArgs, 6 * 16 * sizeof(float))
        CB_LAUNCH(transport_mixed_warp_kernel, 64, TransportArgs, 6 * 64 * sizeof(float))
        CB_LAUNCH(transport_mixed_warp_kernel, 256, TransportArgs, 6 * 256 * sizeof(float))
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace cbg
