// The plain transport kernels in fixed point (transport_fixed_core.cuh; transport.rs:141-210): one cell per thread,
// and one per warp for small calls and gathered cells.
//
// The FP64 form (kernels.cu) is bound by the FP64 pipe: per pair of species 4 FMAs of the diffusion fit, 3
// instructions of its reciprocal and 2 of the mixing sums, and 6 FMAs of Wilke's sums (22.6 k FP64 instructions per
// cell at 53 species, 64 cycles each). Here the fits, their reciprocals and Wilke's sums are integer sums of three
// 4-cycle mad.wide per term; the FP64 pipe keeps the mixing sums over reciprocals (2 per pair).
// Cells outside the range of temperatures or with non-finite amounts take the FP64 form, tables read from global
// memory: 2^19 cells of 53 species above 7,380 K 20.5 ms (5.7 in range, 20.5 in the FP64 kernel), in a mixed field up to
// the sum of both forms.
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "transport_fixed_core.cuh"

namespace cbg {

// Rows k0 .. k0 + Q - 1 of Wilke's sums and their terms of mu (rows k0, k0 + 2 in mu0, the others in mu1).
template <int Q, int LO>
__device__ __forceinline__ void wilke_rows_x(const TransportXTables& tb, int K, int k0, const double* X, const double* r,
                                               const double* Xw, const double* Yw, const double* Zw, int q1, int q2,
                                               int q3, double& mu0, double& mu1) {
    const Word2* a = tb.A2 + k0;
    long long s[Q][3], t[Q][3];
#pragma unroll
    for (int q = 0; q < Q; q++)
#pragma unroll
        for (int i = 0; i < 3; i++) s[q][i] = t[q][i] = 0;
    double xn = Xw[0], yn = Yw[0], zn = Zw[0];
#pragma unroll 1
    for (int j = 0; j < K; j++) {
        const Word2 x{__double2hiint(xn), __double2loint(xn)};
        const Word2 y{__double2hiint(yn), __double2loint(yn)};
        const Word2 z{__double2hiint(zn), __double2loint(zn)};
        if (j + 1 < K) {  // the next species' words on their way under this one's sums
            xn = Xw[j + 1];
            yn = Yw[j + 1];
            zn = Zw[j + 1];
        }
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const Word2 w = a[(size_t)j * K + q];
            dot_term(w, x, s[q][0], t[q][0]);
            dot_term(w, y, s[q][1], t[q][1]);
            dot_term(w, z, s[q][2], t[q][2]);
        }
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const double w = wilke_factor(X[k0 + q], tb.W4[k0 + q]),
                     d = wilke_rcp(mix_value<LO>(s[q][0], t[q][0]), mix_value<LO>(s[q][1], t[q][1]), mix_value<LO>(s[q][2], t[q][2]),
                                   q1, q2, q3, r[k0 + q]);
        if (q & 1) mu1 = fma(w, d, mu1);
        else mu0 = fma(w, d, mu0);
    }
}

// Rows k0 .. k0 + Q - 1 of the diffusion pairs: S_k = sum over j < k of X_j / D_kj (even and odd j apart), and X_k / D_kj
// added to S_j, for every S in the order of its species. One load of X_j and one update of S_j (thread-local arrays,
// mostly in L2) per Q pairs.
template <int Q>
__device__ __forceinline__ void diffusion_rows(const TransportXTables& tb, int k0, const PowersX& L, const double* X, double* S) {
    const PolyX* P[Q];
    double x[Q], s[Q], t[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int k = k0 + q;
        P[q] = tb.diff + (size_t)k * (k - 1) / 2;
        x[q] = X[k];
        s[q] = t[q] = 0.0;
    }
#pragma unroll 1
    for (int j = 0; j < k0; j += 2) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (Q == 1 && h == 1 && j + 1 >= k0) break;  // with Q = 4, k0 is even
            const double xj = X[j + h];
            double sj = S[j + h];
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const PolyX p = P[q][j + h];
                const double R = rcp_fixed(poly_x(p, L), p.rcp_bias);
                if (h) t[q] = fma(xj, R, t[q]);
                else s[q] = fma(xj, R, s[q]);
                sj = fma(x[q], R, sj);
            }
            S[j + h] = sj;
        }
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
#pragma unroll
        for (int i = 0; i < q; i++) {
            const PolyX p = P[q][k0 + i];
            const double R = rcp_fixed(poly_x(p, L), p.rcp_bias);
            if (i & 1) t[q] = fma(x[i], R, t[q]);
            else s[q] = fma(x[i], R, s[q]);
            s[i] = fma(x[q], R, s[i]);  // row i's own sum is complete
        }
        s[q] += t[q];
    }
#pragma unroll
    for (int q = 0; q < Q; q++) S[k0 + q] = s[q];
}

template <int KMAX>
__device__ __forceinline__ bool transport_cell_x(const TransportXTables& tb, const TransportArgs<KMAX>& io, size_t i, size_t o) {
    constexpr int LO = kMixLo<KMAX>;
    const TransportXHeader& H = *tb.H;
    const int K = H.K;
    double N, Tn;
    const double* const* amounts = transport_inputs(H, io, i, N, Tn);
    if (!(Tn >= H.Tn_lo && Tn < H.Tn_hi)) return false;
    double X[KMAX], r[KMAX], Xw[KMAX], Y[KMAX], Z[KMAX], S[KMAX];
    double s = 0.0;
    int mx = 0;
    for (int k = 0; k < K - 1; k++) {
        X[k] = amounts[k][i];
        s += X[k];
        mx = max(mx, __double2hiint(X[k]) & 0x7fffffff);
    }
    X[K - 1] = N - s;
    mx = max(mx, __double2hiint(X[K - 1]) & 0x7fffffff);
    // the largest amount between 1e-150 and 1e150: every other is finite
    if (mx < 0x20ca2fe7 || mx >= 0x5f138d35 || !(N - N == 0.0)) return false;
    const PowersX L = log_powers(H, Tn);
    const double VT = sqrt(Tn);
    // Sums over species as the sum over even and the sum over odd ones (half the roundings).
    double M0 = 0.0, M1 = 0.0;
    for (int k = 0; k + 1 < K; k += 2) {
        M0 = fma(tb.W[k], X[k], M0);
        M1 = fma(tb.W[k + 1], X[k + 1], M1);
    }
    if (K & 1) M0 = fma(tb.W[K - 1], X[K - 1], M0);
    const double MN = M0 + M1;

    // Conductivity (transport.rs:141-146).
    double A0 = 0.0, B0 = 0.0, A1 = 0.0, B1 = 0.0;
    auto conductivity = [&](int k, double& A, double& B) {
        const PolyX P = tb.cond[k];
        const long long d = poly_x(P, L);
        const double x = X[k];
        A = fma(x, fix_to_dbl(d, kDq - P.sp), A);
        B = fma(x, rcp_fixed(d, P.rcp_bias), B);
    };
#pragma unroll 1
    for (int k = 0; k + 1 < K; k += 2) {
        conductivity(k, A0, B0);
        conductivity(k + 1, A1, B1);
    }
    if (K & 1) conductivity(K - 1, A0, B0);
    io.out[0][o] = conductivity_of(A0 + A1, B0 + B1, N, VT);

    // 1 / v'_k, and X, X / v', X / v'^2 as words
    int my = 0, mz = 0;
    for (int k = 0; k < K; k++) {
        const PolyX P = tb.visc[k];
        r[k] = rcp_fixed(poly_x(P, L), P.rcp_bias);
        Y[k] = __dmul_rn(X[k], r[k]);
        Z[k] = __dmul_rn(Y[k], r[k]);
        my = max(my, __double2hiint(Y[k]) & 0x7fffffff);
        mz = max(mz, __double2hiint(Z[k]) & 0x7fffffff);
    }
    const int qx = kMixXq<KMAX> - exponent_above(mx), qy = kMixXq<KMAX> - exponent_above(my),
              qz = kMixXq<KMAX> - exponent_above(mz);
    for (int k = 0; k < K; k++) {
        const Word2 x = split_word<LO>(dbl_to_fix(X[k], qx)), y = split_word<LO>(dbl_to_fix(Y[k], qy)),
                    z = split_word<LO>(dbl_to_fix(Z[k], qz));
        Xw[k] = __hiloint2double(x.hi, x.lo);
        Y[k] = __hiloint2double(y.hi, y.lo);
        Z[k] = __hiloint2double(z.hi, z.lo);
    }
    const int unit = H.a_shift + 1 - 2 * LO;  // of the sums, with the words' positions
    // Two independent parts, the mixing rule on the integer pipe alone and the diffusion on both: half of each
    // sub-partition's warps take them in the other order, so that both pipes have work at any time (131,072 cells at 250
    // species 54.0 -> 44.3 ms; at 10 species the loops are too short to gain).
    const bool swap = KMAX > 16 && ((threadIdx.x >> 7) & 1);
#pragma unroll 1
    for (int part = 0; part < 2; part++) {
        int k = 0;
        if ((part == 0) != swap) {  // viscosity (transport.rs:148-158)
            double mu0 = 0.0, mu1 = 0.0;  // even and odd species
#pragma unroll 1
            for (; k + 4 <= K; k += 4) wilke_rows_x<4, LO>(tb, K, k, X, r, Xw, Y, Z, unit + qx, unit + qy, unit + qz, mu0, mu1);
#pragma unroll 1
            for (; k + 2 <= K; k += 2) wilke_rows_x<2, LO>(tb, K, k, X, r, Xw, Y, Z, unit + qx, unit + qy, unit + qz, mu0, mu1);
            if (k < K) wilke_rows_x<1, LO>(tb, K, k, X, r, Xw, Y, Z, unit + qx, unit + qy, unit + qz, mu0, mu1);
            io.out[1][o] = VT * (mu0 + mu1);
        } else {  // mixture-averaged diffusion (transport.rs:162-177)
#pragma unroll 1
            for (; k + 4 <= K; k += 4) diffusion_rows<4>(tb, k, L, X, S);
#pragma unroll 1
            for (; k < K; k++) diffusion_rows<1>(tb, k, L, X, S);
        }
    }
    for (int k = 0; k < K; k++) io.out[2 + k][o] = diffusion_x(MN, VT, tb.W[k], X[k], S[k]);
    return true;
}

template <int KMAX>
__device__ __noinline__ void transport_cell_f64(const TransportArgs<KMAX>& io, size_t i, size_t o) {
    transport_cell<KMAX>(io.f64_tab, io, i, o);
}

template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(kTransportXBlock<KMAX>) transport_x_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                                                     const __grid_constant__ TransportArgs<KMAX> io,
                                                                     size_t n, int* status) {
    const EndAfterPrevious last;
    __shared__ uint64_t bar;
    if (SMEM) {
        if (!stage_to_shared(cb_dsmem, gtab, tab_bytes, &bar, status)) return;
    } else {
        load_math(gtab);
    }
    const TransportXTables tb(SMEM ? cb_dsmem : gtab);
    if (io.count) n = min(n, (size_t)*io.count);
    for (size_t b = (size_t)blockIdx.x * blockDim.x; b < n; b += (size_t)gridDim.x * blockDim.x) {
        const size_t j = b + threadIdx.x;
        if (j >= n) continue;
        const size_t i = io.index ? (size_t)(io.index[j] & kIndexMask) : j, o = (io.flags & kCompactOut) ? j : i;
        if (!transport_cell_x<KMAX>(tb, io, i, o)) transport_cell_f64<KMAX>(io, i, o);
    }
}

// ---------------------------------------------------------------------------------------------------
// One cell per warp, every sum in the thread form's order (transport_cell_warp's division of the work).
// TEAM warps (a block of its own) share the cell in calls of at most a cell per SM, 1 otherwise.
template <int KMAX>
constexpr size_t kTeamScratch = 4 * KMAX + 32 * (KMAX + 1) > kWarpScratch<KMAX> ? 4 * KMAX + 32 * (KMAX + 1) : kWarpScratch<KMAX>;

template <int TEAM, int KMAX>
__device__ __forceinline__ bool transport_cell_x_warp(const TransportXTables& tb, const TransportArgs<KMAX>& io, size_t i,
                                                      size_t o, double* sh, bool second) {
    constexpr int kStep = 32 * TEAM;
    const int lane = TEAM == 1 ? threadIdx.x & 31 : threadIdx.x, lane32 = threadIdx.x & 31;
    constexpr int LO = kMixLo<KMAX>;
    const TransportXHeader& H = *tb.H;
    const int K = H.K;
    double N, Tn;
    const double* const* amounts = transport_inputs(H, io, i, N, Tn);
    if (!(Tn >= H.Tn_lo && Tn < H.Tn_hi)) return false;
    double* X = sh;
    double* v = sh + KMAX;
    double* Y = sh + 2 * KMAX;
    double* Z = sh + 3 * KMAX;
    double* T = sh + 4 * KMAX;
    int mx = 0;
    for (int k = lane; k < K - 1; k += kStep) {
        X[k] = amounts[k][i];
        mx = max(mx, __double2hiint(X[k]) & 0x7fffffff);
    }
    team_sync<TEAM>();
    double xb = 0.0;
    if (lane == 0) {
        double s = 0.0;
        for (int k = 0; k < K - 1; k++) s += X[k];
        xb = N - s;
        X[K - 1] = xb;
        mx = max(mx, __double2hiint(xb) & 0x7fffffff);
    }
    team_sync<TEAM>();
    if (TEAM > 1)  // every warp over all species
        for (int k = lane32; k < K; k += 32) mx = max(mx, __double2hiint(X[k]) & 0x7fffffff);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (mx < 0x20ca2fe7 || mx >= 0x5f138d35 || !(N - N == 0.0)) return false;
    const PowersX L = log_powers(H, Tn);
    const double VT = sqrt(Tn);
    for (int k = lane; k < K; k += kStep) {
        const PolyX P = tb.cond[k];
        const long long d = poly_x(P, L);
        v[k] = fix_to_dbl(d, kDq - P.sp);
        Y[k] = rcp_fixed(d, P.rcp_bias);
    }
    team_sync<TEAM>();
    double acc = 0.0;  // lanes 0-2: the even species of the three sums, lanes 3-5: the odd ones
    if (lane < 6) {
        const double* src = lane % 3 == 0 ? tb.W : lane % 3 == 1 ? v : Y;
#pragma unroll 4
        for (int k = lane / 3; k < K; k += 2) acc = fma(src[k], X[k], acc);
    }
    acc += __shfl_sync(0xffffffffu, acc, (lane + 3) & 31);  // used by lanes 0-2
    const double MN = team_value<TEAM>(acc, T, lane);
    const double Ac = __shfl_sync(0xffffffffu, acc, 1);
    const double Bc = __shfl_sync(0xffffffffu, acc, 2);
    team_sync<TEAM>();
    if (lane == 0) transport_out(io, 0, second)[o] = conductivity_of(Ac, Bc, N, VT);

    int my = 0, mz = 0;
    for (int k = lane; k < K; k += kStep) {
        const PolyX P = tb.visc[k];
        v[k] = rcp_fixed(poly_x(P, L), P.rcp_bias);  // 1 / v'
        Y[k] = __dmul_rn(X[k], v[k]);
        Z[k] = __dmul_rn(Y[k], v[k]);
        my = max(my, __double2hiint(Y[k]) & 0x7fffffff);
        mz = max(mz, __double2hiint(Z[k]) & 0x7fffffff);
    }
    if (TEAM > 1) {
        __syncthreads();
        for (int k = lane32; k < K; k += 32) {
            my = max(my, __double2hiint(Y[k]) & 0x7fffffff);
            mz = max(mz, __double2hiint(Z[k]) & 0x7fffffff);
        }
        __syncthreads();
    }
    my = __reduce_max_sync(0xffffffffu, my);
    mz = __reduce_max_sync(0xffffffffu, mz);
    const int qx = kMixXq<KMAX> - exponent_above(mx), qy = kMixXq<KMAX> - exponent_above(my),
              qz = kMixXq<KMAX> - exponent_above(mz);
    double* Xw = T;  // the tile holds X's words and the viscosity terms until the diffusion
    double* U = T + KMAX;
    for (int k = lane; k < K; k += kStep) {
        const Word2 x = split_word<LO>(dbl_to_fix(X[k], qx)), y = split_word<LO>(dbl_to_fix(Y[k], qy)),
                    z = split_word<LO>(dbl_to_fix(Z[k], qz));
        Xw[k] = __hiloint2double(x.hi, x.lo);
        Y[k] = __hiloint2double(y.hi, y.lo);
        Z[k] = __hiloint2double(z.hi, z.lo);
    }
    team_sync<TEAM>();
    const int unit = H.a_shift + 1 - 2 * LO;
#pragma unroll 1
    for (int k = lane; k < K; k += kStep) {
        const Word2* a = tb.A2 + k;
        long long s[3] = {0, 0, 0}, t[3] = {0, 0, 0};
#pragma unroll 2
        for (int j = 0; j < K; j++) {
            const Word2 w = a[(size_t)j * K];
            dot_term(w, Word2{__double2hiint(Xw[j]), __double2loint(Xw[j])}, s[0], t[0]);
            dot_term(w, Word2{__double2hiint(Y[j]), __double2loint(Y[j])}, s[1], t[1]);
            dot_term(w, Word2{__double2hiint(Z[j]), __double2loint(Z[j])}, s[2], t[2]);
        }
        U[2 * k] = wilke_factor(X[k], tb.W4[k]);
        U[2 * k + 1] = wilke_rcp(mix_value<LO>(s[0], t[0]), mix_value<LO>(s[1], t[1]), mix_value<LO>(s[2], t[2]), unit + qx,
                                 unit + qy, unit + qz, v[k]);
    }
    team_sync<TEAM>();
    double mu = 0.0;
    if (lane < 2) {
#pragma unroll 4
        for (int k = lane; k < K; k += 2) mu = fma(U[2 * k], U[2 * k + 1], mu);
    }
    mu += __shfl_sync(0xffffffffu, mu, 1);
    if (lane == 0) transport_out(io, 1, second)[o] = VT * mu;
    team_sync<TEAM>();

    // Diffusion, in tiles of 32 rows by 32 columns of pairs: lanes on consecutive pairs of a row (consecutive table
    // records) leave the reciprocals in the tile, then lanes on rows add theirs, then lanes on columns.
    double* S = Y;
    if (TEAM > 1) {  // bands of 32 rows: all warps evaluate the pairs, one adds the rows' sums, the others the columns'
        constexpr int LD = KMAX + 1;
        for (int base = 0; base < K; base += 32) {
            const int rows = min(32, K - base);
            for (int q = lane >> 5; q < rows; q += TEAM) {
                const int k = base + q;
                const PolyX* P = tb.diff + (size_t)k * (k - 1) / 2;
#pragma unroll 2
                for (int c = lane32; c < k; c += 32) {
                    const PolyX p = P[c];
                    T[q * LD + c] = rcp_fixed(poly_x(p, L), p.rcp_bias);
                }
            }
            __syncthreads();
            if (lane < 32) {
                if (lane < rows) {
                    const int k = base + lane;
                    const double* Trow = T + lane * LD;
                    double sa = 0.0, sb = 0.0;
                    int c = 0;
#pragma unroll 4
                    for (; c + 1 < k; c += 2) {
                        sa = fma(X[c], Trow[c], sa);
                        sb = fma(X[c + 1], Trow[c + 1], sb);
                    }
                    if (c < k) sa = fma(X[c], Trow[c], sa);
                    double s1 = sa + sb;
                    for (int q = lane + 1; q < rows; q++) s1 = fma(X[base + q], T[q * LD + k], s1);
                    S[k] = s1;
                }
            } else {
                for (int c = lane - 32; c < base; c += kStep - 32) {
                    double s1 = S[c];
#pragma unroll 4
                    for (int q = 0; q < rows; q++) s1 = fma(X[base + q], T[q * LD + c], s1);
                    S[c] = s1;
                }
            }
            __syncthreads();
        }
        for (int k = lane; k < K; k += kStep)
            transport_out(io, 2 + k, second)[o] = diffusion_x(MN, VT, tb.W[k], X[k], S[k]);
        return true;
    }
#pragma unroll 1
    for (int b = 0; 32 * b < K; b++) {
        const int r = 32 * b + lane, rows = min(32, K - 32 * b);
        double sa = 0.0, sb = 0.0;
#pragma unroll 1
        for (int t = 0; t <= b; t++) {
            const int j0 = 32 * t, jc = j0 + lane;
            const PolyX* P = tb.diff + (size_t)(32 * b) * (32 * b - 1) / 2 + jc;  // pair (32 b, jc); row k + 1 is k records on
            if (t < b) {
#pragma unroll 4
                for (int q = 0; q < rows; q++) {
                    const PolyX p = P[(size_t)q * (32 * b) + q * (q - 1) / 2];
                    T[33 * q + lane] = rcp_fixed(poly_x(p, L), p.rcp_bias);
                }
            } else {
#pragma unroll 1
                for (int q = 1; q < rows; q++) {
                    if (lane < q) {
                        const PolyX p = P[(size_t)q * (32 * b) + q * (q - 1) / 2];
                        T[33 * q + lane] = rcp_fixed(poly_x(p, L), p.rcp_bias);
                    }
                }
            }
            __syncwarp();
            const int columns = r < K ? min(32, r - j0) : 0;  // j0 is even: even columns in sa, odd ones in sb
            const double* Trow = T + 33 * lane;
            int c = 0;
#pragma unroll 4
            for (; c + 1 < columns; c += 2) {
                sa = fma(X[j0 + c], Trow[c], sa);
                sb = fma(X[j0 + c + 1], Trow[c + 1], sb);
            }
            if (c < columns) sa = fma(X[j0 + c], Trow[c], sa);
            if (t == b && r < K) S[r] = sa + sb;
            __syncwarp();
            if (jc < K) {
                double s = S[jc];
#pragma unroll 4
                for (int q = t == b ? lane + 1 : 0; q < rows; q++) s = fma(X[32 * b + q], T[33 * q + lane], s);
                S[jc] = s;
            }
            __syncwarp();
        }
    }
    for (int k = lane; k < K; k += 32) transport_out(io, 2 + k, second)[o] = diffusion_x(MN, VT, tb.W[k], X[k], S[k]);
    return true;
}

constexpr int kWarpCellWarpsX = 16;  // cells per block, as many as fit in shared memory

template <int KMAX>
__device__ __noinline__ void transport_cell_f64_warp(const TransportArgs<KMAX>& io, size_t i, size_t o, double* sh,
                                                     bool second) {
    transport_cell_warp<KMAX>(io.f64_tab, io, i, o, sh, second);
}

template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(32 * kWarpCellWarpsX) transport_x_warp_kernel(const uint8_t* __restrict__ gtab,
                                                                             uint32_t tab_bytes,
                                                                             const __grid_constant__ TransportArgs<KMAX> io,
                                                                             size_t n, int* status) {
    const EndAfterPrevious last;
    __shared__ uint64_t bar;
    if (SMEM) {
        if (!stage_to_shared(cb_dsmem, gtab, tab_bytes, &bar, status)) return;
    } else {
        load_math(gtab);
    }
    const TransportXTables tb(SMEM ? cb_dsmem : gtab);
    double* sh = reinterpret_cast<double*>(cb_dsmem + warp_table_bytes(SMEM, tab_bytes)) +
                 (size_t)(threadIdx.x >> 5) * kWarpScratch<KMAX>;
    if (io.count && !io.index2) n = min(n, (size_t)*io.count);
    const size_t warps = (size_t)gridDim.x * (blockDim.x >> 5);
    for (size_t j = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); j < n; j += warps) {
        const bool second = io.index2 && j >= io.n1;
        const size_t i = second ? (size_t)(io.index2[j - io.n1] & kIndexMask) : io.index ? (size_t)(io.index[j] & kIndexMask) : j;
        const size_t o = second ? j - io.n1 : (io.flags & kCompactOut) ? j : i;
        if (!transport_cell_x_warp<1, KMAX>(tb, io, i, o, sh, second)) {
            __syncwarp();
            transport_cell_f64_warp<KMAX>(io, i, o, sh, second);
        }
        __syncwarp();  // the scratch is reused by the warp's next cell
    }
}

template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(32 * kTeamWarps) transport_x_team_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                                                           const __grid_constant__ TransportArgs<KMAX> io,
                                                                           size_t n, int* status) {
    const EndAfterPrevious last;
    __shared__ uint64_t bar;
    if (SMEM) {
        if (!stage_to_shared(cb_dsmem, gtab, tab_bytes, &bar, status)) return;
    } else {
        load_math(gtab);
    }
    const TransportXTables tb(SMEM ? cb_dsmem : gtab);
    double* sh = reinterpret_cast<double*>(cb_dsmem + warp_table_bytes(SMEM, tab_bytes));
    if (io.count && !io.index2) n = min(n, (size_t)*io.count);
    for (size_t j = blockIdx.x; j < n; j += gridDim.x) {
        const bool second = io.index2 && j >= io.n1;
        const size_t i = second ? (size_t)(io.index2[j - io.n1] & kIndexMask) : io.index ? (size_t)(io.index[j] & kIndexMask) : j;
        const size_t o = second ? j - io.n1 : (io.flags & kCompactOut) ? j : i;
        const bool done = transport_cell_x_warp<kTeamWarps, KMAX>(tb, io, i, o, sh, second);
        __syncthreads();
        if (!done && threadIdx.x < 32) transport_cell_f64_warp<KMAX>(io, i, o, sh, second);
        __syncthreads();  // the scratch is reused by the block's next cell
    }
}

namespace {
// Calls and gathered launches of up to a cell per SM go one cell per block of eight warps: one state 27, 70 -> 53 and
// 700 -> 205 us (10, 53, 250 species), where Wilke's rows and the pairs of a band of rows take all lanes at once; the
// sums keep their lanes and order.
// Calls and gathered launches of up to this many cells per SM go one cell per warp: a thread's cell takes 55, 460 and
// 18,000 us however few there are (10, 53, 250 species), a warp's 30, 70 and 660 us and then 9, 34 and 480 ns per
// cell; beyond these lines the thread form is the faster.
template <int KMAX>
constexpr size_t kWarpCellsPerSmX = KMAX == 16 ? 24 : KMAX == 64 ? 96 : 256;

template <int KMAX>
cudaError_t launch_transport_xk(const uint8_t* tab, uint32_t tab_bytes, const TransportArgs<KMAX>& io, size_t n,
                                cudaStream_t st, int* status) {
    if (n <= (size_t)sm_count()) {
        const size_t scratch = kTeamScratch<KMAX> * sizeof(double);
        const bool smem = warp_table_bytes(true, tab_bytes) + scratch <= (size_t)max_table_smem();
        const size_t bytes = warp_table_bytes(smem, tab_bytes) + scratch;
        auto kern = smem ? transport_x_team_kernel<KMAX, true> : transport_x_team_kernel<KMAX, false>;
        const cudaError_t e = allow_shared(kern);
        if (e != cudaSuccess) return e;
        return launch_one(kern, n, 32 * kTeamWarps, bytes, st, tab, tab_bytes, io, n, status);
    }
    if (n <= (size_t)sm_count() * kWarpCellsPerSmX<KMAX>) {
        const size_t share = (n + sm_count() - 1) / sm_count(), scratch = kWarpScratch<KMAX> * sizeof(double);
        const bool smem = warp_table_bytes(true, tab_bytes) + 4 * scratch <= (size_t)max_table_smem();
        int warps = share < (size_t)kWarpCellWarpsX ? (int)share : kWarpCellWarpsX;
        while (warps > 1 && warp_table_bytes(smem, tab_bytes) + warps * scratch > (size_t)max_table_smem()) warps--;
        const size_t bytes = warp_table_bytes(smem, tab_bytes) + warps * scratch;
        auto kern = smem ? transport_x_warp_kernel<KMAX, true> : transport_x_warp_kernel<KMAX, false>;
        const cudaError_t e = allow_shared(kern);
        if (e != cudaSuccess) return e;
        int per_sm = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, bytes);
        if (per_sm < 1) per_sm = 1;
        size_t grid = (size_t)sm_count() * per_sm;
        const size_t want = (n + warps - 1) / warps;
        if (want < grid) grid = want ? want : 1;
        return launch_one(kern, grid, 32 * warps, bytes, st, tab, tab_bytes, io, n, status);
    }
    return launch_table_kernel<kTransportXBlock<KMAX>>(transport_x_kernel<KMAX, true>, transport_x_kernel<KMAX, false>, tab,
                                                 tab_bytes, io, n, kMathBytes, false, st, status);
}
}  // namespace

cudaError_t launch_transport_x(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                               cudaStream_t st, int* status) {
    switch (kmax) {
    case 16: return launch_transport_xk<16>(tab, tab_bytes, *static_cast<const TransportArgs<16>*>(args), n, st, status);
    case 64: return launch_transport_xk<64>(tab, tab_bytes, *static_cast<const TransportArgs<64>*>(args), n, st, status);
    case 256:
        return launch_transport_xk<256>(tab, tab_bytes, *static_cast<const TransportArgs<256>*>(args), n, st, status);
    default: return cudaErrorInvalidValue;
    }
}
size_t transport_x_warp_cells(int kmax) {
    return (size_t)sm_count() * (kmax == 16 ? kWarpCellsPerSmX<16> : kmax == 64 ? kWarpCellsPerSmX<64> : kWarpCellsPerSmX<256>);
}
template <int KMAX>
static size_t wave_transport_xk(uint32_t tab_bytes) {
    return wave_of<kTransportXBlock<KMAX>>(transport_x_kernel<KMAX, true>, transport_x_kernel<KMAX, false>, tab_bytes, kMathBytes);
}
size_t wave_transport_x(int kmax, uint32_t tab_bytes) {
    return kmax == 16 ? wave_transport_xk<16>(tab_bytes) : kmax == 64 ? wave_transport_xk<64>(tab_bytes)
                                                                    : kmax == 256 ? wave_transport_xk<256>(tab_bytes) : 0;
}

cudaError_t set_stage_wait_polls_tx(long long polls) { return cudaMemcpyToSymbol(g_stage_wait_polls, &polls, sizeof polls); }

}  // namespace cbg
