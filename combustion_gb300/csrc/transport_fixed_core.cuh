// Pieces of the plain transport program in fixed point, shared by its thread-per-cell and warp-per-cell kernels
// (transport_fixed.cu) so that both give a cell the same bits: the fitted polynomials, their reciprocals and
// Wilke's mixing sums are exact integer sums rounded once; the FP64 sums over species run in one order.
//
// With v'_k = v_k W_k^(-1/4), Wilke's denominator sum_j X_j (a_kj + b_kj v_k / v_j)^2 (transport.rs:148-158) is
// sum_j a_kj^2 X_j (1 + v'_k / v'_j)^2, since b_kj = a_kj (W_j / W_k)^(1/4): one matrix for three dot products.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fixed_math.cuh"
#include "kernels.h"
#include "tables_fixed.h"
#include "transport_cell.cuh"

namespace cbg {

struct TransportXTables {
    const TransportXHeader* H;
    const PolyX *cond, *visc, *diff;
    const double *W, *W4;
    const Word2* A2;
    __device__ explicit TransportXTables(const uint8_t* tab)
        : H(reinterpret_cast<const TransportXHeader*>(tab + kMathBytes)),
          cond(reinterpret_cast<const PolyX*>(tab + H->off_cond)), visc(reinterpret_cast<const PolyX*>(tab + H->off_visc)),
          diff(reinterpret_cast<const PolyX*>(tab + H->off_diff)), W(reinterpret_cast<const double*>(tab + H->off_W)),
          W4(reinterpret_cast<const double*>(tab + H->off_W4)), A2(reinterpret_cast<const Word2*>(tab + H->off_A2)) {}
};

struct PowersX {
    Word2 l[4];  // (L / 2^pw)^1 .. ^4
};
__device__ __forceinline__ PowersX log_powers(const TransportXHeader& H, double Tn) {
    const double L1 = log64(Tn), L2 = L1 * L1, L3 = L2 * L1, L4 = L3 * L1;
    PowersX p;
    p.l[0] = split_word<kPlo>(dbl_to_fix(L1, kLpq + kPlo - H.pw));
    p.l[1] = split_word<kPlo>(dbl_to_fix(L2, kLpq + kPlo - 2 * H.pw));
    p.l[2] = split_word<kPlo>(dbl_to_fix(L3, kLpq + kPlo - 3 * H.pw));
    p.l[3] = split_word<kPlo>(dbl_to_fix(L4, kLpq + kPlo - 4 * H.pw));
    return p;
}
__device__ __forceinline__ long long poly_x(const PolyX& P, const PowersX& L) {
    long long s1 = 0, s2 = 0;
#pragma unroll
    for (int m = 0; m < 4; m++) dot_term(P.p[m], L.l[m], s1, s2);
    static_assert(kPpq + kLpq == kDq - 3, "word positions");
    return P.p0 + (s1 << 3) + ((s2 + (1ll << (kPlo - 4))) >> (kPlo - 3));
}

// Exponent e with |x| < 2^e of the largest of finite doubles, from the maximum of their high words' magnitudes.
__device__ __forceinline__ int exponent_above(int largest_hi) { return (largest_hi >> 20) - 1022; }

// mu's term X_k v_k^2 / den_k = X_k W_k^(1/2) / (s3 + r (2 s2 + r s1)), r = 1 / v'_k, of the three sums over j (unit
// 2^-q each), as a factor and a reciprocal.
__device__ __forceinline__ double wilke_factor(double Xk, double W4k) { return __dmul_rn(Xk, W4k); }
__device__ __forceinline__ double wilke_rcp(long long s1, long long s2, long long s3, int q1, int q2, int q3, double r) {
    return rcp64(fma(r, fma(r, fix_to_dbl(s1, q1), fix_to_dbl(s2, q2 - 1)), fix_to_dbl(s3, q3)));
}
// rho D_k of its mixing sum (transport.rs:176).
__device__ __forceinline__ double diffusion_x(double MN, double VT, double W, double X, double S) {
    return __dmul_rn(__dmul_rn(fma(-W, X, MN), VT), rcp64(S));
}
// The three sums' accumulators to values in one unit (one bit finer than the hi-hi products').
template <int LO>
__device__ __forceinline__ long long mix_value(long long s1, long long s2) {
    return (s1 << 1) + ((s2 + (1ll << (LO - 2))) >> (LO - 1));
}

}  // namespace cbg
