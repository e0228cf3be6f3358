// Pieces of the plain rates program in its fixed-point form, shared by its thread-per-cell and
// warp-per-cell kernels (kernels_fixed.cu): what depends on the temperature alone as 64-bit fixed-point
// logarithms on the integer pipe (fixed_math.cuh), the rate of progress and its accumulation in FP64.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fixed_math.cuh"
#include "kernels.h"
#include "rates_core.cuh"
#include "tables_fixed.h"

namespace cbg {

struct RatesXTables {
    const RatesXHeader* H;
    const SpeciesX* species;
    const ThermoX* thermo;
    const ReactionX* reactions;
    const FalloffX* falloff;
    const Word2* eff;
    const int32_t* eff_q;
    const int32_t *csr_start, *csr;
    __device__ explicit RatesXTables(const uint8_t* tab)
        : H(reinterpret_cast<const RatesXHeader*>(tab + kMathBytes + kFixMathBytes)),
          species(reinterpret_cast<const SpeciesX*>(tab + H->off_species)),
          thermo(reinterpret_cast<const ThermoX*>(tab + H->off_thermo)),
          reactions(reinterpret_cast<const ReactionX*>(tab + H->off_reactions)),
          falloff(reinterpret_cast<const FalloffX*>(tab + H->off_falloff)),
          eff(reinterpret_cast<const Word2*>(tab + H->off_eff)),
          eff_q(reinterpret_cast<const int32_t*>(tab + H->off_eff_q)),
          csr_start(reinterpret_cast<const int32_t*>(tab + H->off_csr_start)),
          csr(reinterpret_cast<const int32_t*>(tab + H->off_csr)) {}
};

// A cell's temperature in fixed point.
struct TempsX {
    double T;
    Word2 l, r, p[4];   // log2 T, 1/T, (T / 2^pw)^i with pw = 11 below kFixTmid, else 13
    long long lc0;      // log2(P0 / (R T)), Qy
};

__device__ __forceinline__ TempsX make_temps(const RatesXHeader& H, double T, double rcpT) {
    TempsX t;
    t.T = T;
    int e;
    const long long f = log2_frac(T, e);
    t.l = split_word(((long long)e << (kLq + kLo)) + ((f + 32) >> 6));
    t.lc0 = H.lC0 - (((long long)e << kYq) + ((f + (1ll << 10)) >> 11));
    // 1/T with the residual of its FP64 value
    t.r = split_word(dbl_to_fix(rcpT, kRq + kLo) + dbl_to_fix(rcpT * fma(-T, rcpT, 1.0), kRq + kLo));
    const int pw = T < kFixTmid ? 11 : 13;
    const double T2 = T * T, T3 = T * T2, T4 = T2 * T2;
    t.p[0] = split_word(dbl_to_fix(T, kPq + kLo - pw));
    t.p[1] = split_word(dbl_to_fix(T2, kPq + kLo - 2 * pw));
    t.p[2] = split_word(dbl_to_fix(T3, kPq + kLo - 3 * pw));
    t.p[3] = split_word(dbl_to_fix(T4, kPq + kLo - 4 * pw));
    return t;
}

// log2 of a rate constant, Qy.
__device__ __forceinline__ long long arrhenius_log2(const ArrheniusX& a, const TempsX& t) {
    long long s1 = a.a, s2 = 0;
    dot_term(a.b, t.l, s1, s2);
    dot_term(a.e, t.r, s1, s2);
    return dot_value(s1, s2);
}
// min(f32::MAX, A T^power), as the FP64 form's arrhenius.
static __device__ __noinline__ double rate_exact(int power, double A, double T) {
    const double T2 = T * T, rcpT = __drcp_rn(T);
    double f = 1.0;
    switch (power) {
    case kRcpT2: f = rcpT * rcpT; break;
    case kRcpT: f = rcpT; break;
    case kT4: f = T2 * T2; break;
    case kT3: f = T * T2; break;
    case kT2: f = T2; break;
    case kT: f = T; break;
    }
    return min_pos(kF32Max, f * A);
}
// min(f32::MAX, k) of reaction.rs:138.
__device__ __forceinline__ double rate_constant(const ArrheniusX& a, const TempsX& t) {
    return rate_fix(arrhenius_log2(a, t));
}

// The table piece at T (SpeciesX): 0 for T <= split (lib.rs:15; never for a NaN split).
__device__ __forceinline__ int piece_x(double split, double T) {
    return bits(T) <= bits(split) && (bits(split) >> 52) < 0x7ff ? 0 : __double2hiint(T) < (1023 + 11) << 20 ? 1 : 2;
}

// The cross products of two dot products with word positions a (Qy) and b (3 bits below) as a number in Qy. Each of four
// terms of b is below 2^58 + 2^58 (a coefficient's high word is below 2^30, a power's at most 2^30, low words at most
// 2^28), so their sum, below 2^61, is not shifted up; a's two terms are below 2^60.2 together. (The high words' sums may
// wrap on their way: the total is in range.)
__device__ __forceinline__ long long low_words(long long a2, long long b2) {
    return (b2 + (a2 >> 3) + (1ll << (kLo - 4))) >> (kLo - 3);
}

// Gibbs energy over RT (reaction.rs:75-110) in base-2 units, Qy.
__device__ __forceinline__ long long gibbs_log2(const SpeciesX& s, const TempsX& t) {
    const int set = piece_x(s.split, t.T);
    const Word2* g = s.g[set];
    long long a1 = s.g0[set], a2 = 0, b1 = 0, b2 = 0;
    dot_term(g[0], t.l, a1, a2);
    dot_term(g[1], t.r, a1, a2);
#pragma unroll
    for (int i = 0; i < 4; i++) dot_term(g[2 + i], t.p[i], b1, b2);  // Q(kGq + kPq), 3 bits below Qy
    static_assert(kGq + kPq == kYq - 3 && kBq + kLq == kYq && kEq + kRq == kYq, "word positions");
    return a1 + (b1 << 3) + low_words(a2, b2);
}

// h / RT and cp / R of a species.
__device__ __forceinline__ double enthalpy_x(const ThermoX& s, int set, const TempsX& t) {
    const Word2* h = s.h[set];
    long long a1 = s.h0[set], a2 = 0, b1 = 0, b2 = 0;
    dot_term(h[4], t.r, a1, a2);
#pragma unroll
    for (int i = 0; i < 4; i++) dot_term(h[i], t.p[i], b1, b2);
    return fix_to_dbl(a1 + (b1 << 3) + low_words(a2, b2), kYq);
}
__device__ __forceinline__ double heat_capacity_x(const ThermoX& s, int set, const TempsX& t) {
    const Word2* c = s.cp[set];
    long long b1 = 0, b2 = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) dot_term(c[i], t.p[i], b1, b2);
    return fix_to_dbl(s.cp0[set] + (b1 << 3) + low_words(0, b2), kYq);
}

// The Troe forward coefficient in the general case (reaction.rs:160-193).
static __device__ __noinline__ double troe_general(const RatesXHeader& H, const FalloffX& f, long long y0, long long yi,
                                                   double lF, double M) {
    const double k0 = rate_fix(y0);
    double Pr, kinf;
    if (f.flags & kKinfConst) {
        Pr = M * k0;
        kinf = f.ainf;
    } else {
        const double ki = rate_fix(yi);
        Pr = div64(M * k0, ki + kF32MinPos);
        kinf = f.ainf * ki;
    }
    const double Cc = fma(-0.67, lF, -H.l10_04);
    const double Nn = fma(-1.27, lF, H.l10_075);
    const double lPrC = log2_dbl(Pr + kF32MinPos) + Cc;
    const double f1 = div64(lPrC, fma(-0.14, lPrC, Nn));
    const double Fb = exp2_dbl(div64(lF, fma(f1, f1, 1.0)));
    return div64((Fb * kinf) * Pr, Pr + 1.0);
}

// Forward coefficient of one reaction: k, k M, or the falloff-blended value (reaction.rs:149-203).
template <int MODEL>
__device__ __forceinline__ double forward_x(const RatesXHeader& H, const ArrheniusX& k, const FalloffX* fo,
                                            const TempsX& t, double rcpT, double M) {
    if constexpr (MODEL == 4) {  // Troe (reaction.rs:160-193), logarithms in base 2
        const FalloffX& f = *fo;
        double lF;
        if (f.flags & kFcentConst) {
            lF = f.l2_fcent;
        } else {
            double F = 0.0;
            if (f.flags & kTermT3) F = f.c1mA * exp2_dbl(t.T * f.c3);
            if (f.flags & kTermT1) F += f.cA * exp2_dbl(t.T * f.c1);
            if (f.flags & kTermAConst) F += f.cA;
            if (f.flags & kTermT2) F += exp2_dbl(f.cmT2 * rcpT);
            lF = log2_dbl(F);
        }
        const long long y0 = arrhenius_log2(f.k0, t), yi = f.flags & kKinfConst ? 0 : arrhenius_log2(k, t);
        // log2 Pr = log2 M + log2 k0 - log2 k_inf, and k = F A_inf k_inf Pr / (1 + Pr) by its logarithm, while
        // neither coefficient is capped at f32::MAX and f32::MIN_POSITIVE vanishes next to k_inf and Pr
        // (nor k0 a constant: its y0 is above all others)
        if (!(M > 1e-200 && M < 1e200) || y0 >= (127ll << kYq) || yi >= (127ll << kYq) || yi < -(60ll << kYq))
            return troe_general(H, f, y0, yi, lF, M);
        const long long lPr = log2_fix(M) + y0 - yi;
        if (lPr < -(60ll << kYq) || lPr > (1000ll << kYq)) return troe_general(H, f, y0, yi, lF, M);
        const double Cc = fma(-0.67, lF, -H.l10_04);
        const double Nn = fma(-1.27, lF, H.l10_075);
        const double lPrC = fix_to_dbl(lPr, kYq) + Cc;
        const double f1 = div64(lPrC, fma(-0.14, lPrC, Nn));
        const double lFb = div64(lF, fma(f1, f1, 1.0));
        if (!(lFb > -1000.0 && lFb < 1000.0)) return troe_general(H, f, y0, yi, lF, M);
        return exp2_fix(dbl_to_fix(lFb, kYq) + f.lainf + yi + lPr - log2_fix(exp2_core(lPr) + 1.0));
    } else if constexpr (MODEL == 3) {  // Lindemann (reaction.rs:153-159)
        const double Ck0 = M * rate_constant(fo->k0, t);
        const double ki = rate_constant(k, t);
        return div64(Ck0 * ki, (Ck0 + ki) + kF32MinPos);
    } else if constexpr (MODEL == 5) {  // SRI: the commented formula of reaction.rs:194-203
        const FalloffX& f = *fo;
        const double k0 = rate_constant(f.k0, t);
        const double ki = rate_constant(k, t);
        const double Pr = div64(M * k0, ki + kF32MinPos);
        const double lP = log2_dbl(Pr + kF32MinPos) * 0.69314718055994530942;  // natural
        double base = exp2_dbl(f.smrC * t.T);
        if (f.sri_flags & kSriA) base = fma(f.sA, exp2_dbl(f.smB * rcpT), base);
        double F = exp2_dbl(log2_dbl(base) * rcp64(fma(lP, lP, 1.0)));
        if (f.sri_flags & kSriD) F = f.sD * F;
        if (f.sri_flags & kSriE) F *= exp2_dbl(f.sE * log2_dbl(t.T));
        return div64((F * ki) * Pr, Pr + 1.0);
    } else if constexpr (MODEL == 2) {  // three-body (reaction.rs:152)
        return rate_constant(k, t) * M;
    } else {
        return rate_constant(k, t);
    }
}

// Logarithm of one net species' factor of 1/Kc: the exponent of its capped Gibbs exponential.
__device__ __forceinline__ long long gibbs_term(const RatesXHeader& H, long long g, bool consumed) {
    const long long v = consumed ? -g : g, cap = consumed ? H.lcbrt : H.lM3;
    return v < cap ? v : cap;
}

// One reaction (reaction.rs:149-327) of a cell with arrays C (FP64 concentrations) and g (Gibbs energies, Qy),
// its rate added to the species rates (w) or handed to emit(orig, cR). The cell's arrays are far away
// (thread-local memory in L2): everything a reaction reads from them is loaded at its start, so that one wait
// runs under its rate constant.
// REVERSIBLE: models other than 1. forward(k): the forward coefficient from the reaction's constants.
template <bool REVERSIBLE, bool SUM, class CellT, class Forward, class Emit>
__device__ __forceinline__ void reaction_x(const RatesXTables& tb, int r, const CellT& c, double* w, Forward forward,
                                           Emit emit) {
    const RatesXHeader& H = *tb.H;
    const ReactionX& x = tb.reactions[r];
    const uint4 idx = *reinterpret_cast<const uint4*>(x.r_k);
    const uint32_t shape = x.shape;
    const int msn = (int)((shape / kShapeMsn) & 7) - 2;
    long long y = msn == 0 ? 0 : msn == 1 ? c.t.lc0 : msn == -1 ? -c.t.lc0 : -2 * c.t.lc0;
    if (!(shape & kShapeGeneral)) {
        const int net = (int)((shape / kShapeNet) & 7);
        const int r0 = idx.x & 255, r1 = (idx.x >> 8) & 255, p0 = idx.y & 255, p1 = (idx.y >> 8) & 255;
        const bool r2 = shape & kShapeR2, p2 = shape & kShapeP2;
        const double cr0 = c.C[r0], cr1 = r2 ? c.C[r1] : 0.0;
        double cp0 = 0.0, cp1 = 0.0;
        long long g[4];
        double wk[4];
        if (REVERSIBLE) {
            cp0 = c.C[p0];
            if (p2) cp1 = c.C[p1];
#pragma unroll
            for (int j = 0; j < 4; j++) g[j] = j < net ? c.g[(idx.z >> (8 * j)) & 255] : 0;
        }
        if (SUM) {
#pragma unroll
            for (int j = 0; j < 4; j++) wk[j] = j < net ? w[(idx.z >> (8 * j)) & 255] : 0.0;
        }
        const double kf = forward(x.k);
        double pK = 0.0;
        if (REVERSIBLE) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (j < net) {
                    const long long v = gibbs_term(H, g[j], shape & (kShapeNeg << j));
                    y += shape & (kShapeTwo << j) ? 2 * v : v;
                }
            }
            pK = exp2_fix(y);
        }
        // The FP64 tail by shape, one real branch: predicated-off FP64 instructions occupy the pipe too.
        double cR = 0.0;
        double nu[4];
        if (SUM) {
#pragma unroll
            for (int j = 0; j < 4; j++)  // +-1 or +-2
                nu[j] = __hiloint2double((int)((0x3ff00000u + ((shape >> (9 + j)) & 1) * 0x100000u) | (((shape >> (5 + j)) & 1) << 31)), 0);
        }
#define CB_TAIL(R2, P2, NET)                                        \
    do {                                                            \
        double a = R2 ? cr0 * cr1 : cr0;                            \
        if (REVERSIBLE) a = fma(-pK, P2 ? cp0 * cp1 : cp0, a);      \
        cR = kf * a;                                                \
        if (SUM) {                                                  \
            for (int j = 0; j < NET; j++) wk[j] = fma(nu[j], cR, wk[j]); \
        }                                                           \
    } while (0);                                                    \
    break
        switch (shape & (SUM ? 31 : 3)) {
        case 0: CB_TAIL(0, 0, 0);
        case 1: CB_TAIL(1, 0, 0);
        case 2: CB_TAIL(0, 1, 0);
        case 3: CB_TAIL(1, 1, 0);
        case 4: CB_TAIL(0, 0, 1);
        case 5: CB_TAIL(1, 0, 1);
        case 6: CB_TAIL(0, 1, 1);
        case 7: CB_TAIL(1, 1, 1);
        case 8: CB_TAIL(0, 0, 2);
        case 9: CB_TAIL(1, 0, 2);
        case 10: CB_TAIL(0, 1, 2);
        case 11: CB_TAIL(1, 1, 2);
        case 12: CB_TAIL(0, 0, 3);
        case 13: CB_TAIL(1, 0, 3);
        case 14: CB_TAIL(0, 1, 3);
        case 15: CB_TAIL(1, 1, 3);
        case 16: CB_TAIL(0, 0, 4);
        case 17: CB_TAIL(1, 0, 4);
        case 18: CB_TAIL(0, 1, 4);
        default: CB_TAIL(1, 1, 4);
        }
#undef CB_TAIL
        if (SUM) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < net) w[(idx.z >> (8 * j)) & 255] = wk[j];
        } else {
            emit(x.orig, cR);
        }
        return;
    }
    const double kf = x.k.e.lo == kExactRate ? rate_exact(x.k.b.lo, __longlong_as_double(x.k.a), c.t.T) : forward(x.k);
    double Rf = 1.0, Pp = 1.0;
#pragma unroll 1
    for (int q = 0; q < kMaxSide; q++) {
#pragma unroll 1
        for (int m = 0; m < x.r_n[q]; m++) Rf *= c.C[x.r_k[q]];
#pragma unroll 1
        for (int m = 0; m < x.p_n[q]; m++) Pp *= c.C[x.p_k[q]];
    }
    if (REVERSIBLE) {
#pragma unroll 1
        for (int q = 0; q < kMaxNet; q++) {
            const int nu = x.net_n[q];
            if (nu) y += (nu < 0 ? -nu : nu) * gibbs_term(H, c.g[x.net_k[q]], nu < 0);
        }
        Rf = fma(-exp2_fix(y), Pp, Rf);
    }
    const double cR = kf * Rf;
    if (SUM) {
#pragma unroll 1
        for (int q = 0; q < kMaxNet; q++)
            if (x.net_n[q]) w[x.net_k[q]] = fma(small_int_to_double(x.net_n[q]), cR, w[x.net_k[q]]);
    } else {
        emit(x.orig, cR);
    }
}

}  // namespace cbg
