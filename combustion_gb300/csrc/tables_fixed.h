// Tables of the plain rates kernels' fixed-point form (fixed_math.cuh, kernels.cu), built by
// fixed_tables.cpp from the FP64 tables (tables.h) of the same mechanism.
//
// Everything that depends on the temperature alone (rate constants, Gibbs energies) is evaluated as a
// base-2 logarithm in 64-bit fixed point on the integer pipe; the third-body sums are fixed-point dot
// products. Numbers are Qn: the integer times 2^-n. A product term keeps each factor as two signed
// 32-bit words, value = (hi 2^29 + lo) 2^-(q + 29) with |lo| <= 2^28, hi Qq.
#pragma once
#include <stdint.h>

#include "tables.h"

namespace cbg {

constexpr int kExpTable = 1024, kLogTable = 512;
struct FixMath {
    uint64_t exp2t[kExpTable];  // 2^(j/1024), Q62
    int64_t log2c[kLogTable];   // -log2(rc[j] / 4096), Q62
    uint32_t rc[kLogTable];     // nearest 12-bit reciprocal of 1 + (j + 1/2) / 512, Q12
};
constexpr int kFixMathBytes = (int)sizeof(FixMath);
static_assert(kFixMathBytes % kAlign == 0, "fixed-point tables must keep the blob sections aligned");

// Bounds of the fixed-point form. A cell takes it for T in [Tmin, kFixTmax), Tmin the lowest of kFixTmin over which every
// constant of the mechanism fits its word (fixed_tables.cpp checks; without one the FP64 form runs). The words of 1 / T
// hold 65 K; large exponents over T may not (100 K at 53 and 250 species of the generator).
constexpr double kFixTmin[] = {65.0, 100.0, 200.0}, kFixTmax = 8192.0, kFixTmid = 2048.0;
constexpr int kYq = 51;    // base-2 logarithms: |y| < 2^12
constexpr int kLo = 29;    // bits of a low word
constexpr int kLq = 27;    // log2 T, hi word (log2 T < 13)
constexpr int kBq = 24;    // its factor, |.| < 64
constexpr int kRq = 37;    // 1 / T, hi word (1/T <= 1/65)
constexpr int kEq = 14;    // its factor, |.| < 2^17
constexpr int kPq = 30;    // (T / 2^p)^i, hi word, p = 11 below 2048 K and 13 above
constexpr int kGq = 18;    // its factor, |.| < 4096
// Third-body sums: C_k / S (S a power of two above both totals) in 60 bits, efficiencies - 1 of four rows in units of
// 2^-(q + kThirdLo), q the largest (at most 29) that keeps their high words below 2^31 and the sum of a row's below 2^33:
// then the cross products' sum stays below 2^63. The dropped products of low words are below 2^-(q + 32) S each; the sum's
// error is below that of FP64 FMAs for every efficiency that is accepted (of 61 beside 52 of 0.5 to 3 at most 1.9e-16 of
// M, FP64 9.2e-16; with one unit for the whole mechanism and 29-bit low words 4e-15).
constexpr int kThirdLo = 30;
constexpr double kMaxEff = 128.0;  // of |efficiency - 1|

struct Word2 {
    int32_t hi, lo;
};

// log2 of k = exp(beta ln T + mEa / T + ln A). Coefficients that FP64 holds exactly, or to a rounding or two, are not
// taken through a logarithm (whose last bit is 1.5e-16 of k):
//  - a constant is `a` = the bits of A + kConstRate with no factors. As a logarithm it lies above every other one's
//    (A = 2^-500 .. 2^499 gives 2,046 .. 4,046, the others are below kMaxRate), where rate_slow finds it;
//  - a constant times a whole power of T, of an elementary reaction, is the bits of A, the power (Factor) in b.lo and
//    e.lo = kExactRate, in a reaction of general shape. (Where a third body multiplies it, its sum is the more exact for
//    being in fixed point, and the logarithm's error is no more than that gains.)
struct ArrheniusX {
    Word2 b, e;  // factors of log2 T and 1 / T
    int64_t a;   // Qy
};
constexpr int64_t kConstRate = 1000ll << kYq, kConstRateMin = 2046ll << kYq;
constexpr double kMaxRate = 2000.0;  // of |log2 k|
constexpr int32_t kExactRate = 1 << 29;  // no balanced low word

// Shape flags of a reaction (ReactionX::shape).
enum Shape : uint32_t {
    kShapeR2 = 1,        // two reactant factors (else one)
    kShapeP2 = 2,        // two product factors (else one)
    kShapeNet = 4,       // net species: bits 2-4 (1 .. 4)
    kShapeNeg = 32,      // bit 5 + j: net species j is consumed
    kShapeTwo = 512,     // bit 9 + j: by two
    kShapeMsn = 8192,    // minus the net order, plus 2: bits 13-15
    kShapeGeneral = 65536  // none of the above but the order: the lists below with their multiplicities
};
struct ReactionX {  // 64 bytes
    ArrheniusX k;
    uint32_t shape;
    int32_t orig;
    // up to two factors on each side (a doubled species twice) and four net species changing by one or two,
    // or (kShapeGeneral) distinct species with the multiplicities that follow
    uint8_t r_k[kMaxSide], p_k[kMaxSide], net_k[kMaxNet];
    int8_t r_n[kMaxSide], p_n[kMaxSide], net_n[kMaxNet];
};
static_assert(sizeof(ReactionX) == 64, "four 16-byte loads");

// One per reaction of models 2-5, in reaction order (three-body entries unused). Exponents and
// logarithms in base 2.
struct FalloffX {
    ArrheniusX k0;
    double ainf, c1mA, cA, c3, c1, cmT2, l2_fcent;
    int64_t lainf;          // log2(ainf), Qy
    int32_t flags, sri_flags;
    double sA, smB, smrC, sD, sE;
};

// Gibbs energy over RT in base-2 units: piece 0 for T <= split, else 1 below kFixTmid and 2 above (the
// same polynomial in (T / 2^11) and (T / 2^13)).
struct SpeciesX {
    double split;
    int64_t g0[3];
    Word2 g[3][6];  // factors of log2 T, 1/T, (T/2^p)^1 .. ^4
    int32_t need_exp, need_exp_neg;
};

// h / RT (powers 1 .. 4 of T / 2^p, then 1/T) and cp / R, pieces as SpeciesX::g.
struct ThermoX {
    double split, dtE;
    int64_t h0[3], cp0[3];  // Qy
    Word2 h[3][5];          // factors of (T/2^p)^1 .. ^4, 1/T
    Word2 cp[3][4];
};

struct RatesXHeader {
    int32_t K, A, R, n_eff, total_bytes, off_species, off_thermo, off_reactions, off_falloff, off_eff;
    int32_t off_eff_q;  // q of every four rows
    int32_t off_csr_start, off_csr;  // per species the reactions that change it, in order: [K + 1]; r << 8 | nu
    int32_t group_end[6];
    int64_t lM3, lcbrt, lC0;  // log2 of the Gibbs exponentials' caps and of P0 / R, Qy
    double l10_04, l10_075;   // 0.4 and 0.75 log2(10)
    double Tmin;
};

// ---- transport --------------------------------------------------------------------------------------
// A fitted polynomial D = P0 + P1 L + .. + P4 L^4 in L = ln(T/T0), over 2^sp so that it lies in (2^-6, 1) over
// the fixed-point temperature range: the widest of these that its mechanism's polynomials allow and whose L need no larger
// 2^pw than the narrowest's (at T0 = 1,000 K 136 to 7,380 K, |L| < 2).
constexpr double kFixTransportT[][2] = {{136.0, 7380.0}, {160.0, 6000.0}, {200.0, 5000.0}, {200.0, 4000.0}};
constexpr int kLpq = 29;  // (L / 2^pw)^m, hi word
constexpr int kPpq = 28;  // its coefficient, |.| < 4
constexpr int kPlo = 30;  // bits of their low words
constexpr int kDq = 60;   // D 2^-sp
struct alignas(16) PolyX {  // three 16-byte loads
    Word2 p[4];
    int64_t p0;
    int32_t sp, rcp_bias;  // D = d 2^(sp - 60), 1/D = R 2^-(56 + sp) (rcp_fixed): its exponent bias
};
static_assert(sizeof(PolyX) == 48, "three 16-byte loads");

// Words of the Wilke sums: a^2 (column j: the rows k, so that rows in registers or lanes read consecutive words) times
// a cell's X, X/v', X/v'^2 over their largest. A product of low words is dropped: below 2^-57 of the largest term with 64
// species. Sums over 256 leave fewer bits; with 27 low ones (54-bit words) it is below 2^-56, and coherent traces beside a
// main species put viscosities at 250 species off by 6e-16, as FP64 sums (29 of 54 and 55 bits: 2^-53 and 1.4e-14).
template <int KMAX>
constexpr int kMixLo = KMAX <= 64 ? 29 : 27;
template <int KMAX>
constexpr int kMixAq = KMAX <= 64 ? 56 : 54;  // |a^2| 2^a_shift < 2^this
template <int KMAX>
constexpr int kMixXq = KMAX <= 64 ? 57 : 54;  // |X| over a power of two above the largest, < 2^this

struct TransportXHeader {
    int32_t K, n_pairs, total_bytes, pw;
    int32_t off_cond, off_visc, off_W, off_W4, off_diff, off_A2;  // polynomials, W, sqrt(W), pairs, a^2 by columns
    int32_t a_shift, pad;
    double T0, Tn_lo, Tn_hi, pad2;
};

}  // namespace cbg
