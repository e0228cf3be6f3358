// Fixed-point tables of the plain rates kernels (tables_fixed.h) from a mechanism's packed FP64 tables.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <iterator>
#include <vector>

#include "kernels.h"
#include "mechanism.hpp"
#include "tables_fixed.h"

namespace cbg {
namespace {

const long double kLog2e = 1.0L / std::log(2.0L);

bool to_fix(long double x, int q, long double limit, int64_t& v) {
    if (!(std::fabs(x) < limit)) return false;
    v = (int64_t)std::llround(std::ldexp(x, q));
    return true;
}
Word2 words(int64_t v, int lo = kLo) {
    Word2 w;
    w.hi = (int32_t)((v + (1ll << (lo - 1))) >> lo);
    w.lo = (int32_t)(v - ((int64_t)w.hi << lo));
    return w;
}
bool to_words(long double x, int q_hi, long double limit, Word2& w, int lo = kLo) {
    int64_t v;
    if (!to_fix(x, q_hi + lo, limit, v)) return false;
    w = words(v, lo);
    return true;
}

// k = exp(x) or A times a power of T, as log2 k; `bound` receives the largest |log2 k| over the fixed-point temperature
// range. `constant`: a constant as itself (kConstRate).
bool arrhenius_fix(const Arrhenius& a, double Tmin, ArrheniusX& f, long double& bound, bool constant) {
    static const int power[] = {0, -2, -1, 4, 3, 2, 1};  // Factor
    const long double beta = a.has_x ? (long double)a.beta : (long double)power[a.factor];
    const long double e = a.has_x ? (long double)a.mEa * kLog2e : 0.0L;
    if (!a.has_x && !(a.A >= std::ldexp(1.0, -500) && a.A < std::ldexp(1.0, 500))) return false;
    if (!a.has_x && a.factor == kNone && constant) {
        f.b = f.e = {0, 0};
        std::memcpy(&f.a, &a.A, sizeof f.a);
        f.a += kConstRate;
        return true;
    }
    const long double l = a.has_x ? (long double)a.lnA * kLog2e : std::log2((long double)a.A);
    bound = std::fabs(l) + std::fabs(beta) * 13.0L + std::fabs(e) / (long double)Tmin;
    return to_words(beta, kBq, 64.0L, f.b) && to_words(e, kEq, 131000.0L, f.e) && to_fix(l, kYq, 4000.0L, f.a) &&
           bound < (long double)kMaxRate;
}

template <class T>
int32_t put(std::vector<uint8_t>& b, const T* p, size_t n) {
    while (b.size() % kAlign) b.push_back(0);
    const int32_t off = (int32_t)b.size();
    b.insert(b.end(), reinterpret_cast<const uint8_t*>(p), reinterpret_cast<const uint8_t*>(p + n));
    return off;
}

}  // namespace

FixMath make_fix_math() {
    FixMath t;
    for (int j = 0; j < kExpTable; j++) {
        const long double x = std::ldexp(std::exp2((long double)j / kExpTable), 62);
        t.exp2t[j] = (uint64_t)std::floor(x + 0.5L);
    }
    for (int j = 0; j < kLogTable; j++) {
        const long double c = 1.0L + (j + 0.5L) / kLogTable;
        t.rc[j] = (uint32_t)std::llround(4096.0L / c);
        t.log2c[j] = (int64_t)std::llround(std::ldexp(-std::log2((long double)t.rc[j] / 4096.0L), 62));
    }
    return t;
}

namespace {
bool build_rates(HostMechanism& m, double Tmin) {
    m.rates_fixed_blob.clear();
    const uint8_t* blob = m.rates_blob.data();
    RatesHeader H;
    std::memcpy(&H, blob + kMathBytes, sizeof H);
    const int K = H.K, A = H.A, R = H.R;
    if (K > 256) return false;
    auto at = [&](int32_t off, size_t i, size_t size, void* out) { std::memcpy(out, blob + off + i * size, size); };
    RatesXHeader X;
    std::memset(&X, 0, sizeof X);
    X.K = K;
    X.A = A;
    X.R = R;
    X.n_eff = H.n_eff;
    std::memcpy(X.group_end, H.group_end, sizeof X.group_end);
    X.Tmin = Tmin;
    X.l10_04 = (double)(0.4L * std::log2(10.0L));
    X.l10_075 = (double)(0.75L * std::log2(10.0L));
    if (!to_fix(std::log2((long double)H.M3), kYq, 4000.0L, X.lM3) ||
        !to_fix(std::log2((long double)H.cbrt_max), kYq, 4000.0L, X.lcbrt) ||
        !to_fix(std::log2((long double)H.C0), kYq, 4000.0L, X.lC0))
        return false;

    // Gibbs energies: g0 + g1 ln T + g2 T + g3 T^2 + g4 T^3 + g5 T^4 + g6 / T over RT, in base-2 units
    std::vector<Species> species(K);
    std::vector<SpeciesX> sx(K);
    std::vector<long double> g_bound(K, 0.0L);
    for (int k = 0; k < K; k++) {
        at(H.off_species, k, sizeof(Species), &species[k]);
        const Species& s = species[k];
        SpeciesX& f = sx[k];
        std::memset(&f, 0, sizeof f);
        f.split = s.split;
        f.need_exp = s.need_exp;
        f.need_exp_neg = s.need_exp_neg;
        if (!(s.need_exp | s.need_exp_neg)) continue;
        if (!std::isnan(s.split) && !(s.split < kFixTmid)) return false;
        for (int set = 0; set < 3; set++) {
            const double* g = s.g[std::isnan(s.split) ? 0 : set == 0 ? 0 : 1];
            const int p = set == 2 ? 13 : 11;
            long double b = std::fabs((long double)g[0]) * kLog2e + std::fabs((long double)g[1]) * 13.0L +
                            std::fabs((long double)g[6]) * kLog2e / (long double)Tmin;
            bool ok = to_fix((long double)g[0] * kLog2e, kYq, 2000.0L, f.g0[set]) &&
                      to_words((long double)g[1], kBq, 64.0L, f.g[set][0]) &&
                      to_words((long double)g[6] * kLog2e, kEq, 131000.0L, f.g[set][1]);
            for (int i = 1; i <= 4 && ok; i++) {
                const long double c = std::ldexp((long double)g[1 + i] * kLog2e, p * i);
                ok = to_words(c, kGq, 4000.0L, f.g[set][1 + i]);
                b += std::fabs(c);
            }
            if (!ok) return false;
            g_bound[k] = std::max(g_bound[k], b);
        }
    }

    // h / RT and cp / R
    std::vector<ThermoX> tx(K);
    for (int k = 0; k < K; k++) {
        const Species& s = species[k];
        ThermoX& f = tx[k];
        std::memset(&f, 0, sizeof f);
        f.split = s.split;
        f.dtE = s.dtE;
        if (!std::isnan(s.split) && !(s.split < kFixTmid)) return false;
        for (int set = 0; set < 3; set++) {
            const int piece = std::isnan(s.split) ? 0 : set == 0 ? 0 : 1, p = set == 2 ? 13 : 11;
            const double *h = s.h[piece], *cp = s.cp[piece];
            bool ok = to_fix((long double)h[0], kYq, 500.0L, f.h0[set]) &&
                      to_fix((long double)cp[0], kYq, 500.0L, f.cp0[set]) &&
                      to_words((long double)h[5], kEq, 131000.0L, f.h[set][4]);
            for (int i = 1; i <= 4 && ok; i++)
                ok = to_words(std::ldexp((long double)h[i], p * i), kGq, 500.0L, f.h[set][i - 1]) &&
                     to_words(std::ldexp((long double)cp[i], p * i), kGq, 500.0L, f.cp[set][i - 1]);
            if (!ok) return false;
        }
    }

    std::vector<Reaction> rx(R);
    std::vector<ReactionX> fx(R);
    const int third = H.group_end[1];  // models 2-5 follow
    std::vector<FalloffX> ff(R > third ? R - third : 0);
    for (int r = 0; r < R; r++) {
        at(H.off_reactions, r, sizeof(Reaction), &rx[r]);
        const Reaction& x = rx[r];
        ReactionX& f = fx[r];
        std::memset(&f, 0, sizeof f);
        f.orig = x.orig;
        int factors_r = 0, factors_p = 0;
        bool small = x.n_net >= 1 && x.n_net <= 4;
        for (int i = 0; i < x.n_r; i++) factors_r += x.r_n[i];
        for (int i = 0; i < x.n_p; i++) factors_p += x.p_n[i];
        for (int i = 0; i < x.n_net; i++) small &= std::abs((int)x.net_n[i]) <= 2;
        small &= factors_r <= 2 && (x.model == 1 || factors_p <= 2);
        const bool power = x.model <= 1 && !x.k.has_x && x.k.factor != kNone;  // A T^n
        small &= !power;
        f.shape = (uint32_t)(x.minus_sigma_net + 2) * kShapeMsn;
        if (x.model == 1 && (x.minus_sigma_net < -2 || x.minus_sigma_net > 5)) f.shape = 0;  // unused there
        if (small) {
            auto expand = [](uint8_t* out, const uint16_t* k, const int8_t* n, int count) {
                for (int i = 0, q = 0; i < count; i++)
                    for (int m = 0; m < n[i] && q < 2; m++) out[q++] = (uint8_t)k[i];
            };
            expand(f.r_k, x.r_k, x.r_n, x.n_r);
            expand(f.p_k, x.p_k, x.p_n, x.n_p);
            if (factors_r == 2) f.shape |= kShapeR2;
            if (factors_p == 2) f.shape |= kShapeP2;
            f.shape |= (uint32_t)x.n_net * kShapeNet;
            for (int i = 0; i < x.n_net; i++) {
                f.net_k[i] = (uint8_t)x.net_k[i];
                if (x.net_n[i] < 0) f.shape |= (uint32_t)kShapeNeg << i;
                if (std::abs((int)x.net_n[i]) == 2) f.shape |= (uint32_t)kShapeTwo << i;
            }
        } else {
            f.shape |= kShapeGeneral;
            for (int i = 0; i < kMaxSide; i++) {
                f.r_k[i] = (uint8_t)x.r_k[i];
                f.p_k[i] = (uint8_t)x.p_k[i];
                f.r_n[i] = i < x.n_r ? x.r_n[i] : 0;
                f.p_n[i] = i < x.n_p ? x.p_n[i] : 0;
            }
            for (int i = 0; i < kMaxNet; i++) {
                f.net_k[i] = (uint8_t)x.net_k[i];
                f.net_n[i] = i < x.n_net ? x.net_n[i] : 0;
            }
        }
        long double bound = 0.0L;
        Falloff fo;
        if (x.falloff >= 0) at(H.off_falloff, x.falloff, sizeof fo, &fo);
        const bool const_k = x.model == 4 && (fo.flags & kKinfConst);
        if (!const_k && !arrhenius_fix(x.k, Tmin, f.k, bound, true)) return false;
        if (power) {
            f.k.b = {0, x.k.factor};
            f.k.e = {0, kExactRate};
            std::memcpy(&f.k.a, &x.k.A, sizeof f.k.a);
        }
        if (x.model != 1) {  // the equilibrium constant's logarithm stays in range
            long double b = 2.0L * (30.0L + 13.0L);
            for (int i = 0; i < x.n_net; i++) b += std::abs((int)x.net_n[i]) * g_bound[x.net_k[i]];
            if (!(b < 4000.0L)) return false;
        }
        if (r >= third) {
            FalloffX& g = ff[r - third];
            std::memset(&g, 0, sizeof g);
            if (x.falloff >= 0) {
                // (of a Troe reaction when k_inf is a constant too: otherwise their logarithms are added)
                if (!arrhenius_fix(fo.k0, Tmin, g.k0, bound, x.model != 4 || const_k)) return false;
                g.ainf = fo.ainf;
                if (x.model == 4 && (!(fo.ainf > 0.) || !to_fix(std::log2((long double)fo.ainf), kYq, 1000.0L, g.lainf)))
                    return false;
                g.c1mA = fo.c1mA;
                g.cA = fo.cA;
                g.c3 = (double)((long double)fo.c3 * kLog2e);
                g.c1 = (double)((long double)fo.c1 * kLog2e);
                g.cmT2 = (double)((long double)fo.cmT2 * kLog2e);
                g.l2_fcent = (double)((long double)fo.ln_fcent * kLog2e);
                g.flags = fo.flags;
                g.sri_flags = fo.sri_flags;
                g.sA = fo.sA;
                g.smB = (double)((long double)fo.smB * kLog2e);
                g.smrC = (double)((long double)fo.smrC * kLog2e);
                g.sD = fo.sD;
                g.sE = fo.sE;
            }
        }
    }

    // third-body efficiencies minus one, rows padded to a multiple of 4 like the FP64 table's, a unit for every four
    const size_t n_e = (size_t)(H.n_eff + 3) / 4 * 4 * K;
    std::vector<double> eff(n_e);
    if (n_e) std::memcpy(eff.data(), blob + H.off_eff, n_e * sizeof(double));
    std::vector<Word2> ef(n_e);
    std::vector<int32_t> eq(n_e / K / 4);
    for (size_t g = 0; g < eq.size(); g++) {
        const double* e = &eff[4 * g * K];
        long double largest = 0.0L, sum = 0.0L;
        for (int row = 0; row < 4; row++) {
            long double s = 0.0L;
            for (int k = 0; k < K; k++) {
                largest = std::max(largest, std::fabs((long double)e[row * K + k]));
                s += std::fabs((long double)e[row * K + k]);
            }
            sum = std::max(sum, s);
        }
        if (!(largest < (long double)kMaxEff)) return false;
        int q = 29;
        while (std::ldexp(largest, q) > 2147483646.0L || std::ldexp(sum, q) + K > std::ldexp(1.0L, 33)) q--;
        for (int i = 0; i < 4 * K; i++)
            ef[4 * g * K + i] = words((int64_t)std::llround(std::ldexp((long double)e[i], q + kThirdLo)), kThirdLo);
        eq[g] = q;
    }

    std::vector<uint8_t>& b = m.rates_fixed_blob;
    b.insert(b.end(), blob, blob + kMathBytes);  // the FP64 functions' tables, then the fixed-point ones
    const FixMath fm = make_fix_math();
    put(b, &fm, 1);
    const int32_t off_header = put(b, &X, 1);
    if (off_header != kMathBytes + kFixMathBytes) return false;
    X.off_species = put(b, sx.data(), sx.size());
    X.off_thermo = put(b, tx.data(), tx.size());
    X.off_reactions = put(b, fx.data(), fx.size());
    X.off_falloff = put(b, ff.data(), ff.size());
    X.off_eff = put(b, ef.data(), ef.size());
    X.off_eff_q = put(b, eq.data(), eq.size());
    std::vector<int32_t> start(K + 1, 0), lists;
    for (int k = 0; k < K; k++) {
        for (int r = 0; r < R; r++)
            for (int i = 0; i < rx[r].n_net; i++)
                if (rx[r].net_k[i] == k) lists.push_back((r << 8) | (rx[r].net_n[i] & 0xff));
        start[k + 1] = (int32_t)lists.size();
    }
    X.off_csr_start = put(b, start.data(), start.size());
    X.off_csr = put(b, lists.data(), lists.size());
    while (b.size() % kAlign) b.push_back(0);
    X.total_bytes = (int32_t)b.size();
    std::memcpy(b.data() + off_header, &X, sizeof X);
    return true;
}
}  // namespace

bool build_rates_fixed(HostMechanism& m) {
    for (double Tmin : kFixTmin)
        if (build_rates(m, Tmin)) return true;
    return false;
}

namespace {

// A polynomial over the fixed-point temperature range: positive, within a factor of 2^5, coefficients that fit.
bool poly_fix(const double* P, double Tn_lo, double Tn_hi, int pw, long double scale, PolyX& f) {
    long double lo = 1e300L, hi = 0.0L;
    const long double a = std::log((long double)Tn_lo), b = std::log((long double)Tn_hi);
    for (int i = 0; i <= 256; i++) {
        const long double L = a + (b - a) * i / 256.0L;
        const long double D = scale * (P[0] + L * (P[1] + L * (P[2] + L * (P[3] + L * (long double)P[4]))));
        lo = std::min(lo, D);
        hi = std::max(hi, D);
    }
    if (!(lo > 1e-290L) || !(hi < 1e290L)) return false;
    int e;
    std::frexp((double)(hi * 1.0001L), &e);  // hi < 2^e
    if (!(lo > std::ldexp(1.0L, e - 5))) return false;
    f.sp = e;
    f.rcp_bias = 1022 + 63 - 56 - e;
    if (!to_fix(std::ldexp((long double)P[0] * scale, -e), kDq, 4.0L, f.p0)) return false;
    for (int m = 1; m <= 4; m++)
        if (!to_words(std::ldexp((long double)P[m] * scale, pw * m - e), kPpq, 4.0L, f.p[m - 1], kPlo)) return false;
    return true;
}

// Bits of 2^pw above |ln(T/T0)|.
int log_power(double Tn_lo, double Tn_hi) {
    const double Lmax = std::max(std::fabs(std::log(Tn_lo)), std::fabs(std::log(Tn_hi)));
    int pw = 0;
    while (std::ldexp(1.0, pw) <= Lmax) pw++;
    return pw;
}

bool build_transport(HostMechanism& m, double Tmin, double Tmax) {
    m.transport_fixed_blob.clear();
    const uint8_t* blob = m.transport_blob.data();
    TransportHeader H;
    std::memcpy(&H, blob + kMathBytes, sizeof H);
    const int K = H.K;
    if (K > 256) return false;
    auto doubles = [&](int32_t off, size_t n) {
        std::vector<double> v(n);
        std::memcpy(v.data(), blob + off, n * sizeof(double));
        return v;
    };
    const std::vector<double> cond = doubles(H.off_cond, (size_t)K * 5), visc = doubles(H.off_visc, (size_t)K * 5);
    const std::vector<double> W = doubles(H.off_W, K), diff = doubles(H.off_diff, (size_t)H.n_pairs * 5);
    const std::vector<double> A2 = doubles(H.off_A2, (size_t)K * K), AB = doubles(H.off_AB, (size_t)K * K);
    const std::vector<double> B2 = doubles(H.off_B2, (size_t)K * K);
    TransportXHeader X;
    std::memset(&X, 0, sizeof X);
    X.K = K;
    X.n_pairs = H.n_pairs;
    X.T0 = H.T0;
    X.Tn_lo = Tmin / H.T0;
    X.Tn_hi = Tmax / H.T0;
    X.pw = log_power(X.Tn_lo, X.Tn_hi);
    const double* narrowest = std::end(kFixTransportT)[-1];
    if (X.pw > 4 || X.pw != log_power(narrowest[0] / H.T0, narrowest[1] / H.T0)) return false;
    std::vector<PolyX> pc(K), pv(K), pd(std::max(H.n_pairs, 1));
    std::memset(pc.data(), 0, pc.size() * sizeof(PolyX));
    std::memset(pv.data(), 0, pv.size() * sizeof(PolyX));
    std::memset(pd.data(), 0, pd.size() * sizeof(PolyX));
    std::vector<double> W4(K);
    std::vector<long double> w4(K);  // W^(1/4)
    for (int k = 0; k < K; k++) {
        w4[k] = std::sqrt(std::sqrt((long double)m.W[k]));
        W4[k] = (double)std::sqrt((long double)m.W[k]);
        if (!poly_fix(&cond[(size_t)k * 5], X.Tn_lo, X.Tn_hi, X.pw, 1.0, pc[k])) return false;
        if (!poly_fix(&visc[(size_t)k * 5], X.Tn_lo, X.Tn_hi, X.pw, 1.0L / w4[k], pv[k])) return false;
    }
    for (int p = 0; p < H.n_pairs; p++)
        if (!poly_fix(&diff[(size_t)p * 5], X.Tn_lo, X.Tn_hi, X.pw, 1.0, pd[p])) return false;
    // b_kj = a_kj (W_j / W_k)^(1/4) to FP64 rounding (a constant that the reference's builder folds to 0 or 1 is
    // not); |a^2| to the words' position
    double largest = 0.;
    for (int k = 0; k < K; k++)
        for (int j = 0; j < K; j++) {
            const size_t i = (size_t)k * K + j;
            const long double r = w4[j] / w4[k], a2 = A2[i];
            if (!(A2[i] > 0.) || std::fabs(AB[i] / (2.0L * a2 * r) - 1.0L) > 2e-15L || std::fabs(B2[i] / (a2 * r * r) - 1.0L) > 2e-15L)
                return false;
            largest = std::max(largest, A2[i]);
        }
    const bool wide = kmax_for(K, m.n_eff) > 64;  // the kernels' words go by their capacity
    const int bits = wide ? kMixAq<256> : kMixAq<64>, low = wide ? kMixLo<256> : kMixLo<64>;
    const int sum_bits = 2 * low - (wide ? kMixXq<256> : kMixXq<64>);  // high words' products: a row of a^2 over 2^this
    double row = 0.;
    for (int k = 0; k < K; k++) {
        double sum = 0.;
        for (int j = 0; j < K; j++) sum += A2[(size_t)k * K + j];
        row = std::max(row, sum);
    }
    X.a_shift = bits;
    while (std::ldexp(largest, X.a_shift) >= std::ldexp(1.0, bits)) X.a_shift--;
    while (std::ldexp(largest, X.a_shift + 1) < std::ldexp(1.0, bits)) X.a_shift++;
    while (std::ldexp(row, X.a_shift - sum_bits) >= 0.95 * std::ldexp(1.0, 62)) X.a_shift--;  // (the sums are doubled)
    std::vector<Word2> a2((size_t)K * K);
    for (int k = 0; k < K; k++)
        for (int j = 0; j < K; j++)
            a2[(size_t)j * K + k] =
                words((int64_t)std::llround(std::ldexp((long double)A2[(size_t)k * K + j], X.a_shift)), low);

    std::vector<uint8_t>& b = m.transport_fixed_blob;
    b.insert(b.end(), blob, blob + kMathBytes);
    const int32_t off_header = put(b, &X, 1);
    if (off_header != kMathBytes) return false;
    X.off_cond = put(b, pc.data(), pc.size());
    X.off_visc = put(b, pv.data(), pv.size());
    X.off_W = put(b, W.data(), W.size());
    X.off_W4 = put(b, W4.data(), W4.size());
    X.off_diff = put(b, pd.data(), pd.size());
    X.off_A2 = put(b, a2.data(), a2.size());
    while (b.size() % kAlign) b.push_back(0);
    X.total_bytes = (int32_t)b.size();
    std::memcpy(b.data() + off_header, &X, sizeof X);
    return true;
}
}  // namespace

bool build_transport_fixed(HostMechanism& m) {
    for (const double* T : kFixTransportT)
        if (build_transport(m, T[0], T[1])) return true;
    return false;
}

}  // namespace cbg
