// Per-reaction evaluation of the evaluation kernels (pjg_wave.cuh, pjg_tile.cu).
//
// rxn_terms() evaluates one reaction at one state: forward rate constant
// (get_simple_arrhenius_rates :2642, PLOG :2084, Chebyshev :1904 of
// pyjac/core/rate_subs.py), reverse rate through the equilibrium constant
// (:1627), mass-action rates of progress (:1170-1509), third-body and
// fall-off pressure modification (:1510-1626, :1788-2641), and, when DER is
// set, the reaction's analytical derivative terms (create_jacobian.py
// dRopi_dnj :4169-4522, dci_*_dnj :3558-4168, dRopidT :2589-3108,
// dRopidE :1458-1594, dci_*_dT :2117-2588, dci_*_dE :362-880).
//
// The caller owns the accumulation: species rates get nu_k * net, species row
// k of the Jacobian gets nu_k * (g_j ci) in column j, nu_k * d0 (times V / T) in
// column T, nu_k * (d1 - net) (constant pressure; else nu_k * d1) in column E,
// nu_k * coef_l * X in the columns of the third-body list, and
// nu_k * (gns ci + cns X) in every species column (the bath-gas terms, gathered
// per row).
//
// The temperature derivative of a reaction's Gibbs sum needs no array of its
// own: d b_k / dT = (h_k / (R T) - 1) / T, so sum nu_k d b_k / dT follows from
// the reaction's enthalpy dH = sum nu_k h_k (at constant volume, with energies,
// the -1 drops out), which is also its weight in row T of the Jacobian.
//
// Per-state arrays are read through an accessor with operator[] (a strided
// view of global memory, or a shared-memory pointer).
#pragma once
#include "pjg_math.cuh"
#include "pjg_tables.cuh"

namespace pjg {

// nu * x for a warp-uniform small integer nu without an int->double conversion
// -x by flipping the sign bit on the integer pipe: a value that only feeds a
// reduction cannot fold the negation into an FP64 instruction
__device__ __forceinline__ double negi(double x)
{
    return __hiloint2double(__double2hiint(x) ^ 0x80000000, __double2loint(x));
}

__device__ __forceinline__ double nux(int nu, double x)
{
    switch (nu) {
    case 1: return x;
    case -1: return negi(x);
    case 2: return x + x;
    case -2: return negi(x + x);
    case 0: return 0.0;
    }
    return (double)nu * x;
}

// acc + nu * x
__device__ __forceinline__ double addnu(double acc, int nu, double x)
{
    switch (nu) {
    case 1: return acc + x;
    case -1: return acc - x;
    case 2: return fma(2.0, x, acc);
    case -2: return fma(-2.0, x, acc);
    case 0: return acc;
    }
    return fma((double)nu, x, acc);
}

// scalars of one thermochemical state used by every reaction
struct StateVars {
    double T;       // temperature (unclamped: explicit factors of the Jacobian)
    double Tc;      // T clamped to [100, 10000] K (rate evaluation)
    double logT, Tinv;  // of Tc
    double ls, tis;     // the same in units of the exponential's table step
    double Tjinv;   // 1 / T
    double V, P;
    double PoRT;    // P / (R T)
    double rt_inv;  // 1 / (R T)
    double kB, kC;  // T sum nu d b / dT = dH kB - (sum nu) kC
    double h_ns;    // enthalpy (energy) of the bath gas
    double logP;    // ln P (PLOG / Chebyshev mechanisms only)
    bool conp;
    // every |b_k| <= EvalArgs::kc_split_max = 690 / (the mechanism's largest
    // sum |nu| of a reversible reaction) and the bath gas's concentration is
    // not negative: 1 / Kc is the product of the participants' exp(+-b_k) (no
    // partial product past e^690, so the reference's clamp of sum nu b at
    // 690.78 never acts); else exp(-sum nu b) per reaction from b_k
    bool split;
    const double* etab;  // fexp table (shared memory)
};

// the values derived from T, Tc, Tinv and conp; ls is log2(Tc) times a power of
// two and tis one quotient, so that neither is rounded twice
template <bool DER>
__device__ __forceinline__ void set_scaled(StateVars& sv, double lg2T, double tis)
{
    sv.ls = __dmul_rn(lg2T, (double)PJG_EXP_TAB);
    sv.tis = tis;
    sv.kC = sv.conp ? __dmul_rn(sv.T, sv.Tinv) : 0.0;
    sv.kB = DER ? __dmul_rn(__dmul_rn(__dmul_rn(sv.T, sv.Tinv), sv.Tinv), 1.0 / RU) : 0.0;
}

// decoded reaction header
struct RxnHead {
    int flags, nsp, thd_off, thd_cnt, auxo, list, bint, fbint;
    unsigned ent[PJG_MAXSP];
    const double* p;
};

__device__ __forceinline__ void load_head(const RxnRec* R, RxnHead& h)
{
    const int4 h0 = __ldg(reinterpret_cast<const int4*>(R));
    const int4 h1 = __ldg(reinterpret_cast<const int4*>(R) + 1);
    h.flags = h0.x;
    h.nsp = h0.y;
    h.thd_off = h0.z;
    h.thd_cnt = h0.w;
    h.auxo = h1.x;
    h.list = h1.y;
    h.bint = h1.z;
    h.fbint = h1.w;
    const uint4 e0 = __ldg(reinterpret_cast<const uint4*>(R) + 2);
    const uint4 e1 = __ldg(reinterpret_cast<const uint4*>(R) + 3);
    h.ent[0] = e0.x; h.ent[1] = e0.y; h.ent[2] = e0.z; h.ent[3] = e0.w;
    h.ent[4] = e1.x; h.ent[5] = e1.y; h.ent[6] = e1.z; h.ent[7] = e1.w;
    h.p = R->p;
}

struct RxnTerms {
    double net;              // pressure-modified net rate of progress
    double w;                // sum nu_k hw_k, the weight in row T
    double g[PJG_MAXSP];     // d (rf - rr) / d c_j for participant j
    double gns;              // the same for the bath gas (0 if absent)
    double ci_;              // pressure modification (1 without third body)
    // temperature column (times V / T) and extra-variable column terms; at
    // constant pressure the latter without -net, which sums to -wdot over a
    // row's reactions
    double d0, d1;
    double X;                // third-body column factor, Rnet d ci / d [M]
};

// the weight in row T from the reaction's enthalpy: sum over the species rows
// of nu_k (h_k - h_ns W_k / W_ns), which is sum nu_k h_k where mass is conserved
__device__ __forceinline__ double row_t_weight(int flags, const double* p, double dH, int nu_sum, double h_ns)
{
    return (flags & RX_WEREAL) ? fma(-h_ns, (double)nu_sum - ldg(p + P_WE), dH) : dH;
}

// T sum nu_k d b_k / dT
__device__ __forceinline__ double gibbs_slope(const StateVars& sv, double dH, int nu_sum)
{
    const double x = __dmul_rn(dH, sv.kB);
    return nu_sum ? addnu(x, -nu_sum, sv.kC) : x;
}

// mulpow with rounded products: the rates of progress must not depend on
// how the compiler contracts them into later FMAs, which differs between the
// kernel kinds (the Jacobian kernel's rates equal the rates kernel's bit for
// bit)
__device__ __forceinline__ double mulpow_rn(double acc, double v, int p)
{
    if (p == 0) return acc;
    if (p == 1) return __dmul_rn(acc, v);
    if (p == 2) return __dmul_rn(acc, __dmul_rn(v, v));
    return __dmul_rn(acc, powi(v, p));
}

// Stoichiometry of a reaction as rxn_terms() reads it: from the record
// (RunStoich) or fixed at compile time by a coefficient pattern
// (PatStoich<MaPattern<...>>, the record's entries stored in the pattern's
// order).
struct RunStoich {
    __device__ static int nsp(const RxnHead& h) { return h.nsp; }
    __device__ static int nuf(const RxnHead& h, int e) { return ent_nuf(h.ent[e]); }
    __device__ static int nur(const RxnHead& h, int e) { return ent_nur(h.ent[e]); }
};
template <class PT>
struct PatStoich {
    __device__ static constexpr int nsp(const RxnHead&) { return PT::n; }
    __device__ static constexpr int nuf(const RxnHead&, int e) { return PT::nuf(e); }
    __device__ static constexpr int nur(const RxnHead&, int e) { return PT::nur(e); }
};

// exp(-sum nu b) as the product of the participants' per-species factors
// exp(b_k)^-nu (nu < 0) and exp(-b_k)^nu (nu > 0), where StateVars::split
// holds (no partial product then passes e^690).
template <class ST, class ARR>
__device__ __forceinline__ double inv_kc_split(const RxnHead& h, const ARR& ep, const ARR& em)
{
    double r = 1.0;
    bool first = true;
#pragma unroll
    for (int e = 0; e < PJG_MAXSP; ++e) {
        if (e >= ST::nsp(h)) break;
        const int nu = ST::nur(h, e) - ST::nuf(h, e);
        if (nu == 0) continue;
        const int k = ent_spec(h.ent[e]);
        const double f = nu < 0 ? ep[k] : em[k];
        const int na = nu < 0 ? -nu : nu;
        const double fn = na == 1 ? f : (na == 2 ? __dmul_rn(f, f) : powi(f, na));
        r = first ? fn : __dmul_rn(r, fn);
        first = false;
    }
    return r;
}

// [M] and log10 [M] of the third-body lists that several reactions share
// (pjg_capi.cu numbers them): from the tile's arrays, formed once per state, ...
template <class ARR>
struct MLists {
    ARR m;
    int n;
    template <class FORM>
    __device__ __forceinline__ double conc(int l, FORM&&)
    {
        return m[l];
    }
    __device__ __forceinline__ double log10(int l, double) { return m[n + l]; }
};
// ... or kept from the last reaction (the packing lets them follow one another)
struct MLast {
    int list = -1, list_log = -1;
    double M = 0.0, lgM = 0.0;
    template <class FORM>
    __device__ __forceinline__ double conc(int l, FORM&& form)
    {
        if (l != list) {
            M = form();
            list = l;
        }
        return M;
    }
    __device__ __forceinline__ double log10(int l, double m)
    {
        if (l != list_log) {
            lgM = __dmul_rn(log(m), INV_LN10);
            list_log = l;
        }
        return lgM;
    }
};

struct FallState {
    double Pr, Fi, A, B, Fc, lnFc, X, lnQ, kratio, logPr;
    double inv1, ci0, rabs;  // 1 / (1 + Pr), Fi / (1 + Pr), Troe 1 / (A^2 + B^2)
    double e1, e2, e3;  // Troe exponentials at the clamped temperature
};

template <bool DER, class ST = RunStoich, class ARR, class ML>
__device__ __forceinline__ void rxn_terms(const RxnHead& h, const double* aux,
                                          const int* thd_spec, const double* thd_coef, int last,
                                          const StateVars& sv, const ARR& conc, const ARR& bk,
                                          const ARR& ep, const ARR& em, const ARR& hk,
                                          ML& ml, RxnTerms& o)
{
    const int flags = h.flags, nsp = ST::nsp(h);
    const double* p = h.p;
    const int form = RX_FORM(flags);
    const bool rev = flags & RX_REV;
    const double Tc = sv.Tc, Tjinv = sv.Tjinv;
    const double* et = sv.etab;

    // forward rate constant and its log-derivatives (dl: T d ln kf / dT)
    double kf, dl = 0.0, dlnkf_dlnP = 0.0;
    if (form <= FORM_ARR) {
        kf = arrhenius(form, ldg(p + P_A), h.bint, ldg(p + P_B), ldg(p + P_TA), Tc, sv.Tinv, sv.ls, sv.tis,
                       et);
        if (DER) dl = fma(ldg(p + P_TA), Tjinv, ldg(p + P_B));
    } else if (form == FORM_PLOG) {
        kf = gexp(plog_logk(aux + h.auxo, sv.logT, sv.Tinv, sv.logP, Tjinv, &dl, &dlnkf_dlnP), et);
        dl *= sv.T;
    } else {
        const double l10 = cheb_log10k(aux + h.auxo, sv.Tinv, sv.logP, Tjinv, &dl, &dlnkf_dlnP);
        kf = fexp(LN10 * min_pos(EXP_MAX, l10), et);
        dl *= LN10 * sv.T;
        dlnkf_dlnP *= LN10;
    }
    // reaction enthalpy; reverse rate: kr = kf / Kc, Kc = (P_atm/R)^nu_sum exp(sum nu b)
    int nu_sum = 0;
    double dH = 0.0;
    if (DER) {
#pragma unroll
        for (int e = 0; e < PJG_MAXSP; ++e) {
            if (e >= nsp) break;
            const int nu = ST::nur(h, e) - ST::nuf(h, e);
            if (nu == 0) continue;
            nu_sum += nu;
            dH = addnu(dH, nu, hk[ent_spec(h.ent[e])]);
        }
        o.w = row_t_weight(flags, p, dH, nu_sum, sv.h_ns);
    }
    double kr = 0.0;
    if (rev) {
        double ikc;
        if (sv.split) {
            ikc = inv_kc_split<ST>(h, ep, em);
        } else {
            double Bsum = 0.0;
#pragma unroll
            for (int e = 0; e < PJG_MAXSP; ++e) {
                if (e >= nsp) break;
                const int nu = ST::nur(h, e) - ST::nuf(h, e);
                if (nu != 0) Bsum = addnu(Bsum, nu, bk[ent_spec(h.ent[e])]);
            }
            ikc = fexp(-min_pos(EXP_MAX, Bsum), et);
        }
        kr = __dmul_rn(__dmul_rn(kf, ldg(p + P_PSUM)), ikc);
    }
    // rates of progress (mass action on raw concentrations)
    double rf = kf, rr = kr;
#pragma unroll
    for (int e = 0; e < PJG_MAXSP; ++e) {
        if (e >= nsp) break;
        const double c = conc[ent_spec(h.ent[e])];
        rf = mulpow_rn(rf, c, ST::nuf(h, e));
        if (rev) rr = mulpow_rn(rr, c, ST::nur(h, e));
    }
    // third-body / fall-off pressure modification
    const int thd = RX_THD(flags);
    const int blend = RX_BLEND(flags);
    const bool chem = flags & RX_CHEM;
    double ci = 1.0, M = 0.0;
    FallState fs;
    fs.Pr = 0.0; fs.Fi = 1.0; fs.A = 0.0; fs.B = 0.0; fs.Fc = 1.0; fs.lnFc = 0.0; fs.X = 0.0;
    fs.lnQ = 0.0; fs.kratio = 0.0; fs.e1 = 0.0; fs.e2 = 0.0; fs.e3 = 0.0; fs.logPr = 0.0;
    fs.inv1 = 0.0; fs.ci0 = 0.0; fs.rabs = 0.0;
    if (thd) {
        auto form_m = [&]() -> double {
            double m = sv.PoRT * ldg(p + P_FLAG);
            for (int l = 0; l < h.thd_cnt; ++l)
                m = fma(__ldg(thd_coef + h.thd_off + l), conc[__ldg(thd_spec + h.thd_off + l)], m);
            return m;
        };
        M = h.list >= 0 ? ml.conc(h.list, form_m) : form_m();
        if (blend == BL_NONE) {
            ci = M;
        } else {
            // k0 / kinf, in one exponential where both are, and its logarithm
            double lnr = 0.0;
            bool has_lnr = flags & RX_RATIO;
            if (has_lnr) {
                lnr = fma(-ldg(p + P_RTA), sv.tis, fma(ldg(p + P_RB), sv.ls, ldg(p + P_RA)));
                fs.kratio = fexp_s(lnr, h.fbint, et);
                lnr = __dadd_rn(lnr, ldg(p + P_RN));
            } else {
                const double kfall = arrhenius(RX_FFORM(flags), ldg(p + P_FA), h.fbint, ldg(p + P_FB),
                                               ldg(p + P_FTA), Tc, sv.Tinv, sv.ls, sv.tis, et);
                fs.kratio = chem ? kf / kfall : kfall / kf;
            }
            fs.Pr = __dmul_rn(M, fs.kratio);
            fs.inv1 = 1.0 / __dadd_rn(1.0, fs.Pr);
            // log10 Pr from the logarithms where k0 / kinf is one exponential and
            // Pr >= 1e-300; else the logarithm of the guarded Pr
            if (blend == BL_TROE || blend == BL_SRI) {
                if (has_lnr && __double_as_longlong(fs.Pr) >= __double_as_longlong(SMALL)) {
                    const double lgM = h.list >= 0 ? ml.log10(h.list, M) : __dmul_rn(log(M), INV_LN10);
                    fs.logPr = fma(lnr, kExpStep * INV_LN10, lgM);
                } else {
                    fs.logPr = __dmul_rn(log(gsmall(fs.Pr)), INV_LN10);
                }
            }
            if (blend == BL_TROE) {
                const double logPr = fs.logPr;
                const double ta = ldg(p + P_F0), tcs = -(Tc * kExpScale);
                fs.e1 = fexp_s(__dmul_rn(tcs, ldg(p + P_F1)), 0, et);
                fs.e3 = fexp_s(__dmul_rn(tcs, ldg(p + P_F3)), 0, et);
                double Fc = fma(ta, fs.e1, __dmul_rn(1.0 - ta, fs.e3));
                if (flags & RX_T2) {
                    fs.e2 = fexp_s(__dmul_rn(-ldg(p + P_F2), sv.tis), 0, et);
                    Fc = __dadd_rn(Fc, fs.e2);
                }
                fs.lnFc = log(gsmall(Fc));
                const double logFc = __dmul_rn(fs.lnFc, INV_LN10);
                fs.B = fma(-1.1762, logFc, fma(-0.14, logPr, 0.806));
                fs.A = fma(-0.67, logFc, __dsub_rn(logPr, 0.4));
                fs.Fc = Fc;
                const double B2 = __dmul_rn(fs.B, fs.B);
                fs.rabs = 1.0 / fma(fs.A, fs.A, B2);
                fs.Fi = fexp_s(__dmul_rn(__dmul_rn(B2, fs.rabs), __dmul_rn(fs.lnFc, kExpScale)), 0, et);
            } else if (blend == BL_SRI) {
                const double logPr = fs.logPr;
                fs.X = 1.0 / fma(logPr, logPr, 1.0);
                fs.e1 = fexp_s(__dmul_rn(-ldg(p + P_F1), sv.tis), 0, et);
                fs.e3 = gexp(-Tc / ldg(p + P_F2), et);
                const double Q = fma(ldg(p + P_F0), fs.e1, fs.e3);
                fs.lnQ = log(Q);
                double Fi = fexp(__dmul_rn(fs.X, fs.lnQ), et);
                if (flags & RX_SRID) Fi = __dmul_rn(Fi, ldg(p + P_F3));
                if (flags & RX_SRIE) {
                    const double e = ldg(p + P_F4);
                    const int ie = (int)e;
                    Fi = __dmul_rn(Fi, (flags & RX_SRIEINT) ? (ie < 0 ? powi(sv.Tinv, -ie) : powi(Tc, ie))
                                                            : pow(Tc, e));
                }
                fs.Fi = Fi;
            }
            fs.ci0 = __dmul_rn(fs.Fi, fs.inv1);
            ci = chem ? fs.ci0 : __dmul_rn(fs.ci0, fs.Pr);
        }
    }
    double Rnet = rf;
    if (rev) Rnet = __dsub_rn(Rnet, rr);
    o.net = thd ? __dmul_rn(Rnet, ci) : Rnet;
    if (!DER) return;

    const double T = sv.T, V = sv.V, P = sv.P, PoRT = sv.PoRT, rt_inv = sv.rt_inv;
    const bool conp = sv.conp;
    const double kr_ = rev ? kr : 0.0;
    double cg[PJG_MAXSP];
#pragma unroll
    for (int e = 0; e < PJG_MAXSP; ++e) cg[e] = e < nsp ? gsmall(conc[ent_spec(h.ent[e])]) : 1.0;
    // d R / d c_j for every participant j (dRopidnj :4169-4522)
    double gns = 0.0;
#pragma unroll
    for (int j = 0; j < PJG_MAXSP; ++j) {
        if (j >= nsp) break;
        const int nfj = ST::nuf(h, j), nrj = ST::nur(h, j);
        double gf = 0.0, gr = 0.0;
        if (nfj) {
            double S = nux(nfj, kf);
#pragma unroll
            for (int e = 0; e < PJG_MAXSP; ++e) {
                if (e >= nsp) break;
                S = mulpow(S, cg[e], ST::nuf(h, e) - (e == j));
            }
            gf = S;
        }
        if (rev && nrj) {
            double S = nux(nrj, kr_);
#pragma unroll
            for (int e = 0; e < PJG_MAXSP; ++e) {
                if (e >= nsp) break;
                S = mulpow(S, cg[e], ST::nur(h, e) - (e == j));
            }
            gr = S;
        }
        o.g[j] = gf - gr;
        if (ent_spec(h.ent[j]) == last) gns = o.g[j];
    }
    o.gns = gns;
    const double ci_ = thd ? ci : 1.0;
    o.ci_ = ci_;
    // Fall-off derivative shared by the n, T and E columns: d ci / dx given
    // d Pr / dx and the direct part of d ln Fi / dx.  With dlnF = d ln Fi / d ln Pr
    // and ci = Fi Pr / (1 + Pr), d ci = Fi / (1 + Pr) (d Pr (1 / (1 + Pr) + dlnF)
    // + Pr direct); chemically activated, ci = Fi / (1 + Pr).
    double dlnF = 0.0;
    const bool fall = thd && blend != BL_NONE;
    if (blend == BL_TROE)
        dlnF = -2.0 * fs.A * fs.B * fs.lnFc * fma(0.14, fs.A, fs.B) * INV_LN10 * (fs.rabs * fs.rabs);
    else if (blend == BL_SRI)
        dlnF = -2.0 * INV_LN10 * fs.X * fs.X * fs.logPr * fs.lnQ;
    const double slope = chem ? dlnF / gsmall(fs.Pr) - fs.inv1 : dlnF + fs.inv1;
    auto dci = [&](double dPr, double direct) -> double {
        return fs.ci0 * fma(dPr, slope, chem ? direct : fs.Pr * direct);
    };
    const double dMfac = fall ? fs.ci0 * (fs.kratio * slope) : 1.0;
    o.X = Rnet * dMfac;
    const double mod = ldg(p + P_MOD);
    const bool hasns = flags & RX_HASNS;
    // temperature column times T / V (dRopi_dT :2589-3108, dci_*_dT :2117-2588):
    // rf dl - rr (dl - T dB) = Rnet dl + rr T dB
    double d0 = rev ? fma(rr, gibbs_slope(sv, dH, nu_sum), Rnet * dl) : rf * dl;
    d0 = d0 * ci_;
    if (hasns) d0 = fma(-gns * ci_, PoRT, d0);
    // extra-variable column (dRopi_dE :1458-1594, dci_*_dE :362-880)
    double d1 = 0.0;
    if (conp) {
        int nuf = -2, nur = -2;
#pragma unroll
        for (int e = 0; e < PJG_MAXSP; ++e) {
            if (e >= nsp) break;
            nuf += ST::nuf(h, e);
            nur += ST::nur(h, e);
        }
        d1 = (-nux(nuf, rf) + (rev ? nux(nur, rr) : 0.0)) * ci_;
    } else if (form >= FORM_PLOG) {
        d1 = V * ci_ * Rnet * dlnkf_dlnP / P;
    }
    if (hasns) d1 = fma(__dmul_rn(gns, ci_), conp ? PoRT : __dmul_rn(V, rt_inv), d1);
    if (thd) {
        const double dM = -PoRT * mod;  // T d [M] / dT
        if (blend == BL_NONE) {
            d0 = fma(dM, Rnet, d0);
            if (conp) {
                if (thd != THD_UNITY) d1 = fma(fma(mod, PoRT, -M), Rnet, d1);
            } else {
                d1 = fma(__dmul_rn(V, Rnet), __dmul_rn(mod, rt_inv), d1);
            }
        } else {
            double Rb, RTa;
            if (flags & RX_RATIO) {
                Rb = ldg(p + P_RB);
                RTa = ldg(p + P_RTA);
            } else {
                Rb = ldg(p + P_FB) - ldg(p + P_B);
                RTa = ldg(p + P_FTA) - ldg(p + P_TA);
                if (chem) {
                    Rb = -Rb;
                    RTa = -RTa;
                }
            }
            const double theta = fma(RTa, Tjinv, Rb);  // T d ln (k0 / kinf) / dT
            double direct = 0.0;  // T times the explicit part
            if (blend == BL_TROE) {
                const double absq = fma(fs.A, fs.A, fs.B * fs.B);
                const double ta = ldg(p + P_F0), t1 = ldg(p + P_F1), t2 = ldg(p + P_F2),
                             t3 = ldg(p + P_F3);
                // the explicit T derivative uses the unclamped T, as the reference
                const bool same = T == Tc;
                const double x1 = same ? fs.e1 : gexp(-1.0 * T * t1, et);
                const double x3 = same ? fs.e3 : gexp(-1.0 * T * t3, et);
                double dFc = T * ((ta - 1.0) * t3 * x3 - ta * t1 * x1);
                if (flags & RX_T2) dFc = fma(t2 * Tjinv, same ? fs.e2 : gexp(-1.0 * t2 * Tjinv, et), dFc);
                direct = -fs.B * dFc *
                         (2.0 * fs.A * (1.1762 * fs.A + -0.67 * fs.B) * fs.lnFc - fs.B * absq * LN10) *
                         (fs.rabs * fs.rabs * INV_LN10) / fs.Fc;
            } else if (blend == BL_SRI) {
                const double sa = ldg(p + P_F0), sb = ldg(p + P_F1), sc = ldg(p + P_F2);
                const double Q = fma(sa, fs.e1, fs.e3);
                const double dQ = sa * sb * Tjinv * fs.e1 - T * fs.e3 / sc;
                direct = fs.X * dQ / Q + ldg(p + P_F4);
            }
            d0 = fma(dci(fma(fs.Pr, theta, dM * fs.kratio), direct), Rnet, d0);
            const double modp = (conp ? (thd == THD_UNITY ? 0.0 : mod) * PoRT : mod * rt_inv) * fs.kratio;
            const double dPr = conp && thd != THD_UNITY ? modp - fs.Pr : modp;
            d1 = fma(dci(dPr, 0.0) * (conp ? 1.0 : V), Rnet, d1);
        }
    }
    o.d0 = d0;
    o.d1 = d1;
}

// ------------------------------------------------------------------------
// Reactions A + B <=> C + D (is_e22 in pjg_capi.cu: four distinct species
// with unit coefficients, reversible, Arrhenius form, no third body,
// nu_sum = 0), entries stored reactants first.  The same arithmetic as
// rxn_terms() for this case with every stoichiometric branch resolved at
// compile time: kr = kf exp(-sum nu b) (the (P_atm/R)^0 factor is 1),
// d R / d c_j is one product per participant, and ci = 1.
struct E22Head {
    int flags, bint;
    int s[4];  // reactant, reactant, product, product
    const double* p;
};

__device__ __forceinline__ void load_e22(const RxnRec* R, E22Head& h)
{
    const int4 h0 = __ldg(reinterpret_cast<const int4*>(R));
    const int4 h1 = __ldg(reinterpret_cast<const int4*>(R) + 1);
    const uint4 e0 = __ldg(reinterpret_cast<const uint4*>(R) + 2);
    h.flags = h0.x;
    h.bint = h1.z;
    h.s[0] = ent_spec(e0.x);
    h.s[1] = ent_spec(e0.y);
    h.s[2] = ent_spec(e0.z);
    h.s[3] = ent_spec(e0.w);
    h.p = R->p;
}

struct E22Terms {
    double net;   // rate of progress
    double w;     // weight in row T
    double g[4];  // d net / d c_j of the four participants
    double gns;   // the same for the bath gas (0 if it does not take part)
    double d0, d1;
};

// the per-state values an elementary reaction reads: concentrations, the 1 / Kc
// factors exp(b) of the reactants and exp(-b) of the products (where the state
// is not split, the four b), enthalpies
struct E22Vals {
    double c[4], x[4], h[4];
};

template <bool DER, class ARR>
__device__ __forceinline__ void e22_fetch(const E22Head& h, bool split, const ARR& conc, const ARR& ep,
                                          const ARR& em, const ARR& hk, E22Vals& v)
{
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v.c[q] = conc[h.s[q]];
        v.x[q] = (q < 2 || !split) ? ep[h.s[q]] : em[h.s[q]];  // ep holds b if !split
        if (DER) v.h[q] = hk[h.s[q]];
    }
}

// The derivatives by one participant are the partial products of the rates of
// progress.  Rounded products and one FMA for the difference, the same in every
// kernel kind: the Jacobian's rates equal the rates kernel's bit for bit.
template <bool DER>
__device__ __forceinline__ void e22_terms(const E22Head& h, const E22Vals& v, int last, const StateVars& sv,
                                          E22Terms& o)
{
    const double* p = h.p;
    const double b = ldg(p + P_B), Ta = ldg(p + P_TA);
    const double kf = arrhenius(RX_FORM(h.flags), ldg(p + P_A), h.bint, b, Ta, sv.Tc, sv.Tinv, sv.ls, sv.tis,
                                sv.etab);
    double ikc;  // 1 / Kc = exp(-sum nu b)
    if (sv.split) {
        ikc = __dmul_rn(__dmul_rn(v.x[0], v.x[1]), __dmul_rn(v.x[2], v.x[3]));
    } else {
        const double Bsum = (v.x[2] + v.x[3]) - (v.x[0] + v.x[1]);
        ikc = fexp(-min_pos(EXP_MAX, Bsum), sv.etab);
    }
    const double kr = __dmul_rn(kf, ikc);
    const double f1 = __dmul_rn(kf, v.c[0]), f2 = __dmul_rn(kr, v.c[2]);
    const double rr = __dmul_rn(f2, v.c[3]);
    o.net = fma(f1, v.c[1], negi(rr));
    if (!DER) return;
    if (sv.split) {
        o.g[0] = __dmul_rn(kf, v.c[1]);
        o.g[1] = f1;
        o.g[2] = negi(__dmul_rn(kr, v.c[3]));
        o.g[3] = negi(f2);
    } else {  // a concentration may be negative here
        o.g[0] = __dmul_rn(kf, gsmall(v.c[1]));
        o.g[1] = __dmul_rn(kf, gsmall(v.c[0]));
        o.g[2] = negi(__dmul_rn(kr, gsmall(v.c[3])));
        o.g[3] = negi(__dmul_rn(kr, gsmall(v.c[2])));
    }
    const double dH = (v.h[2] + v.h[3]) - (v.h[0] + v.h[1]);
    o.w = row_t_weight(h.flags, p, dH, 0, sv.h_ns);
    double gns = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (h.s[j] == last) gns = o.g[j];
    o.gns = gns;
    // rf dl - rr (dl - T dB) = net dl + rr T dB
    o.d0 = fma(rr, __dmul_rn(dH, sv.kB), __dmul_rn(o.net, fma(Ta, sv.Tjinv, b)));
    o.d1 = 0.0;
    if (h.flags & RX_HASNS) {
        o.d0 = fma(negi(gns), sv.PoRT, o.d0);
        o.d1 = __dmul_rn(gns, sv.conp ? sv.PoRT : __dmul_rn(sv.V, sv.rt_inv));
    }
}

// ------------------------------------------------------------------------
// Other mass-action reactions without a third body, in a few fixed
// stoichiometric patterns (MaPattern below; pjg_capi.cu order_reactions packs
// each pattern's reactions together, entries in the pattern's order:
// reactants by coefficient, then species on both sides, then products by
// coefficient).  The arithmetic
// of rxn_terms() for such a reaction with every coefficient known at compile
// time.  Up to five entries.
template <bool REV, int F0, int R0, int F1, int R1, int F2 = 0, int R2 = 0, int F3 = 0, int R3 = 0,
          int F4 = 0, int R4 = 0>
struct MaPattern {
    static constexpr bool rev = REV;
    static constexpr int n = 2 + (F2 || R2) + (F3 || R3) + (F4 || R4);
    __host__ __device__ static constexpr int nuf(int e)
    {
        return e == 0 ? F0 : e == 1 ? F1 : e == 2 ? F2 : e == 3 ? F3 : F4;
    }
    __host__ __device__ static constexpr int nur(int e)
    {
        return e == 0 ? R0 : e == 1 ? R1 : e == 2 ? R2 : e == 3 ? R3 : R4;
    }
    __host__ __device__ static constexpr int sumf() { return F0 + F1 + F2 + F3 + F4; }
    __host__ __device__ static constexpr int sumr() { return R0 + R1 + R2 + R3 + R4; }
};

// the patterns, in the order their reactions are packed (kMaPatterns of them)
using MaP0 = MaPattern<false, 1, 0, 1, 0, 0, 1, 0, 1, 0, 1>;  // A + B => C + D + E
using MaP1 = MaPattern<true, 1, 0, 1, 0, 0, 1, 0, 1, 0, 1>;   // A + B <=> C + D + E
using MaP2 = MaPattern<true, 1, 0, 1, 0, 0, 2>;               // A + B <=> 2 C
using MaP3 = MaPattern<true, 2, 0, 0, 1, 0, 1>;               // 2 A <=> B + C
using MaP4 = MaPattern<true, 1, 0, 1, 0, 1, 0, 0, 1, 0, 1>;   // A + B + C <=> D + E
using MaP5 = MaPattern<true, 1, 0, 1, 0, 0, 1, 0, 2>;         // A + B <=> C + 2 D
using MaP6 = MaPattern<true, 1, 0, 2, 0, 0, 1, 0, 1>;         // A + 2 B <=> C + D
using MaP7 = MaPattern<false, 1, 0, 1, 0, 0, 1, 0, 1>;        // A + B => C + D
using MaP8 = MaPattern<true, 1, 0, 1, 1, 0, 1>;               // A + X <=> B + X
using MaP9 = MaPattern<true, 1, 0, 1, 0, 1, 1, 0, 1>;         // A + B + X <=> C + X
constexpr int kMaPatterns = 10;

// coefficient patterns of reactions with a third body or fall-off, evaluated
// by the general code (rxn_terms) compiled per pattern (PatStoich)
using TpP0 = MaPattern<true, 1, 0, 1, 0, 0, 1>;  // A + B (+M) <=> C
using TpP1 = MaPattern<true, 1, 0, 0, 1, 0, 1>;  // A (+M) <=> B + C
using TpP2 = MaPattern<true, 2, 0, 0, 1>;        // 2 A (+M) <=> B
constexpr int kTpPatterns = 3;

// acc * v^p for a compile-time p (0, 1 or 2), rounded products
template <int P>
__device__ __forceinline__ double mulpow_rn(double acc, double v)
{
    if (P == 0) return acc;
    if (P == 1) return __dmul_rn(acc, v);
    return __dmul_rn(acc, __dmul_rn(v, v));
}

struct MaTerms {
    double net, w;
    double g[5];
    double gns;
    double d0, d1;
};

template <class PT, bool DER, class ARR>
__device__ __forceinline__ void ma_terms(const RxnHead& h, int last, const StateVars& sv,
                                         const ARR& conc, const ARR& bk, const ARR& ep,
                                         const ARR& em, const ARR& hk, MaTerms& o)
{
    constexpr int N = PT::n;
    const double* p = h.p;
    const double b = ldg(p + P_B), Ta = ldg(p + P_TA);
    const double kf = arrhenius(RX_FORM(h.flags), ldg(p + P_A), h.bint, b, Ta, sv.Tc, sv.Tinv, sv.ls, sv.tis,
                                sv.etab);
    int sp[N];
    double c[N];
#pragma unroll
    for (int e = 0; e < N; ++e) {
        sp[e] = ent_spec(h.ent[e]);
        c[e] = conc[sp[e]];
    }
    constexpr int nu_sum = PT::sumr() - PT::sumf();
    double dH = 0.0;
    if (DER) {
        bool first = true;  // the first term starts the sum
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int nu = PT::nur(e) - PT::nuf(e);
            if (nu == 0) continue;
            dH = first ? nux(nu, hk[sp[e]]) : addnu(dH, nu, hk[sp[e]]);
            first = false;
        }
        o.w = row_t_weight(h.flags, p, dH, nu_sum, sv.h_ns);
    }
    double kr = 0.0;
    if (PT::rev) {
        double ikc;
        if (sv.split) {
            ikc = inv_kc_split<PatStoich<PT>>(h, ep, em);
        } else {
            double Bsum = 0.0;
            bool first = true;
#pragma unroll
            for (int e = 0; e < N; ++e) {
                const int nu = PT::nur(e) - PT::nuf(e);
                if (nu == 0) continue;
                Bsum = first ? nux(nu, bk[sp[e]]) : addnu(Bsum, nu, bk[sp[e]]);
                first = false;
            }
            ikc = fexp(-min_pos(EXP_MAX, Bsum), sv.etab);
        }
        kr = __dmul_rn(__dmul_rn(kf, ldg(p + P_PSUM)), ikc);
    }
    // rounded products and difference: the rate of progress is the same in
    // every kernel kind (see e22_terms)
    double rf = kf, rr = kr;
#pragma unroll
    for (int e = 0; e < N; ++e) {
        if (PT::nuf(e) == 1) rf = mulpow_rn<1>(rf, c[e]);
        if (PT::nuf(e) == 2) rf = mulpow_rn<2>(rf, c[e]);
        if (PT::rev && PT::nur(e) == 1) rr = mulpow_rn<1>(rr, c[e]);
        if (PT::rev && PT::nur(e) == 2) rr = mulpow_rn<2>(rr, c[e]);
    }
    o.net = PT::rev ? __dsub_rn(rf, rr) : rf;
    if (!DER) return;
    const double dl = fma(Ta, sv.Tjinv, b);
    double cg[N];
#pragma unroll
    for (int e = 0; e < N; ++e) cg[e] = gsmall(c[e]);
    double gns = 0.0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        double gf = 0.0, gr = 0.0;
        if (PT::nuf(j)) {
            double S = PT::nuf(j) == 2 ? kf + kf : kf;
#pragma unroll
            for (int e = 0; e < N; ++e) {
                const int q = PT::nuf(e) - (e == j);
                if (q == 1) S = S * cg[e];
                if (q == 2) S = S * (cg[e] * cg[e]);
            }
            gf = S;
        }
        if (PT::rev && PT::nur(j)) {
            double S = PT::nur(j) == 2 ? kr + kr : kr;
#pragma unroll
            for (int e = 0; e < N; ++e) {
                const int q = PT::nur(e) - (e == j);
                if (q == 1) S = S * cg[e];
                if (q == 2) S = S * (cg[e] * cg[e]);
            }
            gr = S;
        }
        o.g[j] = gf - gr;
        if (sp[j] == last) gns = o.g[j];
    }
    o.gns = gns;
    const bool hasns = h.flags & RX_HASNS;
    // rf dl - rr (dl - T dB) = net dl + rr T dB
    double d0 = PT::rev ? fma(rr, gibbs_slope(sv, dH, nu_sum), o.net * dl) : rf * dl;
    if (hasns) d0 = fma(negi(gns), sv.PoRT, d0);
    double d1 = 0.0;
    if (sv.conp) d1 = -nux(PT::sumf() - 2, rf) + (PT::rev ? nux(PT::sumr() - 2, rr) : 0.0);
    if (hasns) d1 = fma(gns, sv.conp ? sv.PoRT : __dmul_rn(sv.V, sv.rt_inv), d1);
    o.d0 = d0;
    o.d1 = d1;
}

}  // namespace pjg
