// Fused FP64 species-rate and analytical-Jacobian kernels for sm_103a.
//
// One thread evaluates one thermochemical state end to end.  All threads of a
// warp walk the same reaction list, so mechanism records are read with
// warp-uniform addresses (broadcast loads, no divergence on reaction type);
// state data are laid out state-innermost so that every per-state access of a
// warp is one coalesced 256-byte transaction.
//
// Species rates restate pyJac's sub-kernel chain (pyjac/core/rate_subs.py
// get_specrates_kernel :3026-3278) as one pass over the reactions: forward rate
// (get_simple_arrhenius_rates :2642, PLOG :2084, Chebyshev :1904), third-body
// concentration (:1788), reduced pressure and Lindemann/Troe/SRI blending
// (:2251-2641), equilibrium constant and reverse rate (:1627), rates of progress
// (:1170-1509) and the net-production scatter (:1079), then molar, temperature and
// extra-variable rates (:709-1076).  Intermediates stay in registers instead of a
// global working buffer.
//
// The Jacobian restates create_jacobian.py (:285-4522) the same way: in the
// reaction pass each reaction adds its d(rop)/dn_j block, its third-body /
// fall-off terms and its T / extra-variable column terms; terms through the
// bath-gas concentration (the "_ns" kernels) are the same for every species
// column and are gathered per row; rows T and E are assembled afterwards from
// the species block (dTdot_dnj :3382, dEdot_dnj :3266, dTdotdT :1847,
// dEdotdT :2001, dTdotdE :1595, dEdotdE :1740).
//
// Numeric guards are the reference's (pyjac/core/instruction_creator.py:370-478):
// T clamped to [100, 10000] K for rate evaluation, V >= 1e-30, moles and
// concentrations in derivative products >= 1e-300, exp(min(x, 690.775527898)),
// log(max(x, 1e-300)).  (The derivatives of A + B <=> C + D take the rates' own
// products where no concentration is negative: moles there are >= 1e-300
// already, and V > 1 or a vanishing bath gas may put a concentration below.)  As
// in the reference, the explicit T, V, P factors of the Jacobian blocks use the
// unclamped state values.
//
// FP64 instruction count is the cost that matters on GB300 (2 FP64 FMA per clock
// per SM): quotients of the NASA polynomials come precomputed in the species
// records, Troe's Fcent^(1/(1+(A/B)^2)) is exp(X ln Fcent) with ln Fcent shared
// with log10 Fcent, fall-off derivative factors are formed once per reaction,
// stoichiometric multiplications by +-1/+-2 are adds, and d(rop)/dc products
// skip zero exponents instead of dividing.  Rows T and E of the Jacobian are
// summed per reaction (d R_i / d c_j times the reaction's enthalpy, and times
// sum nu) instead of over the species block, which is not read back; the
// exponentials take their integer part on the integer pipe (fexp_s).  FP64
// instructions per GRI state, ncu: Jacobian 27,817 -> 21,085, rates 11,255 ->
// 9,619; 1M states dense F 68.5 -> 60.8 ms, rates 21.9 -> 19.0 ms.  The rates keep
// the FP64 pipe 84 % busy.  The Jacobian keeps it 61 % busy and waits for its
// per-state arrays, reductions and spilled registers (396 bytes of stores and 528
// of loads): four blocks of 128 registers per SM, 28 % of the accesses that reach
// L2 hit, DRAM moves 5.3x the output.  J^T v: 82 %.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "pjg_eval.cuh"
#include "pjg_math.cuh"
#include "pjg_rxn.cuh"

namespace pjg {

// One of the per-state arrays of ns entries.  The rates kernel keeps a pointer
// for each of its 6; the other two keep one base and a 32-bit first entry each
// (element k lies first + k strides of bytes from the state's place).  With
// pointers the Jacobian kernel's 13 arrays spilled 636 bytes of stores and 1,260
// of loads, now 396 and 528: GRI-Mech 3.0, dense F, 200,000 states 11.96 ->
// 11.68 ms, H2/O2 155,648 states 875 -> 847 us.  The rates kernel lost by the
// change (GRI, 200,000 states 3.88 -> 3.98 ms).
struct PtrView {
    double* b;
    int64_t ld;
    __device__ __forceinline__ PtrView(double* base, int64_t stride, int first) : b(base + first * stride), ld(stride) {}
    __device__ __forceinline__ double& operator[](int k) const { return b[k * ld]; }
};
struct BaseView {
    char* b;
    uint32_t st, first;  // the stride fits 32 bits: the working buffer's budget
    __device__ __forceinline__ BaseView(double* base, int64_t stride, int first_)
        : b(reinterpret_cast<char*>(base)), st((uint32_t)stride * sizeof(double)), first(first_) {}
    __device__ __forceinline__ double& operator[](int k) const
    {
        return *reinterpret_cast<double*>(b + (uint64_t)(first + k) * st);
    }
};

// Registers against warps, 1M GRI states dense F: 3 blocks per SM 75.4 ms, 4
// 63.0, 5 65.2.  A launch that leaves at most two blocks to an SM has the
// registers for no spills at all (H2/O2, 38,000 states: 293 -> 282 us), so the
// Jacobian kernel comes in that form, too.  And a mechanism whose state arrays
// are large (tiles of 32 states do not fit shared memory) gains nothing from a
// fourth block: 500 species, sparse F, 58,368 states at three blocks 69 ms, 77,824
// at four 121; compiled for three it takes 67.
#ifndef PJG_VJP_MINB
#define PJG_VJP_MINB 3  // resident 128-thread blocks per SM requested for the J^T v kernel
#endif

#ifndef PJG_JAC_MINB
#define PJG_JAC_MINB 4  // resident 128-thread blocks per SM requested for the Jacobian kernel
#endif

constexpr int kFewBlocks = 2, kLargeBlocks = 3;

#ifndef PJG_RATES_MINB
#define PJG_RATES_MINB 6  // resident 128-thread blocks per SM requested for the species-rate kernel
#endif

constexpr int kPostUnroll = 8;

// stoichiometry of the elementary class A + B <=> C + D
struct E22Stoich {
    __device__ static constexpr int nsp(const RxnHead&) { return 4; }
    __device__ static constexpr int nuf(const RxnHead&, int e) { return e < 2; }
    __device__ static constexpr int nur(const RxnHead&, int e) { return e >= 2; }
};

// One thread per state; the per-state arrays and accumulators live in global
// scratch (state-innermost, so a warp's accesses are coalesced).
template <int KIND, int MINB>  // KIND_RATES, KIND_JAC, KIND_VJP; resident blocks per SM asked for
__global__ void __launch_bounds__(PJG_BLOCK, MINB) wave_kernel(const EvalArgs a)
{
    __shared__ double etab[PJG_EXP_TAB];
    fill_exp_table(etab);
    __syncthreads();
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= a.n) return;  // no block-wide synchronisation below
    constexpr bool JAC = KIND == KIND_JAC;
    constexpr bool VJP = KIND == KIND_VJP;
    constexpr bool DER = JAC || VJP;  // derivative terms needed
    constexpr int kArr = tile_arrays(KIND);
    const int ns = a.ns, last = ns - 1;
    using SV = std::conditional_t<DER, BaseView, PtrView>;
    auto arr = [&](int which) -> SV { return SV(a.scratch + s, a.sc_ld, which * ns); };
    auto vec = [&](int v) -> SV { return arr(kArr + v); };
    const SV conc = arr(ARR_CONC), ep = arr(ARR_EP), em = arr(ARR_EM);
    const SV& bk = ep;  // b_k until the state's split is known (then exp(b_k) if it holds)
    const SV hk = DER ? arr(ARR_H) : vec(VEC_H), vt = VJP ? arr(ARR_VT) : conc;
    const SV sums = vec(0);  // by entry of the vector space (third-body sums)
    const SV wdot = vec(VEC_WDOT), cpa = vec(VEC_CP), dcpa = vec(VEC_DCP), nsrow = vec(VEC_NS);
    const SV rT = vec(VEC_RT), rE = vec(VEC_RE), cT = vec(VEC_CT), cE = vec(VEC_CE);
    // Additions are fire-and-forget reductions (red.global.add.f64): the thread
    // does not wait for the accumulator's old value.  Only this thread updates
    // its state's entries, and one thread's operations on one address apply in
    // program order, so every entry sums its reactions in a fixed order; the
    // sums are read back from L2 after a fence.  The first addition to an entry
    // of the output is a plain store (marked by the host, which knows the
    // order), so the output needs no zeroing pass.
    auto accum = [&](const SV& v, int k, double x) { atomicAdd(&v[k], x); };
    auto rd = [&](const SV& v, int k) -> double { return __ldcg(&v[k]); };
    double* accs = a.acc + s;  // Jacobian only
    auto add = [&](unsigned sl, double x) {
        if (sl == TGT_MASK) return;
        double* p = accs + (int64_t)(sl & TGT_MASK) * a.acc_ld;
        if (sl & TGT_FIRST) *p = x;
        else atomicAdd(p, x);
    };
    const bool conp = a.conp;
    const double* ph = a.phi + s * a.phi_ss;
    const double T = ph[0];
    const double Tc = fmin(10000.0, fmax(100.0, T));
    const double logT = log(Tc), Tinv = 1.0 / Tc;
    const double lg2T = log2(Tc), tis = kExpScale / Tc;
    const double E = ph[a.phi_sj];
    const double prm = a.param[s];
    const double V = conp ? E : prm;
    const double P = conp ? prm : E;
    const double Vinv = 1.0 / fmax(1e-30, V);
    const double logP = a.need_logP ? log(P) : 0.0;
    const double Tjinv = 1.0 / T;
    const double rt_inv = 1.0 / (RU * T);  // unclamped, as the reference's thd concentration
    const double PoRT = P * rt_inv;
    StateVars sv;
    sv.T = T; sv.Tc = Tc; sv.logT = logT; sv.Tinv = Tinv; sv.Tjinv = Tjinv;
    sv.V = V; sv.P = P; sv.PoRT = PoRT; sv.rt_inv = rt_inv; sv.logP = logP; sv.conp = conp;
    set_scaled<DER>(sv, lg2T, tis);
    sv.etab = etab;

    // concentrations (rate_subs.py get_concentrations :597-706)
    double nsum = 0.0;
    for (int k = 0; k < last; ++k) {
        const double nk = gsmall(ph[(int64_t)(2 + k) * a.phi_sj]);
        nsum = nsum + nk;
        conc[k] = nk * Vinv;
    }
    conc[last] = P / (RU * Tc) + -1.0 * gsmall(nsum) * Vinv;
    for (int k = 0; k < ns; ++k) {
        wdot[k] = 0.0;
        if (DER) nsrow[k] = 0.0;
        if (JAC) {
            rT[k] = 0.0;
            rE[k] = 0.0;
            cT[k] = 0.0;
            cE[k] = 0.0;
        }
    }
    if (DER)
        for (int k = vec_arrays(KIND) * ns; k < a.sc.n_vec; ++k) sums[k] = 0.0;
    if (JAC)
#pragma unroll 8
        for (int q = 0; q < a.wt.n_zero; ++q) accs[(int64_t)__ldg(a.wt.zero + q) * a.acc_ld] = 0.0;

    // thermo: Gibbs functions for Kc, cp, h (+ derivatives); the Gibbs functions'
    // exponentials, the factors of 1 / Kc (StateVars::split)
    bool split = __double2hiint(conc[last]) >= 0;
    for (int k = 0; k < ns; ++k) {
        const Thermo t = thermo<DER>(a.sp + (int64_t)k * PJG_SP_DOUBLES, Tc, logT, Tinv, conp);
        ep[k] = t.b;
        split = split && abs_le(t.b, a.kc_split_max);
        hk[k] = t.h;
        cpa[k] = t.cp;
        if (DER) dcpa[k] = t.dcp;
    }
    const double h_ns = DER ? hk[last] : 0.0, cp_ns = DER ? cpa[last] : 0.0;
    sv.h_ns = h_ns;
    sv.split = split;
    if (split) {
        for (int k = 0; k < ns; ++k) {
            const double b = ep[k];
            ep[k] = fexp(b, etab);
            em[k] = fexp(-b, etab);
        }
    }
    // J^T v: rows T and E of J are linear in the species rows, so v folds into
    // species weights vt_k = v_k + alpha * (h_k - h_ns W_k / W_ns)
    // + beta * (1 - W_k / W_ns) known before the reactions (cp_tot needs no
    // rates); the species part of the product accumulates in VEC_NS.
    double vt_c0 = 0.0, v1 = 0.0, vout0 = 0.0, vout1 = 0.0, vNS = 0.0, cp_tot_v = 0.0;
    if (VJP) {
        const double* vv = a.v + s * a.phi_ss;
        const double v0 = vv[0];
        v1 = vv[a.phi_sj];
        double ct = 0.0;
        for (int k = 0; k < ns; ++k) ct = fma(conc[k], cpa[k], ct);
        cp_tot_v = ct;
        const double extra = conp ? V : P, fixed = conp ? P : V;
        vt_c0 = v0 + v1 * extra * Tjinv;
        const double alpha = -vt_c0 / (V * ct), beta = v1 * T * RU / fixed;
        for (int k = 0; k < last; ++k) {
            const double* rec = a.sp + (int64_t)k * PJG_SP_DOUBLES;
            vt[k] = vv[(int64_t)(2 + k) * a.phi_sj] + alpha * (hk[k] - h_ns * ldg(rec + SP_MW)) +
                    beta * ldg(rec + SP_OMW);
        }
        vt[last] = 0.0;
    }

    // [M] and log10 [M] of the list of the last third-body reaction that shares
    // it (such reactions follow one another)
    MLast ml;

    const bool approx = a.jac_approx;
    // what one reaction adds; g holds d net / d c_j with the pressure modification
    auto scatter = [&](auto st_tag, const RxnHead& h, int i, double net, double w_t, const double* g, double d0,
                       double d1, double gns, double X) {
        using ST = decltype(st_tag);
        const int nsp = ST::nsp(h), flags = h.flags, thd = RX_THD(flags);
        int sp[PJG_MAXSP];
#pragma unroll
        for (int e = 0; e < PJG_MAXSP; ++e) {
            if (e >= nsp) break;
            sp[e] = ent_spec(h.ent[e]);
            const int nu = ST::nur(h, e) - ST::nuf(h, e);
            if (nu) accum(wdot, sp[e], nux(nu, net));
        }
        if (!DER) return;
        const bool hasns = (flags & RX_HASNS) && !approx, has_d1 = rxn_has_d1(flags);
        const bool listed = thd && h.list >= 0;  // a shared list
        const int n_l = thd && !listed ? h.thd_cnt : 0;
        const int* tb = a.wt.tb + (listed ? __ldg(a.wt.tb_off + i) : 0);
        if (VJP) {
            double w = 0.0;
#pragma unroll
            for (int e = 0; e < PJG_MAXSP; ++e) {
                if (e >= nsp) break;
                const int nu = ST::nur(h, e) - ST::nuf(h, e);
                if (nu) w = e == 0 ? nux(nu, vt[sp[e]]) : addnu(w, nu, vt[sp[e]]);
            }
#pragma unroll
            for (int e = 0; e < PJG_MAXSP; ++e) {
                if (e >= nsp) break;
                if (sp[e] != last) accum(nsrow, sp[e], w * g[e]);
            }
            if (listed) accum(sums, __ldg(tb), w * X);
            for (int l = 0; l < n_l; ++l) {
                const int j = __ldg(a.thd_spec + h.thd_off + l);
                const double x = __dmul_rn(__ldg(a.thd_coef + h.thd_off + l), w * X);
                if (j != last) accum(nsrow, j, x);
                else if (!approx) vNS = vNS + x;
            }
            if (hasns) vNS = fma(w, gns, vNS);
            vout0 = fma(w, d0, vout0);
            if (has_d1) vout1 = fma(w, d1, vout1);
            return;
        }
        const unsigned* slots = a.wt.slots + __ldg(a.wt.slot_off + i);
        int nu_sum = 0;
#pragma unroll
        for (int ka = 0; ka < PJG_MAXSP; ++ka) {
            if (ka >= nsp) break;
            const int nu = ST::nur(h, ka) - ST::nuf(h, ka);
            nu_sum += nu;
            if (nu == 0 || sp[ka] == last) continue;
#pragma unroll
            for (int e = 0; e < PJG_MAXSP; ++e) {
                if (e >= nsp) break;
                add(__ldg(slots + ka * (nsp + n_l) + e), nux(nu, g[e]));
            }
            accum(cT, sp[ka], nux(nu, d0));
            if (has_d1) accum(cE, sp[ka], nux(nu, d1));
            if (hasns) accum(nsrow, sp[ka], nux(nu, gns));
            if (listed) accum(sums, __ldg(tb + ka), nux(nu, X));
        }
        const bool we = flags & RX_WE, real = flags & RX_WEREAL;
        const double wE = real ? ldg(h.p + P_WE) : 0.0;
#pragma unroll
        for (int e = 0; e < PJG_MAXSP; ++e) {
            if (e >= nsp) break;
            if (sp[e] == last || (!(flags & RX_REV) && ST::nuf(h, e) == 0)) continue;
            accum(rT, sp[e], __dmul_rn(w_t, g[e]));
            if (we) accum(rE, sp[e], real ? __dmul_rn(wE, g[e]) : nux(nu_sum, g[e]));
        }
        if (listed) {
            accum(sums, __ldg(tb + nsp), __dmul_rn(w_t, X));
            if (we) accum(sums, __ldg(tb + nsp + 1), real ? __dmul_rn(wE, X) : nux(nu_sum, X));
        }
        for (int l = 0; l < n_l; ++l) {
            const int j = __ldg(a.thd_spec + h.thd_off + l);
            const double x = __dmul_rn(__ldg(a.thd_coef + h.thd_off + l), X);
            if (j == last && approx) continue;
#pragma unroll
            for (int ka = 0; ka < PJG_MAXSP; ++ka) {
                if (ka >= nsp) break;
                const int nu = ST::nur(h, ka) - ST::nuf(h, ka);
                if (nu == 0 || sp[ka] == last) continue;
                if (j == last) accum(nsrow, sp[ka], nux(nu, x));
                else add(__ldg(slots + ka * (nsp + n_l) + nsp + l), nux(nu, x));
            }
            if (j == last) continue;
            accum(rT, j, __dmul_rn(w_t, x));
            if (we) accum(rE, j, real ? __dmul_rn(wE, x) : nux(nu_sum, x));
        }
    };

    // ------------------------------------- reactions A + B <=> C + D (packed first)
    // the next reaction's record and per-state values are loaded while this
    // one computes
    {
        const int n22 = a.cls_off[1];
        E22Head hn;
        E22Vals vn;
        if (n22 > 0) {
            load_e22(a.rxn, hn);
            e22_fetch<DER>(hn, split, conc, ep, em, hk, vn);
        }
        for (int i = 0; i < n22; ++i) {
            const E22Head h = hn;
            const E22Vals v = vn;
            if (i + 1 < n22) {
                load_e22(a.rxn + i + 1, hn);
                e22_fetch<DER>(hn, split, conc, ep, em, hk, vn);
            }
            E22Terms o;
            e22_terms<DER>(h, v, last, sv, o);
            RxnHead r;
            r.flags = h.flags;
            r.p = h.p;
            r.thd_cnt = 0;
            r.list = -1;
#pragma unroll
            for (int e = 0; e < 4; ++e) r.ent[e] = (unsigned)h.s[e];
            scatter(E22Stoich{}, r, i, o.net, o.w, o.g, o.d0, o.d1, o.gns, 0.0);
        }
    }
    // the next reaction's record and values, brought nearer while this one computes
    auto touch = [&](const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); };
    auto prefetch = [&](int i) {
        const RxnRec* R = a.rxn + (i + 1 < a.nr ? i + 1 : i);
        touch(reinterpret_cast<const char*>(R) + 128);
        const int n = __ldg(&R->nspec);
        for (int e = 0; e < n; ++e) {
            const int k = ent_spec(__ldg(&R->ent[e]));
            touch(&conc[k]);
            touch(&ep[k]);
            touch(&em[k]);
            if (DER) touch(&hk[k]);
        }
    };
    // ------------------------- other mass-action reactions in fixed patterns
    auto ma_range = [&](auto tag, int c) {
        using PT = decltype(tag);
        for (int i = a.cls_off[c]; i < a.cls_off[c + 1]; ++i) {
            RxnHead h;
            load_head(a.rxn + i, h);
            prefetch(i);
            MaTerms o;
            ma_terms<PT, DER>(h, last, sv, conc, bk, ep, em, hk, o);
            scatter(PatStoich<PT>{}, h, i, o.net, o.w, o.g, o.d0, o.d1, o.gns, 0.0);
        }
    };
    ma_range(MaP0{}, 1);
    ma_range(MaP1{}, 2);
    ma_range(MaP2{}, 3);
    ma_range(MaP3{}, 4);
    ma_range(MaP4{}, 5);
    ma_range(MaP5{}, 6);
    ma_range(MaP6{}, 7);
    ma_range(MaP7{}, 8);
    ma_range(MaP8{}, 9);
    ma_range(MaP9{}, 10);
    // ------------------------------------------------------- other reactions
    // (the general code; third-body and fall-off reactions of the patterns
    // TpP0..TpP2 compiled per pattern, the rest reading their coefficients)
    auto general = [&](auto st_tag, int c) {
        using ST = decltype(st_tag);
        for (int i = a.cls_off[c]; i < a.cls_off[c + 1]; ++i) {
            RxnHead h;
            load_head(a.rxn + i, h);
            prefetch(i);
            RxnTerms o;
            rxn_terms<DER, ST>(h, a.aux, a.thd_spec, a.thd_coef, last, sv, conc, bk, ep, em, hk, ml, o);
            double gci[PJG_MAXSP];
            if (DER) {
                const bool thd = RX_THD(h.flags) != THD_NONE;
#pragma unroll
                for (int e = 0; e < PJG_MAXSP; ++e)
                    if (e < ST::nsp(h)) gci[e] = thd ? __dmul_rn(o.g[e], o.ci_) : o.g[e];
            }
            scatter(ST{}, h, i, o.net, o.w, gci, o.d0, o.d1, o.gns * o.ci_, o.X);
        }
    };
    general(PatStoich<TpP0>{}, 11);
    general(PatStoich<TpP1>{}, 12);
    general(PatStoich<TpP2>{}, 13);
    general(RunStoich{}, 14);

    __threadfence();

    // ------------------------ third-body columns, temperature and E rates
    if (DER) {
        for (int q0 = 0; q0 < a.wt.n_post; q0 += kPostUnroll) {
            int4 it[kPostUnroll];
            double x[kPostUnroll];
#pragma unroll
            for (int e = 0; e < kPostUnroll; ++e)
                it[e] = __ldg(reinterpret_cast<const int4*>(a.wt.post + (q0 + e < a.wt.n_post ? q0 + e : q0)));
#pragma unroll
            for (int e = 0; e < kPostUnroll; ++e) x[e] = rd(sums, it[e].x);
#pragma unroll
            for (int e = 0; e < kPostUnroll; ++e) {
                if (q0 + e >= a.wt.n_post) break;
                const unsigned tgt = (unsigned)it[e].y;
                const double y = __dmul_rn(__hiloint2double(it[e].w, it[e].z), x[e]);
                // J^T v has no output entries among the targets
                if (!JAC || (tgt & TGT_VEC)) accum(sums, (int)(tgt & TGT_MASK), y);
                else add(tgt, y);
            }
        }
        __threadfence();
    }
    // sums over species in partial sums (the order of the tile kernels)
    const int n_parts = sum_parts(ns);
    double upper = 0.0, lower = 0.0, dE = 0.0, dTsum = 0.0, dTsum1 = 0.0;
    for (int w = 0; w < n_parts; ++w) {
        double pu = 0.0, pl = 0.0, pe = 0.0, pt = 0.0, p1 = 0.0;
#pragma unroll 4
        for (int k = w; k < ns; k += n_parts) {
            const double w_k = rd(wdot, k), cpk = cpa[k], ck = conc[k];
            pu = fma(hk[k], w_k, pu);
            pl = fma(ck, cpk, pl);
            pe = fma(ldg(a.sp + (int64_t)k * PJG_SP_DOUBLES + SP_OMW), w_k, pe);  // omw of the bath gas is 0
            if (DER) {
                pt = fma(cp_ns * Tjinv - dcpa[k], ck, pt);
                p1 = fma(cpk - cp_ns, ck, p1);
            }
        }
        upper = w ? upper + pu : pu;
        lower = w ? lower + pl : pl;
        dE = w ? dE + pe : pe;
        dTsum = w ? dTsum + pt : pt;
        dTsum1 = w ? dTsum1 + p1 : p1;
    }
    const double inv_cp = 1.0 / lower;
    const double Tdot = -upper * inv_cp;
    const double Vval = fmax(1e-30, V);
    if (a.dphi) {
        double* o = a.dphi + s * a.dphi_ss;
        double Edot;
        if (conp) {
            Edot = Vval * Tdot / Tc;
            Edot = Edot + Vval * dE * Tc * RU / P;
        } else {
            Edot = P * Tdot / Tc;
            Edot = Edot + Tc * RU * dE;
        }
        o[0] = Tdot;
        o[a.dphi_sj] = Edot;
        for (int k = 0; k < last; ++k) o[(int64_t)(2 + k) * a.dphi_sj] = Vval * rd(wdot, k);
    }
    if (VJP) {
        // constant parts of columns T and E (from rows T, E of dTdot_dT :1847,
        // dEdotdT :2001, dTdotdE :1595, dEdotdE :1740) and the species columns'
        // bath-gas and d cp_tot / dn_j terms
        const double extra = conp ? V : P, ct = cp_tot_v;
        for (int q = 0; q < a.n_ns_post; ++q)
            vNS = fma(__ldg(&a.ns_post[q].coef), rd(sums, (int)__ldg(&a.ns_post[q].src)), vNS);
        double wsum = 0.0, omws = 0.0, hws = 0.0, vws = 0.0;
        for (int k = 0; k < last; ++k) {
            const double* rec = a.sp + (int64_t)k * PJG_SP_DOUBLES;
            const double mw = ldg(rec + SP_MW), omw = ldg(rec + SP_OMW);
            const double w_k = rd(wdot, k), cpk = cpa[k];
            wsum = wsum + w_k * (-cpk + mw * cp_ns);
            omws = fma(omw, w_k, omws);
            hws = fma(hk[k] - h_ns * mw, w_k, hws);
            vws = fma(vt[k], w_k, vws);
        }
        if (conp) vout1 = vout1 - vws;  // the reactions' -net of column E
        const double C0 = vt_c0 * (Tdot * dTsum + wsum) / ct - v1 * extra * Tdot * Tjinv * Tjinv +
                          v1 * RU * (conp ? V / P : 1.0) * omws;
        double C1 = conp ? vt_c0 * (Tdot * dTsum1 + hws) / (ct * V) : -vt_c0 * Tdot * cp_ns * rt_inv / ct;
        C1 += v1 * Tdot * Tjinv;
        const double gam = -vt_c0 * Tdot / (V * ct);
        double* o = a.vjp + s * a.phi_ss;
        o[0] = fma(vout0, V * Tjinv, C0);  // the reactions' terms of column T leave V / T out
        o[a.phi_sj] = vout1 + C1;
        for (int j = 0; j < last; ++j)
            o[(int64_t)(2 + j) * a.phi_sj] = rd(nsrow, j) - vNS + gam * (cpa[j] - cp_ns);
        return;
    }
    if (!JAC) return;

    // ------------------------------------------- assemble rows T and E
    // Both rows are linear in the species rows, so each reaction has added its
    // share (w_i d R_i / d c_j, with w_i = sum_k nu_ki hw_k for row T and
    // sum_k nu_ki (1 - W_k / W_ns) = sum nu for row E); the bath-gas terms, the
    // same for every species column, take one sum per state.
    const int64_t ald = a.acc_ld;
    const double fixed = conp ? P : V, extra = conp ? V : P;
    const double Vjinv = V >= 1e-30 ? Vinv : 1.0 / V;
    const double inv_vcp = Vjinv * inv_cp;
    const double eTj = extra * Tjinv, VTj = V * Tjinv, TRf = T * RU / fixed;
    for (int q = 0; q < a.n_ns; ++q) {
        const double mv = negi(rd(nsrow, __ldg(a.ns_rows + q)));
        if (!nonzero(mv)) continue;
        const int* sl = a.ns_slots + q * last;
#pragma unroll 8
        for (int j = 0; j < last; ++j) {
            const int t = __ldg(sl + j);
            if (t >= 0) atomicAdd(accs + (int64_t)t * ald, mv);
        }
    }
    // T column of rows T, E and E column of rows T, E; column E of a species
    // row: at constant pressure the terms leave out -net of each reaction, in
    // sum -wdot_k
    double rate_sum = 0.0, sumT = 0.0, spec1 = 0.0, sumE1 = 0.0, nsT = 0.0, nsE = 0.0;
    for (int w = 0; w < n_parts; ++w) {
        double pr = 0.0, pt = 0.0, ps = 0.0, pe = 0.0, pnt = 0.0, pne = 0.0;
#pragma unroll 2
        for (int k = w; k < last; k += n_parts) {
            const double* rec = a.sp + (int64_t)k * PJG_SP_DOUBLES;
            const double mw = ldg(rec + SP_MW), omw = ldg(rec + SP_OMW);
            const int sl0 = __ldg(a.sp_slots + 2 * k), sl1 = __ldg(a.sp_slots + 2 * k + 1);
            const double w_k = rd(wdot, k), cpk = cpa[k], hwk = fma(-h_ns, mw, hk[k]);
            const double ct = rd(cT, k), ce = rd(cE, k), ek = conp ? ce - w_k : ce;
            if (sl0 >= 0) accs[(int64_t)sl0 * ald] = ct * VTj;
            if (sl1 >= 0) accs[(int64_t)sl1 * ald] = ek;
            const double vk = sl0 >= 0 ? ct * Tjinv : 0.0;  // J_kT / V
            const double Jk1 = sl1 >= 0 ? ek : 0.0;
            pr = fma(-vk, hwk, pr);
            pr = fma(w_k, fma(mw, cp_ns, -cpk), pr);
            pt = fma(omw, conp ? fma(Tjinv, w_k, vk) : fma(T, vk, w_k), pt);
            ps = fma(hwk, conp ? Jk1 - w_k : Jk1, ps);
            pe = fma(omw, Jk1, pe);
        }
        for (int q = w; q < a.n_ns; q += n_parts) {
            const int k = __ldg(a.ns_rows + q);
            const double v = rd(nsrow, k);
            pnt = fma(fma(-h_ns, ldg(a.sp + (int64_t)k * PJG_SP_DOUBLES + SP_MW), hk[k]), v, pnt);
            pne = fma(ldg(a.sp + (int64_t)k * PJG_SP_DOUBLES + SP_OMW), v, pne);
        }
        rate_sum = w ? rate_sum + pr : pr;
        sumT = w ? sumT + pt : pt;
        spec1 = w ? spec1 + ps : ps;
        sumE1 = w ? sumE1 + pe : pe;
        nsT = w ? nsT + pnt : pnt;
        nsE = w ? nsE + pne : pne;
    }
    const bool summed = a.col_list == nullptr;
    if (!summed) __threadfence();  // the species block is read back below
#pragma unroll 2
    for (int j = 0; j < last; ++j) {
        double sT, sE;
        if (summed) {
            sT = rd(rT, j) - nsT;
            sE = rd(rE, j) - nsE;
        } else {
            sT = 0.0;
            sE = 0.0;
            const int c0 = __ldg(a.col_off + j), c1 = __ldg(a.col_off + j + 1);
            for (int q = c0; q < c1; ++q) {
                const int2 e = __ldg(a.col_list + q);
                const double Jkj = __ldcg(accs + (int64_t)e.y * ald);
                sT = fma(fma(-h_ns, ldg(a.sp + (int64_t)e.x * PJG_SP_DOUBLES + SP_MW), hk[e.x]), Jkj, sT);
                sE = fma(ldg(a.sp + (int64_t)e.x * PJG_SP_DOUBLES + SP_OMW), Jkj, sE);
            }
        }
        const double J0 = -1.0 * (sT + Tdot * (cpa[j] + -1.0 * cp_ns)) * inv_vcp;
        accs[(int64_t)__ldg(a.cj_slots + 2 * j) * ald] = J0;
        accs[(int64_t)__ldg(a.cj_slots + 2 * j + 1) * ald] = TRf * sE + eTj * J0;
    }
    const double J00 = (Tdot * dTsum + rate_sum) * inv_cp;
    double J10;
    if (conp) {
        J10 = V * Tjinv * (J00 - Tjinv * Tdot);
        J10 = J10 + RU * T * V * sumT / P;
    } else {
        J10 = P * (J00 - Tdot * Tjinv) * Tjinv;
        J10 = J10 + RU * sumT;
    }
    double J01;
    if (conp) {
        J01 = (Tdot * dTsum1 - spec1) * inv_vcp;
    } else {
        J01 = -((Tdot * cp_ns * rt_inv) * inv_cp);
        J01 = J01 - (spec1 * Vjinv) * inv_cp;
    }
    double J11 = TRf * sumE1;
    J11 = J11 + (extra * J01 + Tdot) * Tjinv;
    accs[(int64_t)a.s00 * ald] = J00;
    accs[(int64_t)a.s10 * ald] = J10;
    accs[(int64_t)a.s01 * ald] = J01;
    accs[(int64_t)a.s11 * ald] = J11;
}

// One translation unit instantiates each form (pjg_eval.cu, pjg_jac*.cu), so that
// they compile in parallel.
template <int KIND, int MINB>
void wave_launch(const EvalArgs& a, unsigned grid, cudaStream_t st);
template <int KIND, int MINB>
const void* wave_fn();

#define PJG_WAVE_INSTANCE(KIND, MINB)                                                  \
    template <>                                                                        \
    void pjg::wave_launch<KIND, MINB>(const EvalArgs& a, unsigned grid, cudaStream_t st) \
    {                                                                                  \
        pjg::wave_kernel<KIND, MINB><<<grid, PJG_BLOCK, 0, st>>>(a);                   \
    }                                                                                  \
    template <>                                                                        \
    const void* pjg::wave_fn<KIND, MINB>()                                             \
    {                                                                                  \
        return (const void*)pjg::wave_kernel<KIND, MINB>;                              \
    }

#define PJG_WAVE_DECLARE(KIND, MINB)                                                   \
    template <>                                                                        \
    void wave_launch<KIND, MINB>(const EvalArgs& a, unsigned grid, cudaStream_t st);   \
    template <>                                                                        \
    const void* wave_fn<KIND, MINB>();
PJG_WAVE_DECLARE(KIND_RATES, PJG_RATES_MINB)
PJG_WAVE_DECLARE(KIND_VJP, PJG_VJP_MINB)
PJG_WAVE_DECLARE(KIND_JAC, PJG_JAC_MINB)
PJG_WAVE_DECLARE(KIND_JAC, kFewBlocks)
PJG_WAVE_DECLARE(KIND_JAC, kLargeBlocks)
#undef PJG_WAVE_DECLARE

}  // namespace pjg
