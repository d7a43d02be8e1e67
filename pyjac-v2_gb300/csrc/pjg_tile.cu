// Species-rate, Jacobian and J^T v kernels for batches below a wave of the
// thread-per-state kernels (pjg_wave.cuh): the same reaction code (pjg_rxn.cuh),
// the sums over reactions and species in the same order.  The rates are equal bit
// for bit, the Jacobian but for the contraction of a few products; of J^T v, columns
// T and E and the bath-gas term of every column are summed per worker first, so
// their last bits depend on the tile's shape.
#include <cuda_runtime.h>

#include <type_traits>

#include "pjg_eval.cuh"
#include "pjg_math.cuh"
#include "pjg_rxn.cuh"

using namespace pjg;

namespace {

constexpr int kPostUnroll = 8;
constexpr int kNsParts = 4;  // pieces of a row of bath-gas terms

// one state's view of an array of the tile: entry k at b[k << slog]
struct TA {
    double* b;
    int slog;
    __device__ __forceinline__ double& operator[](int k) const { return b[k << slog]; }
};

// Explicit global-space accesses: the targets' address space is not known to
// the compiler (a generic FP64 atomic tests for shared memory and loops there).
__device__ __forceinline__ void st_global(uint64_t p, double x)
{
    asm volatile("st.global.f64 [%0], %1;" ::"l"(p), "d"(x) : "memory");
}
__device__ __forceinline__ void red_global(uint64_t p, double x)
{
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(x) : "memory");
}

// A tile of S states is evaluated by W warps (EvalArgs, pjg_eval.cuh): the
// reactions come in batches, one per worker; a worker leaves its reaction's
// terms in shared memory, and after a barrier the batch's additions to the
// Jacobian and the rates are made from there, every target by one worker, in
// the reactions' order.  So each of these sums has one fixed order, whatever S and
// W, and the additions are fire-and-forget reductions (red.global.add.f64) that
// take no FP64 instruction.
//
// The arrays that the reactions read (concentrations, 1 / Kc factors, weights)
// stay in shared memory.  With a thread per state and these arrays in global
// memory, 16 warps per SM held 2.2 MB of them: 45 % of the warps' time went
// into waiting for L1 misses (hit rate 18 %), and a batch smaller than one
// wave (77,824 states) left SMs or lanes idle and took as long as a whole one.
// GRI-Mech 3.0 on GB300, before -> here: dense Jacobian C, 200 states 2,370 ->
// 131 us; sparse F, 10,007 states 2,694 -> 1,031 us; rates C, 1,000 states 720 ->
// 137 us; the 500-species mechanism's sparse Jacobian C, 4,096 states 60.9 ->
// 13.8 ms.  Tiles of 32 states keep the FP64 pipe 61 % busy where they fill the SMs
// (37 % of the 10,007 states' time, nine of whose 313 tiles run a second round): what
// is left are the phases between the reactions and waits on shared memory.  Tiles
// of a few states wait on the barriers between a batch's reactions and its
// additions (half to two thirds of the stalls), those of 500 species on instruction
// fetch and barriers.
template <int KIND>  // KIND_RATES, KIND_JAC, KIND_VJP
__global__ void __launch_bounds__(32 * kTileWarps, KIND == KIND_RATES ? 3 : 2)
    tile_kernel(const EvalArgs a)
{
    constexpr bool JAC = KIND == KIND_JAC;
    constexpr bool VJP = KIND == KIND_VJP;
    constexpr bool DER = JAC || VJP;  // derivative terms needed
    extern __shared__ double smem[];
    double* etab = smem;
    int* nosplit = reinterpret_cast<int*>(smem + PJG_EXP_TAB);  // one per state
    const int ns = a.ns, last = ns - 1;
    const int slog = a.sc.slog, S = 1 << slog, wpw = 32 >> slog;  // states, workers per warp
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int st = lane & (S - 1), grp = lane >> slog, wk = warp * wpw + grp, G = a.sc.warps * wpw;
    // the worker's lanes: they share its items, so they refill them together
    const unsigned own_lanes = ((slog == 5 ? 0u : 1u << S) - 1u) << (grp << slog);
    constexpr int kArr = tile_arrays(KIND);
    const int cap = item_stage(slog);
    uint2* stage = reinterpret_cast<uint2*>(smem + kTileStatic / sizeof(double)) + wk * cap;
    double* arrays = smem + kTileStatic / sizeof(double) + G * cap + st;
    auto arr = [&](int which) -> TA { return TA{arrays + ((which * ns) << slog), slog}; };
    const TA conc = arr(ARR_CONC), ep = arr(ARR_EP), em = arr(ARR_EM);
    const TA& bk = ep;  // b_k until the state's split is known (then exp(b_k) if it holds)
    const TA hk = DER ? arr(ARR_H) : conc, vt = VJP ? arr(ARR_VT) : conc;
    MLists<TA> ml{TA{arrays + ((kArr * ns) << slog), slog}, a.n_m};
    double* buf = arrays + ((kArr * ns + 2 * a.n_m) << slog);
    double* red = buf - st;  // per-state values between the reaction phases
    double* vec = a.scratch + (int64_t)blockIdx.x * a.sc.n_vec * S + st;
    auto vat = [&](int v, int k) -> double* { return vec + ((v * ns + k) << slog); };
    auto rd = [&](int v, int k) -> double { return __ldcg(vat(v, k)); };
    const bool conp = a.conp;

    fill_exp_table(etab);
    const int64_t tiles = (a.n + S - 1) >> slog;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t s_raw = (tile << slog) + st;
        const bool live = s_raw < a.n;
        const int64_t s = live ? s_raw : a.n - 1;  // a tile's surplus lanes repeat the last state
        // a surplus lane's Jacobian goes to the slice's unread last entry
        double* unread = vec + ((a.sc.n_vec - 1) << slog);
        double* accs = JAC ? (live ? a.acc + s * a.acc_ss : unread) : nullptr;
        const int64_t acc_ld = live ? a.acc_ld : 0;
        const uint64_t acc_g = __cvta_generic_to_global(accs), ld_bytes = (uint64_t)acc_ld * sizeof(double);
        const uint64_t vec_g = __cvta_generic_to_global(vec);
        // target += x, or its first addition
        auto apply = [&](unsigned tgt, double x) {
            const uint64_t p = (tgt & TGT_VEC) || !JAC ? vec_g + (uint64_t)(tgt & TGT_MASK) * (8u << slog)
                                                       : acc_g + (uint64_t)(tgt & TGT_MASK) * ld_bytes;
            if (tgt & TGT_FIRST) st_global(p, x);
            else red_global(p, x);
        };
        if (threadIdx.x < S) nosplit[threadIdx.x] = 0;
        __syncthreads();  // also: the previous tile is done with shared memory and the slice

        const double* ph = a.phi + s * a.phi_ss;
        const double T = ph[0];
        const double Tc = fmin(10000.0, fmax(100.0, T));
        const double E = ph[a.phi_sj];
        const double prm = a.param[s];
        const double V = conp ? E : prm;
        const double P = conp ? prm : E;
        // each worker takes a few of the state's quotients and logarithms
        enum { Q_LOGT = 0, Q_TINV, Q_TJINV, Q_VINV, Q_RT, Q_LOGP, Q_LG2T, Q_TIS, Q_N };
        for (int q = wk; q < Q_N; q += G) {
            double x = 0.0;
            if (q == Q_LOGT) x = log(Tc);
            else if (q == Q_LG2T) x = log2(Tc);
            else if (q == Q_LOGP) x = a.need_logP ? log(P) : 0.0;
            else
                x = (q == Q_TIS ? kExpScale : 1.0) / (q == Q_TIS ? Tc : q == Q_TINV ? Tc : q == Q_TJINV ? T : q == Q_VINV ? fmax(1e-30, V) : RU * T);
            red[(q << slog) + st] = x;
        }
        __syncthreads();
        const double logT = red[(Q_LOGT << slog) + st], Tinv = red[(Q_TINV << slog) + st];
        const double Tjinv = red[(Q_TJINV << slog) + st], Vinv = red[(Q_VINV << slog) + st];
        const double rt_inv = red[(Q_RT << slog) + st];  // unclamped, as the reference's thd concentration
        const double logP = red[(Q_LOGP << slog) + st];
        const double PoRT = P * rt_inv;
        StateVars sv;
        sv.T = T; sv.Tc = Tc; sv.logT = logT; sv.Tinv = Tinv; sv.Tjinv = Tjinv;
        sv.V = V; sv.P = P; sv.PoRT = PoRT; sv.rt_inv = rt_inv; sv.logP = logP; sv.conp = conp;
        set_scaled<DER>(sv, red[(Q_LG2T << slog) + st], red[(Q_TIS << slog) + st]);
        sv.etab = etab;

        // concentrations (rate_subs.py get_concentrations :597-706) by every
        // worker but the first, which sums the moles for the bath gas
        if (wk == 0) {
            double nsum = 0.0;
            for (int k = 0; k < last; ++k) nsum = nsum + gsmall(ph[(int64_t)(2 + k) * a.phi_sj]);
            const double cl = P / (RU * Tc) + -1.0 * gsmall(nsum) * Vinv;
            conc[last] = cl;
            if (__double2hiint(cl) < 0) nosplit[st] = 1;
        } else {
            for (int k = wk - 1; k < last; k += G - 1) conc[k] = gsmall(ph[(int64_t)(2 + k) * a.phi_sj]) * Vinv;
        }
        // thermo: Gibbs functions for Kc, cp, h (+ derivatives)
        for (int k = wk; k < ns; k += G) {
            const Thermo t = thermo<DER>(a.sp + (int64_t)k * PJG_SP_DOUBLES, Tc, logT, Tinv, conp);
            ep[k] = t.b;
            if (!abs_le(t.b, a.kc_split_max)) nosplit[st] = 1;
            *vat(VEC_CP, k) = t.cp;
            *vat(VEC_H, k) = t.h;
            if (DER) {
                hk[k] = t.h;
                *vat(VEC_DCP, k) = t.dcp;
            }
        }
        __syncthreads();
        const double h_ns = DER ? hk[last] : 0.0, cp_ns = DER ? rd(VEC_CP, last) : 0.0;
        sv.h_ns = h_ns;
        // the Gibbs functions' exponentials, the factors of 1 / Kc (StateVars::split)
        const bool split = nosplit[st] == 0;
        sv.split = split;
        if (split) {
            for (int k = wk; k < ns; k += G) {
                const double b = ep[k];
                ep[k] = fexp(b, etab);
                em[k] = fexp(-b, etab);
            }
        }
        // [M] of the third-body lists that several reactions share, and its logarithm
        for (int l = wk; l < a.n_m; l += G) {
            const int4 e = __ldg(a.m_lists + l);
            double M = e.z ? PoRT : 0.0;
            for (int q = e.x; q < e.x + e.y; ++q) M = fma(__ldg(a.thd_coef + q), conc[__ldg(a.thd_spec + q)], M);
            ml.m[l] = M;
            ml.m[a.n_m + l] = e.w ? __dmul_rn(log(M), INV_LN10) : 0.0;  // log10
        }
        // J^T v: rows T and E of J are linear in the species rows, so v folds into
        // species weights vt_k = v_k + alpha * (h_k - h_ns W_k / W_ns)
        // + beta * (1 - W_k / W_ns) known before the reactions (cp_tot needs no
        // rates); the species part of the product accumulates in VEC_NS.
        double vt_c0 = 0.0, v1 = 0.0, vout0 = 0.0, vout1 = 0.0, vNS = 0.0, cp_tot_v = 0.0;
        if (VJP) {
            if (wk == 0) {
                double ct = 0.0;
                for (int k = 0; k < ns; ++k) ct = fma(conc[k], rd(VEC_CP, k), ct);
                red[st] = ct;
            }
            __syncthreads();
            const double* vv = a.v + s * a.phi_ss;
            const double v0 = vv[0];
            v1 = vv[a.phi_sj];
            cp_tot_v = red[st];
            const double extra = conp ? V : P, fixed = conp ? P : V;
            vt_c0 = v0 + v1 * extra * Tjinv;
            const double alpha = -vt_c0 / (V * cp_tot_v), beta = v1 * T * RU / fixed;
            for (int k = wk; k < ns; k += G) {
                const double* rec = a.sp + (int64_t)k * PJG_SP_DOUBLES;
                vt[k] = k == last ? 0.0
                                  : vv[(int64_t)(2 + k) * a.phi_sj] +
                                        alpha * (hk[k] - h_ns * ldg(rec + SP_MW)) + beta * ldg(rec + SP_OMW);
            }
        }
        __syncthreads();

        // ---------------------------------------------------- the reactions
        if (wk < 2) buf[(wk * a.sc.buf_terms) << slog] = 0.0;  // term 0 of both buffers
        __syncthreads();
        // A batch's terms go to one of two buffers in turn, so one barrier per
        // batch is enough.
        const bool approx = a.jac_approx;
        for (int bt = 0; bt < a.sc.n_batch; ++bt) {
            double* cur = buf + (bt & 1 ? a.sc.buf_terms << slog : 0);
            // the additions' first items, copied to shared memory meanwhile
            const int* off = a.sc.item_off + RUN_N * (bt * G + wk);
            const int q_begin = __ldg(off), q_end = __ldg(off + RUN_N);
            auto fill = [&](int from) {
                for (int e = 2 * st; e < cap && from + e < q_end; e += 2 * S) {
                    const unsigned d = (unsigned)__cvta_generic_to_shared(stage + e);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(a.sc.items + from + e) : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            __syncwarp();  // the warp's lanes are done with the last batch's items
            fill(q_begin);
            for (int rd_ = 0; rd_ < a.sc.rounds; ++rd_) {
                const int4 task = __ldg(a.sc.tasks + (bt * a.sc.rounds + rd_) * a.sc.warps + warp);
                const int i = task.y + grp;
                if (grp >= task.z) continue;
                const RxnRec* R = a.rxn + i;
                double* out = cur + (__ldg(a.sc.term_off + i) << slog);
                auto put = [&](double x) {
                    *out = x;
                    out += S;
                };
                if (task.x == 0) {
                    E22Head h;
                    E22Vals v;
                    E22Terms o;
                    load_e22(R, h);
                    e22_fetch<DER>(h, split, conc, ep, em, hk, v);
                    e22_terms<DER>(h, v, last, sv, o);
                    if (!DER) {
                        put(o.net);
                    } else {
                        const double w = VJP ? (vt[h.s[2]] + vt[h.s[3]]) - (vt[h.s[0]] + vt[h.s[1]]) : o.w;
                        const bool hasns = (h.flags & RX_HASNS) && !approx;
                        if (JAC) {
                            put(w);
                            put(o.net);
                            put(o.d0);
#pragma unroll
                            for (int e = 0; e < 4; ++e) put(o.g[e]);
                            if (hasns) put(o.gns);
                            if (h.flags & RX_HASNS) put(o.d1);
                            if (h.flags & RX_WEREAL) put(ldg(h.p + P_WE));
                        } else {
                            put(o.net);
#pragma unroll
                            for (int e = 0; e < 4; ++e) put(w * o.g[e]);
                            if (hasns) vNS = fma(w, o.gns, vNS);
                            vout0 = fma(w, o.d0, vout0);
                            if (h.flags & RX_HASNS) vout1 = fma(w, o.d1, vout1);
                        }
                    }
                } else {
                    // other mass-action reactions in fixed patterns
                    auto ma = [&](auto tag) {
                        using PT = decltype(tag);
                        constexpr int N = PT::n;
                        RxnHead h;
                        load_head(R, h);
                        MaTerms o;
                        ma_terms<PT, DER>(h, last, sv, conc, bk, ep, em, hk, o);
                        if (!DER) {
                            put(o.net);
                            return;
                        }
                        double w = o.w;
                        if (VJP) {
                            w = 0.0;
#pragma unroll
                            for (int e = 0; e < N; ++e) {
                                const int nu = PT::nur(e) - PT::nuf(e), k = ent_spec(h.ent[e]);
                                if (nu) w = e == 0 ? nux(nu, vt[k]) : addnu(w, nu, vt[k]);
                            }
                        }
                        const bool hasns = (h.flags & RX_HASNS) && !approx;
                        if (JAC) {
                            put(w);
                            put(o.net);
                            put(o.d0);
#pragma unroll
                            for (int e = 0; e < N; ++e) put(o.g[e]);
                            if (hasns) put(o.gns);
                            put(o.d1);
                            if (h.flags & RX_WEREAL) put(ldg(h.p + P_WE));
                        } else {
                            put(o.net);
#pragma unroll
                            for (int e = 0; e < N; ++e) put(w * o.g[e]);
                            if (hasns) vNS = fma(w, o.gns, vNS);
                            vout0 = fma(w, o.d0, vout0);
                            vout1 = fma(w, o.d1, vout1);
                        }
                    };
                    // the general code: third-body and fall-off reactions of the
                    // patterns TpP0..TpP2 compiled per pattern, the rest reading
                    // their coefficients
                    auto general = [&](auto tag) {
                        using ST = decltype(tag);
                        RxnHead h;
                        load_head(R, h);
                        RxnTerms o;
                        rxn_terms<DER, ST>(h, a.aux, a.thd_spec, a.thd_coef, last, sv, conc, bk, ep, em, hk, ml, o);
                        if (!DER) {
                            put(o.net);
                            return;
                        }
                        const int nsp = ST::nsp(h), thd = RX_THD(h.flags);
                        double w = o.w;
                        if (VJP) {
                            w = 0.0;
#pragma unroll
                            for (int e = 0; e < PJG_MAXSP; ++e) {
                                if (e >= nsp) break;
                                const int nu = ST::nur(h, e) - ST::nuf(h, e);
                                if (nu != 0) w = addnu(w, nu, vt[ent_spec(h.ent[e])]);
                            }
                        }
                        const bool hasns = (h.flags & RX_HASNS) && !approx;
                        if (JAC) {
                            put(w);
                            put(o.net);
                            put(o.d0);
                            // d R / d c_j times the pressure modification (exactly 1
                            // without a third body)
#pragma unroll
                            for (int e = 0; e < PJG_MAXSP; ++e) {
                                if (e >= nsp) break;
                                put(thd ? __dmul_rn(o.g[e], o.ci_) : o.g[e]);
                            }
                            if (hasns) put(o.gns * o.ci_);
                            put(o.d1);
                            if (thd && h.list >= 0) put(o.X);
                            else if (thd)
                                for (int l = 0; l < h.thd_cnt; ++l) put(__dmul_rn(__ldg(a.thd_coef + h.thd_off + l), o.X));
                            if (h.flags & RX_WEREAL) put(ldg(h.p + P_WE));
                        } else {
                            put(o.net);
                            const double wc = w * o.ci_;
#pragma unroll
                            for (int e = 0; e < PJG_MAXSP; ++e) {
                                if (e >= nsp) break;
                                put(wc * o.g[e]);
                            }
                            if (thd && h.list >= 0) put(w * o.X);
                            else if (thd)
                                for (int l = 0; l < h.thd_cnt; ++l) {
                                    const double x = __dmul_rn(__ldg(a.thd_coef + h.thd_off + l), w * o.X);
                                    put(x);
                                    if (__ldg(a.thd_spec + h.thd_off + l) == last && !approx) vNS = vNS + x;
                                }
                            if (hasns) vNS = fma(wc, o.gns, vNS);
                            vout0 = fma(w, o.d0, vout0);
                            vout1 = fma(w, o.d1, vout1);
                        }
                    };
                    switch (task.x) {
                    case 1: ma(MaP0{}); break;
                    case 2: ma(MaP1{}); break;
                    case 3: ma(MaP2{}); break;
                    case 4: ma(MaP3{}); break;
                    case 5: ma(MaP4{}); break;
                    case 6: ma(MaP5{}); break;
                    case 7: ma(MaP6{}); break;
                    case 8: ma(MaP7{}); break;
                    case 9: ma(MaP8{}); break;
                    case 10: ma(MaP9{}); break;
                    case 11: general(PatStoich<TpP0>{}); break;
                    case 12: general(PatStoich<TpP1>{}); break;
                    case 13: general(PatStoich<TpP2>{}); break;
                    default: general(RunStoich{}); break;
                    }
                }
            }
            // the batch's additions
            int qs[RUN_N];
#pragma unroll
            for (int r = 0; r < RUN_N; ++r) qs[r] = __ldg(off + 1 + r);
            const char* src = reinterpret_cast<const char*>(buf + (bt & 1 ? a.sc.buf_terms << slog : 0));
            auto term = [&](unsigned o) -> double { return *reinterpret_cast<const double*>(src + o); };
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // (the barrier also shows a warp's staged items to its other lanes)
            int q = q_begin, limit = q_begin + cap;
            auto run = [&](auto kind, int q1) {
                constexpr int R = decltype(kind)::value;
                constexpr bool VEC = R != RUN_SLOT && R != RUN_SLOT_FIRST;
                constexpr bool FIRST = R == RUN_SLOT_FIRST || R == RUN_VEC_FIRST || R == RUN_PROD_FIRST;
#pragma unroll 1
                for (; q < q1; q += kItemUnroll) {
                    if (q == limit) {  // the next items of a long batch
                        __syncwarp(own_lanes);
                        fill(q);
                        asm volatile("cp.async.wait_all;" ::: "memory");
                        __syncwarp(own_lanes);
                        limit = q + cap;
                    }
                    uint2 it[kItemUnroll];
#pragma unroll
                    for (int e = 0; e < kItemUnroll; e += 2) {
                        const uint4 w = *reinterpret_cast<const uint4*>(stage + (q - limit + cap) + e);
                        it[e] = make_uint2(w.x, w.y);
                        it[e + 1] = make_uint2(w.z, w.w);
                    }
                    double x[kItemUnroll];
#pragma unroll
                    for (int e = 0; e < kItemUnroll; ++e) {
                        x[e] = term(it[e].y & kItemOff);
                        if (R == RUN_PROD || R == RUN_PROD_FIRST)
                            x[e] = __dmul_rn(term((it[e].y & kItemOff) - (item_q(it[e].y) << (slog + 3))), x[e]);
                        else if (R == RUN_GENERAL)
                            x[e] = nux(item_q(it[e].y), x[e]);
                        else
                            x[e] = __hiloint2double(__double2hiint(x[e]) ^ (it[e].y & 0x80000000u), __double2loint(x[e]));
                    }
#pragma unroll
                    for (int e = 0; e < kItemUnroll; ++e) {
                        if (R == RUN_GENERAL) {
                            apply(it[e].x, x[e]);
                        } else {
                            const uint64_t p = VEC ? vec_g + (uint64_t)it[e].x * (8u << slog)
                                                   : acc_g + (uint64_t)it[e].x * ld_bytes;
                            if (FIRST) st_global(p, x[e]);
                            else red_global(p, x[e]);
                        }
                    }
                }
            };
            if (JAC) run(std::integral_constant<int, RUN_SLOT_FIRST>{}, qs[RUN_SLOT_FIRST]);
            run(std::integral_constant<int, RUN_VEC_FIRST>{}, qs[RUN_VEC_FIRST]);
            if (JAC) run(std::integral_constant<int, RUN_SLOT>{}, qs[RUN_SLOT]);
            run(std::integral_constant<int, RUN_VEC>{}, qs[RUN_VEC]);
            if (JAC) {
                run(std::integral_constant<int, RUN_PROD_FIRST>{}, qs[RUN_PROD_FIRST]);
                run(std::integral_constant<int, RUN_PROD>{}, qs[RUN_PROD]);
            }
            run(std::integral_constant<int, RUN_GENERAL>{}, qs[RUN_GENERAL]);
        }
        __threadfence();
        __syncthreads();

        // ------------------------ third-body columns, temperature and E rates
        const int post_end = __ldg(a.sc.post_off + wk + 1);
        for (int q0 = __ldg(a.sc.post_off + wk); q0 < post_end; q0 += kPostUnroll) {
            int4 it[kPostUnroll];
            double x[kPostUnroll];
#pragma unroll
            for (int e = 0; e < kPostUnroll; ++e)
                it[e] = __ldg(reinterpret_cast<const int4*>(a.sc.post + (q0 + e < post_end ? q0 + e : post_end - 1)));
#pragma unroll
            for (int e = 0; e < kPostUnroll; ++e) x[e] = __ldcg(vec + (it[e].x << slog));
#pragma unroll
            for (int e = 0; e < kPostUnroll; ++e)
                if (q0 + e < post_end) apply((unsigned)it[e].y, __dmul_rn(__hiloint2double(it[e].w, it[e].z), x[e]));
        }
        // Sums over species: n_parts workers take every n_parts-th species each,
        // then one adds their partial sums, so the order does not depend on the
        // tile's shape.
        const int n_parts = sum_parts(ns);
        enum { R_UPPER = 0, R_LOWER, R_DE, R_DT, R_DT1, R_A, R_RATE = R_A, R_SUMT, R_SPEC, R_SUME, R_NST, R_NSE, R_N };
        double* parts = red + (R_N << slog) + st;
        auto rsum = [&](int which) -> double& { return red[(which << slog) + st]; };
        auto part = [&](int which, int w) -> double& { return parts[((which < R_A ? which : which - R_A) * kParts + w) << slog]; };
        if (wk < n_parts) {
            double upper = 0.0, lower = 0.0, dE = 0.0, dT = 0.0, dT1 = 0.0;
#pragma unroll 2
            for (int k = wk; k < ns; k += n_parts) {
                const double w_k = rd(VEC_WDOT, k), cpk = rd(VEC_CP, k), ck = conc[k];
                upper = fma(rd(VEC_H, k), w_k, upper);
                lower = fma(ck, cpk, lower);
                dE = fma(ldg(a.sp + (int64_t)k * PJG_SP_DOUBLES + SP_OMW), w_k, dE);  // omw of the bath gas is 0
                if (DER) {
                    // (cp_ns / T - dcp_k) c_k, (cp_k - cp_ns) c_k
                    dT = fma(cp_ns * Tjinv - rd(VEC_DCP, k), ck, dT);
                    dT1 = fma(cpk - cp_ns, ck, dT1);
                }
            }
            part(R_UPPER, wk) = upper;
            part(R_LOWER, wk) = lower;
            part(R_DE, wk) = dE;
            if (DER) {
                part(R_DT, wk) = dT;
                part(R_DT1, wk) = dT1;
            }
        }
        auto combine = [&](int from, int to) {
            __syncthreads();
            const int q = from + wk;
            if (q < to) {
                double x = part(q, 0);
                for (int w = 1; w < n_parts; ++w) x = x + part(q, w);
                rsum(q) = q == R_LOWER ? 1.0 / x : x;
            }
        };
        if (VJP) {
            // the workers' sums of columns T, E and of the bath-gas terms
            double* own = parts + ((R_A * kParts) << slog);
            const int stride = G << slog;
            own[wk << slog] = vout0;
            own[stride + (wk << slog)] = vout1;
            own[2 * stride + (wk << slog)] = vNS;
        }
        if (JAC) __threadfence();
        combine(R_UPPER, DER ? R_A : R_DT);
        __syncthreads();
        const double inv_cp = rsum(R_LOWER);
        const double Tdot = -rsum(R_UPPER) * inv_cp;
        const double Vval = fmax(1e-30, V);
        if (a.dphi && live) {
            double* o = a.dphi + s * a.dphi_ss;
            if (wk == 0) {
                const double dE = rsum(R_DE);
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
            }
            for (int k = wk; k < last; k += G) o[(int64_t)(2 + k) * a.dphi_sj] = Vval * rd(VEC_WDOT, k);
        }
        if (VJP) {
            // constant parts of columns T and E (from rows T, E of dTdot_dT :1847,
            // dEdotdT :2001, dTdotdE :1595, dEdotdE :1740) and the species columns'
            // bath-gas and d cp_tot / dn_j terms
            const double* own = parts + ((R_A * kParts) << slog);
            const int stride = G << slog;
            const double ct = cp_tot_v;
            double* o = a.vjp + s * a.phi_ss;
            double sNS = 0.0;
            for (int q = 0; q < G; ++q) sNS = sNS + own[2 * stride + (q << slog)];
            for (int q = 0; q < a.n_ns_post; ++q)
                sNS = fma(__ldg(&a.ns_post[q].coef), __ldcg(vec + (__ldg(&a.ns_post[q].src) << slog)), sNS);
            if (wk == 0) {
                const double extra = conp ? V : P;
                double s0 = 0.0, s1 = 0.0;
                for (int q = 0; q < G; ++q) {
                    s0 = s0 + own[q << slog];
                    s1 = s1 + own[stride + (q << slog)];
                }
                s0 = s0 * (V * Tjinv);  // the reactions' terms of column T leave V / T out
                double wsum = 0.0, omws = 0.0, hws = 0.0, vws = 0.0;
                for (int k = 0; k < last; ++k) {
                    const double* rec = a.sp + (int64_t)k * PJG_SP_DOUBLES;
                    const double mw = ldg(rec + SP_MW), omw = ldg(rec + SP_OMW);
                    const double wkk = rd(VEC_WDOT, k), cpk = rd(VEC_CP, k);
                    wsum = wsum + wkk * (-cpk + mw * cp_ns);
                    omws = fma(omw, wkk, omws);
                    hws = fma(rd(VEC_H, k) - h_ns * mw, wkk, hws);
                    vws = fma(vt[k], wkk, vws);
                }
                if (conp) s1 = s1 - vws;  // the reactions' -net of column E
                const double C0 = vt_c0 * (Tdot * rsum(R_DT) + wsum) / ct - v1 * extra * Tdot * Tjinv * Tjinv +
                                  v1 * RU * (conp ? V / P : 1.0) * omws;
                double C1 = conp ? vt_c0 * (Tdot * rsum(R_DT1) + hws) / (ct * V)
                                 : -vt_c0 * Tdot * cp_ns * rt_inv / ct;
                C1 += v1 * Tdot * Tjinv;
                if (live) {
                    o[0] = s0 + C0;
                    o[a.phi_sj] = s1 + C1;
                }
            }
            const double gam = -vt_c0 * Tdot / (V * ct);
            if (live)
                for (int j = wk; j < last; j += G)
                    o[(int64_t)(2 + j) * a.phi_sj] = rd(VEC_NS, j) - sNS + gam * (rd(VEC_CP, j) - cp_ns);
        }
        if (JAC) {
            // ------------------------------------------- assemble rows T and E
            // Both rows are linear in the species rows, so each reaction has added
            // its share (w_i d R_i / d c_j, with w_i = sum_k nu_ki hw_k for row T
            // and sum_k nu_ki (1 - W_k / W_ns) = sum nu for row E); the bath-gas
            // terms, the same for every species column, take one sum per state.
            const double fixed = conp ? P : V, extra = conp ? V : P;
            const double Vjinv = V >= 1e-30 ? Vinv : 1.0 / V;
            const double inv_vcp = Vjinv * inv_cp;
            const double eTj = extra * Tjinv, VTj = V * Tjinv;
            // the bath-gas terms of each row, subtracted from every species column
            for (int q = wk; q < a.n_ns * kNsParts; q += G) {
                const int row = q / kNsParts, j0 = (q - row * kNsParts) * last / kNsParts,
                          j1 = (q - row * kNsParts + 1) * last / kNsParts;
                const double mv = negi(rd(VEC_NS, __ldg(a.ns_rows + row)));
                if (!nonzero(mv)) continue;
                const int* sl = a.ns_slots + row * last;
#pragma unroll 8
                for (int j = j0; j < j1; ++j) {
                    const int t = __ldg(sl + j);
                    if (t >= 0) red_global(acc_g + (uint64_t)(unsigned)t * ld_bytes, mv);
                }
            }
            // T column of rows T, E and E column of rows T, E; column E of a
            // species row: at constant pressure the terms leave out -net of each
            // reaction, in sum -wdot_k
            if (wk < n_parts) {
                double rate_sum = 0.0, sumT = 0.0, spec1 = 0.0, sumE1 = 0.0, nsT = 0.0, nsE = 0.0;
#pragma unroll 2
                for (int k = wk; k < last; k += n_parts) {
                    const double* rec = a.sp + (int64_t)k * PJG_SP_DOUBLES;
                    const double mw = ldg(rec + SP_MW), omw = ldg(rec + SP_OMW);
                    const double w_k = rd(VEC_WDOT, k), cpk = rd(VEC_CP, k), hwk = fma(-h_ns, mw, hk[k]);
                    const double vk = __ldg(a.sp_slots + 2 * k) >= 0 ? rd(VEC_CT, k) * Tjinv : 0.0;  // J_kT / V
                    const double ce = rd(VEC_CE, k);
                    const double Jk1 = __ldg(a.sp_slots + 2 * k + 1) >= 0 ? (conp ? ce - w_k : ce) : 0.0;
                    rate_sum = fma(-vk, hwk, rate_sum);
                    rate_sum = fma(w_k, fma(mw, cp_ns, -cpk), rate_sum);
                    sumT = fma(omw, conp ? fma(Tjinv, w_k, vk) : fma(T, vk, w_k), sumT);
                    spec1 = fma(hwk, conp ? Jk1 - w_k : Jk1, spec1);
                    sumE1 = fma(omw, Jk1, sumE1);
                }
                for (int q = wk; q < a.n_ns; q += n_parts) {
                    const int k = __ldg(a.ns_rows + q);
                    const double v = rd(VEC_NS, k);
                    nsT = fma(fma(-h_ns, ldg(a.sp + (int64_t)k * PJG_SP_DOUBLES + SP_MW), hk[k]), v, nsT);
                    nsE = fma(ldg(a.sp + (int64_t)k * PJG_SP_DOUBLES + SP_OMW), v, nsE);
                }
                part(R_RATE, wk) = rate_sum;
                part(R_SUMT, wk) = sumT;
                part(R_SPEC, wk) = spec1;
                part(R_SUME, wk) = sumE1;
                part(R_NST, wk) = nsT;
                part(R_NSE, wk) = nsE;
            }
            for (int k = wk; k < last; k += G) {
                const int sl0 = __ldg(a.sp_slots + 2 * k), sl1 = __ldg(a.sp_slots + 2 * k + 1);
                if (sl0 >= 0) accs[(int64_t)sl0 * acc_ld] = rd(VEC_CT, k) * VTj;
                if (sl1 >= 0) accs[(int64_t)sl1 * acc_ld] = conp ? rd(VEC_CE, k) - rd(VEC_WDOT, k) : rd(VEC_CE, k);
            }
            const bool summed = a.col_list == nullptr;
            if (!summed) __threadfence();  // the species block is read back below
            combine(R_A, R_N);
            __syncthreads();
            const double TRf = T * RU / fixed;
            for (int j = wk; j < last; j += G) {
                double sT, sE;
                if (summed) {
                    sT = rd(VEC_RT, j) - rsum(R_NST);
                    sE = rd(VEC_RE, j) - rsum(R_NSE);
                } else {
                    sT = 0.0;
                    sE = 0.0;
                    const int c0 = __ldg(a.col_off + j), c1 = __ldg(a.col_off + j + 1);
                    for (int q = c0; q < c1; ++q) {
                        const int2 e = __ldg(a.col_list + q);
                        const double Jkj = __ldcg(accs + (int64_t)e.y * acc_ld);
                        sT = fma(fma(-h_ns, ldg(a.sp + (int64_t)e.x * PJG_SP_DOUBLES + SP_MW), hk[e.x]), Jkj, sT);
                        sE = fma(ldg(a.sp + (int64_t)e.x * PJG_SP_DOUBLES + SP_OMW), Jkj, sE);
                    }
                }
                const double J0 = -1.0 * (sT + Tdot * (rd(VEC_CP, j) + -1.0 * cp_ns)) * inv_vcp;
                accs[(int64_t)__ldg(a.cj_slots + 2 * j) * acc_ld] = J0;
                accs[(int64_t)__ldg(a.cj_slots + 2 * j + 1) * acc_ld] = TRf * sE + eTj * J0;
            }
            if (wk == 0) {
                const double J00 = (Tdot * rsum(R_DT) + rsum(R_RATE)) * inv_cp;
                double J10;
                if (conp) {
                    J10 = V * Tjinv * (J00 - Tjinv * Tdot);
                    J10 = J10 + RU * T * V * rsum(R_SUMT) / P;
                } else {
                    J10 = P * (J00 - Tdot * Tjinv) * Tjinv;
                    J10 = J10 + RU * rsum(R_SUMT);
                }
                double J01;
                if (conp) {
                    J01 = (Tdot * rsum(R_DT1) - rsum(R_SPEC)) * inv_vcp;
                } else {
                    J01 = -((Tdot * cp_ns * rt_inv) * inv_cp);
                    J01 = J01 - (rsum(R_SPEC) * Vjinv) * inv_cp;
                }
                double J11 = TRf * rsum(R_SUME);
                J11 = J11 + (extra * J01 + Tdot) * Tjinv;
                accs[(int64_t)a.s00 * acc_ld] = J00;
                accs[(int64_t)a.s10 * acc_ld] = J10;
                accs[(int64_t)a.s01 * acc_ld] = J01;
                accs[(int64_t)a.s11 * acc_ld] = J11;
            }
        }
    }
}

}  // namespace

size_t pjg_tile_smem(int kind, int ns, int n_m, int slog, int buf_terms)
{
    return kTileStatic + stage_bytes(slog) +
           (((size_t)tile_arrays(kind) * ns + 2 * (size_t)n_m + 2 * (size_t)buf_terms) << slog) * sizeof(double);
}

namespace {

const void* kernel_of(int kind)
{
    return kind == KIND_JAC ? (const void*)tile_kernel<KIND_JAC>
           : kind == KIND_VJP ? (const void*)tile_kernel<KIND_VJP> : (const void*)tile_kernel<KIND_RATES>;
}


}  // namespace

int pjg_tile_blocks_per_sm(int kind, size_t smem)
{
    int b = 0;
    const void* fn = kernel_of(kind);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, 32 * kTileWarps, smem) != cudaSuccess)
        return 1;
    return b > 0 ? b : 1;
}

int pjg_launch_tile(const EvalArgs& a, int kind, int grid, void* stream)
{
    if (a.n <= 0) return 0;
    const cudaStream_t st = (cudaStream_t)stream;
    const size_t smem = pjg_tile_smem(kind, a.ns, a.n_m, a.sc.slog, a.sc.buf_terms);
    const int threads = 32 * kTileWarps;
    pjg_launch_err = cudaFuncSetAttribute(kernel_of(kind), cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    if (pjg_launch_err != cudaSuccess) return -2;
    if (kind == KIND_JAC) tile_kernel<KIND_JAC><<<grid, threads, smem, st>>>(a);
    else if (kind == KIND_VJP) tile_kernel<KIND_VJP><<<grid, threads, smem, st>>>(a);
    else tile_kernel<KIND_RATES><<<grid, threads, smem, st>>>(a);
    pjg_launch_err = cudaGetLastError();
    return pjg_launch_err == cudaSuccess ? 0 : -2;
}
