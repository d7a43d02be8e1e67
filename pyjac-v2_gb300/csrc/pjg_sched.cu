// Work schedules of the evaluation kernels (host code): which worker of a
// tile's block evaluates which reaction when, and which worker makes which
// addition (Schedule, pjg_eval.cuh).
//
// Reactions are taken in packed order: a task is up to 32 / S consecutive
// reactions of one class (one warp's workers run the same code), a batch up to
// rounds * W consecutive tasks whose terms fit the buffer.  All additions to
// one target stay with one worker, in reaction order, so that every sum has
// that order whatever the tile's shape; the targets go to the least-loaded
// worker, longest first.
#include <algorithm>
#include <cmath>
#include <map>
#include <queue>
#include <set>

#include "pjg_eval.cuh"

namespace {

struct Item {
    unsigned target;
    int t, q;   // term; factor, or the second term's distance
    bool prod;
};

// workers of targets (dense numbers) by their numbers of additions
void deal(const std::vector<int>& count, int G, std::vector<int>& owner)
{
    std::vector<std::pair<int, int>> by;
    for (int t = 0; t < (int)count.size(); ++t)
        if (count[t]) by.push_back({-count[t], t});
    std::sort(by.begin(), by.end());
    std::priority_queue<std::pair<int, int>, std::vector<std::pair<int, int>>, std::greater<std::pair<int, int>>> load;
    for (int g = 0; g < G; ++g) load.push({0, g});
    owner.assign(count.size(), 0);
    for (auto& x : by) {
        auto [n, g] = load.top();
        load.pop();
        owner[x.second] = g;
        load.push({n - x.first, g});
    }
}

}  // namespace

bool sched_build(const SchedInput& in, int slog, int warps, int rounds, int buf_terms, SchedHost& o)
{
    const int S = 1 << slog, wpw = 32 / S, G = warps * wpw;
    const int ns = in.ns, last = ns - 1, kind = in.kind;
    const std::vector<RxnRec>& rx = *in.rxn;
    const int nr = (int)rx.size();
    const bool jac = kind == KIND_JAC, vjp = kind == KIND_VJP;
    o.slog = slog;
    o.warps = warps;
    o.rounds = rounds;
    o.buf_terms = buf_terms;
    o.n_vec = vec_arrays(kind) * ns;

    // third-body sums: one per (list, species row) and two per list (Jacobian:
    // rows T and E), one per list (J^T v)
    std::map<std::pair<int, int>, unsigned> sum_of;  // (list offset, row; ns: row T, ns + 1: row E)
    auto tb_sum = [&](int list, int row) -> unsigned {
        auto it = sum_of.find({list, row});
        if (it != sum_of.end()) return it->second;
        return sum_of[{list, row}] = (unsigned)o.n_vec++;
    };
    std::vector<char> seen_vec;  // marks of scratch entries added to
    std::vector<char> seen_slot;
    if (jac) {
        int top = 0;
        for (int sl : *in.slot) top = std::max(top, sl + 1);
        seen_slot.assign(top, 0);
    }
    auto first = [&](unsigned t) -> unsigned {
        std::vector<char>& seen = (t & TGT_VEC) ? seen_vec : seen_slot;
        const unsigned i = t & TGT_MASK;
        if (i >= seen.size()) seen.resize(2 * i + 1, 0);  // scratch entries
        if (seen[i]) return t;
        seen[i] = 1;
        return t | TGT_FIRST;
    };
    auto vec_t = [&](int v, int k) -> unsigned { return TGT_VEC | (unsigned)(v * ns + k); };
    auto slot_of = [&](int k, int j) -> int { return (*in.slot)[(size_t)k * last + j]; };

    auto has_ns = [&](const RxnRec& R) { return (R.flags & RX_HASNS) && !in.jac_approx; };
    auto terms_of = [&](const RxnRec& R) {
        if (vjp) return 1 + R.nspec + rxn_x_terms(R);
        if (!jac) return 1;
        return 3 + R.nspec + (has_ns(R) ? 1 : 0) + (rxn_has_d1(R.flags) ? 1 : 0) + rxn_x_terms(R) +
               ((R.flags & RX_WEREAL) ? 1 : 0);
    };

    o.term_off.assign(std::max(nr, 1), 0);
    std::vector<std::vector<Item>> batches;
    const int n_slot = jac ? (int)seen_slot.size() : 0;
    auto dense = [&](unsigned t) { return (int)(t & TGT_MASK) + ((t & TGT_VEC) ? n_slot : 0); };
    std::set<unsigned> general;  // targets with a factor other than 1 and -1
    int i = 0;
    while (i < nr) {
        // one batch
        int terms = 1, b0 = i;  // term 0 is zero
        std::vector<int4> tasks;
        while (i < nr && (int)tasks.size() < warps * rounds) {
            const int cl = (*in.cls)[i];
            int cnt = 0, t = 0;
            while (cnt < wpw && i + cnt < nr && (*in.cls)[i + cnt] == cl) {
                const int q = terms_of(rx[i + cnt]);
                if (terms + t + q > buf_terms) break;
                t += q;
                ++cnt;
            }
            if (!cnt) break;
            int off = terms;
            for (int e = 0; e < cnt; ++e) {
                o.term_off[i + e] = off;
                off += terms_of(rx[i + e]);
            }
            tasks.push_back(make_int4(cl, i, cnt, 0));
            terms = off;
            i += cnt;
        }
        if (tasks.empty()) return false;  // one reaction's terms pass the buffer
        while ((int)tasks.size() < warps * rounds) tasks.push_back(make_int4(0, 0, 0, 0));
        o.tasks.insert(o.tasks.end(), tasks.begin(), tasks.end());
        ++o.n_batch;
        // its additions
        std::vector<Item> items;
        auto scaled = [&](unsigned target, int t, int q) {
            items.push_back({target, t, q, false});
            if (q != 1 && q != -1) general.insert(target);
        };
        auto product = [&](unsigned target, int t, int t2) {
            items.push_back({target, t, t - t2, true});
        };
        for (int r = b0; r < i; ++r) {
            const RxnRec& R = rx[r];
            const int n = R.nspec, base = o.term_off[r];
            const int n_x = rxn_x_terms(R);  // 1: summed per list; else one per entry of the list
            const bool thd = n_x > 0, summed = R.list >= 0;
            const int t_net = jac ? base + 1 : base, t_g = jac ? base + 3 : base + 1;
            int sp[PJG_MAXSP], nu[PJG_MAXSP], nu_sum = 0;
            bool zero[PJG_MAXSP];  // d net / d c_j is zero by itself
            for (int e = 0; e < n; ++e) {
                sp[e] = ent_spec(R.ent[e]);
                nu[e] = ent_nur(R.ent[e]) - ent_nuf(R.ent[e]);
                nu_sum += nu[e];
                zero[e] = !(R.flags & RX_REV) && ent_nuf(R.ent[e]) == 0;
                if (nu[e]) scaled(vec_t(VEC_WDOT, sp[e]), t_net, nu[e]);
            }
            o.wave_slot_off.push_back((int)o.wave_slots.size());
            o.wave_tb_off.push_back((int)o.wave_tb.size());
            if (vjp) {
                if (summed) o.wave_tb.push_back((int)tb_sum(R.thd_off, 0));
                for (int e = 0; e < n; ++e)
                    if (sp[e] != last && !zero[e]) scaled(vec_t(VEC_NS, sp[e]), t_g + e, 1);
                if (summed) scaled(TGT_VEC | tb_sum(R.thd_off, 0), t_g + n, 1);
                else
                    for (int l = 0; l < n_x; ++l)
                        if ((*in.thd_spec)[R.thd_off + l] != last && (*in.thd_coef)[R.thd_off + l] != 0.0)
                            scaled(vec_t(VEC_NS, (*in.thd_spec)[R.thd_off + l]), t_g + n + l, 1);
            }
            if (!jac) continue;
            int t = t_g + n;
            const int t_ns = has_ns(R) ? t++ : -1, t_d1 = rxn_has_d1(R.flags) ? t++ : -1,
                      t_x = t, t_we = t + n_x;
            const bool we_term = R.flags & RX_WEREAL;
            if (summed) {
                for (int a = 0; a < n; ++a)
                    o.wave_tb.push_back(sp[a] == last || !nu[a] ? -1 : (int)tb_sum(R.thd_off, sp[a]));
                o.wave_tb.push_back((int)tb_sum(R.thd_off, ns));
                o.wave_tb.push_back(R.flags & RX_WE ? (int)tb_sum(R.thd_off, ns + 1) : -1);
            }
            // the thread-per-state kernel's slots: per participant, one per
            // participant and one per entry of an unshared third-body list
            const int n_l = summed ? 0 : n_x, row = n + n_l;
            o.wave_slots.resize(o.wave_slots.size() + n * row, TGT_MASK);
            unsigned* wave = o.wave_slots.data() + o.wave_slots.size() - n * row;
            for (int a = 0; a < n; ++a) {
                if (sp[a] == last || !nu[a]) continue;
                for (int e = 0; e < n; ++e) {
                    if (sp[e] == last || zero[e]) continue;
                    if (slot_of(sp[a], sp[e]) >= 0) wave[a * row + e] = (unsigned)slot_of(sp[a], sp[e]);
                    const int sl = slot_of(sp[a], sp[e]);
                    if (sl < 0) o.left_out = true;
                    else scaled((unsigned)sl, t_g + e, nu[a]);
                }
                scaled(vec_t(VEC_CT, sp[a]), base + 2, nu[a]);
                if (t_d1 >= 0) scaled(vec_t(VEC_CE, sp[a]), t_d1, nu[a]);
                if (t_ns >= 0) scaled(vec_t(VEC_NS, sp[a]), t_ns, nu[a]);
                if (summed) scaled(TGT_VEC | tb_sum(R.thd_off, sp[a]), t_x, nu[a]);
                for (int l = 0; l < n_l; ++l) {
                    const int j = (*in.thd_spec)[R.thd_off + l];
                    if ((*in.thd_coef)[R.thd_off + l] == 0.0) continue;
                    if (j == last) {
                        if (!in.jac_approx) scaled(vec_t(VEC_NS, sp[a]), t_x + l, nu[a]);
                        continue;
                    }
                    const int sl = slot_of(sp[a], j);
                    if (sl < 0) o.left_out = true;
                    else scaled((unsigned)sl, t_x + l, nu[a]);
                    if (sl >= 0) wave[a * row + n + l] = (unsigned)sl;
                }
            }
            auto row_e = [&](unsigned target, int src) {
                if (!(R.flags & RX_WE)) return;
                if (we_term) product(target, src, t_we);
                else scaled(target, src, nu_sum);
            };
            for (int e = 0; e < n; ++e) {
                if (sp[e] == last || zero[e]) continue;
                product(vec_t(VEC_RT, sp[e]), t_g + e, base);
                row_e(vec_t(VEC_RE, sp[e]), t_g + e);
            }
            if (summed) {
                product(TGT_VEC | tb_sum(R.thd_off, ns), t_x, base);
                if (R.flags & RX_WE) row_e(TGT_VEC | tb_sum(R.thd_off, ns + 1), t_x);
            }
            for (int l = 0; l < n_l; ++l) {
                const int j = (*in.thd_spec)[R.thd_off + l];
                if ((*in.thd_coef)[R.thd_off + l] == 0.0 || j == last) continue;
                product(vec_t(VEC_RT, j), t_x + l, base);
                row_e(vec_t(VEC_RE, j), t_x + l);
            }
        }
        for (Item& x : items) x.target = first(x.target);
        if (jac) {  // the same marks in the thread-per-state kernel's slots
            size_t q = 0;
            for (int r = b0; r < i; ++r)
                for (int e = o.wave_slot_off[r]; e < (r + 1 < (int)o.wave_slot_off.size() ? o.wave_slot_off[r + 1] : (int)o.wave_slots.size()); ++e) {
                    unsigned& sl = o.wave_slots[e];
                    if (sl == TGT_MASK) continue;
                    while (items[q].prod || (items[q].target & TGT_VEC) || (items[q].target & TGT_MASK) != sl) ++q;
                    sl = items[q++].target;
                }
        }
        batches.push_back(std::move(items));
    }
    // the third-body columns, after the reactions: coefficient x sum
    std::vector<PostItem> post;
    std::map<int, int> lists;  // offset -> reaction with that list
    for (int r = 0; r < nr; ++r)
        if (rx[r].list >= 0) lists.emplace(rx[r].thd_off, r);
    for (auto& kv : sum_of) {
        const RxnRec& R = rx[lists[kv.first.first]];
        const int row = kv.first.second;
        for (int l = R.thd_off; l < R.thd_off + R.thd_cnt; ++l) {
            const int j = (*in.thd_spec)[l];
            const double c = (*in.thd_coef)[l];
            if (c == 0.0) continue;
            if (j == last) {
                if (in.jac_approx) continue;
                if (vjp) o.ns_post.push_back({kv.second, 0u, c});
                else if (row < last) post.push_back({kv.second, vec_t(VEC_NS, row), c});
                continue;
            }
            if (vjp) {
                post.push_back({kv.second, vec_t(VEC_NS, j), c});
            } else if (row < last) {
                const int sl = slot_of(row, j);
                if (sl < 0) o.left_out = true;
                else post.push_back({kv.second, (unsigned)sl, c});
            } else if (row >= ns) {
                post.push_back({kv.second, vec_t(row == ns ? VEC_RT : VEC_RE, j), c});
            }
        }
    }
    for (PostItem& x : post) x.target = first(x.target);
    o.wave_post = post;
    // what nothing is added to is set to zero by items of term 0, spread over
    // the batches
    if (batches.empty()) {
        batches.emplace_back();
        o.tasks.assign(warps * rounds, make_int4(0, 0, 0, 0));
        o.n_batch = 1;
    }
    size_t next_batch = 0;
    auto zero = [&](unsigned target) {
        if (!(first(target) & TGT_FIRST)) return;
        batches[next_batch++ % batches.size()].push_back({target | TGT_FIRST, 0, 1, false});
    };
    std::vector<int> vecs = {VEC_WDOT};
    if (vjp) vecs.push_back(VEC_NS);
    if (jac) vecs.insert(vecs.end(), {VEC_NS, VEC_RT, VEC_RE, VEC_CT, VEC_CE});
    for (int v : vecs)
        for (int k = 0; k < ns; ++k) zero(vec_t(v, k));
    if (jac)
        for (int sl : *in.slot)
            if (sl >= 0) {
                if (!seen_slot[sl]) o.wave_zero.push_back((unsigned)sl);
                zero((unsigned)sl);
            }
    std::vector<int> count(n_slot + o.n_vec, 0), owner;
    size_t n_items = 0;
    for (const auto& items : batches) {
        for (const Item& x : items) ++count[dense(x.target)];
        n_items += items.size();
    }
    deal(count, G, owner);
    const unsigned unread = (unsigned)o.n_vec++;  // the slice's last entry
    // a batch's items by worker and run, each run in order (a counting sort)
    o.item_off.assign(1, 0);
    o.items.reserve(n_items * 5 / 4 + 64);
    std::vector<int> at(G * RUN_N + 1), key;
    std::vector<int> sorted;
    for (const auto& items : batches) {
        key.resize(items.size());
        sorted.resize(items.size());
        std::fill(at.begin(), at.end(), 0);
        for (size_t i = 0; i < items.size(); ++i) {
            const Item& x = items[i];
            const bool fi = x.target & TGT_FIRST, vec = x.target & TGT_VEC;
            const int run = x.prod ? (fi ? RUN_PROD_FIRST : RUN_PROD)
                            : !general.empty() && general.count(x.target & ~TGT_FIRST) ? RUN_GENERAL
                            : vec ? (fi ? RUN_VEC_FIRST : RUN_VEC) : (fi ? RUN_SLOT_FIRST : RUN_SLOT);
            key[i] = owner[dense(x.target)] * RUN_N + run;
            ++at[key[i] + 1];
        }
        for (size_t q = 1; q < at.size(); ++q) at[q] += at[q - 1];
        std::vector<int> put(at.begin(), at.end() - 1);
        for (size_t i = 0; i < items.size(); ++i) sorted[put[key[i]]++] = (int)i;
        for (int q = 0; q < G * RUN_N; ++q) {
            const int r = q % RUN_N;
            const size_t from = o.items.size();
            for (int j = at[q]; j < at[q + 1]; ++j) {
                const Item& x = items[sorted[j]];
                const unsigned idx = x.target & TGT_MASK, off = (unsigned)(x.t * S * (int)sizeof(double));
                if (r == RUN_PROD || r == RUN_PROD_FIRST)
                    o.items.push_back(make_uint2(idx, off | (((unsigned)x.q & 0x7ffu) << 20)));
                else if (r == RUN_GENERAL)
                    o.items.push_back(make_uint2(x.target, off | (((unsigned)x.q & 0x7ffu) << 20)));
                else
                    o.items.push_back(make_uint2(idx, off | (x.q < 0 ? 1u << 31 : 0u)));
            }
            while ((o.items.size() - from) % kItemUnroll)
                o.items.push_back(r == RUN_SLOT_FIRST ? o.items.back() : r == RUN_SLOT ? make_uint2(o.items.back().x, 0u)
                                  : r == RUN_GENERAL ? make_uint2(unread | TGT_VEC | TGT_FIRST, 1u << 20) : make_uint2(unread, 0u));
            o.item_off.push_back((int)o.items.size());
        }
    }
    o.items.insert(o.items.end(), kItemUnroll, make_uint2(unread, 0u));  // loaded ahead, not used
    std::vector<int> post_count(n_slot + o.n_vec, 0), post_owner;
    for (const PostItem& x : post) ++post_count[dense(x.target)];
    deal(post_count, G, post_owner);
    std::vector<std::vector<PostItem>> of(G);
    for (const PostItem& x : post) of[post_owner[dense(x.target)]].push_back(x);
    o.post_off.assign(1, 0);
    for (const auto& l : of) {
        o.post.insert(o.post.end(), l.begin(), l.end());
        o.post_off.push_back((int)o.post.size());
    }
    return true;
}
