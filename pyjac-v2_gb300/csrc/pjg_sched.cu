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
//
// The additions themselves do not depend on the tile's shape: sched_adds lists
// them once per kind and output layout (the thread-per-state kernel's tables
// among them), sched_build deals them out for one shape.  Both in one cost the
// first Jacobian call of GRI-Mech 3.0 2.1 ms on the host and each further shape
// 0.9, with the 500-species mechanism 137 and 75 (dense; sparse 46 and 20); now
// 0.7 and 0.3, 25 and 12 (sparse 8 and 3.5).
#include <algorithm>
#include <cmath>
#include <map>
#include <queue>

#include "pjg_eval.cuh"

namespace {

// Workers of targets (dense numbers) by their numbers of additions, `order`
// holding the targets longest first: the least-loaded worker, the lowest of
// several.  Where only single additions are left, that is filling level by
// level.
void deal(const std::vector<int>& count, const std::vector<int>& order, int G, std::vector<int>& owner)
{
    std::priority_queue<std::pair<int, int>, std::vector<std::pair<int, int>>, std::greater<std::pair<int, int>>> heap;
    for (int g = 0; g < G; ++g) heap.push({0, g});
    owner.assign(count.size(), 0);
    size_t x = 0;
    for (; x < order.size() && count[order[x]] > 1; ++x) {
        auto [n, g] = heap.top();
        heap.pop();
        owner[order[x]] = g;
        heap.push({n + count[order[x]], g});
    }
    std::vector<int> load(G);
    int level = heap.top().first;
    for (; !heap.empty(); heap.pop()) load[heap.top().second] = heap.top().first;
    for (; x < order.size(); ++level)
        for (int g = 0; g < G && x < order.size(); ++g)
            if (load[g] == level) {
                ++load[g];
                owner[order[x++]] = g;
            }
}

// the targets that something is added to, longest first
std::vector<int> longest_first(const std::vector<int>& count)
{
    int top = 0;
    for (int c : count) top = std::max(top, c);
    std::vector<size_t> at(top + 2, 0);
    for (int c : count) ++at[top - c + 1];
    for (int q = 0; q <= top; ++q) at[q + 1] += at[q];
    std::vector<int> order(at[top]);  // of count >= 1
    for (int t = 0; t < (int)count.size(); ++t)
        if (count[t]) order[at[top - count[t]]++] = t;
    return order;
}

}  // namespace

void sched_adds(const SchedInput& in, SchedAdds& o)
{
    const int ns = in.ns, last = ns - 1, kind = in.kind;
    const std::vector<RxnRec>& rx = *in.rxn;
    const int nr = (int)rx.size();
    const bool jac = kind == KIND_JAC, vjp = kind == KIND_VJP;
    o.kind = kind;
    o.n_vec = vec_arrays(kind) * ns;
    o.cls = *in.cls;

    // third-body sums: one per (list, species row) and two per list (Jacobian:
    // rows T and E), one per list (J^T v)
    std::map<std::pair<int, int>, unsigned> sum_of;  // (list offset, row; ns: row T, ns + 1: row E)
    auto tb_sum = [&](int list, int row) -> unsigned {
        auto it = sum_of.find({list, row});
        if (it != sum_of.end()) return it->second;
        return sum_of[{list, row}] = (unsigned)o.n_vec++;
    };
    o.n_slot = 0;
    if (jac)
        for (int sl : *in.slot) o.n_slot = std::max(o.n_slot, sl + 1);
    std::vector<char> seen_vec, seen_slot(o.n_slot, 0);  // marks of targets added to
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

    std::vector<unsigned> general;  // targets with a factor other than 1 and -1
    auto scaled = [&](unsigned target, int t, int q) {
        o.items.push_back({first(target), t, q, false});
        if (q != 1 && q != -1) general.push_back(target);
    };
    auto product = [&](unsigned target, int t, int t2) {
        o.items.push_back({first(target), t, t - t2, true});
    };
    auto add_slot = [&](int sl, int t, int q, unsigned& wave) {
        if (sl < 0) {
            o.left_out = true;
            return;
        }
        scaled((unsigned)sl, t, q);
        wave = o.items.back().target;
    };
    for (int r = 0; r < nr; ++r) {
        const RxnRec& R = rx[r];
        const int n = R.nspec;
        const int n_x = rxn_x_terms(R);  // 1: summed per list; else one per entry of the list
        const bool summed = R.list >= 0;
        const int t_net = jac ? 1 : 0, t_g = jac ? 3 : 1;
        o.terms.push_back(vjp ? 1 + n + n_x
                          : !jac ? 1
                                 : 3 + n + (has_ns(R) ? 1 : 0) + (rxn_has_d1(R.flags) ? 1 : 0) + n_x +
                                       ((R.flags & RX_WEREAL) ? 1 : 0));
        o.item_off.push_back((int)o.items.size());
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
                add_slot(slot_of(sp[a], sp[e]), t_g + e, nu[a], wave[a * row + e]);
            }
            scaled(vec_t(VEC_CT, sp[a]), 2, nu[a]);
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
                add_slot(slot_of(sp[a], j), t_x + l, nu[a], wave[a * row + n + l]);
            }
        }
        auto row_e = [&](unsigned target, int src) {
            if (!(R.flags & RX_WE)) return;
            if (we_term) product(target, src, t_we);
            else scaled(target, src, nu_sum);
        };
        for (int e = 0; e < n; ++e) {
            if (sp[e] == last || zero[e]) continue;
            product(vec_t(VEC_RT, sp[e]), t_g + e, 0);
            row_e(vec_t(VEC_RE, sp[e]), t_g + e);
        }
        if (summed) {
            product(TGT_VEC | tb_sum(R.thd_off, ns), t_x, 0);
            if (R.flags & RX_WE) row_e(TGT_VEC | tb_sum(R.thd_off, ns + 1), t_x);
        }
        for (int l = 0; l < n_l; ++l) {
            const int j = (*in.thd_spec)[R.thd_off + l];
            if ((*in.thd_coef)[R.thd_off + l] == 0.0 || j == last) continue;
            product(vec_t(VEC_RT, j), t_x + l, 0);
            row_e(vec_t(VEC_RE, j), t_x + l);
        }
    }
    o.item_off.push_back((int)o.items.size());
    // the third-body columns, after the reactions: coefficient x sum
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
                else if (row < last) o.post.push_back({kv.second, vec_t(VEC_NS, row), c});
                continue;
            }
            if (vjp) {
                o.post.push_back({kv.second, vec_t(VEC_NS, j), c});
            } else if (row < last) {
                const int sl = slot_of(row, j);
                if (sl < 0) o.left_out = true;
                else o.post.push_back({kv.second, (unsigned)sl, c});
            } else if (row >= ns) {
                o.post.push_back({kv.second, vec_t(row == ns ? VEC_RT : VEC_RE, j), c});
            }
        }
    }
    for (PostItem& x : o.post) x.target = first(x.target);
    // what nothing is added to is set to zero
    auto zero = [&](unsigned target) {
        if (first(target) & TGT_FIRST) o.zeros.push_back(target);
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
    o.general.assign(general.empty() ? 0 : o.n_slot + o.n_vec, 0);
    for (unsigned t : general) o.general[o.dense(t)] = 1;
    o.count.assign(o.n_slot + o.n_vec, 0);
    for (const SchedAdds::Item& x : o.items) ++o.count[o.dense(x.target)];
    for (unsigned t : o.zeros) ++o.count[o.dense(t)];
    o.order = longest_first(o.count);
    o.unread = (unsigned)o.n_vec++;  // the slice's last entry
}

bool sched_build(const SchedAdds& in, int slog, int rounds, int buf_terms, SchedHost& o)
{
    const int S = 1 << slog, wpw = 32 / S, G = kTileWarps * wpw;
    const int nr = (int)in.terms.size();
    o.n_batch = 0;
    // batches of tasks
    o.term_off.assign(std::max(nr, 1), 0);
    std::vector<int> batch_r = {0};  // first reactions of the batches
    for (int i = 0; i < nr;) {
        int terms = 1, n_tasks = 0;  // term 0 is zero
        while (i < nr && n_tasks < kTileWarps * rounds) {
            const int cl = in.cls[i], i0 = i;
            while (i < nr && i - i0 < wpw && in.cls[i] == cl && terms + in.terms[i] <= buf_terms) {
                o.term_off[i] = terms;
                terms += in.terms[i++];
            }
            if (i == i0) break;
            o.tasks.push_back(make_int4(cl, i0, i - i0, 0));
            ++n_tasks;
        }
        if (!n_tasks) return false;  // one reaction's terms pass the buffer
        o.tasks.resize(o.tasks.size() + kTileWarps * rounds - n_tasks, make_int4(0, 0, 0, 0));
        ++o.n_batch;
        batch_r.push_back(i);
    }
    if (!nr) {  // one empty batch, for the zeros
        o.tasks.assign(kTileWarps * rounds, make_int4(0, 0, 0, 0));
        o.n_batch = 1;
        batch_r.push_back(0);
    }
    std::vector<int> owner;
    deal(in.count, in.order, G, owner);
    // a batch's items by worker and run, each run in order (a counting sort);
    // the zeros are items of term 0, spread over the batches
    o.item_off.assign(1, 0);
    o.items.reserve((in.items.size() + in.zeros.size()) * 5 / 4 + 64);
    std::vector<int> at(G * RUN_N + 1), put, key;
    std::vector<SchedAdds::Item> items, sorted;
    for (int b = 0; b < o.n_batch; ++b) {
        items.clear();
        for (int r = batch_r[b]; r < batch_r[b + 1]; ++r)
            for (int q = in.item_off[r]; q < in.item_off[r + 1]; ++q) {
                items.push_back(in.items[q]);
                items.back().t += o.term_off[r];
            }
        for (size_t q = b; q < in.zeros.size(); q += o.n_batch) items.push_back({in.zeros[q] | TGT_FIRST, 0, 1, false});
        key.resize(items.size());
        sorted.resize(items.size());
        std::fill(at.begin(), at.end(), 0);
        for (size_t i = 0; i < items.size(); ++i) {
            const SchedAdds::Item& x = items[i];
            const bool fi = x.target & TGT_FIRST, vec = x.target & TGT_VEC;
            const int d = in.dense(x.target);
            const int run = x.prod ? (fi ? RUN_PROD_FIRST : RUN_PROD)
                            : !in.general.empty() && in.general[d] ? RUN_GENERAL
                            : vec ? (fi ? RUN_VEC_FIRST : RUN_VEC) : (fi ? RUN_SLOT_FIRST : RUN_SLOT);
            key[i] = owner[d] * RUN_N + run;
            ++at[key[i] + 1];
        }
        for (size_t q = 1; q < at.size(); ++q) at[q] += at[q - 1];
        put.assign(at.begin(), at.end() - 1);
        for (size_t i = 0; i < items.size(); ++i) sorted[put[key[i]]++] = items[i];
        for (int q = 0; q < G * RUN_N; ++q) {
            const int r = q % RUN_N;
            const size_t from = o.items.size();
            for (int j = at[q]; j < at[q + 1]; ++j) {
                const SchedAdds::Item& x = sorted[j];
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
                                  : r == RUN_GENERAL ? make_uint2(in.unread | TGT_VEC | TGT_FIRST, 1u << 20) : make_uint2(in.unread, 0u));
            o.item_off.push_back((int)o.items.size());
        }
    }
    o.items.insert(o.items.end(), kItemUnroll, make_uint2(in.unread, 0u));  // loaded ahead, not used
    std::vector<int> post_count(in.n_slot + in.n_vec, 0), post_owner;
    for (const PostItem& x : in.post) ++post_count[in.dense(x.target)];
    deal(post_count, longest_first(post_count), G, post_owner);
    std::vector<std::vector<PostItem>> of(G);
    for (const PostItem& x : in.post) of[post_owner[in.dense(x.target)]].push_back(x);
    o.post_off.assign(1, 0);
    for (const auto& l : of) {
        o.post.insert(o.post.end(), l.begin(), l.end());
        o.post_off.push_back((int)o.post.size());
    }
    return true;
}
