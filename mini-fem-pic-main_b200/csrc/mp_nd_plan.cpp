// Host side of the sparse direct solve: nested dissection of K's graph, the
// tile structure of its factor and the task list of the device kernels.
#include "mp_nd.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <exception>
#include <future>
#include <limits>
#include <numeric>

namespace mp {

namespace {

// A part of the dissection: a separator, or a leaf.
struct Part {
    std::vector<int> v;
};

struct Dissection {
    const std::vector<long long> &ptr;
    const std::vector<int> &col;
    const std::vector<double> &pos;
    std::vector<std::atomic<int>> label;  // which side of which cut a vertex is on (unique ids, read across threads)
    std::atomic<int> next_label{1};

    Dissection(int n, const std::vector<long long> &p, const std::vector<int> &c, const std::vector<double> &x)
        : ptr(p), col(c), pos(x), label(n) {
        for (auto &l : label) l.store(0, std::memory_order_relaxed);
    }

    // Splits s by coordinate planes into compact runs (in place), so that a
    // subdomain's neighbours among a separator's vertices fill few tiles.
    void compact(int *s, int m) const {
        if (m <= 8) return;
        int ax;
        double lo, hi;
        extent(s, m, ax, lo, hi);
        if (!(hi > lo)) return;
        std::stable_sort(s, s + m, [&](int a, int b) { return pos[3 * (size_t)a + ax] < pos[3 * (size_t)b + ax]; });
        const double eps = 1e-9 * (hi - lo);
        int h = m / 2, best = -1;
        for (int i = 1; i < m; i++)
            if (pos[3 * (size_t)s[i] + ax] > pos[3 * (size_t)s[i - 1] + ax] + eps &&
                (best < 0 || std::abs(2 * i - m) < std::abs(2 * best - m)))
                best = i;
        if (best > 0) h = best;
        compact(s, h);
        compact(s + h, m - h);
    }

    // longest axis of s's bounding box
    void extent(const int *s, int m, int &ax, double &lo, double &hi) const {
        double l[3], h[3];
        for (int d = 0; d < 3; d++) l[d] = h[d] = pos[3 * (size_t)s[0] + d];
        for (int i = 1; i < m; i++)
            for (int d = 0; d < 3; d++) {
                const double x = pos[3 * (size_t)s[i] + d];
                l[d] = std::min(l[d], x);
                h[d] = std::max(h[d], x);
            }
        ax = 0;
        for (int d = 1; d < 3; d++)
            if (h[d] - l[d] > (h[ax] - l[ax]) * (1 + 1e-9)) ax = d;
        lo = l[ax];
        hi = h[ax];
    }

    // Breadth-first levels of s from a far vertex: the coordinate of a part
    // whose vertices' positions do not tell them apart.  Unreached vertices
    // get the highest level.
    void levels(const std::vector<int> &s, std::vector<double> &x) {
        const int in = next_label.fetch_add(2);
        std::vector<int> queue;
        int start = s[0];
        for (int pass = 0; pass < 2; pass++) {
            for (int v : s) label[v].store(in, std::memory_order_relaxed);
            queue.assign(1, start);
            label[start].store(in + 1, std::memory_order_relaxed);
            std::vector<int> depth(1, 0);
            for (size_t q = 0; q < queue.size(); q++) {
                const int v = queue[q];
                for (long long k = ptr[v]; k < ptr[v + 1]; k++)
                    if (label[col[k]].load(std::memory_order_relaxed) == in) {
                        label[col[k]].store(in + 1, std::memory_order_relaxed);
                        queue.push_back(col[k]);
                        depth.push_back(depth[q] + 1);
                    }
            }
            start = queue.back();
            if (pass == 1) {
                const double far = depth.back() + 2;
                for (int v : s) x[v] = far;
                for (size_t q = 0; q < queue.size(); q++) x[queue[q]] = depth[q];
            }
        }
    }

    // Cuts s at coordinate x(v) >= c: a = below, sep = the others with a
    // neighbour in a, b = the rest.
    template <typename X>
    void cut(const std::vector<int> &s, X x, double c, std::vector<int> &a, std::vector<int> &sep,
             std::vector<int> &b) {
        const int id = next_label.fetch_add(1);
        a.clear();
        sep.clear();
        b.clear();
        for (int v : s)
            if (x(v) < c) {
                a.push_back(v);
                label[v].store(id, std::memory_order_relaxed);
            }
        for (int v : s) {
            if (x(v) < c) continue;
            bool touch = false;
            for (long long k = ptr[v]; k < ptr[v + 1] && !touch; k++)
                touch = label[col[k]].load(std::memory_order_relaxed) == id;
            (touch ? sep : b).push_back(v);
        }
    }

    // the median of x over s, and cuts there; false when one side stays empty
    template <typename X>
    bool halve(const std::vector<int> &s, X x, std::vector<int> &a, std::vector<int> &sep, std::vector<int> &b) {
        std::vector<double> xs(s.size());
        for (size_t i = 0; i < s.size(); i++) xs[i] = x(s[i]);
        std::nth_element(xs.begin(), xs.begin() + xs.size() / 2, xs.end());
        const double med = xs[xs.size() / 2];
        const auto mm = std::minmax_element(xs.begin(), xs.end());
        const double eps = 1e-9 * (*mm.second - *mm.first);
        double c = med;
        if (!(*mm.first < med - eps)) {  // nothing below the median's plane: take the next plane
            c = std::numeric_limits<double>::infinity();
            for (double v : xs)
                if (v > med + eps) c = std::min(c, v);
            if (!std::isfinite(c)) return false;
        }
        cut(s, x, c - eps, a, sep, b);
        return !a.empty() && !b.empty();
    }

    void run(std::vector<int> s, int depth, std::vector<Part> &out) {
        std::vector<int> a, sep, b;
        bool ok = false;
        if ((int)s.size() > ND_LEAF) {
            int ax;
            double lo, hi;
            extent(s.data(), (int)s.size(), ax, lo, hi);
            if (hi > lo) ok = halve(s, [&](int v) { return pos[3 * (size_t)v + ax]; }, a, sep, b);
            if (!ok) {
                std::vector<double> x(label.size());
                levels(s, x);
                ok = halve(s, [&](int v) { return x[v]; }, a, sep, b);
            }
            if (ok && 2 * sep.size() > s.size()) ok = false;  // nothing gained by this cut
        }
        if (!ok) {
            compact(s.data(), (int)s.size());
            out.push_back(Part{std::move(s)});
            return;
        }
        s.clear();
        s.shrink_to_fit();
        if (depth < 3 && a.size() + b.size() > 4000) {
            std::vector<Part> pa;
            std::future<void> f;
            try {
                f = std::async(std::launch::async, [&] { run(std::move(a), depth + 1, pa); });
            } catch (const std::exception &) {  // no thread can be had: one side after the other
            }
            if (!f.valid()) run(std::move(a), depth + 1, pa);
            std::vector<Part> pb;
            run(std::move(b), depth + 1, pb);
            if (f.valid()) f.get();
            for (auto &p : pa) out.push_back(std::move(p));
            for (auto &p : pb) out.push_back(std::move(p));
        } else {
            run(std::move(a), depth + 1, out);
            run(std::move(b), depth + 1, out);
        }
        if (!sep.empty()) {
            compact(sep.data(), (int)sep.size());
            out.push_back(Part{std::move(sep)});
        }
    }
};

}  // namespace

bool nd_build_plan(int n, const std::vector<long long> &ptr, const std::vector<int> &col,
                   const std::vector<long long> &slot, const std::vector<double> &pos, long long max_products,
                   NdPlan &plan) {
    plan = NdPlan();
    plan.n = n;
    std::vector<Part> parts;
    {
        Dissection d(n, ptr, col, pos);
        std::vector<int> all(n);
        std::iota(all.begin(), all.end(), 0);
        d.run(std::move(all), 0, parts);
    }
    // tile columns in postorder: a part's vertices in near-equal runs of at most 64
    std::vector<std::vector<int>> verts;
    for (const Part &p : parts) {
        const int m = (int)p.v.size(), k = (m + ND_TILE - 1) / ND_TILE;
        for (int i = 0, o = 0; i < k; i++) {
            const int w = m / k + (i < m % k);
            verts.emplace_back(p.v.begin() + o, p.v.begin() + o + w);
            o += w;
        }
    }
    const int nc = plan.ncol = (int)verts.size();
    std::vector<int> at(n), in(n);  // tile column (postorder) and row of each unknown
    for (int J = 0; J < nc; J++)
        for (int r = 0; r < (int)verts[J].size(); r++) {
            at[verts[J][r]] = J;
            in[verts[J][r]] = r;
        }
    // block symbolic factorization: a column's rows go up to its first one
    std::vector<std::vector<int>> st(nc);
    for (int J = 0; J < nc; J++)
        for (int v : verts[J])
            for (long long k = ptr[v]; k < ptr[v + 1]; k++)
                if (at[col[k]] > J) st[J].push_back(at[col[k]]);
    long long products = 0;
    for (int J = 0; J < nc; J++) {
        auto &s = st[J];
        std::sort(s.begin(), s.end());
        s.erase(std::unique(s.begin(), s.end()), s.end());
        products += (long long)s.size() * (s.size() + 3) / 2;
        if (products > max_products) return false;
        if (!s.empty()) st[s[0]].insert(st[s[0]].end(), s.begin() + 1, s.end());
    }
    // rank: columns on the longest way up from a column; columns are numbered
    // by falling rank, so a column's rows all come after it and the columns on
    // the longest chain come first
    std::vector<int> rank(nc, 1), dep(nc, 1);
    for (int J = nc - 1; J >= 0; J--)
        for (int I : st[J]) rank[J] = std::max(rank[J], rank[I] + 1);
    for (int J = 0; J < nc; J++)
        for (int I : st[J]) dep[I] = std::max(dep[I], dep[J] + 1);
    std::vector<int> order(nc), num(nc);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return rank[a] > rank[b]; });
    for (int k = 0; k < nc; k++) num[order[k]] = k;
    plan.chain = nc ? rank[order[0]] : 0;
    plan.products = products;
    plan.perm.assign((size_t)nc * ND_TILE, -1);
    plan.width.resize(nc);
    plan.tile_ptr.assign(nc + 1, 0);
    std::vector<int> rk(nc), dp(nc);
    for (int J = 0; J < nc; J++) {
        const int o = order[J];
        plan.width[J] = (int)verts[o].size();
        std::copy(verts[o].begin(), verts[o].end(), plan.perm.begin() + (size_t)J * ND_TILE);
        rk[J] = rank[o];
        dp[J] = dep[o];
        plan.tile_ptr[J + 1] = plan.tile_ptr[J] + 1 + (int)st[o].size();
    }
    const int nt = plan.ntile = plan.tile_ptr[nc];
    plan.tile_row.resize(nt);
    plan.tile_col.resize(nt);
    plan.row_ptr.assign(nc + 1, 0);
    for (int J = 0; J < nc; J++) {
        int *t = plan.tile_row.data() + plan.tile_ptr[J];
        *t++ = J;
        for (int I : st[order[J]]) *t++ = num[I];
        std::sort(plan.tile_row.data() + plan.tile_ptr[J] + 1, t);
        for (int k = plan.tile_ptr[J]; k < plan.tile_ptr[J + 1]; k++) {
            plan.tile_col[k] = J;
            if (plan.tile_row[k] != J) plan.row_ptr[plan.tile_row[k] + 1]++;
        }
    }
    for (int I = 0; I < nc; I++) plan.row_ptr[I + 1] += plan.row_ptr[I];
    plan.row_tile.resize(plan.row_ptr[nc]);
    {
        std::vector<int> fill(plan.row_ptr.begin(), plan.row_ptr.end() - 1);
        for (int t = 0; t < nt; t++)
            if (plan.tile_row[t] != plan.tile_col[t]) plan.row_tile[fill[plan.tile_row[t]]++] = t;
    }
    auto find = [&](int I, int J) {  // tile (I, J), -1 if there is none
        const int *b = plan.tile_row.data() + plan.tile_ptr[J], *e = plan.tile_row.data() + plan.tile_ptr[J + 1];
        const int *p = std::lower_bound(b, e, I);
        return p != e && *p == I ? (int)(p - plan.tile_row.data()) : -1;
    };
    // K's entries by tile (the diagonal tiles' lower triangle)
    std::vector<int> ent_ptr(nt + 1, 0);
    {
        std::vector<int> where;
        std::vector<uint16_t> pos_in;
        std::vector<int> src;
        where.reserve(col.size() / 2 + n);
        pos_in.reserve(col.size() / 2 + n);
        src.reserve(col.size() / 2 + n);
        for (int J = 0; J < nc; J++)
            for (int v : verts[order[J]]) {
                int lastI = -1, lastT = -1;
                for (long long k = ptr[v]; k < ptr[v + 1]; k++) {
                    const int w = col[k], I = num[at[w]];
                    if (I < J || (I == J && in[w] < in[v])) continue;
                    if (I != lastI) {
                        lastI = I;
                        lastT = find(I, J);
                    }
                    where.push_back(lastT);
                    pos_in.push_back((uint16_t)nd_at(in[w], in[v]));
                    src.push_back((int)slot[k]);
                    ent_ptr[lastT + 1]++;
                }
            }
        for (int t = 0; t < nt; t++) ent_ptr[t + 1] += ent_ptr[t];
        plan.ent_src.resize(where.size());
        plan.ent_at.resize(where.size());
        std::vector<int> fill(ent_ptr.begin(), ent_ptr.end() - 1);
        for (size_t k = 0; k < where.size(); k++) {
            const int o = fill[where[k]]++;
            plan.ent_src[o] = src[k];
            plan.ent_at[o] = pos_in[k];
        }
    }
    // products of each tile, by ascending summed column
    std::vector<int> prod_ptr(nt + 1, 0);
    std::vector<NdItem> prod;
    {
        for (int pass = 0; pass < 2; pass++) {
            std::vector<int> fill(prod_ptr.begin(), prod_ptr.end() - 1);
            if (pass) prod.resize(prod_ptr[nt]);
            for (int K = 0; K < nc; K++) {
                const int b = plan.tile_ptr[K] + 1, e = plan.tile_ptr[K + 1];
                const int kb = (plan.width[K] + 7) / 8;
                for (int j = b; j < e; j++) {
                    // rows of column J = row(j) that column K also holds: both ascending
                    const int J = plan.tile_row[j];
                    int t = plan.tile_ptr[J];
                    for (int i = j; i < e; i++) {
                        while (plan.tile_row[t] != plan.tile_row[i]) t++;
                        if (pass) prod[fill[t]++] = NdItem{i, j, K, kb};
                        else prod_ptr[t + 1]++;
                    }
                }
            }
            if (!pass)
                for (int t = 0; t < nt; t++) prod_ptr[t + 1] += prod_ptr[t];
        }
    }
    // Tasks, by falling rank: of each rank the diagonal tasks, then the others,
    // then the partial tasks whose last product's column is one rank higher.  A
    // task's needs are then all formed by tasks before it: tiles of columns of
    // higher rank (formed in their own rank's group or, for a diagonal task's
    // second tile, with the diagonal tasks one rank on), the diagonal blocks of
    // its own group, and partial sums at least one group back.
    const int top = plan.chain;
    std::vector<std::vector<NdTask>> diag(top + 1), off(top + 1), part(top + 1);
    std::vector<std::vector<NdItem>> lists;  // a task's items, indexed by item0 until they are laid out
    std::vector<char> fused(nt, 0);
    auto begin = [&](int row, int col) {
        NdTask t{};
        t.row = row;
        t.col = col;
        t.pred = t.tile = t.xtile = -1;
        t.rblocks = (int16_t)((plan.width[row] + 7) / 8);
        t.cblocks = (int16_t)((plan.width[col] + 7) / 8);
        t.item0 = (int)lists.size();
        lists.push_back({NdItem{-1, ND_BEGIN, col, 0}});
        return t;
    };
    auto scratch = [&] { return nt + plan.nscratch++; };
    // moves the early products of task t (list `l`) to partial tasks
    auto split = [&](NdTask &t, const std::vector<NdItem> &l) {
        int early = 0;
        while (early < (int)l.size() && rk[l[early].col] > rk[t.col] + ND_NEAR) early++;
        if (early < ND_SPLIT_FROM) early = 0;
        const int pieces = (early + ND_SPLIT - 1) / ND_SPLIT;
        for (int i = 0, o = 0; i < pieces; i++) {
            const int m = early / pieces + (i < early % pieces);
            NdTask q = begin(t.row, t.col);
            q.pred = t.pred;
            q.pblocks = t.pblocks;
            q.partial = 1;
            q.tile = scratch();
            lists[t.item0].push_back(NdItem{q.tile, ND_ADD, nc + q.tile - nt, 8});
            bool x = false;
            for (int k = o; k < o + m; k++) x = x || (t.row == t.col && l[k].b >= 0);
            if (x) {
                q.xtile = scratch();
                lists[t.item0].push_back(NdItem{q.xtile, ND_ADDX, nc + q.xtile - nt, 8});
            }
            lists[q.item0].insert(lists[q.item0].end(), l.begin() + o, l.begin() + o + m);
            o += m;
            part[rk[l[o - 1].col] - 1].push_back(q);
        }
        lists[t.item0].insert(lists[t.item0].end(), l.begin() + early, l.end());
    };
    for (int J = 0; J < nc; J++) {
        NdTask t = begin(J, J);
        t.tile = plan.tile_ptr[J];
        t.ent0 = ent_ptr[t.tile];
        t.ent1 = ent_ptr[t.tile + 1];
        // the latest of the columns just before J on a chain: forming its tile here saves the
        // chain one hand-over between SMs
        for (int q = plan.row_ptr[J]; q < plan.row_ptr[J + 1]; q++) {
            const int P = plan.tile_col[plan.row_tile[q]];
            if (rk[P] == rk[J] + 1 && (t.pred < 0 || dp[P] > dp[t.pred])) {
                t.pred = P;
                t.xtile = plan.row_tile[q];
            }
        }
        if (t.pred >= 0) t.pblocks = (int16_t)((plan.width[t.pred] + 7) / 8);
        std::vector<NdItem> l;
        for (int q = prod_ptr[t.tile]; q < prod_ptr[t.tile + 1]; q++) {
            NdItem it = prod[q];
            if (it.col == t.pred) continue;  // taken from the tile formed here
            it.b = t.pred >= 0 ? find(t.pred, it.col) : -1;
            if (it.b < 0) it.b = ND_DIAG_ONLY;
            l.push_back(it);
        }
        split(t, l);
        if (t.pred >= 0) {
            fused[t.xtile] = 1;
            lists[t.item0].push_back(NdItem{plan.tile_ptr[t.pred], ND_INV, t.pred, (plan.width[t.pred] + 7) / 8});
            t.xent0 = ent_ptr[t.xtile];
            t.xent1 = ent_ptr[t.xtile + 1];
        }
        diag[rk[J]].push_back(t);
    }
    for (int J = 0; J < nc; J++)
        for (int k = plan.tile_ptr[J] + 1; k < plan.tile_ptr[J + 1]; k++) {
            if (fused[k]) continue;  // formed by a diagonal task
            NdTask t = begin(plan.tile_row[k], J);
            t.tile = k;
            t.ent0 = ent_ptr[k];
            t.ent1 = ent_ptr[k + 1];
            split(t, std::vector<NdItem>(prod.begin() + prod_ptr[k], prod.begin() + prod_ptr[k + 1]));
            lists[t.item0].push_back(NdItem{plan.tile_ptr[J], ND_INV, J, (plan.width[J] + 7) / 8});
            off[rk[J]].push_back(t);
        }
    for (int r = top; r >= 0; r--)
        for (auto *group : {&diag[r], &off[r], &part[r]})
            for (NdTask t : *group) {
                const std::vector<NdItem> &l = lists[t.item0];
                t.item0 = (int)plan.item.size();
                plan.item.insert(plan.item.end(), l.begin(), l.end());
                t.item1 = (int)plan.item.size();
                plan.task.push_back(t);
            }
    return true;
}

}  // namespace mp
