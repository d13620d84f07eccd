// symbolic.cpp -- once-per-topology analysis on the host: Ybus pattern and
// assembly map, fill-reducing ordering of the buses, symbolic block LU of the
// Newton Jacobian, its Crout gather lists and level schedules, and the map
// from factor block positions to Ybus slots used by the Jacobian fill.
#include <algorithm>
#include <numeric>
#include <queue>
#include <string>
#include <vector>

#include "gbpf_internal.h"

namespace gbpf {

int YPattern::find(int r, int c) const {
    auto b = col.begin() + rowptr[r], e = col.begin() + rowptr[r + 1];
    auto it = std::lower_bound(b, e, c);
    return (it != e && *it == c) ? (int)(it - col.begin()) : -1;
}

// Pattern of calcYbusSp_eficinte (GPU/sistema.h:705-758): four stamps per
// branch and one shunt per bus, duplicates summed.  Slot contributions are
// listed in the order Eigen's setFromTriplets adds them: the stamps of branch
// 0 (de,para), (para,de), (de,de), (para,para), then branch 1, ..., then the
// bus shunts.
YPattern build_ypattern(const Grid &g) {
    YPattern y;
    const int n = g.nB;
    y.n = n;
    std::vector<std::vector<int>> rows(n);
    for (int k = 0; k < n; k++) rows[k].push_back(k);
    for (int b = 0; b < g.nL; b++) {
        const int f = g.de[b] - 1, t = g.para[b] - 1;
        rows[f].push_back(t);
        rows[t].push_back(f);
    }
    y.rowptr.assign(n + 1, 0);
    for (int k = 0; k < n; k++) {
        auto &r = rows[k];
        std::sort(r.begin(), r.end());
        r.erase(std::unique(r.begin(), r.end()), r.end());
        y.rowptr[k + 1] = y.rowptr[k] + (int)r.size();
    }
    y.nnz = y.rowptr[n];
    y.col.resize(y.nnz);
    for (int k = 0; k < n; k++) std::copy(rows[k].begin(), rows[k].end(), y.col.begin() + y.rowptr[k]);
    y.diag.resize(n);
    for (int k = 0; k < n; k++) y.diag[k] = y.find(k, k);
    // contributions in triplet order
    std::vector<int> cnt(y.nnz, 0);
    std::vector<std::pair<int, int>> trip;  // (slot, source)
    trip.reserve(4 * g.nL + n);
    for (int b = 0; b < g.nL; b++) {
        const int f = g.de[b] - 1, t = g.para[b] - 1;
        trip.push_back({y.find(f, t), 4 * b + 0});
        trip.push_back({y.find(t, f), 4 * b + 1});
        trip.push_back({y.find(f, f), 4 * b + 2});
        trip.push_back({y.find(t, t), 4 * b + 3});
    }
    for (int k = 0; k < n; k++) trip.push_back({y.diag[k], -1 - k});
    for (auto &p : trip) cnt[p.first]++;
    y.cptr.assign(y.nnz + 1, 0);
    for (int s = 0; s < y.nnz; s++) y.cptr[s + 1] = y.cptr[s] + cnt[s];
    y.csrc.resize(trip.size());
    std::vector<int> fill(y.cptr.begin(), y.cptr.end() - 1);
    for (auto &p : trip) y.csrc[fill[p.first]++] = p.second;
    return y;
}

// Minimum degree on an explicit elimination graph (ties broken by the lower
// index), giving the order in which blocks are eliminated.
std::vector<int> min_degree_order(int n, const std::vector<std::vector<int>> &adj0) {
    std::vector<std::vector<int>> adj(adj0);
    std::vector<int> deg(n), mark(n, 0), done(n, 0), order;
    order.reserve(n);
    int stamp = 0;
    using E = std::pair<int, int>;
    std::priority_queue<E, std::vector<E>, std::greater<E>> pq;
    for (int i = 0; i < n; i++) { deg[i] = (int)adj[i].size(); pq.push({deg[i], i}); }
    std::vector<int> nb, tmp;
    while ((int)order.size() < n) {
        E e = pq.top();
        pq.pop();
        const int p = e.second;
        if (done[p] || e.first != deg[p]) continue;
        done[p] = 1;
        order.push_back(p);
        nb.clear();
        for (int v : adj[p]) if (!done[v]) nb.push_back(v);
        for (int u : nb) {
            ++stamp;
            mark[u] = stamp;
            tmp.clear();
            for (int v : adj[u]) if (v != p && !done[v] && mark[v] != stamp) { mark[v] = stamp; tmp.push_back(v); }
            for (int v : nb) if (mark[v] != stamp) { mark[v] = stamp; tmp.push_back(v); }
            adj[u] = tmp;
            deg[u] = (int)tmp.size();
            pq.push({deg[u], u});
        }
        adj[p].clear();
        adj[p].shrink_to_fit();
    }
    return order;
}

// Shorter elimination tree at no extra fill (Jess and Kees, "A data structure
// for parallel L/U decomposition", IEEE Trans. Computers C-31, 1982): the
// filled graph of `ord` is chordal, and eliminating, round after round, a
// maximal independent set of its simplicial vertices (neighbourhood a clique)
// is a perfect elimination order of it -- no fill beyond that of `ord` -- whose
// elimination tree is as short as such an order allows.  Every round becomes
// one level of the factor's schedule, and each level costs the Newton kernels a
// barrier and a chain of dependent 2x2 products, so fewer levels is less
// latency per iteration (118-bus grid: 30 -> 21 levels, same factor).
// Within a round the vertices keep their order in `ord`.
std::vector<int> reduce_height(int n, const std::vector<std::vector<int>> &adj, const std::vector<int> &ord) {
    std::vector<int> pos(n);
    for (int i = 0; i < n; i++) pos[ord[i]] = i;
    // filled graph: elimination of ord on a copy of the graph (sorted adjacency)
    std::vector<std::vector<int>> F(n);
    {
        std::vector<std::vector<int>> up(n);  // higher neighbours, by position
        for (int v = 0; v < n; v++)
            for (int w : adj[v]) if (pos[w] > pos[v]) up[v].push_back(w);
        std::vector<int> mark(n, -1);
        for (int i = 0; i < n; i++) {
            const int v = ord[i];
            auto &u = up[v];
            std::sort(u.begin(), u.end(), [&](int a, int b) { return pos[a] < pos[b]; });
            u.erase(std::unique(u.begin(), u.end()), u.end());
            for (int w : u) { F[v].push_back(w); F[w].push_back(v); }
            if (u.empty()) continue;
            // the lowest higher neighbour inherits the rest (elimination-tree parent)
            const int p = u[0];
            auto &pu = up[p];
            for (size_t k = 1; k < u.size(); k++) pu.push_back(u[k]);
            (void)mark;
        }
        for (auto &f : F) {
            std::sort(f.begin(), f.end());
            f.erase(std::unique(f.begin(), f.end()), f.end());
        }
    }
    std::vector<char> alive(n, 1), simp(n, 0), dirty(n, 1);
    std::vector<int> deg(n);
    for (int v = 0; v < n; v++) deg[v] = (int)F[v].size();
    auto adjacent = [&](int a, int b) { return std::binary_search(F[a].begin(), F[a].end(), b); };
    auto simplicial = [&](int v) {
        std::vector<int> nb;
        for (int w : F[v]) if (alive[w]) nb.push_back(w);
        for (size_t x = 0; x < nb.size(); x++)
            for (size_t z = x + 1; z < nb.size(); z++)
                if (!adjacent(nb[x], nb[z])) return false;
        return true;
    };
    std::vector<int> out, cand, blocked(n, -1);
    out.reserve(n);
    int left = n, round = 0;
    while (left > 0) {
        cand.clear();
        for (int i = 0; i < n; i++) {
            const int v = ord[i];
            if (!alive[v]) continue;
            if (dirty[v]) { simp[v] = simplicial(v); dirty[v] = 0; }
            if (simp[v]) cand.push_back(v);
        }
        // maximal independent set, lowest degree first, ties in ord order
        std::stable_sort(cand.begin(), cand.end(), [&](int a, int b) { return deg[a] < deg[b]; });
        std::vector<int> chosen;
        for (int v : cand) {
            if (blocked[v] == round) continue;
            chosen.push_back(v);
            blocked[v] = round;
            for (int w : F[v]) if (alive[w]) blocked[w] = round;
        }
        std::sort(chosen.begin(), chosen.end(), [&](int a, int b) { return pos[a] < pos[b]; });
        for (int v : chosen) {
            alive[v] = 0;
            left--;
            out.push_back(v);
            for (int w : F[v]) if (alive[w]) { dirty[w] = 1; deg[w]--; }
        }
        round++;
    }
    return out;
}

Symbolic analyse(const Grid &g, const YPattern &y, std::string *why) {
    Symbolic S;
    const int nB = g.nB, s = g.slack - 1, n = nB - 1;
    S.n = n;
    // bus graph without the slack
    std::vector<int> cidx(nB, -1), cbus;
    for (int k = 0; k < nB; k++) if (k != s) { cidx[k] = (int)cbus.size(); cbus.push_back(k); }
    std::vector<std::vector<int>> adj(n);
    for (int k = 0; k < nB; k++) {
        if (k == s) continue;
        for (int p = y.rowptr[k]; p < y.rowptr[k + 1]; p++) {
            const int m = y.col[p];
            if (m == s || m == k) continue;
            adj[cidx[k]].push_back(cidx[m]);
        }
    }
    std::vector<int> ord = reduce_height(n, adj, min_degree_order(n, adj));
    S.bus_of_blk.resize(n);
    S.blk_of_bus.assign(nB, -1);
    for (int b = 0; b < n; b++) {
        S.bus_of_blk[b] = cbus[ord[b]];
        S.blk_of_bus[cbus[ord[b]]] = b;
    }
    // lower structure of A in the new order: for column j, rows i > j
    std::vector<std::vector<int>> alow(n);
    for (int k = 0; k < nB; k++) {
        if (k == s) continue;
        const int bk = S.blk_of_bus[k];
        for (int p = y.rowptr[k]; p < y.rowptr[k + 1]; p++) {
            const int m = y.col[p];
            if (m == s || m == k) continue;
            const int bm = S.blk_of_bus[m];
            if (bm > bk) alow[bk].push_back(bm);
        }
    }
    // symbolic factorisation: struct(j) = alow(j) U (struct(c) \ {j}) over the
    // elimination-tree children c of j
    std::vector<std::vector<int>> st(n), children(n);
    std::vector<int> mark(n, -1);
    for (int j = 0; j < n; j++) {
        std::vector<int> &out = st[j];
        mark[j] = j;
        for (int i : alow[j]) if (mark[i] != j) { mark[i] = j; out.push_back(i); }
        for (int c : children[j])
            for (int i : st[c]) if (i != j && mark[i] != j) { mark[i] = j; out.push_back(i); }
        std::sort(out.begin(), out.end());
        if (!out.empty()) children[out[0]].push_back(j);
    }
    S.up_ptr.assign(n + 1, 0);
    for (int j = 0; j < n; j++) S.up_ptr[j + 1] = S.up_ptr[j] + (int)st[j].size();
    S.nup = S.up_ptr[n];
    S.up_col.resize(S.nup);
    for (int j = 0; j < n; j++) std::copy(st[j].begin(), st[j].end(), S.up_col.begin() + S.up_ptr[j]);
    auto pos_in = [&](int j, int i) -> int {
        auto b = S.up_col.begin() + S.up_ptr[j], e = S.up_col.begin() + S.up_ptr[j + 1];
        auto it = std::lower_bound(b, e, i);
        return (it != e && *it == i) ? (int)(it - S.up_col.begin()) : -1;
    };
    // row structures rs(j) = {k : j in idx(k)}, k ascending, with positions
    std::vector<int> rcnt(n, 0);
    for (int p = 0; p < S.nup; p++) rcnt[S.up_col[p]]++;
    S.dg_ptr.assign(n + 1, 0);
    for (int j = 0; j < n; j++) S.dg_ptr[j + 1] = S.dg_ptr[j] + rcnt[j];
    S.dg_pos.resize(S.nup);
    S.dg_k.resize(S.nup);
    {
        std::vector<int> f(S.dg_ptr.begin(), S.dg_ptr.end() - 1);
        for (int k = 0; k < n; k++)
            for (int p = S.up_ptr[k]; p < S.up_ptr[k + 1]; p++) {
                const int j = S.up_col[p];
                S.dg_pos[f[j]] = p;
                S.dg_k[f[j]] = k;
                f[j]++;
            }
    }
    // off-diagonal gather pairs: for k, a < b in idx(k): entry (j = idx(k)[a], i = idx(k)[b])
    std::vector<long long> ocnt(S.nup, 0);
    for (int k = 0; k < n; k++)
        for (int a = S.up_ptr[k]; a < S.up_ptr[k + 1]; a++)
            for (int b = a + 1; b < S.up_ptr[k + 1]; b++) {
                const int p = pos_in(S.up_col[a], S.up_col[b]);
                if (p < 0) { if (why) *why = "symbolic factorisation is not closed under fill"; return Symbolic(); }
                ocnt[p]++;
            }
    S.og_ptr.assign(S.nup + 1, 0);
    for (int p = 0; p < S.nup; p++) S.og_ptr[p + 1] = S.og_ptr[p] + ocnt[p];
    const long long npairs = S.og_ptr[S.nup];
    S.og_a.resize(npairs);
    S.og_b.resize(npairs);
    S.og_k.resize(npairs);
    {
        std::vector<long long> f(S.og_ptr.begin(), S.og_ptr.end() - 1);
        for (int k = 0; k < n; k++)
            for (int a = S.up_ptr[k]; a < S.up_ptr[k + 1]; a++)
                for (int b = a + 1; b < S.up_ptr[k + 1]; b++) {
                    const int p = pos_in(S.up_col[a], S.up_col[b]);
                    S.og_a[f[p]] = a;
                    S.og_b[f[p]] = b;
                    S.og_k[f[p]] = k;
                    f[p]++;
                }
    }
    // level schedules
    std::vector<int> fl(n, 0), bl(n, 0);
    int nfl = 0, nbl = 0;
    for (int j = 0; j < n; j++) {
        int l = 0;
        for (int q = S.dg_ptr[j]; q < S.dg_ptr[j + 1]; q++) l = std::max(l, fl[S.dg_k[q]] + 1);
        fl[j] = l;
        nfl = std::max(nfl, l + 1);
    }
    for (int j = n - 1; j >= 0; j--) {
        int l = 0;
        for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++) l = std::max(l, bl[S.up_col[p]] + 1);
        bl[j] = l;
        nbl = std::max(nbl, l + 1);
    }
    auto bucket = [n](const std::vector<int> &lev, int nl, std::vector<int> &ptr, std::vector<int> &steps) {
        ptr.assign(nl + 1, 0);
        for (int j = 0; j < n; j++) ptr[lev[j] + 1]++;
        for (int l = 0; l < nl; l++) ptr[l + 1] += ptr[l];
        steps.resize(n);
        std::vector<int> f(ptr.begin(), ptr.end() - 1);
        for (int j = 0; j < n; j++) steps[f[lev[j]]++] = j;
    };
    bucket(fl, nfl, S.flev_ptr, S.flev_steps);
    bucket(bl, nbl, S.blev_ptr, S.blev_steps);
    S.fent_ptr.assign(nfl + 1, 0);
    S.fent_p.clear();
    S.fent_j.clear();
    for (int l = 0; l < nfl; l++) {
        for (int t = S.flev_ptr[l]; t < S.flev_ptr[l + 1]; t++) {
            const int j = S.flev_steps[t];
            for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++) { S.fent_p.push_back(p); S.fent_j.push_back(j); }
        }
        S.fent_ptr[l + 1] = (int)S.fent_p.size();
    }
    // Jacobian fill map over factor block positions
    const int nq = n + 2 * S.nup;
    S.ysl.resize(nq);
    S.rbus.resize(nq);
    S.cbus.resize(nq);
    for (int j = 0; j < n; j++) {
        const int bj = S.bus_of_blk[j];
        S.ysl[j] = y.diag[bj];
        S.rbus[j] = bj;
        S.cbus[j] = bj;
    }
    for (int j = 0; j < n; j++)
        for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++) {
            const int bi = S.bus_of_blk[S.up_col[p]], bj = S.bus_of_blk[j];
            const int ql = n + p, qu = n + S.nup + p;
            S.ysl[ql] = y.find(bi, bj);  // L(i,j): row bus i, column bus j
            S.rbus[ql] = bi;
            S.cbus[ql] = bj;
            S.ysl[qu] = y.find(bj, bi);  // U(j,i): row bus j, column bus i
            S.rbus[qu] = bj;
            S.cbus[qu] = bi;
        }
    return S;
}

namespace {

// How the items (pivots, entries or rows) of one level run on one CTA -- 2^g
// lanes (quads of lanes) an item, dealt round to 2^lw warps -- and what that is
// estimated to take, in cycles.  An FP64 instruction holds its quarter of the
// SM 64 cycles a warp whatever lanes are active (measured: 64 cycles with one
// warp, 19 a warp with four or more), so the estimate is the instructions of
// the fullest quarter; FP32 levels are chains of latencies.  `ops` =
// multiply-adds of one list element on one lane, `sums` = values a group of
// lanes adds up.
struct Lanes {
    int g = 0, quad = 0, lw = 0, passes = 1;
    double cost = 0;
};
Lanes pick_lanes(long long count, long long longest, long long total, int ops, int sums, int fixed, int mem,
                 bool fp64) {
    Lanes best;
    if (!count) return best;
    best.cost = 1e30;
    const double mean = (double)total / count;
    for (int quad = 0; quad <= (fp64 && sums > 2 ? 1 : 0); quad++)
        for (int g = 0; g <= (quad ? 3 : 5); g++) {
            if (g && (1LL << (g - 1)) >= longest) break;
            const int per = quad ? 4 : 1;
            for (int lw = 0; (1 << lw) <= kClusterThreads / 32; lw++) {
                const long long cap = (32LL >> g) / per << lw, passes = (count + cap - 1) / cap;
                if (quad && passes > 1) continue;
                const double longest_walk = (double)((longest + (1LL << g) - 1) >> g);
                const double walk =
                    passes > 1 ? std::min(longest_walk, 0.5 * longest_walk + 0.5 * mean / (1 << g)) : longest_walk;
                const double instr = fixed / (double)(per > 1 ? 2 : 1) + walk * ops / per + g * sums / (double)per;
                const long long warps = std::min<long long>(1LL << lw, count);
                const double chain = mem + walk * ((quad ? 130 : 90) + 0.5 * mem) + g * (quad ? 30 : 40);
                const double cost = fp64 ? passes * ((warps + 3) / 4 * instr * 64 + chain)
                                         : passes * (chain + (warps + 3) / 4 * instr * 2);
                if (cost < best.cost) {
                    best.g = g;
                    best.quad = quad;
                    best.lw = lw;
                    best.passes = (int)passes;
                    best.cost = cost;
                }
            }
        }
    return best;
}

}  // namespace

namespace {

size_t up128(size_t x) { return (x + 127) / 128 * 128; }

// The levels of a choice of segment and tail.
struct ClusterSplit {
    std::vector<std::vector<int>> f1, fs, bs, b1;  // steps of every level
};

struct ClusterBuilder {
    const Symbolic &S;
    const int n, ctas, td;
    const bool fp64;
    const size_t limit, b4, b2;
    int tail_ctas;

    // k of the lists ascends: the elements below t are a prefix
    int dg_cut(int j, int t) const {
        return (int)(std::lower_bound(S.dg_k.begin() + S.dg_ptr[j], S.dg_k.begin() + S.dg_ptr[j + 1], t) -
                     S.dg_k.begin());
    }
    long long og_cut(int p, int t) const {
        return (long long)(std::lower_bound(S.og_k.begin() + S.og_ptr[p], S.og_k.begin() + S.og_ptr[p + 1], t) -
                           S.og_k.begin());
    }
    ClusterSplit split(int t0) const {
        ClusterSplit R;
        std::vector<int> lv(n, 0);
        auto add = [](std::vector<std::vector<int>> &v, int l, int j) {
            if ((int)v.size() <= l) v.resize(l + 1);
            v[l].push_back(j);
        };
        for (int j = 0; j < td; j++) {
            int l = 0;
            for (int q = j < t0 ? S.dg_ptr[j] : dg_cut(j, t0); q < S.dg_ptr[j + 1]; q++)
                l = std::max(l, lv[S.dg_k[q]] + 1);
            lv[j] = l;
            add(j < t0 ? R.f1 : R.fs, l, j);
        }
        for (int j = td - 1; j >= 0; j--) {
            int l = 0;
            for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++)
                if (S.up_col[p] < (j < t0 ? t0 : td)) l = std::max(l, lv[S.up_col[p]] + 1);
            lv[j] = l;
            add(j < t0 ? R.b1 : R.bs, l, j);
        }
        return R;
    }
    size_t seg_bytes(int t0) const {
        return up128(((size_t)(td - t0) + 2 * (size_t)(S.up_ptr[td] - S.up_ptr[t0])) * b4);
    }
    size_t vec_bytes(int t0) const { return up128((size_t)(n - t0) * b2); }
    size_t tail_bytes() const { return td < n ? up128(tail_blocks(n - td, tail_ctas) * b4) : 0; }
    // estimated cycles of one pass with the segment from t0 on (the tail's are
    // the same for every choice), and bytes of CTA 0's schedule
    double estimate(int t0, size_t &bytes) const {
        const ClusterSplit L = split(t0);
        const size_t per = S.nup <= 65536 && n <= 65536 ? 4 : 8;
        double items0 = 0, pairs0 = 0;  // of CTA 0
        // what a level takes besides its work: on the cluster a store, a cluster
        // barrier and a load from L2 (2,650 cycles measured; the barrier alone 380
        // to 480, with the store 1,760), in the segment two block barriers and the
        // loads between them
        const double clus = 3000, seg = 400;
        auto fwd = [&](const std::vector<int> &steps, bool in_seg, int share) {
            long long md = 0, sd = 0, ne = 0, me = 0, se = 0;
            for (int j : steps) {
                const int c = in_seg ? dg_cut(j, t0) : S.dg_ptr[j];
                md = std::max<long long>(md, S.dg_ptr[j + 1] - c);
                sd += S.dg_ptr[j + 1] - c;
                for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++) {
                    const long long k = S.og_ptr[p + 1] - (in_seg ? og_cut(p, t0) : S.og_ptr[p]);
                    me = std::max(me, k);
                    se += k;
                    ne++;
                }
            }
            const long long np = steps.size();
            items0 += (double)(np + ne) / share;
            pairs0 += (double)(sd + se) / share + (np < share ? md : 0);
            const int mem = in_seg ? 60 : 700;
            const Lanes a = pick_lanes((np + share - 1) / share, md, (sd + share - 1) / share, 12, 6, 20, mem, fp64);
            const Lanes b = pick_lanes((ne + share - 1) / share, me, (se + share - 1) / share, 16, 8, 8, mem, fp64);
            return std::max(a.cost, b.cost) + (fp64 ? 0.25 * std::min(a.cost, b.cost) : 0);
        };
        double c = 0;
        for (const auto &l : L.f1) c += clus + fwd(l, false, ctas);
        // (FP64 segment levels measured at about twice the estimate: with 1 / 1.4 /
        // 2 / 3 here a 1,888-bus solve takes 0.630 / 0.607 / 0.603 / 0.623 ms, a
        // filled 236-bus grid 0.82 / 0.70 / 0.71 / 0.65, its 170-bus kin 0.59 /
        // 0.59 / 0.53 / 0.54)
        for (const auto &l : L.fs) c += seg + fwd(l, true, 1) * (fp64 ? 2.0 : 1.0);
        c += L.bs.size() * (seg + 300.0) + L.b1.size() * (0.8 * clus);
        if (t0 < td && td < n) {
            // the segment's updates of the tail, on CTA 0
            long long ne = 0, me = 0, se = 0;
            for (int p = S.up_ptr[td]; p < S.nup; p++) {
                const long long k = og_cut(p, td) - og_cut(p, t0);
                ne += k > 0;
                me = std::max(me, k);
                se += k;
            }
            c += pick_lanes(ne, me, se, 16, 8, 0, 60, false).cost + (tail_ctas > 1 ? 2 * clus : 0);
            items0 += ne;
            pairs0 += se;
        }
        // the gather into segment and tail, and the backward rows
        for (int p = S.up_ptr[t0]; p < S.nup; p++) {
            const double k = (double)(og_cut(p, t0) - S.og_ptr[p]);
            items0 += (k > 0) / (double)ctas;
            pairs0 += k / ctas;
        }
        items0 += (double)t0 / ctas + (td - t0);
        pairs0 += (double)S.up_ptr[t0] / ctas + (S.up_ptr[td] - S.up_ptr[t0]);
        bytes = (size_t)(16 * items0 + per * pairs0) + 32 * (L.f1.size() + L.fs.size()) + 16 * (L.bs.size() + L.b1.size());
        return c;
    }
    ClusterSchedule build(int t0) const;
};

// One level's entries: position, list length, pivot's index in the level (or
// what the record's last field is to hold).
struct LevelEnt { int p, len, piv; };

ClusterSchedule ClusterBuilder::build(int t0) const {
    const ClusterSplit L = split(t0);
    const int ctas = t0 == 0 && tail_ctas == 1 ? 1 : this->ctas;  // CTA 0 does it all
    ClusterSchedule R;
    R.ctas = ctas;
    R.t0 = t0;
    R.td = td;
    R.tail_ctas = tail_ctas;
    R.nf1 = (int)L.f1.size(); R.nfs = (int)L.fs.size(); R.nbs = (int)L.bs.size(); R.nb1 = (int)L.b1.size();
    std::vector<std::vector<int>> part(ctas);
    const size_t heads = 8 * (size_t)(R.nf1 + 1 + R.nfs + 1);
    for (auto &b : part) b.assign(heads + 4 * (size_t)(R.nbs + R.nb1), 0);
    const int W = kClusterThreads / 32;
    R.packed = S.nup <= 65536 && n <= 65536;
    auto pair = [&](std::vector<int> &b, int x, int y) {
        if (R.packed) b.push_back((int)((unsigned)y << 16 | (unsigned)x));
        else { b.push_back(x); b.push_back(y); }
    };
    // index of the list element that the next pair() of b makes
    auto at = [&](std::vector<int> &b) {
        if (!R.packed && b.size() % 2) b.push_back(0);
        return (int)(R.packed ? b.size() : b.size() / 2);
    };
    auto pad4 = [](std::vector<int> &b) { while (b.size() % 4) b.push_back(0); };
    // kind 0: cluster level, 1: the gather into segment and tail, 2: segment
    // level, 3: the segment's gather into the tail.  Steps [from, to) of the
    // lists belong to it.
    using Piv = std::pair<int, int>;
    auto put_level = [&](std::vector<int> &b, size_t head, const std::vector<Piv> &piv, std::vector<LevelEnt> &ent,
                         int kind) {
        const int from = kind < 2 ? 0 : t0, to = kind == 0 || kind == 2 ? n : kind == 1 ? t0 : td;
        auto dg_of = [&](int j) {
            return std::make_pair(from ? dg_cut(j, from) : S.dg_ptr[j], to < n ? dg_cut(j, to) : S.dg_ptr[j + 1]);
        };
        auto og_of = [&](int p) {
            return std::make_pair(from ? og_cut(p, from) : S.og_ptr[p], to < n ? og_cut(p, to) : S.og_ptr[p + 1]);
        };
        // longest lists first, so that the lanes of a warp walk alike
        std::vector<int> ord(piv.size()), back(piv.size());
        for (size_t i = 0; i < ord.size(); i++) ord[i] = (int)i;
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int c) {
            const auto x = dg_of(piv[a].first), y = dg_of(piv[c].first);
            return x.second - x.first > y.second - y.first;
        });
        for (size_t i = 0; i < ord.size(); i++) back[ord[i]] = (int)i;
        std::stable_sort(ent.begin(), ent.end(), [](const LevelEnt &a, const LevelEnt &c) { return a.len > c.len; });
        long long md = 0, sd = 0, me = 0, se = 0;
        pad4(b);
        const int op = (int)b.size();
        b.resize(b.size() + 4 * piv.size());
        for (size_t i = 0; i < ord.size(); i++) {
            const int j = piv[ord[i]].first;
            const auto r = dg_of(j);
            const int q0 = at(b);
            int *rec = &b[op + 4 * i];
            rec[0] = j;
            rec[1] = q0;
            rec[2] = q0 + r.second - r.first;
            rec[3] = piv[ord[i]].second;
            for (int q = r.first; q < r.second; q++) pair(b, S.dg_pos[q], S.dg_k[q]);
            md = std::max<long long>(md, r.second - r.first);
            sd += r.second - r.first;
        }
        pad4(b);
        const int oe = (int)b.size();
        b.resize(b.size() + 4 * ent.size());
        for (size_t i = 0; i < ent.size(); i++) {
            const auto r = og_of(ent[i].p);
            const int q0 = at(b);
            int *rec = &b[oe + 4 * i];
            rec[0] = ent[i].p;
            rec[1] = q0;
            rec[2] = q0 + (int)(r.second - r.first);
            rec[3] = kind == 0 ? back[ent[i].piv] : ent[i].piv;
            for (long long q = r.first; q < r.second; q++) pair(b, S.og_a[q], S.og_b[q]);
            me = std::max<long long>(me, r.second - r.first);
            se += r.second - r.first;
        }
        // (the segment's gather into the tail keeps a block on one lane)
        const int mem = kind < 2 ? 700 : 60;
        const Lanes a = pick_lanes((long long)piv.size(), md, sd, 12, 6, kind & 1 ? 0 : 20, mem, fp64 && kind != 3);
        const Lanes e = pick_lanes((long long)ent.size(), me, se, 16, 8, kind & 1 ? 0 : 8, mem, fp64 && kind != 3);
        // the entries start on the warp after the pivots'
        const int rot = (W - std::min<int>(1 << a.lw, (int)piv.size())) % W;
        int *h = &b[head];
        h[0] = (int)piv.size(); h[1] = (int)ent.size(); h[2] = op; h[3] = oe;
        h[4] = a.g | e.g << 3 | a.quad << 6 | e.quad << 7 | a.lw << 8 | e.lw << 11 | (e.passes == 1) << 14 | rot << 16;
        if (kind == 0) R.max_pivots = std::max(R.max_pivots, (int)piv.size());
    };
    for (int l = 0; l < R.nf1; l++) {
        const std::vector<int> &st = L.f1[l];
        std::vector<std::vector<Piv>> piv(ctas);
        std::vector<std::vector<LevelEnt>> ent(ctas);
        auto ents = [&](int j, int at, std::vector<LevelEnt> &out) {
            for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++)
                out.push_back({p, (int)(S.og_ptr[p + 1] - S.og_ptr[p]), at});
        };
        if ((int)st.size() >= ctas) {
            // a pivot and its entries on one CTA, the heaviest first to the least loaded
            std::vector<std::pair<long long, int>> w;
            for (int j : st) {
                long long k = 4 + S.dg_ptr[j + 1] - S.dg_ptr[j];
                for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++) k += 2 + 2 * (S.og_ptr[p + 1] - S.og_ptr[p]);
                w.push_back({-k, j});
            }
            std::sort(w.begin(), w.end());
            std::priority_queue<std::pair<long long, int>, std::vector<std::pair<long long, int>>, std::greater<>> q;
            for (int c = 0; c < ctas; c++) q.push({0, c});
            for (const auto &x : w) {
                auto t = q.top();
                q.pop();
                piv[t.second].push_back({x.second, 1});
                ents(x.second, (int)piv[t.second].size() - 1, ent[t.second]);
                t.first -= x.first;
                q.push(t);
            }
        } else {
            // fewer pivots than CTAs: the level's entries in runs of about equal
            // work, and every CTA with an entry of a pivot computes that pivot
            // for itself (the first one stores it)
            std::vector<LevelEnt> all;
            for (size_t i = 0; i < st.size(); i++) ents(st[i], (int)i, all);
            long long total = 0, run = 0;
            for (const auto &e : all) total += 1 + e.len;
            std::vector<int> first(st.size(), -1);
            std::vector<std::vector<int>> pos(ctas, std::vector<int>(st.size(), -1));
            for (const auto &e : all) {
                const int c = (int)std::min<long long>(ctas - 1, run * ctas / std::max<long long>(total, 1));
                run += 1 + e.len;
                if (pos[c][e.piv] < 0) {
                    pos[c][e.piv] = (int)piv[c].size();
                    piv[c].push_back({st[e.piv], first[e.piv] < 0});
                    if (first[e.piv] < 0) first[e.piv] = c;
                }
                ent[c].push_back({e.p, e.len, pos[c][e.piv]});
            }
            for (size_t i = 0; i < st.size(); i++)
                if (first[i] < 0) piv[(int)i % ctas].push_back({st[i], 1});  // a pivot without entries
        }
        for (int c = 0; c < ctas; c++) put_level(part[c], 8 * (size_t)l, piv[c], ent[c], 0);
    }
    {
        // the cluster's updates of the segment's and the tail's blocks, spread
        // over all CTAs
        std::vector<std::vector<Piv>> piv(ctas);
        std::vector<std::vector<LevelEnt>> ent(ctas);
        for (int j = t0, c = 0; j < n; j++, c++) piv[c % ctas].push_back({j, 1});
        std::vector<std::pair<long long, int>> w;
        for (int p = S.up_ptr[t0]; p < S.nup; p++) {
            const long long k = og_cut(p, t0) - S.og_ptr[p];
            if (k) w.push_back({-k, p});
        }
        std::sort(w.begin(), w.end());
        for (size_t i = 0; i < w.size(); i++) ent[i % ctas].push_back({w[i].second, (int)-w[i].first, 0});
        for (int q = 0; q < ctas; q++) put_level(part[q], 8 * (size_t)R.nf1, piv[q], ent[q], 1);
    }
    for (int l = 0; l < R.nfs; l++) {
        std::vector<Piv> piv;
        std::vector<LevelEnt> ent;
        for (int j : L.fs[l]) {
            piv.push_back({j, 1});
            for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++)
                ent.push_back({p, (int)(S.og_ptr[p + 1] - og_cut(p, t0)), j});
        }
        put_level(part[0], 8 * (size_t)(R.nf1 + 1 + l), piv, ent, 2);
    }
    if (t0 < td && td < n) {
        std::vector<Piv> piv;
        std::vector<LevelEnt> ent;
        for (int j = td; j < n; j++)
            if (dg_cut(j, td) > dg_cut(j, t0)) piv.push_back({j, 1});
        for (int j = td; j < n; j++)
            for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++) {
                const long long k = og_cut(p, td) - og_cut(p, t0);
                if (k) ent.push_back({p, (int)k, (S.up_col[p] - td) << 16 | (j - td)});
            }
        put_level(part[0], 8 * (size_t)(R.nf1 + 1 + R.nfs), piv, ent, 3);
    }
    for (int l = 0; l < R.nbs + R.nb1; l++) {
        const bool in_seg = l < R.nbs;
        std::vector<int> ord = in_seg ? L.bs[l] : L.b1[l - R.nbs];
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int c) {
            return S.up_ptr[a + 1] - S.up_ptr[a] > S.up_ptr[c + 1] - S.up_ptr[c];
        });
        for (int c = 0; c < (in_seg ? 1 : ctas); c++) {
            std::vector<int> &b = part[c];
            std::vector<int> mine;
            for (size_t i = c; i < ord.size(); i += in_seg ? 1 : ctas) mine.push_back(ord[i]);
            pad4(b);
            const int o = (int)b.size();
            b.resize(b.size() + 4 * mine.size());
            long long mu = 0, su = 0;
            for (size_t i = 0; i < mine.size(); i++) {
                const int j = mine[i], k = S.up_ptr[j + 1] - S.up_ptr[j];
                const int q0 = at(b);
                int *rec = &b[o + 4 * i];
                rec[0] = j;
                rec[1] = q0;
                rec[2] = q0 + k;
                for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1]; p++) pair(b, p, S.up_col[p]);
                mu = std::max<long long>(mu, k);
                su += k;
            }
            const Lanes a = pick_lanes((long long)mine.size(), mu, su, 4, 2, 4, in_seg ? 60 : 700, fp64);
            int *h = &b[heads + 4 * (size_t)l];
            h[0] = (int)mine.size(); h[1] = o; h[2] = a.g | a.lw << 8;
        }
    }
    R.off.push_back(0);
    for (auto &b : part) {
        pad4(b);
        R.blob.insert(R.blob.end(), b.begin(), b.end());
        R.off.push_back((int)R.blob.size());
        R.max_ints = std::max(R.max_ints, (int)b.size());
    }
    R.inv_bytes = up128(b4 * (size_t)R.max_pivots);
    R.seg_bytes = seg_bytes(t0);
    R.vec_bytes = vec_bytes(t0);
    R.tail_bytes = tail_bytes();
    const size_t used = R.inv_bytes + R.seg_bytes + R.vec_bytes + R.tail_bytes;
    R.sched_bytes = used + 4 * (size_t)R.max_ints <= limit ? 4 * (size_t)R.max_ints : 0;
    return R;
}

}  // namespace

// The schedule with the tail from td on.
static ClusterSchedule schedule_with_tail(const Symbolic &S, int ctas, int td, bool fp64, size_t limit) {
    const int n = S.n;
    // FP64: one SM's pipe cannot carry a tail of this size (8 multiply-adds a
    // block and step at two a cycle), so its columns go round the cluster
    const ClusterBuilder B{S, n, ctas, td, fp64, limit, fp64 ? 32u : 16u, fp64 ? 16u : 8u, fp64 && td < n ? ctas : 1};
    // the cheapest segment (by estimate) whose schedule fits shared memory
    // beside it; if none does, the cheapest, its schedule in global memory
    std::vector<std::pair<double, int>> fits, rest;
    for (int m = 0;; m = std::min(td, std::max(m + 8, m + m / 2))) {
        const int t0 = td - m;
        const size_t used = B.seg_bytes(t0) + B.vec_bytes(t0) + B.tail_bytes();
        if (used > limit) break;
        size_t bytes = 0;
        const double c = B.estimate(t0, bytes);
        (used + bytes <= limit ? fits : rest).push_back({c, t0});
        if (m == td) break;
    }
    std::sort(fits.begin(), fits.end());
    std::sort(rest.begin(), rest.end());
    ClusterSchedule best;
    for (const auto *v : {&fits, &rest})
        for (const auto &c : *v) {
            ClusterSchedule R = B.build(c.second);
            if (R.inv_bytes + R.seg_bytes + R.vec_bytes + R.tail_bytes > limit) continue;
            if (R.sched_bytes) return R;
            if (!best.ctas) best = std::move(R);
            if (v == &rest) return best;
        }
    return best;
}

ClusterSchedule cluster_schedule(const Symbolic &S, int ctas, bool fp64, size_t limit) {
    const int n = S.n;
    int td = n;
    while (td > 0 && n - td < (fp64 ? kTailMax : kTailMax32) && S.up_ptr[td] - S.up_ptr[td - 1] == n - td) td--;
    // the whole dense trailing block, or less of it where the schedule would
    // not fit shared memory beside it (15,104 buses in FP32: 2.00 ms a solve
    // with the schedule in global memory, 1.8 with a tail of 53 instead of 61)
    ClusterSchedule first;
    for (; n - td >= kTailMin; td += 8) {
        ClusterSchedule R = schedule_with_tail(S, ctas, td, fp64, limit);
        if (R.sched_bytes) return R;
        if (!first.ctas) first = std::move(R);
    }
    return first.ctas ? first : schedule_with_tail(S, ctas, n, fp64, limit);
}

}  // namespace gbpf

extern "C" gbpf_status gbpf_grid_analyse(const gbpf_grid *h, long long info[8]) {
    if (!h || !info) return GBPF_E_ARG;
    const gbpf::Grid &g = h->g;
    if (g.nB < 2 || g.slack < 1) return GBPF_E_INPUT;
    const gbpf::YPattern y = gbpf::build_ypattern(g);
    std::string why;
    const gbpf::Symbolic S = gbpf::analyse(g, y, &why);
    if (S.n != g.nB - 1) {
        gbpf::set_error("symbolic analysis failed: " + why);
        return GBPF_E_INPUT;
    }
    long long jblocks = 0;
    for (int q = 0; q < S.n + 2 * S.nup; q++) jblocks += S.ysl[q] >= 0;
    // closure: every pair target (a, b) of entry p lies in an earlier step's row
    bool closed = true;
    for (int j = 0; j < S.n && closed; j++)
        for (int p = S.up_ptr[j]; p < S.up_ptr[j + 1] && closed; p++)
            for (long long r = S.og_ptr[p]; r < S.og_ptr[p + 1]; r++)
                if (S.og_a[r] >= S.up_ptr[j] || S.og_b[r] >= S.up_ptr[j]) { closed = false; break; }
    info[0] = S.n;
    info[1] = S.nup;
    info[2] = S.pairs();
    info[3] = (long long)S.flev_ptr.size() - 1;
    info[4] = (long long)S.blev_ptr.size() - 1;
    info[5] = y.nnz;
    info[6] = jblocks;
    info[7] = closed ? 1 : 0;
    return GBPF_OK;
}
