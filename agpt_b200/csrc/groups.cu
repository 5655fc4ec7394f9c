// Launch groups straight from a radix trie.
//
// A launch group is a forest of char positions in depth-first order.  Its rows come in runs -- the chars of one radix edge
// are consecutive rows with one parent run, one subtree end, one unit -- and a trie has an order of magnitude fewer edges
// than chars.  So everything that needs decisions (depth-first order, units, packing, subtree ends, ancestor chains'
// offsets, the dK/dV reduction list, mass weights) is done per run on the host, one packed copy goes up, and a kernel
// writes what the training step reads per row.  Arrays are those of the char-level path (trie_char_tree, plan_create,
// groups_create), which walked 1.7M positions for what 92,000 edges say: 199 -> 18 ms from a 60k-token corpus to its group.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "../../include/agpt_b200.h"
#include "internal.h"

namespace {

struct RunGroup {
    std::vector<int32_t> rid, prun, unit, qoff;          // radix id, parent run (-1: root), unit, first row (E + 1 entries)
    std::vector<uint8_t> trained;
    int32_t n_units = 0;
    int64_t rows() const { return qoff.empty() ? 0 : qoff.back(); }
    bool full(const agpt_trie *t, int32_t r) const { return rows() + t->edge_len[r] >= (1LL << 31) - 256; }      // ask before add
    int32_t add(const agpt_trie *t, int32_t r, int32_t parent, int32_t u, bool tr) {
        if (qoff.empty()) qoff.push_back(0);
        rid.push_back(r); prun.push_back(parent); unit.push_back(u); trained.push_back(tr);
        qoff.push_back(qoff.back() + t->edge_len[r]);
        return (int32_t)rid.size() - 1;
    }
};

// Radix nodes in depth-first order: siblings by their first char position.
struct RadixOrder {
    std::vector<int32_t> at, rank, end;      // node at each place, place of each node, one past the node's subtree (places)
    std::vector<int64_t> rows;               // char positions of each node's subtree
    std::vector<int32_t> kids;               // children of each node
};
int radix_order(const agpt_trie *t, RadixOrder &o) {
    const int32_t R = t->radix_count;
    for (int32_t r = 1; r < R; r++)
        if (t->parent[r] < 0 || t->parent[r] >= r) return agpt_set_error(AGPT_E_ARG, "trie_groups: radix node %d does not follow its parent", r);
    o.at.assign(R > 1 ? R - 1 : 0, 0); o.rank.assign(R, 0); o.end.assign(R, 0); o.rows.assign(R, 0); o.kids.assign(R, 0);
    std::vector<int32_t> size(R, 0), next(R, 0);
    for (int32_t r = R - 1; r >= 1; r--) {
        size[r] += 1; o.rows[r] += t->edge_len[r];
        size[t->parent[r]] += size[r]; o.rows[t->parent[r]] += o.rows[r]; o.kids[t->parent[r]]++;
    }
    // char positions follow (endpoint depth, id): visiting the nodes in that order hands every parent its children in order
    std::vector<int64_t> first(t->n_depth_files + 1, 0);
    for (int32_t r = 1; r < R; r++) first[t->endpoint_depth[r] + 1]++;
    for (int d = 0; d < t->n_depth_files; d++) first[d + 1] += first[d];
    std::vector<int32_t> by(R > 1 ? R - 1 : 0);
    for (int32_t r = 1; r < R; r++) by[first[t->endpoint_depth[r]]++] = r;
    // a child's endpoint lies deeper than its parent's, so parents are placed first
    for (int32_t r : by) {
        const int32_t p = t->parent[r], at = next[p];
        next[p] += size[r];
        o.rank[r] = at; o.at[at] = r; o.end[r] = at + size[r];
        next[r] = at + 1;
    }
    return AGPT_OK;
}

__global__ void __launch_bounds__(256) expand_runs_kernel(const int32_t *__restrict__ qoff, const int32_t *__restrict__ fd, const int32_t *__restrict__ ld,
                                                           const int32_t *__restrict__ send, const int32_t *__restrict__ unit, const int32_t *__restrict__ first,
                                                           const float *__restrict__ mw, const uint8_t *__restrict__ tr, int runs, int seq_len,
                                                           int32_t *__restrict__ pos, int32_t *__restrict__ q2n, int32_t *__restrict__ edge_first,
                                                           int64_t *__restrict__ unit_row, float *__restrict__ mass, float *__restrict__ trained,
                                                           int32_t *__restrict__ depth, int32_t *__restrict__ sub_end) {
    const int e = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (e >= runs) return;
    const int q0 = qoff[e], len = qoff[e + 1] - q0;
    for (int j = threadIdx.x & 31; j < len; j += 32) {
        const int r = q0 + j;
        pos[r] = min(max(fd[e] + j - 1, 0), seq_len - 1);
        q2n[r] = e; edge_first[r] = first[e]; unit_row[r] = unit[e];
        if (mass) mass[r] = mw[e];
        if (trained) trained[r] = tr[e] ? 1.f : 0.f;
        depth[r] = ld[e] + j; sub_end[r] = send[e];
    }
}

// ancestor chain of the first row of every tile, root side first: up its own run, then run by run
__global__ void __launch_bounds__(128) tile_chain_kernel(const int32_t *__restrict__ qoff, const int32_t *__restrict__ prun, const int32_t *__restrict__ send,
                                                          const int64_t *__restrict__ chain_off, const int32_t *__restrict__ tile_start, int runs, int64_t tiles,
                                                          int32_t *__restrict__ ids, int32_t *__restrict__ ends) {
    const int64_t t = (int64_t)blockIdx.x * 128 + threadIdx.x;
    if (t >= tiles) return;
    int row = tile_start[t], lo = 0, hi = runs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (qoff[mid] <= row) lo = mid; else hi = mid - 1;
    }
    int e = lo, a = row - 1;                   // the next ancestor
    for (int64_t j = chain_off[t + 1] - 1; j >= chain_off[t]; j--) {
        if (a < qoff[e]) { e = prun[e]; a = qoff[e + 1] - 1; }
        ids[j] = a; ends[j] = send[e];
        a--;
    }
}

int64_t up16(int64_t x) { return (x + 15) & ~(int64_t)15; }

}  // namespace

struct agpt_run_groups {
    const agpt_trie *trie = nullptr;
    std::vector<RunGroup> groups;
    // of the group made ready last
    int64_t ready = -1;
    std::unique_ptr<uint8_t[], agpt_big_free> staging;
    int64_t staged = 0;
    agpt_plan *plan = nullptr;
    bool even = false;                        // of the plans made from here on
    agpt_run_group_info info;
    int64_t at_prun = 0, at_fd = 0, at_ld = 0, at_send = 0, at_unit = 0, at_first = 0, at_mw = 0, at_tr = 0, at_choff = 0, at_items[4] = {0, 0, 0, 0},
            at_multi = 0, at_mcount = 0, at_mfirst = 0, at_ts = 0, at_depth = 0, at_subend = 0, at_cid = 0, at_cend = 0;
    ~agpt_run_groups() { delete plan; }
};

extern "C" int agpt_b200_trie_groups_create(const agpt_trie *t, int level, int64_t unit_cap, int n_ranks, int rank, int64_t group_rows,
                                            agpt_run_groups **out) try {
    if (!t || !out || (level != 1 && level != 2) || n_ranks < 1 || rank < 0 || rank >= n_ranks || group_rows < 1)
        return agpt_set_error(AGPT_E_ARG, "trie_groups: bad argument");
    RadixOrder o;
    if (int rc = radix_order(t, o)) return rc;
    // units as ranges of places, in depth-first order (agpt_b200_plan_units and the deeper cut of units_capped, per run)
    std::vector<std::pair<int32_t, int32_t>> units, stack;
    const int32_t places = (int32_t)o.at.size();
    auto rows_of = [&](int32_t b, int32_t e) {
        int64_t n = 0;
        for (int32_t i = b; i < e; i = o.end[o.at[i]]) n += o.end[o.at[i]] <= e ? o.rows[o.at[i]] : (int64_t)t->edge_len[o.at[i]];
        return n;
    };
    auto cut = [&](int32_t b, int32_t e, bool whole) {       // whole: [b, e) is one subtree
        if (unit_cap <= 0 || !whole) { units.emplace_back(b, e); return; }
        stack.clear();
        stack.emplace_back(b, e);
        while (!stack.empty()) {
            const auto [x, y] = stack.back();
            stack.pop_back();
            if (o.rows[o.at[x]] <= unit_cap) { units.emplace_back(x, y); continue; }
            int32_t j = x;                                       // the unary chain at the top
            while (j + 1 < y && o.end[o.at[j + 1]] == y) j++;
            if (j + 1 >= y) { units.emplace_back(x, y); continue; }
            units.emplace_back(x, j + 1);
            const size_t from = stack.size();
            for (int32_t c = j + 1; c < y; c = o.end[o.at[c]]) stack.emplace_back(c, o.end[o.at[c]]);
            std::reverse(stack.begin() + from, stack.end());
        }
    };
    for (int32_t a = 0; a < places; a = o.end[o.at[a]]) {
        const int32_t r = o.at[a], e = o.end[r];
        // a depth-1 char with a single child stays with it: its edge runs on, or it has one child edge
        if (level == 1 || t->edge_len[r] > 1 || o.kids[r] == 1) { cut(a, e, true); continue; }
        units.emplace_back(a, a + 1);
        for (int32_t c = a + 1; c < e; c = o.end[o.at[c]]) cut(c, o.end[o.at[c]], true);
    }
    std::vector<int64_t> weight(units.size());
    for (size_t u = 0; u < units.size(); u++) weight[u] = rows_of(units[u].first, units[u].second);
    std::vector<int32_t> owner(units.size(), 0);
    if (int rc = agpt_b200_partition_lpt(weight.data(), (int64_t)units.size(), n_ranks, owner.data())) return rc;

    auto G = std::make_unique<agpt_run_groups>();
    G->trie = t;
    RunGroup cur;
    auto flush = [&]() { if (cur.rows()) { G->groups.push_back(std::move(cur)); cur = RunGroup(); } };
    std::vector<int32_t> chain;
    for (size_t u = 0; u < units.size(); u++) {
        if (owner[u] != rank) continue;
        const int32_t b = units[u].first, e = units[u].second;
        // a unit that does not start at the root carries its ancestors as context rows (attended, not trained)
        chain.clear();
        int64_t k = 0;
        for (int32_t p = t->parent[o.at[b]]; p > 0; p = t->parent[p]) { chain.push_back(p); k += t->edge_len[p]; }
        if (cur.rows() && cur.rows() + k + weight[u] > group_rows) flush();
        if (cur.rows() + k + weight[u] >= (1LL << 31) - 256) return agpt_set_error(AGPT_E_LIMIT, "trie_groups: more than 2^31 rows in one group");
        const int32_t unit = cur.n_units++;
        int32_t above = -1;
        for (size_t i = chain.size(); i-- > 0;) above = cur.add(t, chain[i], above, unit, false);
        const int32_t off = (int32_t)cur.rid.size();
        for (int32_t i = b; i < e; i++) {
            const int32_t r = o.at[i], p = t->parent[r];
            cur.add(t, r, i == b ? above : (p == 0 || o.rank[p] < b ? -1 : off + o.rank[p] - b), unit, true);
        }
    }
    flush();
    *out = G.release();
    return AGPT_OK;
} AGPT_CATCH("trie_groups_create")

// The group of a set of radix nodes closed under "parent" (a sampled training unit): rows in depth-first order, one unit.
// order: a depth-first rank per radix node (agpt_b200_trie_ranks), kept by the caller between samples.
extern "C" int agpt_b200_trie_ranks(const agpt_trie *t, int32_t *rank_out) try {
    if (!t || !rank_out) return agpt_set_error(AGPT_E_ARG, "trie_ranks: null");
    RadixOrder o;
    if (int rc = radix_order(t, o)) return rc;
    std::copy(o.rank.begin(), o.rank.end(), rank_out);
    return AGPT_OK;
} AGPT_CATCH("trie_ranks")

extern "C" int agpt_b200_trie_sample_group(const agpt_trie *t, const int32_t *rank, const int32_t *nodes, int64_t n_nodes, const int32_t *context,
                                           int64_t n_context, agpt_run_groups **out) try {
    if (!t || !rank || !nodes || !out || n_nodes < 1 || n_context < 0 || (n_context && !context)) return agpt_set_error(AGPT_E_ARG, "trie_sample_group: bad argument");
    std::vector<std::pair<int32_t, int32_t>> by((size_t)n_nodes);        // (rank, node)
    for (int64_t i = 0; i < n_nodes; i++) {
        if (nodes[i] < 1 || nodes[i] >= t->radix_count) return agpt_set_error(AGPT_E_ARG, "trie_sample_group: node %d out of range", nodes[i]);
        by[i] = {rank[nodes[i]], nodes[i]};
    }
    std::sort(by.begin(), by.end());
    std::vector<int32_t> ctx(context, context + n_context);
    std::sort(ctx.begin(), ctx.end());
    auto G = std::make_unique<agpt_run_groups>();
    G->trie = t;
    G->groups.emplace_back();
    RunGroup &g = G->groups[0];
    g.n_units = 1;
    std::vector<std::pair<int32_t, int32_t>> open;                        // (node, run) from the root to the current place
    for (const auto &x : by) {
        const int32_t r = x.second, p = t->parent[r];
        while (!open.empty() && open.back().first != p) open.pop_back();
        if (p > 0 && open.empty()) return agpt_set_error(AGPT_E_ARG, "the node set is not closed under parent");
        if (g.full(t, r)) return agpt_set_error(AGPT_E_LIMIT, "trie_sample_group: more than 2^31 rows");
        const int32_t e = g.add(t, r, p > 0 ? open.back().second : -1, 0, !std::binary_search(ctx.begin(), ctx.end(), r));
        open.emplace_back(r, e);
    }
    *out = G.release();
    return AGPT_OK;
} AGPT_CATCH("trie_sample_group")

extern "C" int64_t agpt_b200_trie_groups_count(const agpt_run_groups *G) { return G ? (int64_t)G->groups.size() : 0; }
extern "C" void agpt_b200_trie_groups_free(agpt_run_groups *G) { delete G; }
extern "C" int agpt_b200_trie_groups_even(agpt_run_groups *G, int even) {
    if (!G) return agpt_set_error(AGPT_E_ARG, "trie_groups_even: null");
    G->even = even != 0;
    return AGPT_OK;
}

extern "C" int agpt_b200_trie_group_prepare(agpt_run_groups *G, int64_t i, int tile_m, int mass_mode, int seq_len, agpt_run_group_info *out) try {
    if (!G || !out || i < 0 || i >= (int64_t)G->groups.size() || seq_len < 1 || mass_mode < 0 || mass_mode > 3 || (tile_m != 32 && tile_m != 64 && tile_m != 128))
        return agpt_set_error(AGPT_E_ARG, "trie_group_prepare: bad argument");
    const RunGroup &g = G->groups[i];
    const agpt_trie *t = G->trie;
    const int32_t E = (int32_t)g.rid.size();
    const int64_t n = g.rows(), M = tile_m;
    G->ready = -1;                              // until this one is complete
    delete G->plan;
    G->plan = nullptr;
    agpt_plan *P = G->plan = new agpt_plan();
    P->n = n; P->tile_m = tile_m; P->even = G->even;
    P->lazy = true;
    P->run_qoff.assign(g.qoff.begin(), g.qoff.end()); P->run_parent = g.prun;
    std::vector<int32_t> &ld = P->run_depth, &send = P->run_end;
    ld.resize(E); send.assign(E, 0);
    bool roots = false;
    for (int32_t e = 0; e < E; e++) ld[e] = g.prun[e] < 0 ? 1 : ld[g.prun[e]] + (g.qoff[g.prun[e] + 1] - g.qoff[g.prun[e]]);
    for (int32_t e = E - 1; e >= 0; e--) {
        if (send[e] < g.qoff[e + 1]) send[e] = g.qoff[e + 1];
        const int32_t p = g.prun[e];
        if (p >= 0) send[p] = std::max(send[p], send[e]); else roots = true;
    }
    // sums of the bytes model: every char but an edge's last has one child, the last has some if the subtree goes on
    P->n_groups = roots ? 1 : 0;
    for (int32_t e = 0; e < E; e++) {
        const int64_t len = g.qoff[e + 1] - g.qoff[e], d0 = ld[e];
        P->max_depth = std::max<int32_t>(P->max_depth, (int32_t)(d0 + len - 1));
        P->sum_depth += len * d0 + len * (len - 1) / 2;
        const int64_t inner = len - (send[e] > g.qoff[e + 1] ? 0 : 1);
        P->n_groups += inner; P->sum_group_prefix += inner * d0 + inner * (inner - 1) / 2;
    }
    // tiles, as agpt_b200_plan_create cuts them: depths grow along a run, so only its first row in reach can be a better end
    std::vector<int32_t> &ts = P->tile_start;
    ts.reserve(n / 32 + 2);
    P->chain_off.reserve(n / 32 + 2);
    P->chain_off.push_back(0);
    int64_t e0 = 0;                             // the run of the tile's first row
    for (int64_t r0 = 0; r0 < n;) {
        ts.push_back((int32_t)r0);
        int64_t k = std::min(M, n - r0), e1 = e0;
        if (tile_m == 64 && !P->even && r0 + M < n) {
            while (g.qoff[e1 + 1] <= r0 + 32) e1++;
            int64_t b = g.qoff[e1] == r0 + 32 ? e1 : e1 + 1;            // the first run from row 32 on that does not hang on the one before it
            while (b < E && g.prun[b] == b - 1) b++;
            const int64_t branch = (b < E ? (int64_t)g.qoff[b] : n) - r0;
            if (branch > M) {
                k = agpt_tile_of_chain(branch);
                while (g.qoff[e1 + 1] <= r0 + k) e1++;
            } else {
                int64_t best = INT64_MAX;
                for (int64_t e = e1; e < E && g.qoff[e] <= r0 + M; e++) {
                    const int64_t c = std::max<int64_t>(g.qoff[e] - r0, 32), v = agpt_tile_cost((int32_t)(ld[e] + (r0 + c - g.qoff[e])), c);
                    if (v <= best) { best = v; k = c; e1 = e; }
                }
            }
        } else while (e1 < E && g.qoff[e1 + 1] <= r0 + k) e1++;
        const int64_t chain = ld[e0] + (r0 - g.qoff[e0]) - 1;
        P->chain_off.push_back(P->chain_off.back() + chain);
        P->max_keys = std::max(P->max_keys, (int32_t)(chain + k));
        r0 += k; e0 = e1;
    }
    P->n_tiles = (int64_t)ts.size();
    ts.push_back((int32_t)n);
    P->chain_rows = P->chain_off[P->n_tiles];
    // reduction work list: the rows whose subtree reaches into later tiles, ordered by their last tile (a counting sort)
    {
        const int32_t SEG = P->even ? (int32_t)P->n_tiles : AGPT_REDUCE_SEG;
        std::vector<int64_t> start(P->n_tiles + 1, 0);
        std::vector<int32_t> last_tile(E);      // tile of the last row of a run's subtree
        {   // of every run's last row first; a run's subtree ends with a run's last row
            std::vector<int32_t> run_end_tile(E);
            for (int32_t e = 0, t = 0; e < E; e++) {
                while (ts[t + 1] < g.qoff[e + 1]) t++;
                run_end_tile[e] = t;
            }
            for (int32_t e = E - 1; e >= 0; e--) last_tile[e] = run_end_tile[e];
            for (int32_t e = E - 1; e >= 0; e--)
                if (g.prun[e] >= 0) last_tile[g.prun[e]] = std::max(last_tile[g.prun[e]], last_tile[e]);
        }
        // f(first row, one past the last row, first tile, last tile): the rows of a run that lie in one tile
        auto each = [&](auto &&f) {
            int32_t t = 0;
            for (int32_t e = 0; e < E; e++) {
                const int32_t t1 = last_tile[e], last = std::min(g.qoff[e + 1], ts[t1]);
                while (ts[t + 1] <= g.qoff[e]) t++;
                for (int32_t a = g.qoff[e], u = t; a < last; u++) {
                    const int32_t b = std::min(last, ts[u + 1]);
                    f(a, b, u + 1, t1);
                    a = b;
                }
            }
        };
        each([&](int32_t a, int32_t b, int32_t t0, int32_t t1) {
            for (int32_t s = t0; s <= t1; s += SEG) start[std::min(t1, s + SEG - 1) + 1] += b - a;
        });
        for (int64_t tl = 0; tl < P->n_tiles; tl++) start[tl + 1] += start[tl];
        const size_t items = (size_t)start[P->n_tiles];
        P->item_node.resize(items); P->item_t0.resize(items); P->item_t1.resize(items); P->item_slot.resize(items);
        each([&](int32_t a, int32_t b, int32_t t0, int32_t t1) {
            const int32_t nseg = (t1 - t0 + SEG) / SEG;
            P->n_reduce_nodes += b - a;
            if (nseg == 1) {
                int64_t at = start[t1];
                start[t1] += b - a;
                for (; a < b; a++, at++) { P->item_node[at] = a; P->item_t0[at] = t0; P->item_t1[at] = t1; P->item_slot[at] = -1; }
                return;
            }
            for (; a < b; a++) {
                P->multi_node.push_back(a); P->multi_first.push_back(P->n_multi_items); P->multi_count.push_back(nseg);
                for (int32_t s = t0; s <= t1; s += SEG) {
                    const int32_t end = std::min(t1, s + SEG - 1);
                    const int64_t at = start[end]++;
                    P->item_node[at] = a; P->item_t0[at] = s; P->item_t1[at] = end; P->item_slot[at] = (int32_t)P->n_multi_items++;
                }
            }
        });
    }

    // layout: what is copied up, then what the kernels write
    int64_t at = 0;
    auto take = [&](int64_t bytes) { const int64_t p = at; at += up16(bytes); return p; };
    agpt_run_group_info &o = G->info;
    o = agpt_run_group_info();
    o.n = n; o.n_loss_nodes = E; o.n_units = g.n_units;
    o.qoff = take((int64_t)(E + 1) * 4); o.rid = take((int64_t)E * 4);
    G->at_prun = take((int64_t)E * 4); G->at_fd = take((int64_t)E * 4); G->at_ld = take((int64_t)E * 4); G->at_send = take((int64_t)E * 4);
    G->at_unit = take((int64_t)E * 4); G->at_first = take((int64_t)E * 4); G->at_mw = take((int64_t)E * 4); G->at_tr = take(E);
    G->at_choff = take((P->n_tiles + 1) * 8); G->at_ts = take((P->n_tiles + 1) * 4);
    const std::vector<int32_t> *items[4] = {&P->item_node, &P->item_t0, &P->item_t1, &P->item_slot};
    for (int k = 0; k < 4; k++) G->at_items[k] = take((int64_t)items[k]->size() * 4);
    const int64_t nm = (int64_t)P->multi_node.size();
    G->at_multi = take(nm * 4); G->at_mcount = take(nm * 4); G->at_mfirst = take(nm * 8);
    o.unit_off = take((int64_t)(g.n_units + 1) * 8);
    o.tokens = take(n * 4);
    G->staged = at;
    bool all = true;
    int64_t n_trained = 0, deepest = 0;
    for (int32_t e = 0; e < E; e++) {
        const int64_t len = g.qoff[e + 1] - g.qoff[e];
        if (g.trained[e]) n_trained += len; else all = false;
        deepest = std::max<int64_t>(deepest, t->first_char_depth[g.rid[e]] + len - 1);
    }
    o.n_trained = n_trained;
    o.n_pos = (int32_t)std::min<int64_t>(std::max<int64_t>(deepest - 1, 0), seq_len - 1) + 1;
    o.pos = take(n * 4); o.q2n = take(n * 4); o.edge_first = take(n * 4); o.unit_of_row = take(n * 8);
    o.mass_w = mass_mode ? take(n * 4) : -1;
    o.trained = all ? -1 : take(n * 4);
    G->at_depth = take(n * 4); G->at_subend = take(n * 4); G->at_cid = take(P->chain_rows * 4); G->at_cend = take(P->chain_rows * 4);
    o.bytes = std::max<int64_t>(at, 16);
    o.seq_len = seq_len;

    G->staging.reset((uint8_t *)agpt_big_alloc((size_t)std::max<int64_t>(G->staged, 16)));
    if (!G->staging) return agpt_set_error(AGPT_E_NOMEM, "trie_group_prepare: out of host memory");
    uint8_t *s = G->staging.get();
    auto put = [&](int64_t where, const void *src, int64_t bytes) { if (bytes) memcpy(s + where, src, (size_t)bytes); };
    put(o.qoff, g.qoff.data(), (int64_t)(E + 1) * 4); put(o.rid, g.rid.data(), (int64_t)E * 4);
    put(G->at_prun, g.prun.data(), (int64_t)E * 4); put(G->at_ld, ld.data(), (int64_t)E * 4); put(G->at_send, send.data(), (int64_t)E * 4);
    put(G->at_unit, g.unit.data(), (int64_t)E * 4); put(G->at_tr, g.trained.data(), E);
    put(G->at_choff, P->chain_off.data(), (P->n_tiles + 1) * 8); put(G->at_ts, P->tile_start.data(), (P->n_tiles + 1) * 4);
    for (int k = 0; k < 4; k++) put(G->at_items[k], items[k]->data(), (int64_t)items[k]->size() * 4);
    put(G->at_multi, P->multi_node.data(), nm * 4); put(G->at_mcount, P->multi_count.data(), nm * 4); put(G->at_mfirst, P->multi_first.data(), nm * 8);
    int32_t *fd = (int32_t *)(s + G->at_fd), *first = (int32_t *)(s + G->at_first), *tok = (int32_t *)(s + o.tokens);
    int64_t *uoff = (int64_t *)(s + o.unit_off);
    for (int32_t e = 0, u = 0; e < E; e++) {
        const int32_t r = g.rid[e];
        fd[e] = t->first_char_depth[r];
        // first row of the rows of one radix edge that follow each other (two units may share an edge at their border)
        first[e] = e > 0 && g.rid[e - 1] == r ? first[e - 1] : g.qoff[e];
        memcpy(tok + g.qoff[e], t->edge_tok.data() + t->edge_off[r], (size_t)(g.qoff[e + 1] - g.qoff[e]) * 4);
        for (; u <= g.unit[e]; u++) uoff[u] = g.qoff[e];
    }
    uoff[g.n_units] = n;
    if (mass_mode) {
        std::vector<int32_t> em(E), el(E);
        for (int32_t e = 0; e < E; e++) { em[e] = t->edge_mass[g.rid[e]]; el[e] = g.qoff[e + 1] - g.qoff[e]; }
        if (int rc = agpt_mass_weights_per_node(em.data(), el.data(), g.unit.data(), g.trained.data(), E, std::max(1, g.n_units), mass_mode, (float *)(s + G->at_mw)))
            return rc;
    }
    G->ready = i;
    *out = o;
    return AGPT_OK;
} AGPT_CATCH("trie_group_prepare")

extern "C" int agpt_b200_trie_group_upload(agpt_run_groups *G, int device, void *d_buffer, void *stream, agpt_plan **plan_out) {
    if (!G || G->ready < 0 || !G->plan || !d_buffer || !plan_out || device < 0) return agpt_set_error(AGPT_E_ARG, "trie_group_upload: nothing prepared");
    const agpt_run_group_info &o = G->info;
    agpt_plan *P = G->plan;
    uint8_t *d = (uint8_t *)d_buffer;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t err = cudaSetDevice(device);
    if (err == cudaSuccess) err = cudaMemcpyAsync(d, G->staging.get(), (size_t)G->staged, cudaMemcpyHostToDevice, st);
    if (err != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "trie_group_upload: %s", cudaGetErrorString(err));
    auto i32 = [&](int64_t at) { return (int32_t *)(d + at); };
    const int E = (int)o.n_loss_nodes;
    P->device = device; P->external = true;
    P->d_depth = i32(G->at_depth); P->d_sub_end = i32(G->at_subend); P->d_chain_ids = i32(G->at_cid); P->d_chain_end = i32(G->at_cend);
    P->d_chain_off = (int64_t *)(d + G->at_choff); P->d_tile_start = i32(G->at_ts);
    P->d_item_node = i32(G->at_items[0]); P->d_item_t0 = i32(G->at_items[1]); P->d_item_t1 = i32(G->at_items[2]); P->d_item_slot = i32(G->at_items[3]);
    P->d_multi_node = i32(G->at_multi); P->d_multi_count = i32(G->at_mcount); P->d_multi_first = (int64_t *)(d + G->at_mfirst);
    expand_runs_kernel<<<(E + 7) / 8, 256, 0, st>>>(i32(o.qoff), i32(G->at_fd), i32(G->at_ld), i32(G->at_send), i32(G->at_unit), i32(G->at_first),
                                                    (const float *)(d + G->at_mw), d + G->at_tr, E, o.seq_len, i32(o.pos), i32(o.q2n), i32(o.edge_first),
                                                    (int64_t *)(d + o.unit_of_row), o.mass_w < 0 ? nullptr : (float *)(d + o.mass_w),
                                                    o.trained < 0 ? nullptr : (float *)(d + o.trained), P->d_depth, P->d_sub_end);
    tile_chain_kernel<<<(unsigned)((P->n_tiles + 127) / 128), 128, 0, st>>>(i32(o.qoff), i32(G->at_prun), i32(G->at_send), P->d_chain_off, P->d_tile_start, E, P->n_tiles,
                                                                            P->d_chain_ids, P->d_chain_end);
    err = cudaGetLastError();
    if (err != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "trie_group_upload: %s", cudaGetErrorString(err));
    *plan_out = P;
    G->plan = nullptr; G->ready = -1;
    G->staging.reset();
    return AGPT_OK;
}
