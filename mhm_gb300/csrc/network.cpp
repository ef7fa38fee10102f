// network.cpp -- routing blocks and routing order (host).
#include "network.h"

#include <algorithm>
#include <numeric>

namespace mhm {

bool build_route_network(int32_t L, int32_t n_outlets, const int32_t *net_perm, const int32_t *from_n,
                         const int32_t *to_n, int32_t cap, RouteNetwork &o, std::string &err)
{
    o = RouteNetwork{};
    if (L < 1 || n_outlets < 1 || n_outlets > L) {
        err = "network: need n_nodes >= 1 and 1 <= n_outlets <= n_nodes";
        return false;
    }
    cap = std::max(kRouteUps, std::min(cap, kRouteBlock));
    const int32_t nl = L - n_outlets;
    o.n_nodes = L;
    o.n_links = nl;
    std::vector<int32_t> rank(nl, -1), down(L, -1);
    for (int32_t r = 0; r < nl; ++r) {
        const int32_t i = net_perm[r] - 1;
        if (i < 0 || i >= nl || rank[i] != -1) {
            err = "network: netPerm is not a permutation of the links";
            return false;
        }
        rank[i] = r;
    }
    for (int32_t i = 0; i < nl; ++i) {
        const int32_t f = from_n[i] - 1, t = to_n[i] - 1;
        if (f < 0 || f >= L || t < 0 || t >= L || f == t) {
            err = "network: fromN/toN out of range or self loop";
            return false;
        }
        if (down[f] != -1) {
            err = "network: a node is the source of two links";
            return false;
        }
        down[f] = t;
    }
    // upstream nodes of each node in rank order of their links, and the nodes
    // in rank order of their own link (sinks last): upstream before downstream
    std::vector<std::vector<int32_t>> ups(L);
    std::vector<int32_t> topo, topo_of(L, -1), above(L, 0); // above: links of the longest river into a node
    for (int32_t r = 0; r < nl; ++r) {
        const int32_t i = net_perm[r] - 1, f = from_n[i] - 1;
        ups[to_n[i] - 1].push_back(f);
        above[to_n[i] - 1] = std::max(above[to_n[i] - 1], above[f] + 1);
        topo_of[f] = (int32_t)topo.size();
        topo.push_back(f);
    }
    o.depth = *std::max_element(above.begin(), above.end());
    for (int32_t v = 0; v < L; ++v)
        if (down[v] < 0) {
            topo_of[v] = (int32_t)topo.size();
            topo.push_back(v);
        }
    for (int32_t v = 0; v < L; ++v)
        for (int32_t u : ups[v])
            if (topo_of[u] >= topo_of[v]) {
                err = "network: netPerm is not a topological order of the links";
                return false;
            }
    const int32_t special_outlet = (nl > 0) ? to_n[net_perm[nl - 1] - 1] - 1 : -1;

    // trunk: nodes whose subtree holds more than `cap` nodes or a hub (a node
    // with more than kRouteUps upstream links); what is left are subtrees of
    // at most `cap` nodes
    std::vector<int32_t> size(L, 1);
    std::vector<uint8_t> hub(L, 0), trunk(L, 0);
    for (int32_t v : topo) {
        hub[v] = (int32_t)ups[v].size() > kRouteUps;
        for (int32_t u : ups[v]) {
            size[v] += size[u];
            trunk[v] |= trunk[u];
        }
        trunk[v] |= hub[v] || size[v] > cap;
    }
    // pieces: piece[v], a piece's nodes upstream first; `level` 0 for whole
    // subtrees, for a stretch of the trunk one more than any piece draining into it
    struct Piece {
        std::vector<int32_t> nodes;
        int32_t n_ext = 0, level = 0;
    };
    std::vector<Piece> pieces;
    std::vector<int32_t> piece(L, -1);
    for (size_t k = topo.size(); k-- > 0;) { // downstream first: a subtree's root opens its piece
        const int32_t v = topo[k];
        if (trunk[v]) continue;
        if (down[v] >= 0 && !trunk[down[v]]) {
            piece[v] = piece[down[v]];
        } else {
            piece[v] = (int32_t)pieces.size();
            pieces.emplace_back();
        }
    }
    for (int32_t v : topo)
        if (!trunk[v]) pieces[piece[v]].nodes.push_back(v);
    // trunk: every node continues the stretch of its longest upstream trunk
    // branch until the stretch is full; all other links are cut
    std::vector<int32_t> height(L, 0);
    for (int32_t v : topo) {
        if (!trunk[v]) continue;
        int32_t main = -1;
        for (int32_t u : ups[v])
            if (trunk[u] && (main < 0 || height[u] > height[main])) main = u;
        height[v] = main < 0 ? 1 : height[main] + 1;
        const int32_t n_cut = (int32_t)ups[v].size() - (main >= 0 ? 1 : 0);
        int32_t p = main >= 0 ? piece[main] : -1;
        if (hub[v] || p < 0 || (int32_t)pieces[p].nodes.size() >= cap || pieces[p].n_ext + n_cut > cap) {
            p = (int32_t)pieces.size();
            pieces.emplace_back();
            if (!hub[v]) pieces[p].n_ext = (int32_t)ups[v].size();
        } else {
            pieces[p].n_ext += n_cut;
        }
        piece[v] = p;
        pieces[p].nodes.push_back(v);
    }
    std::vector<int32_t> order(pieces.size());
    std::iota(order.begin(), order.end(), 0);
    auto last = [&](int32_t p) { return topo_of[pieces[p].nodes.back()]; };
    std::sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return last(a) < last(b); });
    for (int32_t p : order)
        for (int32_t v : pieces[p].nodes)
            for (int32_t u : ups[v])
                if (piece[u] != p) pieces[p].level = std::max(pieces[p].level, pieces[piece[u]].level + 1);
    // blocks: pieces of one level, filled in the order of the place they drain into
    auto drains_to = [&](int32_t p) {
        const int32_t d = down[pieces[p].nodes.back()];
        return d < 0 ? L : topo_of[d];
    };
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
        if (pieces[a].level != pieces[b].level) return pieces[a].level < pieces[b].level;
        return drains_to(a) < drains_to(b);
    });
    std::vector<std::vector<int32_t>> blocks;
    int32_t fill = 0, fill_ext = 0, blk_level = -1;
    for (int32_t p : order) {
        const int32_t n = (int32_t)pieces[p].nodes.size(), e = pieces[p].n_ext;
        if (pieces[p].level != blk_level || fill + n > cap || fill_ext + e > cap) {
            blocks.emplace_back();
            fill = fill_ext = 0;
            blk_level = pieces[p].level;
        }
        fill += n;
        fill_ext += e;
        blocks.back().push_back(p);
    }
    // lags: the distance to the piece's last node, counted back from the piece's
    // longest, so that a link inside a piece is always one tick
    std::vector<int32_t> lag(L, 0), pos_in(L, 0);
    for (const Piece &pc : pieces) {
        int32_t deepest = 0;
        for (size_t k = pc.nodes.size(); k-- > 0;) {
            const int32_t v = pc.nodes[k];
            lag[v] = k + 1 == pc.nodes.size() ? 0 : lag[down[v]] + 1;
            deepest = std::max(deepest, lag[v]);
        }
        for (int32_t v : pc.nodes) lag[v] = deepest - lag[v];
    }
    o.n_blocks = (int32_t)blocks.size();
    o.pos_of_node.assign(L, 0);
    o.node_of_pos.reserve(L);
    o.pos_export.assign(L, -1);
    o.blk_ptr.push_back(0);
    std::vector<int32_t> export_of(L, -1);
    for (const auto &blk : blocks) {
        std::vector<int32_t> nodes;
        for (int32_t p : blk) nodes.insert(nodes.end(), pieces[p].nodes.begin(), pieces[p].nodes.end());
        // by lag: neighbouring threads work on the same step
        std::stable_sort(nodes.begin(), nodes.end(), [&](int32_t a, int32_t b) { return lag[a] < lag[b]; });
        for (size_t k = 0; k < nodes.size(); ++k) {
            const int32_t v = nodes[k], pos = (int32_t)o.node_of_pos.size();
            pos_in[v] = (int32_t)k;
            o.pos_of_node[v] = pos;
            o.node_of_pos.push_back(v);
            if (down[v] >= 0 && piece[down[v]] != piece[v]) o.pos_export[pos] = export_of[v] = o.n_exports++;
        }
        o.blk_ptr.push_back((int32_t)o.node_of_pos.size());
        o.blk_lag.push_back(lag[nodes.back()]);
    }
    o.ext_ptr.push_back(0);
    o.pos_ups.assign((size_t)L * kRouteUps, -1);
    o.pos_flags.assign(L, 0);
    o.pos_lag.resize(L);
    o.hub_ptr.push_back(0);
    for (int32_t b = 0; b < o.n_blocks; ++b) {
        for (int32_t pos = o.blk_ptr[b]; pos < o.blk_ptr[b + 1]; ++pos) {
            const int32_t v = o.node_of_pos[pos];
            o.pos_lag[pos] = lag[v];
            int16_t *up = &o.pos_ups[(size_t)pos * kRouteUps];
            if (hub[v]) {
                const int32_t h = (int32_t)o.hub_ptr.size() - 1;
                up[0] = -2;
                up[1] = (int16_t)(h & 0x7fff);
                up[2] = (int16_t)(h >> 15);
                for (int32_t u : ups[v]) o.hub_ups.push_back(export_of[u]);
                o.hub_ptr.push_back((int32_t)o.hub_ups.size());
            } else {
                int j = 0;
                for (int32_t u : ups[v]) {
                    if (piece[u] == piece[v]) {
                        up[j++] = (int16_t)pos_in[u];
                    } else {
                        up[j++] = (int16_t)(kRouteBlock + (int32_t)o.ext_export.size() - o.ext_ptr[b]);
                        o.ext_export.push_back(export_of[u]);
                        o.ext_lag.push_back(lag[v]);
                    }
                }
            }
            int8_t fl = 0;
            if (down[v] >= 0) fl |= 3; // a link adds its own qOUT (mo_mrm_routing.f90:445)
            if (v == special_outlet) fl |= 2; // mo_mrm_routing.f90:466-467
            o.pos_flags[pos] = fl;
        }
        o.ext_ptr.push_back((int32_t)o.ext_export.size());
    }
    o.link_pos.assign(nl, 0);
    for (int32_t i = 0; i < nl; ++i) o.link_pos[i] = o.pos_of_node[from_n[i] - 1];
    return true;
}

bool routing_order(int32_t L, int32_t n_outlets, const int32_t *from_n, const int32_t *to_n, int32_t *net_perm,
                   int32_t *r_order, std::string &err)
{
    const int32_t nl = L - n_outlets;
    for (int32_t i = 0; i < L; ++i) net_perm[i] = r_order[i] = -9999;
    if (L <= 1) return true;
    if (nl < 0) {
        err = "routing_order: n_outlets > n_nodes";
        return false;
    }
    // pending[i]: number of unranked links draining into fromN(i) (self excluded,
    // as in the reference's jj == ii test).
    std::vector<int32_t> pending(nl, 0);
    std::vector<std::vector<int32_t>> into(L); // links whose toN is node v
    for (int32_t j = 0; j < nl; ++j) {
        const int32_t t = to_n[j] - 1;
        if (t < 0 || t >= L) {
            err = "routing_order: toN out of range";
            return false;
        }
        into[t].push_back(j);
    }
    std::vector<std::vector<int32_t>> feeds(nl); // feeds[j]: links i with fromN(i) == toN(j)
    for (int32_t i = 0; i < nl; ++i) {
        const int32_t f = from_n[i] - 1;
        if (f < 0 || f >= L) {
            err = "routing_order: fromN out of range";
            return false;
        }
        for (int32_t j : into[f])
            if (j != i) {
                pending[i]++;
                feeds[j].push_back(i);
            }
    }
    std::vector<int32_t> rank(nl, 0);
    int32_t kk = 0;
    std::vector<int32_t> unranked;
    for (int32_t i = 0; i < nl; ++i) {
        if (pending[i] == 0) {
            rank[i] = ++kk; // headwaters in link order
        } else {
            unranked.push_back(i);
        }
    }
    for (int32_t i = 0; i < nl; ++i)
        if (rank[i] > 0)
            for (int32_t d : feeds[i]) pending[d]--;
    // sweeps in link order; a link ranked earlier in the same sweep counts
    while (!unranked.empty()) {
        std::vector<int32_t> rest;
        bool progress = false;
        for (int32_t i : unranked) {
            if (pending[i] == 0) {
                rank[i] = ++kk;
                progress = true;
                for (int32_t d : feeds[i]) pending[d]--;
            } else {
                rest.push_back(i);
            }
        }
        if (!progress) {
            err = "routing_order: network has a cycle";
            return false;
        }
        unranked.swap(rest);
    }
    for (int32_t i = 0; i < nl; ++i) {
        r_order[i] = rank[i];
        net_perm[rank[i] - 1] = i + 1;
    }
    return true;
}

bool network_topology(int32_t nrows, int32_t ncols, const int32_t *id2d, int32_t n_cells, const int32_t *cell_row,
                      const int32_t *cell_col, const int32_t *fdir, int32_t *from_n, int32_t *to_n, int32_t *n_links,
                      std::string &err)
{
    for (int32_t k = 0; k < n_cells; ++k) from_n[k] = to_n[k] = -9999; // nodata_i4
    int32_t nl = 0;
    for (int32_t k = 0; k < n_cells; ++k) {
        // row / column offsets of the ESRI D8 codes, as moveDownOneCell
        // steps them (src/mRM/mo_mrm_net_startup.f90:1768-1801); any other
        // code leaves the cell where it is
        int32_t di = 0, dj = 0;
        switch (fdir[k]) {
        case 1: dj = 1; break;
        case 2: di = 1; dj = 1; break;
        case 4: di = 1; break;
        case 8: di = 1; dj = -1; break;
        case 16: dj = -1; break;
        case 32: di = -1; dj = -1; break;
        case 64: di = -1; break;
        case 128: di = -1; dj = 1; break;
        default: break;
        }
        const int32_t i = cell_row[k] + di, j = cell_col[k] + dj; // 1-based
        if (i < 1 || i > nrows || j < 1 || j > ncols) {
            err = "network_topology: flow direction of cell " + std::to_string(k + 1) + " leaves the grid";
            return false;
        }
        const int32_t to = id2d[(size_t)(j - 1) * nrows + (i - 1)];
        if (to == k + 1) continue; // points at itself: an outlet
        if (to < 1 || to > n_cells) {
            err = "network_topology: flow direction of cell " + std::to_string(k + 1) + " leaves the mask";
            return false;
        }
        from_n[nl] = k + 1;
        to_n[nl] = to;
        ++nl;
    }
    *n_links = nl;
    return true;
}

} // namespace mhm
