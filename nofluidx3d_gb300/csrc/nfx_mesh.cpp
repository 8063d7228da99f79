// Host-side mesh plan: locality reordering, tiles and per-tetra reference quantities.
//
// The reference keeps the user's node and tetra order and recomputes the inverse reference
// edge matrix every step (tetra.cl:47-53). Here, once at set-up:
//  * nodes are sorted along a Morton (Z-order) curve of their reference positions, and tetrahedra
//    along the Morton curve of their centroids, so a run of consecutive tetrahedra touches a
//    compact set of nodes;
//  * tetrahedra are grouped into tiles of at most tile_tets (128, 256 or 512) elements and
//    min(tile_tets, 256) distinct nodes by greedy region growing: a tile starts at the first
//    unassigned tetra along the Morton curve and repeatedly takes the adjacent tetra that adds
//    the fewest new nodes, so tiles are compact and share few nodes (every node entry of a tile
//    costs a displacement gather and three accumulator atomics per step). Each tetra's corners
//    are stored as 8-bit indices into its tile's node list, plus the tile's incidence list
//    (corners grouped by node) for the fixed-order force sums. Local node numbers and the order of
//    the sums are chosen so that the warps' shared-memory reads meet few bank conflicts: on the
//    Kuhn spheres the law's corner reads cost 90 passes a tile instead of 126, the force sums' 99
//    instead of 173 and their list entries 38 instead of 61 (64, 75 and 30 without any conflict);
//  * Dm^-1 (inverse of the reference edge matrix [X1-X0, X2-X0, X3-X0]) and the signed
//    reference volume V0 = det(Dm)/6 (TetraCell.py:33-41) are computed in double and stored
//    as float;
//  * reference positions are split into float hi + lo parts.
// Corner order within a tetra is the user's, so node 0 of each tetra stays the base node of
// the reference's elastic kernel (tetra.cl:31-35).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <functional>
#include <numeric>
#include <thread>

#include "nfx_internal.h"

namespace nfx {

namespace {

inline uint64_t spread3(uint64_t x) {
    x &= 0x1fffff;  // 21 bits
    x = (x | (x << 32)) & 0x1f00000000ffffULL;
    x = (x | (x << 16)) & 0x1f0000ff0000ffULL;
    x = (x | (x << 8)) & 0x100f00f00f00f00fULL;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ULL;
    x = (x | (x << 2)) & 0x1249249249249249ULL;
    return x;
}

inline uint64_t morton3(uint64_t x, uint64_t y, uint64_t z) { return spread3(x) | (spread3(y) << 1) | (spread3(z) << 2); }

struct Quant {
    double lo[3];
    double inv_h;
    uint64_t q(double v, int d) const {
        double s = (v - lo[d]) * inv_h;
        if (!(s > 0)) s = 0;
        if (s > 2097151.0) s = 2097151.0;
        return (uint64_t)s;
    }
};

// Greedy region-growing tiles (see the file comment). seed_order: the tetrahedra in Morton
// order. Appends each tile's tetrahedra to tets and the tiles' end offsets to tile_end.
// Candidates are kept in five FIFO buckets by the number of nodes they would add (0..4); a
// bucket entry is stale when the tetra was assigned or its count dropped since it was pushed.
void grow_tiles(int64_t np, int64_t nt, const uint32_t* T, const std::vector<int64_t>& seed_order, int tile_tets,
                int nodes_max, std::vector<uint32_t>& tets, std::vector<int64_t>& tile_end) {
    std::vector<int64_t> off((size_t)np + 1, 0);  // node -> incident tetrahedra (CSR)
    for (int64_t i = 0; i < 4 * nt; i++) off[(size_t)T[i] + 1]++;
    for (int64_t i = 0; i < np; i++) off[i + 1] += off[i];
    std::vector<uint32_t> adj((size_t)(4 * nt));
    {
        std::vector<int64_t> fill(off.begin(), off.end() - 1);
        for (int64_t k = 0; k < 4; k++)
            for (int64_t t = 0; t < nt; t++) adj[fill[T[k * nt + t]]++] = (uint32_t)t;
    }
    std::vector<uint8_t> assigned((size_t)nt, 0), newc((size_t)nt, 0);
    std::vector<int64_t> node_stamp((size_t)np, -1), tet_stamp((size_t)nt, -1);
    std::vector<uint32_t> bucket[5];
    size_t head[5];
    tets.clear();
    tets.reserve((size_t)nt);
    tile_end.clear();
    int64_t seed = 0, tile = 0;
    for (;;) {
        while (seed < nt && assigned[seed_order[seed]]) seed++;
        if (seed == nt) break;
        for (int b = 0; b < 5; b++) {
            bucket[b].clear();
            head[b] = 0;
        }
        int nodes = 0, cnt = 0;
        auto new_nodes = [&](uint32_t t) {
            int c = 0;
            for (int k = 0; k < 4; k++) c += node_stamp[T[k * nt + t]] != tile;
            return c;
        };
        auto add = [&](uint32_t t) {
            assigned[t] = 1;
            tets.push_back(t);
            cnt++;
            for (int k = 0; k < 4; k++) {
                const uint32_t n = T[k * nt + t];
                if (node_stamp[n] == tile) continue;
                node_stamp[n] = tile;
                nodes++;
                for (int64_t a = off[n]; a < off[n + 1]; a++) {
                    const uint32_t t2 = adj[a];
                    if (assigned[t2]) continue;
                    if (tet_stamp[t2] != tile) {
                        tet_stamp[t2] = tile;
                        newc[t2] = (uint8_t)new_nodes(t2);
                    } else if (newc[t2] > 0) {
                        newc[t2]--;
                    }
                    bucket[newc[t2]].push_back(t2);
                }
            }
        };
        add((uint32_t)seed_order[seed]);
        while (cnt < tile_tets) {
            int64_t pick = -1;
            for (int b = 0; b < 5 && pick < 0; b++) {
                if (nodes + b > nodes_max) break;
                while (head[b] < bucket[b].size()) {
                    const uint32_t t = bucket[b][head[b]++];
                    if (!assigned[t] && tet_stamp[t] == tile && newc[t] == b) {
                        pick = t;
                        break;
                    }
                }
            }
            if (pick < 0) {  // nothing adjacent fits: the next unassigned tetra along the curve
                while (seed < nt && assigned[seed_order[seed]]) seed++;
                if (seed == nt) break;
                const uint32_t t = (uint32_t)seed_order[seed];
                if (nodes + new_nodes(t) > nodes_max) break;
                pick = t;
            }
            add((uint32_t)pick);
        }
        tile_end.push_back((int64_t)tets.size());
        tile++;
    }
}

// Shared-memory bank groups. A 16-byte read of a warp is served eight lanes (a quarter) at a time and
// costs one pass per distinct address that falls on the most used of the eight 16-byte bank groups.
constexpr int BANK_GROUPS = 8;

// Local numbers for a tile's nodes. rank lists them by falling incidence count; every run of eight in
// that order is a quarter of a warp in the force sums, and stays one (equal counts end together).
// Within a quarter the nodes are permuted so that the tetrahedra of a quarter (eight consecutive
// ones) find their k-th corners in different bank groups: loc[node] % 8 is the group. corner[4 j + k]:
// node of corner k of tetra j.
void number_nodes(int cnt, int nn, const uint16_t* corner, const std::vector<uint32_t>& rank, std::vector<uint16_t>& loc,
                  std::vector<uint16_t>& w) {
    // w[a * nn + b]: how often a and b are read by the same quarter at the same corner
    w.assign((size_t)nn * nn, 0);
    for (int j = 0; j < cnt; j += BANK_GROUPS)
        for (int k = 0; k < 4; k++) {
            const int n = std::min(BANK_GROUPS, cnt - j);
            for (int x = 0; x < n; x++)
                for (int y = 0; y < x; y++) {
                    const int a = corner[4 * (j + x) + k], c = corner[4 * (j + y) + k];
                    if (a == c) continue;
                    w[(size_t)a * nn + c]++;
                    w[(size_t)c * nn + a]++;
                }
        }
    uint16_t group[BANK_GROUPS][TILE_NODES_MAX / BANK_GROUPS];  // the nodes of each group so far
    int held[BANK_GROUPS] = {};
    int cost[BANK_GROUPS][BANK_GROUPS];  // [node of the quarter][group]
    for (int q = 0; q < nn; q += BANK_GROUPS) {
        const int n = std::min(BANK_GROUPS, nn - q);
        for (int x = 0; x < n; x++)
            for (int g = 0; g < n; g++) {
                cost[x][g] = 0;
                for (int o = 0; o < held[g]; o++) cost[x][g] += w[(size_t)rank[q + x] * nn + group[g][o]];
            }
        int at[BANK_GROUPS];  // group of each node: in order, then improved by swaps
        for (int x = 0; x < n; x++) at[x] = x;
        for (bool better = true; better;) {
            better = false;
            for (int x = 0; x < n; x++)
                for (int y = 0; y < x; y++)
                    if (cost[x][at[y]] + cost[y][at[x]] < cost[x][at[x]] + cost[y][at[y]]) {
                        std::swap(at[x], at[y]);
                        better = true;
                    }
        }
        for (int x = 0; x < n; x++) {
            loc[rank[q + x]] = (uint16_t)(q + at[x]);
            group[at[x]][held[at[x]]++] = (uint16_t)rank[q + x];
        }
    }
}

// Order in which the n <= 8 nodes of a quarter take their corner forces, one each per round: slots[begin[l]
// .. begin[l + 1]) are node l's corner slots (corner * T + tetra, bank group tetra % 8), put into that order.
// Each round matches nodes to different bank groups as far as their remaining corners allow
// (augmenting paths, the groups in most demand first); what is left over takes the least used.
void order_corners(uint16_t* slots, const uint32_t* begin, int n, std::vector<uint16_t>& sorted) {
    int left[BANK_GROUPS][BANK_GROUPS] = {}, next[BANK_GROUPS][BANK_GROUPS], demand[BANK_GROUPS] = {};
    uint32_t rounds = 0;
    sorted.resize(begin[n] - begin[0]);  // each node's slots by bank group; next: the first not yet taken
    for (int l = 0; l < n; l++) {
        rounds = std::max(rounds, begin[l + 1] - begin[l]);
        for (uint32_t i = begin[l]; i < begin[l + 1]; i++) left[l][slots[i] % BANK_GROUPS]++;
        int pos = (int)(begin[l] - begin[0]), fill[BANK_GROUPS];
        for (int g = 0; g < BANK_GROUPS; g++) {
            next[l][g] = fill[g] = pos;
            pos += left[l][g];
            demand[g] += left[l][g];
        }
        for (uint32_t i = begin[l]; i < begin[l + 1]; i++) sorted[fill[slots[i] % BANK_GROUPS]++] = slots[i];
    }
    unsigned has[BANK_GROUPS] = {};  // per group: the nodes that still have a corner in it, as bits
    for (int l = 0; l < n; l++)
        for (int g = 0; g < BANK_GROUPS; g++) has[g] |= (unsigned)(left[l][g] > 0) << l;
    int order[BANK_GROUPS];
    for (int g = 0; g < BANK_GROUPS; g++) order[g] = g;
    for (uint32_t r = 0; r < rounds; r++) {
        int take[BANK_GROUPS], load[BANK_GROUPS] = {};
        std::fill(take, take + BANK_GROUPS, -1);
        for (int i = 1; i < BANK_GROUPS; i++)  // nearly sorted from the round before
            for (int k = i; k > 0 && demand[order[k]] > demand[order[k - 1]]; k--) std::swap(order[k], order[k - 1]);
        unsigned taken = 0, open_nodes = 0;
        for (int g = 0; g < BANK_GROUPS; g++) open_nodes |= has[g];
        for (int oi = 0; oi < BANK_GROUPS && demand[order[oi]] > 0 && taken != open_nodes; oi++) {
            const int g0 = order[oi];
            const unsigned open = has[g0] & ~taken;
            if (open) {  // a node without a group yet
                const int l = __builtin_ctz(open);
                take[l] = g0;
                taken |= 1u << l;
                continue;
            }
            // match the group to a node all the same, moving other groups' nodes along
            unsigned seen = 0;
            auto place = [&](auto&& self, int g) -> bool {
                for (unsigned open; (open = has[g] & ~seen) != 0;) {
                    const int l = __builtin_ctz(open);
                    seen |= 1u << l;
                    if (take[l] < 0 || self(self, take[l])) {
                        take[l] = g;
                        taken |= 1u << l;
                        return true;
                    }
                }
                return false;
            };
            place(place, g0);
        }
        for (int l = 0; l < n; l++)
            if (take[l] >= 0) load[take[l]]++;
        for (int l = 0; l < n; l++) {
            if (r >= begin[l + 1] - begin[l]) continue;
            if (take[l] < 0) {
                int best = -1;
                for (int g = 0; g < BANK_GROUPS; g++)
                    if (left[l][g] && (best < 0 || load[g] < load[best])) best = g;
                take[l] = best;
                load[best]++;
            }
            const int g = take[l];
            slots[begin[l] + r] = sorted[next[l][g]++];
            if (--left[l][g] == 0) has[g] &= ~(1u << l);
            demand[g]--;
        }
    }
}

}  // namespace

bool in_parallel(int64_t n, int threads, const std::function<void(int64_t, int64_t)>& work) {
    const int64_t parts = std::max<int64_t>(1, std::min<int64_t>(threads, n / 4));
    std::atomic<bool> failed{false};
    auto part = [&](int64_t k) {
        try {
            work(n * k / parts, n * (k + 1) / parts);
        } catch (...) {
            failed = true;
        }
    };
    std::vector<std::thread> pool;
    int64_t k = 1;
    try {
        for (; k < parts; k++) pool.emplace_back(part, k);
    } catch (...) {  // no more threads: the parts without one run here
    }
    part(0);
    for (; k < parts; k++) part(k);
    for (auto& t : pool) t.join();
    return !failed;
}

bool build_mesh_plan(int64_t np, int64_t nt, const double* P, const uint32_t* T, int tile_tets, MeshPlan& plan,
                     std::string& err, int threads) {
    if (tile_tets != 64 && tile_tets != 128 && tile_tets != 256 && tile_tets != 512) {
        err = "tile size must be 64, 128, 256 or 512";
        return false;
    }
    if (np <= 0 || nt <= 0) {
        err = "mesh needs at least one node and one tetra";
        return false;
    }
    if (np > (int64_t)0x7fffffff || nt > (int64_t)0x7fffffff) {
        err = "mesh too large (more than 2^31-1 nodes or tetrahedra)";
        return false;
    }
    for (int64_t t = 0; t < 4 * nt; t++) {
        if ((int64_t)T[t] >= np) {
            err = "tetra corner index out of range";
            return false;
        }
    }
    for (int64_t i = 0; i < 3 * np; i++) {
        if (!std::isfinite(P[i])) {
            err = "non-finite node position";
            return false;
        }
    }
    plan = MeshPlan();
    plan.np = np;
    plan.nt = nt;
    plan.tile_tets = tile_tets;
    const int64_t nodes_max = std::min<int64_t>(TILE_NODES_MAX, tile_tets);

    // quantisation: cell size ~ mean node spacing
    Quant Q;
    double hi[3];
    for (int d = 0; d < 3; d++) {
        Q.lo[d] = P[d * np];
        hi[d] = P[d * np];
        for (int64_t i = 1; i < np; i++) {
            Q.lo[d] = std::min(Q.lo[d], P[d * np + i]);
            hi[d] = std::max(hi[d], P[d * np + i]);
        }
    }
    double vol = 1.0;
    for (int d = 0; d < 3; d++) vol *= std::max(hi[d] - Q.lo[d], 1e-12);
    double h = std::cbrt(vol / (double)np);
    if (!(h > 0)) h = 1.0;
    Q.inv_h = 1.0 / h;

    // nodes
    std::vector<uint64_t> nkey(np);
    for (int64_t i = 0; i < np; i++)
        nkey[i] = morton3(Q.q(P[i], 0), Q.q(P[np + i], 1), Q.q(P[2 * np + i], 2));
    plan.node_user.resize(np);
    std::iota(plan.node_user.begin(), plan.node_user.end(), 0);
    std::stable_sort(plan.node_user.begin(), plan.node_user.end(),
                     [&](int64_t a, int64_t b) { return nkey[a] < nkey[b]; });
    plan.node_int.resize(np);
    for (int64_t i = 0; i < np; i++) plan.node_int[plan.node_user[i]] = i;

    // tetrahedra, by centroid
    std::vector<uint64_t> tkey(nt);
    for (int64_t t = 0; t < nt; t++) {
        double c[3] = {0, 0, 0};
        for (int k = 0; k < 4; k++) {
            const int64_t n = T[k * nt + t];
            for (int d = 0; d < 3; d++) c[d] += 0.25 * P[d * np + n];
        }
        tkey[t] = morton3(Q.q(c[0], 0), Q.q(c[1], 1), Q.q(c[2], 2));
    }
    std::vector<int64_t> order(nt);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int64_t a, int64_t b) { return tkey[a] < tkey[b]; });

    // Tiles at a fixed stride: tile b owns tetra slots [b*T, b*T + T) and node-list entries
    // [b*NMAX, b*NMAX + NMAX); unused slots and entries are zero padding (a padding tetra has
    // Dm^-1 = 0 and V0 = 0 and produces no force; a padding node entry has count 0). Kernels can
    // then address a tile's data without first loading its offsets.
    const int64_t T_ = tile_tets, NM_ = nodes_max;
    std::vector<uint32_t> tile_tets_list;
    std::vector<int64_t> tile_end;
    grow_tiles(np, nt, T, order, tile_tets, (int)nodes_max, tile_tets_list, tile_end);
    order.assign(tile_tets_list.begin(), tile_tets_list.end());  // tetrahedra in tile order
    const int64_t nti = (int64_t)tile_end.size();
    std::vector<int64_t> slot_user((size_t)(nti * T_), -1);  // tetra slot -> user tetra (-1: padding)
    plan.lconn.assign(4 * (size_t)(nti * T_), 0);
    plan.tile_nodes.assign(2 * (size_t)(nti * NM_), 0u);
    plan.tile_meta.assign((size_t)nti, 0u);
    std::vector<std::vector<uint16_t>> inc_of_tile((size_t)nti);
    // Tiles do not depend on one another: build_tiles makes those of [b0, b1).
    auto build_tiles = [&](int64_t b0, int64_t b1) {
        std::vector<uint32_t> ids;
        ids.reserve(4 * (size_t)tile_tets);
        // the tile's working arrays, kept from tile to tile: with allocations of their own for each, threads
        // planning small meshes side by side waited for the allocator (eight meshes of 14k tetras 10 ms)
        std::vector<uint16_t> corner, weights, loc_of, slots, sorted;
        std::vector<uint32_t> cnt_by_id, by_count, node_at, begin, fill, first;
        for (int64_t b = b0; b < b1; b++) {
            const int64_t t0 = b > 0 ? tile_end[b - 1] : 0;
            const int64_t cnt = tile_end[b] - t0;
            ids.clear();
            for (int64_t j = 0; j < cnt; j++) {
                const int64_t ut = order[t0 + j];
                for (int k = 0; k < 4; k++) ids.push_back((uint32_t)plan.node_int[T[k * nt + ut]]);
            }
            std::sort(ids.begin(), ids.end());
            ids.erase(std::unique(ids.begin(), ids.end()), ids.end());
            const size_t nn = ids.size();
            const size_t s0 = (size_t)(b * T_);
            // Local node order: by incidence count, largest first (ties by node index). The thread of
            // local node q sums its corners in a loop, and a warp runs as many iterations as its
            // largest count, so grouping similar counts into the same warp saves iterations. Eight at
            // a time they are permuted against bank conflicts (number_nodes).
            corner.resize(4 * (size_t)cnt);
            cnt_by_id.assign(nn, 0);
            for (int64_t j = 0; j < cnt; j++)
                for (int k = 0; k < 4; k++) {
                    const uint32_t g = (uint32_t)plan.node_int[T[k * nt + order[t0 + j]]];
                    const uint16_t a = (uint16_t)(std::lower_bound(ids.begin(), ids.end(), g) - ids.begin());
                    corner[4 * j + k] = a;
                    cnt_by_id[a]++;
                }
            by_count.resize(nn);
            std::iota(by_count.begin(), by_count.end(), 0u);
            std::sort(by_count.begin(), by_count.end(), [&](uint32_t a, uint32_t c) {
                return cnt_by_id[a] != cnt_by_id[c] ? cnt_by_id[a] > cnt_by_id[c] : a < c;
            });
            loc_of.resize(nn);
            number_nodes((int)cnt, (int)nn, corner.data(), by_count, loc_of, weights);
            node_at.resize(nn);  // local number -> position in ids
            for (size_t a = 0; a < nn; a++) node_at[loc_of[a]] = (uint32_t)a;
            slots.resize(4 * (size_t)cnt);  // corner slots by local node, in (tet, corner) order
            begin.assign(nn + 1, 0);
            for (size_t a = 0; a < nn; a++) begin[loc_of[a] + 1] = cnt_by_id[a];
            for (size_t q = 0; q < nn; q++) begin[q + 1] += begin[q];
            fill.assign(begin.begin(), begin.end() - 1);
            for (int64_t j = 0; j < cnt; j++) {
                slot_user[s0 + j] = order[t0 + j];
                for (int k = 0; k < 4; k++) {
                    const uint16_t loc = loc_of[corner[4 * j + k]];
                    plan.lconn[4 * (s0 + j) + k] = (uint8_t)loc;
                    slots[fill[loc]++] = (uint16_t)(k * T_ + j);
                }
            }
            // Incidence list of the tile: the local nodes of a quarter side by side, eight entries per
            // round, a node's entries one round apart; a node with fewer than its quarter's most has
            // unused entries.
            first.resize(nn);
            std::vector<uint16_t> inc;
            inc.reserve(6 * (size_t)cnt);
            for (size_t w = 0; w < nn; w += 4 * BANK_GROUPS) {
                const int nq = (int)std::min<size_t>(4, (nn - w + BANK_GROUPS - 1) / BANK_GROUPS);
                int rounds[4] = {};
                for (int u = 0; u < nq; u++) {
                    const size_t q = w + u * BANK_GROUPS;
                    const int n = (int)std::min<size_t>(BANK_GROUPS, nn - q);
                    for (int l = 0; l < n; l++) rounds[u] = std::max(rounds[u], (int)(begin[q + l + 1] - begin[q + l]));
                    order_corners(slots.data(), begin.data() + q, n, sorted);
                }
                // the quarters of a warp read their lists in step: lay them out so that as few as possible
                // start in the same bank group
                int perm[4] = {0, 1, 2, 3}, best[4] = {0, 1, 2, 3}, best_cost = -1;
                do {
                    int cost = 0, at[4], pos = (int)(inc.size() / BANK_GROUPS);
                    for (int u = 0; u < nq; u++) {
                        at[perm[u]] = pos;
                        pos += rounds[perm[u]];
                    }
                    for (int u = 0; u < nq; u++)
                        for (int v = 0; v < u; v++)
                            if ((at[u] - at[v]) % BANK_GROUPS == 0) cost += std::min(rounds[u], rounds[v]);
                    if (best_cost < 0 || cost < best_cost) {
                        best_cost = cost;
                        std::copy(perm, perm + 4, best);
                    }
                } while (best_cost > 0 && std::next_permutation(perm, perm + nq));
                for (int v = 0; v < nq; v++) {
                    const int u = best[v];
                    const size_t base = inc.size();
                    inc.resize(base + (size_t)rounds[u] * BANK_GROUPS, 0);
                    for (int l = 0; l < BANK_GROUPS && w + u * BANK_GROUPS + l < nn; l++) {
                        const size_t q = w + u * BANK_GROUPS + l;
                        first[q] = (uint32_t)(base + l);
                        for (uint32_t i = begin[q]; i < begin[q + 1]; i++)
                            inc[base + (i - begin[q]) * BANK_GROUPS + l] = (uint16_t)(16 * slots[i]);
                    }
                }
            }
            inc_of_tile[b] = std::move(inc);
            for (size_t q = 0; q < nn; q++) {
                plan.tile_nodes[2 * (b * NM_ + q)] = ids[node_at[q]];
                plan.tile_nodes[2 * (b * NM_ + q) + 1] = (first[q] << 16) | (begin[q + 1] - begin[q]);
            }
            plan.tile_meta[b] = (uint32_t)cnt | ((uint32_t)nn << 16);
        }
    };
    if (!in_parallel(nti, threads, build_tiles)) {
        err = "out of memory";
        return false;
    }
    const int64_t b = nti;
    plan.ntiles = b;
    plan.nslots = b * T_;
    {
        // the tiles' incidence lists at one stride, that of the longest
        size_t longest = BANK_GROUPS;
        for (const auto& v : inc_of_tile) longest = std::max(longest, v.size());
        plan.inc_stride = (int)longest;
        plan.tile_inc.assign((size_t)b * longest, 0);
        for (int64_t q = 0; q < b; q++) std::copy(inc_of_tile[q].begin(), inc_of_tile[q].end(), &plan.tile_inc[q * longest]);
    }
    {
        // the most tiles any node appears in sets the per-tile bound of the fixed-point sums
        std::vector<int32_t> tiles_of((size_t)np, 0);
        for (int64_t q = 0; q < b; q++) {
            const int64_t nn = plan.tile_meta[q] >> 16;
            for (int64_t e = 0; e < nn; e++) tiles_of[plan.tile_nodes[2 * (q * NM_ + e)]]++;
        }
        plan.max_tiles_per_node = std::max(1, *std::max_element(tiles_of.begin(), tiles_of.end()));
        plan.all_nodes_used = *std::min_element(tiles_of.begin(), tiles_of.end()) > 0;
        plan.fix_max = force_fix_bound(plan.max_tiles_per_node);
    }
    plan.tet_user = std::move(slot_user);
    plan.tile_tet_begin.resize(b + 1);
    plan.tile_node_begin.resize(b + 1);
    for (int64_t q = 0; q <= b; q++) {
        plan.tile_tet_begin[q] = (int32_t)(q * T_);
        plan.tile_node_begin[q] = (int32_t)(q * NM_);
    }

    // per-tetra Dm^-1 and V0 (slot order; padding slots stay zero), and the lumped nodal masses of
    // density 1 that VelocityVerlet2 uses: a quarter of every tetra's V0 to each of its corners
    // (SimulationLegacy.py:911-924)
    plan.dmi.assign(12 * (size_t)plan.nslots, 0.0f);
    std::vector<double> mass((size_t)np, 0.0);
    for (int64_t it = 0; it < plan.nslots; it++) {
        const int64_t ut = plan.tet_user[it];
        if (ut < 0) continue;
        const int64_t n0 = T[ut];
        double M[9];  // columns X_k - X_0
        for (int k = 0; k < 3; k++) {
            const int64_t nk = T[(k + 1) * nt + ut];
            for (int d = 0; d < 3; d++) M[3 * d + k] = P[d * np + nk] - P[d * np + n0];
        }
        const double A[9] = {M[4] * M[8] - M[5] * M[7], M[2] * M[7] - M[1] * M[8], M[1] * M[5] - M[2] * M[4],
                             M[5] * M[6] - M[3] * M[8], M[0] * M[8] - M[2] * M[6], M[2] * M[3] - M[0] * M[5],
                             M[3] * M[7] - M[4] * M[6], M[1] * M[6] - M[0] * M[7], M[0] * M[4] - M[1] * M[3]};
        const double det = M[0] * A[0] + M[1] * A[3] + M[2] * A[6];
        if (det == 0.0 || !std::isfinite(det)) {
            err = "degenerate tetra (zero reference volume) at index " + std::to_string(ut);
            return false;
        }
        float* o = &plan.dmi[12 * it];
        for (int k = 0; k < 9; k++) o[k] = (float)(A[k] / det);
        o[9] = (float)(det / 6.0);
        for (int k = 0; k < 4; k++) mass[T[k * nt + ut]] += 0.25 * (det / 6.0);
    }

    // reference positions, hi/lo, internal order
    plan.Xh.assign(4 * (size_t)np, 0.0f);
    plan.Xl.assign(4 * (size_t)np, 0.0f);
    for (int64_t i = 0; i < np; i++) {
        const int64_t u = plan.node_user[i];
        for (int d = 0; d < 3; d++) {
            const double x = P[d * np + u];
            const float h32 = (float)x;
            plan.Xh[4 * i + d] = h32;
            plan.Xl[4 * i + d] = (float)(x - (double)h32);
        }
        // the unused fourth lane carries the inverse lumped mass (density 1); 0 for a node no
        // tetra touches
        const double m = mass[u];
        plan.Xh[4 * i + 3] = m != 0.0 ? (float)(1.0 / m) : 0.0f;
    }

    // bounding box of every node block's reference positions, rounded outwards to float
    const int64_t nb = (np + NODE_BLOCK - 1) / NODE_BLOCK;
    plan.block_box.assign(8 * (size_t)nb, 0.0f);
    for (int64_t q = 0; q < nb; q++) {
        double lo[3] = {HUGE_VAL, HUGE_VAL, HUGE_VAL}, hi[3] = {-HUGE_VAL, -HUGE_VAL, -HUGE_VAL};
        for (int64_t i = q * NODE_BLOCK; i < std::min<int64_t>(np, (q + 1) * NODE_BLOCK); i++) {
            const int64_t u = plan.node_user[i];
            for (int d = 0; d < 3; d++) {
                lo[d] = std::min(lo[d], P[d * np + u]);
                hi[d] = std::max(hi[d], P[d * np + u]);
            }
        }
        for (int d = 0; d < 3; d++) {
            float l = (float)lo[d], h = (float)hi[d];
            if ((double)l > lo[d]) l = std::nextafter(l, -HUGE_VALF);
            if ((double)h < hi[d]) h = std::nextafter(h, HUGE_VALF);
            plan.block_box[8 * q + d] = l;
            plan.block_box[8 * q + 4 + d] = h;
        }
    }
    return true;
}

}  // namespace nfx
