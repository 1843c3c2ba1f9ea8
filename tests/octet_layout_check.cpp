// The octet storage of the off-diagonal blocks (build_layout in
// nricp_b200/csrc/host.cpp), which the assembly writes and the solve reads: see
// tests/test_octet_layouts.py.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <initializer_list>
#include <random>
#include <set>
#include <vector>

#include "../nricp_b200/csrc/host.hpp"

using namespace nricp_b200;

extern "C" void nricp_default_level(NricpLevelSettings*) {}  // report_json only

namespace {

int failures = 0;
void expect(bool ok, const char* what, int N, int level) {
    if (ok || failures > 20) return;
    ++failures;
    std::printf("%s: %d nodes, level %d\n", what, N, level);
}

void check_level(const TemplateGraph& g, int level, int V) {
    const LevelLayout L = build_layout(g, level, V);
    const int N = L.node_count, B = static_cast<int>(L.offdiag_nodes.size() / 2), octets = (N + 7) / 8;
    // a node's entries: the blocks that touch it, in block order
    std::vector<std::vector<int>> entries(N);  // block * 2 + (1: its second node)
    for (int k = 0; k < B; ++k) {
        entries[L.offdiag_nodes[k * 2]].push_back(k * 2);
        entries[L.offdiag_nodes[k * 2 + 1]].push_back(k * 2 + 1);
    }
    bool steps = static_cast<int>(L.sell_begin.size()) == octets + 1 && L.sell_begin[0] == 0;
    for (int o = 0; o < octets && steps; ++o) {
        size_t most = 0;
        for (int n = o * 8; n < std::min(N, o * 8 + 8); ++n) {
            most = std::max(most, entries[n].size());
            steps &= L.row_begin[n + 1] - L.row_begin[n] == static_cast<int>(entries[n].size());
        }
        steps &= L.sell_begin[o + 1] - L.sell_begin[o] == static_cast<int>(most);
    }
    expect(steps, "an octet has as many steps as its longest row", N, level);
    if (!steps) return;
    expect(static_cast<int>(L.sell_nodes.size()) == L.sell_begin[octets] * 8 &&
               static_cast<int>(L.sell_slots.size()) == 2 * B, "sizes", N, level);
    std::set<int> used;
    bool places = true, nodes = true;
    for (int k = 0; k < B; ++k)
        for (int side = 0; side < 2; ++side) {
            const int node = L.offdiag_nodes[k * 2 + side], other = L.offdiag_nodes[k * 2 + 1 - side];
            const int place = L.sell_slots[k * 2 + side];
            places &= place >= 0 && place < static_cast<int>(L.sell_nodes.size()) && used.insert(place).second;
            if (!places) break;
            // in the node's octet and column, below the node's own degree
            const int t = place / 8 - L.sell_begin[node / 8];
            places &= place % 8 == node % 8 && t >= 0 && t < static_cast<int>(entries[node].size());
            nodes &= L.sell_nodes[place] == other;
        }
    expect(places, "every block has two places of its own, in its nodes' rows", N, level);
    expect(nodes, "a place names the block's other node", N, level);
    bool padding = true;  // a place without a block is read, not multiplied: a node of the graph
    for (size_t p = 0; p < L.sell_nodes.size(); ++p)
        if (!used.count(static_cast<int>(p))) padding &= L.sell_nodes[p] >= 0 && L.sell_nodes[p] < N;
    expect(padding, "padding names a node", N, level);
    // the device keeps one smoothness edge per block, as its first node sees it
    std::set<int> with_edge;
    bool edges = true;
    for (int e = 0; e < L.edge_count; ++e) {
        const int k = L.edge_block[e];
        edges &= k >= 0 && k < B && with_edge.insert(k).second && L.offdiag_nodes[k * 2] == L.edges[e * 2] &&
                 L.offdiag_nodes[k * 2 + 1] == L.edges[e * 2 + 1];
    }
    expect(edges, "a block has one edge at most, in its nodes' order", N, level);
}

}  // namespace

int main() {
    for (int nodes : {1, 2, 7, 8, 9, 15, 16, 17, 63, 65, 300})
        for (int k : {1, 2, 4, 8})
            for (int neighbours : {0, 3, 8}) {
                const int V = std::max(40, nodes * 5);
                std::mt19937_64 rng(static_cast<uint64_t>(nodes) * 131 + k * 7 + neighbours);
                std::normal_distribution<double> normal;
                std::vector<double> p(static_cast<size_t>(V) * 3);
                for (double& x : p) x = normal(rng);
                TemplateGraph g = build_template_graph(p.data(), V, 2, nodes, 2, k, neighbours);
                if (V >= 300) {  // a node in two slots, a zero weight
                    Binding& twice = g.levels.back().bindings[7];
                    if (twice.count >= 3) twice.nodes[2] = twice.nodes[0];
                    Binding& weightless = g.levels.back().bindings[8];
                    if (weightless.count >= 2) weightless.weights[1] = 0.0;
                }
                for (int l = 0; l < static_cast<int>(g.levels.size()); ++l) check_level(g, l, V);
            }
    std::printf(failures ? "FAILED\n" : "ok\n");
    return failures ? 1 : 0;
}
