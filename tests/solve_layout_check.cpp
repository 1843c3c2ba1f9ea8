// The solve's use of shared memory (nricp_b200/csrc/solve_layout.hpp) over every
// graph size and number of CTAs: see tests/test_solve_layout.py.
#include <cstdio>
#include <initializer_list>

#include "../nricp_b200/csrc/solve_layout.hpp"

using namespace nricp_b200;

namespace {

int failures = 0;
void expect(bool ok, const char* what, int nodes, int ctas) {
    if (ok || failures > 20) return;
    ++failures;
    std::printf("%s: %d nodes, %d CTAs\n", what, nodes, ctas);
}

}  // namespace

int main() {
    constexpr int kNodes = 32768;  // the most a level may have
    for (int n = 1; n <= kNodes; ++n) {
        for (int ctas = 1; ctas <= 16; ctas *= 2) {
            const int cap = pcg_owned_capacity(n, ctas);
            expect(cap % 8 == 0 && (long)cap * ctas >= n, "every node is owned", n, ctas);
            const PcgPlacement p = pcg_place(n, ctas, kPcgMaxSmemFloats);
            expect(p.floats <= kPcgMaxSmemFloats, "a cluster's arrays fit", n, ctas);
            // only what the instance reads is taken: the damped diagonal blocks
            // are in shared memory with everything else or not at all
            const int slots = 12 * ((n + 7) / 8), u = (n * 6 + 3) / 4 * 4;
            const int read = slots + (p.u_shared ? u : 0) + (p.vectors_shared ? cap * 44 : 0) +
                             (p.inverse_shared ? cap * 36 : 0) + (p.all() ? cap * 36 : 0);
            expect(p.floats == read, "nothing is taken that is not read", n, ctas);
            expect(p.all() == (slots + u + cap * (44 + 72) <= kPcgMaxSmemFloats), "all arrays where they fit", n, ctas);
        }
        // the whole device: what the kernel carves, array by array
        for (int ctas : {16, 64, 97, 98, 132, 148, 160}) {
            const int cap = (n + 8 * ctas - 1) / (8 * ctas) * 8;
            const long u = 6L * cap, gathered = 16L * 16 * 64, x_r = 2 * 2 * 6L * cap, p_s_w = 3 * 6L * cap;
            const long degrees = cap + 2L * (cap / 8), blocks = 2 * 36L * cap;
            const bool fits = u + gathered + x_r + p_s_w + degrees + blocks <= kPcgMaxSmemFloats;
            if (!fits) expect(!pcg_grid_fits(n, ctas), "a grid that does not fit is declined", n, ctas);
        }
        expect(pcg_grid_fits(n, 148) && pcg_grid_fits(n, 98), "a grid that fits is taken", n, 148);
    }
    expect(!pcg_grid_fits(kNodes, 97), "97 SMs are too few for the largest graph", kNodes, 97);
    std::printf(failures ? "FAILED\n" : "ok\n");
    return failures ? 1 : 0;
}
