// The linear solve's partition of a graph over CTAs and its use of their shared
// memory (pcg_solve in wrap_kernels.cu).
#pragma once

#ifdef __CUDACC__
#define NRICP_HOST_DEVICE __host__ __device__
#else
#define NRICP_HOST_DEVICE
#endif

namespace nricp_b200 {

// Rows are grouped into segments of kSegNodes nodes (24 rows: one pass of a
// warp; 4-node segments balance the warps better than 8-node ones, 0.90 s
// against 0.93 s per 64-wrap batch, and 16-node ones are slower).  A segment is
// the unit of reduction: one warp forms the segment's FP64 partial dot products
// in a fixed lane order, and every CTA sums the segments' partials in a fixed
// order.  A CTA owns a contiguous run of octets (eight nodes, two segments), so
// the number of CTAs only decides which CTA computes which segment, never the
// order of any sum: a wrap's solve is bit-identical for every cluster size, by
// the whole device, and with it alone and in any batch.
constexpr int kSegNodes = 4;
constexpr int kOctet = 8;  // nodes a warp multiplies at a time (24 of its lanes)

constexpr int kPcgThreads = 512;
constexpr int kPcgWarps = kPcgThreads / 32;
// Shared floats per owned node: X, R (2 x 6 FP64), P, S, W (18), its row's
// entry count and (one per octet each) the octet's first step and steps, padded.
constexpr int kPcgVectorFloats = 44;
constexpr int kPcgBlockFloats = 36;  // its damped diagonal block; and its inverse
// Dynamic shared memory of every solve launch: all there is.  A solve CTA holds
// its SM alone (512 threads of 128 registers), and what the vectors leave
// holds off-diagonal blocks.
constexpr int kPcgMaxSmemBytes = 225 * 1024;
constexpr int kPcgMaxSmemFloats = kPcgMaxSmemBytes / 4;
constexpr int kGatherSteps = 16;  // steps whose u a warp of a grid solve gathers at a time

NRICP_HOST_DEVICE inline int pcg_segments(int nodes) { return (nodes + kSegNodes - 1) / kSegNodes; }
NRICP_HOST_DEVICE inline int pcg_octets(int nodes) { return (nodes + kOctet - 1) / kOctet; }
// FP64 slots for the segments' three partials (two segments per octet)
NRICP_HOST_DEVICE inline int pcg_slot_doubles(int nodes) { return 6 * pcg_octets(nodes); }

// Owned-node capacity of one CTA when `ranks` CTAs share the solve.
NRICP_HOST_DEVICE inline int pcg_owned_capacity(int nodes, int ranks) {
    return (pcg_octets(nodes) + ranks - 1) / ranks * kOctet;
}

// Placement for one wrap within the launch's shared memory, in this order:
// the segment slots always, the all-node direction copy U if it fits (the
// matvec reads it ~20 times per row), the owned rows' vectors, the inverses of
// their diagonal blocks, if all of these fit those blocks themselves, and what
// is left for the last steps of every owned octet's off-diagonal blocks.
// Whatever does not fit lives in the wrap's global scratch, and the diagonal
// blocks are then read from the system; the arithmetic is the same.  (The
// instance without all arrays in shared memory never reads the blocks there.
// With their 36 to 54 KB left to off-diagonal steps an iteration takes, 3,000
// nodes on 8 CTAs, 26.4 -> 25.2 us; 3,100 30.3 -> 28.9; 4,200 on 16 25.6 -> 24.9.)
struct PcgPlacement {
    bool u_shared, vectors_shared, diagonal_shared, inverse_shared;
    int floats;  // shared floats used before the blocks
    NRICP_HOST_DEVICE bool all() const { return diagonal_shared; }
};
NRICP_HOST_DEVICE inline PcgPlacement pcg_place(int nodes, int ranks, int budget_floats) {
    PcgPlacement p;
    int used = pcg_slot_doubles(nodes) * 2;
    const int u = (nodes * 6 + 3) & ~3;
    const int cap = pcg_owned_capacity(nodes, ranks);
    auto take = [&](int floats) {
        const bool fits = used + floats <= budget_floats;
        if (fits) used += floats;
        return fits;
    };
    p.u_shared = take(u);
    p.vectors_shared = take(cap * kPcgVectorFloats);
    p.inverse_shared = take(cap * kPcgBlockFloats);
    p.diagonal_shared = p.u_shared && p.vectors_shared && p.inverse_shared && take(cap * kPcgBlockFloats);
    p.floats = used;
    return p;
}

// A whole-device solve's CTA holds every array of its rows in shared memory: u,
// the vectors, the diagonal blocks, their inverses, and the u its warps gather.
NRICP_HOST_DEVICE inline int pcg_grid_floats(int nodes, int ctas) {
    return pcg_owned_capacity(nodes, ctas) * (6 + kPcgVectorFloats + 2 * kPcgBlockFloats) +
           kPcgWarps * kGatherSteps * 64;
}
// 32,768 nodes fit 98 CTAs and more; a device with fewer SMs solves them by
// clusters.
NRICP_HOST_DEVICE inline bool pcg_grid_fits(int nodes, int ctas) {
    return pcg_grid_floats(nodes, ctas) <= kPcgMaxSmemFloats;
}

}  // namespace nricp_b200
