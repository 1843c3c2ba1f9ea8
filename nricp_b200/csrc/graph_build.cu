// The template graphs of many wraps at once on the device: farthest-point
// seeds, the nearest-node bindings of every vertex and the k-NN node edges of
// every level (src/core/graph.cpp:41-76, src/core/sampling.cpp:17-143).
//
// Every value is the host build's to the bit: the same FP64 operations in the
// same order, each rounded on its own (no contraction), and the same tie
// rules -- the first maximum for the seeds, (squared distance, index) for the
// bindings, (distance, index) for the edges.  Only the scan orders differ,
// and none of the rules depends on them.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>

#include "async.cuh"
#include "graph_build.hpp"
#include "per_device.hpp"
#include "resources.hpp"
#include "session.hpp"
#include "staging.hpp"

namespace nricp_b200 {

namespace cg = cooperative_groups;

namespace {

constexpr int kBindThreads = 128;
constexpr int kTile = 512;            // nodes staged in shared memory per pass
constexpr int kMaxEdgeNeighbours = 16;

__device__ inline double sq_rn(const double* a, const double* b) {  // sampling.cpp:17-19
    const double x = __dsub_rn(a[0], b[0]), y = __dsub_rn(a[1], b[1]), z = __dsub_rn(a[2], b[2]);
    return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

// Farthest-point seeds (sampling.cpp:47-88): seeds[0] = 0, then repeatedly the
// point farthest from all seeds so far, the first of equals.  A chain of
// thousands of dependent steps, so a step's latency is all that counts: one
// thread-block cluster per template (templates[blockIdx.y]), the points split in
// contiguous chunks over its CTAs and at most kPer to a thread, coordinates in
// shared memory, distances to the nearest seed in registers.  Per step: every
// thread updates its points; a distance's bits order like the distance (it is
// never negative), so a warp finds its farthest point with three integer
// reductions instead of shuffling candidates; the CTA's first warp does the
// same over the warps and sends the CTA's candidate to every CTA with
// asynchronous stores that complete on the receiver's mbarrier (two sets of
// slots in turn); and every warp takes the same winner from the slots.
// The tie rule makes the winner the same for any split.  30,000 points, 2,000
// seeds: 6.0 ms with shuffled candidates and a cluster barrier, now 2.0 ms;
// 100,130 points, 10,000 seeds: 291 ms in one block, now 18 ms.
constexpr int kFpsThreads = 1024;
constexpr int kFpsMaxPer = 8;                                         // points per thread at most
constexpr int kFpsClusterPoints = 16 * kFpsThreads * kFpsMaxPer;      // 131,072

struct alignas(16) FpsCandidate {
    unsigned long long key;  // the distance's bits
    long index;
    double x, y, z, pad;
};

// The warp's largest (key, then smallest index), in every lane.
__device__ __forceinline__ void warp_farthest(unsigned long long& key, int& index) {
    const uint32_t high = (uint32_t)(key >> 32), low = (uint32_t)key;
    const uint32_t top = __reduce_max_sync(0xffffffffu, high);
    const uint32_t next = __reduce_max_sync(0xffffffffu, high == top ? low : 0u);
    const bool mine = high == top && low == next;
    index = __reduce_min_sync(0xffffffffu, mine ? index : INT_MAX);
    key = ((unsigned long long)top << 32) | next;
}

template <int kPer>
__global__ void __launch_bounds__(kFpsThreads, 1) k_fps(const double* __restrict__ points,
                                                     const long* __restrict__ point_offset,
                                                     const int* __restrict__ point_count,
                                                     const int* __restrict__ seed_count,
                                                     const long* __restrict__ seed_offset,
                                                     const int* __restrict__ templates, int* __restrict__ seeds_all,
                                                     int* __restrict__ failed, int tries) {
    cg::cluster_group cluster = cg::this_cluster();
    const int t = templates[blockIdx.y];
    const int n = point_count[t];
    const int count = min(seed_count[t], n);
    if (n <= 0 || count <= 0) return;  // the same for the whole cluster
    const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
    const int chunk = (n + ranks - 1) / ranks;  // <= kFpsThreads * kPer
    const int c0 = rank * chunk, here = max(0, min(n, c0 + chunk) - c0);
    const double* p = points + point_offset[t] * 3;
    int* seeds = seeds_all + seed_offset[t];
    extern __shared__ double coordinates[];  // x, y, z of the chunk
    double* const sx = coordinates;
    double* const sy = sx + chunk;
    double* const sz = sy + chunk;
    __shared__ FpsCandidate slots[2][16];
    __shared__ unsigned long long warp_key[kFpsThreads / 32];
    __shared__ int warp_index[kFpsThreads / 32];
    __shared__ alignas(8) unsigned long long arrived[2];  // mbarriers
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < here * 3; i += kFpsThreads) {
        const double x = p[(long)c0 * 3 + i];
        (i % 3 == 0 ? sx : (i % 3 == 1 ? sy : sz))[i / 3] = x;
    }
    if (threadIdx.x == 0) {
        mbar_init(&arrived[0], 1);
        mbar_init(&arrived[1], 1);
    }
    cluster.sync();
    double near[kPer];
    const int peer = min(lane, ranks - 1);
    const uint32_t peer_slots = peer_address(slots, peer), peer_arrived = peer_address(arrived, peer);
    if (rank == 0 && threadIdx.x == 0) seeds[0] = 0;
    double c[3] = {p[0], p[1], p[2]};
    bool timed_out = false;
    for (int s = 0;; ++s) {
        unsigned long long key = 0;
        int index = INT_MAX;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int i = threadIdx.x + k * kFpsThreads;
            if (i >= here) continue;
            const double q[3] = {sx[i], sy[i], sz[i]};
            const double d = sq_rn(q, c);
            const double m = s == 0 ? d : (near[k] < d ? near[k] : d);
            near[k] = m;
            const unsigned long long bits = (unsigned long long)__double_as_longlong(m);
            if (bits > key || index == INT_MAX) {  // indices grow with k: the first of equals stays
                key = bits;
                index = c0 + i;
            }
        }
        if (s + 1 >= count) break;
        const int set = s & 1;
        if (threadIdx.x == 0 && ranks > 1) mbar_arrive_expect(&arrived[set], ranks * (int)sizeof(FpsCandidate));
        warp_farthest(key, index);
        if (lane == 0) {
            warp_key[warp] = key;
            warp_index[warp] = index;
        }
        if (__syncthreads_or(timed_out)) break;
        if (warp == 0) {
            key = warp_key[lane];  // 32 warps
            index = warp_index[lane];
            warp_farthest(key, index);
            const int at = index == INT_MAX ? 0 : index - c0;  // an empty chunk's candidate loses to any other
            if (ranks > 1) {
                if (lane < ranks) {
                    const uint32_t dst = peer_slots + (uint32_t)(set * 16 + rank) * (uint32_t)sizeof(FpsCandidate);
                    const uint32_t bar = peer_arrived + set * 8;
                    store_to_peer(dst, __longlong_as_double((long long)key), __longlong_as_double((long long)index), bar);
                    store_to_peer(dst + 16, sx[at], sy[at], bar);
                    store_to_peer(dst + 32, sz[at], 0.0, bar);
                }
            } else if (lane == 0) {
                slots[set][0] = FpsCandidate{key, index, sx[at], sy[at], sz[at], 0.0};
            }
        }
        int win = 0;
        if (ranks > 1) {
            if (!mbar_wait(&arrived[set], (s >> 1) & 1, tries)) timed_out = true;
            key = lane < ranks ? slots[set][lane].key : 0;
            index = lane < ranks ? (int)slots[set][lane].index : INT_MAX;
            const int own = index;
            warp_farthest(key, index);
            win = __ffs(__ballot_sync(0xffffffffu, lane < ranks && own == index)) - 1;
        } else {
            __syncthreads();
        }
        const FpsCandidate& w = slots[set][max(win, 0)];
        if (rank == 0 && threadIdx.x == 0 && !timed_out) seeds[s + 1] = (int)w.index;
        c[0] = w.x;
        c[1] = w.y;
        c[2] = w.z;
    }
    // a wait that ran out, the last step's too; the peers' run out in turn
    if (__syncthreads_or(timed_out)) {
        if (threadIdx.x == 0) atomicOr(failed, 1);
        for (int i = 0; i < 256; ++i) __nanosleep(10000);  // the stores in flight (2.6 ms)
    }
    // no CTA leaves while another may still write into its shared memory
    cluster.sync();
}

// The same for a template of more points, by one block: distances in global
// memory.
__global__ void __launch_bounds__(kFpsThreads, 1) k_fps_block(const double* __restrict__ points,
                                                           const long* __restrict__ point_offset,
                                                           const int* __restrict__ point_count,
                                                           const int* __restrict__ seed_count,
                                                           const long* __restrict__ seed_offset,
                                                           const int* __restrict__ templates,
                                                           double* __restrict__ nearest_all,
                                                           int* __restrict__ seeds_all) {
    const int t = templates[blockIdx.x];
    const int n = point_count[t];
    const int count = min(seed_count[t], n);
    if (n <= 0 || count <= 0) return;
    const double* p = points + point_offset[t] * 3;
    double* nearest = nearest_all + point_offset[t];
    int* seeds = seeds_all + seed_offset[t];
    __shared__ unsigned long long warp_key[kFpsThreads / 32];
    __shared__ int warp_index[kFpsThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) seeds[0] = 0;
    int chosen = 0;
    for (int s = 0; s + 1 < count; ++s) {
        const double c[3] = {p[(long)chosen * 3], p[(long)chosen * 3 + 1], p[(long)chosen * 3 + 2]};
        unsigned long long key = 0;
        int index = INT_MAX;
        for (int i = threadIdx.x; i < n; i += kFpsThreads) {
            const double d = sq_rn(p + (long)i * 3, c);
            const double m = s == 0 ? d : (nearest[i] < d ? nearest[i] : d);
            nearest[i] = m;
            const unsigned long long bits = (unsigned long long)__double_as_longlong(m);
            if (bits > key || index == INT_MAX) {
                key = bits;
                index = i;
            }
        }
        warp_farthest(key, index);
        if (lane == 0) {
            warp_key[warp] = key;
            warp_index[warp] = index;
        }
        __syncthreads();
        key = warp_key[lane];
        index = warp_index[lane];
        warp_farthest(key, index);
        chosen = index;
        if (threadIdx.x == 0) seeds[s + 1] = chosen;
        __syncthreads();
    }
}

// (sq, idx) kept sorted ascending, at most `capacity` entries, entries offered
// in increasing index (sampling.cpp:23-42).
__device__ inline void keep(double* sq, int* idx, int& held, int capacity, double value, int entry) {
    if (held == capacity && !(value < sq[capacity - 1] || (value == sq[capacity - 1] && entry < idx[capacity - 1])))
        return;
    int at = held < capacity ? held++ : capacity - 1;
    while (at > 0 && (sq[at - 1] > value || (sq[at - 1] == value && idx[at - 1] > entry))) {
        sq[at] = sq[at - 1];
        idx[at] = idx[at - 1];
        --at;
    }
    sq[at] = value;
    idx[at] = entry;
}

// The `wanted` smallest (value, entry) of a group of G lanes' sorted lists, in
// every lane's (sq, idx) places 0 .. wanted - 1.  Values and entries of
// different lanes differ in the entry, so each round has one winner.
template <int G, int kMost>
__device__ inline void merge_lists(double* sq, int* idx, int held, int wanted) {
    double out_sq[kMost];
    int out_idx[kMost];
    int head = 0;
    for (int k = 0; k < wanted; ++k) {
        const double mine = head < held ? sq[head] : 1e300;
        const int my_entry = head < held ? idx[head] : INT_MAX;
        double v = mine;
        int e = my_entry;
        for (int o = G / 2; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oe = __shfl_xor_sync(0xffffffffu, e, o);
            if (ov < v || (ov == v && oe < e)) {
                v = ov;
                e = oe;
            }
        }
        out_sq[k] = v;
        out_idx[k] = e;
        if (e == my_entry && head < held) ++head;
    }
    for (int k = 0; k < wanted; ++k) {
        sq[k] = out_sq[k];
        idx[k] = out_idx[k];
    }
}

// A lane's K nearest so far in registers, ascending, equal values in the order
// they came (increasing entries).
template <int K>
struct Nearest {
    double sq[K];
    int idx[K];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            sq[k] = 1e300;
            idx[k] = INT_MAX;
        }
    }
    __device__ __forceinline__ void offer(double value, int entry) {
        if (!(value < sq[K - 1])) return;
#pragma unroll
        for (int k = K - 1; k >= 0; --k) {
            if (k > 0 && value < sq[k - 1]) {
                sq[k] = sq[k - 1];
                idx[k] = idx[k - 1];
            } else if (value < sq[k]) {
                sq[k] = value;
                idx[k] = entry;
            }
        }
    }
    __device__ __forceinline__ void drop_first() {
#pragma unroll
        for (int k = 0; k + 1 < K; ++k) {
            sq[k] = sq[k + 1];
            idx[k] = idx[k + 1];
        }
        sq[K - 1] = 1e300;
        idx[K - 1] = INT_MAX;
    }
};

// A group of kBindLanes lanes per (template, vertex) for one level: its K
// nearest nodes and weights (1 - d / d_max)^2, normalised (sampling.cpp:
// 90-143).  The nearest under (squared distance, index) are a strict total
// order, so each lane scans every kBindLanes-th node and the lists merge to the
// scan's own answer.
constexpr int kBindLanes = 8;
template <int K>
__device__ __forceinline__ void bind_vertices_of(const double* p, int n, int nc, const int* seeds, long out_at,
                                                 int* bind_nodes, double* bind_weights, double (*tile)[kTile]) {
    constexpr int kVertices = kBindThreads / kBindLanes;
    const int v = blockIdx.x * kVertices + threadIdx.x / kBindLanes, part = threadIdx.x % kBindLanes;
    Nearest<K> list;
    list.clear();
    double q[3] = {0.0, 0.0, 0.0};
    if (v < n) { q[0] = p[(long)v * 3]; q[1] = p[(long)v * 3 + 1]; q[2] = p[(long)v * 3 + 2]; }
    for (int base = 0; base < nc; base += kTile) {
        const int m = min(kTile, nc - base);
        __syncthreads();
        for (int j = threadIdx.x; j < m; j += kBindThreads)
            for (int k = 0; k < 3; ++k) tile[k][j] = p[(long)seeds[base + j] * 3 + k];
        __syncthreads();
        if (v < n)
            for (int j = part; j < m; j += kBindLanes) {
                const double node[3] = {tile[0][j], tile[1][j], tile[2][j]};
                list.offer(sq_rn(q, node), base + j);
            }
    }
    // the group's K nearest: K rounds, the lane that holds the winner drops it
    double sq[K];
    int idx[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double value = list.sq[0];
        int entry = list.idx[0];
        for (int o = kBindLanes / 2; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, value, o);
            const int oe = __shfl_xor_sync(0xffffffffu, entry, o);
            if (ov < value || (ov == value && oe < entry)) {
                value = ov;
                entry = oe;
            }
        }
        if (entry == list.idx[0]) list.drop_first();
        sq[k] = value;
        idx[k] = entry;
    }
    if (v >= n || part != 0) return;
    const double dmax = __dsqrt_rn(sq[K - 1]);
    double w[K];
    double total = 0.0;
#pragma unroll
    for (int s = 0; s < K; ++s) {
        const double distance = __dsqrt_rn(sq[s]);
        const double ratio = dmax > 0.0 ? __ddiv_rn(distance, dmax) : 0.0;
        const double falloff = __dsub_rn(1.0, ratio);
        w[s] = __dmul_rn(falloff, falloff);
        total = __dadd_rn(total, w[s]);
    }
    const long at = out_at + (long)v * NRICP_MAX_SLOTS;
#pragma unroll
    for (int s = 0; s < NRICP_MAX_SLOTS; ++s) {
        bind_nodes[at + s] = s < K ? idx[s < K ? s : 0] : -1;
        bind_weights[at + s] =
            s < K ? (total > 0.0 ? __ddiv_rn(w[s < K ? s : 0], total) : __ddiv_rn(1.0, (double)K)) : 0.0;
    }
}

__global__ void __launch_bounds__(kBindThreads) k_bind(const double* __restrict__ points,
                                                       const long* __restrict__ point_offset,
                                                       const int* __restrict__ point_count,
                                                       const int* __restrict__ seeds_all,
                                                       const long* __restrict__ seed_offset,
                                                       const int* __restrict__ level_nodes,
                                                       const int* __restrict__ support_of,
                                                       const long* __restrict__ bind_offset,
                                                       int* __restrict__ bind_nodes,
                                                       double* __restrict__ bind_weights) {
    const int t = blockIdx.y;
    const int n = point_count[t], nc = level_nodes[t];
    if (nc <= 0 || (long)blockIdx.x * (kBindThreads / kBindLanes) >= n) return;
    const double* p = points + point_offset[t] * 3;
    const int* seeds = seeds_all + seed_offset[t];
    __shared__ double tile[3][kTile];
    static_assert(NRICP_MAX_SLOTS == 8, "a case per support");
#define NRICP_BIND(K) \
    case K: bind_vertices_of<K>(p, n, nc, seeds, bind_offset[t], bind_nodes, bind_weights, tile); break;
    switch (support_of[t]) {  // 1 to 8, the same for a template
        NRICP_BIND(1) NRICP_BIND(2) NRICP_BIND(3) NRICP_BIND(4) NRICP_BIND(5) NRICP_BIND(6) NRICP_BIND(7)
        NRICP_BIND(8)
    }
#undef NRICP_BIND
}

// A warp per (template, node) for one level: the `taken` nearest other nodes
// by (distance, index) (graph.cpp:11-39), each lane scanning every 32nd.  A
// square well above the square of a lane's last kept distance cannot be kept,
// and is not rooted.
__global__ void __launch_bounds__(kBindThreads) k_neighbours(const double* __restrict__ points,
                                                             const long* __restrict__ point_offset,
                                                             const int* __restrict__ seeds_all,
                                                             const long* __restrict__ seed_offset,
                                                             const int* __restrict__ level_nodes,
                                                             const int* __restrict__ taken_of,
                                                             const long* __restrict__ edge_offset,
                                                             int* __restrict__ neighbours) {
    constexpr int kNodes = kBindThreads / 32;
    const int t = blockIdx.y;
    const int nc = level_nodes[t];
    if ((long)blockIdx.x * kNodes >= nc) return;
    const int i = blockIdx.x * kNodes + threadIdx.x / 32, lane = threadIdx.x % 32;
    const double* p = points + point_offset[t] * 3;
    const int* seeds = seeds_all + seed_offset[t];
    const int taken = taken_of[t];
    __shared__ double tile[3][kTile];
    double dist[kMaxEdgeNeighbours];
    int idx[kMaxEdgeNeighbours];
    int held = 0;
    double reach = 1e300;  // a square above this is not kept
    double q[3] = {0.0, 0.0, 0.0};
    if (i < nc) {
        const long s = seeds[i];
        q[0] = p[s * 3]; q[1] = p[s * 3 + 1]; q[2] = p[s * 3 + 2];
    }
    for (int base = 0; base < nc; base += kTile) {
        const int m = min(kTile, nc - base);
        __syncthreads();
        for (int j = threadIdx.x; j < m; j += kBindThreads)
            for (int k = 0; k < 3; ++k) tile[k][j] = p[(long)seeds[base + j] * 3 + k];
        __syncthreads();
        if (i < nc && taken > 0)
            for (int j = lane; j < m; j += 32) {
                const int o = base + j;
                if (o == i) continue;
                const double node[3] = {tile[0][j], tile[1][j], tile[2][j]};
                const double square = sq_rn(q, node);
                if (square > reach) continue;
                keep(dist, idx, held, taken, __dsqrt_rn(square), o);
                if (held == taken && dist[taken - 1] > 1e-150) reach = dist[taken - 1] * dist[taken - 1] * (1.0 + 1e-12);
            }
    }
    merge_lists<32, kMaxEdgeNeighbours>(dist, idx, held, taken);
    if (i < nc && lane < taken) neighbours[edge_offset[t] + (long)i * taken + lane] = idx[lane];
}

int blocks(long n, int threads) { return static_cast<int>((n + threads - 1) / threads); }

// Small host arrays that go up in one copy: each at a 256-byte offset.
class Packed {
public:
    template <typename T>
    size_t add(const std::vector<T>& v) {
        const size_t at = bytes_.size();
        bytes_.resize((at + sizeof(T) * std::max<size_t>(1, v.size()) + 255) & ~size_t(255));
        if (!v.empty()) std::memcpy(bytes_.data() + at, v.data(), sizeof(T) * v.size());
        return at;
    }
    const std::vector<char>& bytes() const { return bytes_; }

private:
    std::vector<char> bytes_;
};

}  // namespace

bool device_graph_supported(int edge_neighbours) { return edge_neighbours <= kMaxEdgeNeighbours; }

std::vector<TemplateGraph> device_template_graphs(const std::vector<GraphRequest>& requests,
                                                  cudaStream_t stream, int wait_tries) {
    const int W = static_cast<int>(requests.size());
    std::vector<TemplateGraph> out(W);
    if (W == 0) return out;
    // host: normalisation (mesh.cpp:174-187) and the sizes of every level
    std::vector<long> point_offset(W), seed_offset(W);
    std::vector<int> point_count(W), seed_count(W);
    std::vector<std::vector<int>> level_sizes(W);
    long total_points = 0, total_seeds = 0;
    int max_levels = 0, max_points = 0;
    for (int t = 0; t < W; ++t) {
        const GraphRequest& r = requests[t];
        point_offset[t] = total_points;
        point_count[t] = r.count;
        total_points += r.count;
        const int levels = std::max(1, r.levels);
        int most = 0;
        for (int l = 0; l < levels; ++l) {
            level_sizes[t].push_back(level_node_count(l, r.nodes_initial, r.growth, r.count));
            most = std::max(most, level_sizes[t].back());
        }
        most = std::min(most, r.count);
        seed_offset[t] = total_seeds;
        seed_count[t] = most;
        total_seeds += most;
        max_levels = std::max(max_levels, levels);
        max_points = std::max(max_points, r.count);
    }
    // every level's sizes, on the host
    struct LevelPlan {
        std::vector<int> nodes, support, taken;
        std::vector<long> eoff;
        long edge_total = 0;
        int max_nodes = 0;
    };
    std::vector<LevelPlan> plan(max_levels);
    long all_edges = 0;
    std::vector<long> edge_base(max_levels + 1, 0);
    for (int l = 0; l < max_levels; ++l) {
        LevelPlan& p = plan[l];
        p.nodes.assign(W, 0);
        p.support.assign(W, 1);
        p.taken.assign(W, 0);
        p.eoff.assign(W, 0);
        for (int t = 0; t < W; ++t) {
            const GraphRequest& r = requests[t];
            if (l >= static_cast<int>(level_sizes[t].size())) continue;
            p.nodes[t] = std::min(level_sizes[t][l], seed_count[t]);
            p.support[t] = std::max(1, std::min({r.max_nodes, p.nodes[t], NRICP_MAX_SLOTS}));
            p.taken[t] = p.nodes[t] > 1 && r.edge_neighbours > 0 ? std::min(r.edge_neighbours, p.nodes[t] - 1) : 0;
            p.eoff[t] = p.edge_total;
            p.edge_total += static_cast<long>(p.nodes[t]) * p.taken[t];
            p.max_nodes = std::max(p.max_nodes, p.nodes[t]);
        }
        edge_base[l + 1] = edge_base[l] + std::max<long>(1, p.edge_total);
        all_edges = edge_base[l + 1];
    }

    // Every template normalised on its own host thread, into page-locked
    // memory, where the downloads land too: the points and the small arrays,
    // the seeds, then per level the bindings' nodes and weights, then every
    // level's neighbour lists.
    const long bind_entries = std::max<long>(1, total_points * NRICP_MAX_SLOTS);
    auto rounded = [](size_t bytes) { return (bytes + 255) & ~size_t(255); };
    const size_t point_bytes = rounded(sizeof(double) * 3 * std::max<long>(1, total_points));
    const size_t seed_bytes = rounded(sizeof(int) * std::max<long>(1, total_seeds));
    const size_t level_bytes = (sizeof(int32_t) + sizeof(double)) * bind_entries;
    StagingLease lease(point_bytes + seed_bytes + level_bytes * max_levels + sizeof(int) * all_edges);
    double* points = reinterpret_cast<double*>(lease.data());
    char* const down = lease.data() + point_bytes;
    int* seeds = reinterpret_cast<int*>(down);
    auto host_nodes = [&](int l) { return reinterpret_cast<int32_t*>(down + seed_bytes + level_bytes * l); };
    auto host_weights = [&](int l) {
        return reinterpret_cast<double*>(down + seed_bytes + level_bytes * l + sizeof(int32_t) * bind_entries);
    };
    int* host_neigh = reinterpret_cast<int*>(down + seed_bytes + level_bytes * max_levels);
#pragma omp parallel for schedule(dynamic, 1) if (W > 1)
    for (int t = 0; t < W; ++t) {
        const GraphRequest& r = requests[t];
        TemplateGraph& g = out[t];
        compute_normalization(r.points, r.count, g.center, &g.scale);
        normalized_into(r.points, r.count, g.center, g.scale, points + point_offset[t] * 3);
    }

    // seeds: a cluster of 1-16 CTAs per template, at most two points per
    // thread while every template's CTAs fit on the device at once, else four
    // (a CTA takes its SM); past 16 CTAs up to eight; one block beyond 131,072
    // points.  One launch per cluster size and points per thread; the launches
    // touch different templates, so each runs on a stream of its own.
    int device = 0, sms = 148;
    check(cudaGetDevice(&device), "device");
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "device");
    auto cluster_log2 = [](int n, int per) {
        int g = 0;
        while (g < 4 && (1 << g) * kFpsThreads * per < n) ++g;
        return g;
    };
    long ctas = 0;
    for (int t = 0; t < W; ++t) ctas += 1 << cluster_log2(point_count[t], 2);
    const int target = ctas <= sms ? 2 : 4;
    constexpr int kClasses = 5 * 4;  // cluster 1 .. 16 by 1, 2, 4, 8 points per thread
    std::vector<std::vector<int>> by_class(kClasses);
    std::vector<int> single, chunk(kClasses, 0);
    for (int t = 0; t < W; ++t) {
        if (point_count[t] > kFpsClusterPoints) {
            single.push_back(t);
            continue;
        }
        const int g = cluster_log2(point_count[t], target);
        const int here = (point_count[t] + (1 << g) - 1) >> g;
        int per = 0;
        while ((1 << per) * kFpsThreads < here) ++per;
        by_class[g * 4 + per].push_back(t);
        chunk[g * 4 + per] = std::max(chunk[g * 4 + per], here);
    }
    // the small arrays and the points go up in two copies
    Packed packed;
    const size_t o_point_offset = packed.add(point_offset), o_point_count = packed.add(point_count);
    const size_t o_seed_count = packed.add(seed_count), o_seed_offset = packed.add(seed_offset);
    std::vector<long> bind_offset(W);
    for (int t = 0; t < W; ++t) bind_offset[t] = point_offset[t] * NRICP_MAX_SLOTS;
    const size_t o_bind_offset = packed.add(bind_offset), o_single = packed.add(single);
    std::vector<size_t> o_class(kClasses), o_nodes(max_levels), o_support(max_levels), o_taken(max_levels),
        o_eoff(max_levels);
    for (int k = 0; k < kClasses; ++k) o_class[k] = packed.add(by_class[k]);
    for (int l = 0; l < max_levels; ++l) {
        o_nodes[l] = packed.add(plan[l].nodes);
        o_support[l] = packed.add(plan[l].support);
        o_taken[l] = packed.add(plan[l].taken);
        o_eoff[l] = packed.add(plan[l].eoff);
    }
    size_t device_bytes = 0;
    auto piece = [&](size_t bytes) {
        const size_t at = device_bytes;
        device_bytes += rounded(bytes);
        return at;
    };
    const size_t o_packed = piece(packed.bytes().size()), o_points = piece(point_bytes), o_seeds = piece(seed_bytes);
    const size_t o_failed = piece(sizeof(int));
    const size_t o_nearest = piece(single.empty() ? 0 : sizeof(double) * total_points);
    const size_t o_bind_nodes = piece(sizeof(int32_t) * bind_entries * max_levels);
    const size_t o_bind_weights = piece(sizeof(double) * bind_entries * max_levels);
    const size_t o_neigh = piece(sizeof(int) * all_edges);
    PoolBuffer memory(device_bytes, stream, "cudaMallocFromPoolAsync(graph build)");
    const char* meta = memory.data() + o_packed;
    auto ints = [&](size_t at) { return reinterpret_cast<const int*>(meta + at); };
    auto longs = [&](size_t at) { return reinterpret_cast<const long*>(meta + at); };
    double* d_points = reinterpret_cast<double*>(memory.data() + o_points);
    int* d_seeds = reinterpret_cast<int*>(memory.data() + o_seeds);
    int* d_failed = reinterpret_cast<int*>(memory.data() + o_failed);
    double* d_nearest = reinterpret_cast<double*>(memory.data() + o_nearest);
    int32_t* d_bind_nodes = reinterpret_cast<int32_t*>(memory.data() + o_bind_nodes);
    double* d_bind_weights = reinterpret_cast<double*>(memory.data() + o_bind_weights);
    int* d_neigh = reinterpret_cast<int*>(memory.data() + o_neigh);
    int failed = 0;
    check(cudaMemcpyAsync(memory.data() + o_packed, packed.bytes().data(), packed.bytes().size(),
                          cudaMemcpyHostToDevice, stream), "upload");
    check(cudaMemcpyAsync(d_points, points, sizeof(double) * 3 * total_points, cudaMemcpyHostToDevice, stream),
          "upload");
    {
        using FpsKernel = decltype(&k_fps<1>);
        static const FpsKernel kernels[4] = {k_fps<1>, k_fps<2>, k_fps<4>, k_fps<8>};
        static PerDevice<bool>& enabled = *new PerDevice<bool>;
        enabled.of(device, [] {
            for (int k = 0; k < 4; ++k) {
                check(cudaFuncSetAttribute(kernels[k], cudaFuncAttributeNonPortableClusterSizeAllowed, 1),
                      "farthest-point seeds' attributes");
                check(cudaFuncSetAttribute(kernels[k], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           24 * kFpsThreads * (1 << k)), "farthest-point seeds' attributes");
            }
            return true;
        });
        check(cudaMemsetAsync(d_failed, 0, sizeof(int), stream), "farthest-point seeds");
        // where a wait runs out the rest of the seeds stay the first point:
        // the kernels that follow read points by them before the host knows
        check(cudaMemsetAsync(d_seeds, 0, seed_bytes, stream), "farthest-point seeds");
        cudaEvent_t fork = nullptr;
        check(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming), "event");
        check(cudaEventRecord(fork, stream), "event");
        std::vector<StreamLease> lanes;
        auto beside = [&](auto&& launch) {  // on a stream of its own, joined afterwards
            lanes.push_back(StreamLease::take());
            const cudaStream_t lane = lanes.back();
            cudaEvent_t join;
            check(cudaEventCreateWithFlags(&join, cudaEventDisableTiming), "event");
            check(cudaStreamWaitEvent(lane, fork, 0), "wait");
            launch(lane);
            check(cudaEventRecord(join, lane), "event");
            check(cudaStreamWaitEvent(stream, join, 0), "wait");
            cudaEventDestroy(join);  // released once its work is done
        };
        for (int k = 0; k < kClasses; ++k) {
            if (by_class[k].empty()) continue;
            beside([&](cudaStream_t lane) {
                cudaLaunchConfig_t config = {};
                config.gridDim = dim3(1 << (k / 4), static_cast<unsigned>(by_class[k].size()));
                config.blockDim = dim3(kFpsThreads);
                config.dynamicSmemBytes = static_cast<size_t>(24) * chunk[k];
                config.stream = lane;
                cudaLaunchAttribute attribute[1];
                attribute[0].id = cudaLaunchAttributeClusterDimension;
                attribute[0].val.clusterDim.x = 1 << (k / 4);
                attribute[0].val.clusterDim.y = 1;
                attribute[0].val.clusterDim.z = 1;
                config.attrs = attribute;
                config.numAttrs = 1;
                check(cudaLaunchKernelEx(&config, kernels[k % 4], (const double*)d_points,
                                         longs(o_point_offset), ints(o_point_count), ints(o_seed_count),
                                         longs(o_seed_offset), ints(o_class[k]), d_seeds, d_failed, wait_tries),
                      "farthest-point seeds");
            });
        }
        if (!single.empty())
            beside([&](cudaStream_t lane) {
                k_fps_block<<<static_cast<int>(single.size()), kFpsThreads, 0, lane>>>(
                    d_points, longs(o_point_offset), ints(o_point_count), ints(o_seed_count), longs(o_seed_offset),
                    ints(o_single), d_nearest, d_seeds);
            });
        cudaEventDestroy(fork);
    }
    check(cudaGetLastError(), "farthest-point seeds");
    check(cudaMemcpyAsync(seeds, d_seeds, sizeof(int) * std::max<long>(1, total_seeds), cudaMemcpyDeviceToHost,
                          stream), "download seeds");

    // per level: bindings and neighbour lists of every template in one launch each
    for (int l = 0; l < max_levels; ++l) {
        const LevelPlan& p = plan[l];
        int32_t* level_nodes = d_bind_nodes + bind_entries * l;
        double* level_weights = d_bind_weights + bind_entries * l;
        int* level_neigh = d_neigh + edge_base[l];
        k_bind<<<dim3(blocks(max_points, kBindThreads / kBindLanes), W), kBindThreads, 0, stream>>>(
            d_points, longs(o_point_offset), ints(o_point_count), d_seeds, longs(o_seed_offset), ints(o_nodes[l]),
            ints(o_support[l]), longs(o_bind_offset), level_nodes, level_weights);
        check(cudaGetLastError(), "bindings");
        if (p.max_nodes > 0)
            k_neighbours<<<dim3(blocks(p.max_nodes, kBindThreads / 32), W), kBindThreads, 0, stream>>>(
                d_points, longs(o_point_offset), d_seeds, longs(o_seed_offset), ints(o_nodes[l]), ints(o_taken[l]),
                longs(o_eoff[l]), level_neigh);
        check(cudaGetLastError(), "node edges");
        check(cudaMemcpyAsync(host_nodes(l), level_nodes, sizeof(int32_t) * bind_entries, cudaMemcpyDeviceToHost,
                              stream), "download bindings");
        check(cudaMemcpyAsync(host_weights(l), level_weights, sizeof(double) * bind_entries, cudaMemcpyDeviceToHost,
                              stream), "download bindings");
        if (p.edge_total > 0)
            check(cudaMemcpyAsync(host_neigh + edge_base[l], level_neigh, sizeof(int) * p.edge_total,
                                  cudaMemcpyDeviceToHost, stream), "download edges");
    }
    check(cudaMemcpyAsync(&failed, d_failed, sizeof(int), cudaMemcpyDeviceToHost, stream), "download");
    check(cudaStreamSynchronize(stream), "graph build");
    if (failed) throw StateError("a wait inside the farthest-point seeds ran out");

    // host: the graphs in the host build's form, one template per thread
#pragma omp parallel for schedule(dynamic, 1) if (W > 1)
    for (int t = 0; t < W; ++t) {
        TemplateGraph& g = out[t];
        const int levels = static_cast<int>(level_sizes[t].size());
        for (int l = 0; l < levels; ++l) {
            GraphLevel level;
            const int n = std::min(level_sizes[t][l], seed_count[t]);
            level.template_index.assign(seeds + seed_offset[t], seeds + seed_offset[t] + n);
            level.rest.resize(static_cast<size_t>(n) * 3);
            for (int i = 0; i < n; ++i)
                for (int k = 0; k < 3; ++k)
                    level.rest[i * 3 + k] = points[(point_offset[t] + level.template_index[i]) * 3 + k];
            level.bindings.resize(point_count[t]);
            const int32_t* nodes = host_nodes(l);
            const double* weights = host_weights(l);
            for (int v = 0; v < point_count[t]; ++v) {
                Binding& b = level.bindings[v];
                const long at = (point_offset[t] + v) * NRICP_MAX_SLOTS;
                for (int s = 0; s < NRICP_MAX_SLOTS; ++s) {
                    b.nodes[s] = nodes[at + s];
                    b.weights[s] = weights[at + s];
                }
                b.count = plan[l].support[t];
            }
            const int taken = plan[l].taken[t];
            const int* neigh = host_neigh + edge_base[l] + plan[l].eoff[t];
            std::vector<std::pair<int, int>> pairs;
            pairs.reserve(static_cast<size_t>(n) * taken);
            for (int i = 0; i < n; ++i)
                for (int k = 0; k < taken; ++k) {
                    const int o = neigh[static_cast<long>(i) * taken + k];
                    pairs.emplace_back(std::min(i, o), std::max(i, o));
                }
            std::sort(pairs.begin(), pairs.end());
            pairs.erase(std::unique(pairs.begin(), pairs.end()), pairs.end());
            level.edges.reserve(pairs.size() * 2);
            for (auto& p : pairs) {
                level.edges.push_back(p.first);
                level.edges.push_back(p.second);
            }
            g.levels.push_back(std::move(level));
        }
    }
    return out;
}

}  // namespace nricp_b200
