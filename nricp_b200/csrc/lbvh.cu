// The target's Morton-code LBVH: build and closest-point query.
//
// Build (once per target, all on the device): FP32 triangle centroids and
// scene bounds, 30-bit Morton codes with the reference's quantisation
// (src/cuda/lbvh.cu:146-168), a stable LSD radix sort of (code, index) written
// here (8-bit digits, warps ranking their keys by ballots), Karras' split search
// with index tie-breaking (lbvh.cu:177-245), and a bottom-up box fit with the
// fence + arrival-counter protocol (no waiting: the second child to arrive
// merges), straight into the traversal layout, with each child's box stored in its parent (64 B per internal node = one L2 line pair), so a
// visit costs one 64-byte load instead of three dependent ones.
//
// Query (a group of lanes per template vertex): the previous correspondence's triangle
// seeds the search radius, the traversal prunes FP32 boxes with a fixed-depth
// stack whose overflow is reported (never silently pruned), and every
// triangle it reaches is measured with the reference's FP64 closest-point
// routine (src/geometry/closest_point.cpp:24-121), so the winner, its point,
// normal and distance are those of an FP64 brute-force scan.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "per_device.hpp"

namespace nricp_b200 {

void check(cudaError_t status, const char* what);  // throws CudaError (session.cu)

namespace {

constexpr int kThreads = 256;
constexpr int kSortItems = 8;                       // keys per thread per tile
constexpr int kSortTile = kThreads * kSortItems;    // 2048 keys
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;             // 256 bins, one per thread
// Up to this many tiles every tile's block sums the tiles' counts itself; past
// it a scan kernel does (each block's sum would pass 10 us).
constexpr int kTilesSummed = 128;

int blocks_for(long n, int threads = kThreads) { return (int)((n + threads - 1) / threads); }

__device__ inline uint32_t expand_bits(uint32_t v) {  // lbvh.cu:132-139
    v &= 0x000003ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// Floats as integers in the same order (negative ones flipped), so that the
// scene bounds are integer atomics: minima and maxima are exact in any order.
__device__ inline uint32_t ordered_bits(float x) {
    const uint32_t b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ inline float ordered_float(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// Triangle centroids from FP32 copies of the corners ((a+b+c)/3 with each
// operation rounded on its own, as lbvh.cu:44-45 evaluates it), and their
// bounds: three ordered minima, then three ordered maxima, complemented so
// that all six start from 0xff bytes.  (Folding the blocks' partial bounds in
// one thread took 85 to 108 us, a third of a hierarchy export.)
__global__ void k_centroids(const double* __restrict__ points, const int32_t* __restrict__ faces,
                            int count, float* __restrict__ centroids, uint32_t* __restrict__ ordered) {
    // bounds start at +-3.4e38, and a centroid that is no number does not count
    const uint32_t start = ordered_bits(3.4e38f), start_max = ~ordered_bits(-3.4e38f);
    uint32_t best[6] = {start, start, start, start_max, start_max, start_max};
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (long)gridDim.x * blockDim.x) {
        const int32_t* f = faces + t * 3;
        for (int k = 0; k < 3; ++k) {
            const float a = __double2float_rn(points[(long)f[0] * 3 + k]);
            const float b = __double2float_rn(points[(long)f[1] * 3 + k]);
            const float c = __double2float_rn(points[(long)f[2] * 3 + k]);
            const float m = __fdiv_rn(__fadd_rn(__fadd_rn(a, b), c), 3.0f);
            centroids[t * 3 + k] = m;
            if (m != m) continue;
            const uint32_t o = ordered_bits(m);
            best[k] = min(best[k], o);
            best[3 + k] = min(best[3 + k], ~o);
        }
    }
    for (int k = 0; k < 6; ++k) best[k] = __reduce_min_sync(0xffffffffu, best[k]);
    __shared__ uint32_t warp_best[6][kThreads / 32];
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 6; ++k) warp_best[k][threadIdx.x >> 5] = best[k];
    __syncthreads();
    if (threadIdx.x < 6) {
        uint32_t x = warp_best[threadIdx.x][0];
        for (int i = 1; i < kThreads / 32; ++i) x = min(x, warp_best[threadIdx.x][i]);
        atomicMin(ordered + threadIdx.x, x);
    }
}

// Morton codes in the caller's numbering, the identity permutation, the bounds
// as floats, and the first sort pass's digit counts: a block per sort tile.
__global__ void k_morton(const float* __restrict__ centroids, int count, const uint32_t* __restrict__ ordered,
                         float* __restrict__ bounds_out, uint32_t* __restrict__ codes, uint32_t* __restrict__ order,
                         uint32_t* __restrict__ counts) {
    __shared__ uint32_t bins[kRadix];
    bins[threadIdx.x] = 0;
    __syncthreads();
    float lo[3], scale[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = ordered_float(ordered[k]);
        const float hi = ordered_float(~ordered[3 + k]);
        const float extent = __fsub_rn(hi, lo[k]);
        scale[k] = extent > 1e-10f ? __fdiv_rn(1023.0f, extent) : 0.0f;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            bounds_out[k] = lo[k];
            bounds_out[3 + k] = hi;
        }
    }
    const long base = (long)blockIdx.x * kSortTile;
    for (int i = threadIdx.x; i < kSortTile; i += kThreads) {
        const long t = base + i;
        if (t >= count) break;
        uint32_t q[3];
        for (int k = 0; k < 3; ++k)
            q[k] = (uint32_t)fminf(1023.0f, fmaxf(0.0f, __fmul_rn(__fsub_rn(centroids[t * 3 + k], lo[k]), scale[k])));
        const uint32_t code = (expand_bits(q[2]) << 2) | (expand_bits(q[1]) << 1) | expand_bits(q[0]);
        codes[t] = code;
        order[t] = (uint32_t)t;
        atomicAdd(&bins[code & (kRadix - 1)], 1u);
    }
    __syncthreads();
    counts[(long)blockIdx.x * kRadix + threadIdx.x] = bins[threadIdx.x];
}

// ---- stable LSD radix sort of (key, value), 8-bit digits ---------------------
//
// Per pass: each 2,048-key tile's digit counts (tile-major), then a scatter
// whose block finds its tile's place for every digit by summing the tiles'
// counts, a thread per digit -- or, past kTilesSummed tiles, reads the sums a
// scan kernel left.  Eight-bit digits sort 30-bit codes in four passes; with
// 4-bit digits it was eight passes of three kernels each, 60 % of the build.

__global__ void k_radix_counts(const uint32_t* __restrict__ keys, long count, int shift,
                               uint32_t* __restrict__ counts) {
    __shared__ uint32_t bins[kRadix];
    bins[threadIdx.x] = 0;
    __syncthreads();
    const long base = (long)blockIdx.x * kSortTile;
    for (int i = threadIdx.x; i < kSortTile; i += kThreads)
        if (base + i < count) atomicAdd(&bins[(keys[base + i] >> shift) & (kRadix - 1)], 1u);
    __syncthreads();
    counts[(long)blockIdx.x * kRadix + threadIdx.x] = bins[threadIdx.x];
}

// A block per digit: its counts over the tiles become exclusive sums, the
// digit's total goes after the last tile's row.
__global__ void k_radix_sums(uint32_t* __restrict__ counts, int tiles) {
    __shared__ uint32_t warp_sum[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t running = 0;
    for (int base = 0; base < tiles; base += kThreads) {
        const int t = base + threadIdx.x;
        const uint32_t c = t < tiles ? counts[(long)t * kRadix + blockIdx.x] : 0;
        uint32_t x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        uint32_t before = 0, all = 0;
        for (int i = 0; i < kThreads / 32; ++i) {
            if (i < warp) before += warp_sum[i];
            all += warp_sum[i];
        }
        if (t < tiles) counts[(long)t * kRadix + blockIdx.x] = running + before + x - c;
        running += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) counts[(long)tiles * kRadix + blockIdx.x] = running;
}

// Each warp owns 256 consecutive keys of the tile and ranks them 32 at a time
// in order, so equal digits keep their input order.
__global__ void __launch_bounds__(kThreads) k_radix_scatter(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ values_in, long count, int shift,
    const uint32_t* __restrict__ counts, int tiles, int summed, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ values_out) {
    constexpr int kWarps = kThreads / 32;
    __shared__ uint32_t held[kWarps][kRadix];  // a warp's keys of each digit so far; then its place for the digit
    __shared__ uint32_t warp_sum[kWarps];
    __shared__ alignas(16) uint32_t part[2][4][kRadix];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, digit = threadIdx.x;
    for (int i = 0; i < kWarps; ++i) held[i][digit] = 0;
    // this tile's keys before it per digit, and the digit's total
    uint32_t before = 0, total = 0;
    if (summed) {
        before = counts[(long)blockIdx.x * kRadix + digit];
        total = counts[(long)tiles * kRadix + digit];
    } else {
        // four digits and every fourth tile per thread
        const int quad = threadIdx.x & 63, row = threadIdx.x >> 6;
        uint4 b4 = make_uint4(0, 0, 0, 0), t4 = b4;
#pragma unroll 8
        for (int t = row; t < tiles; t += 4) {
            const uint4 c = reinterpret_cast<const uint4*>(counts + (long)t * kRadix)[quad];
            t4.x += c.x; t4.y += c.y; t4.z += c.z; t4.w += c.w;
            if (t < (int)blockIdx.x) { b4.x += c.x; b4.y += c.y; b4.z += c.z; b4.w += c.w; }
        }
        reinterpret_cast<uint4*>(part[0][row])[quad] = b4;
        reinterpret_cast<uint4*>(part[1][row])[quad] = t4;
        __syncthreads();
        for (int i = 0; i < 4; ++i) {
            before += part[0][i][digit];
            total += part[1][i][digit];
        }
    }
    uint32_t x = total;  // exclusive scan of the totals over the digits
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    uint32_t place = before + x - total;
    for (int i = 0; i < warp; ++i) place += warp_sum[i];
    // ranks within the warp's keys
    const long base = (long)blockIdx.x * kSortTile + warp * (kSortTile / kWarps) + lane;
    uint32_t k[kSortItems], v[kSortItems], rank[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const long at = base + i * 32;
        k[i] = at < count ? keys_in[at] : 0xffffffffu;
        v[i] = at < count ? values_in[at] : 0;
    }
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const bool on = base + i * 32 < count;
        const uint32_t d = (k[i] >> shift) & (kRadix - 1);
        uint32_t same = __ballot_sync(0xffffffffu, on);  // the lanes with this digit
#pragma unroll
        for (int bit = 0; bit < kRadixBits; ++bit) {
            const uint32_t set = __ballot_sync(0xffffffffu, (d >> bit) & 1u);
            same &= ((d >> bit) & 1u) ? set : ~set;
        }
        const uint32_t ahead = on ? held[warp][d] : 0;
        rank[i] = ahead + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (on && (same >> lane) == 1u) held[warp][d] = rank[i] + 1;  // its last lane
        __syncwarp();
    }
    __syncthreads();
    // each warp's place for the digit
    for (int i = 0; i < kWarps; ++i) {
        const uint32_t c = held[i][digit];
        held[i][digit] = place;
        place += c;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        if (base + i * 32 >= count) continue;
        const uint32_t at = held[warp][(k[i] >> shift) & (kRadix - 1)] + rank[i];
        keys_out[at] = k[i];
        values_out[at] = v[i];
    }
}

size_t radix_count_bytes(long n) {
    return sizeof(uint32_t) * kRadix * (size_t)((n + kSortTile - 1) / kSortTile + 1);
}

// Sorts by the low `bits` bits between the two buffer pairs; returns the pair
// that holds the result.  `counted`: the first pass's counts are there.
int radix_sort(uint32_t* const keys[2], uint32_t* const values[2], long n, int bits, bool counted, uint32_t* counts,
               cudaStream_t stream) {
    const int tiles = (int)((n + kSortTile - 1) / kSortTile);
    const int summed = tiles > kTilesSummed ? 1 : 0;
    int cur = 0;
    for (int shift = 0; shift < bits; shift += kRadixBits) {
        if (shift > 0 || !counted) k_radix_counts<<<tiles, kThreads, 0, stream>>>(keys[cur], n, shift, counts);
        if (summed) k_radix_sums<<<kRadix, kThreads, 0, stream>>>(counts, tiles);
        k_radix_scatter<<<tiles, kThreads, 0, stream>>>(keys[cur], values[cur], n, shift, counts, tiles, summed,
                                                        keys[1 - cur], values[1 - cur]);
        cur = 1 - cur;
    }
    return cur;
}

int radix_sort_launches(long n, int bits, bool counted) {
    const int passes = (bits + kRadixBits - 1) / kRadixBits;
    return passes * ((n + kSortTile - 1) / kSortTile > kTilesSummed ? 3 : 2) - (counted ? 1 : 0);
}

constexpr int kCodeBits = 30;

// Centroids, bounds, codes and the sort, shared by the build and the export:
// returns the buffer pair with the sorted codes (with 30-bit codes the first).
int sorted_codes(const double* points, const int32_t* faces, int n, float* centroids, uint32_t* ordered, float* bounds,
                 uint32_t* const keys[2], uint32_t* const values[2], uint32_t* counts, cudaStream_t stream) {
    const int blocks = blocks_for(n);
    cudaMemsetAsync(ordered, 0xff, sizeof(uint32_t) * 6, stream);
    k_centroids<<<blocks < 592 ? blocks : 592, kThreads, 0, stream>>>(points, faces, n, centroids, ordered);
    k_morton<<<blocks_for(n, kSortTile), kThreads, 0, stream>>>(centroids, n, ordered, bounds, keys[0], values[0],
                                                                counts);
    return radix_sort(keys, values, n, kCodeBits, true, counts, stream);
}

// ---- Karras build --------------------------------------------------------

__device__ inline int lcp(const uint32_t* codes, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = codes[i], b = codes[j];
    if (a == b) return 32 + __clz((uint32_t)(i ^ j));
    return __clz(a ^ b);
}

// Internal node i covers a range and splits it (lbvh.cu:190-245).  Children
// are written in the reference's numbering: a leaf is its sorted position
// (< n), an internal node is n + index.  `left` and `right` are for exports
// (may be null); `parent` (may be null) holds, for every child, twice its
// parent's index, plus one for a right child, and -1 for the root.
__global__ void k_karras(const uint32_t* __restrict__ codes, int n, int32_t* __restrict__ left,
                         int32_t* __restrict__ right, int32_t* __restrict__ parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int pp = lcp(codes, n, i, i - 1);
    const int pn = lcp(codes, n, i, i + 1);
    const int dir = pn > pp ? 1 : -1;
    const int pmin = pp < pn ? pp : pn;
    int span = 2;
    while (lcp(codes, n, i, i + span * dir) > pmin) span *= 2;
    int last = 0;
    for (int step = span / 2; step >= 1; step /= 2)
        if (lcp(codes, n, i, i + (last + step) * dir) > pmin) last += step;
    const int j = i + last * dir;
    const int rl = i < j ? i : j, rr = i < j ? j : i;
    const int np = lcp(codes, n, rl, rr);
    int offset = 0, step = rr - rl;
    do {
        step = (step + 1) / 2;
        if (lcp(codes, n, rl, rl + offset + step) > np) offset += step;
    } while (step > 1);
    const int split = rl + offset;
    const int lc = rl == split ? rl : n + split;
    const int rc = split + 1 == rr ? rr : n + split + 1;
    if (left) {
        left[i] = lc;
        right[i] = rc;
    }
    if (parent) {
        parent[lc] = 2 * i;
        parent[rc] = 2 * i + 1;
        if (i == 0) parent[n] = -1;
    }
}

// The traversal layout, bottom up in one pass.  A leaf is packed (80 bytes: its
// FP64 corners and triangle) and its box taken from the FP32 corners; then each
// child writes its box and code into its half of its parent's node (4 float4:
// left box lo and hi, right box lo and hi, the two children), and the second to
// arrive goes on with the union.  The fence makes a half visible before its
// arrival is counted, and nothing ever waits.  (Boxes in an array of their own,
// packed by two more kernels, took 190 us at 494,000 triangles,
// now 103.)
__global__ void k_refit(const double* __restrict__ points, const int32_t* __restrict__ faces,
                        const uint32_t* __restrict__ order, int n, const int32_t* __restrict__ parent,
                        uint32_t* __restrict__ arrivals, float4* __restrict__ nodes, float4* __restrict__ leaves) {
    const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf >= n) return;
    const int tri = (int)order[leaf];
    const int32_t* f = faces + (long)tri * 3;
    double c[9];
    for (int k = 0; k < 3; ++k)
        for (int a = 0; a < 3; ++a) c[k * 3 + a] = points[(long)f[k] * 3 + a];
    double2* l = reinterpret_cast<double2*>(leaves) + (long)leaf * kLeafFloat4s;
    l[0] = make_double2(c[0], c[1]);
    l[1] = make_double2(c[2], c[3]);
    l[2] = make_double2(c[4], c[5]);
    l[3] = make_double2(c[6], c[7]);
    l[4] = make_double2(c[8], __longlong_as_double((long long)tri));
    if (n == 1) return;
    float lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        const float x = __double2float_rn(c[k]), y = __double2float_rn(c[3 + k]), z = __double2float_rn(c[6 + k]);
        lo[k] = fminf(x, fminf(y, z));
        hi[k] = fmaxf(x, fmaxf(y, z));
    }
    uint32_t code = kLeafBit | (uint32_t)leaf;
    int up = parent[leaf];
    for (int depth = 0; depth < 2 * n + 2 && up >= 0; ++depth) {
        const int p = up >> 1, side = up & 1;
        float* node = reinterpret_cast<float*>(nodes + (long)p * 4);
        float2* mine = reinterpret_cast<float2*>(node + side * 6);
        mine[0] = make_float2(lo[0], lo[1]);
        mine[1] = make_float2(lo[2], hi[0]);
        mine[2] = make_float2(hi[1], hi[2]);
        node[12 + side] = __uint_as_float(code);
        __threadfence();
        if (atomicAdd(&arrivals[p], 1u) != 1u) return;
        __threadfence();
        const float2* other = reinterpret_cast<const float2*>(node + (1 - side) * 6);
        const float2 o0 = __ldcg(other), o1 = __ldcg(other + 1), o2 = __ldcg(other + 2);
        lo[0] = fminf(lo[0], o0.x); lo[1] = fminf(lo[1], o0.y); lo[2] = fminf(lo[2], o1.x);
        hi[0] = fmaxf(hi[0], o1.y); hi[1] = fmaxf(hi[1], o2.x); hi[2] = fmaxf(hi[2], o2.y);
        code = (uint32_t)p;
        up = parent[n + p];
    }
}

}  // namespace

size_t lbvh_scratch_bytes(int n) {
    // the carve sequence of lbvh_build, each piece rounded up to 256 bytes
    const size_t pieces[] = {
        sizeof(float) * 3 * (size_t)n,                 // centroids
        64,                                            // bounds, ordered
        64,                                            // bounds
        sizeof(uint32_t) * (size_t)n, sizeof(uint32_t) * (size_t)n,  // keys x2
        sizeof(uint32_t) * (size_t)n, sizeof(uint32_t) * (size_t)n,  // values x2
        radix_count_bytes(n),                          // digit counts
        sizeof(int32_t) * (size_t)n, sizeof(int32_t) * (size_t)n,    // left, right (export)
        sizeof(int32_t) * 2 * (size_t)n,               // parent
        sizeof(uint32_t) * (size_t)n,                  // arrivals
    };
    size_t total = 0;
    for (size_t bytes : pieces) total += (bytes + 255) & ~size_t(255);
    return total + 256;
}

// Builds the hierarchy over `n` target triangles into `nodes` ((n-1) x 4
// float4) and `leaves` (n x kLeafFloat4s float4) using `scratch`; optionally exports the
// canonical arrays (sorted codes, permutation, Karras children) for parity
// tests.  Returns the encoded root.
uint32_t lbvh_build(const double* points, const int32_t* faces, int n, void* scratch,
                    float4* nodes, float4* leaves, cudaStream_t stream, LbvhExport* out) {
    char* base = static_cast<char*>(scratch);
    auto carve = [&base](size_t bytes) {
        char* p = base;
        base += (bytes + 255) & ~size_t(255);
        return p;
    };
    float* centroids = reinterpret_cast<float*>(carve(sizeof(float) * 3 * n));
    uint32_t* ordered = reinterpret_cast<uint32_t*>(carve(64));
    float* bounds = reinterpret_cast<float*>(carve(64));
    uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * n)),
                         reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * n))};
    uint32_t* values[2] = {reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * n)),
                           reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * n))};
    uint32_t* counts = reinterpret_cast<uint32_t*>(carve(radix_count_bytes(n)));
    int32_t* left = reinterpret_cast<int32_t*>(carve(sizeof(int32_t) * n));
    int32_t* right = reinterpret_cast<int32_t*>(carve(sizeof(int32_t) * n));
    int32_t* parent = reinterpret_cast<int32_t*>(carve(sizeof(int32_t) * 2 * n));
    uint32_t* arrivals = reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * n));

    const int cur = sorted_codes(points, faces, n, centroids, ordered, bounds, keys, values, counts, stream);
    const uint32_t* codes = keys[cur];
    const uint32_t* order = values[cur];
    if (n > 1) {
        cudaMemsetAsync(arrivals, 0, sizeof(uint32_t) * n, stream);
        k_karras<<<blocks_for(n - 1), kThreads, 0, stream>>>(codes, n, out ? left : nullptr, out ? right : nullptr,
                                                             parent);
    }
    k_refit<<<blocks_for(n), kThreads, 0, stream>>>(points, faces, order, n, parent, arrivals, nodes, leaves);
    if (out) {
        cudaMemcpyAsync(out->codes, codes, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, stream);
        cudaMemcpyAsync(out->order, order, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, stream);
        if (n > 1) {
            cudaMemcpyAsync(out->left, left, sizeof(int32_t) * (n - 1), cudaMemcpyDeviceToHost, stream);
            cudaMemcpyAsync(out->right, right, sizeof(int32_t) * (n - 1), cudaMemcpyDeviceToHost, stream);
        }
        cudaMemcpyAsync(out->bounds, bounds, sizeof(float) * 6, cudaMemcpyDeviceToHost, stream);
    }
    return n > 1 ? 0u : (kLeafBit | 0u);
}

int lbvh_build_launches(int n) { return 2 + radix_sort_launches(n, kCodeBits, true) + (n > 1 ? 2 : 1); }

// ---------------------------------------------------------------------------
// Target ingestion: normalisation and vertex normals on the device
// ---------------------------------------------------------------------------
//
// The target arrives in the caller's units.  Its points are moved into the
// normalised frame in place, (p - center) * scale per coordinate with the two
// roundings of the host's normalisation (mesh.cpp:183-187), and its
// area-weighted vertex normals (mesh.cpp:71-88) are summed per vertex over
// its faces in ascending face order, as the host's face loop adds them, then
// normalised -- so both are bit-identical to the host's.  A vertex's faces
// come from a stable sort of the (vertex, face) corner pairs by vertex.

namespace {

__global__ void k_normalize(double* __restrict__ p, long count, double cx, double cy, double cz,
                            double scale) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const int k = (int)(i % 3);
    const double c = k == 0 ? cx : (k == 1 ? cy : cz);
    p[i] = __dmul_rn(__dsub_rn(p[i], c), scale);
}

__global__ void k_corner_keys(const int32_t* __restrict__ faces, long corners, uint32_t* __restrict__ keys,
                              uint32_t* __restrict__ values) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= corners) return;
    keys[i] = (uint32_t)faces[i];
    values[i] = (uint32_t)(i / 3);
}

__device__ inline long lower_bound_key(const uint32_t* __restrict__ keys, long n, uint32_t x) {
    long lo = 0, hi = n;
    while (lo < hi) {
        const long mid = (lo + hi) >> 1;
        if (keys[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

__global__ void k_target_normals(const double* __restrict__ p, int n, const int32_t* __restrict__ faces,
                                 const uint32_t* __restrict__ keys, const uint32_t* __restrict__ face_of,
                                 long corners, double* __restrict__ normals) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const long j0 = lower_bound_key(keys, corners, (uint32_t)v);
    const long j1 = lower_bound_key(keys, corners, (uint32_t)v + 1u);
    double t0 = 0.0, t1 = 0.0, t2 = 0.0;
    for (long j = j0; j < j1; ++j) {
        const int32_t* f = faces + (long)face_of[j] * 3;
        const double* a = p + (long)f[0] * 3;
        const double* b = p + (long)f[1] * 3;
        const double* c = p + (long)f[2] * 3;
        const double e10 = __dsub_rn(b[0], a[0]), e11 = __dsub_rn(b[1], a[1]), e12 = __dsub_rn(b[2], a[2]);
        const double e20 = __dsub_rn(c[0], a[0]), e21 = __dsub_rn(c[1], a[1]), e22 = __dsub_rn(c[2], a[2]);
        t0 = __dadd_rn(t0, __dsub_rn(__dmul_rn(e11, e22), __dmul_rn(e12, e21)));
        t1 = __dadd_rn(t1, __dsub_rn(__dmul_rn(e12, e20), __dmul_rn(e10, e22)));
        t2 = __dadd_rn(t2, __dsub_rn(__dmul_rn(e10, e21), __dmul_rn(e11, e20)));
    }
    const double length =
        __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(t0, t0), __dmul_rn(t1, t1)), __dmul_rn(t2, t2)));
    double* out = normals + (long)v * 3;
    if (length > 0.0) {
        out[0] = __ddiv_rn(t0, length);
        out[1] = __ddiv_rn(t1, length);
        out[2] = __ddiv_rn(t2, length);
    } else {
        out[0] = out[1] = out[2] = 0.0;
    }
}

// Key bits that cover vertex indices below n.
int corner_key_bits(int n) {
    int bits = 1;
    while (bits < 32 && (1u << bits) < (uint32_t)n) ++bits;
    return bits;
}

}  // namespace

size_t ingest_scratch_bytes(int n, int F) {
    const size_t corners = (size_t)F * 3;
    const size_t pieces[] = {sizeof(uint32_t) * corners, sizeof(uint32_t) * corners,
                             sizeof(uint32_t) * corners, sizeof(uint32_t) * corners,
                             radix_count_bytes((long)corners)};
    size_t total = 0;
    for (size_t bytes : pieces) total += (bytes + 255) & ~size_t(255);
    (void)n;
    return total + 256;
}

int ingest_launches(int n, int F) {
    return 2 + (F > 0 ? 1 + radix_sort_launches((long)F * 3, corner_key_bits(n), false) : 0);
}

void ingest_target(double* points, int n, const int32_t* faces, int F, const double center[3], double scale,
                   double* normals, void* scratch, cudaStream_t stream) {
    k_normalize<<<blocks_for((long)n * 3), kThreads, 0, stream>>>(points, (long)n * 3, center[0], center[1],
                                                                  center[2], scale);
    const long corners = (long)F * 3;
    char* base = static_cast<char*>(scratch);
    auto carve = [&base](size_t bytes) {
        char* q = base;
        base += (bytes + 255) & ~size_t(255);
        return q;
    };
    uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * corners)),
                         reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * corners))};
    uint32_t* values[2] = {reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * corners)),
                           reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * corners))};
    uint32_t* counts = reinterpret_cast<uint32_t*>(carve(radix_count_bytes(corners)));
    int cur = 0;
    if (F > 0) {
        k_corner_keys<<<blocks_for(corners), kThreads, 0, stream>>>(faces, corners, keys[0], values[0]);
        cur = radix_sort(keys, values, corners, corner_key_bits(n), false, counts, stream);
    }
    k_target_normals<<<blocks_for(n), kThreads, 0, stream>>>(points, n, faces, keys[cur], values[cur], corners,
                                                             normals);
}

// ---------------------------------------------------------------------------
// Closest-point query
// ---------------------------------------------------------------------------

__device__ inline float box_distance(F3 p, float lx, float ly, float lz, float hx, float hy,
                                     float hz) {
    const float dx = fmaxf(fmaxf(lx - p.x, p.x - hx), 0.0f);
    const float dy = fmaxf(fmaxf(ly - p.y, p.y - hy), 0.0f);
    const float dz = fmaxf(fmaxf(lz - p.z, p.z - hz), 0.0f);
    return dx * dx + dy * dy + dz * dz;
}

// FP64 closest point with barycentrics, the reference routine's exact steps
// (closest_point.cpp:24-121), with every product and sum rounded on its own so
// the result matches the host build bit for bit.
__device__ inline double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ inline double da(double a, double b) { return __dadd_rn(a, b); }
__device__ inline double ds(double a, double b) { return __dsub_rn(a, b); }
__device__ inline D3 vsub(D3 a, D3 b) { return {ds(a.x, b.x), ds(a.y, b.y), ds(a.z, b.z)}; }
__device__ inline D3 vadd(D3 a, D3 b) { return {da(a.x, b.x), da(a.y, b.y), da(a.z, b.z)}; }
__device__ inline D3 vmul(D3 a, double s) { return {dm(a.x, s), dm(a.y, s), dm(a.z, s)}; }
__device__ inline double vdot(D3 a, D3 b) { return da(da(dm(a.x, b.x), dm(a.y, b.y)), dm(a.z, b.z)); }

__device__ D3 closest_point_fp64(D3 p, D3 a, D3 b, D3 c, double* bary) {
    const D3 ab = vsub(b, a), ac = vsub(c, a), ap = vsub(p, a);
    const double d1 = vdot(ab, ap), d2 = vdot(ac, ap);
    if (d1 <= 0.0 && d2 <= 0.0) { bary[0] = 1; bary[1] = 0; bary[2] = 0; return a; }
    const D3 bp = vsub(p, b);
    const double d3 = vdot(ab, bp), d4 = vdot(ac, bp);
    if (d3 >= 0.0 && d4 <= d3) { bary[0] = 0; bary[1] = 1; bary[2] = 0; return b; }
    const double vc = ds(dm(d1, d4), dm(d3, d2));
    if (vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0) {
        const double den = ds(d1, d3);
        const double v = den != 0.0 ? __ddiv_rn(d1, den) : 0.0;
        bary[0] = ds(1.0, v); bary[1] = v; bary[2] = 0.0;
        return vadd(a, vmul(ab, v));
    }
    const D3 cp = vsub(p, c);
    const double d5 = vdot(ab, cp), d6 = vdot(ac, cp);
    if (d6 >= 0.0 && d5 <= d6) { bary[0] = 0; bary[1] = 0; bary[2] = 1; return c; }
    const double vb = ds(dm(d5, d2), dm(d1, d6));
    if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) {
        const double den = ds(d2, d6);
        const double w = den != 0.0 ? __ddiv_rn(d2, den) : 0.0;
        bary[0] = ds(1.0, w); bary[1] = 0.0; bary[2] = w;
        return vadd(a, vmul(ac, w));
    }
    const double va = ds(dm(d3, d6), dm(d5, d4));
    if (va <= 0.0 && ds(d4, d3) >= 0.0 && ds(d5, d6) >= 0.0) {
        const double den = da(ds(d4, d3), ds(d5, d6));
        const double w = den != 0.0 ? __ddiv_rn(ds(d4, d3), den) : 0.0;
        bary[0] = 0.0; bary[1] = ds(1.0, w); bary[2] = w;
        return vadd(b, vmul(vsub(c, b), w));
    }
    const double den = da(da(va, vb), vc);
    if (fabs(den) < 1e-300) { bary[0] = 1; bary[1] = 0; bary[2] = 0; return a; }
    const double v = __ddiv_rn(vb, den), w = __ddiv_rn(vc, den);
    bary[0] = ds(ds(1.0, v), w); bary[1] = v; bary[2] = w;
    return vadd(vadd(a, vmul(ab, v)), vmul(ac, w));
}

__device__ inline D3 vnormalized(D3 a) {
    const double length = __dsqrt_rn(vdot(a, a));
    if (!(length > 0.0)) return {0.0, 0.0, 0.0};
    return {__ddiv_rn(a.x, length), __ddiv_rn(a.y, length), __ddiv_rn(a.z, length)};
}

// Robust weight, src/energy/robust.cpp:30-58.
__device__ inline double robust_weight(int kernel, double squared, double threshold) {
    if (squared < 0.0) squared = 0.0;
    if (kernel == 1) {
        if (threshold <= 0.0) return 1.0;
        if (squared <= threshold * threshold) return 1.0;
        return threshold / sqrt(squared);
    }
    if (kernel == 2) {
        if (threshold <= 0.0) return 1.0;
        const double ratio = squared / (threshold * threshold);
        const double den = 1.0 + ratio;
        return 1.0 / (den * den);
    }
    return 1.0;
}

// FP64 squared distance from q to triangle `tri` of the target.
__device__ inline double triangle_distance_fp64(const WrapDev& w, D3 q, int tri) {
    const int32_t* f = w.tgt_faces + (long)tri * 3;
    double bary[3];
    const D3 c = closest_point_fp64(q, load_d3(w.tgt_points, f[0]), load_d3(w.tgt_points, f[1]),
                                    load_d3(w.tgt_points, f[2]), bary);
    const D3 d = vsub(c, q);
    return vdot(d, d);
}

// FP64 squared distance from q to the triangle of leaf `leaf` (its corners
// are stored in FP64), and the triangle's index.
__device__ inline double leaf_distance(const WrapDev& w, int leaf, D3 q, int* tri) {
    const double2* l = reinterpret_cast<const double2*>(w.bvh_leaves) + (long)leaf * (kLeafFloat4s);
    const double2 l0 = __ldg(l), l1 = __ldg(l + 1), l2 = __ldg(l + 2), l3 = __ldg(l + 3),
                  l4 = __ldg(l + 4);
    *tri = (int)__double_as_longlong(l4.y);
    double bary[3];
    const D3 c = closest_point_fp64(q, {l0.x, l0.y, l1.x}, {l1.y, l2.x, l2.y}, {l3.x, l3.y, l4.x}, bary);
    const D3 d = vsub(c, q);
    return vdot(d, d);
}

// Nearest target triangle for `q`: the FP64 brute-force answer (smallest
// FP64 distance from the reference's closest-point routine, exact ties to the
// lowest triangle index), found by walking the hierarchy.  Boxes are pruned
// in FP32, which is well conditioned (a box distance is a clamp and three
// squares), with `w.rank_window` of slack, far above the rounding of the FP32
// boxes and query; every triangle reached is measured in FP64 -- an FP32
// closest-point routine can misplace its point on thin sliver triangles by
// far more than any fixed window.  `seed` is a triangle whose distance bounds
// the search from the start.  Returns the winner, or -1.
__device__ int nearest_triangle(const WrapDev& w, F3 q, D3 q64, int seed, int* overflow) {
    const double slack = (double)w.rank_window;
    double best = 1e300;     // FP64 squared distance of the best triangle so far
    float bound = 3.4e38f;   // FP32 pruning radius^2: (sqrt(best) + slack)^2, rounded up
    int best_tri = -1;
    auto consider = [&](int tri, double d) {
        if (d < best || (d == best && tri < best_tri)) {
            best = d;
            best_tri = tri;
            const double r = sqrt(best) + slack;
            bound = __double2float_ru(r * r);
        }
    };
    if (seed >= 0 && seed < w.F) consider(seed, triangle_distance_fp64(w, q64, seed));
    uint32_t stack[kStackDepth];
    float stack_d[kStackDepth];
    int sp = 0;
    uint32_t node = (uint32_t)w.bvh_root;
    // A tree visits each node at most once; the cap only guards against a
    // corrupt hierarchy, which it reports instead of looping.
    const long step_limit = 4L * (long)w.F + 1024;
    long steps = 0;
    while (true) {
        if (++steps > step_limit) {
            *overflow = 1;
            break;
        }
        if (node & kLeafBit) {
            int tri;
            const double d = leaf_distance(w, (int)(node & ~kLeafBit), q64, &tri);
            if (tri != seed) consider(tri, d);
        } else {
            const float4* nd = w.bvh_nodes + (long)node * 4;
            const float4 n0 = __ldg(nd), n1 = __ldg(nd + 1), n2 = __ldg(nd + 2), n3 = __ldg(nd + 3);
            const float dl = box_distance(q, n0.x, n0.y, n0.z, n0.w, n1.x, n1.y);
            const float dr = box_distance(q, n1.z, n1.w, n2.x, n2.y, n2.z, n2.w);
            const uint32_t cl = __float_as_uint(n3.x), cr = __float_as_uint(n3.y);
            const bool hl = dl < bound, hr = dr < bound;
            if (hl && hr) {
                const bool left_first = dl <= dr;
                if (sp < kStackDepth) {
                    stack[sp] = left_first ? cr : cl;
                    stack_d[sp] = left_first ? dr : dl;
                    ++sp;
                } else {
                    *overflow = 1;
                }
                node = left_first ? cl : cr;
                continue;
            }
            if (hl) { node = cl; continue; }
            if (hr) { node = cr; continue; }
        }
        // pop the next subtree that can still hold something closer
        bool found = false;
        while (sp > 0) {
            --sp;
            if (stack_d[sp] < bound) { node = stack[sp]; found = true; break; }
        }
        if (!found) break;
    }
    return best_tri;
}

// Walks longer than this many steps put their vertex on the wrap's list for
// its next query, where a warp walks it (a vertex over a hole in the target,
// or above the fan of slivers at a lat-long pole, stays far from the nearest
// triangles and walks hundreds to thousands of steps query after query).
constexpr long kLongWalk = 256;
// Lanes per query for `total` queries on a grid of `resident` threads: the
// widest groups that keep the grid about as busy.  A walk's time is its chain of
// dependent rounds, so a few queries want wide groups; many queries fill the
// device anyway, and narrower groups visit fewer subtrees that a bound found
// meanwhile would have pruned.
__host__ __device__ inline int group_lanes(long total, long resident) {
    return total * 16 <= resident * 2 ? 16 : (total * 8 <= resident * 4 ? 8 : 4);
}

// The warps' stacks of pending subtrees: 1,024 entries per warp, shared by its
// groups of G lanes.
constexpr int kWarpStack = 1024;

// The nearest triangle for `q` found by a group of G lanes of a warp (each
// group its own query): the same pruning and the same winner rule as
// `nearest_triangle`, so the same answer, with up to G pending subtrees taken
// from the stack at a time, so that a walk takes several times fewer dependent
// rounds.  All 32 lanes call it together, and a warp's groups run their rounds
// side by side until the last is done; `on` is false for a group without a
// query.  `nodes` / `dists` are the group's stack (kWarpStack * G / 32
// entries).  Should the stack not hold a round's children, the rest of the
// walk is left to one lane (`*unfinished`), seeded with the winner so far,
// which is returned.  Every lane of a group returns the same triangle; `*work`
// is the entries taken.
template <int G>
__device__ int nearest_triangle_group(const WrapDev& w, bool on, F3 q, D3 q64, int seed, uint32_t* nodes,
                                      float* dists, int* overflow, bool* unfinished, long* work) {
    constexpr int kStack = kWarpStack * G / 32;
    const int lane = threadIdx.x & 31, at_group = lane & (G - 1);
    const uint32_t group = (G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u)) << (lane - at_group);
    const uint32_t below = group & ((1u << lane) - 1u);
    const double slack = on ? (double)w.rank_window : 0.0;
    double best = 1e300;
    int best_tri = -1;
    float bound = 3.4e38f;
    if (on && seed >= 0 && seed < w.F) {
        best = triangle_distance_fp64(w, q64, seed);
        best_tri = seed;
        const double r = sqrt(best) + slack;
        bound = __double2float_ru(r * r);
    }
    // The stack holds pending internal nodes from its bottom up and pending
    // leaves from its top down; a round takes one kind for the whole warp, so
    // that the FP64 measurement and the box tests do not run by turns under
    // half-empty masks.
    const uint32_t root = on ? (uint32_t)w.bvh_root : 0;
    if (on && at_group == 0) {
        nodes[(root & kLeafBit) ? kStack - 1 : 0] = root;
        dists[(root & kLeafBit) ? kStack - 1 : 0] = 0.0f;
    }
    int inner = on && !(root & kLeafBit) ? 1 : 0;  // the same in a group's lanes
    int leaves = on && (root & kLeafBit) ? 1 : 0;
    const long round_limit = on ? 4L * (long)w.F + 1024 : 0;
    long rounds = 0, taken = 0;
    *unfinished = false;
    __syncwarp();
    while (__any_sync(0xffffffffu, inner + leaves > 0)) {
        if (inner + leaves > 0 && ++rounds > round_limit) {  // a corrupt hierarchy: report, do not loop
            *overflow = 1;
            inner = leaves = 0;
        }
        // leaves once some group can fill its lanes with them, or nothing else is left
        if (__any_sync(0xffffffffu, leaves >= G) || !__any_sync(0xffffffffu, inner > 0)) {
            // FP64 distances, then the group's winner under the exact rule
            const int take = leaves < G ? leaves : G;
            const int first = kStack - leaves;
            leaves -= take;
            taken += take;
            double d = 1e300;
            int tri = 0x7fffffff;
            if (at_group < take && dists[first + at_group] < bound) {
                int t;
                const double x = leaf_distance(w, (int)(nodes[first + at_group] & ~kLeafBit), q64, &t);
                if (t != seed) {
                    d = x;
                    tri = t;
                }
            }
            for (int o = G / 2; o > 0; o >>= 1) {
                const double od = __shfl_xor_sync(0xffffffffu, d, o);
                const int ot = __shfl_xor_sync(0xffffffffu, tri, o);
                if (od < d || (od == d && ot < tri)) {
                    d = od;
                    tri = ot;
                }
            }
            if (d < best || (d == best && tri < best_tri)) {
                best = d;
                best_tri = tri;
                const double r = sqrt(best) + slack;
                bound = __double2float_ru(r * r);
            }
            continue;
        }
        const int take = inner < G ? inner : G;
        inner -= take;
        taken += take;
        bool push[2] = {false, false};  // left, right child
        uint32_t child[2] = {0, 0};
        float dist[2] = {0.0f, 0.0f};
        if (at_group < take && dists[inner + at_group] < bound) {
            const float4* nd = w.bvh_nodes + (long)nodes[inner + at_group] * 4;
            const float4 n0 = __ldg(nd), n1 = __ldg(nd + 1), n2 = __ldg(nd + 2), n3 = __ldg(nd + 3);
            dist[0] = box_distance(q, n0.x, n0.y, n0.z, n0.w, n1.x, n1.y);
            dist[1] = box_distance(q, n1.z, n1.w, n2.x, n2.y, n2.z, n2.w);
            child[0] = __float_as_uint(n3.x);
            child[1] = __float_as_uint(n3.y);
            // the nearer child second: it is taken first
            if (dist[0] < dist[1]) {
                const float x = dist[0]; dist[0] = dist[1]; dist[1] = x;
                const uint32_t y = child[0]; child[0] = child[1]; child[1] = y;
            }
            push[0] = dist[0] < bound;
            push[1] = dist[1] < bound;
        }
        __syncwarp();
        // each kind's place: the lanes' farther children, then their nearer ones
        int new_inner = 0, new_leaves = 0, place[2] = {0, 0};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const bool leaf = (child[k] & kLeafBit) != 0;
            const uint32_t to_inner = __ballot_sync(0xffffffffu, push[k] && !leaf) & group;
            const uint32_t to_leaves = __ballot_sync(0xffffffffu, push[k] && leaf) & group;
            place[k] = leaf ? kStack - 1 - (leaves + new_leaves + __popc(to_leaves & below))
                            : inner + new_inner + __popc(to_inner & below);
            new_inner += __popc(to_inner);
            new_leaves += __popc(to_leaves);
        }
        if (inner + new_inner + leaves + new_leaves > kStack) {  // the rest by one lane, from the winner so far
            *unfinished = true;
            inner = leaves = 0;
        } else {
#pragma unroll
            for (int k = 0; k < 2; ++k)
                if (push[k]) {
                    nodes[place[k]] = child[k];
                    dists[place[k]] = dist[k];
                }
            inner += new_inner;
            leaves += new_leaves;
        }
        __syncwarp();
    }
    *work = taken;
    return best_tri;
}

__device__ inline bool queries(int phase) {
    return phase == kPhaseTransfer || phase == kPhaseRefresh || phase == kPhaseFinal;
}

// The correspondence of template vertex v to triangle `tri` (-1: none), with
// the filters in the order the reference applies them
// (correspondence.cpp:35-80) and the reweighting of route_a.cpp:19-38.
__device__ void store_correspondence(const WrapDev& w, int level, int v, int tri) {
    uint8_t code = 0;
    D3 point = {0, 0, 0}, normal = {0, 0, 0};
    double distance = 0.0, robust = 1.0;
    if (tri >= 0) {
        const D3 q = load_d3(w.deformed, v);
        const int32_t* f = w.tgt_faces + (long)tri * 3;
        double bary[3];
        point = closest_point_fp64(q, load_d3(w.tgt_points, f[0]), load_d3(w.tgt_points, f[1]),
                                   load_d3(w.tgt_points, f[2]), bary);
        const D3 d = vsub(point, q);
        distance = __dsqrt_rn(vdot(d, d));
        const D3 n0 = load_d3(w.tgt_normals, f[0]), n1 = load_d3(w.tgt_normals, f[1]),
                 n2 = load_d3(w.tgt_normals, f[2]);
        normal = vnormalized(vadd(vadd(vmul(n0, bary[0]), vmul(n1, bary[1])), vmul(n2, bary[2])));
        if (distance > w.distance_threshold) {
            code = 1;
        } else if (vdot(load_d3(w.qnormals, v), normal) < w.min_normal_cosine) {
            code = 2;
        } else if (distance > 0.0) {
            const D3 offset = vsub(q, point);
            const double slope = __ddiv_rn(fabs(vdot(normal, offset)), distance);
            if (slope < w.min_slope) code = 3;
        }
        if (code == 0) {
            const D3 o = vsub(q, point);
            const double squared = vdot(o, o);
            const double threshold = w.robust_threshold[level];
            robust = threshold > 0.0 ? robust_weight(w.robust_kernel[level], squared, threshold) : 1.0;
        }
    } else {
        code = 1;
    }
    store_d3(w.corr_point, v, point);
    store_d3(w.corr_normal, v, normal);
    w.corr_distance[v] = distance;
    w.corr_triangle[v] = tri;
    w.corr_code[v] = code;
    w.robust[v] = robust;
}

// A masked vertex keeps its previous triangle and takes no correspondence.
__device__ inline void store_masked(const WrapDev& w, int v) {
    store_d3(w.corr_point, v, {0, 0, 0});
    store_d3(w.corr_normal, v, {0, 0, 0});
    w.corr_distance[v] = 0.0;
    w.corr_code[v] = 4;
    w.robust[v] = 1.0;
}

// Puts vertex v on the wrap's list of long walks for its next query (list
// 1 - long_cur), unless the list is full.
__device__ inline void list_long_walk(const WrapDev& w, int next, int v) {
    const int at = atomicAdd(w.long_count + next, 1);
    if (at < kLongCap) {
        w.long_list[next * kLongCap + at] = v;
        w.long_flag[(long)next * w.V + v] = 1;
    }
}

// The closest points of every querying wrap, as queues over a grid that fits on
// the device at once.  First, the vertices whose walk was long at the wrap's
// previous query (its list), a warp each.  Then every other vertex of every
// querying wrap, in wrap then vertex order, handed out to whichever warp is
// free, a group of 4, 8 or 16 lanes per vertex (group_lanes).  A thread per
// vertex left a launch waiting for a chain of a few hundred dependent fetches
// with a few lanes of each warp alive; groups cut the chain and share its
// fetches: the queries of a 25,000-vertex wrap onto 394,000 triangles took
// 18.7 ms, now 5.8; of 16 uneven wraps in a batch 70 ms, now 32.  A walk longer
// than kLongWalk lists its vertex for the wrap's next query.
// counter[0]: the vertices' queue head; counter[1]: the long walks'; both
// start at 0.
__global__ void __launch_bounds__(128) k_query_queue(const WrapDev* __restrict__ wraps, int wrap_count,
                                                    int* __restrict__ counter) {
    extern __shared__ float4 query_shared[];  // 4 warps' stacks, then 2 x (wrap_count + 1) ints
    uint32_t* stack_nodes = reinterpret_cast<uint32_t*>(query_shared);
    float* stack_dists = reinterpret_cast<float*>(stack_nodes + 4 * kWarpStack);
    int* first = reinterpret_cast<int*>(stack_dists + 4 * kWarpStack);  // each wrap's first vertex item
    int* first_long = first + wrap_count + 1;                             // and first long-walk item
    for (int i = threadIdx.x; i < wrap_count; i += blockDim.x) {
        const WrapDev& w = wraps[i];
        const bool on = queries(w.control->tick_phase);
        first[i + 1] = on ? w.V : 0;
        first_long[i + 1] = on ? min(w.long_count[w.control->long_cur], kLongCap) : 0;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // inclusive scans by warp 0, 32 wraps at a time
        const int lane = threadIdx.x;
        for (int k = 0; k < 2; ++k) {
            int* f = k == 0 ? first : first_long;
            int carry = 0;
            for (int base = 0; base < wrap_count; base += 32) {
                int x = base + lane < wrap_count ? f[base + lane + 1] : 0;
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (base + lane < wrap_count) f[base + lane + 1] = carry + x;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) f[0] = 0;
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    auto wrap_of = [&](const int* f, int item) {  // the last wrap whose first item is <= item
        int lo = 0, hi = wrap_count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (f[mid] <= item) lo = mid; else hi = mid - 1;
        }
        return lo;
    };
    uint32_t* const warp_nodes = stack_nodes + (threadIdx.x >> 5) * kWarpStack;
    float* const warp_dists = stack_dists + (threadIdx.x >> 5) * kWarpStack;
    // ---- the listed long walks, a warp each ----
    {
        const int total = first_long[wrap_count];
        while (true) {
            int item = 0;
            if (lane == 0) item = atomicAdd(counter + 1, 1);
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= total) break;
            const int wi = wrap_of(first_long, item);
            const WrapDev& w = wraps[wi];
            const int cur = w.control->long_cur;
            const int v = w.long_list[cur * kLongCap + item - first_long[wi]];
            const float4 q32 = w.deformed32[v];
            const F3 q = {q32.x, q32.y, q32.z};
            const D3 q64 = load_d3(w.deformed, v);
            int overflow = 0;
            bool unfinished = false;
            long work = 0;
            int tri = nearest_triangle_group<32>(w, true, q, q64, w.corr_triangle[v], warp_nodes, warp_dists,
                                                 &overflow, &unfinished, &work);
            if (lane == 0) {
                if (unfinished) tri = nearest_triangle(w, q, q64, tri, &overflow);
                if (overflow) atomicOr(&w.control->error, kErrorTraversal);
                store_correspondence(w, w.control->level, v, tri);
                if (unfinished || work > kLongWalk) list_long_walk(w, 1 - cur, v);
            }
            __syncwarp();
        }
    }
    // ---- every other vertex, a group of lanes each ----
    const int total = first[wrap_count];
    auto others = [&](auto lanes) {
        constexpr int G = decltype(lanes)::value;
        constexpr int kGroups = 32 / G;
        const int group = lane / G;
        while (true) {
            int base = 0;
            if (lane == 0) base = atomicAdd(counter, kGroups);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= total) break;
            const int item = min(base + group, total - 1);
            const int wi = wrap_of(first, item);
            const WrapDev& w = wraps[wi];
            const int v = item - first[wi];
            const int cur = w.control->long_cur;
            const bool mine = base + group < total;
            const bool masked = w.mask && !w.mask[v];
            const bool on = mine && !masked && !w.long_flag[(long)cur * w.V + v];  // flagged: a warp's walk, above
            const float4 q32 = w.deformed32[v];
            const F3 q = {q32.x, q32.y, q32.z};
            const D3 q64 = load_d3(w.deformed, v);
            int overflow = 0;
            bool unfinished = false;
            long work = 0;
            int tri = nearest_triangle_group<G>(w, on, q, q64, w.corr_triangle[v],
                                                warp_nodes + group * (kWarpStack / kGroups),
                                                warp_dists + group * (kWarpStack / kGroups), &overflow, &unfinished,
                                                &work);
            if (lane % G == 0) {
                if (on) {
                    if (unfinished) tri = nearest_triangle(w, q, q64, tri, &overflow);
                    if (overflow) atomicOr(&w.control->error, kErrorTraversal);
                    store_correspondence(w, w.control->level, v, tri);
                    if (unfinished || work > kLongWalk) list_long_walk(w, 1 - cur, v);
                } else if (mine && masked) {
                    store_masked(w, v);
                }
            }
            __syncwarp();
        }
    };
    const int lanes = group_lanes(total, (long)gridDim.x * blockDim.x);
    if (lanes == 16) {
        others(std::integral_constant<int, 16>{});
    } else if (lanes == 8) {
        others(std::integral_constant<int, 8>{});
    } else {
        others(std::integral_constant<int, 4>{});
    }
}

// Stand-alone query over a prepared hierarchy (parity tests and the
// `closest_points` entry point): a group of G lanes per query.
template <int G>
__global__ void __launch_bounds__(128) k_closest_points(const WrapDev* __restrict__ wraps,
                                                       const double* __restrict__ queries, int count,
                                                       double* __restrict__ out_points,
                                                       double* __restrict__ out_normals,
                                                       double* __restrict__ out_distances,
                                                       int32_t* __restrict__ out_triangles,
                                                       int* __restrict__ overflow_flag) {
    __shared__ uint32_t stack_nodes[4 * kWarpStack];
    __shared__ float stack_dists[4 * kWarpStack];
    const WrapDev& w = wraps[0];
    const int group = threadIdx.x / G;
    const int i = blockIdx.x * (128 / G) + group;
    const bool on = i < count;
    const D3 q = on ? load_d3(queries, i) : D3{0.0, 0.0, 0.0};
    const F3 q32 = {__double2float_rn(q.x), __double2float_rn(q.y), __double2float_rn(q.z)};
    int overflow = 0;
    bool unfinished = false;
    long work = 0;
    constexpr int kStack = kWarpStack * G / 32;
    int tri = nearest_triangle_group<G>(w, on, q32, q, -1, stack_nodes + group * kStack, stack_dists + group * kStack,
                                        &overflow, &unfinished, &work);
    if (!on || threadIdx.x % G != 0) return;
    if (unfinished) tri = nearest_triangle(w, q32, q, tri, &overflow);
    if (overflow) atomicOr(overflow_flag, 1);
    D3 point = {0, 0, 0}, normal = {0, 0, 0};
    double distance = 0.0;
    if (tri >= 0) {
        const int32_t* f = w.tgt_faces + (long)tri * 3;
        double bary[3];
        point = closest_point_fp64(q, load_d3(w.tgt_points, f[0]), load_d3(w.tgt_points, f[1]),
                                   load_d3(w.tgt_points, f[2]), bary);
        const D3 d = vsub(point, q);
        distance = __dsqrt_rn(vdot(d, d));
        normal = vnormalized(vadd(vadd(vmul(load_d3(w.tgt_normals, f[0]), bary[0]),
                                       vmul(load_d3(w.tgt_normals, f[1]), bary[1])),
                                  vmul(load_d3(w.tgt_normals, f[2]), bary[2])));
    }
    store_d3(out_points, i, point);
    store_d3(out_normals, i, normal);
    out_distances[i] = distance;
    out_triangles[i] = tri;
}

// Blocks of 128 threads of `kernel` that fit on the current device at once.
template <typename Kernel>
static int resident_blocks(PerDevice<int>& of_device, Kernel kernel, size_t shared_bytes) {
    int device = 0;
    check(cudaGetDevice(&device), "device");
    return of_device.of(device, [&] {
        int sms = 0, per_sm = 0;
        check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "device");
        check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 128, shared_bytes), "occupancy");
        const int blocks = sms * (per_sm > 0 ? per_sm : 1);
        return blocks > 0 ? blocks : 1;
    });
}

void launch_query(const WrapDev* wraps, int wrap_count, cudaStream_t stream, int* counter) {
    // the warps' stacks, then two scans over the wraps (1024 at most)
    constexpr size_t kStackBytes = (sizeof(uint32_t) + sizeof(float)) * kWarpStack * 4;
    static PerDevice<int>& of_device = *new PerDevice<int>;
    const int resident = resident_blocks(of_device, k_query_queue, kStackBytes + 2 * sizeof(int) * 1025);
    cudaMemsetAsync(counter, 0, 2 * sizeof(int), stream);
    k_query_queue<<<resident, 128, kStackBytes + 2 * sizeof(int) * (wrap_count + 1), stream>>>(
        wraps, wrap_count, counter);
}

void launch_closest_points(const WrapDev* wrap, const double* queries, int count,
                           double* points, double* normals, double* distances, int32_t* triangles,
                           int* overflow, cudaStream_t stream) {
    static PerDevice<int>& of_device = *new PerDevice<int>;
    const long resident = 128L * resident_blocks(of_device, k_closest_points<8>, 0);
    auto launch = [&](auto kernel, int lanes) {
        kernel<<<blocks_for((long)count * lanes, 128), 128, 0, stream>>>(wrap, queries, count, points, normals, distances,
                                                                   triangles, overflow);
    };
    const int lanes = group_lanes(count, resident);
    if (lanes == 16) {
        launch(k_closest_points<16>, 16);
    } else if (lanes == 8) {
        launch(k_closest_points<8>, 8);
    } else {
        launch(k_closest_points<4>, 4);
    }
}

}  // namespace nricp_b200

namespace nricp_b200 {

namespace {

// Out-of-range face indices would make the centroid pass read outside the
// caller's vertex buffer; this pass only records that they exist.
__global__ void k_check_faces(const int32_t* __restrict__ faces, int count, int vertex_count,
                              int* __restrict__ flag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count * 3) return;
    const int v = faces[i];
    if (v < 0 || v >= vertex_count) atomicOr(flag, 1);
}

}  // namespace

size_t lbvh_export_scratch_bytes(int n) {
    const size_t pieces[] = {
        sizeof(float) * 3 * (size_t)n,            // centroids
        64,                                       // bounds, ordered
        sizeof(uint32_t) * (size_t)n,             // second key buffer
        sizeof(uint32_t) * (size_t)n,             // second value buffer
        radix_count_bytes(n),                     // digit counts
        256,                                      // validation flag
    };
    size_t total = 0;
    for (size_t bytes : pieces) total += (bytes + 255) & ~size_t(255);
    return total;
}

// The canonical arrays of the hierarchy (sorted codes, permutation, Karras
// children, centroid bounds) straight into caller-owned device buffers, with
// every intermediate in `scratch`.  The sort ping-pongs between the caller's
// code/permutation buffers and a scratch pair; with an even number of passes
// the result lands in the caller's.  Returns false when a face index is out of
// range (nothing past the check reads the vertices then).
bool lbvh_export_to_device(const double* points, int vertex_count, const int32_t* faces, int n,
                           void* scratch, uint32_t* codes, uint32_t* order, int32_t* left,
                           int32_t* right, float* bounds, cudaStream_t stream) {
    char* base = static_cast<char*>(scratch);
    auto carve = [&base](size_t bytes) {
        char* p = base;
        base += (bytes + 255) & ~size_t(255);
        return p;
    };
    float* centroids = reinterpret_cast<float*>(carve(sizeof(float) * 3 * n));
    uint32_t* ordered = reinterpret_cast<uint32_t*>(carve(64));
    uint32_t* keys[2] = {codes, reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * n))};
    uint32_t* values[2] = {order, reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * n))};
    uint32_t* counts = reinterpret_cast<uint32_t*>(carve(radix_count_bytes(n)));
    int* flag = reinterpret_cast<int*>(carve(256));

    // the array keeps the previous call's contents: clear what starts at zero
    check(cudaMemsetAsync(flag, 0, sizeof(int), stream), "hierarchy export: clearing the flag");
    k_check_faces<<<blocks_for((long)n * 3), kThreads, 0, stream>>>(faces, n, vertex_count, flag);
    check(cudaGetLastError(), "hierarchy export: face check");
    int host_flag = 0;
    check(cudaMemcpyAsync(&host_flag, flag, sizeof(int), cudaMemcpyDeviceToHost, stream),
          "hierarchy export: reading the flag");
    // the caller's stream is synchronised here, on every call
    check(cudaStreamSynchronize(stream), "hierarchy export: face check");
    if (host_flag) return false;

    // an even number of passes: the sorted arrays are back in the caller's buffers
    static_assert((kCodeBits + kRadixBits - 1) / kRadixBits % 2 == 0, "the result is in the first pair");
    sorted_codes(points, faces, n, centroids, ordered, bounds, keys, values, counts, stream);
    if (n > 1) k_karras<<<blocks_for(n - 1), kThreads, 0, stream>>>(codes, n, left, right, nullptr);
    return true;
}

}  // namespace nricp_b200
