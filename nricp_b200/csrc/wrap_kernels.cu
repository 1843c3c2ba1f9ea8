// The per-tick kernels of the device schedule.
//
// One tick advances every wrap of a batch by one unit of the schedule the
// reference's session runs (src/cuda/session.cu:404-576) -- a correspondence
// refresh, or one damped solve attempt with its candidate system -- and every
// kernel below serves all wraps at once: blockIdx.y is the wrap, and a wrap
// whose phase does not need a kernel leaves it immediately.  The decision
// kernel at the end of the tick is the only writer of the schedule's scalars,
// so the host never sits in the loop: it replays the tick (a CUDA graph) and
// polls one pinned flag.
//
// Reductions are fixed-order (per-block partials, then a fixed tree), so a
// wrap's result does not depend on which other wraps share its batch.
#include <cmath>

#include "async.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "per_device.hpp"
#include "solve_layout.hpp"

#include <cooperative_groups.h>

namespace nricp_b200 {

void check(cudaError_t status, const char* what);  // throws CudaError (session.cu)

namespace cg = cooperative_groups;

namespace {

int current_device() {
    int device = 0;
    check(cudaGetDevice(&device), "device");
    return device;
}

constexpr int kVertexThreads = 256;
constexpr int kNodeThreads = 256;   // 8 warps = 8 nodes per block
constexpr int kEdgeSums = 128;      // edges per partial sum of the smoothness energy
constexpr int kStatsThreads = 512;

// Which branch of a tick handles a wrap: part 0 every wrap (one chain), 1 the
// wraps that started the tick in a solve, 2 the others.  The phase at the
// tick's start decides, so a wrap that one branch's decision moves on is not
// picked up by the other branch in the same tick.
__device__ inline bool in_part(const WrapControl& c, int part) {
    return part == 0 || (part == 1) == (c.tick_phase == kPhaseSolve);
}
__device__ inline int blocks_of_dev(long n, int threads) { return (int)((n + threads - 1) / threads); }

// Most wraps of a batch are smaller than the largest, and in any tick only
// some of them have work for a given kernel; a grid sized for the largest wrap
// times the wraps launches mostly blocks that return at once.  Instead a
// kernel's work is a list of virtual blocks -- block x of wrap y, exactly the
// blocks the full grid would run to some effect -- which a grid that fits on
// the device walks in order.  Each virtual block does the same work, with
// the same reductions and the same partial slots, as that block of the full
// grid, so results do not change.  need(w) gives the virtual blocks of wrap w
// (0: none this tick); body(wrap index, x) runs one.  The launch gives
// (wrap_count + 1) ints of dynamic shared memory.  kShared: the body uses
// shared memory, so the block meets at a barrier between virtual blocks;
// bodies without it let each warp go on to the next virtual block at once.
template <bool kShared, typename Need, typename Body>
__device__ __forceinline__ void over_virtual_blocks(const WrapDev* __restrict__ wraps, int wrap_count, Need need,
                                                    Body body) {
    extern __shared__ int first[];  // each wrap's first virtual block
    for (int i = threadIdx.x; i < wrap_count; i += blockDim.x) first[i + 1] = need(wraps[i]);
    __syncthreads();
    if (threadIdx.x < 32) {  // inclusive scan by warp 0, 32 wraps at a time
        const int lane = threadIdx.x;
        int carry = 0;
        for (int base = 0; base < wrap_count; base += 32) {
            int x = base + lane < wrap_count ? first[base + lane + 1] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (base + lane < wrap_count) first[base + lane + 1] = carry + x;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) first[0] = 0;
    }
    __syncthreads();
    const int total = first[wrap_count];
    for (int vb = blockIdx.x; vb < total; vb += gridDim.x) {
        int lo = 0, hi = wrap_count - 1;  // the last wrap whose first block is <= vb
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first[mid] <= vb) lo = mid; else hi = mid - 1;
        }
        body(lo, vb - first[lo]);
        if (kShared) __syncthreads();  // shared memory of one virtual block before the next
    }
}

__device__ inline bool refresh_like(int phase) {
    return phase == kPhaseTransfer || phase == kPhaseRefresh || phase == kPhaseFinal;
}
// Which state buffer the kernels of this tick evaluate: the candidate for a
// solve attempt, the freshly transferred state at a level start, else the
// accepted one.
__device__ inline int eval_buffer(const WrapControl& c) {
    return (c.phase == kPhaseSolve || c.phase == kPhaseTransfer) ? 1 - c.state : c.state;
}
__device__ inline bool has_candidate(const WrapControl& c) {
    return c.phase != kPhaseSolve || c.pcg_ok;
}
// Whether this tick evaluates the energy (everything but the final query).
__device__ inline bool computes_energy(const WrapControl& c) {
    return (c.phase == kPhaseTransfer || c.phase == kPhaseRefresh || c.phase == kPhaseSolve) &&
           has_candidate(c);
}
// Whether this tick assembles a system.  Route C's translation-only matrix
// does not depend on the state, so it is assembled once per refresh.
__device__ inline bool assembles(const WrapControl& c) {
    if (c.phase == kPhaseTransfer || c.phase == kPhaseRefresh) return true;
    return c.phase == kPhaseSolve && c.route == 0 && c.pcg_ok;
}

// ---- FP64 with every operation rounded on its own (host-identical) --------
__device__ inline double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ inline double da(double a, double b) { return __dadd_rn(a, b); }
__device__ inline double ds(double a, double b) { return __dsub_rn(a, b); }
__device__ inline D3 rsub(D3 a, D3 b) { return {ds(a.x, b.x), ds(a.y, b.y), ds(a.z, b.z)}; }
__device__ inline D3 radd(D3 a, D3 b) { return {da(a.x, b.x), da(a.y, b.y), da(a.z, b.z)}; }
__device__ inline D3 rmul(D3 a, double s) { return {dm(a.x, s), dm(a.y, s), dm(a.z, s)}; }
__device__ inline double rdot(D3 a, D3 b) { return da(da(dm(a.x, b.x), dm(a.y, b.y)), dm(a.z, b.z)); }
__device__ inline D3 rcross(D3 a, D3 b) {
    return {ds(dm(a.y, b.z), dm(a.z, b.y)), ds(dm(a.z, b.x), dm(a.x, b.z)),
            ds(dm(a.x, b.y), dm(a.y, b.x))};
}
__device__ inline D3 rmat(const double* m, D3 v) {
    return {da(da(dm(m[0], v.x), dm(m[1], v.y)), dm(m[2], v.z)),
            da(da(dm(m[3], v.x), dm(m[4], v.y)), dm(m[5], v.z)),
            da(da(dm(m[6], v.x), dm(m[7], v.y)), dm(m[8], v.z))};
}

// ---- rotations (src/core/rotation.h, quaternion.h), FP64 -------------------
__device__ inline void mat_mul(const double* a, const double* b, double* out) {
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) {
            double sum = 0.0;
            for (int k = 0; k < 3; ++k) sum = da(sum, dm(a[r * 3 + k], b[k * 3 + c]));
            out[r * 3 + c] = sum;
        }
}
__device__ inline void skew(D3 w, double* m) {
    m[0] = 0.0; m[1] = -w.z; m[2] = w.y; m[3] = w.z; m[4] = 0.0; m[5] = -w.x;
    m[6] = -w.y; m[7] = w.x; m[8] = 0.0;
}
__device__ inline void exp_so3(D3 w, double* out) {  // rotation.h:29-47
    const double t2 = rdot(w, w);
    double h[9], h2[9];
    skew(w, h);
    mat_mul(h, h, h2);
    for (int i = 0; i < 9; ++i) out[i] = (i % 4 == 0) ? 1.0 : 0.0;
    if (t2 < 1e-24) {
        for (int i = 0; i < 9; ++i) out[i] = da(out[i], da(h[i], dm(0.5, h2[i])));
        return;
    }
    const double t = sqrt(t2);
    const double a = sin(t) / t;
    const double b = (1.0 - cos(t)) / t2;
    for (int i = 0; i < 9; ++i) out[i] = da(out[i], da(dm(a, h[i]), dm(b, h2[i])));
}
struct Quat { double w, x, y, z; };
__device__ inline Quat quat_from_matrix(const double* m) {  // quaternion.h:49-76
    const double trace = m[0] + m[4] + m[8];
    if (trace > 0.0) {
        const double s = sqrt(trace + 1.0) * 2.0;
        return {0.25 * s, (m[7] - m[5]) / s, (m[2] - m[6]) / s, (m[3] - m[1]) / s};
    }
    if (m[0] > m[4] && m[0] > m[8]) {
        const double s = sqrt(1.0 + m[0] - m[4] - m[8]) * 2.0;
        return {(m[7] - m[5]) / s, 0.25 * s, (m[1] + m[3]) / s, (m[2] + m[6]) / s};
    }
    if (m[4] > m[8]) {
        const double s = sqrt(1.0 + m[4] - m[0] - m[8]) * 2.0;
        return {(m[2] - m[6]) / s, (m[1] + m[3]) / s, 0.25 * s, (m[5] + m[7]) / s};
    }
    const double s = sqrt(1.0 + m[8] - m[0] - m[4]) * 2.0;
    return {(m[3] - m[1]) / s, (m[2] + m[6]) / s, (m[5] + m[7]) / s, 0.25 * s};
}
__device__ inline void matrix_from_quat(Quat q, double* m) {  // quaternion.h:78-94
    m[0] = 1.0 - 2.0 * (q.y * q.y + q.z * q.z);
    m[1] = 2.0 * (q.x * q.y - q.z * q.w);
    m[2] = 2.0 * (q.x * q.z + q.y * q.w);
    m[3] = 2.0 * (q.x * q.y + q.z * q.w);
    m[4] = 1.0 - 2.0 * (q.x * q.x + q.z * q.z);
    m[5] = 2.0 * (q.y * q.z - q.x * q.w);
    m[6] = 2.0 * (q.x * q.z - q.y * q.w);
    m[7] = 2.0 * (q.y * q.z + q.x * q.w);
    m[8] = 1.0 - 2.0 * (q.x * q.x + q.y * q.y);
}
__device__ inline D3 log_so3(const double* m) {  // rotation.h:51-63
    Quat q = quat_from_matrix(m);
    double len = sqrt(q.w * q.w + q.x * q.x + q.y * q.y + q.z * q.z);
    if (len > 0.0) { q.w /= len; q.x /= len; q.y /= len; q.z /= len; }
    else { q = {1.0, 0.0, 0.0, 0.0}; }
    if (q.w < 0.0) { q.w = -q.w; q.x = -q.x; q.y = -q.y; q.z = -q.z; }
    const double l = sqrt(q.x * q.x + q.y * q.y + q.z * q.z);
    if (l < 1e-12) return {0.0, 0.0, 0.0};
    const double angle = 2.0 * atan2(l, q.w);
    return {q.x * (angle / l), q.y * (angle / l), q.z * (angle / l)};
}
__device__ inline void left_jacobian_inverse(D3 w, double* out) {  // rotation.h:71-105
    const double t2 = dot(w, w);
    double h[9], h2[9];
    skew(w, h);
    mat_mul(h, h, h2);
    if (t2 < 1e-12) {
        for (int i = 0; i < 9; ++i)
            out[i] = ((i % 4 == 0) ? 1.0 : 0.0) - 0.5 * h[i] + (1.0 / 12.0) * h2[i];
        return;
    }
    const double t = sqrt(t2);
    if (t > 3.14159265358979323846 - 1e-6) {
        for (int i = 0; i < 9; ++i) out[i] = ((i % 4 == 0) ? 1.0 : 0.0) - 0.5 * h[i];
        return;
    }
    const double second = 1.0 / t2 - (1.0 + cos(t)) / (2.0 * t * sin(t));
    for (int i = 0; i < 9; ++i) out[i] = ((i % 4 == 0) ? 1.0 : 0.0) - 0.5 * h[i] + second * h2[i];
}

// ---- reductions ------------------------------------------------------------
template <typename T>
__device__ inline T warp_sum(T v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Warp sums of N values at once, by recursive halving: at lane distance
// o = 16, 8, .., 1 each lane keeps half of its values (the upper half when
// its lane bit o is set) and adds its partner's copy of that half.  Each
// total is formed by the same additions as `warp_sum` of that value (x + y
// and y + x round alike), so the bits are the same, with ~N shuffles instead
// of 5N.  Afterwards this lane holds the totals of values
// [first, first + count) in v[0 .. count).
template <int N, int O = 16, typename T, typename Add>
__device__ __forceinline__ void warp_sum_halving(T* v, int lane, int& first, int& count, Add add) {
    if constexpr (O >= 1) {
        constexpr int H = (N + 1) / 2;
        const bool upper = (lane & O) != 0;
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const T lo = v[i];
            const T hi = i + H < N ? v[i + H] : T(0);
            v[i] = add(upper ? hi : lo, __shfl_xor_sync(0xffffffffu, upper ? lo : hi, O));
        }
        if (upper) {
            first += H;
            count = count > H ? count - H : 0;
        } else {
            count = count < H ? count : H;
        }
        warp_sum_halving<H, O / 2>(v, lane, first, count, add);
    }
}
template <int N>
__device__ __forceinline__ void warp_sum_halving(float* v, int lane, int& first, int& count) {
    warp_sum_halving<N, 16>(v, lane, first, count, [](float a, float b) { return a + b; });
}
// Where warp_sum_halving leaves the totals, without the sums.
template <int N, int O = 16>
__device__ __forceinline__ void halving_place(int lane, int& first, int& count) {
    if constexpr (O >= 1) {
        constexpr int H = (N + 1) / 2;
        if (lane & O) {
            first += H;
            count = count > H ? count - H : 0;
        } else {
            count = count < H ? count : H;
        }
        halving_place<H, O / 2>(lane, first, count);
    }
}
// Block sums of N values in a fixed order, two barriers for all of them; the
// first warp's lanes hold the totals.  `scratch` is kThreadsT / 32 x N doubles.
template <int kThreadsT, int N>
__device__ inline void block_sums(double* v, double* scratch) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = 0; k < N; ++k) v[k] = warp_sum(v[k]);
    __syncthreads();
    if (lane == 0)
        for (int k = 0; k < N; ++k) scratch[warp * N + k] = v[k];
    __syncthreads();
    if (warp == 0)
        for (int k = 0; k < N; ++k) v[k] = warp_sum(lane < kThreadsT / 32 ? scratch[lane * N + k] : 0.0);
}

// ---- symmetric 6x6 accumulation in the upper triangle ----------------------
// d[k] for (r, c), r <= c, row-major over the upper triangle.
__device__ inline int tri_index(int r, int c) { return r * 6 - r * (r - 1) / 2 + (c - r); }

// D += coef * [ |a|^2 I - a a^T, [a]x ; [a]x^T, I ]  (sum over the three rows
// of an offset residual whose node-local offset is `a`)
__device__ inline void add_offset_block(float* d, F3 a, float coef) {
    const float aa = dot(a, a);
    const float av[3] = {a.x, a.y, a.z};
    for (int r = 0; r < 3; ++r)
        for (int c = r; c < 3; ++c) d[tri_index(r, c)] += coef * ((r == c ? aa : 0.0f) - av[r] * av[c]);
    // [a]x = [[0,-az,ay],[az,0,-ax],[-ay,ax,0]] in rows 0-2, columns 3-5
    d[tri_index(0, 4)] += -coef * a.z; d[tri_index(0, 5)] += coef * a.y;
    d[tri_index(1, 3)] += coef * a.z;  d[tri_index(1, 5)] += -coef * a.x;
    d[tri_index(2, 3)] += -coef * a.y; d[tri_index(2, 4)] += coef * a.x;
    d[tri_index(3, 3)] += coef; d[tri_index(4, 4)] += coef; d[tri_index(5, 5)] += coef;
}
// D += coef * u u^T for a 6-vector u
__device__ inline void add_rank_one(float* d, const float* u, float coef) {
    for (int r = 0; r < 6; ++r)
        for (int c = r; c < 6; ++c) d[tri_index(r, c)] += coef * u[r] * u[c];
}

}  // namespace

// ---------------------------------------------------------------------------
// statistics (deform_ops.cu:135-182 / correspondence.cpp:82-94)
// ---------------------------------------------------------------------------
constexpr int kStatsBins = 2048;
constexpr int kStatsKept = 2048;
// The statistics pass at a tick's start (final_mode 0) also takes the tick's
// phase snapshot.
__global__ void __launch_bounds__(kStatsThreads) k_stats(const WrapDev* __restrict__ wraps, int final_mode) {
    const WrapDev& w = wraps[blockIdx.y * gridDim.x + blockIdx.x];
    const WrapControl c = *w.control;
    if (!final_mode && threadIdx.x == 0) {
        w.control->tick_phase = c.phase;
        *w.solve_arrivals = 0;
    }
    CorrStats* target = nullptr;
    int level = -1;
    if (final_mode) {
        if (c.tick_phase != kPhaseFinal || c.phase != kPhaseFinal) return;
        target = w.final_stats;
    } else {
        if (c.stats_pending == 0) return;
        level = c.stats_pending - 1;
        target = w.level_stats + level;
    }
    constexpr int kWarps = kStatsThreads / 32;
    __shared__ double scratch[kWarps * 7];
    __shared__ int hist[kStatsBins];
    __shared__ unsigned long long kept[kStatsKept];
    __shared__ double totals_s[6];
    __shared__ unsigned long long low_s, high_s, maximum_s;
    __shared__ int warp_count[kWarps], bin_s, rank_s, count_s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // counts per outcome, and the accepted distances' sum and extremes (a
    // distance is never negative, so its bits order like the distance)
    double sums[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    unsigned long long low = ~0ull, high = 0ull;
    double maximum = 0.0;
#pragma unroll 4
    for (int v = threadIdx.x; v < w.V; v += kStatsThreads) {
        const int code = w.corr_code[v];
        const double d = w.corr_distance[v];
        for (int k = 0; k < 5; ++k)
            if (code == k) sums[k] += 1.0;
        if (code == 0) {
            sums[5] += d;
            const unsigned long long bits = (unsigned long long)__double_as_longlong(d);
            low = min(low, bits);
            high = max(high, bits);
            maximum = fmax(maximum, d);
        }
    }
    if (threadIdx.x == 0) {
        low_s = ~0ull;
        high_s = maximum_s = 0ull;
    }
    block_sums<kStatsThreads, 6>(sums, scratch);
    for (int o = 16; o > 0; o >>= 1) {
        low = min(low, __shfl_xor_sync(0xffffffffu, low, o));
        high = max(high, __shfl_xor_sync(0xffffffffu, high, o));
        maximum = fmax(maximum, __shfl_xor_sync(0xffffffffu, maximum, o));
    }
    if (lane == 0) {
        atomicMin(&low_s, low);
        atomicMax(&high_s, high);
        atomicMax(&maximum_s, (unsigned long long)__double_as_longlong(maximum));
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < 6; ++k) totals_s[k] = sums[k];
    __syncthreads();
    int totals[5];
    for (int k = 0; k < 5; ++k) totals[k] = (int)totals_s[k];
    const double total_sum = totals_s[5];
    const int accepted = totals[0];
    const double total_max = __longlong_as_double((long long)maximum_s);
    // p95 = the floor(0.95 (n - 1))-th smallest accepted distance: the range
    // of the bits that holds it, split into 2,048 equal bins and narrowed to
    // the rank's bin until a bin is one value; once a bin's distances fit in
    // shared memory they are kept there.  (Eight passes of 8 bits over the
    // vertices, the first two counting into a few bins only, took 750 us for
    // 100,000 vertices.)
    double p95 = 0.0;
    if (accepted > 0) {
        double pi = 0.95 * (double)(accepted - 1);
        if (pi > (double)(accepted - 1)) pi = (double)(accepted - 1);
        int rank = (int)pi, in_shared = -1;
        unsigned long long from = low_s, span = high_s - low_s;  // the value lies in [from, from + span]
        while (span > 0) {
            const int bits = 64 - __clzll((long long)span);
            const int shift = bits > 11 ? bits - 11 : 0;
            for (int i = threadIdx.x; i < kStatsBins; i += kStatsThreads) hist[i] = 0;
            __syncthreads();
            // every accepted distance's place in the range, or every kept one's
            auto each = [&](auto&& body) {
                if (in_shared >= 0) {
                    for (int i = threadIdx.x; i < in_shared; i += kStatsThreads) body(kept[i] - from, kept[i]);
                } else {
#pragma unroll 4
                    for (int v = threadIdx.x; v < w.V; v += kStatsThreads) {
                        const int code = w.corr_code[v];
                        const unsigned long long b = (unsigned long long)__double_as_longlong(w.corr_distance[v]);
                        if (code == 0 && b >= from) body(b - from, b);
                    }
                }
            };
            each([&](unsigned long long at, unsigned long long) {
                if (at <= span) atomicAdd(&hist[at >> shift], 1);
            });
            __syncthreads();
            // the bin of the rank: each thread four bins, a scan over the threads
            constexpr int kPer = kStatsBins / kStatsThreads;
            int mine = 0;
            for (int k = 0; k < kPer; ++k) mine += hist[threadIdx.x * kPer + k];
            int before = mine;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += y;
            }
            if (lane == 31) warp_count[warp] = before;
            __syncthreads();
            before -= mine;
            for (int i = 0; i < warp; ++i) before += warp_count[i];
            if (rank >= before && rank < before + mine) {  // one thread's
                int at = rank - before, k = 0;
                while (at >= hist[threadIdx.x * kPer + k]) at -= hist[threadIdx.x * kPer + k++];
                bin_s = threadIdx.x * kPer + k;
                rank_s = at;
                count_s = 0;
            }
            __syncthreads();
            const unsigned long long next = from + ((unsigned long long)bin_s << shift);
            const unsigned long long width = (1ull << shift) - 1;  // the bin's last value, from its first
            const int there = hist[bin_s];
            if (width > 0 && in_shared < 0 && there <= kStatsKept) {
                each([&](unsigned long long, unsigned long long b) {
                    if (b >= next && b - next <= width) kept[atomicAdd(&count_s, 1)] = b;
                });
                in_shared = there;
            }
            rank = rank_s;
            from = next;
            span = width;
            __syncthreads();
        }
        p95 = __longlong_as_double((long long)from);
    }
    if (threadIdx.x == 0) {
        CorrStats s;
        s.total = totals[0] + totals[1] + totals[2] + totals[3] + totals[4];
        s.accepted = accepted;
        s.rejected_distance = totals[1];
        s.rejected_normal = totals[2];
        s.rejected_slope = totals[3];
        s.rejected_masked = totals[4];
        s.mean = accepted > 0 ? total_sum / accepted : 0.0;
        s.p95 = p95;
        s.max = accepted > 0 ? total_max : 0.0;
        *target = s;
        if (!final_mode) {
            w.records[level].correspondence_mean = s.mean;
            w.control->last_corr_mean = s.mean;
            w.control->stats_pending = 0;
        }
    }
}

// ---------------------------------------------------------------------------
// node prologue: level warm start (deformation.cpp:141-203) and FP32 copies
// ---------------------------------------------------------------------------
__device__ __forceinline__ void k_prologue_body(const WrapDev& w, int part, int bx) {
    const WrapControl c = *w.control;
    if (!in_part(c, part)) return;
    if (!refresh_like(c.phase)) return;
    const LevelDev& L = w.levels[c.level];
    const int n = bx * blockDim.x + threadIdx.x;
    if (n >= L.node_count) return;
    double R[9];
    if (c.phase == kPhaseTransfer) {
        const LevelDev& from = w.levels[c.level - 1];
        const double* src_rot = w.rot[c.state];
        const double* src_trans = w.trans[c.state];
        const int count = L.transfer_counts[n];
        const int* nodes = L.transfer_nodes + n * 4;
        const double* weights = L.transfer_weights + n * 4;
        D3 t = {0.0, 0.0, 0.0};
        if (count > 0) {
            int heaviest = nodes[0];
            double hw = weights[0];
            for (int s = 1; s < count; ++s)
                if (weights[s] > hw) { hw = weights[s]; heaviest = nodes[s]; }
            const Quat ref = quat_from_matrix(src_rot + heaviest * 9);
            Quat b = {0.0, 0.0, 0.0, 0.0};
            D3 position = {0.0, 0.0, 0.0};
            const D3 g = load_d3(L.rest, n);
            for (int s = 0; s < count; ++s) {
                const int src = nodes[s];
                const double wt = weights[s];
                Quat q = quat_from_matrix(src_rot + src * 9);
                if (q.w * ref.w + q.x * ref.x + q.y * ref.y + q.z * ref.z < 0.0) {
                    q.w = -q.w; q.x = -q.x; q.y = -q.y; q.z = -q.z;
                }
                b.w += q.w * wt; b.x += q.x * wt; b.y += q.y * wt; b.z += q.z * wt;
                const D3 gs = load_d3(from.rest, src);
                const D3 applied = radd(radd(rmat(src_rot + src * 9, rsub(g, gs)), gs),
                                        load_d3(src_trans, src));
                position = radd(position, rmul(applied, wt));
            }
            const double len = sqrt(b.w * b.w + b.x * b.x + b.y * b.y + b.z * b.z);
            if (len > 1e-8) {
                const Quat nb = {b.w / len, b.x / len, b.y / len, b.z / len};
                matrix_from_quat(nb, R);
            } else {
                matrix_from_quat(ref, R);
            }
            t = rsub(position, g);
        } else {
            for (int i = 0; i < 9; ++i) R[i] = (i % 4 == 0) ? 1.0 : 0.0;
        }
        double* dst = w.rot[1 - c.state] + n * 9;
        for (int i = 0; i < 9; ++i) dst[i] = R[i];
        store_d3(w.trans[1 - c.state], n, t);
    } else {
        const double* src = w.rot[c.state] + n * 9;
        for (int i = 0; i < 9; ++i) R[i] = src[i];
    }
    for (int i = 0; i < 9; ++i) w.rot32[n * 9 + i] = (float)R[i];
}

__global__ void k_prologue(const WrapDev* __restrict__ wraps, int wrap_count, int part) {
    over_virtual_blocks<false>(
        wraps, wrap_count,
        [&](const WrapDev& w) {
            const WrapControl c = *w.control;
            return in_part(c, part) ? (refresh_like(c.phase) ? blocks_of_dev(w.levels[c.level].node_count, 128) : 0) : 0;
        },
        [&](int wi, int bx) { k_prologue_body(wraps[wi], part, bx); });
}

// ---------------------------------------------------------------------------
// route C: Horn's closed-form rotation (local_global.cu:188-302), FP64
// ---------------------------------------------------------------------------
__device__ inline void horn_rotation(const double* S, double* R) {
    const double sxx = S[0], sxy = S[1], sxz = S[2], syx = S[3], syy = S[4], syz = S[5];
    const double szx = S[6], szy = S[7], szz = S[8];
    double a[4][4];
    a[0][0] = sxx + syy + szz; a[0][1] = syz - szy; a[0][2] = szx - sxz; a[0][3] = sxy - syx;
    a[1][1] = sxx - syy - szz; a[1][2] = sxy + syx; a[1][3] = szx + sxz;
    a[2][2] = -sxx + syy - szz; a[2][3] = syz + szy;
    a[3][3] = -sxx - syy + szz;
    for (int r = 1; r < 4; ++r)
        for (int c = 0; c < r; ++c) a[r][c] = a[c][r];
    double v[4][4];
    for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c) v[r][c] = r == c ? 1.0 : 0.0;
    for (int sweep = 0; sweep < 50; ++sweep) {
        double off = 0.0, diag = 0.0;
        for (int r = 0; r < 4; ++r) {
            diag += a[r][r] * a[r][r];
            for (int c = r + 1; c < 4; ++c) off += a[r][c] * a[r][c];
        }
        if (off <= 1e-30 * diag || off == 0.0) break;
        for (int p = 0; p < 3; ++p)
            for (int q = p + 1; q < 4; ++q) {
                if (a[p][q] == 0.0) continue;
                const double theta = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
                const double sign = theta >= 0.0 ? 1.0 : -1.0;
                const double t = sign / (fabs(theta) + sqrt(theta * theta + 1.0));
                const double cs = 1.0 / sqrt(t * t + 1.0);
                const double sn = t * cs;
                for (int k = 0; k < 4; ++k) {
                    const double f = a[k][p], s2 = a[k][q];
                    a[k][p] = cs * f - sn * s2; a[k][q] = sn * f + cs * s2;
                }
                for (int k = 0; k < 4; ++k) {
                    const double f = a[p][k], s2 = a[q][k];
                    a[p][k] = cs * f - sn * s2; a[q][k] = sn * f + cs * s2;
                }
                for (int k = 0; k < 4; ++k) {
                    const double f = v[k][p], s2 = v[k][q];
                    v[k][p] = cs * f - sn * s2; v[k][q] = sn * f + cs * s2;
                }
            }
    }
    int best = 0;
    for (int i = 1; i < 4; ++i)
        if (a[i][i] > a[best][best]) best = i;
    const double qw = v[0][best], qx = v[1][best], qy = v[2][best], qz = v[3][best];
    const double len = sqrt(qw * qw + qx * qx + qy * qy + qz * qz);
    if (!(len > 0.0)) {
        for (int i = 0; i < 9; ++i) R[i] = (i % 4 == 0) ? 1.0 : 0.0;
        return;
    }
    const double w_ = qw / len, x = qx / len, y = qy / len, z = qz / len;
    R[0] = w_ * w_ + x * x - y * y - z * z; R[1] = 2.0 * (x * y - w_ * z); R[2] = 2.0 * (x * z + w_ * y);
    R[3] = 2.0 * (x * y + w_ * z); R[4] = w_ * w_ - x * x + y * y - z * z; R[5] = 2.0 * (y * z - w_ * x);
    R[6] = 2.0 * (x * z - w_ * y); R[7] = 2.0 * (y * z + w_ * x); R[8] = w_ * w_ - x * x - y * y + z * z;
}

constexpr double kRotationRelaxation = 0.2;  // local_global.cu:18

// The weighted rigid fit of point pairs (fit_rigid, deformation.cpp:86-139):
// weights clamped at zero, weighted centroids, the covariance
// sum w (p - cp)(q - cq)^T, the proper rotation that best maps the sources
// onto the targets, and t = cq - R cp.  The reference takes the rotation
// from an SVD with the reflection corrected; Horn's quaternion (the top
// eigenvector of the 4x4 matrix built from the covariance, Jacobi in FP64)
// is the same rotation.  One block, FP64 sums in a fixed order.
constexpr int kRigidThreads = 1024;
__global__ void __launch_bounds__(kRigidThreads) k_fit_rigid(const double* __restrict__ src,
                                                            const double* __restrict__ dst,
                                                            const double* __restrict__ weights, int n,
                                                            double* __restrict__ out) {
    __shared__ double scratch[kRigidThreads / 32 * 9];
    __shared__ double total[9];
    double sums[7] = {0, 0, 0, 0, 0, 0, 0};  // w, w p, w q
    for (int i = threadIdx.x; i < n; i += kRigidThreads) {
        const double w = fmax(0.0, weights[i]);
        sums[0] += w;
        for (int k = 0; k < 3; ++k) {
            sums[1 + k] += src[(long)i * 3 + k] * w;
            sums[4 + k] += dst[(long)i * 3 + k] * w;
        }
    }
    block_sums<kRigidThreads, 7>(sums, scratch);
    if (threadIdx.x == 0)
        for (int k = 0; k < 7; ++k) total[k] = sums[k];
    __syncthreads();
    double R[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    if (!(total[0] > 0.0)) {
        if (threadIdx.x == 0)
            for (int k = 0; k < 12; ++k) out[k] = k < 9 ? R[k] : 0.0;
        return;
    }
    const double cp[3] = {total[1] / total[0], total[2] / total[0], total[3] / total[0]};
    const double cq[3] = {total[4] / total[0], total[5] / total[0], total[6] / total[0]};
    double S[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = threadIdx.x; i < n; i += kRigidThreads) {
        const double w = fmax(0.0, weights[i]);
        if (w == 0.0) continue;
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q) S[r * 3 + q] += w * (src[(long)i * 3 + r] - cp[r]) * (dst[(long)i * 3 + q] - cq[q]);
    }
    block_sums<kRigidThreads, 9>(S, scratch);
    if (threadIdx.x == 0) {
        horn_rotation(S, R);
        for (int k = 0; k < 9; ++k) out[k] = R[k];
        for (int r = 0; r < 3; ++r) out[9 + r] = cq[r] - (R[r * 3] * cp[0] + R[r * 3 + 1] * cp[1] + R[r * 3 + 2] * cp[2]);
    }
}

// Warp per node: the correlation of the influences that mention the node
// (bound vertices' data and landmark rows, edges it is the first endpoint of),
// Horn's rotation, and the under-relaxed update into the candidate buffer.
__device__ __forceinline__ void k_c_fit_body(const WrapDev& w, int part, int bx) {
    const WrapControl c = *w.control;
    if (!in_part(c, part)) return;
    if (c.phase != kPhaseSolve || c.route != 1) return;
    const LevelDev& L = w.levels[c.level];
    const int node = (bx * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (node >= L.node_count) return;
    const double* wt = w.weights[c.level];
    const double data_weight = wt[0] + wt[1];  // local_global.cu:546
    const double* T = w.trans[c.state];
    const D3 g = load_d3(L.rest, node);
    const D3 tn = load_d3(T, node);
    double S[9];
    for (int i = 0; i < 9; ++i) S[i] = 0.0;
    // the lane's first edge, read while its first binding is on its way
    const int edge_first = L.node_edge_begin[node] + lane, edge_end = L.node_edge_begin[node + 1];
    D3 edge_src, edge_dst;
    auto load_edge = [&](int i) {  // false: the node is the edge's second
        const int e = L.node_edge_list[i];
        const int a = L.edges[e * 2], b = L.edges[e * 2 + 1];
        if (a != node) return false;
        const D3 gb = load_d3(L.rest, b);
        edge_src = gb - g;
        edge_dst = gb + load_d3(T, b) - g - tn;
        return true;
    };
    const bool near = edge_first < edge_end && load_edge(edge_first);
    for (int i = L.gather_begin[node] + lane; i < L.gather_begin[node + 1]; i += 32) {
        const int entry = L.gather_entry[i];
        const int v = entry / kMaxSlots;
        const double own = L.bind_weights[entry];
        const D3 src = load_d3(w.tpl, v) - g;
        const D3 point = load_d3(w.corr_point, v);
        const double robust = w.robust[v];
        if (w.corr_code[v] == 0) {
            const D3 dst = point - g - tn;
            const double s = data_weight * robust * own;
            const double xs[3] = {src.x, src.y, src.z}, ys[3] = {dst.x, dst.y, dst.z};
            for (int r = 0; r < 3; ++r)
                for (int q = 0; q < 3; ++q) S[r * 3 + q] += s * xs[r] * ys[q];
        }
        if (wt[4] > 0.0 && w.lm_flag[v]) {
            const D3 dst = load_d3(w.lm_target, v) - g - tn;
            const double s = wt[4] * own;
            const double xs[3] = {src.x, src.y, src.z}, ys[3] = {dst.x, dst.y, dst.z};
            for (int r = 0; r < 3; ++r)
                for (int q = 0; q < 3; ++q) S[r * 3 + q] += s * xs[r] * ys[q];
        }
    }
    auto add_edge = [&] {
        const double xs[3] = {edge_src.x, edge_src.y, edge_src.z}, ys[3] = {edge_dst.x, edge_dst.y, edge_dst.z};
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q) S[r * 3 + q] += wt[2] * xs[r] * ys[q];
    };
    if (near) add_edge();
    for (int i = edge_first + 32; i < edge_end; i += 32)
        if (load_edge(i)) add_edge();
    for (int i = 0; i < 9; ++i) S[i] = warp_sum(S[i]);
    if (lane == 0) {
        double fit[9], cur[9], curT[9], rel[9], step[9], out[9];
        horn_rotation(S, fit);
        for (int i = 0; i < 9; ++i) cur[i] = w.rot[c.state][node * 9 + i];
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q) curT[r * 3 + q] = cur[q * 3 + r];
        mat_mul(fit, curT, rel);
        const D3 omega = log_so3(rel);
        exp_so3(omega * kRotationRelaxation, step);
        mat_mul(step, cur, out);
        for (int i = 0; i < 9; ++i) w.rot[1 - c.state][node * 9 + i] = out[i];
        store_d3(w.trans[1 - c.state], node, tn);
    }
}

__global__ void k_c_fit(const WrapDev* __restrict__ wraps, int wrap_count, int part) {
    over_virtual_blocks<false>(
        wraps, wrap_count,
        [&](const WrapDev& w) {
            const WrapControl c = *w.control;
            return in_part(c, part) ? ((c.phase == kPhaseSolve && c.route == 1) ? blocks_of_dev(w.levels[c.level].node_count * 32, kNodeThreads) : 0) : 0;
        },
        [&](int wi, int bx) { k_c_fit_body(wraps[wi], part, bx); });
}

// Every vertex deformed by the fitted rotations, once for the right-hand side
// that follows (the candidate's evaluation overwrites it).  The nodes' warps
// did this for each binding again: up to eight dependent reads of a rotation
// per entry.  8k vertices, 130 ticks: a step 23.8 -> 22.2 ms, with the fit's and
// this kernel's first edges read beside the bindings.
__device__ __forceinline__ void k_c_deform_body(const WrapDev& w, int part, int bx) {
    const WrapControl c = *w.control;
    if (!in_part(c, part)) return;
    if (c.phase != kPhaseSolve || c.route != 1) return;
    const LevelDev& L = w.levels[c.level];
    const int v = bx * blockDim.x + threadIdx.x;
    if (v >= w.V) return;
    const double* Rc = w.rot[1 - c.state];
    const double* Tc = w.trans[1 - c.state];
    const D3 p = load_d3(w.tpl, v);
    D3 deformed = {0.0, 0.0, 0.0};
    const int count = L.bind_counts[v];
    for (int s = 0; s < count; ++s) {
        const int j = L.bind_nodes[v * kMaxSlots + s];
        const double ws = L.bind_weights[v * kMaxSlots + s];
        const D3 gj = load_d3(L.rest, j);
        deformed = deformed + (mul3(Rc + j * 9, p - gj) + gj + load_d3(Tc, j)) * ws;
    }
    store_d3(w.deformed, v, deformed);
}

__global__ void __launch_bounds__(kVertexThreads) k_c_deform(const WrapDev* __restrict__ wraps, int wrap_count, int part) {
    over_virtual_blocks<false>(
        wraps, wrap_count,
        [&](const WrapDev& w) {
            const WrapControl c = *w.control;
            return in_part(c, part) && c.phase == kPhaseSolve && c.route == 1 ? blocks_of_dev(w.V, kVertexThreads) : 0;
        },
        [&](int wi, int bx) { k_c_deform_body(wraps[wi], part, bx); });
}

// Warp per node: the translation-only right-hand side with the fitted
// rotations (local_global.cu:317-438); the rotation half is exactly zero.
__device__ __forceinline__ void k_c_rhs_body(const WrapDev& w, int part, int bx) {
    const WrapControl c = *w.control;
    if (!in_part(c, part)) return;
    if (c.phase != kPhaseSolve || c.route != 1) return;
    const LevelDev& L = w.levels[c.level];
    const int node = (bx * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (node >= L.node_count) return;
    const double* wt = w.weights[c.level];
    const double* Rc = w.rot[1 - c.state];
    const double* Tc = w.trans[1 - c.state];
    double local[3] = {0.0, 0.0, 0.0};
    // the lane's first edge, read while its first binding is on its way
    const int edge_first = L.node_edge_begin[node] + lane, edge_end = L.node_edge_begin[node + 1];
    double sign = 0.0;
    auto edge_difference = [&](int i) {
        const int e = L.node_edge_list[i];
        const int a = L.edges[e * 2], b = L.edges[e * 2 + 1];
        const D3 ga = load_d3(L.rest, a), gb = load_d3(L.rest, b);
        sign = a == node ? 1.0 : -1.0;
        return mul3(Rc + a * 9, gb - ga) + ga + load_d3(Tc, a) - gb - load_d3(Tc, b);
    };
    D3 diff = {0.0, 0.0, 0.0};
    if (edge_first < edge_end) diff = edge_difference(edge_first);
    for (int i = L.gather_begin[node] + lane; i < L.gather_begin[node + 1]; i += 32) {
        const int entry = L.gather_entry[i];
        const int v = entry / kMaxSlots;
        const double own = L.bind_weights[entry];
        const D3 deformed = load_d3(w.deformed, v);
        const D3 point = load_d3(w.corr_point, v);
        const D3 n = load_d3(w.corr_normal, v);
        const double u = w.robust[v];
        if (w.corr_code[v] == 0) {
            const D3 off = deformed - point;
            if (wt[0] > 0.0) {
                const double s = wt[0] * u * own;
                local[0] -= s * off.x; local[1] -= s * off.y; local[2] -= s * off.z;
            }
            if (wt[1] > 0.0) {
                const double s = wt[1] * u * own * dot(n, off);
                local[0] -= s * n.x; local[1] -= s * n.y; local[2] -= s * n.z;
            }
        }
        if (wt[4] > 0.0 && w.lm_flag[v]) {
            const D3 o = deformed - load_d3(w.lm_target, v);
            const double s = wt[4] * own;
            local[0] -= s * o.x; local[1] -= s * o.y; local[2] -= s * o.z;
        }
    }
    for (int i = edge_first; i < edge_end; i += 32) {
        if (i != edge_first) diff = edge_difference(i);
        local[0] -= sign * wt[2] * diff.x;
        local[1] -= sign * wt[2] * diff.y;
        local[2] -= sign * wt[2] * diff.z;
    }
    for (int i = 0; i < 3; ++i) local[i] = warp_sum(local[i]);
    if (lane == 0) {
        const D3 t = load_d3(Tc, node);
        float* r = w.rhs[c.system] + node * 6;
        r[0] = r[1] = r[2] = 0.0f;
        r[3] = (float)(local[0] - wt[3] * t.x);
        r[4] = (float)(local[1] - wt[3] * t.y);
        r[5] = (float)(local[2] - wt[3] * t.z);
    }
}

__global__ void k_c_rhs(const WrapDev* __restrict__ wraps, int wrap_count, int part) {
    over_virtual_blocks<false>(
        wraps, wrap_count,
        [&](const WrapDev& w) {
            const WrapControl c = *w.control;
            return in_part(c, part) ? ((c.phase == kPhaseSolve && c.route == 1) ? blocks_of_dev(w.levels[c.level].node_count * 32, kNodeThreads) : 0) : 0;
        },
        [&](int wi, int bx) { k_c_rhs_body(wraps[wi], part, bx); });
}

// ---------------------------------------------------------------------------
// the damped solve: block-Jacobi PCG by a cluster of CTAs per wrap, or by the whole
// device (pcg_solver.cu:15-241)
// FP32 blocks and matvec, FP64 solution / residual / dots.
// ---------------------------------------------------------------------------
__device__ inline bool cholesky6(float* a) {
    for (int r = 0; r < 6; ++r)
        for (int c = 0; c <= r; ++c) {
            float sum = a[r * 6 + c];
            for (int k = 0; k < c; ++k) sum -= a[r * 6 + k] * a[c * 6 + k];
            if (r == c) {
                if (!(sum > 0.0f)) return false;
                a[r * 6 + c] = sqrtf(sum);
            } else {
                a[r * 6 + c] = sum / a[c * 6 + c];
            }
        }
    return true;
}

// The solve's reductions -- the dot products, the residual norm, the Krylov
// scalars and the x and r vectors -- are FP64.  A build with
// NRICP_FP32_REDUCTIONS defined rounds every one of those operations to FP32
// instead (each FP64 result of a sum or product of FP32 values rounded to
// FP32 is the correctly rounded FP32 result): a variant for measuring what
// the FP64 reductions buy, never the shipped library.
#ifdef NRICP_FP32_REDUCTIONS
__device__ __forceinline__ double rnd(double x) { return (double)__double2float_rn(x); }
#else
__device__ __forceinline__ double rnd(double x) { return x; }
#endif
__device__ __forceinline__ double warp_sum_rnd(double v) {
    for (int o = 16; o > 0; o >>= 1) v = rnd(v + __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// Inverse of a 6x6 SPD block from its Cholesky factor L (lower): L^-T L^-1.
__device__ inline void cholesky_inverse6(const float* l, float* inv) {
    float li[36];
    for (int i = 0; i < 36; ++i) li[i] = 0.0f;
    for (int c = 0; c < 6; ++c) {
        li[c * 6 + c] = 1.0f / l[c * 6 + c];
        for (int r = c + 1; r < 6; ++r) {
            float s = 0.0f;
            for (int k = c; k < r; ++k) s -= l[r * 6 + k] * li[k * 6 + c];
            li[r * 6 + c] = s / l[r * 6 + r];
        }
    }
    for (int r = 0; r < 6; ++r)
        for (int q = 0; q < 6; ++q) {
            float s = 0.0f;
            for (int k = r > q ? r : q; k < 6; ++k) s += li[k * 6 + r] * li[k * 6 + q];
            inv[r * 6 + q] = s;
        }
}

// Rows 2p and 2p + 1 of a 6x6 block (twelve floats in three float4) times a
// node's six values.  The order of the operations is spelt out, so that every
// placement gives the same bits: of the first two products, a diagonal block's
// second is fused onto its first, an off-diagonal block's first onto its
// second; the other four follow left to right.
struct RowPair { float a, b; };
template <bool kDiagonal>
__device__ __forceinline__ float row_dot(float x0, float x1, float x2, float x3, float x4, float x5, float2 u0,
                                         float2 u1, float2 u2) {
    float y = kDiagonal ? __fmaf_rn(x1, u0.y, __fmul_rn(x0, u0.x)) : __fmaf_rn(x0, u0.x, __fmul_rn(x1, u0.y));
    y = __fmaf_rn(x2, u1.x, y);
    y = __fmaf_rn(x3, u1.y, y);
    y = __fmaf_rn(x4, u2.x, y);
    return __fmaf_rn(x5, u2.y, y);
}
template <bool kDiagonal>
__device__ __forceinline__ RowPair row_pair_dot(float4 b0, float4 b1, float4 b2, const float* u) {
    const float2* v = reinterpret_cast<const float2*>(u);
    const float2 u0 = v[0], u1 = v[1], u2 = v[2];
    return {row_dot<kDiagonal>(b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, u0, u1, u2),
            row_dot<kDiagonal>(b1.z, b1.w, b2.x, b2.y, b2.z, b2.w, u0, u1, u2)};
}

// Sixteen bytes from global memory (past the L1) to shared memory, and the wait
// for all that the thread has under way.
__device__ __forceinline__ void copy_16_async(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(shared_address(dst)),
                 "l"(__cvta_generic_to_global(src))
                 : "memory");
}
__device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One thread's part of a meeting of a cooperative grid's CTAs: counts its CTA
// in and waits, at most `polls` times, until `target` have come.
__device__ __forceinline__ bool grid_arrive_and_wait(unsigned* arrivals, unsigned target, int polls) {
    // the release covers what the CTA's threads wrote before the block barrier;
    // the polls are plain, and one fence after the last orders what follows
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrivals) : "memory");
    for (int i = 0; i < polls; ++i) {
        unsigned seen;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrivals) : "memory");
        if (seen >= target) {
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            return true;
        }
    }
    return false;
}

// A few steps of an octet's blocks from global memory, in registers.
constexpr int kStepsAhead = 4;
struct StepBlocks {
    float4 b[kStepsAhead][3];
    int node[kStepsAhead];
};

// The damped solve (pcg_solver.cu:15-241): (A + lambda diag-scale) x = b,
// x0 = 0, block-Jacobi preconditioner from the Cholesky factor of each damped
// 6x6 diagonal block (with the reference's jitter retry), stop at
// |r| / |b| <= tolerance or after the iteration cap.  One thread-block
// cluster per wrap (blockIdx.y), any cluster size.
//
// The recurrence is the single-reduction form of preconditioned CG
// (Chronopoulos & Gear, 1989): with u = M^-1 r and w = A u, the three inner
// products (r,u), (w,u), (r,r) of an iteration are formed together, so an
// iteration needs one exchange of partial sums and one exchange of u:
//
//   gamma = (r,u), delta = (w,u); beta = gamma / gamma_prev;
//   alpha = gamma / (delta - beta gamma / alpha_prev)   (beta = 0 first);
//   p = u + beta p;  s = w + beta s;  x += alpha p;  r -= alpha s.
//
// FP32 blocks, matvec, p, s, u and w; FP64 x, r, the inner products and the
// scalars.  Each CTA sends its slice of u as one bulk copy per peer through
// distributed shared memory, and each octet's partial sums with asynchronous
// stores; both complete on an mbarrier of the receiver, so a CTA waits only for
// its data, and the loop has no cluster barrier.  What is received is not
// overwritten early: a peer sends its next u after it has every CTA's sums,
// which each CTA sends after reading u; and its next sums after it has every
// CTA's u, which each CTA sends after reading the sums.
//
// kAllShared: every array of the placement is in shared memory (the compiler
// then addresses it as such); the other instance decides at run time.
//
// kGrid: the CTAs are a cooperative grid over the whole device instead of a
// cluster, for a graph whose rows are worth more SMs than a cluster has.  u
// (eight floats a node) and the segments' sums are then in global memory, and
// the CTAs meet at a counter in global memory twice per iteration; a CTA holds
// so few rows that its own arrays are always in shared memory.
//
// Every wait has a limit (`tries`).  A CTA whose wait ran out sets
// kErrorSolveWait, upon which the decision kernel ends the wrap; it first waits
// for the copies it has started, and its peers' waits run out in turn.
template <bool kAllShared, bool kGrid>
__device__ __forceinline__ void pcg_solve(const WrapDev& w, const WrapControl& c, const PcgPlacement& place,
                                          int budget_floats, int tries) {
    static_assert(kAllShared || !kGrid, "a grid whose rows would not fit is not launched (pcg_grid_fits)");
    cg::cluster_group cluster = cg::this_cluster();
    const LevelDev& L = w.levels[c.level];
    const int N = L.node_count;
    const int rank = kGrid ? (int)blockIdx.x : (int)cluster.block_rank();
    const int ranks = kGrid ? (int)gridDim.x : (int)cluster.num_blocks();
    const int segs = pcg_segments(N);
    const int octets = pcg_octets(N);
    const int cap = pcg_owned_capacity(N, ranks);
    const int o0 = min(octets, rank * (cap / kOctet));
    const int o1 = min(octets, o0 + cap / kOctet);
    const int n0 = o0 * kOctet;
    const int n1 = min(N, o1 * kOctet);
    int own = n1 > n0 ? n1 - n0 : 0;
    const int rows = own * 6;

    extern __shared__ float4 dynamic_shared[];
    double* slots;  // 3 per segment, in every CTA
    float* cursor;
    float *U, *own_u;  // u of every node; of the owned rows
    float* gathered = nullptr;
    if (kGrid) {
        slots = w.pcg_sums;
        U = w.pcg_u;
        cursor = reinterpret_cast<float*>(dynamic_shared);
        own_u = cursor;
        cursor += cap * 6;
        gathered = cursor;  // a warp's steps' u
        cursor += kPcgWarps * kGatherSteps * 64;
    } else {
        slots = reinterpret_cast<double*>(dynamic_shared);
        cursor = reinterpret_cast<float*>(slots + pcg_slot_doubles(N));
        if (kAllShared || place.u_shared) {
            U = cursor;
            cursor += (N * 6 + 3) & ~3;
        } else {
            U = w.pcg_u;
        }
        own_u = U + n0 * 6;
    }
    double *X, *R;
    float *Minv, *P, *S, *Wv;
    int* degrees = nullptr;  // per owned node; then per owned octet its first step and its steps
    float* diagonal = nullptr;
    if (kAllShared || place.vectors_shared) {
        X = reinterpret_cast<double*>(cursor);
        R = X + cap * 6;
        P = reinterpret_cast<float*>(R + cap * 6);
        S = P + cap * 6;
        Wv = S + cap * 6;
        degrees = reinterpret_cast<int*>(Wv + cap * 6);
        cursor += cap * kPcgVectorFloats;
    } else {
        X = w.pcg_x + n0 * 6;
        R = w.pcg_r + n0 * 6;
        P = w.pcg_p + n0 * 6;
        S = w.pcg_s + n0 * 6;
        Wv = w.pcg_ap + n0 * 6;
    }
    if (kAllShared) {
        diagonal = cursor;
        cursor += cap * kPcgBlockFloats;
    }
    if (kAllShared || place.inverse_shared) {
        Minv = cursor;
        cursor += cap * kPcgBlockFloats;
    } else {
        Minv = w.factor + n0 * 36;
    }
    const float* __restrict__ D = w.diag[c.system];
    const float4* __restrict__ B = reinterpret_cast<const float4*>(w.offdiag[c.system]);
    const float* __restrict__ b = w.rhs[c.system];
    const int* __restrict__ row_begin = L.row_begin;
    const int* __restrict__ sell_begin = L.sell_begin;
    const int* __restrict__ sell_nodes = L.sell_nodes;
    constexpr int kStepFloat4s = kStepFloats / 4;
    const float damping = (float)c.damping;
    const bool scaled = w.diagonal_damping != 0;
    const int max_iterations = w.pcg_max_iterations;
    const double tolerance = w.pcg_tolerance;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ double red[3][kPcgWarps];
    // mbarriers: the cached blocks; an iteration's partial sums; its u
    __shared__ alignas(8) unsigned long long blocks_arrived, sums_arrived, u_arrived;
    __shared__ int cached_s, listed_s;
    bool timed_out = false;  // a wait of this thread ran out

    // ---- the last steps of every owned octet's blocks into the shared
    //      memory that is left, as many as fit, by bulk copies that run under
    //      the factorisation below ----
    if (warp == 0) {
        int most = 0;
        for (int o = o0 + lane; o < o1; o += 32) most = max(most, sell_begin[o + 1] - sell_begin[o]);
        most = __reduce_max_sync(0xffffffffu, most);
        // a grid keeps the other nodes of every step if they fit (a node of very
        // many neighbours may prevent it), a cluster of the cached ones
        const int room = budget_floats - place.floats;
        const bool list_all = kGrid && (long)(o1 - o0) * most * kOctet <= room;
        const int left = list_all ? room - (o1 - o0) * most * kOctet : room;
        const int each = kGrid ? kStepFloats : kStepFloats + kOctet;
        const int cached = o1 > o0 ? max(0, min(most, left / ((o1 - o0) * each))) : 0;
        const int listed = kGrid ? (list_all ? most : 0) : cached;  // steps whose nodes are kept
        if (lane == 0) {
            cached_s = cached;
            listed_s = listed;
            mbar_init(&blocks_arrived, 1);
            mbar_init(&sums_arrived, kPcgWarps);
            mbar_init(&u_arrived, 1);
        }
        __syncwarp();
        int bytes = 0;
        for (int o = o0 + lane; o < o1; o += 32) {
            const int steps = sell_begin[o + 1] - sell_begin[o];
            bytes += (min(cached, steps) * kStepFloats + min(listed, steps) * kOctet) * (int)sizeof(float);
        }
        bytes = __reduce_add_sync(0xffffffffu, bytes);
        if (lane == 0) mbar_arrive_expect(&blocks_arrived, bytes);
        __syncwarp();
        float* block_room = cursor;
        float* node_room = cursor + (long)(o1 - o0) * cached * kStepFloats;
        for (int o = o0 + lane; o < o1; o += 32) {
            const int end = sell_begin[o + 1], steps = end - sell_begin[o];
            const int count = min(cached, steps), nodes = min(listed, steps);
            if (count > 0)
                bulk_to_shared(block_room + (long)(o - o0) * cached * kStepFloats, B + (long)(end - count) * kStepFloat4s,
                               count * kStepFloats * (int)sizeof(float), &blocks_arrived);
            if (nodes > 0)
                bulk_to_shared(node_room + (o - o0) * listed * kOctet, sell_nodes + (long)(end - nodes) * kOctet,
                               nodes * kOctet * (int)sizeof(float), &blocks_arrived);
        }
    }

    // a diagonal entry damped (spelt out, so that every instance rounds alike)
    auto damped = [&](float x) {
        const float scale = scaled ? fmaxf(x, 1e-12f) : 1.0f;
        return __fmaf_rn(damping, scale, x);
    };
    // ---- damped diagonal blocks and their inverses (route A's damped():
    //      scale = max(D_rr, 1e-12)); Cholesky with the reference's jitter ----
    for (int m = threadIdx.x; m < own; m += blockDim.x) {
        const int n = n0 + m;
        float blk[36];
        for (int i = 0; i < 36; ++i) blk[i] = D[n * 36 + i];
        for (int r = 0; r < 6; ++r) blk[r * 7] = damped(blk[r * 7]);
        if (kAllShared) {  // stored as a step's block
            float* to = diagonal + block_base(m);
            for (int i = 0; i < 36; ++i) to[block_at(i / 6, i % 6)] = blk[i];
            degrees[m] = row_begin[n + 1] - row_begin[n];
            if (m % kOctet == 0) {
                const int first = sell_begin[n / kOctet];
                degrees[cap + m / kOctet * 2] = first;
                degrees[cap + m / kOctet * 2 + 1] = sell_begin[n / kOctet + 1] - first;
            }
        }
        float jitter = 0.0f;
        bool ok = false;
        for (int attempt = 0; attempt < 8 && !ok; ++attempt) {
            float cand[36];
            for (int i = 0; i < 36; ++i) cand[i] = blk[i];
            for (int r = 0; r < 6; ++r) cand[r * 7] += jitter;
            if (cholesky6(cand)) {
                cholesky_inverse6(cand, Minv + m * 36);
                ok = true;
            }
            jitter = jitter == 0.0f ? 1e-6f : jitter * 10.0f;
        }
        if (!ok)
            for (int i = 0; i < 36; ++i) Minv[m * 36 + i] = (i % 7 == 0) ? 1.0f : 0.0f;
    }
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
        X[i] = 0.0;
        R[i] = (double)b[n0 * 6 + i];
        P[i] = 0.0f;
        S[i] = 0.0f;
    }
    // every CTA's rows and mbarriers are ready
    if (kGrid) __syncthreads();
    else cluster.sync();

    const int cached = cached_s, listed = listed_s;
    const float4* cached_blocks = reinterpret_cast<const float4*>(cursor);
    const int* cached_nodes = reinterpret_cast<const int*>(cursor + (long)(o1 - o0) * cached * kStepFloats);
    // The lists of nodes among what was copied are indices: without them no
    // product is formed.
    const bool incomplete = __syncthreads_or(!mbar_wait(&blocks_arrived, 0, tries));
    auto give_up = [&]() {
        if (threadIdx.x == 0) atomicOr(&w.control->error, kErrorSolveWait);
        mbar_wait(&blocks_arrived, 0, kWaitTries);  // this CTA's own copies
        for (int i = 0; i < 256; ++i) __nanosleep(10000);  // and those it sent to its peers (2.6 ms)
    };
    if (incomplete) {
        give_up();
        own = 0;  // skips the loop
    }

    // The CTAs that own rows; the others only wait at the end.  (Where u is
    // global the loop meets at cluster barriers, and so does the end.)
    const int active = (octets * kOctet + cap - 1) / cap;
    const bool u_shared = !kGrid && (kAllShared || place.u_shared);
    const int u_bytes = ((N * 6 + 3) & ~3) * (int)sizeof(float);  // of every row
    const int own_bytes = (rank == active - 1 ? u_bytes : n1 * 24) - n0 * 24;
    const int peer = kGrid ? 0 : min(lane, active - 1);
    const uint32_t peer_slots = kGrid ? 0 : peer_address(slots, peer);
    const uint32_t peer_sums_arrived = kGrid ? 0 : peer_address(&sums_arrived, peer);
    unsigned meetings = 0;  // the grid's, so far
    auto meet = [&]() {     // every active CTA's writes before it are visible after it
        __syncthreads();
        ++meetings;
        if (threadIdx.x == 0 && !grid_arrive_and_wait(w.solve_arrivals, meetings * (unsigned)active, tries * kPollsPerTry))
            timed_out = true;
        // the other threads learn of a wait that ran out at the totals' barrier
        __syncthreads();
    };

    // One segment's rows per warp at a time: `update` forms r[i], then
    // u = M^-1 r into this CTA's copy.
    auto segment_rows = [&](auto update) {
        for (int sl = warp; sl * 24 < rows; sl += kPcgWarps) {
            const int i = sl * 24 + lane;
            const bool on = lane < 24 && i < rows;
            if (on) update(i);
            __syncwarp();
            if (on) {
                const int m = sl * 4 + lane / 6, r = lane % 6;
                const float* mi = Minv + m * 36 + r * 6;
                float z = 0.0f;
                for (int q = 0; q < 6; ++q) z += mi[q] * (float)R[m * 6 + q];
                own_u[i] = z;
                if (kGrid) __stcg(U + (long)(n0 + m) * 8 + r, z);
            }
        }
    };
    // The slice of u into every other CTA's copy: one bulk copy per peer,
    // which completes on the peer's mbarrier.
    auto share_u = [&]() {
        if (kGrid) {
            meet();
            return;
        }
        if (!u_shared) {
            __threadfence();  // the global copy: visible device-wide first
            cluster.sync();
            return;
        }
        if (active > 1) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (active > 1 && warp == 0) {
            if (lane == 0) mbar_arrive_expect(&u_arrived, u_bytes - own_bytes);
            if (lane < active && lane != rank)
                bulk_to_peer(peer_address(U, lane) + n0 * 24, U + n0 * 6, own_bytes, peer_address(&u_arrived, lane));
        }
    };
    // A few streamed steps of octet o (its first `streamed`) into registers.
    const int i_node = lane / 3, p_row = lane - i_node * 3;
    StepBlocks ahead;
    // Past the end they are zeros: values left over from an earlier fetch would
    // hold their registers through the whole iteration.
    auto fetch = [&](int first, int t, int end) {
#pragma unroll
        for (int k = 0; k < kStepsAhead; ++k) {
            const bool there = t + k < end;
            const float4* at = B + (long)(first + t + k) * kStepFloat4s + lane;
            const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (!kGrid) ahead.node[k] = there ? __ldg(sell_nodes + (long)(first + t + k) * kOctet + i_node) : 0;
            ahead.b[k][0] = there ? __ldg(at) : zero;
            ahead.b[k][1] = there ? __ldg(at + 24) : zero;
            ahead.b[k][2] = there ? __ldg(at + 48) : zero;
        }
    };
    struct OctetShape { int first, steps, streamed, degree; };
    auto octet_shape = [&](int o) {
        OctetShape x;
        const int n = o * kOctet + i_node;
        const bool on = lane < 24 && n < N;
        int steps;
        x.degree = 0;
        if (kAllShared) {
            x.first = degrees[cap + (o - o0) * 2];
            steps = degrees[cap + (o - o0) * 2 + 1];
            if (on) x.degree = degrees[n - n0];
        } else {
            x.first = sell_begin[o];
            steps = sell_begin[o + 1] - x.first;
            if (on) x.degree = row_begin[n + 1] - row_begin[n];
        }
        x.steps = steps;
        x.streamed = max(0, steps - cached);
        return x;
    };
    // The warp's first streamed steps do not depend on u: they are fetched
    // before the wait for it.
    OctetShape shape = {0, 0, 0, 0};
    auto fetch_first = [&]() {
        if (o0 + warp < o1) {
            shape = octet_shape(o0 + warp);
            if (!kGrid) fetch(shape.first, 0, min(shape.streamed, shape.degree));
        }
    };
    if (own > 0) {
        segment_rows([](int) {});
        share_u();
        fetch_first();
    }

    double gamma_prev = 0.0, alpha_prev = 0.0, bnorm = 0.0, residual = 0.0, surely_above = 0.0;
    int iterations = 0;
    bool converged = false;
    for (int it = 0; own > 0; ++it) {
        if (u_shared && active > 1 && !mbar_wait(&u_arrived, it & 1, tries)) timed_out = true;
        // ---- w = A u for the owned rows, an octet per warp at a time: lane
        //      3i + p multiplies rows 2p and 2p + 1 of the octet's node i ----
        for (int o = o0 + warp; o < o1; o += kPcgWarps) {
            const int n = o * kOctet + i_node;
            const bool on = lane < 24 && n < N;
            if (o != o0 + warp) {
                shape = octet_shape(o);
                if (!kGrid) fetch(shape.first, 0, min(shape.streamed, shape.degree));
            }
            RowPair y = {0.0f, 0.0f};
            if (kAllShared) {
                if (on) {
                    const float4* at = reinterpret_cast<const float4*>(diagonal) + (long)(o - o0) * kStepFloat4s + lane;
                    y = row_pair_dot<true>(at[0], at[24], at[48], own_u + (n - n0) * 6);
                }
            } else if (on) {
                const float4* d4 = reinterpret_cast<const float4*>(D + (long)n * 36) + p_row * 3;
                float4 q0 = __ldg(d4), q1 = __ldg(d4 + 1), q2 = __ldg(d4 + 2);
                auto damp = [&](float& x) { x = damped(x); };
                damp(p_row == 0 ? q0.x : (p_row == 1 ? q0.z : q1.x));  // (2p, 2p) and (2p + 1, 2p + 1)
                damp(p_row == 0 ? q1.w : (p_row == 1 ? q2.y : q2.w));
                y = row_pair_dot<true>(q0, q1, q2, U + n * 6);
            }
            const float4* const cached_at = cached_blocks + (long)(o - o0) * cached * kStepFloat4s + lane;
            const int* const listed_at = cached_nodes + (o - o0) * listed * kOctet;
            // steps [t, t + kStepsAhead) below `end`, added in order: dot(k)
            // gives the products of step t + k
            auto add_steps = [&](int t, int end, auto&& dot) {
                RowPair part[kStepsAhead];
#pragma unroll
                for (int k = 0; k < kStepsAhead; ++k) part[k] = dot(k);
#pragma unroll
                for (int k = 0; k < kStepsAhead; ++k)
                    if (t + k < end) {
                        y.a += part[k].a;
                        y.b += part[k].b;
                    }
            };
            if constexpr (kGrid) {
                // kGatherSteps steps at a time: the warp copies all their u
                // from global memory at once (one latency instead of one per
                // group of steps), then multiplies from shared memory
                float* const room = gathered + warp * kGatherSteps * 64;
                for (int base = 0; base < shape.steps; base += kGatherSteps) {
                    const int last = min(shape.degree, base + kGatherSteps);
                    const int streamed = min(shape.streamed, last);
                    fetch(shape.first, base, streamed);
#pragma unroll
                    for (int j = 0; j < kGatherSteps / 2; ++j) {
                        const int step = 2 * j + (lane >> 4), half = lane & 1, node = (lane >> 1) & 7;
                        if (base + step < shape.steps)
                        {
                            const int at = (base + step) * kOctet + node;
                            const int id = listed > 0 ? listed_at[at] : __ldg(sell_nodes + (long)shape.first * kOctet + at);
                            copy_16_async(room + step * 64 + node * 8 + half * 4, U + (long)id * 8 + half * 4);
                        }
                    }
                    wait_copies();
                    __syncwarp();
                    const float* const mine = room + i_node * 8;
                    for (int t = base; t < streamed; t += kStepsAhead) {
                        add_steps(t, streamed, [&](int k) {
                            return row_pair_dot<false>(ahead.b[k][0], ahead.b[k][1], ahead.b[k][2],
                                                       mine + min(t + k - base, kGatherSteps - 1) * 64);
                        });
                        fetch(shape.first, t + kStepsAhead, streamed);
                    }
                    for (int t = max(base, shape.streamed); t < last; t += kStepsAhead)
                        add_steps(t, last, [&](int k) {
                            const int tk = min(t + k, last - 1);  // past the end: the last one again, not added
                            const float4* at = cached_at + (long)(tk - shape.streamed) * kStepFloat4s;
                            return row_pair_dot<false>(at[0], at[24], at[48], mine + (tk - base) * 64);
                        });
                    __syncwarp();  // read before the next steps' copies
                }
            } else {
                const int streamed = min(shape.streamed, shape.degree);
                for (int t = 0; t < streamed; t += kStepsAhead) {
                    add_steps(t, streamed, [&](int k) {
                        return row_pair_dot<false>(ahead.b[k][0], ahead.b[k][1], ahead.b[k][2],
                                                   U + ahead.node[k] * 6);
                    });
                    fetch(shape.first, t + kStepsAhead, streamed);
                }
                const int* const node = listed_at + i_node;
                const int end = shape.degree - shape.streamed;
                for (int t = 0; t < end; t += kStepsAhead) {
                    // every load of the group before its first product
                    int at[kStepsAhead], other[kStepsAhead];
#pragma unroll
                    for (int k = 0; k < kStepsAhead; ++k) at[k] = min(t + k, end - 1);  // past the end: not added
#pragma unroll
                    for (int k = 0; k < kStepsAhead; ++k) other[k] = node[at[k] * kOctet] * 6;
                    float4 b[kStepsAhead][3];
                    float2 u[kStepsAhead][3];
#pragma unroll
                    for (int k = 0; k < kStepsAhead; ++k)
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            b[k][j] = cached_at[at[k] * kStepFloat4s + 24 * j];
                            u[k][j] = reinterpret_cast<const float2*>(U + other[k])[j];
                        }
                    add_steps(t, end, [&](int k) {
                        return RowPair{row_dot<false>(b[k][0].x, b[k][0].y, b[k][0].z, b[k][0].w, b[k][1].x, b[k][1].y,
                                                      u[k][0], u[k][1], u[k][2]),
                                       row_dot<false>(b[k][1].z, b[k][1].w, b[k][2].x, b[k][2].y, b[k][2].z, b[k][2].w,
                                                      u[k][0], u[k][1], u[k][2])};
                    });
                }
            }
            const int first_row = (o * kOctet - n0) * 6;
            if (on) *reinterpret_cast<float2*>(Wv + first_row + 2 * lane) = make_float2(y.a, y.b);
            __syncwarp();
            // the two segments' partials of (r,u), (w,u), (r,r), a row per
            // lane; the six sums end in lanes 0, 4, 8, 16, 20 and 24
            double v[6];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = first_row + h * 24 + lane;
                double ui = 0.0, ri = 0.0, wi = 0.0;
                if (lane < 24 && k < rows) {
                    ui = (double)own_u[k];
                    ri = R[k];
                    wi = (double)Wv[k];
                }
                v[3 * h] = rnd(ri * ui);
                v[3 * h + 1] = rnd(wi * ui);
                v[3 * h + 2] = rnd(ri * ri);
            }
            int held = 0, count = 6;
            warp_sum_halving<6, 16>(v, lane, held, count, [](double x, double z) { return rnd(x + z); });
            if constexpr (kGrid) {
                const int third = (lane >> 2) & 3;  // lanes 0, 4, 8, 16, 20, 24 hold sums 0 .. 5
                if ((lane & 3) == 0 && third < 3) __stcg(slots + 6 * o + (lane >> 4) * 3 + third, v[0]);
            } else {
                double partial[6];
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    partial[k] = __shfl_sync(0xffffffffu, v[0], (k >= 3 ? 16 : 0) + (k % 3) * 4);
                if (active == 1) {
                    if (lane == 0)
                        for (int k = 0; k < 6; ++k) slots[6 * o + k] = partial[k];
                } else if (lane < active) {  // lane q stores the partials in CTA q's slots
                    const uint32_t dst = peer_slots + 48 * o;
                    store_to_peer(dst, partial[0], partial[1], peer_sums_arrived);
                    store_to_peer(dst + 16, partial[2], partial[3], peer_sums_arrived);
                    store_to_peer(dst + 32, partial[4], partial[5], peer_sums_arrived);
                }
            }
        }
        if (kGrid) {
            meet();
        } else {
            __syncwarp();
            if (threadIdx.x == 0) {
                mbar_arrive_expect(&sums_arrived, active > 1 ? 48 * octets : 0);
            } else if (lane == 0) {
                mbar_arrive(&sums_arrived);
            }
            if (!mbar_wait(&sums_arrived, it & 1, tries)) timed_out = true;
        }
        // ---- totals over every segment, in one fixed order in every CTA:
        //      each warp its stride of the segments, then every warp the same
        //      butterfly over the warps' sums ----
        double gamma, delta, rr_total;
        {
            double v[3] = {0.0, 0.0, 0.0};
            if (warp * 32 < segs) {
#pragma unroll 4
                for (int sg = threadIdx.x; sg < segs; sg += kPcgThreads)
                    for (int k = 0; k < 3; ++k)
                        v[k] = rnd(v[k] + (kGrid ? __ldcg(slots + 3 * sg + k) : slots[3 * sg + k]));
                int held = 0, count = 3;
                warp_sum_halving<3, 16>(v, lane, held, count, [](double x, double z) { return rnd(x + z); });
            }
            // the sums end in lanes 0, 8 and 16
            if (lane == 0 || lane == 8 || lane == 16) red[lane >> 3][warp] = v[0];
            const bool failed = __syncthreads_or(timed_out);
            double a = red[lane >> 4][lane & 15], b2 = red[2][lane & 15];
            static_assert(kPcgWarps == 16, "a half warp per sum");
            for (int o = 8; o > 0; o >>= 1) {
                a = rnd(a + __shfl_xor_sync(0xffffffffu, a, o));
                b2 = rnd(b2 + __shfl_xor_sync(0xffffffffu, b2, o));
            }
            gamma = __shfl_sync(0xffffffffu, a, 0);
            delta = __shfl_sync(0xffffffffu, a, 16);
            rr_total = b2;
            if (failed) {  // uniform over the CTA; its peers' waits run out in turn
                give_up();
                break;
            }
        }
        if (it == 0) {
            bnorm = rnd(sqrt(rr_total));
            if (!(bnorm > 0.0)) { converged = true; residual = 0.0; break; }
            // |r|^2 above this is surely not converged: the comparison below
            // without its root and quotient
            const double limit = tolerance * bnorm;
            surely_above = limit > 1e-140 ? limit * limit * (1.0 + 1e-6) : 1e300;
        }
        const bool capped = it >= max_iterations;
        if (capped || !(rr_total > surely_above)) {
            residual = rnd(rnd(sqrt(rr_total)) / bnorm);
            if (residual <= tolerance) { converged = true; break; }
            if (capped) break;
        }
        const double beta = it == 0 ? 0.0 : rnd(gamma / gamma_prev);
        const double denominator = it == 0 ? delta : rnd(delta - rnd(rnd(beta * gamma) / alpha_prev));
        if (!(fabs(denominator) > 1e-300)) {
            residual = rnd(rnd(sqrt(rr_total)) / bnorm);
            break;
        }
        const double alpha = rnd(gamma / denominator);
        gamma_prev = gamma;
        alpha_prev = alpha;
        // ---- p, s, x, r for the owned rows; then u = M^-1 r, shared ----
        segment_rows([&](int i) {
            const float pn = (float)((double)own_u[i] + rnd(beta * (double)P[i]));
            const float sn = (float)((double)Wv[i] + rnd(beta * (double)S[i]));
            P[i] = pn;
            S[i] = sn;
            X[i] = rnd(X[i] + rnd(alpha * (double)pn));
            R[i] = rnd(R[i] - rnd(alpha * (double)sn));
        });
        share_u();
        fetch_first();
        iterations = it + 1;
    }
    if (rank == 0 && threadIdx.x == 0) {
        w.control->pcg_ok = converged ? 1 : 0;
        w.control->pcg_iterations = iterations;
        w.control->pcg_residual = residual;
    }
    if (converged) {
        // candidate = retract(accepted, delta): R <- exp([w]) R, t <- t + u
        // (deformation.cpp:19-32).  Route C's rotation half is zero and its
        // rotations were already fitted into the candidate buffer.
        for (int m = threadIdx.x; m < own; m += blockDim.x) {
            const int n = n0 + m;
            const double* x = X + m * 6;
            const D3 tcur = load_d3(w.trans[c.state], n);
            store_d3(w.trans[1 - c.state], n, {tcur.x + x[3], tcur.y + x[4], tcur.z + x[5]});
            double out[9];
            if (c.route == 0) {
                double e[9];
                exp_so3({x[0], x[1], x[2]}, e);
                mat_mul(e, w.rot[c.state] + n * 9, out);
                for (int i = 0; i < 9; ++i) w.rot[1 - c.state][n * 9 + i] = out[i];
            } else {
                for (int i = 0; i < 9; ++i) out[i] = w.rot[1 - c.state][n * 9 + i];
            }
            for (int i = 0; i < 9; ++i) w.rot32[n * 9 + i] = (float)out[i];
            for (int k = 0; k < 6; ++k) w.delta[n * 6 + k] = x[k];
        }
    }
    // no CTA may exit while another can still write into its shared memory
    if (!kGrid && u_shared) {
        cluster.sync();
    } else if (!kGrid) {
        // The loop has met at this barrier, so a CTA whose wait ran out would
        // pair with the others' next meeting and exit while they go on to send
        // it their sums.  It meets them until every CTA has left the loop,
        // which their waits for its own sums see to.
        __shared__ int all_left_s;
        if (threadIdx.x == 0) atomicAdd(w.solve_arrivals, 1u);  // after the last that this CTA has sent
        for (;;) {
            cluster.sync();
            if (threadIdx.x == 0) {
                unsigned left;
                asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(left) : "l"(w.solve_arrivals) : "memory");
                all_left_s = left >= (unsigned)ranks;
            }
            __syncthreads();
            if (all_left_s) break;
        }
    } else {
        __syncthreads();
        if (threadIdx.x == 0)  // initialised again for the block's next wrap
            for (void* bar : {(void*)&blocks_arrived, (void*)&sums_arrived, (void*)&u_arrived}) mbar_invalidate(bar);
    }
}

// Whether the grid kernel takes a wrap's solve this tick (both kernels ask):
// its graph has more than `grid_nodes` nodes for every wrap that the grid would
// take one after the other, and no smaller solve needs SMs at the same time.
__device__ inline bool grid_takes(const WrapDev* wraps, int wrap_count, int nodes, int grid_nodes) {
    if (grid_nodes <= 0 || nodes <= grid_nodes) return false;
    int solving = 0, large = 0;
    for (int i = 0; i < wrap_count; ++i) {
        const WrapControl* c = wraps[i].control;
        if (c->tick_phase != kPhaseSolve || c->phase != kPhaseSolve) continue;
        ++solving;
        large += wraps[i].levels[c->level].node_count > grid_nodes ? 1 : 0;
    }
    return solving == large && nodes > grid_nodes * large;
}

// The wraps the grid takes, one after the other over the whole device.
__global__ void __launch_bounds__(kPcgThreads, 1) k_pcg_grid(const WrapDev* __restrict__ wraps, int wrap_count,
                                                          int grid_nodes, int budget_floats, int tries) {
    for (int i = 0; i < wrap_count; ++i) {
        const WrapDev& w = wraps[i];
        const WrapControl c = *w.control;
        if (c.tick_phase != kPhaseSolve || c.phase != kPhaseSolve) continue;
        const int N = w.levels[c.level].node_count;
        if (!grid_takes(wraps, wrap_count, N, grid_nodes)) continue;
        PcgPlacement place = {};
        place.floats = pcg_grid_floats(N, (int)gridDim.x);
        pcg_solve<true, true>(w, c, place, budget_floats, tries);
        __syncthreads();  // shared memory of one wrap before the next
    }
}

__global__ void __launch_bounds__(kPcgThreads, 1) k_pcg(const WrapDev* __restrict__ wraps,
                                                     const int* __restrict__ index,
                                                     int budget_floats, int wrap_count, int grid_nodes, int tries) {
    const int slot = index ? index[blockIdx.y] : (int)blockIdx.y;
    if (slot < 0) return;  // an empty entry of a class launch; uniform across the cluster
    const WrapDev& w = wraps[slot];
    const WrapControl c = *w.control;
    if (c.tick_phase != kPhaseSolve || c.phase != kPhaseSolve) return;  // uniform across the cluster
    if (grid_takes(wraps, wrap_count, w.levels[c.level].node_count, grid_nodes)) return;
    const PcgPlacement place =
        pcg_place(w.levels[c.level].node_count, (int)cg::this_cluster().num_blocks(), budget_floats);
    if (place.all()) {
        pcg_solve<true, false>(w, c, place, budget_floats, tries);
    } else {
        pcg_solve<false, false>(w, c, place, budget_floats, tries);
    }
}

// ---------------------------------------------------------------------------
// deformation evaluation (deformation.cpp:55-68) and the deformed template's
// vertex normals (mesh.cpp:71-88)
// ---------------------------------------------------------------------------
// The deformed position of vertex v under the state being evaluated.
__device__ __forceinline__ D3 evaluate_vertex(const WrapDev& w, const LevelDev& L, const WrapControl& c, int v) {
    const int buf = eval_buffer(c);
    const double* R = w.rot[buf];
    const double* T = w.trans[buf];
    const D3 p = load_d3(w.tpl, v);
    D3 sum = {0.0, 0.0, 0.0};
    const int count = L.bind_counts[v];
    for (int s = 0; s < count; ++s) {
        const int j = L.bind_nodes[v * kMaxSlots + s];
        const double wt = L.bind_weights[v * kMaxSlots + s];
        const D3 g = load_d3(L.rest, j);
        const D3 applied = radd(radd(rmat(R + j * 9, rsub(p, g)), g), load_d3(T, j));
        sum = radd(sum, rmul(applied, wt));
    }
    if (count == 0) sum = p;
    store_d3(w.deformed, v, sum);
    w.deformed32[v] = make_float4((float)sum.x, (float)sum.y, (float)sum.z, 0.0f);
    return sum;
}

__device__ __forceinline__ void k_evaluate_body(const WrapDev& w, int part, int bx) {
    const WrapControl c = *w.control;
    if (!in_part(c, part)) return;
    if (c.phase == kPhaseDone || !has_candidate(c)) return;
    const int v = bx * blockDim.x + threadIdx.x;
    if (v < w.V) evaluate_vertex(w, w.levels[c.level], c, v);
}

__global__ void k_evaluate(const WrapDev* __restrict__ wraps, int wrap_count, int part) {
    over_virtual_blocks<false>(
        wraps, wrap_count,
        [&](const WrapDev& w) {
            const WrapControl c = *w.control;
            return in_part(c, part) ? ((c.phase != kPhaseDone && has_candidate(c)) ? blocks_of_dev(w.V, kVertexThreads) : 0) : 0;
        },
        [&](int wi, int bx) { k_evaluate_body(wraps[wi], part, bx); });
}

// A thread per vertex; a vertex of more faces than kWideFan (the poles of a
// lat-long template have hundreds) is its warp's: the lanes form the faces'
// normals, which are then added in face order, as the thread's loop would.
// (One thread's loop over a pole's 224 faces held the kernel for 68 us.)
constexpr int kWideFan = 24;
__device__ __forceinline__ D3 face_normal(const WrapDev& w, int i) {
    const int32_t* f = w.tpl_faces + (long)w.vf_faces[i] * 3;
    const D3 a = load_d3(w.deformed, f[0]);
    const D3 b = load_d3(w.deformed, f[1]);
    const D3 c = load_d3(w.deformed, f[2]);
    return rcross(rsub(b, a), rsub(c, a));
}
__device__ __forceinline__ void k_normals_body(const WrapDev& w, int part, int bx) {
    const WrapControl c = *w.control;
    if (!in_part(c, part)) return;
    if (!refresh_like(c.phase)) return;
    const int v = bx * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const int begin = v < w.V ? w.vf_begin[v] : 0, end = v < w.V ? w.vf_begin[v + 1] : 0;
    const bool wide = end - begin > kWideFan;
    D3 n = {0.0, 0.0, 0.0};
    if (!wide)
        for (int i = begin; i < end; ++i) n = radd(n, face_normal(w, i));
    uint32_t fans = __ballot_sync(0xffffffffu, wide);
    while (fans) {
        const int owner = __ffs(fans) - 1;
        fans &= fans - 1;
        const int b = __shfl_sync(0xffffffffu, begin, owner), e = __shfl_sync(0xffffffffu, end, owner);
        D3 sum = {0.0, 0.0, 0.0};
        for (int base = b; base < e; base += 32) {
            D3 x = {0.0, 0.0, 0.0};
            if (base + lane < e) x = face_normal(w, base + lane);
            const int here = min(32, e - base);
            for (int k = 0; k < here; ++k)
                sum = radd(sum, {__shfl_sync(0xffffffffu, x.x, k), __shfl_sync(0xffffffffu, x.y, k),
                                 __shfl_sync(0xffffffffu, x.z, k)});
        }
        if (lane == owner) n = sum;
    }
    if (v >= w.V) return;
    const double len = __dsqrt_rn(rdot(n, n));
    if (len > 0.0) n = {__ddiv_rn(n.x, len), __ddiv_rn(n.y, len), __ddiv_rn(n.z, len)};
    else n = {0.0, 0.0, 0.0};
    store_d3(w.qnormals, v, n);
}

__global__ void k_normals(const WrapDev* __restrict__ wraps, int wrap_count, int part) {
    over_virtual_blocks<false>(
        wraps, wrap_count,
        [&](const WrapDev& w) {
            const WrapControl c = *w.control;
            return in_part(c, part) ? (refresh_like(c.phase) ? blocks_of_dev(w.V, kVertexThreads) : 0) : 0;
        },
        [&](int wi, int bx) { k_normals_body(wraps[wi], part, bx); });
}

// ---------------------------------------------------------------------------
// per-vertex residuals, the data and landmark energies (FP64), and the FP32
// residual records the assembly reads (fused_assembly.cpp:185-216, 262-280)
// ---------------------------------------------------------------------------
// The node-local offset R (p_v - g_node) of vertex v bound to `node`, FP32.
__device__ inline F3 node_offset32(const WrapDev& w, const LevelDev& L, int node, int v) {
    const D3 p = load_d3(w.tpl, v) - load_d3(L.rest, node);
    return mul3f(w.rot32 + node * 9, {(float)p.x, (float)p.y, (float)p.z});
}

// A node's anchor term (energy.cpp:239-271): its energy, and what it adds to
// the node's diagonal block and right-hand side (twelve floats: the upper
// triangle of the rotation block, the rotation half, the translation half).
__device__ __forceinline__ void anchor_term(const WrapDev& w, const WrapControl& c, int node) {
    const double weight = w.weights[c.level][3];
    double energy = 0.0;
    if (weight > 0.0) {
        const int buf = eval_buffer(c);
        const D3 om = log_so3(w.rot[buf] + node * 9);
        const D3 t = load_d3(w.trans[buf], node);
        const double sc = sqrt(weight);
        const double vals[6] = {sc * om.x, sc * om.y, sc * om.z, sc * t.x, sc * t.y, sc * t.z};
        for (int k = 0; k < 6; ++k) energy += vals[k] * vals[k];
        if (assembles(c)) {
            double J[9];
            left_jacobian_inverse(om, J);
            float* out = w.anchor32 + node * 12;
            int at = 0;
            for (int r = 0; r < 3; ++r)
                for (int q = r; q < 3; ++q) {
                    double s = 0.0;
                    for (int k = 0; k < 3; ++k) s += J[k * 3 + r] * J[k * 3 + q];
                    out[at++] = (float)(weight * s);
                }
            for (int r = 0; r < 3; ++r) {
                double s = 0.0;
                for (int k = 0; k < 3; ++k) s += J[k * 3 + r] * (k == 0 ? om.x : k == 1 ? om.y : om.z);
                out[at++] = (float)(weight * s);
            }
            out[9] = (float)(weight * t.x);
            out[10] = (float)(weight * t.y);
            out[11] = (float)(weight * t.z);
        }
    }
    w.node_partials[node] = energy;  // the decision kernel sums them
}

// kEvaluate: the vertex is deformed first (the solve chain; the refresh chain
// has deformed it before its query).  The blocks past the vertices' take the
// nodes' anchor terms, a thread each: FP64 logarithms and Jacobians of several
// thousand cycles, which in the node assembly held a whole warp per node.
template <bool kEvaluate>
__device__ __forceinline__ void k_residual_body(const WrapDev& w, int part, int bx) {
    const WrapControl c = *w.control;
    if (!in_part(c, part)) return;
    if (!computes_energy(c)) return;
    const LevelDev& L = w.levels[c.level];
    const int vertex_blocks = blocks_of_dev(w.V, kVertexThreads);
    if (bx >= vertex_blocks) {
        const int node = (bx - vertex_blocks) * kVertexThreads + threadIdx.x;
        if (node < L.node_count) anchor_term(w, c, node);
        return;
    }
    const int v = bx * blockDim.x + threadIdx.x;
    const double* wt = w.weights[c.level];
    double e[3] = {0.0, 0.0, 0.0};  // point to point, plane, landmark
    if (v < w.V) {
        float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = r0;
        const bool bound = L.bind_counts[v] > 0;
        const D3 q = kEvaluate ? evaluate_vertex(w, L, c, v) : load_d3(w.deformed, v);
        if (bound && w.corr_code[v] == 0) {
            const D3 y = load_d3(w.corr_point, v);
            const D3 o = rsub(q, y);
            const double u = fmax(0.0, w.robust[v]);
            const D3 n = load_d3(w.corr_normal, v);
            if (wt[0] > 0.0) {
                const double s = sqrt(wt[0] * u);
                const D3 so = rmul(o, s);
                e[0] = da(da(dm(so.x, so.x), dm(so.y, so.y)), dm(so.z, so.z));
                r0 = make_float4((float)o.x, (float)o.y, (float)o.z, (float)(wt[0] * u));
            } else {
                r0 = make_float4((float)o.x, (float)o.y, (float)o.z, 0.0f);
            }
            if (wt[1] > 0.0) {
                const double s = sqrt(wt[1] * u);
                const double value = dm(s, rdot(n, o));
                e[1] = dm(value, value);
                r1 = make_float4((float)n.x, (float)n.y, (float)n.z, (float)(wt[1] * u));
            }
        }
        if (bound && wt[4] > 0.0 && w.lm_flag[v]) {
            const D3 o = rsub(q, load_d3(w.lm_target, v));
            const double s = sqrt(wt[4]);
            const D3 so = rmul(o, s);
            e[2] = da(da(dm(so.x, so.x), dm(so.y, so.y)), dm(so.z, so.z));
            r2 = make_float4((float)o.x, (float)o.y, (float)o.z, (float)wt[4]);
        }
        if (assembles(c)) {
            w.residual32[v] = r0;
            w.resid_aux32[v] = r1;
            if (w.L > 0) w.lm_resid32[v] = r2;
            // each binding's offset and FP32 weight, once for the node and pair
            // assembly that follow
            if (bound)
                for (int k = 0; k < L.bind_counts[v]; ++k) {
                    const int node = L.bind_nodes[v * kMaxSlots + k];
                    if (node < 0) continue;
                    const F3 a = node_offset32(w, L, node, v);
                    w.offsets32[v * kMaxSlots + k] =
                        make_float4(a.x, a.y, a.z, (float)L.bind_weights[v * kMaxSlots + k]);
                }
        }
    }
    __shared__ double scratch[kVertexThreads / 32 * 3];
    block_sums<kVertexThreads, 3>(e, scratch);
    if (threadIdx.x == 0) {
        double* p = w.partials + (long)bx * kPartialStride;
        p[0] = e[0]; p[1] = e[1]; p[2] = e[2];
    }
}

template <bool kEvaluate>
__global__ void __launch_bounds__(kVertexThreads) k_residual(const WrapDev* __restrict__ wraps, int wrap_count, int part) {
    over_virtual_blocks<true>(
        wraps, wrap_count,
        [&](const WrapDev& w) {
            const WrapControl c = *w.control;
            if (!in_part(c, part) || !computes_energy(c)) return 0;
            return blocks_of_dev(w.V, kVertexThreads) + blocks_of_dev(w.levels[c.level].node_count, kVertexThreads);
        },
        [&](int wi, int bx) { k_residual_body<kEvaluate>(wraps[wi], part, bx); });
}

// ---------------------------------------------------------------------------
// Gauss-Newton blocks in one launch: a warp per node for the diagonal block and
// the right-hand side (data, landmark, incident smoothness edges, anchor), then
// a warp per off-diagonal block (the vertices its node pair shares, and the
// smoothness edge between them).  Closed forms of sum_rows J^T J for an offset
// residual replace the reference's row-by-row outer products.
// ---------------------------------------------------------------------------

// What one binding or one shared vertex adds is read through an index, so each
// lane keeps the next entry's data and the index after it in flight while it
// adds the current one.
struct NodeEntry {
    float4 a, r0, r1, r2;
};
__device__ __forceinline__ NodeEntry load_entry(const WrapDev& w, int entry, bool landmarks) {
    NodeEntry x;
    const int v = entry / kMaxSlots;
    x.a = __ldg(w.offsets32 + entry);
    x.r0 = __ldg(w.residual32 + v);
    x.r1 = __ldg(w.resid_aux32 + v);
    x.r2 = landmarks ? __ldg(w.lm_resid32 + v) : make_float4(0.f, 0.f, 0.f, 0.f);
    return x;
}

// One incident smoothness edge as a node sees it: its energy is stored if the
// node is its first (the decision kernel sums them), and what the block and the
// right-hand side need of it is returned.
struct EdgeTerms {
    F3 difference, arm;
    int role;  // 0 none, 1 the edge's first node, 2 its second
};
__device__ __forceinline__ EdgeTerms edge_terms(const WrapDev& w, const WrapControl& c, const LevelDev& L, int e,
                                                int a, int b, int node, bool build) {
    EdgeTerms t;
    t.role = 0;
    t.difference = t.arm = F3{0.0f, 0.0f, 0.0f};
    const double weight = w.weights[c.level][2];
    double energy = 0.0;
    if (weight > 0.0) {
        const int buf = eval_buffer(c);
        const double* R = w.rot[buf];
        const double* T = w.trans[buf];
        const D3 ga = load_d3(L.rest, a), gb = load_d3(L.rest, b);
        const D3 gd = rsub(gb, ga);
        const D3 field_a = radd(radd(rmat(R + a * 9, gd), ga), load_d3(T, a));
        const D3 field_b = radd(gb, load_d3(T, b));
        const D3 diff = rsub(field_a, field_b);
        const D3 scaled = rmul(diff, sqrt(weight));
        energy = da(da(dm(scaled.x, scaled.x), dm(scaled.y, scaled.y)), dm(scaled.z, scaled.z));
        if (build) {
            t.difference = F3{(float)diff.x, (float)diff.y, (float)diff.z};
            t.role = 2;
            if (a == node) {
                t.role = 1;
                t.arm = mul3f(w.rot32 + a * 9, {(float)gd.x, (float)gd.y, (float)gd.z});
            }
        }
    }
    if (a == node) w.edge_partials[e] = energy;
    return t;
}

// What the node's loop over its bindings has nothing to do with is loaded ahead
// of it: the lane's first edge (few nodes have more than 32) is reduced to six
// numbers while the first binding's data are on their way, so that the chain
// list -> edge -> positions and rotations does not follow the loop's own.
__device__ __forceinline__ void assemble_node(const WrapDev& w, const WrapControl& c, int node) {
    const bool build = assembles(c);
    const LevelDev& L = w.levels[c.level];
    const int lane = threadIdx.x & 31;
    const double* wt = w.weights[c.level];
    const int next = 1 - c.system;
    const int edge_first = L.node_edge_begin[node] + lane, edge_end = L.node_edge_begin[node + 1];
    const int edge = edge_first < edge_end ? L.node_edge_list[edge_first] : -1;
    EdgeTerms near;
    near.role = 0;
    near.difference = near.arm = F3{0.0f, 0.0f, 0.0f};
    float d[21], g[6];
    for (int i = 0; i < 21; ++i) d[i] = 0.0f;
    for (int i = 0; i < 6; ++i) g[i] = 0.0f;
    if (build) {
        const int end = L.gather_begin[node + 1];
        const bool landmarks = w.L > 0;
        int i = L.gather_begin[node] + lane;
        int after = i + 32 < end ? L.gather_entry[i + 32] : 0;
        NodeEntry ahead;
        const int entry = i < end ? L.gather_entry[i] : 0;
        const int ea = edge >= 0 ? L.edges[edge * 2] : 0, eb = edge >= 0 ? L.edges[edge * 2 + 1] : 0;
        if (i < end) ahead = load_entry(w, entry, landmarks);
        if (edge >= 0) near = edge_terms(w, c, L, edge, ea, eb, node, true);
        for (; i < end; i += 32) {
            const NodeEntry x = ahead;
            if (i + 32 < end) ahead = load_entry(w, after, landmarks);
            if (i + 64 < end) after = L.gather_entry[i + 64];
            const float wgt = x.a.w;
            const F3 a = {x.a.x, x.a.y, x.a.z};
            if (x.r0.w > 0.0f) {  // point to point
                const F3 o = {x.r0.x, x.r0.y, x.r0.z};
                add_offset_block(d, a, x.r0.w * wgt * wgt);
                const F3 ao = cross(a, o);
                const float s = x.r0.w * wgt;
                g[0] -= s * ao.x; g[1] -= s * ao.y; g[2] -= s * ao.z;
                g[3] -= s * o.x; g[4] -= s * o.y; g[5] -= s * o.z;
            }
            if (x.r1.w > 0.0f) {  // point to plane
                const F3 n = {x.r1.x, x.r1.y, x.r1.z};
                const F3 an = cross(a, n);
                const float u[6] = {an.x, an.y, an.z, n.x, n.y, n.z};
                add_rank_one(d, u, x.r1.w * wgt * wgt);
                const float pv = dot(n, F3{x.r0.x, x.r0.y, x.r0.z});
                const float s = x.r1.w * wgt * pv;
                for (int k = 0; k < 6; ++k) g[k] -= s * u[k];
            }
            if (x.r2.w > 0.0f) {  // landmark
                const F3 o = {x.r2.x, x.r2.y, x.r2.z};
                add_offset_block(d, a, x.r2.w * wgt * wgt);
                const F3 ao = cross(a, o);
                const float s = x.r2.w * wgt;
                g[0] -= s * ao.x; g[1] -= s * ao.y; g[2] -= s * ao.z;
                g[3] -= s * o.x; g[4] -= s * o.y; g[5] -= s * o.z;
            }
        }
    } else if (edge >= 0) {
        edge_terms(w, c, L, edge, L.edges[edge * 2], L.edges[edge * 2 + 1], node, false);
    }
    // the incident smoothness edges
    const float ws = (float)wt[2];
    auto add_edge = [&](const EdgeTerms& t) {
        if (t.role == 0) return;
        const F3 dv = t.difference;
        if (t.role == 1) {
            add_offset_block(d, t.arm, ws);
            const F3 cd = cross(t.arm, dv);
            g[0] -= ws * cd.x; g[1] -= ws * cd.y; g[2] -= ws * cd.z;
            g[3] -= ws * dv.x; g[4] -= ws * dv.y; g[5] -= ws * dv.z;
        } else {
            d[tri_index(3, 3)] += ws; d[tri_index(4, 4)] += ws; d[tri_index(5, 5)] += ws;
            g[3] += ws * dv.x; g[4] += ws * dv.y; g[5] += ws * dv.z;
        }
    };
    add_edge(near);
    for (int i = edge_first + 32; i < edge_end; i += 32) {
        const int e = L.node_edge_list[i];
        add_edge(edge_terms(w, c, L, e, L.edges[e * 2], L.edges[e * 2 + 1], node, build));
    }
    if (!build) return;
    if (lane == 0 && wt[3] > 0.0) {  // the anchor term, formed with the residuals
        const float* x = w.anchor32 + node * 12;
        int at = 0;
        for (int r = 0; r < 3; ++r)
            for (int q = r; q < 3; ++q) d[tri_index(r, q)] += x[at++];
        for (int r = 0; r < 3; ++r) g[r] -= x[at++];
        d[tri_index(3, 3)] += (float)wt[3]; d[tri_index(4, 4)] += (float)wt[3];
        d[tri_index(5, 5)] += (float)wt[3];
        g[3] -= x[9]; g[4] -= x[10]; g[5] -= x[11];
    }
    // the 21 upper-triangle sums and the 6 of the rhs, spread over the
    // lanes; each lane stores what it holds
    float v[27];
    for (int i = 0; i < 21; ++i) v[i] = d[i];
    for (int i = 0; i < 6; ++i) v[21 + i] = g[i];
    int first = 0, count = 27;
    warp_sum_halving<27>(v, lane, first, count);
    if (count > 0) {
        float* D = w.diag[next] + node * 36;
        float* G = w.rhs[next] + node * 6;
        const bool restricted = c.route == 1;
        const int j = first;
        if (j < 21) {
            int r = 0;
            while (tri_index(r + 1, r + 1) <= j) ++r;  // row of upper-triangle entry j
            const int q = j - tri_index(r, r) + r;
            float value = v[0];
            if (restricted && (r < 3 || q < 3)) value = (r == q) ? 1.0f : 0.0f;
            D[r * 6 + q] = value;
            D[q * 6 + r] = value;
        } else {
            const int k = j - 21;
            G[k] = (restricted && k < 3) ? 0.0f : v[0];
        }
    }
}

// Off-diagonal block k: the lanes stride over the vertices its node pair
// shares (none past pair_count), each with a 6x6 block in registers, then one
// halving reduction; the smoothness edge of the pair is added to the sums (it
// took a kernel of its own before, which read and wrote the blocks again with
// a thread per edge: 28 us of latency in every tick).
struct PairEntry {
    float4 a, b, r0, r1;
    float lm;
};
__device__ __forceinline__ PairEntry load_pair(const WrapDev& w, int code, bool landmarks) {
    PairEntry x;
    const int v = code >> 6, sa = (code >> 3) & 7, sb = code & 7;
    x.a = __ldg(w.offsets32 + v * kMaxSlots + sa);
    x.b = __ldg(w.offsets32 + v * kMaxSlots + sb);
    x.r0 = __ldg(w.residual32 + v);
    x.r1 = __ldg(w.resid_aux32 + v);
    x.lm = landmarks ? __ldg(&w.lm_resid32[v].w) : 0.0f;
    return x;
}

__device__ __forceinline__ void assemble_block(const WrapDev& w, const WrapControl& c, int k) {
    const LevelDev& L = w.levels[c.level];
    const int lane = threadIdx.x & 31;
    float blk[36];
    for (int i = 0; i < 36; ++i) blk[i] = 0.0f;
    const bool pair = k < L.pair_count;
    // what the loop has nothing to do with is loaded ahead of it
    const int edge = L.block_edge[k];
    const int slot = L.sell_slots[k * 2], mirror = L.sell_slots[k * 2 + 1];
    const float ws = edge >= 0 && w.weights[c.level][2] > 0.0 ? (float)w.weights[c.level][2] : 0.0f;
    const bool arm = ws > 0.0f && c.route == 0;
    F3 cv = {0.0f, 0.0f, 0.0f};
    // of the smoothness edge's term, ws * [[0, -[c]x], [0, -I]]: c = R_a (g_b - g_a)
    auto edge_arm = [&](int a, int b) {
        const D3 gd = rsub(load_d3(L.rest, b), load_d3(L.rest, a));
        cv = mul3f(w.rot32 + a * 9, {(float)gd.x, (float)gd.y, (float)gd.z});
    };
    if (pair) {
        const int end = L.pair_begin[k + 1];
        const bool landmarks = w.L > 0;
        int i = L.pair_begin[k] + lane;
        int after = i + 32 < end ? L.pair_entry[i + 32] : 0;
        PairEntry ahead;
        const int entry = i < end ? L.pair_entry[i] : 0;
        const int ea = arm ? L.edges[edge * 2] : 0, eb = arm ? L.edges[edge * 2 + 1] : 0;
        if (i < end) ahead = load_pair(w, entry, landmarks);
        if (arm) edge_arm(ea, eb);
        for (; i < end; i += 32) {
            const PairEntry x = ahead;
            if (i + 32 < end) ahead = load_pair(w, after, landmarks);
            if (i + 64 < end) after = L.pair_entry[i + 64];
            const float wa = x.a.w, wb = x.b.w;
            const F3 aa = {x.a.x, x.a.y, x.a.z};
            const F3 ab = {x.b.x, x.b.y, x.b.z};
            const float coef = (x.r0.w + x.lm) * wa * wb;  // p2p and landmark share the form
            if (coef > 0.0f) {
                // [ (aa.ab) I - ab aa^T, [aa]x ; [ab]x^T, I ]
                const float dp = dot(aa, ab);
                const float av[3] = {aa.x, aa.y, aa.z}, bv[3] = {ab.x, ab.y, ab.z};
                for (int r = 0; r < 3; ++r)
                    for (int q = 0; q < 3; ++q)
                        blk[r * 6 + q] += coef * ((r == q ? dp : 0.0f) - bv[r] * av[q]);
                blk[0 * 6 + 4] += -coef * aa.z; blk[0 * 6 + 5] += coef * aa.y;
                blk[1 * 6 + 3] += coef * aa.z;  blk[1 * 6 + 5] += -coef * aa.x;
                blk[2 * 6 + 3] += -coef * aa.y; blk[2 * 6 + 4] += coef * aa.x;
                // [ab]x^T = -[ab]x in rows 3-5, columns 0-2
                blk[3 * 6 + 1] += coef * ab.z;  blk[3 * 6 + 2] += -coef * ab.y;
                blk[4 * 6 + 0] += -coef * ab.z; blk[4 * 6 + 2] += coef * ab.x;
                blk[5 * 6 + 0] += coef * ab.y;  blk[5 * 6 + 1] += -coef * ab.x;
                blk[3 * 6 + 3] += coef; blk[4 * 6 + 4] += coef; blk[5 * 6 + 5] += coef;
            }
            if (x.r1.w > 0.0f) {
                const F3 n = {x.r1.x, x.r1.y, x.r1.z};
                const F3 ca = cross(aa, n), cb = cross(ab, n);
                const float ua[6] = {ca.x, ca.y, ca.z, n.x, n.y, n.z};
                const float ub[6] = {cb.x, cb.y, cb.z, n.x, n.y, n.z};
                const float s = x.r1.w * wa * wb;
                for (int r = 0; r < 6; ++r)
                    for (int q = 0; q < 6; ++q) blk[r * 6 + q] += s * ua[r] * ub[q];
            }
        }
    } else if (arm) {
        edge_arm(L.edges[edge * 2], L.edges[edge * 2 + 1]);
    }
    // the 36 sums spread over the lanes (two each at most); each lane stores
    // what it holds, both ways
    int first = 0, count = 36;
    if (pair) warp_sum_halving<36>(blk, lane, first, count);
    else halving_place<36>(lane, first, count);
    float* A = w.offdiag[1 - c.system] + block_base(slot);
    float* T = w.offdiag[1 - c.system] + block_base(mirror);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (i >= count) break;
        const int j = first + i, r = j / 6, q = j - r * 6;
        float value = (c.route == 1 && (r < 3 || q < 3)) ? 0.0f : blk[i];
        if (edge >= 0) {
            float term = 0.0f;
            if (r >= 3) {
                if (r == q) term = -ws;
            } else if (q >= 3 && q - 3 != r) {
                // row r, column q of -[c]x: c's remaining component, its sign
                // alternating around the cycle
                const int other = 3 - r - (q - 3);
                const float x = other == 0 ? cv.x : (other == 1 ? cv.y : cv.z);
                term = (q - 3 == (r + 1) % 3) ? ws * x : -ws * x;
            }
            value = pair ? value + term : term;
        }
        A[block_at(r, q)] = value;
        T[block_at(q, r)] = value;
    }
}

// Blocks of eight warps: the nodes', then the off-diagonal blocks'.
__device__ __forceinline__ void k_assemble_body(const WrapDev& w, int part, int bx) {
    const WrapControl c = *w.control;
    if (!in_part(c, part)) return;
    if (!computes_energy(c)) return;
    const LevelDev& L = w.levels[c.level];
    const int node_blocks = blocks_of_dev((long)L.node_count * 32, kNodeThreads);
    const int warp = threadIdx.x >> 5;
    if (bx < node_blocks) {
        const int node = bx * (kNodeThreads / 32) + warp;
        if (node < L.node_count) assemble_node(w, c, node);
    } else if (assembles(c)) {
        const int k = (bx - node_blocks) * (kNodeThreads / 32) + warp;
        if (k < L.offdiag_count) assemble_block(w, c, k);
    }
}

// Two blocks per SM (127 registers, no spills): three spill (80 registers; a
// batch of 16 wraps 54 against 46 ms of assembly), one leaves too few warps
// (68 ms).
__global__ void __launch_bounds__(kNodeThreads, 2) k_assemble(const WrapDev* __restrict__ wraps, int wrap_count, int part) {
    over_virtual_blocks<false>(
        wraps, wrap_count,
        [&](const WrapDev& w) {
            const WrapControl c = *w.control;
            if (!in_part(c, part) || !computes_energy(c)) return 0;
            const LevelDev& L = w.levels[c.level];
            return blocks_of_dev((long)L.node_count * 32, kNodeThreads) +
                   (assembles(c) ? blocks_of_dev((long)L.offdiag_count * 32, kNodeThreads) : 0);
        },
        [&](int wi, int bx) { k_assemble_body(wraps[wi], part, bx); });
}

// ---------------------------------------------------------------------------
// the decision: the schedule of route_a.cpp:99-190 / session.cu:404-576,
// taken on the device from FP64 energies
// ---------------------------------------------------------------------------
__device__ inline double relative_change(double before, double after) {  // route_shared.h:24-26
    return (before - after) / fmax(fabs(before), 1e-12);
}

constexpr int kDecideThreads = 256;
constexpr int kMaxEdgeSums = 512;  // a multiple of kDecideThreads
__global__ void __launch_bounds__(kDecideThreads) k_decide(const WrapDev* __restrict__ wraps, int part) {
    const WrapDev& w = wraps[blockIdx.x];
    WrapControl* ctl = w.control;
    if (part != 0 && (part == 1) != (ctl->tick_phase == kPhaseSolve)) return;
    const int phase = ctl->phase;
    if (phase == kPhaseDone) return;
    constexpr int kWarps = kDecideThreads / 32;
    __shared__ double scratch[kWarps * kEnergyKinds];
    __shared__ double edge_sums[kMaxEdgeSums];
    __shared__ double parts_s[kEnergyKinds];
    const WrapControl c0 = *ctl;
    if (computes_energy(c0)) {
        const LevelDev& L = w.levels[c0.level];
        const int vb = (w.V + kVertexThreads - 1) / kVertexThreads;
        const int eb = (L.edge_count + kEdgeSums - 1) / kEdgeSums;
        const int nb = (L.node_count + kNodeThreads / 32 - 1) / (kNodeThreads / 32);
        double s[kEnergyKinds] = {0, 0, 0, 0, 0};
        for (int i = threadIdx.x; i < vb; i += blockDim.x) {
            s[0] += w.partials[(long)i * kPartialStride];
            s[1] += w.partials[(long)i * kPartialStride + 1];
            s[4] += w.partials[(long)i * kPartialStride + 2];
        }
        // Each 128 edges' smoothness energy, summed in the order of a block
        // sum over 128 threads: a butterfly within each 32 (zero past the last
        // edge), then ((w0 + w2) + (w1 + w3)).  A warp takes 128 edges at a
        // time with coalesced loads; thread i then adds sum i, i + 256, ...
        // (one thread per 128 edges, summing 128 values of its own, took 6 us).
        const int lane = threadIdx.x & 31;
        for (int base = 0; base < eb; base += kMaxEdgeSums) {
            const int here = min(kMaxEdgeSums, eb - base);
            for (int i = threadIdx.x >> 5; i < here; i += kWarps) {
                double x[4];
                for (int j = 0; j < 4; ++j) {
                    const int e = (base + i) * kEdgeSums + j * 32 + lane;
                    x[j] = e < L.edge_count ? w.edge_partials[e] : 0.0;
                }
                for (int o = 16; o > 0; o >>= 1)
                    for (int j = 0; j < 4; ++j) x[j] += __shfl_xor_sync(0xffffffffu, x[j], o);
                if (lane == 0) edge_sums[i] = (x[0] + x[2]) + (x[1] + x[3]);
            }
            __syncthreads();
            for (int i = threadIdx.x; i < here; i += blockDim.x) s[2] += edge_sums[i];
            __syncthreads();
        }
        for (int i = threadIdx.x; i < nb; i += blockDim.x) {
            // node block i's anchor energy, summed in the order of a block sum
            // over 8 warps (node 8i + j in lane 0 of warp j; the other lanes'
            // zeros change nothing)
            static_assert(kNodeThreads == 8 * 32, "eight nodes per partial sum");
            double v[8];
            for (int j = 0; j < 8; ++j) {
                const int n = i * 8 + j;
                v[j] = n < L.node_count ? w.node_partials[n] : 0.0;
            }
            s[3] += ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
        }
        block_sums<kDecideThreads, kEnergyKinds>(s, scratch);
        if (threadIdx.x == 0)
            for (int k = 0; k < kEnergyKinds; ++k) parts_s[k] = s[k];
    }
    // the long walks this tick's query took from its list are done: clear
    // their flags and empty the list, which the next query but one fills
    const bool queried = c0.tick_phase == kPhaseTransfer || c0.tick_phase == kPhaseRefresh ||
                         c0.tick_phase == kPhaseFinal;
    if (queried) {
        const int cur = c0.long_cur;
        const int taken = min(w.long_count[cur], kLongCap);
        for (int i = threadIdx.x; i < taken; i += blockDim.x)
            w.long_flag[(long)cur * w.V + w.long_list[cur * kLongCap + i]] = 0;
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    WrapControl c = c0;
    c.steps += 1;
    if (queried) {
        w.long_count[c.long_cur] = 0;
        c.long_cur ^= 1;
    }
    const double total = parts_s[0] + parts_s[1] + parts_s[2] + parts_s[3] + parts_s[4];
    LevelRecord& rec = w.records[c.level];
    if (c.phase == kPhaseSolve) {
        rec.solves += 1;
        rec.pcg_iterations += c.pcg_iterations;
    }
    if (refresh_like(c.phase)) rec.queries += 1;
    if (assembles(c)) rec.assemblies += 1;
    bool close_outer = false;
    if (c.phase == kPhaseTransfer || c.phase == kPhaseRefresh) {
        if (c.phase == kPhaseTransfer) c.state = 1 - c.state;
        c.system = 1 - c.system;
        c.energy = total;
        for (int k = 0; k < kEnergyKinds; ++k) c.energy_parts[k] = parts_s[k];
        if (c.outer == 0) rec.energy_start = total;
        c.phase = kPhaseSolve;
        c.inner = 0;
        c.attempt = 0;
    } else if (c.phase == kPhaseSolve) {
        bool end_inner = false;
        if (!c.pcg_ok) {
            c.damping *= w.damping_increase;
            c.attempt += 1;
            end_inner = c.attempt >= w.max_attempts;
        } else {
            c.candidate_energy = total;
            for (int k = 0; k < kEnergyKinds; ++k) c.candidate_parts[k] = parts_s[k];
            if (total < c.energy) {
                c.state = 1 - c.state;
                if (c.route == 0) c.system = 1 - c.system;
                c.damping = fmax(c.damping * w.damping_decrease, 1e-12);
                c.inner += 1;
                rec.inner_iterations += 1;
                const double improvement = relative_change(c.energy, total);
                c.energy = total;
                for (int k = 0; k < kEnergyKinds; ++k) c.energy_parts[k] = parts_s[k];
                c.attempt = 0;
                end_inner = improvement <= w.inner_tol[c.level] || c.inner >= w.max_inner[c.level];
            } else {
                c.damping *= w.damping_increase;
                c.attempt += 1;
                end_inner = c.attempt >= w.max_attempts;
            }
        }
        close_outer = end_inner;
    } else if (c.phase == kPhaseFinal) {
        c.phase = kPhaseDone;
    }
    if (close_outer) {  // route_a.cpp:171-181
        rec.energy_end = c.energy;
        rec.outer_iterations += 1;
        bool converged = false;
        if (c.outer > 0 && relative_change(c.previous_level_energy, c.energy) <= w.outer_tol[c.level]) {
            converged = true;
            rec.converged = 1;
        } else {
            c.previous_level_energy = c.energy;
        }
        c.outer += 1;
        if (converged || c.outer >= w.max_outer[c.level]) {
            c.stats_pending = c.level + 1;
            if (c.level + 1 < c.level_count) {
                c.level += 1;
                c.phase = kPhaseTransfer;
                c.damping = w.initial_damping;
                c.outer = 0;
                c.previous_level_energy = 0.0;
                LevelRecord& next = w.records[c.level];
                next.level = c.level;
                next.nodes = w.levels[c.level].node_count;
            } else {
                c.phase = kPhaseFinal;
            }
        } else {
            c.phase = kPhaseRefresh;
        }
        c.inner = 0;
        c.attempt = 0;
    }
    if (c.error & kErrorSolveWait) c.phase = kPhaseDone;  // the host reports it
    *ctl = c;
}

// ---------------------------------------------------------------------------
// host launch of one tick
// ---------------------------------------------------------------------------
// Grids of the virtual-block kernels: as many blocks as fit on the device
// at once (occupancy of each kernel at its block size, times the SMs).
struct VirtualGrids {
    int prologue, c_fit, c_deform, c_rhs, evaluate, normals, residual, candidate, assemble;
};
const VirtualGrids& virtual_grids() {
    static PerDevice<VirtualGrids>& grids = *new PerDevice<VirtualGrids>;
    const int device = current_device();
    return grids.of(device, [device] {
        int sms = 148;
        check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "device");
        auto fit = [sms](auto kernel, int threads) {
            int per_sm = 0;
            check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, sizeof(int) * 1025),
                  "occupancy");
            return sms * (per_sm > 0 ? per_sm : 1);
        };
        VirtualGrids g;
        g.prologue = fit(k_prologue, 128);
        g.c_fit = fit(k_c_fit, kNodeThreads);
        g.c_deform = fit(k_c_deform, kVertexThreads);
        g.c_rhs = fit(k_c_rhs, kNodeThreads);
        g.evaluate = fit(k_evaluate, kVertexThreads);
        g.normals = fit(k_normals, kVertexThreads);
        g.residual = fit(k_residual<false>, kVertexThreads);
        g.candidate = fit(k_residual<true>, kVertexThreads);
        g.assemble = fit(k_assemble, kNodeThreads);
        return g;
    });
}

void launch_tick(const WrapDev* wraps, const TickShape& s, cudaStream_t stream,
                 KernelTimers* timers) {
    const int W = s.wraps;
    const VirtualGrids& grids = virtual_grids();
    const size_t virtual_smem = sizeof(int) * (W + 1);
    const bool timed = timers && timers->active;
    // statistics of a finished level, and every wrap's phase at the tick's start
    k_stats<<<dim3(1, W), kStatsThreads, 0, stream>>>(wraps, 0);
    // A wrap that starts the tick in a solve runs the solve chain (Horn fit,
    // PCG, candidate evaluation, energy and system, decision); any other runs
    // the refresh chain (warm start, evaluation, normals, closest points,
    // energy and system, decision).  The chains touch different wraps, so
    // with a side stream they run as two parallel branches of the tick.  A
    // timed tick runs them one after the other, so that each kernel group's
    // time is its own.
    const bool split = s.side_stream != nullptr && !timed;
    const int solve_part = split ? 1 : 0, refresh_part = split ? 2 : 0;
    cudaStream_t refresh = split ? s.side_stream : stream;
    // evaluate: the solve chain's kernel deforms the candidate's vertices too
    // (a timed tick's refresh chain has done it, for either kind of wrap)
    auto assemble_and_decide = [&](int part, bool evaluate, cudaStream_t on) {
        if (timed) cudaEventRecord(timers->assemble_begin, on);
        if (evaluate) {
            k_residual<true><<<grids.candidate, kVertexThreads, virtual_smem, on>>>(wraps, W, part);
        } else {
            k_residual<false><<<grids.residual, kVertexThreads, virtual_smem, on>>>(wraps, W, part);
        }
        k_assemble<<<grids.assemble, kNodeThreads, virtual_smem, on>>>(wraps, W, part);
        if (timed) cudaEventRecord(timers->assemble_end, on);
        k_decide<<<W, kDecideThreads, 0, on>>>(wraps, part);
    };
    if (split) {
        cudaEventRecord(s.side_fork, stream);
        cudaStreamWaitEvent(refresh, s.side_fork, 0);
    }

    // ---- the solve chain ----
    if (s.route_c) {
        k_c_fit<<<grids.c_fit, kNodeThreads, virtual_smem, stream>>>(wraps, W, solve_part);
        k_c_deform<<<grids.c_deform, kVertexThreads, virtual_smem, stream>>>(wraps, W, solve_part);
        k_c_rhs<<<grids.c_rhs, kNodeThreads, virtual_smem, stream>>>(wraps, W, solve_part);
    }
    if (timed) cudaEventRecord(timers->pcg_begin, stream);
    auto launch_pcg = [&](int cluster, int count, const int* index, cudaStream_t on) {
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(cluster, count);
        config.blockDim = dim3(kPcgThreads);
        config.dynamicSmemBytes = kPcgMaxSmemBytes;
        config.stream = on;
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeClusterDimension;
        attribute[0].val.clusterDim.x = cluster;
        attribute[0].val.clusterDim.y = 1;
        attribute[0].val.clusterDim.z = 1;
        config.attrs = attribute;
        config.numAttrs = 1;
        cudaLaunchKernelEx(&config, k_pcg, wraps, index, kPcgMaxSmemFloats, W, s.grid_nodes,
                           s.wait_tries);
    };
    if (s.grid_nodes > 0) {
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(s.grid_ctas);
        config.blockDim = dim3(kPcgThreads);
        config.dynamicSmemBytes = kPcgMaxSmemBytes;
        config.stream = stream;
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeCooperative;
        attribute[0].val.cooperative = 1;
        config.attrs = attribute;
        config.numAttrs = 1;
        cudaLaunchKernelEx(&config, k_pcg_grid, wraps, W, s.grid_nodes, kPcgMaxSmemFloats,
                           s.wait_tries);
    }
    if (s.pcg_groups <= 0) {
        launch_pcg(s.pcg_cluster, W, nullptr, stream);
    } else {
        // fork: every class launch after everything before it on `stream`
        cudaEventRecord(s.pcg_fork, stream);
        for (int g = 1; g < s.pcg_groups; ++g) {
            cudaStreamWaitEvent(s.pcg_streams[g], s.pcg_fork, 0);
            launch_pcg(s.pcg_group_cluster[g], s.pcg_group_count[g], s.pcg_group_index[g], s.pcg_streams[g]);
            cudaEventRecord(s.pcg_join[g], s.pcg_streams[g]);
        }
        launch_pcg(s.pcg_group_cluster[0], s.pcg_group_count[0], s.pcg_group_index[0], stream);
        for (int g = 1; g < s.pcg_groups; ++g) cudaStreamWaitEvent(stream, s.pcg_join[g], 0);
    }
    if (timed) cudaEventRecord(timers->pcg_end, stream);
    if (split) assemble_and_decide(solve_part, true, stream);

    // ---- the refresh chain ----
    k_prologue<<<grids.prologue, 128, virtual_smem, refresh>>>(wraps, W, refresh_part);
    k_evaluate<<<grids.evaluate, kVertexThreads, virtual_smem, refresh>>>(wraps, W, refresh_part);
    k_normals<<<grids.normals, kVertexThreads, virtual_smem, refresh>>>(wraps, W, refresh_part);
    if (timed) cudaEventRecord(timers->query_begin, refresh);
    launch_query(wraps, W, refresh, s.query_counter);
    if (timed) cudaEventRecord(timers->query_end, refresh);
    k_stats<<<dim3(1, W), kStatsThreads, 0, refresh>>>(wraps, 1);
    assemble_and_decide(refresh_part, false, refresh);
    if (split) {
        cudaEventRecord(s.side_join, refresh);
        cudaStreamWaitEvent(stream, s.side_join, 0);
    }
}

int tick_kernel_launches(const TickShape& s, bool timed) {
    // stats twice, [fit, deform, rhs,] solve launches, prologue, evaluate, normals,
    // query, residual, assembly, decision; an untimed tick with a side stream
    // runs the last three in each branch
    return 9 + (s.route_c ? 3 : 0) + (s.grid_nodes > 0 ? 1 : 0) + (s.pcg_groups > 0 ? s.pcg_groups : 1) + (s.side_stream && !timed ? 3 : 0);
}

// Cluster size of the solve for a wrap of `nodes` nodes in a class: a power of
// two with about 128 nodes (an octet per warp) per CTA, at most 16 CTAs (the
// non-portable maximum, enabled here), halved `shift` times; shift -1: about 64
// nodes.  An iteration's shared-memory reads fall with the rows per CTA: us per
// iteration with 64 / 128 nodes a CTA: 200 nodes 4.40 / 5.51, 544 nodes 4.97 /
// 5.48; with 32 nodes a CTA 200 nodes take 4.15, the whole step no less.
int pcg_class_cluster(int nodes, int shift) {
    const int per_cta = shift < 0 ? 64 : 128;
    int ranks = 1;
    while (ranks < 16 && ranks * per_cta < nodes) ranks *= 2;
    return std::max(1, shift > 0 ? ranks >> shift : ranks);
}

void pcg_enable() {
    static PerDevice<bool>& enabled = *new PerDevice<bool>;
    enabled.of(current_device(), [] {
        check(cudaFuncSetAttribute(k_pcg, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "solve attributes");
        check(cudaFuncSetAttribute(k_pcg, cudaFuncAttributeMaxDynamicSharedMemorySize, kPcgMaxSmemBytes),
              "solve attributes");
        check(cudaFuncSetAttribute(k_pcg_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, kPcgMaxSmemBytes),
              "solve attributes");
        return true;
    });
}

// One over the clusters that run at once: a cluster's CTAs sit in one group of
// SMs, so that, say, twelve clusters of sixteen do not fit on 148 SMs.
double pcg_cluster_share(int cluster) {
    struct Shares {
        double of[5];
    };
    static PerDevice<Shares>& of_device = *new PerDevice<Shares>;
    const Shares& shares = of_device.of(current_device(), [] {
        pcg_enable();
        Shares s{};
        for (int i = 0; i < 5; ++i) {
            cudaLaunchConfig_t config = {};
            config.gridDim = dim3(1 << i);
            config.blockDim = dim3(kPcgThreads);
            config.dynamicSmemBytes = kPcgMaxSmemBytes;
            cudaLaunchAttribute attribute[1];
            attribute[0].id = cudaLaunchAttributeClusterDimension;
            attribute[0].val.clusterDim.x = 1 << i;
            attribute[0].val.clusterDim.y = 1;
            attribute[0].val.clusterDim.z = 1;
            config.attrs = attribute;
            config.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, k_pcg, &config) != cudaSuccess) {
                cudaGetLastError();  // not a size for this device: it takes all of it
                clusters = 0;
            }
            s.of[i] = 1.0 / std::max(1, clusters);
        }
        return s;
    });
    int i = 0;
    while (i < 4 && (1 << i) < cluster) ++i;
    return shares.of[i];
}

// Graphs above this many nodes (per wrap the grid takes) are solved by the
// whole device.  An iteration of a 16-CTA cluster grows with the rows per CTA,
// the grid's is mostly its two meetings: 6.9 against 9.9 us at 1,000 nodes with
// 6 bindings, 10.2 against 10.3 at 2,000; with 8 bindings 8.7 against 10.8 at
// 1,250, 16 against 12.5 at 2,500, 34 against 14 at 5,000, 73 against 18 at
// 10,000.
constexpr int kGridNodes = 2000;
// Wraps a tick may hold with the grid solve among its launches: it is of use to
// few large wraps only, and a launch without work costs each tick 3 us.  A
// batch's step with / without it, ms (6 bindings): 2,500 + 200 nodes 40.5 /
// 42.8; 5,000 + 1,000 68.3 / 93.1; 2,500 + 3 of 800 46.3 / 47.1; 5,000 + 3 of
// 1,500 86.5 / 102.3; 2,500 + 7 of 500 48.6 / 48.8; 5,000 + 7 of 1,200 90.2 /
// 111.0; 2 of 5,000 + 6 of 500 104.0 / 110.9; and where it is of least use, 4 of
// 4,000 107.8 / 109.4, 3 of 5,000 121.7 / 120.9, 8 of 2,100 124.3 / 122.2.  A
// server's two lanes, a request of 2,500 nodes in one and five small ones in the
// other, 99 / 98; of 5,000 nodes 167 / 192.
constexpr int kGridWraps = 8;
void grid_solve_shape(TickShape& shape) {
    shape.grid_nodes = shape.max_nodes > kGridNodes && shape.wraps <= kGridWraps ? kGridNodes : 0;
    shape.grid_ctas = 0;
    if (!shape.grid_nodes) return;
    pcg_enable();
    const int device = current_device();
    int sms = 0, cooperative = 0, per_sm = 0;
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "device");
    check(cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device), "device");
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pcg_grid, kPcgThreads, kPcgMaxSmemBytes),
          "occupancy");
    if (!cooperative || per_sm < 1 || !pcg_grid_fits(shape.max_nodes, sms)) {
        shape.grid_nodes = 0;
        return;
    }
    shape.grid_ctas = sms;
}

int pcg_max_nodes() { return 32768; }

// A wrap's template vertices under a state, in the caller's units
// (mesh.cpp:189-193): the operations of the host's evaluation, each rounded on
// its own, so the bits are the host's.  (The host took 2 ms for 25,000 vertices
// on one core, and as long again at every step a session redraws.)
__global__ void __launch_bounds__(kVertexThreads) k_caller_vertices(const WrapDev* __restrict__ wrap, int level,
                                                                    int buffer, double cx, double cy, double cz,
                                                                    double scale, double* __restrict__ out) {
    const WrapDev& w = *wrap;
    const int v = blockIdx.x * kVertexThreads + threadIdx.x;
    if (v >= w.V) return;
    const LevelDev& L = w.levels[level];
    const double* R = w.rot[buffer];
    const double* T = w.trans[buffer];
    const D3 p = load_d3(w.tpl, v);
    D3 sum = {0.0, 0.0, 0.0};
    const int count = L.bind_counts[v];
    for (int s = 0; s < count; ++s) {
        const int j = L.bind_nodes[v * kMaxSlots + s];
        const D3 g = load_d3(L.rest, j);
        const D3 applied = radd(radd(rmat(R + j * 9, rsub(p, g)), g), load_d3(T, j));
        sum = radd(sum, rmul(applied, L.bind_weights[v * kMaxSlots + s]));
    }
    store_d3(out, v, {da(__ddiv_rn(sum.x, scale), cx), da(__ddiv_rn(sum.y, scale), cy), da(__ddiv_rn(sum.z, scale), cz)});
}

void launch_caller_vertices(const WrapDev* wrap, int vertices, int level, int buffer, const double center[3],
                            double scale, double* out, cudaStream_t stream) {
    k_caller_vertices<<<(vertices + kVertexThreads - 1) / kVertexThreads, kVertexThreads, 0, stream>>>(
        wrap, level, buffer, center[0], center[1], center[2], scale, out);
}

void launch_fit_rigid(const double* src, const double* dst, const double* weights, int n, double* out,
                      cudaStream_t stream) {
    k_fit_rigid<<<1, kRigidThreads, 0, stream>>>(src, dst, weights, n, out);
}

}  // namespace nricp_b200
